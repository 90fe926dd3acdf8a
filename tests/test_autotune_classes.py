"""The split-K autotuner's classes tell apart outputs that one 128 x 128 CTA covers but that
run in different tiles (no GPU needed): 24 x 24 (1 x 3 blocks of 32 x 8, bucket 1), 128 x 8
(4 blocks, bucket 2) and 128 x 128 (64 blocks, bucket 6), k = 1000 (63 k tiles, bucket 5).  A
line without the last bucket stands for those that have no line of their own."""
import pytest

import libuw12_b200 as L


@pytest.fixture(autouse=True)
def clean_table():
    L.autotune_clear()
    L.autotune(L.AUTOTUNE_OFF)
    yield
    L.autotune_clear()
    L.autotune(L.AUTOTUNE_OFF)


def test_outputs_of_one_cta_are_told_apart(tmp_path):
    src = tmp_path / "table.txt"
    src.write_text("# header\n1 5 8 0.1 1\n1 5 2 0.2 6\n1 5 3 0.3\n")
    L.autotune(L.AUTOTUNE_USE, str(src))
    out = tmp_path / "saved.txt"
    L.autotune_save(str(out))
    for path in (src, out):
        L.autotune_clear()
        L.autotune(L.AUTOTUNE_USE, str(path))
        assert L.autotune_size() == 3
        assert L.autotune_lookup(24, 24, 1000) == 8
        assert L.autotune_lookup(128, 128, 1000) == 2
        assert L.autotune_lookup(128, 8, 1000) == 3
        assert L.autotune_lookup(128, 128, 2000) == 0


@pytest.mark.parametrize("bucket", ["-2", "63"])
def test_block_bucket_out_of_range(tmp_path, bucket):
    bad = tmp_path / "bad.txt"
    bad.write_text(f"1 5 8 0.1 {bucket}\n")
    with pytest.raises(L.UW12CudaError, match="malformed line 1"):
        L.autotune(L.AUTOTUNE_USE, str(bad))
