"""The split-K autotuner measures 24 x 24 and 128 x 128 outputs, one CTA of 128 x 128 both
but different tiles of the kernel, each for itself, also where a table of an earlier build
gives both one split; the products agree with numpy (1e-13 relative to sum |a||b|, as in
tests/test_gpu_gemm.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("old_table", [False, True])
def test_each_output_has_its_own_class(uw12lib, cuda_device, tmp_path, old_table):
    import torch
    L = uw12lib
    rng = np.random.default_rng(3)
    k = 6000  # 375 k tiles, bucket 8
    path = tmp_path / "old.txt"
    path.write_text("1 8 5 0.1\n")
    L.autotune_clear()
    try:
        L.autotune(L.AUTOTUNE_TUNE, str(path) if old_table else None)
        for n, m in enumerate((24, 128), start=1):
            A, B = rng.standard_normal((m, k)), rng.standard_normal((k, m))
            dA = torch.from_numpy(np.asfortranarray(A).reshape(-1, order="F")).cuda()
            dB = torch.from_numpy(np.asfortranarray(B).reshape(-1, order="F")).cuda()
            dC = torch.full((m * m,), np.nan, dtype=torch.float64, device="cuda")
            L.dgemm(m, m, k, 1.0, dA.data_ptr(), m, False, dB.data_ptr(), k, False, 0.0,
                    dC.data_ptr(), m)
            torch.cuda.synchronize()
            assert L.autotune_size() == n + old_table
            C = dC.cpu().numpy().reshape((m, m), order="F")
            assert np.all(np.abs(C - A @ B) <= 1e-13 * (np.abs(A) @ np.abs(B)))
    finally:
        L.autotune_clear()
        L.autotune(L.AUTOTUNE_OFF)
