// Orbital pairs and their shards (csrc/kernels.cuh).  With arguments a c n: the first
// orbital of every shard and the last one's end.  Without: checks over all small cases.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "kernels.cuh"

using namespace uw12b;

int main(int argc, char** argv) {
  if (argc == 4) {
    const size_t a = std::atoi(argv[1]), c = std::atoi(argv[2]), n = std::atoi(argv[3]);
    for (size_t i = 0; i <= n; ++i) std::printf("%zu\n", pair_bound(a, c, i, n));
    return 0;
  }
  for (size_t a = 1; a <= 40; ++a)
    for (size_t c = 0; c <= 6; ++c)
      for (size_t n = 1; n <= 16; ++n) {
        const size_t o = c + a;
        const double even = double(pair_count(a, c, o)) / double(n);
        if (pair_bound(a, c, 0, n) != 0 || pair_bound(a, c, n, n) != o) return 1;
        for (size_t i = 0; i < n; ++i) {
          const size_t lo = pair_bound(a, c, i, n), hi = pair_bound(a, c, i + 1, n);
          if (hi < lo) return 2;
          // each end is within half an orbital's pairs of its even place
          const double has = double(pair_count(a, c, hi) - pair_count(a, c, lo));
          if (has > even + double(a) || has < even - double(a)) return 3;
          // columns of a range of the distinct-pair order: one per pair, mirror images shared
          const PairColumns q = PairColumns::of((long long)a, (long long)c, (long long)lo,
                                                (long long)(hi - lo));
          std::set<long long> seen;
          for (size_t k = lo; k < hi; ++k)
            for (size_t j = 0; j < a; ++j) seen.insert(q.column((long long)j, (long long)k));
          if ((long long)seen.size() != q.count()) return 4;
          if (!seen.empty() && (*seen.begin() != 0 || *seen.rbegin() != q.count() - 1)) return 5;
        }
      }
  std::puts("ok");
  return 0;
}
