// The grid solvers' team (common.cuh: Team) on host threads: reductions and
// barriers in a row, every thread checking every result.  Built with
// ThreadSanitizer, which reports any access to a shared variable that no
// barrier orders.  exit 0: all results right and nothing reported.
#include "cuda_threads.hpp"

#include "team.inc"

using namespace cup2d;

int main() {
  constexpr unsigned kCtas = 2;
  static Team teams[kCtas];
  static double slots[kRedWords * kCtas];
  static unsigned counter = 0;
  static int abort_flag = 0, wrong = 0;
  host::launch(kCtas, kSolveThreads, [&] {
    Team& B = teams[blockIdx.x];
    if (threadIdx.x == 0) B.init(blockIdx.x, kCtas, &counter, slots, &abort_flag, 300000000000ull, nullptr);
    __syncthreads();
    const unsigned id = blockIdx.x * kSolveThreads + threadIdx.x, n = kCtas * kSolveThreads;
    const double sum = 0.5 * n * (n - 1);
    bool ok = true;
    for (int k = 0; k < 3; ++k) {
      const double one[1] = {(double)id + k};
      ok = B.reduce<1>(one, 0u, 0) && B.out[0] == sum + (double)n * k && ok;
      ok = B.sync(0) && ok;
      const double four[4] = {(double)id, 1.0, 2.0 * id, (double)k};
      ok = B.reduce<4>(four, 0x1u, 0) && B.out[0] == n - 1 && B.out[1] == n && B.out[2] == 2.0 * sum &&
           B.out[3] == (double)n * k && ok;
      const double six[6] = {(double)id, (double)id, 1.0, 1.0, 1.0, (double)(id + k)};
      ok = B.reduce<6>(six, 0x23u, 0) && B.out[0] == n - 1 && B.out[4] == n && B.out[5] == n - 1 + k && ok;
    }
    if (!ok) __atomic_store_n(&wrong, 1, __ATOMIC_RELAXED);
  });
  if (wrong || abort_flag) {
    std::printf("wrong result\n");
    return 1;
  }
  return 0;
}
