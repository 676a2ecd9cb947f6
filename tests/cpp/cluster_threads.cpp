// The cluster solver's team (cluster_team.cuh) on host threads, with waits that
// are made to run out.  argv: the CTA whose wait runs out and the reductions in
// which it does (none: an undisturbed run).  The body has the solver's order of
// barriers and reductions and branches on what the reductions return, so that a
// CTA with a wrong sum takes another branch than the others.  Checked: no CTA
// posts into the shared memory of one that has left, all leave behind the same
// barrier and agree why, and an undisturbed run has the right sums.
#include <set>

#include "cuda_threads.hpp"

namespace host {
constexpr unsigned kCtas = 3, kArena = 1u << 16;  // "addresses": a CTA's rank times kArena, plus the place in its memory
alignas(16) unsigned char arena[kCtas][kArena];
int gone[kCtas], posted_to_gone = 0;
int blind_cta = -1;
std::set<unsigned> blind;  // tags that blind_cta never sees
pthread_barrier_t cluster;
inline void store_check(uint32_t a) {
  if (__atomic_load_n(&gone[a / kArena], __ATOMIC_SEQ_CST)) __atomic_store_n(&posted_to_gone, 1, __ATOMIC_RELAXED);
}
}  // namespace host

namespace cup2d {
inline uint32_t smem_u32(const void* p) { return (uint32_t)((const unsigned char*)p - &host::arena[0][0]); }
inline uint32_t cluster_addr(uint32_t local, unsigned rank) { return local % host::kArena + rank * host::kArena; }
inline unsigned long long* words(uint32_t a) { return reinterpret_cast<unsigned long long*>(&host::arena[0][0] + a); }
inline void st_cluster_words(uint32_t a, unsigned long long x, unsigned long long y) {
  host::store_check(a);
  __atomic_store_n(words(a), x, __ATOMIC_RELAXED);
  __atomic_store_n(words(a) + 1, y, __ATOMIC_RELAXED);
}
inline ulonglong2 ld_words(uint32_t a) {
  ulonglong2 v{__atomic_load_n(words(a), __ATOMIC_RELAXED), __atomic_load_n(words(a) + 1, __ATOMIC_RELAXED)};
  const unsigned cta = a / host::kArena;
  if ((int)cta == host::blind_cta && host::blind.count((unsigned)(v.x >> 32))) v.x = v.y = 0ull;
  sched_yield();
  return v;
}
inline void st_cluster_u32(uint32_t a, unsigned v) {
  host::store_check(a);
  __atomic_store_n(reinterpret_cast<unsigned*>(words(a)), v, __ATOMIC_RELAXED);
}
inline unsigned ld_cta_u32(uint32_t a) { return __atomic_load_n(reinterpret_cast<unsigned*>(words(a)), __ATOMIC_RELAXED); }
inline void cluster_barrier() { pthread_barrier_wait(&host::cluster); }
}  // namespace cup2d

#include "cluster.inc"

using namespace cup2d;

int main(int argc, char** argv) {
  if (argc > 1) host::blind_cta = std::atoi(argv[1]);
  for (int i = 2; i < argc; ++i) host::blind.insert((unsigned)std::atoi(argv[i]));
  constexpr unsigned kCtas = host::kCtas;
  pthread_barrier_init(&host::cluster, nullptr, kCtas * kClThreads);
  static unsigned barriers[kCtas], wrong = 0;
  static int left[kCtas];
  host::launch(kCtas, kClThreads, [&] {
    const unsigned rank = blockIdx.x;
    ClusterPosts& S = *reinterpret_cast<ClusterPosts*>(host::arena[rank]);
    ClusterTeam team{S, rank, kCtas, 0u, 0u};
    S.clear();
    const double n = (double)kCtas * kClThreads, id = rank * (double)kClThreads + threadIdx.x;
    bool ok = team.sync(), lost = false, refreshed = false;
    const auto sum = [&](double per) {  // of `per` over the threads, and the largest id
      const double v[2] = {per, id};
      double o[2];
      team.reduce(v, 0x2u, o);
      ok = ok && o[1] == n - 1.0;
      return o[0];
    };
    double s = sum(1.0);               // the mean of b
    s += sum(1.0);                     // the residual
    int k = 0;
    for (; s == 2.0 * n && k < 6; ++k) {
      if ((lost = !team.sync())) break;  // behind pass A
      sum(2.0);                          // pass B
      if ((lost = !team.sync())) break;  // behind pass C
      const double d = sum(0.5);         // pass D
      const double e = sum(d == 0.5 * n ? 1.0 : 2.0);  // pass E
      if (e != n) break;                 // "not a number", or the deadline
      if (k == 2 || e < n) {             // a true residual
        if ((lost = !team.sync())) break;
        const double r = sum(3.0);
        refreshed = true;
        if (r != 3.0 * n) break;         // "converged"
      }
    }
    if (!lost) lost = !team.sync();
    if (!lost) {
      ok = ok && sum(4.0) == 4.0 * n && refreshed && k == 6;
      lost = !team.sync();
    }
    __syncthreads();
    if (host::blind_cta < 0 && (!ok || lost)) __atomic_store_n(&wrong, 1u, __ATOMIC_RELAXED);
    if (threadIdx.x == 0) {
      barriers[rank] = team.barriers;
      left[rank] = lost ? 1 : 0;
      __atomic_store_n(&host::gone[rank], 1, __ATOMIC_SEQ_CST);
    }
  });
  bool same = true;
  for (unsigned r = 1; r < kCtas; ++r) same = same && barriers[r] == barriers[0] && left[r] == left[0];
  const bool expect = host::blind_cta >= 0;
  std::printf("left behind barrier %u, lost %d\n", barriers[0], left[0]);
  return host::posted_to_gone || wrong || !same || (left[0] != 0) != expect;
}
