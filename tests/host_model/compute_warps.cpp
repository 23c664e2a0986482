// One compute thread of k_list_two_fp64 (csrc/lbm_kernels_fp64.cu, as written
// there), with waits that arrive or run out: a thread follows a run record only
// after the wait for it has succeeded, and ends only after the previous launch.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../lbm-benchmark-kernels_b200/csrc/lbm_kernels.cuh"

namespace lbm {

constexpr int kPairThreads = kListTile + 32;
template <int R, int kWords>
struct PairShared {
  PairRec<R> item{};
  uint64_t named = 0, go = 0, even = 0;
};
struct Index {
  unsigned x;
} threadIdx{5}, blockIdx{1};
uint32_t records[2 * 64];
bool namedArrives, goArrives;
bool chained;
std::vector<const uint32_t*> followed;
uint64_t* g_go;

bool mbar_wait_bounded(uint64_t* bar, uint32_t) { return bar == g_go ? goArrives : namedArrives; }
void mbar_arrive(uint64_t*) {}
int atomicOr(int* p, int v) { return *p |= v; }
void __syncwarp() {}
void chain_wait() { chained = true; }
template <class Sh>
void pair_init(Sh* sh) {
  sh->item.tile = 2;
  g_go = &sh->go;
}
template <class... A>
void pair_service(A...) {}
const uint32_t* run_row(const uint32_t* run, int, uint32_t& off) {
  followed.push_back(run);
  off = 0;
  return run;
}
template <bool kPush, bool kLast>
void two_grid_node(const ListArgs&, const Trt<double>&, const double*, double*, int, const uint32_t*, uint32_t) {}

#define __launch_bounds__(...)
#define __shared__
#include "extracted.inc"  // pair_even_done, the waits, k_list_two_fp64

}  // namespace lbm

int main(int argc, char** argv) {
  using namespace lbm;
  const bool push = atoi(argv[1]);
  namedArrives = atoi(argv[2]);
  goArrives = atoi(argv[3]);
  int err = 0;
  ListArgs a{};
  a.nFluid = 4 * kListTile;
  a.err = &err;
  PairArgs<3> p{};
  p.nTiles = 4;
  if (push)
    k_list_two_fp64<true>(a, p, Trt<double>{}, 64);
  else
    k_list_two_fp64<false>(a, p, Trt<double>{}, 64);
  std::vector<const uint32_t*> want;
  if (namedArrives) want.push_back(records);
  if (namedArrives && goArrives) want.push_back(records + 64);
  const bool ok = followed == want && chained && (err != 0) == !(namedArrives && goArrives);
  if (!ok) std::printf("%zu records followed (%zu arrived), error word %d\n", followed.size(), want.size(), err);
  return !ok;
}
