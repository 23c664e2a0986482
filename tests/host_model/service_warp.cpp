// The service warp of a fused pair (pair_serve, pair_ready of csrc/lbm_pair.cuh,
// as written there) run by 32 host threads that keep vector clocks by the rules
// of the PTX memory model: an acquire load orders what follows it in its own
// lane only, a vote orders nothing, __syncwarp orders the lanes, an arrival
// publishes what is ordered before the arriving lane. The even step of every
// group that the odd item depends on has to be ordered before the `go` barrier
// that the compute warps wait for.
#include <cuda_runtime.h>

#include <array>
#include <atomic>
#include <barrier>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

#include "../../lbm-benchmark-kernels_b200/csrc/lbm_kernels.cuh"

namespace model {

constexpr int kLanes = 32, kGroups = 40;
using Clock = std::array<int, kLanes + kGroups>;  // lanes, then the writers of the even groups
void join(Clock& a, const Clock& b) {
  for (size_t k = 0; k < a.size(); ++k) a[k] = std::max(a[k], b[k]);
}

std::mutex lock;
std::map<const void*, Clock> published;  // by release operations, per location
std::array<Clock, kLanes> clocks;
std::barrier<> meet(kLanes);
std::array<int, kLanes> ballot;
int polls, readyAfter;
const uint32_t* counters;
uint32_t done;  // tiles done per group from poll readyAfter on

struct Index {
  unsigned x;
};
thread_local Index thread;
int lane() { return (int)thread.x - lbm::kListTile; }

void syncwarp() {
  meet.arrive_and_wait();
  {
    std::lock_guard<std::mutex> hold(lock);
    for (const Clock& c : clocks) join(clocks[lane()], c);
  }
  meet.arrive_and_wait();
}
bool vote(bool v, bool all) {
  ballot[lane()] = v;
  meet.arrive_and_wait();
  int n = 0;
  for (int b : ballot) n += b;
  meet.arrive_and_wait();
  return all ? n == kLanes : n > 0;
}

}  // namespace model

namespace lbm {

using std::min;
constexpr uint32_t kPairSpinLimit = 1u << 20;
uint32_t ld_acquire(const uint32_t* p) {
  std::lock_guard<std::mutex> hold(model::lock);
  if (++model::polls <= model::readyAfter) return 0;
  model::join(model::clocks[model::lane()], model::published[p]);
  return model::done;
}
uint32_t ld_relaxed(const uint32_t* p) { return *p; }
void red_release(uint32_t*, uint32_t) {}
void mbar_arrive(uint64_t* bar) {
  std::lock_guard<std::mutex> hold(model::lock);
  model::join(model::published[bar], model::clocks[model::lane()]);
}
void mbar_expect_tx(uint64_t*, uint32_t) {}
bool mbar_wait_bounded(uint64_t*, uint32_t) { return true; }
void bulk_g2s(void*, const void*, uint32_t, uint64_t*) {}
void bulk_prefetch_l2(const void*, uint32_t) {}
void chain_wait() {}
template <class T>
T __ldg(const T* p) { return *p; }
uint32_t atomicInc(uint32_t*, uint32_t) { return 0; }
uint32_t atomicAdd(uint32_t*, uint32_t) { return 0; }
int atomicOr(int* p, int v) { std::lock_guard<std::mutex> hold(model::lock); return *p |= v; }

#define threadIdx model::thread
#define __syncwarp model::syncwarp
#define __all_sync(mask, v) model::vote(v, true)
#define __any_sync(mask, v) model::vote(v, false)
#define asm
#define volatile(...)
#include "extracted.inc"  // PairShared, pair_ready, pair_serve
#undef volatile
#undef asm

}  // namespace lbm

int main(int argc, char** argv) {
  // groups of 2 tiles; the odd item depends on `a` + `b` + `c` of them
  const int ranges[3] = {argc > 1 ? atoi(argv[1]) : 1, argc > 2 ? atoi(argv[2]) : 1, argc > 3 ? atoi(argv[3]) : 1};
  model::readyAfter = argc > 4 ? atoi(argv[4]) : 0;
  model::done = 2;
  std::vector<uint32_t> count(model::kGroups + 2, 0);
  std::vector<lbm::PairItem> items(200);
  lbm::PairItem& it = items[100];
  it.tile = 3;
  uint32_t lo = 0;
  for (int r = 0; r < 3; ++r) {
    it.lo[r] = lo;
    it.n[r] = ranges[r];
    lo += ranges[r];
  }
  for (int g = 0; g < model::kGroups; ++g) {
    model::Clock c{};
    c[model::kLanes + g] = 1;  // the even step of the group's tiles
    model::published[&count[g]] = c;
  }
  for (auto& c : model::clocks) c.fill(0);
  lbm::PairArgs<3> p{};
  p.items = items.data();
  p.count = count.data();
  p.launches = count.data() + model::kGroups;
  p.nItems = 200;
  p.nTiles = 2 * model::kGroups;
  p.shift = 1;
  static lbm::PairShared<3, 4> sh;
  int err = 0;
  std::vector<std::thread> lanes;
  for (int l = 0; l < model::kLanes; ++l)
    lanes.emplace_back([&, l] {
      model::thread.x = lbm::kListTile + l;
      lbm::pair_serve(&sh, p, [](const lbm::PairItem&) -> const void* { return nullptr; }, &err, 100u);
    });
  for (auto& t : lanes) t.join();
  int bad = err != 0;
  for (uint32_t g = 0; g < lo; ++g)
    if (model::published[&sh.go][model::kLanes + g] != 1) {
      std::printf("group %u is not ordered before the odd step\n", g);
      bad = 1;
    }
  return bad;
}
