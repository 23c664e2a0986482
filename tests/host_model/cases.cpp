// Cases of the host layer on the model of fake_runtime.hpp: `cases NAME` runs
// one and returns 0 if everything held. The step launchers are stand-ins that
// look, when their stream runs, at what the kernels would read.
#include "fake_runtime.hpp"

#include <string>

#include "../../include/lbm_b200.h"
#include "../../lbm-benchmark-kernels_b200/csrc/lbm_batch.cuh"
#include "../../lbm-benchmark-kernels_b200/csrc/lbm_kernels.cuh"
#include "../../lbm-benchmark-kernels_b200/csrc/lbm_mem.cuh"

namespace {

int g_bad = 0;
int g_steps = 0;             // launches of one step of batches that have run
double g_pairMs = 1.5;       // what a fused launch takes; a step of its own: 1
int g_pairs = 0;             // fused launches of batches that have run
bool g_waitRunsOut = false;  // the next steps set the error word
void check(bool ok, const char* what) {
  if (ok) return;
  std::printf("not so: %s\n", what);
  ++g_bad;
}

// The interior work items of the AA odd step that aa_interior_items gives out.
std::vector<int> odd_items() { return {0, 3, ~0, 5, ~1}; }
std::vector<int> odd_cells() {
  std::vector<int> c(256);
  for (int k = 0; k < 256; ++k) c[k] = 7 * k + 1;
  return c;
}

struct Lattice {
  LatticeDesc ld{};
  std::vector<int> mask;
  Lattice(int nx, int ny, int nz) : mask((size_t)nx * ny * nz, LAT_CELL_FLUID) {
    ld.Dims[0] = nx;
    ld.Dims[1] = ny;
    ld.Dims[2] = nz;
    ld.Lattice = mask.data();
    ld.nCells = ld.nFluid = nx * ny * nz;
    ld.PeriodicX = ld.PeriodicY = ld.PeriodicZ = 1;
    ld.Name = "fluid";
  }
};

KernelData* full_array(Lattice& lat) {
  Parameters p{};
  KernelData* kd = nullptr;
  D3Q19CudaAaInit_AaSoA(&lat.ld, &kd, &p);
  return kd;
}

CaseData a_case() {
  CaseData cd{};
  cd.Omega = 1.2;
  cd.MaxIterations = 2;
  return cd;
}

}  // namespace

namespace lbm {

long long aa_interior_block_count(const AaArgs&) { return 8; }
bool aa_shell_needed(const AaArgs&) { return false; }
void aa_interior_items(const AaArgs&, const uint32_t*, std::vector<int>& items, std::vector<int>& cells) {
  items = odd_items();
  cells = odd_cells();
}
AaPairGeom aa_pair_geom(const AaArgs& a) {
  AaPairGeom g{};
  g.tpp = 1;
  g.nX = (uint32_t)a.nX;
  return g;
}
int aa_resident_tiles() { return 0; }
int aa_pair_resident() { return 4; }
void aa_pair_schedule(const AaArgs&, const AaPairGeom& g, int, std::vector<AaPairItem>& items) {
  items.assign(g.nX + 2, AaPairItem{});
  for (size_t k = 0; k < items.size(); ++k) items[k].tile = (uint32_t)k;
}
void aa_pair_fp64(const AaArgs& a, const AaPairArgs& q, const Trt<double>&, cudaStream_t s) {
  fake::launch(s, [=] {
    for (uint32_t k = 0; k < q.p.nItems; ++k) check(q.p.items[k].tile == k, "the fused pair reads its items");
    check(*q.p.count == 0, "the counters start at zero");
    a.f[0] += 1.0;
  });
}
void aa_even_fp64(const AaArgs& a, const Trt<double>&, cudaStream_t s) {
  fake::launch(s, [=] { a.f[0] += 1.0; });
}
void aa_odd_interior_fp64(const AaArgs&, const Trt<double>&, const int* items, int nItems, const int* cells,
                          cudaStream_t s) {
  fake::launch(s, [=] {
    check(std::vector<int>(items, items + nItems) == odd_items(), "the odd step reads its work items");
    const std::vector<int> want = odd_cells();
    check(std::vector<int>(cells, cells + want.size()) == want, "the odd step reads its cell lists");
  });
}

// The list layout of a lattice of fluid cells, and the tables of a batch.
long long list_build_device(const int*, const int dims[3], const int*, int, const int*, int, uint32_t* grid, uint32_t*,
                            long long, cudaStream_t s, const char**) {
  const int n = dims[0] * dims[1] * dims[2];
  fake::launch(s, [=] {
    for (int k = 0; k < n; ++k) grid[k] = (uint32_t)k;
  });
  cudaStreamSynchronize(s);
  return n;
}
int list_runs_device(const uint32_t*, int nFluid, cudaStream_t s, uint32_t** runs, uint32_t** runOff, size_t* runBytes) {
  cudaStreamSynchronize(s);
  const int tiles = (nFluid + kListTile - 1) / kListTile;
  *runBytes = 64 * (size_t)tiles;
  const cudaError_t e = dev_alloc(runs, *runBytes);
  if (e != cudaSuccess) return (int)e;
  return (int)dev_alloc(runOff, sizeof(uint32_t) * (tiles + 1));
}
int list_resident_tiles(int) { return 0; }
int list_pair_resident(int) { return 4; }
double pair_schedule(const uint32_t*, const uint32_t*, int nTiles, int, double, std::vector<PairItem>& items) {
  items.assign(nTiles + 2, PairItem{});
  for (size_t k = 0; k < items.size(); ++k) items[k].tile = (uint32_t)k;
  return 0.0;
}
void list_pair_fp64(const ListArgs& a, const PairArgs<3>& p, const Trt<double>&, cudaStream_t s) {
  fake::launch(s, [=] {
    for (uint32_t k = 0; k < p.nItems; ++k) check(p.items[k].tile == k, "the fused pair reads its items");
    a.f[0] += 1.0;
  });
}
void list_pull_fp64(const ListArgs& a, const Trt<double>&, cudaStream_t s) {
  fake::launch(s, [=] { a.g[0] = a.f[0] + 1.0; });
}
void list_tile_reach(const uint32_t*, int nFluid, long long, uint32_t* reach, cudaStream_t s) {
  fake::launch(s, [=] {
    for (int t = 0; t < (nFluid + kListTile - 1) / kListTile; ++t)
      for (int c = 0; c < 6; ++c) reach[6 * t + c] = (uint32_t)t;
  });
}
void batch_pad_adjacency(uint32_t*, int, long long, cudaStream_t) {}
void batch_build_tiles(const BatchDomain*, const int*, int nTiles, BatchTile* out, cudaStream_t s) {
  fake::launch(s, [=] { std::memset((void*)out, 0, sizeof(BatchTile) * nTiles); });
}
uint32_t batch_odd_order(const uint32_t*, int nTiles, std::vector<BatchOdd>& odd) {
  odd.resize(nTiles);
  return 0;
}
void batch_build_items(const BatchDomain*, const int*, int nTiles, uint32_t lead, PairItem* items, cudaStream_t s) {
  fake::launch(s, [=] { std::memset((void*)items, 0, sizeof(PairItem) * (nTiles + lead)); });
}
int batch_pair_resident(int) { return 16; }
void batch_even_lp(const BatchArgs& a, const BatchLaunch&, int, cudaStream_t s) {
  fake::launch(s, [=] {
    if (g_waitRunsOut) *a.err |= 1;
    g_steps += *a.nTiles > 0;
    fake::now += 1.0;
    for (int t = 0; t < *a.nTiles; ++t) check(a.tiles[t].nCells == 0, "the step reads its tile records");
  });
}
void batch_pair_lp(const BatchPairArgs& a, int grid, cudaStream_t s) {
  fake::launch(s, [=] {
    const PairArgs<3> p = *a.pair;
    check((uint32_t)grid >= p.nItems, "the grid covers the items");
    for (uint32_t k = 0; k < p.nItems; ++k) check(p.items[k].tile == 0, "the pair reads its items");
    for (uint32_t k = 0; k < p.nTiles; ++k) check(a.tiles[k].nCells == 0, "the pair reads its tile records");
    for (uint32_t k = 0; k < ((p.nTiles - 1) >> p.shift) + 3; ++k) check(p.count[k] == 0, "the counters start at zero");
    ++g_pairs;
    fake::now += g_pairMs;
  });
}
void batch_odd_lp(const BatchArgs& a, const BatchLaunch& l, int grid, cudaStream_t s) { batch_even_lp(a, l, grid, s); }
void batch_moments(const BatchArgs&, int, double*, const int*, const int*, int slots, double* out, cudaStream_t s) {
  fake::launch(s, [=] {
    for (int k = 0; k < 4 * slots; ++k) out[k] = 1.0;
  });
}

}  // namespace lbm

namespace {

// The first half step of a whole-lattice instance on the caller's own stream.
void first_slab_step(int how) {
  Lattice lat(6, 5, 4);
  KernelData* kd = full_array(lat);
  cudaStream_t mine;
  cudaStreamCreateWithFlags(&mine, cudaStreamNonBlocking);
  CaseData cd = a_case();
  int rc = 0;
  if (how == 0) rc = lbm_aa_slab_odd_part(kd, &cd, 0, mine);
  if (how == 1) rc = lbm_aa_slab_step(kd, &cd, 1, mine);
  if (how == 2) rc = lbm_aa_slab_step(kd, &cd, 0, mine) | lbm_aa_slab_step(kd, &cd, 1, mine);
  check(rc == 0, "the step is accepted");
  cudaStreamSynchronize(mine);
  D3Q19CudaAaDeinit_AaSoA(&lat.ld, &kd);
}

// The same captured into a graph: nothing is allocated, copied or waited for.
void first_slab_step_captured() {
  Lattice lat(6, 5, 4);
  KernelData* kd = full_array(lat);
  cudaStream_t mine;
  cudaStreamCreateWithFlags(&mine, cudaStreamNonBlocking);
  CaseData cd = a_case();
  const size_t blocks = fake::blocks.size();
  cudaStreamBeginCapture(mine, cudaStreamCaptureModeGlobal);
  fake::calls = 0;
  check(lbm_aa_slab_step(kd, &cd, 0, mine) == 0 && lbm_aa_slab_step(kd, &cd, 1, mine) == 0, "the steps are accepted");
  check(fake::calls == 0 && fake::blocks.size() == blocks, "a step is a launch and nothing else");
  cudaGraph_t g;
  cudaGraphExec_t e;
  cudaStreamEndCapture(mine, &g);
  cudaGraphInstantiate(&e, g, 0);
  cudaGraphLaunch(e, mine);
  cudaStreamSynchronize(mine);
  cudaGraphExecDestroy(e);
  cudaGraphDestroy(g);
  D3Q19CudaAaDeinit_AaSoA(&lat.ld, &kd);
}

// Deinit of an instance whose steps are under way, with another device current.
void deinit_from_another_device() {
  Lattice lat(6, 5, 4);
  KernelData* kd = full_array(lat);
  CaseData cd = a_case();
  check(lbm_b200_step_device(kd, &cd, 4) == 0, "the steps are accepted");
  cudaSetDevice(1);
  D3Q19CudaAaDeinit_AaSoA(&lat.ld, &kd);
  check(fake::device == 1, "the caller's device stays current");
  check(fake::blocks.empty(), "the instance's memory is given back");
  fake::run_device(0);  // what the free did not wait for uses the memory now
}

// A wait inside a step runs out: what is read back afterwards says so.
void batch_results_of_a_lost_state() {
  Lattice lat(6, 5, 4);
  void* b = lbm_batch_create(1, 1.0, 4);
  const int slot = lbm_batch_add(b, &lat.ld, 1.2, 0.1875, 1e-5);
  check(slot == 0, "the domain is admitted");
  std::vector<double> sums(16), field(19 * 6 * 5 * 4);
  const char* path = "/dev/null";
  for (int graph = 0; graph < 2; ++graph) {
    check(lbm_batch_step(b, 2, graph) == 0, "the steps are accepted");
    check(lbm_batch_moments(b, sums.data()) == 0 && sums[0] == 1.0, "the sums of a good state");
    check(lbm_batch_get_field(b, slot, field.data()) == 0, "the field of a good state");
    check(lbm_batch_checkpoint_save(b, slot, path) == 0, "the checkpoint of a good state");
  }
  g_waitRunsOut = true;
  check(lbm_batch_step(b, 2, 1) == 0, "the steps are accepted");
  check(lbm_batch_moments(b, sums.data()) == -7, "no sums of a lost state");
  check(lbm_batch_get_field(b, slot, field.data()) == -7, "no field of a lost state");
  check(lbm_batch_checkpoint_save(b, slot, path) == -7, "no checkpoint of a lost state");
  check(lbm_batch_sync(b) == -7, "sync reports it too");
  lbm_batch_destroy(b);
}

// A domain is admitted to a running batch, or leaves it, with memory for k more
// allocations. The others go on, and nothing of a refused one stays.
void batch_without_memory() {
  Lattice first(32, 32, 32), next(72, 71, 70);
  auto steps = [](void* b, const char* what) {
    for (int graph = 0; graph < 2; ++graph)
      check(lbm_batch_step(b, 2, graph) == 0 && lbm_batch_sync(b) == 0, what);
  };
  for (int k = 0; k == 0 || fake::failed; ++k) {
    void* b = lbm_batch_create(1, 1.0, 4);
    check(lbm_batch_add(b, &first.ld, 1.2, 0.1875, 1e-5) == 0, "the first domain is admitted");
    g_pairs = 0;
    steps(b, "it steps");
    check(g_pairs == 2, "in fused pairs");
    const size_t used = lbm_batch_bytes_used(b), blocks = fake::blocks.size();
    fake::failed = false;
    fake::failAfter = k;
    const int slot = lbm_batch_add(b, &next.ld, 1.2, 0.1875, 1e-5);
    fake::failAfter = -1;
    if (slot < 0) {
      check(lbm_batch_active_domains(b) == 1 && lbm_batch_bytes_used(b) == used, "the refused domain does not count");
      check(fake::blocks.size() <= blocks, "its memory is given back");
      steps(b, "the steps go on");
      check(lbm_batch_add(b, &next.ld, 1.2, 0.1875, 1e-5) == 1, "it is admitted later");
    }
    steps(b, "the steps go on with it");
    fake::failAfter = 0;
    check(lbm_batch_remove(b, 0) == 0, "a domain may leave without memory");
    fake::failAfter = -1;
    steps(b, "the steps go on without it");
    lbm_batch_destroy(b);
    check(fake::blocks.empty(), "the batch's memory is given back");
  }
}

// Steps of an empty batch do nothing; those of the domain that comes next do.
void batch_steps_while_empty() {
  Lattice lat(6, 5, 4);
  void* b = lbm_batch_create(1, 1.0, 4);
  for (int again = 0; again < 2; ++again) {
    check(lbm_batch_step(b, 2, 1) == 0 && lbm_batch_sync(b) == 0, "an empty batch steps");
    check(lbm_batch_add(b, &lat.ld, 1.2, 0.1875, 1e-5) == 0, "the domain is admitted");
    g_steps = 0;
    check(lbm_batch_step(b, 2, 1) == 0 && lbm_batch_sync(b) == 0 && g_steps == 2, "the domain steps");
    check(lbm_batch_remove(b, 0) == 0, "the domain leaves");
    check(lbm_batch_step(b, 4, 1) == 0 && lbm_batch_sync(b) == 0, "an empty batch steps");
    check(lbm_batch_add(b, &lat.ld, 1.2, 0.1875, 1e-5) == 0, "the domain is admitted");
    g_steps = 0;
    check(lbm_batch_step(b, 4, 1) == 0 && lbm_batch_sync(b) == 0 && g_steps == 4, "the domain steps");
    check(lbm_batch_remove(b, 0) == 0, "the domain leaves");
  }
  lbm_batch_destroy(b);
}

// Copies from pageable memory may read it as late as the stream gets to them:
// what they read has to be there until then.
void uploads_outlive_the_call(const char* what) {
  fake::staged = false;
  const std::string kind = what;
  Lattice lat(16, 10, 8);
  Parameters p{};
  CaseData cd = a_case();
  KernelData* kd = nullptr;
  if (kind == "batch") {
    void* b = lbm_batch_create(1, 1.0, 4);
    check(lbm_batch_add(b, &lat.ld, 1.2, 0.1875, 1e-5) == 0 && lbm_batch_step(b, 2, 1) == 0 && lbm_batch_sync(b) == 0,
          "a domain steps");
    lbm_batch_destroy(b);
    return;
  }
  if (kind == "full") D3Q19CudaAaInit_AaSoA(&lat.ld, &kd, &p);
  if (kind == "list") D3Q19CudaListAaPvInit_PushSoA(&lat.ld, &kd, &p);
  if (kind == "slab") kd = lbm_aa_slab_init(&lat.ld, 0, 8, 1, 1, &p);
  if (kind == "list slab") kd = lbm_aa_list_slab_init(&lat.ld, 0, 8, 1, 1, &p);
  check(kd != nullptr, "the instance is there");
  if (kind == "full" || kind == "list") check(lbm_b200_step_device(kd, &cd, 4) == 0, "the steps are accepted");
  if (kind == "slab") check(lbm_aa_slab_step(kd, &cd, 1, nullptr) == 0, "the step is accepted");
  fake::run_device(0);
  lbm_aa_slab_deinit(kd);
}

// The PDF arrays whose pointers the library gives out are blocks of their own:
// memory of a pool has no IPC handle and is not mapped to peers.
void state_pointer_is_a_block() {
  Lattice lat(6, 5, 4);
  Parameters p{};
  for (int row = 0; row < 2; ++row) {
    KernelData* kd = nullptr;
    if (row == 0) D3Q19CudaListAaPvInit_PushSoA(&lat.ld, &kd, &p);
    if (row == 1) D3Q19CudaListInit_PullSoA(&lat.ld, &kd, &p);
    CaseData cd = a_case();
    for (int k = 0; k < 2; ++k) {  // both grids of the two-grid row
      double* pdfs = nullptr;
      check(lbm_b200_device_state(kd, &pdfs, nullptr, nullptr, nullptr) == 0, "the state has a pointer");
      const auto it = fake::blocks.find(pdfs);
      check(it != fake::blocks.end() && !it->second.pool, "it is a block from cudaMalloc");
      check(lbm_b200_step_device(kd, &cd, 1) == 0, "the step is accepted");
    }
    D3Q19CudaListAaPvDeinit_PushSoA(&lat.ld, &kd);
    check(lbm_b200_release_memory() == 0 && fake::blocks.empty(), "the instance's memory is given back");
  }
}

// Freed blocks are kept for the next of about their size, up to a bound, per
// device, and go when memory is short.
void kept_blocks() {
  const size_t MB = 1 << 20;
  auto kept = [] {
    size_t n = 0;
    for (const auto& b : fake::blocks) n += b.second.bytes;
    return n;
  };
  void *a, *b, *c;
  lbm::dev_alloc_block(&a, 8 * MB);
  lbm::dev_free(a);
  lbm::dev_alloc_block(&b, 7 * MB);
  check(b == a, "a block is used again");
  lbm::dev_free(b);
  lbm::dev_alloc_block(&b, 6 * MB);
  check(b != a, "not for a much smaller one");
  lbm::dev_alloc_block(&c, 9 * MB);
  check(c != a, "not for a larger one");
  fake::device = 1;
  void* d;
  lbm::dev_alloc_block(&d, 8 * MB);
  check(d != a, "not on another device");
  lbm::dev_free(d);
  lbm::dev_free(c);
  lbm::dev_free(b);
  check(lbm_b200_release_memory() == 0 && kept() == 23 * MB, "the current device's are given back");
  fake::device = 0;
  check(lbm_b200_release_memory() == 0 && kept() == 0, "and the other's");
  std::vector<void*> many(30);
  for (void*& p : many) lbm::dev_alloc_block(&p, 5 * MB);
  for (void* p : many) lbm::dev_free(p);
  check(kept() <= 64 * MB && kept() > 50 * MB, "what is kept is bounded");
  lbm::dev_alloc_block(&a, 65 * MB);
  lbm::dev_free(a);
  check(kept() <= 64 * MB, "a larger block is not kept");
  fake::capacity = 70 * MB;
  check(lbm::dev_alloc_block(&a, 66 * MB) == cudaSuccess && kept() == 66 * MB, "what is kept makes room");
  lbm::dev_free(a);
  lbm::dev_alloc_block(&a, 40 * MB);
  lbm::dev_free(a);
  check(lbm::dev_alloc(&b, 60 * MB) == cudaSuccess && kept() == 60 * MB, "for the pool's too");
  check(lbm::dev_alloc(&c, 60 * MB) == cudaErrorMemoryAllocation && !c, "no memory is an error");
  lbm::dev_free(b);
}

// The tuner leaves the batch on the faster of fused pairs and the best steps
// apart, whatever a launch shape asked for before it.
void batch_tune_keeps_the_fastest() {
  Lattice large(32, 32, 32), small(16, 10, 8);
  for (double pairMs : {1.5, 2.5, 1.5})
    for (int shaped = 0; shaped < 2; ++shaped) {
      g_pairMs = pairMs;
      void* b = lbm_batch_create(1, 1.0, 4);
      check(lbm_batch_add(b, &large.ld, 1.2, 0.1875, 1e-5) == 0, "the domain is admitted");
      if (shaped) check(lbm_batch_set_launch(b, 2, 128, 0) == 0, "a launch shape is taken");
      for (int graph = 0; graph < 2; ++graph) {
        g_pairs = g_steps = 0;
        check(lbm_batch_step(b, 2, graph) == 0 && lbm_batch_sync(b) == 0, "the domain steps");
        check(shaped ? g_steps == 2 && g_pairs == 0 : g_pairs == 1 && g_steps == 0, "in the shape asked for");
      }
      double rows[64 * 5];
      check(lbm_batch_tune(b, 4, rows, 64) == 36, "every launch shape is timed");
      for (int graph = 0; graph < 2; ++graph) {
        g_pairs = g_steps = 0;
        check(lbm_batch_step(b, 2, graph) == 0 && lbm_batch_sync(b) == 0, "the domain steps");
        check(pairMs < 2 ? g_pairs == 1 && g_steps == 0 : g_steps == 2 && g_pairs == 0, "in the fastest way");
      }
      lbm_batch_destroy(b);
    }
  // a batch that has no fused form
  void* b = lbm_batch_create(1, 1.0, 4);
  check(lbm_batch_add(b, &small.ld, 1.2, 0.1875, 1e-5) == 0, "the domain is admitted");
  check(lbm_batch_tune(b, 4, nullptr, 64) == 36, "every launch shape is timed");
  check(lbm_batch_add(b, &large.ld, 1.2, 0.1875, 1e-5) == 1, "a large one joins");
  g_pairs = g_steps = 0;
  check(lbm_batch_step(b, 2, 1) == 0 && lbm_batch_sync(b) == 0 && g_pairs == 1 && g_steps == 0, "it steps fused");
  lbm_batch_destroy(b);
}

const std::map<std::string, std::function<void()>> kCases = {
    {"first_odd_part", [] { first_slab_step(0); }},
    {"first_odd_half", [] { first_slab_step(1); }},
    {"first_even_half", [] { first_slab_step(2); }},
    {"first_slab_step_captured", first_slab_step_captured},
    {"deinit_from_another_device", deinit_from_another_device},
    {"state_pointer_is_a_block", state_pointer_is_a_block},
    {"kept_blocks", kept_blocks},
    {"uploads_full", [] { uploads_outlive_the_call("full"); }},
    {"uploads_list", [] { uploads_outlive_the_call("list"); }},
    {"uploads_slab", [] { uploads_outlive_the_call("slab"); }},
    {"uploads_list_slab", [] { uploads_outlive_the_call("list slab"); }},
    {"uploads_batch", [] { uploads_outlive_the_call("batch"); }},
    {"batch_results_of_a_lost_state", batch_results_of_a_lost_state},
    {"batch_without_memory", batch_without_memory},
    {"batch_steps_while_empty", batch_steps_while_empty},
    {"batch_tune_keeps_the_fastest", batch_tune_keeps_the_fastest},
};

}  // namespace

int main(int argc, char** argv) {
  const auto it = kCases.find(argc > 1 ? argv[1] : "");
  if (it == kCases.end()) {
    std::printf("unknown case\n");
    return 2;
  }
  it->second();
  return g_bad != 0;
}
