// lbm_batch.cu -- host side of the batched list AA form (include/lbm_b200.h,
// "Batched domains"): admission of domains under an HBM budget, the device
// tile/domain tables, CUDA-graph replay of whole step sequences, the FP64
// per-domain sums, and the launch autotuner.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "../../include/lbm_b200.h"
#include "lbm_batch.cuh"
#include "lbm_host.h"
#include "lbm_mem.cuh"

namespace {

using lbm::Q;
using lbm::QM;

const char* g_batchError = "";

#define BCK(call)                                                          \
  do {                                                                     \
    cudaError_t e_ = (call);                                               \
    if (e_ != cudaSuccess) {                                               \
      g_batchError = cudaGetErrorString(e_);                               \
      cudaGetLastError(); /* reported here, not by the next launch check */ \
      std::fprintf(stderr, "lbm batch: %s: %s\n", #call, g_batchError);   \
      return -(int)e_ - 1000;                                              \
    }                                                                      \
  } while (0)

double weight_of(int d) {
  const int c2 = lbm::cx(d) * lbm::cx(d) + lbm::cy(d) * lbm::cy(d) + lbm::cz(d) * lbm::cz(d);
  return c2 == 0 ? 1.0 / 3.0 : (c2 == 1 ? 1.0 / 18.0 : 1.0 / 36.0);
}
double f16_scale_of(int d) { return d == lbm::DC ? 32768.0 : (weight_of(d) > 0.05 ? 262144.0 : 524288.0); }

struct DomainSlot {
  bool active = false;
  lbm::BatchDomain dev{};  // as uploaded to the device table
  void* pdfs = nullptr;
  uint32_t* runs = nullptr;    // run-compressed adjacency
  uint32_t* runOff = nullptr;
  lbm::BatchOdd* odd = nullptr;
  uint32_t ahead = 0;          // batch_odd_order
  int nTiles = 0;
  size_t bytes = 0;
  int dims[3] = {0, 0, 0};
  std::vector<uint32_t> grid;  // lattice cell -> node (for field access)
  double omega = 1.0, lambda = 1.0 / 12.0, xforce = 0.0;
};

struct Batch {
  int storage;
  size_t elemBytes;
  size_t budget, used = 0;
  int maxSlots, maxTiles;
  std::vector<DomainSlot> slots;
  std::vector<int> tileDomHost;
  int nTiles = 0;
  cudaStream_t stream = nullptr;
  lbm::BatchDomain* dDoms = nullptr;
  int* dTileDom = nullptr;
  lbm::BatchTile* dTiles = nullptr;  // tile records, capacity tileCap
  int tileCap = 0;
  int gridTiles = 0;  // grid of the one-block-per-tile launches (>= nTiles)
  int* dNTiles = nullptr;
  int* dErr = nullptr;
  double* dPartials = nullptr;
  int* dDomTileStart = nullptr;
  int* dDomTileCount = nullptr;
  double* dMoments = nullptr;  // 4 per slot, then the error word
  lbm::BatchLaunch evenL{256, 1, 0}, oddL{256, 1, 0};
  bool separate = false;             // launches of their own for even and odd steps were asked for
  lbm::PairArgs<3> pair{};           // fused pairs (nItems 0: none), as uploaded to dPair
  lbm::PairArgs<3>* dPair = nullptr;
  lbm::PairItem* dItems = nullptr;   // capacity itemCap
  uint32_t* dCount = nullptr;        // as many groups as itemCap items can have
  uint32_t itemCap = 0, gridItems = 0;
  std::vector<double> sums;          // dMoments on the host
  std::map<int, cudaGraphExec_t> graphs;  // steps -> instantiated graph
  long long launches = 0;
  int numSMs = 148;
};

lbm::BatchArgs args_of(const Batch* b, const lbm::BatchLaunch& l) {
  lbm::BatchArgs a;
  a.doms = b->dDoms;
  a.tileDom = b->dTileDom;
  a.tiles = b->dTiles;
  a.nTiles = b->dNTiles;
  a.err = b->dErr;
  a.storage = b->storage;
  a.nodesPerThread = l.nodesPerThread;
  a.blockNodes = l.threads * l.nodesPerThread;
  return a;
}

void drop_graphs(Batch* b) {
  for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
  b->graphs.clear();
}

// Tables of fused pairs of nItems items. False without memory for them, which is
// no reason to refuse a domain: the steps are launches of their own then.
bool reserve_pairs(Batch* b, uint32_t nItems) {
  if (nItems <= b->itemCap) return true;
  lbm::dev_free(b->dItems);  // the caller has waited for the steps
  lbm::dev_free(b->dCount);
  b->dItems = nullptr;
  b->dCount = nullptr;
  b->itemCap = 0;
  const uint32_t cap = nItems + nItems / 2;
  if (lbm::dev_alloc(&b->dItems, sizeof(lbm::PairItem) * (size_t)cap) != cudaSuccess ||
      lbm::dev_alloc(&b->dCount, sizeof(uint32_t) * ((size_t)cap / 8 + 4)) != cudaSuccess) {  // groups of 8 or more
    cudaGetLastError();
    lbm::dev_free(b->dItems);
    b->dItems = nullptr;
    return false;
  }
  b->itemCap = cap;
  return true;
}

// Fused pairs (two steps in one launch) for the tables just published, where
// they are the faster way.
//
// The lead of the even steps: the blocks that run at once beyond what the
// domain that needs it most needs its even tiles ahead; all tiles in a smaller
// batch (FP32, 73905 / 17191 tiles, us per step: 459 / 105.1 at 740 resident
// blocks, 470 / 105.9 at 925, 478 / 106.2 at 1110, 507 / 111 at 1400). The PDFs
// in between have to stay in 2/5 of L2 as for one lattice.
//
// Worth it once the PDFs outgrow half of L2; below, both launches find them
// there. us per step, a launch per step / fused: FP32 49 MB 14.9 / 16.3, 85 MB
// 33.2 / 29.5, 104 MB 41.8 / 35.4, 334 MB 128.5 / 107.6; FP16 24 MB 13.6 / 14.9,
// 43 MB 23.7 / 24.7, 52 MB 31.1 / 30.7, 167 MB 101.1 / 93.4.
int publish_pairs(Batch* b, uint32_t ahead) {
  const uint32_t n = static_cast<uint32_t>(b->nTiles);
  const uint32_t margin = std::max<uint32_t>(lbm::batch_pair_resident(b->storage), 2u << lbm::pair_group_shift(n));
  const uint32_t lead = std::min(n, margin + ahead);
  int dev = 0, l2 = 0;
  BCK(cudaGetDevice(&dev));
  BCK(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev));
  const uint32_t nItems = n + lead;
  const bool fused = (double)n * lbm::kBatchTileNodes * Q * b->elemBytes > 0.5 * l2 &&
                     (double)lead * lbm::kBatchTileNodes * Q * b->elemBytes <= 0.4 * l2 && reserve_pairs(b, nItems);
  if (fused != (b->pair.nItems > 0)) drop_graphs(b);
  b->pair.nItems = 0;
  if (!fused) return 0;
  if (nItems > b->gridItems || nItems < b->gridItems / 2) {
    drop_graphs(b);
    b->gridItems = nItems + nItems / 8;
  }
  const int shift = lbm::pair_group_shift(n);
  const size_t groups = ((n - 1) >> shift) + 1;
  b->pair.items = b->dItems;
  b->pair.count = b->dCount;
  b->pair.launches = b->dCount + groups;
  b->pair.nTiles = n;
  b->pair.shift = shift;
  b->pair.prefetch = 0;
  b->pair.nItems = nItems;
  BCK(cudaMemsetAsync(b->dCount, 0, sizeof(uint32_t) * (groups + 2), b->stream));
  BCK(cudaMemcpyAsync(b->dPair, &b->pair, sizeof(b->pair), cudaMemcpyHostToDevice, b->stream));
  lbm::batch_build_items(b->dDoms, b->dTileDom, b->nTiles, lead, b->dItems, b->stream);
  BCK(cudaGetLastError());
  return 0;
}

// Rebuilds the tile table, the per-domain tile ranges and the tile records
// after a change of membership (stream-ordered uploads, then a device pass
// that fills the records). What can fail for want of memory comes first and
// leaves the tables published before as they are.
int publish(Batch* b) {
  std::vector<int> start(b->maxSlots, 0), count(b->maxSlots, 0);
  uint32_t ahead = 0;
  int n = 0;
  for (int s = 0; s < b->maxSlots; ++s) {
    const DomainSlot& d = b->slots[s];
    if (!d.active) continue;
    start[s] = n;
    count[s] = d.nTiles;
    ahead = std::max(ahead, d.ahead);
    n += d.nTiles;
  }
  if (n > b->maxTiles) return -3;
  BCK(cudaStreamSynchronize(b->stream));
  if (n > b->tileCap) {
    const int cap = std::min(b->maxTiles, std::max(n + n / 2, 1024));
    lbm::BatchTile* tiles = nullptr;
    BCK(lbm::dev_alloc(&tiles, sizeof(lbm::BatchTile) * (size_t)cap));
    // graphs captured with the old records go
    drop_graphs(b);
    lbm::dev_free(b->dTiles);
    b->dTiles = tiles;
    b->tileCap = cap;
  }
  b->nTiles = n;
  b->tileDomHost.clear();
  for (int s = 0; s < b->maxSlots; ++s) {
    DomainSlot& d = b->slots[s];
    if (!d.active) continue;
    d.dev.tileStart = start[s];
    b->tileDomHost.insert(b->tileDomHost.end(), d.nTiles, s);
    BCK(cudaMemcpyAsync(b->dDoms + s, &d.dev, sizeof(lbm::BatchDomain), cudaMemcpyHostToDevice, b->stream));
  }
  if (b->nTiles)
    BCK(cudaMemcpyAsync(b->dTileDom, b->tileDomHost.data(), sizeof(int) * b->nTiles, cudaMemcpyHostToDevice,
                        b->stream));
  // the grid of one-block-per-tile launches keeps some headroom, so that
  // graphs survive admissions; it is resized (and graphs dropped) when the
  // table outgrows it or shrinks below half of it
  if (b->nTiles > b->gridTiles || b->nTiles < b->gridTiles / 2) {
    const int g = std::max(b->nTiles + b->nTiles / 8, 64);
    if (g != b->gridTiles) {
      drop_graphs(b);
      b->gridTiles = g;
    }
  }
  BCK(cudaMemcpyAsync(b->dNTiles, &b->nTiles, sizeof(int), cudaMemcpyHostToDevice, b->stream));
  BCK(cudaMemcpyAsync(b->dDomTileStart, start.data(), sizeof(int) * b->maxSlots, cudaMemcpyHostToDevice, b->stream));
  BCK(cudaMemcpyAsync(b->dDomTileCount, count.data(), sizeof(int) * b->maxSlots, cudaMemcpyHostToDevice, b->stream));
  lbm::batch_build_tiles(b->dDoms, b->dTileDom, b->nTiles, b->dTiles, b->stream);
  BCK(cudaGetLastError());
  const int rc = publish_pairs(b, ahead);
  if (rc) return rc;
  // the host vectors above are read by the copies: wait before they go away
  BCK(cudaStreamSynchronize(b->stream));
  return 0;
}

void free_domain(DomainSlot& d) {
  lbm::dev_free(d.pdfs);
  lbm::dev_free(d.runs);
  lbm::dev_free(d.runOff);
  lbm::dev_free(d.odd);
  d = DomainSlot();
}

bool fused(const Batch* b) { return b->pair.nItems > 0 && !b->separate; }

int enqueue(Batch* b, int nsteps) {
  if (b->nTiles == 0) return 0;
  if (fused(b)) {
    const lbm::BatchPairArgs a{b->dTiles, b->dPair, b->dErr, b->storage};
    for (int it = 0; it < nsteps; it += 2) {
      lbm::batch_pair_lp(a, (int)b->gridItems, b->stream);
      ++b->launches;
    }
    BCK(cudaGetLastError());
    return 0;
  }
  const lbm::BatchArgs ae = args_of(b, b->evenL), ao = args_of(b, b->oddL);
  for (int it = 0; it < nsteps; it += 2) {
    lbm::batch_even_lp(ae, b->evenL, b->evenL.blocks ? b->evenL.blocks : b->gridTiles, b->stream);
    lbm::batch_odd_lp(ao, b->oddL, b->oddL.blocks ? b->oddL.blocks : b->gridTiles, b->stream);
    b->launches += 2;
  }
  BCK(cudaGetLastError());
  return 0;
}

// -7 if a wait inside a step gave up (the steps' blocks wait for one another):
// the PDFs, and what was copied from them, are no state of the update.
int lost_state(int err) {
  if (err == 0) return 0;
  g_batchError = "a device wait exceeded its limit";
  return -7;
}

// Waits for what the stream holds; lost_state of the device error word.
int finish(Batch* b) {
  int err = 0;
  BCK(cudaMemcpyAsync(&err, b->dErr, sizeof(int), cudaMemcpyDeviceToHost, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  return lost_state(err);
}

// Bound on a domain's device bytes: PDFs plus the adjacency (full rows
// while the run-compressed form is built from them; the runs never exceed
// the full rows plus a 48-byte header per tile).
size_t domain_bytes(const Batch* b, long long nCells) {
  return (size_t)nCells * Q * b->elemBytes + (size_t)nCells * QM * 4 +
         (size_t)(nCells / lbm::kBatchTileNodes) * lbm::kRunHdrWords * 4;
}

lbm::TrtW trt_of(double omega, double lambda, double xforce) {
  lbm::TrtW t;
  t.omegaEven = (float)omega;
  t.omegaOdd = (float)(1.0 / (0.5 + lambda / (1.0 / omega - 0.5)));
  t.fx1 = (float)(3.0 * (1.0 / 18.0) * xforce);
  t.fx2 = (float)(3.0 * (1.0 / 36.0) * xforce);
  return t;
}

// The device arrays of a domain of lattice `ld`, into slot d (on failure the
// caller frees what is there).
int build_domain(Batch* b, const LatticeDesc* ld, long long nCells, DomainSlot& d) {
  // what is needed while building; goes when the stream has finished with it
  struct Scratch {
    cudaStream_t s;
    uint32_t *adj = nullptr, *grid = nullptr, *reach = nullptr;
    int* mask = nullptr;
    ~Scratch() {
      cudaStreamSynchronize(s);
      lbm::dev_free(adj);
      lbm::dev_free(grid);
      lbm::dev_free(reach);
      lbm::dev_free(mask);
    }
  };
  const int nFluid = ld->nFluid, nTiles = (int)(nCells / lbm::kBatchTileNodes);
  const long ncell = (long)ld->Dims[0] * ld->Dims[1] * ld->Dims[2];
  std::vector<uint32_t> reach;
  std::vector<lbm::BatchOdd> odd;
  d = DomainSlot();
  d.grid.resize(ncell);
  Scratch tmp{b->stream};
  BCK(lbm::dev_alloc(&d.pdfs, (size_t)nCells * Q * b->elemBytes));
  // numbering and adjacency built on the device (lbm_build.cu); padding
  // nodes then point at their own slots so that every entry is in range;
  // the steps read the run-compressed form, built from it
  BCK(lbm::dev_alloc(&tmp.adj, (size_t)nCells * QM * 4));
  BCK(lbm::dev_alloc(&tmp.mask, sizeof(int) * ncell));
  BCK(lbm::dev_alloc(&tmp.grid, sizeof(uint32_t) * ncell));
  BCK(cudaMemcpyAsync(tmp.mask, ld->Lattice, sizeof(int) * ncell, cudaMemcpyHostToDevice, b->stream));
  const int blk[3] = {0, 0, 0}, per[3] = {ld->PeriodicX, ld->PeriodicY, ld->PeriodicZ};
  const char* berr = "";
  const long long nf = lbm::list_build_device(tmp.mask, ld->Dims, per, 0, blk, (int)nCells, tmp.grid, tmp.adj, nCells,
                                              b->stream, &berr);
  if (nf != nFluid) {
    g_batchError = nf < 0 ? berr : "the mask's fluid cell count differs from the lattice's";
    cudaGetLastError();
    return -6;
  }
  lbm::batch_pad_adjacency(tmp.adj, nFluid, nCells, b->stream);
  BCK(cudaMemcpyAsync(d.grid.data(), tmp.grid, sizeof(uint32_t) * ncell, cudaMemcpyDeviceToHost, b->stream));
  for (int t = 0; t < 3 * nTiles; ++t) reach.insert(reach.end(), {1u, 0u});  // no node: reaches nothing
  if (nFluid > 0) {
    BCK(lbm::dev_alloc(&tmp.reach, sizeof(uint32_t) * reach.size()));
    lbm::list_tile_reach(tmp.adj, nFluid, nCells, tmp.reach, b->stream);
    BCK(cudaMemcpyAsync(reach.data(), tmp.reach, sizeof(uint32_t) * reach.size(), cudaMemcpyDeviceToHost, b->stream));
  }
  size_t runBytes = 0;
  if (lbm::list_runs_device(tmp.adj, (int)nCells, b->stream, &d.runs, &d.runOff, &runBytes)) {
    g_batchError = "building the run-compressed adjacency failed";
    cudaGetLastError();
    return -6;
  }
  BCK(cudaStreamSynchronize(b->stream));
  d.ahead = lbm::batch_odd_order(reach.data(), nTiles, odd);
  BCK(lbm::dev_alloc(&d.odd, sizeof(lbm::BatchOdd) * odd.size()));
  BCK(cudaMemcpyAsync(d.odd, odd.data(), sizeof(lbm::BatchOdd) * odd.size(), cudaMemcpyHostToDevice, b->stream));
  d.nTiles = nTiles;
  for (int i = 0; i < 3; ++i) d.dims[i] = ld->Dims[i];
  d.dev.f = d.pdfs;
  d.dev.runs = d.runs;
  d.dev.runOff = d.runOff;
  d.dev.nCells = nCells;
  d.dev.nFluid = nFluid;
  d.dev.odd = d.odd;
  return 0;
}

// Domain checkpoint: header (host byte order), then the slot's PDF array as
// the device holds it (storage format, tile padding included).
struct DomCkpt {
  char magic[8];  // "LBMBDOM1"
  int32_t storage, nFluid;
  int32_t dims[3], reserved;
  int64_t nCells;
  double omega, lambda, xforce;
  uint64_t checksum;
};
const char kDomMagic[8] = {'L', 'B', 'M', 'B', 'D', 'O', 'M', '1'};

uint64_t dom_fnv1a64(const void* data, size_t n) {
  const unsigned char* p = static_cast<const unsigned char*>(data);
  uint64_t h = 1469598103934665603ull;
  for (size_t k = 0; k < n; ++k) {
    h ^= p[k];
    h *= 1099511628211ull;
  }
  return h;
}

DomCkpt dom_header_of(const Batch* b, const DomainSlot& d) {
  DomCkpt c;
  std::memset(&c, 0, sizeof(c));
  std::memcpy(c.magic, kDomMagic, 8);
  c.storage = b->storage;
  c.nFluid = d.dev.nFluid;
  for (int i = 0; i < 3; ++i) c.dims[i] = d.dims[i];
  c.nCells = d.dev.nCells;
  c.omega = d.omega;
  c.lambda = d.lambda;
  c.xforce = d.xforce;
  return c;
}
}  // namespace

extern "C" {

const char* lbm_batch_last_error(void) { return g_batchError; }

int lbm_batch_reset(void* h, int slot);

void* lbm_batch_create(int storage, double budgetGB, int maxDomains) {
  if (storage != lbm::kStoreF32 && storage != lbm::kStoreF16) {
    g_batchError = "batched domains support storage fp32 (1) and fp16 (2)";
    return nullptr;
  }
  Batch* b = new Batch();
  b->storage = storage;
  b->elemBytes = storage == lbm::kStoreF32 ? 4 : 2;
  b->budget = (size_t)(budgetGB * 1e9);
  b->maxSlots = maxDomains > 0 ? maxDomains : 1024;
  b->slots.resize(b->maxSlots);
  const size_t perTile = domain_bytes(b, lbm::kBatchTileNodes);
  b->maxTiles = (int)std::min<size_t>(b->budget / perTile + (size_t)b->maxSlots, (size_t)1 << 26);
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&b->numSMs, cudaDevAttrMultiProcessorCount, dev);
  bool ok = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) == cudaSuccess &&
            lbm::dev_alloc(&b->dDoms, sizeof(lbm::BatchDomain) * b->maxSlots) == cudaSuccess &&
            lbm::dev_alloc(&b->dTileDom, sizeof(int) * b->maxTiles) == cudaSuccess &&
            lbm::dev_alloc(&b->dNTiles, sizeof(int)) == cudaSuccess &&
            lbm::dev_alloc(&b->dErr, sizeof(int)) == cudaSuccess &&
            lbm::dev_alloc(&b->dPair, sizeof(lbm::PairArgs<3>)) == cudaSuccess &&
            lbm::dev_alloc(&b->dPartials, sizeof(double) * 4 * (size_t)b->maxTiles) == cudaSuccess &&
            lbm::dev_alloc(&b->dDomTileStart, sizeof(int) * b->maxSlots) == cudaSuccess &&
            lbm::dev_alloc(&b->dDomTileCount, sizeof(int) * b->maxSlots) == cudaSuccess &&
            lbm::dev_alloc(&b->dMoments, sizeof(double) * (4 * (size_t)b->maxSlots + 1)) == cudaSuccess &&
            cudaMemsetAsync(b->dErr, 0, sizeof(int), b->stream) == cudaSuccess &&
            cudaMemsetAsync(b->dNTiles, 0, sizeof(int), b->stream) == cudaSuccess;
  if (!ok) {
    g_batchError = "device allocation of the batch tables failed";
    delete b;
    return nullptr;
  }
  b->evenL.blocks = b->oddL.blocks = 0;  // one block per tile until tuned
  return b;
}

void lbm_batch_destroy(void* h) {
  Batch* b = static_cast<Batch*>(h);
  if (!b) return;
  cudaStreamSynchronize(b->stream);
  drop_graphs(b);
  for (auto& s : b->slots) free_domain(s);
  lbm::dev_free(b->dPair);
  lbm::dev_free(b->dItems);
  lbm::dev_free(b->dCount);
  lbm::dev_free(b->dDoms);
  lbm::dev_free(b->dTileDom);
  lbm::dev_free(b->dTiles);
  lbm::dev_free(b->dNTiles);
  lbm::dev_free(b->dErr);
  lbm::dev_free(b->dPartials);
  lbm::dev_free(b->dDomTileStart);
  lbm::dev_free(b->dDomTileCount);
  lbm::dev_free(b->dMoments);
  cudaStreamDestroy(b->stream);
  delete b;
}

// Admits a domain; returns its slot, -1 when the HBM budget is exhausted,
// -2 when every slot is taken, or another negative code on errors. The PDFs
// start at rest (f = w, rho = 1, u = 0).
int lbm_batch_add(void* h, const LatticeDesc* ld, double omega, double lambda, double xforce) {
  Batch* b = static_cast<Batch*>(h);
  if (!(omega > 0.0 && omega < 2.0) || !(lambda > 0.0)) return -4;
  int slot = -1;
  for (int s = 0; s < b->maxSlots; ++s)
    if (!b->slots[s].active) { slot = s; break; }
  if (slot < 0) return -2;
  const int nFluid = ld->nFluid;
  const long long nCells = ((long long)std::max(nFluid, 1) + lbm::kBatchTileNodes - 1) / lbm::kBatchTileNodes *
                           lbm::kBatchTileNodes;
  const size_t bytes = domain_bytes(b, nCells);
  if (b->used + bytes > b->budget) return -1;
  if ((uint64_t)nCells * Q >= (1ull << 32)) return -5;

  DomainSlot& d = b->slots[slot];
  int rc = build_domain(b, ld, nCells, d);
  if (rc == 0) {
    d.active = true;
    d.bytes = bytes;
    d.omega = omega;
    d.lambda = lambda;
    d.xforce = xforce;
    d.dev.trt = trt_of(omega, lambda, xforce);
    b->used += bytes;
    rc = lbm_batch_reset(h, slot);
    if (rc == 0) rc = publish(b);
    if (rc == 0) return slot;
    b->used -= bytes;
  }
  cudaStreamSynchronize(b->stream);
  free_domain(d);
  return rc;
}

int lbm_batch_remove(void* h, int slot) {
  Batch* b = static_cast<Batch*>(h);
  if (slot < 0 || slot >= b->maxSlots || !b->slots[slot].active) return -1;
  BCK(cudaStreamSynchronize(b->stream));
  b->used -= b->slots[slot].bytes;
  free_domain(b->slots[slot]);
  return publish(b);
}

// PDFs of a slot back to rest, f = w (stream-ordered).
int lbm_batch_reset(void* h, int slot) {
  Batch* b = static_cast<Batch*>(h);
  DomainSlot& d = b->slots[slot];
  const size_t nc = (size_t)d.dev.nCells;
  // both storage formats hold deviations from w: rest is all zero bits
  BCK(cudaMemsetAsync(d.pdfs, 0, nc * Q * b->elemBytes, b->stream));
  return 0;
}

// Enqueues nsteps time steps (rounded up to even) of every active domain.
// With use_graph, sequences are captured once per length into a CUDA graph
// and replayed (the kernels read the tables from device memory, so the graph
// stays valid when domains come and go).
int lbm_batch_step(void* h, int nsteps, int use_graph) {
  Batch* b = static_cast<Batch*>(h);
  nsteps += nsteps & 1;
  if (nsteps <= 0) return 0;
  if (b->nTiles == 0) return 0;  // nothing to capture that would hold for later domains
  if (!use_graph) return enqueue(b, nsteps);
  auto it = b->graphs.find(nsteps);
  if (it == b->graphs.end()) {
    cudaGraph_t g;
    BCK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    const long long before = b->launches;
    enqueue(b, nsteps);
    b->launches = before;
    BCK(cudaStreamEndCapture(b->stream, &g));
    cudaGraphExec_t ge;
    BCK(cudaGraphInstantiate(&ge, g, 0));
    cudaGraphDestroy(g);
    it = b->graphs.emplace(nsteps, ge).first;
  }
  BCK(cudaGraphLaunch(it->second, b->stream));
  b->launches += fused(b) ? nsteps / 2 : nsteps;
  return 0;
}

int lbm_batch_sync(void* h) {
  return finish(static_cast<Batch*>(h));
}

// FP64 sums {rho, jx, jy, jz} of every slot into out (maxDomains x 4,
// inactive slots 0). Synchronises.
int lbm_batch_moments(void* h, double* out) {
  Batch* b = static_cast<Batch*>(h);
  const lbm::BatchArgs a = args_of(b, b->evenL);
  BCK(cudaMemsetAsync(b->dMoments, 0, sizeof(double) * 4 * b->maxSlots, b->stream));
  if (b->nTiles > 0)
    lbm::batch_moments(a, b->nTiles, b->dPartials, b->dDomTileStart, b->dDomTileCount, b->maxSlots, b->dMoments,
                       b->stream);
  BCK(cudaGetLastError());
  // the error word in the same copy: one of its own costs 8 us more, and
  // page-locked memory for it 2 to 5 ms when a batch is made
  const size_t n = 4 * (size_t)b->maxSlots;
  b->sums.resize(n + 1);
  BCK(cudaMemcpyAsync(b->dMoments + n, b->dErr, sizeof(int), cudaMemcpyDeviceToDevice, b->stream));
  BCK(cudaMemcpyAsync(b->sums.data(), b->dMoments, sizeof(double) * (n + 1), cudaMemcpyDeviceToHost, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  int err;
  std::memcpy(&err, &b->sums[n], sizeof(int));
  if (err == 0) std::memcpy(out, b->sums.data(), sizeof(double) * n);
  return lost_state(err);
}

// Logical PDFs of a slot (cells x fastest, 19 per cell, obstacles untouched)
// after the last completed even/odd pair.
int lbm_batch_get_field(void* h, int slot, double* out) {
  Batch* b = static_cast<Batch*>(h);
  DomainSlot& d = b->slots[slot];
  if (!d.active) return -1;
  const size_t nc = (size_t)d.dev.nCells;
  std::vector<unsigned char> raw(nc * Q * b->elemBytes);
  BCK(cudaMemcpyAsync(raw.data(), d.pdfs, raw.size(), cudaMemcpyDeviceToHost, b->stream));
  const int rc = finish(b);
  if (rc) return rc;
  const long ncell = (long)d.dims[0] * d.dims[1] * d.dims[2];
  for (long c = 0; c < ncell; ++c) {
    const uint32_t n = d.grid[c];
    if (n == 0xffffffffu) continue;
    for (int q = 0; q < Q; ++q) {
      const size_t k = (size_t)q * nc + n;
      double v;
      if (b->storage == lbm::kStoreF32)
        v = weight_of(q) + (double)reinterpret_cast<const float*>(raw.data())[k];
      else
        v = weight_of(q) + (double)lbmh_f16_to_f32(reinterpret_cast<const uint16_t*>(raw.data())[k]) / f16_scale_of(q);
      out[c * Q + q] = v;
    }
  }
  return 0;
}

int lbm_batch_set_field(void* h, int slot, const double* in) {
  Batch* b = static_cast<Batch*>(h);
  DomainSlot& d = b->slots[slot];
  if (!d.active) return -1;
  const size_t nc = (size_t)d.dev.nCells;
  std::vector<unsigned char> raw(nc * Q * b->elemBytes);
  BCK(cudaMemcpyAsync(raw.data(), d.pdfs, raw.size(), cudaMemcpyDeviceToHost, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  const long ncell = (long)d.dims[0] * d.dims[1] * d.dims[2];
  for (long c = 0; c < ncell; ++c) {
    const uint32_t n = d.grid[c];
    if (n == 0xffffffffu) continue;
    for (int q = 0; q < Q; ++q) {
      const size_t k = (size_t)q * nc + n;
      if (b->storage == lbm::kStoreF32)
        reinterpret_cast<float*>(raw.data())[k] = (float)(in[c * Q + q] - weight_of(q));
      else
        reinterpret_cast<uint16_t*>(raw.data())[k] =
            lbmh_f32_to_f16((float)((in[c * Q + q] - weight_of(q)) * f16_scale_of(q)));
    }
  }
  BCK(cudaMemcpyAsync(d.pdfs, raw.data(), raw.size(), cudaMemcpyHostToDevice, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  return 0;
}

int lbm_batch_set_launch(void* h, int which, int threads, int blocks) {
  Batch* b = static_cast<Batch*>(h);
  if (threads != 64 && threads != 128 && threads != 256) return -1;
  if (blocks < 0) return -1;
  lbm::BatchLaunch l{threads, lbm::kBatchTileNodes / threads, blocks};
  if (which == 0 || which == 2) b->evenL = l;
  if (which == 1 || which == 2) b->oddL = l;
  b->separate = true;
  drop_graphs(b);
  return 0;
}

void lbm_batch_get_launch(void* h, int* out6) {
  Batch* b = static_cast<Batch*>(h);
  out6[0] = b->evenL.threads;
  out6[1] = b->evenL.nodesPerThread;
  out6[2] = b->evenL.blocks;
  out6[3] = b->oddL.threads;
  out6[4] = b->oddL.nodesPerThread;
  out6[5] = b->oddL.blocks;
}

// Device time (ms) of nsteps steps of the active domains (CUDA events on the
// batch stream, direct launches).
int lbm_batch_time_steps(void* h, int nsteps, double* ms) {
  Batch* b = static_cast<Batch*>(h);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  BCK(cudaStreamSynchronize(b->stream));
  cudaEventRecord(e0, b->stream);
  int rc = enqueue(b, nsteps);
  cudaEventRecord(e1, b->stream);
  cudaEventSynchronize(e1);
  float f = 0.f;
  cudaEventElapsedTime(&f, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms = f;
  return rc;
}

// Autotuner: times each (block size, nodes per thread, grid) candidate --
// grids of 2..6 persistent blocks per SM, or one block per tile -- on the current batch for `trialSteps` steps, separately for the
// even and the odd kernel (each candidate runs whole even/odd pairs with the
// other kernel on its current setting), then fused pairs against the best of
// these where the batch has them, and keeps the fastest. Advances the domains
// by the trial steps. results (optional): rows of
// {which, threads, nodesPerThread, blocks, ms} for every candidate; returns the
// number of rows written (at most maxRows).
int lbm_batch_tune(void* h, int trialSteps, double* results, int maxRows) {
  Batch* b = static_cast<Batch*>(h);
  const int threadsC[3] = {256, 128, 64};
  const int perSM[6] = {0, 2, 3, 4, 5, 6};  // 0: one block per tile
  int rows = 0;
  const bool asked = b->separate;
  b->separate = true;
  for (int which = 0; which < 2; ++which) {
    double bestMs = 1e300;
    lbm::BatchLaunch best = which == 0 ? b->evenL : b->oddL;
    for (int ti = 0; ti < 3; ++ti)
      for (int pi = 0; pi < 6; ++pi) {
        lbm::BatchLaunch l{threadsC[ti], lbm::kBatchTileNodes / threadsC[ti], perSM[pi] * b->numSMs};
        if (which == 0) b->evenL = l; else b->oddL = l;
        double ms = 0.0;
        if (lbm_batch_time_steps(h, 2, &ms) != 0) continue;  // warm
        if (lbm_batch_time_steps(h, trialSteps, &ms) != 0) continue;
        if (results && rows < maxRows) {
          double* r = results + 5 * rows;
          r[0] = which; r[1] = l.threads; r[2] = l.nodesPerThread; r[3] = l.blocks; r[4] = ms;
        }
        ++rows;
        if (ms < bestMs) { bestMs = ms; best = l; }
      }
    if (which == 0) b->evenL = best; else b->oddL = best;
  }
  b->separate = asked;
  if (b->pair.nItems > 0) {
    // both steps of a pair in one launch against the best launches apart
    double apart = 0.0, fusedMs = 0.0;
    b->separate = true;
    bool timed = lbm_batch_time_steps(h, trialSteps, &apart) == 0;
    b->separate = false;
    timed = timed && lbm_batch_time_steps(h, 2, &fusedMs) == 0;  // warm
    timed = timed && lbm_batch_time_steps(h, trialSteps, &fusedMs) == 0;
    b->separate = timed ? apart < fusedMs : asked;
  }
  drop_graphs(b);
  return std::min(rows, maxRows);
}

int lbm_batch_checkpoint_save(void* h, int slot, const char* path) {
  Batch* b = static_cast<Batch*>(h);
  if (slot < 0 || slot >= b->maxSlots || !b->slots[slot].active) return -1;
  DomainSlot& d = b->slots[slot];
  std::vector<unsigned char> raw((size_t)d.dev.nCells * Q * b->elemBytes);
  BCK(cudaMemcpyAsync(raw.data(), d.pdfs, raw.size(), cudaMemcpyDeviceToHost, b->stream));
  const int rc = finish(b);
  if (rc) return rc;
  DomCkpt c = dom_header_of(b, d);
  c.checksum = dom_fnv1a64(raw.data(), raw.size());
  FILE* fh = std::fopen(path, "wb");
  if (!fh) { g_batchError = "cannot open the checkpoint file"; return -1; }
  const bool ok = std::fwrite(&c, sizeof(c), 1, fh) == 1 && std::fwrite(raw.data(), 1, raw.size(), fh) == raw.size();
  if (std::fclose(fh) != 0 || !ok) { g_batchError = "writing the checkpoint file failed"; return -1; }
  return 0;
}

int lbm_batch_checkpoint_load(void* h, int slot, const char* path) {
  Batch* b = static_cast<Batch*>(h);
  if (slot < 0 || slot >= b->maxSlots || !b->slots[slot].active) return -1;
  DomainSlot& d = b->slots[slot];
  FILE* fh = std::fopen(path, "rb");
  if (!fh) { g_batchError = "cannot open the checkpoint file"; return -1; }
  DomCkpt c;
  const DomCkpt want = dom_header_of(b, d);
  if (std::fread(&c, sizeof(c), 1, fh) != 1 || std::memcmp(c.magic, kDomMagic, 8) != 0) {
    std::fclose(fh);
    g_batchError = "not a domain checkpoint";
    return -2;
  }
  bool same = c.storage == want.storage && c.nFluid == want.nFluid && c.nCells == want.nCells &&
              c.omega == want.omega && c.lambda == want.lambda && c.xforce == want.xforce;
  for (int i = 0; i < 3; ++i) same = same && c.dims[i] == want.dims[i];
  if (!same) {
    std::fclose(fh);
    g_batchError = "the checkpoint belongs to a domain of another lattice, storage or relaxation";
    return -2;
  }
  std::vector<unsigned char> raw((size_t)d.dev.nCells * Q * b->elemBytes);
  const bool ok = std::fread(raw.data(), 1, raw.size(), fh) == raw.size();
  std::fclose(fh);
  if (!ok) { g_batchError = "the checkpoint file is truncated"; return -1; }
  if (dom_fnv1a64(raw.data(), raw.size()) != c.checksum) { g_batchError = "checkpoint checksum mismatch"; return -3; }
  BCK(cudaMemcpyAsync(d.pdfs, raw.data(), raw.size(), cudaMemcpyHostToDevice, b->stream));
  BCK(cudaStreamSynchronize(b->stream));
  return 0;
}

size_t lbm_batch_bytes_used(void* h) { return static_cast<Batch*>(h)->used; }
long long lbm_batch_launches(void* h) { return static_cast<Batch*>(h)->launches; }
int lbm_batch_active_domains(void* h) {
  Batch* b = static_cast<Batch*>(h);
  int n = 0;
  for (auto& s : b->slots) n += s.active ? 1 : 0;
  return n;
}
int lbm_batch_fluid_nodes(void* h, int slot) {
  Batch* b = static_cast<Batch*>(h);
  return (slot >= 0 && slot < b->maxSlots && b->slots[slot].active) ? b->slots[slot].dev.nFluid : -1;
}

}  // extern "C"
