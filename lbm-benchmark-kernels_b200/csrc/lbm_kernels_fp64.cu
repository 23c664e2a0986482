// lbm_kernels_fp64.cu -- FP64 D3Q19 TRT time-step kernels for sm_100a.
//
// Compiled with --fmad=false: every add and multiply rounds on its own, in the
// reference's scalar order (lbm_d3q19.cuh), so the PDFs are bit-identical to
// the reference's scalar CPU kernels.
//
// One thread per lattice cell (full array) or fluid node (lists). The work is
// HBM bound: a time step moves 19 PDFs in and 19 out per fluid node; no
// tensor-core path applies (the collision is not a contraction).
//
// Body force. The reference adds f_i += 3 w_i c_ix F to every logical PDF of a
// fluid node after each step (KernelAddBodyForce, src/Kernel.c:759-803) in a
// separate pass. Here the increment travels with the data instead:
//  * AA kernels: the even step stores plain post-collision values; the odd
//    step adds the increment of each PDF when it loads it (the logical
//    post-even PDF) and adds the increment of its destination when it stores
//    it (a PDF that bounces back becomes direction inv(i), so it gets the
//    increment of inv(i)). After every even/odd pair the device state equals
//    the reference's state bit for bit.
//  * pull kernel: the increment is added at the store.
// Obstacle cells are skipped in both AA steps. The reference relaxes them in
// its odd step and then overwrites what they wrote with the fix-up lists
// (src/BenchKernelD3Q19Aa.c:301-311,501-511); here periodic wraps and bounce
// back are resolved at the load/store itself, so no fix-up pass exists.
#include <algorithm>
#include <atomic>
#include <utility>
#include <vector>

#include "lbm_bulk.cuh"
#include "lbm_kernels.cuh"
#include "lbm_pair.cuh"

namespace lbm {

// ---------------------------------------------------------------------------
// Full array, AA pattern.

__device__ __forceinline__ int aa_cell(const AaArgs& a, int x, int y, int z) {
  return (x + 1) * a.xs + (y + 1) * a.pitch + z + kZOff;
}

// Offset of the neighbour in direction d, in cells.
__device__ __forceinline__ int aa_off(const AaArgs& a, int d) { return cx(d) * a.xs + cy(d) * a.pitch + cz(d); }

// Cell of x + c_d with every out-of-range coordinate wrapped (the reference
// wraps all crossed axes once one periodic axis is crossed,
// src/BenchKernelD3Q19AaCommon.c:522-578). Only called for links that do
// reach a fluid node, i.e. in-range or periodic ones.
__device__ __forceinline__ int aa_wrapped(const AaArgs& a, int x, int y, int z, int d) {
  int nx = x + cx(d), ny = y + cy(d), nz = z + cz(d);
  // across a halo face the neighbour slab's cell is mirrored in the ghost plane
  nx = nx < 0 ? (a.haloLo ? -1 : a.nX - 1) : (nx >= a.nX ? (a.haloHi ? a.nX : 0) : nx);
  ny = ny < 0 ? a.nY - 1 : (ny >= a.nY ? 0 : ny);
  nz = nz < 0 ? a.nZ - 1 : (nz >= a.nZ ? 0 : nz);
  return aa_cell(a, nx, ny, nz);
}

// A reversed link (bit set) is open when x + c_d leaves the domain only
// through non-periodic faces: the PDF then goes to the ghost layer, as in the
// reference, instead of bouncing back.
__device__ __forceinline__ bool aa_open(const AaArgs& a, int x, int y, int z, int d) {
  int nx = x + cx(d), ny = y + cy(d), nz = z + cz(d);
  // crossing a halo face leaves the lattice only where it is the periodic x boundary
  bool ox = (nx < 0 && (!a.haloLo || a.crossLo)) || (nx >= a.nX && (!a.haloHi || a.crossHi));
  bool oy = ny < 0 || ny >= a.nY, oz = nz < 0 || nz >= a.nZ;
  bool crossesPeriodic = (ox && a.perX) || (oy && a.perY) || (oz && a.perZ);
  return (ox || oy || oz) && !crossesPeriodic;
}

// One block per 256 z-cells of a row (longer contiguous segments per plane),
// 4 resident blocks per SM (64 registers): 0.816 ms against 0.824 ms for
// 128-cell blocks and 0.850 ms for 32 x 4 blocks at 256^3 on B200.
constexpr int kAaEvenBlock = 256;
__global__ void __launch_bounds__(kAaEvenBlock, 1024 / kAaEvenBlock) k_aa_even_fp64(const AaArgs a, const Trt<double> t) {
  const int z = blockIdx.x * kAaEvenBlock + threadIdx.x;
  const int y = blockIdx.y;
  const int x = blockIdx.z + a.xBase;
  if (z >= a.nZ || y >= a.nY) return;
  const int c = aa_cell(a, x, y, z);
  if (!(__ldg(a.link + c) & kFluidBit)) return;
  double* const f = a.f + c;
  double* const fs = launder(f);
  const long long S = a.dstride;
  // local collide; the post-collision PDF of direction d goes to slot inv(d)
  trt_update(t, [&](int d) { return f[d * S]; }, [&](int d, double v) { fs[inv(d) * S] = v; });
}

// Odd step. Node x reads its incoming f_i from slot (x + c_j, j), j = inv(i)
// (the AA pattern: the slots a node reads are the slots it writes), plus the
// body-force increment of that post-even logical PDF; it writes f_i to slot
// (x + c_i, i) with the increment of i, or -- bounced back at a wall -- to
// its own slot (x, inv(i)) with the increment of inv(i).
//
// Two launches share the step. The interior launch takes every cell whose
// links leave the domain, if at all, only through periodic faces
// (aa_interior_range): the z faces when z is periodic, and the x and y faces
// too when every axis is periodic and no x face is a halo face (then the
// face launch has no cells left). A link through such a face moves by a
// fixed -/+ n cells along each crossed axis. (Taking the periodic x faces of
// a channel, periodic in x only, into the interior saves nothing: the face
// launch still runs for its wall faces, and the interior pays for the wrap
// tests of two more axes -- 256^3 channel odd step 0.873 + 0.029 ms against
// 0.862 + 0.029 ms; on the fully periodic box the face launch goes away,
// 0.813 + 0.039 -> 0.824 ms.) Interior cells are sorted on the
// host by their link words: a cell without reversed links is "direct" (every
// address is the neighbour's slot), the others are "general" (each address
// is a select between the neighbour's slot and the node's own slot). The
// launch runs a list of work items in x-plane order: for each plane, the
// blocks (128 z-cells of one row) that hold at least one direct cell --
// these skip the general cells in them -- then chunks of 128 of the plane's
// general cells, one thread per cell. So the select-free path covers every
// direct cell, also those next to a wall (in a 256^3 channel a split by
// whole blocks sends 27 % of the cells, every block with one wall-adjacent
// cell, down the general path; the general cells are 1.6 %), and a general
// cell runs while the direct blocks of its plane touch the same 32-byte
// sectors, so its scattered accesses (a column of wall-adjacent cells is
// `pitch` apart) hit L2 instead of DRAM. Blocks without fluid cells are not
// launched. In both paths the 19 loads are issued together. The face kernel
// takes the shell (x and y faces, and z faces unless z is periodic):
// links that leave the domain wrap periodically on every crossed axis, or,
// at a non-periodic face, go to the ghost layer (an "open" link), as in the
// reference.
//
// Cells of different nodes never share a slot in the odd step (each node
// reads and writes only its own links' slots), so the work items and the
// two launches may run in any order.

// Interior blocks of the odd step: kAaBZ z-cells x kAaBY rows of one x plane
// (128 threads). A 128-cell row segment per plane: interior 0.811 ms against
// 0.818 ms for 64 x 2 and 0.830 ms for 32 x 4 blocks (256^3 fluid box, B200).
constexpr int kAaBZ = 128, kAaBY = 1;

// Whether the interior launch takes the whole lattice (see above).
__host__ __device__ __forceinline__ bool aa_interior_all(const AaArgs& a) {
  return a.perX && a.perY && a.perZ && !a.haloLo && !a.haloHi;
}

// The interior ranges [lo, hi] of x, y and z (see above).
struct AaRange {
  int x0, x1, y0, y1, z0, z1;
};
__host__ __device__ __forceinline__ AaRange aa_interior_range(const AaArgs& a) {
  AaRange r;
  const bool all = aa_interior_all(a);
  r.x0 = all ? 0 : 1;
  r.x1 = all ? a.nX - 1 : a.nX - 2;
  r.y0 = all ? 0 : 1;
  r.y1 = all ? a.nY - 1 : a.nY - 2;
  r.z0 = a.perZ ? 0 : 1;
  r.z1 = a.perZ ? a.nZ - 1 : a.nZ - 2;
  return r;
}

// Interior blocks start at z = 0 whatever the interior's first z: row
// element kZOff + z then puts each warp's 32 cells on whole 32-byte sectors
// (with walls in z, a start at z = 1 made every warp's z-aligned accesses
// span one sector more); threads off the interior range return.
__host__ __device__ __forceinline__ int aa_interior_zblocks(const AaArgs& a) { return (a.nZ + kAaBZ - 1) / kAaBZ; }

// Interior block `id` of the list: (bz, by, bx) with bz fastest.
__device__ __forceinline__ void aa_interior_block(const AaArgs& a, const AaRange& r, int id, int& z, int& y,
                                                  int& x) {
  const int gz = aa_interior_zblocks(a), gy = (r.y1 - r.y0 + 1 + kAaBY - 1) / kAaBY;
  const int bz = id % gz, rest = id / gz;
  z = bz * kAaBZ + threadIdx.x;
  y = r.y0 + (rest % gy) * kAaBY + threadIdx.y;
  x = r.x0 + rest / gy;
}

// The periodic wraps of an interior cell, decided once per cell: a link with
// c_a = -1 leaving through the low face of axis a moves +n_a cells along a,
// one with c_a = +1 through the high face moves -n_a. ZWrap: only z faces
// are reached (interior cells are off the x and y faces, and off the z faces
// unless z is periodic); XyzWrap: the interior is the whole lattice.
struct ZWrap {
  int down, up;
  __device__ __forceinline__ ZWrap(const AaArgs& a, int z)
      : down(z == 0 ? a.nZ : 0), up(z == a.nZ - 1 ? -a.nZ : 0) {}
  __device__ __forceinline__ int operator()(int d) const { return cz(d) < 0 ? down : (cz(d) > 0 ? up : 0); }
};
struct XyzWrap {
  const AaArgs& a;
  unsigned m;  // bits 0-5: x == 0, x == nX - 1, y == 0, y == nY - 1, z == 0, z == nZ - 1
  __device__ __forceinline__ XyzWrap(const AaArgs& a_, int x, int y, int z)
      : a(a_),
        m((x == 0) | (x == a_.nX - 1) << 1 | (y == 0) << 2 | (y == a_.nY - 1) << 3 | (z == 0) << 4 |
          (z == a_.nZ - 1) << 5) {}
  __device__ __forceinline__ int operator()(int d) const {
    int o = 0;
    if (cx(d) < 0 && (m & 1u)) o += a.nX * a.xs;
    if (cx(d) > 0 && (m & 2u)) o -= a.nX * a.xs;
    if (cy(d) < 0 && (m & 4u)) o += a.nY * a.pitch;
    if (cy(d) > 0 && (m & 8u)) o -= a.nY * a.pitch;
    if (cz(d) < 0 && (m & 16u)) o += a.nZ;
    if (cz(d) > 0 && (m & 32u)) o -= a.nZ;
    return o;
  }
};
template <bool kXY>
__device__ __forceinline__ auto aa_wrap(const AaArgs& a, int x, int y, int z) {
  if constexpr (kXY)
    return XyzWrap(a, x, y, z);
  else
    return ZWrap(a, z);
}

// A general cell (interior, fluid, at least one reversed link).
template <bool kXY>
__device__ __noinline__ void aa_odd_general_cell(const AaArgs& a, const Trt<double>& t, int c) {
  // cell index -> (x, y, z): planes of xs cells, rows of pitch cells,
  // interior z = 0 at element kZOff (x and y only matter to XyzWrap)
  int x = 0, y = 0, z;
  if constexpr (kXY) {
    const int rem = c % a.xs;
    x = c / a.xs - 1;
    y = rem / a.pitch - 1;
    z = rem % a.pitch - kZOff;
  } else {
    z = c % a.pitch - kZOff;
  }
  const uint32_t w = __ldg(a.link + c);
  double* const fb = a.f + c;
  const auto wrap = aa_wrap<kXY>(a, x, y, z);
  const int S = (int)a.dstride;
  auto load = [&](int d) -> double {
    if (d == DC) return fb[a.ldOff[DC]] + t.force[DC];
    const int j = inv(d);
    const bool rev = (w >> j) & 1u;
    return fb[rev ? d * S : a.ldOff[d] + wrap(j)] + t.force[d];
  };
  auto store = [&](int d, double v) {
    double* const fs = launder(fb);
    if (d == DC) {
      fs[a.stOff[DC]] = v + t.force[DC];
      return;
    }
    const int j = inv(d);
    const bool rev = (w >> d) & 1u;
    fs[rev ? j * S : a.stOff[d] + wrap(d)] = v + (rev ? t.force[j] : t.force[d]);
  };
  trt_update(t, load, store);
}

// Work item `items[blockIdx.x]`: >= 0 a block id (direct cells), < 0 the
// general-cell chunk ~item (cells[128 * chunk + thread], -1 = none).
// Launch bounds: 7 resident blocks of 128 threads per SM (measured fastest
// among 1-8 on B200; the general path spills a few values into L1 under that
// cap). Direct addresses are the cell's base pointer plus a per-direction
// offset from the parameter bank (and the periodic wraps), so no
// per-direction address stays live in registers; store addresses come from a
// laundered base pointer, apart from the load addresses, so those need not
// stay live across the collision.
template <bool kXY>
__global__ void __launch_bounds__(128, 7)
    k_aa_odd_interior_fp64(const __grid_constant__ AaArgs a, const __grid_constant__ Trt<double> t, const int* items,
                           const int* cells) {
  const int item = __ldg(items + blockIdx.x);
  if (item < 0) {
    const int c = __ldg(cells + (size_t)(~item) * 128 + threadIdx.y * kAaBZ + threadIdx.x);
    if (c >= 0) aa_odd_general_cell<kXY>(a, t, c);
    return;
  }
  const AaRange r = aa_interior_range(a);
  int x, y, z;
  aa_interior_block(a, r, item, z, y, x);
  if (z < r.z0 || z > r.z1 || y > r.y1) return;
  const int c = aa_cell(a, x, y, z);
  const uint32_t w = __ldg(a.link + c);
  if ((w & (kFluidBit | kLinkBits)) != kFluidBit) return;  // solid, or a general cell (own item)
  double* const fb = a.f + c;
  const auto wrap = aa_wrap<kXY>(a, x, y, z);
  trt_update(t, [&](int d) -> double { return fb[a.ldOff[d] + wrap(inv(d))] + t.force[d]; },
             [&](int d, double v) { launder(fb)[a.stOff[d] + wrap(d)] = v + t.force[d]; });
}

// Cell of shell index i: the x faces (all y, z), then the y faces (inner x,
// all z), then -- when z is not periodic -- the z faces (inner x and y). A
// one-cell-thin axis has a single face. The arithmetic is 32-bit unsigned:
// the layout holds fewer than 2^31 PDFs, so every product and index here is
// below 2^31.
__device__ __forceinline__ void aa_shell_cell(const AaArgs& a, long long i64, int& x, int& y, int& z) {
  const unsigned i = static_cast<unsigned>(i64);
  const unsigned nY = a.nY, nZ = a.nZ;
  const unsigned sx = a.nX > 1 ? 2 : 1, sy = a.nY > 1 ? 2 : 1;
  const unsigned mx = a.nX > 2 ? a.nX - 2 : 0, my = a.nY > 2 ? a.nY - 2 : 0;
  const unsigned nA = sx * nY * nZ, nB = sy * mx * nZ;
  if (i < nA) {
    x = (i / (nY * nZ)) == 0 ? 0 : a.nX - 1;
    const unsigned r = i % (nY * nZ);
    y = (int)(r / nZ);
    z = (int)(r % nZ);
  } else if (i < nA + nB) {
    const unsigned j = i - nA;
    y = (j / (mx * nZ)) == 0 ? 0 : a.nY - 1;
    const unsigned r = j % (mx * nZ);
    x = 1 + (int)(r / nZ);
    z = (int)(r % nZ);
  } else {
    const unsigned k = i - nA - nB;
    z = (k / (mx * my)) == 0 ? 0 : a.nZ - 1;
    const unsigned r = k % (mx * my);
    x = 1 + (int)(r / my);
    y = 1 + (int)(r % my);
  }
}

__global__ void __launch_bounds__(128) k_aa_odd_face_fp64(const AaArgs a, const Trt<double> t, long long nShell) {
  const long long i = static_cast<long long>(blockIdx.x) * 128 + threadIdx.x;
  if (i >= nShell) return;
  int x, y, z;
  aa_shell_cell(a, i, x, y, z);
  const int c = aa_cell(a, x, y, z);
  const uint32_t w = __ldg(a.link + c);
  if (!(w & kFluidBit)) return;
  const long long S = a.dstride;
  double* const f = a.f;
  auto load = [&](int d) -> double {
    if (d == DC) return f[DC * S + c] + t.force[DC];
    const int j = inv(d);
    const bool rev = (w >> j) & 1u;
    const bool open = rev && aa_open(a, x, y, z, j);
    const int nb = rev ? c + aa_off(a, j) : aa_wrapped(a, x, y, z, j);
    return f[(rev && !open) ? d * S + c : j * S + nb] + t.force[d];
  };
  auto store = [&](int d, double v) {
    if (d == DC) {
      f[DC * S + c] = v + t.force[DC];
      return;
    }
    const int j = inv(d);
    const bool rev = (w >> d) & 1u;
    if (!rev) {
      f[d * S + aa_wrapped(a, x, y, z, d)] = v + t.force[d];
    } else if (aa_open(a, x, y, z, d)) {
      // open face: the PDF leaves into the ghost layer; the node's own slot
      // of direction inv(d) keeps its even-step value and gets its increment
      f[d * S + c + aa_off(a, d)] = v;
      f[j * S + c] = f[j * S + c] + t.force[j];
    } else {
      f[j * S + c] = v + t.force[j];
    }
  };
  trt_update(t, load, store);
}

// ---------------------------------------------------------------------------
// The fused pair of a whole lattice (lbm_pair.cuh).

// The odd step of a warp of cells of which at least one has a reversed link:
// every address is a select between the neighbour's slot and the node's own.
struct NoWrap {
  __device__ __forceinline__ int operator()(int) const { return 0; }
};
template <class Wrap>
__device__ __forceinline__ void aa_odd_select(const AaArgs& a, const Trt<double>& t, int c, uint32_t w,
                                              const Wrap& wrap) {
  double* const fb = a.f + c;
  const int S = (int)a.dstride;
  auto load = [&](int d) -> double {
    if (d == DC) return fb[a.ldOff[DC]] + t.force[DC];
    const int j = inv(d);
    return fb[(w >> j) & 1u ? d * S : a.ldOff[d] + wrap(j)] + t.force[d];
  };
  auto store = [&](int d, double v) {
    double* const fs = launder(fb);
    if (d == DC) {
      __stcs(fs + a.stOff[DC], v + t.force[DC]);
      return;
    }
    const int j = inv(d);
    const bool rev = (w >> d) & 1u;
    __stcs(fs + (rev ? j * S : a.stOff[d] + wrap(d)), v + (rev ? t.force[j] : t.force[d]));
  };
  trt_update(t, load, store);
}

// The same on a lattice with open faces: a reversed link may also leave into
// the ghost layer, as in the face kernel.
__device__ __noinline__ void aa_odd_open_cell(const AaArgs& a, const Trt<double>& t, int c, int x, int y, int z,
                                              uint32_t w) {
  const long long S = a.dstride;
  double* const f = a.f;
  auto load = [&](int d) -> double {
    if (d == DC) return f[DC * S + c] + t.force[DC];
    const int j = inv(d);
    const bool rev = (w >> j) & 1u;
    const bool open = rev && aa_open(a, x, y, z, j);
    const int nb = rev ? c + aa_off(a, j) : aa_wrapped(a, x, y, z, j);
    return f[(rev && !open) ? d * S + c : j * S + nb] + t.force[d];
  };
  auto store = [&](int d, double v) {
    if (d == DC) {
      f[DC * S + c] = v + t.force[DC];
      return;
    }
    const int j = inv(d);
    const bool rev = (w >> d) & 1u;
    if (!rev) {
      f[d * S + aa_wrapped(a, x, y, z, d)] = v + t.force[d];
    } else if (aa_open(a, x, y, z, d)) {
      f[d * S + c + aa_off(a, d)] = v;
      f[j * S + c] = f[j * S + c] + t.force[j];
    } else {
      f[j * S + c] = v + t.force[j];
    }
  };
  trt_update(t, load, store);
}

__device__ __forceinline__ uint32_t fast_div(uint32_t n, const FastDiv& v) {
  return static_cast<uint32_t>((static_cast<uint64_t>(n) * v.mul) >> v.shift);
}

// Even position k -> x plane and first cell (in plane order) of its tile.
__device__ __forceinline__ void aa_pair_tile(const AaPairGeom& g, uint32_t k, uint32_t& x, uint32_t& cell0) {
  const uint32_t s = fast_div(k, g.byStrip);
  const uint32_t r = k - s * g.byStrip.d;
  const bool last = (s + 1) * g.J >= g.tpp;
  const uint32_t width = last ? g.byLast.d : g.J;
  x = last ? fast_div(r, g.byLast) : fast_div(r, g.byJ);
  cell0 = (s * g.J + r - x * width) * kListTile;
}

// The even step of cell c (link word w). The loads do not wait for the word
// (solid cells' slots exist; nothing is stored there).
__device__ __forceinline__ void aa_pair_even_cell(const AaArgs& a, const Trt<double>& t, int c, uint32_t w) {
  const double* const f = a.f + c;
  double* const fs = launder(a.f + c);
  const uint64_t keep = l2_keep_policy();
  const long long S = a.dstride;
  trt_update(t, [&](int d) { return __ldcs(f + d * S); },
             [&](int d, double v) {
               if (w & kFluidBit) st_keep(fs + inv(d) * S, v, keep);
             });
}

// What a warp's odd step has to provide for: any reversed link, any fluid cell
// on a face of the lattice.
struct AaWarpKind {
  bool wall, face;
};
__device__ __forceinline__ AaWarpKind aa_warp_kind(const AaArgs& a, int x, int y, int z, uint32_t w) {
  const bool fluid = w & kFluidBit;
  AaWarpKind k;
  k.wall = __any_sync(0xffffffffu, fluid && (w & kLinkBits));
  k.face = __any_sync(0xffffffffu, fluid && XyzWrap(a, x, y, z).m != 0u);
  return k;
}
__device__ __forceinline__ void aa_pair_odd_cell(const AaArgs& a, const Trt<double>& t, int c, int x, int y, int z,
                                                 uint32_t w, const AaWarpKind& kind, int openFaces) {
  if (!(w & kFluidBit)) return;
  if (!kind.wall) {
    double* const fb = a.f + c;
    const XyzWrap wrap(a, x, y, z);
    trt_update(t, [&](int d) -> double { return fb[a.ldOff[d] + wrap(inv(d))] + t.force[d]; },
               [&](int d, double v) { __stcs(launder(fb) + (a.stOff[d] + wrap(d)), v + t.force[d]); });
  } else if (!kind.face) {
    aa_odd_select(a, t, c, w, NoWrap());
  } else if (!openFaces) {
    aa_odd_select(a, t, c, w, XyzWrap(a, x, y, z));
  } else {
    aa_odd_open_cell(a, t, c, x, y, z, w);
  }
}

// One thread per cell of a tile of 256 consecutive cells of an x plane in
// (y, z) order, so that rows of any length fill the warps (64^3, whose 64-cell
// rows left half to three quarters of the threads of row-shaped blocks idle).
// A warp without reversed links takes the odd step by fixed offsets and the
// periodic wraps of its cells' positions (XyzWrap); a warp with any takes a
// selecting path for all its cells, without the wraps where none lies on a face
// of the lattice. Open faces have a path of their own, out of line. Channel 203
// x 190 x 197: 0.277 ms per step; one selecting path with the wraps 0.287; that
// path out of line 0.35; lists of the wall cells as a second pass 0.32 (two
// launches 0.412).
// Even loads do not wait for the link word that says whether the cell is
// fluid (solid cells' slots exist; nothing is stored there): 0.310 against
// 0.319 ms on that channel, 0.189 / 0.194 at 85 % fluid cells, 0.176 / 0.174
// at 40 %.
// 72 registers spill 52 bytes, more in the open-face function. Bound by L2
// requests and their latency as the list pair: 256^3 fluid box 0.818 -> 0.597 ms per step (28.1 GFLUP/s, half the HBM bytes), 64^3 channel
// 0.0220 -> 0.0106, 128 x 112 x 120 blocks, periodic, 0.101 -> 0.064.
__global__ void __launch_bounds__(kPairThreads, 3)
    k_aa_pair_fp64(const __grid_constant__ AaArgs a, const __grid_constant__ AaPairArgs q,
                   const __grid_constant__ Trt<double> t) {
  __shared__ PairShared<9, 4> sh;  // nothing staged
  pair_init(&sh);
  const uint32_t k = blockIdx.x;
  if (threadIdx.x >= kListTile) {
    pair_service(&sh, q.p, nullptr, a.err, k);
    return;
  }
  chain_wait();
  if (k < q.p.nTiles) {
    uint32_t x, i;
    aa_pair_tile(q.g, k, x, i);
    i += threadIdx.x;
    if (i < q.g.plane) {
      const uint32_t y = fast_div(i, q.g.byZ), z = i - y * q.g.byZ.d;
      const int c = aa_cell(a, x, y, z);
      aa_pair_even_cell(a, t, c, __ldg(a.link + c));
    }
    pair_even_done(&sh);
  }
  if (!pair_odd_named(&sh, a.err)) return;
  const uint32_t x = sh.item.extra, i = sh.item.tile + threadIdx.x;
  const uint32_t y = fast_div(i, q.g.byZ), z = i - y * q.g.byZ.d;
  const int c = aa_cell(a, x, y, z);
  const uint32_t w = i < q.g.plane ? __ldg(a.link + c) : 0u;
  const AaWarpKind kind = aa_warp_kind(a, x, y, z, w);
  if (pair_odd_turn(&sh, a.err)) aa_pair_odd_cell(a, t, c, x, y, z, w, kind, q.openFaces);
}

// Small lattices (lbm_pair.cuh): block b on tile b for all pairs of the launch.
__global__ void __launch_bounds__(kListTile, 3)
    k_aa_resident_fp64(const __grid_constant__ AaArgs a, const __grid_constant__ AaPairGeom g, int openFaces,
                       const __grid_constant__ ResidentArgs r, const __grid_constant__ Trt<double> t) {
  __shared__ int ok;
  chain_wait();
  uint32_t x, i;
  aa_pair_tile(g, blockIdx.x, x, i);
  i += threadIdx.x;
  const uint32_t y = fast_div(i, g.byZ), z = i - y * g.byZ.d;
  const int c = aa_cell(a, x, y, z);
  const uint32_t w = i < g.plane ? __ldg(a.link + c) : 0u;
  const AaWarpKind kind = aa_warp_kind(a, x, y, z, w);
  for (int p = 0; p < r.pairs; ++p) {
    if (i < g.plane) aa_pair_even_cell(a, t, c, w);
    if (!resident_meet(r, 2 * p + 1, a.err, &ok)) return;
    aa_pair_odd_cell(a, t, c, x, y, z, w, kind, openFaces);
    if (!resident_meet(r, 2 * p + 2, a.err, &ok)) return;
  }
}

// Two steps of a two-grid full-array row in one launch: the tiles, order and
// waits of the AA pair, the first step from grid f into g and the second back
// (k_list_two_fp64 says why, with the same 3/4 of the HBM traffic; tiles of
// consecutive cells fill the warps of short rows). ms per step, one launch each
// / one for two: pull 256^3 fluid box 0.891 / 0.749, 128 x 112 x 120 box 0.110 /
// 0.082, periodic blocks 0.132 / 0.088, 64^3 0.0205 / 0.0114; push 0.857 / 0.748,
// 0.100 / 0.079, 0.113 / 0.080, 0.0174 / 0.0112 (push with streaming loads 10 %
// slower). Warps with wall cells take one selecting path, wraps included.

// A warp with wall cells and open faces, as k_fa_push_fp64 and k_fa_pull_fp64.
template <bool kPush>
__device__ __noinline__ void fa_general_cell(const AaArgs& a, const Trt<double>& t, const double* f, double* g0, int c,
                                             int x, int y, int z, uint32_t w) {
  const long long S = a.dstride;
  double* const g = launder(g0);
  trt_update(t, [&](int d) -> double { return kPush ? f[d * S + c] : f[a.ldOff[d] + c]; },
             [&](int e, double v) {
               if (!kPush || e == DC) g[e * S + c] = v + t.force[e];
               if (e == DC) return;
               const int j = inv(e);
               const int n = c + aa_off(a, e);
               if (!((w >> e) & 1u)) {
                 const int q = aa_wrapped(a, x, y, z, e);
                 if (kPush)
                   g[e * S + q] = v + t.force[e];
                 else if (q != n)
                   g[e * S + q - aa_off(a, e)] = v + t.force[e];  // periodic image's ghost slot
               } else {
                 double* const s = g + j * S + (kPush ? c : n);
                 *s = (aa_open(a, x, y, z, e) ? *s : v) + t.force[j];
               }
             });
}

template <bool kPush, bool kLast>
__device__ __forceinline__ void fa_pair_cell(const AaArgs& a, const Trt<double>& t, const double* f, double* g, int c,
                                             int x, int y, int z, uint32_t w, int openFaces) {
  const AaWarpKind kind = aa_warp_kind(a, x, y, z, w);
  if (!(w & kFluidBit)) return;
  if (kind.wall && kind.face && openFaces) {
    fa_general_cell<kPush>(a, t, f, g, c, x, y, z, w);
    return;
  }
  const int S = (int)a.dstride;
  const double* const fb = f + c;
  const uint64_t keep = l2_keep_policy();
  auto put = [&](int o, double v) {
    double* const q = launder(g + c) + o;
    if (kLast)
      __stcs(q, v);
    else
      st_keep(q, v, keep);
  };
  auto load = [&](int d) -> double { return kPush ? fb[d * S] : fb[a.ldOff[d]]; };
  if (!kind.wall) {
    const XyzWrap wrap(a, x, y, z);
    trt_update(t, load, [&](int e, double v) {
      if (kPush) {
        put(a.stOff[e] + wrap(e), v + t.force[e]);
      } else {
        put(e * S, v + t.force[e]);
        const int o = wrap(e);
        if (o != 0) put(e * S + o, v + t.force[e]);  // periodic image's ghost slot
      }
    });
  } else {
    const XyzWrap wrap(a, x, y, z);
    trt_update(t, load, [&](int e, double v) {
      const int j = inv(e);
      const bool rev = e != DC && ((w >> e) & 1u);
      if (kPush) {
        put(rev ? j * S : a.stOff[e] + wrap(e), v + (rev ? t.force[j] : t.force[e]));
      } else {
        put(e * S, v + t.force[e]);
        if (rev) put(j * S + aa_off(a, e), v + t.force[j]);  // wall slot
        const int o = wrap(e);
        if (!rev && o != 0) put(e * S + o, v + t.force[e]);  // periodic image's ghost slot
      }
    });
  }
}

template <bool kPush>
__global__ void __launch_bounds__(kPairThreads, 3)
    k_fa_two_fp64(const __grid_constant__ AaArgs a, const __grid_constant__ AaPairArgs q,
                  const __grid_constant__ Trt<double> t) {
  __shared__ PairShared<9, 4> sh;  // nothing staged
  pair_init(&sh);
  const uint32_t k = blockIdx.x;
  if (threadIdx.x >= kListTile) {
    pair_service(&sh, q.p, nullptr, a.err, k);
    return;
  }
  chain_wait();
  if (k < q.p.nTiles) {
    uint32_t x, i;
    aa_pair_tile(q.g, k, x, i);
    i += threadIdx.x;
    const uint32_t y = fast_div(i, q.g.byZ), z = i - y * q.g.byZ.d;
    const int c = aa_cell(a, x, y, z);
    fa_pair_cell<kPush, false>(a, t, a.f, a.g, c, x, y, z, i < q.g.plane ? __ldg(a.link + c) : 0u,
                               q.openFaces);
    pair_even_done(&sh);
  }
  if (!pair_odd_named(&sh, a.err)) return;
  const uint32_t x = sh.item.extra, i = sh.item.tile + threadIdx.x;
  const uint32_t y = fast_div(i, q.g.byZ), z = i - y * q.g.byZ.d;
  const int c = aa_cell(a, x, y, z);
  const uint32_t w = i < q.g.plane ? __ldg(a.link + c) : 0u;
  if (pair_odd_turn(&sh, a.err)) fa_pair_cell<kPush, true>(a, t, a.g, a.f, c, x, y, z, w, q.openFaces);
}

static FastDiv fast_div_of(uint32_t d) {
  // ceil(log2 d) bits: exact for n < 2^31
  uint32_t l = 0;
  while ((1ull << l) < d) ++l;
  return FastDiv{d, static_cast<uint32_t>((1ull << (31 + l)) / d + 1), 31 + l};
}

// Strips: an odd tile needs the tiles of the neighbouring rows in three
// planes, so with whole planes one after the other the PDFs of two planes wait
// in L2. Planes of more than kWholePlane tiles go in strips of about
// kStripTiles tiles of each plane; a tile at a strip's edge needs the next
// strip and comes late (its PDFs are read again). Measured, ms per step
// (fluid boxes): 256 tiles per plane, whole 0.597, strips of 128 0.627, of 86
// 0.612; 352 tiles: 0.647, 0.690 (176), 0.662 (88); 625 tiles: 0.739, 0.711
// (209), 0.683 (90); 900: 0.770, 0.703 (225), 0.697 (90). Two launches: 0.818,
// 0.891, 0.946, 0.893.
constexpr uint32_t kWholePlane = 384, kStripTiles = 96;

AaPairGeom aa_pair_geom(const AaArgs& a) {
  AaPairGeom g;
  g.plane = static_cast<uint32_t>(a.nY) * static_cast<uint32_t>(a.nZ);
  g.tpp = (g.plane + kListTile - 1) / kListTile;
  g.nX = static_cast<uint32_t>(a.nX);
  // rows either side of a tile, in tiles: a strip is several times as wide
  const uint32_t halo = (2 * static_cast<uint32_t>(a.nZ) + kListTile) / kListTile;
  const uint32_t width = std::max(kStripTiles, 8 * halo);
  const uint32_t strips = g.tpp <= kWholePlane ? 1 : (g.tpp + width - 1) / width;
  g.J = (g.tpp + strips - 1) / strips;
  const uint32_t lastStrip = (g.tpp - 1) / g.J;
  g.byStrip = fast_div_of(g.J * g.nX);
  g.byJ = fast_div_of(g.J);
  g.byLast = fast_div_of(g.tpp - lastStrip * g.J);
  g.byZ = fast_div_of(static_cast<uint32_t>(a.nZ));
  return g;
}

void aa_pair_schedule(const AaArgs& a, const AaPairGeom& g, int margin, std::vector<AaPairItem>& items) {
  const uint32_t nTiles = g.nX * g.tpp, lastStrip = (g.tpp - 1) / g.J;
  const int shift = pair_group_shift(nTiles);
  auto width = [&](uint32_t s) { return s == lastStrip ? g.tpp - s * g.J : g.J; };
  auto position = [&](uint32_t x, uint32_t j) {
    const uint32_t s = j / g.J;
    return s * g.J * g.nX + x * width(s) + (j - s * g.J);
  };
  struct Range {
    uint32_t lo, hi;
  };
  std::vector<AaPairItem> work(nTiles);
  std::vector<uint32_t> need(nTiles), home(nTiles);
  std::vector<Range> reach, pos;
  for (uint32_t j = 0; j < g.tpp; ++j) {
    // tiles of a plane that the tile's cells reach in y and z, wrapping at the
    // plane's ends whether or not a link does; a link to the row before or
    // after may wrap in z, so up to two rows away, and split at strip ends
    reach.clear();
    auto add = [&](long long cell0, long long cell1) {
      const uint32_t t0 = (uint32_t)(cell0 / kListTile), t1 = (uint32_t)(cell1 / kListTile);
      for (uint32_t s = t0 / g.J; s <= t1 / g.J; ++s)
        reach.push_back({std::max(t0, s * g.J), std::min(t1, s * g.J + width(s) - 1)});
    };
    const long long n = g.plane, i0 = (long long)j * kListTile - 2LL * a.nZ;
    const long long i1 = std::min<long long>(n, (long long)(j + 1) * kListTile) - 1 + 2LL * a.nZ;
    if (i1 - i0 + 1 >= n) {
      add(0, n - 1);
    } else {
      add(std::max(i0, 0ll), std::min(i1, n - 1));
      if (i0 < 0) add(n + i0, n - 1);
      if (i1 >= n) add(0, i1 - n);
    }
    for (uint32_t x = 0; x < g.nX; ++x) {
      const uint32_t t = x * g.tpp + j;
      AaPairItem& it = work[t];
      it = AaPairItem{};
      it.tile = j * kListTile;
      it.extra = x;
      home[t] = position(x, j);
      pos.clear();
      for (uint32_t dx = 0; dx < 3; ++dx) {
        const uint32_t px = (x + g.nX + dx - 1) % g.nX;
        for (const Range& v : reach) {
          pos.push_back({position(px, v.lo) >> shift, position(px, v.hi) >> shift});
          need[t] = std::max(need[t], position(px, v.hi));
        }
      }
      std::sort(pos.begin(), pos.end(), [](const Range& u, const Range& v) { return u.lo < v.lo; });
      size_t m = 0;
      for (const Range& v : pos) {
        if (m && v.lo <= pos[m - 1].hi + 1)
          pos[m - 1].hi = std::max(pos[m - 1].hi, v.hi);
        else
          pos[m++] = v;
      }
      if (m > 9) {  // more pieces than a record holds: wait for every even tile
        m = 1;
        pos[0] = {0, (nTiles - 1) >> shift};
        need[t] = nTiles - 1;
      }
      for (size_t r = 0; r < m; ++r) {
        it.lo[r] = pos[r].lo;
        it.n[r] = pos[r].hi - pos[r].lo + 1;
      }
    }
  }
  pair_order(work, need, home, nTiles, static_cast<size_t>(margin), 0.0, items);
}

void fa_two_fp64(const AaArgs& a, const AaPairArgs& q, const Trt<double>& t, bool push, cudaStream_t s) {
  if (push)
    launch_chained(k_fa_two_fp64<true>, q.p.nItems, kPairThreads, 0, s, a, q, t);
  else
    launch_chained(k_fa_two_fp64<false>, q.p.nItems, kPairThreads, 0, s, a, q, t);
}

int aa_resident_tiles() {
  static std::atomic<int> n{0};
  return resident_tiles(n, k_aa_resident_fp64, kListTile, 2);
}

void aa_resident_fp64(const AaArgs& a, const AaPairGeom& g, int openFaces, const ResidentArgs& r,
                      const Trt<double>& t, cudaStream_t s) {
  launch_together(k_aa_resident_fp64, g.nX * g.tpp, kListTile, s, a, g, openFaces, r, t);
}

int aa_pair_resident() {
  static std::atomic<int> n{0};
  return prefetch_distance(n, k_aa_pair_fp64, kPairThreads, true);
}

void aa_pair_fp64(const AaArgs& a, const AaPairArgs& q, const Trt<double>& t, cudaStream_t s) {
  if (q.p.nItems > 0) launch_chained(k_aa_pair_fp64, q.p.nItems, kPairThreads, 0, s, a, q, t);
}

// ---------------------------------------------------------------------------
// x-slab halo messages.

// The 5 directions with c_x = +1 (E, NE, SE, TE, BE) and c_x = -1 (W, NW, SW,
// TW, BW), in the order of a message.
__device__ __forceinline__ int halo_dir(int k, bool plusX) {
  return plusX ? (k == 0 ? E : k == 1 ? NE : k == 2 ? SE : k == 3 ? TE : BE)
               : (k == 0 ? W : k == 1 ? NW : k == 2 ? SW : k == 3 ? TW : BW);
}

// plane: local x of the plane (-1 and nX are the ghost planes); plusX: which
// five directions; mode: 0 copy the slots into buf; 1 (phase-0 unpack into a
// ghost plane) and 2 (phase-1 unpack into a face plane) copy out of buf, but
// only into the slots the odd step exchanges through the face:
//  1: a ghost slot (g, y, z, d) is read and written by the face cell whose
//     direct link d lands on it, (y - c_dy, z - c_dz) wrapped on the face;
//     other ghost slots keep what they hold (open-face values);
//  2: a face slot (y, z, d) was written by the neighbour only if this slab's
//     cell reaches the neighbour's cell through the direct link inv(d); where
//     that link is reversed (a wall or an open face behind the halo face),
//     this slab's own odd step wrote the slot (bounce back) and keeps it.
__global__ void k_aa_halo(const AaArgs a, int plane, bool plusX, int mode, double* buf) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long face = (long long)a.nY * a.nZ;
  if (i >= 5 * face) return;
  const int k = (int)(i / face);
  const int y = (int)(i % face / a.nZ), z = (int)(i % a.nZ);
  const int d = halo_dir(k, plusX);
  const long long cell = (long long)(plane + 1) * a.xs + (long long)(y + 1) * a.pitch + z + kZOff;
  const long long slot = d * a.dstride + cell;
  if (mode == 0) {
    buf[i] = a.f[slot];
    return;
  }
  bool take;
  if (mode == 1) {
    const int rx = plane < 0 ? 0 : a.nX - 1;
    int ry = (y - cy(d)) % a.nY, rz = (z - cz(d)) % a.nZ;
    ry += ry < 0 ? a.nY : 0;
    rz += rz < 0 ? a.nZ : 0;
    const uint32_t w = a.link[(long long)(rx + 1) * a.xs + (long long)(ry + 1) * a.pitch + rz + kZOff];
    take = (w & kFluidBit) && !((w >> d) & 1u);
  } else {
    const uint32_t w = a.link[cell];
    take = (w & kFluidBit) && !((w >> inv(d)) & 1u);
  }
  if (take) a.f[slot] = buf[i];
}

// Side 1 (x = nX-1 face): the cells of this slab cross it with c_x = +1, the
// neighbour's with c_x = -1; side 0 the other way round.
void aa_halo_pack(const AaArgs& a, int side, int phase, double* buf, cudaStream_t s) {
  const long long n = 5LL * a.nY * a.nZ;
  const int plane = phase == 0 ? (side == 0 ? 0 : a.nX - 1) : (side == 0 ? -1 : a.nX);
  // phase 0: the face plane's slots the neighbour streams through (pointing
  // into this slab); phase 1: the ghost plane's slots this slab streamed into
  const bool plusX = phase == 0 ? side == 0 : side == 1;
  if (n > 0) k_aa_halo<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, plane, plusX, 0, buf);
}

void aa_halo_unpack(const AaArgs& a, int side, int phase, const double* buf, cudaStream_t s) {
  const long long n = 5LL * a.nY * a.nZ;
  const int plane = phase == 0 ? (side == 0 ? -1 : a.nX) : (side == 0 ? 0 : a.nX - 1);
  const bool plusX = phase == 0 ? side == 1 : side == 0;
  if (n > 0)
    k_aa_halo<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(a, plane, plusX, phase == 0 ? 1 : 2,
                                                           const_cast<double*>(buf));
}

// ---------------------------------------------------------------------------
// Two-grid full array (src/BenchKernelD3Q19.c:114-344) on the AA layout and
// link words, one thread per cell, obstacles skipped. The reference's
// bounce-back and periodic fix-up lists (src/BenchKernelD3Q19Common.c:
// 531-660), which copy slots after each step, and its body-force pass, which
// adds 3 w_i c_ix F through the logical node view, are folded into the
// stores; the result in every slot some fluid node views is the reference's
// bit for bit (tests against the oracle and the reference).

// Blocks of the two-grid steps: kFaBZ z-cells x kFaBY rows of one x plane.
// 32 x 4: push 0.860 / pull 0.897 ms at 256^3 (fluid box) against 0.867 /
// 0.925 for 64 x 2 and 0.887 / 0.986 for 128 x 1 (unlike the AA steps, whose
// longer row segments won).
constexpr int kFaBZ = 32, kFaBY = 4;

// Push: node x's own PDFs in from grid f; PDF d out to (x + c_d, d) of grid g
// (across a periodic face: the wrapped cell). A wall sends it back to the
// node's own slot inv(d); an open face leaves that slot untouched by the step,
// so only the force increment is added to what the grid held.
__global__ void __launch_bounds__(128) k_fa_push_fp64(const AaArgs a, const Trt<double> t) {
  chain_wait();
  const int z = blockIdx.x * kFaBZ + threadIdx.x;
  const int y = blockIdx.y * kFaBY + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= a.nZ || y >= a.nY) return;
  const int c = aa_cell(a, x, y, z);
  const uint32_t w = __ldg(a.link + c);
  if (!(w & kFluidBit)) return;
  const long long S = a.dstride;
  const double* const f = a.f + c;
  double* const g = launder(a.g);
  // a cell off every face with all links direct writes each PDF to x + c_d
  // without wrap or bounce logic (a warp-uniform branch for most warps)
  const bool inner = !(w & kLinkBits) && x > 0 && x < a.nX - 1 && y > 0 && y < a.nY - 1 && z > 0 && z < a.nZ - 1;
  if (inner) {
    trt_update(t, [&](int d) { return f[d * S]; },
               [&](int d, double v) { g[d * S + c + aa_off(a, d)] = v + t.force[d]; });
    return;
  }
  auto store = [&](int d, double v) {
    if (d == DC) {
      g[DC * S + c] = v + t.force[DC];
      return;
    }
    const int j = inv(d);
    if (!((w >> d) & 1u))
      g[d * S + aa_wrapped(a, x, y, z, d)] = v + t.force[d];
    else if (aa_open(a, x, y, z, d))
      g[j * S + c] = g[j * S + c] + t.force[j];
    else
      g[j * S + c] = v + t.force[j];
  };
  trt_update(t, [&](int d) { return f[d * S]; }, store);
}

// Pull: PDF d in from (x - c_d, d) of grid f (the slot the previous step
// filled for this node, ghost cells included); own PDFs out to grid g. For a
// link e that the next step pulls through a ghost or wall slot, the copy the
// reference's fix-up list makes is written directly: a wall slot (x + c_e,
// inv(e)) gets this node's PDF e (bounce back), the ghost slot of the periodic
// image q = wrap(x + c_e) gets it at (q - c_e, e), and an open slot only gets
// the force increment.
__global__ void __launch_bounds__(128) k_fa_pull_fp64(const AaArgs a, const Trt<double> t) {
  chain_wait();
  const int z = blockIdx.x * kFaBZ + threadIdx.x;
  const int y = blockIdx.y * kFaBY + threadIdx.y;
  const int x = blockIdx.z;
  if (z >= a.nZ || y >= a.nY) return;
  const int c = aa_cell(a, x, y, z);
  const uint32_t w = __ldg(a.link + c);
  if (!(w & kFluidBit)) return;
  const long long S = a.dstride;
  const double* const f = a.f;
  double* const g = launder(a.g);
  auto load = [&](int d) -> double { return f[d * S + c - aa_off(a, d)]; };
  // a cell off every face with all links direct has no periodic image, wall
  // or open-face slot to write: its 19 stores are its own slots (the check is
  // uniform across most warps; 0.946 -> 0.896 ms per step at 256^3)
  const bool inner = !(w & kLinkBits) && x > 0 && x < a.nX - 1 && y > 0 && y < a.nY - 1 && z > 0 && z < a.nZ - 1;
  if (inner) {
    trt_update(t, load, [&](int e, double v) { g[e * S + c] = v + t.force[e]; });
    return;
  }
  auto store = [&](int e, double v) {
    g[e * S + c] = v + t.force[e];
    if (e == DC) return;
    const int j = inv(e);
    if (!((w >> e) & 1u)) {
      const int q = aa_wrapped(a, x, y, z, e);
      const int n = c + aa_off(a, e);
      if (q != n) g[e * S + q - aa_off(a, e)] = v + t.force[e];  // periodic image's ghost slot
    } else if (aa_open(a, x, y, z, e)) {
      g[j * S + c + aa_off(a, e)] = g[j * S + c + aa_off(a, e)] + t.force[j];
    } else {
      g[j * S + c + aa_off(a, e)] = v + t.force[j];
    }
  };
  trt_update(t, load, store);
}

void fa_push_fp64(const AaArgs& a, const Trt<double>& t, cudaStream_t s) {
  launch_chained(k_fa_push_fp64, dim3((a.nZ + kFaBZ - 1) / kFaBZ, (a.nY + kFaBY - 1) / kFaBY, a.nX),
                 dim3(kFaBZ, kFaBY), 0, s, a, t);
}
void fa_pull_fp64(const AaArgs& a, const Trt<double>& t, cudaStream_t s) {
  launch_chained(k_fa_pull_fp64, dim3((a.nZ + kFaBZ - 1) / kFaBZ, (a.nY + kFaBY - 1) / kFaBY, a.nX),
                 dim3(kFaBZ, kFaBY), 0, s, a, t);
}

long long aa_shell_cells(const AaArgs& a) {
  const long long sx = a.nX > 1 ? 2 : 1, sy = a.nY > 1 ? 2 : 1, sz = a.nZ > 1 ? 2 : 1;
  const long long mx = a.nX > 2 ? a.nX - 2 : 0, my = a.nY > 2 ? a.nY - 2 : 0;
  return sx * a.nY * a.nZ + sy * mx * a.nZ + (a.perZ ? 0 : sz * mx * my);
}

bool aa_has_interior(const AaArgs& a) {
  const AaRange r = aa_interior_range(a);
  return r.x1 >= r.x0 && r.y1 >= r.y0 && r.z1 >= r.z0;
}

long long aa_interior_block_count(const AaArgs& a) {
  if (!aa_has_interior(a)) return 0;
  const AaRange r = aa_interior_range(a);
  return (long long)aa_interior_zblocks(a) * ((r.y1 - r.y0 + 1 + kAaBY - 1) / kAaBY) * (r.x1 - r.x0 + 1);
}

// Whether the face kernel has work: the shell (x and y faces, z faces unless
// z is periodic) lies outside the interior range unless the interior is the
// whole lattice.
bool aa_shell_needed(const AaArgs& a) { return !aa_interior_all(a) && aa_shell_cells(a) > 0; }

void aa_interior_items(const AaArgs& a, const uint32_t* link, std::vector<int>& items, std::vector<int>& cells) {
  items.clear();
  cells.clear();
  const long long n = aa_interior_block_count(a);
  if (n == 0) return;
  const AaRange r = aa_interior_range(a);
  const int gz = aa_interior_zblocks(a), gy = (r.y1 - r.y0 + 1 + kAaBY - 1) / kAaBY;
  const long long perPlane = (long long)gz * gy;
  auto word = [&](int x, int y, int z) { return link[(long long)(x + 1) * a.xs + (long long)(y + 1) * a.pitch + z + kZOff]; };
  for (int x = r.x0; x <= r.x1; ++x) {
    // the plane's blocks holding direct cells (block ids: bz fastest, then by, then x)
    for (long long k = 0; k < perPlane; ++k) {
      const int bz = (int)(k % gz), by = (int)(k / gz);
      bool direct = false;
      for (int ty = 0; ty < kAaBY && !direct; ++ty) {
        const int y = r.y0 + by * kAaBY + ty;
        if (y > r.y1) break;
        for (int tz = 0; tz < kAaBZ; ++tz) {
          const int z = bz * kAaBZ + tz;
          if (z < r.z0) continue;
          if (z > r.z1) break;
          if ((word(x, y, z) & (kFluidBit | kLinkBits)) == kFluidBit) { direct = true; break; }
        }
      }
      if (direct) items.push_back((int)((x - r.x0) * perPlane + k));
    }
    // then the plane's general cells in chunks of 128
    const size_t first = cells.size();
    for (int y = r.y0; y <= r.y1; ++y)
      for (int z = r.z0; z <= r.z1; ++z) {
        const uint32_t w = word(x, y, z);
        if ((w & kFluidBit) && (w & kLinkBits)) cells.push_back((x + 1) * a.xs + (y + 1) * a.pitch + z + kZOff);
      }
    while ((cells.size() - first) % 128) cells.push_back(-1);
    for (size_t c = first; c < cells.size(); c += 128) items.push_back(~(int)(c / 128));
  }
}

void aa_even_fp64(const AaArgs& a, const Trt<double>& t, cudaStream_t s) {
  AaArgs b = a;
  b.xBase = 0;
  k_aa_even_fp64<<<dim3((a.nZ + kAaEvenBlock - 1) / kAaEvenBlock, a.nY, a.nX), kAaEvenBlock, 0, s>>>(b, t);
}

void aa_even_fp64_planes(const AaArgs& a, const Trt<double>& t, int x0, int x1, cudaStream_t s) {
  if (x1 <= x0) return;
  AaArgs b = a;
  b.xBase = x0;
  k_aa_even_fp64<<<dim3((a.nZ + kAaEvenBlock - 1) / kAaEvenBlock, a.nY, x1 - x0), kAaEvenBlock, 0, s>>>(b, t);
}

void aa_odd_interior_fp64(const AaArgs& a, const Trt<double>& t, const int* items, int nItems, const int* cells,
                          cudaStream_t s) {
  if (nItems <= 0) return;
  if (aa_interior_all(a))
    k_aa_odd_interior_fp64<true><<<nItems, dim3(kAaBZ, kAaBY), 0, s>>>(a, t, items, cells);
  else
    k_aa_odd_interior_fp64<false><<<nItems, dim3(kAaBZ, kAaBY), 0, s>>>(a, t, items, cells);
}

void aa_odd_face_fp64(const AaArgs& a, const Trt<double>& t, cudaStream_t s) {
  const long long n = aa_shell_cells(a);
  if (n > 0) k_aa_odd_face_fp64<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(a, t, n);
}

// ---------------------------------------------------------------------------
// Fluid-node lists.

// 4 blocks of 256 threads per SM (64 registers, no spills)
__global__ void __launch_bounds__(kListTile, 4) k_list_even_fp64(const ListArgs a, const Trt<double> t) {
  chain_next();
  chain_wait();
  const int n = (blockIdx.x + a.tileBase) * kListTile + threadIdx.x;
  if (n >= a.nFluid) return;
  double* const f = a.f + n;
  double* const fs = launder(f);
  const long long S = a.nCells;
  trt_update(t, [&](int d) { return f[d * S]; }, [&](int d, double v) { fs[inv(d) * S] = v; });
}

// L2 prefetch of the PDF regions that the block of tile u will touch: for
// each of the 18 links, the 256 slots from the link of the tile's first node
// on (consecutive nodes mostly reach consecutive slots), and the tile's own
// rest-direction slots; one lane per region, clamped to the PDF array. The
// tile's run record was prefetched into L2 half a resident wave earlier.
__device__ __forceinline__ void prefetch_tile_pdfs(const ListArgs& a, unsigned u, int lane) {
  if (lane >= Q) return;
  const unsigned long long first =
      lane == DC ? (unsigned long long)DC * a.nCells + (unsigned long long)u * kListTile
                 : a.runs[(size_t)a.runOff[u] * 4 + kRunHdrWords + lane];
  const unsigned long long endB = (unsigned long long)Q * a.nCells * 8ull / 16ull * 16ull;
  const unsigned long long b0 = first * 8ull / 16ull * 16ull;
  if (b0 >= endB) return;
  unsigned long long len = kListTile * 8ull + 16ull;
  if (b0 + len > endB) len = endB - b0;
  if (len >= 16) bulk_prefetch_l2(reinterpret_cast<const char*>(a.f) + b0, static_cast<uint32_t>(len / 16 * 16));
}

// 3 blocks of 256 threads per SM. The adjacency comes run-compressed (one
// row per run of consecutive nodes, see kRunHdrWords): at the 256^3 sphere
// packing 0.49 rows per node, 35 instead of 72 bytes per node. The block's
// gathers are latency-bound at this occupancy (80 registers; a 64-register
// build spills and is slower), so warp 2 prefetches into L2 the PDF regions
// of the tile half a resident wave ahead (the run records are one wave
// ahead): 0.395 -> 0.371 ms at the 256^3 packing. Measured distances: one
// wave 0.386 ms, two waves 0.435, a quarter wave 0.377.
__global__ void __launch_bounds__(kListTile, 3) k_list_odd_fp64(const ListArgs a, const Trt<double> t) {
  __shared__ alignas(128) uint32_t srun[kRunTileWords];
  __shared__ alignas(8) uint64_t bar;
  __shared__ int ok;
  if (!stage_run_tile(a, srun, &bar, &ok)) return;
  const unsigned tile = blockIdx.x + static_cast<unsigned>(a.tileBase);
  const unsigned pdfAhead = static_cast<unsigned>(a.prefetch) / 2;
  if (threadIdx.x >= 64 && threadIdx.x < 96 && pdfAhead > 0 &&
      tile + pdfAhead < static_cast<unsigned>((a.nFluid + kListTile - 1) / kListTile))
    prefetch_tile_pdfs(a, tile + pdfAhead, threadIdx.x - 64);
  const int n = static_cast<int>(tile) * kListTile + threadIdx.x;
  if (n >= a.nFluid) return;
  uint32_t off;
  const uint32_t* e = run_row(srun, threadIdx.x, off);  // link d = e[d] + off
  double* const f = a.f;
  const long long S = a.nCells;

  // incoming f_d (the post-even logical PDF) through link inv(d), plus its
  // body-force increment
  auto load = [&](int d) -> double {
    return (d == DC ? f[DC * S + n] : f[e[inv(d)] + off]) + t.force[d];
  };
  // outgoing f_d through link d; a link that points back to the node itself
  // is a bounce back: the PDF becomes direction inv(d) of this node and gets
  // the increment of inv(d)
  auto store = [&](int d, double v) {
    if (d == DC) { f[DC * S + n] = v + t.force[DC]; return; }
    const uint32_t dst = reinterpret_cast<const volatile uint32_t*>(e)[d] + off;  // re-read: keeps no 64-bit addresses live across the collision
    const int j = inv(d);
    const bool bounce = dst == static_cast<uint32_t>(j * S + n);
    f[dst] = v + (bounce ? t.force[j] : t.force[d]);
  };
  trt_update(t, load, store);
}

// The two steps of node n in the fused kernels: the arithmetic of the two
// kernels above, with the cache hints of lbm_pair.cuh.
__device__ __forceinline__ void pair_even_node(const ListArgs& a, const Trt<double>& t, int n) {
  const long long S = a.nCells;
  const double* const f = a.f + n;
  double* const fs = launder(a.f + n);
  const uint64_t keep = l2_keep_policy();
  trt_update(t, [&](int d) { return __ldcs(f + d * S); },
             [&](int d, double v) { st_keep(fs + inv(d) * S, v, keep); });
}
__device__ __forceinline__ void pair_odd_node(const ListArgs& a, const Trt<double>& t, int n, const uint32_t* e,
                                              uint32_t off) {
  const long long S = a.nCells;
  double* const f = a.f;
  auto load = [&](int d) -> double { return (d == DC ? f[DC * S + n] : f[e[inv(d)] + off]) + t.force[d]; };
  auto store = [&](int d, double v) {
    if (d == DC) { __stcs(f + DC * S + n, v + t.force[DC]); return; }
    const uint32_t dst = reinterpret_cast<const volatile uint32_t*>(e)[d] + off;
    const int j = inv(d);
    const bool bounce = dst == static_cast<uint32_t>(j * S + n);
    __stcs(f + dst, v + (bounce ? t.force[j] : t.force[d]));
  };
  trt_update(t, load, store);
}

// The fused pair (lbm_pair.cuh). The parameters are read in place
// (__grid_constant__), which fits both steps into the 72 registers of 3 blocks of
// 288 threads per SM but for 16 bytes of spills. What bounds it: L2 and the
// fabric between its halves (the odd step's gathers and scatters touch 1.2-1.5 sectors per
// sector of payload; without any waiting the 256^3 packing would take 0.247 ms
// per step), then the waits.
__global__ void __launch_bounds__(kPairThreads, 3)
    k_list_pair_fp64(const __grid_constant__ ListArgs a, const __grid_constant__ PairArgs<3> p,
                     const __grid_constant__ Trt<double> t) {
  __shared__ ListPairShared sh;
  pair_init(&sh);
  const uint32_t k = blockIdx.x;
  if (threadIdx.x >= kListTile) {
    pair_service(&sh, p, a.runs, a.err, k);
    return;
  }
  chain_wait();
  if (k < p.nTiles) {
    const int n = static_cast<int>(k) * kListTile + threadIdx.x;
    if (n < a.nFluid) pair_even_node(a, t, n);
    pair_even_done(&sh);
  }
  if (!pair_odd_turn(&sh, a.err)) return;
  const int n = static_cast<int>(sh.item.tile) * kListTile + threadIdx.x;
  if (n >= a.nFluid) return;
  uint32_t off;
  const uint32_t* e = run_row(sh.run, threadIdx.x, off);
  pair_odd_node(a, t, n, e, off);
}

// Small domains (lbm_pair.cuh): block b on tile b for all pairs of the launch.
__global__ void __launch_bounds__(kListTile, 3)
    k_list_resident_fp64(const __grid_constant__ ListArgs a, const __grid_constant__ ResidentArgs r,
                         const __grid_constant__ Trt<double> t) {
  __shared__ alignas(128) uint32_t srun[kRunTileWords];
  __shared__ alignas(8) uint64_t bar;
  __shared__ int ok;
  if (!stage_run_tile(a, srun, &bar, &ok)) return;
  const int n = static_cast<int>(blockIdx.x) * kListTile + threadIdx.x;
  uint32_t off = 0;
  const uint32_t* e = run_row(srun, threadIdx.x, off);
  for (int p = 0; p < r.pairs; ++p) {
    if (n < a.nFluid) pair_even_node(a, t, n);
    if (!resident_meet(r, 2 * p + 1, a.err, &ok)) return;
    if (n < a.nFluid) pair_odd_node(a, t, n, e, off);
    if (!resident_meet(r, 2 * p + 2, a.err, &ok)) return;
  }
}

__global__ void __launch_bounds__(kListTile) k_list_pull_fp64(const ListArgs a, const Trt<double> t) {
  __shared__ alignas(128) uint32_t srun[kRunTileWords];
  __shared__ alignas(8) uint64_t bar;
  __shared__ int ok;
  if (!stage_run_tile(a, srun, &bar, &ok)) return;
  const int n = (blockIdx.x + a.tileBase) * kListTile + threadIdx.x;
  if (n >= a.nFluid) return;
  uint32_t off;
  const uint32_t* e = run_row(srun, threadIdx.x, off);  // link d = e[d] + off (run-compressed pull adjacency)
  const long long S = a.nCells;
  // one pass: the gathers are issued together and the 19 outputs are
  // contiguous stores to the second grid
  double f[Q], o[Q];
  f[DC] = a.f[DC * S + n];
#pragma unroll
  for (int d = 0; d < QM; ++d) f[d] = a.f[e[d] + off];
  trt_collide(t, f, o);
#pragma unroll
  for (int d = 0; d < Q; ++d) a.g[d * S + n] = o[d] + t.force[d];
}

// Two-grid list push (src/BenchKernelD3Q19List.c:114-320, PROP_MODEL_PUSH):
// the node's own 19 PDFs from the source grid, each post-collision PDF
// written through the push adjacency into the destination grid with the
// body-force increment of the slot's direction (a bounce back lands in the
// node's own slot inv(d) and gets the increment of inv(d)). The own PDFs do
// not depend on the adjacency: their loads are issued before the wait for
// the tile's run record, so the two latencies overlap.
__global__ void __launch_bounds__(kListTile, 3) k_list_push_fp64(const ListArgs a, const Trt<double> t) {
  __shared__ alignas(128) uint32_t srun[kRunTileWords];
  __shared__ alignas(8) uint64_t bar;
  __shared__ int ok;
  if (!stage_run_tile_issue(a, srun, &bar, &ok)) return;
  const int n = (blockIdx.x + a.tileBase) * kListTile + threadIdx.x;
  const long long S = a.nCells;
  double x[Q];
  if (n < a.nFluid) {
    const double* const f = a.f + n;
#pragma unroll
    for (int d = 0; d < Q; ++d) x[d] = f[d * S];
  }
  if (!stage_run_tile_wait(a, &bar) || n >= a.nFluid) return;
  uint32_t off;
  const uint32_t* e = run_row(srun, threadIdx.x, off);
  double* const g = a.g;
  auto store = [&](int d, double v) {
    if (d == DC) { g[DC * S + n] = v + t.force[DC]; return; }
    const uint32_t dst = reinterpret_cast<const volatile uint32_t*>(e)[d] + off;
    const int j = inv(d);
    const bool bounce = dst == static_cast<uint32_t>(j * S + n);
    g[dst] = v + (bounce ? t.force[j] : t.force[d]);
  };
  trt_update(t, [&](int d) { return x[d]; }, store);
}

// Two steps of a two-grid list row in one launch (lbm_pair.cuh): block k steps
// its first tile from grid f into grid g, then a tile two planes back from g
// into f once the first steps of all tiles that its links reach are done (they
// wrote the slots of g it reads and have read the slots of f it writes). The
// second step finds g in L2: per two steps HBM sees f read and written and g
// written, 3/4 of two launches' traffic. ms per step, one launch each / one for
// two: pull 256^3 packing 0.355 / 0.313, 160^3 0.0939 / 0.0770, 96^3 0.0268 /
// 0.0210; push 0.407 / 0.377, 0.1034 / 0.0910, 0.0284 / 0.0240. Loads ask for
// no early eviction: the second step overwrites the lines of f that the first
// one read, and a push into lines that have left L2 reads them back for the
// sectors it fills in part (push with streaming loads: 0.433 ms). Both tiles'
// run records are staged, in dynamic shared memory sized to the instance's
// largest record (the rest of the 256 KB holds the loads in flight).
template <bool kPush, bool kLast>
__device__ __forceinline__ void two_grid_node(const ListArgs& a, const Trt<double>& t, const double* src, double* dst,
                                              int n, const uint32_t* e, uint32_t off) {
  const long long S = a.nCells;
  const uint64_t keep = l2_keep_policy();
  auto put = [&](double* q, double v) {
    if (kLast)
      __stcs(q, v);
    else
      st_keep(q, v, keep);
  };
  auto load = [&](int d) -> double { return kPush || d == DC ? src[d * S + n] : src[e[d] + off]; };
  trt_update(t, load, [&](int d, double v) {
    if (!kPush || d == DC) {
      put(launder(dst) + d * S + n, v + t.force[d]);
      return;
    }
    const uint32_t to = reinterpret_cast<const volatile uint32_t*>(e)[d] + off;
    const int j = inv(d);
    const bool bounce = to == static_cast<uint32_t>(j * S + n);
    put(dst + to, v + (bounce ? t.force[j] : t.force[d]));
  });
}

template <bool kPush>
__global__ void __launch_bounds__(kPairThreads, 3)
    k_list_two_fp64(const __grid_constant__ ListArgs a, const __grid_constant__ PairArgs<3> p,
                    const __grid_constant__ Trt<double> t, uint32_t recordWords) {
  extern __shared__ __align__(128) uint32_t records[];
  __shared__ PairShared<3, 4> sh;
  pair_init(&sh);
  const uint32_t k = blockIdx.x;
  if (threadIdx.x >= kListTile) {
    pair_service(&sh, p, a.runs, a.err, k, records + recordWords, records);
    return;
  }
  if (k < p.nTiles) {
    const int n = static_cast<int>(k) * kListTile + threadIdx.x;
    const bool named = pair_named(&sh, a.err);  // the first tile's run record
    chain_wait();
    if (!named) return;
    if (n < a.nFluid) {
      uint32_t off;
      const uint32_t* e = run_row(records, threadIdx.x, off);
      two_grid_node<kPush, false>(a, t, a.f, a.g, n, e, off);
    }
    pair_even_done(&sh);
  } else {
    chain_wait();
  }
  if (!pair_odd_turn(&sh, a.err)) return;
  const int n = static_cast<int>(sh.item.tile) * kListTile + threadIdx.x;
  if (n >= a.nFluid) return;
  uint32_t off;
  const uint32_t* e = run_row(records + recordWords, threadIdx.x, off);
  two_grid_node<kPush, true>(a, t, a.g, a.f, n, e, off);
}

// Shared memory of the two records, each 128-byte aligned.
static uint32_t two_record_words(uint32_t recordBytes) { return (recordBytes + 127u) / 128u * 32u; }
template <bool kPush>
static size_t two_smem(uint32_t recordBytes) {
  // the opt-in is a per-device attribute, set once to the most any record needs
  // (concurrent first calls set the same value)
  constexpr int kMaxDevices = 64;
  static std::atomic<bool> set[kMaxDevices];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= kMaxDevices || !set[dev].load(std::memory_order_acquire)) {
    cudaFuncSetAttribute(k_list_two_fp64<kPush>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(2 * sizeof(uint32_t) * two_record_words(kRunTileWords * 4)));
    if (dev < kMaxDevices) set[dev].store(true, std::memory_order_release);
  }
  return 2 * sizeof(uint32_t) * two_record_words(recordBytes);
}

template <typename E>
__global__ void k_slot_gather(const E* __restrict__ f, const uint32_t* __restrict__ idx, long long n,
                              E* __restrict__ buf) {
  const long long k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) buf[k] = f[idx[k]];
}

template <typename E>
__global__ void k_slot_scatter(E* __restrict__ f, const uint32_t* __restrict__ idx, long long n,
                               const E* __restrict__ buf) {
  const long long k = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k < n) f[idx[k]] = buf[k];
}

template <typename E>
static void slot_move(bool gather, void* f, const uint32_t* idx, long long n, void* buf, cudaStream_t s) {
  const unsigned blocks = (unsigned)((n + 255) / 256);
  if (gather)
    k_slot_gather<E><<<blocks, 256, 0, s>>>(static_cast<const E*>(f), idx, n, static_cast<E*>(buf));
  else
    k_slot_scatter<E><<<blocks, 256, 0, s>>>(static_cast<E*>(f), idx, n, static_cast<const E*>(buf));
}

static void slot_move_bytes(bool gather, void* f, const uint32_t* idx, long long n, void* buf, int elemBytes,
                            cudaStream_t s) {
  if (n <= 0) return;
  if (elemBytes == 8)
    slot_move<unsigned long long>(gather, f, idx, n, buf, s);
  else if (elemBytes == 4)
    slot_move<unsigned int>(gather, f, idx, n, buf, s);
  else if (elemBytes == 2)
    slot_move<unsigned short>(gather, f, idx, n, buf, s);
}

void slot_gather(const void* f, const uint32_t* idx, long long n, void* buf, int elemBytes, cudaStream_t s) {
  slot_move_bytes(true, const_cast<void*>(f), idx, n, buf, elemBytes, s);
}

void slot_scatter(void* f, const uint32_t* idx, long long n, const void* buf, int elemBytes, cudaStream_t s) {
  slot_move_bytes(false, f, idx, n, const_cast<void*>(buf), elemBytes, s);
}

static unsigned list_blocks(const ListArgs& a) { return (a.nFluid + kListTile - 1) / kListTile; }

void list_even_fp64(const ListArgs& a, const Trt<double>& t, cudaStream_t s) {
  ListArgs b = a;
  b.tileBase = 0;
  if (a.nFluid > 0) launch_chained(k_list_even_fp64, list_blocks(b), kListTile, 0, s, b, t);
}

void list_even_fp64_tiles(const ListArgs& a, const Trt<double>& t, int t0, int t1, cudaStream_t s) {
  if (a.nFluid <= 0 || t1 <= t0) return;
  ListArgs b = a;
  b.tileBase = t0;
  launch_chained(k_list_even_fp64, (unsigned)(t1 - t0), kListTile, 0, s, b, t);
}
static std::atomic<int> g_oddAhead{0};

void list_odd_fp64(const ListArgs& a, const Trt<double>& t, cudaStream_t s) {
  if (a.nFluid <= 0) return;
  ListArgs b = a;
  b.tileBase = 0;
  b.prefetch = prefetch_distance(g_oddAhead, k_list_odd_fp64, kListTile, a.prefetch != 0);
  launch_chained(k_list_odd_fp64, list_blocks(b), kListTile, 0, s, b, t);
}

void list_odd_fp64_tiles(const ListArgs& a, const Trt<double>& t, int t0, int t1, cudaStream_t s) {
  if (a.nFluid <= 0 || t1 <= t0) return;
  ListArgs b = a;
  b.tileBase = t0;
  b.prefetch = prefetch_distance(g_oddAhead, k_list_odd_fp64, kListTile, a.prefetch != 0);
  launch_chained(k_list_odd_fp64, (unsigned)(t1 - t0), kListTile, 0, s, b, t);
}
void list_pair_fp64(const ListArgs& a, const PairArgs<3>& p, const Trt<double>& t, cudaStream_t s) {
  if (p.nItems > 0) launch_chained(k_list_pair_fp64, p.nItems, kPairThreads, 0, s, a, p, t);
}
void list_resident_fp64(const ListArgs& a, const ResidentArgs& r, const Trt<double>& t, cudaStream_t s) {
  ListArgs b = a;
  b.tileBase = 0;
  b.prefetch = 0;
  launch_together(k_list_resident_fp64, list_blocks(b), kListTile, s, b, r, t);
}
int list_resident_tiles_fp64() {
  static std::atomic<int> n{0};
  return resident_tiles(n, k_list_resident_fp64, kListTile, 2);
}
int list_pair_resident_fp64() {
  static std::atomic<int> n{0};
  return prefetch_distance(n, k_list_pair_fp64, kPairThreads, true);
}
int list_two_resident(bool push, uint32_t recordBytes) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (push)
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_list_two_fp64<true>, kPairThreads, two_smem<true>(recordBytes));
  else
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_list_two_fp64<false>, kPairThreads,
                                                  two_smem<false>(recordBytes));
  return sms * per;
}
void list_two_fp64(const ListArgs& a, const PairArgs<3>& p, const Trt<double>& t, bool push, uint32_t recordBytes,
                   cudaStream_t s) {
  const uint32_t words = two_record_words(recordBytes);
  if (push)
    launch_chained(k_list_two_fp64<true>, p.nItems, kPairThreads, two_smem<true>(recordBytes), s, a, p, t, words);
  else
    launch_chained(k_list_two_fp64<false>, p.nItems, kPairThreads, two_smem<false>(recordBytes), s, a, p, t, words);
}
void list_pull_fp64(const ListArgs& a, const Trt<double>& t, cudaStream_t s) {
  // no adjacency prefetch: with the full adjacency it slowed this kernel by
  // 8 % on a 256^3 sphere packing
  if (a.nFluid <= 0) return;
  ListArgs b = a;
  b.prefetch = 0;
  launch_chained(k_list_pull_fp64, list_blocks(b), kListTile, 0, s, b, t);
}
void list_push_fp64(const ListArgs& a, const Trt<double>& t, cudaStream_t s) {
  static std::atomic<int> ahead{0};
  if (a.nFluid <= 0) return;
  ListArgs b = a;
  b.prefetch = prefetch_distance(ahead, k_list_push_fp64, kListTile, a.prefetch != 0);
  launch_chained(k_list_push_fp64, list_blocks(b), kListTile, 0, s, b, t);
}

}  // namespace lbm
