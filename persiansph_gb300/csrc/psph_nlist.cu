// Per-step neighbour lists (replaces the candidate arrays SMPairs / FSMPairs /
// NSMPairs of MainNeighbourSearch, Source/Domain.cpp:808-945).
//
// Each particle scans the sorted ranges of its 3x3(x3) cell block once per step
// (the rows and x-slabs of it that can reach the support) and keeps the
// candidates inside the kernel support, tested in FP32 on
// (cell offset, FP32 offset) separations with a margin on r^2 (0.02 % for the
// FP32C form, 0.4 % for the FP64 form); the pair kernels then apply the exact
// test of their form. Lists are written in 16-byte chunks of 4 entries, chunk-
// major across particles (nl_index / nl_slot), so every store and every
// reader's load covers whole 32-byte sectors. The scan is cheap integer/FP32
// work; the pair kernels then walk lists of nearly equal length instead of
// branching per candidate.
//
// With one h everywhere and many particles (nlist_pair_kernel) a lane scans for two
// particles of one cell at once; otherwise (nlist_kernel) for one particle, and
// with few particles (nlist_cells_kernel) a lane takes one cell of one particle.
//
// Staged form (nlist_staged_kernel, one h everywhere, x not periodic): a block
// first copies the candidate positions of its particles' neighbour cells into
// shared memory with TMA bulk copies, then scans them there. The block's 256
// particles are consecutive in cell order, so they occupy one row of cells
// (or the end of one row and the start of the next); for each such home row
// and each of the 3 (2D) or 9 (3D) neighbouring rows, the cells within one of
// the home cells' x-range form one contiguous range of sorted particles: one
// bulk copy each. A block whose ranges do not fit the staging buffer, or
// whose particles span more rows or instances, scans global memory as before.
#include <algorithm>

#include "psph_pairs.cuh"
#include "psph_tma.cuh"

namespace psph {

namespace {

constexpr int kNT = 128;
constexpr int kOver = 4;  // a masked group reads up to 3 candidates past its cell's end: room behind the offsets

// Shared pieces of both scans. The 8-slot entry ring of a lane is
// lane-interleaved (slot s of lane l at ring[s][l], so the per-candidate
// stores are bank-conflict free); it holds the chunk being filled and the next
// one, and a completed chunk goes out as one 16-byte store.
struct ListWriter {
  int* rp;    // this lane's slot 0; slot s at rp[s * kNT]
  int4* out;  // the next chunk to write; chunk c of particle i at nl + c * stride + nl_slot(i)
  int k = 0;  // entries kept
  // the entry goes to the next free slot for every candidate and is kept (k
  // advances) only when the candidate is inside
  __device__ __forceinline__ void put(int e, bool in) {
    rp[(k & 7) * kNT] = e;
    k += in ? 1 : 0;
  }
  // after at most 4 candidates that started at count k0: the chunk k0 / 4, if
  // they completed it and it fits the capacity
  __device__ __forceinline__ void flush(int k0, int cap, int N) {
    if (((k0 ^ k) & 4) && k0 < cap) {
      const int b = (k0 & 4) * kNT;
      __stcs(out, make_int4(rp[b], rp[b + kNT], rp[b + 2 * kNT], rp[b + 3 * kNT]));
      out += N;
    }
  }
  __device__ __forceinline__ void finish(int cap, int* count) {
    if (k <= cap && (k & 3)) {  // last, partial chunk
      const int b = (k & 4) * kNT;
      __stcs(out, make_int4(rp[b], rp[b + kNT], rp[b + 2 * kNT], rp[b + 3 * kNT]));
    }
    *count = (k <= cap) ? k : -1;
  }
};

// Rows of cells and x-slabs of cells whose nearest point lies outside the
// support are skipped (cells are sorted slab by slab, xsub slabs along x).
// The bound assumes the in-cell offset lies in [0, cell size), which holds
// away from the grid faces (ListGenerate clamps only there); a neighbour
// cell's clamped particles lie beyond its outer face, farther than the slab
// they are counted in. Returns false when the row is out of reach, else the
// slabs in reach along x, counted from the first slab of the particle's cell.
__device__ __forceinline__ bool slab_reach(float ox, float gy, float gz, float thr_cull, float inv_sw, int* slo,
                                           int* shi) {
  const float rx2 = thr_cull - gy * gy - gz * gz;
  if (rx2 < 0.f) return false;
  const float rx = sqrtf(rx2);
  *slo = (int)floorf((ox - rx) * inv_sw - 1e-3f);
  *shi = (int)floorf((ox + rx) * inv_sw + 1e-3f);
  return true;
}

// One particle's list: the candidates of its 3x3(x3) cell block inside the
// support, tested in FP32 on (cell offset, FP32 offset) separations.
template <int DIM, bool UNIFORM_H>
__device__ __forceinline__ void list_one(const DevView& v, int i, float margin, int* rp) {
  const int cell = v.S.cellid[i];
  if (cell < 0) {
    v.S.nl_count[i] = 0;
    return;
  }
  const Persist& P = cur_persist(v);
  const PClass& C = v.cls[P.cls[i]];
  const GridDev& g = grid_of(v, C.inst);
  // a fixed particle's list holds free particles only (it has no other pairs)
  const bool fixed = !C.is_free && !v.o.list_all, free_half = fixed && v.o.xsub == 1, by_sign = fixed && !free_half;
  const float3 cs = cell_size_f(g);
  float4 oi = v.S.OFF32[i];
  oi.w = fabsf(oi.w);  // (its sign says whether the particle is fixed)
  const float cf = (float)g.cellfac;
  // support test r^2 <= (Cellfac hb)^2 margin; with one h everywhere it is a constant
  const float thr_u = cf * cf * oi.w * oi.w * margin;
  const int N = v.nl_stride, cap = v.o.nl_cap;
  const CellCoord c = decode(g, cell);
  const float4* __restrict__ off = v.S.OFF32;
  ListWriter w{rp, reinterpret_cast<int4*>(v.S.nl) + nl_slot(i)};
  const bool inner = c.x > 0 && c.x < g.nc[0] - 1 && c.y > 0 && c.y < g.nc[1] - 1 &&
                     (DIM == 2 || (c.z > 0 && c.z < g.nc[2] - 1));
  const bool cull = UNIFORM_H && inner;
  const float thr_cull = thr_u * 1.0001f;
  const int xs = v.o.xsub;
  const int* __restrict__ sstart = v.S.sstart;  // two bins per slab: its free, then its fixed particles
  const float inv_sw = (float)xs / cs.x;  // 1 / slab width
  const int zlo = (DIM == 3) ? -1 : 0, zhi = (DIM == 3) ? 1 : 0;
  for (int dz = zlo; dz <= zhi; ++dz) {
    int z = c.z + dz;
    if (g.periodic[2]) z = (z + g.nc[2]) % g.nc[2];
    else if (z < 0 || z >= g.nc[2]) continue;
    const float gz = (DIM == 3) ? (dz < 0 ? oi.z : (dz > 0 ? cs.z - oi.z : 0.f)) : 0.f;
    for (int dy = -1; dy <= 1; ++dy) {
      int y = c.y + dy;
      if (g.periodic[1]) y = (y + g.nc[1]) % g.nc[1];
      else if (y < 0 || y >= g.nc[1]) continue;
      const float gy = dy < 0 ? oi.y : (dy > 0 ? cs.y - oi.y : 0.f);
      const int base = g.cell_base + (z * g.nc[1] + y) * g.nc[0];
      const int cyz = (dy + 1) << 2 | (dz + 1) << 4;
      const float cy = -(float)dy * cs.y, cz = -(float)dz * cs.z;  // exact: dy, dz in {-1, 0, 1}
      int slo = -xs, shi = 2 * xs - 1;
      if (cull) {
        int lo_, hi_;
        if (!slab_reach(oi.x, gy, gz, thr_cull, inv_sw, &lo_, &hi_)) continue;
        slo = max(slo, lo_);
        shi = min(shi, hi_);
      }
      // the row's three cells in one walk, as in scan_two
      int lo0, hi0, lo1, hi1, lo2, hi2;
      auto range = [&](int dx, int& lo, int& hi) {
        lo = hi = 0;
        int x = c.x + dx;
        if (g.periodic[0]) x = (x + g.nc[0]) % g.nc[0];
        else if (x < 0 || x >= g.nc[0]) return;
        const int s0 = max(slo - dx * xs, 0), s1 = min(shi - dx * xs, xs - 1);
        if (s0 > s1) return;
        const unsigned bin = sort_bin(base + x, xs, s0);
        lo = sstart[bin];
        hi = sstart[free_half ? bin + 1 : sort_bin(base + x, xs, s1 + 1)];
      };
      range(-1, lo0, hi0);
      range(0, lo1, hi1);
      range(1, lo2, hi2);
      const bool home = dy == 0 && dz == 0;
      // i's position relative to a cell's origin: x_i - x_j = a - off_j (one
      // rounding away from rel_pos's form, which the pair kernels apply exactly;
      // the list's margin covers the difference)
      const float ay = oi.y + cy, az = oi.z + cz;
      float ax = oi.x + cs.x;
      int tag = (int)((unsigned)cyz << kCodeShift), cell_k = 0, j = lo0, end = hi0;
      auto next_cell = [&]() {
        while (j >= end && cell_k < 2) {
          ++cell_k;
          j = cell_k == 1 ? lo1 : lo2;
          end = cell_k == 1 ? hi1 : hi2;
          ax = cell_k == 1 ? oi.x : oi.x - cs.x;
          tag += 1 << kCodeShift;
        }
      };
      next_cell();
      while (j < end) {
        const int m = end - j;
        bool in[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 oj = off[j + e];  // (past the cell's end: another particle's, masked)
          const float x0 = ax - oj.x, x1 = ay - oj.y, x2 = az - oj.z;
          float d2 = __fmaf_rn(x1, x1, x0 * x0);
          if (DIM == 3) d2 = __fmaf_rn(x2, x2, d2);
          float thr = thr_u;
          if (!UNIFORM_H) {
            const float hb = 0.5f * (oi.w + fabsf(oj.w));
            thr = cf * cf * hb * hb * margin;
          }
          in[e] = d2 <= thr && m > e;
          if (home) in[e] = in[e] && j + e != i;
          if (by_sign) in[e] = in[e] && !(oj.w < 0.f);
        }
        const int k0 = w.k;
#pragma unroll
        for (int e = 0; e < 4; ++e) w.put((j + e) | tag, in[e]);
        w.flush(k0, cap, N);
        j += 4;
        if (j >= end) {
          j = end;
          next_cell();
        }
      }
    }
  }
  w.finish(cap, v.S.nl_count + i);
}

template <int DIM, bool UNIFORM_H>
__global__ void __launch_bounds__(kNT, 8) nlist_kernel(DevView v, float margin) {
  __shared__ int ring[8][kNT];
  if (v.sc->all_stop || !v.sc->rebuild) return;  // lists with a skin: kept from the last rebuild
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= v.sc->n) return;
  list_one<DIM, UNIFORM_H>(v, i, margin, &ring[0][threadIdx.x]);
}

// Few particles: 2^lg lanes to a particle, one cell of its block to a lane (9 of
// 16 lanes in 2D, 27 of 32 in 3D). A lane alone walks the cells one after the
// other, each of them a wait for its bounds and one for its candidates: 22 us for
// any number of particles up to 100k in 2D. Here the cells wait together; the
// lanes' hits, a bit each, get their places from a prefix over the group, in the
// same order. A cell with more candidates than bits sends its group's particle to
// the walk of one lane.
template <int DIM>
constexpr int kCellLanesLog2 = DIM == 2 ? 4 : 5;

template <int DIM, bool UNIFORM_H>
__global__ void __launch_bounds__(kNT) nlist_cells_kernel(DevView v, float margin) {
  __shared__ int ring[8][kNT];
  const StepScalars* sc = v.sc;
  if (sc->all_stop || !sc->rebuild) return;
  constexpr int L = 1 << kCellLanesLog2<DIM>, NC = DIM == 2 ? 9 : 27;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, sub = lane & (L - 1);
  const int i = (blockIdx.x * kNT + threadIdx.x) >> kCellLanesLog2<DIM>;
  const bool on = i < sc->n;
  const int cell = on ? v.S.cellid[i] : -1;
  unsigned long long hits = 0ull;
  int lo = 0, hi = 0, tag = 0;
  if (cell >= 0 && sub < NC) {
    const PClass& C = v.cls[cur_persist(v).cls[i]];
    const GridDev& g = grid_of(v, C.inst);
    const bool fixed = !C.is_free && !v.o.list_all;  // lists free particles only
    const CellCoord c = decode(g, cell);
    const int dx = sub % 3 - 1, dy = sub / 3 % 3 - 1, dz = DIM == 3 ? sub / 9 - 1 : 0;
    int q[3] = {c.x + dx, c.y + dy, c.z + dz};
    bool in = true;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      if (g.periodic[d]) q[d] = (q[d] + g.nc[d]) % g.nc[d];
      else in = in && q[d] >= 0 && q[d] < g.nc[d];
    }
    if (in) {
      const int b = g.cell_base + (q[2] * g.nc[1] + q[1]) * g.nc[0] + q[0];
      lo = v.S.start[b];
      hi = v.S.start[b + 1];
    }
    tag = (int)((unsigned)cell_code(dx, dy, dz) << kCodeShift);
    const float3 cs = cell_size_f(g);
    const float4 oi = v.S.OFF32[i];
    const float hi_ = fabsf(oi.w), cf = (float)g.cellfac;
    const float thr_u = cf * cf * hi_ * hi_ * margin;
    const float ax = oi.x - (float)dx * cs.x, ay = oi.y - (float)dy * cs.y, az = oi.z - (float)dz * cs.z;
    const int m = min(hi - lo, 64);
    for (int k0 = 0; k0 < m; k0 += 4) {
      unsigned four = 0u;
#pragma unroll
      for (int e = 0; e < 4; ++e) {  // (past the cell's end: another particle's, or the room behind the offsets)
        const int j = lo + k0 + e;
        const float4 oj = v.S.OFF32[j];
        const float x0 = ax - oj.x, x1 = ay - oj.y, x2 = az - oj.z;
        float d2 = __fmaf_rn(x1, x1, x0 * x0);  // the other walks' arithmetic
        if (DIM == 3) d2 = __fmaf_rn(x2, x2, d2);
        float thr = thr_u;
        if (!UNIFORM_H) {
          const float hb = 0.5f * (hi_ + fabsf(oj.w));
          thr = cf * cf * hb * hb * margin;
        }
        if (d2 <= thr && j < hi && j != i && !(fixed && oj.w < 0.f)) four |= 1u << e;
      }
      hits |= (unsigned long long)four << k0;
    }
  }
  const unsigned group = (L == 32 ? full : (1u << L) - 1u) << (lane - sub);
  const bool walk = __ballot_sync(full, hi - lo > 64) & group;
  int incl = __popcll(hits);
  const int own = incl;
#pragma unroll
  for (int o = 1; o < L; o <<= 1) {
    const int y = __shfl_up_sync(full, incl, o, L);
    if (sub >= o) incl += y;
  }
  const int total = __shfl_sync(full, incl, L - 1, L), cap = v.o.nl_cap;
  if (!on) return;
  if (walk) {
    if (sub == 0) list_one<DIM, UNIFORM_H>(v, i, margin, &ring[0][threadIdx.x]);
    return;
  }
  if (total <= cap)
    for (int k = incl - own; hits; hits &= hits - 1ull, ++k)
      v.S.nl[nl_index(v.nl_stride, i, k)] = (lo + __ffsll((long long)hits) - 1) | tag;
  if (sub == 0) v.S.nl_count[i] = total <= cap ? total : -1;
}

// Where the scan reads a candidate's FP32 offset: global memory, or the
// block's staged copy (row k of the lane's home row: smem index j + delta[k]).
struct GlobalCands {
  const float4* __restrict__ off;
  __device__ __forceinline__ void home(int) {}
  __device__ __forceinline__ void row(int) {}
  __device__ __forceinline__ float4 at(int j) const { return off[j]; }
};
template <int RPH>
struct StagedCands {
  uint32_t sbase;     // shared address of the staged offsets
  const int* delta;   // smem index - global index, per home row (2) x neighbour row (RPH)
  int row_a;          // the first home row (z * ny + y); the second is the next one
  int hsel = 0, d = 0;
  __device__ __forceinline__ void home(int r) { hsel = (r == row_a) ? 0 : RPH; }
  __device__ __forceinline__ void row(int k) { d = delta[hsel + k]; }
  __device__ __forceinline__ float4 at(int j) const { return tma::lds128(sbase + 16u * (uint32_t)(j + d)); }
};

template <int DIM, class Cands>
__device__ __forceinline__ void scan_two(const DevView& v, int ia, int n, float margin, Cands cand,
                                         int (*ring)[8][kNT]);

// One h everywhere: a lane builds the lists of sorted particles 2t and 2t+1
// when they share a cell. Both scan the same cell block, so each candidate is
// loaded once and tested against both, and the rows and slabs walked are the
// union of the two particles' reach. The odd particles whose cell starts at
// them (listed by the sort, nl_rest of them in S.rest) get a lane of their
// own in the first nr blocks of the grid, which the hardware starts first, so
// their scans run beside the pairs instead of after them.
template <int DIM>
__global__ void __launch_bounds__(kNT, 8) nlist_pair_kernel(DevView v, float margin, int nr) {
  __shared__ int ring[2][8][kNT];
  const StepScalars* sc = v.sc;
  if (sc->all_stop || !sc->rebuild) return;
  if ((int)blockIdx.x < nr) {
    const int m = min(sc->nl_rest, v.ncap);
    for (int q = blockIdx.x * kNT + threadIdx.x; q < m; q += nr * kNT)
      list_one<DIM, true>(v, v.S.rest[q], margin, &ring[0][0][threadIdx.x]);
    return;
  }
  const int n = sc->n;
  const int t = (blockIdx.x - nr) * kNT + threadIdx.x;
  scan_two<DIM>(v, 2 * t, n, margin, GlobalCands{v.S.OFF32}, ring);
}

// The two-particle scan of sorted particles ia and ia + 1 (one lane).
template <int DIM, class Cands>
__device__ __forceinline__ void scan_two(const DevView& v, int ia, int n, float margin, Cands cand,
                                         int (*ring)[8][kNT]) {
  const int ib = ia + 1;
  if (ia >= n) return;
  const int cell = v.S.cellid[ia];
  const int cellb = ib < n ? v.S.cellid[ib] : -1;
  const bool pair = cell >= 0 && cellb == cell;
  if (ib < n && cellb < 0) v.S.nl_count[ib] = 0;  // in no cell (sorted after every cell)
  if (cell < 0) {
    v.S.nl_count[ia] = 0;
    return;
  }
  const Persist& P = cur_persist(v);
  const PClass& C = v.cls[P.cls[ia]];
  const GridDev& g = grid_of(v, C.inst);
  // a fixed particle lists free candidates only: two fixed ones scan the free
  // half of each cell (one slab per cell), otherwise the candidates' signs tell
  const bool fixed_a = !C.is_free && !v.o.list_all;
  const bool fixed_b = pair ? !v.cls[P.cls[ib]].is_free && !v.o.list_all : fixed_a;
  const bool free_half = fixed_a && fixed_b && v.o.xsub == 1, by_sign = (fixed_a || fixed_b) && !free_half;
  const float3 cs = cell_size_f(g);
  // particle b far away when it is not paired: its tests always fail
  constexpr float kFar = 1e18f;
  const float4 oa = v.S.OFF32[ia];
  const float4 ob = pair ? v.S.OFF32[ib] : make_float4(kFar, kFar, kFar, oa.w);
  const float cf = (float)g.cellfac;
  const float thr = cf * cf * oa.w * oa.w * margin;
  const int N = v.nl_stride, cap = v.o.nl_cap;
  const CellCoord c = decode(g, cell);
  cand.home(c.z * g.nc[1] + c.y);
  int4* const nl4 = reinterpret_cast<int4*>(v.S.nl);
  ListWriter wa{&ring[0][0][threadIdx.x], nl4 + nl_slot(ia)};
  ListWriter wb{&ring[1][0][threadIdx.x], nl4 + nl_slot(ib)};
  const int zlo_ = (DIM == 3) ? -1 : 0;
  const bool cull = c.x > 0 && c.x < g.nc[0] - 1 && c.y > 0 && c.y < g.nc[1] - 1 &&
                    (DIM == 2 || (c.z > 0 && c.z < g.nc[2] - 1));
  const float thr_cull = thr * 1.0001f;
  const int xs = v.o.xsub;
  const int* __restrict__ sstart = v.S.sstart;  // two bins per slab: its free, then its fixed particles
  const float inv_sw = (float)xs / cs.x;
  const float2 AXm = make_float2(oa.x + cs.x, ob.x + cs.x), AX0 = make_float2(oa.x, ob.x),
               AXp = make_float2(oa.x - cs.x, ob.x - cs.x);
  const int zlo = (DIM == 3) ? -1 : 0, zhi = (DIM == 3) ? 1 : 0;
  for (int dz = zlo; dz <= zhi; ++dz) {
    int z = c.z + dz;
    if (g.periodic[2]) z = (z + g.nc[2]) % g.nc[2];
    else if (z < 0 || z >= g.nc[2]) continue;
    const float gza = (DIM == 3) ? (dz < 0 ? oa.z : (dz > 0 ? cs.z - oa.z : 0.f)) : 0.f;
    const float gzb = (DIM == 3) ? (dz < 0 ? ob.z : (dz > 0 ? cs.z - ob.z : 0.f)) : 0.f;
    for (int dy = -1; dy <= 1; ++dy) {
      int y = c.y + dy;
      if (g.periodic[1]) y = (y + g.nc[1]) % g.nc[1];
      else if (y < 0 || y >= g.nc[1]) continue;
      const float gya = dy < 0 ? oa.y : (dy > 0 ? cs.y - oa.y : 0.f);
      const float gyb = dy < 0 ? ob.y : (dy > 0 ? cs.y - ob.y : 0.f);
      const int base = g.cell_base + (z * g.nc[1] + y) * g.nc[0];
      const int cyz = (dy + 1) << 2 | (dz + 1) << 4;
      const float cy = -(float)dy * cs.y, cz = -(float)dz * cs.z;
      cand.row(3 * (dz - zlo_) + (dy + 1));
      int slo = -xs, shi = 2 * xs - 1;
      if (cull) {  // the union of the two particles' reach
        int la, ha, lb, hb;
        const bool ra = slab_reach(oa.x, gya, gza, thr_cull, inv_sw, &la, &ha);
        const bool rb = pair && slab_reach(ob.x, gyb, gzb, thr_cull, inv_sw, &lb, &hb);
        if (!ra && !rb) continue;
        if (!ra) la = lb, ha = hb;
        else if (rb) la = min(la, lb), ha = max(ha, hb);
        slo = max(slo, la);
        shi = min(shi, ha);
      }
      // The row's three cells as candidate ranges, walked in one loop: the lanes
      // of a warp lie in neighbouring cells of one row, whose sums over three cells
      // are nearly equal where the single cells' counts are not (a lattice puts two
      // or three planes into a cell's width). A group of 4 candidates never spans
      // two cells; the last one of a cell is partly masked. Bound by issue slots:
      // with a loop per cell 21 of 32 lanes were active (1.0M particles in 3D: 420 us,
      // this walk 360; 177k: 143, now 110).
      int lo0, hi0, lo1, hi1, lo2, hi2;
      auto range = [&](int dx, int& lo, int& hi) {
        lo = hi = 0;
        int x = c.x + dx;
        if (g.periodic[0]) x = (x + g.nc[0]) % g.nc[0];
        else if (x < 0 || x >= g.nc[0]) return;
        const int s0 = max(slo - dx * xs, 0), s1 = min(shi - dx * xs, xs - 1);
        if (s0 > s1) return;
        const unsigned bin = sort_bin(base + x, xs, s0);
        lo = sstart[bin];
        hi = sstart[free_half ? bin + 1 : sort_bin(base + x, xs, s1 + 1)];
      };
      range(-1, lo0, hi0);
      range(0, lo1, hi1);
      range(1, lo2, hi2);
      const bool home = dy == 0 && dz == 0;  // neither particle lists itself
      const float2 AY = make_float2(oa.y + cy, ob.y + cy), AZ = make_float2(oa.z + cz, ob.z + cz);
      const float2 M1 = make_float2(-1.f, -1.f);
      float2 AX = AXm;
      int tag = (int)((unsigned)cyz << kCodeShift), cell_k = 0, j = lo0, end = hi0;
      auto next_cell = [&]() {
        while (j >= end && cell_k < 2) {
          ++cell_k;
          j = cell_k == 1 ? lo1 : lo2;
          end = cell_k == 1 ? hi1 : hi2;
          AX = cell_k == 1 ? AX0 : AXp;
          tag += 1 << kCodeShift;
        }
      };
      next_cell();
      while (j < end) {
        const int m = end - j;  // candidates left in the cell
        bool ia_[4], ib_[4];
        float w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // both particles' separations in packed FP32x2 arithmetic: a - off_j
          // as fma(off_j, -1, a) (one rounding, the subtraction's), then the
          // squared distances, one instruction for both particles' values
          const float4 oj = cand.at(j + e);  // (past the cell's end: another particle's, masked)
          const float2 ex = __ffma2_rn(make_float2(oj.x, oj.x), M1, AX);
          const float2 ey = __ffma2_rn(make_float2(oj.y, oj.y), M1, AY);
          float2 d2 = __fmul2_rn(ex, ex);
          d2 = __ffma2_rn(ey, ey, d2);
          if (DIM == 3) {
            const float2 ez = __ffma2_rn(make_float2(oj.z, oj.z), M1, AZ);
            d2 = __ffma2_rn(ez, ez, d2);
          }
          ia_[e] = d2.x <= thr && m > e;
          ib_[e] = d2.y <= thr && m > e;
          w[e] = oj.w;
        }
        if (home) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ia_[e] = ia_[e] && j + e != ia;
            ib_[e] = ib_[e] && j + e != ib;
          }
        }
        if (by_sign) {  // fixed particles among the candidates of a fixed one (their h is negative)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            ia_[e] = ia_[e] && !(fixed_a && w[e] < 0.f);
            ib_[e] = ib_[e] && !(fixed_b && w[e] < 0.f);
          }
        }
        const int ka = wa.k, kb = wb.k;
#pragma unroll
        for (int e = 0; e < 4; ++e) wa.put((j + e) | tag, ia_[e]);
#pragma unroll
        for (int e = 0; e < 4; ++e) wb.put((j + e) | tag, ib_[e]);
        wa.flush(ka, cap, N);
        wb.flush(kb, cap, N);
        j += 4;
        if (j >= end) {
          j = end;
          next_cell();
        }
      }
    }
  }
  wa.finish(cap, v.S.nl_count + ia);
  if (pair) wb.finish(cap, v.S.nl_count + ib);
}

// Staged form of nlist_pair_kernel (see the file header). Warp 0 plans the
// block's copies: the home rows of its particles and, per home row and
// neighbour row, the sorted range of the cells within one of the home cells'
// x-range; lane 0 arms the mbarrier with the total bytes and each planning lane
// issues its range's bulk copy. Every thread waits for the copies with a time
// limit; a thread whose wait gives up sets ST_STAGE_TIMEOUT, scans global
// memory instead, and waits again (bounded) before the block exits, so no copy
// lands in shared memory the block no longer owns.
constexpr unsigned long long kStageWaitNs = 1000000000ull;

template <int DIM>
__global__ void __launch_bounds__(kNT, 4) nlist_staged_kernel(DevView v, float margin, int nr, int cap_stage) {
  constexpr int RPH = (DIM == 3) ? 9 : 3;  // neighbour rows per home row
  __shared__ int ring[2][8][kNT];
  __shared__ int s_delta[2 * RPH];
  __shared__ int s_row_a, s_mode;
  __shared__ __align__(8) uint64_t s_bar;
  extern __shared__ float4 s_off[];
  StepScalars* sc = v.sc;
  if (sc->all_stop || !sc->rebuild) return;
  if ((int)blockIdx.x < nr) {
    const int m = min(sc->nl_rest, v.ncap);
    for (int q = blockIdx.x * kNT + threadIdx.x; q < m; q += nr * kNT)
      list_one<DIM, true>(v, v.S.rest[q], margin, &ring[0][0][threadIdx.x]);
    return;
  }
  const int n = sc->n;
  const int b = blockIdx.x - nr;
  const int p0 = 2 * b * kNT;
  if (threadIdx.x == 0) {
    tma::mbar_init(&s_bar, 1);
    tma::mbar_init_fence();
  }
  // plan (warp 0): lane q < nh * RPH owns the range of home row q / RPH and
  // neighbour row q % RPH
  int seg_lo = 0, cnt = 0, off = 0, total = 0;
  if (threadIdx.x < 32) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x;
    const int last = min(p0 + 2 * kNT, min(n, sc->n_cells)) - 1;
    bool ok = p0 <= last;
    const int ca = ok ? v.S.cellid[p0] : -1, cl = ok ? v.S.cellid[last] : -1;
    ok = ok && ca >= 0 && cl >= 0;
    const Persist& P = cur_persist(v);
    const int inst = ok ? v.cls[P.cls[p0]].inst : 0;
    ok = ok && v.cls[P.cls[last]].inst == inst;
    const GridDev& g = grid_of(v, inst);
    ok = ok && !g.periodic[0];
    const CellCoord A = decode(g, ok ? ca : g.cell_base), L = decode(g, ok ? cl : g.cell_base);
    const int ra = A.z * g.nc[1] + A.y, rl = L.z * g.nc[1] + L.y;
    const int nh = (rl == ra) ? 1 : (rl == ra + 1 ? 2 : 0);
    ok = ok && nh > 0;
    if (ok && lane < nh * RPH) {
      const int h = lane / RPH, k = lane % RPH;
      const int hy = h ? L.y : A.y, hz = h ? L.z : A.z;
      const int xlo = h ? 0 : A.x, xhi = (nh == 1 || h) ? L.x : g.nc[0] - 1;
      const int dz = (DIM == 3) ? k / 3 - 1 : 0, dy = k % 3 - 1;
      int y = hy + dy, z = hz + dz;
      bool in = true;
      if (g.periodic[1]) y = (y + g.nc[1]) % g.nc[1];
      else if (y < 0 || y >= g.nc[1]) in = false;
      if (g.periodic[2]) z = (z + g.nc[2]) % g.nc[2];
      else if (z < 0 || z >= g.nc[2]) in = false;
      if (in) {
        const int base = g.cell_base + (z * g.nc[1] + y) * g.nc[0];
        seg_lo = v.S.start[base + max(xlo - 1, 0)];
        cnt = v.S.start[base + min(xhi + 1, g.nc[0] - 1) + 1] - seg_lo;
      }
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(full, incl, o);
      if (lane >= o) incl += y;
    }
    total = __shfl_sync(full, incl, 31);
    off = incl - cnt;
    ok = ok && total > 0 && total <= cap_stage;
    if (lane < 2 * RPH) s_delta[lane] = off - seg_lo;
    if (lane == 0) {
      s_row_a = ra;
      s_mode = ok;
    }
    if (!ok) cnt = 0;
  }
  __syncthreads();  // the plan and the initialised mbarrier
  const bool staged = s_mode;
  const uint32_t sbase = tma::smem_u32(s_off);
  if (staged && threadIdx.x < 32) {
    if (threadIdx.x == 0) tma::mbar_expect_tx(&s_bar, 16u * (uint32_t)total);
    __syncwarp();
    if (cnt > 0) tma::bulk_g2s(sbase + 16u * (uint32_t)off, v.S.OFF32 + seg_lo, 16u * (uint32_t)cnt, &s_bar);
  }
  bool use_stage = staged;
  if (staged && !tma::mbar_wait_bounded(&s_bar, 0, kStageWaitNs)) {
    atomicOr(&sc->status, ST_STAGE_TIMEOUT);
    use_stage = false;
  }
  const int t = b * kNT + threadIdx.x;
  if (use_stage) scan_two<DIM>(v, 2 * t, n, margin, StagedCands<RPH>{sbase, s_delta, s_row_a}, ring);
  else scan_two<DIM>(v, 2 * t, n, margin, GlobalCands{v.S.OFF32}, ring);
  if (staged && !use_stage) tma::mbar_wait_bounded(&s_bar, 0, kStageWaitNs);
}

// Deepest staging (Options::nlist_stage): 64 KB of FP32 offsets per block
// (one home row of ~256 particles and its neighbour rows take ~2,600 in the
// 3D dam break).
constexpr int kStageCapMax = 4096;

}  // namespace

void nlist_configure() {
  const int bytes = (kStageCapMax + kOver) * (int)sizeof(float4);
  cudaFuncSetAttribute(nlist_staged_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  cudaFuncSetAttribute(nlist_staged_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

void launch_nlist(const DevView& v, cudaStream_t st) {
  // a superset of the support: the pair kernels apply the exact test (FP32 in
  // the FP32C form, FP64 in the plain form)
  // with a skin s the lists hold every pair within (1 + s) of the support
  const float margin = v.o.fp32 ? 1.0002f * (1.f + v.o.skin) * (1.f + v.o.skin) : 1.004f;
  // A lane to a cell while the lanes of all particles fit the SMs at once (2,048
  // an SM): 920 particles in 2D 10 us against 24, 5k 8 and 21; with 86k, four
  // times as many as fit, 33 against 24.
  const int cell_lanes = v.o.dim == 2 ? kCellLanesLog2<2> : kCellLanesLog2<3>;
  const long long lanes = (long long)v.ncap << cell_lanes;
  if (v.o.nlist_stage == 0 && lanes <= 2048ll * sm_count()) {
    const int nb = lanes > 0 ? (int)((lanes + kNT - 1) / kNT) : 1;
    if (v.o.dim == 2 && v.o.uniform_h) nlist_cells_kernel<2, true><<<nb, kNT, 0, st>>>(v, margin);
    else if (v.o.dim == 2) nlist_cells_kernel<2, false><<<nb, kNT, 0, st>>>(v, margin);
    else if (v.o.uniform_h) nlist_cells_kernel<3, true><<<nb, kNT, 0, st>>>(v, margin);
    else nlist_cells_kernel<3, false><<<nb, kNT, 0, st>>>(v, margin);
    return;
  }
  // A lane to a particle while the lanes of two particles would fit the SMs at once
  // (1,024 an SM, 311k particles on 152): then there are too few of them to cover each
  // other's waits, where more take the shared loads and tests of two. One lane and two,
  // us: 3D 177k 86 and 106, 242k 101 and 121, 309k 137 and 146 | 392k 155 and 150, 464k
  // 182 and 180, 1.0M 388 and 349 (at 564k one is ahead once more, 220 and 233); 2D 86k
  // 18 and 22, 171k 23 and 27, 265k 32 and 30 | 359k 39 and 41, 515k 51 and 49, 907k 84
  // and 78. Between 265k and 360k they differ by less than a run does.
  if (v.o.uniform_h && v.o.nlist_stage == 0 && v.ncap <= 2048ll * sm_count()) {
    const int nb = (v.ncap + kNT - 1) / kNT;
    if (v.o.dim == 2) nlist_kernel<2, true><<<nb, kNT, 0, st>>>(v, margin);
    else nlist_kernel<3, true><<<nb, kNT, 0, st>>>(v, margin);
    return;
  }
  if (v.o.uniform_h) {  // two particles per lane; the leftovers' blocks first
    const int half = (v.ncap + 1) / 2;
    const int nr = 2 * sm_count();
    const int nb = nr + (half > 0 ? (half + kNT - 1) / kNT : 1);
    const int cap = min(v.o.nlist_stage, kStageCapMax);
    if (cap > 0 && !v.o.any_periodic_x) {
      const size_t smem = (size_t)(cap + kOver) * sizeof(float4);
      if (v.o.dim == 2) nlist_staged_kernel<2><<<nb, kNT, smem, st>>>(v, margin, nr, cap);
      else nlist_staged_kernel<3><<<nb, kNT, smem, st>>>(v, margin, nr, cap);
      return;
    }
    if (v.o.dim == 2) nlist_pair_kernel<2><<<nb, kNT, 0, st>>>(v, margin, nr);
    else nlist_pair_kernel<3><<<nb, kNT, 0, st>>>(v, margin, nr);
    return;
  }
  const int nb = v.ncap > 0 ? (v.ncap + kNT - 1) / kNT : 1;
  if (v.o.dim == 2) nlist_kernel<2, false><<<nb, kNT, 0, st>>>(v, margin);
  else nlist_kernel<3, false><<<nb, kNT, 0, st>>>(v, margin);
}

}  // namespace psph
