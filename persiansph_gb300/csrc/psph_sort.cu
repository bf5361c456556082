// Cell list as a deterministic counting sort (replaces CellReset + ListGenerate,
// Source/Domain.cpp:662-806, and the per-step pair arrays of MainNeighbourSearch).
//
//   bin      cell key per particle, exactly ListGenerate's floor/clamp rule;
//            each cell is split into xsub slabs along x and each slab into its
//            free and its fixed particles (the key counts them: (cell * xsub +
//            slab) * 2 + fixed), so the particles of a cell lie in x-slab order,
//            free ones first: the neighbour-list walk can skip slabs out of
//            reach, a fixed particle's walk the fixed ones (it has no pairs with
//            them), and warps hold fewer particles of both kinds;
//            key = nbins (= 2 xsub ncells) for a particle that ListGenerate
//            would drop into a periodic ghost column (it then sits in no list),
//            nbins+1 for one that CheckParticleLeave removed. The counting
//            atomic's old value is the particle's slot inside its segment.
//   scan     exclusive prefix of the counts; the sorted state's particle counts.
//   scatter  into the slots; per-cell segment starts (start[c] = start of c's
//            first slab) for everything that walks whole cells, the particles
//            the neighbour-list scan handles one per lane, the counts cleared.
//   reorder  deterministic order inside each segment: by original index, so the
//            sorted state depends only on positions, never on atomic timing;
//            each particle's fields move to that place (HBM-bound), with its
//            FP32 copies and the list of the fixed particles.
// A cell takes 64 bytes: 8 bins (4 slabs, free and fixed) in the counts and in their
// scan, 17 GB at the limit of 2^28 cells (half of it with one bin for both kinds).
// Four launches (five with more than 131,072 bins): launches are what counts up
// to 100k particles. With six 5k particles took 40 us, so 31; 920 in the FP32C
// form, their copies included, 37 and 25.
#include <algorithm>
#include <cstdio>

#include "psph_copies.cuh"

namespace psph {

namespace {

constexpr int kBT = 256;

__global__ void bin_kernel(DevView v, const uint8_t* __restrict__ alive, unsigned* __restrict__ key,
                           int* __restrict__ count, int* __restrict__ slot_of, StepScalars* sc, int dim, int xsub) {
  if (sc->all_stop || !sc->rebuild) return;
  const Persist& P = cur_persist(v);
  const int n = sc->n;
  const unsigned nbins = sort_bin(v.total_cells, xsub, 0);
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->nl_rest = sc->n_walls = 0;  // counted by the scatter and the reorder
  const unsigned orphan_key = nbins, dead_key = nbins + 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    unsigned k;
    if (!alive[i]) {
      k = dead_key;
    } else {
      const PClass& C = v.cls[P.cls[i]];
      const GridDev& g = grid_of(v, C.inst);
      const double4_32a x = P.X4[i];
      const double xs[3] = {x.x, x.y, x.z};
      int c[3] = {0, 0, 0};
      bool orphan = false, out = false;
      for (int d = 0; d < dim; ++d) {
        int cd = cell_floor(g, d, xs[d]);  // ListGenerate's rule
        if (cd < 0) {
          if ((g.blpf[d] - xs[d]) <= g.hmax) cd = 0;
          else out = true;
        }
        if (cd >= g.cn_ref[d]) {
          if ((xs[d] - g.trpr[d]) <= g.hmax) cd = g.cn_ref[d] - 1;
          else out = true;
        }
        if (cd >= g.nc[d]) orphan = true;  // periodic ghost column: overwritten by the copy
        c[d] = cd;
      }
      if (out) {
        atomicOr(&sc->status, ST_OUT_OF_GRID);
        k = dead_key;
      } else if (orphan) {
        k = orphan_key;
      } else {
        int slab = 0;
        if (xsub > 1) {  // x-slab inside the cell (clamped for particles outside it), in FP32
          const float ox = d2f_bits(x.x - g.blpf[0]) - (float)c[0] * g.cell_size32[0];
          slab = min(max((int)floorf(ox * (float)xsub * g.inv_cell_size32[0]), 0), xsub - 1);
        }
        k = sort_bin(g.cell_base + (c[2] * g.nc[1] + c[1]) * g.nc[0] + c[0], xsub, slab) + (C.is_free ? 0 : 1);
      }
    }
    key[i] = k;
    // one atomic per distinct cell of the warp: consecutive particles (sorted
    // by the previous step) mostly share their cell
    const unsigned peers = __match_any_sync(__activemask(), k);
    const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&count[k], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    slot_of[i] = base + __popc(peers & ((1u << lane) - 1u));
  }
}

// Exclusive scan of `in` (len entries; psph_bins.cuh has its shape).

// A thread's entries, from `first` (a multiple of 8), as 16-byte accesses: entry by
// entry a warp's accesses are 32 bytes apart (the sort of 86k particles into 167k bins
// 41 us, so 37; of 957k into 2.4M 117 and 109).
__device__ __forceinline__ void load_entries(const int* __restrict__ in, unsigned first, unsigned len, int (&v)[kScanPer]) {
  static_assert(kScanPer == 8, "two int4");
  if (scan_full(first, kScanPer, len)) {
    const int4 a = *reinterpret_cast<const int4*>(in + first), b = *reinterpret_cast<const int4*>(in + first + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
#pragma unroll
    for (unsigned e = 0; e < kScanPer; ++e) v[e] = (first + e < len) ? in[first + e] : 0;
  }
}
// their exclusive prefixes from `at`
__device__ __forceinline__ void store_prefixes(int* __restrict__ out, unsigned first, unsigned len, int at,
                                               const int (&v)[kScanPer]) {
  int p[kScanPer];
#pragma unroll
  for (unsigned e = 0; e < kScanPer; ++e) {
    p[e] = at;
    at += v[e];
  }
  if (scan_full(first, kScanPer, len)) {
    *reinterpret_cast<int4*>(out + first) = make_int4(p[0], p[1], p[2], p[3]);
    *reinterpret_cast<int4*>(out + first + 4) = make_int4(p[4], p[5], p[6], p[7]);
  } else {
#pragma unroll
    for (unsigned e = 0; e < kScanPer; ++e)
      if (first + e < len) out[first + e] = p[e];
  }
}

// A block's scan: v[] the thread's entries; returns the exclusive prefix of the
// thread's first one in the block, *total the block's sum (in every thread).
__device__ __forceinline__ int block_scan(const int (&v)[kScanPer], int* total) {
  __shared__ int warp_tot[33];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  int own = 0;
#pragma unroll
  for (unsigned e = 0; e < kScanPer; ++e) own += v[e];
  int incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    int s = warp_tot[lane];
    int si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, si, o);
      if (lane >= o) si += y;
    }
    warp_tot[lane] = si - s;  // exclusive warp offsets
    if (lane == 31) warp_tot[32] = si;
  }
  __syncthreads();
  *total = warp_tot[32];
  return incl - own + warp_tot[w];
}

// The sum of `part` over the block, in every thread.
__device__ __forceinline__ int block_sum(int part) {
  __shared__ int warp_sum[32];
  const int lane = threadIdx.x & 31;
  part = __reduce_add_sync(0xffffffffu, part);
  if (lane == 0) warp_sum[threadIdx.x >> 5] = part;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, warp_sum[lane]);
}

// The cell sort's scan knows the sorted state's counts, and makes its buffer the
// current one: nothing but the reorder, which knows, reads it in between. at is
// the prefix of entry i (len = bins + 2: the orphans' and the removed particles'
// segments come last).
__device__ __forceinline__ void sorted_counts(StepScalars* sc, unsigned i, unsigned len, int at) {
  if (i == len - 2) sc->n_cells = at;
  if (i == len - 1) {
    sc->n_old = sc->n;
    sc->n = at;
    sc->buf ^= 1;
  }
}
__device__ __forceinline__ void sorted_counts4(StepScalars* sc, unsigned i, unsigned len, int4 at) {
  if (i + 4 < len - 1 || i >= len) return;
  sorted_counts(sc, i, len, at.x);
  sorted_counts(sc, i + 1, len, at.y);
  sorted_counts(sc, i + 2, len, at.z);
  sorted_counts(sc, i + 3, len, at.w);
}

// Few blocks: each sums the entries before its own itself, so that one launch
// does it (up to 16 blocks, 131,072 bins: the last one reads 480 KB, 3 us, where
// a second launch costs as much).
constexpr unsigned kScanWhole = 16;
__global__ void __launch_bounds__(1024) scan_whole(const int* __restrict__ in, int* __restrict__ out, unsigned len,
                                                   StepScalars* sc) {
  if (sc && (sc->all_stop || !sc->rebuild)) return;  // the cell sort's scan, on a step without a rebuild
  const unsigned t = threadIdx.x, first = scan_first(blockIdx.x, t);
  int before = 0;
#pragma unroll 4
  for (unsigned i = t; i < blockIdx.x * (kScanBlock / 4); i += 1024) {
    const int4 q = reinterpret_cast<const int4*>(in)[i];
    before += q.x + q.y + q.z + q.w;
  }
  int v[kScanPer], total;
  load_entries(in, first, len, v);
  before = block_sum(before);
  int at = before + block_scan(v, &total);
  store_prefixes(out, first, len, at, v);
  if (sc && first < len) {
    sorted_counts4(sc, first, len, make_int4(at, at + v[0], at + v[0] + v[1], at + v[0] + v[1] + v[2]));
    at += v[0] + v[1] + v[2] + v[3];
    sorted_counts4(sc, first + 4, len, make_int4(at, at + v[4], at + v[4] + v[5], at + v[4] + v[5] + v[6]));
  }
  if (blockIdx.x == gridDim.x - 1 && t == 0) out[len] = before + total;
}

// Many blocks, phase 1: each block's own scan, its total to sums.
__global__ void __launch_bounds__(1024) scan_blocks(const int* __restrict__ in, int* __restrict__ out,
                                                    int* __restrict__ sums, unsigned len, const StepScalars* sc) {
  if (sc && (sc->all_stop || !sc->rebuild)) return;
  const unsigned first = scan_first(blockIdx.x, threadIdx.x);
  int v[kScanPer], total;
  load_entries(in, first, len, v);
  const int at = block_scan(v, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
  store_prefixes(out, first, len, at, v);
}

// Phase 2: every block adds the totals of the blocks before it; the last one
// writes the grand total.
__global__ void __launch_bounds__(1024) scan_add(int* __restrict__ out, const int* __restrict__ sums, unsigned len,
                                                 StepScalars* sc) {
  if (sc && (sc->all_stop || !sc->rebuild)) return;
  const unsigned t = threadIdx.x;
  int before = 0;
  for (unsigned b = t; b < blockIdx.x; b += 1024) before += sums[b];
  before = block_sum(before);
  // four consecutive entries, twice: 16-byte accesses that follow one another
#pragma unroll
  for (unsigned h = 0; h < kScanPer / 4; ++h) {
    const unsigned i = blockIdx.x * kScanBlock + h * 4096 + 4 * t;
    if (scan_full(i, 4, len)) {
      int4 q = *reinterpret_cast<int4*>(out + i);
      q.x += before; q.y += before; q.z += before; q.w += before;
      *reinterpret_cast<int4*>(out + i) = q;
      if (sc) sorted_counts4(sc, i, len, q);
    } else {
      int4 q = make_int4(0, 0, 0, 0);
      int* const e = &q.x;
      for (unsigned k = 0; k < 4 && i + k < len; ++k) out[i + k] = e[k] = out[i + k] + before;
      if (sc) sorted_counts4(sc, i, len, q);
    }
  }
  if (blockIdx.x == gridDim.x - 1 && t == 0) out[len] = before + sums[blockIdx.x];
}

void scan_launch(const int* in, int* out, unsigned len, int* sums, StepScalars* sc, cudaStream_t st) {
  const unsigned nb = scan_blocks_for(len);
  if (nb <= kScanWhole) {
    scan_whole<<<nb, 1024, 0, st>>>(in, out, len, sc);
  } else {
    scan_blocks<<<nb, 1024, 0, st>>>(in, out, sums, len, sc);
    scan_add<<<nb, 1024, 0, st>>>(out, sums, len, sc);
  }
}

// Particles into their slots, each with its original index (which the reorder ranks
// by: a read of it through the slot was a second wait per member); and what the scan makes known: per-cell segment
// starts from the bin starts (start[c] = sstart[c * 2 xsub] for c <= ncells, and
// the orphan / dead / total boundaries after them), and the particles the
// two-per-lane neighbour-list scan leaves to a lane of their own: lanes take
// sorted particles 2t and 2t+1 together when they share a cell, so the odd
// particles left are exactly the cells' first particles at odd indices (into
// rest, at most cap). The counts are cleared for the next sort.
__global__ void scatter_kernel(DevView v, const unsigned* __restrict__ key, const int* __restrict__ sstart,
                               const int* __restrict__ slot_of, int2* __restrict__ tmp_perm, int* __restrict__ count,
                               int* __restrict__ start, int ncells, int xsub, StepScalars* sc,
                               int* __restrict__ rest, int cap) {
  if (sc->all_stop || !sc->rebuild) return;
  const int n = sc->n_old;  // (the scan has counted the sorted state's n)
  const int tid = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  const int lane = threadIdx.x & 31;
  const int* __restrict__ orig = next_persist(v).orig;  // (the scan has made the sorted state's buffer the current one)
  for (int i = tid; i < n; i += stride) tmp_perm[sstart[key[i]] + slot_of[i]] = make_int2(i, orig[i]);
  const size_t per = 2 * (size_t)xsub, nbins = per * ncells;
  for (size_t i = tid; i < nbins + 2; i += stride) count[i] = 0;
  for (int c0 = tid - lane; c0 < ncells + 3; c0 += stride) {
    const int c = c0 + lane;
    if (c <= ncells) start[c] = sstart[c * per];
    else if (c <= ncells + 2) start[c] = sstart[nbins + (c - ncells)];
    bool odd_first = false;
    int s0 = 0;
    if (c < ncells) {
      s0 = sstart[c * per];
      odd_first = (s0 & 1) && sstart[(c + 1) * per] > s0;
    }
    const unsigned want = __ballot_sync(0xffffffffu, odd_first);  // (c0 is the warp's)
    if (odd_first) {  // one atomic per warp
      const int leader = __ffs(want) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(&sc->nl_rest, __popc(want));
      base = __shfl_sync(want, base, leader);
      const int slot = base + __popc(want & ((1u << lane) - 1u));
      if (slot < cap) rest[slot] = s0;
    }
  }
}

// One thread per scattered particle i: its place s is its segment's start plus
// the number of the segment's particles with a smaller original index; then its
// fields move there (a solid's 3x3 tensors stay where they are: tensor_row).
// With it go the FP32 offset from the cell's origin, an FP32C fluid's copies, and
// the list of the fixed particles (written by warps of places that ascend, so
// that a warp of the list lies close together).
__global__ void __launch_bounds__(kBT) reorder_kernel(DevView v, const int2* __restrict__ tmp_perm, const unsigned* __restrict__ key, const int* __restrict__ start, int* __restrict__ cellid,
                               uint8_t* __restrict__ alive, StepScalars* sc, unsigned nbins, int xsub, int dyn_mu) {
  if (sc->all_stop || !sc->rebuild) return;
  const Persist& src = next_persist(v);  // (the scan has made the sorted state's buffer the current one)
  const Persist& dst = cur_persist(v);
  const int n_new = sc->n;  // the removed particles' segment comes last
  const bool fluid32 = v.o.fp32 && !v.o.has_solid;
  const bool copies = fluid32 && v.o.skin == 0.f;  // (with a skin: skin_offsets_kernel)
  const bool list_walls = !fluid32 || v.o.dim == 2;  // (the 3D FP32C walls are interpolated where they lie)
  __shared__ int before[kBT / 32];  // walls of the block's warps before each
  __shared__ int list_at;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int q0 = blockIdx.x * kBT; q0 < n_new; q0 += gridDim.x * kBT) {
    const int q = q0 + threadIdx.x;
    int wall = -1;  // this thread's particle, if fixed
    if (q < n_new) {
      const int2 own = tmp_perm[q];
      const int i = own.x, mine = own.y;
      const unsigned k = key[i];
      const int lo = start[k], hi = start[k + 1];
      int s = lo;
      for (int t = lo; t < hi; ++t) s += tmp_perm[t].y < mine;
      const double4_32a xs = src.X4[i], vs = src.V4[i];
      dst.X4[s] = xs;
      dst.V4[s] = vs;
      dst.H4[s] = src.H4[i];
      if (src.H4b) dst.H4b[s] = src.H4b[i];
      const int cls = src.cls[i];
      dst.cls[s] = cls;
      if (dyn_mu) dst.mu[s] = src.mu[i];
      const bool is_free = v.cls[cls].is_free;
      // FP32 offset from the cell origin (absolute position outside any cell)
      const float h = is_free ? d2f_rn(v.cls[cls].h) : -d2f_rn(v.cls[cls].h);
      float4 off;
      if (k < nbins) {
        const GridDev& g = grid_of(v, v.cls[cls].inst);
        const int lk = (int)(k / sort_bin(1, xsub, 0)) - g.cell_base;
        const int cx = lk % g.nc[0], t = lk / g.nc[0], cy = t % g.nc[1], cz = t / g.nc[1];
        off = make_float4(d2f_rn(xs.x - (g.blpf[0] + i2d_small(cx) * g.cell_size[0])),
                          d2f_rn(xs.y - (g.blpf[1] + i2d_small(cy) * g.cell_size[1])),
                          v.o.dim == 3 ? d2f_rn(xs.z - (g.blpf[2] + i2d_small(cz) * g.cell_size[2])) : 0.f, h);
      } else {
        off = make_float4(d2f_rn(xs.x), d2f_rn(xs.y), d2f_rn(xs.z), h);
      }
      v.S.OFF32[s] = off;
      if (v.o.skin > 0.f)  // displacements are measured from here (FP32, truncated)
        v.S.OFFREF[s] = make_float4(d2f_bits(xs.x), d2f_bits(xs.y), d2f_bits(xs.z), 0.f);
      if (copies) fluid_copies32(v, dst, s, cls, xs.w, vs, off, 0);
      dst.orig[s] = mine;
      if (src.io) dst.io[s] = src.io[i];
      cellid[s] = (k < nbins) ? (int)(k / sort_bin(1, xsub, 0)) : -1;
      alive[s] = 1;
      if (!is_free) wall = s;
    }
    if (!list_walls) continue;
    // the block's walls, by one atomic: parts of some hundred in sorted order
    const unsigned m = __ballot_sync(0xffffffffu, wall >= 0);
    if (lane == 0) before[warp] = __popc(m);
    if (__syncthreads_or(m != 0) == 0) continue;
    if (threadIdx.x == 0) {
      int sum = 0;
      for (int w = 0; w < kBT / 32; ++w) {
        const int c = before[w];
        before[w] = sum;
        sum += c;
      }
      list_at = atomicAdd(&sc->n_walls, sum);
    }
    __syncthreads();
    if (wall >= 0) v.S.walls[list_at + before[warp] + __popc(m & ((1u << lane) - 1u))] = wall;
    __syncthreads();
  }
}

// Neighbour lists with a skin: on every step an FP32C fluid's copies, the FP32
// offsets of the particles from their cells' origins (the cells of the last rebuild), and
// each particle's cell in the reference's grid (ListGenerate's floor and
// clamp on the FP64 position, Source/Domain.cpp:669-691), which orients the
// wall pressure's pairs as the reference's neighbour search does.
__global__ void skin_offsets_kernel(DevView v) {
  const StepScalars* sc = v.sc;
  if (sc->all_stop) return;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= sc->n) return;
  const Persist& P = cur_persist(v);
  const PClass& C = v.cls[P.cls[s]];
  const double4_32a xs = P.X4[s];
  const float h = C.is_free ? d2f_rn(C.h) : -d2f_rn(C.h);
  const int cell = v.S.cellid[s];
  float4 off;
  if (cell >= 0) {
    const GridDev& g = grid_of(v, C.inst);
    const int lk = cell - g.cell_base;
    const int cx = lk % g.nc[0], t = lk / g.nc[0], cy = t % g.nc[1], cz = t / g.nc[1];
    off = make_float4(d2f_rn(xs.x - (g.blpf[0] + i2d_small(cx) * g.cell_size[0])),
                      d2f_rn(xs.y - (g.blpf[1] + i2d_small(cy) * g.cell_size[1])),
                      v.o.dim == 3 ? d2f_rn(xs.z - (g.blpf[2] + i2d_small(cz) * g.cell_size[2])) : 0.f, h);
  } else {
    off = make_float4(d2f_rn(xs.x), d2f_rn(xs.y), d2f_rn(xs.z), h);
  }
  v.S.OFF32[s] = off;
  const GridDev& r = v.grids_ref[C.inst];
  const double xd[3] = {xs.x, xs.y, xs.z};
  int q[3] = {0, 0, 0};
  for (int d = 0; d < v.o.dim; ++d) {
    const int k = cell_floor(r, d, xd[d]);
    q[d] = min(max(k, 0), r.cn_ref[d] - 1);  // clamped as ListGenerate clamps the particles just outside
  }
  const int rc = q[0] | (q[1] << 10) | (q[2] << 20);
  v.S.refcell[s] = rc;
  if (v.o.fp32 && !v.o.has_solid) fluid_copies32(v, P, s, P.cls[s], xs.w, P.V4[s], off, rc);
}

// now: the next cell sort runs (a sort outside the step loop); next_step:
// the next step sorts and lists again (with a skin, whose lists would
// otherwise be kept)
__global__ void mark_rebuild_kernel(StepScalars* sc, int now, int next_step) {
  if (now) sc->rebuild = 1;
  if (next_step) sc->force_rebuild = 1;
}

inline int grid_for(int n) {
  int b = (n + kBT - 1) / kBT;
  return b < 1 ? 1 : b;
}

}  // namespace

void launch_skin_offsets(const DevView& v, cudaStream_t st) {
  skin_offsets_kernel<<<grid_for(v.ncap), kBT, 0, st>>>(v);
}

void launch_mark_rebuild(const DevView& v, bool now, bool next_step, cudaStream_t st) {
  mark_rebuild_kernel<<<1, 1, 0, st>>>(v.sc, now ? 1 : 0, next_step ? 1 : 0);
}

void launch_sort(const DevView& v, cudaStream_t st) {
  const Scratch& S = v.S;
  const int ncells = v.total_cells;
  const int xsub = v.o.xsub;
  const unsigned nbins = sort_bin(ncells, xsub, 0), len = nbins + 2;
  // with a skin most steps skip the sort: few enough blocks that skipping is cheap
  // (6.7M particles: 67 us a step for the skipped launches, 25 so)
  const int gp = v.o.skin > 0.f ? std::min(grid_for(v.ncap), 4096) : grid_for(v.ncap);
  // S.count is zero here (allocated so, and cleared behind every scan)
  bin_kernel<<<gp, kBT, 0, st>>>(v, v.alive, S.key, S.count, S.slot, v.sc, v.o.dim, xsub);
  scan_launch(S.count, S.sstart, len, S.block_sums, v.sc, st);
  scatter_kernel<<<gp, kBT, 0, st>>>(v, S.key, S.sstart, S.slot, S.tmp_perm, S.count, S.start, ncells, xsub, v.sc, S.rest,
                                     v.ncap);
  reorder_kernel<<<gp, kBT, 0, st>>>(v, S.tmp_perm, S.key, S.sstart, S.cellid, v.alive, v.sc, nbins, xsub,
                                     v.o.dyn_mu);
}

int sort_launches(const DevView& v) { return scan_blocks_for(sort_bin(v.total_cells, v.o.xsub, 0) + 2) <= kScanWhole ? 4 : 5; }

}  // namespace psph

namespace psph {

// Exclusive prefix of in[0..len) into out[0..len], out[len] = total, using
// block_sums (>= ceil(len/1024) entries) as scratch. Used by the pair export
// that takes its scratch from caller-owned or static device memory.
void launch_exclusive_scan(const int* in, int* out, int len, int* block_sums, cudaStream_t st) {
  scan_launch(in, out, len, block_sums, nullptr, st);
}

}  // namespace psph
