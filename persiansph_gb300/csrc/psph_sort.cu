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
//   scan     exclusive prefix of the counts (block scans, then each block adds
//            the totals before it and clears the counts for the next sort).
//   scatter  into the slots.
//   reorder  deterministic order inside each segment: by original index, so the
//            sorted state depends only on positions, never on atomic timing;
//            each particle's fields move to that place (HBM-bound).
//   starts   per-cell segment starts (start[c] = start of c's first slab) for
//            everything that walks whole cells, the particles the neighbour-list
//            scan handles one per lane, and the new counts and buffer.
// Six launches (eleven with separate clearing, scan of totals, ranking and
// finish kernels): 57 -> 44 us for 86k particles, where launches are what counts.
#include <algorithm>
#include <cstdio>

#include "psph_device.cuh"

namespace psph {

namespace {

constexpr int kBT = 256;

__global__ void bin_kernel(DevView v, const uint8_t* __restrict__ alive, int* __restrict__ key,
                           int* __restrict__ count, int* __restrict__ slot_of, StepScalars* sc, int dim, int xsub) {
  if (sc->all_stop || !sc->rebuild) return;
  const Persist& P = cur_persist(v);
  const int n = sc->n;
  const int nbins = 2 * v.total_cells * xsub;
  if (blockIdx.x == 0 && threadIdx.x == 0) sc->nl_rest = 0;  // cell_starts_kernel counts them
  const int orphan_key = nbins, dead_key = nbins + 1;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    int k;
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
        k = 2 * ((g.cell_base + (c[2] * g.nc[1] + c[1]) * g.nc[0] + c[0]) * xsub + slab) + (C.is_free ? 0 : 1);
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

// Phase 1: in-block exclusive scan of `in` (len entries), block totals to sums.
// A thread takes kScanPer consecutive entries, a block kScanBlock: few enough
// totals that phase 2 needs no scan of them in between.
constexpr int kScanPer = 8, kScanBlock = 1024 * kScanPer;
__global__ void __launch_bounds__(1024) scan_blocks(const int* __restrict__ in, int* __restrict__ out,
                                                    int* __restrict__ sums, int len, const StepScalars* sc) {
  if (sc && (sc->all_stop || !sc->rebuild)) return;  // the cell sort's scan, on a step without a rebuild
  __shared__ int warp_tot[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int first = blockIdx.x * kScanBlock + t * kScanPer;
  int v[kScanPer], own = 0;
#pragma unroll
  for (int e = 0; e < kScanPer; ++e) v[e] = (first + e < len) ? in[first + e] : 0;
#pragma unroll
  for (int e = 0; e < kScanPer; ++e) own += v[e];
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
    if (lane == 31) sums[blockIdx.x] = si;
  }
  __syncthreads();
  int at = incl - own + warp_tot[w];
#pragma unroll
  for (int e = 0; e < kScanPer; ++e) {
    if (first + e < len) out[first + e] = at;
    at += v[e];
  }
}

// Phase 2: every block adds the totals of the blocks before it; the last one
// writes the grand total. clear (if given): entries set to zero behind the scan.
__global__ void __launch_bounds__(1024) scan_add(int* __restrict__ out, const int* __restrict__ sums, int len,
                                                 int* __restrict__ clear, const StepScalars* sc) {
  if (sc && (sc->all_stop || !sc->rebuild)) return;
  __shared__ int part[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  int before = 0;
  for (int b = t; b < (int)blockIdx.x; b += 1024) before += sums[b];
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) part[w] = before;
  __syncthreads();
  before = __reduce_add_sync(0xffffffffu, part[lane]);
#pragma unroll
  for (int e = 0; e < kScanPer; ++e) {
    const int i = blockIdx.x * kScanBlock + e * 1024 + t;
    if (i < len) {
      out[i] += before;
      if (clear) clear[i] = 0;
    }
  }
  if (blockIdx.x == gridDim.x - 1 && t == 0) out[len] = before + sums[blockIdx.x];
}

inline int scan_blocks_for(int len) { return len > kScanBlock ? (len - 1) / kScanBlock + 1 : 1; }

__global__ void scatter_kernel(const int* __restrict__ key, const int* __restrict__ start,
                               const int* __restrict__ slot_of, int* __restrict__ tmp_perm, const StepScalars* sc) {
  if (sc->all_stop || !sc->rebuild) return;
  const int n = sc->n;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    tmp_perm[start[key[i]] + slot_of[i]] = i;
}

// One thread per scattered particle i: its place s is its segment's start plus
// the number of the segment's particles with a smaller original index; then its
// fields move there (a solid's 3x3 tensors stay where they are: tensor_row).
__global__ void reorder_kernel(DevView v, const int* __restrict__ tmp_perm, const int* __restrict__ key, const int* __restrict__ start, int* __restrict__ cellid,
                               uint8_t* __restrict__ alive, const StepScalars* sc, int nbins, int xsub, int dyn_mu) {
  if (sc->all_stop || !sc->rebuild) return;
  const Persist& src = cur_persist(v);
  const Persist& dst = next_persist(v);
  const int n_new = start[nbins + 1];  // the removed particles' segment comes last
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n_new; q += gridDim.x * blockDim.x) {
    const int i = tmp_perm[q];
    const int k = key[i];
    const int lo = start[k], hi = start[k + 1];
    const int mine = src.orig[i];
    int s = lo;
    for (int t = lo; t < hi; ++t) s += src.orig[tmp_perm[t]] < mine;
    dst.X4[s] = src.X4[i];
    dst.V4[s] = src.V4[i];
    dst.H4[s] = src.H4[i];
    if (src.H4b) dst.H4b[s] = src.H4b[i];
    const int cls = src.cls[i];
    dst.cls[s] = cls;
    {
      // FP32 offset from the cell origin (absolute position outside any cell)
      const double4_32a xs = src.X4[i];
      const float h = v.cls[cls].is_free ? d2f_rn(v.cls[cls].h) : -d2f_rn(v.cls[cls].h);
      if (k < nbins) {
        const GridDev& g = grid_of(v, v.cls[cls].inst);
        const int lk = k / (2 * xsub) - g.cell_base;
        const int cx = lk % g.nc[0], t = lk / g.nc[0], cy = t % g.nc[1], cz = t / g.nc[1];
        v.S.OFF32[s] = make_float4(d2f_rn(xs.x - (g.blpf[0] + i2d_small(cx) * g.cell_size[0])),
                                   d2f_rn(xs.y - (g.blpf[1] + i2d_small(cy) * g.cell_size[1])),
                                   v.o.dim == 3 ? d2f_rn(xs.z - (g.blpf[2] + i2d_small(cz) * g.cell_size[2])) : 0.f, h);
      } else {
        v.S.OFF32[s] = make_float4(d2f_rn(xs.x), d2f_rn(xs.y), d2f_rn(xs.z), h);
      }
      if (v.o.skin > 0.f)  // displacements are measured from here (FP32, truncated)
        v.S.OFFREF[s] = make_float4(d2f_bits(xs.x), d2f_bits(xs.y), d2f_bits(xs.z), 0.f);
    }
    dst.orig[s] = mine;
    if (src.io) dst.io[s] = src.io[i];
    cellid[s] = (k < nbins) ? k / (2 * xsub) : -1;
    alive[s] = 1;
    if (dyn_mu) dst.mu[s] = src.mu[i];
  }
}

// Per-cell segment starts from the bin starts: start[c] = sstart[c * 2 xsub] for
// c <= ncells, and the orphan / dead / total boundaries after them; the sorted
// state's counts and buffer. Also lists the particles the two-per-lane
// neighbour-list scan leaves to a lane of their own: lanes take sorted particles
// 2t and 2t+1 together when they share a cell, so the odd particles left are
// exactly the cells' first particles at odd indices (into rest, at most cap).
__global__ void cell_starts_kernel(const int* __restrict__ sstart, int* __restrict__ start, int ncells, int xsub,
                                   StepScalars* sc, int* __restrict__ rest, int cap) {
  if (sc->all_stop || !sc->rebuild) return;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const size_t per = 2 * (size_t)xsub, nbins = per * ncells;
  if (c <= ncells) start[c] = sstart[c * per];
  else if (c <= ncells + 2) start[c] = sstart[nbins + (c - ncells)];
  if (c == 0) {
    sc->n_cells = sstart[nbins];
    sc->n = sstart[nbins + 1];
    sc->buf ^= 1;
  }
  bool odd_first = false;
  int s0 = 0;
  if (c < ncells) {
    s0 = sstart[c * per];
    odd_first = (s0 & 1) && sstart[(c + 1) * per] > s0;
  }
  const unsigned want = __ballot_sync(0xffffffffu, odd_first);  // every lane of the grid gets here
  if (odd_first) {  // one atomic per warp
    const int lane = threadIdx.x & 31, leader = __ffs(want) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&sc->nl_rest, __popc(want));
    base = __shfl_sync(want, base, leader);
    const int slot = base + __popc(want & ((1u << lane) - 1u));
    if (slot < cap) rest[slot] = s0;
  }
}

// Neighbour lists with a skin: on every step the FP32 offsets of the
// particles from their cells' origins (the cells of the last rebuild), and
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
  if (cell >= 0) {
    const GridDev& g = grid_of(v, C.inst);
    const int lk = cell - g.cell_base;
    const int cx = lk % g.nc[0], t = lk / g.nc[0], cy = t % g.nc[1], cz = t / g.nc[1];
    v.S.OFF32[s] = make_float4(d2f_rn(xs.x - (g.blpf[0] + i2d_small(cx) * g.cell_size[0])),
                               d2f_rn(xs.y - (g.blpf[1] + i2d_small(cy) * g.cell_size[1])),
                               v.o.dim == 3 ? d2f_rn(xs.z - (g.blpf[2] + i2d_small(cz) * g.cell_size[2])) : 0.f, h);
  } else {
    v.S.OFF32[s] = make_float4(d2f_rn(xs.x), d2f_rn(xs.y), d2f_rn(xs.z), h);
  }
  const GridDev& r = v.grids_ref[C.inst];
  const double xd[3] = {xs.x, xs.y, xs.z};
  int q[3] = {0, 0, 0};
  for (int d = 0; d < v.o.dim; ++d) {
    const int k = cell_floor(r, d, xd[d]);
    q[d] = min(max(k, 0), r.cn_ref[d] - 1);  // clamped as ListGenerate clamps the particles just outside
  }
  v.S.refcell[s] = q[0] | (q[1] << 10) | (q[2] << 20);
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
  const int nbins = 2 * ncells * xsub;
  const int len = nbins + 2;
  // with a skin most steps skip the sort: few enough blocks that skipping is cheap
  // (6.7M particles: 67 us a step for the skipped launches, 25 so)
  const int gp = v.o.skin > 0.f ? std::min(grid_for(v.ncap), 4096) : grid_for(v.ncap);
  // S.count is zero here (allocated so, and cleared behind every scan)
  bin_kernel<<<gp, kBT, 0, st>>>(v, v.alive, S.key, S.count, S.slot, v.sc, v.o.dim, xsub);
  const int nb = scan_blocks_for(len);
  scan_blocks<<<nb, 1024, 0, st>>>(S.count, S.sstart, S.block_sums, len, v.sc);
  scan_add<<<nb, 1024, 0, st>>>(S.sstart, S.block_sums, len, S.count, v.sc);
  scatter_kernel<<<gp, kBT, 0, st>>>(S.key, S.sstart, S.slot, S.tmp_perm, v.sc);
  reorder_kernel<<<gp, kBT, 0, st>>>(v, S.tmp_perm, S.key, S.sstart, S.cellid, v.alive, v.sc, nbins, xsub,
                                     v.o.dyn_mu);
  cell_starts_kernel<<<grid_for(ncells + 3), kBT, 0, st>>>(S.sstart, S.start, ncells, xsub, v.sc, S.tmp_perm, v.ncap);
}

}  // namespace psph

namespace psph {

// Exclusive prefix of in[0..len) into out[0..len], out[len] = total, using
// block_sums (>= ceil(len/1024) entries) as scratch. Used by the pair export
// that takes its scratch from caller-owned or static device memory.
void launch_exclusive_scan(const int* in, int* out, int len, int* block_sums, cudaStream_t st) {
  const int nb = scan_blocks_for(len);
  scan_blocks<<<nb, 1024, 0, st>>>(in, out, block_sums, len, nullptr);
  scan_add<<<nb, 1024, 0, st>>>(out, block_sums, len, nullptr, nullptr);
}

}  // namespace psph
