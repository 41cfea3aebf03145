// gb_uf.cu -- PNUM connectivity on the GPU.
//
// Semantics of PerformMerge (pnummerge.f90:279-385) with UnionFind
// (datastructures.f90:26-215): two boxes are connected when their closed
// extents overlap (edge and corner touches count); the root of a component is
// its smallest box index; after the final reduction the non-singleton roots
// are numbered 1..R in index order and singletons keep label 0; the
// component count is R + #singletons.
//
// Candidate pairs come from a closed-range tile binning (every box is listed
// in each tile its closed extent touches, so two touching boxes share at
// least one tile).  Tiles of up to UF_WARP_BOXES boxes (nearly all: the grid
// is sized for about 32 boxes per tile) are taken one per warp; larger tiles
// are taken one per CTA.  A lane keeps its boxes in registers and meets the
// tile's boxes one after the other, each read from shared memory by all lanes
// at once.  Pairs that meet are united in shared memory first, so a tile adds
// to the global forest one edge per box that is not its local root, and not
// one per pair.  Global edges are hooked with atomicCAS, the larger root
// under the smaller, so the surviving root is the component minimum whatever
// the order of the hooks.  Pointer jumping then flattens the forest.
#include "gb_internal.h"
#include "gb_scan.cuh"

#define UF_SMEM_BOXES 1024
#define UF_WARP_BOXES 128  // tiles up to this size go one per warp, four boxes per lane
#define UF_LB (UF_WARP_BOXES / 32)
#define UF_WARPS 8         // warps per CTA of the per-warp kernels
#define KID_UF 30

__device__ __forceinline__ int uf_find(int* parent, int x) {
  // Path halving.  Parents only ever point to smaller indices, so writing a
  // grandparent is always a valid ancestor even under concurrent updates.
  int guard = 0;
  while (true) {
    const int p = parent[x];
    if (p == x || guard++ > (1 << 26)) return x;
    const int gp = parent[p];
    if (gp != p) atomicMin(&parent[x], gp);
    x = gp == p ? p : gp;
  }
}

__device__ __forceinline__ void uf_unite(int* parent, int a, int b, DStatus* st) {
  for (int it = 0; it < (1 << 24); ++it) {
    a = uf_find(parent, a);
    b = uf_find(parent, b);
    if (a == b) return;
    if (a > b) { const int t = a; a = b; b = t; }
    const int old = atomicCAS(&parent[b], b, a);
    if (old == b) return;
  }
  gb_set_error(st, GB_ERR_TIMEOUT, KID_UF, 0);
}

__global__ void k_uf_init(int* parent, unsigned char* touched, long long n) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    parent[i] = (int)i;
    touched[i] = 0;
  }
}

__device__ __forceinline__ bool closed_overlap(int4 a, int4 b) {
  return a.x <= b.z && b.x <= a.z && a.y <= b.w && b.y <= a.w;  // both boxes are valid
}

// Shared-memory union-find over a tile's boxes (indices into the tile).
__device__ __forceinline__ int sm_find(const int* sp, int x) {
  for (int guard = 0; guard <= UF_SMEM_BOXES; ++guard) {
    const int p = *(volatile const int*)&sp[x];
    if (p == x) break;
    x = p;
  }
  return x;
}
__device__ __forceinline__ void sm_unite(int* sp, int a, int b) {
  for (int it = 0; it < (1 << 16); ++it) {  // a failed hook means another one succeeded
    a = sm_find(sp, a);
    b = sm_find(sp, b);
    if (a == b) return;
    if (a > b) { const int t = a; a = b; b = t; }
    if (atomicCAS(&sp[b], b, a) == b) return;
  }
}

// Box i of a tile's component whose smallest box index is m: touched, and
// joined to m.  A box that lies in this tile alone is seen by no other tile,
// and nothing is ever hooked under it (it is not its component's smallest
// box), so it takes m as its parent with a plain store; only boxes over
// several tiles walk and hook the forest.
__device__ __forceinline__ void tile_edge(int* parent, unsigned char* touched, int i, int4 b, int m, int g, DStatus* st) {
  touched[i] = 1;
  if (i == m) return;
  if ((b.x >> g) == (b.z >> g) && (b.y >> g) == (b.w >> g)) parent[i] = m;
  else uf_unite(parent, i, m, st);
}

// Boxes of a tile in shared memory, for the warp or the CTA that has it.
template <int N>
struct TileBoxes {
  int4 box[N];
  int idx[N];
};

// One warp's tiles of at most UF_WARP_BOXES boxes (in a grid stride over all
// warps; larger tiles are left to the per-CTA kernels): the boxes go to
// shared memory and, four per lane, to registers.  32 boxes of the tile at a
// time are read by all lanes at once and tested against the lanes' own, the
// outcomes kept as bits; then met(j, a0, m) is called with the pairs of the
// lane's box j (bit i of m: it meets box a0 + i < j), so that the work per
// pair runs on all lanes together and not lane by lane as pairs turn up
// (5500 -> 2900 instructions a tile).  Finally done(k, hit): the lane's boxes
// that met any (bit u: box u * 32 + lane).
template <typename Begin, typename Met, typename Done>
__device__ __forceinline__ void warp_tiles(const DLayer* raw, const DLayer* bin, TileBoxes<UF_WARP_BOXES>* tb, Begin begin,
                                           Met met, Done done) {
  const int4* boxes = raw->boxes;
  const int* idx = (const int*)bin->pcs;
  TileBoxes<UF_WARP_BOXES>& s = tb[gb_warp()];
  const int lane = gb_lane();
  const long long nt = bin->ntiles;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long t = (long long)blockIdx.x * (blockDim.x >> 5) + gb_warp(); t < nt; t += nwarps) {
    const int k = bin->tcount[t];
    if (k < 2 || k > UF_WARP_BOXES) continue;
    const int* ti = idx + bin->tstart[t];
    int4 bb[UF_LB];
#pragma unroll
    for (int u = 0; u < UF_LB; ++u) {
      const int j = u * 32 + lane;
      bb[u] = make_int4(INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN);
      if (j < k) {
        const int i = ti[j];
        bb[u] = boxes[i];
        s.idx[j] = i;
        s.box[j] = bb[u];
      }
    }
    begin(k, t);
    __syncwarp();
    unsigned hit = 0;
#pragma unroll
    for (int w = 0; w < UF_LB; ++w) {
      if (w * 32 + 1 >= k) break;  // warp-uniform, as the tests on k below
      unsigned m[UF_LB];
#pragma unroll
      for (int u = 0; u < UF_LB; ++u) m[u] = 0;
      const int na = min(32, k - w * 32);
      for (int i = 0; i < na; ++i) {
        const int4 ba = s.box[w * 32 + i];
#pragma unroll
        for (int u = w; u < UF_LB; ++u)
          if (u * 32 < k && closed_overlap(ba, bb[u])) m[u] |= 1u << i;
      }
      m[w] &= (1u << lane) - 1u;  // earlier boxes only
      unsigned all = 0;
#pragma unroll
      for (int u = w; u < UF_LB; ++u) {
        if (u * 32 >= k) break;
        if (u * 32 + lane >= k) m[u] = 0;  // no box: the inverted one held there meets a box that spans all of int32
        if (m[u]) {
          hit |= 1u << u;
          met(u * 32 + lane, w * 32, m[u]);
        }
        all |= m[u];
      }
      hit |= ((__reduce_or_sync(0xffffffffu, all) >> lane) & 1u) << w;
    }
    __syncwarp();
    done(k, hit);
    __syncwarp();  // the next tile overwrites the warp's boxes
  }
}

__global__ void __launch_bounds__(UF_WARPS * 32) k_uf_tile_warp(const DLayer* raw, const DLayer* bin, int* parent,
                                                              unsigned char* touched, DStatus* st) {
  __shared__ TileBoxes<UF_WARP_BOXES> tb[UF_WARPS];
  __shared__ int sparent[UF_WARPS][UF_WARP_BOXES];
  __shared__ int least[UF_WARPS][UF_WARP_BOXES];  // smallest box index per component
  if (st->err) return;
  const TileBoxes<UF_WARP_BOXES>& s = tb[gb_warp()];
  int* const sp = sparent[gb_warp()];
  int* const lm = least[gb_warp()];
  const int lane = gb_lane(), g = bin->g;
  warp_tiles(
      raw, bin, tb,
      [&](int k, long long) {
        for (int j = lane; j < k; j += 32) {
          sp[j] = j;
          lm[j] = INT32_MAX;
        }
      },
      [&](int j, int a0, unsigned m) {
        for (; m; m &= m - 1) sm_unite(sp, a0 + __ffs(m) - 1, j);
      },
      [&](int, unsigned hit) {
        int r[UF_LB];
#pragma unroll
        for (int u = 0; u < UF_LB; ++u)
          if ((hit >> u) & 1) {
            r[u] = sm_find(sp, u * 32 + lane);
            atomicMin(&lm[r[u]], s.idx[u * 32 + lane]);
          }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < UF_LB; ++u)
          if ((hit >> u) & 1) tile_edge(parent, touched, s.idx[u * 32 + lane], s.box[u * 32 + lane], lm[r[u]], g, st);
      });
}

// Tiles of more than UF_WARP_BOXES boxes, one per CTA (a grid stride over the
// tiles; the others are skipped without a barrier).  Up to UF_SMEM_BOXES boxes
// the CTA keeps four per thread in registers, as a warp does; the boxes of
// larger tiles are read from global memory for every pair, and
// pair(ia, ba, ib, bb) then has no place in shared memory (j = -1).
template <typename Begin, typename Pair, typename Done>
__device__ __forceinline__ void cta_tiles(const DLayer* raw, const DLayer* bin, TileBoxes<UF_SMEM_BOXES>& s, Begin begin,
                                          Pair pair, Done done) {
  constexpr int NT = 256, LB = UF_SMEM_BOXES / NT;
  const int4* boxes = raw->boxes;
  const int* idx = (const int*)bin->pcs;
  for (long long t = blockIdx.x; t < bin->ntiles; t += gridDim.x) {
    const int k = bin->tcount[t];
    if (k <= UF_WARP_BOXES) continue;
    const int* ti = idx + bin->tstart[t];
    __syncthreads();  // the previous tile's boxes are no longer read
    begin(k, t);
    if (k > UF_SMEM_BOXES) {
      const int nw = NT >> 5;
      for (int a = gb_warp(); a < k; a += nw) {
        const int ia = ti[a];
        const int4 ba = boxes[ia];
        for (int b = a + 1 + gb_lane(); b < k; b += 32) {
          const int ib = ti[b];
          const int4 bb = boxes[ib];
          if (closed_overlap(ba, bb)) pair(-1, -1, ia, ba, ib, bb);
        }
      }
      continue;
    }
    int4 bb[LB];
#pragma unroll
    for (int u = 0; u < LB; ++u) {
      const int j = u * NT + threadIdx.x;
      bb[u] = make_int4(INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN);
      if (j < k) {
        const int i = ti[j];
        bb[u] = boxes[i];
        s.idx[j] = i;
        s.box[j] = bb[u];
      }
    }
    __syncthreads();
    for (int a = 0; a + 1 < k; ++a) {
      const int4 ba = s.box[a];
#pragma unroll
      for (int u = 0; u < LB; ++u) {
        if (u * NT + NT - 1 <= a || u * NT >= k) continue;  // uniform
        const int j = u * NT + threadIdx.x;
        // a < j < k, in one comparison
        if ((unsigned)(j - a - 1) < (unsigned)(k - a - 1) && closed_overlap(ba, bb[u])) pair(a, j, s.idx[a], ba, s.idx[j], bb[u]);
      }
    }
    __syncthreads();
    done(k);
  }
}

__global__ void __launch_bounds__(256) k_uf_tile(const DLayer* raw, const DLayer* bin, int* parent,
                                                 unsigned char* touched, DStatus* st) {
  __shared__ TileBoxes<UF_SMEM_BOXES> s;
  __shared__ int sp[UF_SMEM_BOXES];
  __shared__ int least[UF_SMEM_BOXES];
  __shared__ unsigned char met[UF_SMEM_BOXES];
  if (st->err) return;
  const int g = bin->g;
  cta_tiles(
      raw, bin, s,
      [&](int k, long long) {
        for (int j = threadIdx.x; j < min(k, UF_SMEM_BOXES); j += blockDim.x) {
          sp[j] = j;
          least[j] = INT32_MAX;
          met[j] = 0;
        }
      },
      [&](int a, int b, int ia, int4, int ib, int4) {
        if (a < 0) {
          touched[ia] = 1;
          touched[ib] = 1;
          uf_unite(parent, ia, ib, st);
        } else {
          met[a] = 1;
          met[b] = 1;
          sm_unite(sp, a, b);
        }
      },
      [&](int k) {
        for (int j = threadIdx.x; j < k; j += blockDim.x)
          if (met[j]) atomicMin(&least[sm_find(sp, j)], s.idx[j]);
        __syncthreads();
        for (int j = threadIdx.x; j < k; j += blockDim.x)
          if (met[j]) tile_edge(parent, touched, s.idx[j], s.box[j], least[sm_find(sp, j)], g, st);
      });
}

// Overlap statistics (ComputeInteractionsCPU, pnummerge.f90:483-562, and
// FindSingletonsCPU, :388-482).  Every pair meeting with closed bounds marks
// both boxes as non-singletons.  A pair overlapping with positive area is
// counted once: in the tile holding the lower-left corner of its
// intersection (both boxes are binned there, being closed-range binned).
__device__ __forceinline__ bool strict_overlap(int4 a, int4 b) {
  return max(a.x, b.x) < min(a.z, b.z) && max(a.y, b.y) < min(a.w, b.w);
}
__device__ __forceinline__ bool counted_here(int4 ba, int4 bb, int g, int tx, int ty) {
  return strict_overlap(ba, bb) && (max(ba.x, bb.x) >> g) == tx && (max(ba.y, bb.y) >> g) == ty;
}
__device__ __forceinline__ void tile_xy(const DLayer* bin, long long t, int* tx, int* ty) {
  const int4 w = bin->win[0];
  const long long li = t - bin->tbase[0];
  *tx = w.x + (int)(li % w.z);
  *ty = w.y + (int)(li / w.z);
}

__global__ void __launch_bounds__(UF_WARPS * 32) k_pair_stats_warp(const DLayer* raw, const DLayer* bin, int g,
                                                                 unsigned char* touched,
                                                                 unsigned long long* strict, DStatus* st) {
  __shared__ TileBoxes<UF_WARP_BOXES> tb[UF_WARPS];
  if (st->err) return;
  const TileBoxes<UF_WARP_BOXES>& s = tb[gb_warp()];
  int tx = 0, ty = 0;
  unsigned long long cnt = 0;
  warp_tiles(
      raw, bin, tb, [&](int, long long t) { tile_xy(bin, t, &tx, &ty); },
      [&](int j, int a0, unsigned m) {
        const int4 b = s.box[j];
        for (; m; m &= m - 1)
          if (counted_here(s.box[a0 + __ffs(m) - 1], b, g, tx, ty)) ++cnt;
      },
      [&](int, unsigned hit) {
#pragma unroll
        for (int u = 0; u < UF_LB; ++u)
          if ((hit >> u) & 1) touched[s.idx[u * 32 + gb_lane()]] = 1;
      });
  cnt = gb_warp_sum(cnt);
  if (gb_lane() == 0 && cnt) atomicAdd(strict, cnt);
}

// Tiles of more than UF_WARP_BOXES boxes, one per CTA.
__global__ void __launch_bounds__(256) k_pair_stats(const DLayer* raw, const DLayer* bin, int g,
                                                    unsigned char* touched, unsigned long long* strict,
                                                    DStatus* st) {
  __shared__ TileBoxes<UF_SMEM_BOXES> s;
  __shared__ unsigned char met[UF_SMEM_BOXES];
  if (st->err) return;
  int tx = 0, ty = 0;
  unsigned long long cnt = 0;
  cta_tiles(
      raw, bin, s,
      [&](int k, long long t) {
        tile_xy(bin, t, &tx, &ty);
        for (int j = threadIdx.x; j < min(k, UF_SMEM_BOXES); j += blockDim.x) met[j] = 0;
      },
      [&](int a, int b, int ia, int4 ba, int ib, int4 bb) {
        if (a < 0) {
          touched[ia] = 1;
          touched[ib] = 1;
        } else {
          met[a] = 1;
          met[b] = 1;
        }
        if (counted_here(ba, bb, g, tx, ty)) ++cnt;
      },
      [&](int k) {
        for (int j = threadIdx.x; j < k; j += blockDim.x)
          if (met[j]) touched[s.idx[j]] = 1;
      });
  cnt = gb_warp_sum(cnt);
  if (gb_lane() == 0 && cnt) atomicAdd(strict, cnt);
}

__global__ void k_singletons(const unsigned char* touched, long long n, unsigned char* mask,
                             unsigned long long* nsingle) {
  unsigned long long ns = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const unsigned char s = touched[i] ? 0 : 1;
    if (mask) mask[i] = s;
    ns += s;
  }
  ns = gb_warp_sum(ns);
  if (gb_lane() == 0 && ns) atomicAdd(nsingle, ns);
}

__global__ void k_uf_flatten(int* parent, const unsigned char* touched, int* flag, long long n,
                             long long* nsingle) {
  long long ns = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = uf_find(parent, (int)i);
    parent[i] = r;
    flag[i] = (touched[i] && r == (int)i) ? 1 : 0;
    ns += touched[i] ? 0 : 1;
  }
  ns = gb_warp_sum(ns);
  if (gb_lane() == 0 && ns) atomicAdd((unsigned long long*)nsingle, (unsigned long long)ns);
}

__global__ void k_uf_label(const int* parent, const unsigned char* touched, const long long* map,
                           long long* labels, long long n, const long long* nroots,
                           const long long* nsingle, long long* ncomp) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    labels[i] = touched[i] ? map[parent[i]] + 1 : 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *ncomp = *nroots + *nsingle;
}

__global__ void k_zero_ll(long long* p, int n) {
  if (threadIdx.x < n) p[threadIdx.x] = 0;
}
__global__ void k_set_ptrs(long long* slots, int* flag, long long* map, long long n) {
  slots[8] = (long long)flag;
  slots[9] = (long long)map;
  slots[10] = n;
}

void gb_launch_pair_stats(GbCtx& c, const DLayer* raw, DLayer* binidx, int g, unsigned char* touched,
                          long long n, unsigned long long* strict_dev, unsigned long long* single_dev,
                          unsigned char* mask_dev) {
  cudaMemsetAsync(touched, 0, (size_t)n, c.stream);
  cudaMemsetAsync(strict_dev, 0, 8, c.stream);
  cudaMemsetAsync(single_dev, 0, 8, c.stream);
  k_pair_stats_warp<<<c.nsm * 8, UF_WARPS * 32, 0, c.stream>>>(raw, binidx, g, touched, strict_dev, c.st);
  k_pair_stats<<<c.nsm * 4, 256, 0, c.stream>>>(raw, binidx, g, touched, strict_dev, c.st);
  k_singletons<<<c.work_blocks, 256, 0, c.stream>>>(touched, n, mask_dev, single_dev);
  c.launches += 3;
}

void gb_launch_components(GbCtx& c, const DLayer* raw, DLayer* binidx, int* parent,
                          unsigned char* touched, long long* labels, long long n,
                          long long* out_ncomp_dev, int* flag_tmp, long long* map_tmp) {
  const int wb = c.work_blocks;
  long long* sl = c.dscal;  // [4] nsingle, [5] nroots, [8..10] scan pointer slots
  k_zero_ll<<<1, 32, 0, c.stream>>>(sl + 4, 2);
  k_uf_init<<<wb, 256, 0, c.stream>>>(parent, touched, n);
  k_uf_tile_warp<<<c.nsm * 8, UF_WARPS * 32, 0, c.stream>>>(raw, binidx, parent, touched, c.st);
  k_uf_tile<<<c.nsm * 4, 256, 0, c.stream>>>(raw, binidx, parent, touched, c.st);
  k_uf_flatten<<<wb, 256, 0, c.stream>>>(parent, touched, flag_tmp, n, sl + 4);
  k_set_ptrs<<<1, 1, 0, c.stream>>>(sl, flag_tmp, map_tmp, n);
  gb_launch_scan_i32(c, (int* const*)&sl[8], (long long* const*)&sl[9], &sl[10], sl + 5);
  k_uf_label<<<wb, 256, 0, c.stream>>>(parent, touched, map_tmp, labels, n, sl + 5, sl + 4,
                                       out_ncomp_dev);
}
