// gb_bin.cu -- device-sized scans, tile windows and the binning (split) pass.
//
// Binning is a counting sort of box pieces by tile: per-cell bounding boxes
// give a dense tile window, every (grown) box adds one to each tile it covers,
// an exclusive scan turns counts into starts, and a scatter writes the clipped
// 8-byte tile-relative pieces.  The order of pieces inside a tile is not
// significant: the tile kernel is order independent.
#include "gb_internal.h"
#include "gb_scan.cuh"

#define KID_BBOX 10
#define KID_WINDOW 11
#define KID_ALLOC 12
#define KID_SCAN 13
#define KID_EXPORT 14
#define KID_FRAME 50

// Setup kernels of a layer's chain are a few microseconds of launch and memory
// latency each, so they are few: a binning of raw boxes is five launches
// (setup, count, two of the scan, scatter; thirteen took 12 us more on an
// idle chip), a Boolean three beside the tile kernel's, an export three.

// ------------------------------------------------------------------ scans
// What the last block of the first scan launch does with the total.
enum ScanHook { SCAN_TOTAL, SCAN_BIN, SCAN_EXPORT };
struct ScanEnd {
  int hook;
  long long* total;  // may be null
  DLayer* out;       // SCAN_BIN: its pieces (elem bytes each) are allocated
  int elem;
  const DLayer* src;  // SCAN_EXPORT: its tiles
  long long* dscal;   // SCAN_EXPORT: [0] box array, [1] offsets, [2] total
  DStatus* st;
};

__device__ void scan_end(const ScanEnd& e, long long total) {
  if (e.total) *e.total = total;
  if (e.hook == SCAN_BIN) {
    if (e.st->err) return;
    DLayer* O = e.out;
    O->pcs = (unsigned long long*)gb_arena_alloc(e.st, (unsigned long long)(total + 1) * e.elem, KID_ALLOC);
    O->nused = total;
    O->ntot = total;
    if (!O->pcs) O->ntiles = 0;
  } else if (e.hook == SCAN_EXPORT) {
    e.dscal[0] = e.dscal[1] = 0;
    e.dscal[2] = e.st->err ? 0 : total;
    if (e.st->err) return;
    e.dscal[1] = (long long)gb_arena_alloc(e.st, (unsigned long long)(e.src->ntiles + 1) * 8, KID_EXPORT);
    if (e.dscal[1]) e.dscal[0] = (long long)gb_arena_alloc(e.st, (unsigned long long)(total + 1) * 16, KID_EXPORT);
  }
}

// Partial sums per block; the last block to finish scans them.  part: the
// partial sums, then a ticket that is 0 between launches.
__global__ void k_scan1(int* const* inp, const long long* np, long long* part, ScanEnd e) {
  __shared__ long long tmp[33];
  __shared__ bool last;
  const int* __restrict__ in = *inp;
  const long long n = in ? *np : 0;
  const long long chunk = (n + gridDim.x - 1) / gridDim.x;
  const long long beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  long long s = 0;
  for (long long i = beg + threadIdx.x; i < end; i += blockDim.x) s += in[i];
  s = gb_block_sum(s, tmp);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd((unsigned long long*)&part[GB_SCAN_BLOCKS], 1ull) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const long long v = threadIdx.x < gridDim.x ? __ldcg(&part[threadIdx.x]) : 0;
  long long tot;
  const long long ex = gb_block_excl(v, tmp, &tot);
  if (threadIdx.x < gridDim.x) part[threadIdx.x] = ex;
  if (threadIdx.x == 0) {
    part[GB_SCAN_BLOCKS] = 0;
    scan_end(e, tot);
  }
}

// zero: the counts are cleared once read (a scatter counts them up again).
__global__ void k_scan2(int* const* inp, long long* const* outp, const long long* np, const long long* part, int zero) {
  __shared__ long long tmp[33];
  constexpr int IT = 8;
  int* in = *inp;
  long long* __restrict__ out = *outp;
  const long long n = (in && out) ? *np : 0;
  const long long chunk = (n + gridDim.x - 1) / gridDim.x;
  const long long beg = blockIdx.x * chunk, end = min(n, beg + chunk);
  long long carry = part[blockIdx.x];
  for (long long base = beg; base < end; base += (long long)blockDim.x * IT) {
    long long v[IT];
    long long s = 0;
    const long long my = base + (long long)threadIdx.x * IT;
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      v[k] = (my + k < end) ? in[my + k] : 0;
      s += v[k];
    }
    long long tot;
    long long ex = gb_block_excl(s, tmp, &tot);
    long long run = carry + ex;
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      if (my + k < end) {
        out[my + k] = run;
        if (zero) in[my + k] = 0;
      }
      run += v[k];
    }
    carry += tot;
  }
}

static void launch_scan(GbCtx& c, int* const* in_field, long long* const* out_field, const long long* n_dev,
                        const ScanEnd& e, int zero) {
  k_scan1<<<GB_SCAN_BLOCKS, GB_SCAN_THREADS, 0, c.stream>>>(in_field, n_dev, c.scan_part, e);
  k_scan2<<<GB_SCAN_BLOCKS, GB_SCAN_THREADS, 0, c.stream>>>(in_field, out_field, n_dev, c.scan_part, zero);
}

void gb_launch_scan_i32(GbCtx& c, int* const* in_field, long long* const* out_field,
                        const long long* n_dev, long long* total_dev) {
  ScanEnd e = {};
  e.hook = SCAN_TOTAL;
  e.total = total_dev;
  launch_scan(c, in_field, out_field, n_dev, e, 0);
}

// ------------------------------------------------------------------ arena
__global__ void k_arena_reset(DStatus* st, unsigned long long mark) {
  st->arena_off = mark;
}
void gb_launch_arena_reset(GbCtx& c, unsigned long long mark) {
  k_arena_reset<<<1, 1, 0, c.stream>>>(c.st, mark);
}

// ------------------------------------------------------------------ bbox
__device__ __forceinline__ bool grow_box(int4 b, int E, int N, int W, int S, int4& o) {
  // box_grow_directional (geometry.f90:184-193): x2+=E, y2+=N, x1-=W, y1-=S.
  long long x1 = (long long)b.x - W, y1 = (long long)b.y - S;
  long long x2 = (long long)b.z + E, y2 = (long long)b.w + N;
  if (!(b.x < b.z && b.y < b.w) || x1 >= x2 || y1 >= y2 || x1 < INT32_MIN || y1 < INT32_MIN ||
      x2 > INT32_MAX || y2 > INT32_MAX)
    return false;
  o = make_int4((int)x1, (int)y1, (int)x2, (int)y2);
  return true;
}

#define BIN_CELLS 16384  // cells that a one-block setup kernel fills itself

// A fresh descriptor with its per-cell arrays (one thread); false when the
// context has failed or the arena is full (the descriptor is empty then).
__device__ bool layer_fresh(DLayer* O, int ncell, int g, int binned, DStatus* st) {
  DLayer z;
  memset(&z, 0, sizeof(z));
  z.ncell = ncell;
  z.g = g;
  z.binned = binned;
  const unsigned long long c16 = ((unsigned long long)ncell * 16 + 255) & ~255ull,
                           c8 = ((unsigned long long)(ncell + 1) * 8 + 255) & ~255ull;
  char* p = st->err ? nullptr : (char*)gb_arena_alloc(st, 2 * c16 + 3 * c8, KID_ALLOC);
  if (p) {
    z.cbox = (int4*)p;
    z.win = (int4*)(p + c16);
    z.cell_count = (long long*)(p + 2 * c16);
    z.cell_area = (long long*)(p + 2 * c16 + c8);
    z.tbase = (long long*)(p + 2 * c16 + 2 * c8);
  }
  *O = z;
  return p != nullptr;
}

__device__ __forceinline__ int4 bbox_none() { return make_int4(INT32_MAX, INT32_MAX, INT32_MIN, INT32_MIN); }

// A fresh binned layer with empty bounding boxes (up to BIN_CELLS cells are
// filled here, more by k_cbox_fill).
__global__ void k_bin_init(DLayer* O, int ncell, int g, DStatus* st) {
  __shared__ bool ok;
  if (threadIdx.x == 0) ok = layer_fresh(O, ncell, g, 1, st);
  __syncthreads();
  if (!ok || ncell > BIN_CELLS) return;
  for (int k = threadIdx.x; k < ncell; k += blockDim.x) {
    O->cbox[k] = bbox_none();
    O->cell_count[k] = 0;
    O->cell_area[k] = 0;
  }
}

__global__ void k_cbox_fill(DLayer* O, int ncell, DStatus* st) {
  if (st->err) return;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < ncell; k += gridDim.x * blockDim.x) {
    O->cbox[k] = bbox_none();
    O->cell_count[k] = 0;
    O->cell_area[k] = 0;
  }
}

__device__ __forceinline__ void warp_bbox_atomic(int4* dst, int x1, int y1, int x2, int y2) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x1 = min(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y1 = min(y1, __shfl_xor_sync(0xffffffffu, y1, o));
    x2 = max(x2, __shfl_xor_sync(0xffffffffu, x2, o));
    y2 = max(y2, __shfl_xor_sync(0xffffffffu, y2, o));
  }
  if (gb_lane() == 0 && x1 <= x2) {
    atomicMin(&dst->x, x1);
    atomicMin(&dst->y, y1);
    atomicMax(&dst->z, x2);
    atomicMax(&dst->w, y2);
  }
}

// Raw-source kernels walk the boxes in one contiguous chunk per warp (the
// boxes divided evenly over the grid's warps, in multiples of 32), 32
// consecutive boxes per step (coalesced), BIN_LD steps loaded before any is
// processed.  The cell of a box comes from one search of the cell
// offsets at the chunk's start; after that a lane only steps past the cells
// that end before its box (cells are sorted and hold many boxes, so nearly
// always none), which removes the dependent chain of a binary search per box.
#define BIN_LD 4

template <int LD, typename F>
__device__ __forceinline__ void walk_raw_boxes(const int4* bx, const long long* coff, int ncell, long long n, F f) {
  const int lane = gb_lane();
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  const long long ch = max(32ll, (((n + nw - 1) / nw) + 31) & ~31ll);
  for (long long c0 = ((long long)blockIdx.x * (blockDim.x >> 5) + gb_warp()) * ch; c0 < n; c0 += nw * ch) {
    const long long c1 = min(n, c0 + ch);
    int k = 0;
    long long hi = 0;
    if (lane == 0) {
      k = gb_find_cell(coff, ncell, c0);
      hi = coff[k + 1];
    }
    k = __shfl_sync(0xffffffffu, k, 0);
    hi = __shfl_sync(0xffffffffu, hi, 0);
    for (long long b0 = c0; b0 < c1; b0 += 32 * LD) {
      int4 ld[LD];
#pragma unroll
      for (int u = 0; u < LD; ++u) {
        const long long i = b0 + 32 * u + lane;
        if (i < c1) ld[u] = bx[i];
      }
#pragma unroll
      for (int u = 0; u < LD; ++u) {
        const long long b = b0 + 32 * u;
        if (b >= c1) break;  // warp-uniform
        const long long i = b + lane;
        int kl = k;
        long long hl = hi;
        if (i < c1)
          while (i >= hl && kl + 1 < ncell) {
            ++kl;
            hl = coff[kl + 1];
          }
        f(i, i < c1, ld[u], kl);  // called by all lanes (warp collectives allowed)
        k = __shfl_sync(0xffffffffu, kl, 31);  // the last lane holds the furthest cell
        hi = __shfl_sync(0xffffffffu, hl, 31);
      }
    }
  }
}

// Raw source.  A lane keeps the bounds of its boxes in registers while the
// warp stays in one cell; the warp adds them to the cell's box when the cell
// ends, the block at its end, so a large cell takes four atomics per block
// and not four per 32 boxes (12M boxes of one cell: 1000 -> 40 us; four
// same-address atomics per 32 boxes had bound it, HBM's share is 29 us).
// Bounds that the cell's box already holds take no atomic.  A step whose
// lanes straddle cells adds its boxes lane by lane.
__device__ __forceinline__ void bbox_add(int4* dst, int4 b) {
  const int4 cur = __ldcg(dst);  // bounds only widen, so an old value costs at most an atomic
  if (b.x < cur.x) atomicMin(&dst->x, b.x);
  if (b.y < cur.y) atomicMin(&dst->y, b.y);
  if (b.z > cur.z) atomicMax(&dst->z, b.z);
  if (b.w > cur.w) atomicMax(&dst->w, b.w);
}
__device__ __forceinline__ int4 bbox_join(int4 a, int4 b) {
  return make_int4(min(a.x, b.x), min(a.y, b.y), max(a.z, b.z), max(a.w, b.w));
}
__device__ __forceinline__ int4 bbox_warp(int4 a) {
  a.x = __reduce_min_sync(0xffffffffu, a.x);
  a.y = __reduce_min_sync(0xffffffffu, a.y);
  a.z = __reduce_max_sync(0xffffffffu, a.z);
  a.w = __reduce_max_sync(0xffffffffu, a.w);
  return a;
}

__global__ void __launch_bounds__(256) k_bbox_raw(const DLayer* S, DLayer* O, int ncell, int E, int N, int W, int Sg,
                                                  DStatus* st) {
  __shared__ int4 wb[8];
  __shared__ int wk[8];
  __shared__ bool failed;
  // other blocks report errors meanwhile: one read for the whole block, whose warps' bounds meet at the end.  A raw
  // layer's own boxes (S == O) are taken whatever the status: the layer may be used after the error is cleared
  if (threadIdx.x == 0) failed = S != O && *(volatile int*)&st->err != 0;
  __syncthreads();
  if (failed) return;
  int4* const cb = O->cbox;
  int kc = -1;  // the cell whose bounds the warp holds
  int4 acc = bbox_none();
  walk_raw_boxes<BIN_LD>(S->boxes, S->coff, ncell, S->nbox, [&](long long i, bool valid_i, int4 box, int k) {
    int4 g = bbox_none();
    if (valid_i && !grow_box(box, E, N, W, Sg, g)) {
      gb_set_error(st, GB_ERR_INVALID_BOX, KID_BBOX, i);
      if (S == O) O->bad = i + 1;
      g = bbox_none();
    }
    const int k0 = __shfl_sync(0xffffffffu, k, 0);
    const bool same = __all_sync(0xffffffffu, !valid_i || k == k0);
    if (!same || k0 != kc) {
      const int4 r = bbox_warp(acc);
      if (gb_lane() == 0 && kc >= 0 && r.x <= r.z) bbox_add(&cb[kc], r);
      acc = bbox_none();
      kc = same ? k0 : -1;
    }
    if (same) acc = bbox_join(acc, g);
    else if (valid_i && g.x <= g.z) bbox_add(&cb[k], g);
  });
  acc = bbox_warp(acc);
  if (gb_lane() == 0) {
    wb[gb_warp()] = acc;
    wk[gb_warp()] = acc.x <= acc.z ? kc : -1;
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // the block's warps hold neighbouring chunks: nearly always one cell
    for (int w = 0; w < 8; ++w) {
      if (wk[w] < 0) continue;
      int4 b = wb[w];
      for (int v = w + 1; v < 8; ++v)
        if (wk[v] == wk[w]) {
          b = bbox_join(b, wb[v]);
          wk[v] = -1;
        }
      bbox_add(&cb[wk[w]], b);
    }
  }
}

__device__ __forceinline__ void tile_of_index(const DLayer* L, long long t, int& k, int& tx, int& ty) {
  k = gb_find_cell(L->tbase, L->ncell, t);
  const int4 w = L->win[k];
  const long long li = t - L->tbase[k];
  tx = w.x + (int)(li % w.z);
  ty = w.y + (int)(li / w.z);
}

// Who takes a tile of a binned source: a warp, or with few tiles a block.
struct TileTeam {
  bool block;
  long long first, step;  // tiles
  int at, size;           // the thread's first piece and the step
  __device__ explicit TileTeam(long long nt) : block(nt <= gridDim.x) {
    const int wpb = blockDim.x >> 5;
    first = block ? (long long)blockIdx.x : (long long)blockIdx.x * wpb + gb_warp();
    step = block ? (long long)gridDim.x : (long long)gridDim.x * wpb;
    at = block ? (int)threadIdx.x : gb_lane();
    size = block ? (int)blockDim.x : 32;
  }
  __device__ __forceinline__ void sync() const {
    if (block) __syncthreads();
    else __syncwarp();
  }
};

// Binned source: a warp or a block per source tile.
__global__ void __launch_bounds__(256) k_bbox_bin(const DLayer* S, DLayer* O, int E, int N, int W, int Sg, DStatus* st) {
  if (st->err) return;
  const long long nt = S->ntiles;
  const int g = S->g;
  const TileTeam team(nt);
  for (long long t = team.first; t < nt; t += team.step) {
    const int cnt = S->tcount[t];
    if (cnt == 0) continue;
    int k, tx, ty;
    tile_of_index(S, t, k, tx, ty);
    const unsigned long long* p = S->pcs + S->tstart[t];
    const int ox = tx << g, oy = ty << g;
    int x1 = INT32_MAX, y1 = INT32_MAX, x2 = INT32_MIN, y2 = INT32_MIN;
    for (int j = team.at; j < cnt; j += team.size) {
      int a, b, c, d;
      gb_unpack(p[j], a, b, c, d);
      int4 gbx;
      if (!grow_box(make_int4(ox + a, oy + b, ox + c, oy + d), E, N, W, Sg, gbx)) {
        gb_set_error(st, GB_ERR_INVALID_BOX, KID_BBOX, t);
        continue;
      }
      x1 = min(x1, gbx.x); y1 = min(y1, gbx.y); x2 = max(x2, gbx.z); y2 = max(y2, gbx.w);
    }
    warp_bbox_atomic(&O->cbox[k], x1, y1, x2, y2);
  }
}

// ------------------------------------------------------------------ windows
// One block: per-cell tile window from the cell bbox, scan into tbase,
// allocate the per-tile arrays and clear the counts.  closed=1 uses closed
// tile ranges (x2 >> g).
__device__ void window_block(DLayer* O, int ncell, int g, int closed, DStatus* st) {
  __shared__ long long tmp[33];
  __shared__ long long carry;
  __shared__ int* counts;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < ncell; base += blockDim.x) {
    const int k = base + threadIdx.x;
    long long nt = 0;
    if (k < ncell) {
      int4 b = O->cbox[k];
      int4 w = make_int4(0, 0, 0, 0);
      if (b.x <= b.z && b.y <= b.w && (closed || (b.x < b.z && b.y < b.w))) {
        const int tx0 = gb_floor_shift(b.x, g), ty0 = gb_floor_shift(b.y, g);
        const int tx1 = closed ? gb_floor_shift(b.z, g) : gb_floor_shift(b.z - 1, g);
        const int ty1 = closed ? gb_floor_shift(b.w, g) : gb_floor_shift(b.w - 1, g);
        w = make_int4(tx0, ty0, tx1 - tx0 + 1, ty1 - ty0 + 1);
        nt = (long long)w.z * w.w;
      }
      O->win[k] = w;
    }
    long long tot;
    long long ex = gb_block_excl(nt, tmp, &tot);
    if (k < ncell) O->tbase[k] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const long long total = carry;
    counts = nullptr;
    O->tbase[ncell] = total;
    O->ntiles = total;
    O->g = g;
    O->binned = 1;
    if (total > GB_MAX_TILES_PER_OP) {
      gb_set_error(st, GB_ERR_CAPACITY, KID_WINDOW, total);
      O->ntiles = 0;
    } else {
      const unsigned long long b8 = ((unsigned long long)(total + 1) * 8 + 255) & ~255ull;
      char* p = (char*)gb_arena_alloc(st, b8 + (unsigned long long)(total + 1) * 4, KID_ALLOC);
      if (p) {
        O->tstart = (long long*)p;
        counts = O->tcount = (int*)(p + b8);
      } else {
        O->ntiles = 0;
      }
    }
  }
  __syncthreads();
  if (!counts) return;
  int4* z = reinterpret_cast<int4*>(counts);  // the allocation is whole 256 bytes
  for (long long i = threadIdx.x; i < (carry + 3) / 4; i += blockDim.x) z[i] = make_int4(0, 0, 0, 0);
}

__global__ void __launch_bounds__(1024) k_window(DLayer* O, int ncell, int g, int closed, DStatus* st) {
  if (st->err) return;
  window_block(O, ncell, g, closed, st);
}

// One block, raw source, boxes not shrunk, at most BIN_CELLS cells: the cells'
// bounding boxes are the source's, grown, so the binning needs no pass over
// the boxes for them.
__global__ void __launch_bounds__(1024) k_bin_setup(const DLayer* S, DLayer* O, int ncell, int g, int closed, int E, int N,
                                                    int W, int Sg, DStatus* st) {
  __shared__ bool ok;
  if (threadIdx.x == 0) {
    ok = layer_fresh(O, ncell, g, 1, st);
    if (ok && S->bad) {  // reported again, as a pass over the boxes would
      gb_set_error(st, GB_ERR_INVALID_BOX, KID_BBOX, S->bad - 1);
      ok = false;
    }
  }
  __syncthreads();
  const bool go = ok;
  __syncthreads();  // read by all before a thread clears it below
  if (!go) return;
  for (int k = threadIdx.x; k < ncell; k += blockDim.x) {
    const int4 b = S->cbox[k];
    int4 o = bbox_none();
    if (b.x <= b.z && !grow_box(b, E, N, W, Sg, o)) {  // past int32: so is a box at that bound
      gb_set_error(st, GB_ERR_INVALID_BOX, KID_BBOX, S->coff[k]);
      ok = false;
    }
    O->cbox[k] = o;
    O->cell_count[k] = 0;
    O->cell_area[k] = 0;
  }
  __syncthreads();
  if (ok) window_block(O, ncell, g, closed, st);
}

// ------------------------------------------------------------------ count / scatter
// MODE 0: half-open tile ranges, packed pieces; MODE 1: closed ranges, int index payload.
// Raw source, one contiguous chunk of boxes per block.  The tiles of the
// chunk's cells are counted in shared memory (up to SPLIT_SM tiles; layers of
// a few hundred tiles had been bound by global atomics on those few counters:
// 1M boxes over 400 tiles, count 173 -> 15 us, scatter 178 -> 25 us).  Count:
// the block adds its counts to the layer's once.  Scatter: the block counts
// its chunk, reserves each tile's slots with one atomic, and places the
// pieces on a second walk over the chunk.  A chunk over more tiles takes its
// slots from the global counters, which many tiles spread.  A box over more
// than SPLIT_WIDE tiles (the one-box frames of an erosion's cells cover them
// all) is left to the whole block after the walk: one lane had walked its tiles
// in series (1200 tiles, 280 us), and blocks of 512 such frames took 140 us.
#define SPLIT_SM 8192
#define SPLIT_SM_MIN 32768  // smaller layers: the counters see few atomics, and the second walk costs more
#define SPLIT_WIDE 8
#define SPLIT_NWIDE 64  // wide boxes of one chunk held for the block; more are walked by their lanes

struct SplitBox {
  int4 b;
  long long idx;
  int k;
};

// Tile ranges of a box in its cell: half-open extents (MODE 0) or closed.
template <int MODE>
__device__ __forceinline__ int4 box_tiles(int4 b, int g) {
  return make_int4(gb_floor_shift(b.x, g), gb_floor_shift(b.y, g), gb_floor_shift(MODE ? b.z : b.z - 1, g),
                   gb_floor_shift(MODE ? b.w : b.w - 1, g));
}

template <int MODE>
__device__ __forceinline__ void put_piece(DLayer* O, long long pos, int4 b, long long idx, int tx, int ty, int g) {
  if (MODE == 0) {
    const int ox = tx << g, oy = ty << g;
    const int x1 = max(b.x, ox) - ox, y1 = max(b.y, oy) - oy;
    const int x2 = (int)(min((long long)b.z, (long long)ox + (1ll << g)) - ox);
    const int y2 = (int)(min((long long)b.w, (long long)oy + (1ll << g)) - oy);
    O->pcs[pos] = gb_pack(x1, y1, x2, y2);
  } else {
    ((int*)O->pcs)[pos] = (int)idx;
  }
}

template <int MODE, bool SCATTER>
__global__ void __launch_bounds__(256) k_split_raw(const DLayer* S, DLayer* O, int ncell, int g, int E, int N, int W,
                                                   int Sg, DStatus* st) {
  __shared__ int hist[SPLIT_SM];
  __shared__ SplitBox wide[SPLIT_NWIDE];
  __shared__ int nwide;
  if (st->err) return;
  const long long n = S->nbox;
  const int4* const bx = S->boxes;
  const long long* const coff = S->coff;
  const int4* const win = O->win;
  const long long* const tbase = O->tbase;
  int* const tcount = O->tcount;
  const long long* const tstart = O->tstart;
  const int nt = blockDim.x, tid = threadIdx.x;
  // few boxes are spread over the blocks (they may all be wide), many in whole warps
  const long long even = (n + gridDim.x - 1) / gridDim.x;
  const long long ch = n < SPLIT_SM_MIN ? even : (even + nt - 1) / nt * nt;
  const long long c0 = (long long)blockIdx.x * ch, c1 = min(n, c0 + ch);
  if (c0 >= n) return;
  const int k0 = gb_find_cell(coff, ncell, c0), k1 = gb_find_cell(coff, ncell, c1 - 1);
  const long long r0 = tbase[k0], nr = tbase[k1 + 1] - r0;
  const bool sm = nr <= SPLIT_SM && n >= SPLIT_SM_MIN;
  if (sm)
    for (int i = tid; i < (int)nr; i += nt) hist[i] = 0;
  // one tile of a box: count it (PLACE = 0) or take its slot and write the piece
  auto visit = [&](bool place, int4 b, long long idx, int tx, int ty, long long t) {
    if (!place) {
      if (sm) atomicAdd(&hist[t - r0], 1);
      else atomicAdd(&tcount[t], 1);
    } else {
      const int slot = sm ? atomicAdd(&hist[t - r0], 1) : atomicAdd(&tcount[t], 1);
      put_piece<MODE>(O, tstart[t] + slot, b, idx, tx, ty, g);
    }
  };
  auto walk = [&](bool place) {
    if (tid == 0) nwide = 0;
    __syncthreads();
    int kc = -1;
    int4 w = make_int4(0, 0, 0, 0);
    long long tb = 0;
    for (long long i0 = c0 + tid; i0 < c1; i0 += (long long)nt * BIN_LD) {
      int4 ld[BIN_LD];
#pragma unroll
      for (int u = 0; u < BIN_LD; ++u)
        if (i0 + (long long)u * nt < c1) ld[u] = bx[i0 + (long long)u * nt];
#pragma unroll
      for (int u = 0; u < BIN_LD; ++u) {
        const long long i = i0 + (long long)u * nt;
        if (i >= c1) break;
        int4 b;
        if (!grow_box(ld[u], E, N, W, Sg, b)) continue;  // invalid: reported by k_bbox_raw
        if (kc < 0 || i >= coff[kc + 1]) {
          kc = k0 == k1 ? k0 : k0 + gb_find_cell(coff + k0, k1 + 1 - k0, i);
          w = win[kc];
          tb = tbase[kc];
        }
        const int4 q = box_tiles<MODE>(b, g);
        if ((long long)(q.z - q.x + 1) * (q.w - q.y + 1) > SPLIT_WIDE) {
          const int at = atomicAdd(&nwide, 1);
          if (at < SPLIT_NWIDE) {
            wide[at].b = b;
            wide[at].idx = i;
            wide[at].k = kc;
            continue;
          }
        }
        for (int ty = q.y; ty <= q.w; ++ty)
          for (int tx = q.x; tx <= q.z; ++tx)
            visit(place, b, i, tx, ty, tb + (long long)(ty - w.y) * w.z + (tx - w.x));
      }
    }
    __syncthreads();
    const int nb = min(nwide, SPLIT_NWIDE);
    for (int j = 0; j < nb; ++j) {
      const SplitBox s = wide[j];
      const int4 q = box_tiles<MODE>(s.b, g), ws = win[s.k];
      const long long sx = q.z - q.x + 1, tot = sx * (q.w - q.y + 1);
      for (long long v = tid; v < tot; v += nt) {
        const int ty = q.y + (int)(v / sx), tx = q.x + (int)(v % sx);
        visit(place, s.b, s.idx, tx, ty, tbase[s.k] + (long long)(ty - ws.y) * ws.z + (tx - ws.x));
      }
    }
    __syncthreads();
  };
  if (!SCATTER) {
    walk(false);
    if (sm)
      for (int i = tid; i < (int)nr; i += nt)
        if (hist[i]) atomicAdd(&tcount[r0 + i], hist[i]);
    return;
  }
  if (sm) {
    walk(false);
    for (int i = tid; i < (int)nr; i += nt)
      if (hist[i]) hist[i] = atomicAdd(&tcount[r0 + i], hist[i]);
    __syncthreads();
  }
  walk(true);
}

// Binned source, a warp or a block per source tile.  A grown piece of one tile lies in
// the tile of the target that the source tile maps to and its eight neighbours
// (the same grid, grown by less than a tile), so the team keeps nine counters:
// count adds them to the layer's at the end; scatter counts its tile, reserves
// nine ranges and places the pieces in a second walk.  (Global atomics for
// every group of 32 pieces and target tile, pieces on tile edges one by one:
// count 247, scatter 378 us per 512 cells of an OP1 deck; now 132 and 260.)  Other pieces take their slots from the layer's counters.
template <bool SCATTER>
__global__ void __launch_bounds__(256) k_split_bin(const DLayer* S, DLayer* O, int g, int E, int N, int W, int Sg,
                                                   DStatus* st) {
  __shared__ int near[8][9];
  if (st->err) return;
  const long long nt = S->ntiles;
  const int sg = S->g;
  const TileTeam team(nt);
  int* const cn = near[team.block ? 0 : gb_warp()];
  int* const tcount = O->tcount;
  const long long* const tstart = O->tstart;
  for (long long t = team.first; t < nt; t += team.step) {
    const int cnt = S->tcount[t];
    if (cnt == 0) continue;
    int k, tx, ty;
    tile_of_index(S, t, k, tx, ty);
    const unsigned long long* p = S->pcs + S->tstart[t];
    const int ox = tx << sg, oy = ty << sg;
    const int4 w = O->win[k];
    const long long tb = O->tbase[k];
    const bool same = sg == g;
    auto index = [&](int x, int y) { return tb + (long long)(y - w.y) * w.z + (x - w.x); };
    if (team.at < 9) cn[team.at] = 0;
    team.sync();
    auto walk = [&](bool place) {
      for (int j = team.at; j < cnt; j += team.size) {
        int a, b, c, d;
        gb_unpack(p[j], a, b, c, d);
        int4 o;
        if (!grow_box(make_int4(ox + a, oy + b, ox + c, oy + d), E, N, W, Sg, o)) continue;
        const int4 q = box_tiles<0>(o, g);
        const bool in9 = same && q.x >= tx - 1 && q.z <= tx + 1 && q.y >= ty - 1 && q.w <= ty + 1;
        for (int y = q.y; y <= q.w; ++y)
          for (int x = q.x; x <= q.z; ++x) {
            if (in9) {
              const int i = (y - ty + 1) * 3 + (x - tx + 1);
              const int s = atomicAdd(&cn[i], 1);
              if (place) put_piece<0>(O, tstart[index(x, y)] + s, o, 0, x, y, g);
            } else if (SCATTER ? place : !place) {
              const int s = atomicAdd(&tcount[index(x, y)], 1);
              if (place) put_piece<0>(O, tstart[index(x, y)] + s, o, 0, x, y, g);
            }
          }
      }
      team.sync();
    };
    walk(false);
    const int i9 = team.at;
    if (i9 < 9 && cn[i9]) {
      const int base = atomicAdd(&tcount[index(tx + i9 % 3 - 1, ty + i9 / 3 - 1)], cn[i9]);
      if (SCATTER) cn[i9] = base;
    }
    team.sync();
    if (SCATTER) walk(true);
  }
}

// ------------------------------------------------------------------ launchers
static void launch_bin_common(GbCtx& c, const DLayer* src, int src_binned, DLayer* out, int ncell,
                              int g, int E, int N, int W, int S, int mode) {
  const int wb = c.work_blocks, T = 256;
  if (!src_binned && ncell <= BIN_CELLS && E >= 0 && N >= 0 && W >= 0 && S >= 0) {
    k_bin_setup<<<1, 1024, 0, c.stream>>>(src, out, ncell, g, mode, E, N, W, S, c.st);
  } else {
    k_bin_init<<<1, 1024, 0, c.stream>>>(out, ncell, g, c.st);
    if (ncell > BIN_CELLS) k_cbox_fill<<<(ncell + 255) / 256, 256, 0, c.stream>>>(out, ncell, c.st);
    if (src_binned) k_bbox_bin<<<wb, T, 0, c.stream>>>(src, out, E, N, W, S, c.st);
    else k_bbox_raw<<<wb, T, 0, c.stream>>>(src, out, ncell, E, N, W, S, c.st);
    k_window<<<1, 1024, 0, c.stream>>>(out, ncell, g, mode, c.st);
  }
  if (mode == 0) {
    if (src_binned) k_split_bin<false><<<wb, T, 0, c.stream>>>(src, out, g, E, N, W, S, c.st);
    else k_split_raw<0, false><<<wb, T, 0, c.stream>>>(src, out, ncell, g, E, N, W, S, c.st);
  } else {
    k_split_raw<1, false><<<wb, T, 0, c.stream>>>(src, out, ncell, g, 0, 0, 0, 0, c.st);
  }
  ScanEnd e = {};
  e.hook = SCAN_BIN;
  e.total = &out->npcs;
  e.out = out;
  e.elem = mode == 0 ? 8 : 4;
  e.st = c.st;
  launch_scan(c, &out->tcount, &out->tstart, &out->ntiles, e, 1);
  if (mode == 0) {
    if (src_binned) k_split_bin<true><<<wb, T, 0, c.stream>>>(src, out, g, E, N, W, S, c.st);
    else k_split_raw<0, true><<<wb, T, 0, c.stream>>>(src, out, ncell, g, E, N, W, S, c.st);
  } else {
    k_split_raw<1, true><<<wb, T, 0, c.stream>>>(src, out, ncell, g, 0, 0, 0, 0, c.st);
  }
}

void gb_launch_rebin(GbCtx& c, const DLayer* src, int src_binned, DLayer* out, int ncell, int g,
                     int E, int N, int W, int S) {
  launch_bin_common(c, src, src_binned, out, ncell, g, E, N, W, S, 0);
}

void gb_launch_bin_index(GbCtx& c, const DLayer* src, DLayer* out, int ncell, int g) {
  launch_bin_common(c, src, 0, out, ncell, g, 0, 0, 0, 0, 1);
}

// Per-cell bounding box of a raw layer (no grow) into its own cbox, which
// starts empty.
void gb_launch_cell_bbox_fill(GbCtx& c, DLayer* L, int ncell) {
  k_bbox_raw<<<c.work_blocks, 256, 0, c.stream>>>(L, L, ncell, 0, 0, 0, 0, c.st);
}

// A raw layer's descriptor, per-cell arrays empty; one_cell: its offsets too.
__global__ void k_raw_desc(DLayer* d, DLayer v, bool one_cell) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0) {
    *d = v;
    if (one_cell) {
      v.coff[0] = 0;
      v.coff[1] = v.nbox;
    }
  }
  if (k < v.ncell) {
    v.cbox[k] = bbox_none();
    v.cell_count[k] = 0;
    v.cell_area[k] = 0;
  }
}

void gb_launch_raw_desc(GbCtx& c, DLayer* d, const DLayer& v, bool one_cell) {
  k_raw_desc<<<(v.ncell + 255) / 256, 256, 0, c.stream>>>(d, v, one_cell);
}

// Frame of an erosion: per cell the cell bbox grown by t (a superset of
// bbox(P) (+) t is all the construction needs); empty cells get a unit box,
// which leaves their (empty) result unchanged.  A fresh raw layer, one block.
__global__ void __launch_bounds__(1024) k_frame(const DLayer* P, DLayer* F, int ncell, int g, int t, DStatus* st) {
  __shared__ bool ok;
  if (threadIdx.x == 0) {
    ok = layer_fresh(F, ncell, g, 0, st);
    if (ok) {
      F->boxes = (int4*)gb_arena_alloc(st, (unsigned long long)ncell * 16, KID_FRAME);
      F->coff = (long long*)gb_arena_alloc(st, (unsigned long long)(ncell + 1) * 8, KID_FRAME);
      F->nbox = ncell;
      ok = F->boxes && F->coff;
      if (ok) F->coff[ncell] = ncell;
    }
  }
  __syncthreads();
  if (!ok) return;
  for (int k = threadIdx.x; k < ncell; k += blockDim.x) {
    const int4 b = P->cbox[k];
    int4 o = make_int4(0, 0, 1, 1);
    if (b.x < b.z && b.y < b.w) {
      const long long x1 = (long long)b.x - t, y1 = (long long)b.y - t;
      const long long x2 = (long long)b.z + t, y2 = (long long)b.w + t;
      if (x1 < INT32_MIN || y1 < INT32_MIN || x2 > INT32_MAX || y2 > INT32_MAX) {
        gb_set_error(st, GB_ERR_INVALID_BOX, KID_FRAME, k);
      } else {
        o = make_int4((int)x1, (int)y1, (int)x2, (int)y2);
      }
    }
    F->boxes[k] = o;
    F->coff[k] = k;
    F->cbox[k] = o;
    F->cell_count[k] = 1;
    F->cell_area[k] = 0;
  }
}

void gb_launch_frame(GbCtx& c, const DLayer* P, DLayer* F, int ncell, int g, int t) {
  k_frame<<<1, 1024, 0, c.stream>>>(P, F, ncell, g, t, c.st);
}

// ------------------------------------------------------------------ Boolean op setup
__device__ __forceinline__ int tile_index_in(const DLayer* L, int k, int tx, int ty, long long* t) {
  if (L == nullptr) return 0;
  const int4 w = L->win[k];
  if (tx < w.x || ty < w.y || tx >= w.x + w.z || ty >= w.y + w.w) return 0;
  *t = L->tbase[k] + (long long)(ty - w.y) * w.z + (tx - w.x);
  return 1;
}

// Output window per cell: the union of both windows for OR / XOR, A's window
// otherwise (AND, NOT and MERGE results lie inside A).  One block: the fresh
// result layer, its windows and per-tile arrays, its output pool, and the tile
// kernel's work counters at zero.
// Output pool (factor > 0): factor x (pieces of A + pieces of B) plus a
// little per tile.  Each tile reserves exactly its strip count from the pool
// cursor (nused) once it knows it, so no per-tile slack is needed; a tile
// that no longer fits takes its slots from the arena directly (atomically),
// at an offset relative to the pool base.
__global__ void __launch_bounds__(1024) k_bool_window(int op, const DLayer* A, const DLayer* B, DLayer* O, int ncell, int g,
                                                      int factor, bool descs, long long* counter, DStatus* st) {
  __shared__ long long tmp[33];
  __shared__ long long carry;
  __shared__ bool ok;
  if (threadIdx.x == 0) {
    carry = 0;
    counter[0] = 0;
    counter[2] = 0;
    ok = layer_fresh(O, ncell, g, 1, st);
  }
  __syncthreads();
  if (!ok) return;
  for (int base = 0; base < ncell; base += blockDim.x) {
    const int k = base + threadIdx.x;
    long long nt = 0;
    if (k < ncell) {
      int4 wa = A->win[k];
      int4 w = wa;
      if ((op == GB_OP_OR || op == GB_OP_XOR) && B) {
        int4 wb = B->win[k];
        if (wa.z == 0 || wa.w == 0) w = wb;
        else if (wb.z > 0 && wb.w > 0) {
          const int x0 = min(wa.x, wb.x), y0 = min(wa.y, wb.y);
          const int x1 = max(wa.x + wa.z, wb.x + wb.z), y1 = max(wa.y + wa.w, wb.y + wb.w);
          w = make_int4(x0, y0, x1 - x0, y1 - y0);
        }
      }
      if (w.z <= 0 || w.w <= 0) w = make_int4(0, 0, 0, 0);
      O->win[k] = w;
      O->cell_count[k] = 0;
      O->cell_area[k] = 0;
      O->cbox[k] = make_int4(w.x << g, w.y << g, (w.x + w.z) << g, (w.y + w.w) << g);
      nt = (long long)w.z * w.w;
    }
    long long tot;
    long long ex = gb_block_excl(nt, tmp, &tot);
    if (k < ncell) O->tbase[k] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const long long total = carry;
    O->tbase[ncell] = total;
    O->ntiles = total;
    if (total > GB_MAX_TILES_PER_OP) {
      gb_set_error(st, GB_ERR_CAPACITY, KID_WINDOW, total);
      O->ntiles = 0;
      return;
    }
    const unsigned long long b8 = ((unsigned long long)(total + 1) * 8 + 255) & ~255ull,
                             b4 = ((unsigned long long)(total + 1) * 4 + 255) & ~255ull;
    char* p = (char*)gb_arena_alloc(st, b8 + b4 + (descs ? (unsigned long long)(total + 1) * sizeof(TileDesc) : 0), KID_ALLOC);
    if (!p) {
      O->ntiles = 0;
      return;
    }
    O->tstart = (long long*)p;
    O->tcount = (int*)(p + b8);
    O->tdesc = descs ? (TileDesc*)(p + b8 + b4) : nullptr;
    if (factor <= 0) return;
    const long long na = A->ntot, nb = B && op != GB_OP_MERGE ? B->ntot : 0;
    O->npcs = (na + nb) * factor + 16 * total + 64;
    O->pcs = (unsigned long long*)gb_arena_alloc(st, (unsigned long long)O->npcs * 8, KID_ALLOC);
    if (!O->pcs) O->ntiles = 0;
  }
}

// Every output tile's cell and the operands' pieces of that tile, so the tile
// kernel looks a tile up with one load.  Only B's pieces of a two-operand op.
__global__ void k_tile_descs(int op, const DLayer* A, const DLayer* B, DLayer* O, DStatus* st) {
  if (st->err) return;
  const long long n = O->ntiles;
  const bool useB = B && op != GB_OP_MERGE && op != GB_OP_OVERLAP;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int k = gb_find_cell(O->tbase, O->ncell, t);
    const int4 w = O->win[k];
    const long long li = t - O->tbase[k];
    const int tx = w.x + (int)(li % w.z), ty = w.y + (int)(li / w.z);
    TileDesc d;
    d.cell = k;
    d.nA = d.nB = d.pad = 0;
    d.offA = d.offB = 0;
    long long ta = 0, tb = 0;
    if (tile_index_in(A, k, tx, ty, &ta)) {
      d.nA = A->tcount[ta];
      d.offA = A->tstart[ta];
    }
    if (useB && tile_index_in(B, k, tx, ty, &tb)) {
      d.nB = B->tcount[tb];
      d.offB = B->tstart[tb];
    }
    O->tdesc[t] = d;
  }
}

void gb_launch_bool_setup(GbCtx& c, int op, const DLayer* A, const DLayer* B, DLayer* O, int ncell,
                          int g, int alloc_slots) {
  // One cell: the tile kernel looks its tiles up in two loads more than a descriptor takes, while the tile before
  // is stitched, so a launch less is worth more (an AND of 1237 and 911 boxes 208 -> 203 us, 40 served requests 1992 ->
  // 1954 us).  Not in area mode (no slots), which has nothing to hide the loads, nor on smaller grids than the default,
  // whose tiles are more and smaller (300000 boxes, two layers: XOR on grid 2^10 67.2 -> 58.1 ms, on 2^12 6.4 -> 5.9).
  const bool descs = ncell > 1 || !alloc_slots || g < 16;
  k_bool_window<<<1, 1024, 0, c.stream>>>(op, A, B, O, ncell, g, alloc_slots ? c.cap_factor : 0, descs, c.tile_counter, c.st);
  if (descs) k_tile_descs<<<c.work_blocks, 256, 0, c.stream>>>(op, A, B, O, c.st);
}

// ------------------------------------------------------------------ export
// Slots of c.dscal used by the export: [0] = int4* array, [1] = offsets*, [2] = total.
// One contiguous chunk of output boxes per warp; the tile of the first comes
// from a search of the offsets, after that a lane steps over the tiles that
// end before its box.  (A warp per tile left the chip idle on few dense tiles:
// 3.1M strips of 400 tiles 136 us, now 20.)
__global__ void __launch_bounds__(256) k_export(const DLayer* L, const long long* dscal, DStatus* st) {
  if (st->err) return;
  int4* out = (int4*)dscal[0];
  const long long* off = (const long long*)dscal[1];
  if (!out || !off) return;
  const long long nt = L->ntiles, n = dscal[2];
  const int g = L->g, lane = gb_lane();
  const long long nw = (long long)gridDim.x * (blockDim.x >> 5);
  const long long ch = max(32ll, (((n + nw - 1) / nw) + 31) & ~31ll);
  const long long c0 = ((long long)blockIdx.x * (blockDim.x >> 5) + gb_warp()) * ch, c1 = min(n, c0 + ch);
  long long t = -1, hi = 0;
  const unsigned long long* p = nullptr;  // pieces of tile t, less its first output index
  int ox = 0, oy = 0;
  for (long long i = c0 + lane; i < c1; i += 32) {
    if (i >= hi) {
      long long lo = t < 0 ? 0 : t, e = nt;  // off[lo] <= i, off[e] > i (or the end)
      if (t >= 0 && t + 1 < nt && (t + 2 >= nt || i < off[t + 2])) lo = t + 1;
      else
        while (e - lo > 1) {
          const long long mid = (lo + e) >> 1;
          if (off[mid] <= i) lo = mid;
          else e = mid;
        }
      t = lo;
      hi = t + 1 < nt ? off[t + 1] : n;
      int k, tx, ty;
      tile_of_index(L, t, k, tx, ty);
      p = L->pcs + L->tstart[t] - off[t];
      ox = tx << g;
      oy = ty << g;
    }
    int a, b, c, d;
    gb_unpack(p[i], a, b, c, d);
    out[i] = make_int4(ox + a, oy + b, ox + c, oy + d);
  }
}

// Per-cell digest of a binned layer: the sum (mod 2^64) of gb_strip_hash over
// its strips in global coordinates.  A sum is independent of the strip order,
// so two layers with the same canonical strips per cell have equal digests
// whatever order their tiles were written in.  One warp per tile.
__global__ void k_cell_digest(const DLayer* L, unsigned long long* out, int stride) {
  const long long nt = L->ntiles;
  const int g = L->g;
  const int wpb = blockDim.x >> 5;
  for (long long t = (long long)blockIdx.x * wpb + gb_warp(); t < nt; t += (long long)gridDim.x * wpb) {
    const int cnt = L->tcount[t];
    if (cnt == 0) continue;
    int k, tx, ty;
    tile_of_index(L, t, k, tx, ty);
    const unsigned long long* p = L->pcs + L->tstart[t];
    const int ox = tx << g, oy = ty << g;
    unsigned long long h = 0;
#pragma unroll 4
    for (int j = gb_lane(); j < cnt; j += 32) {
      int a, b, cc, d;
      gb_unpack(p[j], a, b, cc, d);
      h += gb_strip_hash(ox + a, oy + b, ox + cc, oy + d);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
    if (gb_lane() == 0) atomicAdd(&out[(size_t)k * stride], h);
  }
}

void gb_launch_digest(GbCtx& c, const DLayer* L, unsigned long long* out, int stride) {
  k_cell_digest<<<c.work_blocks, 256, 0, c.stream>>>(L, out, stride);
}

void gb_launch_export(GbCtx& c, const DLayer* L, int4** out_ptr_dev, long long* total_dev) {
  (void)out_ptr_dev;
  (void)total_dev;
  ScanEnd e = {};
  e.hook = SCAN_EXPORT;
  e.src = L;
  e.dscal = c.dscal;
  e.st = c.st;
  launch_scan(c, (int* const*)&L->tcount, (long long* const*)&c.dscal[1], &L->ntiles, e, 0);
  k_export<<<c.work_blocks, 256, 0, c.stream>>>(L, c.dscal, c.st);
}
