// gb_tile.cu -- the scanline Boolean kernel.
//
// Persistent CTAs (three per SM, 8 warps each) pull output tiles from a
// device work counter.
// For a tile it computes the canonical strips of pred(A, B) inside the tile:
// at every x the maximal y-intervals of the region, merged along x while
// unchanged -- the decomposition heal_boxes emits (polygon_fracture.f90:
// 805-1004), here for any Boolean predicate on the two coverages.
//
// Per tile:
//  A. Ranks.  The distinct x and y values of the tile's pieces are marked in
//     two 2^g+1-bit shared-memory bitmaps; prefix popcounts give every value
//     its rank.  x ranks number the x-slabs (elementary columns of the
//     sweep), y ranks the elementary y-intervals.
//  B. Sub-bands.  The x-slabs are grouped 63 at a time; sub-band s owns
//     slabs [63s, 63s+63) as rows 1..63 of a 64-bit word and sees slab 63s-1
//     as row 0.  Every piece is listed in each sub-band its slab range
//     touches (a counting sort in shared memory).
//  C. One warp per sub-band.  The y ranks of the sub-band's members are
//     compressed again (a bitmap over tile y ranks), and each member ORs its
//     row mask into one 64-bit word per local y column (separately for A and
//     B).  R = pred(A, B) word-wise gives the region for 64 slabs at once.
//     With V = R ^ (R << 1) (the rows where a column changes), a run of R
//     over columns [c1, c2] at row r is unchanged from row r-1 iff
//     V[c1-1 .. c2+1] has bit r clear; a segmented OR-scan along the columns
//     (a linear recurrence F_c = a_c | (b_c & F_{c-1}) evaluated with a warp
//     scan) delivers that OR at each run's last column for all 64 rows at
//     once.  A strip piece starts wherever the run changed; it ends at the
//     next change.  Pieces reaching row 63 are "open", pieces starting at
//     row 1 with no change from row 0 are "continuations".  The scan pass
//     leaves each column's local prefix of the recurrence, the count pass
//     each column's piece starts, so the passes after them do not evaluate
//     it again.  The pieces are dealt to the lanes 32 at a time in (column,
//     row) order, so a column with many pieces does not hold up the warp; a
//     piece's 16-byte record goes to the CTA's record region at its index.
//     A sub-band with more columns or y ranks than a warp's buffer holds is
//     wide: the tile's wide ones are swept afterwards, tall ones of few columns
//     by single warps with a layout for more y ranks, the others by teams of
//     warps with larger buffers.
//  D. Stitch.  The records come into shared memory in one bulk copy.  Each
//     continuation is linked to the open piece of the previous sub-band with
//     the same y-interval; every chain head becomes one strip.  The output
//     slots are reserved while the links are made.  Strips are written in
//     (sub-band, column, row) order, so the output of a tile is
//     deterministic.
// Layers of few tiles: one tile per CTA would leave most of the chip idle, so a
// cluster's CTAs then share tiles (k_tile<false, TILE_SPLIT>): each ranks the whole
// tile, takes a contiguous share of the sub-bands through phases B to D, and
// chains that run on into the next CTA's share are followed through a table of
// that CTA's continuations.  These CTAs meet at two hardware cluster barriers.
// Otherwise no CTA ever waits on another CTA.  The only other waits are on the
// CTA's own mbarrier for the bulk copies of phases A and D; each is bounded (a poll
// limit, then GB_ERR_TIMEOUT and the CTA leaves after its copies land).
#include <algorithm>
#include <cstdio>
#include <mutex>

#include "gb_internal.h"
#include "gb_scan.cuh"

#define TK_NW 8
#define TK_NT (TK_NW * 32)
#define TK_WMAX 2052  // words of a bitmap over 0..65536, whole 16-byte groups
#define TK_PMAX 1028
#define TK_XYV (2 * TK_WMAX + 2 * TK_PMAX)
#define TK_NSBMAX 1042
#define TK_SBS 256
#define TK_MDS 128   // sub-bands whose metadata fits in the bitmap region after phase B
#define TK_MD_INTS (TK_MDS * 4 + (TK_MDS + 2) * 2 + TK_MDS * 2 * 2)  // sbinfo, sbh, sbct, sbol, sbrec
// Per-warp sweep buffers of phase C (6 KB a warp): bitmap words over the tile's y ranks, columns.  A sub-band
// that needs more is wide; the wide ones of a tile are swept after the others by teams of 2, 4 or 8 warps with their
// buffers together (levels 1..3), so their words stay in shared memory too.  Standard-cell tiles (2700 boxes of
// each layer) have 160..290 columns in nearly every sub-band: with their words in the global scratch, and a walk
// back over them for every piece, XOR of two 1M-box layers took 2337 us, now 1898 us.
// The wide buffers keep a bitmap's prefix popcounts per 64-bit word and the run starts in the bitmap's place, so they
// hold more y ranks.  A tile whose y ranks are too many for level 0 though its sub-bands have few columns (3000 small
// random boxes and more) has them swept by single warps with such a buffer (level 0 of the wide form): one CTA, XOR of
// 3000 and 3000 boxes of one tile 704 us by teams, now 381; 484 such tiles 1737 and 1047.  In the common form the 64-bit
// ranks cost 3% of an OP1 deck.
#define TK_LBW 188
#define TK_LVN 132
#define TK_LCN 128
#define TK_WLEVELS 3
#define TK_MC 128   // sub-band members kept in the per-warp member cache (8 bytes each)
#define TK_MLD 2    // member records loaded per lane before the first is used (per 1024-cell deck: 4 -> 2
                    // records 30.88 -> 30.59 ms)
#define TK_DU 2     // pieces per thread and step of phase D when the records stay in the scratch
#define TK_LD 2     // independent global loads in flight per thread in the streaming loops
// Columns of a member painted on its own lane; the rest are spread over the warp (device time of a 1024-cell deck
// at 0 / 1 / 2 columns: 30.34 / 30.29 / 30.66 ms; of the wide sub-bands of two 1M-box layers 607 / 592 / 579 us a
// tile).
#define TK_DIRECT (WIDE ? 2 : 1)
#define KID_TILE 20

// A strip piece of one sub-band, 16 bytes, stored downward from the top of
// the CTA scratch.  x: y1 rank | cont << 30 | open << 31; y: y2 rank | low 15
// bits of the head rank << 17; z: first x-slab | high bits of the head rank
// << 17; w: end x-slab.  Ranks and slabs are below 2^17.
struct PieceRec {
  int x, y, z, w;
};
__device__ __forceinline__ int pr_ylo(const PieceRec& p) { return p.x & 0x1ffff; }
__device__ __forceinline__ int pr_yhi(const PieceRec& p) { return p.y & 0x1ffff; }
__device__ __forceinline__ int pr_slo(const PieceRec& p) { return p.z & 0x1ffff; }
__device__ __forceinline__ int pr_shi(const PieceRec& p) { return p.w; }
__device__ __forceinline__ bool pr_cont(const PieceRec& p) { return (p.x >> 30) & 1; }
__device__ __forceinline__ int pr_hrank(const PieceRec& p) {
  return (int)(((unsigned)p.y >> 17) | (((unsigned)p.z >> 17) << 15));
}

// A pointer that is known to lie in shared memory: accesses through one that could lie elsewhere too are slower (a
// tile's pieces and ranks, which large tiles keep in the scratch, and its members' counters: a 1024-cell deck 26.84 ->
// 26.07 ms).
template <typename T>
__device__ __forceinline__ T* in_shared(T* p) {
  __builtin_assume(__isShared(p));
  return p;
}

// A tile to process: its index, cell and the two operands' pieces.
struct TileRef {
  long long tile;
  const unsigned long long* pa;
  const unsigned long long* pb;
  int nA, nB, cell, pad;
};

struct TileSmem {
  union {  // phases A-B: value bitmaps and their prefix popcounts; then what is below
    struct {
      unsigned xb[TK_WMAX], yb[TK_WMAX];
      unsigned xp[TK_PMAX], yp[TK_PMAX];  // prefix popcount per 2 words
    };
    int xyv[TK_XYV];  // sub-band metadata, hand-out order, wide lists, x / y value tables
  };
  int sbc_s[TK_SBS + 2];  // per sub-band member counts / cursors (scratch when more sub-bands)
  union {  // phase C: per-warp sweep buffers; phase D: piece records and chain links
    struct {
      unsigned lb[TK_NW][TK_LBW];
      unsigned lp[TK_NW][TK_LBW];
      int lv[TK_NW][TK_LVN];
      unsigned long long ca[TK_NW][TK_LCN];
      unsigned long long cb[TK_NW][TK_LCN];
      // member cache: first row | end row << 7 | owner << 14 | y1 rank << 15, y2 rank << 32 (rows 0..64,
      // ranks below 2^17)
      unsigned long long mc[TK_NW][TK_MC];
      unsigned srow[TK_NW][64][TK_LCN / 32];  // run starts, row-major (transposed)
    };
    unsigned char dbuf[1];
    int4 dbuf_align;  // the region starts on 16 bytes: bulk copies and int4 records land in it
  };
  int sbnext;                            // next sub-band to hand to a warp
  int nwide[TK_WLEVELS + 2];             // sub-bands that the wide form takes at each level (listed in xyv)
  int narrow;                            // sub-bands swept at level 1 that level 0 could have held
  int hint;                              // the previous tile was mostly wide: start at level 1
  unsigned long long mbar;               // completion of phase D's bulk copies (one phase per tile)
  long long tmp64[40];
  long long tile;
  const unsigned long long* pa;
  const unsigned long long* pb;
  int nA, nB, cell, err;
  int rsplit;  // some sub-band's piece records did not fit the record region (allocated below instead)
  TileRef nx;   // the next tile, reserved and looked up during this tile's phase D
  int have_nx;
  long long nxi;  // a work item reserved but not looked up yet (-1: none)
  long long obase;
  DStatus* st;
  // up: bytes allocated from the lower half of the scratch; down: strip pieces so far, whose records sit at
  // their piece index in the upper half (the record region)
  unsigned long long up, down;
  int t16, t16o;  // the x / y value tables lie in xyv at word t16o, 16 bits a value, t16 x values; t16 0: Xt, Yt
  int* Xt;
  int* Yt;
  int4* rk;
  int4* mem;  // member records: x1-slab | owner<<31, x2-slab, y1 rank, y2 rank
  int4* sbinfo;  // per sub-band: piece base, piece count, open-list byte offset, open count
  int* sbh;      // heads per sub-band, then their exclusive scan
  int* sbct;     // continuation pieces per sub-band
  int* sbc;      // per sub-band member counts / cursors (sbc_s or scratch)
  int** sbol;    // open list (then continuation list) per sub-band
  PieceRec** sbrec;  // strip pieces per sub-band (global piece index = sbinfo.x + local index)
  int* succ;
  int q0, nsbg;  // a shared tile: the CTA's first sub-band, the tile's sub-bands
  unsigned long long area;  // area mode: the CTA's share of the tile
  int2* cont;    // a shared tile: the CTA's continuations from the CTA before it (ordinal, end)
};

// A tile shared by several CTAs: what a CTA tells the others, at the start of its scratch.
struct SplitPub {
  int err;          // 1 until the CTA's strips are known
  int H;            // strips that start in its share
  int nc;           // continuations: (ordinal among the open pieces of the CTA before, end), in order
  int pad;
  int2* cont;       // end >= 0: end slab; else -1 - (ordinal among its own open pieces)
  long long obase;  // first CTA of the tile: the output slots (-1: none)
};
#define TK_PUB_BYTES 64
static_assert(sizeof(SplitPub) <= TK_PUB_BYTES, "published words");
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n barrier.cluster.wait.acquire;" ::: "memory");
}

// Where a chain that is open at the end of CTA `me`'s share ends: open ordinal
// o is looked up among the continuations of the CTAs after it.  pub(j) is CTA
// j's words, ka the tile's CTAs, nsbg its sub-bands.
__device__ __forceinline__ int split_end(const char* pub0, unsigned long long scr, int me, int ka, int nsbg, int o) {
  for (int j = me + 1; j < ka; ++j) {
    const SplitPub* p = reinterpret_cast<const SplitPub*>(pub0 + (size_t)j * scr);
    const int2* c = (const int2*)__ldcg((const unsigned long long*)&p->cont);
    int lo = 0, hi = __ldcg(&p->nc);
    while (lo < hi) {  // first continuation of ordinal >= o
      const int mid = (lo + hi) >> 1;
      if (__ldcg(&c[mid].x) < o) lo = mid + 1;
      else hi = mid;
    }
    const bool found = lo < __ldcg(&p->nc) && __ldcg(&c[lo].x) == o;
    if (!found) return 63 * (int)((long long)nsbg * j / ka);  // it ends where that share starts
    const int e = __ldcg(&c[lo].y);
    if (e >= 0) return e;
    o = -1 - e;
  }
  return 0;  // not reached: the last share has no open pieces
}
// Wide lists of phase C, alternating by level, behind the metadata and the hand-out order in xyv; then the value
// tables, when they fit.
#define TK_WLIST(s, level, nsb) ((s).xyv + TK_MD_INTS + TK_SBS + ((level) & 1) * ((nsb) + 2))
static_assert(TK_MD_INTS + TK_SBS + 2 * (TK_NSBMAX + 2) <= TK_XYV, "wide lists");

// The values of x and y ranks, as the start or the end of an interval.  16 bits hold 0..65536: no interval ends at 0
// (stored for 65536) and none starts at 65536.
struct TileXY {
  const unsigned short *x16, *y16;
  const int *x, *y;
  bool on;
  __device__ __forceinline__ explicit TileXY(const TileSmem& s)
      : x16(reinterpret_cast<const unsigned short*>(s.xyv + s.t16o)), y16(x16 + s.t16), x(s.Xt), y(s.Yt), on(s.t16 != 0) {}
  __device__ __forceinline__ int x0(int r) const { return on ? x16[r] : x[r]; }
  __device__ __forceinline__ int y0(int r) const { return on ? y16[r] : y[r]; }
  __device__ __forceinline__ int x1(int r) const { return on ? ((x16[r] + 0xffff) & 0xffff) + 1 : x[r]; }
  __device__ __forceinline__ int y1(int r) const { return on ? ((y16[r] + 0xffff) & 0xffff) + 1 : y[r]; }
};

// Sweep buffer of the wide form at level 0..3: columns, bitmap words, cached members.
__host__ __device__ constexpr int wide_cols(int level) {
  return level == 0 ? TK_LCN : level == 1 ? 288 : level == 2 ? 640 : 1024;
}
__host__ __device__ constexpr int wide_lbw(int level) { return level == 0 ? 420 : level == 1 ? 844 : level == 2 ? 1724 : 2052; }
__host__ __device__ constexpr int wide_mc(int level) { return level == 0 ? TK_MC : level == 1 ? 176 : level == 2 ? 168 : 488; }
constexpr int wide_bytes(int level) {
  return wide_cols(level) * 16 + wide_mc(level) * 8 + wide_lbw(level) * 6 + (wide_cols(level) + 4) * 4;
}
// The bitmap and its prefixes are dead after the raster: the run starts lie at the end of their place, and the packed
// counts (pf) of up to 512 columns reach from the member cache into its start.
constexpr bool wide_fits(int level) {
  const int cols = wide_cols(level), packed = cols < 512 ? cols : 512;
  return (packed - wide_mc(level)) * 8 + 64 * (cols / 32) * 4 <= wide_lbw(level) * 6;
}
constexpr int TK_WBUF = 6128;  // level 0's bytes per warp; 2, 4 or 8 warps' buffers together at the levels above
static_assert(wide_bytes(0) <= TK_WBUF && wide_bytes(1) <= 2 * TK_WBUF && wide_bytes(2) <= 4 * TK_WBUF &&
                  wide_bytes(3) <= 8 * TK_WBUF && wide_fits(0) && wide_fits(1) && wide_fits(2) && wide_fits(3) &&
                  TK_WBUF % 16 == 0,
              "wide sweep buffers");
static_assert(sizeof(((TileSmem*)0)->lb) + sizeof(((TileSmem*)0)->lp) + sizeof(((TileSmem*)0)->lv) +
                      sizeof(((TileSmem*)0)->ca) + sizeof(((TileSmem*)0)->cb) + sizeof(((TileSmem*)0)->mc) +
                      sizeof(((TileSmem*)0)->srow) ==
                  TK_NW * TK_WBUF,
              "sweep buffers");

#include <cstddef>
// Bulk asynchronous copies need 16-byte aligned shared-memory addresses, and
// the staged ranks, piece records and sub-band metadata are read as int4.
static_assert(offsetof(TileSmem, dbuf) % 16 == 0, "phase C/D region must start on 16 bytes");
static_assert(offsetof(TileSmem, xyv) % 16 == 0, "bitmaps are cleared 16 bytes at a time");
static_assert(offsetof(TileSmem, ca) % 16 == 0 && offsetof(TileSmem, srow) % 16 == 0, "per-warp arrays");


__device__ __forceinline__ unsigned long long gb_pred(int op, unsigned long long a, unsigned long long b) {
  switch (op) {
    case GB_OP_XOR: return a ^ b;
    case GB_OP_AND: return a & b;
    case GB_OP_NOT: return a & ~b;
    case GB_OP_OVERLAP: return b;  // b holds the rows covered a second time
    default: return a | b;  // OR, MERGE (B empty)
  }
}

// Single-layer AND: a row bit painted into a column that already had it is
// recorded in the second word array (atomics make the order of two paints of
// the same cell irrelevant), so b ends as the cells covered at least twice.
__device__ __forceinline__ void paint_twice(unsigned* a, unsigned* b, int c, unsigned mlo, unsigned mhi) {
  if (mlo) {
    const unsigned o = atomicOr(&a[2 * c], mlo) & mlo;
    if (o) atomicOr(&b[2 * c], o);
  }
  if (mhi) {
    const unsigned o = atomicOr(&a[2 * c + 1], mhi) & mhi;
    if (o) atomicOr(&b[2 * c + 1], o);
  }
}

__device__ __forceinline__ int bm_rank(const unsigned* bits, const unsigned* pref, int v) {
  const int w = v >> 5;
  return (int)pref[w] + __popc(bits[w] & ((1u << (v & 31)) - 1u));
}
// rank with a prefix stored once per 2 words
__device__ __forceinline__ int bm_rank2(const unsigned* bits, const unsigned* pref2, int v) {
  const unsigned long long b = reinterpret_cast<const unsigned long long*>(bits)[v >> 6];
  return (int)pref2[v >> 6] + __popcll(b & ((1ull << (v & 63)) - 1ull));
}
// Exclusive scan over the CTA with one barrier (gb_block_excl has four).  slot: TK_NW words that nobody writes
// between this barrier and the next.  With it, the bitmap words of the prefix pass kept in registers (8 a thread) and
// cleared 16 bytes at a time, and a rank from one 64-bit word, a 1024-cell deck takes 29.06 and not 30.28 ms.
template <typename T>
__device__ __forceinline__ T tile_excl(T v, T* slot, T* total) {
  T tot;
  T ex = gb_warp_excl(v, &tot);
  if (gb_lane() == 0) slot[gb_warp()] = tot;
  __syncthreads();
  tot = 0;
#pragma unroll
  for (int i = 0; i < TK_NW; ++i) {
    const T x = slot[i];
    if (i < gb_warp()) ex += x;
    tot += x;
  }
  *total = tot;
  return ex;
}

__device__ __forceinline__ unsigned long long vchg(unsigned long long r) { return (r ^ (r << 1)) & ~1ull; }

// ---- bulk copies of phase D (global scratch -> shared memory, completing on an mbarrier)
#define TK_SPIN_LIMIT (1 << 22)
#define KID_TILE_COPY 22
__device__ __forceinline__ unsigned tk_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tk_bulk(void* dst, const void* src, unsigned bytes, unsigned mbar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   tk_smem(dst)),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}
// bounded wait for the given phase parity; false after `limit` polls
__device__ __forceinline__ bool tk_wait(unsigned mbar, unsigned parity, int limit) {
  for (int i = 0; i < limit; ++i) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Allocation in the lower half of the CTA's scratch (one thread calls it).
// When a dense tile outgrows it, the allocation spills into the work arena
// (released with the operation); only an exhausted arena is an error.
__device__ __forceinline__ void* sc_up(TileSmem& s, char* base, unsigned long long half,
                                       unsigned long long bytes) {
  const unsigned long long off = atomicAdd(&s.up, (bytes + 15ull) & ~15ull);
  if (off + bytes > half) {
    void* p = s.st ? gb_arena_alloc_atomic(s.st, bytes, KID_TILE) : nullptr;
    if (!p) s.err = 1;
    return p;
  }
  return base + off;
}


// Output tile t: its cell, and where A's and B's pieces of that tile start.  A Boolean result carries a
// descriptor per tile (one load); other callers' layers are looked up through the cell windows.
__device__ __forceinline__ void tile_lookup(int op, const DLayer* A, const DLayer* B, const DLayer* O, long long t,
                                            TileRef& r) {
  r.tile = t;
  r.nA = r.nB = 0;
  r.pa = r.pb = nullptr;
  r.cell = 0;
  if (t >= O->ntiles) return;
  if (O->tdesc) {
    const TileDesc d = O->tdesc[t];
    r.cell = d.cell;
    r.nA = d.nA;
    r.nB = d.nB;
    if (d.nA) r.pa = A->pcs + d.offA;
    if (d.nB) r.pb = B->pcs + d.offB;
    return;
  }
  const int k = gb_find_cell(O->tbase, O->ncell, t);
  const int4 w = O->win[k];
  const unsigned li = (unsigned)(t - O->tbase[k]);  // below GB_MAX_TILES_PER_OP
  const int tx = w.x + (int)(li % (unsigned)w.z), ty = w.y + (int)(li / (unsigned)w.z);
  r.cell = k;
  const int4 wa = A->win[k];
  if (tx >= wa.x && ty >= wa.y && tx < wa.x + wa.z && ty < wa.y + wa.w) {
    const long long ta = A->tbase[k] + (long long)(ty - wa.y) * wa.z + (tx - wa.x);
    r.nA = A->tcount[ta];
    r.pa = A->pcs + A->tstart[ta];
  }
  if (B && op != GB_OP_MERGE && op != GB_OP_OVERLAP) {
    const int4 wb = B->win[k];
    if (tx >= wb.x && ty >= wb.y && tx < wb.x + wb.z && ty < wb.y + wb.w) {
      const long long tb = B->tbase[k] + (long long)(ty - wb.y) * wb.z + (tx - wb.x);
      r.nB = B->tcount[tb];
      r.pb = B->pcs + B->tstart[tb];
    }
  }
}

// The 2, 4 or 8 warps of a team of level 1..3 meet (hardware barriers 1..4); at level 0 a team is a warp.
__device__ __forceinline__ void team_sync(int level) {
  __syncwarp();
  if (level == 0) return;
  asm volatile("bar.sync %0, %1;" ::"r"(1 + (gb_warp() >> level)), "r"(32 << level) : "memory");
}

// TIMING: the phase counters of gb_tile_timing are compiled in (tctr non-null
// then); the production instance has none of that code.
// WIDE: the level's larger buffers (level 0..3).  Returns false, with nothing
// done, when the sub-band needs the next level's buffers; at the last level
// columns beyond them spill to the scratch.
// FORM: what the kernel does with a tile (below).
enum TileForm {
  TILE_WHOLE,  // strips, one tile per CTA
  TILE_SPLIT,  // strips, CTAs of a cluster share a tile
  TILE_AREA    // the area alone: no strips, so no chains either, and CTAs share a tile without meeting
};
template <bool TIMING, bool WIDE, int FORM>
__device__ __forceinline__ bool tile_subband(TileSmem& s, int op, int sb, int nsb, int Ny, int nA, char* base,
                             unsigned long long scr, int level, long long* tctr) {
  if (!TIMING) tctr = nullptr;
  // a wide sub-band's warps (1, 2, 4 or 8: a team) share its members and columns
  const int lane = gb_lane(), wid = gb_warp();
  const int T = WIDE ? 32 << level : 32, tl = WIDE ? (int)threadIdx.x & (T - 1) : lane;
  const int wt = WIDE ? tl >> 5 : 0, lead = WIDE ? wid & ~((1 << level) - 1) : 0;
  auto tsync = [&]() {
    if (WIDE) team_sync(level);
    else __syncwarp();
  };
  long long q0 = tctr ? clock64() : 0;
  const long long qstart = q0;
#define TSTEP(k)                                                           \
  if (tctr && tl == 0) {                                                 \
    const long long q1 = clock64();                                        \
    atomicAdd((unsigned long long*)&tctr[k], (unsigned long long)(q1 - q0)); \
    q0 = q1;                                                               \
  }
  const unsigned long long half = scr >> 1;
  const int beg = sb ? s.sbc[sb - 1] : 0, end = s.sbc[sb];
  const int m = end - beg;
  if (m == 0) {
    if (tl == 0) {
      s.sbinfo[sb] = make_int4(0, 0, 0, 0);
      s.sbh[sb] = 0;
      s.sbct[sb] = 0;
      s.sbol[sb] = nullptr;
      s.sbrec[sb] = nullptr;
    }
    return true;
  }
  const int gsb = FORM != TILE_WHOLE ? s.q0 + sb : sb;  // of the tile; sb and nsb count the CTA's share
  const int rowbase = 63 * gsb - 1;
  const int nwy = ((Ny - 1) >> 5) + 1;
  const int lcn = WIDE ? wide_cols(level) : TK_LCN, mcn = WIDE ? wide_mc(level) : TK_MC;
  if (nwy > (WIDE ? wide_lbw(level) : TK_LBW)) return false;  // the last level holds any tile's y ranks
  unsigned long long *ca, *cb, *mc;
  unsigned *lb, *lp, *srow;
  int* lv;
  const int srw = WIDE ? lcn >> 5 : TK_LCN / 32;  // words per row of srow
  if (WIDE) {
    ca = reinterpret_cast<unsigned long long*>(s.dbuf + (size_t)lead * TK_WBUF);
    cb = ca + lcn;
    mc = cb + lcn;
    lb = reinterpret_cast<unsigned*>(mc + mcn);
    lp = lb + wide_lbw(level);
    lv = reinterpret_cast<int*>(lp + wide_lbw(level) / 2);
    srow = reinterpret_cast<unsigned*>(lv) - 64 * srw;
  } else {
    ca = s.ca[wid];
    cb = s.cb[wid];
    mc = s.mc[wid];
    lb = s.lb[wid];
    lp = s.lp[wid];
    lv = s.lv[wid];
    srow = s.srow[wid][0];
  }
  const bool cache = m <= mcn;
  unsigned long long* const lb64 = reinterpret_cast<unsigned long long*>(lb);
  const int nw = WIDE ? (nwy + 1) >> 1 : nwy;  // words with a prefix: of 64 ranks in the wide form, else of 32
  for (int w = tl; w < nw; w += T) {
    if (WIDE) lb64[w] = 0;
    else lb[w] = 0;
  }
  tsync();
  for (int j0 = 0; j0 < m; j0 += T * TK_MLD) {
    int4 rr[TK_MLD];
#pragma unroll
    for (int u = 0; u < TK_MLD; ++u) {
      const int j = j0 + u * T + tl;
      rr[u] = j < m ? s.mem[beg + j] : make_int4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < TK_MLD; ++u) {
      const int j = j0 + u * T + tl;
      if (j < m) {
        const int4 r = rr[u];
        if (cache) {
          const unsigned lo = (unsigned)max((r.x & 0x7fffffff) - rowbase, 0), hi = (unsigned)min(r.y - rowbase, 64);
          mc[j] = (unsigned long long)(lo | (hi << 7) | (((unsigned)r.x >> 31) << 14) | ((unsigned)r.z << 15)) |
                         ((unsigned long long)(unsigned)r.w << 32);
        }
        atomicOr(&lb[r.z >> 5], 1u << (r.z & 31));
        atomicOr(&lb[r.w >> 5], 1u << (r.w & 31));
      }
    }
  }
  tsync();
  int nl;
  {
    const int per = WIDE ? ((nw + T - 1) / T) | 1 : (nw + 31) >> 5, w0 = min(nw, tl * per), w1 = min(nw, w0 + per);
    int cnt = 0;
    for (int w = w0; w < w1; ++w) cnt += WIDE ? __popcll(lb64[w]) : __popc(lb[w]);
    int tot;
    int ex = gb_warp_excl(cnt, &tot);
    if (WIDE) {
      if (lane == 0) s.tmp64[wid] = tot;
      tsync();
      tot = 0;
      for (int i = 0; i < T >> 5; ++i) {
        const int v = (int)s.tmp64[lead + i];
        if (i < wt) ex += v;
        tot += v;
      }
    }
    for (int w = w0; w < w1; ++w) { lp[w] = ex; ex += WIDE ? __popcll(lb64[w]) : __popc(lb[w]); }
    nl = tot;
  }
  const int L = nl - 1;
  TSTEP(0)
  if (tctr && tl == 0) {
    atomicAdd((unsigned long long*)&tctr[6], (unsigned long long)m);
    atomicAdd((unsigned long long*)&tctr[7], (unsigned long long)L);
  }
  if (L > lcn) {
    if (!WIDE || level < TK_WLEVELS) return false;
    if (tl == 0) {
      s.tmp64[8 + lead] = (long long)sc_up(s, base, half, (unsigned long long)nl * 4);
      s.tmp64[9 + lead] = (long long)sc_up(s, base, half, (unsigned long long)L * 16);
    }
    tsync();
    const long long pv = s.tmp64[8 + lead], pc = s.tmp64[9 + lead];
    if (!pv || !pc) return true;  // s.err is set
    lv = (int*)pv;
    ca = (unsigned long long*)pc;
    cb = ca + L;
  }
  if (WIDE && level == 1 && tl == 0 && L <= TK_LCN && nwy <= wide_lbw(0)) atomicAdd(&s.narrow, 1);
  // ---- rasterise: one member per lane; each column word is updated as two
  // 32-bit halves with native shared-memory atomicOr
  // columns per lane; an odd count keeps the lanes' 8-byte words on different banks
  const int per = WIDE ? ((L + T - 1) / T) | 1 : (L + 31) >> 5, c0 = min(L, tl * per), c1e = min(L, c0 + per);
  for (int c = c0; c < c1e; ++c) { ca[c] = 0; cb[c] = 0; }
  tsync();
  // 32 members at a time: the (member, column) pairs of the group are spread
  // evenly over the lanes (a warp scan of the spans; the member of a pair from
  // a warp-wide mask of the members' first pairs), so one long member does not
  // serialise a lane.  A five-step shuffle search in the mask's place: 31.27 ms
  // a 1024-cell deck and not 30.28; in the wide form it is the faster one (592
  // against 798 us a tile, the registers).
  long long qa = tctr ? clock64() : 0, qsetup = 0, qpaint = 0;
  for (int jb = 32 * wt; jb < m; jb += T) {
    const int j = jb + lane;
    int lc1 = 0, span = 0, own = 0;
    unsigned long long mk = 0;
    if (j < m) {
      int lo, hi, yz, yw;
      if (cache) {
        const unsigned long long e = mc[j];
        const unsigned e0 = (unsigned)e;
        lo = (int)(e0 & 127u);
        hi = (int)((e0 >> 7) & 127u);
        own = (int)((e0 >> 14) & 1u);
        yz = (int)(e0 >> 15);
        yw = (int)(e >> 32);
      } else {
        const int4 r = s.mem[beg + j];
        own = (r.x >> 31) & 1;
        lo = max((r.x & 0x7fffffff) - rowbase, 0);
        hi = min(r.y - rowbase, 64);
        yz = r.z;
        yw = r.w;
      }
      mk = (hi >= 64 ? ~0ull : ((1ull << hi) - 1ull)) & (~0ull << lo);
      lc1 = WIDE ? bm_rank2(lb, lp, yz) : bm_rank(lb, lp, yz);
      const int lc2 = WIDE ? bm_rank2(lb, lp, yw) : bm_rank(lb, lp, yw);
      span = lc2 - lc1;
      lv[lc1] = yz;  // a column's bound comes from every member that has it: the same value
      lv[lc2] = yw;
    }
    // direct: the first TK_DIRECT columns of every member on its own lane
    {
      unsigned* col = (unsigned*)(own ? cb : ca);
      const unsigned mlo = (unsigned)mk, mhi = (unsigned)(mk >> 32);
      const int d = min(span, TK_DIRECT);
      if (op == GB_OP_OVERLAP) {
        for (int c = lc1; c < lc1 + d; ++c) paint_twice((unsigned*)ca, (unsigned*)cb, c, mlo, mhi);
      } else {
        for (int c = lc1; c < lc1 + d; ++c) {
          if (mlo) atomicOr(&col[2 * c], mlo);
          if (mhi) atomicOr(&col[2 * c + 1], mhi);
        }
      }
    }
    if (tctr) { const long long qb = clock64(); qsetup += qb - qa; qa = qb; }
    // remainder of long members: (member, column) pairs spread over the lanes
    const int rest = max(span - TK_DIRECT, 0);
    if (__any_sync(0xffffffffu, rest > 0)) {
      const int incl = gb_warp_incl(rest);
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      const int cm = ((lc1 + TK_DIRECT - (incl - rest)) << 1) | own;  // a pair's column less its index; the operand
      // the lanes with pairs, in order: lane i keeps the i-th (the bytes lie in srow, unused until the transposition)
      const unsigned le = 0xffffffffu >> (31 - lane);
      int src = 0, seen = 0;
      if (!WIDE) {
        unsigned char* const order = reinterpret_cast<unsigned char*>(srow);
        const unsigned has = __ballot_sync(0xffffffffu, rest > 0);
        if (rest > 0) order[__popc(has & (le >> 1))] = (unsigned char)lane;
        __syncwarp();
        src = order[lane];
        __syncwarp();
      }
      if (tctr && lane == 0) atomicAdd((unsigned long long*)&tctr[12], (unsigned long long)total);
      for (int k0 = 0; k0 < total; k0 += 32) {  // warp-uniform trip count
        const int k = k0 + lane;
        int o = 0;  // owner lane
        if (WIDE) {  // the first whose inclusive prefix exceeds k
#pragma unroll
          for (int st2 = 16; st2 > 0; st2 >>= 1) {
            const int v = __shfl_sync(0xffffffffu, incl, o + st2 - 1);
            if (v <= k) o += st2;
          }
        } else {  // of the lanes with pairs the last that starts at or before k: a bit for each start in [k0, k0 + 32)
          const unsigned d = (unsigned)(incl - rest - k0);
          const unsigned starts = __reduce_or_sync(0xffffffffu, rest > 0 && d < 32u ? 1u << d : 0u);
          o = __shfl_sync(0xffffffffu, src, seen + __popc(starts & le) - 1);
          seen += __popc(starts);
        }
        const int cm_o = __shfl_sync(0xffffffffu, cm, o);
        const unsigned long long mk_o = __shfl_sync(0xffffffffu, mk, o);
        if (k < total) {
          unsigned* col = (unsigned*)((cm_o & 1) ? cb : ca);
          const int c = (cm_o >> 1) + k;
          if (op == GB_OP_OVERLAP) {
            paint_twice((unsigned*)ca, (unsigned*)cb, c, (unsigned)mk_o, (unsigned)(mk_o >> 32));
          } else {
            if ((unsigned)mk_o) atomicOr(&col[2 * c], (unsigned)mk_o);
            if ((unsigned)(mk_o >> 32)) atomicOr(&col[2 * c + 1], (unsigned)(mk_o >> 32));
          }
        }
      }
    }
    if (tctr) { const long long qb = clock64(); qpaint += qb - qa; qa = qb; }
  }
  tsync();
  if (tctr && tl == 0) {
    atomicAdd((unsigned long long*)&tctr[8], (unsigned long long)qsetup);
    atomicAdd((unsigned long long*)&tctr[9], (unsigned long long)qpaint);
  }
  unsigned long long rany = 0;
  for (int c = c0; c < c1e; ++c) {
    const unsigned long long r = gb_pred(op, ca[c], cb[c]);
    ca[c] = r;
    rany |= r;
  }
  // No region in rows 1..63: the sub-band has no strip pieces (row 0 belongs to
  // the previous sub-band, and its runs matter only to continuations here).
  bool any = __any_sync(0xffffffffu, (rany & ~1ull) != 0ull);
  if (WIDE) {
    if (lane == 0) s.tmp64[8 + wid] = any;
    tsync();
    for (int i = 0; i < T >> 5; ++i) any |= s.tmp64[8 + lead + i] != 0;
  }
  if (!any) {
    TSTEP(1)
    if (tl == 0) {
      s.sbinfo[sb] = make_int4(0, 0, 0, 0);
      s.sbh[sb] = 0;
      s.sbct[sb] = 0;
      s.sbol[sb] = nullptr;
      s.sbrec[sb] = nullptr;
    }
    __syncwarp();
    return true;
  }
  __syncwarp();
  if (FORM == TILE_AREA) {
    // per column its height times the width of its runs of rows 1..63 (row 0 is the sub-band before's)
    const TileXY xy(s);
    long long area = 0;
    for (int c = c0; c < c1e; ++c) {
      unsigned long long rr = ca[c] & ~1ull;
      if (!rr) continue;
      int w = 0;
      while (rr) {
        const int r1 = __ffsll((long long)rr) - 1;
        const int r2 = r1 + __ffsll((long long)~(rr >> r1)) - 1;  // shifted-in zeros (r1 >= 1) end a run at row 63
        w += xy.x1(rowbase + r2) - xy.x0(rowbase + r1);
        rr = r2 >= 64 ? 0ull : rr & (~0ull << r2);
      }
      area += (long long)w * (xy.y1(lv[c + 1]) - xy.y0(lv[c]));
    }
    area = gb_warp_sum(area);
    if (lane == 0) atomicAdd(&s.area, (unsigned long long)area);
    __syncwarp();
    return true;
  }
  TSTEP(1)
  // ---- run starts S_c = R_c & ~R_{c-1}, transposed to one column bitmap per row
  const bool tr = !WIDE || L <= lcn;
  if (tr) {
    const int nb = (L + 31) >> 5;
    for (int b = wt; b < nb; b += T >> 5) {
      const int c = (b << 5) + lane;
      const unsigned long long Rc = c < L ? ca[c] : 0ull;
      const unsigned long long Rm = (c >= 1 && c - 1 < L) ? ca[c - 1] : 0ull;
      const unsigned long long S = Rc & ~Rm;
      unsigned lo = (unsigned)S, hi = (unsigned)(S >> 32);
#pragma unroll
      for (int j = 16; j > 0; j >>= 1) {
        const unsigned m0 = j == 16 ? 0x0000FFFFu : j == 8 ? 0x00FF00FFu : j == 4 ? 0x0F0F0F0Fu
                          : j == 2 ? 0x33333333u : 0x55555555u;
        const unsigned tlo = __shfl_xor_sync(0xffffffffu, lo, j);
        const unsigned thi = __shfl_xor_sync(0xffffffffu, hi, j);
        if (lane & j) {
          lo = ((tlo & ~m0) >> j) | (lo & ~m0);
          hi = ((thi & ~m0) >> j) | (hi & ~m0);
        } else {
          lo = (lo & m0) | ((tlo & m0) << j);
          hi = (hi & m0) | ((thi & m0) << j);
        }
      }
      srow[lane * srw + b] = lo;
      srow[(32 + lane) * srw + b] = hi;
    }
    if (!WIDE) __syncwarp();  // a team's columns meet at the barriers below
  }
  TSTEP(5)

  // ---- forward segmented OR-scan over the columns (bit-parallel over rows)
  auto R = [&](int c) -> unsigned long long { return (c < 0 || c >= L) ? 0ull : ca[c]; };
  unsigned long long FA = 0ull, FB = ~0ull;
  {
    unsigned long long Rm1 = R(c0 - 1);
    for (int c = c0; c < c1e; ++c) {
      const unsigned long long Rc = ca[c];
      const unsigned long long Sc = Rc & ~Rm1;
      const unsigned long long a = Rc & (vchg(Rc) | (Sc & vchg(Rm1)));
      const unsigned long long b = Rc & Rm1;
      FA = a | (b & FA);
      FB = b & FB;
      cb[c] = FA;  // local prefix: F_c = FA_c | (FB_c & carry-in)
      Rm1 = Rc;
    }
  }
  unsigned long long IA = FA, IB = FB;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long pA = __shfl_up_sync(0xffffffffu, IA, o);
    const unsigned long long pB = __shfl_up_sync(0xffffffffu, IB, o);
    if (lane >= o) { IA = IA | (IB & pA); IB = IB & pB; }
  }
  unsigned long long Fin = __shfl_up_sync(0xffffffffu, IA, 1);
  if (lane == 0) Fin = 0ull;
  if (WIDE) {
    if (lane == 31) {
      s.tmp64[wid] = (long long)IA;
      s.tmp64[16 + wid] = (long long)IB;
    }
    tsync();
    unsigned long long Fw = 0ull;  // into the warp's columns
    for (int i = 0; i < wt; ++i) Fw = (unsigned long long)s.tmp64[lead + i] | ((unsigned long long)s.tmp64[16 + lead + i] & Fw);
    unsigned long long Bin = __shfl_up_sync(0xffffffffu, IB, 1);
    if (lane == 0) Bin = ~0ull;
    Fin |= Bin & Fw;
  }
  const bool last_sb = gsb == (FORM != TILE_WHOLE ? s.nsbg : nsb) - 1;
  TSTEP(2)

  // ---- count pieces / opens / heads
  // Packed counts: pieces and heads (at most 64 x 512 each) in 16 bits, opens, continuations and row-0 ends (at
  // most 512 each) in 10 bits.  pf[c] becomes the counts before column c; it lies in the member cache (and the
  // bitmap words behind it in the wide buffers), dead after the raster.
  const bool packed = !WIDE || L <= 512;
  unsigned long long* const pf = mc;
  int* const pos = reinterpret_cast<int*>(mc);
  int np = 0, no = 0, ncn = 0, nz = 0;
  unsigned long long pv = 0;
  {
    unsigned long long Rm1 = R(c0 - 1), fb = ~0ull;
    for (int c = c0; c < c1e; ++c) {
      const unsigned long long Rc = ca[c], Rp1 = R(c + 1);
      const unsigned long long Ec = Rc & ~Rp1;
      fb &= Rc & Rm1;
      const unsigned long long F = cb[c] | (fb & Fin);
      const unsigned long long Chg = (F | vchg(Rp1)) & Ec;
      const unsigned long long Z = (Chg | 2ull) & Ec & ~1ull;
      cb[c] = Z | ((Chg >> 1) & 1ull);  // bit 0 of Z is always clear
      const int pc = __popcll(Z);
      const int open = !last_sb && (Ec >> 63);
      const int cont = (gsb > 0) && ((Z >> 1) & 1ull) && !((Chg >> 1) & 1ull);
      if (packed) {
        pf[c] = pv;
        pv += ((unsigned long long)(unsigned)((int)(Ec & 1ull) << 20 | cont << 10 | open) << 32) |
              (unsigned)(pc | (pc - cont) << 16);
      } else {
        np += pc;
        no += open;
        ncn += cont;
        nz += (int)(Ec & 1ull);
      }
      Rm1 = Rc;
    }
  }
  int totP, totO, totH, totC, totZ;
  // runs at row 0 are the runs at row 63 of the previous sub-band, both in y
  // order: a continuation's ordinal among them indexes that sub-band's open list
  int posZ = 0, posP = 0, posO = 0, posC = 0;
  if (packed) {
    unsigned long long t;
    unsigned long long e = gb_warp_excl(pv, &t);
    if (WIDE) {
      if (lane == 0) s.tmp64[8 + wid] = (long long)t;
      tsync();
      t = 0;
      for (int i = 0; i < T >> 5; ++i) {
        const unsigned long long v = (unsigned long long)s.tmp64[8 + lead + i];
        if (i < wt) e += v;
        t += v;
      }
    }
    for (int c = c0; c < c1e; ++c) pf[c] += e;
    totP = (int)(t & 0xffffu);
    totH = (int)((t >> 16) & 0xffffu);
    totO = (int)((t >> 32) & 0x3ffu);
    totC = (int)((t >> 42) & 0x3ffu);
    if (!WIDE) __syncwarp();
  } else {
    // only in a team: every thread's counts before its columns (pos, in pf's place: the sweeps' words there are
    // dead), behind the other warps' totals
    posZ = gb_warp_excl(nz, &totZ);
    posP = gb_warp_excl(np, &totP);
    posO = gb_warp_excl(no, &totO);
    posC = gb_warp_excl(ncn, &totC);
    if (lane == 0) {
      s.tmp64[8 + wid] = (long long)totP << 32 | totO;
      s.tmp64[24 + wid] = (long long)totC << 32 | totZ;
    }
    tsync();
    totP = totO = totC = 0;
    for (int i = 0; i < T >> 5; ++i) {
      const long long po = s.tmp64[8 + lead + i], cz = s.tmp64[24 + lead + i];
      const int vp = (int)(po >> 32), vo = (int)po, vc = (int)(cz >> 32);
      if (i < wt) { posP += vp; posO += vo; posC += vc; posZ += (int)cz; }
      totP += vp;
      totO += vo;
      totC += vc;
    }
    totH = totP - totC;
    pos[tl] = posP;
    pos[T + tl] = posO;
    pos[2 * T + tl] = posC;
    pos[3 * T + tl] = posZ;
  }
  int pbase = 0;
  unsigned long long obase = 0, rbase = 0;
  if (tl == 0) {
    pbase = (int)atomicAdd(&s.down, (unsigned long long)totP);
    if (totP > 0) {
      // the record region is the upper half of the scratch, indexed by piece
      const unsigned long long rh = half & ~15ull;
      void* p;
      if ((unsigned long long)(pbase + totP) * sizeof(PieceRec) <= scr - rh) {
        p = base + rh + (size_t)pbase * sizeof(PieceRec);
      } else {
        p = sc_up(s, base, half, (unsigned long long)totP * sizeof(PieceRec));
        s.rsplit = 1;
      }
      rbase = (unsigned long long)p;
      if (!p) pbase = -1;
    }
    if (totO + totC > 0 && pbase >= 0) {
      void* p = sc_up(s, base, half, (unsigned long long)(totO + 2 * totC) * 4);
      obase = (unsigned long long)p;
      if (!p) pbase = -1;
    }
  }
  if (WIDE) {
    if (tl == 0) {
      s.tmp64[lead] = pbase;
      s.tmp64[32 + lead] = (long long)obase;
      s.tmp64[16 + lead] = (long long)rbase;
    }
    tsync();
    pbase = (int)s.tmp64[lead];
    obase = (unsigned long long)s.tmp64[32 + lead];
    rbase = (unsigned long long)s.tmp64[16 + lead];
  } else {
    pbase = __shfl_sync(0xffffffffu, pbase, 0);
    obase = __shfl_sync(0xffffffffu, obase, 0);
    rbase = __shfl_sync(0xffffffffu, rbase, 0);
  }
  if (pbase < 0) return true;
  PieceRec* recs = (PieceRec*)rbase;
  int* olist = (int*)obase;  // open pieces, then continuation pieces, each in y order, then the latter's ordinals
  TSTEP(3)

  // ---- write pieces, dealt to the lanes 32 at a time in (column, row) order: piece k's column is found by a
  // binary search over the columns' packed counts (of more than 512 columns: over the threads'
  // counts, and a walk over that thread's columns), its row is its rank among the column's piece starts
  {
    for (int k0 = 0; k0 < totP; k0 += T) {  // uniform trip count
      const int k = k0 + tl;
      int j = 0, o = 0, h = 0, q = 0, z = 0, c = 0;
      if (packed) {
        const unsigned* p32 = reinterpret_cast<const unsigned*>(pf);
#pragma unroll
        for (int st2 = WIDE ? 256 : TK_LCN / 2; st2 > 0; st2 >>= 1)
          if (c + st2 < L && (int)(p32[2 * (c + st2)] & 0xffffu) <= k) c += st2;
        const unsigned long long e = pf[c];
        j = k - (int)(e & 0xffffu);
        h = (int)((e >> 16) & 0xffffu);
        o = (int)((e >> 32) & 0x3ffu);
        q = (int)((e >> 42) & 0x3ffu);
        z = (int)((e >> 52) & 0x3ffu);
      } else {
        int ow = 0;  // owner: the last thread whose columns start at or before piece k
        for (int st2 = T >> 1; st2 > 0; st2 >>= 1)
          if (pos[ow + st2] <= k) ow += st2;
        j = pos[ow];
        o = pos[T + ow];
        q = pos[2 * T + ow];
        z = pos[3 * T + ow];
        h = j - q;
        j = k - j;
        c = min(L, ow * per);
      }
      if (k < totP) {
        unsigned long long zs, Z, Ec;
        int contc;
        for (;;) {  // the owner's columns before the piece's own: their pieces, opens, continuations, row-0 ends
          zs = cb[c];
          Z = zs & ~1ull;
          Ec = ca[c] & ~R(c + 1);
          contc = (gsb > 0) && ((Z >> 1) & 1ull) && !(zs & 1ull);
          if (packed) break;
          const int pc = __popcll(Z);
          if (j < pc) break;
          j -= pc;
          h += pc - contc;
          q += contc;
          o += (!last_sb && (Ec >> 63)) ? 1 : 0;
          z += (int)(Ec & 1ull);
          ++c;
        }
        unsigned long long Zr = Z;
        for (int i = 0; i < j; ++i) Zr &= Zr - 1;
        const int r = __ffsll((long long)Zr) - 1;
        h += j - ((contc && r > 1) ? 1 : 0);  // the column's continuation (row 1) is not a head
        const unsigned long long above = (r >= 63) ? 0ull : ((Z | ~Ec) & (~0ull << (r + 1)));
        const int rend = above ? (__ffsll((long long)above) - 1) : 64;
        int cs = c;
        if (tr) {
          int b = c >> 5;
          unsigned mk = srow[r * srw + b] & (0xFFFFFFFFu >> (31 - (c & 31)));
          while (!mk && b > 0) mk = srow[r * srw + --b];
          cs = (b << 5) + 31 - __clz(mk);
        } else {
          while (cs > 0) {
            const unsigned long long S2 = ca[cs] & ~ca[cs - 1];
            if ((S2 >> r) & 1ull) break;
            --cs;
          }
        }
        const int cont = (r == 1) && contc;
        const int open = (rend == 64) && !last_sb;
        const int p = pbase + k;
        PieceRec pr;
        const unsigned hr = (unsigned)h;
        pr.x = lv[cs] | (cont << 30) | (open << 31);
        pr.y = lv[c + 1] | (int)((hr & 0x7fffu) << 17);
        pr.z = (rowbase + r) | (int)((hr >> 15) << 17);
        pr.w = rowbase + rend;
        recs[k] = pr;
        if (open) olist[o] = p;
        if (cont) {
          olist[totO + q] = p;
          olist[totO + totC + q] = z;
        }
      }
    }
  }
  TSTEP(4)
  if (tctr && tl == 0) {  // wide sub-bands: count and cycles
    const long long q1 = clock64();
    atomicAdd((unsigned long long*)&tctr[28 + (WIDE ? 0 : 2)], 1ull);
    atomicAdd((unsigned long long*)&tctr[29 + (WIDE ? 0 : 2)], (unsigned long long)(q1 - qstart));
  }
  if (tl == 0) {
    s.sbinfo[sb] = make_int4(pbase, totP, totO, 0);
    s.sbol[sb] = (int*)obase;
    s.sbrec[sb] = recs;
    s.sbh[sb] = totH;
    s.sbct[sb] = totC;
  }
  return true;
#undef TSTEP
}

// Phase D's emission for a tile whose piece records stay in the scratch: TK_DU pieces per thread and step, so
// that the loads of one (record, table values) overlap those of the others.  A strip's chain runs through as many
// sub-bands as the strip spans, so its links are what bounds the step: on chip (16 bits, sl16) a hop takes an L1
// latency and not L2's.  Out of line: its registers stay out of the kernel's main path.  Returns the area.
template <bool SPLIT>
__device__ __noinline__ long long tile_emit_scratch(TileSmem& s, const char* recs, int NP, int nsb,
                                                    unsigned long long* outp, bool sl16,
                                                    const char* pub0, unsigned long long scr, int me, int ka) {
  const PieceRec* rg = reinterpret_cast<const PieceRec*>(recs);
  const unsigned short* s16 = reinterpret_cast<const unsigned short*>(s.dbuf);
  const int* s32 = s.succ;
  const TileXY xy(s);
  auto rec = [&](int q) -> PieceRec {
    if (!s.rsplit) return rg[q];
    int sb = 0;  // some records lie elsewhere: the sub-band that holds piece q
    for (; sb < nsb - 1; ++sb) {
      const int4 inf = s.sbinfo[sb];
      if (q >= inf.x && q < inf.x + inf.y) break;
    }
    return s.sbrec[sb][q - s.sbinfo[sb].x];
  };
  auto next = [&](int q) -> int {
    if (!sl16) return s32[q];
    const int v = s16[q];
    return v == 0xffff ? -1 : v;
  };
  long long area = 0;
  for (int p0 = threadIdx.x; p0 < NP; p0 += TK_DU * TK_NT) {
    PieceRec r[TK_DU];
    int nx[TK_DU];
#pragma unroll
    for (int u = 0; u < TK_DU; ++u) {
      const int p = p0 + u * TK_NT;
      r[u].x = 1 << 30;  // past the end: as a continuation, skipped
      nx[u] = -1;
      if (p < NP) {
        r[u] = rec(p);
        nx[u] = next(p);
      }
    }
#pragma unroll
    for (int u = 0; u < TK_DU; ++u) {
      if (pr_cont(r[u])) continue;
      int q = -1, guard = 0;
      while (nx[u] >= 0 && guard++ <= nsb) {
        q = nx[u];
        nx[u] = next(q);
      }
      if (q >= 0) r[u].w = rec(q).w;
      if (SPLIT && nx[u] <= -2) r[u].w = split_end(pub0, scr, me, ka, s.nsbg, -2 - nx[u]);
    }
#pragma unroll
    for (int u = 0; u < TK_DU; ++u) {
      if (pr_cont(r[u])) continue;
      const int slo = pr_slo(r[u]);
      const int xs = xy.x0(slo), xe = xy.x1(pr_shi(r[u])), ylo = xy.y0(pr_ylo(r[u])), yhi = xy.y1(pr_yhi(r[u]));
      if (outp) outp[s.sbh[slo / 63 - (SPLIT ? s.q0 : 0)] + pr_hrank(r[u])] = gb_pack(xs, ylo, xe, yhi);
      area += (long long)(xe - xs) * (long long)(yhi - ylo);
    }
  }
  return area;
}

// Levels first..3 of phase C: the wide sub-bands that were listed for the level, by teams of warps that share a
// buffer.  Called by the whole CTA after level 0.  Out of line: its registers stay out of the kernel's narrow path.
template <bool TIMING, int FORM>
__device__ __noinline__ void tile_wide(TileSmem& s, int op, int first, int nsb, int Ny, int nA, char* base,
                                       unsigned long long scr, long long* tctr) {
  for (int level = first; level <= TK_WLEVELS; ++level) {
    __syncthreads();
    const int todo = s.err ? 0 : s.nwide[level];
    if (todo == 0) break;  // uniform: neither changes before the next barrier
    if (threadIdx.x == 0) s.sbnext = 0;
    __syncthreads();
    const int lead = gb_warp() & ~((1 << level) - 1);
    const bool one = (threadIdx.x & ((32 << level) - 1)) == 0;  // of the team
    for (;;) {
      team_sync(level);  // the sub-band before is done with the team's words
      if (one) {
        const int k = atomicAdd(&s.sbnext, 1), w = *(volatile int*)&s.nwide[level + 1];
        // once three of four were too wide for the level, the rest are listed for the next without a try
        s.tmp64[24 + lead] = k | (w >= TK_NW && w * 4 >= k * 3 ? 1ll << 32 : 0ll);
      }
      team_sync(level);
      const long long e = s.tmp64[24 + lead];
      const int k = (int)e;
      if (k >= todo) break;
      const int sb = TK_WLIST(s, level, nsb)[k];
      if ((e >> 32 || !tile_subband<TIMING, true, FORM>(s, op, sb, nsb, Ny, nA, base, scr, level, tctr)) && one)
        TK_WLIST(s, level + 1, nsb)[atomicAdd(&s.nwide[level + 1], 1)] = sb;
    }
  }
}

// The output pool is sized for the worst case (cap_factor x input pieces) and
// tiles reserve exactly what they emit.  When nothing was allocated in the
// arena after the pool (no overflow, no scratch spill), the unused tail goes
// back to the arena, so a chain of operators keeps only what it produced.  One
// thread of the kernel's last CTA.
__device__ void pool_trim(DLayer* O, DStatus* st) {
  if (*(volatile int*)&st->err || !O->pcs) return;
  const unsigned long long start = (unsigned long long)((char*)O->pcs - st->arena_base);
  const unsigned long long end = start + (((unsigned long long)O->npcs * 8ull + 255ull) & ~255ull);
  const long long nused = (long long)__ldcg((const unsigned long long*)&O->nused);
  if (__ldcg(&st->arena_off) != end || nused > O->npcs) return;
  const long long used = nused > 0 ? nused : 0;
  st->arena_off = start + (((unsigned long long)used * 8ull + 255ull) & ~255ull);
  O->npcs = used;
}

// CTAs per tile for a layer of nt tiles when `ctas` CTAs can share (a multiple
// of 8; 0: never): as many as the chip holds, at least two, else 1.  Sharing
// repeats the ranking (a quarter of a small tile's time), so it pays while it
// fills idle CTAs and not beyond.  XOR of two standard-cell layers, one CTA per
// tile and shared: 9 tiles 1350 -> 541 us, 25 tiles 1400 -> 553 us, 81 tiles
// 1485 -> 776 us; area of 144 tiles (50000 boxes) 198 -> 161 us.
__device__ __forceinline__ int tile_share(long long nt, int ctas) {
  return nt * 8 <= ctas ? (ctas ? 8 : 1) : nt * 4 <= ctas ? 4 : nt * 2 <= ctas ? 2 : 1;
}

// TILE_SPLIT: clusters of 8 CTAs, groups of `share` of them take a tile each;
// every CTA passes two cluster barriers and takes one tile at most.
// TILE_AREA: the work counter hands out (tile, share) pairs.  Klee's measure
// needs the columns' rows and no strips: without the scans, the records and
// the stitch, 12M boxes took 2077 us in all and not 2606 (1648 with the steps
// since).
template <bool TIMING, int FORM>
__global__ void __launch_bounds__(TK_NT, 3)
k_tile(int op, const DLayer* A, const DLayer* B, DLayer* O, int g, char* scratch,
       unsigned long long scr, long long* counter, DStatus* st, int split_ctas) {
  extern __shared__ __align__(16) unsigned char smraw[];
  TileSmem& s = *reinterpret_cast<TileSmem*>(smraw);
  const int tid = threadIdx.x;
  char* base = scratch + (size_t)blockIdx.x * scr;
  const unsigned long long half = scr >> 1;
  const int W = ((1 << g) >> 5) + 1;
  constexpr bool timing = TIMING;
  long long tA = 0, tB = 0, tC = 0, tD = 0, t0 = 0;
  constexpr bool SPLIT = FORM == TILE_SPLIT, AREA = FORM == TILE_AREA;
  const int share = tile_share(O->ntiles, split_ctas);
  if (!AREA && (share > 1) != SPLIT) return;  // the other launch takes the layer (the same on every CTA)
  // a shared tile: the CTA's place among the tile's CTAs, the first one's scratch
  int me = SPLIT ? (int)blockIdx.x % share : 0;
  const char* const pub0 = scratch + (size_t)(blockIdx.x - me) * scr;
  SplitPub* const pub = reinterpret_cast<SplitPub*>(base);
  int ka = 1;  // CTAs that have a part of the tile
  if (SPLIT && tid == 0) {
    pub->err = 1;  // until the CTA has its strips
    __threadfence();
  }
  const unsigned mbar = tk_smem(&s.mbar);
  unsigned mph = 0;  // parity of the mbarrier phase the next bulk copies complete
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s.have_nx = 0;
    s.nxi = -1;
    s.hint = 0;
  }
  for (;;) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // before this tile's bulk copies
    __syncthreads();
    if (tid == 0) {
      s.st = st;
      TileRef r;
      // work item i of the counter: a tile, in area mode a tile and a share of it (their number is 1, 2, 4 or 8)
      auto item = [&](long long i, TileRef& q) {
        tile_lookup(op, A, B, O, AREA ? i >> (__ffs(share) - 1) : i, q);
        if (AREA) q.pad = (int)i & (share - 1);
      };
      const bool reserved = s.have_nx;
      s.have_nx = 0;
      if (reserved) r = s.nx;
      else if (SPLIT) tile_lookup(op, A, B, O, blockIdx.x / share, r);
      else if (st->err) item(1ll << 62, r);
      else {
        // Empty tiles one behind the other are done by this thread alone.  While many are left, the next item is
        // reserved before one is looked up (1000 boxes on 2^24 tiles: 51.6 ms with the block's barriers for every
        // tile); not at the end, where a tile reserved behind another would keep other CTAs idle.
        auto reserve = [&]() { return (long long)atomicAdd((unsigned long long*)counter, 1ull); };
        long long i = s.nxi >= 0 ? s.nxi : reserve(), j = -1;
        for (;;) {
          item(i, r);
          if (r.tile >= O->ntiles || r.nA + r.nB) break;
          if (!AREA) { O->tcount[r.tile] = 0; O->tstart[r.tile] = 0; }
          i = j >= 0 ? j : reserve();
          j = r.tile + 4ll * gridDim.x < O->ntiles ? reserve() : -1;
        }
        s.nxi = j;
      }
      if (st->err && !SPLIT) r.tile = 1ll << 62;  // an error stops the CTA, a reserved tile too
      s.tile = r.tile;
      s.nA = r.nA;
      s.nB = r.nB;
      s.pa = r.pa;
      s.pb = r.pb;
      s.cell = r.cell;
      s.up = SPLIT ? TK_PUB_BYTES : 0;
      s.sbc = s.sbc_s;
      s.down = 0;
      s.err = SPLIT && st->err;
      s.rsplit = 0;
      if (AREA) {
        s.q0 = r.pad;  // the CTA's place, until its sub-bands are known
        s.area = 0;
      }
    }
    __syncthreads();
    if (AREA) me = s.q0;
    const long long t = s.tile;
    if (!SPLIT && t >= O->ntiles) break;
    const int nA = s.nA, nB = s.nB, P = nA + nB;
    if (SPLIT && (t >= O->ntiles || P == 0 || s.err)) {  // the same for the tile's CTAs, but for s.err: published
      if (tid == 0 && me == 0 && t < O->ntiles) { O->tcount[t] = 0; O->tstart[t] = 0; }
      cluster_sync();
      cluster_sync();
      break;
    }
    if (P == 0) {
      if (!AREA && tid == 0) { O->tcount[t] = 0; O->tstart[t] = 0; }
      continue;
    }
    if (timing) t0 = clock64();
    // ---- A: tile ranks
    // Pieces of a tile with at most ~2000 pieces are staged in the (still unused) phase C/D region by
    // bulk copies, their ranks kept next to them; each operand starts at the source's offset modulo 16
    // bytes so both ends of the copy are 16-byte aligned, a leading / trailing odd piece is loaded plainly.
    constexpr int DB = (int)(sizeof(s.lb) + sizeof(s.lp) + sizeof(s.lv) + sizeof(s.ca) + sizeof(s.cb) +
                             sizeof(s.mc) + sizeof(s.srow));
    const unsigned long long* pa = s.pa;
    const unsigned long long* pb = s.pb;
    // A pieces at sp + offA, B pieces at sp + offB: offsets of the parity of the source addresses' 8-byte
    // index, so a piece and its copy agree modulo 16 bytes
    const int offA = nA ? (int)(((uintptr_t)pa >> 3) & 1) : 0;
    const int pbit = nB ? (int)(((uintptr_t)pb >> 3) & 1) : 0;
    const int offB = offA + nA + (((offA + nA) & 1) != pbit ? 1 : 0);
    const int rkoff = ((offB + nB) * 8 + 15) & ~15;  // bytes
    const bool pst = rkoff + P * 16 <= DB;
    unsigned long long* sp = reinterpret_cast<unsigned long long*>(s.dbuf);
    int4* srk = reinterpret_cast<int4*>(s.dbuf + rkoff);
    if (pst) {
      // bulk parts [a0, a1) of A and [b0, b1) of B: even counts of pieces starting on 16-byte addresses
      const int a0 = offA & 1, a1 = nA > a0 ? a0 + ((nA - a0) & ~1) : a0;
      const int b0 = pbit, b1 = nB > b0 ? b0 + ((nB - b0) & ~1) : b0;
      if (tid == 0) {
        const unsigned bytes = (unsigned)(a1 - a0 + b1 - b0) * 8u;
        asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(mbar),
                     "r"(bytes)
                     : "memory");
        if (a1 > a0) tk_bulk(sp + offA + a0, pa + a0, (unsigned)(a1 - a0) * 8u, mbar);
        if (b1 > b0) tk_bulk(sp + offB + b0, pb + b0, (unsigned)(b1 - b0) * 8u, mbar);
      }
      // the first / last piece of an operand when it lies outside the bulk part
      if (tid < 4) {
        const int i = (tid & 1) ? ((tid < 2 ? nA : nB) - 1) : 0;
        if (tid < 2 && nA && (i < a0 || i >= a1)) sp[offA + i] = pa[i];
        if (tid >= 2 && nB && (i < b0 || i >= b1)) sp[offB + i] = pb[i];
      }
    }
    for (int w = tid; w < 2 * TK_WMAX / 4; w += TK_NT) reinterpret_cast<int4*>(s.xb)[w] = make_int4(0, 0, 0, 0);
    for (int i = tid; i < TK_SBS + 2; i += TK_NT) s.sbc_s[i] = 0;
    if (pst) {
      const bool ok = tk_wait(mbar, mph, TK_SPIN_LIMIT);
      mph ^= 1u;
      if (__syncthreads_or(!ok)) {
        if (tid == 0) gb_set_error(st, GB_ERR_TIMEOUT, KID_TILE_COPY, t);
        tk_wait(mbar, mph ^ 1u, TK_SPIN_LIMIT);  // let copies in flight land before the CTA exits
        return;
      }
    } else {
      __syncthreads();
    }
    // piece i of the tile, staged or not
    auto piece_s = [&](int i) { return in_shared(sp)[i + (i < nA ? offA : offB - nA)]; };
    auto piece_g = [&](int i) { return i < nA ? pa[i] : pb[i - nA]; };
    // pieces are read TK_LD at a time per thread, so their loads overlap
    auto mark = [&](auto at) {
      for (int i0 = tid; i0 < P; i0 += TK_LD * TK_NT) {
        unsigned long long pk[TK_LD];
#pragma unroll
        for (int u = 0; u < TK_LD; ++u) {
          const int i = i0 + u * TK_NT;
          pk[u] = i < P ? at(i) : 0ull;
        }
#pragma unroll
        for (int u = 0; u < TK_LD; ++u) {
          if (i0 + u * TK_NT < P) {
            int x1, y1, x2, y2;
            gb_unpack(pk[u], x1, y1, x2, y2);
            atomicOr(&s.xb[x1 >> 5], 1u << (x1 & 31));
            atomicOr(&s.xb[x2 >> 5], 1u << (x2 & 31));
            atomicOr(&s.yb[y1 >> 5], 1u << (y1 & 31));
            atomicOr(&s.yb[y2 >> 5], 1u << (y2 & 31));
          }
        }
      }
    };
    if (pst) mark(piece_s);
    else mark(piece_g);
    __syncthreads();
    int Nx, Ny, t16o;
    // The value tables fit on chip (9232 values less 4 a sub-band): phase B writes them from the pieces' ranks, and
    // they stay there.  Walking the bitmaps' bits into the scratch and copying the tables back for phase D took 4 us
    // of a 1024-cell deck's 58 us a tile (28.10 -> 27.22 ms).
    bool t16;
    {
      // eight words of each bitmap a thread, in registers; the last thread has the word of 65536 too
      const uint4* const x4 = reinterpret_cast<const uint4*>(s.xb) + tid * 2;
      const uint4* const y4 = reinterpret_cast<const uint4*>(s.yb) + tid * 2;
      const uint4 xa = x4[0], xc = x4[1], ya = y4[0], yc = y4[1];
      const int x0 = __popc(xa.x) + __popc(xa.y), x1 = x0 + __popc(xa.z) + __popc(xa.w),
                x2 = x1 + __popc(xc.x) + __popc(xc.y), x3 = x2 + __popc(xc.z) + __popc(xc.w);
      const int y0 = __popc(ya.x) + __popc(ya.y), y1 = y0 + __popc(ya.z) + __popc(ya.w),
                y2 = y1 + __popc(yc.x) + __popc(yc.y), y3 = y2 + __popc(yc.z) + __popc(yc.w);
      int ex = x3, ey = y3;
      if (tid == TK_NT - 1) {
        ex += (int)(s.xb[8 * TK_NT] & 1u);
        ey += (int)(s.yb[8 * TK_NT] & 1u);
      }
      long long tot;
      const long long before = tile_excl((long long)ex | ((long long)ey << 32), s.tmp64, &tot);
      const unsigned ox = (unsigned)before, oy = (unsigned)(before >> 32);
      reinterpret_cast<uint4*>(s.xp)[tid] = make_uint4(ox, ox + x0, ox + x1, ox + x2);
      reinterpret_cast<uint4*>(s.yp)[tid] = make_uint4(oy, oy + y0, oy + y1, oy + y2);
      if (tid == TK_NT - 1) {
        s.xp[4 * TK_NT] = ox + x3;
        s.yp[4 * TK_NT] = oy + y3;
      }
      Nx = (int)(tot & 0xffffffffll);
      Ny = (int)(tot >> 32);
      t16o = TK_MD_INTS + TK_SBS + 2 * ((Nx - 1 + 62) / 63 + 2);
      t16 = Nx + Ny <= 2 * (TK_XYV - t16o);
      if (tid == 0) {
        s.t16 = t16 ? Nx : 0;
        s.t16o = t16o;
        if (!t16) s.Xt = (int*)sc_up(s, base, half, (unsigned long long)Nx * 4);
      }
      if (tid == 32 && !t16) s.Yt = (int*)sc_up(s, base, half, (unsigned long long)Ny * 4);
      if (tid == 64) s.rk = pst ? srk : (int4*)sc_up(s, base, half, (unsigned long long)P * 16);
      __syncthreads();
      if (!t16 && !s.err) {
        // value tables in the scratch, one word per thread in turn (set bits are spread, so
        // the threads stay balanced); the rank of a word's first bit comes
        // from the per-2-word prefix
        int* xt = s.Xt;
        int* yt = s.Yt;
        for (int w = tid; w < W; w += TK_NT) {
          unsigned bx = s.xb[w], by = s.yb[w];
          if (bx) {
            int k = (int)s.xp[w >> 1] + ((w & 1) ? __popc(s.xb[w - 1]) : 0);
            while (bx) { const int b = __ffs(bx) - 1; bx &= bx - 1; xt[k++] = (w << 5) + b; }
          }
          if (by) {
            int k = (int)s.yp[w >> 1] + ((w & 1) ? __popc(s.yb[w - 1]) : 0);
            while (by) { const int b = __ffs(by) - 1; by &= by - 1; yt[k++] = (w << 5) + b; }
          }
        }
      }
    }
    const int nslab = Nx - 1;
    const int nsbg = (nslab + 62) / 63;
    int q0 = 0, q1 = nsbg;  // the CTA's sub-bands
    if (SPLIT || AREA) {
      ka = min(share, nsbg);
      q0 = (int)((long long)nsbg * min(me, ka) / ka);
      q1 = (int)((long long)nsbg * min(me + 1, ka) / ka);
      if (tid == 0) {
        s.q0 = q0;
        s.nsbg = nsbg;
      }
    }
    const int nsb = q1 - q0;
    if (timing) { __syncthreads(); const long long t1 = clock64(); tA += t1 - t0; t0 = t1; }
    // ---- B: sub-band membership (counting sort in shared memory)
    if (nsb > TK_SBS) {  // else the counters were cleared with the bitmaps
      if (tid == 0) {
        int* p = (int*)sc_up(s, base, half, (unsigned long long)(nsb + 2) * 4);
        s.sbc = p ? p : s.sbc_s;  // null only after an error (s.err set); the tile is then abandoned
      }
      __syncthreads();
      for (int i = tid; i <= nsb && s.sbc != s.sbc_s; i += TK_NT) s.sbc[i] = 0;
      __syncthreads();
    }
    auto count = [&](auto at, int4* rk) {
      for (int i0 = tid; i0 < P; i0 += TK_LD * TK_NT) {
        unsigned long long pk[TK_LD];
#pragma unroll
        for (int u = 0; u < TK_LD; ++u) {
          const int i = i0 + u * TK_NT;
          pk[u] = i < P ? at(i) : 0ull;
        }
#pragma unroll
        for (int u = 0; u < TK_LD; ++u) {
          const int i = i0 + u * TK_NT;
          if (i < P) {
            int x1, y1, x2, y2;
            gb_unpack(pk[u], x1, y1, x2, y2);
            const int r1 = bm_rank2(s.xb, s.xp, x1), r2 = bm_rank2(s.xb, s.xp, x2);
            const int lo = max(r1 / 63, q0), hi = min(q1 - 1, r2 / 63);
            int c1 = 0, c2 = 0;
            if (FORM == TILE_WHOLE || lo <= hi) {
              c1 = bm_rank2(s.yb, s.yp, y1);
              c2 = bm_rank2(s.yb, s.yp, y2);
            }
            rk[i] = make_int4(r1, r2, c1, c2);
            if (lo <= hi) {  // the changes of the member count along the sub-bands
              if (nsb <= TK_SBS) {
                atomicAdd(&s.sbc_s[lo - q0], 1);
                atomicSub(&s.sbc_s[hi - q0 + 1], 1);
              } else {
                atomicAdd(&s.sbc[lo - q0], 1);
                atomicSub(&s.sbc[hi - q0 + 1], 1);
              }
            }
          }
        }
      }
    };
    if (!s.err) {
      if (pst) count(piece_s, in_shared(srk));
      else count(piece_g, s.rk);
    }
    __syncthreads();
    int M = 0;
    {
      // sub-band q starts at the sum of the counts before it, which the changes d_j give as the sum of (q - j) d_j:
      // one scan of d_j and j d_j (the sums of j d_j in the upper half, a borrow from it for a negative lower half).
      // Counting every sub-band of a piece: a 1024-cell deck 27.03 ms and not 26.84, phase B of two 1M-box layers 100
      // us a tile and not 87.
      const int nsbv = s.err ? 0 : nsb;  // after an error the counters are not valid
      long long carry = 0;
      for (int b0 = 0; b0 < nsbv; b0 += TK_NT) {
        const int q = b0 + tid;
        const long long d = q < nsbv ? s.sbc[q] : 0;
        long long tot;
        const long long ex = carry + tile_excl((d * q << 32) + d, s.tmp64 + 8, &tot);
        if (q < nsbv) s.sbc[q] = q * (int)ex - (int)((ex - (int)ex) >> 32);
        carry += tot;
        if (nsbv > TK_NT) __syncthreads();
      }
      M = nsbv * (int)carry - (int)((carry - (int)carry) >> 32);
    }
    if (tid == 0) {
      s.mem = (int4*)sc_up(s, base, half, (unsigned long long)M * 16);
      if (nsb <= TK_MDS) {  // the value bitmaps are dead now: keep the metadata on chip
        char* q = reinterpret_cast<char*>(s.xyv);
        s.sbinfo = (int4*)q; q += TK_MDS * 16;
        s.sbol = (int**)q; q += TK_MDS * 8;
        s.sbrec = (PieceRec**)q; q += TK_MDS * 8;
        s.sbh = (int*)q; q += (TK_MDS + 2) * 4;
        s.sbct = (int*)q;
      } else {
        s.sbinfo = (int4*)sc_up(s, base, half, (unsigned long long)nsb * 16);
        s.sbh = (int*)sc_up(s, base, half, (unsigned long long)nsb * 4 + 4);
        s.sbct = (int*)sc_up(s, base, half, (unsigned long long)nsb * 4 + 4);
        s.sbol = (int**)sc_up(s, base, half, (unsigned long long)nsb * 8 + 8);
        s.sbrec = (PieceRec**)sc_up(s, base, half, (unsigned long long)nsb * 8 + 8);
      }
    }
    __syncthreads();
    auto scatter = [&](auto at, const int4* rkp) {
      int4* memp = s.mem;
      unsigned short* const x16 = reinterpret_cast<unsigned short*>(s.xyv + t16o);
      unsigned short* const y16 = x16 + Nx;
      for (int i0 = tid; i0 < P; i0 += TK_LD * TK_NT) {
        int4 rr[TK_LD];
#pragma unroll
        for (int u = 0; u < TK_LD; ++u) {
          const int i = i0 + u * TK_NT;
          rr[u] = i < P ? rkp[i] : make_int4(0, -1, 0, 0);
          if (t16 && i < P) {
            int x1, y1, x2, y2;
            gb_unpack(at(i), x1, y1, x2, y2);
            x16[rr[u].x] = (unsigned short)x1;
            x16[rr[u].y] = (unsigned short)x2;
            if (FORM == TILE_WHOLE || max(rr[u].x / 63, q0) <= min(q1 - 1, rr[u].y / 63)) {
              y16[rr[u].z] = (unsigned short)y1;
              y16[rr[u].w] = (unsigned short)y2;
            }
          }
        }
#pragma unroll
        for (int u = 0; u < TK_LD; ++u) {
          const int i = i0 + u * TK_NT;
          if (i < P) {
            const int4 r = rr[u];
            const int lo = max(r.x / 63, q0), hi = min(q1 - 1, r.y / 63);
            const int4 rec = make_int4(r.x | (i >= nA ? (int)0x80000000 : 0), r.y, r.z, r.w);
            if (nsb <= TK_SBS) {
              for (int q = lo; q <= hi; ++q) memp[atomicAdd(&s.sbc_s[q - q0], 1)] = rec;
            } else {
              for (int q = lo; q <= hi; ++q) memp[atomicAdd(&s.sbc[q - q0], 1)] = rec;
            }
          }
        }
      }
    };
    if (!s.err) {
      if (pst) scatter(piece_s, in_shared(srk));
      else scatter(piece_g, s.rk);
    }
    __syncthreads();
    if (timing) { const long long t1 = clock64(); tB += t1 - t0; t0 = t1; }
    // ---- C: one warp per sub-band, handed out dynamically, the ones with the most members first
    // (longest processing time first: the phase ends with the last sub-band, so the large ones must
    // not come last).  The order lies behind the metadata.
    // Eight lanes rank a sub-band: a 1024-cell deck 27.22 -> 27.00 ms.
    int* const ord = s.xyv + TK_MD_INTS;
    const bool lpt = !s.err && nsb > TK_NW && nsb <= TK_SBS;
    if (lpt) {
      for (int b0 = 0; b0 < nsb; b0 += TK_NT / 8) {  // eight lanes rank a sub-band
        const int q = b0 + (tid >> 3);
        int r = 0;
        if (q < nsb) {
          const int mq = s.sbc[q] - (q ? s.sbc[q - 1] : 0);
          for (int j = tid & 7; j < nsb; j += 8) {
            const int mj = s.sbc[j] - (j ? s.sbc[j - 1] : 0);
            r += mj > mq || (mj == mq && j < q);
          }
        }
        r += __shfl_xor_sync(0xffffffffu, r, 1);
        r += __shfl_xor_sync(0xffffffffu, r, 2);
        r += __shfl_xor_sync(0xffffffffu, r, 4);
        if (q < nsb && (tid & 7) == 0) ord[r] = q;
      }
    }
    if (tid < TK_WLEVELS + 2) s.nwide[tid] = 0;
    if (tid == 0) {
      s.sbnext = 0;
      s.narrow = 0;
    }
    __syncthreads();
    // level 0: every warp with its own buffer.  Wide sub-bands are listed for level 1; once three of four have
    // been wide (or when the previous tile's were), the rest are listed without a try.  Those of a tile with more y
    // ranks than the buffer holds are listed for the wide form's level 0 while its buffer holds them.
    const int nwy = ((Ny - 1) >> 5) + 1;
    const bool mostly = s.hint != 0, tall = nwy > TK_LBW && nwy <= wide_lbw(0);
    const int first = tall && !mostly ? 0 : 1;  // level of the listed ones
    if (!s.err) {
      for (;;) {
        int k = 0;
        bool list = mostly || tall;
        if (gb_lane() == 0) {
          k = atomicAdd(&s.sbnext, 1);
          const int w = *(volatile int*)&s.nwide[1];
          list |= w >= TK_NW && w * 4 >= k * 3;
        }
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= nsb) break;
        const int sb = lpt ? ord[k] : k;
        if (__any_sync(0xffffffffu, list) ||
            !tile_subband<TIMING, false, FORM>(s, op, sb, nsb, Ny, nA, base, scr, 0, timing ? counter + 24 : nullptr)) {
          if (gb_lane() == 0) TK_WLIST(s, first, nsb)[atomicAdd(&s.nwide[first], 1)] = sb;
        }
      }
    }
    __syncthreads();
    if (s.nwide[first]) tile_wide<TIMING, FORM>(s, op, first, nsb, Ny, nA, base, scr, timing ? counter + 24 : nullptr);
    if (tid == 0 && !s.err) s.hint = mostly ? s.narrow * 4 <= nsb : s.nwide[1] * 4 >= nsb * 3;
    if (AREA) {
      __syncthreads();
      if (tid == 0) {
        if (s.err) gb_set_error(st, GB_ERR_CAPACITY, KID_TILE, (long long)scr * 2);
        else atomicAdd((unsigned long long*)&O->cell_area[s.cell], s.area);
        if (me == 0) atomicAdd((unsigned long long*)&counter[8], (unsigned long long)P * 8ull);
      }
      continue;
    }
    // the bulk copies of phase D (async proxy) read the records written above and overwrite shared
    // memory written in phases A-C (generic proxy)
    asm volatile("fence.proxy.async.global;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (timing) {
      const long long t1 = clock64();
      tC += t1 - t0;
      if (tid == 0) {  // phase C per tile, by the tile's sub-band count: 1, 2-3, 4-7, 8-15, 16-31, 32+
        const int bk = nsb <= 1 ? 0 : nsb <= 3 ? 1 : nsb <= 7 ? 2 : nsb <= 15 ? 3 : nsb <= 31 ? 4 : 5;
        atomicAdd((unsigned long long*)&counter[40 + bk], 1ull);
        atomicAdd((unsigned long long*)&counter[46 + bk], (unsigned long long)(t1 - t0));
      }
      t0 = t1;
    }
    // ---- D: stitch and emit.  Piece records and chain links are staged in
    // shared memory that phases A-C no longer use.
    const int NP = (int)s.down;
    constexpr int DBYTES = (int)(sizeof(s.lb) + sizeof(s.lp) + sizeof(s.lv) + sizeof(s.ca) + sizeof(s.cb) +
                                 sizeof(s.mc) + sizeof(s.srow));
    const bool prs = (long long)NP * 20 <= DBYTES;
    // chain links of a tile whose records stay in the scratch: 16 bits each on chip when they fit
    const bool sl16 = !SPLIT && !prs && NP * 2 <= DBYTES;
    if (tid == 0 && !s.err && !prs && !sl16) s.succ = (int*)sc_up(s, base, half, (unsigned long long)NP * 4 + 4);
    const int nc0 = SPLIT && me > 0 && nsb > 0 && !s.err ? s.sbct[0] : 0;  // continuations from the CTA before
    if (SPLIT && tid == 0 && nc0) s.cont = (int2*)sc_up(s, base, half, (unsigned long long)nc0 * 8);
    __syncthreads();
    if (s.err) {
      if (tid == 0) {
        if (me == 0) {
          O->tcount[t] = 0;
          O->tstart[t] = 0;
        }
        gb_set_error(st, GB_ERR_CAPACITY, KID_TILE, (long long)scr * 2);
      }
      if (SPLIT) {
        cluster_sync();
        cluster_sync();
        break;
      }
      continue;
    }
    // the next tile's reservation (the work counter) and its descriptor load run on the last thread while
    // the bulk copies below land
    if (!SPLIT && tid == TK_NT - 1 && !st->err) {
      tile_lookup(op, A, B, O, s.nxi >= 0 ? s.nxi : (long long)atomicAdd((unsigned long long*)counter, 1ull), s.nx);
      s.nxi = -1;
      s.have_nx = 1;
    }
    PieceRec* PR = prs ? reinterpret_cast<PieceRec*>(s.dbuf) : nullptr;
    int* succ = prs ? reinterpret_cast<int*>(s.dbuf + (size_t)NP * 16) : s.succ;
    const int wid = gb_warp(), lane = gb_lane();
    // piece records of every sub-band into shared memory by bulk copies
    // (all 16-byte aligned: records are 16 bytes, scratch allocations are rounded to 16 bytes)
    if (prs && NP > 0) {
      if (tid == 0) {
        const unsigned bytes = (unsigned)NP * 16u;
        asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(mbar),
                     "r"(bytes)
                     : "memory");
      }
      if (!s.rsplit) {
        if (tid == 0) tk_bulk(PR, base + (half & ~15ull), (unsigned)NP * 16u, mbar);
      } else if (wid == 0) {
        for (int sb = lane; sb < nsb; sb += 32) {
          const int4 inf = s.sbinfo[sb];
          if (inf.y > 0) tk_bulk(PR + inf.x, s.sbrec[sb], (unsigned)inf.y * 16u, mbar);
        }
      }
      const bool ok = tk_wait(mbar, mph, TK_SPIN_LIMIT);
      mph ^= 1u;
      if (__syncthreads_or(!ok)) {
        if (tid == 0) gb_set_error(st, GB_ERR_TIMEOUT, KID_TILE_COPY, t);
        tk_wait(mbar, mph ^ 1u, TK_SPIN_LIMIT);  // let copies in flight land before the CTA exits
        return;
      }
    }
    unsigned short* const succ16 = reinterpret_cast<unsigned short*>(s.dbuf);
    if (sl16)
      for (int p = tid; p < NP; p += TK_NT) succ16[p] = 0xffffu;
    else
      for (int p = tid; p < NP; p += TK_NT) succ[p] = -1;
    int H = 0;
    {
      for (int b0 = 0; b0 < nsb; b0 += TK_NT) {
        const int q = b0 + tid;
        int tot;
        const int ex = tile_excl(q < nsb ? s.sbh[q] : 0, reinterpret_cast<int*>(s.tmp64 + 16), &tot);
        if (q < nsb) s.sbh[q] = H + ex;
        H += tot;
        if (nsb > TK_NT) __syncthreads();
      }
    }
    if (nsb <= 0) __syncthreads();  // else the scan's barrier: the links are cleared
    if (!SPLIT && tid == TK_NT - 32) {  // read after the links' barrier
      s.obase = -1;
      if (H > 0) {
        atomicAdd((unsigned long long*)&O->ntot, (unsigned long long)H);
        const long long o = (long long)atomicAdd((unsigned long long*)&O->nused, (unsigned long long)H);
        if (o + H <= O->npcs) {
          s.obase = o;
        } else {
          unsigned long long* p =
              (unsigned long long*)gb_arena_alloc_atomic(st, (unsigned long long)H * 8ull, KID_TILE + 1);
          if (p) s.obase = (long long)(p - O->pcs);
        }
      }
    }
    // link every continuation piece to the open piece of the previous
    // sub-band: its row-0 ordinal indexes that sub-band's open list directly
    for (int sb = 1 + wid; sb < nsb; sb += TK_NW) {
      const int nc = s.sbct[sb];
      if (!nc) continue;
      const int* cl = s.sbol[sb] + s.sbinfo[sb].z;
      const int4 pinf = s.sbinfo[sb - 1];
      const int* ol = s.sbol[sb - 1];
      for (int k = lane; k < nc; k += 32) {
        const int p = cl[k], ord = cl[nc + k];
        if (ord < pinf.z) {
          if (sl16) succ16[ol[ord]] = (unsigned short)p;
          else succ[ol[ord]] = p;
        } else gb_set_error(st, GB_ERR_INTERNAL, KID_TILE, t);
      }
    }
    if (SPLIT && me < ka - 1 && nsb > 0) {  // open at the end of the share: -2 - ordinal
      const int no = s.sbinfo[nsb - 1].z;
      const int* ol = s.sbol[nsb - 1];
      for (int k = tid; k < no; k += TK_NT) succ[ol[k]] = -2 - k;
    }
    __syncthreads();
    if (SPLIT) {
      if (nc0) {  // where the chains that come in end
        const int* cl = s.sbol[0] + s.sbinfo[0].z;
        const PieceRec* rg = reinterpret_cast<const PieceRec*>(base + (half & ~15ull));
        for (int k = tid; k < nc0; k += TK_NT) {
          int q = cl[k], e, guard = 0;
          while ((e = succ[q]) >= 0 && guard++ <= nsb) q = e;
          if (e > -2) {
            if (prs) e = pr_shi(PR[q]);
            else if (!s.rsplit) e = pr_shi(rg[q]);
            else {
              int sb = 0;
              for (; sb < nsb - 1; ++sb)
                if (q >= s.sbinfo[sb].x && q < s.sbinfo[sb].x + s.sbinfo[sb].y) break;
              e = pr_shi(s.sbrec[sb][q - s.sbinfo[sb].x]);
            }
          } else {
            e += 1;  // -1 - ordinal
          }
          s.cont[k] = make_int2(cl[nc0 + k], e);
        }
      }
      if (tid == 0) {
        pub->H = H;
        pub->nc = nc0;
        pub->cont = s.cont;
        pub->err = 0;
      }
      cluster_sync();
      int before = 0, total = 0, bad = 0;
      for (int j = 0; j < ka; ++j) {
        const SplitPub* pj = reinterpret_cast<const SplitPub*>(pub0 + (size_t)j * scr);
        const int h = __ldcg(&pj->H);
        bad |= __ldcg(&pj->err);
        if (j < me) before += h;
        total += h;
      }
      if (me == 0 && tid == 0) {
        long long o = -1;
        if (total > 0 && !bad) {
          atomicAdd((unsigned long long*)&O->ntot, (unsigned long long)total);
          o = (long long)atomicAdd((unsigned long long*)&O->nused, (unsigned long long)total);
          if (o + total > O->npcs) {
            unsigned long long* p =
                (unsigned long long*)gb_arena_alloc_atomic(st, (unsigned long long)total * 8ull, KID_TILE + 1);
            o = p ? (long long)(p - O->pcs) : -1;
          }
        }
        pub->obase = o;
      }
      cluster_sync();
      if (bad) {  // a CTA of the tile failed and said so
        if (tid == 0 && me == 0) {
          O->tcount[t] = 0;
          O->tstart[t] = 0;
        }
        break;
      }
      H = total;
      if (tid == 0) s.obase = __ldcg(&reinterpret_cast<const SplitPub*>(pub0)->obase);
      for (int q = tid; q < nsb; q += TK_NT) s.sbh[q] += before;
      __syncthreads();
    }
    const long long obase = s.obase;
    const TileXY xy(s);
    unsigned long long* outp = obase >= 0 ? O->pcs + obase : nullptr;
    long long area = 0;
    if (prs) {
      // records on chip: every thread takes pieces in turn; a piece's sub-band is its first slab / 63
      // (its first row is 1..63 of that sub-band)
      for (int p = tid; p < NP; p += TK_NT) {
        const PieceRec pr = PR[p];
        if (pr_cont(pr)) continue;
        int q = p, guard = 0;
        while (succ[q] >= 0 && guard++ <= nsb) q = succ[q];
        int shi = q == p ? pr_shi(pr) : pr_shi(PR[q]);
        if (SPLIT && succ[q] <= -2) shi = split_end(pub0, scr, me, ka, nsbg, -2 - succ[q]);
        const int slo = pr_slo(pr);
        const int xs = xy.x0(slo), xe = xy.x1(shi), ylo = xy.y0(pr_ylo(pr)), yhi = xy.y1(pr_yhi(pr));
        const int pos = s.sbh[slo / 63 - q0] + pr_hrank(pr);
        if (outp) outp[pos] = gb_pack(xs, ylo, xe, yhi);
        area += (long long)(xe - xs) * (long long)(yhi - ylo);
      }
    } else {
      area = tile_emit_scratch<SPLIT>(s, base + (half & ~15ull), NP, nsb, outp, sl16, pub0, scr, me, ka);
    }
    {
      long long tot;
      tile_excl(area, s.tmp64 + 24, &tot);
      area = tot;
    }
    if (SPLIT && tid == 0 && me > 0) atomicAdd((unsigned long long*)&O->cell_area[s.cell], (unsigned long long)area);
    if (tid == 0 && me == 0) {
      O->tcount[t] = obase >= 0 ? H : 0;
      O->tstart[t] = obase >= 0 ? obase : 0;
      atomicAdd((unsigned long long*)&O->cell_area[s.cell], (unsigned long long)area);
      atomicAdd((unsigned long long*)&O->cell_count[s.cell], (unsigned long long)H);
      if (timing) {
        const long long t1 = clock64();
        tD += t1 - t0;
        atomicAdd((unsigned long long*)&counter[20], 1ull);
        atomicAdd((unsigned long long*)&counter[21], (unsigned long long)P);
        atomicAdd((unsigned long long*)&counter[22], (unsigned long long)nsb);
        atomicAdd((unsigned long long*)&counter[23], (unsigned long long)NP);
      }
      atomicAdd((unsigned long long*)&counter[8], (unsigned long long)P * 8ull);
      atomicAdd((unsigned long long*)&counter[9], (unsigned long long)H * 8ull);
    }
    if (SPLIT) break;
  }
  if (!AREA && tid == 0) {  // the last CTA to finish gives the pool's tail back
    __threadfence();
    if (atomicAdd((unsigned long long*)&counter[2], 1ull) == gridDim.x - 1) {
      __threadfence();
      pool_trim(O, st);
    }
  }
  if (timing && threadIdx.x == 0) {
    atomicAdd((unsigned long long*)&counter[16], (unsigned long long)tA);
    atomicAdd((unsigned long long*)&counter[17], (unsigned long long)tB);
    atomicAdd((unsigned long long*)&counter[18], (unsigned long long)tC);
    atomicAdd((unsigned long long*)&counter[19], (unsigned long long)tD);
  }
}

static cudaLaunchConfig_t split_config(GbCtx& c, cudaLaunchAttribute* at, int ctas) {
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = 8;
  at->val.clusterDim.y = at->val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3(TK_NT);
  cfg.dynamicSmemBytes = c.tile_smem;
  cfg.stream = c.stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

void gb_tile_setup(GbCtx& c) {
  c.tile_smem = sizeof(TileSmem);
  cudaFuncSetAttribute(k_tile<false, TILE_WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.tile_smem);
  cudaFuncSetAttribute(k_tile<true, TILE_WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.tile_smem);
  cudaFuncSetAttribute(k_tile<false, TILE_SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.tile_smem);
  cudaFuncSetAttribute(k_tile<false, TILE_AREA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.tile_smem);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tile<false, TILE_WHOLE>, TK_NT, c.tile_smem);
  c.tile_blocks = c.nsm * (per_sm > 0 ? per_sm : 1);
  // clusters of 8 CTAs that the chip holds at once
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = split_config(c, &at, c.tile_blocks / 8 * 8);
  int ncl = 0;
  if (cudaOccupancyMaxActiveClusters(&ncl, k_tile<false, TILE_SPLIT>, &cfg) != cudaSuccess) {
    cudaGetLastError();
    ncl = 0;
  }
  c.split_ctas = std::min(ncl, c.tile_blocks / 8) * 8;
}

void gb_launch_tile_bool(GbCtx& c, int op, const DLayer* A, const DLayer* B, DLayer* O, int g, bool area) {
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (c.prof) {
    if (c.prof_used + 2 > c.prof_ev.size()) {
      for (int i = 0; i < 64; ++i) {
        cudaEvent_t e;
        cudaEventCreate(&e);
        c.prof_ev.push_back(e);
      }
    }
    e0 = c.prof_ev[c.prof_used++];
    e1 = c.prof_ev[c.prof_used++];
    // inside a stream capture only an external record becomes a real event node
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(c.stream, &cs);
    c.prof_flags = cs == cudaStreamCaptureStatusActive ? cudaEventRecordExternal : 0;
    cudaEventRecordWithFlags(e0, c.stream, c.prof_flags);
  }
  // which of the two launches takes the layer depends on its tiles, which the device knows
  if (area) {
    k_tile<false, TILE_AREA><<<c.tile_blocks, TK_NT, c.tile_smem, c.stream>>>(
        op, A, B, O, g, c.tile_scratch, c.tile_scr_bytes, c.tile_counter, c.st, c.tile_blocks);
  } else if (c.timing) {
    k_tile<true, TILE_WHOLE><<<c.tile_blocks, TK_NT, c.tile_smem, c.stream>>>(
        op, A, B, O, g, c.tile_scratch, c.tile_scr_bytes, c.tile_counter, c.st, 0);
  } else {
    if (c.split_ctas) {
      cudaLaunchAttribute at;
      const cudaLaunchConfig_t cfg = split_config(c, &at, c.split_ctas);
      cudaLaunchKernelEx(&cfg, k_tile<false, TILE_SPLIT>, op, A, B, O, g, c.tile_scratch,
                         (unsigned long long)c.tile_scr_bytes, c.tile_counter, c.st, c.split_ctas);
      ++c.launches;
    }
    k_tile<false, TILE_WHOLE><<<c.tile_blocks, TK_NT, c.tile_smem, c.stream>>>(
        op, A, B, O, g, c.tile_scratch, c.tile_scr_bytes, c.tile_counter, c.st, c.split_ctas);
  }
  if (c.prof) cudaEventRecordWithFlags(e1, c.stream, c.prof_flags);
  ++c.launches;
}

// ===================================================================== no-allocation entry point
// gb_bool_tile_noalloc: the scanline Boolean for callers that cannot allocate
// device memory -- code running where cudaMalloc is not permitted on the
// request path (a serving loop that has reserved its whole device budget up
// front, a host that must not take the allocator's implicit device-wide
// synchronisation, or a Fortran/C caller that only owns the buffers it
// passes).  It computes the canonical strips of pred(A, B) for boxes that all
// lie inside one 65536-dbu tile, entirely in memory reserved statically in
// this library: every GPU that loads libgbool.so holds this storage until the
// process exits.
//
// Limits: nA + nB <= GB_NA_MAX_IN boxes (nA alone for MERGE, which ignores
// B), at most GB_NA_MAX_OUT result strips, and the CTA scratch of
// GB_NA_SCRATCH bytes.  Beyond any of them the call returns GB_ERR_CAPACITY;
// a result with more strips than the caller's out_cap does too.  On every
// status other than GB_OK, *d_count (and *d_area when given) is -1.
//
// All calls share the static storage (each call re-initialises what must
// start at zero and keeps the last call's contents otherwise), so calls whose
// work overlaps on the GPU -- on different streams, or from different host
// threads -- race and must be serialised by the caller.  Every call waits for
// its stream to finish before it returns.
//
// Set-up: the first call on a device resolves the device addresses of the
// static storage with cudaGetSymbolAddress (with that device current) and
// sets the kernel's shared-memory attribute; later calls on that device reuse
// them.
#define GB_NA_MAX_IN 16384
#define GB_NA_MAX_OUT 65536
#define GB_NA_SCRATCH (8u << 20)
#define GB_NA_MAX_DEV 64

// What the host reads back after a call, in one copy: the status and the
// result's strip count (also when it exceeds the caller's buffer).
struct NoAllocResult {
  DStatus st;       // status; its arena is empty (no spill space)
  long long nout;   // strips of the result
};

struct NoAllocState {
  NoAllocResult res;
  DLayer L[3];                              // A, B, result
  long long ctr[64];                        // work counters of the tile kernel
  int4 win[3];
  long long tbase[3][2];
  long long tstart[3][2];
  int tcount[3][2];
  long long cell_count[3];
  long long cell_area[3];
  int4 cbox[3];
  unsigned long long pcs_in[GB_NA_MAX_IN];  // packed pieces of A then B
  unsigned long long pcs_out[GB_NA_MAX_OUT];
};

static __device__ __align__(256) NoAllocState g_na_state;
static __device__ __align__(256) char g_na_scratch[GB_NA_SCRATCH];

static NoAllocState* g_na_state_ptr[GB_NA_MAX_DEV];
static char* g_na_scratch_ptr[GB_NA_MAX_DEV];
static std::mutex g_na_mu;

// Re-initialise the shared state and pack the inputs (one block).  Every box
// must lie inside the tile of the first box; otherwise the status says so.
// MERGE reads A only.
__global__ void k_na_prep(NoAllocState* S, int op, const int4* A, int nA, const int4* B, int nB, int g) {
  __shared__ int bad;
  __shared__ int tx0, ty0;
  if (op == GB_OP_MERGE) nB = 0;
  if (threadIdx.x == 0) {
    bad = 0;
    const int4 f = nA ? A[0] : (nB ? B[0] : make_int4(0, 0, 1, 1));
    tx0 = gb_floor_shift(f.x, g);
    ty0 = gb_floor_shift(f.y, g);
    memset(&S->res, 0, sizeof(S->res));  // empty arena: spills report GB_ERR_CAPACITY
    for (int i = 0; i < 64; ++i) S->ctr[i] = 0;
  }
  __syncthreads();
  const int n = nA + nB;
  const int ox = tx0 << g, oy = ty0 << g;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int4 b = i < nA ? A[i] : B[i - nA];
    const bool ok = b.x < b.z && b.y < b.w && gb_floor_shift(b.x, g) == tx0 &&
                    gb_floor_shift(b.z - 1, g) == tx0 && gb_floor_shift(b.y, g) == ty0 &&
                    gb_floor_shift(b.w - 1, g) == ty0;
    if (!ok) { atomicOr(&bad, 1); continue; }
    S->pcs_in[i] = gb_pack(b.x - ox, b.y - oy, b.z - ox, b.w - oy);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (bad) gb_set_error(&S->res.st, GB_ERR_INVALID_BOX, 60, 0);
    for (int l = 0; l < 3; ++l) {
      DLayer& d = S->L[l];
      memset(&d, 0, sizeof(d));
      d.ncell = 1;
      d.g = g;
      d.binned = 1;
      S->win[l] = make_int4(tx0, ty0, 1, 1);
      S->tbase[l][0] = 0;
      S->tbase[l][1] = 1;
      S->cell_count[l] = 0;
      S->cell_area[l] = 0;
      S->cbox[l] = make_int4(ox, oy, ox + (1 << g), oy + (1 << g));
      d.win = &S->win[l];
      d.tbase = S->tbase[l];
      d.tstart = S->tstart[l];
      d.tcount = S->tcount[l];
      d.cell_count = &S->cell_count[l];
      d.cell_area = &S->cell_area[l];
      d.cbox = &S->cbox[l];
      d.ntiles = 1;
    }
    S->L[0].pcs = S->pcs_in;
    S->tstart[0][0] = 0;
    S->tcount[0][0] = nA;
    S->L[0].npcs = S->L[0].nused = S->L[0].ntot = nA;
    S->L[1].pcs = S->pcs_in;
    S->tstart[1][0] = nA;
    S->tcount[1][0] = nB;
    S->L[1].npcs = S->L[1].nused = S->L[1].ntot = nB;
    S->L[2].pcs = S->pcs_out;
    S->L[2].npcs = GB_NA_MAX_OUT;
    S->tstart[2][0] = 0;
    S->tcount[2][0] = 0;
    if (bad) S->L[2].ntiles = 0;  // nothing runs on invalid input
  }
}

// Unpack the result into the caller's buffer; *count = strips, or -1 when the
// call failed or the buffer is too small.  The strip count also goes to the
// state, for the host.
__global__ void k_na_export(NoAllocState* S, int4* out, long long cap, long long* count, long long* area) {
  const DLayer& O = S->L[2];
  const long long n = O.ntiles ? O.tcount[0] : 0;
  const bool ok = S->res.st.err == 0 && n <= cap;
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    *count = ok ? n : -1;
    if (area) *area = ok ? S->cell_area[2] : -1;
  }
  if (!ok) {
    if (threadIdx.x == 0 && blockIdx.x == 0) S->res.nout = n;
    return;
  }
  const int4 w = S->win[2];
  const int ox = w.x << O.g, oy = w.y << O.g;
  const unsigned long long* p = O.pcs + O.tstart[0];
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    int a, b, c, d;
    gb_unpack(p[i], a, b, c, d);
    out[i] = make_int4(ox + a, oy + b, ox + c, oy + d);
  }
  if (threadIdx.x == 0 && blockIdx.x == 0) S->res.nout = n;
}

// *d_count = -1 (and *d_area) for a call refused before its kernels run.
static int na_refuse(int code, long long* d_count, long long* d_area, cudaStream_t s) {
  if (d_count) cudaMemsetAsync(d_count, 0xff, sizeof(long long), s);
  if (d_area) cudaMemsetAsync(d_area, 0xff, sizeof(long long), s);
  if (d_count || d_area) cudaStreamSynchronize(s);
  return code;
}

extern "C" int gb_bool_tile_noalloc(int op, const int4* d_A, int nA, const int4* d_B, int nB, int4* d_out,
                                    long long out_cap, long long* d_count, long long* d_area, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  if (op == GB_OP_MERGE) nB = nB < 0 ? nB : 0;
  if (op < GB_OP_XOR || op > GB_OP_MERGE || nA < 0 || nB < 0 || out_cap < 0 || !d_out || !d_count ||
      (nA && !d_A) || (nB && !d_B))
    return na_refuse(GB_ERR_ARG, d_count, d_area, s);
  if ((long long)nA + nB > GB_NA_MAX_IN) {
    fprintf(stderr, "gb_bool_tile_noalloc: %lld input boxes exceed the static limit of %d\n",
            (long long)nA + nB, GB_NA_MAX_IN);
    return na_refuse(GB_ERR_CAPACITY, d_count, d_area, s);
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= GB_NA_MAX_DEV)
    return na_refuse(GB_ERR_CUDA, d_count, d_area, s);
  NoAllocState* S;
  char* scr;
  {
    std::lock_guard<std::mutex> lk(g_na_mu);
    if (!g_na_state_ptr[dev]) {
      void* a = nullptr;
      void* b = nullptr;
      if (cudaGetSymbolAddress(&a, g_na_state) != cudaSuccess ||
          cudaGetSymbolAddress(&b, g_na_scratch) != cudaSuccess) {
        fprintf(stderr, "gb_bool_tile_noalloc: cudaGetSymbolAddress failed on device %d\n", dev);
        return na_refuse(GB_ERR_CUDA, d_count, d_area, s);
      }
      if (cudaFuncSetAttribute(k_tile<false, TILE_WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem)) !=
          cudaSuccess)
        return na_refuse(GB_ERR_CUDA, d_count, d_area, s);
      g_na_state_ptr[dev] = (NoAllocState*)a;
      g_na_scratch_ptr[dev] = (char*)b;
    }
    S = g_na_state_ptr[dev];
    scr = g_na_scratch_ptr[dev];
  }
  // each launch reports its own error (no reliance on the thread's last-error state)
  const int g = 16;
  {
    void* args[] = {&S, &op, &d_A, &nA, &d_B, &nB, (void*)&g};
    if (cudaLaunchKernel((const void*)k_na_prep, dim3(1), dim3(256), args, 0, s) != cudaSuccess)
      return na_refuse(GB_ERR_CUDA, d_count, d_area, s);
  }
  {
    DLayer* la = &S->L[0];
    DLayer* lb = &S->L[1];
    DLayer* lo = &S->L[2];
    int gg = g;
    unsigned long long scr_bytes = GB_NA_SCRATCH;
    long long* ctr = S->ctr;
    DStatus* st = &S->res.st;
    int split = 0;
    void* args[] = {&op, &la, &lb, &lo, &gg, &scr, &scr_bytes, &ctr, &st, &split};
    if (cudaLaunchKernel((const void*)k_tile<false, TILE_WHOLE>, dim3(1), dim3(TK_NT), args, sizeof(TileSmem), s) != cudaSuccess)
      return na_refuse(GB_ERR_CUDA, d_count, d_area, s);
  }
  {
    void* args[] = {&S, &d_out, &out_cap, &d_count, &d_area};
    if (cudaLaunchKernel((const void*)k_na_export, dim3(8), dim3(256), args, 0, s) != cudaSuccess)
      return na_refuse(GB_ERR_CUDA, d_count, d_area, s);
  }
  NoAllocResult hr;
  if (cudaMemcpyAsync(&hr, &S->res, sizeof(hr), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
      cudaStreamSynchronize(s) != cudaSuccess)
    return GB_ERR_CUDA;
  if (hr.st.err == GB_ERR_CAPACITY)
    fprintf(stderr, "gb_bool_tile_noalloc: result exceeds the static limits (%d strips, %u scratch bytes)\n",
            GB_NA_MAX_OUT, GB_NA_SCRATCH);
  if (hr.st.err) return hr.st.err;
  if (hr.nout > out_cap) {
    fprintf(stderr, "gb_bool_tile_noalloc: %lld result strips exceed out_cap %lld\n", hr.nout, out_cap);
    return GB_ERR_CAPACITY;
  }
  return GB_OK;
}
