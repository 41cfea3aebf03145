// gb_snap.cu -- SNAP layer streams on the device: the box codec of
// box_codec.f90 (CompressBoxesUsingCodec :616-698, DecompressBoxesUsingCodec
// :446-525) over 65536-box chunks, the Snappy raw format that
// snappy_api.cpp:9-37 applies to each chunk's codec bytes, and the .snap file
// of serialization.f90:15-130 (SaveCompressedStreamToDisk /
// RestoreCompressedStreamFromDisk).
//
// Encoding, per chunk (one 1024-thread CTA):
//   * widths, then heights of the non-square boxes, go into an open-addressing
//     table (16384 slots in shared memory; a chunk with more than 8192
//     distinct values is redone with a 131072-slot table in global memory)
//     that keeps each value's first position; a bitmap of first positions
//     with prefix popcounts gives each value its 1-based order of first
//     appearance, the codec's dictionary index, stored per box;
//   * blocks of 1024 boxes then size and write their records: a box's record
//     (infobyte, zigzag varint anchor deltas, the width / height as a varint
//     when new or an int16 index when seen before) depends only on the
//     previous box, the previous non-square box and the two ranks, and lands
//     at the sum of the sizes of the blocks and boxes before it.  One launch
//     sizes the blocks, a second writes them through shared memory.
// Snappy: each 65536-byte fragment of a chunk's codec bytes is compressed by
// one CTA with the fragment in shared memory.  A position's candidate is the
// latest earlier position with the same 11-bit hash of its 4 bytes; 32 warps
// find the candidates of 12288 positions (each warp's last positions per hash,
// a scan of these over the warps, then every warp through its positions), and
// mark those whose first 8 bytes match.  One warp takes the greedy parse from
// mark to mark, extends a match 32 bytes per step and emits Snappy literal /
// copy elements.  Fragments are concatenated behind the chunk's length
// preamble.  Decoding takes one CTA per chunk through the elements (all
// element forms of the format are accepted), with the last 32 KB of output in
// a shared-memory ring for the copies and long literals copied by the CTA.
// Decoding the codec.  Record boundaries: a record's length follows from its
// bytes, so a chain started anywhere falls in with the true one after a few
// records.  Every 128-byte segment guesses its first record by a chain from
// 96 bytes before it and walks to its end; one CTA per chunk then redoes the
// segments whose guess is not where the segment before them ended, until all
// agree, and the record counts give every segment its first record's number.
// Boxes: blocks of 1024 records sum their anchor deltas and dictionary
// entries, then every block adds up the blocks before it and rebuilds its
// boxes, with the dictionary entries looked up by block.
#include <cstdio>
#include <cstring>
#include <vector>

#include "gbool.h"
#include "gb_internal.h"

#define SN_CHUNK 65536  // boxes per chunk (box_codec.f90:227)
#define SN_FRAG 65536   // Snappy fragment (bytes)
#define SN_FCAP ((SN_FRAG + SN_FRAG / 6 + 64 + 15) / 16 * 16)
#define SN_T 1024       // threads of the per-chunk CTAs
#define SN_REC_MAX 31   // longest record of a valid box (1 + 5 + 5 + 10 + 10)
#define SN_MIN_MATCH 8  // shortest copy the compressor emits
#define SN_CODEC_VERSION 1
#define SN_LAYER_STATE_PNUM 4
#define KID_SNAP_ENC 60
#define KID_SNAP_BOUNDS 61
#define KID_SNAP_DEC 62
#define KID_SNAPPY_C 63
#define KID_SNAPPY_D 64

namespace {

// ---------------------------------------------------------------- helpers
__device__ __forceinline__ unsigned sn_zigzag(int v) {  // box_codec.f90:334-349 (fits 32 bits)
  return v < 0 ? (unsigned)(-(long long)v * 2 - 1) : (unsigned)v * 2u;
}
__device__ __forceinline__ int sn_unzigzag(unsigned long long v) {  // box_codec.f90:351-356
  return (int)(unsigned)((v >> 1) ^ (0ull - (v & 1ull)));
}
__host__ __device__ __forceinline__ int sn_vlen(unsigned long long v) {
  int n = 1;
  while (v >= 128ull) {
    v >>= 7;
    ++n;
  }
  return n;
}
__device__ __forceinline__ unsigned char* sn_put_varint(unsigned char* o, unsigned long long v) {
  while (v >= 128ull) {
    *o++ = (unsigned char)(v | 128ull);
    v >>= 7;
  }
  *o++ = (unsigned char)v;
  return o;
}
// varint at p (at most 10 bytes); *k receives its length, 0 when malformed
__device__ __forceinline__ unsigned long long sn_get_varint(const unsigned char* p, int* k) {
  unsigned long long r = 0;
  for (int i = 0; i < 10; ++i) {
    const unsigned b = p[i];
    r |= (unsigned long long)(b & 127u) << (7 * i);
    if (!(b & 128u)) {
      *k = i + 1;
      return r;
    }
  }
  *k = 0;
  return 0;
}

// len bytes from src to dst, thread t of nt: 16-byte groups of the destination, each from five aligned source words
// that lie inside [src, src + len); the ends byte by byte.
__device__ __forceinline__ void sn_copy(unsigned char* dst, const unsigned char* src, long long len, int t, int nt) {
  const long long i0 = 3 + ((16 - ((uintptr_t)(dst + 3) & 15)) & 15);
  const long long ng = len >= i0 + 20 ? (len - i0 - 20) / 16 + 1 : 0;
  const int sh = 8 * (int)((uintptr_t)(src + i0) & 3);
  const unsigned* s32 = reinterpret_cast<const unsigned*>(src + i0 - ((uintptr_t)(src + i0) & 3));
#pragma unroll 4
  for (long long g = t; g < ng; g += nt) {
    unsigned w[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) w[j] = s32[4 * g + j];
    *reinterpret_cast<uint4*>(dst + i0 + 16 * g) =
        make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh), __funnelshift_r(w[2], w[3], sh),
                   __funnelshift_r(w[3], w[4], sh));
  }
  for (long long i = t; i < (ng ? i0 : len); i += nt) dst[i] = src[i];
  if (ng)
    for (long long i = i0 + 16 * ng + t; i < len; i += nt) dst[i] = src[i];
}

// ---------------------------------------------------------------- block scans
struct SumS {
  unsigned a;
};
struct LastS {  // last valid value (has = 0: none)
  int has, val;
};
struct Sum4 {
  unsigned x, y, nw, nh;
};
struct Last2 {
  int w, h;  // 0 = none
};
__device__ __forceinline__ SumS op(SumS p, SumS q) { return {p.a + q.a}; }
__device__ __forceinline__ LastS op(LastS p, LastS q) { return q.has ? q : p; }
__device__ __forceinline__ Sum4 op(Sum4 p, Sum4 q) { return {p.x + q.x, p.y + q.y, p.nw + q.nw, p.nh + q.nh}; }
__device__ __forceinline__ Last2 op(Last2 p, Last2 q) { return {q.w ? q.w : p.w, q.h ? q.h : p.h}; }
__device__ __forceinline__ SumS shup(SumS v, int d) { return {__shfl_up_sync(0xffffffffu, v.a, d)}; }
__device__ __forceinline__ LastS shup(LastS v, int d) {
  return {__shfl_up_sync(0xffffffffu, v.has, d), __shfl_up_sync(0xffffffffu, v.val, d)};
}
__device__ __forceinline__ Sum4 shup(Sum4 v, int d) {
  return {__shfl_up_sync(0xffffffffu, v.x, d), __shfl_up_sync(0xffffffffu, v.y, d),
          __shfl_up_sync(0xffffffffu, v.nw, d), __shfl_up_sync(0xffffffffu, v.nh, d)};
}
__device__ __forceinline__ Last2 shup(Last2 v, int d) {
  return {__shfl_up_sync(0xffffffffu, v.w, d), __shfl_up_sync(0xffffffffu, v.h, d)};
}

// Exclusive block scan (all threads of the block call it); buf holds 32
// entries and must not be reused by the next call (callers alternate two).
// *tot receives the block total.
template <class T>
__device__ __forceinline__ T block_excl(T x, T ident, T* buf, T* tot) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  T inc = x;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const T o = shup(inc, d);
    if (lane >= d) inc = op(o, inc);
  }
  if (lane == 31) buf[wid] = inc;
  __syncthreads();
  if (wid == 0) {
    T v = lane < nw ? buf[lane] : ident;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const T o = shup(v, d);
      if (lane >= d) v = op(o, v);
    }
    if (lane < nw) buf[lane] = v;
  }
  __syncthreads();
  T ex = shup(inc, 1);
  if (lane == 0) ex = ident;
  *tot = buf[nw - 1];
  return wid ? op(buf[wid - 1], ex) : ex;
}

// ---------------------------------------------------------------- encoder: dictionary ranks
// Open-addressing table of one chunk: slot = (first position << 32) | value,
// empty = all ones (positions are below 65536, so an occupied slot never has
// an all-ones high word).  Inserting an existing value lowers its position
// with atomicMin on the whole word, which keeps the value.
#define SN_EMPTY 0xffffffffffffffffull
#define SN_STAB_SLOTS 16384  // shared table: at most 8192 distinct values
#define SN_GTAB_SLOTS 131072 // global table (a chunk has at most 65536 values)

__device__ __forceinline__ unsigned sn_slot(int v, unsigned mask) { return ((unsigned)v * 0x9E3779B1u >> 15) & mask; }

// inserts (v, j); false when the table holds `limit` values already
__device__ __forceinline__ bool tab_insert(unsigned long long* tab, unsigned mask, int v, unsigned j,
                                           unsigned* ndist, unsigned limit) {
  const unsigned long long mine = ((unsigned long long)j << 32) | (unsigned)v;
  unsigned s = sn_slot(v, mask);
  for (unsigned probe = 0; probe <= mask; ++probe) {
    unsigned long long cur = *(volatile unsigned long long*)&tab[s];
    if (cur == SN_EMPTY) {
      if (*(volatile unsigned*)ndist >= limit) return false;
      cur = atomicCAS(&tab[s], SN_EMPTY, mine);
      if (cur == SN_EMPTY) {
        atomicAdd(ndist, 1u);
        return true;
      }
    }
    if ((unsigned)cur == (unsigned)v) {
      if ((unsigned)(cur >> 32) > j) atomicMin(&tab[s], mine);
      return true;
    }
    s = (s + 1u) & mask;
  }
  return false;
}

// first position of v (the value must be in the table)
__device__ __forceinline__ unsigned tab_first(const unsigned long long* tab, unsigned mask, int v) {
  unsigned s = sn_slot(v, mask);
  for (unsigned probe = 0; probe <= mask; ++probe) {
    const unsigned long long cur = *(const volatile unsigned long long*)&tab[s];
    if (cur == SN_EMPTY) break;
    if ((unsigned)cur == (unsigned)v) return (unsigned)(cur >> 32);
    s = (s + 1u) & mask;
  }
  return 0xffffffffu;
}

// 1-based order of first appearance of the value first seen at position p
__device__ __forceinline__ unsigned sn_rank(const unsigned* bits, const unsigned* pre, unsigned p) {
  return pre[p >> 5] + __popc(bits[p >> 5] & ((1u << (p & 31)) - 1u)) + 1u;
}

// Dictionary ranks of one chunk's widths (blockIdx.y 0: ranks[b]) or of its
// non-square boxes' heights (1: ranks[n + b]) per CTA = order of first
// appearance | first << 31.  A CTA takes most of an SM's shared memory, so
// chunks fill the chip in waves; half a chunk per CTA leaves less of the last
// one idle, and SN_RLD boxes are loaded ahead of their inserts (184 chunks:
// 388 -> 173 us).  GT: 131072-slot tables in global memory for the chunks in list
// (one table per CTA), else 16384-slot shared tables (chunk = block index);
// a chunk with more values than a shared table holds goes to ovf_list.
#define SN_RLD 4
template <bool GT>
__global__ void __launch_bounds__(SN_T, 1)
k_enc_rank(const int4* __restrict__ boxes, long long n, const int* __restrict__ list, int nlist,
           unsigned long long* gtab, unsigned* __restrict__ ranks, int* ovf_list, int* ovf_count, DStatus* st) {
  extern __shared__ __align__(16) unsigned char sm[];
  constexpr unsigned SLOTS = GT ? SN_GTAB_SLOTS : SN_STAB_SLOTS;
  constexpr unsigned MASK = SLOTS - 1u;
  constexpr unsigned LIMIT = GT ? SLOTS : SLOTS / 2;
  unsigned char* q = sm;
  unsigned long long* tab;
  if (GT) {
    tab = gtab + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * SLOTS;
  } else {
    tab = (unsigned long long*)q;
    q += SLOTS * 8;
  }
  unsigned* bits = (unsigned*)q;  // [2048] first-position bitmap
  unsigned* pre = bits + 2048;    // [2048] exclusive popcounts
  int* wsum = (int*)(pre + 2048); // [32]
  unsigned* flags = (unsigned*)(wsum + 32);  // distinct values, overflow
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const long long nchunks = (n + SN_CHUNK - 1) / SN_CHUNK;
  const long long nitems = GT ? nlist : nchunks;
  const int which = blockIdx.y;
  for (long long li = blockIdx.x; li < nitems; li += gridDim.x) {
    if (GT && li >= list[which - 2]) break;  // the widths' and the heights' lists alternate behind their counts
    const long long c = GT ? list[2 * li + which] : li;
    const long long b0 = c * SN_CHUNK;
    const int nb = (int)min((long long)SN_CHUNK, n - b0);
    bool ovf = false;
    {
      for (unsigned i = t; i < SLOTS; i += SN_T) tab[i] = SN_EMPTY;
      for (int i = t; i < 2048; i += SN_T) bits[i] = 0;
      if (t < 2) flags[t] = 0;
      __syncthreads();
      bool full = false;
      for (int j0 = t; j0 < nb && !full; j0 += SN_RLD * SN_T) {
        int4 ld[SN_RLD];
#pragma unroll
        for (int u = 0; u < SN_RLD; ++u)
          if (j0 + u * SN_T < nb) ld[u] = boxes[b0 + j0 + u * SN_T];
#pragma unroll
        for (int u = 0; u < SN_RLD; ++u) {
          const int j = j0 + u * SN_T;
          const int4 b = ld[u];
          const int w = (int)((unsigned)b.z - (unsigned)b.x), h = (int)((unsigned)b.w - (unsigned)b.y);
          if (full || j >= nb || (which && w == h)) continue;
          if (!tab_insert(tab, MASK, which ? h : w, (unsigned)j, &flags[0], LIMIT)) {
            flags[1] = 1;
            full = true;
          }
        }
      }
      __syncthreads();
      ovf = *(volatile unsigned*)&flags[1] != 0;
    }
    if (!ovf) {  // uniform
      for (unsigned i = t; i < SLOTS; i += SN_T) {
        const unsigned long long cur = *(volatile unsigned long long*)&tab[i];
        if (cur != SN_EMPTY) {
          const unsigned p = (unsigned)(cur >> 32);
          atomicOr(&bits[p >> 5], 1u << (p & 31));
        }
      }
      __syncthreads();
      {  // exclusive popcount prefix, two words per thread
        const int pc = __popc(bits[2 * t]) + __popc(bits[2 * t + 1]);
        int inc = pc;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, inc, d);
          if (lane >= d) inc += o;
        }
        if (lane == 31) wsum[wid] = inc;
        __syncthreads();
        if (wid == 0) {
          int v = wsum[lane];
#pragma unroll
          for (int d = 1; d < 32; d <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d) v += o;
          }
          wsum[lane] = v;
        }
        __syncthreads();
        const int ex = inc - pc + (wid ? wsum[wid - 1] : 0);
        pre[2 * t] = (unsigned)ex;
        pre[2 * t + 1] = (unsigned)ex + __popc(bits[2 * t]);
      }
      __syncthreads();
      unsigned* out = ranks + (which ? n : 0) + b0;
      for (int j0 = t; j0 < nb; j0 += SN_RLD * SN_T) {
        int4 ld[SN_RLD];
#pragma unroll
        for (int u = 0; u < SN_RLD; ++u)
          if (j0 + u * SN_T < nb) ld[u] = boxes[b0 + j0 + u * SN_T];
#pragma unroll
        for (int u = 0; u < SN_RLD; ++u) {
          const int j = j0 + u * SN_T;
          const int4 b = ld[u];
          const int w = (int)((unsigned)b.z - (unsigned)b.x), h = (int)((unsigned)b.w - (unsigned)b.y);
          if (j >= nb || (which && w == h)) continue;
          const unsigned p = tab_first(tab, MASK, which ? h : w);
          if (p >= SN_CHUNK) {
            gb_set_error(st, GB_ERR_INTERNAL, KID_SNAP_ENC, b0 + j);
            continue;
          }
          out[j] = sn_rank(bits, pre, p) | ((p == (unsigned)j) ? 0x80000000u : 0u);
        }
      }
      __syncthreads();
    }
    if (ovf && t == 0) {
      if (GT)
        gb_set_error(st, GB_ERR_INTERNAL, KID_SNAP_ENC, c);
      else
        ovf_list[2 * atomicAdd(&ovf_count[which], 1) + which] = (int)c;
    }
    __syncthreads();
  }
}

// Codec records from the ranks, SN_RB boxes per block, four consecutive ones
// per thread.  WRITE: the block's records are put together in shared memory
// and copied to raw at the chunk's offset plus the sizes of the blocks before
// it; else bsize[block] receives the block's byte count.  (One CTA per chunk,
// 64 steps behind one another, took 369 us for the sizes and 606 us for the
// records of 184 chunks, written byte by byte.)
#define SN_RB 1024
#define SN_RT 256
#define SN_BPC (SN_CHUNK / SN_RB)  // blocks per chunk: 64
template <bool WRITE>
__global__ void __launch_bounds__(SN_RT)
k_enc_emit(const int4* __restrict__ boxes, long long n, const unsigned* __restrict__ ranks, int* __restrict__ bsize,
           const long long* __restrict__ raw_off, unsigned char* __restrict__ raw, DStatus* st) {
  __shared__ SumS bufS[32];
  __shared__ LastS bufL[32];
  __shared__ int s_back, s_off;
  extern __shared__ __align__(16) unsigned char sm[];  // WRITE: SN_RB * SN_REC_MAX bytes
  const long long c = blockIdx.x / SN_BPC;
  const int kb = blockIdx.x % SN_BPC, t = threadIdx.x;
  const long long b0 = c * SN_CHUNK;
  const int nb = (int)min((long long)SN_CHUNK, n - b0);
  const int j0 = kb * SN_RB;
  if (j0 >= nb) {
    if (!WRITE && t == 0) bsize[blockIdx.x] = 0;
    return;
  }
  const int4* bx = boxes + b0;
  int4 b[5];  // the box before the thread's four, then these
  LastS lh{0, 0};
#pragma unroll
  for (int u = 0; u < 5; ++u) {
    const int j = j0 + 4 * t + u - 1;
    b[u] = j >= 0 && j < nb ? bx[j] : make_int4(0, 0, 0, 0);
  }
  int w[4], h[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    w[u] = (int)((unsigned)b[u + 1].z - (unsigned)b[u + 1].x);
    h[u] = (int)((unsigned)b[u + 1].w - (unsigned)b[u + 1].y);
    lh = op(lh, LastS{j0 + 4 * t + u < nb && w[u] != h[u], h[u]});
  }
  // the last non-square box of the chunk before this block, searched backwards when the block needs it
  LastS before{0, 0};
  if (t == 0) s_back = -1;
  if (__syncthreads_or(lh.has) && j0 > 0) {
    for (int e = j0; e > 0; e -= SN_RT) {
      const int j = e - 1 - t;
      if (j >= 0) {
        const int4 q = bx[j];
        if ((unsigned)q.z - (unsigned)q.x != (unsigned)q.w - (unsigned)q.y) atomicMax(&s_back, j);
      }
      __syncthreads();
      const int found = s_back;
      __syncthreads();
      if (found >= 0) break;
    }
    if (s_back >= 0) {
      const int4 q = bx[s_back];
      before = LastS{1, (int)((unsigned)q.w - (unsigned)q.y)};
    }
  }
  LastS tl;
  LastS ph = op(before, block_excl(lh, LastS{0, 0}, bufL, &tl));
  unsigned info[4], wr[4], hr[4], size = 0;
  int dx[4], dy[4];
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int j = j0 + 4 * t + u;
    info[u] = wr[u] = hr[u] = 0;
    dx[u] = dy[u] = 0;
    if (j >= nb) continue;
    const int4 q = b[u + 1], pb = b[u];  // the anchor cursor starts at 0 and follows x1 (b[0] is 0 at the chunk's start)
    const bool sq = w[u] == h[u];
    const int pw = (int)((unsigned)pb.z - (unsigned)pb.x);
    dx[u] = (int)((unsigned)q.x - (unsigned)pb.x);
    dy[u] = (int)((unsigned)q.y - (unsigned)pb.y);
    if (sq) info[u] |= 16;
    if (dx[u]) info[u] |= 32;
    if (dy[u]) info[u] |= 64;
    const unsigned rw = ranks[b0 + j];
    wr[u] = rw & 0x7fffffffu;
    if (j == 0 || w[u] != pw) info[u] |= (rw >> 31) ? 3u : 1u;
    if (!sq) {
      const unsigned rh = ranks[n + b0 + j];
      hr[u] = rh & 0x7fffffffu;
      if (!ph.has || ph.val != h[u]) info[u] |= (rh >> 31) ? 12u : 4u;
      ph = LastS{1, h[u]};
    }
    size += 1;
    if (info[u] & 32) size += sn_vlen(sn_zigzag(dx[u]));
    if (info[u] & 64) size += sn_vlen(sn_zigzag(dy[u]));
    if (info[u] & 1) size += (info[u] & 2) ? sn_vlen((unsigned long long)(long long)w[u]) : 2;
    if (info[u] & 4) size += (info[u] & 8) ? sn_vlen((unsigned long long)(long long)h[u]) : 2;
  }
  SumS ts;
  const SumS ex = block_excl(SumS{size}, SumS{0}, bufS, &ts);
  if (!WRITE) {
    if (t == 0) bsize[blockIdx.x] = (int)ts.a;
    return;
  }
  if (t < 32) {  // sizes of the chunk's blocks before this one, and of all (checked by its last block)
    int v = 0, all = 0;
    for (int j = t; j < SN_BPC; j += 32) {
      const int x = bsize[c * SN_BPC + j];
      v += j < kb ? x : 0;
      all += x;
    }
    v = __reduce_add_sync(0xffffffffu, v);
    all = __reduce_add_sync(0xffffffffu, all);
    if (t == 0) {
      s_off = v;
      if (j0 + SN_RB >= nb && ((long long)v + ts.a != all || all != raw_off[c + 1] - raw_off[c]))
        gb_set_error(st, GB_ERR_INTERNAL, KID_SNAP_ENC, c);
    }
  }
  unsigned char* o = sm + ex.a;
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    if (j0 + 4 * t + u >= nb) break;
    *o++ = (unsigned char)info[u];
    if (info[u] & 32) o = sn_put_varint(o, sn_zigzag(dx[u]));
    if (info[u] & 64) o = sn_put_varint(o, sn_zigzag(dy[u]));
    if (info[u] & 1) {
      if (info[u] & 2) {
        o = sn_put_varint(o, (unsigned long long)(long long)w[u]);
      } else {  // int16 index, little-endian (wraps above 32767 as the reference's int16 does)
        *o++ = (unsigned char)wr[u];
        *o++ = (unsigned char)(wr[u] >> 8);
      }
    }
    if (info[u] & 4) {
      if (info[u] & 8) {
        o = sn_put_varint(o, (unsigned long long)(long long)h[u]);
      } else {
        *o++ = (unsigned char)hr[u];
        *o++ = (unsigned char)(hr[u] >> 8);
      }
    }
  }
  __syncthreads();
  sn_copy(raw + raw_off[c] + s_off, sm, ts.a, t, SN_RT);
}

// Chunk sizes from the block sizes (one warp per chunk).
__global__ void k_enc_sizes(const int* __restrict__ bsize, long long nchunks, long long* __restrict__ raw_size) {
  const long long c = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (c >= nchunks) return;
  int v = 0;
  for (int j = threadIdx.x & 31; j < SN_BPC; j += 32) v += bsize[c * SN_BPC + j];
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) raw_size[c] = v;
}

// ---------------------------------------------------------------- codec decoder
// Record boundaries by guessed segments (see the top).  The walk of a chunk
// is a serial chain of 65536 lengths (one CTA per chunk with one walking
// thread: 1774 us for 184 chunks); segments make it some 4000 chains of about
// 15 records per chunk, and the guesses cost 10 more each.  A block stages 256
// segments (32 KB) with the continuation bits of their bytes, so a length is
// one byte and three words from shared memory and then register work.
#define SN_SEG 128
#define SN_WARM 96        // a guess starts this many bytes before its segment
#define SN_SEGT 256       // segments (threads) per block
#define SN_SEGB (SN_SEG * SN_SEGT)
#define SN_LOOK 64        // bytes staged past the block (more than a record's length)
#define SN_STG (SN_WARM + SN_SEGB + SN_LOOK)
#define SN_LMAX 41           // longest record the decoder accepts (1 + 4 x 10)
#define SN_DEAD 0xffffffffu  // no chain reaches the segment (a malformed record lies before)

// Length of the record whose infobyte is `info`, from the continuation bits
// of the bytes behind it; 0 when a varint is longer than 10 bytes.
__device__ __forceinline__ int sn_len(unsigned info, unsigned long long cont) {
  int l = 1;
  bool bad = false;
  auto varint = [&](bool on) {
    const int k = __ffs(~(unsigned)cont);  // 0 or beyond 10: too long
    const bool ok = (unsigned)(k - 1) < 10u;
    bad |= on && !ok;
    const int u = on && ok ? k : 0;
    cont >>= u;
    l += u;
  };
  varint(info & 32);
  varint(info & 64);
  varint((info & 3) == 3);
  if ((info & 3) == 1) {
    cont >>= 2;
    l += 2;
  }
  const bool hf = (info & 20) == 4;
  varint(hf && (info & 8));
  if (hf && !(info & 8)) l += 2;
  return bad ? 0 : l;
}

struct SegStage {  // a block's bytes; byte pos of the chunk is at buf[pos - pos0]
  __align__(16) unsigned char buf[SN_STG + 32];
  unsigned cont[SN_STG / 32 + 4];
};

// Bytes [first, first + SN_STG) of the chunk (zeros outside [0, L)) and their
// continuation bits.  Returns the chunk position of buf[0].
__device__ __forceinline__ long long seg_stage(SegStage& s, const unsigned char* base, long long L, long long first) {
  // 16-byte groups of the source, so buf[0] lies up to 15 bytes before `first`
  const int sh = (int)((uintptr_t)(base + first) & 15);
  const long long p0 = first - sh;
  constexpr int U = 3;  // groups in flight per thread
  for (int i0 = threadIdx.x * 16; i0 < SN_STG + 32; i0 += U * SN_SEGT * 16) {
    uint4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * SN_SEGT * 16;
      const long long p = p0 + i;
      v[u] = make_uint4(0, 0, 0, 0);
      if (i >= SN_STG + 32) continue;
      if (p >= 0 && p + 16 <= L) {
        v[u] = *reinterpret_cast<const uint4*>(base + p);
      } else if (p + 16 > 0 && p < L) {
        unsigned w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (p + j >= 0 && p + j < L) w[j >> 2] |= (unsigned)base[p + j] << (8 * (j & 3));
        v[u] = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * SN_SEGT * 16 < SN_STG + 32) *reinterpret_cast<uint4*>(s.buf + i0 + u * SN_SEGT * 16) = v[u];
  }
  __syncthreads();
  for (int w = threadIdx.x; w < SN_STG / 32 + 4; w += SN_SEGT) {
    unsigned m = 0;
    if (w < SN_STG / 32 + 1) {
      const unsigned* q = reinterpret_cast<const unsigned*>(s.buf) + w * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) m |= ((((q[j] >> 7) & 0x01010101u) * 0x10204080u) >> 28) << (4 * j);  // 4 top bits
    }
    s.cont[w] = m;
  }
  __syncthreads();
  return p0;
}

__device__ __forceinline__ int seg_len(const SegStage& s, int b) {
  const int w = (b + 1) >> 5, sh = (b + 1) & 31;
  const unsigned c0 = s.cont[w], c1 = s.cont[w + 1], c2 = s.cont[w + 2];
  const unsigned long long cont =
      ((unsigned long long)__funnelshift_r(c1, c2, sh) << 32) | __funnelshift_r(c0, c1, sh);
  return sn_len(s.buf[b], cont);
}

// Grid (chunks, blocks of the largest chunk): chunks can be more than a grid's y
// holds (65535).  blk[c] is the number of blocks of the chunks before c, so
// segment arrays are indexed by blk[c] + blockIdx.y.
__global__ void __launch_bounds__(SN_SEGT)
k_seg_guess(const unsigned char* __restrict__ raw, const long long* __restrict__ raw_off,
            const long long* __restrict__ raw_len, const long long* __restrict__ blk, unsigned* __restrict__ entry, unsigned* __restrict__ exit_, unsigned* __restrict__ cnt) {
  __shared__ SegStage s;
  const int c = blockIdx.x;
  const long long L = raw_len[c], blk0 = blk[c], start = (long long)blockIdx.y * SN_SEGB;
  if (blk0 + blockIdx.y >= blk[c + 1]) return;
  const long long p0 = seg_stage(s, raw + raw_off[c], L, start - SN_WARM);
  const int s0 = (int)(start - p0) + (int)threadIdx.x * SN_SEG, s1 = s0 + SN_SEG;
  const int lim = (int)min((long long)s1, L - p0);
  int b = s0;
  if (start + threadIdx.x > 0) {
    b = s0 - SN_WARM;
    while (b < s0) b += max(1, seg_len(s, b));
  }
  const size_t g = (size_t)(blk0 + blockIdx.y) * SN_SEGT + threadIdx.x;
  entry[g] = (unsigned)(p0 + b);
  unsigned n = 0;
  bool bad = false;
  while (b < lim) {
    const int l = seg_len(s, b);
    if (!l) {
      bad = true;
      break;
    }
    b += l;
    ++n;
  }
  exit_[g] = bad ? SN_DEAD : (unsigned)(p0 + b);
  cnt[g] = n;
}

// The segments from k0 on by table, for chains that do not fall in with the
// true one by themselves: records of one length whose bytes also parse out of
// step, as rows of equal boxes at some pitches are (20 e0 03 20 e0 03 ...).
// Each of SN_TABT threads goes backwards through its segment and leaves, for
// every byte, the records of a chain from there and where it ends; one thread
// then follows the chain from segment to segment.  (4M squares in rows at a
// pitch of 240 decode in 1.2 ms; with rounds of walks alone, each right for one
// more segment of a chunk, in 704 ms; with one serial walk a chunk in 1.6 ms.)
#define SN_ROUNDS 2   // rounds of walks before the table: layouts in Morton order need none or one
#define SN_TABT 256   // segments of a step of the table
#define SN_TABW 130   // a segment's entries, one word more than its bytes for the banks
#define SN_TEND 255   // the chain meets a malformed record
#define SN_TAB_SMEM (SN_TABT * SN_TABW * 2 + (SN_TABT + 1) * 4)
static_assert(SN_SEG + SN_LMAX < SN_TEND, "an entry's end is a byte");

// 4 bytes from chunk position p (on a word of memory), zeros outside [0, L)
__device__ __forceinline__ unsigned seg_word(const unsigned char* base, long long L, long long p) {
  if (p >= 0 && p + 4 <= L) return *reinterpret_cast<const unsigned*>(base + p);
  unsigned w = 0;
  for (int j = 0; j < 4; ++j)
    if (p + j >= 0 && p + j < L) w |= (unsigned)base[p + j] << (8 * j);
  return w;
}

__device__ __noinline__ void seg_table(const unsigned char* base, long long L, int k0, int nseg, unsigned* entry,
                                       const unsigned* exit_, unsigned* cnt, unsigned char* sm) {
  unsigned short* const tab = reinterpret_cast<unsigned short*>(sm);  // records << 8 | end, from the segment's start
  int* const ent = reinterpret_cast<int*>(tab + SN_TABT * SN_TABW);   // entries of the step's segments, -1: none
  const int t = threadIdx.x;
  if (t == 0) {
    const unsigned e = exit_[k0 - 1];
    ent[SN_TABT] = e == SN_DEAD ? -1 : (int)(e - (unsigned)k0 * SN_SEG);
  }
  for (; k0 < nseg; k0 += SN_TABT) {
    const int k = k0 + t, ns = min(SN_TABT, nseg - k0);
    const long long s0 = (long long)k * SN_SEG;
    unsigned short* const my = tab + t * SN_TABW;
    const int lim = (int)min((long long)SN_SEG, L - s0);
    if (t < ns) {
      const int mis = (int)((uintptr_t)(base + s0) & 3);
      unsigned long long cont = 0;  // continuation bits of the bytes behind the current one
#pragma unroll 4
      for (int i = (SN_SEG + SN_LMAX + 6) / 4; i >= 0; --i) {
        const unsigned w = seg_word(base, L, s0 - mis + 4 * i);
#pragma unroll
        for (int j = 3; j >= 0; --j) {
          const int b = 4 * i + j - mis;
          const unsigned v = (w >> (8 * j)) & 255u;
          if (b >= 0 && b < lim) {
            const int l = sn_len(v, cont), x = b + l;
            my[b] = (unsigned short)(!l ? SN_TEND : x >= lim ? (1 << 8) + x : (1 << 8) + my[x]);
          }
          cont = (cont << 1) | (v >> 7);
        }
      }
    }
    __syncthreads();
    if (t == 0) {
      int e = ent[SN_TABT];
      for (int q = 0; q < ns; ++q) {
        ent[q] = e;
        if (e < 0 || (long long)(k0 + q) * SN_SEG + e >= L) continue;  // the stream ends before the entry: no record
        const int x = tab[q * SN_TABW + e] & 255;
        e = x == SN_TEND ? -1 : x - SN_SEG;
        if (e < 0) e = -1;  // the last segment's: not used
      }
      ent[SN_TABT] = e;
    }
    __syncthreads();
    if (t < ns) {
      const int e = ent[t];
      entry[k] = e < 0 ? SN_DEAD : (unsigned)(s0 + e);
      cnt[k] = e < 0 || e >= lim ? 0u : (unsigned)(my[e] >> 8);
    }
    __syncthreads();  // the next step writes the table
  }
}

// One CTA per chunk: segments whose guess does not follow from the segment
// before them are walked again, a few times, until all agree (segment k is
// right after at most k rounds); what then still disagrees is settled by table.
// cnt becomes the number of the segment's first record.  The chunk is malformed
// when the chain holds fewer records than it has boxes.
__global__ void __launch_bounds__(SN_T)
k_seg_settle(const unsigned char* __restrict__ raw, const long long* __restrict__ raw_off,
             const long long* __restrict__ raw_len, const long long* __restrict__ blk, long long n, unsigned* entry,
             unsigned* exit_, unsigned* cnt, DStatus* st) {
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ SumS buf[2][32];
  __shared__ int s_first;
  const int c = blockIdx.x;
  const int nb = (int)min((long long)SN_CHUNK, n - (long long)c * SN_CHUNK);
  const long long L = raw_len[c];
  const unsigned char* base = raw + raw_off[c];
  // segments that start inside the stream (records lie in its first SN_CHUNK * SN_LMAX bytes)
  const int nseg = (int)((min(L, (long long)SN_CHUNK * SN_LMAX) + SN_SEG - 1) / SN_SEG);
  entry += blk[c] * SN_SEGT;
  exit_ += blk[c] * SN_SEGT;
  cnt += blk[c] * SN_SEGT;
  if (threadIdx.x == 0) s_first = nseg;
  for (int round = 0;; ++round) {
    int first = nseg;  // the thread's first segment that does not follow
    for (int k = threadIdx.x; k < nseg; k += SN_T) {
      const unsigned e = k ? *(volatile unsigned*)&exit_[k - 1] : 0u;
      if (entry[k] == e) continue;
      first = min(first, k);
      if (round == SN_ROUNDS) break;
      entry[k] = e;
      unsigned m = 0, x = e;
      if (e != SN_DEAD) {
        long long p = e;
        const long long lim = min(L, (long long)(k + 1) * SN_SEG);
        while (p < lim) {
          // continuation bits of the next bytes: 16 are nearly always enough (a record that needs more is too long
          // when the others are set), else as many as a record can use
          unsigned long long cont = 0;
          for (int j = 0; j < 16; ++j) {
            const long long q = p + 1 + j;
            if (q < L) cont |= (unsigned long long)(base[q] >> 7) << j;
          }
          int l = sn_len(base[p], cont | ~0xffffull);
          if (!l) {
            for (int j = 16; j < SN_LMAX; ++j) {
              const long long q = p + 1 + j;
              if (q < L) cont |= (unsigned long long)(base[q] >> 7) << j;
            }
            l = sn_len(base[p], cont);
          }
          if (!l) break;
          p += l;
          ++m;
        }
        x = p < lim ? SN_DEAD : (unsigned)p;
      }
      cnt[k] = m;
      *(volatile unsigned*)&exit_[k] = x;
    }
    if (!__syncthreads_or(first < nseg)) break;
    if (round == SN_ROUNDS) {
      atomicMin(&s_first, first);
      __syncthreads();
      seg_table(base, L, s_first, nseg, entry, exit_, cnt, sm);
      break;
    }
  }
  unsigned carry = 0;
  for (int k0 = 0, it = 0; k0 < nseg; k0 += SN_T, ++it) {
    const int k = k0 + (int)threadIdx.x;
    SumS tot;
    const SumS ex = block_excl(SumS{k < nseg ? cnt[k] : 0u}, SumS{0}, buf[it & 1], &tot);
    if (k < nseg) cnt[k] = carry + ex.a;
    carry += tot.a;
  }
  if (threadIdx.x == 0 && carry < (unsigned)nb) gb_set_error(st, GB_ERR_CORRUPT, KID_SNAP_BOUNDS, c);
}

// rec[c * SN_CHUNK + r] = offset of record r in the chunk: every segment marks
// its records' bytes, the block writes the marked offsets in order.
__global__ void __launch_bounds__(SN_SEGT)
k_seg_records(const unsigned char* __restrict__ raw, const long long* __restrict__ raw_off,
              const long long* __restrict__ raw_len, const long long* __restrict__ blk, long long n, const unsigned* __restrict__ entry, const unsigned* __restrict__ first, unsigned* __restrict__ rec,
              DStatus* st) {
  __shared__ SegStage s;
  __shared__ unsigned mark[SN_SEGB / 32];
  __shared__ SumS buf[32];
  const int c = blockIdx.x;
  const int nb = (int)min((long long)SN_CHUNK, n - (long long)c * SN_CHUNK);
  const long long L = raw_len[c], blk0 = blk[c], start = (long long)blockIdx.y * SN_SEGB;
  if (blk0 + blockIdx.y >= blk[c + 1]) return;
  const size_t g0 = (size_t)(blk0 + blockIdx.y) * SN_SEGT, g = g0 + threadIdx.x;
  if (first[g0] >= (unsigned)nb) return;  // uniform: the chunk's records end before this block
  for (int i = threadIdx.x; i < SN_SEGB / 32; i += SN_SEGT) mark[i] = 0;
  const long long p0 = seg_stage(s, raw + raw_off[c], L, start - SN_WARM);
  const int o = (int)(start - p0);  // buf index of the block's first byte
  const unsigned e = entry[g];
  if (e != SN_DEAD) {
    int b = (int)((long long)e - p0);
    const int lim = (int)min((long long)(o + ((int)threadIdx.x + 1) * SN_SEG), L - p0);
    unsigned r = first[g];
    while (b < lim && r < (unsigned)nb) {
      const int l = seg_len(s, b);
      if (!l) break;
      atomicOr(&mark[(b - o) >> 5], 1u << ((b - o) & 31));
      b += l;
      if (++r == (unsigned)nb && p0 + b > L) gb_set_error(st, GB_ERR_CORRUPT, KID_SNAP_BOUNDS, c);  // past the stream
    }
  }
  __syncthreads();
  // words of mark in order: SN_SEGB / 32 / SN_SEGT per thread
  constexpr int WPT = SN_SEGB / 32 / SN_SEGT;
  unsigned m = 0;
#pragma unroll
  for (int j = 0; j < WPT; ++j) m += __popc(mark[threadIdx.x * WPT + j]);
  SumS tot;
  const SumS ex = block_excl(SumS{m}, SumS{0}, buf, &tot);
  unsigned* out = rec + (long long)c * SN_CHUNK + first[g0] + ex.a;
#pragma unroll
  for (int j = 0; j < WPT; ++j) {
    const int w = threadIdx.x * WPT + j;
    for (unsigned v = mark[w]; v; v &= v - 1) *out++ = (unsigned)(start + w * 32 + __ffs(v) - 1);
  }
}

// Records to boxes, SN_RB records per block, four consecutive ones per thread.
// Pass 0 leaves the block's sums (anchor deltas, dictionary entries, last
// width and height set) and its dictionary entries, in the block's own part of
// the dictionary; pass 1 adds up the blocks of the chunk before it and writes
// the boxes.  The chunk's 64 steps in one CTA, each behind the scans of the
// one before, took 459 us for 184 chunks.
#define SN_REL (1 << 30)  // a "last set" code: the block's own entry, 1-based; else SN_ABS | index, 0 = none
#define SN_ABS (1 << 29)
struct RecBlock {
  unsigned dx, dy, nw, nh;
  int lw, lh, pad0, pad1;
};

struct RecFields {
  unsigned info;
  int dx, dy, wv, hv;
  __device__ __forceinline__ int wsel() const { return (info & 1) ? ((info & 2) ? 1 : 2) : 0; }
  __device__ __forceinline__ int hsel() const { return (info & 20) == 4 ? ((info & 8) ? 1 : 2) : 0; }
};

__device__ __forceinline__ RecFields rec_parse(const unsigned char* p) {
  RecFields f{p[0], 0, 0, 0, 0};
  int i = 1, k;
  if (f.info & 32) {
    f.dx = sn_unzigzag(sn_get_varint(p + i, &k));
    i += k;
  }
  if (f.info & 64) {
    f.dy = sn_unzigzag(sn_get_varint(p + i, &k));
    i += k;
  }
  if (f.info & 1) {
    if (f.info & 2) {
      f.wv = (int)(unsigned)sn_get_varint(p + i, &k);
      i += k;
    } else {
      f.wv = (short)(unsigned short)(p[i] | (p[i + 1] << 8));
      i += 2;
    }
  }
  if ((f.info & 20) == 4) {
    if (f.info & 8)
      f.hv = (int)(unsigned)sn_get_varint(p + i, &k);
    else
      f.hv = (short)(unsigned short)(p[i] | (p[i + 1] << 8));
  }
  return f;
}

template <bool WRITE>
__global__ void __launch_bounds__(SN_RT)
k_codec_decode(const unsigned char* __restrict__ raw, const long long* __restrict__ raw_off,
               const unsigned* __restrict__ rec, long long n, int* dict, RecBlock* blocks, int4* __restrict__ out,
               DStatus* st) {
  __shared__ Sum4 bufA[32];
  __shared__ Last2 bufB[32];
  __shared__ unsigned pnw[64], pnh[64];  // entries of the chunk's blocks before block j
  __shared__ RecBlock pre;               // sums of the blocks before this one, last codes made absolute
  __shared__ int s_skip;
  const long long c = blockIdx.x / SN_BPC;
  const int kb = blockIdx.x % SN_BPC, t = threadIdx.x;
  const long long b0 = c * SN_CHUNK;
  const int nb = (int)min((long long)SN_CHUNK, n - b0);
  const int j0 = kb * SN_RB;
  if (j0 >= nb) return;
  if (t == 0) s_skip = *(volatile int*)&st->err;  // the boundaries (or the Snappy layer) were malformed
  if (WRITE && t < 32) {
    unsigned dx = 0, dy = 0, nw = 0, nh = 0;
    int lw = 0, lh = 0;
    for (int h = 0; h < 2; ++h) {  // blocks 0..31, then 32..63
      const int j = h * 32 + t;
      RecBlock q{0, 0, 0, 0, 0, 0, 0, 0};
      if (j < kb) q = blocks[c * SN_BPC + j];
      SumS e[4] = {{q.dx}, {q.dy}, {q.nw}, {q.nh}};
#pragma unroll
      for (int d = 1; d < 32; d <<= 1)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const SumS o = shup(e[x], d);
          if (t >= d) e[x].a += o.a;
        }
      pnw[j] = nw + e[2].a - q.nw;
      pnh[j] = nh + e[3].a - q.nh;
      const unsigned mw = __ballot_sync(0xffffffffu, q.lw != 0), mh = __ballot_sync(0xffffffffu, q.lh != 0);
      // the last block that sets a width (height), its own entries counted from the blocks before it; an index
      // outside the entries up to that block sets none (the block reports its record)
      int aw = q.lw & SN_REL ? (int)pnw[j] + (q.lw & ~SN_REL) : (short)(q.lw & 0xffff);
      int ah = q.lh & SN_REL ? (int)pnh[j] + (q.lh & ~SN_REL) : (short)(q.lh & 0xffff);
      if (aw < 1 || aw > (int)(pnw[j] + q.nw)) aw = 0;
      if (ah < 1 || ah > (int)(pnh[j] + q.nh)) ah = 0;
      const int sw = __shfl_sync(0xffffffffu, aw, mw ? 31 - __clz(mw) : 0);
      const int sh = __shfl_sync(0xffffffffu, ah, mh ? 31 - __clz(mh) : 0);
      if (mw) lw = sw;
      if (mh) lh = sh;
      dx += __shfl_sync(0xffffffffu, e[0].a, 31);
      dy += __shfl_sync(0xffffffffu, e[1].a, 31);
      nw += __shfl_sync(0xffffffffu, e[2].a, 31);
      nh += __shfl_sync(0xffffffffu, e[3].a, 31);
    }
    if (t == 0) pre = RecBlock{dx, dy, nw, nh, lw, lh, 0, 0};
  }
  __syncthreads();
  if (s_skip) return;
  const unsigned char* base = raw + raw_off[c];
  int* const dw = dict + c * 2 * SN_CHUNK;
  int* const dh = dw + SN_CHUNK;
  RecFields f[4];
  Sum4 sum{0, 0, 0, 0};
  {
    unsigned at[4];
    const int j = j0 + 4 * t;
    if (j + 4 <= nb) {
      const uint4 q = *reinterpret_cast<const uint4*>(rec + b0 + j);
      at[0] = q.x;
      at[1] = q.y;
      at[2] = q.z;
      at[3] = q.w;
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u) at[u] = j + u < nb ? rec[b0 + j + u] : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      f[u] = RecFields{0, 0, 0, 0, 0};
      if (j + u < nb) f[u] = rec_parse(base + at[u]);
      sum = op(sum, Sum4{(unsigned)f[u].dx, (unsigned)f[u].dy, f[u].wsel() == 1 ? 1u : 0u, f[u].hsel() == 1 ? 1u : 0u});
    }
  }
  Sum4 tA;
  Sum4 ea = block_excl(sum, Sum4{0, 0, 0, 0}, bufA, &tA);
  if (!WRITE) {
    Last2 last{0, 0};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (f[u].wsel() == 1) {
        dw[j0 + ea.nw] = f[u].wv;
        last.w = SN_REL | (int)++ea.nw;
      } else if (f[u].wsel() == 2) {
        last.w = SN_ABS | (f[u].wv & 0xffff);
      }
      if (f[u].hsel() == 1) {
        dh[j0 + ea.nh] = f[u].hv;
        last.h = SN_REL | (int)++ea.nh;
      } else if (f[u].hsel() == 2) {
        last.h = SN_ABS | (f[u].hv & 0xffff);
      }
    }
    Last2 tB;
    block_excl(last, Last2{0, 0}, bufB, &tB);
    if (t == 0) blocks[c * SN_BPC + kb] = RecBlock{tA.x, tA.y, tA.nw, tA.nh, tB.w, tB.h, 0, 0};
    return;
  }
  ea = op(Sum4{pre.dx, pre.dy, pre.nw, pre.nh}, ea);
  // the dictionary index every record sets (0: none); an index outside the entries so far is malformed
  int wi[4], hi[4], bad = 0;
  Last2 last{0, 0};
  {
    Sum4 e = ea;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      wi[u] = hi[u] = 0;
      if (f[u].wsel() == 1) {
        wi[u] = (int)++e.nw;
      } else if (f[u].wsel() == 2) {
        if (f[u].wv < 1 || f[u].wv > (int)e.nw) bad |= 1 << u;
        else wi[u] = f[u].wv;
      }
      if (f[u].hsel() == 1) {
        hi[u] = (int)++e.nh;
      } else if (f[u].hsel() == 2) {
        if (f[u].hv < 1 || f[u].hv > (int)e.nh) bad |= 1 << u;
        else hi[u] = f[u].hv;
      }
      last = op(last, Last2{wi[u], hi[u]});
    }
  }
  Last2 tB;
  Last2 cur = op(Last2{pre.lw, pre.lh}, block_excl(last, Last2{0, 0}, bufB, &tB));
  auto entry_at = [&](const int* d, const unsigned* p, int idx) {  // entry idx (1-based) of the chunk's dictionary
    int j = 0;
#pragma unroll
    for (int s2 = 32; s2 > 0; s2 >>= 1)
      if (j + s2 <= kb && (int)p[j + s2] < idx) j += s2;
    return d[j * SN_RB + idx - 1 - (int)p[j]];
  };
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int j = j0 + 4 * t + u;
    ea.x += (unsigned)f[u].dx;
    ea.y += (unsigned)f[u].dy;
    cur = op(cur, Last2{wi[u], hi[u]});
    if (j >= nb) break;
    int w = 0, h = 0;
    if (cur.w < 1) bad |= 1 << u;
    else w = entry_at(dw, pnw, cur.w);
    if (f[u].info & 16) h = w;
    else if (cur.h < 1) bad |= 1 << u;
    else h = entry_at(dh, pnh, cur.h);
    if ((bad >> u) & 1) gb_set_error(st, GB_ERR_CORRUPT, KID_SNAP_DEC, b0 + j);
    out[b0 + j] = make_int4((int)ea.x, (int)ea.y, (int)(ea.x + (unsigned)w), (int)(ea.y + (unsigned)h));
  }
}

// ---------------------------------------------------------------- Snappy
// Writes one Snappy copy element of 4..64 bytes (lane 0 only); returns its size.
__device__ __forceinline__ int sn_copy_piece(unsigned char* o, unsigned off, int len, bool write) {
  if (len <= 11 && off < 2048u) {
    if (write) {
      o[0] = (unsigned char)(1u | ((unsigned)(len - 4) << 2) | ((off >> 8) << 5));
      o[1] = (unsigned char)off;
    }
    return 2;
  }
  if (write) {
    o[0] = (unsigned char)(2u | ((unsigned)(len - 1) << 2));
    o[1] = (unsigned char)off;
    o[2] = (unsigned char)(off >> 8);
  }
  return 3;
}

// One CTA per fragment (see the top; one warp per fragment, 2048 steps of 32
// positions behind one another and bytes copied singly, took 1950 us for 1600
// fragments, this 620 us: bound by shared memory, 74% of its wavefronts, the
// hash tables' random 2-byte accesses most of them; match_any in every step
// cost 1097 us, the scan one hash at a time 838 us).  fsrc / flen: the fragment's bytes in raw; the compressed
// elements go to fout + f * SN_FCAP, their count to flout.
#define SN_CT 1024
#define SN_CW (SN_CT / 32)
#define SN_SUB 12288  // positions whose candidates are held at once
struct SnapFrag {
  __align__(16) unsigned char buf[SN_FRAG + 32];  // the fragment at buf[sh], sh = its address modulo 16
  __align__(16) unsigned short tab[SN_CW][2048];  // latest position + 1 per hash (positions with 4 bytes left are < 65533)
  unsigned short last[2048];        // the same before the current SN_SUB positions
  unsigned short cand[SN_SUB];     // candidates of the marked positions
  unsigned mark[SN_SUB / 32];      // positions whose candidate matches SN_MIN_MATCH bytes
  int o, lit, fail;
};

__global__ void __launch_bounds__(SN_CT, 1)
k_snappy_compress(const unsigned char* __restrict__ raw, const long long* __restrict__ fsrc,
                  const int* __restrict__ flen, unsigned char* __restrict__ fout, int* __restrict__ flout,
                  DStatus* st) {
  extern __shared__ __align__(16) unsigned char sm[];
  SnapFrag& s = *reinterpret_cast<SnapFrag*>(sm);
  const int t = threadIdx.x, wid = t >> 5, lane = t & 31;
  const long long f = blockIdx.x;
  const unsigned char* src = raw + fsrc[f];
  const int fl = flen[f];
  unsigned char* out = fout + f * SN_FCAP;
  const int sh = (int)((uintptr_t)src & 15);
#pragma unroll 4
  for (int i = t * 16; i < SN_FRAG + 32; i += SN_CT * 16) {
    const int q = i - sh;  // fragment position of the group
    uint4 v = make_uint4(0, 0, 0, 0);
    if (q >= 0 && q + 16 <= fl) {
      v = *reinterpret_cast<const uint4*>(src + q);
    } else if (q + 16 > 0 && q < fl) {
      unsigned w[4] = {0, 0, 0, 0};
#pragma unroll
      for (int j = 0; j < 16; ++j)
        if (q + j >= 0 && q + j < fl) w[j >> 2] |= (unsigned)src[q + j] << (8 * (j & 3));
      v = make_uint4(w[0], w[1], w[2], w[3]);
    }
    *reinterpret_cast<uint4*>(s.buf + i) = v;
  }
  // Cleared once: what the tables hold of earlier positions is never above `last`, from which the running maximum
  // starts, nor at a later position, so it changes nothing.  (Cleared for every 8192 positions, the positions whose
  // candidates were held at once: 12M boxes encoded in 1320 us, now 1284.)
  for (int i = t; i < SN_CW * 2048 * 2 / 16; i += SN_CT) reinterpret_cast<uint4*>(s.tab)[i] = make_uint4(0, 0, 0, 0);
  for (int i = t; i < 2048; i += SN_CT) s.last[i] = 0;
  if (t == 0) s.fail = 0;
  __syncthreads();
  const unsigned* b32 = reinterpret_cast<const unsigned*>(s.buf);
  const unsigned char* by = s.buf + sh;
  auto ld32 = [&](int q) -> unsigned {  // the 4 bytes from position q (staged: q + 8 <= fl + 16)
    const int i = q + sh;
    return __funnelshift_r(b32[i >> 2], b32[(i >> 2) + 1], 8 * (i & 3));
  };
  unsigned short* tab = s.tab[wid];
  int o = 0, p = 0, lit = 0;  // the parse (warp 0)
  for (int h0 = 0; h0 + 4 <= fl; h0 += SN_SUB) {
    const int q0 = h0 + wid * (SN_SUB / SN_CW);
    const int q1 = min(q0 + SN_SUB / SN_CW, fl - 3);  // positions with 4 bytes left
    for (int i = t; i < SN_SUB / 32; i += SN_CT) s.mark[i] = 0;
    __syncwarp();
    unsigned val[SN_SUB / SN_CT];  // the 4 bytes from each of the lane's positions, for both searches (1277 -> 1239 us)
#pragma unroll
    for (int i = 0; i < SN_SUB / SN_CT; ++i) {  // the warp's latest position per hash
      const int b = q0 + i * 32;
      if (b >= q1) break;
      const int q = b + lane;
      const bool has = q < q1;
      val[i] = ld32(min(q, fl - 4));
      const unsigned h = (val[i] * 0x9E3779B1u) >> 21;
      bool again = has;
      while (__any_sync(0xffffffffu, again)) {  // lanes of one hash: the highest position stays
        if (again) tab[h] = (unsigned short)(q + 1);
        __syncwarp();
        again = has && tab[h] < (unsigned short)(q + 1);
        __syncwarp();
      }
    }
    __syncthreads();
    {  // before each warp's positions: a running maximum over the warps, two hashes per thread
      static_assert(SN_CT == 1024, "one word of two hashes per thread");
      unsigned run = reinterpret_cast<unsigned*>(s.last)[t];
#pragma unroll 8
      for (int w = 0; w < SN_CW; ++w) {
        unsigned* e = reinterpret_cast<unsigned*>(s.tab[w]) + t;
        const unsigned x = *e;
        *e = run;
        run = __vmaxu2(run, x);
      }
      reinterpret_cast<unsigned*>(s.last)[t] = run;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SN_SUB / SN_CT; ++i) {
      const int b = q0 + i * 32;
      if (b >= q1) break;
      const int q = b + lane;
      const bool has = q < q1;
      const unsigned v = val[i];
      const unsigned h = (v * 0x9E3779B1u) >> 21;
      unsigned cand = has ? tab[h] : 0u;  // 1-based
      __syncwarp();
      if (has) tab[h] = (unsigned short)(q + 1);
      __syncwarp();
      // lanes of one hash (one step in five): the latest lower lane is the candidate, the highest lane stays
      if (__any_sync(0xffffffffu, has && tab[h] != (unsigned short)(q + 1))) {
        const unsigned peers = __match_any_sync(0xffffffffu, has ? h : 0x10000u + lane);
        const unsigned lower = peers & ((1u << lane) - 1u);
        if (lower) cand = (unsigned)(b + 31 - __clz(lower)) + 1u;
        if (has && (peers >> lane) == 1u) tab[h] = (unsigned short)(q + 1);
        __syncwarp();
      }
      // a candidate counts when its first 8 bytes match (shorter copies are not emitted)
      const bool ok = has && q + SN_MIN_MATCH <= fl && cand && ld32((int)cand - 1) == v &&
                      ld32((int)cand + 3) == ld32(q + 4);
      const unsigned okm = __ballot_sync(0xffffffffu, ok);
      if (ok) s.cand[q - h0] = (unsigned short)(cand - 1);
      if (lane == 0 && okm) s.mark[(b - h0) >> 5] = okm;
    }
    __syncthreads();
    if (wid == 0) {
      const int hend = min(h0 + SN_SUB, fl - 3);
      while (p < hend && !s.fail) {
        // the next marked position at or after p, 32 words of marks at a time
        const int w0 = (p - h0) >> 5, w = w0 + lane;
        unsigned m = w < SN_SUB / 32 ? s.mark[w] : 0u;
        if (lane == 0) m &= 0xffffffffu << (p & 31);
        const unsigned any = __ballot_sync(0xffffffffu, m != 0);
        if (!any) {
          p = min(hend, h0 + ((w0 + 32) << 5));
          continue;
        }
        const int l0 = __ffs(any) - 1;
        p = h0 + ((w0 + l0) << 5) + __ffs(__shfl_sync(0xffffffffu, m, l0)) - 1;
        const int qs = s.cand[p - h0];
        int L = SN_MIN_MATCH;
        for (;;) {
          const int a = p + L + lane;
          const bool eq = a < fl && by[qs + L + lane] == by[a];
          const unsigned ne = __ballot_sync(0xffffffffu, !eq);
          if (ne) {
            L += __ffs(ne) - 1;
            break;
          }
          L += 32;
        }
        // pending literal
        if (p > lit) {
          const int len = p - lit;
          const unsigned mm = (unsigned)len - 1u;
          const int nb = mm < 60u ? 0 : mm < 256u ? 1 : 2;
          if (o + 1 + nb + len + 3 * ((L + 59) / 60) > SN_FCAP) {
            if (lane == 0) s.fail = 1;
            __syncwarp();
            break;
          }
          if (lane == 0) {
            out[o] = (unsigned char)(nb ? (59 + nb) << 2 : mm << 2);
            for (int i = 0; i < nb; ++i) out[o + 1 + i] = (unsigned char)(mm >> (8 * i));
          }
          sn_copy(out + o + 1 + nb, by + lit, len, lane, 32);
          o += 1 + nb + len;
        }
        {
          const unsigned off = (unsigned)(p - qs);
          int rem = L;
          while (rem >= 68) {
            o += sn_copy_piece(out + o, off, 64, lane == 0);
            rem -= 64;
          }
          if (rem > 64) {
            o += sn_copy_piece(out + o, off, 60, lane == 0);
            rem -= 60;
          }
          o += sn_copy_piece(out + o, off, rem, lane == 0);
        }
        p += L;
        lit = p;
      }
    }
    __syncthreads();  // the next positions overwrite marks, candidates and tables
    if (s.fail) break;
  }
  if (t == 0) {
    s.o = o;
    s.lit = lit;
  }
  __syncthreads();
  o = s.o;
  lit = s.lit;
  int bad = s.fail;
  if (!bad && fl > lit) {  // the last literal, by the whole CTA
    const int len = fl - lit;
    const unsigned mm = (unsigned)len - 1u;
    const int nb = mm < 60u ? 0 : mm < 256u ? 1 : 2;
    if (o + 1 + nb + len > SN_FCAP) {
      bad = 1;
    } else {
      if (t == 0) {
        out[o] = (unsigned char)(nb ? (59 + nb) << 2 : mm << 2);
        for (int i = 0; i < nb; ++i) out[o + 1 + i] = (unsigned char)(mm >> (8 * i));
      }
      sn_copy(out + o + 1 + nb, by + lit, len, t, SN_CT);
      o += 1 + nb + len;
    }
  }
  if (t == 0) {
    if (bad) gb_set_error(st, GB_ERR_INTERNAL, KID_SNAPPY_C, f);
    flout[f] = bad ? 0 : o;
  }
}

// Chunk preambles and fragment copies into the final stream.  One CTA per
// fragment; fdst[f] is the fragment's destination, pre_at / pre_val the
// chunks' preamble positions and values.
__global__ void k_snappy_gather(const unsigned char* __restrict__ fout, const int* __restrict__ flout,
                                const long long* __restrict__ fdst, long long nfrag,
                                const long long* __restrict__ pre_at, const long long* __restrict__ pre_val,
                                long long nchunks, unsigned char* __restrict__ dst) {
  const long long f = blockIdx.x;
  if (f < nfrag) {
    sn_copy(dst + fdst[f], fout + f * SN_FCAP, flout[f], threadIdx.x, blockDim.x);
  }
  if (blockIdx.x == 0)
    for (long long c = threadIdx.x; c < nchunks; c += blockDim.x) sn_put_varint(dst + pre_at[c], (unsigned long long)pre_val[c]);
}

// One CTA per chunk: Snappy raw stream -> codec bytes.  Warp 0 takes the
// elements; a literal of SN_LONG bytes or more is copied by the whole CTA, 16
// bytes per thread and step (a chunk of 65536-byte literals, as a stream
// without repeats has them, had one warp copy 1 byte per lane: 1892 us for
// 184 chunks).  Element tags are read from a 4 KB staging copy of the input;
// copies whose source lies in the last 32 KB of output are read from a
// shared-memory ring of it (older sources from global memory).
#define SN_RING 32768
#define SN_STAGE 4096
#define SN_LONG 1024
#define SN_DT 256
__global__ void __launch_bounds__(SN_DT)
k_snappy_decompress(const unsigned char* __restrict__ in_all, const long long* __restrict__ in_off,
                    const long long* __restrict__ in_len, unsigned char* out_all, const long long* __restrict__ out_off,
                    const long long* __restrict__ out_len, long long nchunks, DStatus* st) {
  extern __shared__ __align__(16) unsigned char dsm[];
  unsigned char* ring = dsm;           // output byte x at ring[(x + ra) % SN_RING] for the last SN_RING bytes
  unsigned char* stg = dsm + SN_RING;  // input bytes [sb, sb + SN_STAGE)
  __shared__ long long s_lit[3];       // a long literal: input position, output position, length (0: done)
  const int lane = threadIdx.x & 31;
  const long long c = blockIdx.x;
  if (c >= nchunks) return;
  const unsigned char* in = in_all + in_off[c];
  const long long len = in_len[c];
  unsigned char* out = out_all + out_off[c];
  const long long want = out_len[c];
  const int ra = (int)((uintptr_t)out & 15);  // ring and output agree modulo 16 bytes
  long long sb = -(long long)SN_STAGE - 8;
  auto stage = [&](long long p) {  // bytes p .. p + 7 staged (warp 0)
    if (p < sb || p + 8 > sb + SN_STAGE) {
      sb = p - (long long)((uintptr_t)(in + p) & 15);
      __syncwarp();
      for (int i0 = 0; i0 < SN_STAGE; i0 += 32 * 16 * 4) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const long long q = sb + i0 + u * 512 + lane * 16;
          v[u] = make_uint4(0, 0, 0, 0);
          if (q >= 0 && q + 16 <= len) {
            v[u] = *reinterpret_cast<const uint4*>(in + q);
          } else if (q + 16 > 0 && q < len) {
            unsigned w[4] = {0, 0, 0, 0};
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (q + j >= 0 && q + j < len) w[j >> 2] |= (unsigned)in[q + j] << (8 * (j & 3));
            v[u] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<uint4*>(stg + i0 + u * 512 + lane * 16) = v[u];
      }
      __syncwarp();
    }
  };
  int bad = 0;
  long long p = 0, o = 0;
  if (threadIdx.x < 32) {
    stage(0);
    unsigned long long v = 0;
    int k = 0;
    for (int i = 0; i < 5 && i < len; ++i) {
      const unsigned b = stg[i - sb];
      v |= (unsigned long long)(b & 127u) << (7 * i);
      if (!(b & 128u)) {
        k = i + 1;
        break;
      }
    }
    if (!k || (long long)v != want) bad = 1;
    p = k;
  }
  for (;;) {
    if (threadIdx.x < 32) {
      long long lit = 0;
      while (!bad && p < len) {
        stage(p);
        const unsigned tag = stg[p - sb];
        const unsigned char* tb = stg + (p - sb) + 1;  // up to 4 bytes after the tag
        ++p;
        const unsigned tt = tag & 3u;
        if (tt == 0) {
          long long m = tag >> 2;
          if (m >= 60) {
            const int nb = (int)m - 59;
            if (p + nb > len) {
              bad = 1;
              break;
            }
            m = 0;
            for (int i = 0; i < nb; ++i) m |= (long long)tb[i] << (8 * i);
            p += nb;
          }
          const long long L = m + 1;
          if (p + L > len || o + L > want) {
            bad = 1;
            break;
          }
          if (L >= SN_LONG) {
            lit = L;
            break;
          }
          for (long long i0 = 0; i0 < L; i0 += 128) {
            unsigned char v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const long long i = i0 + u * 32 + lane;
              v[u] = i < L ? in[p + i] : 0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const long long i = i0 + u * 32 + lane;
              if (i < L) {
                out[o + i] = v[u];
                ring[(o + i + ra) & (SN_RING - 1)] = v[u];
              }
            }
          }
          p += L;
          o += L;
        } else {
          long long L, off;
          if (tt == 1) {
            if (p + 1 > len) {
              bad = 1;
              break;
            }
            L = 4 + ((tag >> 2) & 7u);
            off = ((long long)(tag >> 5) << 8) | tb[0];
            p += 1;
          } else if (tt == 2) {
            if (p + 2 > len) {
              bad = 1;
              break;
            }
            L = 1 + (tag >> 2);
            off = (long long)tb[0] | ((long long)tb[1] << 8);
            p += 2;
          } else {
            if (p + 4 > len) {
              bad = 1;
              break;
            }
            L = 1 + (tag >> 2);
            off = (long long)tb[0] | ((long long)tb[1] << 8) | ((long long)tb[2] << 16) | ((long long)tb[3] << 24);
            p += 4;
          }
          if (off == 0 || off > o || o + L > want) {
            bad = 1;
            break;
          }
          // byte o + i repeats the period [o - off, o): every source precedes this element
          if (off + L <= SN_RING) {
            for (long long i = lane; i < L; i += 32) {
              const unsigned char v = ring[(o - off + (i < off ? i : i % off) + ra) & (SN_RING - 1)];
              out[o + i] = v;
              ring[(o + i + ra) & (SN_RING - 1)] = v;
            }
          } else {
            for (long long i = lane; i < L; i += 32) {
              const unsigned char v = out[o - off + (i < off ? i : i % off)];
              out[o + i] = v;
              ring[(o + i + ra) & (SN_RING - 1)] = v;
            }
          }
          o += L;
        }
        __syncwarp();
      }
      if (lane == 0) {
        s_lit[0] = p;
        s_lit[1] = o;
        s_lit[2] = lit;
      }
    }
    __syncthreads();
    const long long lp = s_lit[0], lo = s_lit[1], L = s_lit[2];
    if (L == 0) break;
    const long long keep = L - SN_RING;  // only the last SN_RING bytes stay in the ring
    auto put = [&](long long i) {
      const unsigned char v = in[lp + i];
      out[lo + i] = v;
      if (i >= keep) ring[(lo + i + ra) & (SN_RING - 1)] = v;
    };
    // body: 16-byte groups of the output, each from five aligned source words inside the literal
    const long long i0 = 3 + ((16 - ((uintptr_t)(out + lo + 3) & 15)) & 15);
    const long long ng = L >= i0 + 20 ? (L - i0 - 20) / 16 + 1 : 0;
    const unsigned char* src = in + lp + i0;
    const int sh = 8 * (int)((uintptr_t)src & 3);
    const unsigned* s32 = reinterpret_cast<const unsigned*>(src - ((uintptr_t)src & 3));
#pragma unroll 4
    for (long long g = threadIdx.x; g < ng; g += SN_DT) {
      unsigned w[5];
#pragma unroll
      for (int j = 0; j < 5; ++j) w[j] = s32[4 * g + j];
      const uint4 v = make_uint4(__funnelshift_r(w[0], w[1], sh), __funnelshift_r(w[1], w[2], sh),
                                 __funnelshift_r(w[2], w[3], sh), __funnelshift_r(w[3], w[4], sh));
      const long long i = i0 + 16 * g;
      *reinterpret_cast<uint4*>(out + lo + i) = v;
      if (i >= keep) *reinterpret_cast<uint4*>(ring + ((lo + i + ra) & (SN_RING - 1))) = v;
      else if (i + 16 > keep)
        for (int j = 0; j < 16; ++j) put(i + j);
    }
    for (long long i = threadIdx.x; i < (ng ? i0 : L); i += SN_DT) put(i);
    if (ng)
      for (long long i = i0 + 16 * ng + threadIdx.x; i < L; i += SN_DT) put(i);
    __syncthreads();
    p = lp + L;
    o = lo + L;
  }
  if (threadIdx.x == 0 && (bad || o != want)) gb_set_error(st, GB_ERR_CORRUPT, KID_SNAPPY_D, c);
}

// ---------------------------------------------------------------- host side
struct DevMem {  // scratch from the context's pool, freed on scope exit
  GbCtx& c;
  std::vector<void*> ptrs;
  explicit DevMem(GbCtx& ctx) : c(ctx) {}
  ~DevMem() {
    for (void* p : ptrs) gb_tmp_free(c, p);
  }
  template <class T>
  T* get(size_t count) {
    void* p = gb_tmp_alloc(c, std::max<size_t>(count * sizeof(T), 16));
    if (p) ptrs.push_back(p);
    return (T*)p;
  }
};

size_t rank_smem(bool gt) { return (gt ? 0 : (size_t)SN_STAB_SLOTS * 8) + 2 * 2048 * 4 + 32 * 4 + 16; }

long long nchunks_of(long long n) { return (n + SN_CHUNK - 1) / SN_CHUNK; }

// Encodes n device boxes: chunk table (num_boxes, raw_byte_size,
// compressed_size) into meta, the chunks' data concatenated into d_out.
int snap_encode(gb_context* ctx, const int4* d_boxes, long long n, int method, unsigned char* d_out, long long cap,
                long long* meta, long long* total) {
  GbCtx& c = ctx->c;
  const long long nch = nchunks_of(n);
  *total = 0;
  if (nch == 0) return GB_OK;
  DevMem M(c);
  long long* d_rsize = M.get<long long>(nch);
  long long* d_roff = M.get<long long>(nch + 1);
  int* d_ovf = M.get<int>(2 * nch + 2);  // the widths' and heights' counts of chunks that need global tables, then these
  unsigned* d_rank = M.get<unsigned>((size_t)2 * n);
  int* d_bsize = M.get<int>((size_t)nch * SN_BPC);
  if (!d_rsize || !d_roff || !d_ovf || !d_rank || !d_bsize) return gbi::set_err(ctx, GB_ERR_OOM, "snap encode scratch");
  cudaMemsetAsync(d_ovf, 0, 2 * sizeof(int), c.stream);
  const size_t sm_s = rank_smem(false), sm_g = rank_smem(true), sm_e = (size_t)SN_RB * SN_REC_MAX;
  const unsigned eb = (unsigned)(nch * SN_BPC);
  std::vector<long long> rsize(nch), roff(nch + 1, 0);
  int novf[2] = {0, 0};
  auto sizes = [&]() -> bool {  // block and chunk sizes from the ranks; the chunks' to the host
    k_enc_emit<false><<<eb, SN_RT, 0, c.stream>>>(d_boxes, n, d_rank, d_bsize, nullptr, nullptr, c.st);
    k_enc_sizes<<<(unsigned)((nch + 7) / 8), 256, 0, c.stream>>>(d_bsize, nch, d_rsize);
    c.launches += 2;
    cudaMemcpyAsync(rsize.data(), d_rsize, nch * 8, cudaMemcpyDeviceToHost, c.stream);
    return cudaStreamSynchronize(c.stream) == cudaSuccess;
  };
  cudaFuncSetAttribute((const void*)k_enc_rank<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_s);
  k_enc_rank<false><<<dim3((unsigned)nch, 2), SN_T, sm_s, c.stream>>>(d_boxes, n, nullptr, 0, nullptr, d_rank, d_ovf + 2,
                                                                      d_ovf, c.st);
  ++c.launches;
  cudaMemcpyAsync(novf, d_ovf, sizeof(novf), cudaMemcpyDeviceToHost, c.stream);
  if (!sizes()) return gbi::set_err(ctx, GB_ERR_CUDA, "snap encode (sizes)");
  if (novf[0] || novf[1]) {  // the listed chunks again with global tables
    const int gblocks = std::min(std::max(novf[0], novf[1]), std::max(1, c.nsm));
    unsigned long long* gtab = M.get<unsigned long long>((size_t)2 * gblocks * SN_GTAB_SLOTS);
    if (!gtab) return gbi::set_err(ctx, GB_ERR_OOM, "snap encode tables");
    k_enc_rank<true><<<dim3(gblocks, 2), SN_T, sm_g, c.stream>>>(d_boxes, n, d_ovf + 2, (int)nch, gtab, d_rank, nullptr,
                                                                 nullptr, c.st);
    ++c.launches;
    if (!sizes()) return gbi::set_err(ctx, GB_ERR_CUDA, "snap encode (sizes)");
  }
  {
    int e = gb_sync(ctx, nullptr);
    if (e) return e;
  }
  for (long long i = 0; i < nch; ++i) roff[i + 1] = roff[i] + rsize[i];
  const long long rtot = roff[nch];
  unsigned char* d_raw = method == 0 ? nullptr : M.get<unsigned char>((size_t)rtot + 16);
  if (method == 0 && rtot > cap) return gbi::set_err(ctx, GB_ERR_CAPACITY, "snap output buffer too small");
  if (method != 0 && !d_raw) return gbi::set_err(ctx, GB_ERR_OOM, "snap raw buffer");
  unsigned char* rawbuf = method == 0 ? d_out : d_raw;
  cudaMemcpyAsync(d_roff, roff.data(), (nch + 1) * 8, cudaMemcpyHostToDevice, c.stream);
  k_enc_emit<true><<<eb, SN_RT, sm_e, c.stream>>>(d_boxes, n, d_rank, d_bsize, d_roff, rawbuf, c.st);
  ++c.launches;
  if (method == 0) {
    for (long long i = 0; i < nch; ++i) {
      meta[3 * i] = std::min((long long)SN_CHUNK, n - i * SN_CHUNK);
      meta[3 * i + 1] = rsize[i];
      meta[3 * i + 2] = rsize[i];
    }
    *total = rtot;
    return gb_sync(ctx, nullptr);
  }
  // Snappy: fragments of each chunk's codec bytes
  std::vector<long long> fsrc, fchunk;
  std::vector<int> flen;
  for (long long i = 0; i < nch; ++i)
    for (long long f0 = 0; f0 < rsize[i]; f0 += SN_FRAG) {
      fsrc.push_back(roff[i] + f0);
      flen.push_back((int)std::min((long long)SN_FRAG, rsize[i] - f0));
      fchunk.push_back(i);
    }
  const long long nfrag = (long long)fsrc.size();
  long long* d_fsrc = M.get<long long>(nfrag + 1);
  int* d_flen = M.get<int>(nfrag + 1);
  int* d_flout = M.get<int>(nfrag + 1);
  long long* d_fdst = M.get<long long>(nfrag + 1);
  long long* d_pre = M.get<long long>(2 * nch);
  unsigned char* d_fout = M.get<unsigned char>((size_t)std::max(nfrag, 1ll) * SN_FCAP);
  if (!d_fsrc || !d_flen || !d_flout || !d_fdst || !d_pre || !d_fout) return gbi::set_err(ctx, GB_ERR_OOM, "snappy scratch");
  if (nfrag) {
    cudaMemcpyAsync(d_fsrc, fsrc.data(), nfrag * 8, cudaMemcpyHostToDevice, c.stream);
    cudaMemcpyAsync(d_flen, flen.data(), nfrag * 4, cudaMemcpyHostToDevice, c.stream);
    cudaFuncSetAttribute((const void*)k_snappy_compress, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(SnapFrag));
    k_snappy_compress<<<(unsigned)nfrag, SN_CT, sizeof(SnapFrag), c.stream>>>(d_raw, d_fsrc, d_flen, d_fout, d_flout, c.st);
    ++c.launches;
  }
  std::vector<int> flout(nfrag);
  if (nfrag) cudaMemcpyAsync(flout.data(), d_flout, nfrag * 4, cudaMemcpyDeviceToHost, c.stream);
  {
    int e = gb_sync(ctx, nullptr);
    if (e) return e;
  }
  std::vector<long long> fdst(nfrag), pre(2 * nch);
  long long at = 0, fi = 0;
  for (long long i = 0; i < nch; ++i) {
    pre[i] = at;
    pre[nch + i] = rsize[i];
    const long long start = at;
    at += sn_vlen((unsigned long long)rsize[i]);
    for (; fi < nfrag && fchunk[fi] == i; ++fi) {
      fdst[fi] = at;
      at += flout[fi];
    }
    meta[3 * i] = std::min((long long)SN_CHUNK, n - i * SN_CHUNK);
    meta[3 * i + 1] = rsize[i];
    meta[3 * i + 2] = at - start;
  }
  if (at > cap) return gbi::set_err(ctx, GB_ERR_CAPACITY, "snap output buffer too small");
  if (nfrag) cudaMemcpyAsync(d_fdst, fdst.data(), nfrag * 8, cudaMemcpyHostToDevice, c.stream);
  cudaMemcpyAsync(d_pre, pre.data(), 2 * nch * 8, cudaMemcpyHostToDevice, c.stream);
  k_snappy_gather<<<(unsigned)std::max(nfrag, 1ll), 256, 0, c.stream>>>(d_fout, d_flout, d_fdst, nfrag, d_pre,
                                                                       d_pre + nch, nch, d_out);
  ++c.launches;
  *total = at;
  return gb_sync(ctx, nullptr);
}

// Decodes the concatenated chunk data (device) described by meta.
int snap_decode(gb_context* ctx, const unsigned char* d_data, const long long* meta, long long nch, int method,
                int4* d_boxes) {
  GbCtx& c = ctx->c;
  if (nch == 0) return GB_OK;
  long long n = 0;
  std::vector<long long> roff(nch + 1, 0), coff(nch + 1, 0), rlen(nch), clen(nch);
  for (long long i = 0; i < nch; ++i) {
    if (meta[3 * i] < 0 || meta[3 * i] > SN_CHUNK || (i + 1 < nch && meta[3 * i] != SN_CHUNK) || meta[3 * i + 1] < 0 ||
        meta[3 * i + 2] < 0)
      return gbi::set_err(ctx, GB_ERR_CORRUPT, "snap chunk table");
    n += meta[3 * i];
    rlen[i] = meta[3 * i + 1];
    clen[i] = meta[3 * i + 2];
    roff[i + 1] = roff[i] + rlen[i];
    coff[i + 1] = coff[i] + clen[i];
  }
  if (method == 0)
    for (long long i = 0; i < nch; ++i)
      if (rlen[i] != clen[i]) return gbi::set_err(ctx, GB_ERR_CORRUPT, "snap chunk sizes");
  DevMem M(c);
  std::vector<long long> sblk(nch + 1, 0);  // blocks of segments before each chunk
  for (long long i = 0; i < nch; ++i)
    sblk[i + 1] = sblk[i] + (std::min(rlen[i], (long long)SN_CHUNK * SN_LMAX) + SN_SEGB - 1) / SN_SEGB;
  const size_t nseg = (size_t)std::max(sblk[nch], 1ll) * SN_SEGT;
  long long* d_tab = M.get<long long>(5 * (nch + 1));
  unsigned* d_rec = M.get<unsigned>((size_t)nch * SN_CHUNK);
  int* d_dict = M.get<int>((size_t)nch * 2 * SN_CHUNK);
  unsigned* d_seg = M.get<unsigned>(3 * nseg);  // entries, exits, counts
  RecBlock* d_blk = M.get<RecBlock>((size_t)nch * SN_BPC);
  unsigned char* d_raw = method == 0 ? nullptr : M.get<unsigned char>((size_t)roff[nch] + 16);
  if (!d_tab || !d_rec || !d_dict || !d_seg || !d_blk || (method != 0 && !d_raw)) return gbi::set_err(ctx, GB_ERR_OOM, "snap decode scratch");
  std::vector<long long> tab(5 * (nch + 1));
  std::copy(roff.begin(), roff.end(), tab.begin());
  std::copy(coff.begin(), coff.end(), tab.begin() + (nch + 1));
  std::copy(rlen.begin(), rlen.end(), tab.begin() + 2 * (nch + 1));
  std::copy(clen.begin(), clen.end(), tab.begin() + 3 * (nch + 1));
  std::copy(sblk.begin(), sblk.end(), tab.begin() + 4 * (nch + 1));
  cudaMemcpyAsync(d_tab, tab.data(), tab.size() * 8, cudaMemcpyHostToDevice, c.stream);
  const long long* d_roff = d_tab;
  const long long* d_coff = d_tab + (nch + 1);
  const long long* d_rlen = d_tab + 2 * (nch + 1);
  const long long* d_clen = d_tab + 3 * (nch + 1);
  const long long* d_sblk = d_tab + 4 * (nch + 1);
  const unsigned char* raw = d_data;
  if (method != 0) {
    cudaFuncSetAttribute((const void*)k_snappy_decompress, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         SN_RING + SN_STAGE);
    k_snappy_decompress<<<(unsigned)nch, SN_DT, SN_RING + SN_STAGE, c.stream>>>(d_data, d_coff, d_clen, d_raw, d_roff,
                                                                             d_rlen, nch, c.st);
    ++c.launches;
    raw = d_raw;
  }
  long long most = 0;  // blocks of the largest chunk
  for (long long i = 0; i < nch; ++i) most = std::max(most, sblk[i + 1] - sblk[i]);
  const dim3 sgrid((unsigned)nch, (unsigned)most);
  if (most) {
    k_seg_guess<<<sgrid, SN_SEGT, 0, c.stream>>>(raw, d_roff, d_rlen, d_sblk, d_seg, d_seg + nseg, d_seg + 2 * nseg);
    ++c.launches;
  }
  cudaFuncSetAttribute((const void*)k_seg_settle, cudaFuncAttributeMaxDynamicSharedMemorySize, SN_TAB_SMEM);
  k_seg_settle<<<(unsigned)nch, SN_T, SN_TAB_SMEM, c.stream>>>(raw, d_roff, d_rlen, d_sblk, n, d_seg, d_seg + nseg, d_seg + 2 * nseg,
                                                     c.st);
  if (most) {
    k_seg_records<<<sgrid, SN_SEGT, 0, c.stream>>>(raw, d_roff, d_rlen, d_sblk, n, d_seg, d_seg + 2 * nseg, d_rec, c.st);
    ++c.launches;
  }
  const unsigned rb = (unsigned)(nch * SN_BPC);
  k_codec_decode<false><<<rb, SN_RT, 0, c.stream>>>(raw, d_roff, d_rec, n, d_dict, d_blk, d_boxes, c.st);
  k_codec_decode<true><<<rb, SN_RT, 0, c.stream>>>(raw, d_roff, d_rec, n, d_dict, d_blk, d_boxes, c.st);
  c.launches += 3;
  return gb_sync(ctx, nullptr);
}

bool write_all(FILE* f, const void* p, size_t n) { return n == 0 || fwrite(p, 1, n, f) == n; }

}  // namespace

extern "C" int gb_snap_max_bytes(long long n, long long* bytes) {
  if (n < 0 || !bytes) return GB_ERR_ARG;
  const long long nch = nchunks_of(n);
  const long long raw = n * SN_REC_MAX;
  *bytes = raw + raw / 6 + nch * 64 + (raw / SN_FRAG + nch) * 64 + 64;
  return GB_OK;
}

extern "C" int gb_compress_boxes_to_stream(gb_context* ctx, const c_box* d_boxes, long long n, int method,
                                           unsigned char* d_out, long long cap, long long* chunk_meta, long long* total) {
  if (!ctx || n < 0 || !total || (n > 0 && (!d_boxes || !d_out || !chunk_meta))) return GB_ERR_ARG;
  if (method != 0 && method != 1) return gbi::set_err(ctx, GB_ERR_ARG, "compression method: 0 (codec only) or 1 (Snappy)");
  if (n > 0xffffffffll || ((uintptr_t)d_boxes & 15u)) return GB_ERR_ARG;
  std::lock_guard<std::mutex> lk(ctx->mu);
  return snap_encode(ctx, (const int4*)d_boxes, n, method, d_out, cap, chunk_meta, total);
}

extern "C" int gb_decompress_stream_to_boxes(gb_context* ctx, const unsigned char* d_data, const long long* chunk_meta,
                                             long long num_chunks, int method, c_box* d_boxes) {
  if (!ctx || num_chunks < 0 || (num_chunks > 0 && (!d_data || !chunk_meta || !d_boxes))) return GB_ERR_ARG;
  if (method != 0 && method != 1) return gbi::set_err(ctx, GB_ERR_ARG, "compression method: 0 (codec only) or 1 (Snappy)");
  if ((uintptr_t)d_boxes & 15u) return GB_ERR_ARG;
  std::lock_guard<std::mutex> lk(ctx->mu);
  return snap_decode(ctx, d_data, chunk_meta, num_chunks, method, (int4*)d_boxes);
}

extern "C" int gb_save_layer_to_snap(gb_context* ctx, const char* path, const c_box* d_boxes, long long n, int method,
                                     int layer_properties, const long long* pnum) {
  if (!ctx || !path || n < 0 || (n > 0 && !d_boxes)) return GB_ERR_ARG;
  long long cap = 0;
  gb_snap_max_bytes(n, &cap);
  const long long nch = nchunks_of(n);
  std::vector<long long> meta(3 * std::max(nch, 1ll));
  unsigned char* d_out = nullptr;
  if (n > 0 && gb_dev_alloc(ctx->c, (void**)&d_out, (size_t)cap) != cudaSuccess) return gbi::set_err(ctx, GB_ERR_OOM, "snap output buffer");
  long long total = 0;
  int e = n > 0 ? gb_compress_boxes_to_stream(ctx, d_boxes, n, method, d_out, cap, meta.data(), &total) : GB_OK;
  if (e == GB_OK && (method != 0 && method != 1)) e = gbi::set_err(ctx, GB_ERR_ARG, "compression method");
  std::vector<unsigned char> data((size_t)total);
  if (e == GB_OK && total > 0 &&
      cudaMemcpyAsync(data.data(), d_out, (size_t)total, cudaMemcpyDeviceToHost, ctx->c.stream) != cudaSuccess)
    e = GB_ERR_CUDA;
  if (e == GB_OK && cudaStreamSynchronize(ctx->c.stream) != cudaSuccess) e = GB_ERR_CUDA;
  if (d_out) cudaFree(d_out);
  if (e) return e;
  FILE* f = fopen(path, "wb");
  if (!f) return gbi::set_err(ctx, GB_ERR_ARG, "cannot open the .snap file for writing");
  // serialization.f90:27-48: version, properties, totals, [PNUM table], chunks, offset table, its position.
  // As SaveLayerToSnap (diskdesign_impl.f90:63-67) the R-tree bit is not saved; the PNUM bit says
  // whether the table follows, which is what RestoreCompressedStreamFromDisk reads.
  layer_properties &= ~8;
  layer_properties = pnum ? (layer_properties | SN_LAYER_STATE_PNUM) : (layer_properties & ~SN_LAYER_STATE_PNUM);
  const int ver = SN_CODEC_VERSION;
  bool ok = write_all(f, &ver, 4) && write_all(f, &layer_properties, 4) && write_all(f, &n, 8) &&
            write_all(f, &nch, 8) && write_all(f, &method, 4);
  long long pos = 28;
  if (ok && pnum) {
    ok = write_all(f, pnum, (size_t)n * 8);
    pos += n * 8;
  }
  std::vector<long long> offs(nch);
  long long dpos = 0;
  for (long long i = 0; ok && i < nch; ++i) {
    offs[i] = pos + 1;  // 1-based stream positions
    ok = write_all(f, &meta[3 * i], 24) && write_all(f, data.data() + dpos, (size_t)meta[3 * i + 2]);
    dpos += meta[3 * i + 2];
    pos += 24 + meta[3 * i + 2];
  }
  const long long table = pos + 1;
  ok = ok && write_all(f, offs.data(), (size_t)nch * 8) && write_all(f, &table, 8);
  ok = (fclose(f) == 0) && ok;
  return ok ? GB_OK : gbi::set_err(ctx, GB_ERR_ARG, "write to the .snap file failed");
}

namespace {
struct SnapFile {
  int ver = 0, props = 0, method = 0;
  long long total = 0, nch = 0;
  long long pnum_at = -1;
  std::vector<long long> meta;
  std::vector<unsigned char> data;
};

int read_snap(const char* path, SnapFile& S, bool with_data, std::string* why) {
  FILE* f = fopen(path, "rb");
  if (!f) {
    *why = "cannot open the .snap file";
    return GB_ERR_ARG;
  }
  fseek(f, 0, SEEK_END);
  const long long size = ftell(f);
  fseek(f, 0, SEEK_SET);
  if (size == 0) {  // serialization.f90:98-103: an empty file is an empty layer
    fclose(f);
    return GB_OK;
  }
  auto rd = [&](void* p, size_t k) { return k == 0 || fread(p, 1, k, f) == k; };
  bool ok = rd(&S.ver, 4) && rd(&S.props, 4) && rd(&S.total, 8) && rd(&S.nch, 8) && rd(&S.method, 4);
  if (!ok || S.total < 0 || S.nch < 0 || S.nch != nchunks_of(S.total) || S.total > 0xffffffffll) {
    fclose(f);
    *why = "malformed .snap header";
    return GB_ERR_CORRUPT;
  }
  long long pos = 28;
  if (S.props & SN_LAYER_STATE_PNUM) {
    S.pnum_at = pos;
    pos += 8 * S.total;
    fseek(f, pos, SEEK_SET);
  }
  S.meta.resize(3 * S.nch);
  long long dbytes = 0;
  std::vector<long long> at(S.nch);
  for (long long i = 0; ok && i < S.nch; ++i) {
    ok = rd(&S.meta[3 * i], 24) && S.meta[3 * i + 2] >= 0 && pos + 24 + S.meta[3 * i + 2] <= size;
    at[i] = pos + 24;
    pos += 24 + S.meta[3 * i + 2];
    dbytes += S.meta[3 * i + 2];
    if (ok) fseek(f, pos, SEEK_SET);
  }
  if (ok && with_data) {
    S.data.resize((size_t)dbytes);
    long long d = 0;
    for (long long i = 0; ok && i < S.nch; ++i) {
      fseek(f, at[i], SEEK_SET);
      ok = rd(S.data.data() + d, (size_t)S.meta[3 * i + 2]);
      d += S.meta[3 * i + 2];
    }
  }
  fclose(f);
  if (!ok) {
    *why = "truncated .snap file";
    return GB_ERR_CORRUPT;
  }
  return GB_OK;
}
}  // namespace

extern "C" int gb_snap_file_info(const char* path, long long* total_boxes, long long* num_chunks, int* method,
                                 int* layer_properties) {
  if (!path) return GB_ERR_ARG;
  SnapFile S;
  std::string why;
  const int e = read_snap(path, S, false, &why);
  if (e) return e;
  if (total_boxes) *total_boxes = S.total;
  if (num_chunks) *num_chunks = S.nch;
  if (method) *method = S.method;
  if (layer_properties) *layer_properties = S.props;
  return GB_OK;
}

extern "C" int gb_restore_snap_to_layer(gb_context* ctx, const char* path, c_box* d_boxes, long long cap, long long* n,
                                        long long* pnum) {
  if (!ctx || !path || !n) return GB_ERR_ARG;
  SnapFile S;
  std::string why;
  int e = read_snap(path, S, true, &why);
  if (e) return gbi::set_err(ctx, e, why.c_str());
  *n = S.total;
  if (S.total > cap || (S.total > 0 && !d_boxes)) return gbi::set_err(ctx, GB_ERR_CAPACITY, "box buffer too small");
  if (S.method != 0 && S.method != 1)
    return gbi::set_err(ctx, GB_ERR_ARG, "compression method of the file is not Snappy (ZLIB/ZSTD are not supported)");
  if (pnum && S.pnum_at >= 0) {
    FILE* f = fopen(path, "rb");
    const bool ok = f && fseek(f, S.pnum_at, SEEK_SET) == 0 && fread(pnum, 8, (size_t)S.total, f) == (size_t)S.total;
    if (f) fclose(f);
    if (!ok) return gbi::set_err(ctx, GB_ERR_CORRUPT, "truncated PNUM table");
  }
  if (S.total == 0) return GB_OK;
  unsigned char* d_data = nullptr;
  if (gb_dev_alloc(ctx->c, (void**)&d_data, std::max<size_t>(S.data.size(), 16)) != cudaSuccess)
    return gbi::set_err(ctx, GB_ERR_OOM, "snap data buffer");
  cudaMemcpyAsync(d_data, S.data.data(), S.data.size(), cudaMemcpyHostToDevice, ctx->c.stream);
  e = gb_decompress_stream_to_boxes(ctx, d_data, S.meta.data(), S.nch, S.method, d_boxes);
  cudaStreamSynchronize(ctx->c.stream);
  cudaFree(d_data);
  return e;
}
