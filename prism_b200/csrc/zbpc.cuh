// ZBPC lossless coder for the bit-plane buffer, byte-exact with the
// reference (src/encoder/zbpc.cu, include/encoder/RZE.hpp,
// d_zero_elimination.hpp, d_repetition_elimination.hpp).
//
// Stream layout: int64 plane-buffer size, uint16 csize[chunks], the chunk
// payloads back to back, zero padding to 8 bytes.  Chunks are 16 KiB pieces of
// each host plane (level 3 planes 0..31 first, then levels 2, 1, 0).  A chunk
// payload is either the raw bytes (csize == osize) or
//   [nonzero bytes][RE1 bytes][RE2 bytes][RE3 bytes][4-byte bitmap][osize:u16]
// where the zero-elimination bitmap (2048 B, bit i = byte i != 0, LSB first)
// is itself repetition-eliminated three times (2048 -> 256 -> 32 -> 4 bytes;
// a byte is kept iff it differs from its predecessor, byte -1 being 0).
// An all-zero chunk is just its 2-byte osize.
//
// B200 mapping.  Encode: chunks are coded independently into a plane-sized
// buffer, their offsets scanned, the payloads gathered (below); an entry point
// without scratch has a one-launch form with tickets and a decoupled look-back
// over a per-chunk status word (bounded spin: a stuck predecessor sets an
// error flag instead of hanging).  Decode: offsets come from a scan of the
// size table; one CTA per coded chunk rebuilds the bitmaps from the tail and
// expands the bytes (a fill-forward is an inclusive popcount prefix).
#pragma once
#include "chain.cuh"
#include "geometry.h"

namespace prism_b200 {

constexpr int kZThreads = 512;
constexpr int kZWarps = kZThreads / 32;

struct ChunkLoc {
  int level;        // host level (3 = coarsest, first in the stream)
  int64_t plane;
  int64_t offset;   // chunk index within the plane
  int64_t base;     // byte offset in the plane buffer
  int osize;
  bool last_of_plane;
};

// Chunk counts fit 32 bits (a plane buffer of 2^32 chunks would be 64 TB),
// so the plane/offset split is a 32-bit division (a 64-bit one is a long
// software sequence, run by every thread for every chunk).
__host__ __device__ __forceinline__ ChunkLoc locate_chunk(const Geometry& g, int64_t id) {
  ChunkLoc c;
  int64_t real = id;
  int l = 3;
  while (l > 0 && real >= g.chunks_level[l]) real -= g.chunks_level[l--];
  const uint32_t cpp = (uint32_t)(g.chunks_level[l] >> 5), r32 = (uint32_t)real;
  const uint32_t plane = r32 / cpp;
  c.level = l;
  c.plane = plane;
  c.offset = r32 - plane * cpp;
  int64_t b = 0;
  for (int i = 3; i > l; --i) b += g.hastride[i] << 5;
  c.base = b + c.plane * g.hastride[l] + c.offset * kChunk;
  int64_t rem = g.hastride[l] - c.offset * kChunk;
  c.osize = (int)(rem < kChunk ? rem : kChunk);
  c.last_of_plane = c.offset == cpp - 1;
  return c;
}

// Chunk holding byte `off` of the plane buffer (host placement: level 3's 32
// planes first, each plane cut into 16 KiB chunks; chunk ids follow the
// bytes).  Offsets past the buffer map past the last chunk.
__host__ __device__ __forceinline__ int64_t chunk_of_byte(const Geometry& g, int64_t off) {
  int64_t hb = 0, cb = 0;
  for (int l = 3; l >= 0; --l) {
    const int64_t span = g.hastride[l] << 5;
    if (off < hb + span || l == 0) {
      const int64_t rel = off - hb, p = rel / g.hastride[l];
      return cb + p * (g.chunks_level[l] >> 5) + (rel - p * g.hastride[l]) / kChunk;
    }
    hb += span;
    cb += g.chunks_level[l];
  }
  return 0;
}

// Host placement of a byte of the plane buffer: its chunk, the chunk's level,
// plane and byte range.  The byte is given with the level and plane whose
// device placement it was computed from; the two placements drift apart by a
// few bytes per plane, so the chunk is that plane's or a near one's and the
// walk below takes a step or none (no division).
struct HostChunk {
  int64_t id, begin, end;
  int level, plane;
};
__host__ __device__ __forceinline__ int64_t host_stride(const Geometry& g, int l) {
  return l == 0 ? g.hastride[0] : (l == 1 ? g.hastride[1] : (l == 2 ? g.hastride[2] : g.hastride[3]));
}
__host__ __device__ __forceinline__ HostChunk chunk_near(const Geometry& g, int level, int plane, int64_t off) {
  const int64_t h3 = g.hastride[3] << 5, h2 = h3 + (g.hastride[2] << 5), h1 = h2 + (g.hastride[1] << 5);
  int l = level, p = plane;
  int64_t stride = host_stride(g, l);
  int64_t base = (l == 3 ? 0 : (l == 2 ? h3 : (l == 1 ? h2 : h1))) + p * stride;
  while (off < base) {
    if (p == 0) {
      p = 31;
      stride = host_stride(g, ++l);
    } else {
      --p;
    }
    base -= stride;
  }
  while (off >= base + stride && !(l == 0 && p == 31)) {
    base += stride;
    if (p == 31) {
      p = 0;
      stride = host_stride(g, --l);
    } else {
      ++p;
    }
  }
  const int64_t k = (off - base) >> 14;
  static_assert(kChunk == 1 << 14, "chunk index by shift");
  HostChunk c;
  c.level = l;
  c.plane = p;
  c.begin = base + k * kChunk;
  c.end = c.begin + kChunk < base + stride ? c.begin + kChunk : base + stride;
  const int64_t c3 = g.chunks_level[3], c2 = c3 + g.chunks_level[2], c1 = c2 + g.chunks_level[1];
  const int64_t per = (l == 0 ? g.chunks_level[0] : (l == 1 ? g.chunks_level[1] : (l == 2 ? g.chunks_level[2] : c3))) >> 5;
  c.id = (l == 3 ? 0 : (l == 2 ? c3 : (l == 1 ? c2 : c1))) + p * per + k;
  return c;
}

// ---- block-wide helpers (512 threads) ----
__device__ __forceinline__ int warp_incl_scan(int v, int lane) {
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    int t = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += t;
  }
  return v;
}

// exclusive prefix over the block; *total receives the block sum.  Two
// barriers; scratch must not be reused before the next barrier.
__device__ __forceinline__ int block_excl_scan(int v, int* scratch, int* total) {
  int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = warp_incl_scan(v, lane);
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  int w = lane < kZWarps ? scratch[lane] : 0;
  int wi = warp_incl_scan(w, lane);
  int before = __shfl_sync(0xffffffffu, wi - w, warp);
  *total = __shfl_sync(0xffffffffu, wi, kZWarps - 1);
  __syncthreads();
  return before + incl - v;
}

struct EncodeShared {
  uint8_t in[kChunk + 16];
  // payload staging: nonzero bytes (< osize) plus up to 2048 + 256 + 32 + 6
  // bitmap bytes before the size check can reject the encoding
  uint8_t out[kChunk + 2048 + 512 + 16];
  uint8_t bm0[2048];
  uint8_t bm1[256];
  uint8_t bm2[32];
  uint8_t bm3[4];
  int scratch[40];
  long long ticket;
  long long excl;
  int csz;
};

// Copy n bytes from shared memory to an arbitrarily aligned global address:
// head bytes, then aligned 32-bit words (each assembled from two aligned
// shared words), then the tail.
__device__ __forceinline__ void copy_out(uint8_t* dst, const uint8_t* src, int n) {
  const int tid = threadIdx.x;
  int head = (int)((4 - ((uintptr_t)dst & 3)) & 3);
  if (head > n) head = n;
  if (tid < head) dst[tid] = src[tid];
  const int words = (n - head) >> 2;
  uint32_t* dw = reinterpret_cast<uint32_t*>(dst + head);
  const int sh = head & 3;
  const uint32_t* sw = reinterpret_cast<const uint32_t*>(src);
  for (int w = tid; w < words; w += kZThreads) {
    if (sh == 0) {
      dw[w] = sw[w];
    } else {
      // bytes head + 4w .. +3 = words w and w+1 shifted by sh bytes
      uint32_t lo = sw[w], hi = sw[w + 1];
      dw[w] = __funnelshift_r(lo, hi, 8 * sh);
    }
  }
  const int done = head + 4 * words;
  if (tid < n - done) dst[done + tid] = src[done + tid];
}

// Encode chunk `id` of one field (status is that field's slice, so the
// look-back ends at the field's first chunk).  All 512 threads of the CTA
// call this; it ends with a barrier.
__device__ __forceinline__ void encode_chunk(EncodeShared& sh, const uint8_t* __restrict__ planes, const Geometry& g,
                                             uint8_t* __restrict__ stream, unsigned long long* __restrict__ status,
                                             const int64_t id, uint64_t* __restrict__ comp_size_bp,
                                             uint64_t* __restrict__ lossless_size, int* __restrict__ error_flag,
                                             long long spin_limit) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t chunks = g.chunks;
  uint16_t* sizes = reinterpret_cast<uint16_t*>(stream + 8);
  uint8_t* data_out = stream + 8 + 2 * chunks;
  {
    const ChunkLoc loc = locate_chunk(g, id);
    const int osize = loc.osize;
    // ---- load 32 bytes per thread (base and osize are multiples of 8) ----
    const int b0 = tid * 32;
    uint32_t wds[8];
    {
      const uint2* src = reinterpret_cast<const uint2*>(planes + loc.base + b0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint2 v = make_uint2(0, 0);
        if (b0 + 8 * q < osize) v = __ldg(src + q);
        wds[2 * q] = v.x;
        wds[2 * q + 1] = v.y;
      }
    }
    uint4* in4 = reinterpret_cast<uint4*>(sh.in + b0);
    in4[0] = make_uint4(wds[0], wds[1], wds[2], wds[3]);
    in4[1] = make_uint4(wds[4], wds[5], wds[6], wds[7]);
    // zero elimination bitmap: bit j = byte b0 + j is nonzero
    uint32_t bits = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
      for (int j = 0; j < 4; ++j) bits |= (uint32_t)(((wds[k] >> (8 * j)) & 0xFF) != 0) << (4 * k + j);
    if (b0 + 32 > osize) bits = b0 >= osize ? 0u : bits & ((1u << (osize - b0)) - 1u);
    reinterpret_cast<uint32_t*>(sh.bm0)[tid] = bits;
    int nz_total;
    const int zoff = block_excl_scan(__popc(bits), sh.scratch, &nz_total);
    // ---- decide the encoding; build the payload in sh.out ----
    int csize;
    bool raw = false;
    if (nz_total == 0) {
      csize = 2;
      if (tid == 0) { sh.out[0] = (uint8_t)osize; sh.out[1] = (uint8_t)(osize >> 8); }
    } else if (nz_total + 6 >= osize) {
      raw = true;
      csize = osize;
    } else {
      // nonzero bytes, in order: every thread walks its 32 positions
      {
        int r = zoff;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          if ((bits >> j) & 1u) sh.out[r] = (uint8_t)(wds[j >> 2] >> (8 * (j & 3)));
          r += (bits >> j) & 1u;
        }
      }
      // RE 2048 -> 256: thread t flags bitmap bytes 4t..4t+3 (bm0 is complete
      // since the scan's barriers)
      const uint32_t cur = bits;
      const uint32_t prev_byte = tid == 0 ? 0u : (reinterpret_cast<const uint32_t*>(sh.bm0)[tid - 1] >> 24);
      uint32_t f1 = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t byte = (cur >> (8 * k)) & 0xFF;
        uint32_t before = k == 0 ? prev_byte : ((cur >> (8 * (k - 1))) & 0xFF);
        f1 |= (uint32_t)(byte != before) << k;
      }
      int c1;
      const int r1 = block_excl_scan(__popc(f1), sh.scratch, &c1);
      if (nz_total + c1 + 6 >= osize) {
        raw = true;
        csize = osize;
      } else {
        {
          int r = nz_total + r1;
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if ((f1 >> k) & 1u) sh.out[r++] = (uint8_t)(cur >> (8 * k));
        }
        uint32_t other = __shfl_down_sync(0xffffffffu, f1, 1);
        if ((tid & 1) == 0) sh.bm1[tid >> 1] = (uint8_t)(f1 | (other << 4));
        __syncthreads();
        if (warp == 0) {
          // RE 256 -> 32: lane l flags bm1 bytes 8l..8l+7
          uint32_t f2 = 0;
          uint8_t b1[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) b1[k] = sh.bm1[8 * lane + k];
          uint8_t before = lane == 0 ? 0 : sh.bm1[8 * lane - 1];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            f2 |= (uint32_t)(b1[k] != before) << k;
            before = b1[k];
          }
          int cnt2 = __popc(f2);
          int incl2 = warp_incl_scan(cnt2, lane);
          int c2 = __shfl_sync(0xffffffffu, incl2, 31);
          int r = nz_total + c1 + incl2 - cnt2;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if ((f2 >> k) & 1u) sh.out[r++] = b1[k];
          // RE 32 -> 4: lane l flags bm2 byte l (= f2)
          uint32_t prev2 = __shfl_up_sync(0xffffffffu, f2, 1);
          if (lane == 0) prev2 = 0;
          uint32_t bal = __ballot_sync(0xffffffffu, f2 != prev2);
          int c3 = __popc(bal);
          int pos = nz_total + c1 + c2;
          if ((f2 != prev2)) sh.out[pos + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)f2;
          pos += c3;
          int cs = pos + 6;
          if (lane == 0) sh.csz = cs;
          if (cs < osize) {
            if (lane < 4) sh.out[pos + lane] = (uint8_t)(bal >> (8 * lane));
            if (lane == 0) { sh.out[pos + 4] = (uint8_t)osize; sh.out[pos + 5] = (uint8_t)(osize >> 8); }
          }
        }
        __syncthreads();
        csize = sh.csz;
        if (csize >= osize) { raw = true; csize = osize; }
      }
    }
    // ---- decoupled look-back: flag 1 = local size, flag 2 = inclusive prefix ----
    if (warp == 0) {
      const unsigned long long kAgg = 1ull << 62, kInc = 2ull << 62, kMask = (1ull << 62) - 1;
      if (id == 0) {
        if (lane == 0) { atomicExch(&status[0], kInc | (unsigned long long)csize); sh.excl = 0; }
      } else {
        if (lane == 0) atomicExch(&status[id], kAgg | (unsigned long long)csize);
        long long excl = 0;
        int64_t j = id - 1;
        long long spins = 0;
        bool done = false;
        while (!done) {
          int64_t k = j - lane;
          unsigned long long v = k >= 0 ? 0ull : kInc;
          if (k >= 0) {
            do {
              v = atomicAdd(&status[k], 0ull);
              if (v == 0) {
                if (++spins > spin_limit) { atomicExch(error_flag, 1); v = kInc; }
                else __nanosleep(64);
              }
            } while (v == 0);
          }
          unsigned inc_mask = __ballot_sync(0xffffffffu, (v >> 62) == 2);
          int stop = inc_mask ? __ffs(inc_mask) - 1 : 32;
          long long part = lane <= stop ? (long long)(v & kMask) : 0;
#pragma unroll
          for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
          excl += part;
          if (inc_mask) done = true;
          else j -= 32;
        }
        if (lane == 0) {
          atomicExch(&status[id], kInc | (unsigned long long)(excl + csize));
          sh.excl = excl;
        }
      }
    }
    __syncthreads();
    const long long offs = sh.excl;
    if (tid == 0) {
      sizes[id] = (uint16_t)csize;
      if (loc.last_of_plane) comp_size_bp[(3 - loc.level) * 32 + loc.plane] = (uint64_t)(offs + csize);
      if (id == chunks - 1) *lossless_size = (uint64_t)(offs + csize);
    }
    copy_out(data_out + offs, raw ? sh.in : sh.out, csize);
    __syncthreads();
  }
}

// One-launch encoder (prism_lossless_encode_static): one CTA (512 threads, 32
// bytes each) per 16 KiB chunk, four CTAs per SM, chunks handed out in order by
// a ticket counter.
__global__ void __launch_bounds__(kZThreads, 4)
zbpc_encode_kernel(const uint8_t* __restrict__ planes, Geometry g, uint8_t* __restrict__ stream,
                   unsigned long long* __restrict__ status, unsigned long long* __restrict__ ticket,
                   uint64_t* __restrict__ comp_size_bp, uint64_t* __restrict__ lossless_size,
                   int* __restrict__ error_flag, long long spin_limit) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  EncodeShared& sh = *reinterpret_cast<EncodeShared*>(smem_raw);
  while (true) {
    if (threadIdx.x == 0) sh.ticket = (long long)atomicAdd(ticket, 1ull);
    __syncthreads();
    const int64_t id = sh.ticket;
    if (id >= g.chunks) break;
    encode_chunk(sh, planes, g, stream, status, id, comp_size_bp, lossless_size, error_flag, spin_limit);
  }
}

// stream header + zero padding once the total is known
__global__ void zbpc_finish_kernel(uint8_t* stream, Geometry g, const uint64_t* lossless_size,
                                   uint64_t* padded_size) {
  uint64_t total = 8 + 2 * (uint64_t)g.chunks + *lossless_size;
  uint64_t pad = (8 - total % 8) % 8;
  if (threadIdx.x < pad) stream[total + threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    long long hdr = (long long)g.aligned_size;
    for (int i = 0; i < 8; ++i) stream[i] = (uint8_t)(hdr >> (8 * i));
    *padded_size = total + pad;
  }
}

// ---------------- decode ----------------
// Per-chunk tables of a stream, derived from its size table:
//   coded[k] the k-th coded chunk; an all-zero chunk is 2 bytes, every other
//            chunk has another size (a chunk spans at least 8 bytes)
//   offs[i]  payload offset of chunk i (exclusive prefix sum of the sizes)
//   rank[i]  coded chunks before chunk i (rank[n] = all of them), so the coded
//            chunks of an id range [s, e) are coded[rank[s] .. rank[e])
// A coded entry holds the payload offset and size and the plane-buffer offset
// and size of its chunk (48 + 16 bits each): one 16-byte load tells a CTA
// all it needs.
struct ChunkTable {
  ulonglong2* coded;
  int64_t* offs;
  uint32_t* rank;
};
__host__ __device__ __forceinline__ ChunkTable chunk_table(void* p, int64_t n) {
  ChunkTable t;
  t.coded = reinterpret_cast<ulonglong2*>(p);
  t.offs = reinterpret_cast<int64_t*>(t.coded + n);
  t.rank = reinterpret_cast<uint32_t*>(t.offs + n);
  return t;
}
constexpr int kChunkTableBytes = 28;  // per chunk
inline size_t chunk_table_bytes(int64_t n) { return (size_t)n * kChunkTableBytes + 64; }
__device__ __forceinline__ ulonglong2 pack_coded(uint64_t off, uint32_t csize, uint64_t base, uint32_t osize) {
  return make_ulonglong2(off | (uint64_t)csize << 48, base | (uint64_t)osize << 48);
}
constexpr uint64_t kCodedMask = (1ull << 48) - 1;

constexpr uint32_t kZeroChunkBytes = 2;
constexpr int kScanThreads = 1024, kScanPer = 4, kScanItems = kScanThreads * kScanPer;

// One launch for the whole table: a CTA (`cta` of the field's) scans
// kScanItems sizes and gets the sums before them by reading the earlier part
// of the table itself (16 bits a chunk: 0.5 MB for a 4.3 GB field, from L2),
// which costs less than a second launch or a wait on the CTAs before it.
// each(i, size, off, rank, coded) sees every chunk of the CTA.
template <class F>
__device__ __forceinline__ void scan_chunks(const uint16_t* sizes, const int64_t n, const int cta, F each) {
  __shared__ unsigned long long warp_tot[32], prior_b[32];
  __shared__ unsigned prior_c[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t base = (int64_t)cta * kScanItems;
  const bool vec = (reinterpret_cast<uintptr_t>(sizes) & 7) == 0;  // four sizes a load
  auto four = [&](int64_t i, uint32_t (&v)[4]) {
    if (vec && i + 4 <= n) {
      const uint2 q = *reinterpret_cast<const uint2*>(sizes + i);
      v[0] = q.x & 0xffffu;
      v[1] = q.x >> 16;
      v[2] = q.y & 0xffffu;
      v[3] = q.y >> 16;
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = i + k < n ? sizes[i + k] : kZeroChunkBytes;
    }
  };
  const int64_t i0 = base + (int64_t)tid * kScanPer;
  uint32_t v[kScanPer];
  four(i0, v);
  unsigned long long pb = 0;
  unsigned pc = 0;
#pragma unroll 8
  for (int64_t i = 4 * tid; i < base; i += 4 * kScanThreads) {
    uint32_t w[4];
    four(i, w);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      pb += w[k];
      pc += w[k] != kZeroChunkBytes;
    }
  }
  unsigned long long own = 0;  // bytes (below 2^32 for a CTA's chunks), coded chunks << 32
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) own += v[k] | (unsigned long long)(v[k] != kZeroChunkBytes) << 32;
  unsigned long long incl = own;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const unsigned long long x = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += x;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) pb += __shfl_xor_sync(0xffffffffu, pb, d);
  pc = __reduce_add_sync(0xffffffffu, pc);
  if (lane == 31) {
    warp_tot[warp] = incl;
    prior_b[warp] = pb;
    prior_c[warp] = pc;
  }
  __syncthreads();
  unsigned long long before = lane < warp ? warp_tot[lane] : 0;
  pb = prior_b[lane];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    before += __shfl_xor_sync(0xffffffffu, before, d);
    pb += __shfl_xor_sync(0xffffffffu, pb, d);
  }
  pc = __reduce_add_sync(0xffffffffu, prior_c[lane]);
  before += incl - own;
  unsigned long long off = pb + (before & 0xffffffffu);
  uint32_t rank = pc + (uint32_t)(before >> 32);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    const int64_t i = i0 + k;
    if (i < n) {
      const bool coded = v[k] != kZeroChunkBytes;
      each(i, v[k], off, rank, coded);
      rank += coded;
      off += v[k];
    }
  }
}

// One CTA more than the scan's does open() instead: what else a decode has to
// have before it starts (parameters, cleared flags).
template <class F>
__global__ void __launch_bounds__(kScanThreads)
scan_chunks_kernel(const uint16_t* __restrict__ sizes, Geometry g, ChunkTable t, F open) {
  if (blockIdx.x == gridDim.x - 1) {
    open();
    return;
  }
  scan_chunks(sizes, g.chunks, blockIdx.x, [&](int64_t i, uint32_t size, uint64_t off, uint32_t rank, bool coded) {
    t.offs[i] = (int64_t)off;
    t.rank[i] = rank;
    if (coded) {
      const ChunkLoc loc = locate_chunk(g, i);
      t.coded[rank] = pack_coded(off, size, (uint64_t)loc.base, (uint32_t)loc.osize);
    }
    if (i == g.chunks - 1) t.rank[g.chunks] = rank + coded;
  });
}

// ---------------- encode without look-back ----------------
// The pipelines encode in three launches that wait for nothing on the device:
//   encode_chunks   every chunk's size into the stream's size table and its
//                   payload into the chunk's own place in a plane-sized buffer
//                   (a coded payload is smaller than its chunk; a raw chunk
//                   and an all-zero one need none).  The pipelines own their
//                   plane buffer and encode it in place.
//   scan            the payload offsets (scan_chunks) and the stream's totals
//   gather          the payloads to their offsets in the stream
// Against the one-launch encoder above (tickets, look-back) this moves the
// container twice more through L2, but a chunk costs one barrier when it
// turns out raw, two when it is coded, three when only its last bitmaps decide
// which, no CTA waits for its predecessors,
// and chunks that the bit-plane shuffle knows to be zero are never read.  The
// one-launch encoder stays for the entry point that has no scratch to put
// payloads in.
//
// us for the one-launch encoder -> encode + scan + gather: 384x384x256 double
// at REL 1e-6 (151 MB of planes, 86 MB out) 172 -> 40 + 5 + 32 (floor 36);
// 1024^3 float sparse at ABS 1e-3 (two thirds of 262 K chunks coded) 3468 ->
// 1360 + 22 + 123; 32 uneven float fields 482 -> 85 + 6 + 40.  The encode
// launch waits on the latency of a chunk's loads and barriers; five CTAs an
// SM (48 registers) against 4 / 6 / 8: 40 / 40 / 43 / 67 us and
// 1360 / 1369 / 1422 / 2139 us on the first two.  Fetching the next chunk with
// asynchronous copies meanwhile was slower (1675-1851 us: the staging adds to
// the shared-memory traffic).
constexpr int kEncThreads = 256, kEncWarps = kEncThreads / 32, kEncCtas = 5;

struct EncodeJob {
  const uint8_t* planes;
  uint8_t* slots;   // plane-sized, may be `planes`
  uint16_t* sizes;  // the stream's size table
};

struct EncodeShared2 {
  // payload staging: nonzero bytes (< osize) plus up to 2048 + 256 + 32 + 6
  // bitmap bytes before the size check can reject the encoding
  uint4 out[(kChunk + 2048 + 512) / 16];
  uint32_t compact[16];
  uint8_t bm1[256];
  uint32_t scratch[2][kEncWarps];
  int csz;
};

// bit j = byte j of w is nonzero
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t w) {
  const uint32_t t = (((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) & 0x80808080u;  // bits 7, 15, 23, 31
  return (t * 0x00204081u) >> 28;
}

// nibble of flags -> byte-permute selector that moves the flagged bytes
// down, and 8 x their count
__device__ __forceinline__ uint32_t compact_entry(int nibble) {
  uint32_t sel = 0, kept = 0;
  for (int j = 0; j < 4; ++j)
    if ((nibble >> j) & 1) sel |= (uint32_t)j << (4 * kept++);
  for (uint32_t k = kept; k < 4; ++k) sel |= 4u << (4 * k);
  return sel | (8 * kept) << 16;
}

// The bytes of w (32, flagged by `bits`) that are kept, to out[pos ..]: few
// are stored one by one (read again through L1), otherwise whole words are
// assembled, the words shared with the neighbouring ranges byte by byte.
__device__ __forceinline__ void compact_word(EncodeShared2& sh, const uint32_t (&w)[8], const uint8_t* src, uint32_t bits,
                                             int pos, int most) {
  uint8_t* out = reinterpret_cast<uint8_t*>(sh.out);
  if (most <= 4) {
    for (uint32_t b = bits; b; b &= b - 1) out[pos++] = src[__ffs(b) - 1];
    return;
  }
  uint32_t* o32 = reinterpret_cast<uint32_t*>(sh.out);
  int at = pos >> 2, head = pos & 3, fill = 8 * head;
  uint32_t lo = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t e = sh.compact[(bits >> (4 * q)) & 15u];
    const uint32_t x = __byte_perm(w[q], 0u, e);
    const uint32_t next = fill ? x >> (32 - fill) : 0u;  // what does not fit the open word
    lo |= x << fill;
    fill += e >> 16;
    if (fill >= 32) {
      if (head) {
        for (int j = head; j < 4; ++j) out[4 * at + j] = (uint8_t)(lo >> (8 * j));
        head = 0;
      } else {
        o32[at] = lo;
      }
      ++at;
      fill -= 32;
      lo = next;
    }
  }
  for (int j = head; 8 * j < fill; ++j) out[4 * at + j] = (uint8_t)(lo >> (8 * j));
}

// Encode the chunk of `osize` bytes at `base` of the planes; returns its size
// (uniform).  parity alternates between a CTA's chunks.
__device__ __forceinline__ int encode_chunk_slot(EncodeShared2& sh, const uint8_t* planes, uint8_t* slots,
                                                 const int64_t base, const int osize, const int parity) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint8_t* src = planes + base;
  // words `first` and first + 32 of the 512-word zero-elimination bitmap, 32
  // bytes each
  const int first = 64 * warp + lane;
  uint32_t wa[8], wb[8];
  auto load = [&](uint32_t (&w)[8], int b0) {
    const uint2* p = reinterpret_cast<const uint2*>(src + b0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint2 x = make_uint2(0, 0);
      if (b0 + 8 * q < osize) x = p[q];
      w[2 * q] = x.x;
      w[2 * q + 1] = x.y;
    }
  };
  load(wa, 32 * first);
  load(wb, 32 * first + 1024);
  uint32_t before = 0;  // the bitmap byte before the warp's first
  if (lane == 0 && warp > 0 && 2048 * warp - 8 < osize) {
    const uint2 x = *reinterpret_cast<const uint2*>(src + 2048 * warp - 8);
    before = nonzero_bytes(x.x) | nonzero_bytes(x.y) << 4;
  }
  uint32_t ba = 0, bb = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    ba |= nonzero_bytes(wa[q]) << (4 * q);
    bb |= nonzero_bytes(wb[q]) << (4 * q);
  }
  // flags of the bitmap bytes that differ from their predecessors
  uint32_t prev_a = __shfl_up_sync(0xffffffffu, ba, 1) >> 24, prev_b = __shfl_up_sync(0xffffffffu, bb, 1) >> 24;
  const uint32_t last_a = __shfl_sync(0xffffffffu, ba, 31) >> 24;
  if (lane == 0) {
    prev_a = before;
    prev_b = last_a;
  }
  const uint32_t fa = nonzero_bytes(ba ^ (ba << 8 | prev_a)), fb = nonzero_bytes(bb ^ (bb << 8 | prev_b));
  const uint32_t cnt = __popc(ba) | __popc(bb) << 16, fcnt = __popc(fa) | __popc(fb) << 16;
  uint32_t incl = cnt, fincl = fcnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d), u = __shfl_up_sync(0xffffffffu, fincl, d);
    if (lane >= d) {
      incl += t;
      fincl += u;
    }
  }
  const uint32_t all = __shfl_sync(0xffffffffu, incl, 31), fall = __shfl_sync(0xffffffffu, fincl, 31);
  // (kept bitmap bytes << 16 | nonzero bytes) of the warp; the chunk's sums
  // are at most 2048 and 16384
  uint32_t* scratch = sh.scratch[parity];
  if (lane == 0) scratch[warp] = (all & 0xffffu) + (all >> 16) + (((fall & 0xffffu) + (fall >> 16)) << 16);
  __syncthreads();
  const uint32_t t = lane < kEncWarps ? scratch[lane] : 0u;
  const uint32_t total = __reduce_add_sync(0xffffffffu, t);
  const int nz = (int)(total & 0xffffu), c1 = (int)(total >> 16);
  if (nz == 0) return (int)kZeroChunkBytes;
  if (nz + c1 + 6 >= osize) return osize;
  const uint32_t pre = __reduce_add_sync(0xffffffffu, lane < warp ? t : 0u);
  // nonzero bytes, in order
  uint8_t* out = reinterpret_cast<uint8_t*>(sh.out);
  const uint32_t excl = incl - cnt;
  compact_word(sh, wa, src + 32 * first, ba, (int)(pre & 0xffffu) + (int)(excl & 0xffffu),
               (int)__reduce_max_sync(0xffffffffu, (unsigned)__popc(ba)));
  compact_word(sh, wb, src + 32 * first + 1024, bb,
               (int)(pre & 0xffffu) + (int)(all & 0xffffu) + (int)(excl >> 16),
               (int)__reduce_max_sync(0xffffffffu, (unsigned)__popc(bb)));
  // RE 2048 -> 256: the flagged bitmap bytes
  {
    const uint32_t fexcl = fincl - fcnt;
    int r = nz + (int)(pre >> 16) + (int)(fexcl & 0xffffu);
    for (uint32_t f = fa; f; f &= f - 1) out[r++] = (uint8_t)(ba >> (8 * (__ffs(f) - 1)));
    r = nz + (int)(pre >> 16) + (int)(fall & 0xffffu) + (int)(fexcl >> 16);
    for (uint32_t f = fb; f; f &= f - 1) out[r++] = (uint8_t)(bb >> (8 * (__ffs(f) - 1)));
    const uint32_t oa = __shfl_down_sync(0xffffffffu, fa, 1), ob = __shfl_down_sync(0xffffffffu, fb, 1);
    if ((lane & 1) == 0) {
      sh.bm1[first >> 1] = (uint8_t)(fa | oa << 4);
      sh.bm1[(first >> 1) + 16] = (uint8_t)(fb | ob << 4);
    }
  }
  __syncthreads();
  // The first two parts of the payload leave while warp 0 builds the rest,
  // unless the size check can still reject the encoding: the slot may be the
  // chunk itself, which then stays as it is.
  const int head = nz + c1;
  const bool certain = head + 6 + 256 + 32 < osize;
  const int lead = certain ? head & ~7 : 0;  // bytes the other warps copy
  uint2* dst = reinterpret_cast<uint2*>(slots + base);
  const uint2* o2 = reinterpret_cast<const uint2*>(sh.out);
  int csize = 0;
  if (warp == 0) {
    // RE 256 -> 32: lane l flags bm1 bytes 8l..8l+7
    const uint2 b8 = reinterpret_cast<const uint2*>(sh.bm1)[lane];
    uint32_t last = __shfl_up_sync(0xffffffffu, b8.y, 1) >> 24;
    if (lane == 0) last = 0;
    const uint32_t f2 = nonzero_bytes(b8.x ^ (b8.x << 8 | last)) |
                        nonzero_bytes(b8.y ^ (b8.y << 8 | b8.x >> 24)) << 4;
    const int cnt2 = __popc(f2);
    const int incl2 = warp_incl_scan(cnt2, lane);
    const int c2 = __shfl_sync(0xffffffffu, incl2, 31);
    int r = head + incl2 - cnt2;
    for (uint32_t f = f2; f; f &= f - 1) {
      const int k = __ffs(f) - 1;
      out[r++] = (uint8_t)((k < 4 ? b8.x : b8.y) >> (8 * (k & 3)));
    }
    // RE 32 -> 4: lane l flags bm2 byte l (= f2)
    uint32_t prev2 = __shfl_up_sync(0xffffffffu, f2, 1);
    if (lane == 0) prev2 = 0;
    const uint32_t bal = __ballot_sync(0xffffffffu, f2 != prev2);
    int pos = head + c2;
    if (f2 != prev2) out[pos + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)f2;
    pos += __popc(bal);
    csize = pos + 6;
    if (csize < osize) {
      if (lane < 4) out[pos + lane] = (uint8_t)(bal >> (8 * lane));
      if (lane == 0) {
        out[pos + 4] = (uint8_t)osize;
        out[pos + 5] = (uint8_t)(osize >> 8);
      }
    }
    __syncwarp();
    if (certain)
      for (int i = (lead >> 3) + lane; 8 * i < csize; i += 32) dst[i] = o2[i];
    else if (lane == 0) sh.csz = csize;
  } else {
    for (int i = tid - 32; 8 * i < lead; i += kEncThreads - 32) dst[i] = o2[i];
  }
  if (!certain) {
    __syncthreads();
    csize = sh.csz;
    if (csize >= osize) return osize;
    for (int i = tid; 8 * i < csize; i += kEncThreads) dst[i] = o2[i];
  }
  return csize;  // of warp 0 where `certain`
}

// The chunks of a CTA: rounds of kEncThreads chunk ids (every gridDim.x-th
// one), a thread each; the all-zero ones are done with, the others are listed
// and encoded one after the other by the CTA.  find(item) gives the job,
// geometry and chunk id of an item.
struct EncodeItem {
  EncodeJob job;
  int64_t base;
  uint32_t id;
  int osize;
};
template <class F>
__device__ __forceinline__ void encode_items(EncodeShared2& sh, EncodeItem (&list)[kEncThreads], const uint64_t items,
                                             F find) {
  __shared__ int listed;
  const int tid = threadIdx.x;
  if (tid < 16) sh.compact[tid] = compact_entry(tid);
  int parity = 0;
  for (uint64_t i0 = blockIdx.x; i0 < items; i0 += (uint64_t)gridDim.x * kEncThreads) {
    if (tid == 0) listed = 0;
    __syncthreads();  // also: the previous round's list is no longer read
    const uint64_t i = i0 + (uint64_t)tid * gridDim.x;
    if (i < items) {
      EncodeItem it;
      if (find(i, it)) list[atomicAdd(&listed, 1)] = it;
      else it.job.sizes[it.id] = (uint16_t)kZeroChunkBytes;
    }
    __syncthreads();
    const int n = listed;
    for (int k = 0; k < n; ++k) {
      const EncodeItem& it = list[k];
      const int csize = encode_chunk_slot(sh, it.job.planes, it.job.slots, it.base, it.osize, parity);
      if (tid == 0) it.job.sizes[it.id] = (uint16_t)csize;
      parity ^= 1;
    }
    __syncthreads();
  }
}

constexpr int encode_smem_bytes() { return (int)(sizeof(EncodeShared2) + kEncThreads * sizeof(EncodeItem)); }

// Offsets and totals of an encoded stream: payload offset per chunk, the
// cumulative plane sizes, the header, the zero padding.
struct StreamTotals {
  uint64_t* comp_size_bp;
  uint64_t* lossless_size;
  uint64_t* padded_size;
  int* error_flag;
};
__device__ __forceinline__ void scan_stream(uint8_t* stream, const Geometry& g, int64_t* offs, const StreamTotals& t,
                                            int cta) {
  const int64_t n = g.chunks;
  scan_chunks(reinterpret_cast<const uint16_t*>(stream + 8), n, cta,
              [&](int64_t i, uint32_t size, uint64_t off, uint32_t, bool) {
    offs[i] = (int64_t)off;
    const ChunkLoc loc = locate_chunk(g, i);
    if (loc.last_of_plane) t.comp_size_bp[(3 - loc.level) * 32 + loc.plane] = off + size;
    if (i == n - 1) {
      const uint64_t total = 8 + 2 * (uint64_t)n + off + size, pad = (8 - total % 8) % 8;
      for (uint64_t k = 0; k < pad; ++k) stream[total + k] = 0;
      for (int k = 0; k < 8; ++k) stream[k] = (uint8_t)((uint64_t)g.aligned_size >> (8 * k));
      *t.lossless_size = off + size;
      *t.padded_size = total + pad;
      *t.error_flag = 0;
    }
  });
}
// publish(): the call's results for the host, by the last CTA once its totals
// are written
template <class F>
__global__ void __launch_bounds__(kScanThreads)
scan_stream_kernel(uint8_t* stream, Geometry g, int64_t* offs, StreamTotals t, F publish) {
  chain_wait();
  scan_stream(stream, g, offs, t, blockIdx.x);
  if (blockIdx.x == gridDim.x - 1) {
    __syncthreads();
    publish();
  }
}

// LANES threads (a warp or the CTA) copy n bytes from an 8-byte aligned address
// to an arbitrarily aligned one: head bytes, then aligned 32-bit words (each
// from two source words, loaded once: the second is the next lane's), four in
// flight, then the tail.
template <int LANES>
__device__ __forceinline__ void gather_copy(uint8_t* dst, const uint8_t* src, int n) {
  const int tid = LANES == 32 ? threadIdx.x & 31 : threadIdx.x, lane = threadIdx.x & 31;
  int head = (int)((4 - ((uintptr_t)dst & 3)) & 3);
  if (head > n) head = n;
  const int words = (n - head) >> 2, have = (n + 3) >> 2;  // whole words out, source words
  if (tid < head) dst[tid] = src[tid];
  uint32_t* dw = reinterpret_cast<uint32_t*>(dst + head);
  const uint32_t* sw = reinterpret_cast<const uint32_t*>(src);
#pragma unroll 1
  for (int w0 = tid; w0 - lane < words; w0 += 4 * LANES) {  // warp-uniform trips
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int w = w0 + k * LANES;
      lo[k] = w < have ? sw[w] : 0u;
      hi[k] = (lane == 31 && w + 1 < have) ? sw[w + 1] : 0u;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int w = w0 + k * LANES;
      const uint32_t next = __shfl_down_sync(0xffffffffu, lo[k], 1);
      if (lane != 31) hi[k] = next;
      if (w < words) dw[w] = __funnelshift_r(lo[k], hi[k], 8 * head);
    }
  }
  const int done = head + 4 * words;
  if (tid < n - done) dst[done + tid] = src[done + tid];
}

// Payloads to their places in the stream, in rounds as encode_items: a warp
// takes a payload of up to kWarpPayload bytes (a sparse chunk's is a few
// hundred: 1024^3 floats at ABS 1e-3 took 332 us with the CTA copying them one
// after the other, 123 us now; 384x384x256 doubles 36 -> 32 us), the CTA
// together a larger one, or the one it has on a small field (a warp alone is
// 2-4 us slower on one payload).  The launch's time at limits of 0 / 1 / 2 / 4 /
// 8 / 16 KB (under a profiler, the wait for the scan included): 443 / 276 / 255
// / 241 / 239 / 238 us on the first, 50 / 45 / 47 / 47 / 49 / 48 on the second,
// 47 / 46 / 46 / 47 / 49 / 67 on 32 uneven float fields.
constexpr int kWarpPayload = 4096;
struct GatherItem {
  const uint8_t* src;
  uint8_t* dst;
  int n;
};
template <class F>
__device__ __forceinline__ void gather_items(GatherItem (&list)[kEncThreads], const uint64_t items, const int cta,
                                             const int ncta, F find) {
  __shared__ int listed[2];  // short payloads from the front of the list, the others from its end
  const int tid = threadIdx.x;
  const int short_max = items <= (uint64_t)ncta ? 0 : kWarpPayload;  // one payload a CTA: by the CTA
  for (uint64_t i0 = cta; i0 < items; i0 += (uint64_t)ncta * kEncThreads) {
    if (tid < 2) listed[tid] = 0;
    __syncthreads();
    const uint64_t i = i0 + (uint64_t)tid * ncta;
    if (i < items) {
      GatherItem it;
      if (find(i, it)) {
        if (it.n <= short_max) list[atomicAdd(&listed[0], 1)] = it;
        else list[kEncThreads - 1 - atomicAdd(&listed[1], 1)] = it;
      }
    }
    __syncthreads();
    for (int k = tid >> 5; k < listed[0]; k += kEncWarps) gather_copy<32>(list[k].dst, list[k].src, list[k].n);
    for (int k = 0; k < listed[1]; ++k) {
      const GatherItem& it = list[kEncThreads - 1 - k];
      gather_copy<kEncThreads>(it.dst, it.src, it.n);
    }
    __syncthreads();
  }
}
// Item of chunk `id`; an all-zero chunk's two bytes are written here.
__device__ __forceinline__ bool gather_chunk(const EncodeJob& job, const Geometry& g, uint8_t* stream,
                                             const int64_t* offs, int64_t id, GatherItem& it) {
  const ChunkLoc loc = locate_chunk(g, id);
  it.n = job.sizes[id];
  it.dst = stream + 8 + 2 * g.chunks + offs[id];
  if (it.n == (int)kZeroChunkBytes) {
    it.dst[0] = (uint8_t)loc.osize;
    it.dst[1] = (uint8_t)(loc.osize >> 8);
    return false;
  }
  it.src = (it.n == loc.osize ? job.planes : job.slots) + loc.base;
  return true;
}
// The first `front` CTAs do front(cta) instead (the trailer).
template <class F>
__global__ void __launch_bounds__(kEncThreads)
gather_stream_kernel(const EncodeJob job, Geometry g, uint8_t* stream, const int64_t* offs, int front_ctas,
                     F front) {
  chain_wait();
  __shared__ GatherItem list[kEncThreads];
  if ((int)blockIdx.x < front_ctas) {
    front();
    return;
  }
  gather_items(list, (uint64_t)g.chunks, blockIdx.x - front_ctas, gridDim.x - front_ctas, [&](uint64_t i, GatherItem& it) {
    return gather_chunk(job, g, stream, offs, (int64_t)i, it);
  });
}

constexpr int kDecThreads = 256, kDecWarps = kDecThreads / 32;
constexpr int kDecCtas = 6;  // per SM

struct DecodeShared {
  uint8_t in[kChunk + 32];
  uint4 out[kDecWarps][64];  // 1024 decoded bytes of each warp, on their way to coalesced stores
  uint32_t expand[16];
  uint8_t bm1[256];
  int scan1[kDecWarps], scan2[kDecWarps];
  int p2, flag;
};

// Copy n <= kChunk bytes from an arbitrarily aligned global address to `dst`
// (shared memory, or global memory for a raw chunk) with aligned 32-bit
// loads; no byte past src + n - 1's word is read.  Four words a thread are in
// flight.  Each source word is loaded once: the word after w is the next
// lane's (lane 31 loads it itself).  Whole words are written (n is a multiple
// of 4 for raw chunks; the staging buffer has slack).
__device__ __forceinline__ void copy_words(uint32_t* dw, const uint8_t* src, int n) {
  const int shift = (int)((uintptr_t)src & 3);
  const uint32_t* a = reinterpret_cast<const uint32_t*>(src - shift);
  const int last = (shift + n - 1) >> 2;  // last source word needed
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int w0 = threadIdx.x; 4 * (w0 - lane) < n; w0 += 4 * kDecThreads) {  // warp-uniform trips
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int w = w0 + k * kDecThreads;
      lo[k] = w <= last ? __ldg(a + w) : 0u;
      hi[k] = (lane == 31 && w + 1 <= last) ? __ldg(a + w + 1) : 0u;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int w = w0 + k * kDecThreads;
      const uint32_t next = __shfl_down_sync(0xffffffffu, lo[k], 1);
      if (lane != 31) hi[k] = next;
      if (4 * w < n) dw[w] = __funnelshift_r(lo[k], hi[k], 8 * shift);
    }
  }
}

// Exclusive prefix of two counts below 2^16 packed in `v`, one word of 32
// bitmap bits each: the thread's word of the warp's first 32 words (low half)
// and of its second 32 (high half); a warp's 64 words follow the previous
// warp's.  One barrier; `scratch` must not be in use since the last one.
struct TwoRanks {
  int first, second, total;
};
__device__ __forceinline__ TwoRanks block_two_ranks(uint32_t v, int* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += t;
  }
  const uint32_t all = __shfl_sync(0xffffffffu, incl, 31);
  const int tf = (int)(all & 0xffffu), ts = (int)(all >> 16);
  if (lane == 0) scratch[warp] = tf + ts;
  __syncthreads();
  const int t = lane < kDecWarps ? scratch[lane] : 0;
  const int before = (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane < warp ? t : 0));
  TwoRanks r;
  r.total = (int)__reduce_add_sync(0xffffffffu, (unsigned)t);
  const uint32_t excl = incl - v;
  r.first = before + (int)(excl & 0xffffu);
  r.second = before + tf + (int)(excl >> 16);
  return r;
}

// The 32 plane bytes whose nonzero flags are `bits`, the kept ones from
// in[rank] on, into this lane's part of the warp's staging (16-byte pieces
// swizzled so that eight lanes touch eight bank groups).  Few bytes are
// stored one by one; otherwise four bytes at a time, the next kept bytes
// placed by one byte permute whose selector comes from a 16-entry table.
__device__ __forceinline__ int stage_piece(int p) { return p ^ ((p >> 3) & 1); }
__device__ __forceinline__ void expand_word(const DecodeShared& sh, uint4* stage, uint32_t bits, int rank, int most) {
  const int lane = threadIdx.x & 31;
  uint4 &p0 = stage[stage_piece(2 * lane)], &p1 = stage[stage_piece(2 * lane + 1)];
  if (most <= 4) {
    p0 = p1 = make_uint4(0, 0, 0, 0);
    uint8_t* o = reinterpret_cast<uint8_t*>(stage);
    for (uint32_t b = bits; b; b &= b - 1) {
      const int j = __ffs(b) - 1;
      o[16 * stage_piece(2 * lane + (j >> 4)) + (j & 15)] = sh.in[rank++];
    }
    return;
  }
  const uint32_t* in32 = reinterpret_cast<const uint32_t*>(sh.in);
  int at = rank >> 2, shift = (rank & 3) * 8;
  uint32_t lo = in32[at], hi = in32[at + 1], w[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const uint32_t e = sh.expand[(bits >> (4 * q)) & 15u];
    w[q] = __byte_perm(__funnelshift_r(lo, hi, shift), 0u, e);
    shift += e >> 16;
    if (shift >= 32) {  // at most one word per four kept bytes
      shift -= 32;
      lo = hi;
      hi = in32[++at + 1];
    }
  }
  p0 = make_uint4(w[0], w[1], w[2], w[3]);
  p1 = make_uint4(w[4], w[5], w[6], w[7]);
}

// Which chunks a decode leaves as zeros: the all-zero ones and, when
// begin/end select planes, those outside [begin, end) of their level.  sizes
// == null: every chunk holds bytes (a plane buffer that was not decoded here).
struct ChunkLive {
  const uint16_t* sizes;
  const int* begin;
  const int* end;
  __device__ __forceinline__ bool dead(const HostChunk& c) const {
    if (!sizes) return false;
    const bool zero = __ldg(sizes + c.id) == kZeroChunkBytes;
    return zero || (begin && (c.plane < begin[3 - c.level] || c.plane >= end[3 - c.level]));
  }
};

// Bytes at either end of a dead chunk that the decoder still writes as zeros
// when its reader skips dead chunks: an inverse-shuffle item reads up to this
// many consecutive bytes of a plane and skips them only when one dead chunk
// holds them all.
constexpr int kDeadEdge = 128;

// Decode the chunks of a stream into the plane buffer.  begin/end (device, may
// be null) select the chunks of host planes [begin[3-l], end[3-l]) like
// zbpc_decode_progressive (zbpc.cu:420-423).  Two passes over one grid:
//
// 1. Dead chunks (all-zero or not selected) that the inverse shuffle reaches:
//    per level one range of chunk ids, the selected planes' chunks and those
//    holding the bytes the inverse reads for these planes at their device
//    placement.  A reader that skips dead chunks (ChunkLive) needs zeros only
//    within kDeadEdge bytes of their ends (EDGES); otherwise all-zero chunks
//    are written whole and unselected ones where the inverse reads them.  At
//    common bounds most chunks are all-zero (the leading planes of small
//    codes), and not moving their 16 KB here and in the inverse shuffle is
//    most of what this pass saves.
// 2. The selected coded chunks, from the table, one CTA of 256 threads each.
//    The payload is decoded from its tail: bitmap 4 B -> 32 B -> 256 B ->
//    2048 B (fill-forward: byte i = kept byte rank(i) - 1, rank the inclusive
//    flag count), then every thread expands two words of 32 zero-elimination
//    flags (expand_word); the bytes leave through shared memory in coalesced
//    stores.
//
// What bounds pass 2 is instruction issue and the chain of barriers, not
// memory: on a 1000x777x513 float field at ABS 1e-3 (98 K chunks, two thirds
// of them coded and sparse) 449 us against 1248 us for one pass of 512-thread
// CTAs over every chunk, 32 predicated byte loads a thread and six barriers
// more a chunk; on 128^3 floats at REL 1e-4 8.0 against 11.0 us.
//
// Corrupt chunks raise error_flag = 2.
template <bool EDGES>
__global__ void __launch_bounds__(kDecThreads, kDecCtas)
zbpc_decode_kernel(const uint8_t* __restrict__ stream, uint64_t stream_bytes, const ChunkTable table, Geometry g,
                   uint8_t* __restrict__ planes, const int* __restrict__ begin, const int* __restrict__ end,
                   int* __restrict__ error_flag) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DecodeShared& sh = *reinterpret_cast<DecodeShared*>(smem_raw);
  __shared__ int64_t range_start[4], range_len[4];
  __shared__ uint32_t coded_start[4], coded_len[4];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t chunks = g.chunks;
  const uint16_t* sizes = reinterpret_cast<const uint16_t*>(stream + 8);
  const uint8_t* data_in = stream + 8 + 2 * chunks;
  if (tid < 4) {
    const int l = tid;
    int64_t s = 0, e = 0, cs = 0, ce = 0;  // ids to visit; ids of the selected planes' chunks
    if (!begin) {
      ce = e = l == 0 ? chunks : 0;  // a full decode: every chunk, once
    } else if (begin[3 - l] < end[3 - l]) {
      const int lo = begin[3 - l], hi = end[3 - l];
      int64_t cb = 0;
      for (int i = 3; i > l; --i) cb += g.chunks_level[i];
      const int64_t cpp = g.chunks_level[l] >> 5;
      s = cb + lo * cpp;
      e = cb + hi * cpp;
      // a range may name planes past the level's 32 (or below 0): no other
      // level's chunks are selected by them
      cs = cb + (lo < 0 ? 0 : (lo > 32 ? 32 : lo)) * cpp;
      ce = cb + (hi < 0 ? 0 : (hi > 32 ? 32 : hi)) * cpp;
      const int64_t a = g.daprefix[l] + (int64_t)lo * g.dstride[l], b = g.daprefix[l] + (int64_t)hi * g.dstride[l];
      const int64_t lim = (int64_t)g.aligned_size;
      if (a < b && a < lim) {
        const int64_t f = chunk_of_byte(g, a), t = chunk_of_byte(g, (b < lim ? b : lim) - 1) + 1;
        s = f < s ? f : s;
        e = t > e ? t : e;
      }
      s = s < 0 ? 0 : (s > chunks ? chunks : s);
      e = e < s ? s : (e > chunks ? chunks : e);
    }
    range_start[l] = s;
    range_len[l] = e - s;
    coded_start[l] = table.rank[cs];
    coded_len[l] = table.rank[ce] - table.rank[cs];
  }
  if (tid < 16) {  // nibble of flags -> byte-permute selector (4 = a zero byte) and 8 x kept bytes
    uint32_t sel = 0, kept = 0;
    for (int j = 0; j < 4; ++j) {
      sel |= (((tid >> j) & 1) ? kept : 4u) << (4 * j);
      kept += (tid >> j) & 1;
    }
    sh.expand[tid] = sel | (8 * kept) << 16;
  }
  __syncthreads();

  // ---- dead chunks: a lane classifies one, the warp writes the zeros ----
  const int64_t visits = range_len[0] + range_len[1] + range_len[2] + range_len[3];
  const int64_t warps = (int64_t)gridDim.x * kDecWarps;
  for (int64_t v0 = ((int64_t)blockIdx.x * kDecWarps + warp) * 32; v0 < visits; v0 += warps * 32) {
    const int64_t v = v0 + lane;
    int64_t id = v;
    bool zero = false, unselected = false;
    int64_t cb = 0, ce = 0;
    if (v < visits) {
      int r = 0;
      while (r < 3 && id >= range_len[r]) id -= range_len[r++];
      id += range_start[r];
      const ChunkLoc loc = locate_chunk(g, id);
      cb = loc.base;
      ce = cb + loc.osize;
      if (begin) unselected = loc.plane < begin[3 - loc.level] || loc.plane >= end[3 - loc.level];
      if (!unselected && sizes[id] == kZeroChunkBytes) {
        const uint64_t at = (uint64_t)(8 + 2 * chunks + table.offs[id]);
        const uint8_t* src = data_in + table.offs[id];
        if (at + kZeroChunkBytes > stream_bytes || (src[0] | (src[1] << 8)) != loc.osize) atomicExch(error_flag, 2);
        else zero = true;
      }
    }
    for (unsigned todo = __ballot_sync(0xffffffffu, zero || unselected); todo; todo &= todo - 1) {
      const int from = __ffs(todo) - 1;
      const int64_t b = __shfl_sync(0xffffffffu, cb, from), e = __shfl_sync(0xffffffffu, ce, from);
      const bool all = __shfl_sync(0xffffffffu, (int)zero, from) != 0;
      auto clear = [&](int64_t a, int64_t z) {  // [a, z), multiples of 8
        for (int64_t o = a + 8 * lane; o < z; o += 8 * 32) *reinterpret_cast<uint2*>(planes + o) = make_uint2(0, 0);
      };
      if constexpr (EDGES) {
        // kDeadEdge bytes at each end: 16 lanes of 8 bytes each
        const int64_t o = lane < 16 ? b + 8 * lane : e - kDeadEdge + 8 * (lane - 16);
        if (o >= b && o < e) *reinterpret_cast<uint2*>(planes + o) = make_uint2(0, 0);
        static_assert(kDeadEdge == 16 * 8, "one 8-byte store per lane");
      } else if (all) {
        clear(b, e);
      } else {
        // the inverse reads, per level l, the planes [lo, hi) it selects at
        // their device placement, bytes [daprefix[l] + lo dstride[l],
        // daprefix[l] + hi dstride[l]) (multiples of 8); the rest of this
        // chunk is never read
#pragma unroll 1
        for (int l = 0; l < 4; ++l) {
          const int lo = begin[3 - l], hi = end[3 - l];
          if (lo >= hi) continue;
          const int64_t r0 = g.daprefix[l] + (int64_t)lo * g.dstride[l], r1 = g.daprefix[l] + (int64_t)hi * g.dstride[l];
          clear(b > r0 ? b : r0, e < r1 ? e : r1);
        }
      }
    }
  }

  // ---- coded chunks ----
  const uint32_t coded = coded_len[0] + coded_len[1] + coded_len[2] + coded_len[3];
  auto entry = [&](uint32_t v) {
    int r = 0;
    while (r < 3 && v >= coded_len[r]) v -= coded_len[r++];
    return table.coded[coded_start[r] + v];
  };
  ulonglong2 next = make_ulonglong2(0, 0);
  if (blockIdx.x < coded) next = entry(blockIdx.x);
  for (uint32_t v = blockIdx.x; v < coded; v += gridDim.x) {
    const uint64_t off = next.x & kCodedMask;
    const int csize = (int)(next.x >> 48), osize = (int)(next.y >> 48);
    uint8_t* dst = planes + (next.y & kCodedMask);
    if (v + gridDim.x < coded) next = entry(v + gridDim.x);  // arrives meanwhile
    if (csize > osize || (uint64_t)(8 + 2 * chunks) + off + (uint64_t)csize > stream_bytes) {  // corrupt size table
      if (tid == 0) atomicExch(error_flag, 2);
      continue;
    }
    const uint8_t* src = data_in + off;
    if (csize == osize) {  // raw chunk (osize is a multiple of 8)
      copy_words(reinterpret_cast<uint32_t*>(dst), src, osize);
      continue;
    }
    __syncthreads();  // the previous chunk's payload is no longer read
    copy_words(reinterpret_cast<uint32_t*>(sh.in), src, csize);
    if (tid == 0) sh.flag = 0;
    __syncthreads();
    if (csize < 6 || (sh.in[csize - 2] | (sh.in[csize - 1] << 8)) != osize) {
      if (tid == 0) atomicExch(error_flag, 2);
      continue;
    }
    // ---- warp 0: bm3 (4 B) -> bm2 (32 B) -> bm1 (256 B) ----
    const int rpos = csize - 6;  // start of bm3
    if (warp == 0) {
      const uint32_t bm3 = (uint32_t)sh.in[rpos] | ((uint32_t)sh.in[rpos + 1] << 8) |
                           ((uint32_t)sh.in[rpos + 2] << 16) | ((uint32_t)sh.in[rpos + 3] << 24);
      const int c3 = __popc(bm3);
      const int p3 = rpos - c3;  // RE3 bytes
      // bm2 byte l = kept byte (inclusive rank of flag l) - 1, or 0
      const int rank3 = __popc(bm3 & (0xffffffffu >> (31 - lane)));
      uint32_t b2 = 0;
      if (p3 >= 0 && rank3 > 0) b2 = sh.in[p3 + rank3 - 1];
      // bm2 flags 256 bits: lane l owns flags 8l..8l+7 = byte b2 of lane l
      const int cnt2 = __popc(b2);
      const int incl2 = warp_incl_scan(cnt2, lane);
      const int c2 = __shfl_sync(0xffffffffu, incl2, 31);
      const int p2 = p3 - c2;  // RE2 bytes
      int r = incl2 - cnt2;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        r += (b2 >> k) & 1u;
        sh.bm1[8 * lane + k] = (p2 >= 0 && r > 0) ? sh.in[p2 + r - 1] : 0;
      }
      if (lane == 0) {
        sh.p2 = p2;
        if (p3 < 0 || p2 < 0) sh.flag = 1;
      }
    }
    __syncthreads();
    if (sh.flag) {
      if (tid == 0) atomicExch(error_flag, 2);
      continue;
    }
    // ---- all threads: bm1 (2048 flags) -> the words first and first + 32 of
    // the 512-word bitmap, four flags (bitmap bytes) each ----
    const int first = 64 * warp + lane;
    const uint32_t fa = (sh.bm1[first >> 1] >> (4 * (first & 1))) & 0xFu;
    const uint32_t fb = (sh.bm1[(first >> 1) + 16] >> (4 * (first & 1))) & 0xFu;
    const TwoRanks r1 = block_two_ranks(__popc(fa) | __popc(fb) << 16, sh.scan1);
    const int p1 = sh.p2 - r1.total;  // RE1 bytes
    if (p1 < 0) {
      if (tid == 0) atomicExch(error_flag, 2);
      continue;
    }
    // fill-forward: byte i = RE1 byte (rank(i) - 1), rank inclusive; rank 0 -> 0
    auto word_of = [&](uint32_t f, int r) {
      uint32_t b = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        r += (f >> k) & 1u;
        b |= (uint32_t)(r > 0 ? sh.in[p1 + r - 1] : 0) << (8 * k);
      }
      return b;
    };
    const uint32_t ba = word_of(fa, r1.first), bb = word_of(fb, r1.second);
    const TwoRanks nz = block_two_ranks(__popc(ba) | __popc(bb) << 16, sh.scan2);
    if (nz.total > p1) {
      if (tid == 0) atomicExch(error_flag, 2);
      continue;
    }
    uint4* stage = sh.out[warp];
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const uint32_t bits = half ? bb : ba;
      const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)__popc(bits));
      const int b0 = 2048 * warp + 1024 * half;  // the warp's bytes of this half
      if (b0 >= osize) break;
      uint2* d2 = reinterpret_cast<uint2*>(dst + b0);
      if (most > 0) {
        expand_word(sh, stage, bits, half ? nz.second : nz.first, most);
        __syncwarp();
      }
      const uint2* o2 = reinterpret_cast<const uint2*>(stage);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = 32 * q + lane;
        const uint2 x = most > 0 ? o2[2 * stage_piece(i >> 1) + (i & 1)] : make_uint2(0, 0);
        if (b0 + 8 * i < osize) d2[i] = x;
      }
      __syncwarp();
    }
  }
}

}  // namespace prism_b200
