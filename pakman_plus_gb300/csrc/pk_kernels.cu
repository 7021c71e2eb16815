// sm_103a kernels for PaKman's k-mer counting -> histogram cutoff -> macro-node path.
//
// Pipeline for one read set (FASTA bytes resident in HBM):
//   k_line_scan        newline count per 64 KB tile, first '>' and '>' count
//   k_tile_prefix      exclusive newline prefix over tiles, newlines before the first '>'
//   k_extract          per chunk: roll every k-mer window, histogram of bucket ids (smem)
//   k_col_prefix       per bucket: prefix over chunks; k_bucket_prefix: bucket starts;
//   k_coarse_offsets   each chunk's segment of every coarse region
//   k_scatter_coarse   roll again, keys to their coarse region through shared-memory rings
//   k_scatter_fine     per slice of a coarse region: keys to their bucket, staged by bucket
//   k_giant_chunks     chunk and part items of buckets too large for one CTA
//   k_bucket_table     per bucket: hash-aggregate in smem, sort the distinct keys, write
//                      the (k-mer, count) rows and the count histogram
//   k_cutoff           first minimum of the count histogram over [1, t)
//   k_kept_offsets     kept rows (count >= cutoff) per bucket and their prefix over the buckets
//   k_filter_kept      the kept rows, dense
//   k_macro_nodes      per (k-1)-mer unit: merge the suffix-side and prefix-side
//                      streams of kept k-mers into macro-node records
//   k_wire             initial wiring of every macro-node
//
// A bucket is the leading `bbits` bits of the 2k-bit key, so buckets in index order
// are the table in key order and no global merge is needed.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

#include "pk_internal.h"
#include "pk_wire.cuh"

namespace pk {

typedef unsigned __int128 u128;

#define FULLMASK 0xffffffffu

// ----------------------------------------------------------------- key helpers ----
template <typename K>
struct KeyOps;

template <>
struct KeyOps<uint64_t> {
  static constexpr int W = 8;
  __device__ __forceinline__ static uint64_t mask(int bits) {
    return bits >= 64 ? ~0ull : ((1ull << bits) - 1ull);
  }
  __device__ __forceinline__ static uint64_t shr(uint64_t x, int s) { return s >= 64 ? 0ull : x >> s; }
  __device__ __forceinline__ static uint64_t shl(uint64_t x, int s) { return s >= 64 ? 0ull : x << s; }
  __device__ __forceinline__ static uint32_t low32(uint64_t x) { return (uint32_t)x; }
  __device__ __forceinline__ static uint64_t hash(uint64_t x) { return x * 0x9E3779B97F4A7C15ull; }
  __device__ __forceinline__ static unsigned match(unsigned m, uint64_t x) {
    return __match_any_sync(m, (unsigned long long)x);
  }
  __device__ __forceinline__ static int top_bit(uint64_t x) { return 63 - __clzll((long long)x); }
  __device__ __forceinline__ static uint64_t cas(uint64_t* p, uint64_t cmp, uint64_t val) {
    return atomicCAS(reinterpret_cast<unsigned long long*>(p), (unsigned long long)cmp,
                     (unsigned long long)val);
  }
};

template <>
struct KeyOps<u128> {
  static constexpr int W = 16;
  __device__ __forceinline__ static u128 mask(int bits) {
    return bits >= 128 ? ~(u128)0 : (((u128)1 << bits) - 1);
  }
  __device__ __forceinline__ static u128 shr(u128 x, int s) { return s >= 128 ? (u128)0 : x >> s; }
  __device__ __forceinline__ static u128 shl(u128 x, int s) { return s >= 128 ? (u128)0 : x << s; }
  __device__ __forceinline__ static uint32_t low32(u128 x) { return (uint32_t)(uint64_t)x; }
  __device__ __forceinline__ static uint64_t hash(u128 x) {
    uint64_t lo = (uint64_t)x, hi = (uint64_t)(x >> 64);
    return (lo ^ (hi * 0xC2B2AE3D27D4EB4Full)) * 0x9E3779B97F4A7C15ull;
  }
  __device__ __forceinline__ static unsigned match(unsigned m, u128 x) {
    return __match_any_sync(m, (unsigned long long)x) &
           __match_any_sync(m, (unsigned long long)(x >> 64));
  }
  __device__ __forceinline__ static int top_bit(u128 x) {
    const uint64_t hi = (uint64_t)(x >> 64);
    return hi ? 127 - __clzll((long long)hi) : 63 - __clzll((long long)(uint64_t)x);
  }
  // p in shared memory (named as such: the compiler need not infer it for a 128-bit atomic)
  __device__ __forceinline__ static u128 cas(u128* p, u128 cmp, u128 val) {
    uint64_t lo, hi;
    asm volatile(
        "{\n\t.reg .b128 c, v, o;\n\tmov.b128 c, {%3, %4};\n\tmov.b128 v, {%5, %6};\n\t"
        "atom.shared.cas.b128 o, [%2], c, v;\n\tmov.b128 {%0, %1}, o;\n\t}"
        : "=l"(lo), "=l"(hi)
        : "r"((uint32_t)__cvta_generic_to_shared(p)), "l"((uint64_t)cmp), "l"((uint64_t)(cmp >> 64)),
          "l"((uint64_t)val), "l"((uint64_t)(val >> 64))
        : "memory");
    return ((u128)hi << 64) | lo;
  }
};

// A key loaded through L2 only (data another CTA of the same kernel wrote).
__device__ __forceinline__ uint64_t ldcg_key(const uint64_t* p) {
  return (uint64_t)__ldcg(reinterpret_cast<const unsigned long long*>(p));
}
__device__ __forceinline__ u128 ldcg_key(const u128* p) {
  const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p));
  return ((u128)v.y << 64) | v.x;
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned r;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(r));
  return r;
}

// Look-back words carry all their data themselves: relaxed accesses, coherent in the device.
__device__ __forceinline__ unsigned long long ld_relaxed(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_relaxed(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}


// Decoupled look-back words: status in bits 62-63 (1 = aggregate, 2 = inclusive).
constexpr unsigned long long kLbAgg = 1ull << 62;
constexpr unsigned long long kLbIncl = 2ull << 62;
constexpr unsigned long long kLbVal = (1ull << 62) - 1;
constexpr int kLbSpinLimit = 1 << 24;  // ~1-2 s with the back-off below (the default)
__device__ __forceinline__ int spin_limit(int limit) { return limit > 0 ? limit : kLbSpinLimit; }

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULLMASK, v, o);
  return v;
}

// Waits a little before a look-back word is read again; false when the wait has run out
// (the error bit is set).
__device__ __forceinline__ bool lookback_wait(int& spins, int max_spins, uint32_t* err) {
  if (++spins >= max_spins) {
    if ((threadIdx.x & 31) == 0) atomicOr(err, ERR_LOOKBACK);
    return false;
  }
  __nanosleep(spins < 64 ? 32 : 256);
  return true;
}

// Sum over the words before `idx` of a look-back sequence, by a whole warp (all 32 lanes
// call it and all get the sum).  read(j, value) gives word j's state: 0 unpublished, 1 an
// aggregate, 2 an inclusive prefix.  Each step reads the 32 nearest unread predecessors
// (lane 0 = nearest): it stops at the nearest inclusive word, otherwise adds the aggregates
// up to the first word still unpublished and moves past them.  Waiting is bounded: on
// expiry the partial sum is returned.
template <typename Read>
__device__ __forceinline__ unsigned long long lookback_exclusive(int idx, uint32_t* err, int limit, Read&& read) {
  const int max_spins = spin_limit(limit);
  const int lane = threadIdx.x & 31;
  unsigned long long sum = 0;
  int top = idx - 1;  // nearest predecessor not yet added
  int spins = 0;
  while (top >= 0) {
    const int j = top - lane;
    unsigned long long v = 0;
    const unsigned st = j >= 0 ? read(j, v) : 2u;  // below 0: inclusive 0
    const unsigned waiting = __ballot_sync(FULLMASK, st == 0);
    const unsigned incl = __ballot_sync(FULLMASK, st == 2);
    const int first_wait = waiting ? __ffs(waiting) - 1 : 32;
    const int first_incl = incl ? __ffs(incl) - 1 : 32;
    if (first_incl < first_wait) return sum + warp_sum_u64(lane <= first_incl ? v : 0ull);
    if (first_wait > 0) {
      sum += warp_sum_u64(lane < first_wait ? v : 0ull);
      top -= first_wait;
      spins = 0;
      continue;
    }
    if (!lookback_wait(spins, max_spins, err)) return sum;
  }
  return sum;
}

// Look-back in two levels, for sequences with hundreds of units in flight: a unit publishes
// its value in its own word and adds it to its group of 32; it reads the words before it in
// its group, and looks back over groups (complete ones count as aggregates; the group's
// last unit publishes the inclusive prefix).  Looking back over single units, every unit
// read hundreds of words that all the others were reading too.  (Eight words a lane and
// step instead of one made that worse, 0.37 to 0.91 ms for 8.6M nodes: the reads of the
// same lines are the cost, not their number in a row.)  The words: unit (units), then per
// group the sum (count of published units in bits 48 up) and the inclusive prefix; all zero
// beforehand.
struct GroupFlags {
  unsigned long long *unit, *sum, *incl;
  __device__ GroupFlags(unsigned long long* words, uint32_t units)
      : unit(words), sum(words + units), incl(sum + (units + 31) / 32) {}
};

__device__ __forceinline__ void group_publish(const GroupFlags& w, uint32_t u, unsigned long long mine) {
  st_relaxed(&w.unit[u], kLbAgg | mine);
  atomicAdd(&w.sum[u >> 5], (1ull << 48) | mine);
}

// The sum before unit u.  Its own value is published first, or waited for where another CTA
// publishes it (`mine` = ~0); `publish` false keeps it from the successors (fault injection).
__device__ unsigned long long group_lookback(const GroupFlags& w, uint32_t u, unsigned long long mine,
                                             bool publish, uint32_t* err, int limit) {
  const int lane = threadIdx.x & 31, max_spins = spin_limit(limit);
  const uint32_t g = u >> 5, i = u & 31;
  const bool own = mine != ~0ull;
  if (lane == 0 && publish && own) group_publish(w, u, mine);
  __syncwarp();
  unsigned long long f = 0;
  int spins = 0;
  while (true) {
    const bool wanted = (uint32_t)lane < i || ((uint32_t)lane == i && !own);
    f = wanted ? ld_relaxed(&w.unit[32 * g + lane]) : kLbAgg;
    if (__all_sync(FULLMASK, f != 0)) break;
    if (!lookback_wait(spins, max_spins, err)) return 0;
  }
  if (!own) mine = __shfl_sync(FULLMASK, f, i) & kLbVal;
  const unsigned long long before = warp_sum_u64((uint32_t)lane < i ? f & kLbVal : 0ull);
  const unsigned long long ex = before + lookback_exclusive((int)g, err, limit, [&](int j, unsigned long long& v) {
    const unsigned long long p = ld_relaxed(&w.incl[j]), s = ld_relaxed(&w.sum[j]);
    const bool inclusive = (p >> 62) == 2;
    v = inclusive ? p & kLbVal : s & ((1ull << 48) - 1);
    return inclusive ? 2u : (s >> 48) == 32 ? 1u : 0u;
  });
  if (lane == 0 && publish && i == 31) st_relaxed(&w.incl[g], kLbIncl | (ex + mine));
  return ex;
}

// Block-wide exclusive sum over `nthreads` (multiple of 32, <= 1024) threads.
__device__ __forceinline__ uint32_t block_exclusive_sum(uint32_t v, uint32_t* s_warp, uint32_t& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(FULLMASK, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < nw ? s_warp[lane] : 0;
    uint32_t ws = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(FULLMASK, ws, o);
      if (lane >= o) ws += y;
    }
    if (lane < nw) s_warp[lane] = ws - w;
    if (lane == 31) s_warp[32] = ws;
  }
  __syncthreads();
  uint32_t res = s_warp[warp] + x - v;
  total = s_warp[32];
  __syncthreads();
  return res;
}

// Four input bytes: their 2-bit codes (byte 0 in the top bits of the low byte), a mask of
// the bytes equal to a character (bit 7 of each), and such a mask as four bits.
__device__ __forceinline__ uint32_t pack4_codes(uint32_t w) {
  return ((w >> 1) & 0x03030303u) * 0x40100401u;  // in the top byte
}
__device__ __forceinline__ uint32_t zero_bytes(uint32_t x) {
  return ~(((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x | 0x7f7f7f7fu);
}
__device__ __forceinline__ uint32_t flags4(uint32_t m) {  // bits 7, 15, 23, 31 -> 0..3
  return ((m >> 7) * 0x01020408u) >> 24;
}
// a 16-byte unit's four words of such masks as 16 bits
__device__ __forceinline__ uint32_t flags16(uint32_t m0, uint32_t m1, uint32_t m2, uint32_t m3) {
  return flags4(m0) | (flags4(m1) << 4) | (flags4(m2) << 8) | (flags4(m3) << 12);
}
// base j's code at bits 2(15-j)+1..2(15-j)
__device__ __forceinline__ uint32_t unit_codes(const uint32_t w[4]) {
  const uint32_t hi = __byte_perm(pack4_codes(w[1]), pack4_codes(w[0]), 0x7300);
  const uint32_t lo = __byte_perm(pack4_codes(w[3]), pack4_codes(w[2]), 0x0073);
  return (hi & 0xffff0000u) | (lo & 0xffffu);
}
// byte flags (bit j) of a unit as its bit-2 plane: byte j at bit 2(15-j)
__device__ __forceinline__ uint32_t unit_plane(uint32_t flags) {
  uint32_t x = __brev(flags) >> 16;
  x = (x | (x << 8)) & 0x00ff00ffu;
  x = (x | (x << 4)) & 0x0f0f0f0fu;
  x = (x | (x << 2)) & 0x33333333u;
  return (x | (x << 1)) & 0x55555555u;
}

__device__ __forceinline__ void load_unit(const uint8_t* __restrict__ buf, unsigned long long F,
                                          unsigned long long p, uint32_t w[4]) {
  if (p + 16 <= F) {
    uint4 v = __ldg(reinterpret_cast<const uint4*>(buf + p));
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint32_t x = 0;
      for (int b = 0; b < 4; b++) {
        unsigned long long q = p + 4 * i + b;
        if (q < F) x |= (uint32_t)buf[q] << (8 * b);
      }
      w[i] = x;
    }
  }
}

// ------------------------------------------------------------- line scan (k_line_scan) -
// Newlines per 64 KB tile, the first '>' and the number of '>' bytes.  Bound: the read;
// 407 MB in 95 us (4.3 TB/s) with four loads in flight a thread, 127 us with one.
__global__ void __launch_bounds__(256) k_line_scan(const uint8_t* __restrict__ buf,
                                                   unsigned long long F, uint32_t* tile_nl,
                                                   Scalars* sc, unsigned long long tile0) {
  const unsigned long long tile = tile0 + blockIdx.x;
  const unsigned long long t0 = tile * kTileBytes;
  const unsigned long long t1 = min(t0 + (unsigned long long)kTileBytes, F);
  uint32_t nl = 0, gt = 0;
  unsigned long long first = ~0ull;
  auto scan = [&](const uint32_t w[4], unsigned long long p) {
    uint32_t g[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      nl += __popc(zero_bytes(w[i] ^ 0x0A0A0A0Au));
      g[i] = zero_bytes(w[i] ^ 0x3E3E3E3Eu);
      gt += __popc(g[i]);
    }
    if (first == ~0ull && (g[0] | g[1] | g[2] | g[3])) {
#pragma unroll
      for (int i = 3; i >= 0; i--)
        if (g[i]) first = p + 4 * i + (__ffs(g[i]) - 1) / 8;
    }
  };
  if (t1 - t0 == kTileBytes) {  // whole tiles: four 16-byte loads in flight a thread
    const uint4* __restrict__ v = reinterpret_cast<const uint4*>(buf + t0) + threadIdx.x;
#pragma unroll 1
    for (int o = 0; o < kTileBytes / 16; o += 1024) {
      uint4 x[4];
#pragma unroll
      for (int q = 0; q < 4; q++) x[q] = __ldg(v + o + 256 * q);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t w[4] = {x[q].x, x[q].y, x[q].z, x[q].w};
        scan(w, t0 + 16ull * (o + 256 * q + threadIdx.x));
      }
    }
  } else {
    for (unsigned long long p = t0 + 16ull * threadIdx.x; p < t1; p += 16ull * blockDim.x) {
      uint32_t w[4];
      load_unit(buf, F, p, w);  // a zero byte past F is neither '\n' nor '>'
      scan(w, p);
    }
  }
  __shared__ uint32_t s_nl[8], s_gt[8];
  __shared__ unsigned long long s_first[8];
  for (int o = 16; o > 0; o >>= 1) {
    nl += __shfl_down_sync(FULLMASK, nl, o);
    gt += __shfl_down_sync(FULLMASK, gt, o);
    unsigned long long f2 = __shfl_down_sync(FULLMASK, first, o);
    first = min(first, f2);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { s_nl[warp] = nl; s_gt[warp] = gt; s_first[warp] = first; }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t a = 0, b = 0;
    unsigned long long f = ~0ull;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) { a += s_nl[i]; b += s_gt[i]; f = min(f, s_first[i]); }
    tile_nl[tile] = a;
    if (b) atomicAdd(&sc->n_reads, (unsigned long long)b);
    if (f != ~0ull) atomicMin(&sc->s0, f);
  }
}

// One CTA: exclusive prefix of tile newline counts (in place, plus the grand total at
// [ntiles]) and the number of newlines before the first '>'.
__global__ void __launch_bounds__(1024) k_tile_prefix(const uint8_t* __restrict__ buf,
                                                      unsigned long long F, uint32_t* tile_nl,
                                                      int ntiles, Scalars* sc) {
  __shared__ uint32_t s_warp[33];
  uint32_t carry = 0;
  for (int base = 0; base < ntiles; base += blockDim.x) {
    int i = base + threadIdx.x;
    uint32_t v = i < ntiles ? tile_nl[i] : 0;
    uint32_t tot;
    uint32_t ex = block_exclusive_sum(v, s_warp, tot);
    if (i < ntiles) tile_nl[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) tile_nl[ntiles] = carry;
  __syncthreads();
  // newlines in [tile_start(s0), s0)
  const unsigned long long s0 = sc->s0;
  uint32_t cnt = 0;
  if (s0 < F) {
    const unsigned long long ts = (s0 / kTileBytes) * kTileBytes;
    for (unsigned long long p = ts + threadIdx.x; p < s0; p += blockDim.x) cnt += (buf[p] == '\n');
  }
  uint32_t tot;
  block_exclusive_sum(cnt, s_warp, tot);
  if (threadIdx.x == 0) {
    sc->nl_before_s0 = s0 < F ? tile_nl[s0 / kTileBytes] + tot : carry;
  }
}

// --------------------------------------------------------- k-mer window extraction --
// What a window of the next segment needs of this one: its units' codes with the bit-2
// plane folded in (kmer_shift ORs a byte's code bit 2 into the base before it) and the
// bytes no window may hold.
struct SegTail {
  uint32_t w[4];
  unsigned long long brk;
};

// Codes, line breaks, breakers and bit-2 flags of a 64-byte segment.
__device__ __forceinline__ void decode_segment(const uint32_t w[4][4], bool drop_n, uint32_t codes[4],
                                               unsigned long long& nl, unsigned long long& nn,
                                               unsigned long long& b2) {
  uint32_t l[4], n[4], t[4];
#pragma unroll
  for (int u = 0; u < 4; u++) {
    codes[u] = unit_codes(w[u]);
    l[u] = flags16(zero_bytes(w[u][0] ^ 0x0A0A0A0Au), zero_bytes(w[u][1] ^ 0x0A0A0A0Au),
                   zero_bytes(w[u][2] ^ 0x0A0A0A0Au), zero_bytes(w[u][3] ^ 0x0A0A0A0Au));
    t[u] = flags16((w[u][0] << 4) & 0x80808080u, (w[u][1] << 4) & 0x80808080u, (w[u][2] << 4) & 0x80808080u,
                   (w[u][3] << 4) & 0x80808080u);
    n[u] = 0;
    if (drop_n)
      n[u] = flags16(zero_bytes((w[u][0] | 0x20202020u) ^ 0x6E6E6E6Eu),
                     zero_bytes((w[u][1] | 0x20202020u) ^ 0x6E6E6E6Eu),
                     zero_bytes((w[u][2] | 0x20202020u) ^ 0x6E6E6E6Eu),
                     zero_bytes((w[u][3] | 0x20202020u) ^ 0x6E6E6E6Eu));
  }
  nl = (unsigned long long)(l[0] | (l[1] << 16)) | ((unsigned long long)(l[2] | (l[3] << 16)) << 32);
  nn = (unsigned long long)(n[0] | (n[1] << 16)) | ((unsigned long long)(n[2] | (n[3] << 16)) << 32);
  b2 = (unsigned long long)(t[0] | (t[1] << 16)) | ((unsigned long long)(t[2] | (t[3] << 16)) << 32);
}

// Bits [shift, shift + 64) of the 192-bit string c2:c1:c0 (shift < 128).
__device__ __forceinline__ unsigned long long bits64(uint64_t c0, uint64_t c1, uint64_t c2, int shift) {
  const uint64_t a = shift < 64 ? c0 : c1, b = shift < 64 ? c1 : c2;
  const int t = shift & 63;
  return t ? (a >> t) | (b << (64 - t)) : a;
}

// The k-mer whose newest byte has age sh/2 (sh = 0, 2, .., 30), codes alone.
template <typename KeyT>
__device__ __forceinline__ KeyT window_codes(uint64_t r0, uint64_t r1, uint64_t r2, int sh);
template <>
__device__ __forceinline__ uint64_t window_codes<uint64_t>(uint64_t r0, uint64_t r1, uint64_t, int sh) {
  const uint32_t lo = __funnelshift_r((uint32_t)r0, (uint32_t)(r0 >> 32), sh);
  const uint32_t hi = __funnelshift_r((uint32_t)(r0 >> 32), (uint32_t)r1, sh);
  return (uint64_t)hi << 32 | lo;
}
template <>
__device__ __forceinline__ u128 window_codes<u128>(uint64_t r0, uint64_t r1, uint64_t r2, int sh) {
  const uint64_t lo = window_codes<uint64_t>(r0, r1, 0, sh), hi = window_codes<uint64_t>(r1, r2, 0, sh);
  return ((u128)hi << 64) | lo;
}

// Reference record-start rule: a sequence line ending at `pos` (a newline) must be
// followed by '>' when its line start p satisfies p <= F - m.
__device__ void check_record_start(const uint8_t* __restrict__ buf, unsigned long long F, int m,
                                   unsigned long long pos, uint8_t next, uint32_t* err) {
  if (pos + 1 >= F || next == '>') return;
  long long lim = (long long)F - (long long)m;
  if (lim < 0) return;
  bool counts = true;
  if ((long long)pos > lim) {
    // line start <= lim  <=>  no newline in [lim, pos)
    for (long long q = lim; q < (long long)pos; q++)
      if (buf[q] == '\n') { counts = false; break; }
  }
  if (counts) atomicOr(err, ERR_FORMAT);
}

template <typename KeyT>
__device__ __forceinline__ void guarded_store(KeyT* __restrict__ out, uint32_t idx, KeyT v,
                                              unsigned long long cap, uint32_t* err) {
  if (idx < cap) out[idx] = v;
  else atomicOr(err, ERR_BOUNDS);
}

// Counting pass: per chunk, the bucket histogram of its windows, and the packed units that
// the coarse scatter rolls.  A thread takes a 64-byte segment; 1024 threads a CTA, one CTA
// per SM (its histogram holds up to 2^15 bins).
//
// Bound: issue.  So whole segments are decided at once, in 64-bit masks: line parity is a
// prefix XOR of the line breaks, the windows that hold a breaker are the breakers smeared
// over k - 1 bytes (the run before the segment comes from its left neighbour by shuffle,
// not by decoding 64 bytes again), and what is left is one bit per window.  A window's
// bucket is a funnel shift of the segment's codes aligned to the bucket digits: the digits
// start at key bit 2 or above, and a byte outside the window can only reach key bit 0.
// Bit-2 planes are built only for segments whose sequence bytes have such a bit (N, '\r').
// Bacterial reads (407 MB): 0.66 -> 0.37 ms against testing every window by itself; 25 Mbp
// long-k (1.05 GB, k = 63): 2.93 -> 1.02 ms.  The histogram's shared-memory atomics are
// about half of what is left.
constexpr int kCountT = 1024;
template <bool WIDE>
__global__ void __launch_bounds__(kCountT, 1) k_extract(CountArgs a) {
  constexpr int NW = kCountT / 32;
  extern __shared__ uint32_t s_bins[];
  __shared__ uint32_t s_wpar[NW];
  __shared__ SegTail s_tail[NW];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int B = 1 << a.bbits;
  const int k = a.k;
  const int shift = 2 * k - a.bbits;  // >= 2
  const uint32_t hmask = (uint32_t)(B - 1) << 2;  // byte offset of a bin
  const bool drop_n = a.drop_n != 0;
  const uint8_t* __restrict__ buf = a.fasta;
  const unsigned long long F = a.F;
  const unsigned long long s0 = a.sc->s0;
  const int c = blockIdx.x;

  for (int i = tid; i < B; i += kCountT) s_bins[i] = 0;
  __syncthreads();

  const unsigned long long c0 = (unsigned long long)c * a.chunk;
  const unsigned long long c1 = min(c0 + a.chunk, F);
  uint32_t local = 0;
  if (c0 < c1 && s0 < F) {
    uint32_t carry = (a.tile_nl[c0 / kTileBytes] ^ a.sc->nl_before_s0) & 1u;
    for (unsigned long long base = c0; base < c1; base += (unsigned long long)kCountT * kSegBytes) {
      const unsigned long long seg = base + (unsigned long long)tid * kSegBytes;
      const bool active = seg < c1;
      // the segment before warp 0's first: the last one of the previous step, or decoded
      // from memory at the chunk's start
      SegTail before;
      before.w[0] = before.w[1] = before.w[2] = before.w[3] = 0;
      before.brk = 0;
      if (tid == 0) {
        if (base > c0) {
          before = s_tail[NW - 1];
        } else if (seg >= kSegBytes) {
          uint32_t w[4][4], codes[4];
          unsigned long long nl, nn, b2;
#pragma unroll
          for (int u = 0; u < 4; u++) load_unit(buf, F, seg - kSegBytes + 16ull * u, w[u]);
          decode_segment(w, drop_n, codes, nl, nn, b2);
          before.brk = nl | nn;
          uint32_t up = 0;
#pragma unroll
          for (int u = 3; u >= 0; u--) {
            const uint32_t n = unit_plane((uint32_t)(b2 >> (16 * u)) & 0xffffu);
            before.w[u] = codes[u] | (n << 2) | up;
            up = n >> 30;
          }
        }
      }
      uint32_t w[4][4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        if (active) load_unit(buf, F, seg + 16ull * u, w[u]);
        else w[u][0] = w[u][1] = w[u][2] = w[u][3] = 0;
      }
      uint32_t codes[4];
      unsigned long long nl, nn, b2;
      decode_segment(w, drop_n, codes, nl, nn, b2);
      // parity of the line count at the segment start (block XOR-scan)
      const unsigned bal = __ballot_sync(FULLMASK, __popcll(nl) & 1);
      if (lane == 0) s_wpar[warp] = __popc(bal) & 1u;
      __syncthreads();
      const unsigned wpar = __ballot_sync(FULLMASK, s_wpar[lane] != 0);
      const uint32_t pin = (carry ^ __popc(wpar & ((1u << warp) - 1u)) ^ __popc(bal & lanemask_lt())) & 1u;
      carry ^= __popc(wpar) & 1u;
      // sequence bytes: odd lines, from the first '>' on, inside the buffer
      unsigned long long x = nl;
      x ^= x << 1; x ^= x << 2; x ^= x << 4; x ^= x << 8; x ^= x << 16; x ^= x << 32;
      unsigned long long in = (x << 1) ^ (pin ? ~0ull : 0ull);
      if (seg + kSegBytes > F) in &= active ? (1ull << (F - seg)) - 1ull : 0ull;
      if (seg < s0) in &= s0 - seg >= kSegBytes ? 0ull : ~0ull << (s0 - seg);
      // code bit 2 of sequence bytes, folded into the codes
      const unsigned long long n2 = b2 & in & ~nl;
      SegTail t;
#pragma unroll
      for (int u = 0; u < 4; u++) t.w[u] = codes[u];
      t.brk = nl | nn;
      const unsigned long long g = seg / kSegBytes;
      uint32_t flag = 0, up = 0;
      if (n2) {
        flag = 2;
#pragma unroll
        for (int u = 3; u >= 0; u--) {
          const uint32_t n = unit_plane((uint32_t)(n2 >> (16 * u)) & 0xffffu);
          t.w[u] |= (n << 2) | up;
          up = n >> 30;
          if (active) a.unit_nbits[u * a.nseg + g] = u == 3 ? n | flag : n;
        }
      }
      if (lane == 31) s_tail[warp] = t;
      __syncthreads();
      SegTail pv;
#pragma unroll
      for (int u = 0; u < 4; u++) pv.w[u] = WIDE || u >= 2 ? __shfl_up_sync(FULLMASK, t.w[u], 1) : 0u;
      pv.brk = __shfl_up_sync(FULLMASK, t.brk, 1);
      // the first unit's top bit reaches back into the neighbour's last base: below the digits
      // of any window that ends in the neighbour, inside those that end here
      if (lane == 0) pv = warp ? s_tail[warp - 1] : before;
      if (!active) continue;
      pv.w[3] |= up;
      // windows without a breaker: none among the k - 1 bytes before the newest, or at it
      unsigned long long bad = t.brk;
      {
        int cov = 1;
        while (2 * cov <= k) {
          bad |= bad << cov;
          cov *= 2;
        }
        if (cov < k) bad |= bad << (k - cov);
      }
      const int run = pv.brk ? __clzll((long long)pv.brk) : kSegBytes;  // clean bytes before the segment
      unsigned long long counted = ~bad & in;
      if (run < k - 1) counted &= ~0ull << (k - 1 - run);
      a.unit_windows[g] = counted;
      if (!n2) a.unit_nbits[3 * a.nseg + g] = 0;
      {
        unsigned long long ends = nl & in;  // newlines that end sequence lines
        while (ends) {
          const int q = __ffsll((long long)ends) - 1;
          ends &= ends - 1;
          // the byte after the newline, read from memory (it is in L1)
          const unsigned long long p = seg + q;
          const uint8_t next = p + 1 < F ? __ldg(buf + p + 1) : (uint8_t)'>';
          check_record_start(buf, F, a.lmer_m, p, next, &a.sc->err);
        }
      }
      local += __popcll(counted);
      uint64_t r0 = (uint64_t)pv.w[2] << 32 | pv.w[3], r1 = (uint64_t)pv.w[0] << 32 | pv.w[1], r2 = 0;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        a.unit_codes[u * a.nseg + g] = codes[u];
        if (WIDE) r2 = (r2 << 32) | (r1 >> 32);
        r1 = (r1 << 32) | (r0 >> 32);
        r0 = (r0 << 32) | t.w[u];
        const uint32_t v = (uint32_t)(counted >> (16 * u)) & 0xffffu;
        if (!v) continue;
        // the unit's windows aligned so that age 0's bucket digits start at bit 2
        const unsigned long long q = bits64(r0, r1, r2, shift - 2);
        const uint32_t qlo = (uint32_t)q, qhi = (uint32_t)(q >> 32);
#pragma unroll
        for (int j = 0; j < 16; j++) {
          if ((v >> j) & 1u) {
            const uint32_t o = __funnelshift_r(qlo, qhi, 2 * (15 - j)) & hmask;
            atomicAdd(reinterpret_cast<uint32_t*>(reinterpret_cast<char*>(s_bins) + o), 1u);
          }
        }
      }
    }
  }
  __syncthreads();
  for (int i = tid; i < B; i += kCountT) a.counts[(size_t)c * B + i] = s_bins[i];
  local = __reduce_add_sync(FULLMASK, local);
  if (lane == 0) s_wpar[warp] = local;
  __syncthreads();
  if (warp == 0) {
    const uint32_t n = __reduce_add_sync(FULLMASK, s_wpar[lane]);
    if (lane == 0 && n) atomicAdd(&a.sc->n_windows, (unsigned long long)n);
  }
}

// ----------------------------------------------------- two-pass partition of keys ---
// Pass 1 (k_scatter_coarse): roll the k-mers of a chunk again and append each key to a
// shared-memory ring of its coarse bucket (leading kCoarseBits bits); whole 128-byte
// lines are flushed by warps to the chunk's segment of the coarse region, so global
// stores are lines instead of scattered 8/16-byte writes.
template <typename KeyT>
struct CoarseCfg {
  static constexpr int C = 1 << kCoarseBits;               // coarse buckets
  static constexpr int R = sizeof(KeyT) == 8 ? 128 : 64;    // ring slots per bucket
  static constexpr int FU = 128 / (int)sizeof(KeyT);        // keys per 128-byte line
  // Rings are flushed after every BP window positions of a thread, when an average ring
  // has taken about 80 of its 128 slots (64-bit keys) or 40 of its 64 (128-bit keys); a
  // ring that overflows sends its extra keys straight to global memory.  64-bit keys every
  // 8 positions instead: 0.84 against 0.73 ms (bacterial); 128-bit keys with 512 threads and
  // 16 positions: 3.27 against 2.70 ms (25 Mbp long-k).
  static constexpr int T = 1024;
  static constexpr int BP = sizeof(KeyT) == 8 ? 16 : 8;
  static constexpr size_t smem = sizeof(KeyT) * C * R;
};

// Writes the rings' keys out up to the last whole 128-byte line of the output (all of
// them at the end) and moves what is left to the front, so that a ring's next key goes to
// slot s_w[b] and s_g[b] is where slot 0 belongs.
template <typename KeyT>
__device__ __forceinline__ void coarse_flush(KeyT* ring, uint32_t* w, uint32_t* g, KeyT* __restrict__ out,
                                             bool final_flush, unsigned long long cap, uint32_t* err) {
  using CF = CoarseCfg<KeyT>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = CF::T / 32;
  for (int b = warp; b < CF::C; b += NW) {
    const uint32_t W = w[b], gb = g[b];
    KeyT* rb = ring + b * CF::R;
    uint32_t n = W, left = 0;
    if (W > (uint32_t)CF::R) {
      n = CF::R;  // the ring overflowed: the keys past it went straight to global memory
    } else if (!final_flush) {
      left = min(W, (gb + W) & (uint32_t)(CF::FU - 1));
      n = W - left;
    }
    for (uint32_t x = lane; x < n; x += 32) guarded_store(out, gb + x, rb[x], cap, err);
    if (n) {
      KeyT keep = 0;
      if ((uint32_t)lane < left) keep = rb[n + lane];
      __syncwarp();
      if ((uint32_t)lane < left) rb[lane] = keep;
      if (lane == 0) {
        w[b] = left;
        g[b] = gb + (W - left);
      }
    }
  }
}

// Bound: the shared-memory atomic and ring store of every key.  A window is two funnel
// shifts of the codes (four for 128-bit keys), its coarse bucket one more of the codes
// aligned to the bucket digits; rings start at slot 0 after every flush, which ends at a
// whole line of the output, so an append needs no ring position.  Bacterial reads: 0.91 ->
// 0.73 ms against rolling both planes for every window; 25 Mbp long-k: 4.21 -> 2.70 ms.
template <typename KeyT>
__global__ void __launch_bounds__(CoarseCfg<KeyT>::T, 1)
k_scatter_coarse(CountArgs a, const uint32_t* __restrict__ coff, KeyT* __restrict__ out) {
  using CF = CoarseCfg<KeyT>;
  constexpr bool WIDE = sizeof(KeyT) == 16;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KeyT* ring = reinterpret_cast<KeyT*>(smem_raw);
  __shared__ uint32_t s_w[CF::C], s_g[CF::C];
  const int tid = threadIdx.x;
  const int k = a.k;
  const int cshift = 2 * k - a.cbits;  // coarse bucket = leading cbits bits
  const KeyT kmask = KeyOps<KeyT>::mask(2 * k);
  const unsigned long long F = a.F;
  const unsigned long long s0 = a.sc->s0;
  const int c = blockIdx.x;
  const int Cn = 1 << a.cbits;
  for (int i = tid; i < CF::C; i += CF::T) {
    s_w[i] = 0;
    s_g[i] = i < Cn ? coff[(size_t)c * Cn + i] : 0;
  }
  __syncthreads();
  const unsigned long long c0 = (unsigned long long)c * a.chunk;
  const unsigned long long c1 = min(c0 + a.chunk, F);
  const unsigned long long nseg = a.nseg;
  auto append = [&](KeyT key, uint32_t b) {
    const uint32_t pos = atomicAdd(&s_w[b], 1u);
    if (pos < (uint32_t)CF::R) ring[b * CF::R + pos] = key;
    else guarded_store(out, s_g[b] + pos, key, a.n_keys, &a.sc->err);
  };
  if (c0 < c1 && s0 < F) {
    for (unsigned long long base = c0; base < c1; base += (unsigned long long)CF::T * kSegBytes) {
      const unsigned long long seg = base + (unsigned long long)tid * kSegBytes;
      const bool active = seg < c1;
      const unsigned long long g = seg / kSegBytes;
      // the counting pass's packed units: codes, bit-2 plane and the windows it counted
      // (no FASTA decode, no line parity, no window checks here)
      uint32_t cd[4] = {0, 0, 0, 0};
      unsigned long long counted = 0;
      uint64_t r0 = 0, r1 = 0, r2 = 0;
      uint32_t own = 0, left = 0;  // unit 3's bit-2 words of this segment and the one before
      if (active) {
        counted = __ldg(a.unit_windows + g);
        own = __ldg(a.unit_nbits + 3 * nseg + g);
#pragma unroll
        for (int u = 0; u < 4; u++) cd[u] = __ldg(a.unit_codes + u * nseg + g);
        if (g > 0) {
          r0 = (uint64_t)__ldg(a.unit_codes + 2 * nseg + g - 1) << 32 | __ldg(a.unit_codes + 3 * nseg + g - 1);
          if (WIDE) r1 = (uint64_t)__ldg(a.unit_codes + g - 1) << 32 | __ldg(a.unit_codes + nseg + g - 1);
          left = __ldg(a.unit_nbits + 3 * nseg + g - 1);
        }
      }
      // bit-2 planes are folded into the codes, each byte's bit into the base before it;
      // a window then takes the low bit of its newest base from the plain codes, as the
      // byte after it is not its own
      const bool fold = __any_sync(FULLMASK, own | left);
      if (left) {
        const uint64_t m0 = (uint64_t)__ldg(a.unit_nbits + 2 * nseg + g - 1) << 32 | (left & 0x55555555u);
        r0 |= m0 << 2;
        if (WIDE) {
          const uint64_t m1 = (uint64_t)__ldg(a.unit_nbits + g - 1) << 32 | __ldg(a.unit_nbits + nseg + g - 1);
          r1 |= (m1 << 2) | (m0 >> 62);
        }
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const uint32_t v = (uint32_t)(counted >> (16 * u)) & 0xffffu;
        if (WIDE) r2 = (r2 << 32) | (r1 >> 32);
        r1 = (r1 << 32) | (r0 >> 32);
        r0 = (r0 << 32) | cd[u];
        if (own) r0 |= (uint64_t)(u == 3 ? own & 0x55555555u : __ldg(a.unit_nbits + u * nseg + g)) << 2;
        const unsigned long long q = bits64(r0, r1, r2, cshift);
        const uint32_t qlo = (uint32_t)q, qhi = (uint32_t)(q >> 32);
#pragma unroll
        for (int part = 0; part < 16 / CF::BP; part++) {
          if (!fold) {
#pragma unroll
            for (int jj = 0; jj < CF::BP; jj++) {
              const int j = part * CF::BP + jj, sh = 2 * (15 - j);
              if ((v >> j) & 1u)
                append(window_codes<KeyT>(r0, r1, r2, sh) & kmask,
                       __funnelshift_r(qlo, qhi, sh) & (uint32_t)(Cn - 1));
            }
          } else {
#pragma unroll
            for (int jj = 0; jj < CF::BP; jj++) {
              const int j = part * CF::BP + jj, sh = 2 * (15 - j);
              if ((v >> j) & 1u) {
                const KeyT key = window_codes<KeyT>(r0, r1, r2, sh) & kmask;
                append((key & ~(KeyT)1) | (KeyT)((cd[u] >> sh) & 1u),
                       __funnelshift_r(qlo, qhi, sh) & (uint32_t)(Cn - 1));
              }
            }
          }
          __syncthreads();
          coarse_flush<KeyT>(ring, s_w, s_g, out, false, a.n_keys, &a.sc->err);
          __syncthreads();
        }
      }
    }
  }
  __syncthreads();
  coarse_flush<KeyT>(ring, s_w, s_g, out, true, a.n_keys, &a.sc->err);
}

// Coarse offsets: coff[c][g] = start of chunk c's segment in coarse region g (the
// coarse region is the union of its fine buckets' regions); cstart[g] = region start;
// slice_start[g] = first pass-2 slice of region g.  The counting pass's histogram has 2^hbits
// bins; where that is the partition's 2^pbits buckets or more, their starts and the fine
// scatter's cursors are picked out of its prefix here too.
__global__ void __launch_bounds__(256) k_coarse_offsets(const uint32_t* __restrict__ counts,
                                                        const uint32_t* __restrict__ hstart, int hbits, int pbits,
                                                        int cbits, uint32_t* coff, uint32_t* cstart,
                                                        uint32_t* slice_start, int slice_keys,
                                                        uint32_t* __restrict__ bstart,
                                                        uint32_t* __restrict__ fcur, Scalars* sc) {
  __shared__ uint32_t s_c[1 << kCoarseBits];
  __shared__ uint32_t s_warp[33];
  const int c = blockIdx.x;
  const int Cn = 1 << cbits, fb = hbits - cbits;
  // a warp sums the 2^fb histogram bins of one coarse region at a time
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int g = warp; g < Cn; g += nw) {
    uint32_t sum = 0;
    for (int i = lane; i < (1 << fb); i += 32) sum += counts[((size_t)c << hbits) + ((size_t)g << fb) + i];
    sum = __reduce_add_sync(FULLMASK, sum);
    if (lane == 0) s_c[g] = sum;
  }
  __syncthreads();
  for (int g = threadIdx.x; g < Cn; g += blockDim.x) coff[(size_t)c * Cn + g] = hstart[g << fb] + s_c[g];
  if (pbits <= hbits) {
    const int B = 1 << pbits, d = hbits - pbits;
    for (int i = c * blockDim.x + threadIdx.x; i <= B; i += gridDim.x * blockDim.x) {
      const uint32_t v = hstart[i << d];
      bstart[i] = v;
      if (i < B) fcur[i] = v;
    }
  }
  if (c == 0) {
    static_assert((1 << kCoarseBits) <= 256, "one region per thread");
    const int g = threadIdx.x;
    uint32_t s = 0, e = 0;
    if (g < Cn) {
      s = hstart[g << fb];
      e = hstart[(g + 1) << fb];
      cstart[g] = s;
      if (g == Cn - 1) cstart[Cn] = e;
    }
    uint32_t tot;
    const uint32_t first = block_exclusive_sum((e - s + slice_keys - 1) / slice_keys, s_warp, tot);
    if (g < Cn) slice_start[g] = first;
    if (g == 0) {
      slice_start[Cn] = tot;
      sc->ticket_fine = 0;
    }
  }
}

// Pass 2 (k_scatter_fine): a slice of a coarse region (in chunk order) is counted by
// fine bucket in shared memory, which also gives every key its rank in its bucket; one
// atomic per (slice, fine bucket) reserves a run in the bucket's region; the slice is staged
// by bucket and stored in runs.  Keys stay in registers between the two.  Bound: latency
// between its barriers, at 63 to 66 % of the copy bandwidth.  Bacterial reads (254M keys):
// 1.02 -> 0.91 ms against a second atomic per key for its rank and a binary search in
// global memory for every slice's region.  One CTA of 1024 threads an SM: 0.98 ms; the next
// slice's ticket taken ahead: no change.
// FEW: up to 2^kFewFine fine buckets, where slices of a quarter still give runs of 16 (64-bit)
// or 8 keys: six CTAs an SM instead of two wait at their barriers at other times.  Bacterial
// reads (2^14 buckets, 2^7 fine): 0.90 -> 0.77 ms; three CTAs of 4096-key slices 0.80 ms, of
// 8192 1.28 ms (they spill).  With 2^10 fine buckets 4096-key slices lose (25 Mbp long-k path
// 22.6 -> 26.0 ms).  The line between, quarter against whole slices: 64-bit keys at 2^8 fine
// buckets 0.85 against 0.93 ms (254M keys) and 1.58 against 1.70 ms (472M), at 2^9 3.16 against
// 1.41 ms; 128-bit keys at 2^8 1.23 against 1.20, at 2^9 4.94 against 1.79 ms (195M).  So it
// could lie at 2^8 for 64-bit keys; it is the same for both widths.
constexpr int kFewFine = 7;
template <typename KeyT, bool FEW>
struct FineCfg {
  static constexpr int T = FEW ? 256 : 512;                  // threads
  static constexpr int CTAS = FEW ? 6 : 2;                   // CTAs per SM
  static constexpr int PT = (FEW ? 64 : 128) / (int)sizeof(KeyT);  // keys per thread
  static constexpr int S = T * PT;                           // keys per slice (16 or 64 KB)
  static constexpr int FBMAX = 1 << (FEW ? kFewFine : kMaxPartBits - kCoarseBits);  // fine buckets per coarse
  static constexpr size_t smem = sizeof(KeyT) * S;
};

template <typename KeyT, bool FEW>
__global__ void __launch_bounds__(FineCfg<KeyT, FEW>::T, FineCfg<KeyT, FEW>::CTAS)
k_scatter_fine(const KeyT* __restrict__ in, const uint32_t* __restrict__ cstart,
               const uint32_t* __restrict__ slice_start, uint32_t* fcur, KeyT* __restrict__ out, int k, int bbits,
               int cbits, uint32_t* ticket, unsigned long long cap, uint32_t* err) {
  using FC = FineCfg<KeyT, FEW>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KeyT* stage = reinterpret_cast<KeyT*>(smem_raw);  // the slice grouped by fine bucket
  // per fine bucket: keys, first staged key, and what takes a staged position to its place
  __shared__ uint32_t s_hist[FC::FBMAX], s_loff[FC::FBMAX], s_move[FC::FBMAX];
  __shared__ uint32_t s_warp[33];
  __shared__ uint32_t s_slice, s_g;
  // the region tables live in shared memory: a slice finds its region with one read a lane
  __shared__ uint32_t s_ss[(1 << kCoarseBits) + 1], s_cs[(1 << kCoarseBits) + 1];
  const int tid = threadIdx.x;
  const int Cn = 1 << cbits, fb = bbits - cbits, FB = 1 << fb;
  const int fshift = 2 * k - bbits;
  const uint32_t fmask = (uint32_t)(FB - 1);
  for (int i = tid; i <= Cn; i += FC::T) {
    s_ss[i] = slice_start[i];
    s_cs[i] = cstart[i];
  }
  for (int i = tid; i < FB; i += FC::T) s_hist[i] = 0;
  const uint32_t nslices = slice_start[Cn];
  while (true) {
    __syncthreads();
    if (tid < 32) {
      uint32_t sl = 0;
      if (tid == 0) sl = atomicAdd(ticket, 1u);
      sl = __shfl_sync(FULLMASK, sl, 0);
      uint32_t below = 0;  // regions that start at or before the slice
      for (int i = tid; i < Cn; i += 32) below += s_ss[i] <= sl ? 1u : 0u;
      below = __reduce_add_sync(FULLMASK, below);
      if (tid == 0) {
        s_slice = sl;
        s_g = below - 1;
      }
    }
    __syncthreads();
    const uint32_t sl = s_slice;
    if (sl >= nslices) break;
    const uint32_t g = s_g;
    const uint32_t r0 = s_cs[g] + (sl - s_ss[g]) * FC::S;
    const uint32_t r1 = min(r0 + (uint32_t)FC::S, s_cs[g + 1]);
    const uint32_t m = r1 - r0;
    KeyT xs[FC::PT];
    uint32_t rank[FC::PT / 2];  // a key's rank in its fine bucket, two to a word (a slice has
                                // at most 8192 keys)
#pragma unroll
    for (int q = 0; q < FC::PT; q++) {
      const uint32_t i = q * FC::T + tid;
      xs[q] = i < m ? in[r0 + i] : (KeyT)0;
    }
#pragma unroll
    for (int q = 0; q < FC::PT; q++) {
      const uint32_t i = q * FC::T + tid;
      uint32_t r = 0;
      if (i < m) r = atomicAdd(&s_hist[(uint32_t)(xs[q] >> fshift) & fmask], 1u);
      if (q & 1) rank[q / 2] |= r << 16;
      else rank[q / 2] = r;
    }
    __syncthreads();
    {
      // each thread owns a contiguous run of FB / T fine buckets (at least one)
      constexpr int FPT = (FC::FBMAX + FC::T - 1) / FC::T;
      const int per = (FB + FC::T - 1) / FC::T;
      const int f0 = min(FB, tid * per);
      uint32_t hv[FPT], sum = 0;
#pragma unroll
      for (int q = 0; q < FPT; q++) {
        hv[q] = 0u;
        if (q < per && f0 + q < FB) {
          hv[q] = s_hist[f0 + q];
          s_hist[f0 + q] = 0;  // for the next slice
        }
        sum += hv[q];
      }
      uint32_t tot;
      uint32_t ex = block_exclusive_sum(sum, s_warp, tot);
#pragma unroll
      for (int q = 0; q < FPT; q++) {
        if (q < per && f0 + q < FB) {
          s_loff[f0 + q] = ex;
          s_move[f0 + q] = hv[q] ? atomicAdd(&fcur[(g << fb) + f0 + q], hv[q]) - ex : 0u;
          ex += hv[q];
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < FC::PT; q++) {
      const uint32_t i = q * FC::T + tid;
      if (i < m) {
        const uint32_t r = (q & 1) ? rank[q / 2] >> 16 : rank[q / 2] & 0xffffu;
        stage[s_loff[(uint32_t)(xs[q] >> fshift) & fmask] + r] = xs[q];
      }
    }
    __syncthreads();
    // runs of one fine bucket are contiguous in `stage` and in `out`: coalesced stores
    for (uint32_t i = tid; i < m; i += FC::T) {
      const KeyT x = stage[i];
      guarded_store(out, s_move[(uint32_t)(x >> fshift) & fmask] + i, x, cap, err);
    }
  }
}

// Wide fan-out (2048 fine buckets per coarse region): a slice of 192 KB is
// staged in shared memory so that each fine bucket still gets runs of several keys.
// The slice is read twice (counting, then placing; the second read mostly hits L2),
// four keys per thread per round.
template <typename KeyT>
struct FineBigCfg {
  static constexpr int T = 1024;
  static constexpr int S = (192 * 1024) / (int)sizeof(KeyT);  // keys per slice
  static constexpr int PR = 4;                                 // keys per thread per round
  static constexpr size_t smem = sizeof(KeyT) * S;
};

template <typename KeyT>
__global__ void __launch_bounds__(1024, 1) k_scatter_fine_big(const KeyT* __restrict__ in,
                                                             const uint32_t* __restrict__ cstart,
                                                             const uint32_t* __restrict__ slice_start,
                                                             uint32_t* fcur, KeyT* __restrict__ out,
                                                             int k, int bbits, int cbits, uint32_t* ticket,
                                                             unsigned long long cap, uint32_t* err) {
  using FC = FineBigCfg<KeyT>;
  constexpr int FBMAX = FineCfg<KeyT, false>::FBMAX;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  KeyT* stage = reinterpret_cast<KeyT*>(smem_raw);
  __shared__ uint32_t s_hist[FBMAX], s_loff[FBMAX], s_goff[FBMAX], s_fill[FBMAX];
  __shared__ uint32_t s_warp[33];
  __shared__ uint32_t s_slice, s_g;
  const int tid = threadIdx.x;
  const int Cn = 1 << cbits, fb = bbits - cbits, FB = 1 << fb;
  const int fshift = 2 * k - bbits;
  // the region tables live in shared memory: the slice -> region search of every slice
  // reads no global memory
  __shared__ uint32_t s_ss[(1 << kCoarseBits) + 1], s_cs[(1 << kCoarseBits) + 1];
  for (int i = tid; i <= Cn; i += FC::T) {
    s_ss[i] = slice_start[i];
    s_cs[i] = cstart[i];
  }
  const uint32_t nslices = slice_start[Cn];
  while (true) {
    __syncthreads();
    if (tid == 0) {
      s_slice = atomicAdd(ticket, 1u);
      if (s_slice < nslices) {
        int lo = 0, hi = Cn - 1;  // last g with slice_start[g] <= slice
        while (lo < hi) {
          int mid = (lo + hi + 1) >> 1;
          if (s_ss[mid] <= s_slice) lo = mid; else hi = mid - 1;
        }
        s_g = lo;
      }
    }
    for (int i = tid; i < FB; i += FC::T) { s_hist[i] = 0; s_fill[i] = 0; }
    __syncthreads();
    const uint32_t sl = s_slice;
    if (sl >= nslices) break;
    const uint32_t g = s_g;
    const uint32_t r0 = s_cs[g] + (sl - s_ss[g]) * FC::S;
    const uint32_t r1 = min(r0 + (uint32_t)FC::S, s_cs[g + 1]);
    const uint32_t m = r1 - r0;
    for (uint32_t i0 = 0; i0 < m; i0 += FC::PR * FC::T) {
      KeyT xs[FC::PR];
#pragma unroll
      for (int q = 0; q < FC::PR; q++) {
        const uint32_t i = i0 + q * FC::T + tid;
        xs[q] = i < m ? in[r0 + i] : (KeyT)0;
      }
#pragma unroll
      for (int q = 0; q < FC::PR; q++)
        if (i0 + q * FC::T + tid < m) atomicAdd(&s_hist[(uint32_t)(xs[q] >> fshift) & (uint32_t)(FB - 1)], 1u);
    }
    __syncthreads();
    {
      constexpr int FPT = (FBMAX + FC::T - 1) / FC::T;
      const int per = (FB + FC::T - 1) / FC::T;
      const int f0 = min(FB, tid * per);
      uint32_t hv[FPT], sum = 0;
#pragma unroll
      for (int q = 0; q < FPT; q++) {
        hv[q] = (q < per && f0 + q < FB) ? s_hist[f0 + q] : 0u;
        sum += hv[q];
      }
      uint32_t tot;
      uint32_t ex = block_exclusive_sum(sum, s_warp, tot);
#pragma unroll
      for (int q = 0; q < FPT; q++) {
        if (q < per && f0 + q < FB) {
          s_loff[f0 + q] = ex;
          s_goff[f0 + q] = hv[q] ? atomicAdd(&fcur[(g << fb) + f0 + q], hv[q]) : 0u;
          ex += hv[q];
        }
      }
    }
    __syncthreads();
    for (uint32_t i0 = 0; i0 < m; i0 += FC::PR * FC::T) {
      KeyT xs[FC::PR];
#pragma unroll
      for (int q = 0; q < FC::PR; q++) {
        const uint32_t i = i0 + q * FC::T + tid;
        xs[q] = i < m ? in[r0 + i] : (KeyT)0;
      }
#pragma unroll
      for (int q = 0; q < FC::PR; q++) {
        if (i0 + q * FC::T + tid < m) {
          const uint32_t f = (uint32_t)(xs[q] >> fshift) & (uint32_t)(FB - 1);
          stage[s_loff[f] + atomicAdd(&s_fill[f], 1u)] = xs[q];
        }
      }
    }
    __syncthreads();
    for (uint32_t i = tid; i < m; i += FC::T) {
      const KeyT x = stage[i];
      const uint32_t f = (uint32_t)(x >> fshift) & (uint32_t)(FB - 1);
      guarded_store(out, s_goff[f] + (i - s_loff[f]), x, cap, err);
    }
  }
}

int fine_slice_keys(int wide, int fb) {
  if (fb >= 11) return wide ? FineBigCfg<u128>::S : FineBigCfg<uint64_t>::S;
  if (fb <= kFewFine) return wide ? FineCfg<u128, true>::S : FineCfg<uint64_t, true>::S;
  return wide ? FineCfg<u128, false>::S : FineCfg<uint64_t, false>::S;
}

// Fine bucket sizes when the partition has more digits than the counting pass's
// histogram: slices of each coarse region are counted by their fine digits in shared
// memory and added to bcount[(g << fb) + f].  Bound: reading the keys; a thread keeps eight
// loads in flight (one at a time took 2.43 ms for 568M 128-bit keys).
template <typename KeyT>
__global__ void __launch_bounds__(512, 2) k_fine_count(const KeyT* __restrict__ in,
                                                   const uint32_t* __restrict__ cstart,
                                                   const uint32_t* __restrict__ slice_start,
                                                   uint32_t* bcount, int k, int bbits, int cbits,
                                                   uint32_t* ticket, uint32_t slice_keys) {
  using FC = FineCfg<KeyT, false>;
  constexpr int T = 512, PF = 8;
  __shared__ uint32_t s_hist[FC::FBMAX];
  __shared__ uint32_t s_slice, s_g;
  const int tid = threadIdx.x;
  const int Cn = 1 << cbits, fb = bbits - cbits, FB = 1 << fb;
  const int fshift = 2 * k - bbits;
  // the region tables live in shared memory: a slice finds its region with one read a lane
  __shared__ uint32_t s_ss[(1 << kCoarseBits) + 1], s_cs[(1 << kCoarseBits) + 1];
  for (int i = tid; i <= Cn; i += T) {
    s_ss[i] = slice_start[i];
    s_cs[i] = cstart[i];
  }
  const uint32_t nslices = slice_start[Cn];
  while (true) {
    __syncthreads();
    if (tid < 32) {
      uint32_t sl = 0;
      if (tid == 0) sl = atomicAdd(ticket, 1u);
      sl = __shfl_sync(FULLMASK, sl, 0);
      uint32_t below = 0;  // regions that start at or before the slice
      for (int i = tid; i < Cn; i += 32) below += s_ss[i] <= sl ? 1u : 0u;
      below = __reduce_add_sync(FULLMASK, below);
      if (tid == 0) {
        s_slice = sl;
        s_g = below - 1;
      }
    }
    for (int i = tid; i < FB; i += T) s_hist[i] = 0;
    __syncthreads();
    const uint32_t sl = s_slice;
    if (sl >= nslices) break;
    const uint32_t g = s_g;
    const uint32_t r0 = s_cs[g] + (sl - s_ss[g]) * slice_keys;
    const uint32_t m = min(slice_keys, s_cs[g + 1] - r0);
    for (uint32_t i0 = 0; i0 < m; i0 += PF * T) {
      uint32_t f[PF];
#pragma unroll
      for (int q = 0; q < PF; q++) {
        const uint32_t i = i0 + q * T + tid;
        f[q] = i < m ? (uint32_t)(in[r0 + i] >> fshift) & (uint32_t)(FB - 1) : ~0u;
      }
#pragma unroll
      for (int q = 0; q < PF; q++)
        if (f[q] != ~0u) atomicAdd(&s_hist[f[q]], 1u);
    }
    __syncthreads();
    for (int f = tid; f < FB; f += T)
      if (s_hist[f]) atomicAdd(&bcount[((uint32_t)g << fb) + f], s_hist[f]);
  }
}

// counts[c][b] -> exclusive prefix over chunks (in place); totals into bstart[b].
__global__ void __launch_bounds__(256) k_col_prefix(uint32_t* counts, int grid, int B, uint32_t* totals) {
  // a CTA takes 32 bucket columns; its 8 warps take consecutive bands of chunk rows,
  // sum them (coalesced 128-byte rows), and take their band's offset from the sums of
  // the bands above
  __shared__ uint32_t s_band[8][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int b = blockIdx.x * 32 + lane;
  const int per = (grid + 7) / 8;
  const int c0 = min(grid, warp * per), c1 = min(grid, c0 + per);
  uint32_t sum = 0;
  if (b < B)
    for (int c = c0; c < c1; c++) sum += counts[(size_t)c * B + b];
  s_band[warp][lane] = sum;
  __syncthreads();
  uint32_t run = 0;
  for (int w = 0; w < warp; w++) run += s_band[w][lane];
  if (b < B) {
    for (int c = c0; c < c1; c++) {
      const size_t i = (size_t)c * B + b;
      const uint32_t v = counts[i];
      counts[i] = run;
      run += v;
    }
    if (warp == 7) totals[b] = run;  // the last band ends at the last chunk
  }
}

// Exclusive prefix of bstart[0..B) in place, bstart[B] = total.  One CTA, 16384 entries a
// step: four 16-byte loads a thread and one block scan (B a power of two up to 2^18; a run of
// B / 1024 entries a thread, one after the other, took 140 us at 2^17).
__global__ void __launch_bounds__(1024) k_bucket_prefix(uint32_t* bstart, int B) {
  __shared__ uint32_t s_warp[33];
  uint4* v4 = reinterpret_cast<uint4*>(bstart);  // B is 4 or more
  uint32_t carry = 0;
  for (int base = 0; base < B; base += 16 * 1024) {
    const int i0 = base / 4 + 4 * (int)threadIdx.x;
    uint4 v[4];
    uint32_t sum = 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      v[q] = 4 * (i0 + q) < B ? v4[i0 + q] : make_uint4(0, 0, 0, 0);
      sum += v[q].x + v[q].y + v[q].z + v[q].w;
    }
    uint32_t tot;
    uint32_t run = carry + block_exclusive_sum(sum, s_warp, tot);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint4 o = make_uint4(run, run + v[q].x, run + v[q].x + v[q].y, run + v[q].x + v[q].y + v[q].z);
      run = o.w + v[q].w;
      if (4 * (i0 + q) < B) v4[i0 + q] = o;
    }
    carry += tot;
  }
  if (threadIdx.x == 0) bstart[B] = carry;
}

// ------------------------------------------------------------- per-bucket table ------
template <typename KeyT>
struct BucketCfg;
// Threads, measured with two CTAs on an SM: 64-bit keys 768 (bacterial 1.62 ms; 512 and 1024
// 1.76 ms), 1024 with giant buckets (low-complexity reads: whole path 0.91 against
// 0.99 ms); 128-bit keys 512, whose four keys in
// flight need the registers (25 Mbp long-k, 2^18 buckets: 10.9 ms; 768 with two keys in
// flight 13.7 ms).  Keys per chunk of a giant bucket: one that has more distinct keys than half a
// table stays as it is, and every sub-range of the bucket then reads all its keys.  By the
// substitution rate, windows of 55 low-complexity bases at 1 % have about 3300 distinct ones
// in 32768 and 1050 in 8192, so 128-bit keys (half a table is 2048) take 8192.  6 Mbp, 60x,
// k = 55: 14.6 s with 32768, 0.96 s with 16384, 1.21 s with 8192, 1.52 s with 4096; k = 64, 40x:
// 8.3, 2.4, 1.06 and 1.33 s.  Keys loaded ahead: four (64-bit keys with two 1.84, with eight 1.88 ms).
template <>
struct BucketCfg<uint64_t> {
  static constexpr int H = 8192;   // table slots
  static constexpr int T = 768;    // threads
  static constexpr int TG = 1024;  // threads when there are giant buckets
  static constexpr int PF = 4;     // keys loaded per thread before inserting
  static constexpr int CH = 32768; // keys per chunk of a giant bucket
};
template <>
struct BucketCfg<u128> {
  static constexpr int H = 4096;
  static constexpr int T = 512;
  static constexpr int TG = 512;
  static constexpr int PF = 4;
  static constexpr int CH = 8192;
};

// Two CTAs fit an SM: for 64-bit keys 115 KB each (96 KB of slots, the sort's order and
// bins, the histogram and the pending sub-ranges).
template <typename KeyT>
struct BucketSmem {
  static constexpr int H = BucketCfg<KeyT>::H;
  static constexpr int BINS = 1 << kSortBinBits;
  static constexpr size_t off_key = 0;
  static constexpr size_t off_cnt = off_key + sizeof(KeyT) * H;
  static constexpr size_t off_ord = off_cnt + sizeof(uint32_t) * H;      // slot of every sorted element
  static constexpr size_t off_bin = off_ord + sizeof(uint16_t) * (H / 2);  // sort bins; samples of a split
  static constexpr size_t off_hist = off_bin + sizeof(uint32_t) * BINS;
  static constexpr size_t bytes = off_hist + sizeof(uint32_t) * kTableHist;
  static_assert(sizeof(KeyT) * kSplitSamples <= sizeof(uint32_t) * BINS, "samples share the bins");
};

// Insert (r, c) into the open-addressing table: 0 = r was present, 1 = r is new,
// 2 = no slot within kMaxProbe probes (treated as an overflow of the sub-range).
constexpr int kMaxProbe = 256;
template <typename KeyT>
__device__ __forceinline__ int hash_insert(KeyT* skey, uint32_t* scnt, uint32_t hmask, KeyT r, uint32_t c) {
  const KeyT EMPTY = ~(KeyT)0;
  uint32_t h = (uint32_t)(KeyOps<KeyT>::hash(r) >> 40) & hmask;
  for (int probe = 0; probe < kMaxProbe; probe++) {
    KeyT cur = *(volatile KeyT*)&skey[h];
    if (cur == r) {
      atomicAdd(&scnt[h], c);
      return 0;
    }
    if (cur == EMPTY) {
      KeyT old = KeyOps<KeyT>::cas(&skey[h], EMPTY, r);
      if (old == EMPTY || old == r) {
        atomicAdd(&scnt[h], c);
        return old == EMPTY ? 1 : 0;
      }
    }
    h = (h + 1) & hmask;
  }
  return 2;
}

// Sort bin of a remainder: the top bits below the sub-range's common prefix.
template <typename KeyT>
__device__ __forceinline__ uint32_t sort_bin(KeyT r, int dsh, uint32_t bmask) {
  return (uint32_t)KeyOps<KeyT>::shr(r, dsh) & bmask;
}

// One table row, plus its count in the bucket's histogram of small counts (sbsmall, folded
// into the count histogram when the bucket ends) or in the count histogram (counts below t).
template <typename KeyT>
__device__ __forceinline__ void emit_row(const BucketArgs& a, KeyT* __restrict__ tkeys, unsigned long long row,
                                         KeyT key, uint32_t cnt, uint32_t* shist, uint32_t* sbsmall) {
  if (row < a.cap) {
    tkeys[row] = key;
    a.tcounts[row] = cnt;
  } else {
    atomicOr(&a.sc->err, ERR_BOUNDS);
  }
  if (cnt < (uint32_t)kSmallCounts) {
    atomicAdd(&sbsmall[cnt], 1u);
  } else if (cnt < (uint32_t)a.t) {
    if (cnt < (uint32_t)kTableHist) atomicAdd(&shist[cnt], 1u);
    else atomicAdd(&a.hist[cnt], 1ull);
  }
}

// Chunk items of the giant buckets (one thread per bucket): a bucket of at least
// kGiantKeys keys reserves floor(n / chunk_keys) consecutive chunk items, gfirst[b] the
// first and gcount[b] how many, and marks them as its own in chunk_bucket; the number
// of chunk items ends in sc->n_chunk_items (zero beforehand); gdone = 0.  Its kGiantParts
// part items find it in glist; their look-back words and its small-count histogram, which
// they add to, are zeroed.
__global__ void __launch_bounds__(256) k_giant_chunks(const uint32_t* __restrict__ bstart, int B,
                                                      uint32_t* gfirst, uint32_t* gcount,
                                                      uint32_t* chunk_bucket, uint32_t* gdone,
                                                      unsigned long long* gpart, uint32_t* glist,
                                                      uint32_t* bsmall, uint32_t chunk_keys, Scalars* sc) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= B) return;
  const uint32_t n = bstart[b + 1] - bstart[b];
  const uint32_t c = n >= kGiantKeys ? n / chunk_keys : 0u;
  gdone[b] = 0;
  gcount[b] = c;
  uint32_t g0 = 0;
  if (c) {
    g0 = atomicAdd(&sc->n_chunk_items, c);
    for (uint32_t i = 0; i < c; i++) chunk_bucket[g0 + i] = (uint32_t)b;
    const uint32_t g = atomicAdd(&sc->n_giants, 1u);
    glist[g] = (uint32_t)b;
    for (int i = 0; i < kGiantParts; i++) gpart[(size_t)kGiantParts * g + i] = 0;
    for (int i = 0; i < kSmallCounts; i++) bsmall[(size_t)b * kSmallCounts + i] = 0;
  }
  gfirst[b] = g0;
}

// A shared flag as the whole warp sees it: lanes that read it apart could otherwise leave a
// loop whose warp-wide sum the others still wait in.
__device__ __forceinline__ bool warp_flag(const uint32_t* f) {
  return __any_sync(FULLMASK, *(const volatile uint32_t*)f != 0) != 0;
}

// Empties `slots` slots of the table and the sort bins.
template <typename KeyT, int T>
__device__ __forceinline__ void clear_table(KeyT* skey, uint32_t* scnt, uint32_t* bins, uint32_t slots) {
  for (uint32_t i = threadIdx.x; i < slots; i += T) {
    skey[i] = ~(KeyT)0;
    scnt[i] = 0;
  }
  for (int i = threadIdx.x; i < (1 << kSortBinBits); i += T) bins[i] = 0;
}

// One chunk item: keys [cb, cb + CH) of a giant bucket are aggregated on chip.
// When their distinct keys fit half the table they are written back over the chunk's
// own slots as (remainder, count) pairs -- remainders in slots [cb, cb + u), counts as
// uint32 from slot cb + CH / 2 on -- and chunk_u = u; otherwise the chunk keeps
// its keys and chunk_u = kChunkRaw.  The bucket item reads the pairs in place of the
// keys, so a heavy k-mer's copies are summed by many CTAs instead of one.  The table is
// empty before and after.
template <typename KeyT, int T>
__device__ __forceinline__ void aggregate_chunk(const BucketArgs& a, KeyT* keys_rw, unsigned long long cb,
                                                uint32_t item, uint32_t beta, KeyT rmask, KeyT* skey,
                                                uint32_t* scnt, uint32_t* s_flag, uint32_t* s_cnt) {
  constexpr int H = BucketCfg<KeyT>::H, CH = BucketCfg<KeyT>::CH;
  constexpr int PF = BucketCfg<KeyT>::PF;
  const KeyT EMPTY = ~(KeyT)0;
  const int tid = threadIdx.x, lane = tid & 31;
  for (uint32_t i0 = 0; i0 < (uint32_t)CH; i0 += PF * T) {
    if (warp_flag(s_flag)) break;
    KeyT rr[PF];
#pragma unroll
    for (int q = 0; q < PF; q++) {
      const uint32_t i = i0 + q * T + tid;
      rr[q] = i < (uint32_t)CH ? keys_rw[cb + i] & rmask : EMPTY;
    }
    uint32_t fresh = 0;
#pragma unroll
    for (int q = 0; q < PF; q++) {
      if (rr[q] == EMPTY) continue;
      const int res = hash_insert<KeyT>(skey, scnt, H - 1, rr[q], 1u);
      if (res == 2) *s_flag = 1;
      fresh += res == 1;
    }
    fresh = __reduce_add_sync(FULLMASK, fresh);
    if (lane == 0 && fresh && atomicAdd(s_cnt, fresh) + fresh > (uint32_t)(H / 2)) *s_flag = 1;
  }
  __syncthreads();
  const bool raw = *(volatile uint32_t*)s_flag != 0;
  uint32_t u = kChunkRaw;
  if (!raw) u = *(volatile uint32_t*)s_cnt;
  __syncthreads();
  if (tid == 0) {
    *s_cnt = 0;  // now the write cursor
    *s_flag = 0;
  }
  __syncthreads();
  uint32_t* pc = reinterpret_cast<uint32_t*>(keys_rw + cb + CH / 2);
  for (uint32_t i0 = 0; i0 < (uint32_t)H; i0 += T) {
    const uint32_t i = i0 + tid;
    const KeyT x = i < (uint32_t)H ? skey[i] : EMPTY;
    const bool occ = x != EMPTY;
    const unsigned m = __ballot_sync(FULLMASK, occ);
    if (!m) continue;
    uint32_t o = 0;
    if (lane == 0) o = atomicAdd(s_cnt, (uint32_t)__popc(m));
    o = __shfl_sync(FULLMASK, o, 0) + __popc(m & lanemask_lt());
    if (occ) {
      if (!raw) {
        keys_rw[cb + o] = x;
        pc[o] = scnt[i];
      }
      skey[i] = EMPTY;
      scnt[i] = 0;
    }
  }
  if (tid == 0) a.chunk_u[item] = u;
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    atomicAdd(&a.gdone[beta], 1u);
    *s_cnt = 0;
  }
}

// A giant bucket's part waits (bounded) until the bucket's chunk items are done and returns the
// entries it will read: the chunks' pairs (or keys, where a chunk stayed raw) and the
// keys after the last chunk; `raws` tells whether any chunk stayed raw.  On expiry it sets
// ERR_LOOKBACK and *s_fail.
template <int CH, int T>
__device__ __forceinline__ uint32_t giant_entries(const BucketArgs& a, uint32_t beta, uint32_t n, uint32_t g0,
                                               uint32_t nch, uint32_t* s_warp, uint32_t* s_fail, bool& raws) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    int spins = 0;
    const int max_spins = spin_limit(a.spin_limit);
    while (ld_acquire_u32(&a.gdone[beta]) < nch) {
      if (++spins >= max_spins) {
        atomicOr(&a.sc->err, ERR_LOOKBACK);
        *s_fail = 1;
        break;
      }
      __nanosleep(spins < 64 ? 32 : 256);
    }
  }
  __syncthreads();
  uint32_t part = 0;
  bool raw = false;
  for (uint32_t j = tid; j < nch; j += T) {
    const uint32_t cu = __ldcg(&a.chunk_u[g0 + j]);
    raw |= cu == kChunkRaw;
    part += cu == kChunkRaw ? (uint32_t)CH : cu;
  }
  raws = __syncthreads_or(raw) != 0;
  uint32_t tot;
  block_exclusive_sum(part, s_warp, tot);
  return tot + (n - nch * (uint32_t)CH);
}

// The remainder range [lo, hi) of part `part` of a giant bucket, by thread 0's view in *s_lo
// and *s_end: quantiles of kSplitSamples of the entries that its parts read.  Every part
// takes the same sample and so the same quantiles; equal ones leave parts empty.  A bucket
// with few entries is its first part's alone.  `samp`: kSplitSamples keys, barriers inside.
// One CTA that made every pass over a giant bucket, 16 equal ranges first, took 2.6 of the
// 3.26 ms of the low-complexity reads (36M windows, buckets of up to 5.7M); with the parts on
// as many CTAs the whole path takes 0.92 ms (1.55 ms with quicker passes of one CTA).
template <typename KeyT>
__device__ __forceinline__ void giant_range(const BucketArgs& a, const KeyT* keys_rw, uint32_t base, uint32_t n_eff,
                                            uint32_t g0, uint32_t nch, uint32_t part, KeyT rmask, KeyT rtop,
                                            KeyT* samp, KeyT* s_lo, KeyT* s_end) {
  static_assert(kSplitSamples % kGiantParts == 0, "quantiles are samples");
  constexpr uint32_t PER = kSplitSamples / kGiantParts;
  constexpr int CH = BucketCfg<KeyT>::CH;
  const uint32_t tid = threadIdx.x;
  if (n_eff <= (uint32_t)BucketCfg<KeyT>::H / 2) {
    if (tid == 0) {
      *s_lo = (KeyT)0;
      *s_end = part ? (KeyT)0 : rtop;
    }
    __syncthreads();
    return;
  }
  KeyT mine = 0;
  if (tid < (uint32_t)kSplitSamples) {
    const uint32_t j = (uint32_t)(((unsigned long long)tid * nch) / kSplitSamples);
    const uint32_t len = min(__ldcg(&a.chunk_u[g0 + j]), (uint32_t)CH);  // raw: all of them
    const uint32_t e = len ? (tid * 2654435761u >> 8) % len : 0u;
    mine = ldcg_key(keys_rw + ((unsigned long long)base + (unsigned long long)j * CH + e)) & rmask;
    samp[tid] = mine;
  }
  if (tid == 0) {
    *s_lo = (KeyT)0;
    *s_end = rtop;
  }
  __syncthreads();
  if (tid < (uint32_t)kSplitSamples) {
    uint32_t rank = 0;
    for (uint32_t j = 0; j < (uint32_t)kSplitSamples; j++) {
      const KeyT o = samp[j];
      rank += (o < mine || (o == mine && j < tid)) ? 1u : 0u;
    }
    if (part && rank == part * PER) *s_lo = mine;
    if (rank == (part + 1) * PER) *s_end = mine;  // never reached by the last part
  }
  __syncthreads();
  if (tid < (uint32_t)kSplitSamples) samp[tid] = 0;  // the sort bins again
  __syncthreads();
}

// One hash pass of a giant bucket's sub-range [lo, hi): every warp takes whole chunks of
// pairs (their counts are read only inside the sub-range), then the CTA reads the chunks that
// stayed raw (`raws`: there are any) and the tail keys together.  Loads go through L2, as
// other CTAs wrote the pairs during this kernel: four in flight a thread.
template <typename KeyT, int T>
__device__ __forceinline__ void giant_pass(const BucketArgs& a, const KeyT* keys_rw, uint32_t base, uint32_t n,
                                           uint32_t g0, uint32_t nch, bool raws, bool whole, KeyT lo, KeyT hi,
                                           KeyT rmask, KeyT* skey, uint32_t* scnt, uint32_t hmask, uint32_t ulimit,
                                           uint32_t* bins, int dsh, uint32_t bmask, uint32_t* s_ovf,
                                           uint32_t* s_unew) {
  constexpr int GP = 4;  // loads in flight
  constexpr int CH = BucketCfg<KeyT>::CH;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // entries [i, len) of the chunk at cb, `step` apart, GP at a time
  auto read = [&](unsigned long long cb, uint32_t i0, uint32_t len, uint32_t step, bool pairs) {
    const uint32_t* pc = reinterpret_cast<const uint32_t*>(keys_rw + cb + CH / 2);
    KeyT r[GP];
    uint32_t c[GP];
#pragma unroll
    for (int q = 0; q < GP; q++) {
      const uint32_t i = i0 + q * step;
      r[q] = i < len ? ldcg_key(keys_rw + cb + i) & rmask : ~(KeyT)0;
    }
#pragma unroll
    for (int q = 0; q < GP; q++) {
      const bool in = r[q] != ~(KeyT)0 && (whole || (!(r[q] < lo) && r[q] < hi));
      c[q] = in ? 1u : 0u;
      if (in && pairs) c[q] = __ldcg(pc + i0 + q * step);
    }
    uint32_t fresh = 0;
#pragma unroll
    for (int q = 0; q < GP; q++) {
      if (!c[q]) continue;
      const int res = hash_insert<KeyT>(skey, scnt, hmask, r[q], c[q]);
      if (res == 2) *s_ovf = 1;
      if (res == 1) {
        atomicAdd(&bins[sort_bin<KeyT>(r[q], dsh, bmask)], 1u);
        fresh++;
      }
    }
    fresh = __reduce_add_sync(FULLMASK, fresh);
    if (lane == 0 && fresh && atomicAdd(s_unew, fresh) + fresh > ulimit) *s_ovf = 1;
  };
  for (uint32_t j = warp; j < nch; j += T / 32) {
    const uint32_t len = __ldcg(&a.chunk_u[g0 + j]);
    if (len == kChunkRaw) continue;
    for (uint32_t i0 = 0; i0 < len; i0 += 32 * GP) {
      if (warp_flag(s_ovf)) break;
      read((unsigned long long)base + (unsigned long long)j * CH, i0 + lane, len, 32, true);
    }
  }
  for (uint32_t j = raws ? 0 : nch; j <= nch; j++) {
    if (j < nch && __ldcg(&a.chunk_u[g0 + j]) != kChunkRaw) continue;
    const uint32_t len = j < nch ? (uint32_t)CH : n - nch * (uint32_t)CH;
    for (uint32_t i0 = 0; i0 < len; i0 += GP * T) {
      if (warp_flag(s_ovf)) break;
      read((unsigned long long)base + (unsigned long long)j * CH, i0 + tid, len, T, false);
    }
  }
}

// Asks for the keys [p, q) in L2 (whole 16-byte units of them, at most a megabyte).
template <typename KeyT>
__device__ __forceinline__ void prefetch_l2(const KeyT* p, const KeyT* q) {
  const unsigned long long a = ((unsigned long long)__cvta_generic_to_global(p) + 15) & ~15ull;
  const unsigned long long b = (unsigned long long)__cvta_generic_to_global(q) & ~15ull;
  if (a >= b) return;
  const uint32_t n = (uint32_t)min(b - a, 1ull << 20);
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(n) : "memory");
}

// Exclusive prefix of the sort bins in place (one barrier inside, one after); *s_crowd is
// set when a bin holds more than kBinMax elements.
__device__ __forceinline__ void scan_bins(uint32_t* bins, uint32_t* s_warp, uint32_t* s_crowd) {
  constexpr int NT = (1 << kSortBinBits) / 4;  // threads that take four bins each
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint4 v = make_uint4(0, 0, 0, 0);
  uint32_t x = 0, sum = 0;
  if (tid < NT) {
    v = reinterpret_cast<const uint4*>(bins)[tid];
    sum = v.x + v.y + v.z + v.w;
    if (max(max(v.x, v.y), max(v.z, v.w)) > (uint32_t)kBinMax) *s_crowd = 1;
    x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(FULLMASK, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
  }
  __syncthreads();
  if (tid < NT) {
    uint32_t ex = x - sum;
    for (int w = 0; w < warp; w++) ex += s_warp[w];
    reinterpret_cast<uint4*>(bins)[tid] = make_uint4(ex, ex + v.x, ex + v.x + v.y, ex + v.x + v.y + v.z);
  }
  __syncthreads();
}

// Per bucket: aggregate the bucket's keys into (remainder, count) in an on-chip hash
// table, order the distinct remainders and write them as table rows at the bucket's own
// key range [bstart, bstart + u) ("sparse" table: no inter-bucket dependency).
// Sub-ranges of the bucket are counted one at a time, in key order.  A sub-range is an
// interval [lo, hi) of remainders.  The first split guesses from the distinct/keys ratio
// seen so far; a sub-range whose distinct keys overflow the on-chip table is cut at
// quantiles of a sample of its distinct keys, so skewed buckets (a heavy k-mer and its
// error variants) split evenly.
//
// The distinct keys never leave their slots: a counting sort by their top bits (its
// histogram taken as keys are first inserted) orders slot numbers, and each element's
// rank among its bin, a few keys, gives its row.  Nothing is carried in registers from
// one phase to the next, so 1536 threads fit an SM, which is what hides the hash table's
// shared-memory latency; a bucket takes seven barriers, and the slots it emptied are the
// occupied ones, by the same order.  Bound: issue and shared-memory latency of the
// insertions.  Bacterial reads (254M keys, 45M distinct): 1.97 -> 1.62 ms against sorting
// slots held in registers, 512 threads and 17 barriers a bucket.  The next bucket's keys are
// asked for in L2 while this one's rows are ordered (64-bit keys: whole path 4.19 -> 4.15 ms;
// 128-bit keys: no change; asked for a bucket earlier: less).
template <typename KeyT, bool GIANT, int T>
__global__ void __launch_bounds__(T, 2) k_bucket_table(BucketArgs a) {
  using SM = BucketSmem<KeyT>;
  constexpr int H = SM::H;
  static_assert(H <= BucketCfg<KeyT>::CH, "a chunk's pairs: keys in its first half, counts in its second");
  constexpr int BINS = SM::BINS;
  constexpr int HALF = H / 2;
  constexpr int PF = BucketCfg<KeyT>::PF;
  extern __shared__ __align__(16) unsigned char smem[];
  KeyT* skey = reinterpret_cast<KeyT*>(smem + SM::off_key);
  uint32_t* scnt = reinterpret_cast<uint32_t*>(smem + SM::off_cnt);
  uint16_t* ord = reinterpret_cast<uint16_t*>(smem + SM::off_ord);
  uint32_t* bins = reinterpret_cast<uint32_t*>(smem + SM::off_bin);
  uint32_t* shist = reinterpret_cast<uint32_t*>(smem + SM::off_hist);
  __shared__ uint32_t s_warp[33];
  __shared__ uint32_t s_tk, s_nb[2], s_ovf, s_fail, s_unew, s_crowd;
  __shared__ int s_sp;
  // starts of the pending sub-ranges, the next one last; each ends where the one before it
  // in the list starts (the first at the end of the remainder range)
  __shared__ KeyT s_lo[kBucketStack];
  __shared__ KeyT s_split[kSplitWays];
  __shared__ KeyT s_end;       // end of a giant bucket's part
  __shared__ uint32_t s_before;  // rows of the parts before it
  __shared__ float s_ratio, s_size;  // expected distinct keys and table slots per key
  __shared__ uint32_t s_bsmall[kSmallCounts];  // the current bucket's rows by small count

  const int tid = threadIdx.x, lane = tid & 31;
  const int B = 1 << a.bbits;
  const int rem = 2 * a.k - a.bbits;  // remainder bits below the bucket id
  const KeyT rmask = KeyOps<KeyT>::mask(rem);
  const KeyT rtop = KeyOps<KeyT>::shl((KeyT)1, rem);  // end of the remainder range
  const KeyT EMPTY = ~(KeyT)0;
  const KeyT* __restrict__ keys = reinterpret_cast<const KeyT*>(a.keys);
  KeyT* __restrict__ tkeys = reinterpret_cast<KeyT*>(a.tkeys);

  // Two instantiations are launched back to back and exactly one of them works: GIANT
  // = false when the partition has no giant bucket (it carries none of their code, so
  // the common case keeps its registers), GIANT = true otherwise, taking the chunk
  // items first and then every bucket, so the giant buckets' own passes overlap the
  // other buckets.
  const uint32_t ng = a.gfirst ? a.sc->n_chunk_items : 0u;
  if ((ng != 0) != GIANT) return;
  const uint32_t nci = GIANT ? ng : 0u;
  const uint32_t first_bucket = GIANT ? nci + kGiantParts * a.sc->n_giants : 0u;
  const uint32_t nt = first_bucket + (uint32_t)B;
  uint32_t* ticket = &a.sc->ticket_bucket;
  KeyT* keys_rw = reinterpret_cast<KeyT*>(a.keys);

  const int hbins = a.t < kTableHist ? a.t : kTableHist;
  for (int i = tid; i < hbins; i += T) shist[i] = 0;
  if (tid < kSmallCounts) s_bsmall[tid] = 0;
  clear_table<KeyT, T>(skey, scnt, bins, H);

  // Work tickets: the chunk items of giant buckets first (tickets [0, nci)), then their
  // parts, then the other buckets.  A part waits (bounded) until its bucket's chunks are
  // reduced, and before it writes rows until the parts before it have counted theirs: items
  // of earlier tickets, held by CTAs that wait on still earlier ones, so the waits end.
  // Thread 0 takes the next ticket when a bucket starts and its extent once the bucket's keys
  // are in, so neither is waited for between buckets.
  uint32_t next_t = 0, next_base = 0, next_end = 0;
  bool have_extent = true;
  auto take_ticket = [&]() {
    next_t = atomicAdd(ticket, 1u);
    have_extent = false;
  };
  auto take_extent = [&]() {
    if (have_extent) return;
    have_extent = true;
    if ((!GIANT || next_t >= first_bucket) && next_t < nt) {
      next_base = a.bstart[next_t - first_bucket];
      next_end = a.bstart[next_t - first_bucket + 1];
    }
  };
  // thread 0: the next item and its first sub-ranges
  auto publish = [&]() {
    take_extent();
    s_tk = next_t;
    s_nb[0] = next_base;
    s_nb[1] = next_end;
    s_fail = 0;
    s_ovf = 0;
    s_unew = 0;
    s_crowd = 0;
  };
  const int slog_max = rem < 4 ? rem : 4;  // initial split guess (<= 16 sub-ranges)
  auto push_first = [&](uint32_t n_eff) {
    int slog = 0;
    while (slog < slog_max && (float)(n_eff >> slog) * s_ratio * 1.2f > (float)HALF) slog++;
    int sp = 0;
    for (int j = (1 << slog) - 1; j >= 0; j--) s_lo[sp++] = KeyOps<KeyT>::shl((KeyT)(uint32_t)j, rem - slog);
    s_sp = sp;
  };
  if (tid == 0) {
    // running distinct/keys ratio of this CTA's buckets; read sets at 20x-80x coverage
    // with sub-percent errors start near 0.2 (a high guess splits the first buckets
    // needlessly).  The first bucket's table is sized as if every key were distinct.
    s_ratio = 0.2f;
    s_size = 2.5f;
    take_ticket();
    publish();
    if (!GIANT && next_t < nt) push_first(next_end - next_base);
  }
  __syncthreads();
  while (true) {
    const uint32_t tk = s_tk;
    if (tk >= nt) break;
    if (tid == 0) take_ticket();
    if (GIANT && tk < nci) {
      __syncthreads();
      if (tid == 0) {
        const uint32_t gb = a.chunk_bucket[tk];
        s_nb[0] = gb;
        s_nb[1] = a.bstart[gb] + (tk - a.gfirst[gb]) * (uint32_t)BucketCfg<KeyT>::CH;
      }
      __syncthreads();
      aggregate_chunk<KeyT, T>(a, keys_rw, s_nb[1], tk, s_nb[0], rmask, skey, scnt, &s_ovf, &s_unew);
      __syncthreads();
      if (tid == 0) publish();
      __syncthreads();
      continue;
    }
    // a giant bucket is counted by its parts, one remainder range each; a part reads the
    // chunks' pairs (or keys, where a chunk stayed raw) and the keys after the last chunk;
    // n_eff = entries it reads
    const bool part = GIANT && tk < first_bucket;
    const uint32_t item = tk - nci;  // of a part: its place in gpart
    const uint32_t beta = part ? a.glist[item / kGiantParts] : tk - first_bucket;
    const uint32_t base = part ? a.bstart[beta] : s_nb[0];
    const uint32_t all = (part ? a.bstart[beta + 1] : s_nb[1]) - base;
    const uint32_t g0 = part ? a.gfirst[beta] : 0u;
    const uint32_t nch = GIANT ? a.gcount[beta] : 0u;
    const bool elsewhere = GIANT && !part && nch;  // counted by its parts
    uint32_t n = elsewhere ? 0u : all;
    uint32_t n_eff = n;
    bool failed = false, raws = false;
    if (GIANT) {
      __syncthreads();
      if (part) n_eff = giant_entries<BucketCfg<KeyT>::CH, T>(a, beta, n, g0, nch, s_warp, &s_fail, raws);
      failed = s_fail != 0;  // a giant bucket whose chunks did not finish in time
      if (part && !failed) {
        giant_range<KeyT>(a, keys_rw, base, n_eff, g0, nch, item % kGiantParts, rmask, rtop,
                          reinterpret_cast<KeyT*>(bins), &s_lo[0], &s_end);
        if (s_lo[0] == s_end) n = 0;
      }
      if (tid == 0) {
        if (part) {
          s_sp = 1;
        } else {
          s_end = rtop;
          push_first(n_eff);
        }
      }
      __syncthreads();
    }
    if (!GIANT && n == 0) __syncthreads();  // every thread has read this item before the next is published
    uint32_t acc = 0, before = 0;  // rows written so far; of a part, those before it
    bool placed = !part;
    // a part's first row follows the parts before it; the rows up to its own end (`rows` of
    // its own, when it is known to end with them) are published for the parts after it
    unsigned long long* const word = part ? a.gpart + item : nullptr;
    auto place = [&]() {
      if (tid == 0) {
        unsigned long long w = kLbIncl;
        if (item % kGiantParts) {
          // the parts before may have hundreds of sub-ranges to count, one part after the
          // other, so the limit holds for the time in which no part gets through one
          int spins = 0;
          const int max_spins = spin_limit(a.spin_limit);
          uint32_t beats = 0;  // at the last time that the limit was reached
          while ((w = ld_relaxed(word - 1)) == 0) {
            if (++spins >= max_spins) {
              const uint32_t now = *(const volatile uint32_t*)&a.sc->part_beats;
              if (now == beats) {
                atomicOr(&a.sc->err, ERR_LOOKBACK);
                break;
              }
              beats = now;
              spins = 0;
            }
            __nanosleep(spins < 64 ? 32 : 256);
          }
        }
        s_before = (uint32_t)(w & kLbVal);
      }
      __syncthreads();
      before = s_before;
      acc = before;
      placed = true;
    };
    int attempts = 0;
    while (n && !failed) {
      const int sp = s_sp;
      if (++attempts > kMaxBucketAttempts) { failed = true; break; }
      const KeyT lo = s_lo[sp - 1];
      const KeyT hi = sp > 1 ? s_lo[sp - 2] : GIANT ? s_end : rtop;
      const bool whole = lo == (KeyT)0 && hi == rtop;
      // bits below the interval's common prefix (all its keys share the bits above)
      const KeyT span = lo ^ (hi - (KeyT)1);
      const int psh = span == (KeyT)0 ? 0 : KeyOps<KeyT>::top_bit(span) + 1;
      const int dsh = psh < kSortBinBits ? 0 : psh - kSortBinBits;
      const uint32_t bmask = psh < kSortBinBits ? (1u << psh) - 1u : (uint32_t)BINS - 1u;
      // table sized for the distinct keys expected (2.5x), at least 1024 slots; an
      // overflow of a smaller table than H takes all H, one of H splits the sub-range
      uint32_t Heff = 1024;
      {
        const float uest = (float)n_eff * s_size;
        while ((float)Heff < uest && Heff < (uint32_t)H) Heff <<= 1;
        if (!whole) Heff = H;
      }
      const uint32_t hmask = Heff - 1;
      // --- hash aggregation of this sub-range; it stops as soon as the distinct keys
      //     exceed half the table
      const uint32_t ulimit = Heff / 2;
      if (GIANT && part)
        giant_pass<KeyT, T>(a, keys_rw, base, n, g0, nch, raws, whole, lo, hi, rmask, skey, scnt, hmask, ulimit, bins,
                            dsh, bmask, &s_ovf, &s_unew);
      if (GIANT && part && tid == 0) atomicAdd(&a.sc->part_beats, 1u);
      for (uint32_t i0 = 0; i0 < n && !(GIANT && part); i0 += PF * T) {
        if (warp_flag(&s_ovf)) break;
        KeyT rr[PF];
#pragma unroll
        for (int q = 0; q < PF; q++) {
          const uint32_t i = i0 + q * T + tid;
          rr[q] = i < n ? (keys[base + i] & rmask) : EMPTY;
        }
        uint32_t fresh = 0;  // distinct keys this thread added in this round
#pragma unroll
        for (int q = 0; q < PF; q++) {
          const KeyT r = rr[q];
          if (r != EMPTY && (whole || (!(r < lo) && r < hi))) {
            const int res = hash_insert<KeyT>(skey, scnt, hmask, r, 1u);
            if (res == 2) s_ovf = 1;
            if (res == 1) {
              atomicAdd(&bins[sort_bin<KeyT>(r, dsh, bmask)], 1u);
              fresh++;
            }
          }
        }
        // the distinct-key count grows once per warp and round (one shared atomic per
        // new key cost 7 % of the kernel)
        fresh = __reduce_add_sync(FULLMASK, fresh);
        if (lane == 0 && fresh && atomicAdd(&s_unew, fresh) + fresh > ulimit) s_ovf = 1;
      }
      __syncthreads();
      if (s_ovf) {
        if (Heff == (uint32_t)H) {
          // cut [lo, hi) at quantiles of a sample of the distinct keys in the table
          // (one per sampling thread: the first occupied slot of its stride)
          KeyT* samp = reinterpret_cast<KeyT*>(bins);
          KeyT mine = EMPTY;
          if (tid < kSplitSamples)
            for (int i = tid; i < H && mine == EMPTY; i += kSplitSamples) mine = skey[i];
          __syncthreads();  // the bins' last use in this attempt was the insertion
          if (tid < kSplitSamples) samp[tid] = mine;
          const int m = __syncthreads_count(mine != EMPTY);
          const int ways = m < kSplitWays ? m : kSplitWays;
          if (mine != EMPTY) {
            int rank = 0;
            for (int j = 0; j < kSplitSamples; j++) {
              const KeyT o = samp[j];
              rank += (o != EMPTY && o < mine);
            }
            // splitter w (1 <= w < ways) is the sample of rank floor(w * m / ways)
            for (int w = 1; w < ways; w++)
              if (rank == (w * m) / ways) s_split[w] = mine;
          }
          __syncthreads();
          if (tid == 0) {
            if (ways < 2 || sp - 1 + ways > kBucketStack) {
              s_fail = 1;
            } else {
              // the pieces take the sub-range's place, highest first, so the lowest is next
              int o = sp - 1;
              for (int w = ways - 1; w >= 1; w--) s_lo[o++] = s_split[w];
              s_lo[o++] = lo;
              s_sp = o;
            }
          }
          __syncthreads();
          failed = s_fail != 0;
        } else if (tid == 0) {
          s_size = (float)H;  // the same sub-range again, on all H slots
        }
        __syncthreads();
        clear_table<KeyT, T>(skey, scnt, bins, Heff);
        if (tid == 0) {
          s_ovf = 0;
          s_unew = 0;
        }
        __syncthreads();
        continue;
      }
      const uint32_t u = s_unew;
      if (tid == 0) {
        take_extent();
        if (sizeof(KeyT) == 8 && next_t >= first_bucket && next_t < nt) prefetch_l2(keys + next_base, keys + next_end);
      }
      if (GIANT && !placed) place();
      if (GIANT && part && sp == 1 && tid == 0) st_relaxed(word, kLbIncl | (acc + u));
      // --- order the u distinct remainders: slot numbers go to their bins, in any order
      scan_bins(bins, s_warp, &s_crowd);
      for (uint32_t i = tid; i < Heff; i += T) {
        const KeyT x = skey[i];
        if (x != EMPTY) ord[atomicAdd(&bins[sort_bin<KeyT>(x, dsh, bmask)], 1u)] = (uint16_t)i;
      }
      __syncthreads();  // bins now hold their ends
      const KeyT hi_bits = KeyOps<KeyT>::shl((KeyT)beta, rem);
      if (!s_crowd) {
        // element i of the binned order lands at row b0 + rank, within its bin's rows, so
        // neighbouring threads store to neighbouring rows
        for (uint32_t i = tid; i < u; i += T) {
          const uint32_t slot = ord[i];
          const KeyT x = skey[slot];
          const uint32_t bi = sort_bin<KeyT>(x, dsh, bmask);
          const uint32_t b0 = bi ? bins[bi - 1] : 0u, b1 = bins[bi];
          uint32_t rank = 0;
          for (uint32_t j = b0; j < b1; j++) rank += skey[ord[j]] < x;
          emit_row<KeyT>(a, tkeys, (unsigned long long)base + acc + b0 + rank, hi_bits | x, scnt[slot], shist,
                         s_bsmall);
        }
      } else {
        // a bin above kBinMax: a bitonic sort of the slot numbers by key (0xffff: above all)
        uint32_t P = 2;
        while (P < u) P <<= 1;
        for (uint32_t i = u + tid; i < P; i += T) ord[i] = 0xffffu;
        __syncthreads();
        for (uint32_t k2 = 2; k2 <= P; k2 <<= 1) {
          for (uint32_t j2 = k2 >> 1; j2 > 0; j2 >>= 1) {
            for (uint32_t i = tid; i < P / 2; i += T) {
              const uint32_t x = 2 * i - (i & (j2 - 1)), y = x | j2;
              const uint32_t sx = ord[x], sy = ord[y];
              const KeyT kx = sx == 0xffffu ? EMPTY : skey[sx], ky = sy == 0xffffu ? EMPTY : skey[sy];
              if ((ky < kx) == ((x & k2) == 0) && kx != ky) {
                ord[x] = (uint16_t)sy;
                ord[y] = (uint16_t)sx;
              }
            }
            __syncthreads();
          }
        }
        for (uint32_t i = tid; i < u; i += T) {
          const uint32_t slot = ord[i];
          emit_row<KeyT>(a, tkeys, (unsigned long long)base + acc + i, hi_bits | skey[slot], scnt[slot], shist,
                         s_bsmall);
        }
      }
      acc += u;
      __syncthreads();
      // --- empty the table for the next sub-range or bucket
      for (uint32_t i = tid; i < u; i += T) {
        const uint32_t slot = ord[i];
        skey[slot] = EMPTY;
        scnt[slot] = 0;
      }
      for (int i = tid; i < BINS; i += T) bins[i] = 0;
      if (sp == 1) break;
      if (tid == 0) {
        s_sp = sp - 1;
        s_unew = 0;
        s_crowd = 0;
      }
      __syncthreads();
    }
    if (GIANT && part && (failed || n == 0)) {  // nothing was published yet
      if (!placed) place();
      if (tid == 0) st_relaxed(word, kLbIncl | acc);
    }
    if (failed) {
      if (tid == 0) atomicOr(&a.sc->err, ERR_BUCKET);
      acc = 0;
      before = 0;
    }
    // the bucket's rows by small count (every row was emitted before the last barrier):
    // stored for the kept filter and folded into the count histogram (counts below t)
    if (tid < kSmallCounts) {
      const uint32_t c = s_bsmall[tid];
      uint32_t* bs = a.bsmall + (size_t)beta * kSmallCounts + tid;
      if (part) {
        if (c) atomicAdd(bs, c);
      } else if (a.bsmall && !elsewhere) {
        *bs = c;
      }
      if (c && tid < a.t) atomicAdd(&shist[tid], c);
      s_bsmall[tid] = 0;
    }
    if (tid == 0) {
      // of a giant bucket the last part knows all rows
      if (!elsewhere && (!part || item % kGiantParts == kGiantParts - 1)) a.tu[beta] = acc;
      if (n) {
        atomicAdd(&a.sc->n_unique, (unsigned long long)(acc - before));
        if (!part) s_ratio = 0.5f * s_ratio + 0.5f * ((float)acc / (float)n_eff);
        s_size = 2.5f * s_ratio;
      }
      publish();
      if (!GIANT && next_t < nt) push_first(next_end - next_base);
    }
    __syncthreads();
  }
  __syncthreads();
  for (int i = tid; i < hbins; i += T)
    if (shist[i]) atomicAdd(&a.hist[i], (unsigned long long)shist[i]);
}

// Dense copy of the sparse table: rows of bucket b move to doff[b] (exclusive prefix
// of tu).  mode 0: keys + counts arrays; mode 1: packed KmerPairs records.
template <typename KeyT>
__global__ void __launch_bounds__(256) k_compact_rows(const KeyT* __restrict__ skeys,
                                                      const uint32_t* __restrict__ scounts,
                                                      const uint32_t* __restrict__ bstart,
                                                      const uint32_t* __restrict__ tu,
                                                      const uint32_t* __restrict__ doff, int B,
                                                      KeyT* __restrict__ dkeys,
                                                      uint32_t* __restrict__ dcounts,
                                                      uint32_t* __restrict__ packed, int mode) {
  constexpr int WORDS = (sizeof(KeyT) + 4) / 4;
  for (int b = blockIdx.x; b < B; b += gridDim.x) {
    const uint32_t src = bstart[b], dst = doff[b], u = tu[b];
    for (uint32_t i = threadIdx.x; i < u; i += blockDim.x) {
      const KeyT x = skeys[src + i];
      const uint32_t c = scounts[src + i];
      if (mode == 0) {
        dkeys[dst + i] = x;
        dcounts[dst + i] = c;
      } else {
        uint32_t* o = packed + (size_t)(dst + i) * WORDS;
#pragma unroll
        for (int w = 0; w < WORDS - 1; w++) o[w] = (uint32_t)(x >> (32 * w));
        o[WORDS - 1] = c;
      }
    }
  }
}

// ------------------------------------------------------ histogram (other t) / cutoff --
// Rows by count below t, read in place: bucket b's rows are [bstart[b], bstart[b] + tu[b]).
__global__ void __launch_bounds__(256) k_histogram(const uint32_t* __restrict__ tcounts,
                                                   const uint32_t* __restrict__ bstart,
                                                   const uint32_t* __restrict__ tu, int B, int t,
                                                   unsigned long long* hist) {
  __shared__ uint32_t sh[kHistSmem];
  const int hb = t < kHistSmem ? t : kHistSmem;
  for (int i = threadIdx.x; i < hb; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  for (int b = blockIdx.x; b < B; b += gridDim.x) {
    const uint32_t r0 = bstart[b], u = tu[b];
    for (uint32_t i = threadIdx.x; i < u; i += blockDim.x) {
      const uint32_t c = tcounts[r0 + i];
      if (c < (uint32_t)t) {
        if (c < (uint32_t)kHistSmem) atomicAdd(&sh[c], 1u);
        else atomicAdd(&hist[c], 1ull);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < hb; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], (unsigned long long)sh[i]);
}

// cutoff = first minimum of hist[1..t) (t == 1 -> 1); kept = U - sum(hist[1..cutoff))
__global__ void __launch_bounds__(1024) k_cutoff(const unsigned long long* __restrict__ hist, int t,
                                                 Scalars* sc) {
  __shared__ unsigned long long s_v[32];
  __shared__ int s_i[32];
  unsigned long long best = ~0ull;
  int bi = 0x7fffffff;
  for (int c = 1 + threadIdx.x; c < t; c += blockDim.x) {
    unsigned long long v = hist[c];
    if (v < best || (v == best && c < bi)) { best = v; bi = c; }
  }
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long v2 = __shfl_down_sync(FULLMASK, best, o);
    int i2 = __shfl_down_sync(FULLMASK, bi, o);
    if (v2 < best || (v2 == best && i2 < bi)) { best = v2; bi = i2; }
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { s_v[warp] = best; s_i[warp] = bi; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); w++)
      if (s_v[w] < best || (s_v[w] == best && s_i[w] < bi)) { best = s_v[w]; bi = s_i[w]; }
    const int cut = t > 1 ? bi : 1;
    unsigned long long below = 0;
    for (int c = 1; c < cut && c < t; c++) below += hist[c];
    sc->cutoff = (uint32_t)cut;
    sc->n_kept = sc->n_unique - below;
  }
}

// ----------------------------------------------------------------- macro-nodes -------
template <typename KeyT>
struct MnCfg;
template <>
struct MnCfg<uint64_t> {  // with 256 threads; 128 and 192 threads were 5 to 20 % slower
  static constexpr int CTAS = 6;  // CTAs per SM
};
template <>
struct MnCfg<u128> {
  static constexpr int CTAS = 5;
};

template <typename KeyT>
struct MnSmem {
  static constexpr int CAP = kMnCap;
  static constexpr size_t off_key = 0;
  static constexpr size_t off_cnt = off_key + sizeof(KeyT) * CAP;
  static constexpr size_t off_bin = off_cnt + sizeof(uint32_t) * CAP;
  static constexpr size_t off_ord = off_bin + sizeof(uint16_t) * CAP;
  static constexpr size_t merge_bytes = off_ord + sizeof(uint16_t) * CAP;
  // joined units: node rows, suffix-side node keys, first suffix item of every bin
  static constexpr size_t off_rows = 0;
  static constexpr size_t off_pkey = off_rows + 32 * (kMnJoin + 32);
  static constexpr size_t off_start = off_pkey + sizeof(KeyT) * kMnJoin;
  static constexpr size_t join_bytes = (off_start + sizeof(uint16_t) * (kMnBins + 1) + 15) / 16 * 16;
  static constexpr size_t bytes = merge_bytes > join_bytes ? merge_bytes : join_bytes;
  static_assert(CAP <= 2048, "item numbers have 11 bits");
};

__device__ __forceinline__ uint64_t shfl_xor_key(uint64_t x, int o) {
  return __shfl_xor_sync(FULLMASK, (unsigned long long)x, o);
}
__device__ __forceinline__ u128 shfl_xor_key(u128 x, int o) {
  return ((u128)shfl_xor_key((uint64_t)(x >> 64), o) << 64) | shfl_xor_key((uint64_t)x, o);
}
__device__ __forceinline__ uint64_t shfl_key(uint64_t x, int l) {
  return __shfl_sync(FULLMASK, (unsigned long long)x, l);
}
__device__ __forceinline__ u128 shfl_key(u128 x, int l) {
  return ((u128)shfl_key((uint64_t)(x >> 64), l) << 64) | shfl_key((uint64_t)x, l);
}

template <typename KeyT>
__device__ __forceinline__ uint32_t lower_bound_s(const KeyT* k, uint32_t lo, uint32_t hi, KeyT x) {
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (k[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}
template <typename KeyT>
__device__ __forceinline__ uint32_t upper_bound_s(const KeyT* k, uint32_t lo, uint32_t hi, KeyT x) {
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (!(x < k[mid])) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Counts of table rows [q, q+4) (one 16-byte load when the four rows lie inside the
// count buffer) and the mask of those rows that are inside [r0, e) and kept.
__device__ __forceinline__ uint32_t kept_group(const FilterArgs& a, uint32_t q, uint32_t r0, uint32_t e,
                                               uint32_t cut, uint32_t c[4]) {
  c[0] = c[1] = c[2] = c[3] = 0;
  if (q >= e) return 0;
  if ((unsigned long long)q + 4 <= a.trows) {
    const uint4 v = *reinterpret_cast<const uint4*>(a.tcounts + q);
    c[0] = v.x; c[1] = v.y; c[2] = v.z; c[3] = v.w;
  } else {
#pragma unroll
    for (int t = 0; t < 4; t++)
      if ((unsigned long long)q + t < a.trows) c[t] = a.tcounts[q + t];
  }
  uint32_t m = 0;
#pragma unroll
  for (int t = 0; t < 4; t++)
    if (q + t >= r0 && q + t < e && c[t] >= cut) m |= 1u << t;
  return m;
}

// Kept rows (count >= cutoff) of every table bucket by reading its counts, one warp per
// bucket: where the table kernel's histogram of small counts does not tell (a cutoff above
// it, or a table that did not come from that kernel).
__device__ __forceinline__ bool small_counts_tell(const FilterArgs& a, uint32_t cut) {
  return a.bsmall && cut <= (uint32_t)kSmallCounts;
}

__global__ void __launch_bounds__(256) k_kept_count(FilterArgs a) {
  const uint32_t cut = a.sc->cutoff;
  if (small_counts_tell(a, cut)) return;
  const int lane = threadIdx.x & 31;
  const uint32_t B = 1u << a.bbits, warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < B; b += warps) {
    const uint32_t r0 = a.bstart[b], e = r0 + a.tu[b];
    uint32_t v = 0;
    for (uint32_t g = r0 & ~3u; g < e; g += 128) {
      uint32_t c[4];
      v += __popc(kept_group(a, g + 4 * lane, r0, e, cut, c));
    }
    v = __reduce_add_sync(FULLMASK, v);
    if (lane == 0) a.kcount[b] = v;
  }
}

// Kept rows and their prefix over the buckets, one bucket per thread: a bucket keeps its
// rows minus those counted fewer than cutoff times.  One look-back per 256 buckets, where
// one per bucket inside the filter cost it 0.20 against 0.17 ms (bacterial) and 1.21
// against 0.82 ms (46M kept 63-mers), offsets included.
constexpr int kKeptT = 256;
__global__ void __launch_bounds__(kKeptT) k_kept_offsets(FilterArgs a) {
  __shared__ uint32_t s_warp[33];
  __shared__ uint32_t s_tile;
  __shared__ unsigned long long s_before;
  const uint32_t cut = a.sc->cutoff;
  const uint32_t B = 1u << a.bbits, tiles = (B + kKeptT - 1) / kKeptT;
  if (threadIdx.x == 0) s_tile = atomicAdd(&a.sc->ticket_filter, 1u);
  __syncthreads();
  const uint32_t tile = s_tile, b = tile * kKeptT + threadIdx.x;
  uint32_t v = 0;
  if (b < B) {
    if (small_counts_tell(a, cut)) {
      uint32_t below = 0;
      const uint4* h = reinterpret_cast<const uint4*>(a.bsmall + (size_t)b * kSmallCounts);
      for (uint32_t q = 0; 4 * q < cut; q++) {  // counts 4q .. 4q + 3 (no row counts 0)
        const uint4 c = h[q];
        below += (4 * q > 0 ? c.x : 0u) + (4 * q + 1 < cut ? c.y : 0u) + (4 * q + 2 < cut ? c.z : 0u) +
                 (4 * q + 3 < cut ? c.w : 0u);
      }
      v = a.tu[b] - below;
    } else {
      v = a.kcount[b];
    }
  }
  uint32_t tot;
  const uint32_t ex = block_exclusive_sum(v, s_warp, tot);
  if (threadIdx.x < 32) {
    if (threadIdx.x == 0) st_relaxed(&a.flags[tile], (tile ? kLbAgg : kLbIncl) | (unsigned long long)tot);
    __syncwarp();
    const unsigned long long before = lookback_exclusive((int)tile, &a.sc->err, a.spin_limit,
                                                         [&](int j, unsigned long long& x) {
      const unsigned long long f = ld_relaxed(&a.flags[j]);
      x = f & kLbVal;
      return (unsigned)(f >> 62);
    });
    if (threadIdx.x == 0) {
      if (tile) st_relaxed(&a.flags[tile], kLbIncl | (before + tot));
      s_before = before;
    }
  }
  __syncthreads();
  if (b < B) {
    a.kstart[b] = (uint32_t)s_before + ex;
    a.kcount[b] = v;
  }
}

// Kept rows (count >= cutoff) of every table bucket, written densely in key order --
// the k-mers construct_kmer_histogram hands to macro-node construction -- from the bucket's
// offset (kstart) on, and ksub (kept rows whose next two key bits are < 1, 2, 3).
// One warp per table bucket, with no waits between buckets.  Lane l takes the rows
// [g + 4l, g + 4l + 4) of each 128-row step, with g aligned to four rows, so one 16-byte load
// brings its four counts and lane order is row order.  Bound: the wait for its loads, counts
// and then keys; the next step's counts are under way while this step's keys are waited for:
// 1 Mbp, 30x, whole path 0.748 -> 0.722 ms; bacterial 4.15 -> 4.13 ms (eight rows a lane: 0.736
// and 4.12 ms).  Six CTAs an SM: bacterial 4.105 -> 4.092 ms against the five that its 48
// registers would leave; eight 4.103 ms.
template <typename KeyT>
__global__ void __launch_bounds__(256, 6) k_filter_kept(FilterArgs a) {
  const int lane = threadIdx.x & 31;
  const uint32_t B = 1u << a.bbits, warps = gridDim.x * (blockDim.x >> 5);
  const int rem = 2 * a.k - a.bbits;
  const uint32_t cut = a.sc->cutoff;
  const KeyT* __restrict__ tkeys = reinterpret_cast<const KeyT*>(a.tkeys);
  KeyT* __restrict__ kkeys = reinterpret_cast<KeyT*>(a.kkeys);
  for (uint32_t beta = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; beta < B; beta += warps) {
    const uint32_t r0 = a.bstart[beta], e = r0 + a.tu[beta];
    uint32_t pos = a.kstart[beta];
    uint32_t dl0 = 0, dl1 = 0, dl2 = 0;
    uint32_t next[4];
    auto fetch = [&](uint32_t q) {  // counts of rows [q, q + 4); nothing past the bucket
      if (q >= e) return;
      if ((unsigned long long)q + 4 <= a.trows) {
        const uint4 v = *reinterpret_cast<const uint4*>(a.tcounts + q);
        next[0] = v.x; next[1] = v.y; next[2] = v.z; next[3] = v.w;
      } else {
#pragma unroll
        for (int t = 0; t < 4; t++)
          if ((unsigned long long)q + t < a.trows) next[t] = a.tcounts[q + t];
      }
    };
    const uint32_t g0 = r0 & ~3u;
    fetch(g0 + 4 * lane);
    for (uint32_t g = g0; g < e; g += 128) {
      const uint32_t q = g + 4 * lane;
      uint32_t c[4], m = 0;
#pragma unroll
      for (int t = 0; t < 4; t++) {
        c[t] = next[t];
        if (q + t >= r0 && q + t < e && (unsigned long long)q + t < a.trows && c[t] >= cut) m |= 1u << t;
      }
      KeyT x[4];
#pragma unroll
      for (int t = 0; t < 4; t++)
        if ((m >> t) & 1u) x[t] = tkeys[q + t];
      fetch(q + 128);
      const uint32_t n = __popc(m);
      uint32_t inc = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULLMASK, inc, o);
        if (lane >= o) inc += y;
      }
      uint32_t o = pos + inc - n;
#pragma unroll
      for (int t = 0; t < 4; t++) {
        if (!((m >> t) & 1u)) continue;
        if (o < a.cap) {
          kkeys[o] = x[t];
          a.kcounts[o] = c[t];
        } else {
          atomicOr(&a.sc->err, ERR_BOUNDS);
        }
        o++;
        const uint32_t d2 = (uint32_t)(KeyOps<KeyT>::shr(x[t], rem - 2) & 3);
        dl0 += d2 == 0;
        dl1 += d2 == 1;
        dl2 += d2 == 2;
      }
      pos += __shfl_sync(FULLMASK, inc, 31);
    }
    dl0 = __reduce_add_sync(FULLMASK, dl0);
    dl1 = __reduce_add_sync(FULLMASK, dl1);
    dl2 = __reduce_add_sync(FULLMASK, dl2);
    if (lane == 0) {
      a.ksub[3 * beta + 0] = dl0;
      a.ksub[3 * beta + 1] = dl0 + dl1;
      a.ksub[3 * beta + 2] = dl0 + dl1 + dl2;
    }
  }
}

// Node key of kept row `row` as seen from stream `st`: the prefix (k-1)-mer x >> 2 for
// the suffix-side stream (st == 0), the suffix (k-1)-mer for the others.
template <typename KeyT>
__device__ __forceinline__ KeyT node_key(const KeyT* __restrict__ kk, uint32_t row, int st,
                                         KeyT succ_mask) {
  const KeyT x = kk[row];
  return st == 0 ? (x >> 2) : (x & succ_mask);
}

// first row in [lo, hi) whose node key is > piv
template <typename KeyT>
__device__ uint32_t upper_bound_rows(const KeyT* __restrict__ kk, uint32_t lo, uint32_t hi, int st,
                                     KeyT succ_mask, KeyT piv) {
  while (lo < hi) {
    uint32_t mid = (lo + hi) >> 1;
    if (!(piv < node_key(kk, mid, st, succ_mask))) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Rows of stream st (0: suffix side, 1 + f: prefix side of first base f) of node unit beta,
// the node keys whose top bbits - x bits are beta: stream 0 is the kept rows of table
// buckets [beta << x, (beta + 1) << x); stream 1 + f the kept rows whose leading base is f
// and whose next bits are beta -- whole table buckets when x >= 2, else the half or quarter
// of one bucket that its next-digit offsets mark.  Contiguous kept rows each.
__device__ __forceinline__ void mn_extent(const MnArgs& a, uint32_t beta, int st, uint32_t& r0, uint32_t& r1) {
  const int x = a.xbits;
  if (st == 0) {
    const uint32_t b0 = beta << x, b1 = b0 + (1u << x) - 1;
    r0 = a.kstart[b0];
    r1 = a.kstart[b1] + a.kcount[b1];
    return;
  }
  const uint32_t lead = (uint32_t)(st - 1) << (a.bbits - 2);
  if (x >= 2) {
    const uint32_t b0 = lead | (beta << (x - 2)), b1 = b0 + (1u << (x - 2)) - 1;
    r0 = a.kstart[b0];
    r1 = a.kstart[b1] + a.kcount[b1];
    return;
  }
  const int part = 2 - x;  // bits of beta below the bucket's own
  const uint32_t bp = lead | (beta >> part);
  const uint32_t d0 = (beta & ((1u << part) - 1u)) << x, d1 = d0 + (1u << x);  // of four digits
  const uint32_t b0 = a.kstart[bp];
  r0 = b0 + (d0 ? a.ksub[3 * bp + d0 - 1] : 0u);
  r1 = b0 + (d1 == 4 ? a.kcount[bp] : a.ksub[3 * bp + d1 - 1]);
}

// Units of more rows than one segment holds: counted ahead of all others, by the first
// tickets of the macro-node kernel, so that no other unit waits for a long one.
__device__ __forceinline__ bool mn_big(uint32_t rows, uint32_t fit) { return rows > fit; }
__global__ void __launch_bounds__(256) k_mn_big(MnArgs a, uint32_t fit) {
  const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= 1u << (a.bbits - a.xbits)) return;
  uint32_t rows = 0;
  for (int st = 0; st < 5; st++) {
    uint32_t r0, r1;
    mn_extent(a, u, st, r0, r1);
    if (r1 <= a.kcap && r0 <= r1) rows += r1 - r0;
  }
  if (mn_big(rows, fit)) a.big[atomicAdd(&a.sc->n_big, 1u)] = u;
}

// Per node unit: the suffix-side stream (node = x >> 2, extension = last base) and four
// prefix-side streams (node = x & SUCC_MASK, extension = first base) are each sorted by node
// key; merged they give the unit's macro-nodes in key order.  A unit larger than CAP
// rows is processed in segments split at node-key pivots.
//
// Units whose prefix-side items nearly all find their node on the suffix side are joined by
// lookup (see below); the others are sorted.  There a counting sort on the bits below the unit's
// prefix orders item numbers; an item's rank among its bin (two or three items) is its
// place.  Node heads are ballots, and the thread of a head collects its node's up to eight
// items and stores the node's three rows whole.
//
// Bound: the wait for the units before (without it 8.6M nodes take 0.21 ms and 46M 63-mer
// nodes 1.5 ms): all units in flight wait for the slowest of them, so a lookup is a binary
// search in its bin.  Scanning the bin, a unit of repeats took up to 48 thousand cycles
// against 14 thousand on average, and the 46M nodes 3.54 instead of 2.2 ms.  Bacterial nodes
// (8.6M): 0.39 -> 0.23 ms, 46M nodes of 63-mers 6.95 -> 3.54 ms, against sorting every unit,
// assembling nodes by 4-byte stores into zeroed rows and looking back over single units.
template <typename KeyT>
__global__ void __launch_bounds__(kMnThreads, MnCfg<KeyT>::CTAS) k_macro_nodes(MnArgs a) {
  using SM = MnSmem<KeyT>;
  constexpr int T = kMnThreads, NW = T / 32, CAP = kMnCap, NCH = CAP / 32, JCH = kMnJoin / 32;
  static_assert(JCH <= NCH && JCH <= 32, "a joined unit's chunks");
  extern __shared__ __align__(16) unsigned char smem[];
  KeyT* ikey = reinterpret_cast<KeyT*>(smem + SM::off_key);
  uint32_t* icnt = reinterpret_cast<uint32_t*>(smem + SM::off_cnt);
  // item numbers (low 11 bits) and tags (0-3: suffix by last base, 4-7: prefix by first)
  uint16_t* binned = reinterpret_cast<uint16_t*>(smem + SM::off_bin);  // in bin order
  uint16_t* ord = reinterpret_cast<uint16_t*>(smem + SM::off_ord);     // in node order
  __shared__ uint32_t s_warp[33];
  __shared__ uint32_t s_off[6], s_cur[5], s_end[5], s_segend[5], s_ncur[5], s_nend[5], s_nbeta, s_ntask;
  __shared__ uint32_t s_last, s_nodes;
  __shared__ unsigned long long s_NO;
  __shared__ uint32_t s_bin[kMnBins];  // offset (low 16 bits) and fill (high 16 bits)
  __shared__ uint32_t s_head[NCH], s_first[NCH];  // per 32 positions: head ballot, heads before
  // a joined unit's items whose node has no suffix side
  __shared__ uint32_t s_extra, s_xcnt[32];
  __shared__ KeyT s_xkey[32];
  __shared__ uint8_t s_xf[32];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ubits = a.bbits - a.xbits;
  const uint32_t Bu = 1u << ubits;  // node units
  const int k = a.k;
  const int nb = 2 * (k - 1);
  const KeyT succ_mask = KeyOps<KeyT>::mask(nb);
  const KeyT KINF = ~(KeyT)0;  // above every (k-1)-mer key
  const KeyT* __restrict__ kk = reinterpret_cast<const KeyT*>(a.kkeys);
  KeyT* __restrict__ nkeys = reinterpret_cast<KeyT*>(a.nkeys);
  constexpr uint32_t FIT = kMnFit;  // rows per segment before ties
  // every node key of a unit shares its top ubits bits; the sort bins are the next
  // (at most kMnBinBits) bits
  const int rbits = nb - ubits > 0 ? nb - ubits : 0;
  const int dbits = rbits < kMnBinBits ? rbits : kMnBinBits;
  const int bsh = rbits - dbits;
  const uint32_t bmask = (1u << dbits) - 1u;

  // kept rows beyond the kept buffers, or without a place, were not written: nothing to
  // merge.  (A wait that runs out in this kernel sets the flag too; the units left are taken
  // by the CTAs that run.)
  if (tid == 0) s_nbeta = a.sc->err & (ERR_BOUNDS | ERR_LOOKBACK);
  __syncthreads();
  if (s_nbeta) return;
  __syncthreads();

  // the next ticket's unit and extents, by one warp: first the big units' counts, then
  // every unit in order.  Its rows are asked for in L2 (bacterial path 4.137 -> 4.114 ms)
  const uint32_t nbig = a.sc->n_big;
  auto take_unit = [&]() {
    uint32_t t = 0;
    __syncwarp();
    if (lane == 0) t = atomicAdd(&a.sc->ticket_mn, 1u);
    t = __shfl_sync(FULLMASK, t, 0);
    const uint32_t u = t < nbig ? a.big[t] : t - nbig;
    uint32_t r0 = 0, r1 = 0;
    if (u < Bu && lane < 5) {
      mn_extent(a, u, lane, r0, r1);
      if (r1 > a.kcap || r0 > r1) {  // never read past the kept rows
        atomicOr(&a.sc->err, ERR_BOUNDS);
        r0 = r1 = 0;
      }
    }
    if (lane < 5) {
      prefetch_l2(kk + r0, kk + r1);
      prefetch_l2(a.kcounts + r0, a.kcounts + r1);
      s_ncur[lane] = r0;
      s_nend[lane] = r1;
    }
    if (lane == 0) {
      s_nbeta = u;
      s_ntask = t < nbig;
    }
  };
  if (warp == NW - 1) take_unit();
  __syncthreads();

  while (true) {
    const uint32_t beta = s_nbeta;
    if (beta >= Bu) break;
    // ---- joined units: almost every node has a suffix side (a k-mer starts with it), and
    //      the suffix-side stream is those nodes in order.  Each prefix-side item looks its
    //      node up there, so nothing has to be sorted but the few items whose node has no
    //      suffix side (up to 32; dead ends of the graph).
    const uint32_t c0 = s_ncur[0], n0 = s_nend[0] - c0;
    const uint32_t p1 = s_nend[1] - s_ncur[1], p2 = p1 + s_nend[2] - s_ncur[2], p3 = p2 + s_nend[3] - s_ncur[3],
                   np = p3 + s_nend[4] - s_ncur[4];
    if (n0 > 0 && n0 <= (uint32_t)kMnJoin && np <= (uint32_t)kMnJoin) {
      constexpr int IT = kMnJoin / T;
      uint32_t* rows = reinterpret_cast<uint32_t*>(smem + SM::off_rows);
      KeyT* pkey = reinterpret_cast<KeyT*>(smem + SM::off_pkey);
      uint16_t* start = reinterpret_cast<uint16_t*>(smem + SM::off_start);
      uint32_t scnt[IT], pcnt[IT], pfirst[IT], sbase = 0;  // sbase: last bases, two bits each
      KeyT py[IT];
#pragma unroll
      for (int q = 0; q < IT; q++) {  // prefix side: node key, count, first base
        const uint32_t i = q * T + tid;
        py[q] = 0;
        pcnt[q] = pfirst[q] = 0;
        if (i < np) {
          const int st = (i >= p1) + (i >= p2) + (i >= p3);
          const uint32_t row = s_ncur[st + 1] + (i - (st == 0 ? 0u : st == 1 ? p1 : st == 2 ? p2 : p3));
          py[q] = kk[row] & succ_mask;
          pcnt[q] = a.kcounts[row];
          pfirst[q] = st;
        }
      }
#pragma unroll
      for (int q = 0; q < IT; q++) {  // suffix side: heads, and the first item of every bin
        const uint32_t i = q * T + tid;
        bool head = false;
        scnt[q] = 0;
        if (i < n0) {
          const KeyT x = kk[c0 + i], y = x >> 2;
          scnt[q] = a.kcounts[c0 + i];
          sbase |= (uint32_t)(x & 3) << (2 * q);
          pkey[i] = y;
          uint32_t b = 0;  // bins below the item's that no item before it is in or above
          head = i == 0;
          if (i) {
            const KeyT z = kk[c0 + i - 1] >> 2;
            head = !(z == y);
            b = ((uint32_t)KeyOps<KeyT>::shr(z, bsh) & bmask) + 1;
          }
          const uint32_t mine = (uint32_t)KeyOps<KeyT>::shr(y, bsh) & bmask;
          for (; b <= mine; b++) start[b] = (uint16_t)i;
          if (i == n0 - 1)
            for (b = mine + 1; b <= bmask + 1; b++) start[b] = (uint16_t)n0;
        }
        const unsigned m = __ballot_sync(FULLMASK, head);
        if (lane == 0) s_head[q * NW + warp] = m;
      }
      for (uint32_t i = tid; i < 2 * (n0 + 32); i += T) reinterpret_cast<uint4*>(rows)[i] = make_uint4(0, 0, 0, 0);
      if (tid == 0) s_extra = 0;
      __syncthreads();
      uint32_t at[IT];
#pragma unroll
      for (int q = 0; q < IT; q++) {
        at[q] = n0;
        if (q * T + tid < np) {
          const uint32_t b = (uint32_t)KeyOps<KeyT>::shr(py[q], bsh) & bmask;
          const uint32_t i = lower_bound_s(pkey, start[b], start[b + 1], py[q]);
          if (i < n0 && pkey[i] == py[q]) at[q] = i;
          if (at[q] == n0) {  // a node of its own
            const uint32_t x = atomicAdd(&s_extra, 1u);
            if (x < 32) {
              s_xkey[x] = py[q];
              s_xcnt[x] = pcnt[q];
              s_xf[x] = (uint8_t)pfirst[q];
            }
          }
        }
      }
      __syncthreads();
      const uint32_t E = s_extra;
      if (E <= 32) {
        // heads before every 32 suffix items (lane c of each warp holds chunk c)
        const uint32_t mask = lane < JCH ? s_head[lane] : 0u;
        uint32_t inc = __popc(mask);
#pragma unroll
        for (int o = 1; o < JCH; o <<= 1) {
          const uint32_t y = __shfl_up_sync(FULLMASK, inc, o);
          if (lane >= o) inc += y;
        }
        const uint32_t heads = __shfl_sync(FULLMASK, inc, JCH - 1);
        auto heads_to = [&](uint32_t i) {  // heads among suffix items [0, i] (all lanes call it)
          const uint32_t ch = min(i >> 5, (uint32_t)JCH - 1u);
          const uint32_t m = __shfl_sync(FULLMASK, mask, ch), to = __shfl_sync(FULLMASK, inc, ch) - __popc(m);
          return to + __popc(m & ((2u << (i & 31)) - 1u));
        };
        // nodes that only prefix-side items name, one item per lane: the first of each key,
        // the heads below it and its rank among them
        uint32_t xheads = 0, xrank = 0;
        unsigned xfirst = 0;
        KeyT xk = 0;
        if (E) {
          const bool have = (uint32_t)lane < E;
          xk = have ? s_xkey[lane] : KINF;
          bool dup = false;
          for (uint32_t j = 0; j < E; j++) {
            const KeyT o = shfl_key(xk, j);  // every lane takes part
            dup |= j < (uint32_t)lane && o == xk;
          }
          xfirst = __ballot_sync(FULLMASK, have && !dup);
          for (uint32_t j = 0; j < E; j++) {
            const KeyT o = shfl_key(xk, j);
            xrank += ((xfirst >> j) & 1u) != 0 && o < xk ? 1u : 0u;
          }
          uint32_t i = 0;
          if (have) {
            const uint32_t b = (uint32_t)KeyOps<KeyT>::shr(xk, bsh) & bmask;
            i = lower_bound_s(pkey, start[b], start[b + 1], xk);
          }
          const uint32_t h = heads_to(i ? i - 1 : 0u);
          xheads = i ? h : 0u;
        }
        const uint32_t nodes = heads + __popc(xfirst);
        auto place = [&](uint32_t h) {  // node of the head of rank h (all lanes call it)
          uint32_t n = h;
          for (uint32_t j = 0; j < E; j++) {
            const uint32_t o = __shfl_sync(FULLMASK, xheads, j);
            n += ((xfirst >> j) & 1u) != 0 && o <= h ? 1u : 0u;
          }
          return n;
        };
        if (warp == 0) {
          const unsigned long long ex = group_lookback(GroupFlags(a.flags, Bu), beta, nodes,
                                                       (int)beta != a.withhold_unit, &a.sc->err, a.spin_limit);
          if (lane == 0) s_NO = ex;
          if ((uint32_t)lane < E) rows[8 * (xheads + xrank) + 4 + s_xf[lane]] = s_xcnt[lane];
        }
        uint32_t node[IT];
#pragma unroll
        for (int q = 0; q < IT; q++) {
          const uint32_t i = q * T + tid;
          node[q] = place(heads_to(i) - 1u);
          if (i < n0) rows[8 * node[q] + ((sbase >> (2 * q)) & 3u)] = scnt[q];
          const uint32_t t = place(heads_to(at[q]) - 1u);
          if (i < np && at[q] < n0) rows[8 * t + 4 + pfirst[q]] = pcnt[q];
        }
        __syncthreads();
        const unsigned long long q0 = s_NO;
        if (warp == NW - 1) take_unit();
        if (q0 + nodes <= a.cap) {
#pragma unroll
          for (int q = 0; q < IT; q++) {
            const uint32_t i = q * T + tid;
            if (i < n0 && ((s_head[i >> 5] >> (i & 31)) & 1u)) nkeys[q0 + node[q]] = pkey[i];
          }
          if (warp == 0 && ((xfirst >> lane) & 1u)) nkeys[q0 + xheads + xrank] = xk;
          for (uint32_t i = tid; i < 2 * nodes; i += T)
            reinterpret_cast<uint4*>(i & 1 ? a.npre : a.nsuf)[q0 + (i >> 1)] = reinterpret_cast<const uint4*>(rows)[i];
        } else if (tid == 0) {
          atomicOr(&a.sc->err, ERR_MN_CAPACITY);
        }
        if (tid == 0 && beta == Bu - 1) a.sc->n_nodes = q0 + nodes;
        __syncthreads();
        continue;
      }
    }
    // ---- sorted units, in segments: a count task only counts its nodes (and publishes
    //      them), a big unit's place is known before its segments are written, and a unit of
    //      one segment looks for its place once that is counted
    const bool task = s_ntask != 0;
    const bool big = mn_big(n0 + np, FIT);
    if (tid < 5) {
      s_cur[tid] = s_ncur[tid];
      s_end[tid] = s_nend[tid];
    }
    if (big && !task && warp == 0) {
      const unsigned long long ex = group_lookback(GroupFlags(a.flags, Bu), beta, ~0ull,
                                                   (int)beta != a.withhold_unit, &a.sc->err, a.spin_limit);
      if (lane == 0) s_NO = ex;
    }
    unsigned long long NO = 0, done_nodes = 0;
    while (true) {
      // ---- choose this segment's rows: everything left, or rows up to a pivot key;
      //      lane st of warp 0 handles stream st
      if (warp == 0) {
        __syncwarp();
        const uint32_t c0 = lane < 5 ? s_cur[lane] : 0u, c1 = lane < 5 ? s_end[lane] : 0u;
        const uint32_t rows = __reduce_add_sync(FULLMASK, c1 - c0);
        uint32_t e = c1;
        if (rows > FIT) {
          KeyT piv = KINF;
          const uint32_t take = (uint32_t)((float)(c1 - c0) * (0.9f * (float)FIT / (float)rows));
          if (take >= 1) piv = node_key(kk, c0 + take - 1, lane, succ_mask);
          for (int o = 4; o > 0; o >>= 1) {  // the least of lanes 0..4 (the others hold KINF)
            const KeyT y = shfl_xor_key(piv, o);
            if (y < piv) piv = y;
          }
          piv = shfl_key(piv, 0);
          if (lane < 5 && piv != KINF) e = upper_bound_rows(kk, c0, c1, lane, succ_mask, piv);
        }
        const unsigned more = __ballot_sync(FULLMASK, e != c1);
        uint32_t inc = e - c0;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          const uint32_t y = __shfl_up_sync(FULLMASK, inc, o);
          if (lane >= o) inc += y;
        }
        if (lane < 5) {
          s_segend[lane] = e;
          s_off[lane + 1] = inc;
        }
        if (lane == 0) {
          s_off[0] = 0;
          s_last = more == 0;
        }
      }
      for (int b = tid; b < kMnBins; b += T) s_bin[b] = 0;
      __syncthreads();
      const bool last = s_last != 0;
      uint32_t mm = s_off[5];
      if (mm > (uint32_t)CAP) {  // cannot happen with FIT-sized segments
        if (tid == 0) atomicOr(&a.sc->err, ERR_MN_CAPACITY);
        mm = 0;
      }
      // ---- gather the five sorted runs, counted by sort bin
      const uint32_t o1 = s_off[1], o2 = s_off[2], o3 = s_off[3], o4 = s_off[4];
      for (uint32_t i = tid; i < mm; i += T) {
        const int st = (i >= o1) + (i >= o2) + (i >= o3) + (i >= o4);
        const uint32_t row = s_cur[st] + (i - s_off[st]);
        const KeyT x = kk[row];
        const KeyT y = st == 0 ? (x >> 2) : (x & succ_mask);
        ikey[i] = y;
        icnt[i] = a.kcounts[row];
        ord[i] = (uint16_t)(i | ((st == 0 ? (uint32_t)(x & 3) : (uint32_t)(3 + st)) << 11));
        atomicAdd(&s_bin[(uint32_t)KeyOps<KeyT>::shr(y, bsh) & bmask], 1u);
      }
      __syncthreads();
      // ---- order of the items by node key, ties by run and then position (the stable
      //      merge of the five runs)
      {
        constexpr int BPT = (kMnBins + T - 1) / T;
        uint32_t hv[BPT], hs = 0, hm = 0;
#pragma unroll
        for (int q = 0; q < BPT; q++) {
          const int bi = tid * BPT + q;
          hv[q] = bi < kMnBins ? s_bin[bi] : 0u;
          hs += hv[q];
          hm = max(hm, hv[q]);
        }
        uint32_t tot;
        uint32_t ex = block_exclusive_sum(hs, s_warp, tot);
#pragma unroll
        for (int q = 0; q < BPT; q++) {
          const int bi = tid * BPT + q;
          if (bi < kMnBins) s_bin[bi] = ex;
          ex += hv[q];
        }
        const bool crowded = __syncthreads_or(hm > (uint32_t)kMnBinMax) != 0;
        if (!crowded) {
          for (uint32_t i = tid; i < mm; i += T) {
            const uint32_t o = atomicAdd(&s_bin[(uint32_t)KeyOps<KeyT>::shr(ikey[i], bsh) & bmask], 1u << 16);
            binned[(o & 0xffffu) + (o >> 16)] = ord[i];
          }
          __syncthreads();
          for (uint32_t p = tid; p < mm; p += T) {
            const uint32_t v = binned[p], i = v & 2047u;
            const KeyT x = ikey[i];
            const uint32_t o = s_bin[(uint32_t)KeyOps<KeyT>::shr(x, bsh) & bmask];
            const uint32_t b0 = o & 0xffffu, b1 = b0 + (o >> 16);
            uint32_t rank = 0;
            for (uint32_t j = b0; j < b1; j++) {
              const uint32_t ij = binned[j] & 2047u;
              const KeyT y = ikey[ij];
              rank += (y < x || (!(x < y) && ij < i)) ? 1u : 0u;
            }
            ord[b0 + rank] = (uint16_t)v;
          }
        } else {
          // a crowded bin: merge ranks across the runs
          for (uint32_t i = tid; i < mm; i += T) binned[i] = ord[i];
          __syncthreads();
          for (uint32_t i = tid; i < mm; i += T) {
            const int st = (i >= o1) + (i >= o2) + (i >= o3) + (i >= o4);
            const KeyT x = ikey[i];
            uint32_t rank = i - s_off[st];
            for (int b = 0; b < 5; b++) {
              if (b == st) continue;
              const uint32_t lo = s_off[b], hi = s_off[b + 1];
              rank += (b < st ? upper_bound_s(ikey, lo, hi, x) : lower_bound_s(ikey, lo, hi, x)) - lo;
            }
            ord[rank] = binned[i];
          }
        }
      }
      __syncthreads();
      // ---- node heads: one ballot per 32 positions
      const uint32_t nch = (mm + 31) / 32;
      for (uint32_t ch = warp; ch < nch; ch += NW) {
        const uint32_t r = 32 * ch + lane;
        bool head = false;
        if (r < mm) head = r == 0 || !(ikey[ord[r - 1] & 2047u] == ikey[ord[r] & 2047u]);
        const unsigned m = __ballot_sync(FULLMASK, head);
        if (lane == 0) s_head[ch] = m;
      }
      __syncthreads();
      if (warp == 0) {  // heads before each 32 positions, and the unit's place
        uint32_t run = 0;
        for (uint32_t c0 = 0; c0 < nch; c0 += 32) {
          const uint32_t n = c0 + lane < nch ? __popc(s_head[c0 + lane]) : 0u;
          uint32_t inc = n;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULLMASK, inc, o);
            if (lane >= o) inc += y;
          }
          if (c0 + lane < nch) s_first[c0 + lane] = run + inc - n;
          run += __shfl_sync(FULLMASK, inc, 31);
        }
        if (lane == 0) s_nodes = run;
        if (!big) {
          // A withheld unit (bounded-wait tests) publishes nothing: its successors' waits
          // run out and report ERR_LOOKBACK.
          const unsigned long long ex = group_lookback(GroupFlags(a.flags, Bu), beta, run,
                                                       (int)beta != a.withhold_unit, &a.sc->err, a.spin_limit);
          if (lane == 0) s_NO = ex;
        }
      }
      __syncthreads();
      const uint32_t nodes = s_nodes;
      // the unit's place is published: the next one is taken while this one is written
      if (last && warp == NW - 1) take_unit();
      if (!task) {
        NO = s_NO;
        const unsigned long long q0 = NO + done_nodes;
        if (q0 + nodes <= a.cap) {
          for (uint32_t ch = warp; ch < nch; ch += NW) {
            const uint32_t m = s_head[ch];
            if (!((m >> lane) & 1u)) continue;
            uint32_t r = 32 * ch + lane;
            const unsigned long long q = q0 + s_first[ch] + __popc(m & lanemask_lt());
            uint32_t v = ord[r];
            nkeys[q] = ikey[v & 2047u];
            uint32_t c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
            do {
              const uint32_t n = icnt[v & 2047u], tag = v >> 11;
#pragma unroll
              for (int e = 0; e < 8; e++)
                if (tag == (uint32_t)e) c[e] = n;
              r++;
              if (r >= mm || ((s_head[r >> 5] >> (r & 31)) & 1u)) break;
              v = ord[r];
            } while (true);
            reinterpret_cast<uint4*>(a.nsuf)[q] = make_uint4(c[0], c[1], c[2], c[3]);
            reinterpret_cast<uint4*>(a.npre)[q] = make_uint4(c[4], c[5], c[6], c[7]);
          }
        } else if (tid == 0) {
          atomicOr(&a.sc->err, ERR_MN_CAPACITY);
        }
      }
      done_nodes += nodes;
      __syncthreads();
      if (last) break;
      if (tid < 5) s_cur[tid] = s_segend[tid];
      __syncthreads();
    }
    if (tid == 0) {
      if (task) {
        if ((int)beta != a.withhold_unit) group_publish(GroupFlags(a.flags, Bu), beta, done_nodes);
      } else if (beta == Bu - 1) {
        a.sc->n_nodes = NO + done_nodes;
      }
    }
  }
}

// ------------------------------------------------------- loaded (external) tables --
// Bucket extents of a dense ascending table: bstart[b] = first row whose key's top
// `bbits` bits are >= b, tu[b] = rows of bucket b (the sparse layout with no gaps).
template <typename KeyT>
__global__ void __launch_bounds__(256) k_table_bounds(const KeyT* __restrict__ keys, unsigned long long n,
                                                      int bbits, int rem, uint32_t* bstart) {
  const int B = 1 << bbits;
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > B) return;
  unsigned long long lo = 0, hi = n;
  if (b == B) {
    lo = n;
  } else {
    const KeyT x = KeyOps<KeyT>::shl((KeyT)(uint32_t)b, rem);
    while (lo < hi) {
      const unsigned long long mid = (lo + hi) >> 1;
      if (keys[mid] < x) lo = mid + 1; else hi = mid;
    }
  }
  bstart[b] = (uint32_t)lo;
}

// Rows of a loaded table checked, summed and histogrammed in one read: every row a k-mer
// (below 4^k), above the row before it, with a count.  The first bad row (and the first
// rule it breaks) comes back as 4 * row + rule in chk[0] (all ones: none), the counts' sum
// in chk[1]; hist gets the rows by count below t (null: not wanted).  One read of the rows
// at HBM speed in place of a host loop over them: loading 5.0M rows, taking the cutoff and
// building the graph went from 4460 to 889 us, most of it now the copy from pageable memory.
template <typename KeyT>
__global__ void __launch_bounds__(256) k_table_check(const KeyT* __restrict__ keys,
                                                     const uint32_t* __restrict__ counts, unsigned long long n,
                                                     int k, unsigned long long* __restrict__ chk, int t,
                                                     unsigned long long* __restrict__ hist) {
  __shared__ uint32_t sh[kHistSmem];
  const int hb = hist ? min(t, kHistSmem) : 0;
  for (int i = threadIdx.x; i < hb; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  unsigned long long bad = ~0ull, sum = 0;
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const KeyT x = keys[i];
    const uint32_t c = counts[i];
    unsigned long long rule = 3;
    if (c == 0) rule = 2;
    if (i && !(keys[i - 1] < x)) rule = 1;
    if (KeyOps<KeyT>::shr(x, 2 * k) != (KeyT)0) rule = 0;
    if (rule < 3) bad = min(bad, 4 * i + rule);
    sum += c;
    if (hist && c < (uint32_t)t) {
      if (c < (uint32_t)kHistSmem) atomicAdd(&sh[c], 1u);
      else atomicAdd(&hist[c], 1ull);
    }
  }
  sum = warp_sum_u64(sum);
  if ((threadIdx.x & 31) == 0 && sum) atomicAdd(&chk[1], sum);
  if (bad != ~0ull) atomicMin(&chk[0], bad);
  __syncthreads();
  for (int i = threadIdx.x; i < hb; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], (unsigned long long)sh[i]);
}

__global__ void __launch_bounds__(256) k_table_sizes(const uint32_t* bstart, int B, uint32_t* tu) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < B) tu[b] = bstart[b + 1] - bstart[b];
}

// =================================================================== launchers =====
static std::atomic<unsigned long long> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

static int g_sms = 0;
// SM count the calling thread's launches are sized for: a serving worker running a
// request on an SM partition sets it to the partition's SMs (0: the whole device)
static thread_local int t_sms = 0;
void set_thread_sms(int n) { t_sms = n > 0 ? n : 0; }
int thread_sms(int device_sms) { return t_sms > 0 ? t_sms : device_sms; }

static int sm_count() {
  if (t_sms > 0) return t_sms;
  if (!g_sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_sms <= 0) g_sms = 1;
  }
  return g_sms;
}

size_t bucket_smem_bytes(int wide) {
  return wide ? BucketSmem<u128>::bytes : BucketSmem<uint64_t>::bytes;
}
size_t mn_smem_bytes(int wide) { return wide ? MnSmem<u128>::bytes : MnSmem<uint64_t>::bytes; }
int bucket_ctas_per_sm(int) { return 2; }
int mn_ctas_per_sm(int wide) { return wide ? MnCfg<u128>::CTAS : MnCfg<uint64_t>::CTAS; }

cudaError_t launch_line_tiles(const uint8_t* buf, unsigned long long F, uint32_t* tile_nl, Scalars* sc,
                              unsigned long long tile0, unsigned long long ntiles, cudaStream_t st) {
  if (ntiles > 0) pk::note_launch(), k_line_scan<<<(unsigned)ntiles, 256, 0, st>>>(buf, F, tile_nl, sc, tile0);
  return cudaGetLastError();
}

cudaError_t launch_tile_prefix(const CountArgs& a, cudaStream_t st) {
  const int ntiles = (int)((a.F + kTileBytes - 1) / kTileBytes);
  pk::note_launch(), k_tile_prefix<<<1, 1024, 0, st>>>(a.fasta, a.F, a.tile_nl, ntiles, a.sc);
  return cudaGetLastError();
}

cudaError_t launch_line_scan(const CountArgs& a, cudaStream_t st) {
  const unsigned long long ntiles = (a.F + kTileBytes - 1) / kTileBytes;
  cudaError_t e = launch_line_tiles(a.fasta, a.F, a.tile_nl, a.sc, 0, ntiles, st);
  if (e != cudaSuccess) return e;
  return launch_tile_prefix(a, st);
}

template <bool WIDE>
static cudaError_t launch_extract_t(const CountArgs& a, cudaStream_t st) {
  const size_t smem = sizeof(uint32_t) << a.bbits;
  // the attribute is shared by every thread launching this kernel, so it is always
  // set to the largest histogram (15 partition digits), never to this launch's size
  static bool attr_set = false;  // same value from every thread, so a race is benign
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_extract<WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(sizeof(uint32_t) << kHistBits));
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  pk::note_launch(), k_extract<WIDE><<<a.grid, kCountT, smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_bucket_count(const CountArgs& a, int wide, cudaStream_t st) {
  return wide ? launch_extract_t<true>(a, st) : launch_extract_t<false>(a, st);
}

template <typename KeyT>
static cudaError_t launch_coarse_t(const CountArgs& a, const uint32_t* coff, KeyT* out, cudaStream_t st) {
  const size_t smem = CoarseCfg<KeyT>::smem;
  static bool attr_set = false;  // a constant, so concurrent first calls agree
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_scatter_coarse<KeyT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  pk::note_launch(), k_scatter_coarse<KeyT><<<a.grid, CoarseCfg<KeyT>::T, smem, st>>>(a, coff, out);
  return cudaGetLastError();
}

cudaError_t launch_scatter_coarse(const CountArgs& a, const uint32_t* coff, void* out, int wide,
                                  cudaStream_t st) {
  return wide ? launch_coarse_t<u128>(a, coff, reinterpret_cast<u128*>(out), st)
              : launch_coarse_t<uint64_t>(a, coff, reinterpret_cast<uint64_t*>(out), st);
}

cudaError_t launch_coarse_offsets(const CountArgs& a, int pbits, uint32_t* coff, uint32_t* cstart,
                                  uint32_t* slice_start, int slice_keys, uint32_t* bstart, uint32_t* fcur,
                                  cudaStream_t st) {
  pk::note_launch(), k_coarse_offsets<<<a.grid, 256, 0, st>>>(a.counts, a.bstart, a.bbits, pbits, a.cbits, coff, cstart,
                                                              slice_start, slice_keys, bstart, fcur, a.sc);
  return cudaGetLastError();
}

template <typename KeyT, bool FEW>
static cudaError_t launch_fine_n(const KeyT* in, const uint32_t* cstart, const uint32_t* slice_start,
                                 uint32_t* fcur, KeyT* out, int k, int bbits, int cbits, uint32_t* ticket,
                                 unsigned long long cap, uint32_t* err, cudaStream_t st) {
  using FC = FineCfg<KeyT, FEW>;
  static bool attr_set = false;  // a constant, so concurrent first calls agree
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_scatter_fine<KeyT, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)FC::smem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  pk::note_launch(), k_scatter_fine<KeyT, FEW><<<sm_count() * FC::CTAS, FC::T, FC::smem, st>>>(
      in, cstart, slice_start, fcur, out, k, bbits, cbits, ticket, cap, err);
  return cudaGetLastError();
}

template <typename KeyT>
static cudaError_t launch_fine_t(const KeyT* in, const uint32_t* cstart, const uint32_t* slice_start,
                                 uint32_t* fcur, KeyT* out, int k, int bbits, int cbits, uint32_t* ticket,
                                 unsigned long long cap, uint32_t* err, cudaStream_t st) {
  if (bbits - cbits >= 11) {
    const size_t bsmem = FineBigCfg<KeyT>::smem;
    static bool big_attr_set = false;
    if (!big_attr_set) {
      cudaError_t e = cudaFuncSetAttribute(k_scatter_fine_big<KeyT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)bsmem);
      if (e != cudaSuccess) return e;
      big_attr_set = true;
    }
    pk::note_launch(), k_scatter_fine_big<KeyT><<<sm_count(), FineBigCfg<KeyT>::T, bsmem, st>>>(in, cstart, slice_start, fcur, out, k,
                                                                             bbits, cbits, ticket, cap, err);
    return cudaGetLastError();
  }
  return bbits - cbits <= kFewFine ? launch_fine_n<KeyT, true>(in, cstart, slice_start, fcur, out, k, bbits, cbits, ticket,
                                                              cap, err, st)
                                   : launch_fine_n<KeyT, false>(in, cstart, slice_start, fcur, out, k, bbits, cbits,
                                                               ticket, cap, err, st);
}

cudaError_t launch_scatter_fine(const void* in, const uint32_t* cstart, const uint32_t* slice_start,
                                uint32_t* fcur, void* out, int k, int bbits, int cbits, int wide,
                                uint32_t* ticket, unsigned long long cap, uint32_t* err, cudaStream_t st) {
  return wide ? launch_fine_t<u128>(reinterpret_cast<const u128*>(in), cstart, slice_start, fcur,
                                    reinterpret_cast<u128*>(out), k, bbits, cbits, ticket, cap, err, st)
              : launch_fine_t<uint64_t>(reinterpret_cast<const uint64_t*>(in), cstart, slice_start, fcur,
                                        reinterpret_cast<uint64_t*>(out), k, bbits, cbits, ticket, cap, err,
                                        st);
}

cudaError_t launch_fine_count(const void* in, const uint32_t* cstart, const uint32_t* slice_start,
                              uint32_t* bcount, int k, int bbits, int cbits, int wide, uint32_t* ticket,
                              cudaStream_t st) {
  const uint32_t sk = (uint32_t)fine_slice_keys(wide, bbits - cbits);
  if (wide)
    pk::note_launch(), k_fine_count<u128><<<sm_count() * 2, 512, 0, st>>>(reinterpret_cast<const u128*>(in), cstart, slice_start,
                                                      bcount, k, bbits, cbits, ticket, sk);
  else
    pk::note_launch(), k_fine_count<uint64_t><<<sm_count() * 2, 512, 0, st>>>(reinterpret_cast<const uint64_t*>(in), cstart,
                                                          slice_start, bcount, k, bbits, cbits, ticket, sk);
  return cudaGetLastError();
}

cudaError_t launch_prefix(uint32_t* counts, int B, cudaStream_t st) {
  pk::note_launch(), k_bucket_prefix<<<1, 1024, 0, st>>>(counts, B);
  return cudaGetLastError();
}

cudaError_t launch_bucket_offsets(const CountArgs& a, cudaStream_t st) {
  const int B = 1 << a.bbits;
  pk::note_launch(), k_col_prefix<<<(B + 31) / 32, 256, 0, st>>>(a.counts, a.grid, B, a.bstart);
  pk::note_launch(), k_bucket_prefix<<<1, 1024, 0, st>>>(a.bstart, B);
  return cudaGetLastError();
}


template <typename KeyT>
static cudaError_t launch_bucket_t(const BucketArgs& a, int grid, cudaStream_t st) {
  using BC = BucketCfg<KeyT>;
  const size_t smem = BucketSmem<KeyT>::bytes;
  static bool attr_set = false;  // a constant, so concurrent first calls agree
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_bucket_table<KeyT, false, BC::T>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_bucket_table<KeyT, true, BC::TG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  if (grid <= 0) grid = sm_count() * bucket_ctas_per_sm(sizeof(KeyT) == 16);
  // exactly one of the two works (giant buckets present or not); the other returns
  pk::note_launch(), k_bucket_table<KeyT, false, BC::T><<<grid, BC::T, smem, st>>>(a);
  if (a.gfirst) pk::note_launch(), k_bucket_table<KeyT, true, BC::TG><<<grid, BC::TG, smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_bucket_table(const BucketArgs& a, int wide, int grid, cudaStream_t st) {
  return wide ? launch_bucket_t<u128>(a, grid, st) : launch_bucket_t<uint64_t>(a, grid, st);
}

int chunk_keys(int wide) { return wide ? BucketCfg<u128>::CH : BucketCfg<uint64_t>::CH; }

cudaError_t launch_giant_chunks(const BucketArgs& a, int wide, uint32_t* gfirst, uint32_t* gcount,
                                uint32_t* chunk_bucket, uint32_t* glist, cudaStream_t st) {
  const int B = 1 << a.bbits;
  pk::note_launch(), k_giant_chunks<<<(B + 255) / 256, 256, 0, st>>>(a.bstart, B, gfirst, gcount, chunk_bucket, a.gdone,
                                                                    a.gpart, glist, a.bsmall, (uint32_t)chunk_keys(wide), a.sc);
  return cudaGetLastError();
}

size_t giant_part_bytes(unsigned long long keys) {
  return (keys / kGiantKeys + 1) * (kGiantParts * sizeof(unsigned long long) + sizeof(uint32_t));
}

cudaError_t launch_histogram(const uint32_t* tcounts, const uint32_t* bstart, const uint32_t* tu, int B, int t,
                             unsigned long long* hist, cudaStream_t st) {
  const int most = sm_count() * 8, grid = B < most ? B : most;
  pk::note_launch(), k_histogram<<<grid, 256, 0, st>>>(tcounts, bstart, tu, B, t, hist);
  return cudaGetLastError();
}

cudaError_t launch_cutoff(const unsigned long long* hist, int t, Scalars* sc, cudaStream_t st) {
  pk::note_launch(), k_cutoff<<<1, 1024, 0, st>>>(hist, t, sc);
  return cudaGetLastError();
}

size_t mn_flag_words(int bbits) {
  return (size_t)(1u << bbits) + 2 * (((size_t)(1u << bbits) + 31) / 32);
}

template <typename KeyT>
static cudaError_t launch_filter_t(const FilterArgs& a, bool count_rows, cudaStream_t st) {
  const int B = 1 << a.bbits;
  const int most = sm_count() * 8, grid = std::min((B + 7) / 8, most);
  if (count_rows) pk::note_launch(), k_kept_count<<<grid, 256, 0, st>>>(a);
  pk::note_launch(), k_kept_offsets<<<(B + kKeptT - 1) / kKeptT, kKeptT, 0, st>>>(a);
  pk::note_launch(), k_filter_kept<KeyT><<<grid, 256, 0, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_filter_kept(const FilterArgs& a, int wide, bool count_rows, cudaStream_t st) {
  return wide ? launch_filter_t<u128>(a, count_rows, st) : launch_filter_t<uint64_t>(a, count_rows, st);
}

template <typename KeyT>
static cudaError_t launch_mn_t(const MnArgs& a, int grid, cudaStream_t st) {
  const size_t smem = MnSmem<KeyT>::bytes;
  static bool attr_set = false;  // a constant, so concurrent first calls agree
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(k_macro_nodes<KeyT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr_set = true;
  }
  if (grid <= 0) grid = sm_count() * mn_ctas_per_sm(sizeof(KeyT) == 16);
  const unsigned units = 1u << (a.bbits - a.xbits);
  pk::note_launch(), k_mn_big<<<(units + 255) / 256, 256, 0, st>>>(a, kMnFit);
  pk::note_launch(), k_macro_nodes<KeyT><<<grid, kMnThreads, smem, st>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_macro_nodes(const MnArgs& a, int wide, int grid, cudaStream_t st) {
  return wide ? launch_mn_t<u128>(a, grid, st) : launch_mn_t<uint64_t>(a, grid, st);
}

__global__ void __launch_bounds__(1024) k_copy_prefix(const uint32_t* __restrict__ in,
                                                      uint32_t* __restrict__ out, int B) {
  __shared__ uint32_t s_warp[33];
  uint32_t carry = 0;
  for (int base = 0; base < B; base += blockDim.x) {
    int i = base + threadIdx.x;
    uint32_t v = i < B ? in[i] : 0;
    uint32_t tot;
    uint32_t ex = block_exclusive_sum(v, s_warp, tot);
    if (i < B) out[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) out[B] = carry;
}

cudaError_t launch_row_offsets(const uint32_t* tu, uint32_t* doff, int B, cudaStream_t st) {
  pk::note_launch(), k_copy_prefix<<<1, 1024, 0, st>>>(tu, doff, B);
  return cudaGetLastError();
}

cudaError_t launch_compact_rows(const void* tkeys, const uint32_t* tcounts, const uint32_t* bstart,
                                const uint32_t* tu, const uint32_t* doff, int B, int wide,
                                void* dkeys, uint32_t* dcounts, void* packed, cudaStream_t st) {
  int grid = B < sm_count() * 16 ? B : sm_count() * 16;
  if (grid < 1) grid = 1;
  const int mode = packed ? 1 : 0;
  if (wide)
    pk::note_launch(), k_compact_rows<u128><<<grid, 256, 0, st>>>(reinterpret_cast<const u128*>(tkeys), tcounts, bstart,
                                               tu, doff, B, reinterpret_cast<u128*>(dkeys), dcounts,
                                               reinterpret_cast<uint32_t*>(packed), mode);
  else
    pk::note_launch(), k_compact_rows<uint64_t><<<grid, 256, 0, st>>>(reinterpret_cast<const uint64_t*>(tkeys), tcounts,
                                                   bstart, tu, doff, B,
                                                   reinterpret_cast<uint64_t*>(dkeys), dcounts,
                                                   reinterpret_cast<uint32_t*>(packed), mode);
  return cudaGetLastError();
}

}  // namespace pk

namespace pk {
cudaError_t launch_table_check(const void* keys, const uint32_t* counts, unsigned long long n, int k, int wide,
                               unsigned long long* chk, int t, unsigned long long* hist, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  const unsigned long long want = (n + 255) / 256, most = (unsigned long long)sm_count() * 8;
  const unsigned grid = (unsigned)(want < most ? want : most);
  if (wide)
    pk::note_launch(), k_table_check<u128><<<grid, 256, 0, st>>>((const u128*)keys, counts, n, k, chk, t, hist);
  else
    pk::note_launch(), k_table_check<uint64_t><<<grid, 256, 0, st>>>((const uint64_t*)keys, counts, n, k, chk, t, hist);
  return cudaGetLastError();
}

cudaError_t launch_table_bounds(const void* keys, unsigned long long n, int bbits, int k, uint32_t* bstart,
                                uint32_t* tu, int wide, cudaStream_t st) {
  const int B = 1 << bbits;
  const int rem = 2 * k - bbits;
  const int grid = (B + 1 + 255) / 256;
  if (wide) {
    pk::note_launch(), k_table_bounds<u128><<<grid, 256, 0, st>>>((const u128*)keys, n, bbits, rem, bstart);
    pk::note_launch(), k_table_sizes<<<(B + 255) / 256, 256, 0, st>>>(bstart, B, tu);
  } else {
    pk::note_launch(), k_table_bounds<uint64_t><<<grid, 256, 0, st>>>((const uint64_t*)keys, n, bbits, rem, bstart);
    pk::note_launch(), k_table_sizes<<<(B + 255) / 256, 256, 0, st>>>(bstart, B, tu);
  }
  return cudaGetLastError();
}
}  // namespace pk

// ----------------------------------------------------------------- batch output ----
namespace pk {

// One set of a captured batch: reserve its rows in the batch's macro-node table.
// res = {first row, rows, state}; state 1 ok, 2 table full, 3 device error, 4 nothing kept.
__global__ void k_batch_reserve(const Scalars* sc, unsigned long long* counter, unsigned long long cap,
                                unsigned long long* res) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  if (sc->err != 0) {
    res[0] = 0; res[1] = 0; res[2] = 3;
    return;
  }
  if (sc->n_kept == 0) {
    res[0] = 0; res[1] = 0; res[2] = 4;
    return;
  }
  const unsigned long long m = sc->n_nodes;
  const unsigned long long off = atomicAdd(counter, m);
  if (off + m > cap) {
    res[0] = 0; res[1] = 0; res[2] = 2;
    return;
  }
  res[0] = off; res[1] = m; res[2] = 1;
}

// Copy the set's nodes (key words, 4 suffix and 4 prefix counts) to its reserved rows.
__global__ void __launch_bounds__(256) k_batch_copy(const unsigned long long* __restrict__ nkeys,
                                                    const uint4* __restrict__ nsuf,
                                                    const uint4* __restrict__ npre, int key_words,
                                                    const unsigned long long* res,
                                                    unsigned long long* okeys, uint4* osuf, uint4* opre) {
  if (res[2] != 1) return;
  const unsigned long long off = res[0], m = res[1];
  for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < m;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    for (int w = 0; w < key_words; w++) okeys[(off + i) * key_words + w] = nkeys[i * key_words + w];
    osuf[off + i] = nsuf[i];
    opre[off + i] = npre[i];
  }
}

cudaError_t launch_batch_emit(const Scalars* sc, unsigned long long* counter, unsigned long long cap,
                              unsigned long long* res, const void* nkeys, const void* nsuf, const void* npre,
                              int wide, void* okeys, void* osuf, void* opre, cudaStream_t st) {
  pk::note_launch(), k_batch_reserve<<<1, 32, 0, st>>>(sc, counter, cap, res);
  pk::note_launch(), k_batch_copy<<<sm_count() * 2, 256, 0, st>>>((const unsigned long long*)nkeys, (const uint4*)nsuf,
                                               (const uint4*)npre, wide ? 2 : 1, res,
                                               (unsigned long long*)okeys, (uint4*)osuf, (uint4*)opre);
  return cudaGetLastError();
}

}  // namespace pk

// ------------------------------------------------------------------ initial wiring --
namespace pk {

// One thread per macro-node: the initial wiring of src/wire.cpp:66-121 /
// MacroNode::setup_wiring (includes/distribute_kmers.h:549-655).  Lists: present
// extensions in ascending base code, then the terminal entry (count 1, visit =
// max(other side's visit sum - own side's, 0)); entries ranked by visit then count,
// both descending, equal entries in list order; a two-pointer walk pairs prefix
// visits with suffix visits.
//
// Bound: HBM, by the 168-byte rows it writes.  A thread ranks its two lists in registers
// (five slots a side, compared pairwise) and builds its row in shared memory, and the CTA's
// rows go out as one run of 16-byte stores.  8.57M nodes: 264 us, 6.5 TB/s of rows read and
// written; storing each row from its own thread, with the lists in local memory, took
// 1970 us.  128 nodes a CTA: a multiple of 16 bytes of rows, eight CTAs' rows on an SM.
constexpr int kWireT = 128;                            // nodes per CTA
constexpr int kWireW = (int)(sizeof(WireRow) / 4);     // words of a row (42)

__global__ void __launch_bounds__(kWireT, 8) k_wire(const uint4* __restrict__ nsuf, const uint4* __restrict__ npre,
                                                    unsigned long long m, int coverage,
                                                    uint32_t* __restrict__ out) {
  __shared__ __align__(16) uint32_t s_row[kWireT * kWireW];
  __shared__ int32_t s_sv[kWireT * 5], s_pv[kWireT * 5];  // visits in rank order
  const unsigned long long i0 = blockIdx.x * (unsigned long long)kWireT;
  const unsigned long long i = i0 + threadIdx.x;
  for (int w = threadIdx.x; w < kWireT * kWireW; w += kWireT) s_row[w] = 0;
  __syncthreads();
  if (i < m) {
    const uint4 s4 = __ldcs(nsuf + i), p4 = __ldcs(npre + i);
    const uint32_t sraw[4] = {s4.x, s4.y, s4.z, s4.w}, praw[4] = {p4.x, p4.y, p4.z, p4.w};
    int32_t sv[5], pv[5];
    int ns = 1, np = 1, sc = 0, pc = 0;
    const uint32_t cov = (uint32_t)coverage;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      sv[e] = sraw[e] ? (int32_t)((sraw[e] + cov - 1) / cov) : 0;
      pv[e] = praw[e] ? (int32_t)((praw[e] + cov - 1) / cov) : 0;
      ns += sraw[e] != 0;
      np += praw[e] != 0;
      sc += sv[e];
      pc += pv[e];
    }
    sv[4] = max(pc - sc, 0);
    pv[4] = max(sc - pc, 0);
    int32_t* svis = s_sv + 5 * threadIdx.x;
    int32_t* pvis = s_pv + 5 * threadIdx.x;
    const uint32_t sids = wire_rank(sraw, sv, svis), pids = wire_rank(praw, pv, pvis);
    uint32_t* r = s_row + kWireW * threadIdx.x;
    uint32_t* wire = r + 5;
    uint32_t* begin = r + 5 + 27;
    r[0] = (uint32_t)ns;
    r[1] = (uint32_t)np;
    r[2] = (uint32_t)sv[4];
    r[3] = (uint32_t)pv[4];
    // the ranked lists are consumed front to back: a suffix's offset is what has been
    // taken from it so far, and a prefix's wires are consecutive
    int leftover = sc + sv[4];
    int top_p = 0, top_s = 0, var_p = 0, var_s = 0, wi = 0, first = 0;
    int32_t pcur = pvis[0], scur = svis[0];
    while (leftover > 0 && wi < 9) {
      const int cnt = min(pcur - var_p, scur - var_s);
      wire[3 * wi + 0] = (sids >> (4 * top_s)) & 15u;
      wire[3 * wi + 1] = (uint32_t)var_s;
      wire[3 * wi + 2] = (uint32_t)cnt;
      wi++;
      leftover -= cnt;
      var_p += cnt;
      var_s += cnt;
      if (var_p == pcur) {
        const uint32_t pid = (pids >> (4 * top_p)) & 15u;
        begin[2 * pid + 0] = (uint32_t)first;
        begin[2 * pid + 1] = (uint32_t)(wi - first);
        first = wi;
        var_p = 0;
        top_p = min(top_p + 1, 4);
        pcur = pvis[top_p];
      }
      if (var_s == scur) {
        var_s = 0;
        top_s = min(top_s + 1, 4);
        scur = svis[top_s];
      }
    }
    r[4] = (uint32_t)wi;
  }
  __syncthreads();
  // the CTA's rows, contiguous in `out` (128 rows of 168 bytes start 16-byte aligned)
  const unsigned long long left = m - i0;
  const int words = left < (unsigned long long)kWireT ? (int)left * kWireW : kWireT * kWireW;
  uint32_t* o = out + i0 * kWireW;
  for (int q = threadIdx.x; q < words / 4; q += kWireT)
    __stcs(reinterpret_cast<uint4*>(o) + q, reinterpret_cast<const uint4*>(s_row)[q]);
  for (int w = (words & ~3) + threadIdx.x; w < words; w += kWireT) o[w] = s_row[w];
}

cudaError_t launch_wire(const void* nsuf, const void* npre, unsigned long long m, int coverage, WireRow* out,
                        cudaStream_t st) {
  if (m == 0) return cudaSuccess;
  pk::note_launch(), k_wire<<<(unsigned)((m + kWireT - 1) / kWireT), kWireT, 0, st>>>((const uint4*)nsuf, (const uint4*)npre, m,
                                                                          coverage, (uint32_t*)out);
  return cudaGetLastError();
}

}  // namespace pk

extern "C" uint64_t pk_kernel_launches(void) { return pk::g_launches.load(std::memory_order_relaxed); }
