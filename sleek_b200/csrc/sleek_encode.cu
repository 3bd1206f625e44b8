// sleek_encode.cu -- sm_100a encode kernel (one buffer, and batches of buffers).
//
// Replaces d_encode (include/sleek_common_gpu.h:474-559, 989-1074 of the reference).
// One warp takes a chunk from its first byte to its last, alone: it takes a ticket
// (atomic), has the 16 KB chunk copied to its stage of shared memory (one TMA bulk
// copy), turns the values into codes in place and ORs them into the subchunks' bit
// widths, publishes the chunk's size, packs the codes in place, waits for its place
// in the stream, and stores the packed chunk with one bulk copy.  Fourteen such warps
// share an SM, each with its own stage, with no barrier between them: while some wait
// for memory, others compute, so neither a CTA-wide barrier per chunk nor a pipeline
// of producer, compute and store warps is needed.  A fifteenth warp, the scanner,
// follows the sizes of all chunks (ChunkScan, sleek_device.cuh).
//
// What bounds it: instruction issue and the 14 stages an SM has room for.  A chunk
// costs 2,800 warp instructions (f64 lossless; 5,250 when eight warps shared a chunk,
// because each of them waited at barriers, scanned the widths and shifted the packed
// bytes to their place), and its stage is taken for 8-10 us.  Every wait between the
// published size and the store counts against the stages, so the pack comes before
// the wait for the place, at the alignment the place is expected to have.
// (302 MB f64 field: lossless 144 -> 111 us, eb 1e-4 130 -> 89 us; 26 MB f32 field,
// eb 1e-3: 24.0 -> 13.2 us; 67 MB f32 signal, lossless: 44.6 -> 31.8 us.)
#include <type_traits>

#include "sleek_device.cuh"
#include "sleek_launch.h"

namespace sleek {

// KIND: bit 0 = 64-bit values, bit 1 = lossy
template <int KIND>
using EncVal = typename std::conditional<(KIND & 1) != 0, uint64_t, uint32_t>::type;

constexpr int EW_IN = 64;               // the chunk's bytes begin here in a warp's stage
constexpr int EW_STAGE = EW_IN + CS;    // room before them for the packed chunk's widths and alignment

// ---- phase A: values to codes in place, and the subchunks' widths ------------------

constexpr int EW_G = 4;  // subchunks whose loads, maps and reductions overlap

// Quantizes one group's values (EW_G subchunks, this lane's 16 bytes of each) when
// all of the warp's are ordinary (see quant_plain).  False (nothing written) otherwise.
__device__ __forceinline__ bool quant_group(uint4 (&w)[EW_G], float limit, float inv_scale)
{
  bool odd = false;
#pragma unroll
  for (int u = 0; u < EW_G; ++u)
    odd |= !quant_ordinary(w[u].x, limit) | !quant_ordinary(w[u].y, limit) | !quant_ordinary(w[u].z, limit) |
           !quant_ordinary(w[u].w, limit);
  if (__any_sync(0xffffffffu, odd)) return false;
#pragma unroll
  for (int u = 0; u < EW_G; ++u) {
    w[u] = make_uint4(quant_plain(w[u].x, inv_scale), quant_plain(w[u].y, inv_scale), quant_plain(w[u].z, inv_scale),
                      quant_plain(w[u].w, inv_scale));
  }
  return true;
}

__device__ __forceinline__ bool quant_group(uint4 (&w)[EW_G], float limit, double inv_scale)
{
  bool odd = false;
#pragma unroll
  for (int u = 0; u < EW_G; ++u) odd |= !quant_ordinary(w[u].y, limit) | !quant_ordinary(w[u].w, limit);
  if (__any_sync(0xffffffffu, odd)) return false;
#pragma unroll
  for (int u = 0; u < EW_G; ++u) {
    w[u] = make_uint4(quant_plain(w[u].x, w[u].y, inv_scale), 0u, quant_plain(w[u].z, w[u].w, inv_scale), 0u);
  }
  return true;
}

// This lane's 16 bytes of values to codes, whatever the values are.
template <int KIND>
__device__ __forceinline__ uint4 encode_any(const uint4 w, const QParams& q)
{
  constexpr bool LOSSY = (KIND & 2) != 0;
  if constexpr ((KIND & 1) == 0) {
    return make_uint4(encode_value<LOSSY>(w.x, q), encode_value<LOSSY>(w.y, q), encode_value<LOSSY>(w.z, q),
                      encode_value<LOSSY>(w.w, q));
  } else {
    const uint64_t a = encode_value<LOSSY>((static_cast<uint64_t>(w.y) << 32) | w.x, q);
    const uint64_t b = encode_value<LOSSY>((static_cast<uint64_t>(w.w) << 32) | w.z, q);
    return make_uint4(static_cast<uint32_t>(a), static_cast<uint32_t>(a >> 32), static_cast<uint32_t>(b),
                      static_cast<uint32_t>(b >> 32));
  }
}

// One warp: values to codes for the EW_G subchunks from i0 on (this lane's 16 bytes of
// each to `w`, and if STAGED back to the stage); returns the bit width of subchunk
// `lane` where it is one of them, else 0.  SMALL (and STAGED) keeps the code small: a
// group with values that are not ordinary goes subchunk by subchunk through a loop.
template <int KIND, bool STAGED, bool SMALL>
__device__ __forceinline__ int encode_group(uint8_t* data, uint4 (&w)[EW_G], int i0, const QParams& q, int lane)
{
  constexpr bool LOSSY = (KIND & 2) != 0;
  constexpr bool WIDE = (KIND & 1) != 0;
  uint32_t hi_or = 0, lo_or = 0;  // OR of the codes of subchunk `lane`
  uint4* const p = reinterpret_cast<uint4*>(data + i0 * 512 + lane * 16);
#pragma unroll
  for (int u = 0; u < EW_G; ++u) w[u] = p[32 * u];
  bool done = false;  // (then 64-bit codes are below 2^31)
  if constexpr (LOSSY) {
    if constexpr (WIDE) done = quant_group(w, quant_limit64(q), quant_scale64(q));
    else done = quant_group(w, quant_limit32(q), quant_scale32(q));
    if (SMALL && !done) {
#pragma unroll 1
      for (int u = 0; u < EW_G; ++u) {
        const uint4 v = encode_any<KIND>(p[32 * u], q);
        p[32 * u] = v;
        const uint32_t r = __reduce_or_sync(0xffffffffu, WIDE ? v.x | v.z : v.x | v.y | v.z | v.w);
        if (lane == i0 + u) lo_or = r;
        if (WIDE) {
          const uint32_t h = __reduce_or_sync(0xffffffffu, v.y | v.w);
          if (lane == i0 + u) hi_or = h;
        }
      }
      return hi_or ? 64 - __clz(hi_or) : 32 - __clz(lo_or);
    }
    if (!done) {
#pragma unroll
      for (int u = 0; u < EW_G; ++u) w[u] = encode_any<KIND>(w[u], q);
    }
  } else {
#pragma unroll
    for (int u = 0; u < EW_G; ++u) w[u] = encode_any<KIND>(w[u], q);
  }
  if (WIDE && !done) {
#pragma unroll
    for (int u = 0; u < EW_G; ++u) {
      const uint32_t r = __reduce_or_sync(0xffffffffu, w[u].y | w[u].w);
      if (lane == i0 + u) hi_or = r;
    }
  }
#pragma unroll
  for (int u = 0; u < EW_G; ++u) {
    if (STAGED) p[32 * u] = w[u];
    const uint32_t r = __reduce_or_sync(0xffffffffu, WIDE ? w[u].x | w[u].z : w[u].x | w[u].y | w[u].z | w[u].w);
    if (lane == i0 + u) lo_or = r;
  }
  return hi_or ? 64 - __clz(hi_or) : 32 - __clz(lo_or);
}

// One warp: the staged chunk's values become codes in place (each lane reads and
// writes its own 16 bytes of every subchunk); returns the bit width of subchunk
// `lane`.
//
// SMALL: a batch's warps work on four kinds at once, whose code does not fit the
// instruction cache beside each other; smaller code took a batch of 60 arrays from
// 73.1 to 69.0 us (and the loop below unrolled, which takes 2 % off one kind's
// calls, from 73 to 84 and 105 by twos and fours).
template <int KIND, bool SMALL>
__device__ __forceinline__ int encode_values(uint8_t* data, const QParams& q, int lane)
{
  int ln = 0;
#pragma unroll (SMALL ? 1 : 4)
  for (int i0 = 0; i0 < SC; i0 += EW_G) {
    uint4 w[EW_G];
    ln += encode_group<KIND, true, SMALL>(data, w, i0, q, lane);
  }
  return ln;
}

// ---- phase B: codes to the packed chunk, in place ----------------------------------

// Packs the chunk one subchunk after the other.  `at` is the word being filled
// next; `carry` (lane 0) holds the bits already set in that word: the packed bits
// begin in the middle of a word when the chunk's place in the stream does.
struct Packer {
  uint32_t* at;
  uint32_t carry;
  int half;  // bits of the first word that precede the packed bits (0 or 16)
  int lane;

  // The lane's run of R bits (32 <= R <= 128, low bits first in x0..x3) goes to bit
  // lane * R of the subchunk.  Every word holds bits of at most two lanes: a lane
  // stores the words that its run completes and hands the rest to the next one.
  template <int MINR, int MAXR>
  __device__ __forceinline__ void put(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3, int R)
  {
    const int rs = half + lane * R;
    const int s = rs & 31;
    const int t = s + R;
    const uint32_t y0 = x0 << s;
    const uint32_t y1 = __funnelshift_l(x0, x1, s);
    const uint32_t y2 = __funnelshift_l(x1, x2, s);
    uint32_t y3 = 0u, tail;
    if constexpr (MAXR > 64) {
      y3 = __funnelshift_l(x2, x3, s);
      const uint32_t y4 = __funnelshift_l(x3, 0u, s);
      tail = MINR < 64 && t < 64 ? y1 : (t < 96 ? y2 : (t < 128 ? y3 : y4));
    } else {
      tail = t < 64 ? y1 : y2;
    }
    const uint32_t r = __shfl_sync(0xffffffffu, tail, (lane + 31) & 31);
    uint32_t* const d = at + (rs >> 5);
    d[0] = y0 | (lane == 0 ? carry : r);
    if (MINR >= 64 || t >= 64) d[1] = y1;
    if (MAXR > 64) {
      if (t >= 96) d[2] = y2;
      if (t >= 128) d[3] = y3;
    }
    carry = r;
    at += R;
  }

  // Runs of R < 32 bits: adjacent lanes' runs are joined until they have 32 bits
  // or more, then every 2nd, 4th, ... lane stores.
  __device__ __forceinline__ void put_short(uint32_t run, int R)
  {
    int w = R, step = 1;
    while (2 * w < 32) {
      run |= __shfl_down_sync(0xffffffffu, run, step) << w;
      w *= 2;
      step *= 2;
    }
    const uint32_t n = __shfl_down_sync(0xffffffffu, run, step);
    const uint32_t x0 = run | (n << w);
    const uint32_t x1 = __funnelshift_l(n, 0u, w);
    w *= 2;
    step *= 2;
    const int rs = half + lane * R;
    const int s = rs & 31;
    const int t = s + w;
    const uint32_t y0 = x0 << s;
    const uint32_t y1 = __funnelshift_l(x0, x1, s);
    const uint32_t y2 = __funnelshift_l(x1, 0u, s);
    const uint32_t r = __shfl_sync(0xffffffffu, t < 64 ? y1 : y2, (lane - step) & 31);
    if ((lane & (step - 1)) == 0) {
      uint32_t* const d = at + (rs >> 5);
      d[0] = y0 | (lane == 0 ? carry : r);
      if (t >= 64) d[1] = y1;
    }
    carry = r;
    at += R;
  }

  // A run of R bits (16 <= R < 64) per lane, without a branch on R: runs shorter than
  // a word are joined in pairs, and then every other lane stores.
  __device__ __forceinline__ void put_any(uint32_t x0, uint32_t x1, int R)
  {
    const bool pair = R < 32;
    const uint32_t n = __shfl_down_sync(0xffffffffu, x0, 1);
    if (pair) {
      x0 |= n << R;
      x1 = __funnelshift_l(n, 0u, R);
    }
    const int w = pair ? 2 * R : R;
    const int step = pair ? 2 : 1;
    const int rs = half + lane * R;
    const int s = rs & 31;
    const int t = s + w;
    const uint32_t y0 = x0 << s;
    const uint32_t y1 = __funnelshift_l(x0, x1, s);
    const uint32_t y2 = __funnelshift_l(x1, 0u, s);
    const uint32_t r = __shfl_sync(0xffffffffu, t < 64 ? y1 : y2, (lane - step) & 31);
    uint32_t* const d = at + (rs >> 5);
    if ((lane & (step - 1)) == 0) {
      d[0] = y0 | (lane == 0 ? carry : r);
      if (t >= 64) d[1] = y1;
    }
    carry = r;
    at += R;
  }

  // one subchunk of 32-bit codes, this lane's four
  __device__ __forceinline__ void put32(const uint4 w, int ln)
  {
    if (ln == 0) return;
    if (ln >= 16) {
      wide32(w, ln);
    } else {
      const uint32_t m = 1u << ln;
      const uint32_t a = w.y * m + w.x, b = w.w * m + w.z;  // at most 30 bits each
      if (ln >= 8) put<32, 64>(b * (m * m) + a, __funnelshift_l(b, 0u, 2 * ln), 0u, 0u, 4 * ln);
      else put_short(b * (m * m) + a, 4 * ln);
    }
  }
  // 8 <= ln <= 15
  __device__ __forceinline__ void mid32(const uint4 w, int ln)
  {
    const uint32_t m = 1u << ln;
    const uint32_t a = w.y * m + w.x, b = w.w * m + w.z;
    put<32, 64>(b * (m * m) + a, __funnelshift_l(b, 0u, 2 * ln), 0u, 0u, 4 * ln);
  }
  // 4 <= ln <= 15
  __device__ __forceinline__ void narrow32(const uint4 w, int ln)
  {
    const uint32_t m = 1u << ln;
    const uint32_t a = w.y * m + w.x, b = w.w * m + w.z;
    put_any(b * (m * m) + a, __funnelshift_l(b, 0u, 2 * ln), 4 * ln);
  }
  // 16 <= ln <= 32 (shifts of up to 32: the clamping form)
  __device__ __forceinline__ void wide32(const uint4 w, int ln)
  {
    const uint32_t m = pow2_or_0(ln);
    const uint32_t a0 = w.y * m + w.x, a1 = __funnelshift_lc(w.y, 0u, ln);
    const uint32_t b0 = w.w * m + w.z, b1 = __funnelshift_lc(w.w, 0u, ln);
    const int k = 2 * ln - 32;
    put<64, 128>(a0, b0 * pow2_or_0(k) + a1, __funnelshift_lc(b0, b1, k), __funnelshift_lc(b1, 0u, k), 4 * ln);
  }

  // 8 <= ln <= 32, without a branch: the products and shifts that do not apply are 0
  __device__ __forceinline__ void long32(const uint4 w, int ln)
  {
    const uint32_t m = pow2_or_0(ln);
    const uint32_t a0 = w.y * m + w.x, a1 = __funnelshift_lc(w.y, 0u, ln);
    const uint32_t b0 = w.w * m + w.z, b1 = __funnelshift_lc(w.w, 0u, ln);
    const int k = max(2 * ln - 32, 0);
    const uint32_t x1 = 2 * ln < 32 ? __funnelshift_l(b0, 0u, 2 * ln) : b0 * pow2_or_0(k) + a1;
    put<32, 128>(b0 * pow2_or_0(2 * ln) + a0, x1, __funnelshift_lc(b0, b1, k), __funnelshift_lc(b1, 0u, k), 4 * ln);
  }

  // one subchunk of 64-bit codes, this lane's two
  __device__ __forceinline__ void put64(const uint4 w, int ln)
  {
    if (ln == 0) return;
    if (ln >= 32) wide64(w, ln);
    else if (ln >= 16) narrow64(w, ln);
    else put_short(w.z * (1u << ln) + w.x, 2 * ln);
  }
  // 32 <= ln <= 64
  __device__ __forceinline__ void wide64(const uint4 w, int ln)
  {
    const int k = ln - 32;
    put<64, 128>(w.x, w.z * pow2_or_0(k) + w.y, __funnelshift_lc(w.z, w.w, k), __funnelshift_lc(w.w, 0u, k), 2 * ln);
  }
  // 16 <= ln <= 31
  __device__ __forceinline__ void narrow64(const uint4 w, int ln)
  {
    put<32, 64>(w.z * (1u << ln) + w.x, __funnelshift_l(w.z, 0u, ln), 0u, 0u, 2 * ln);
  }
  // 8 <= ln <= 31
  __device__ __forceinline__ void any64(const uint4 w, int ln)
  {
    put_any(w.z * (1u << ln) + w.x, __funnelshift_l(w.z, 0u, ln), 2 * ln);
  }
};

// One warp: packs the codes staged at `stg + EW_IN` into the chunk's bytes at
// `stg + a` (a < 16, even: the chunk's place in the stream modulo 16): the 32 width
// bytes, the packed bits, the int16 trailer.  In place, subchunk by subchunk: the
// packed bytes of a subchunk end before the codes of the next one begin, and a
// lane's stores follow an exchange that every lane enters with its codes loaded.
template <typename T, bool SMALL>
__device__ __forceinline__ void pack_chunk(uint8_t* stg, int a, int ln, int osize, int lane)
{
  constexpr int B = static_cast<int>(sizeof(T));
  stg[a + lane] = static_cast<uint8_t>(ln);
  Packer k;
  k.lane = lane;
  k.half = (a & 2) * 8;
  k.at = reinterpret_cast<uint32_t*>(stg + ((a + 32) & ~3));
  // the last two widths share the first word with the packed bits
  const uint32_t l2 = __shfl_sync(0xffffffffu, ln, 30) | (__shfl_sync(0xffffffffu, ln, 31) << 8);
  k.carry = k.half ? l2 : 0u;
  const unsigned wide = __ballot_sync(0xffffffffu, ln >= (B == 4 ? 16 : 32));
  const unsigned narrow = __ballot_sync(0xffffffffu, B == 4 ? (ln >= 8 && ln < 16) : (ln >= 16 && ln < 32));
  const unsigned lng = B == 4 ? __ballot_sync(0xffffffffu, ln >= 8) : 0u;
  const unsigned any = __ballot_sync(0xffffffffu, B == 4 ? (ln >= 4 && ln < 16) : (ln >= 8 && ln < 32));
#pragma unroll 1
  for (int i0 = 0; i0 < SC; i0 += EW_G) {
    const uint4* const in = reinterpret_cast<const uint4*>(stg + EW_IN + i0 * 512 + lane * 16);
    uint4 w[EW_G];
    int l[EW_G];
#pragma unroll
    for (int u = 0; u < EW_G; ++u) {
      w[u] = in[32 * u];
      l[u] = __shfl_sync(0xffffffffu, ln, i0 + u);
    }
    constexpr unsigned ALL = (1u << EW_G) - 1u;
    if (((wide >> i0) & ALL) == ALL) {
#pragma unroll
      for (int u = 0; u < EW_G; ++u) {
        if constexpr (B == 4) k.wide32(w[u], l[u]);
        else k.wide64(w[u], l[u]);
      }
    } else if (((narrow >> i0) & ALL) == ALL) {
#pragma unroll
      for (int u = 0; u < EW_G; ++u) {
        if constexpr (B == 4) k.mid32(w[u], l[u]);
        else k.narrow64(w[u], l[u]);
      }
    } else if (B == 4 && ((lng >> i0) & ALL) == ALL) {
#pragma unroll
      for (int u = 0; u < EW_G; ++u) k.long32(w[u], l[u]);
    } else if (((any >> i0) & ALL) == ALL) {
#pragma unroll
      for (int u = 0; u < EW_G; ++u) {
        if constexpr (B == 4) k.narrow32(w[u], l[u]);
        else k.any64(w[u], l[u]);
      }
    } else if constexpr (!SMALL) {
#pragma unroll
      for (int u = 0; u < EW_G; ++u) {
        if constexpr (B == 4) k.put32(w[u], l[u]);
        else k.put64(w[u], l[u]);
      }
    } else {
#pragma unroll 1
      for (int u = 0; u < EW_G; ++u) {
        const int l1 = __shfl_sync(0xffffffffu, ln, i0 + u);
        if constexpr (B == 4) k.put32(in[32 * u], l1);
        else k.put64(in[32 * u], l1);
      }
    }
  }
  if (lane == 0) {
    if (k.half) *k.at = (k.carry & 0xffffu) | (static_cast<uint32_t>(osize) << 16);
    else *reinterpret_cast<int16_t*>(k.at) = static_cast<int16_t>(osize);
  }
}

// Stores the packed chunk at `src` (byte `a` of its 16-byte granule) to its place: one
// bulk copy of the whole granules where the place has the same alignment, else 16-byte
// stores put together from the staged words; the two granules shared with the
// neighbouring chunks two bytes at a time (sizes and places are even).
__device__ __forceinline__ void store_chunk(uint8_t* dst, const uint8_t* src, int a, int csize, int lane)
{
  const int al = static_cast<int>(reinterpret_cast<uintptr_t>(dst) & 15u);
  const int b = (16 - al) & 15;             // chunk bytes before the first whole granule
  const int e = ((al + csize) & ~15) - al;  // and up to the end of the last
  if (al == a) {
    if (lane == 0) {
      tma_store_1d(dst + b, src + b, static_cast<uint32_t>(e - b));
      bulk_commit();
    }
  } else if (((al ^ a) & 7) == 0) {
#pragma unroll 4
    for (int o = b + 16 * lane; o < e; o += 512) {
      const uint2 x = *reinterpret_cast<const uint2*>(src + o), y = *reinterpret_cast<const uint2*>(src + o + 8);
      *reinterpret_cast<uint4*>(dst + o) = make_uint4(x.x, x.y, y.x, y.y);
    }
  } else {
    const int sh = ((a + b) & 2) * 8;
#pragma unroll 2
    for (int o = b + 16 * lane; o < e; o += 512) {
      const uint32_t* const p = reinterpret_cast<const uint32_t*>(src + o - (sh >> 3));
      const uint32_t w0 = p[0], w1 = p[1], w2 = p[2], w3 = p[3], w4 = p[4];
      *reinterpret_cast<uint4*>(dst + o) = make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh),
                                                      __funnelshift_r(w2, w3, sh), __funnelshift_r(w3, w4, sh));
    }
  }
  const int o = lane < 16 ? 2 * lane : e + 2 * (lane - 16);
  if (lane < 16 ? o < b : o < csize)
    *reinterpret_cast<uint16_t*>(dst + o) = *reinterpret_cast<const uint16_t*>(src + o);
}

// ---- the kernel --------------------------------------------------------------------

// What a warp needs to know about its chunk.
struct EncChunk {
  const uint8_t* in;  // its first byte
  uint8_t* out;       // the buffer's stream
  long long* outsize;
  long long g;        // chunk id across the launch
  long long c;        // chunk index within its buffer
  long long chunks;   // chunks of the buffer
  long long insize;   // bytes of the buffer
  QParams q;
  int kind;
  int osize;
};

// Copies the chunk's bytes to `dst` (zero-padded to a full chunk) and waits for
// them: one TMA bulk copy, or, where the input is not 16-byte aligned or the chunk
// is partial, asynchronous copies of the widest elements the address allows.
__device__ __forceinline__ bool load_chunk(uint8_t* dst, const uint8_t* in, int osize, uint64_t* bar, uint32_t& par,
                                           int lane)
{
  const unsigned mis = static_cast<unsigned>(reinterpret_cast<uintptr_t>(in)) & 15u;
  if (mis == 0u && osize == CS) {
    if (lane == 0) {
      mbar_arrive_expect_tx(bar, CS);
      tma_load_1d(dst, in, CS, bar);
    }
    const bool ok = copy_landed(bar, par);
    par ^= 1u;
    return ok;
  }
  auto copy = [&](auto width) {
    constexpr int N = decltype(width)::value;
#pragma unroll 8
    for (int k = 0; k < CS / (32 * N); ++k) {
      const int o = (k * 32 + lane) * N;
      const int have = min(max(osize - o, 0), N);
      cp_async<N>(dst + o, have ? in + o : in, have);
    }
  };
  if (mis == 0u) copy(std::integral_constant<int, 16>{});
  else if (mis == 8u) copy(std::integral_constant<int, 8>{});
  else copy(std::integral_constant<int, 4>{});
  cp_async_wait_all();
  __syncwarp();
  return true;
}

template <int KIND, bool BATCH, int NW, int MINB>
__global__ void __launch_bounds__((NW + 1) * 32, MINB)
    k_encode(const typename std::conditional<BATCH, BatchEncArgs, EncArgs>::type a)
{
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + NW * EW_STAGE);
  long long* const cb = reinterpret_cast<long long*>(bars + NW);
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  uint8_t* const stg = smem + warp * EW_STAGE;
  uint64_t* const bar = bars + warp;

  if (tid == 0) {
    for (int i = 0; i < NW; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
  }
  grid_wait();
  const WsPhase ph = [&]() {
    if constexpr (BATCH) return WsPhase::fixed(a.ws);
    else return WsPhase::of(a.ws, a.flag_cap);
  }();
  uint64_t* const hdr = ph.hdr;
  if constexpr (BATCH) {
    for (int i = tid; i <= a.njobs; i += (NW + 1) * 32) cb[i] = a.chunk_base[i];
  }
  __shared__ unsigned long long s_first;
  __shared__ ScanRing ring;
  // The first tickets are taken for the whole CTA, as many as an even share of a
  // small input leaves it; a ticket is only ever held by a running warp.
  unsigned long long* const tick = reinterpret_cast<unsigned long long*>(&a.ws[WS_TICKET]);
  const long long total = [&]() -> long long {
    if constexpr (BATCH) return a.chunk_base[a.njobs];
    else return (a.insize + CS - 1) / CS;
  }();
  const long long share = (total + gridDim.x - 1) / gridDim.x;
  const int first_n = static_cast<int>(share < NW ? share : NW);
  if (tid == 0) {
    s_first = atomicAdd(tick, static_cast<unsigned long long>(first_n));
    ring.known = 0;
    ring.gone = 0;
  }
  __syncthreads();
  const ChunkScan scan(ph.flags, total, &ring);

  uint32_t par = 0;
  auto job_of = [&](long long g) {  // last job whose first chunk id is <= g (empty jobs are skipped)
    int lo = 0;
    if constexpr (BATCH) {
      int hi = a.njobs - 1;
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (cb[mid] <= g) lo = mid;
        else hi = mid - 1;
      }
    }
    return lo;
  };
  // the 16 KB, 16-byte aligned, that hold nearly all of chunk g if it is a whole one
  auto whole_chunk = [&](long long g) -> const uint8_t* {
    const uint8_t* in;
    long long c = g, insize;
    if constexpr (BATCH) {
      const int lo = job_of(g);
      c = g - cb[lo];
      in = a.jobs[lo].in;
      insize = a.jobs[lo].insize;
    } else {
      in = a.in;
      insize = a.insize;
    }
    if ((c + 1) * CS > insize) return nullptr;
    in += c * CS;
    return in - (reinterpret_cast<uintptr_t>(in) & 15u);
  };
  auto next = [&]() -> long long {
    unsigned long long t = 0;
    if (lane == 0) t = atomicAdd(tick, 1ull);
    return static_cast<long long>(__shfl_sync(0xffffffffu, t, 0));
  };
  if (warp == NW) {
    scan.follow(NW);
    if constexpr (!BATCH) ph.clear_other_share(lane);
  } else {
  long long t = warp < first_n ? static_cast<long long>(s_first) + warp : next();
  while (t < total) {
    EncChunk k;
    long long seg = 0;
    int job = 0;
    if constexpr (BATCH) {
      const int lo = job_of(t);
      const BatchJob& j = a.jobs[lo];
      seg = cb[lo];
      job = lo;
      k.g = t;
      k.c = t - seg;
      k.in = j.in + k.c * CS;
      k.out = j.out;
      k.outsize = j.outsize;
      k.chunks = j.chunks;
      k.insize = j.insize;
      k.q = j.q;
      k.kind = j.kind;
    } else {
      k.g = t;
      k.c = t;
      k.in = a.in + t * CS;
      k.out = a.out;
      k.outsize = a.outsize;
      k.chunks = total;
      k.insize = a.insize;
      k.q = a.q;
      k.kind = KIND;
    }
    k.osize = static_cast<int>(min(static_cast<long long>(CS), k.insize - k.c * CS));

    if (!load_chunk(stg + EW_IN, k.in, k.osize, bar, par, lane)) {
      if (lane == 0) set_status(hdr, ST_TIMEOUT, k.g);
      break;
    }
    int ln;
    if constexpr (KIND >= 0) {
      ln = encode_values<KIND, false>(stg + EW_IN, k.q, lane);
    } else {
      switch (k.kind) {
        case 0: ln = encode_values<0, true>(stg + EW_IN, k.q, lane); break;
        case 1: ln = encode_values<1, true>(stg + EW_IN, k.q, lane); break;
        case 2: ln = encode_values<2, true>(stg + EW_IN, k.q, lane); break;
        default: ln = encode_values<3, true>(stg + EW_IN, k.q, lane); break;
      }
    }
    const bool wide = (KIND >= 0 ? KIND : k.kind) & 1;
    const int wtot = __reduce_add_sync(0xffffffffu, wide ? 2 * ln : 4 * ln);
    const bool comp = 34 + 4 * wtot < k.osize;
    const int csize = comp ? 34 + 4 * wtot : k.osize;
    if (lane == 0) scan.publish(k.g, static_cast<uint32_t>(csize));
    if (!comp) {  // stored as it came: fetched again (the codes took its place), mostly from L2
      fence_proxy_async_smem();
      __syncwarp();
      if (!load_chunk(stg + EW_IN, k.in, k.osize, bar, par, lane)) {
        if (lane == 0) set_status(hdr, ST_TIMEOUT, k.g);
        break;
      }
    }
    // Packed before its place is known, at the alignment that it has if every chunk
    // not placed yet is compressed (a compressed chunk's size is 2 mod 16 for 32-bit
    // values, 2 mod 8 for 64-bit ones).
    int al = 0;
    if (comp) {
      long long guess = 2 * k.c;
      if constexpr (!BATCH) guess = scan.guess(k.g);
      al = static_cast<int>((reinterpret_cast<uintptr_t>(k.out) + 8 + 2 * k.chunks + guess) & 15u);
      if (wide) pack_chunk<uint64_t, BATCH>(stg, al, ln, k.osize, lane);
      else pack_chunk<uint32_t, BATCH>(stg, al, ln, k.osize, lane);
      fence_proxy_async_smem();
      __syncwarp();
    }
    // The chunk about a full round of tickets ahead goes to L2, so that its warp's load
    // takes one L2 round trip, not a queue at HBM that all later chunks' places would
    // wait for.  After the pack, not before: at a kernel's start the first loads of all
    // warps are still under way (302 MB f64 lossless: 108 us against 116 with the
    // prefetch right after the load and 110 without one; batch of 60 arrays: 65.3
    // against 67.5 without one).
    const long long ahead = t + static_cast<long long>(gridDim.x) * NW;
    if (ahead < total) {
      const uint8_t* in = whole_chunk(ahead);
      if (lane == 0 && in != nullptr) prefetch_l2(in, CS);
    }
    long long excl = scan.prefix(k.g, BATCH && k.c > 0 ? seg : 0, hdr);
    if constexpr (BATCH) {
      // the place within the buffer: relative to its first chunk, whose warp tells
      // the others where it is unless they share its group
      if (excl >= 0) {
        uint64_t* const start = a.starts + job;
        if (k.c == 0) {
          if (lane == 0) st_relaxed_u64(start, FLAG_SET | static_cast<uint64_t>(excl));
          excl = 0;
        } else if (seg < k.g / GROUP * GROUP) {
          const uint64_t v = ChunkScan::await(start, hdr);
          excl = v ? excl - static_cast<long long>(v & FLAG_VAL) : -1;
        }
      }
    }
    if (excl < 0 || excl > k.c * CS) {
      if (lane == 0) set_status(hdr, excl < 0 ? ST_TIMEOUT : ST_CAPACITY, k.g);
      break;
    }
    if (lane == 0) {
      if (k.c == k.chunks - 1) {
        if constexpr (BATCH) {  // the buffer is complete: its header and size
          *reinterpret_cast<long long*>(k.out) = k.insize;
          *k.outsize = 8 + 2 * k.chunks + excl + csize;
        } else {
          hdr[WS_TOTAL] = static_cast<uint64_t>(excl + csize);
        }
      }
      *reinterpret_cast<uint16_t*>(k.out + 8 + 2 * k.c) = static_cast<uint16_t>(csize);
    }
    uint8_t* const dst = k.out + 8 + 2 * k.chunks + excl;
    if (comp) store_chunk(dst, stg + al, al, csize, lane);
    else store_shifted<32>(dst, stg + EW_IN, csize, lane);
    t = next();
    // the stage is read before it is refilled
    if (lane == 0) bulk_wait_read();
    fence_proxy_async_smem();
    __syncwarp();
  }
  if (lane == 0) {
    atomicAdd(&ring.gone, 1);
    bulk_wait();
  }
  }

  // ---- epilogue: the last CTA out finishes the outputs -----------------------
  grid_release();
  __syncthreads();
  __shared__ int last_cta;
  if (tid == 0) {
    __threadfence();
    const unsigned long long d = atomicAdd(reinterpret_cast<unsigned long long*>(&a.ws[WS_DONE]), 1ull);
    last_cta = d == gridDim.x - 1;
    if (last_cta) __threadfence();
  }
  __syncthreads();
  if (last_cta) {
    const unsigned long long st = ld_relaxed_u64(&hdr[WS_STATUS]);
    if constexpr (BATCH) {
      // buffers without chunks get their header-only stream; an error anywhere
      // turns every size into -status
      for (int i = tid; i < a.njobs; i += (NW + 1) * 32) {
        const BatchJob& j = a.jobs[i];
        if (st) {
          *j.outsize = -static_cast<long long>(st);
        } else if (j.chunks == 0) {
          *reinterpret_cast<long long*>(j.out) = 0;
          *j.outsize = 8;
        }
      }
    } else if (tid == 0) {
      const long long tot = total ? static_cast<long long>(ld_relaxed_u64(&hdr[WS_TOTAL])) : 0ll;
      *reinterpret_cast<long long*>(a.out) = a.insize;
      *a.outsize = st ? -static_cast<long long>(st) : 8 + 2 * total + tot;
      ph.finish(a.ws, scan_words(total));
    }
  }
}

// ---- few chunks: eight warps per chunk ----------------------------------------------

// For at most ENC_TEAM_CTAS chunks per SM, as many as are resident at once, one per
// CTA: such a call is as long as one chunk's way through the kernel, and eight warps
// take an eighth of the chunk each.  The codes stay in registers from the transform to
// the pack, and a chunk's place is the sum of all flags before it.  (f32 lossless,
// microseconds on the GPU against k_encode's: 4 KB 3.9 / 7.2, 200 KB 5.8 / 9.0, 1 MB
// 5.8 / 9.2, 4.8 MB 7.8 / 10.6, 7 MB 9.1 / 11.1.)
constexpr int ENC_TEAM = 8;
constexpr int ENC_TEAM_CTAS = 4;
static_assert(ENC_TEAM * EW_G == SC, "one group of subchunks per warp");

template <int KIND>
__global__ void __launch_bounds__(ENC_TEAM * 32, ENC_TEAM_CTAS) k_encode_team(const EncArgs a)
{
  using T = EncVal<KIND>;
  constexpr int B = static_cast<int>(sizeof(T));
  constexpr int NT = ENC_TEAM * 32;
  __shared__ __align__(128) uint8_t stg[CS + 64];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_ln[SC];
  __shared__ long long s_chunk, s_excl;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  grid_wait();
  const long long chunks = (a.insize + CS - 1) / CS;  // = gridDim.x, or 0
  // the chunk waits for those before it, so it goes by ticket (a lone one does not)
  long long c = 0;
  if (chunks > 1) {
    if (tid == 0) s_chunk = static_cast<long long>(atomicAdd(reinterpret_cast<unsigned long long*>(&a.ws[WS_TICKET]), 1ull));
  }
  const WsPhase ph = WsPhase::of(a.ws, a.flag_cap);
  __syncthreads();
  if (chunks > 1) c = s_chunk;
  uint32_t* const flags = reinterpret_cast<uint32_t*>(ph.flags);

  if (chunks > 0) {
    const uint8_t* const in = a.in + c * CS;
    const int osize = static_cast<int>(min(static_cast<long long>(CS), a.insize - c * CS));
    const unsigned mis = static_cast<unsigned>(reinterpret_cast<uintptr_t>(in)) & 15u;
    bool wlate = false;
    if (mis == 0u && osize == CS) {
      if (tid == 0) {
        mbar_arrive_expect_tx(&bar, CS);
        tma_load_1d(stg, in, CS, &bar);
      }
      wlate = !copy_landed(&bar, 0);
    } else {  // a warp's own subchunks, zero-padded
      for (int k = 0; k < EW_G * 4; ++k) {
        const int o = (warp * EW_G * 4 + k) * 128 + lane * 4;
        const int have = min(max(osize - o, 0), 4);
        cp_async<4>(stg + o, have ? in + o : in, have);
      }
      cp_async_wait_all();
      __syncwarp();
    }
    uint4 w[EW_G];
    int width = 0;
    if (!wlate) width = encode_group<KIND, false, false>(stg, w, warp * EW_G, a.q, lane);
    if (lane / EW_G == warp) s_ln[lane] = width;
    if (__syncthreads_or(wlate)) {
      if (tid == 0) set_status(ph.hdr, ST_TIMEOUT, c);
    } else {
      const int ln = s_ln[lane];
      const int wc = (B == 4 ? 4 : 2) * ln;  // words of subchunk `lane`
      const int wtot = __reduce_add_sync(0xffffffffu, wc);
      const bool comp = 34 + 4 * wtot < osize;
      const int csize = comp ? 34 + 4 * wtot : osize;
      if (tid == 0) st_relaxed_u32(flags + c, static_cast<uint32_t>(csize));
      if (comp) {
        // every warp has read its part of the stage: the packed chunk takes its place
        Packer k;
        k.lane = lane;
        k.half = 0;
        k.carry = 0;
        k.at = reinterpret_cast<uint32_t*>(stg + 32) + __reduce_add_sync(0xffffffffu, lane < warp * EW_G ? wc : 0);
#pragma unroll
        for (int u = 0; u < EW_G; ++u) {
          const int l = __shfl_sync(0xffffffffu, ln, warp * EW_G + u);
          if constexpr (B == 4) k.put32(w[u], l);
          else k.put64(w[u], l);
        }
        if (warp == ENC_TEAM - 1) {
          stg[lane] = static_cast<uint8_t>(ln);
          if (lane == 0) *reinterpret_cast<int16_t*>(stg + 32 + 4 * wtot) = static_cast<int16_t>(osize);
        }
      }
      if (warp == 0) {
        const long long x = c > 0 ? ChunkScan(ph.flags, chunks, nullptr).prefix_flags(c, ph.hdr) : 0;
        if (lane == 0) s_excl = x;
      }
      __syncthreads();
      const long long excl = s_excl;
      if (excl < 0 || excl > c * CS) {
        if (tid == 0) set_status(ph.hdr, excl < 0 ? ST_TIMEOUT : ST_CAPACITY, c);
      } else {
        store_shifted<NT>(a.out + 8 + 2 * chunks + excl, stg, csize, tid);
        if (tid == 0) {
          *reinterpret_cast<uint16_t*>(a.out + 8 + 2 * c) = static_cast<uint16_t>(csize);
          if (c == chunks - 1) ph.hdr[WS_TOTAL] = static_cast<uint64_t>(excl + csize);
        }
      }
    }
  }
  if (warp == ENC_TEAM - 1) ph.clear_other_share(lane);
  grid_release();
  __syncthreads();
  if (tid == 0) {
    bool last = gridDim.x == 1;
    if (!last) {
      __threadfence();
      last = atomicAdd(reinterpret_cast<unsigned long long*>(&a.ws[WS_DONE]), 1ull) == gridDim.x - 1;
      if (last) __threadfence();
    }
    if (last) {
      const unsigned long long st = ld_relaxed_u64(&ph.hdr[WS_STATUS]);
      const long long tot = chunks ? static_cast<long long>(ld_relaxed_u64(&ph.hdr[WS_TOTAL])) : 0ll;
      *reinterpret_cast<long long*>(a.out) = a.insize;
      *a.outsize = st ? -static_cast<long long>(st) : 8 + 2 * chunks + tot;
      ph.finish(a.ws, scan_words(chunks));
    }
  }
}

// ---- launchers ---------------------------------------------------------------------

// Launch shapes: warps (and stages) per CTA and CTAs per SM.  The largest CTA that
// fits, one per SM, has the most chunks in flight and one scanner warp per SM; the
// others leave room for kernels of other streams, or for the autotuner to pick.
template <int NW_, int MINB_>
struct EncShape {
  static constexpr int NW = NW_;
  static constexpr int MINB = MINB_;
  static constexpr int NT = (NW + 1) * 32;  // + the scanner warp
  static constexpr int SMEM = NW * EW_STAGE + 8 * NW;
};
using EncShape0 = EncShape<14, 1>;  // default
using EncShape1 = EncShape<12, 1>;
using EncShape2 = EncShape<6, 2>;
using EncShape3 = EncShape<4, 3>;
using EncShape4 = EncShape<8, 1>;
constexpr int ENC_SHAPES = 5;
using EncShapeBatch = EncShape<13, 1>;  // + the jobs' first chunk ids
constexpr int ENC_BATCH_SMEM = EncShapeBatch::SMEM + 8 + 8 * (BATCH_MAX_JOBS + 1);

template <int KIND>
static cudaError_t launch_enc_team(const EncArgs& a, int grid, cudaStream_t st)
{
  return launch_after(k_encode_team<KIND>, grid, ENC_TEAM * 32, 0, st, a);
}

template <int KIND, class S>
static cudaError_t launch_enc_k(const EncArgs& a, int grid, cudaStream_t st)
{
  auto k = k_encode<KIND, false, S::NW, S::MINB>;
  static unsigned long long attr = 0;
  cudaError_t e = ensure_smem_attr(k, S::SMEM, &attr);
  if (e != cudaSuccess) return e;
  return launch_after(k, grid, S::NT, S::SMEM, st, a);
}

template <int KIND, class S>
static int enc_occupancy()
{
  auto k = k_encode<KIND, false, S::NW, S::MINB>;
  // the smem attribute must be set before the occupancy query counts dynamic smem
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, S::NT, S::SMEM);
  return n;
}

template <int KIND>
static cudaError_t launch_enc_kind(int shape, const EncArgs& a, int grid, cudaStream_t st)
{
  switch (shape) {
    case 1: return launch_enc_k<KIND, EncShape1>(a, grid, st);
    case 2: return launch_enc_k<KIND, EncShape2>(a, grid, st);
    case 3: return launch_enc_k<KIND, EncShape3>(a, grid, st);
    case 4: return launch_enc_k<KIND, EncShape4>(a, grid, st);
    case ENC_SHAPES: return launch_enc_team<KIND>(a, grid, st);
    default: return launch_enc_k<KIND, EncShape0>(a, grid, st);
  }
}

template <int KIND>
static int enc_occupancy_kind(int shape)
{
  switch (shape) {
    case 1: return enc_occupancy<KIND, EncShape1>();
    case 2: return enc_occupancy<KIND, EncShape2>();
    case 3: return enc_occupancy<KIND, EncShape3>();
    case 4: return enc_occupancy<KIND, EncShape4>();
    case ENC_SHAPES: return ENC_TEAM_CTAS;
    default: return enc_occupancy<KIND, EncShape0>();
  }
}

cudaError_t launch_encode(int width, bool lossy, int shape, const EncArgs& a, int grid, cudaStream_t st)
{
  if (width == 4) return lossy ? launch_enc_kind<2>(shape, a, grid, st) : launch_enc_kind<0>(shape, a, grid, st);
  return lossy ? launch_enc_kind<3>(shape, a, grid, st) : launch_enc_kind<1>(shape, a, grid, st);
}

int encode_blocks_per_sm(int width, bool lossy, int shape)
{
  if (width == 4) return lossy ? enc_occupancy_kind<2>(shape) : enc_occupancy_kind<0>(shape);
  return lossy ? enc_occupancy_kind<3>(shape) : enc_occupancy_kind<1>(shape);
}

int encode_shape_count() { return ENC_SHAPES; }

// index ENC_SHAPES, past the shapes that can be asked for, is k_encode_team: its grid
// has to be the number of chunks
int encode_default_shape(long long chunks, int sms, int ctas)
{
  const int most = ctas > 0 && ctas < ENC_TEAM_CTAS ? ctas : ENC_TEAM_CTAS;
  return chunks <= static_cast<long long>(most) * sms ? ENC_SHAPES : 0;
}

ShapeInfo encode_shape_info(int shape)
{
  switch (shape) {
    case 1: return {EncShape1::NT, EncShape1::NW, EncShape1::NW, EncShape1::MINB};
    case 2: return {EncShape2::NT, EncShape2::NW, EncShape2::NW, EncShape2::MINB};
    case 3: return {EncShape3::NT, EncShape3::NW, EncShape3::NW, EncShape3::MINB};
    case 4: return {EncShape4::NT, EncShape4::NW, EncShape4::NW, EncShape4::MINB};
    default: return {EncShape0::NT, EncShape0::NW, EncShape0::NW, EncShape0::MINB};
  }
}

cudaError_t launch_encode_batch(const BatchEncArgs& a, int grid, cudaStream_t st)
{
  auto k = k_encode<-1, true, EncShapeBatch::NW, EncShapeBatch::MINB>;
  static unsigned long long attr = 0;
  cudaError_t e = ensure_smem_attr(k, ENC_BATCH_SMEM, &attr);
  if (e != cudaSuccess) return e;
  return launch_after(k, grid, EncShapeBatch::NT, ENC_BATCH_SMEM, st, a);
}

int encode_batch_blocks_per_sm()
{
  auto k = k_encode<-1, true, EncShapeBatch::NW, EncShapeBatch::MINB>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, ENC_BATCH_SMEM);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, EncShapeBatch::NT, ENC_BATCH_SMEM);
  return n;
}

}  // namespace sleek
