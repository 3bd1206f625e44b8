// sleek_decode.cu -- sm_100a decode kernels (one buffer, and batches of buffers).
//
// Replaces d_decode (include/sleek_common_gpu.h:688-768, 1199-1279 of the reference).
// Every CTA adds up the size table, so that it knows every chunk's place in the
// stream, and its teams of warps take chunks one by one: the chunk's bytes come to the
// team's stage of shared memory by one TMA bulk copy (of the 16-byte aligned superset,
// so any byte offset works), and the team checks and unpacks them straight into 16-byte
// stores.  No CTA waits for another, and there is no CTA barrier per chunk.  Malformed
// streams set an error status instead of trapping; every wait is bounded.
//
// What bounds it: HBM on large fields (302 MB f64 at eb 1e-4: 73.2 -> 63.3 us, 0.91 of
// the measured copy rate), else the waits at the start (header and table, the first
// chunks' copies) and the ALU pipe (26 MB f32 at eb 1e-3: 17.9 -> 11.6 us; 67 MB f32
// lossless: 29.9 -> 26.4 us; batch of 60 arrays: 61.4 -> 49.3 us).
// A chunk costs 1,740 warp instructions (f64, eb 1e-4; all of the launch's), 2,720 when
// eight warps shared it and each lane took every 32nd value.
#include <type_traits>

#include "sleek_device.cuh"
#include "sleek_launch.h"

namespace sleek {

// a chunk at any byte offset, and the words that the unpacking reads past its end
constexpr int DEC_STAGE = CS + 48;

constexpr int DEC_G = 4;  // subchunks whose loads and shifts overlap

// ---- one chunk ---------------------------------------------------------------------

// This lane's 16 bytes of output values.
__device__ __forceinline__ void store16(uint8_t* o, const uint4 v) { *reinterpret_cast<uint4*>(o) = v; }


// Values of the lane's codes.  W: the codes' widths are below 24 bits (32-bit values)
// or 32 bits (64-bit values), so that no code is an escape.
template <typename T, bool LOSSY, bool W>
__device__ __forceinline__ uint4 decode_codes(const uint4 e, const QParams& q)
{
  if constexpr (sizeof(T) == 4) {
    auto one = [&](uint32_t c) -> uint32_t {
      if constexpr (LOSSY && W) {
        return dequant_plain32(c, q);
      } else {
        return decode_value<LOSSY>(c, q);
      }
    };
    return make_uint4(one(e.x), one(e.y), one(e.z), one(e.w));
  } else {
    auto one = [&](uint32_t l, uint32_t h) -> uint64_t {
      if constexpr (LOSSY && W) {
        return dequant_plain64(l, q);
      } else {
        return decode_value<LOSSY>((static_cast<uint64_t>(h) << 32) | l, q);
      }
    };
    const uint64_t a = one(e.x, e.y), b = one(e.z, e.w);
    return make_uint4(static_cast<uint32_t>(a), static_cast<uint32_t>(a >> 32), static_cast<uint32_t>(b),
                      static_cast<uint32_t>(b >> 32));
  }
}

// The lane's codes of one subchunk of width `ln` whose packed bits begin at `bit` of
// the stage: its 4 (32-bit values) or 2 (64-bit) are adjacent, so they are one run of
// bits, aligned once and then cut at warp-uniform places.
template <int B>
__device__ __forceinline__ uint4 codes_narrow(const uint32_t* w, int bit, int ln, int lane)  // ln <= 15 / 31
{
  const int at = bit + lane * ((16 / B) * ln);
  const uint32_t* const p = w + (at >> 5);
  const uint32_t w0 = p[0], w1 = p[1], w2 = p[2];
  const uint32_t x0 = __funnelshift_r(w0, w1, at), x1 = __funnelshift_r(w1, w2, at);
  const uint32_t m = (1u << ln) - 1u;
  if constexpr (B == 4) {
    const uint32_t y = __funnelshift_r(x0, x1, 2 * ln);
    return make_uint4(x0 & m, (x0 >> ln) & m, y & m, (y >> ln) & m);
  } else {
    return make_uint4(x0 & m, 0u, __funnelshift_r(x0, x1, ln) & m, 0u);
  }
}
template <int B>
__device__ __forceinline__ uint4 codes_wide(const uint32_t* w, int bit, int ln, int lane)  // 16 .. 32 / 32 .. 64
{
  const int at = bit + lane * ((16 / B) * ln);
  const uint32_t* const p = w + (at >> 5);
  const uint32_t w0 = p[0], w1 = p[1], w2 = p[2], w3 = p[3], w4 = p[4];
  const uint32_t x0 = __funnelshift_r(w0, w1, at), x1 = __funnelshift_r(w1, w2, at);
  const uint32_t x2 = __funnelshift_r(w2, w3, at), x3 = __funnelshift_r(w3, w4, at);
  // (shifts of up to 32: the clamping form)
  if constexpr (B == 4) {
    const uint32_t m = pow2_or_0(ln) - 1u;
    const bool far = 3 * ln >= 64;
    return make_uint4(x0 & m, __funnelshift_rc(x0, x1, ln) & m, __funnelshift_rc(x1, x2, 2 * ln - 32) & m,
                      __funnelshift_rc(far ? x2 : x1, far ? x3 : x2, 3 * ln - (far ? 64 : 32)) & m);
  } else {
    const int k = ln - 32;
    const uint32_t m = pow2_or_0(k) - 1u;
    return make_uint4(x0, x1 & m, __funnelshift_rc(x1, x2, k), __funnelshift_rc(x2, x3, k) & m);
  }
}
// one code at bit `at`, of any width
template <typename T>
__device__ __forceinline__ T code_at(const uint32_t* w, int at, int ln)
{
  const uint32_t* const p = w + (at >> 5);
  const uint32_t lo = __funnelshift_r(p[0], p[1], at) & (pow2_or_0(ln) - 1u);
  if constexpr (sizeof(T) == 4) {
    return lo;
  } else {
    const uint32_t hi = ln > 32 ? __funnelshift_r(p[1], p[2], at) & (pow2_or_0(ln - 32) - 1u) : 0u;
    return (static_cast<uint64_t>(hi) << 32) | lo;
  }
}
// 16 raw bytes at any bit offset
__device__ __forceinline__ uint4 codes_full(const uint32_t* w, int bit, int lane)
{
  const int at = bit + lane * 128;
  const uint32_t* const p = w + (at >> 5);
  const uint32_t w0 = p[0], w1 = p[1], w2 = p[2], w3 = p[3], w4 = p[4];
  return make_uint4(__funnelshift_r(w0, w1, at), __funnelshift_r(w1, w2, at), __funnelshift_r(w2, w3, at),
                    __funnelshift_r(w3, w4, at));
}

// A chunk whose output is not 16-byte aligned, or that ends early (a stream's last), with
// the chunk already checked (`ln`: width of subchunk `lane`).  Each lane takes the values
// of 16 aligned bytes of output, which begin `mis` bytes before those of an aligned
// output; the values before a subchunk's first and after its last such granule follow one
// by one, a lane each, for the whole chunk.  (302 MB f64 at eb 1e-4 into a view that begins
// at element 1: 74 us, aligned 64; 26 MB f32 at eb 1e-3 13.7 and 12.6, 67 MB f32 lossless
// 29.7 and 26.6, raw chunks 27.7 and 27.4.  With words at the lanes' own 16 bytes, which
// fill a quarter of each sector per store, 89, 16.2, 29.8 and 30.3; with words moved between
// the lanes by shuffles 99, 16.9, 37 and 27.9.)
template <typename T, bool LOSSY, int TW>
__device__ __forceinline__ void unpack_unaligned(const uint32_t* w, int sft, int ln, int osize, uint8_t* o, const QParams& q,
                                              int cw, int lane)
{
  using V = VT<T>;
  constexpr int B = static_cast<int>(sizeof(T));
  constexpr int P = 16 / B;  // values per lane
  constexpr int NARROW = B == 4 ? 16 : 32;
  const int mis = static_cast<int>(reinterpret_cast<uintptr_t>(o) & 15u);
  const int m = mis / B;
  const bool mine = lane > 0 || mis == 0;  // (else lane 0's first values are the subchunk's before)
  const int last = mine ? osize - 16 - lane * 16 + mis : -1;  // the last subchunk's first byte that has all 16
  const unsigned narrow = __ballot_sync(0xffffffffu, ln < NARROW);
  const unsigned wide = __ballot_sync(0xffffffffu, ln >= NARROW);
#pragma unroll 1
  for (int g = cw; g < SC / DEC_G; g += TW) {
    const int i0 = g * DEC_G;
    const uint32_t lw = __reduce_or_sync(0xffffffffu, (lane / DEC_G) == g ? static_cast<uint32_t>(ln) << (8 * (lane % DEC_G)) : 0u);
    int l[DEC_G], b[DEC_G];
    int bit = 8 * sft + 256 + V::VPS * __reduce_add_sync(0xffffffffu, lane < i0 ? ln : 0);
#pragma unroll
    for (int u = 0; u < DEC_G; ++u) {
      l[u] = static_cast<int>((lw >> (8 * u)) & 0xffu);
      b[u] = bit;
      bit += V::VPS * l[u];
    }
    constexpr unsigned ALL = (1u << DEC_G) - 1u;
    const unsigned nm = (narrow >> i0) & ALL, wm = (wide >> i0) & ALL;
    uint4 e[DEC_G];
    if (nm == ALL) {
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) e[u] = codes_narrow<B>(w, b[u] - m * l[u], l[u], lane);
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) e[u] = decode_codes<T, LOSSY, true>(e[u], q);
    } else if (wm == ALL) {
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) e[u] = codes_wide<B>(w, b[u] - m * l[u], l[u], lane);
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) e[u] = decode_codes<T, LOSSY, false>(e[u], q);
    } else {
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) {
        if ((nm >> u) & 1u) e[u] = codes_narrow<B>(w, b[u] - m * l[u], l[u], lane);
        else e[u] = codes_wide<B>(w, b[u] - m * l[u], l[u], lane);
      }
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) e[u] = decode_codes<T, LOSSY, false>(e[u], q);
    }
#pragma unroll
    for (int u = 0; u < DEC_G; ++u)
      if ((i0 + u) * 512 <= last) store16(o + (i0 + u) * 512 + lane * 16 - mis, e[u]);
  }
  auto one = [&](int at, int bit, int l) { *reinterpret_cast<T*>(o + at) = decode_value<LOSSY>(code_at<T>(w, bit, l), q); };
  const int tail = (osize + mis) & 15;  // the chunk's bytes in the granule that it ends in
  if (tail != 0 && cw == 0) {
    const int at = osize - tail + lane * B;
    const int i = (osize - B) / 512;  // (earlier subchunks' values follow below)
    const int l = __shfl_sync(0xffffffffu, ln, i);
    const int bit = 8 * sft + 256 + V::VPS * __reduce_add_sync(0xffffffffu, lane < i ? ln : 0);
    if (at < osize && at >= i * 512) one(at, bit + (at - i * 512) / B * l, l);
  }
  if (mis != 0) {
    int incl = ln;  // widths up to subchunk `lane`
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += x;
    }
    const int bit = 8 * sft + 256 + V::VPS * (incl - ln);
    for (int j0 = cw * 32; j0 < SC * P; j0 += TW * 32) {
      const int i = (j0 + lane) / P, t = (j0 + lane) % P;
      const int k = t < P - m ? t : V::VPS - P + t;
      const int l = __shfl_sync(0xffffffffu, ln, i);
      const int at = __shfl_sync(0xffffffffu, bit, i) + k * l;
      if (i * 512 + k * B < osize) one(i * 512 + k * B, at, l);
    }
  }
}

// A raw chunk to any output: the output's whole granules, then the words around them.
template <int TW>
__device__ __forceinline__ void copy_raw(const uint32_t* w, int sft, int osize, uint8_t* o, int cw, int lane)
{
  const int mis = static_cast<int>(reinterpret_cast<uintptr_t>(o) & 15u);
  const int b = (16 - mis) & 15;  // bytes before the first granule (the chunk may end earlier)
  const int e = max(b, ((mis + osize) & ~15) - mis);
  for (int at = b + (cw * 32 + lane) * 16; at < e; at += TW * 512) store16(o + at, codes_full(w, 8 * (sft + at), 0));
  if (cw == 0) {
    const int at = lane < 4 ? 4 * lane : e + 4 * (lane - 4);
    if (lane < 4 ? at < min(b, osize) : at < osize && lane < 8)
      *reinterpret_cast<uint32_t*>(o + at) = code_at<uint32_t>(w, 8 * (sft + at), 32);
  }
}

// Decodes one staged chunk (payload at byte `sft` of `stg`, `cs` bytes, `osize` bytes
// out to `o`) with warp `cw` of a team of TW; every warp checks the chunk itself.
// Returns false for a malformed chunk (bit width above the element width, widths not
// adding up to cs, trailer not equal to osize); a raw chunk (cs == osize) is copied.
//
// What bounds it: instruction issue for narrow codes, HBM for wide ones.  A lane takes
// 16 adjacent bytes of output, not every 32nd value: one aligned run of 3 or 5 words
// and one 16-byte store for 4 (2) values, instead of 2 or 3 words, a position and a
// store for each.
template <typename T, bool LOSSY, int TW>
__device__ __forceinline__ bool decode_chunk(const uint8_t* stg, int sft, int cs, int osize, uint8_t* o,
                                             const QParams& q, int cw, int lane)
{
  using V = VT<T>;
  constexpr int B = static_cast<int>(sizeof(T));
  const uint32_t* const w = reinterpret_cast<const uint32_t*>(stg);
  const bool whole = osize == CS && (reinterpret_cast<uintptr_t>(o) & 15u) == 0u;
  if (cs == osize) {
    if (!whole) {
      copy_raw<TW>(w, sft, osize, o, cw, lane);
      return true;
    }
    for (int i = cw; i < SC; i += TW) store16(o + i * 512 + lane * 16, codes_full(w, 8 * sft + i * 4096, lane));
    return true;
  }
  const int ln = stg[sft + lane];
  const int tot = __reduce_add_sync(0xffffffffu, ln * V::VPS);
  bool ok = !__any_sync(0xffffffffu, ln > V::TB) && 34 + tot / 8 == cs;
  if (ok) ok = static_cast<int16_t>(stg[sft + cs - 2] | (stg[sft + cs - 1] << 8)) == osize;
  if (!ok) return false;
  if (!whole) {
    unpack_unaligned<T, LOSSY, TW>(w, sft, ln, osize, o, q, cw, lane);
    return true;
  }
  o += lane * 16;
  // widths of the narrow form, of the wide one, and (32-bit values) without escapes
  constexpr int NARROW = B == 4 ? 16 : 32;
  const unsigned narrow = __ballot_sync(0xffffffffu, ln < NARROW);
  const unsigned wide = __ballot_sync(0xffffffffu, ln >= NARROW);
  const unsigned plain = B == 4 && LOSSY ? __ballot_sync(0xffffffffu, ln < 24) : narrow;
  auto put = [&](int i, const uint4 v) { store16(o + i * 512, v); };
#pragma unroll 1
  for (int g = cw; g < SC / DEC_G; g += TW) {
    const int i0 = g * DEC_G;
    // the group's widths as one warp-uniform word, so that what follows from them
    // is computed once per warp, beside the lanes' own arithmetic
    const uint32_t lw = __reduce_or_sync(0xffffffffu, (lane / DEC_G) == g ? static_cast<uint32_t>(ln) << (8 * (lane % DEC_G)) : 0u);
    int l[DEC_G], b[DEC_G];
    int bit = 8 * sft + 256 + V::VPS * __reduce_add_sync(0xffffffffu, lane < i0 ? ln : 0);
#pragma unroll
    for (int u = 0; u < DEC_G; ++u) {
      l[u] = static_cast<int>((lw >> (8 * u)) & 0xffu);
      b[u] = bit;
      bit += V::VPS * l[u];
    }
    constexpr unsigned ALL = (1u << DEC_G) - 1u;
    const unsigned nm = (narrow >> i0) & ALL, wm = (wide >> i0) & ALL, pm = (plain >> i0) & ALL;
    uint4 e[DEC_G];
    if (nm == ALL) {
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) e[u] = codes_narrow<B>(w, b[u], l[u], lane);
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) put(i0 + u, decode_codes<T, LOSSY, true>(e[u], q));
    } else if (wm == ALL) {
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) e[u] = codes_wide<B>(w, b[u], l[u], lane);
      if (B == 4 && LOSSY && pm == ALL) {
#pragma unroll
        for (int u = 0; u < DEC_G; ++u) put(i0 + u, decode_codes<T, LOSSY, true>(e[u], q));
      } else {
#pragma unroll
        for (int u = 0; u < DEC_G; ++u) put(i0 + u, decode_codes<T, LOSSY, false>(e[u], q));
      }
    } else {
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) {
        if (l[u] < NARROW) e[u] = codes_narrow<B>(w, b[u], l[u], lane);
        else e[u] = codes_wide<B>(w, b[u], l[u], lane);
      }
#pragma unroll
      for (int u = 0; u < DEC_G; ++u) {
        if (!LOSSY || ((pm >> u) & 1u)) put(i0 + u, decode_codes<T, LOSSY, true>(e[u], q));
        else put(i0 + u, decode_codes<T, LOSSY, false>(e[u], q));
      }
    }
  }
  return true;
}

// Barrier among the TW warps of team `team` (named barriers 1 ..); true if any warp
// has `fail`, so that the team leaves together.
template <int TW>
__device__ __forceinline__ bool team_failed(int team, bool fail)
{
  if constexpr (TW == 1) {
    return __any_sync(0xffffffffu, fail);
  } else {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(fail)), "r"(team + 1), "n"(TW * 32)
        : "memory");
    return r != 0;
  }
}

// ---- one buffer --------------------------------------------------------------------

// Chunks' places: every CTA adds up the whole size table, a window of DEC_WINDOW
// chunks (403 MB of output) at a time, into the prefixes before its groups of 64
// chunks, and keeps the table; a chunk's place is its group's prefix plus the sizes of
// the group before it (from L2 instead of shared memory, that took the team 1 us more
// per chunk).
// So any warp can take any chunk, and no CTA waits for another.  (A static range of
// chunks per CTA took 71 us instead of 60 on the 302 MB field: the SMs' ends lay
// between 54 and 71 us.)
constexpr int DEC_GROUPS = 384;
constexpr int DEC_WINDOW = 64 * DEC_GROUPS;

// NTEAM teams of TW warps per CTA, each with one stage.
template <typename T, bool LOSSY, int NTEAM, int TW, int MINB>
__global__ void __launch_bounds__(NTEAM * TW * 32, MINB) k_decode(const DecArgs a)
{
  constexpr int NT = NTEAM * TW * 32;
  constexpr int NW = NT / 32;
  static_assert(NW <= 32, "warps");
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + NTEAM * DEC_STAGE);
  unsigned long long* const sizes8 = reinterpret_cast<unsigned long long*>(bars + 2 * NTEAM);  // the window's size table
  uint32_t* const before = reinterpret_cast<uint32_t*>(sizes8 + DEC_WINDOW / 4);  // per group, from the window's start
  __shared__ uint32_t s_warp[NW];
  __shared__ unsigned long long s_ticket[2][NTEAM];

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int team = warp / TW;
  const int cw = warp % TW;
  if (tid == 0) {
    for (int i = 0; i < 2 * NTEAM; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
  }
  grid_wait();
  const WsPhase ph = WsPhase::of(a.ws, a.flag_cap);  // self-resetting workspace
  uint64_t* const hdr = ph.hdr;
  const uint16_t* const size_in = reinterpret_cast<const uint16_t*>(a.in + 8);

  // The window's size table to `sizes8`, and the sums of its groups into `before` (chunks [w0, end), w0 a
  // multiple of 64): four sizes per 8-byte load, 16 lanes per group.
  auto sum_groups = [&](long long w0, long long end) {
    const int n = static_cast<int>(end - w0);
    const unsigned long long* const s8 = reinterpret_cast<const unsigned long long*>(size_in + w0);
    constexpr int U = 4;  // loads in flight per lane
    for (int k0 = 0; 4 * k0 < n; k0 += U * NT) {
      unsigned long long v[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int k = k0 + u * NT + tid;
        v[u] = 0;
        if (4 * k + 4 <= n) {
          v[u] = s8[k];
        } else {
          for (int x = 0; x < 3; ++x)
            if (4 * k + x < n) v[u] |= static_cast<unsigned long long>(size_in[w0 + 4 * k + x]) << (16 * x);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned long long p2 = (v[u] & 0x0000ffff0000ffffull) + ((v[u] >> 16) & 0x0000ffff0000ffffull);
        uint32_t x = static_cast<uint32_t>(p2) + static_cast<uint32_t>(p2 >> 32);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        const int k = k0 + u * NT + tid;
        if (4 * k < n) sizes8[k] = v[u];
        if ((lane & 15) == 0 && 4 * k < n) before[k / 16] = x;
      }
    }
  };

  // Speculation: when the caller states the output capacity and the stream's
  // length, the chunk count is usually ceil(capacity / CS), and the first window's
  // sizes are added up while the header is still on its way, instead of one
  // dependent round trip after it.  Used only if the header agrees; the reads stay
  // inside the stated stream length.
  const long long g_chunks = a.out_cap > 0 ? chunks_of(a.out_cap) : -1;
  const bool spec = g_chunks > 0 && a.in_len >= 8 + 2 * g_chunks;
  const long long insize = *reinterpret_cast<const long long*>(a.in);
  if (spec) sum_groups(0, min(g_chunks, static_cast<long long>(DEC_WINDOW)));

  // header checks (every CTA reads the 8-byte header)
  const long long chunks_in = insize > 0 ? chunks_of(insize) : 0;
  bool hdr_ok = insize >= 0 && (insize % static_cast<long long>(sizeof(T))) == 0;
  if (a.in_len >= 0 && 8 + 2 * chunks_in > a.in_len) hdr_ok = false;
  const bool cap_ok = a.out_cap < 0 || insize <= a.out_cap;
  if (tid == 0 && blockIdx.x == 0) {
    if (!hdr_ok) set_status(hdr, ST_CORRUPT, -1);
    else if (!cap_ok) set_status(hdr, ST_CAPACITY, -1);
  }
  const long long chunks = hdr_ok && cap_ok ? chunks_in : 0;
  const long long payload_len = a.in_len >= 0 ? a.in_len - 8 - 2 * chunks : -1;
  const uint8_t* const data_in = a.in + 8 + 2 * chunks;

  uint8_t* const stg = smem + team * DEC_STAGE;
  uint64_t* const bar = &bars[2 * team];  // used in turn
  uint32_t par = 0;
  int slot = 0;
  bool left = false;  // a wait of this team gave up

  struct Piece {        // one chunk's bytes in the stream and in the stage
    const uint8_t* src;  // 16-byte aligned
    uint32_t nb;
    int pos, sft, cs;    // cs = 0: the size table does not allow them
  };
  // The first chunks are spread over the CTAs, then each team takes the next one that
  // none has (one warp), or its next in turn (several).
  const long long teams = static_cast<long long>(gridDim.x) * NTEAM;
  long long c = blockIdx.x + static_cast<long long>(team) * gridDim.x;
  unsigned long long ticket = 0;  // drawn by the team's first lane, valid there
  int turn = 0;
  auto draw = [&]() {
    if (lane == 0 && cw == 0 && teams < chunks)
      ticket = teams + atomicAdd(reinterpret_cast<unsigned long long*>(&a.ws[WS_TICKET]), 1ull);
  };
  // the last ticket drawn, for the whole team
  auto drawn = [&]() -> long long {
    if (teams >= chunks) return chunks;
    if constexpr (TW == 1) {
      return static_cast<long long>(__shfl_sync(0xffffffffu, ticket, 0));
    } else {
      if (lane == 0 && cw == 0) s_ticket[turn][team] = ticket;
      team_failed<TW>(team, false);
      const long long t = static_cast<long long>(s_ticket[turn][team]);
      turn ^= 1;
      return t;
    }
  };
  long long wbase = 0;  // payload bytes before the window
  auto place = [&](long long k, long long w0) {
    const int in = static_cast<int>(k & 63);
    // this lane's two sizes of the chunk's group (zeros or an old window's after the last chunk)
    const uint32_t s = reinterpret_cast<const uint32_t*>(sizes8)[static_cast<int>(k - w0) / 64 * 32 + lane];
    uint32_t x = 2 * lane < in ? (s & 0xffffu) : 0u;
    if (2 * lane + 1 < in) x += s >> 16;
    const long long off = wbase + before[(k - w0) / 64] + __reduce_add_sync(0xffffffffu, x);
    const uint32_t pair = __shfl_sync(0xffffffffu, s, in >> 1);
    Piece p;
    p.cs = static_cast<int>(in & 1 ? pair >> 16 : pair & 0xffffu);
    p.pos = 0;
    const uint8_t* const src = data_in + off;
    p.sft = static_cast<int>(reinterpret_cast<uintptr_t>(src) & 15u);
    p.src = src - p.sft;
    p.nb = static_cast<uint32_t>((p.sft + p.cs + 15) & ~15);
    const int os = static_cast<int>(min(static_cast<long long>(CS), insize - k * CS));
    if (p.cs > os || (p.cs < os && p.cs < 34) || (payload_len >= 0 && off + p.cs > payload_len)) p.cs = 0;
    return p;
  };
  auto issue = [&](const Piece& p, uint64_t* b) {
    if (lane == 0 && cw == 0 && p.cs > 0) {
      mbar_arrive_expect_tx(b, p.nb);
      tma_load_1d(stg + p.pos, p.src, p.nb, b);
    }
  };

  for (long long w0 = 0; w0 < chunks; w0 += DEC_WINDOW) {
    const long long wend = min(w0 + DEC_WINDOW, chunks);
    const int groups = static_cast<int>((wend - w0 + 63) / 64);
    if (w0 > 0 || !spec || g_chunks != chunks) {
      __syncthreads();  // the last window's sums are read, or the speculation's written
      sum_groups(w0, wend);
    }
    __syncthreads();
    // exclusive prefixes of the group sums
    uint32_t wtotal = 0;
    for (int g0 = 0; g0 < groups; g0 += NT) {
      const uint32_t v = g0 + tid < groups ? before[g0 + tid] : 0u;
      uint32_t incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      const uint32_t ws = lane < NW ? s_warp[lane] : 0u;
      const uint32_t pre = __reduce_add_sync(0xffffffffu, lane < warp ? ws : 0u);
      if (g0 + tid < groups) before[g0 + tid] = wtotal + pre + incl - v;
      wtotal += __reduce_add_sync(0xffffffffu, ws);
      __syncthreads();
    }

    Piece cur;
    if (c < wend && !left) {
      cur = place(c, w0);
      issue(cur, &bar[slot]);
      draw();
    }
    while (c < wend && !left) {
      // The next chunk's bytes are fetched beside the current ones where both fit
      // (compressed below half), else brought to L2.
      const long long nc = drawn();
      Piece nx;
      bool issued = false;
      if (nc < wend) {
        nx = place(nc, w0);
        if (static_cast<int>(nx.nb) + 16 <= cur.pos) {
          issued = true;
        } else if (cur.pos + static_cast<int>(cur.nb + nx.nb) + 32 <= DEC_STAGE) {
          nx.pos = cur.pos + static_cast<int>(cur.nb) + 16;
          issued = true;
        }
        if (issued) issue(nx, &bar[slot ^ 1]);
        else if (lane == 0 && cw == 0 && nx.cs > 0) prefetch_l2(nx.src, nx.nb);
        draw();
      }
      bool late = false;
      bool ok = cur.cs > 0;
      if (ok) {
        late = !copy_landed(&bar[slot], (par >> slot) & 1u);
        par ^= 1u << slot;
        const int osize = static_cast<int>(min(static_cast<long long>(CS), insize - c * CS));
        uint8_t* const dst = a.out + c * CS;
        if (!late) ok = decode_chunk<T, LOSSY, TW>(stg + cur.pos, cur.sft, cur.cs, osize, dst, a.q, cw, lane);
      }
      report_chunk(hdr, late, ok, cw, lane, c);
      // the stage is read before it is refilled (generic accesses ordered before the TMA write)
      fence_proxy_async_smem();
      left = team_failed<TW>(team, late);
      slot ^= 1;
      c = nc;
      if (c < wend) {
        cur = nx;
        if (!issued && !left) issue(cur, &bar[slot]);
        if (issued && left && cur.cs > 0) mbar_wait_bounded(&bar[slot], (par >> slot) & 1u);  // a copy still landing
      }
    }
    wbase += wtotal;
  }

  // this CTA's share of the flags the previous launch left in the other region
  // (off the start of the kernel: only the next launch reads them)
  if (warp == NW - 1) ph.clear_other_share(lane);

  // ---- epilogue ------------------------------------------------------------------
  grid_release();
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const unsigned long long dn = atomicAdd(reinterpret_cast<unsigned long long*>(&a.ws[WS_DONE]), 1ull);
    if (dn == gridDim.x - 1) {
      __threadfence();
      const unsigned long long st = ld_relaxed_u64(&hdr[WS_STATUS]);
      *a.outsize = st ? -static_cast<long long>(st) : insize;
      ph.finish(a.ws, 0);
    }
  }
}

// ---- batches: a prepass places every chunk, then a persistent kernel decodes them in
// any order, a team per chunk ---------------------------------------------------------

constexpr int DB_TEAMS = 10;
constexpr int DB_TW = 2;  // warps per team
constexpr int DB_NT = DB_TEAMS * DB_TW * 32;
constexpr int DB_SMEM = DB_TEAMS * DEC_STAGE + 8 * DB_TEAMS + 8 * (BATCH_MAX_JOBS + 1);

// Prepass, one CTA per buffer: validates the header and size table and writes each
// chunk's place (byte offset in the stream | size << 48) by an exclusive scan of the
// sizes, 1,024 per step (a step costs two barriers and a round trip to memory: 256
// per step took 6 us more on 16 MB buffers).
constexpr int PRE_NT = 1024;

__global__ void __launch_bounds__(PRE_NT) k_decode_prepass(const BatchDecArgs a)
{
  __shared__ uint32_t wsum[PRE_NT / 32];
  __shared__ int wbad[PRE_NT / 32];
  grid_release();  // at once: the decode kernel, which follows, is set up meanwhile (at the end instead: no change)
  grid_wait();
  const int j = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const BatchJob& job = a.jobs[j];
  const uint8_t* const in = job.in;
  const long long len = job.insize;  // stream bytes, -1 when unknown
  const int elem = (job.kind & 1) ? 8 : 4;
  long long insize = (len < 0 || len >= 8) ? *reinterpret_cast<const long long*>(in) : -1;
  bool ok = insize >= 0 && insize % elem == 0 && insize <= job.cap;
  const long long chunks = ok ? (insize + CS - 1) / CS : 0;
  if (ok && len >= 0 && 8 + 2 * chunks > len) ok = false;
  if (!ok) {
    if (tid == 0) set_status(a.ws, insize > job.cap ? ST_CAPACITY : ST_CORRUPT, j);
    return;
  }
  const uint16_t* const size_in = reinterpret_cast<const uint16_t*>(in + 8);
  unsigned long long* const places = a.places + a.chunk_base[j];
  long long carry = 8 + 2 * chunks;
  int bad = 0;
  for (long long b = 0; b < chunks; b += PRE_NT) {
    const long long c = b + tid;
    uint32_t cs = 0;
    if (c < chunks) {
      cs = size_in[c];
      const uint32_t os = static_cast<uint32_t>(min(static_cast<long long>(CS), insize - c * CS));
      bad |= (cs > os) | (cs == 0) | ((cs < os) & (cs < 34));
    }
    uint32_t incl = cs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    const uint32_t ws = wsum[lane];
    const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? ws : 0u);
    if (c < chunks)
      places[c] = static_cast<unsigned long long>(carry + before + incl - cs) | (static_cast<unsigned long long>(cs) << 48);
    carry += __reduce_add_sync(0xffffffffu, ws);
    __syncthreads();
  }
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) wbad[warp] = bad;
  __syncthreads();
  if (tid == 0) {
    int any = 0;
    for (int w = 0; w < PRE_NT / 32; ++w) any |= wbad[w];
    if (any || (len >= 0 && carry > len)) {
      set_status(a.ws, ST_CORRUPT, j);
    } else {
      a.actual[j] = insize;
      *job.outsize = insize;
    }
  }
}

__global__ void __launch_bounds__(DB_NT, 1) k_decode_batch(const BatchDecArgs a)
{
  extern __shared__ __align__(128) uint8_t smem[];
  uint64_t* const bars = reinterpret_cast<uint64_t*>(smem + DB_TEAMS * DEC_STAGE);
  long long* const cb = reinterpret_cast<long long*>(bars + DB_TEAMS);
  __shared__ unsigned long long s_ticket[2][DB_TEAMS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int team = warp / DB_TW, cw = warp % DB_TW;
  const bool leads = lane == 0 && cw == 0;
  uint64_t* const ws = a.ws;
  if (tid == 0) {
    for (int i = 0; i < DB_TEAMS; ++i) mbar_init(&bars[i], 1);
    mbar_fence_init();
  }
  grid_wait();
  for (int i = tid; i <= a.njobs; i += DB_NT) cb[i] = a.chunk_base[i];
  // the prepass found an error (one thread looks: another CTA may report one meanwhile,
  // and a team's warps have to agree)
  const bool failed_before = __syncthreads_or(tid == 0 && ld_relaxed_u64(&ws[WS_STATUS]) != 0ull) != 0;
  const long long total = cb[a.njobs];
  uint8_t* const stg = smem + team * DEC_STAGE;
  uint64_t* const bar = &bars[team];
  uint32_t par = 0;
  // One chunk's ticket and where it is; the next chunk's are read while the current
  // one is decoded, so that its copy can start at once (61 -> 52 us on 60 arrays of
  // 4 KB to 16 MB).
  struct Item {
    long long c, insize;
    unsigned long long place;
    const uint8_t* in;
    uint8_t* out;
    QParams q;
    int kind;
  };
  unsigned long long ticket = 0;
  int turn = 0;
  auto draw = [&]() {
    if (leads) ticket = atomicAdd(reinterpret_cast<unsigned long long*>(&ws[WS_TICKET]), 1ull);
  };
  auto drawn = [&]() -> long long {
    if (leads) s_ticket[turn][team] = ticket;
    team_failed<DB_TW>(team, false);
    const long long t = static_cast<long long>(s_ticket[turn][team]);
    turn ^= 1;
    return t;
  };
  auto look_up = [&](long long t) {
    Item it;
    it.place = a.places[t];  // 0: the stream holds fewer chunks than its output has room for
    int lo = 0, hi = a.njobs - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (cb[mid] <= t) lo = mid;
      else hi = mid - 1;
    }
    const BatchJob& job = a.jobs[lo];
    it.c = t - cb[lo];
    it.insize = a.actual[lo];
    it.in = job.in;
    it.out = job.out;
    it.q = job.q;
    it.kind = job.kind;
    return it;
  };
  draw();
  long long t = failed_before ? total : drawn();
  Item it;
  if (t < total) it = look_up(t);
  while (t < total) {
    const int cs = static_cast<int>(it.place >> 48);
    const uint8_t* const src = it.in + (it.place & 0xffffffffffffull);
    const int sft = static_cast<int>(reinterpret_cast<uintptr_t>(src) & 15u);
    if (leads && cs > 0) {
      const uint32_t nb = static_cast<uint32_t>((sft + cs + 15) & ~15);
      mbar_arrive_expect_tx(bar, nb);
      tma_load_1d(stg, src - sft, nb, bar);
    }
    draw();
    const Item cur = it;
    const long long ct = t;
    t = drawn();
    if (t < total) it = look_up(t);
    if (cs > 0) {
      const bool late = !copy_landed(bar, par);
      par ^= 1u;
      uint8_t* const out = cur.out + cur.c * CS;
      const int osize = static_cast<int>(min(static_cast<long long>(CS), cur.insize - cur.c * CS));
      bool ok = true;
      if (!late) switch (cur.kind) {
        case 0: ok = decode_chunk<uint32_t, false, DB_TW>(stg, sft, cs, osize, out, cur.q, cw, lane); break;
        case 1: ok = decode_chunk<uint64_t, false, DB_TW>(stg, sft, cs, osize, out, cur.q, cw, lane); break;
        case 2: ok = decode_chunk<uint32_t, true, DB_TW>(stg, sft, cs, osize, out, cur.q, cw, lane); break;
        default: ok = decode_chunk<uint64_t, true, DB_TW>(stg, sft, cs, osize, out, cur.q, cw, lane); break;
      }
      report_chunk(ws, late, ok, cw, lane, ct);
      // the stage is read before it is refilled (generic accesses ordered before the TMA write)
      fence_proxy_async_smem();
      if (team_failed<DB_TW>(team, late)) break;
    }
  }

  // ---- epilogue: an error anywhere turns every size into -status ---------------
  grid_release();
  __syncthreads();
  __shared__ int last_cta;
  if (tid == 0) {
    __threadfence();
    const unsigned long long dn = atomicAdd(reinterpret_cast<unsigned long long*>(&ws[WS_DONE]), 1ull);
    last_cta = dn == gridDim.x - 1;
    if (last_cta) __threadfence();
  }
  __syncthreads();
  if (last_cta) {
    const unsigned long long st = ld_relaxed_u64(&ws[WS_STATUS]);
    if (st)
      for (int i = tid; i < a.njobs; i += DB_NT) *a.jobs[i].outsize = -static_cast<long long>(st);
  }
}

// ---- launchers ---------------------------------------------------------------------

// Launch shapes: teams per CTA, warps per team and CTAs per SM (index = the C ABI's
// shape number).
template <int NTEAM_, int TW_, int MINB_>
struct DecShape {
  static constexpr int NTEAM = NTEAM_;
  static constexpr int TW = TW_;
  static constexpr int MINB = MINB_;
  static constexpr int NT = NTEAM * TW * 32;
  static constexpr int SMEM = NTEAM * DEC_STAGE + 16 * NTEAM + 2 * DEC_WINDOW + 4 * DEC_GROUPS;
};
//
// Shape 0: six chunks in flight per SM, two warps each.  Not more: the 302 MB field at
// eb 1e-4 (75 MB in, 302 MB out) takes 65.8 us with 6 or 7 teams of two and 78 us with
// 8, or with 10 teams of one, whose reads and writes interleave more (71 with 5, 78
// with 4 teams of two, which do not cover the latencies).
using DecShape0 = DecShape<6, 2, 1>;  // default
using DecShape1 = DecShape<10, 1, 1>;
using DecShape2 = DecShape<2, 8, 2>;
constexpr int DEC_SHAPES = 3;
// Index DEC_SHAPES, past the shapes that can be asked for: shape 2 for at most one chunk
// per SM, with the registers of one CTA per SM.  With those of two, some of which are
// spilled, one 4 KB chunk takes 5.03 us on the GPU instead of 4.86, but large inputs that
// ask for shape 2 want two CTAs (302 MB f64 at eb 1e-4 87 us, 110 with one).
using DecShapeSmall = DecShape<2, 8, 1>;

template <typename T, bool LOSSY, class S>
static cudaError_t launch_dec_k(const DecArgs& a, int grid, cudaStream_t st)
{
  auto k = k_decode<T, LOSSY, S::NTEAM, S::TW, S::MINB>;
  static unsigned long long attr = 0;
  cudaError_t e = ensure_smem_attr(k, S::SMEM, &attr);
  if (e != cudaSuccess) return e;
  return launch_after(k, grid, S::NT, S::SMEM, st, a);
}

template <typename T, bool LOSSY, class S>
static int dec_occupancy()
{
  auto k = k_decode<T, LOSSY, S::NTEAM, S::TW, S::MINB>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, S::NT, S::SMEM);
  return n;
}

template <typename T, bool LOSSY>
static cudaError_t launch_dec_kind(int shape, const DecArgs& a, int grid, cudaStream_t st)
{
  switch (shape) {
    case 1: return launch_dec_k<T, LOSSY, DecShape1>(a, grid, st);
    case 2: return launch_dec_k<T, LOSSY, DecShape2>(a, grid, st);
    case DEC_SHAPES: return launch_dec_k<T, LOSSY, DecShapeSmall>(a, grid, st);
    default: return launch_dec_k<T, LOSSY, DecShape0>(a, grid, st);
  }
}

template <typename T, bool LOSSY>
static int dec_occupancy_kind(int shape)
{
  switch (shape) {
    case 1: return dec_occupancy<T, LOSSY, DecShape1>();
    case 2: return dec_occupancy<T, LOSSY, DecShape2>();
    case DEC_SHAPES: return dec_occupancy<T, LOSSY, DecShapeSmall>();
    default: return dec_occupancy<T, LOSSY, DecShape0>();
  }
}

cudaError_t launch_decode(int width, bool lossy, int shape, const DecArgs& a, int grid, cudaStream_t st)
{
  if (width == 4)
    return lossy ? launch_dec_kind<uint32_t, true>(shape, a, grid, st) : launch_dec_kind<uint32_t, false>(shape, a, grid, st);
  return lossy ? launch_dec_kind<uint64_t, true>(shape, a, grid, st) : launch_dec_kind<uint64_t, false>(shape, a, grid, st);
}

int blocks_per_sm(int width, bool lossy, bool enc, int shape)
{
  if (enc) return encode_blocks_per_sm(width, lossy, shape);
  if (width == 4) return lossy ? dec_occupancy_kind<uint32_t, true>(shape) : dec_occupancy_kind<uint32_t, false>(shape);
  return lossy ? dec_occupancy_kind<uint64_t, true>(shape) : dec_occupancy_kind<uint64_t, false>(shape);
}

ShapeInfo shape_info(bool enc, int shape)
{
  if (enc) return encode_shape_info(shape);
  switch (shape) {
    case 1: return {DecShape1::NT, DecShape1::NT / 32, DecShape1::NTEAM, DecShape1::MINB};
    case 2: return {DecShape2::NT, DecShape2::NT / 32, DecShape2::NTEAM, DecShape2::MINB};
    default: return {DecShape0::NT, DecShape0::NT / 32, DecShape0::NTEAM, DecShape0::MINB};
  }
}

int shape_count(bool enc) { return enc ? encode_shape_count() : DEC_SHAPES; }

// Decode with at most one chunk per SM: eight warps share a chunk (f32 lossless,
// microseconds on the GPU against shape 0's: 200 KB 6.0 / 6.5, 1.6 MB 6.1 / 6.4; with more
// chunks its larger CTAs cost more than they gain: 3 MB 7.6 / 6.1).
int default_shape(bool enc, long long chunks, int sms, int ctas)
{
  if (enc) return encode_default_shape(chunks, sms, ctas);
  return chunks <= sms ? DEC_SHAPES : 0;
}

cudaError_t launch_decode_batch(const BatchDecArgs& a, int grid, cudaStream_t st)
{
  cudaError_t e = launch_after(k_decode_prepass, a.njobs, PRE_NT, 0, st, a);
  if (e != cudaSuccess) return e;
  static unsigned long long attr = 0;
  e = ensure_smem_attr(k_decode_batch, DB_SMEM, &attr);
  if (e != cudaSuccess) return e;
  return launch_after(k_decode_batch, grid, DB_NT, DB_SMEM, st, a);
}

int decode_batch_blocks_per_sm()
{
  cudaFuncSetAttribute(k_decode_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, DB_SMEM);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_decode_batch, DB_NT, DB_SMEM);
  return n;
}

}  // namespace sleek
