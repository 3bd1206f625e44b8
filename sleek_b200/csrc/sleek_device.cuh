// sleek_device.cuh -- device building blocks of the sm_100a SLEEK codec.
//
// Everything here is integer / bit arithmetic.  The value transforms restate the
// reference's arithmetic exactly (that is what makes the byte stream identical);
// the data movement (TMA bulk copies to and from shared memory, packing in place,
// bounded waits for the chunks' places) is this project's own.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "sleek_launch.h"

namespace sleek {

constexpr int CS = 16384;          // chunk bytes; fixed by the stream format
constexpr int SC = 32;             // subchunks per chunk; fixed by the stream format

// status codes shared with the C ABI (include/sleek_capi.h)
constexpr unsigned ST_CORRUPT = 5;
constexpr unsigned ST_TIMEOUT = 6;
constexpr unsigned ST_CAPACITY = 9;

// Workspace: 32 header words (u64 each), then the chunks' sizes and their groups'
// sums (ChunkScan).  Words 0 and 1 are the launch's ticket and done counters; two blocks of per-launch results
// (status, total, error position, flags used) follow at words 0-7 and 8-15 (the
// first block shares its first two words with the counters), then the launch
// epoch (word 16) and words the range reduction uses (24-26).  Single-buffer
// launches alternate between the blocks and between two flag regions by epoch
// parity (see WsPhase below); batched launches use block 0 and the first region
// of a workspace cleared before each run.
enum WsWord {
  WS_TICKET = 0, WS_DONE = 1,                                   // counters (words 0, 1)
  WS_STATUS = 2, WS_TOTAL = 3, WS_ERRPOS = 4, WS_USED = 5,      // within a block
  WS_BLOCK = 8,       // words per block
  WS_EPOCH = 16,      // launches completed on this workspace
  WS_MINMAX = 24,     // three words for the range reduction (cleared by its own call)
  WS_HDR_WORDS = 32
};

// a published word whose value may be 0: bit 63 set, the value below
constexpr uint64_t FLAG_SET = 1ull << 63;
constexpr uint64_t FLAG_VAL = FLAG_SET - 1;

constexpr unsigned long long SPIN_TIMEOUT_NS = 4000000000ull;  // 4 s of wall time per wait

// ----------------------------------------------------------------------------
// value traits
// ----------------------------------------------------------------------------
template <typename T> struct VT;
template <> struct VT<uint32_t> {
  static constexpr int TB = 32;            // bits per value
  static constexpr int VPC = CS / 4;       // values per chunk
  static constexpr int VPS = VPC / SC;     // values per subchunk (128)
};
template <> struct VT<uint64_t> {
  static constexpr int TB = 64;
  static constexpr int VPC = CS / 8;
  static constexpr int VPS = VPC / SC;     // 64
};

// ----------------------------------------------------------------------------
// PTX helpers
// ----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long globaltimer_ns()
{
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init()
{
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Tests the phase with the given parity; a thread whose phase is not complete
// is suspended until it completes (or about 0.5 ms pass), so waiting warps do
// not spin on issue slots.
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(500000u)
      : "memory");
  return ok != 0;
}

// Waits for the phase with the given parity; gives up after `limit_ns`.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity,
                                                  unsigned long long limit_ns = SPIN_TIMEOUT_NS)
{
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (globaltimer_ns() - t0 > limit_ns) return false;
  }
  return true;
}

// One warp: the bulk copy counted on `bar` has landed.  False if it has not within
// `limit_ns`; then the warp, which is about to leave, has waited for it once more, so
// that it does not land in shared memory that belongs to another CTA by then.
__device__ __forceinline__ bool copy_landed(uint64_t* bar, uint32_t parity,
                                            unsigned long long limit_ns = SPIN_TIMEOUT_NS)
{
#pragma unroll 1
  for (int k = 0; k < 2; ++k)
    if (__all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, limit_ns))) return k == 0;
  return false;
}

// 1-D bulk copy global -> shared (no multicast); completion counted on `bar`.
__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// 1-D bulk copy shared -> global (16-byte aligned addresses and size), in the
// calling thread's current bulk group.
__device__ __forceinline__ void tma_store_1d(void* dst, const void* src, uint32_t bytes)
{
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)), "r"(bytes)
               : "memory");
}

// Programmatic dependent launch: a kernel launched by launch_after may be set up while
// the kernel before it on the stream still runs.  grid_wait returns once that kernel
// has ended and its writes are visible; nothing in global memory is touched before it.
// grid_release lets the next kernel be set up: at a kernel's end, when its own CTAs are
// through (released at the start, the next kernel's CTAs would hold SMs of other
// streams' kernels while they wait; it gains no more).  A call after a call of the same
// stream takes 2 to 3 us less: 26 MB f32 eb 1e-3 compress 18.3 -> 15.2 us, decompress
// 14.3 -> 11.9; batch of 60 arrays, decompress (memset, prepass, decode) 56.4 -> 51.4.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// brings `bytes` (a multiple of 16, at a 16-byte aligned address) into L2
__device__ __forceinline__ void prefetch_l2(const void* src, uint32_t bytes)
{
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the thread's bulk stores have read their shared memory
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
// the thread's bulk stores are complete
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Asynchronous copy of N = 4, 8 or 16 bytes global -> shared, of which the first
// `have` are read and the rest zero-filled.
template <int N>
__device__ __forceinline__ void cp_async(void* dst, const void* src, int have)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(dst)), "l"(src), "n"(N), "r"(have)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void fence_proxy_async_smem()
{
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// Flags carry their own value, so publishing one needs no ordering against the
// thread's earlier stores (a release would wait for the chunk stores in flight).
__device__ __forceinline__ void st_relaxed_u64(uint64_t* p, uint64_t v)
{
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void st_relaxed_u32(uint32_t* p, uint32_t v)
{
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ uint64_t ld_relaxed_u64(const uint64_t* p)
{
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// records the first error in a counter block; later errors keep the first code
__device__ __forceinline__ void set_status(uint64_t* hdr, unsigned code, long long pos)
{
  if (atomicCAS(reinterpret_cast<unsigned long long*>(&hdr[WS_STATUS]), 0ull, (unsigned long long)code) == 0ull) {
    atomicExch(reinterpret_cast<unsigned long long*>(&hdr[WS_ERRPOS]), (unsigned long long)pos);
  }
}

// What became of a chunk that a team of warps decoded: each warp (`cw` of its team)
// reports its own wait that gave up, since the others' may have ended well; what is
// wrong with the chunk itself they all see, so the first reports it.
__device__ __forceinline__ void report_chunk(uint64_t* hdr, bool late, bool ok, int cw, int lane, long long pos)
{
  if (lane == 0 && (late || (!ok && cw == 0))) set_status(hdr, late ? ST_TIMEOUT : ST_CORRUPT, pos);
}

// ----------------------------------------------------------------------------
// Self-resetting workspace of the single-buffer kernels.  A launch works in
// result block and flag region p = epoch & 1 (both clean when it starts), and
// leaves the other parity clean for the next launch: every CTA clears its share
// of the flags the previous launch used there, and the last CTA resets that
// block and the ticket and done counters, records how many flags this launch
// used, then advances the epoch.  The counters do not depend on the epoch, so a
// CTA takes its first ticket without waiting for the epoch's load.  A workspace
// that starts zeroed therefore needs no clearing between launches on one stream;
// a workspace cleared before every launch (epoch 0) behaves the same.  flag_cap
// is the size of one flag region.
// ----------------------------------------------------------------------------
struct WsPhase {
  uint64_t* hdr;        // this launch's counter block
  uint64_t* hdr_other;  // the other block (the previous launch's)
  uint64_t* flags;      // this launch's flag region
  uint64_t* flags_other;
  uint64_t epoch;
  long long used_other;  // flags the previous launch left in the other region

  // The epoch and the other block's flag count were written by an earlier launch
  // and do not change before every CTA of this one has read them, so they are
  // plain loads, free to overlap the kernel's other start-up loads (a volatile
  // load would order them first: measured -7 % on 26 MB decodes).
  __device__ static WsPhase of(uint64_t* ws, long long flag_cap)
  {
    WsPhase w;
    w.epoch = ws[WS_EPOCH];
    const int p = static_cast<int>(w.epoch & 1u);
    w.hdr = ws + WS_BLOCK * p;
    w.hdr_other = ws + WS_BLOCK * (1 - p);
    w.flags = ws + WS_HDR_WORDS + flag_cap * p;
    w.flags_other = ws + WS_HDR_WORDS + flag_cap * (1 - p);
    w.used_other = static_cast<long long>(w.hdr_other[WS_USED]);
    return w;
  }

  // block 0 and the first flag region, nothing to clear (a workspace cleared
  // before each launch, as the batched launches use it)
  __device__ static WsPhase fixed(uint64_t* ws)
  {
    WsPhase w;
    w.epoch = 0;
    w.hdr = ws;
    w.hdr_other = ws + WS_BLOCK;
    w.flags = ws + WS_HDR_WORDS;
    w.flags_other = w.flags;
    w.used_other = 0;
    return w;
  }

  // this CTA's share of the other region's flags, by the calling warp
  __device__ void clear_other_share(int lane) const
  {
    const long long per = (used_other + gridDim.x - 1) / gridDim.x;
    const long long b = per * blockIdx.x;
    const long long e = min(b + per, used_other);
    for (long long i = b + lane; i < e; i += 32) flags_other[i] = 0ull;
  }

  // the last CTA, one thread, after every CTA has counted itself done (so no
  // ticket or done atomic of this launch is still to come)
  __device__ void finish(uint64_t* ws, long long used) const
  {
    hdr[WS_USED] = static_cast<uint64_t>(used);
#pragma unroll
    for (int i = WS_STATUS; i < WS_BLOCK; ++i) hdr_other[i] = 0ull;
    ws[WS_TICKET] = 0ull;
    ws[WS_DONE] = 0ull;
    __threadfence();
    ws[WS_EPOCH] = epoch + 1u;
  }
};

// ----------------------------------------------------------------------------
// value transforms (restated from include/sleek_common_gpu.h of the reference:
// lossless forward :356-374, inverse :614-632, quantize :776-802, deQuantize
// :1077-1108).  Bit-exactness of the stream depends on these being identical.
// ----------------------------------------------------------------------------
// The reference's forward step, on the rotated word v with exponent field
// E = v >> 24: if E != 0, subtract 2^31, then subtract one more exponent unit if
// the field became 0 or the top bit is set; then (v << 1) ^ (v >> 31 arithmetic).
// Case by case the sum adds 0 (E = 0), 2^31 - 2^24 (1 <= E <= 0x80) or 2^31
// (E > 0x80) mod 2^32, and only the middle case ends with the top bit set.  With
// t = 2 v mod 2^32 that is t, or ~(t - 2^25) in the middle case, which is where
// v - 2^24 is non-negative as a signed number (equal on all 2^32 inputs).
__device__ __forceinline__ uint32_t fwd(uint32_t x)
{
  const uint32_t v = __funnelshift_l(x, x, 1);
  const uint32_t t = v + v;
  return static_cast<int32_t>(v - 0x01000000u) >= 0 ? 0x01ffffffu - t : t;
}

// The same step on 64-bit values (11-bit exponent field), on 32-bit halves: the
// case and the subtraction touch only the high word, so the low word of t is
// inverted or kept.
__device__ __forceinline__ uint64_t fwd(uint64_t x)
{
  const uint32_t h = static_cast<uint32_t>(x >> 32);
  const uint32_t l = static_cast<uint32_t>(x);
  const uint32_t nl = __funnelshift_l(h, l, 1);  // low word of v: rotated left by 1
  uint32_t th = __funnelshift_l(l, h, 2);        // high word of t (v's shifted left once more)
  uint32_t tl = nl + nl;
  if (static_cast<int32_t>(h + h - 0x00200000u) >= 0) {  // v's lowest high bit does not matter here
    th = 0x003fffffu - th;
    tl = ~tl;
  }
  return (static_cast<uint64_t>(th) << 32) | tl;
}

// The inverse, without branches.  With r the code rotated right by 1 (its lowest bit
// on top): an odd code is the middle case's ~(2 w), so r = ~w and v = w + 2^24; an
// even one is 2 v mod 2^32 with the bit that 2 v lost set exactly where the exponent
// field is not 0.
__device__ __forceinline__ uint32_t inv(uint32_t o)
{
  const uint32_t r = __funnelshift_r(o, o, 1);
  const uint32_t even = static_cast<int32_t>(r) >= 0x01000000 ? r + 0x80000000u : r;
  const uint32_t v = static_cast<int32_t>(r) < 0 ? 0x00ffffffu - r : even;
  return __funnelshift_r(v, v, 1);
}

__device__ __forceinline__ uint64_t inv(uint64_t o)
{
  const uint32_t h = static_cast<uint32_t>(o >> 32);
  const uint32_t l = static_cast<uint32_t>(o);
  const uint32_t rh = __funnelshift_r(h, l, 1);
  const uint32_t rl = __funnelshift_r(l, h, 1);
  const uint32_t even = static_cast<int32_t>(rh) >= 0x00200000 ? rh + 0x80000000u : rh;
  const bool odd = static_cast<int32_t>(rh) < 0;
  const uint32_t vh = odd ? 0x001fffffu - rh : even;
  const uint32_t vl = odd ? ~rl : rl;
  const uint32_t xh = __funnelshift_r(vh, vl, 1);
  const uint32_t xl = __funnelshift_r(vl, vh, 1);
  return (static_cast<uint64_t>(xh) << 32) | xl;
}

__device__ __forceinline__ uint32_t quant(uint32_t val, const QParams& q)
{
  const uint32_t a = val & 0x7fffffffu;
  const int ve = static_cast<int>(a >> 23);
  uint32_t enc = 0;
  if (ve >= q.thr_e) {
    enc = a - static_cast<uint32_t>(q.offs);
  } else if (ve >= q.eb_e) {
    const int sh = q.thr_e - ve;
    const uint32_t mant = ((val & 0x007fffffu) | 0x00800000u) + (1u << (sh - 1));
    enc = mant >> sh;
  }
  enc = (enc << 1) | ((~val) >> 31);
  return enc ? enc - 1u : 0u;
}

// 64-bit quantize on 32-bit halves (same arithmetic as the 64-bit form: the
// rounding add carries into the high word, the shift is a funnel shift).
__device__ __forceinline__ uint64_t quant(uint64_t val, const QParams& q)
{
  const uint32_t h = static_cast<uint32_t>(val >> 32);
  const uint32_t l = static_cast<uint32_t>(val);
  const uint32_t ah = h & 0x7fffffffu;
  const int ve = static_cast<int>(ah >> 20);
  uint32_t eh = 0, el = 0;
  if (ve >= q.thr_e) {
    const uint32_t oh = static_cast<uint32_t>(q.offs >> 32);
    const uint32_t ol = static_cast<uint32_t>(q.offs);
    el = l - ol;
    eh = ah - oh - (l < ol ? 1u : 0u);
  } else if (ve >= q.eb_e) {
    const int sh = q.thr_e - ve;  // 1 .. 53
    uint32_t mh = (h & 0x000fffffu) | 0x00100000u;
    uint32_t ml = l;
    const int b = sh - 1;
    if (b < 32) {
      const uint32_t add = 1u << b;
      ml += add;
      mh += ml < add ? 1u : 0u;
    } else {
      mh += 1u << (b - 32);
    }
    if (sh < 32) {
      el = __funnelshift_r(ml, mh, sh);
      eh = mh >> sh;
    } else {
      el = mh >> (sh - 32);
    }
  }
  uint32_t rh = __funnelshift_l(el, eh, 1);
  uint32_t rl = (el << 1) | ((h >> 31) ^ 1u);
  if (rh | rl) {
    rh -= rl == 0u ? 1u : 0u;
    rl -= 1u;
  }
  return (static_cast<uint64_t>(rh) << 32) | rl;
}

__device__ __forceinline__ uint32_t dequant(uint32_t enc, const QParams& q)
{
  if (enc == 0u) return 0u;
  const uint32_t a = (enc + 1u) >> 1;
  uint32_t dec = 0;
  if (a >= (1u << 23)) {
    dec = a + static_cast<uint32_t>(q.offs);
  } else if (a > 0u) {
    const int sh = __clz(a) - 8;
    dec = ((a << sh) & 0x007fffffu) | (static_cast<uint32_t>(q.thr_e - sh) << 23);
  }
  return dec | (enc << 31);
}

// 64-bit dequantize on 32-bit halves.
__device__ __forceinline__ uint64_t dequant(uint64_t enc, const QParams& q)
{
  const uint32_t eh = static_cast<uint32_t>(enc >> 32);
  const uint32_t el = static_cast<uint32_t>(enc);
  if ((eh | el) == 0u) return 0ull;
  const uint32_t tl = el + 1u;                      // (enc + 1) >> 1, wrapping like the 64-bit form
  const uint32_t th = eh + (tl == 0u ? 1u : 0u);
  const uint32_t ah = th >> 1;
  const uint32_t al = __funnelshift_r(tl, th, 1);
  uint32_t dh = 0, dl = 0;
  if (ah >= (1u << 20)) {                            // a >= 2^52: stored losslessly
    const uint32_t oh = static_cast<uint32_t>(q.offs >> 32);
    const uint32_t ol = static_cast<uint32_t>(q.offs);
    dl = al + ol;
    dh = ah + oh + (dl < ol ? 1u : 0u);
  } else if ((ah | al) != 0u) {
    const int lz = ah ? __clz(ah) : 32 + __clz(al);
    const int sh = lz - 11;                          // normalise the leading 1 to bit 52
    if (sh < 32) {
      dh = __funnelshift_l(al, ah, sh);
      dl = al << sh;
    } else {
      dh = al << (sh - 32);
    }
    dh = (dh & 0x000fffffu) | (static_cast<uint32_t>(q.thr_e - sh) << 20);
  }
  dh |= el << 31;                                    // sign from the lowest bit
  return (static_cast<uint64_t>(dh) << 32) | dl;
}

// ----------------------------------------------------------------------------
// The same quantize / dequantize with the rounding division done in floating
// point (the integer forms above stay the definition; these are exact rewrites).
//
// Dequantize: for 0 < a < 2^m the integer form normalises a and sets the
// exponent to thr_e - shift, which is the IEEE value a * 2^(thr_e - bias - m):
// the int -> float conversion of a is exact (a < 2^m) and the power-of-two
// product is exact and normal (its exponent field is at least thr_e - m >= 1).
//
// Quantize: for eb_e <= e < thr_e the integer form computes
// floor((M + 2^(sh-1)) / 2^sh), M the significand with its implicit bit and
// sh = thr_e - e.  With y = |v| * 2^(bias + m - thr_e) = M / 2^sh (exact: a
// power-of-two scaling of a normal number with a normal result, y >= 1/2),
// that is floor(y + 1/2).  y + 1/2 = N / 2^sh with N < 2^(m+2) is exact unless
// N needs m + 2 bits and is odd; then rounding toward minus infinity yields
// (N - 1) / 2^sh, and N odd with sh >= 1 means floor((N - 1) / 2^sh) =
// floor(N / 2^sh).  So trunc(round_down(y + 1/2)) is exact.  Denormal values
// (e = 0) are quantized only when eb_e = 0, where the integer form still adds
// the implicit bit; that case keeps the integer form.
//
// Below eb_e the integer form gives 0, and so does eq without a test: e < eb_e
// means |v| < 2^(eb_e - bias), so y < 2^(eb_e + m - thr_e) = 1/2 (thr_e =
// eb_e + m + 1), y + 1/2 < 1 and its round-down truncates to 0 (a product that
// underflows is rounded, but far below 1/2).
//
// The sign step `e2 = (enc << 1) | !sign; e2 ? e2 - 1 : 0` is written as
// `(enc << 1) - (enc ? sign : 0)`: for enc > 0 both are 2 enc - sign, and for
// enc = 0 both are 0 (e2 is 1 - sign there).
// ----------------------------------------------------------------------------
__device__ __forceinline__ uint32_t quant_fp(uint32_t val, const QParams& q)
{
  if (q.eb_e == 0) return quant(val, q);
  const uint32_t a = val & 0x7fffffffu;
  const int ve = static_cast<int>(a >> 23);
  const float inv_scale = __uint_as_float(static_cast<uint32_t>(277 - q.thr_e) << 23);  // 2^(150 - thr_e)
  const uint32_t eq = __float2uint_rz(__fadd_rd(__fmul_rn(__uint_as_float(a), inv_scale), 0.5f));
  const uint32_t enc = ve >= q.thr_e ? a - static_cast<uint32_t>(q.offs) : eq;
  return (enc << 1) - (enc ? (val >> 31) : 0u);
}

__device__ __forceinline__ uint64_t quant_fp(uint64_t val, const QParams& q)
{
  if (q.eb_e == 0) return quant(val, q);
  const uint64_t a = val & 0x7fffffffffffffffull;
  const int ve = static_cast<int>(a >> 52);
  const double inv_scale = __longlong_as_double(static_cast<long long>(2098 - q.thr_e) << 52);  // 2^(1075 - thr_e)
  const uint64_t eq = __double2ull_rz(__dadd_rd(__dmul_rn(__longlong_as_double(static_cast<long long>(a)), inv_scale), 0.5));
  const uint64_t enc = ve >= q.thr_e ? a - q.offs : eq;
  return (enc << 1) - (enc ? (val >> 63) : 0ull);
}

// (A code of 0 needs no test: a, the product and the sign are 0.  Without the branch
// 2^25 f32 values of random bits at eb 1e-3, nearly all escapes, decode in 48 us, not 68.)
__device__ __forceinline__ uint32_t dequant_fp(uint32_t enc, const QParams& q)
{
  const uint32_t a = (enc + 1u) >> 1;
  const float scale = __uint_as_float(static_cast<uint32_t>(q.thr_e - 23) << 23);  // 2^(thr_e - 150)
  const uint32_t dec = a >= (1u << 23) ? a + static_cast<uint32_t>(q.offs)
                                       : __float_as_uint(__fmul_rn(__uint2float_rn(a), scale));
  return dec | (enc << 31);
}

__device__ __forceinline__ uint64_t dequant_fp(uint64_t enc, const QParams& q)
{
  const uint64_t a = (enc + 1ull) >> 1;
  const double scale = __longlong_as_double(static_cast<long long>(q.thr_e - 52) << 52);  // 2^(thr_e - 1075)
  const uint64_t dec = a >= (1ull << 52) ? a + q.offs
                                         : static_cast<uint64_t>(__double_as_longlong(__dmul_rn(__ull2double_rn(a), scale)));
  return dec | (enc << 63);
}

// The same for codes that cannot be escapes, as every code of a narrow subchunk: with
// z the code's zigzag integer (enc / 2, or -(enc + 1) / 2 for odd codes; its magnitude
// is a above and its sign the value's), the value is z * 2^(thr_e - bias - m), both
// factors and the product exact.  32-bit codes below 2^23, 64-bit ones below 2^32.
__device__ __forceinline__ uint32_t dequant_plain32(uint32_t enc, const QParams& q)
{
  const int z = static_cast<int>((enc >> 1) ^ (0u - (enc & 1u)));
  const float scale = __uint_as_float(static_cast<uint32_t>(q.thr_e - 23) << 23);
  return __float_as_uint(__fmul_rn(__int2float_rn(z), scale));
}

__device__ __forceinline__ uint64_t dequant_plain64(uint32_t enc, const QParams& q)
{
  const int z = static_cast<int>((enc >> 1) ^ (0u - (enc & 1u)));
  const double scale = __longlong_as_double(static_cast<long long>(q.thr_e - 52) << 52);
  return static_cast<uint64_t>(__double_as_longlong(__dmul_rn(__int2double_rn(z), scale)));
}

// Quantize for ordinary values, as nearly all are: |v| below quant_limit, which
// excludes escapes, NaN and infinities (and every value where eb_e = 0, whose integer
// form differs), and for 64-bit values keeps the code below 2^31.  floor(y + 1/2) as
// one fused multiply-add rounded down and its integer part (see above); then
// 2 enc - sign, but 0 for enc = 0.  The 64-bit limit is a high word, compared as a float: words that
// are no number as a float are large.
__device__ __forceinline__ float quant_limit32(const QParams& q)
{
  return q.eb_e ? __uint_as_float(static_cast<uint32_t>(q.thr_e) << 23) : 0.0f;
}
__device__ __forceinline__ float quant_limit64(const QParams& q)
{
  return q.eb_e ? __uint_as_float(static_cast<uint32_t>(q.thr_e - 23) << 20) : 0.0f;
}
__device__ __forceinline__ bool quant_ordinary(uint32_t word, float limit)  // a value, or a 64-bit value's high word
{
  return fabsf(__uint_as_float(word)) < limit;
}
__device__ __forceinline__ uint32_t quant_plain(uint32_t v, float inv_scale)
{
  // t <= 2^23, so 2^23 + t rounded down is 2^23 + floor(t), whose bits are those of
  // 2^23 plus floor(t): no conversion, of which an SM does 16 a cycle (40 MB f32 slab
  // 34.1 -> 33.4 us, batch of 60 arrays 68.1 -> 67.2)
  const float t = __fmaf_rd(fabsf(__uint_as_float(v)), inv_scale, 0.5f);
  const uint32_t e = __float_as_uint(__fadd_rd(t, 8388608.0f));  // + 0x4b000000
  const uint32_t c = 0x6a000000u + static_cast<uint32_t>(static_cast<int32_t>(v) >> 31);  // -2 * 0x4b000000 - sign
  return static_cast<uint32_t>(max(static_cast<int>(2u * e + c), 0));
}
__device__ __forceinline__ uint32_t quant_plain(uint32_t l, uint32_t h, double inv_scale)
{
  const double v = fabs(__hiloint2double(static_cast<int>(h), static_cast<int>(l)));
  const uint32_t e = __double2uint_rz(__fma_rd(v, inv_scale, 0.5));
  return static_cast<uint32_t>(max(static_cast<int>(2u * e - (h >> 31)), 0));
}
__device__ __forceinline__ float quant_scale32(const QParams& q)  // 2^(150 - thr_e)
{
  return __uint_as_float(static_cast<uint32_t>(277 - q.thr_e) << 23);
}
__device__ __forceinline__ double quant_scale64(const QParams& q)  // 2^(1075 - thr_e)
{
  return __longlong_as_double(static_cast<long long>(2098 - q.thr_e) << 52);
}

// 2^n for n < 32, 0 for larger n
__device__ __forceinline__ uint32_t pow2_or_0(int n)
{
  uint32_t r;
  asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(n));
  return r;
}

template <bool LOSSY, typename T>
__device__ __forceinline__ T encode_value(T v, const QParams& q)
{
  if constexpr (LOSSY) return quant_fp(v, q);
  else return fwd(v);
}

template <bool LOSSY, typename T>
__device__ __forceinline__ T decode_value(T v, const QParams& q)
{
  if constexpr (LOSSY) return dequant_fp(v, q);
  else return inv(v);
}

__device__ __forceinline__ long long warp_sum(long long v)
{
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ----------------------------------------------------------------------------
// Encode's placement of chunks.  A chunk publishes its size in a 32-bit flag (0 = not
// yet) and adds it to the sum of its group of 64 consecutive chunks (count in the
// high half).  One warp per CTA, the scanner, follows the groups in order, up to 32
// per poll (2,048 chunks, about as many as are ever in flight), and keeps the
// prefix before each in a ring in shared memory; a chunk's own warp adds the flags
// of its group before it (one 8-byte load per lane).  So a chunk is placed about one
// round trip to L2 after its predecessors are sized, however many they are, and 148
// warps poll the group sums.
// ----------------------------------------------------------------------------
constexpr int GROUP = 64;  // chunks per group
constexpr int RING = 128;  // groups whose prefixes a CTA keeps

// words (8 bytes) of the flags and group sums of `chunks` chunks: at most `chunks`
// (the sums are not used where there is only one group)
__host__ __device__ constexpr long long scan_words(long long chunks)
{
  return (chunks + 1) / 2 + (chunks > GROUP ? (chunks + GROUP - 1) / GROUP : 0);
}

struct ScanRing {
  uint64_t base[RING];  // sizes of all chunks before group i, at i % RING
  long long known;      // groups whose prefix is known: 0 .. known
  int gone;             // warps that have left their chunk loop
};

// Whether the entry of group `own`, read before `known`, was still its own: with
// `known` groups known the scanner is at most writing the 32 after them.
__host__ __device__ constexpr bool ring_holds(long long known, long long own) { return known + 32 < own + RING; }

// The ring and the count of warps that have left change while they are read, and the
// lanes of a warp need not read them at the same time.  So the warp goes on with what
// lane 0 saw: the alignment a chunk is packed at and the branches around warp-wide
// exchanges have to be the same in all lanes.
struct ChunkScan {
  uint32_t* flags;  // per chunk
  uint64_t* sums;   // per group: sum of sizes | count << 32
  long long chunks;
  volatile ScanRing* ring;

  __device__ ChunkScan(uint64_t* region, long long chunks_, ScanRing* ring_)
      : flags(reinterpret_cast<uint32_t*>(region)), sums(region + (chunks_ + 1) / 2), chunks(chunks_), ring(ring_)
  {
  }

  // one thread: the size of chunk `idx` is known
  __device__ void publish(long long idx, uint32_t csize) const
  {
    st_relaxed_u32(flags + idx, csize);
    if (chunks > GROUP)
      asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(sums + idx / GROUP), "l"((1ull << 32) | csize)
                   : "memory");
  }

  // this lane's share of the sizes of chunks [b, e) of one group, and whether they are published
  __device__ bool part(long long b, long long e, int lane, uint32_t* sum) const
  {
    const long long i = b / GROUP * GROUP + 2 * lane;
    const bool in0 = i >= b && i < e, in1 = i + 1 >= b && i + 1 < e;
    uint64_t f = 0;
    if (in0 || in1) f = ld_relaxed_u64(reinterpret_cast<const uint64_t*>(flags + i));
    const uint32_t f0 = in0 ? static_cast<uint32_t>(f) : 0u;
    const uint32_t f1 = in1 ? static_cast<uint32_t>(f >> 32) : 0u;
    *sum = f0 + f1;
    return (!in0 || f0) && (!in1 || f1);
  }

  // The scanner warp: until the prefix of the last group is known or `warps` warps
  // have left (their own waits are bounded).
  __device__ void follow(int warps) const
  {
    const int lane = threadIdx.x & 31;
    const long long last = (chunks + GROUP - 1) / GROUP - 1;
    long long f = 0;
    uint64_t before = 0;
    while (f < last && __any_sync(0xffffffffu, lane == 0 && ring->gone < warps)) {
      const long long h = f + lane;
      const uint64_t v = h < last ? ld_relaxed_u64(sums + h) : 0ull;
      const unsigned no = __ballot_sync(0xffffffffu, (v >> 32) != GROUP);
      const int n = no ? __ffs(no) - 1 : 32;
      if (n == 0) continue;
      uint32_t incl = static_cast<uint32_t>(v);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      if (lane < n) ring->base[(h + 1) % RING] = before + incl;
      before += __shfl_sync(0xffffffffu, incl, n - 1);
      f += n;
      __threadfence_block();
      __syncwarp();
      if (lane == 0) ring->known = f;
    }
  }

  // One warp: the prefix before chunk `idx`, modulo 8 or 16, if every chunk after the
  // last group known so far is compressed (size 2 modulo that); a hint only, but the
  // same in every lane.
  __device__ int guess(long long idx) const
  {
    const long long own = idx / GROUP;
    long long g = ring->known;
    g = g < own ? g : own;
    const long long v = (g > 0 ? static_cast<long long>(ring->base[g % RING]) : 0ll) + 2 * (idx - g * GROUP);
    return __shfl_sync(0xffffffffu, static_cast<int>(v), 0);
  }

  // One warp: the sum of the sizes of all chunks before `idx`, or -1 when a wait
  // exceeded the limit or another CTA reported an error in the counter block.
  // Where `from` lies in the own group, only of chunks [from, idx).
  __device__ long long prefix(long long idx, long long from, const uint64_t* hdr,
                              unsigned long long limit_ns = SPIN_TIMEOUT_NS) const
  {
    const int lane = threadIdx.x & 31;
    const long long own = idx / GROUP;
    long long b = own * GROUP;
    bool need_base = own > 0;
    if (from >= b) {
      b = from;
      need_base = false;
    }
    bool need_own = idx > b;
    long long excl = 0;
    unsigned long long t0 = 0;
    int polls = 0;
    while (true) {
      if (need_own) {
        uint32_t s;
        const bool ok = part(b, idx, lane, &s);
        if (__all_sync(0xffffffffu, ok)) {
          excl += __reduce_add_sync(0xffffffffu, s);
          need_own = false;
        }
      }
      if (need_base && __any_sync(0xffffffffu, lane == 0 && ring->known >= own)) {
        __threadfence_block();
        uint64_t v = ring->base[own % RING];
        __threadfence_block();
        if (__any_sync(0xffffffffu, lane == 0 && ring_holds(ring->known, own))) {
          v = __shfl_sync(0xffffffffu, v, 0);
        } else {  // the entry may be gone: add up the groups
          uint64_t s = 0;
          for (long long h = lane; h < own; h += 32) s += ld_relaxed_u64(sums + h) & 0xffffffffull;
          v = static_cast<uint64_t>(warp_sum(static_cast<long long>(s)));
        }
        excl += static_cast<long long>(v);
        need_base = false;
      }
      if (!need_own && !need_base) return excl;
      // a predecessor has not published yet: back off, bounded in time
      if (++polls == 256) {
        t0 = globaltimer_ns();
      } else if (polls > 256 && (polls & 255) == 0) {
        const bool late = globaltimer_ns() - t0 > limit_ns;
        const bool failed = ld_relaxed_u64(&hdr[WS_STATUS]) != 0ull;
        if (__any_sync(0xffffffffu, late || failed)) return -1;
      }
      __nanosleep(64);
    }
  }

  // One warp: the same from the flags alone, for a few groups, with no scanner.
  __device__ long long prefix_flags(long long idx, const uint64_t* hdr,
                                    unsigned long long limit_ns = SPIN_TIMEOUT_NS) const
  {
    const int lane = threadIdx.x & 31;
    long long excl = 0;
    unsigned long long t0 = 0;
    int polls = 0;
    for (long long b = 0; b < idx; b += GROUP) {
      while (true) {
        uint32_t s;
        const bool ok = part(b, idx < b + GROUP ? idx : b + GROUP, lane, &s);
        if (__all_sync(0xffffffffu, ok)) {
          excl += __reduce_add_sync(0xffffffffu, s);
          break;
        }
        if (++polls == 256) {
          t0 = globaltimer_ns();
        } else if (polls > 256 && (polls & 255) == 0) {
          const bool late = globaltimer_ns() - t0 > limit_ns;
          const bool failed = ld_relaxed_u64(&hdr[WS_STATUS]) != 0ull;
          if (__any_sync(0xffffffffu, late || failed)) return -1;
        }
        __nanosleep(32);
      }
    }
    return excl;
  }

  // One warp: the value another warp puts at `p` (never 0), or 0 when the wait gave up.
  __device__ static uint64_t await(const uint64_t* p, const uint64_t* hdr, unsigned long long limit_ns = SPIN_TIMEOUT_NS)
  {
    unsigned long long t0 = 0;
    for (int polls = 0;; ++polls) {
      const uint64_t v = ld_relaxed_u64(p);
      if (__all_sync(0xffffffffu, v != 0ull)) return __shfl_sync(0xffffffffu, v, 0);
      if (polls == 256) {
        t0 = globaltimer_ns();
      } else if (polls > 256 && (polls & 255) == 0) {
        const bool late = globaltimer_ns() - t0 > limit_ns;
        const bool failed = ld_relaxed_u64(&hdr[WS_STATUS]) != 0ull;
        if (__any_sync(0xffffffffu, late || failed)) return 0ull;
      }
      __nanosleep(64);
    }
  }
};

// ----------------------------------------------------------------------------
// Shifted store: writes `len` bytes from 16-byte aligned shared memory `src`
// to the arbitrary global byte address `dst`.  Whole aligned 16-byte granules
// get one vector store each, funnel-shifted from two aligned shared loads; the
// at most two granules shared with neighbouring chunks are written byte by
// byte.  Called by NT threads with tid = 0 .. NT-1: the warp of a raw chunk
// (NT = 32), the team of a small input's chunk (NT = 256).
// ----------------------------------------------------------------------------
template <int WQ>
__device__ __forceinline__ uint4 shifted_granule(const uint4 x, const uint4 y, int bb8)
{
  // output granule from source granules x = j - 1 and y = j
  const uint32_t w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
  uint4 o;
  o.x = __funnelshift_r(w[WQ + 0], w[WQ + 1], bb8);
  o.y = __funnelshift_r(w[WQ + 1], w[WQ + 2], bb8);
  o.z = __funnelshift_r(w[WQ + 2], w[WQ + 3], bb8);
  o.w = __funnelshift_r(w[WQ + 3], w[WQ + 4], bb8);
  return o;
}

// Granules jf .. jl-1, consecutive lanes on consecutive granules (so a warp's
// loads hit every bank once and its stores fill whole sectors), two granules in
// flight per thread.
template <int WQ, int NT>
__device__ __forceinline__ void shifted_run(uint4* out, const uint4* s4, int jf, int jl, int bb8, int t)
{
  for (int j = jf + t; j < jl; j += 2 * NT) {
    const bool two = j + NT < jl;
    const uint4 x0 = s4[j - 1], y0 = s4[j];
    uint4 x1 = x0, y1 = y0;
    if (two) {
      x1 = s4[j + NT - 1];
      y1 = s4[j + NT];
    }
    out[j] = shifted_granule<WQ>(x0, y0, bb8);
    if (two) out[j + NT] = shifted_granule<WQ>(x1, y1, bb8);
  }
}

template <int NT>
__device__ __forceinline__ void store_shifted(uint8_t* dst, const uint8_t* src, int len, int tid)
{
  const uintptr_t d = reinterpret_cast<uintptr_t>(dst);
  const int sft = static_cast<int>(d & 15u);
  uint8_t* const a0 = dst - sft;
  uint4* const out = reinterpret_cast<uint4*>(a0);
  const uint4* const s4 = reinterpret_cast<const uint4*>(src);
  const int nunits = (sft + len + 15) >> 4;
  const int jf = sft ? 1 : 0;              // first granule entirely inside the chunk
  const int jl = (sft + len) >> 4;         // one past the last such granule
  if (sft == 0) {
    for (int j = tid; j < jl; j += NT) out[j] = s4[j];
  } else {
    const int bo = 16 - sft;
    const int bb8 = (bo & 3) * 8;
    switch (bo >> 2) {
      case 0: shifted_run<0, NT>(out, s4, jf, jl, bb8, tid); break;
      case 1: shifted_run<1, NT>(out, s4, jf, jl, bb8, tid); break;
      case 2: shifted_run<2, NT>(out, s4, jf, jl, bb8, tid); break;
      default: shifted_run<3, NT>(out, s4, jf, jl, bb8, tid); break;
    }
  }
  // edge granules (shared with the neighbouring chunks): one byte per lane of
  // the first warp, lanes 0-15 the first granule, lanes 16-31 the last
  if (tid < 32) {
    int e = -1;
    if (tid < 16) {
      if (sft != 0) e = 0;
    } else {
      const int last = nunits - 1;
      if (last >= jl && !(last == 0 && sft != 0)) e = last;
    }
    if (e >= 0) {
      const int r = 16 * e - sft + (tid & 15);  // source byte of this lane
      if (r >= 0 && r < len) a0[16 * e + (tid & 15)] = src[r];
    }
  }
}

// ----------------------------------------------------------------------------
// host
// ----------------------------------------------------------------------------
// Sets the dynamic shared memory limit of `k` once per device.
template <typename K>
static cudaError_t ensure_smem_attr(K k, int bytes, unsigned long long* done_mask)
{
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (__atomic_load_n(done_mask, __ATOMIC_ACQUIRE) & bit) return cudaSuccess;
  e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) __atomic_fetch_or(done_mask, bit, __ATOMIC_RELEASE);
  return e;
}

// Launches `k` so that its set-up overlaps the end of the kernel before it (grid_wait).
template <typename... P, typename... A>
static cudaError_t launch_after(void (*k)(P...), int grid, int threads, int smem, cudaStream_t st, const A&... a)
{
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3(static_cast<unsigned>(grid));
  c.blockDim = dim3(static_cast<unsigned>(threads));
  c.dynamicSmemBytes = static_cast<size_t>(smem);
  c.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  c.attrs = at;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, k, a...);
}

}  // namespace sleek
