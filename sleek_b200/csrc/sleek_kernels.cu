// sleek_kernels.cu -- sm_100a decode kernels (one buffer, and batches); encode is in
// sleek_encode.cu.
//
// Decode (replaces d_decode, :688-768, 1199-1279): CTAs take contiguous chunk
// ranges in ticket order, sum their ranges' compressed sizes, look back over the
// preceding ranges once, then stream their chunks through a two-stage TMA
// pipeline (each copy is the 16-byte aligned superset of the chunk's bytes); every
// warp checks each chunk itself and unpacks its own subchunks straight into
// coalesced global stores, with no CTA barrier per chunk.  Malformed streams set
// an error status instead of trapping; every wait is bounded in time.
#include "sleek_device.cuh"
#include "sleek_launch.h"

namespace sleek {

// ============================================================================
// decode
// ============================================================================
struct DecChunk {
  long long c;
  long long off;
  int cs;
  int sft;
  int ok;
  int pad_;
};

constexpr int DEC_STAGES = 2;

struct DecMisc {
  uint64_t full[DEC_STAGES];   // chunk bytes landed (TMA tx count)
  uint64_t empty[DEC_STAGES];  // every compute warp is done with the stage's chunk
  DecChunk info[DEC_STAGES];
  long long excl;
  long long vb;
  long long red[NT_MAX_WARPS];
  long long pre[NT_MAX_WARPS];
  int bad[NT_MAX_WARPS];
};

// Streams of at most this many chunks place each CTA's range by summing the size
// table before it directly (at most 64 KB read per CTA from L2, no wait on other
// CTAs) instead of the decoupled look-back, whose chain of polls dominates small
// decodes (26 MB: +32 %) and still costs 2-4 % at 18,432 chunks.
constexpr long long DEC_DIRECT_MAX = 32768;

constexpr int DEC_SMEM = DEC_STAGES * STAGE_BYTES + ((sizeof(DecMisc) + 127) / 128) * 128;

__device__ __forceinline__ uint64_t lds_u64_at_byte(const uint8_t* base, int byte_off)
{
  const uint32_t* w = reinterpret_cast<const uint32_t*>(base);
  const int wi = byte_off >> 2;
  const int sh = (byte_off & 3) * 8;
  const uint32_t lo = __funnelshift_r(w[wi], w[wi + 1], sh);
  const uint32_t hi = __funnelshift_r(w[wi + 1], w[wi + 2], sh);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Decodes one staged chunk (payload at byte `sft` of `stg`, `cs` bytes, `osize`
// bytes out) with the calling warp's share of the work and no CTA barrier: every
// warp reads the 32 bit widths, sums and checks them itself (the same result in
// every warp), then unpacks its subchunks cw, cw + NW, ... with consecutive lanes
// on consecutive values, widths and bit offsets in registers.  Returns false for
// a malformed chunk (bit width above the element width, widths not adding up to
// cs, trailer not equal to osize); a raw chunk (cs == osize) is copied.
template <typename T, bool LOSSY, int NW>
__device__ __forceinline__ bool decode_chunk_warp(const uint8_t* stg, int sft, int cs, int osize, T* o,
                                                  const QParams& q, int cw, int lane)
{
  using V = VT<T>;
  const int nv = osize / static_cast<int>(sizeof(T));
  if (cs == osize) {
    for (int e = cw * 32 + lane; e < nv; e += NW * 32) {
      if constexpr (sizeof(T) == 4) o[e] = lds_u32_at_byte(stg, sft + 4 * e);
      else o[e] = lds_u64_at_byte(stg, sft + 8 * e);
    }
    return true;
  }
  const int ln_l = stg[sft + lane];
  const int bitsw = ln_l * V::VPS;
  const int tot = __reduce_add_sync(0xffffffffu, bitsw);
  bool ok = !__any_sync(0xffffffffu, ln_l > V::TB) && (34 + tot / 8 == cs);
  if (ok) {
    const int16_t tr = static_cast<int16_t>(stg[sft + cs - 2] | (stg[sft + cs - 1] << 8));
    ok = tr == osize;
  }
  if (!ok) return false;
  const uint32_t* const w = reinterpret_cast<const uint32_t*>(stg);
  static_assert(SC % NW == 0, "whole subchunks per warp");
  // full chunks (all but a stream's last) are unpacked without the per-value
  // bound test (f32 lossy decode +11 %); 64-bit chunks whose widths are all at
  // most 32 (typical of lossy streams) extract each value from two words
  // instead of three and dequantize it in 32-bit arithmetic (f64 lossy decode
  // +23 %, then +7-13 %).  A zero width needs no test: its mask is 0, and its
  // reads, like every extraction's, end within 12 bytes of a bit inside the
  // chunk's payload (at most 15 + 16383 + 10 bytes into a stage of 16384 + 64).
  auto unpack = [&](auto full, auto narrow) {
#pragma unroll
    for (int u = 0; u < SC / NW; ++u) {  // unrolled: the subchunks' load chains overlap
      const int i = cw + u * NW;
      const int ln = __shfl_sync(0xffffffffu, ln_l, i);
      const int base = 8 * sft + 256 + __reduce_add_sync(0xffffffffu, lane < i ? bitsw : 0);  // first bit of i
      const int k0 = i * V::VPS;
#pragma unroll
      for (int j = lane; j < V::VPS; j += 32) {
        if (decltype(full)::value || k0 + j < nv) {
          if constexpr (sizeof(T) == 8 && LOSSY && decltype(narrow)::value) {
            o[k0 + j] = dequant_fp_narrow(extract_bits32(w, base + j * ln, ln), q);
          } else {
            T e;
            if constexpr (sizeof(T) == 4 || decltype(narrow)::value) e = extract_bits32(w, base + j * ln, ln);
            else e = extract_bits64(w, base + j * ln, ln);
            o[k0 + j] = decode_value<LOSSY>(e, q);
          }
        }
      }
    }
  };
  if (sizeof(T) == 8 && __all_sync(0xffffffffu, ln_l <= 32)) {
    if (osize == CS) unpack(std::true_type{}, std::true_type{});
    else unpack(std::false_type{}, std::true_type{});
  } else {
    if (osize == CS) unpack(std::true_type{}, std::false_type{});
    else unpack(std::false_type{}, std::false_type{});
  }
  return true;
}

template <typename T, bool LOSSY, int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_decode(const DecArgs a)
{
  using V = VT<T>;
  constexpr int NW = NT / 32;
  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t* const stage0 = smem;
  DecMisc& m = *reinterpret_cast<DecMisc*>(smem + DEC_STAGES * STAGE_BYTES);

  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const WsPhase ph = WsPhase::of(a.ws, a.flag_cap);  // self-resetting workspace
  uint64_t* const hdr = ph.hdr;
  uint64_t* const flags = ph.flags;

  // Speculation: when the caller states the output capacity and the stream's
  // length, the chunk count is usually ceil(capacity / CS), and this CTA's sizes
  // (the prefix before its range, and its range) are read while the header is
  // still on its way, instead of one dependent round trip after it.  Used only if
  // the header agrees; the reads stay inside the stated stream length.
  const long long g_chunks = a.out_cap > 0 ? (a.out_cap + CS - 1) / CS : -1;
  const bool spec = g_chunks > 0 && g_chunks <= DEC_DIRECT_MAX && a.in_len >= 8 + 2 * g_chunks;
  long long s_pre = 0;  // this thread's share of the sizes before the range
  int s_cs = -1;        // this thread's size in the range (ranges of at most NT chunks)
  {
    const uint16_t* const sz = reinterpret_cast<const uint16_t*>(a.in + 8);
    if (spec) {
      const long long kg = (g_chunks + gridDim.x - 1) / gridDim.x;
      const long long c0g = min(static_cast<long long>(blockIdx.x) * kg, g_chunks);
      const long long c1g = min(c0g + kg, g_chunks);
      if (kg <= NT && c0g + tid < c1g) s_cs = sz[c0g + tid];
      const unsigned long long* const s8 = reinterpret_cast<const unsigned long long*>(sz);
      const long long q = c0g >> 2;
      for (long long k = tid; k < q; k += NT) {
        const unsigned long long v = s8[k];
        const unsigned long long p2 = (v & 0x0000ffff0000ffffull) + ((v >> 16) & 0x0000ffff0000ffffull);
        s_pre += static_cast<long long>((p2 & 0xffffffffull) + (p2 >> 32));
      }
      for (long long c = (q << 2) + tid; c < c0g; c += NT) s_pre += sz[c];
    }
  }

  // header checks (every CTA reads the 8-byte header)
  const long long insize = *reinterpret_cast<const long long*>(a.in);
  const long long chunks = insize > 0 ? (insize + CS - 1) / CS : 0;
  bool hdr_ok = insize >= 0 && (insize % static_cast<long long>(sizeof(T))) == 0;
  if (a.in_len >= 0 && 8 + 2 * chunks > a.in_len) hdr_ok = false;
  const bool cap_ok = a.out_cap < 0 || insize <= a.out_cap;
  const long long payload_len = a.in_len >= 0 ? a.in_len - 8 - 2 * chunks : -1;
  const uint16_t* const size_in = reinterpret_cast<const uint16_t*>(a.in + 8);
  const uint8_t* const data_in = a.in + 8 + 2 * chunks;

  if (tid == 0) {
    for (int st = 0; st < DEC_STAGES; ++st) {
      mbar_init(&m.full[st], 1);
      mbar_init(&m.empty[st], NW);  // one arrival per warp
    }
    mbar_fence_init();
    // ranges placed by summing the size table wait on no other CTA, so the
    // block index orders them; the look-back needs ticket order (a CTA waits only
    // on CTAs that started before it)
    m.vb = hdr_ok && cap_ok && chunks <= DEC_DIRECT_MAX
               ? static_cast<long long>(blockIdx.x)
               : static_cast<long long>(atomicAdd(reinterpret_cast<unsigned long long*>(&a.ws[WS_TICKET]), 1ull));
    if (!hdr_ok) set_status(hdr, ST_CORRUPT, -1);
    else if (!cap_ok) set_status(hdr, ST_CAPACITY, -1);
  }
  __syncthreads();

  const bool go = hdr_ok && cap_ok;
  const long long vb = m.vb;
  const long long K = (chunks + gridDim.x - 1) / gridDim.x;
  const long long c0 = go ? min(vb * K, chunks) : 0;
  const long long c1 = go ? min(c0 + K, chunks) : 0;

  // ---- range aggregate + size-table validation ---------------------------------
  {
    const bool direct = go && chunks <= DEC_DIRECT_MAX;
    const bool hit = direct && spec && chunks == g_chunks;  // the speculative reads are this CTA's
    long long sum = 0, pre = 0;
    int bad = 0;
    if (hit && K <= NT) {
      if (c0 + tid < c1) {
        const int cs = s_cs;
        const long long c = c0 + tid;
        const int os = static_cast<int>(min(static_cast<long long>(CS), insize - c * CS));
        bad |= (cs > os) | (cs == 0) | ((cs < os) & (cs < 34));
        sum += cs;
      }
    } else {
      for (long long c = c0 + tid; c < c1; c += NT) {
        const int cs = size_in[c];
        const int os = static_cast<int>(min(static_cast<long long>(CS), insize - c * CS));
        bad |= (cs > os) | (cs == 0) | ((cs < os) & (cs < 34));
        sum += cs;
      }
    }
    if (hit) {
      pre = warp_sum(s_pre);
    } else if (direct) {
      // sizes [0, c0), four per 8-byte load (the table starts 8-byte aligned)
      const unsigned long long* const s8 = reinterpret_cast<const unsigned long long*>(size_in);
      const long long q = c0 >> 2;
      for (long long k = tid; k < q; k += NT) {
        const unsigned long long v = s8[k];
        const unsigned long long p2 = (v & 0x0000ffff0000ffffull) + ((v >> 16) & 0x0000ffff0000ffffull);
        pre += static_cast<long long>((p2 & 0xffffffffull) + (p2 >> 32));
      }
      for (long long c = (q << 2) + tid; c < c0; c += NT) pre += size_in[c];
      pre = warp_sum(pre);
    }
    sum = warp_sum(sum);
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) {
      m.red[warp] = sum;
      m.pre[warp] = pre;
      m.bad[warp] = bad;
    }
    __syncthreads();
    if (warp == 0) {
      long long s2 = lane < NW ? m.red[lane] : 0;
      int b2 = lane < NW ? m.bad[lane] : 0;
      s2 = warp_sum(s2);
      b2 = __any_sync(0xffffffffu, b2);
      if (b2 && lane == 0) set_status(hdr, ST_CORRUPT, c0);
      long long excl = 0;
      if (direct) {
        excl = warp_sum(lane < NW ? m.pre[lane] : 0);
      } else {
        if (lane == 0)
          st_relaxed_u64(&flags[vb], (vb == 0 ? FLAG_INC : FLAG_AGG) | (static_cast<uint64_t>(s2) & FLAG_VAL));
      }
      if (!direct && vb > 0) {
        excl = lookback(flags, vb, 0, hdr);
        if (excl < 0) {
          if (lane == 0) set_status(hdr, ST_TIMEOUT, c0);
        }
        if (lane == 0)
          st_relaxed_u64(&flags[vb], FLAG_INC | (static_cast<uint64_t>(excl >= 0 ? excl + s2 : 0) & FLAG_VAL));
      }
      if (lane == 0) m.excl = b2 ? -1 : excl;
    }
    __syncthreads();
  }

  const long long excl = m.excl;
  if (excl >= 0 && c0 < c1) {
    // producer state (warp 0): offsets and sizes of a window of 32 chunks
    long long wbase = -64, woff = 0, run = excl;
    int wcs = 0;
    auto issue = [&](long long c, int stg) {  // warp 0, warp-uniform
      if (c - wbase >= 32) {
        wbase = c;
        const long long cc = c + lane;
        const int cs = cc < c1 ? static_cast<int>(size_in[cc]) : 0;
        long long incl = cs;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const long long t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        woff = run + incl - cs;
        wcs = cs;
        run += __shfl_sync(0xffffffffu, incl, 31);
      }
      const int l = static_cast<int>(c - wbase);
      const long long off = __shfl_sync(0xffffffffu, woff, l);
      const int cs = __shfl_sync(0xffffffffu, wcs, l);
      if (lane == 0) {
        const uint8_t* src = data_in + off;
        const int sft = static_cast<int>(reinterpret_cast<uintptr_t>(src) & 15u);
        const uint32_t nb = static_cast<uint32_t>((sft + cs + 15) & ~15);
        const bool ok = cs >= 1 && cs <= CS && (payload_len < 0 || off + cs <= payload_len);
        DecChunk& d = m.info[stg];
        d.c = c;
        d.off = off;
        d.cs = cs;
        d.sft = sft;
        d.ok = ok;
        if (ok) {
          mbar_arrive_expect_tx(&m.full[stg], nb);
          tma_load_1d(stage0 + stg * STAGE_BYTES, src - sft, nb, &m.full[stg]);
        } else {
          mbar_arrive(&m.full[stg]);
        }
      }
    };

    // Warp 0 keeps DEC_STAGES - 1 chunks in flight: at chunk it it issues chunk
    // it + DEC_STAGES - 1 into the stage of chunk it - 1, once every warp has
    // released that stage.  No CTA barrier per chunk: each warp waits for its
    // stages itself and releases them with its own arrival; a wait that gives up
    // ends that warp's loop (the others end by their own bounded waits).
    long long issued = c0;   // next chunk warp 0 issues
    bool feeding = true;     // warp 0 still issues
    auto issue_next = [&]() {  // warp 0, warp-uniform
      const int jt = static_cast<int>(issued - c0);
      const int st = jt % DEC_STAGES;
      if (jt >= DEC_STAGES &&
          __any_sync(0xffffffffu, !mbar_wait_bounded(&m.empty[st], ((jt - DEC_STAGES) / DEC_STAGES) & 1))) {
        if (lane == 0) set_status(hdr, ST_TIMEOUT, issued);
        feeding = false;
        return;
      }
      issue(issued, st);
      ++issued;
    };
    if (warp == 0)
      for (int k = 0; k < DEC_STAGES - 1 && issued < c1; ++k) issue_next();
    int it = 0;
    long long c = c0;
    for (; c < c1; ++c, ++it) {
      const int s = it % DEC_STAGES;
      uint8_t* const stg = stage0 + s * STAGE_BYTES;
      if (warp == 0 && feeding && issued < c1) issue_next();

      if (__any_sync(0xffffffffu, !mbar_wait_bounded(&m.full[s], (it / DEC_STAGES) & 1))) {
        if (lane == 0) set_status(hdr, ST_TIMEOUT, c);
        break;
      }

      const DecChunk d = m.info[s];
      const int osize = static_cast<int>(min(static_cast<long long>(CS), insize - c * CS));
      uint8_t* const outc = a.out + c * CS;
      if (!d.ok) {
        if (tid == 0) set_status(hdr, ST_CORRUPT, c);
      } else if (!decode_chunk_warp<T, LOSSY, NW>(stg, d.sft, d.cs, osize, reinterpret_cast<T*>(outc), a.q,
                                                    warp, lane)) {
        if (tid == 0) set_status(hdr, ST_CORRUPT, c);
      }
      // this warp is done with the stage (generic accesses ordered before the next TMA write)
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&m.empty[s]);
    }
    // never leave with a bulk copy still landing in this CTA's shared memory:
    // warp 0 waits for the chunks it issued but did not consume
    if (warp == 0 && lane == 0) {
      for (long long k = c; k < issued; ++k) {
        const int jt = static_cast<int>(k - c0);
        mbar_wait_bounded(&m.full[jt % DEC_STAGES], (jt / DEC_STAGES) & 1);
      }
    }
  }

  // this CTA's share of the flags the previous launch left in the other region
  // (off the start of the kernel: only the next launch reads them)
  if (warp == NW - 1) ph.clear_other_share(lane);

  // ---- epilogue ------------------------------------------------------------------
  __syncthreads();
  if (tid == 0) {
    __threadfence();
    const unsigned long long dn = atomicAdd(reinterpret_cast<unsigned long long*>(&a.ws[WS_DONE]), 1ull);
    if (dn == gridDim.x - 1) {
      __threadfence();
      const unsigned long long st = ld_relaxed_u64(&hdr[WS_STATUS]);
      *a.outsize = st ? -static_cast<long long>(st) : insize;
      ph.finish(a.ws, gridDim.x);
    }
  }
}

// ============================================================================
// batched decode: a prepass places every chunk, then a persistent kernel with a
// producer warp and 8 compute warps decodes chunks in any order
// ============================================================================
constexpr long long NO_CHUNK = 0x7fffffffffffffffll;
constexpr int DB_STAGES = 4;
constexpr int DB_CW = 8;
constexpr int DB_NT = (DB_CW + 1) * 32;
constexpr int DB_MINB = 3;

struct DecBMeta {
  long long g;      // chunk id across the launch, or NO_CHUNK
  uint8_t* out;     // where the chunk's values go
  QParams q;
  int kind;         // bit 0: 64-bit values, bit 1: lossy
  int osize;
  int cs;
  int sft;          // byte offset of the chunk within the staged copy
  int state;        // 0: nothing to decode, 1: decode
  int pad_;
};

struct DecBMisc {
  uint64_t full[DB_STAGES];
  uint64_t empty[DB_STAGES];
  DecBMeta meta[DB_STAGES];
};

constexpr int DB_SMEM = DB_STAGES * STAGE_BYTES + ((sizeof(DecBMisc) + 127) / 128) * 128 + 8 * (BATCH_MAX_JOBS + 1);

// Prepass, one CTA per buffer: validates the header and size table and writes the
// byte offset of every chunk's payload (an exclusive scan of the sizes).
__global__ void __launch_bounds__(256) k_decode_prepass(const BatchDecArgs a)
{
  __shared__ long long wsum[8];
  __shared__ int wbad[8];
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
  long long* const offs = a.offsets + a.chunk_base[j];
  long long carry = 0;
  int bad = 0;
  for (long long b = 0; b < chunks; b += 256) {
    const long long c = b + tid;
    int cs = 0;
    if (c < chunks) {
      cs = size_in[c];
      const int os = static_cast<int>(min(static_cast<long long>(CS), insize - c * CS));
      bad |= (cs > os) | (cs == 0) | ((cs < os) & (cs < 34));
    }
    long long incl = cs;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    long long before = carry;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    if (c < chunks) offs[c] = before + incl - cs;
    long long tile = 0;
    for (int w = 0; w < 8; ++w) tile += wsum[w];
    carry += tile;
    __syncthreads();
  }
  bad = __any_sync(0xffffffffu, bad);
  if (lane == 0) wbad[warp] = bad;
  __syncthreads();
  if (tid == 0) {
    int any = 0;
    for (int w = 0; w < 8; ++w) any |= wbad[w];
    if (any || (len >= 0 && 8 + 2 * chunks + carry > len)) {
      set_status(a.ws, ST_CORRUPT, j);
    } else {
      a.actual[j] = chunks;
      a.actual_insize[j] = insize;
      *job.outsize = insize;
    }
  }
}

__global__ void __launch_bounds__(DB_NT, DB_MINB) k_decode_batch(const BatchDecArgs a)
{
  extern __shared__ __align__(128) uint8_t smem[];
  uint8_t* const stage0 = smem;
  DecBMisc& m = *reinterpret_cast<DecBMisc*>(smem + DB_STAGES * STAGE_BYTES);
  long long* const cb = reinterpret_cast<long long*>(smem + DB_STAGES * STAGE_BYTES +
                                                     ((sizeof(DecBMisc) + 127) / 128) * 128);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint64_t* const ws = a.ws;
  for (int i = tid; i <= a.njobs; i += DB_NT) cb[i] = a.chunk_base[i];
  if (tid == 0) {
    for (int s = 0; s < DB_STAGES; ++s) {
      mbar_init(&m.full[s], 1);
      mbar_init(&m.empty[s], DB_CW);  // one arrival per compute warp
    }
    mbar_fence_init();
  }
  __syncthreads();
  const long long total = cb[a.njobs];
  const bool failed_before = ld_relaxed_u64(&ws[WS_STATUS]) != 0ull;  // the prepass found an error

  if (warp == DB_CW) {
    // ===================== producer warp (lane 0 works, the warp follows) =====================
    unsigned long long* const tick = reinterpret_cast<unsigned long long*>(&ws[WS_TICKET]);
    unsigned issued = 0, issued_par = 0;
    for (int seq = 0;; ++seq) {
      const int s = seq % DB_STAGES;
      if (seq >= DB_STAGES) {
        const bool ok = mbar_wait_bounded(&m.empty[s], ((seq - DB_STAGES) / DB_STAGES) & 1);
        if (__any_sync(0xffffffffu, !ok)) {
          if (lane == 0) set_status(ws, ST_TIMEOUT, -1);
          break;
        }
      }
      long long t = NO_CHUNK;
      if (lane == 0 && !failed_before) t = static_cast<long long>(atomicAdd(tick, 1ull));
      t = __shfl_sync(0xffffffffu, t, 0);
      if (lane == 0) {
        DecBMeta& d = m.meta[s];
        bool copy = false;
        if (t < total) {
          int lo = 0, hi = a.njobs - 1;
          while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (cb[mid] <= t) lo = mid;
            else hi = mid - 1;
          }
          const BatchJob& job = a.jobs[lo];
          const long long c = t - cb[lo];
          const long long chunks = a.actual[lo];
          d.g = t;
          d.state = 0;
          if (c < chunks) {
            const long long insize = a.actual_insize[lo];
            const uint8_t* const data_in = job.in + 8 + 2 * chunks;
            const long long off = a.offsets[t];
            const int cs = reinterpret_cast<const uint16_t*>(job.in + 8)[c];
            const uint8_t* const src = data_in + off;
            const int sft = static_cast<int>(reinterpret_cast<uintptr_t>(src) & 15u);
            d.out = job.out + c * CS;
            d.q = job.q;
            d.kind = job.kind;
            d.osize = static_cast<int>(min(static_cast<long long>(CS), insize - c * CS));
            d.cs = cs;
            d.sft = sft;
            d.state = 1;
            const uint32_t nb = static_cast<uint32_t>((sft + cs + 15) & ~15);
            mbar_arrive_expect_tx(&m.full[s], nb);
            tma_load_1d(stage0 + s * STAGE_BYTES, src - sft, nb, &m.full[s]);
            copy = true;
          }
        } else {
          d.g = NO_CHUNK;
        }
        if (copy) {
          issued |= 1u << s;
          issued_par = (issued_par & ~(1u << s)) | (((seq / DB_STAGES) & 1u) << s);
        } else {
          issued &= ~(1u << s);
          mbar_arrive(&m.full[s]);
        }
      }
      __syncwarp();
      if (t >= total) break;
    }
    if (lane == 0) {
      for (int s = 0; s < DB_STAGES; ++s)
        if (issued & (1u << s)) mbar_wait_bounded(&m.full[s], (issued_par >> s) & 1u);
    }
  } else {
    // ===================== compute warps =====================
    // No CTA barrier: each warp waits for a stage itself, decodes its share of the
    // chunk and frees the stage with its own arrival.  A wait that gives up ends
    // this warp's loop; the others and the producer end by their own bounded waits.
    for (int seq = 0;; ++seq) {
      const int s = seq % DB_STAGES;
      if (__any_sync(0xffffffffu, !mbar_wait_bounded(&m.full[s], (seq / DB_STAGES) & 1))) {
        if (lane == 0) set_status(ws, ST_TIMEOUT, -1);
        break;
      }
      const DecBMeta& d = m.meta[s];
      if (d.g == NO_CHUNK) break;
      if (d.state == 1) {
        const uint8_t* const stg = stage0 + s * STAGE_BYTES;
        bool ok;
        switch (d.kind) {
          case 0: ok = decode_chunk_warp<uint32_t, false, DB_CW>(stg, d.sft, d.cs, d.osize,
                                                                 reinterpret_cast<uint32_t*>(d.out), d.q, warp, lane); break;
          case 1: ok = decode_chunk_warp<uint64_t, false, DB_CW>(stg, d.sft, d.cs, d.osize,
                                                                 reinterpret_cast<uint64_t*>(d.out), d.q, warp, lane); break;
          case 2: ok = decode_chunk_warp<uint32_t, true, DB_CW>(stg, d.sft, d.cs, d.osize,
                                                                reinterpret_cast<uint32_t*>(d.out), d.q, warp, lane); break;
          default: ok = decode_chunk_warp<uint64_t, true, DB_CW>(stg, d.sft, d.cs, d.osize,
                                                                 reinterpret_cast<uint64_t*>(d.out), d.q, warp, lane); break;
        }
        if (!ok && warp == 0 && lane == 0) set_status(ws, ST_CORRUPT, d.g);
      }
      // this warp is done with the stage (generic accesses ordered before the next TMA write)
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&m.empty[s]);
    }
  }

  // ---- epilogue: an error anywhere turns every size into -status ---------------
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

// ============================================================================
// launchers
// ============================================================================
// Decode launch shapes: threads per CTA and the CTAs per SM the registers are
// budgeted for (index = the C ABI's shape number).
template <int NT_, int MINB_>
struct DecShape {
  static constexpr int NT = NT_;
  static constexpr int MINB = MINB_;
};
using DecShape0 = DecShape<256, 4>;  // default
using DecShape1 = DecShape<128, 6>;
using DecShape2 = DecShape<512, 2>;
constexpr int DEC_SHAPES = 3;

template <typename T, bool LOSSY, class S>
static cudaError_t launch_dec_k(const DecArgs& a, int grid, cudaStream_t st)
{
  auto k = k_decode<T, LOSSY, S::NT, S::MINB>;
  static unsigned long long attr = 0;
  cudaError_t e = ensure_smem_attr(k, DEC_SMEM, &attr);
  if (e != cudaSuccess) return e;
  k<<<grid, S::NT, DEC_SMEM, st>>>(a);
  return cudaGetLastError();
}

template <typename T, bool LOSSY, class S>
static int dec_occupancy()
{
  auto k = k_decode<T, LOSSY, S::NT, S::MINB>;
  cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, DEC_SMEM);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, S::NT, DEC_SMEM);
  return n;
}

template <typename T, bool LOSSY>
static cudaError_t launch_dec_kind(int shape, const DecArgs& a, int grid, cudaStream_t st)
{
  switch (shape) {
    case 1: return launch_dec_k<T, LOSSY, DecShape1>(a, grid, st);
    case 2: return launch_dec_k<T, LOSSY, DecShape2>(a, grid, st);
    default: return launch_dec_k<T, LOSSY, DecShape0>(a, grid, st);
  }
}

template <typename T, bool LOSSY>
static int dec_occupancy_kind(int shape)
{
  switch (shape) {
    case 1: return dec_occupancy<T, LOSSY, DecShape1>();
    case 2: return dec_occupancy<T, LOSSY, DecShape2>();
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
    case 1: return {DecShape1::NT, DecShape1::NT / 32, DEC_STAGES, DecShape1::MINB};
    case 2: return {DecShape2::NT, DecShape2::NT / 32, DEC_STAGES, DecShape2::MINB};
    default: return {DecShape0::NT, DecShape0::NT / 32, DEC_STAGES, DecShape0::MINB};
  }
}

int shape_count(bool enc) { return enc ? encode_shape_count() : DEC_SHAPES; }

cudaError_t launch_decode_batch(const BatchDecArgs& a, int grid, cudaStream_t st)
{
  k_decode_prepass<<<a.njobs, 256, 0, st>>>(a);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  static unsigned long long attr = 0;
  e = ensure_smem_attr(k_decode_batch, DB_SMEM, &attr);
  if (e != cudaSuccess) return e;
  k_decode_batch<<<grid, DB_NT, DB_SMEM, st>>>(a);
  return cudaGetLastError();
}

int decode_batch_blocks_per_sm()
{
  cudaFuncSetAttribute(k_decode_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, DB_SMEM);
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_decode_batch, DB_NT, DB_SMEM);
  return n;
}

}  // namespace sleek
