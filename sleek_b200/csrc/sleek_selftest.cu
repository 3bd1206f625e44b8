// sleek_selftest.cu -- device self-tests of the codec's building blocks.
//
// Bounded waits: without faulting or hanging the device, one CTA waits on an
// mbarrier that nothing arrives on, and one warp waits for the size of a preceding
// chunk that nothing publishes, each with a caller-given limit, using the same
// wait helpers as the encode and decode kernels (sleek_device.cuh).  Both must
// give up, report it, and return; the context stays usable.
//
// Chunk scan: the encoder's placing of chunks (ChunkScan) on given sizes, for chunks whose
// group is in the scanner's ring and for those whose entry the ring has lost, and its
// alignment hint read by lanes that arrive one after the other while the ring moves.
//
// Value maps: the transforms, quantizers and dequantizers the kernels compute
// (sleek_device.cuh, rewritten forms) against a literal restatement of the
// reference's integer steps, over every 32-bit word and over every 64-bit
// sign/exponent field with seeded mantissas; mismatches are counted, never
// trapped.
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/sleek_capi.h"
#include "sleek_device.cuh"

namespace sleek {
namespace {

// result[0]: 1 if the mbarrier wait gave up; result[1]: the prefix's return
// value (-1 when it gave up); result[2]: nanoseconds the two waits took
__global__ void __launch_bounds__(32) k_selftest_waits(unsigned long long limit_ns, uint64_t* flags, long long* result)
{
  __shared__ __align__(8) uint64_t bar;
  __shared__ ScanRing ring;
  const int lane = threadIdx.x;
  if (lane == 0) {
    mbar_init(&bar, 1);  // expects one arrival, which never comes
    mbar_fence_init();
  }
  __syncwarp();
  const unsigned long long t0 = globaltimer_ns();
  const bool got = mbar_wait_bounded(&bar, 0, limit_ns);
  // the size of chunk 0 is never published; flags[2..] hold the workspace header
  // that the wait reads for errors (status word 0: none)
  const long long lb = ChunkScan(flags + 2 + WS_HDR_WORDS, 2, &ring).prefix(1, 0, flags + 2, limit_ns);
  const unsigned long long t1 = globaltimer_ns();
  if (lane == 0) {
    result[0] = got ? 0 : 1;
    result[1] = lb;
    result[2] = static_cast<long long>(t1 - t0);
  }
}

// One warp waits for a copy that never lands.  result[0]: 1 if it is told that it has;
// result[2]: nanoseconds
__global__ void __launch_bounds__(32) k_selftest_copy(unsigned long long limit_ns, long long* result)
{
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
  }
  __syncwarp();
  const unsigned long long t0 = globaltimer_ns();
  const bool landed = copy_landed(&bar, 0, limit_ns);
  const unsigned long long t1 = globaltimer_ns();
  if (threadIdx.x == 0) {
    result[0] = landed;
    result[1] = 0;
    result[2] = static_cast<long long>(t1 - t0);
  }
}

// One warp waits for what no other will say, as the encoder's warps do.  `what` 3: the
// prefix of a chunk whose group the scanner never reaches; 4: the flag of a preceding
// chunk (small inputs); 5: the start of a buffer in a batch.  result[0]: what the wait
// returns, result[2]: nanoseconds.  `ws`: a zeroed workspace for 129 chunks.
__global__ void __launch_bounds__(32) k_selftest_place_waits(int what, unsigned long long limit_ns, uint64_t* ws,
                                                             long long* result)
{
  __shared__ ScanRing ring;
  if (threadIdx.x == 0) {
    ring.known = 0;
    ring.gone = 0;
  }
  __syncwarp();
  const ChunkScan scan(ws + WS_HDR_WORDS, 129, &ring);
  const unsigned long long t0 = globaltimer_ns();
  long long r = 0;
  if (what == 3) r = scan.prefix(GROUP, 0, ws, limit_ns);
  else if (what == 4) r = scan.prefix_flags(1, ws, limit_ns);
  else r = static_cast<long long>(ChunkScan::await(ws + WS_HDR_WORDS, ws, limit_ns));
  const unsigned long long t1 = globaltimer_ns();
  if (threadIdx.x == 0) {
    result[0] = r;
    result[1] = 0;
    result[2] = static_cast<long long>(t1 - t0);
  }
}

// Two warps as a decode team: the wait of warp `what` (0 or 1) gives up, the other's
// ends well.  result[0]: the status that the team leaves in `hdr`; result[1]: the
// position; result[2]: nanoseconds
__global__ void __launch_bounds__(64) k_selftest_team(int what, unsigned long long limit_ns, uint64_t* hdr,
                                                      long long* result)
{
  __shared__ __align__(8) uint64_t bars[2];
  const int lane = threadIdx.x & 31, cw = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_fence_init();
    mbar_arrive(&bars[1 - what]);
  }
  __syncthreads();
  const unsigned long long t0 = globaltimer_ns();
  const bool late = __any_sync(0xffffffffu, !mbar_wait_bounded(&bars[cw], 0, limit_ns));
  report_chunk(hdr, late, true, cw, lane, 7);
  __syncthreads();
  if (threadIdx.x == 0) {
    result[0] = static_cast<long long>(ld_relaxed_u64(&hdr[WS_STATUS]));
    result[1] = static_cast<long long>(ld_relaxed_u64(&hdr[WS_ERRPOS]));
    result[2] = static_cast<long long>(globaltimer_ns() - t0);
  }
}

__global__ void __launch_bounds__(256) k_selftest_publish(uint64_t* region, long long chunks, const uint32_t* sizes)
{
  const ChunkScan scan(region, chunks, nullptr);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < chunks; i += gridDim.x * 256ll) scan.publish(i, sizes[i]);
}

// One warp: the scanner's walk over all groups, then the places of chunks `index`.
__global__ void __launch_bounds__(32) k_selftest_places(uint64_t* region, long long chunks, const uint64_t* hdr,
                                                        const long long* index, int n, long long* prefix)
{
  __shared__ ScanRing ring;
  if (threadIdx.x == 0) {
    ring.known = 0;
    ring.gone = 0;
  }
  __syncwarp();
  const ChunkScan scan(region, chunks, &ring);
  scan.follow(1);
  __syncwarp();
  for (int i = 0; i < n; ++i) {
    const long long p = scan.prefix(index[i], 0, hdr);
    if (threadIdx.x == 0) prefix[i] = p;
  }
}

// Warp 1 moves the ring on while the lanes of warp 0, each some 1,000 clocks after the
// one before it, ask for the same chunk's hint: `uneven` counts the answers that are not
// lane 0's.
__global__ void __launch_bounds__(64) k_selftest_hint(int rounds, unsigned* uneven)
{
  __shared__ ScanRing ring;
  __shared__ volatile int done;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    ring.known = 0;
    ring.gone = 0;
    done = 0;
  }
  __syncthreads();
  const long long chunks = 1ll << 40;  // (only the ring is used)
  const ChunkScan scan(nullptr, chunks, &ring);
  if (threadIdx.x >= 32) {
    if (lane == 0) {
      volatile ScanRing* const r = &ring;
      for (long long g = 1; g < 100000 && !done; ++g) {
        r->base[g % RING] = static_cast<uint64_t>(3 * g);
        __threadfence_block();
        r->known = g;
        __nanosleep(100);
      }
    }
  } else {
    unsigned bad = 0;
    for (int i = 0; i < rounds; ++i) {
      const long long t0 = clock64();
      while (clock64() - t0 < 1000ll * lane) {
      }
      const int v = scan.guess(chunks - 1);
      bad += v != __shfl_sync(0xffffffffu, v, 0);
    }
    atomicAdd(uneven, bad);
    __syncwarp();
    if (lane == 0) done = 1;
  }
}

// ----------------------------------------------------------------------------
// Value maps against the reference's integer formulation.  The codec kernels
// compute the forward transform's exponent step as one conditional add, the
// 64-bit maps on 32-bit halves, and quantize / dequantize with the rounding
// division in floating point (sleek_device.cuh).  These are the reference's own
// steps, restated literally in 32- and 64-bit integer arithmetic
// (include/sleek_common_gpu.h: forward :356-374, inverse :614-632, quantize
// :776-802, dequantize :1077-1108), to compare against on the device.
// ----------------------------------------------------------------------------
template <typename U>
__device__ __forceinline__ U lit_fwd(U v)
{
  constexpr int TB = 8 * sizeof(U);
  constexpr U top = sizeof(U) == 4 ? static_cast<U>(0xff000000u) : static_cast<U>(0xffe0000000000000ull);
  constexpr U unit = sizeof(U) == 4 ? static_cast<U>(0x01000000u) : static_cast<U>(0x0020000000000000ull);
  constexpr U sgn = static_cast<U>(1) << (TB - 1);
  v = (v << 1) | (v >> (TB - 1));  // sign to the lowest bit
  if (v & top) {
    v -= sgn;
    if ((v & top) == 0 || v >= sgn) v -= unit;
  }
  return (v << 1) ^ ((v & sgn) ? ~static_cast<U>(0) : static_cast<U>(0));
}

template <typename U>
__device__ __forceinline__ U lit_quant(U val, int eb_e, int thr_e, U offs)
{
  constexpr int TB = 8 * sizeof(U);
  constexpr int M = sizeof(U) == 4 ? 23 : 52;  // mantissa bits
  const U a = val & ~(static_cast<U>(1) << (TB - 1));
  const int e = static_cast<int>(a >> M);
  U enc = 0;
  if (e >= thr_e) {
    enc = a - offs;
  } else if (e >= eb_e) {
    const int sh = thr_e - e;
    U mant = (val & ((static_cast<U>(1) << M) - 1)) | (static_cast<U>(1) << M);
    mant += static_cast<U>(1) << (sh - 1);
    enc = mant >> sh;
  }
  enc = (enc << 1) | ((~val) >> (TB - 1));
  return enc ? enc - 1 : 0;
}

template <typename U>
__device__ __forceinline__ U lit_dequant(U enc, int thr_e, U offs)
{
  constexpr int TB = 8 * sizeof(U);
  constexpr int M = sizeof(U) == 4 ? 23 : 52;
  if (enc == 0) return 0;
  const U a = (enc + 1) >> 1;
  U dec = 0;
  if (a >= (static_cast<U>(1) << M)) {
    dec = a + offs;
  } else if (a > 0) {
    const int lz = sizeof(U) == 4 ? __clz(static_cast<uint32_t>(a)) : __clzll(static_cast<unsigned long long>(a));
    const int sh = lz - (TB - 1 - M);
    dec = (a << sh) & ((static_cast<U>(1) << M) - 1);
    dec |= static_cast<U>(thr_e - sh) << M;
  }
  return dec | (enc << (TB - 1));
}

__device__ __forceinline__ uint64_t mix64(uint64_t x)  // splitmix64 finaliser
{
  x += 0x9e3779b97f4a7c15ull;
  x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
  x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
  return x ^ (x >> 31);
}

// error-bound exponents checked: the smallest, small, mid, large and the largest legal
__constant__ int c_eb32[8] = {0, 1, 2, 24, 100, 127, 200, 230};
__constant__ int c_eb64[9] = {0, 1, 2, 53, 500, 1000, 1023, 1500, 1993};

__device__ __forceinline__ QParams q32(int k)
{
  QParams q;
  q.eb_e = c_eb32[k];
  q.thr_e = q.eb_e + 24;
  q.offs = (static_cast<uint64_t>(q.thr_e) << 23) - (1u << 23);
  return q;
}

__device__ __forceinline__ QParams q64(int k)
{
  QParams q;
  q.eb_e = c_eb64[k];
  q.thr_e = q.eb_e + 53;
  q.offs = (static_cast<uint64_t>(q.thr_e) << 52) - (1ull << 52);
  return q;
}

// a 64-bit word with sign and exponent field `top` (12 bits) and a seeded
// mantissa; the first samples of each field are the mantissa's edge values
__device__ __forceinline__ uint64_t word64(uint64_t top, uint64_t j)
{
  constexpr uint64_t MM = (1ull << 52) - 1;
  uint64_t m;
  switch (j) {
    case 0: m = 0; break;
    case 1: m = 1; break;
    case 2: m = MM; break;
    case 3: m = 1ull << 51; break;
    case 4: m = (1ull << 51) - 1; break;
    default: m = mix64(top * 0x100000000ull + j) & MM;
  }
  return (top << 52) | m;
}

// One check over index space [0, n): counts[check] += mismatches, first[check]
// = the smallest failing index.
template <int CHECK>
__global__ void __launch_bounds__(256) k_selftest_maps(unsigned long long n, unsigned long long* counts,
                                                       unsigned long long* first)
{
  unsigned long long bad = 0, fi = ~0ull;
  const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * blockDim.x;
  for (unsigned long long i = blockIdx.x * static_cast<unsigned long long>(blockDim.x) + threadIdx.x; i < n;
       i += stride) {
    bool ok = true;
    if constexpr (CHECK == 0) {  // f32 forward transform and its inverse, every word
      const uint32_t v = static_cast<uint32_t>(i);
      const uint32_t t = fwd(v);
      ok = t == lit_fwd<uint32_t>(v) && inv(t) == v;
    } else if constexpr (CHECK == 1) {  // f32 quantize, every word x 8 bounds
      const uint32_t v = static_cast<uint32_t>(i);
      const QParams q = q32(static_cast<int>(i >> 32));
      const uint32_t want = lit_quant<uint32_t>(v, q.eb_e, q.thr_e, static_cast<uint32_t>(q.offs));
      ok = quant_fp(v, q) == want &&
           (!quant_ordinary(v, quant_limit32(q)) || quant_plain(v, quant_scale32(q)) == want);
    } else if constexpr (CHECK == 2) {  // f32 dequantize, every code x 8 bounds
      const uint32_t e = static_cast<uint32_t>(i);
      const QParams q = q32(static_cast<int>(i >> 32));
      const uint32_t want = lit_dequant<uint32_t>(e, q.thr_e, static_cast<uint32_t>(q.offs));
      ok = dequant_fp(e, q) == want && (e >= (1u << 23) || dequant_plain32(e, q) == want);
    } else if constexpr (CHECK == 3) {  // f64 forward transform and inverse, every sign/exponent x 2^20
      const uint64_t v = word64(i >> 20, i & 0xfffff);
      const uint64_t t = fwd(v);
      ok = t == lit_fwd<uint64_t>(v) && inv(t) == v;
    } else if constexpr (CHECK == 4) {  // f64 quantize, every sign/exponent x 2^20, x 9 bounds
      const uint64_t v = word64((i >> 20) & 0xfff, i & 0xfffff);
      const QParams q = q64(static_cast<int>(i >> 32));
      const uint64_t want = lit_quant<uint64_t>(v, q.eb_e, q.thr_e, q.offs);
      const uint32_t h = static_cast<uint32_t>(v >> 32);
      ok = quant_fp(v, q) == want && quant(v, q) == want &&
           (!quant_ordinary(h, quant_limit64(q)) || quant_plain(static_cast<uint32_t>(v), h, quant_scale64(q)) == want);
    } else {  // f64 dequantize x 9 bounds: every code below 2^32 (also the plain
              // form), then codes of every bit length
      const QParams q = q64(static_cast<int>((i >> 32) % 9));
      if ((i >> 32) < 9) {
        const uint32_t e = static_cast<uint32_t>(i);
        const uint64_t want = lit_dequant<uint64_t>(e, q.thr_e, q.offs);
        ok = dequant_fp(static_cast<uint64_t>(e), q) == want && dequant_plain64(e, q) == want &&
             dequant(static_cast<uint64_t>(e), q) == want;
      } else {
        const int len = static_cast<int>((i >> 26) & 63) + 1;
        const uint64_t e = (mix64(i) & (len == 64 ? ~0ull : ((1ull << len) - 1))) | (1ull << (len - 1));
        const uint64_t want = lit_dequant<uint64_t>(e, q.thr_e, q.offs);
        ok = dequant_fp(e, q) == want && dequant(e, q) == want;
      }
    }
    if (!ok) {
      ++bad;
      if (i < fi) fi = i;
    }
  }
  if (bad) {
    atomicAdd(&counts[CHECK], bad);
    atomicMin(&first[CHECK], fi);
  }
}

}  // namespace
}  // namespace sleek

extern "C" int sleek_selftest_value_maps(long long* h_counts, long long* h_first)
{
  if (!h_counts) return SLEEK_ERR_INVALID_ARG;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return SLEEK_ERR_NO_DEVICE;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  constexpr int K = SLEEK_SELFTEST_VALUE_CHECKS;
  unsigned long long* d = nullptr;
  int rc = SLEEK_OK;
  if (cudaMalloc(&d, 2 * K * sizeof(unsigned long long)) != cudaSuccess ||
      cudaMemset(d, 0, K * sizeof(unsigned long long)) != cudaSuccess ||
      cudaMemset(d + K, 0xff, K * sizeof(unsigned long long)) != cudaSuccess) {
    rc = SLEEK_ERR_CUDA;
  } else {
    const unsigned grid = static_cast<unsigned>((sms > 0 ? sms : 148) * 8);
    const unsigned long long w32 = 1ull << 32;
    sleek::k_selftest_maps<0><<<grid, 256>>>(w32, d, d + K);
    sleek::k_selftest_maps<1><<<grid, 256>>>(8 * w32, d, d + K);
    sleek::k_selftest_maps<2><<<grid, 256>>>(8 * w32, d, d + K);
    sleek::k_selftest_maps<3><<<grid, 256>>>(w32, d, d + K);
    sleek::k_selftest_maps<4><<<grid, 256>>>(9 * w32, d, d + K);
    sleek::k_selftest_maps<5><<<grid, 256>>>(18 * w32, d, d + K);
    unsigned long long h[2 * K];
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) {
      rc = SLEEK_ERR_CUDA;
    } else {
      for (int k = 0; k < K; ++k) {
        h_counts[k] = static_cast<long long>(h[k]);
        if (h_first) h_first[k] = static_cast<long long>(h[K + k]);
      }
    }
  }
  cudaFree(d);
  if (rc) cudaGetLastError();
  return rc;
}

extern "C" int sleek_selftest_bounded_waits(long long limit_ns, long long* h_result)
{
  if (!h_result || limit_ns <= 0 || limit_ns > 10000000000ll) return SLEEK_ERR_INVALID_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return SLEEK_ERR_NO_DEVICE;
  }
  // [0..1] spare, [2..33] a zeroed workspace header, [34] the flag nobody sets
  const size_t words = 2 + sleek::WS_HDR_WORDS + 1;
  uint64_t* d = nullptr;
  long long* d_res = nullptr;
  int rc = SLEEK_OK;
  if (cudaMalloc(&d, words * sizeof(uint64_t)) != cudaSuccess ||
      cudaMalloc(&d_res, 3 * sizeof(long long)) != cudaSuccess ||
      cudaMemset(d, 0, words * sizeof(uint64_t)) != cudaSuccess) {
    rc = SLEEK_ERR_CUDA;
  } else {
    sleek::k_selftest_waits<<<1, 32>>>(static_cast<unsigned long long>(limit_ns), d, d_res);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(h_result, d_res, 3 * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = SLEEK_ERR_CUDA;
  }
  cudaFree(d);
  cudaFree(d_res);
  if (rc) cudaGetLastError();
  return rc;
}

extern "C" int sleek_selftest_wait(int what, long long limit_ns, long long* h_result)
{
  if (!h_result || what < 0 || what > 5 || limit_ns <= 0 || limit_ns > 1000000000ll) return SLEEK_ERR_INVALID_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return SLEEK_ERR_NO_DEVICE;
  }
  const size_t words = static_cast<size_t>(sleek::WS_HDR_WORDS + sleek::scan_words(129));
  uint64_t* d = nullptr;  // a zeroed workspace
  long long* d_res = nullptr;
  int rc = SLEEK_OK;
  if (cudaMalloc(&d, words * sizeof(uint64_t)) != cudaSuccess ||
      cudaMalloc(&d_res, 3 * sizeof(long long)) != cudaSuccess ||
      cudaMemset(d, 0, words * sizeof(uint64_t)) != cudaSuccess) {
    rc = SLEEK_ERR_CUDA;
  } else {
    const unsigned long long limit = static_cast<unsigned long long>(limit_ns);
    if (what < 2) sleek::k_selftest_team<<<1, 64>>>(what, limit, d, d_res);
    else if (what == 2) sleek::k_selftest_copy<<<1, 32>>>(limit, d_res);
    else sleek::k_selftest_place_waits<<<1, 32>>>(what, limit, d, d_res);
    if (cudaGetLastError() != cudaSuccess || cudaDeviceSynchronize() != cudaSuccess ||
        cudaMemcpy(h_result, d_res, 3 * sizeof(long long), cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = SLEEK_ERR_CUDA;
  }
  cudaFree(d);
  cudaFree(d_res);
  if (rc) cudaGetLastError();
  return rc;
}

extern "C" int sleek_selftest_ring_holds(long long known, long long group) { return sleek::ring_holds(known, group); }

extern "C" int sleek_selftest_chunk_scan(const unsigned* h_sizes, long long chunks, const long long* h_index, int n,
                                         long long* h_prefix, unsigned* h_uneven)
{
  if (!h_sizes || !h_index || !h_prefix || !h_uneven || chunks < 1 || chunks > (1ll << 24) || n < 1 || n > 65536)
    return SLEEK_ERR_INVALID_ARG;
  for (long long i = 0; i < chunks; ++i)
    if (h_sizes[i] < 1 || h_sizes[i] > sleek::CS) return SLEEK_ERR_INVALID_ARG;
  for (int i = 0; i < n; ++i)
    if (h_index[i] < 0 || h_index[i] >= chunks) return SLEEK_ERR_INVALID_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return SLEEK_ERR_NO_DEVICE;
  }
  const size_t region = 8 * static_cast<size_t>(sleek::WS_HDR_WORDS + sleek::scan_words(chunks));
  uint64_t* d = nullptr;  // header, then flags and sums
  uint32_t* d_sizes = nullptr;
  long long* d_index = nullptr;  // the indexes, then the places
  unsigned* d_uneven = nullptr;
  int rc = SLEEK_OK;
  if (cudaMalloc(&d, region) != cudaSuccess || cudaMalloc(&d_sizes, 4 * static_cast<size_t>(chunks)) != cudaSuccess ||
      cudaMalloc(&d_index, 16 * static_cast<size_t>(n)) != cudaSuccess || cudaMalloc(&d_uneven, 4) != cudaSuccess ||
      cudaMemset(d, 0, region) != cudaSuccess || cudaMemset(d_uneven, 0, 4) != cudaSuccess ||
      cudaMemcpy(d_sizes, h_sizes, 4 * static_cast<size_t>(chunks), cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(d_index, h_index, 8 * static_cast<size_t>(n), cudaMemcpyHostToDevice) != cudaSuccess) {
    rc = SLEEK_ERR_CUDA;
  } else {
    uint64_t* const flags = d + sleek::WS_HDR_WORDS;
    sleek::k_selftest_publish<<<64, 256>>>(flags, chunks, d_sizes);
    bool ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
    if (ok) {  // every size is published: the scanner's walk ends
      sleek::k_selftest_places<<<1, 32>>>(flags, chunks, d, d_index, n, d_index + n);
      sleek::k_selftest_hint<<<1, 64>>>(32, d_uneven);
      ok = cudaGetLastError() == cudaSuccess && cudaDeviceSynchronize() == cudaSuccess;
    }
    if (!ok ||
        cudaMemcpy(h_prefix, d_index + n, 8 * static_cast<size_t>(n), cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(h_uneven, d_uneven, 4, cudaMemcpyDeviceToHost) != cudaSuccess)
      rc = SLEEK_ERR_CUDA;
  }
  cudaFree(d);
  cudaFree(d_sizes);
  cudaFree(d_index);
  cudaFree(d_uneven);
  if (rc) cudaGetLastError();
  return rc;
}
