// Channel reductions (bandpass, collapse), zero-DM, downsample, stage-1
// subband, and the boxcar matched-filter S/N epilogue.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "spp_common.cuh"
#include "spp_dmt.cuh"

namespace spp {

static inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }
__host__ __device__ __forceinline__ int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

// Reads sample (t, c) of a raw time-major block as float (any nbits).
template <int NB>
__device__ __forceinline__ float raw_at(const void* in, int64_t nchans, int64_t t, int64_t c,
                                        int bitorder) {
  if (NB == 32) return static_cast<const float*>(in)[t * nchans + c];
  const uint8_t* b = static_cast<const uint8_t*>(in);
  const int64_t bit = (t * nchans + c) * NB;
  return (float)field_of<NB>(b[bit >> 3], (int)c, bitorder);
}

// ---------------------------------------------------------------------------
// bandpass: per-channel sequential float32 sum over samples, in sample order,
// exactly as kernels.extract_bpass's loop (bit-identical).  One thread per
// channel; 8 samples are loaded ahead of the dependent add chain.
// ---------------------------------------------------------------------------
template <int NB>
__global__ void k_bandpass(const void* __restrict__ in, int64_t nchans, int64_t nsamps,
                           int bitorder, float* __restrict__ bpass) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= nchans) return;
  float acc = bpass[c];
  int64_t t = 0;
  for (; t + 8 <= nsamps; t += 8) {
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = raw_at<NB>(in, nchans, t + k, c, bitorder);
#pragma unroll
    for (int k = 0; k < 8; ++k) acc = __fadd_rn(acc, v[k]);
  }
  for (; t < nsamps; ++t) acc = __fadd_rn(acc, raw_at<NB>(in, nchans, t, c, bitorder));
  bpass[c] = acc;
}

// collapse: tim[out_start + t] = f32(sum_c f64(x[t][c])) (kernels.extract_tim)
template <int NB>
__global__ void k_collapse(const void* __restrict__ in, int64_t nchans, int64_t nsamps,
                           int bitorder, float* __restrict__ tim, int64_t out_start) {
  const int64_t t = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= nsamps) return;
  double s = 0.0;
  for (int64_t c = lane; c < nchans; c += 32) s += (double)raw_at<NB>(in, nchans, t, c, bitorder);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) tim[out_start + t] = (float)s;
}

// zero-DM on time-major float32 (kernels.remove_zerodm, core/kernels.py:493-505):
// a block of 8 warps takes 256 samples; each warp sums 32 samples' channels in
// channel order (32 x 32 tiles staged through shared memory, one lane per
// sample), then the block rewrites the 256 spectra with coalesced accesses.
// The result is stored in the input's type: float32 rounds; uint8 keeps the low
// eight bits of the truncated value (what the reference's numba cast of a
// float64 to uint8 yields on x86, where values far above 255 are the norm
// because the bandpass is a channel sum).
__device__ __forceinline__ float zdm_store(float, double v) { return (float)v; }
__device__ __forceinline__ uint8_t zdm_store(uint8_t, double v) {
  return (uint8_t)(uint64_t)(int64_t)v;
}

constexpr int kZdmRows = 256;
template <typename T>
__global__ void __launch_bounds__(kZdmRows)
k_zero_dm(const T* __restrict__ in, T* __restrict__ out, int64_t nchans, int64_t nsamps,
          const float* __restrict__ bpass, const float* __restrict__ chanwts) {
  __shared__ float tile[kZdmRows / 32][32][33];
  __shared__ double zs[kZdmRows];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t tb = (int64_t)blockIdx.x * kZdmRows; tb < nsamps; tb += (int64_t)gridDim.x * kZdmRows) {
    const int64_t t0 = tb + warp * 32;
    double s = 0.0;
    for (int64_t c0 = 0; c0 < nchans; c0 += 32) {
      const int64_t c = c0 + lane;
      for (int r = 0; r < 32; ++r) {
        const int64_t t = t0 + r;
        tile[warp][r][lane] = (t < nsamps && c < nchans) ? (float)in[t * nchans + c] : 0.f;
      }
      __syncwarp();
      const int nc = (nchans - c0) < 32 ? (int)(nchans - c0) : 32;
      for (int j = 0; j < nc; ++j) s = __dadd_rn(s, (double)tile[warp][lane][j]);
      __syncwarp();
    }
    zs[threadIdx.x] = s;
    __syncthreads();
    const int64_t rows = imin64(kZdmRows, nsamps - tb);
    for (int64_t r = 0; r < rows; ++r) {
      const double z = zs[r];
      const T* src = in + (tb + r) * nchans;
      T* dst = out + (tb + r) * nchans;
      for (int64_t c = threadIdx.x; c < nchans; c += kZdmRows) {
        const double t1 = __dmul_rn(z, (double)chanwts[c]);
        const double t2 = __dsub_rn((double)src[c], t1);
        dst[c] = zdm_store(T(), __dadd_rn(t2, (double)bpass[c]));
      }
    }
    __syncthreads();
  }
}

// TimeSeries.apply_boxcar (timeseries.py:296-325) over stats.running_filter
// "mean" (core/stats.py:200-243): the series padded symmetrically (np.pad
// "symmetric", a reflection of period 2n), the mean of each window of
// `width` samples times sqrt(width), rolled by ref_bin.  A CTA computes
// kBoxT consecutive window positions i (pre-roll): it stages the padded samples
// they cover in shared memory, each thread sums its first window in float64
// and slides it across kBoxR positions, and writes out[(i + ref_bin) mod n].
constexpr int kBoxThreads = 256;
constexpr int kBoxR = 16;
constexpr int kBoxT = kBoxThreads * kBoxR;

__device__ __forceinline__ int64_t sym_index(int64_t k, int64_t n) {
  int64_t m = k % (2 * n);
  if (m < 0) m += 2 * n;
  return m < n ? m : 2 * n - 1 - m;
}

__global__ void __launch_bounds__(kBoxThreads)
k_boxcar_filter(const float* __restrict__ in, int64_t n, int width, int64_t pad_left,
                int64_t ref_bin, float* __restrict__ out) {
  extern __shared__ float sx[];  // kBoxT + width - 1
  const int64_t i0 = (int64_t)blockIdx.x * kBoxT;
  const int64_t len = imin64(kBoxT, n - i0) + width - 1;
  for (int64_t k = threadIdx.x; k < len; k += kBoxThreads)
    sx[k] = __ldg(in + sym_index(i0 - pad_left + k, n));
  __syncthreads();
  const int64_t a = (int64_t)threadIdx.x * kBoxR;  // this thread's first position
  if (i0 + a >= n) return;
  const int cnt = (int)imin64(kBoxR, n - i0 - a);
  const double norm = sqrt((double)width);
  double s = 0.0;
  for (int k = 0; k < width; ++k) s += (double)sx[a + k];
  for (int r = 0; r < cnt; ++r) {
    if (r > 0) s = (s + (double)sx[a + r + width - 1]) - (double)sx[a + r - 1];
    const int64_t i = i0 + a + r;
    int64_t j = (i + ref_bin) % n;
    if (j < 0) j += n;
    out[j] = (float)(s / (double)width * norm);
  }
}

// downsample_1d_mean over rows
__global__ void k_downsample(const float* __restrict__ in, int64_t n, int64_t in_stride,
                             int factor, float* __restrict__ out, int64_t out_stride) {
  const int64_t m = n / factor;
  const int64_t row = blockIdx.y;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m;
       i += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int k = 0; k < factor; ++k) s += (double)in[row * in_stride + i * factor + k];
    out[row * out_stride + i] = (float)(s / factor);
  }
}

// downsample_2d_mean_flat
__device__ __forceinline__ float ds_store(float, double v) { return (float)v; }
__device__ __forceinline__ uint8_t ds_store(uint8_t, double v) {
  return (uint8_t)(uint64_t)(int64_t)v;  // numba's float64 -> uint8 cast (truncation)
}

template <typename T>
__global__ void k_downsample_2d(const T* __restrict__ in, int64_t dim1, int64_t dim2,
                                int f1, int f2, T* __restrict__ out) {
  const int64_t n1 = dim1 / f1, n2 = dim2 / f2;
  const int64_t total = n1 * n2;
  const double tot = (double)f1 * f2;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx / n2, j = idx - i * n2;
    double s = 0.0;
    const int64_t pos = dim2 * i * f1 + j * f2;
    for (int a = 0; a < f1; ++a)
      for (int b = 0; b < f2; ++b) s += (double)in[pos + a * dim2 + b];
    out[idx] = ds_store(T(), s / tot);
  }
}

// stage-1 subband (kernels.subband with a zeroed output): atomics into
// out[t][sub], exact for integer input (sums < 2^24).
template <int NB>
__global__ void k_subband(const void* __restrict__ in, int64_t nchans, int64_t nsamps,
                          int bitorder, const int32_t* __restrict__ delays,
                          const int32_t* __restrict__ chan_to_sub, int64_t nsub, int64_t nout,
                          float* __restrict__ out) {
  const int64_t total = nout * nchans;
  for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t t = idx / nchans, c = idx - t * nchans;
    int64_t r = t + delays[c];
    if (r < 0) r += nsamps;
    if (r < 0 || r >= nsamps) continue;
    const int s = chan_to_sub[c];
    if (s < 0 || s >= nsub) continue;
    atomicAdd(out + t * nsub + s, raw_at<NB>(in, nchans, r, c, bitorder));
  }
}

// ---------------------------------------------------------------------------
// Boxcar S/N.  Chunk pass: CTA (chunk k, row r, factor fi) builds the
// downsampled series y over its chunk plus a halo of wmax samples in shared
// memory, scans it to prefix sums, and records per width the best window sum
// starting inside the chunk (smallest start on ties) plus the chunk's sum and
// second central moment.  Final pass merges chunks (Chan et al. 1979 pairwise
// variance) and forms (best - w*mean) / (std*sqrt(w)).
//
// Integer rows run on 32-bit integers wherever that is exact (see k_snr_chunk):
// half the shared memory and no float64 in the window loop.  Threads keep the
// largest window sum only; who holds the chunk's best looks its index up
// afterwards, so a window costs a load and a subtract-and-maximum.  512 int32
// rows x 250001, factors 1/2/4, 9 widths: 2057 -> 979 us (issue 59 %, shared
// loads 48 %, a third of the warps' time at the block's barriers); with the scan's
// runs kept in registers between its passes, the moments' 128-bit arithmetic
// moved past the windows and the index search without dependent steps: 805 us;
// twelve to sixteen loads of a thread in flight, and the subtraction and maximum
// of a window in one instruction: 772 us (one factor: 409 -> 366 us, of them 209
// for loads and scan).  200 float32 rows x 300001, factors 1/2: 867 -> 694 us.
// ---------------------------------------------------------------------------
constexpr int kSnrChunk = 6144;     // downsampled samples per CTA, most
constexpr int kSnrThreads = 256;
constexpr int kSnrMaxW = 4096;
constexpr int kSnrMaxWidths = 32;

struct SnrPart {
  double best;
  int64_t idx;
};

struct SnrCfg {
  int nf, nw, wmax;
  int chunk;      // downsampled samples per CTA
  int smem_words;
  int32_t f[8];
  int32_t w[kSnrMaxWidths];
};

__device__ __forceinline__ double row_val(const void* in, int kind, int64_t i) {
  return kind == SPP_OUT_I32 ? (double)static_cast<const int32_t*>(in)[i]
                             : (double)static_cast<const float*>(in)[i];
}

constexpr int kSnrWarps = kSnrThreads / 32;

__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
#pragma unroll
  for (int w = 0; w < kSnrWarps; ++w) t += red[w];
  return t;
}

// Sum over the warp modulo 2^64, in three pieces whose sums fit 32 bits.
__device__ __forceinline__ long long warp_sum64(long long v) {
  const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)v & 0x3ffffffu);
  const uint32_t mid = __reduce_add_sync(0xffffffffu, (uint32_t)(v >> 26) & 0x3ffffffu);
  const int hi = __reduce_add_sync(0xffffffffu, (int)(v >> 52));
  return (long long)lo + ((long long)mid << 26) + ((long long)hi << 52);
}

// Window arithmetic of the two paths: prefix sums (T), the sum of a window
// (V), the warp's largest one, and the widths taken at a time (kGroup: float64
// twelve, as 256 rows x 100001 and 11 or 24 widths take 7 and 2 % longer by tens;
// integer ten, as twelve cost banks of up to ten widths 2 %).
struct SnrInt {
  static constexpr int kGroup = 10;
  typedef uint32_t T;
  typedef int32_t V;
  __device__ __forceinline__ static V lowest() { return INT_MIN; }
  __device__ __forceinline__ static V window(T b, T a) { return (int32_t)(b - a); }
  __device__ __forceinline__ static V larger(V a, V b) { return max(a, b); }
  // the sum wraps modulo 2^32 as the prefix sums do
  __device__ __forceinline__ static V fold(V m, T b, T a) { return __viaddmax_s32((int32_t)b, (int32_t)(0u - a), m); }
  __device__ __forceinline__ static V warp_max(V v) { return __reduce_max_sync(0xffffffffu, v); }
};
struct SnrF64 {
  static constexpr int kGroup = 12;
  typedef double T;
  typedef double V;
  __device__ __forceinline__ static V lowest() { return -DBL_MAX; }
  __device__ __forceinline__ static V window(T b, T a) { return b - a; }
  __device__ __forceinline__ static V larger(V a, V b) { return b > a ? b : a; }  // ignores NaN
  __device__ __forceinline__ static V fold(V m, T b, T a) { return larger(m, window(b, a)); }
  __device__ __forceinline__ static V warp_max(V v) {
    // ordered 64-bit key, largest high word first, then the low word among equals
    long long k = __double_as_longlong(v);
    k ^= (k >> 63) & 0x7fffffffffffffffll;
    const int hi = (int)(k >> 32);
    const int mh = __reduce_max_sync(0xffffffffu, hi);
    const uint32_t ml = __reduce_max_sync(0xffffffffu, hi == mh ? (uint32_t)k : 0u);
    long long m = ((long long)mh << 32) | ml;
    m ^= (m >> 63) & 0x7fffffffffffffffll;
    return __longlong_as_double(m);
  }
};

// Inclusive scan of s[1..len] in place (s[0] = 0): each thread a run of an odd
// length (distinct banks), then warp and block offsets.
template <typename T>
__device__ __forceinline__ void snr_scan(T* s, int len, T* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = ((len + kSnrThreads - 1) / kSnrThreads) | 1;
  const int a = min(1 + (int)threadIdx.x * per, len + 1), b = min(a + per, len + 1);
  T sum = T(0);
#pragma unroll 5
  for (int j = a; j < b; ++j) sum += s[j];
  T incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  __syncthreads();
  if (lane == 31) red[warp] = incl;
  __syncthreads();
  T run = incl - sum;
  for (int w = 0; w < warp; ++w) run += red[w];
#pragma unroll 5
  for (int j = a; j < b; ++j) {
    run += s[j];
    s[j] = run;
  }
  __syncthreads();
}

// The same for words, each thread's run of PER (odd) held in registers between
// the two passes.  s has 1 + PER * kSnrThreads words; those past the chunk are
// scanned along and mean nothing.
template <int PER>
__device__ __forceinline__ void snr_scan_regs(uint32_t* s, uint32_t* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* p = s + 1 + (int)threadIdx.x * PER;
  uint32_t v[PER];
  uint32_t sum = 0u;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    v[j] = p[j];
    sum += v[j];
  }
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += x;
  }
  if (lane == 31) red[warp] = incl;
  __syncthreads();
  uint32_t run = incl - sum;
#pragma unroll
  for (int w = 0; w < kSnrWarps - 1; ++w) run += w < warp ? red[w] : 0u;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    run += v[j];
    p[j] = run;
  }
  __syncthreads();
}

// Shared words of the widths' search, one set for every group size: a set of its
// own per group size left three float32 CTAs per SM where four fit (100 rows x
// 30000, widths 1 to 512: 51.1 -> 38.2 us; 256 x 100001: 288 -> 241 us).
template <class A>
struct SnrBest {
  typename A::V wbest[kSnrWarps][A::kGroup];
  typename A::V bbest[A::kGroup];
  int bidx[A::kGroup];
};

// Best window of NG widths (from w0) over starts 0..own-1 of the scanned chunk,
// folded into the running best (best, idx) in shared memory; the chunk's first
// sample is at `at` of the CTA's, values are scaled by `scale`.
template <class A, int NG>
__device__ __forceinline__ void snr_window_group(const typename A::T* s, int own, int len,
                                                 const SnrCfg& cfg, int w0, int at, double scale,
                                                 double* best, int* idx, SnrBest<A>& sh) {
  typedef typename A::V V;
  static_assert(NG <= A::kGroup, "widths of a group");
  auto& wbest = sh.wbest;
  auto& bbest = sh.bbest;
  auto& bidx = sh.bidx;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V m[NG];
  const typename A::T* sw[NG];
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    m[g] = A::lowest();
    sw[g] = s + cfg.w[w0 + g] + threadIdx.x;
  }
  const typename A::T* s0 = s + threadIdx.x;
  // starts with every window loaded, four steps of the CTA at a time
  const int full = len == own + cfg.wmax ? own : max(0, min(own, len - cfg.wmax + 1));
  int t = 0;
  for (; t + 4 * kSnrThreads <= full; t += 4 * kSnrThreads) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const typename A::T p0 = s0[t + i * kSnrThreads];
#pragma unroll
      for (int g = 0; g < NG; ++g)
        m[g] = A::fold(m[g], sw[g][t + i * kSnrThreads], p0);
    }
  }
  for (; t + (int)threadIdx.x < own; t += kSnrThreads) {
    const typename A::T p0 = s0[t];
#pragma unroll
    for (int g = 0; g < NG; ++g)
      if (sw[g] + t <= s + len) m[g] = A::larger(m[g], A::window(sw[g][t], p0));
  }
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    const V x = A::warp_max(m[g]);
    if (lane == 0) wbest[warp][g] = x;
  }
  __syncthreads();
  if (threadIdx.x < NG) {
    V x = wbest[0][threadIdx.x];
#pragma unroll
    for (int w = 1; w < kSnrWarps; ++w) x = A::larger(x, wbest[w][threadIdx.x]);
    bbest[threadIdx.x] = x;
    bidx[threadIdx.x] = INT_MAX;
  }
  __syncthreads();
  // the threads that hold a width's best find its first start
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    if (m[g] != bbest[g]) continue;
    const int last = min(own - 1, len - cfg.w[w0 + g]) - (int)threadIdx.x;  // its last start
    int hit = INT_MAX;
#pragma unroll 8
    for (int j = 0; j <= last; j += kSnrThreads)
      hit = min(hit, A::window(sw[g][j], s0[j]) == m[g] ? j : INT_MAX);
    if (hit != INT_MAX) atomicMin(&bidx[g], hit + (int)threadIdx.x);
  }
  __syncthreads();
  if (threadIdx.x < NG && bidx[threadIdx.x] != INT_MAX) {
    const double v = (double)bbest[threadIdx.x] * scale;
    const int i = w0 + threadIdx.x;
    if (idx[i] == INT_MAX || v > best[i]) {
      best[i] = v;
      idx[i] = at + bidx[threadIdx.x];
    }
  }
  __syncthreads();
}

// All widths, kGroup at a time.
template <class A>
__device__ __forceinline__ void snr_windows(const typename A::T* s, int own, int len, const SnrCfg& cfg,
                                            int at, double scale, double* best, int* idx) {
  __shared__ SnrBest<A> sh;
  int w0 = 0;
  for (; w0 + A::kGroup <= cfg.nw; w0 += A::kGroup)
    snr_window_group<A, A::kGroup>(s, own, len, cfg, w0, at, scale, best, idx, sh);
  switch (cfg.nw - w0) {
#define SPP_SNR_CASE(NG)                                                         \
  case NG:                                                                       \
    if constexpr (NG < A::kGroup)                                                \
      snr_window_group<A, NG>(s, own, len, cfg, w0, at, scale, best, idx, sh);   \
    break;
    SPP_SNR_CASE(1) SPP_SNR_CASE(2) SPP_SNR_CASE(3) SPP_SNR_CASE(4) SPP_SNR_CASE(5)
    SPP_SNR_CASE(6) SPP_SNR_CASE(7) SPP_SNR_CASE(8) SPP_SNR_CASE(9) SPP_SNR_CASE(10)
    SPP_SNR_CASE(11)
#undef SPP_SNR_CASE
    default: break;
  }
}

// Sums of F consecutive samples (F = 0: f) for every start of the chunk: prefix
// input, largest sample magnitude, and (of the owned ones) sum and sum of
// squares.  Everything is exact where the caller goes on: f * big <= 2^24, and a
// thread owns 24 sums at most.
template <int F>
__device__ __forceinline__ void snr_load_int(const int32_t* __restrict__ x, int f, int own, int len,
                                             uint32_t* s, uint32_t& big, long long& s1, long long& s2) {
  const int ff = F > 0 ? F : f;
  auto put = [&](int j, int v) {
    s[j + 1] = (uint32_t)v;
    return v;
  };
  auto sum = [&](const int32_t* p, auto load) {
    int v = 0;
#pragma unroll
    for (int q = 0; q < (F > 0 ? F : ff); ++q) {
      const int y = load(p, q);
      big = max(big, (uint32_t)(y < 0 ? 0u - (uint32_t)y : (uint32_t)y));
      v = (int)((uint32_t)v + (uint32_t)y);
    }
    return v;
  };
  auto get = [&](int j) {
    return put(j, sum(x + (int64_t)j * ff, [](const int32_t* p, int q) { return __ldg(p + q); }));
  };
  int a1 = 0;
  auto add = [&](int v) {
    a1 = (int)((uint32_t)a1 + (uint32_t)v);
    s2 += (long long)v * v;
  };
  int j = threadIdx.x;
  if constexpr (F > 0) {
    // twelve or sixteen loads of a thread in flight
    constexpr int B = F == 1 ? 12 : F == 2 ? 8 : 4;
    for (; j - (int)threadIdx.x + B * kSnrThreads <= own; j += B * kSnrThreads) {
      int y[B][F];
#pragma unroll
      for (int i = 0; i < B; ++i)
#pragma unroll
        for (int q = 0; q < F; ++q) y[i][q] = __ldg(x + (int64_t)(j + i * kSnrThreads) * F + q);
#pragma unroll
      for (int i = 0; i < B; ++i)
        add(put(j + i * kSnrThreads, sum(nullptr, [&](const int32_t*, int q) { return y[i][q]; })));
    }
  }
#pragma unroll 4
  for (; j < own; j += kSnrThreads) add(get(j));
  s1 = a1;
#pragma unroll 2
  for (j = own + threadIdx.x; j < len; j += kSnrThreads) get(j);
}

// SUMS (int32 rows): for a power-of-two factor f, y = s / f with s the integer sum of f
// samples.  Where f * |x| <= 2^24 the float32 rounding of y is exact, and where
// f * |x| * wmax < 2^31 window sums are exact differences of prefix sums
// modulo 2^32; the chunk's moments come from 64-bit sums (n * sum(s^2) -
// sum(s)^2 in 128 bits).  Other chunks and float32 rows take float64, in pieces
// that fit the shared memory.
template <int KIND, bool SUMS>
__global__ void __launch_bounds__(kSnrThreads, 4)
k_snr_chunk(const void* __restrict__ in, int64_t n, int64_t in_stride, const SnrCfg cfg,
            int64_t nchunks, SnrPart* __restrict__ parts, double* __restrict__ stats) {
  extern __shared__ __align__(16) uint32_t snr_sm[];
  __shared__ double best[kSnrMaxWidths];
  __shared__ int idx[kSnrMaxWidths];
  __shared__ double red[kSnrWarps];
  __shared__ long long wsum[2][kSnrWarps];
  __shared__ uint32_t scan_red[kSnrWarps];
  const int64_t k = blockIdx.x;
  const int64_t row = blockIdx.y / cfg.nf;
  const int fi = blockIdx.y % cfg.nf;
  const int f = cfg.f[fi];
  const int64_t m = n / f;
  const int64_t i0 = k * cfg.chunk;
  if (i0 >= m) return;
  const int own = (int)imin64(cfg.chunk, m - i0);
  const char* base = static_cast<const char*>(in) + row * in_stride * 4;
  const bool pow2 = (f & (f - 1)) == 0;
  if (threadIdx.x < cfg.nw) {
    best[threadIdx.x] = -DBL_MAX;
    idx[threadIdx.x] = INT_MAX;
  }
  double* st = stats + ((row * cfg.nf + fi) * nchunks + k) * 3;
  bool done = false;
  if constexpr (SUMS) {
    if (pow2) {
      const int len = (int)imin64(own + cfg.wmax, m - i0);
      const int32_t* x = reinterpret_cast<const int32_t*>(base) + i0 * f;
      uint32_t big = 0u;
      long long s1 = 0, s2 = 0;
      if (f == 1) snr_load_int<1>(x, f, own, len, snr_sm, big, s1, s2);
      else if (f == 2) snr_load_int<2>(x, f, own, len, snr_sm, big, s1, s2);
      else if (f == 4) snr_load_int<4>(x, f, own, len, snr_sm, big, s1, s2);
      else snr_load_int<0>(x, f, own, len, snr_sm, big, s1, s2);
      if (threadIdx.x == 0) snr_sm[0] = 0u;
      const unsigned long long top = (unsigned long long)big * (unsigned)f;
      const int wide = top * (unsigned)cfg.wmax >= (1ull << 31) || top > (1ull << 24);
      // a thread's sums are below 24 * 2^24 and 24 * 2^48 unless its values are wide
      s1 = warp_sum64(s1);
      s2 = warp_sum64(s2);
      if ((threadIdx.x & 31) == 0) {
        wsum[0][threadIdx.x >> 5] = s1;
        wsum[1][threadIdx.x >> 5] = s2;
      }
      if (__syncthreads_or(wide) == 0) {
        if (len <= 7 * kSnrThreads) snr_scan_regs<7>(snr_sm, scan_red);
        else if (len <= 13 * kSnrThreads) snr_scan_regs<13>(snr_sm, scan_red);
        else if (len <= 25 * kSnrThreads) snr_scan_regs<25>(snr_sm, scan_red);
        else snr_scan<uint32_t>(snr_sm, len, scan_red);
        snr_windows<SnrInt>(snr_sm, own, len, cfg, 0, 1.0 / (double)f, best, idx);
        done = true;
        if (threadIdx.x == 32) {  // beside the threads that write the widths' bests
          long long S1 = 0, S2 = 0;
          for (int w = 0; w < kSnrWarps; ++w) {
            S1 += wsum[0][w];
            S2 += wsum[1][w];
          }
          const __int128 num = (__int128)S2 * own - (__int128)S1 * S1;
          st[0] = (double)own;
          st[1] = (double)S1 / (double)f;
          st[2] = (double)num / (double)own / ((double)f * (double)f);
        }
      }
    }
  }
  if (!done) {
    double* sy = reinterpret_cast<double*>(snr_sm);
    const int piece = min(cfg.chunk, cfg.smem_words / 2 - cfg.wmax - 1);
    const double inv = 1.0 / (double)f;
    double cnt = 0.0, mean = 0.0, m2 = 0.0;
    for (int p0 = 0; p0 < own; p0 += piece) {
      const int po = min(piece, own - p0);
      const int len = (int)imin64(po + cfg.wmax, m - i0 - p0);
      __syncthreads();
      double s = 0.0;
      for (int j = threadIdx.x; j < len; j += kSnrThreads) {
        // downsampled means rounded to float32 as the reference output dtype; a
        // power-of-two factor divides exactly by multiplying
        double v = 0.0;
        const int64_t x0 = (i0 + p0 + j) * f;
        for (int q = 0; q < f; ++q) v += row_val(base, KIND, x0 + q);
        v = (double)(float)(pow2 ? v * inv : v / f);
        sy[j + 1] = v;
        if (j < po) s += v;
      }
      if (threadIdx.x == 0) sy[0] = 0.0;
      const double tot = block_sum(s, red);
      const double mu = tot / (double)po;
      double q = 0.0;
      for (int j = threadIdx.x; j < po; j += kSnrThreads) {
        const double d = sy[j + 1] - mu;
        q += d * d;
      }
      q = block_sum(q, red);
      // pairwise merge of the pieces' moments (every thread keeps them); nearly all
      // chunks are one piece, and float64 divisions by every thread are a tenth of a
      // short row's time
      if (p0 == 0) {
        cnt = (double)po;
        mean = mu;
        m2 = q;
      } else {
        const double nb = (double)po, d = mu - mean, all = cnt + nb;
        mean += d * nb / all;
        m2 += q + d * d * cnt * nb / all;
        cnt = all;
      }
      if (threadIdx.x == 0) {
        st[0] = cnt;
        st[1] = p0 == 0 ? tot : st[1] + tot;
        st[2] = m2;
      }
      __syncthreads();
      snr_scan<double>(sy, len, red);
      snr_windows<SnrF64>(sy, po, len, cfg, p0, 1.0, best, idx);
    }
  }
  if (threadIdx.x < cfg.nw) {
    SnrPart* p = parts + (((row * cfg.nf + fi) * cfg.nw + threadIdx.x) * nchunks + k);
    p->best = best[threadIdx.x];
    p->idx = idx[threadIdx.x] == INT_MAX ? LLONG_MAX : i0 + idx[threadIdx.x];
  }
}

// `lanes` lanes (a power of two up to the warp) per (row, factor, width): they take
// chunks, moments and maxima merge pairwise.  As many as there are chunks: a warp
// each for rows of one chunk took 390 us for 60000 rows and 8 widths, a third of the
// call (12 us with a lane each).
__global__ void k_snr_final(int64_t n, const SnrCfg cfg, int64_t nrows, int64_t nchunks, int lanes,
                            const SnrPart* __restrict__ parts, const double* __restrict__ stats,
                            float* __restrict__ snr, int32_t* __restrict__ peak,
                            const double* __restrict__ locscale) {
  const int64_t all = nrows * cfg.nf * cfg.nw;
  const int64_t own = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / lanes;
  const int64_t id = imin64(own, all - 1);  // whole warps merge
  const int lane = threadIdx.x & (lanes - 1);
  const int wi = id % cfg.nw;
  const int64_t rf = id / cfg.nw;  // row * nfactors + fi
  const int64_t m = n / cfg.f[rf % cfg.nf];
  const int64_t nck = (m + cfg.chunk - 1) / cfg.chunk;
  double cnt = 0.0, mean = 0.0, m2 = 0.0;
  double best = -DBL_MAX;
  long long bidx = LLONG_MAX;
  for (int64_t k = lane; k < nck; k += lanes) {
    const double* st = stats + (rf * nchunks + k) * 3;
    const double nb = st[0], mb = st[1] / nb;
    const double d = mb - mean, tot = cnt + nb;
    mean += d * nb / tot;
    m2 += st[2] + d * d * cnt * nb / tot;
    cnt = tot;
    const SnrPart p = parts[(rf * cfg.nw + wi) * nchunks + k];
    if (p.idx != LLONG_MAX && (bidx == LLONG_MAX || p.best > best)) {
      best = p.best;
      bidx = p.idx;
    }
  }
  for (int o = lanes / 2; o > 0; o >>= 1) {
    const double nb = __shfl_xor_sync(0xffffffffu, cnt, o);
    const double mb = __shfl_xor_sync(0xffffffffu, mean, o);
    const double qb = __shfl_xor_sync(0xffffffffu, m2, o);
    const double tot = cnt + nb;
    if (nb > 0.0) {
      if (cnt > 0.0) {
        const double d = mb - mean;
        mean += d * nb / tot;
        m2 += qb + d * d * cnt * nb / tot;
      } else {
        mean = mb;
        m2 = qb;
      }
      cnt = tot;
    }
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const long long oi = __shfl_xor_sync(0xffffffffu, bidx, o);
    if (oi != LLONG_MAX && (bidx == LLONG_MAX || ob > best || (ob == best && oi < bidx))) {
      best = ob;
      bidx = oi;
    }
  }
  if (lane != 0 || own >= all) return;
  double sd = cnt > 0 ? sqrt(m2 / cnt) : 0.0;
  if (sd == 0.0) sd = 1.0;
  if (locscale) {  // median / IQR scale
    mean = locscale[rf * 2];
    sd = locscale[rf * 2 + 1];
  }
  const int w = cfg.w[wi];
  snr[id] = bidx == LLONG_MAX ? NAN : (float)((best - (double)w * mean) / (sd * sqrt((double)w)));
  if (peak) peak[id] = bidx == LLONG_MAX ? -1 : (int32_t)bidx;
}

// ---------------------------------------------------------------------------
// Median / IQR of each downsampled row (the S/N epilogue's robust z-score:
// stats.estimate_zscore with loc "median" and scale "iqr", core/stats.py:
// 418-502).  The y values (the same float32 downsampled means as k_snr_chunk)
// are mapped to order-preserving 32-bit keys and the needed order statistics
// are found exactly by radix selection.  Up to six ranks: the two middle values
// (median) and the two neighbours of each quartile's index (q25, q75, linear
// interpolation as numpy's percentile).
//
// A first pass finds the smallest and largest key, so that the 2048 bins of the
// first histogram span the values present (rows of sums share their upper key
// bits: bins by those bits would hold everything at once); two more passes of
// up to 2048 bins per distinct prefix finish any 32-bit range, and passes stop
// once a bin is one key wide.  Rows are split over gridDim.x CTAs whose
// histograms are added in global memory, and the last CTA of a row to finish a
// pass selects: one CTA per row took 2.1 ms for a single row of 262144 samples.
// ---------------------------------------------------------------------------
constexpr int kQThreads = 256;      // row MAD
constexpr int kQBits = 11;
constexpr int kQBins = 1 << kQBits;
constexpr int kQRanks = 6;
constexpr int kQPassThreads = 512;
constexpr int kQSplitRows = 148;    // fewer rows than this are split over CTAs

__device__ __forceinline__ uint32_t f32_key(float v) {
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ float key_f32(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

__device__ __forceinline__ float snr_y(const char* base, int kind, int64_t i, int f, bool pow2,
                                       double inv) {
  double s = 0.0;
  const int64_t x0 = i * f;
  for (int q = 0; q < f; ++q) s += row_val(base, kind, x0 + q);
  return (float)(pow2 ? s * inv : s / f);
}

__device__ __forceinline__ double quantile_lerp(double a, double b, double g) {
  const double diff = b - a;  // numpy _lerp: from the far end when g >= 0.5
  return g >= 0.5 ? b - diff * (1.0 - g) : a + diff * g;
}

// State of one row's selection between passes.
struct QState {
  uint32_t kmin_inv, kmax;  // ~smallest key, largest key (both start at 0: atomicMax)
  uint32_t shift;           // key bits below the bins chosen so far
  uint32_t ndist;
  uint32_t dpre[kQRanks];   // distinct bins (their smallest keys)
  uint32_t slot[kQRanks];   // rank -> distinct bin
  uint32_t left[kQRanks];   // rank within the bin
  uint32_t ctr[4];          // CTAs done, per pass
};

struct QArgs {
  const void* in;
  int kind;
  int64_t n, in_stride;
  QState* st;
  uint32_t* hist;  // per row: kQRanks x kQBins, zeroed per call (split rows only)
  double* locscale;
};

// The row block's values, one per thread and step: f(key) for each.
template <class F>
__device__ __forceinline__ void q_each(const QArgs& a, const SnrCfg& cfg, F&& fn) {
  const int64_t row = blockIdx.y / cfg.nf;
  const int f = cfg.f[blockIdx.y % cfg.nf];
  const int64_t m = a.n / f;
  const char* base = static_cast<const char*>(a.in) + row * a.in_stride * 4;
  const bool pow2 = (f & (f - 1)) == 0;
  const double inv = 1.0 / (double)f;
  const int64_t per = (m + gridDim.x - 1) / gridDim.x;
  const int64_t i1 = imin64(m, per * (blockIdx.x + 1));
#pragma unroll 4
  for (int64_t i = per * blockIdx.x + threadIdx.x; i < i1; i += blockDim.x)
    fn(f32_key(f == 1 ? (float)row_val(base, a.kind, i) : snr_y(base, a.kind, i, f, pow2, inv)));
}

__device__ __forceinline__ void q_range(const QArgs& a, const SnrCfg& cfg, QState& st) {
  uint32_t lo = 0xFFFFFFFFu, hi = 0u;
  q_each(a, cfg, [&](uint32_t k) {
    lo = min(lo, k);
    hi = max(hi, k);
  });
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0 && lo <= hi) {
    atomicMax(&st.kmin_inv, ~lo);
    atomicMax(&st.kmax, hi);
  }
}

// One pass: histogram of the next key bits of the values in the chosen bins,
// then (the row's last CTA) each rank's bin.
template <int PASS, int BITS>
__device__ __forceinline__ void q_pass(const QArgs& a, const SnrCfg& cfg, QState& st) {
  constexpr int kBins = 1 << BITS;
  extern __shared__ uint32_t qhist[];  // (PASS == 0 ? 1 : kQRanks) x kBins
  __shared__ uint32_t dpre[kQRanks], pick[kQRanks], left[kQRanks];
  __shared__ bool last;
  const int f = cfg.f[blockIdx.y % cfg.nf];
  const int64_t m = a.n / f;
  const uint32_t kmin = ~st.kmin_inv;
  const int old = PASS == 0 ? 32 - __clz(st.kmax - kmin) : (int)st.shift;  // bits still open
  if (PASS > 0 && old == 0) return;                                       // selected already
  const int sh = old > BITS ? old - BITS : 0;
  const int nd = PASS == 0 ? 1 : (int)st.ndist;
  if (threadIdx.x < kQRanks) dpre[threadIdx.x] = PASS == 0 ? kmin : st.dpre[threadIdx.x];
  for (int i = threadIdx.x; i < nd * kBins; i += blockDim.x) qhist[i] = 0u;
  __syncthreads();
  if (PASS == 0) {
    q_each(a, cfg, [&](uint32_t k) { atomicAdd(&qhist[(k - kmin) >> sh], 1u); });
  } else {
    const uint32_t span = 1u << old;  // old <= 32 - BITS
    q_each(a, cfg, [&](uint32_t k) {
      for (int d = 0; d < nd; ++d) {
        const uint32_t r = k - dpre[d];
        if (r < span) atomicAdd(&qhist[d * kBins + (r >> sh)], 1u);
      }
    });
  }
  __syncthreads();
  const uint32_t* h = qhist;
  if (gridDim.x > 1) {
    uint32_t* gh = a.hist + ((int64_t)blockIdx.y * 3 + PASS) * kQRanks * kBins;
    for (int i = threadIdx.x; i < nd * kBins; i += blockDim.x)
      if (qhist[i]) atomicAdd(gh + i, qhist[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&st.ctr[PASS], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int i = threadIdx.x; i < nd * kBins; i += blockDim.x) qhist[i] = __ldcg(gh + i);
    __syncthreads();
  }
  // one warp per rank: the bin whose cumulative count passes the rank
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double v25 = (double)(m - 1) * 0.25, v75 = (double)(m - 1) * 0.75;
  const int64_t l25 = (int64_t)floor(v25), l75 = (int64_t)floor(v75);
  if (warp < kQRanks) {
    int64_t r;
    int slot = 0;
    if (PASS == 0) {
      r = warp == 0 ? (m - 1) / 2 : warp == 1 ? m / 2 : warp == 2 ? l25 : warp == 3 ? l25 + 1
          : warp == 4 ? l75 : l75 + 1;
      r = imin64(r, m - 1);
    } else {
      r = st.left[warp];
      slot = (int)st.slot[warp];
    }
    h = qhist + slot * kBins;
    constexpr int per = kBins / 32;
    uint32_t sum = 0;
    for (int j = 0; j < per; ++j) sum += h[lane * per + j];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    const uint32_t excl = incl - sum;
    if ((int64_t)excl <= r && r < (int64_t)incl) {
      int64_t c = excl;
      int d = lane * per;
      for (int j = 0; j < per; ++j, ++d) {
        if (r < c + (int64_t)h[d]) break;
        c += h[d];
      }
      pick[warp] = dpre[slot] + ((uint32_t)d << sh);
      left[warp] = (uint32_t)(r - c);
    }
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  st.shift = (uint32_t)sh;
  int n = 0;
  for (int t = 0; t < kQRanks; ++t) {
    int k = 0;
    while (k < n && st.dpre[k] != pick[t]) ++k;
    if (k == n) st.dpre[n++] = pick[t];
    st.slot[t] = (uint32_t)k;
    st.left[t] = left[t];
  }
  st.ndist = (uint32_t)n;
  if (sh > 0) return;
  float med;
  if (m & 1) {
    med = key_f32(pick[0]);
  } else {
    med = __fmul_rn(__fadd_rn(key_f32(pick[0]), key_f32(pick[1])), 0.5f);
  }
  const double q25 = quantile_lerp((double)key_f32(pick[2]), (double)key_f32(pick[3]), v25 - (double)l25);
  const double q75 = quantile_lerp((double)key_f32(pick[4]), (double)key_f32(pick[5]), v75 - (double)l75);
  double sc = (q75 - q25) / 1.3489795003921634;
  if (fabs(sc) <= 1e-8) sc = 1.0;  // np.isclose(scale, 0) -> 1
  a.locscale[blockIdx.y * 2] = (double)med;
  a.locscale[blockIdx.y * 2 + 1] = sc;
}

__global__ void __launch_bounds__(kQPassThreads) k_q_range(const QArgs a, const SnrCfg cfg) {
  q_range(a, cfg, a.st[blockIdx.y]);
}
template <int PASS>
__global__ void __launch_bounds__(kQPassThreads) k_q_pass(const QArgs a, const SnrCfg cfg) {
  q_pass<PASS, kQBits>(a, cfg, a.st[blockIdx.y]);
}
// All passes of a row in one CTA, its state in shared memory.  Short rows take 256
// bins and, where their keys span all 32 bits, four passes: clearing and scanning
// 2048 bins costs more than a pass over few samples (60000 float32 rows x 200, log-
// normal: 4.62 ms with 2048 bins, 2.83 ms with 256; 1000 x 3000: 111 and 101 us;
// one row of 5000: 22 and 25 us).
constexpr int kQShortRow = 4096;
template <int BITS>
__global__ void __launch_bounds__(kQPassThreads) k_row_quantiles(const QArgs a, const SnrCfg cfg) {
  __shared__ QState st;
  for (int i = threadIdx.x; i < (int)(sizeof(QState) / 4); i += blockDim.x)
    reinterpret_cast<uint32_t*>(&st)[i] = 0u;
  __syncthreads();
  q_range(a, cfg, st);
  __syncthreads();
  q_pass<0, BITS>(a, cfg, st);
  __syncthreads();
  q_pass<1, BITS>(a, cfg, st);
  __syncthreads();
  q_pass<2, BITS>(a, cfg, st);
  if constexpr (3 * BITS < 32) {
    __syncthreads();
    q_pass<3, BITS>(a, cfg, st);
  }
}

// CTAs per (row, factor): enough to fill the chip, 2048 values each at least.
static int q_split(int64_t nrf, int64_t n) {
  if (nrf >= kQSplitRows) return 1;
  return (int)std::max<int64_t>(1, std::min<int64_t>(ceil_div(2 * 148, nrf), n / 2048));
}

static int64_t q_state_bytes(int64_t nrf) { return round_up(nrf * (int64_t)sizeof(QState), 256); }
static int64_t q_workspace(int64_t nrf, int64_t n) {
  return q_split(nrf, n) > 1 ? q_state_bytes(nrf) + nrf * 3 * kQRanks * kQBins * 4 : 0;
}

// Median / IQR scale of `nrf` (row, factor) series; `ws` of q_workspace bytes,
// or nullptr for one CTA per series.
static int launch_quantiles(const void* in, int kind, int64_t nrf, int64_t n, int64_t in_stride,
                            const SnrCfg& cfg, double* locscale, void* ws, cudaStream_t st) {
  const int64_t smem = (int64_t)kQRanks * kQBins * 4;
  QArgs a{in, kind, n, in_stride, nullptr, nullptr, locscale};
  const int split = ws ? q_split(nrf, n) : 1;
  int rc = SPP_OK;
  if (split == 1) {
    const dim3 grid(1, (unsigned)nrf);
    if (n / *std::min_element(cfg.f, cfg.f + cfg.nf) <= kQShortRow) {
      k_row_quantiles<8><<<grid, kQPassThreads, kQRanks * 256 * 4, st>>>(a, cfg);
    } else {
      rc = set_smem_attr(reinterpret_cast<const void*>(k_row_quantiles<kQBits>), smem);
      if (rc) return rc;
      k_row_quantiles<kQBits><<<grid, kQPassThreads, smem, st>>>(a, cfg);
    }
    return cuda_status(cudaGetLastError(), "row quantiles launch");
  }
  rc = cuda_status(cudaMemsetAsync(ws, 0, (size_t)q_workspace(nrf, n), st), "quantile state clear");
  if (!rc) rc = set_smem_attr(reinterpret_cast<const void*>(k_q_pass<1>), smem);
  if (!rc) rc = set_smem_attr(reinterpret_cast<const void*>(k_q_pass<2>), smem);
  if (rc) return rc;
  a.st = static_cast<QState*>(ws);
  a.hist = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(ws) + q_state_bytes(nrf));
  dim3 grid((unsigned)split, (unsigned)nrf);
  k_q_range<<<grid, kQPassThreads, 0, st>>>(a, cfg);
  k_q_pass<0><<<grid, kQPassThreads, kQBins * 4, st>>>(a, cfg);
  k_q_pass<1><<<grid, kQPassThreads, smem, st>>>(a, cfg);
  k_q_pass<2><<<grid, kQPassThreads, smem, st>>>(a, cfg);
  return cuda_status(cudaGetLastError(), "row quantiles launch");
}

// ---------------------------------------------------------------------------
// MatchedFilter (core/filters.py:29-338, kernels.convolve_templates
// core/kernels.py:861-906): the reference correlates the z-scored series with
// each template by FFT over the series repeated to the FFT length N >= n
// (circular_pad_goodsize), the template zero-padded to N, its reference bin
// moved to index 0, time-reversed and normalised to zero mean and unit power
// over all N entries.  That is, for t < n,
//   conv[t] = (sum_j h[j] * z[((t + j - ref) mod N) mod n] - mu * S) / sigma,
// mu = sum(h) / N, sigma = sqrt(sum(h^2) - sum(h)^2 / N), S = sum_{m<N} z[m mod n],
// computed here directly in float64 (the templates are at most a few hundred
// bins) and stored float32 as the reference's convs.
// ---------------------------------------------------------------------------
__global__ void k_zscore(const float* __restrict__ in, int64_t n, const double* __restrict__ ls,
                         float* __restrict__ out) {
  // np.subtract(x, loc, dtype=float32) then np.divide(., scale) into float32
  const float loc = (float)ls[0];
  const double scale = ls[1];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = (float)((double)__fsub_rn(in[i], loc) / scale);
}

// mean and population standard deviation of one row in float64 (loc/scale
// "mean"/"std"), one CTA per row
__global__ void k_row_mean_std(const void* __restrict__ in, int kind, int64_t n, int64_t in_stride,
                               double* __restrict__ ls) {
  __shared__ double red[32];
  const char* base = static_cast<const char*>(in) + (int64_t)blockIdx.x * in_stride * 4;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double s = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += row_val(base, kind, i);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) red[warp] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += red[w];
    red[31] = t / (double)n;
  }
  __syncthreads();
  const double mean = red[31];
  __syncthreads();
  double q = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double d = row_val(base, kind, i) - mean;
    q += d * d;
  }
  for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
  if (lane == 0) red[warp] = q;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += red[w];
    double sd = sqrt(t / (double)n);
    if (fabs(sd) <= 1e-8) sd = 1.0;  // np.isclose(scale, 0) -> 1
    ls[blockIdx.x * 2] = mean;
    ls[blockIdx.x * 2 + 1] = sd;
  }
}

// S = sum_{m < N} z[m mod n] in float64, one CTA
__global__ void k_padded_sum(const float* __restrict__ z, int64_t n, int64_t nfft,
                             double* __restrict__ out) {
  __shared__ double red[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int64_t reps = nfft / n, rem = nfft % n;
  double full = 0.0, part = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = (double)z[i];
    full += v;
    if (i < rem) part += v;
  }
  double t = full * (double)reps + part;
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) red[warp] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double u = 0.0;
    for (int w = 0; w < nw; ++w) u += red[w];
    out[0] = u;
  }
}

// First maximum of convs in flattened (template, sample) order, as np.argmax:
// the float's order-preserving key in the high word and the complement of the
// flat index in the low word, so atomicMax keeps the largest value and, among
// equal values, the smallest index.
__global__ void k_argmax_first(const float* __restrict__ v, int64_t count,
                               unsigned long long* __restrict__ best) {
  __shared__ unsigned long long red[32];
  unsigned long long b = 0ull;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x) {
    const unsigned long long key =
        ((unsigned long long)f32_key(v[i]) << 32) | (unsigned long long)(0xFFFFFFFFu - (uint32_t)i);
    if (key > b) b = key;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long ob = __shfl_xor_sync(0xffffffffu, b, o);
    if (ob > b) b = ob;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = b;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (red[w] > b) b = red[w];
    b = red[0] > b ? red[0] : b;
    atomicMax(best, b);
  }
}

// conv[k][t]: one thread per output sample of one template (blockIdx.y)
__global__ void k_template_conv(const float* __restrict__ z, int64_t n, int64_t nfft,
                                const double* __restrict__ temps, const int32_t* __restrict__ toff,
                                const int32_t* __restrict__ tref, const double* __restrict__ tstat,
                                const double* __restrict__ spad, float* __restrict__ convs) {
  const int k = blockIdx.y;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const double* h = temps + toff[k];
  const int len = toff[k + 1] - toff[k];
  const int64_t ref = tref[k];
  double acc = 0.0;
  int64_t m = t - ref;  // padded index of h[0], taken mod N then mod n
  m %= nfft;
  if (m < 0) m += nfft;
  for (int j = 0; j < len; ++j) {
    acc += h[j] * (double)z[m % n];
    if (++m == nfft) m = 0;
  }
  // tstat[k]: (mu, sigma) of the padded, normalised template
  const double mu = tstat[2 * k], sigma = tstat[2 * k + 1];
  convs[(int64_t)k * n + t] = (float)(sigma > 0.0 ? (acc - mu * spad[0]) / sigma : acc - mu * spad[0]);
}

template <typename F>
static int dispatch_nb(int nbits, F&& f) {
  switch (nbits) {
    case 1: f(std::integral_constant<int, 1>()); return SPP_OK;
    case 2: f(std::integral_constant<int, 2>()); return SPP_OK;
    case 4: f(std::integral_constant<int, 4>()); return SPP_OK;
    case 8: f(std::integral_constant<int, 8>()); return SPP_OK;
    case 32: f(std::integral_constant<int, 32>()); return SPP_OK;
    default: return fail(SPP_ERR_ARG, "nbits must be 1, 2, 4, 8 or 32 (got %d)", nbits);
  }
}

static int check_raw(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps) {
  if (!in) return fail(SPP_ERR_ARG, "null input");
  if (nchans <= 0 || nsamps < 0) return fail(SPP_ERR_ARG, "bad shape");
  if (nbits < 8 && (nchans * nbits) % 8) return fail(SPP_ERR_ARG, "nchans*nbits must be a multiple of 8");
  if (bitorder != SPP_BITORDER_BIG && bitorder != SPP_BITORDER_LITTLE) return fail(SPP_ERR_ARG, "bad bitorder");
  return SPP_OK;
}

}  // namespace spp

using namespace spp;

extern "C" {

int spp_bandpass(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                 float* bpass, void* stream) {
  int rc = check_raw(in, nbits, bitorder, nchans, nsamps);
  if (rc) return rc;
  if (!bpass) return fail(SPP_ERR_ARG, "null bpass");
  if (nsamps == 0) return SPP_OK;
  cudaStream_t st = as_stream(stream);
  const unsigned blocks = (unsigned)ceil_div(nchans, 128);
  rc = dispatch_nb(nbits, [&](auto nb) {
    k_bandpass<decltype(nb)::value><<<blocks, 128, 0, st>>>(in, nchans, nsamps, bitorder, bpass);
  });
  if (rc) return rc;
  return cuda_status(cudaGetLastError(), "bandpass launch");
}

int spp_collapse(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                 float* tim, int64_t out_start, void* stream) {
  int rc = check_raw(in, nbits, bitorder, nchans, nsamps);
  if (rc) return rc;
  if (!tim || out_start < 0) return fail(SPP_ERR_ARG, "bad output");
  if (nsamps == 0) return SPP_OK;
  cudaStream_t st = as_stream(stream);
  const unsigned blocks = (unsigned)ceil_div(nsamps, 8);
  rc = dispatch_nb(nbits, [&](auto nb) {
    k_collapse<decltype(nb)::value><<<blocks, 256, 0, st>>>(in, nchans, nsamps, bitorder, tim, out_start);
  });
  if (rc) return rc;
  return cuda_status(cudaGetLastError(), "collapse launch");
}

int spp_zero_dm(const float* in, float* out, int64_t nchans, int64_t nsamps, const float* bpass,
                const float* chanwts, void* stream) {
  if (!in || !out || !bpass || !chanwts) return fail(SPP_ERR_ARG, "null pointer");
  if (nchans <= 0 || nsamps < 0) return fail(SPP_ERR_ARG, "bad shape");
  if (nsamps == 0) return SPP_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(nsamps, kZdmRows), 148 * 6);
  k_zero_dm<float><<<blocks, kZdmRows, 0, as_stream(stream)>>>(in, out, nchans, nsamps, bpass,
                                                               chanwts);
  return cuda_status(cudaGetLastError(), "zero_dm launch");
}

int spp_zero_dm_u8(const uint8_t* in, uint8_t* out, int64_t nchans, int64_t nsamps,
                   const float* bpass, const float* chanwts, void* stream) {
  if (!in || !out || !bpass || !chanwts) return fail(SPP_ERR_ARG, "null pointer");
  if (nchans <= 0 || nsamps < 0) return fail(SPP_ERR_ARG, "bad shape");
  if (nsamps == 0) return SPP_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(nsamps, kZdmRows), 148 * 6);
  k_zero_dm<uint8_t><<<blocks, kZdmRows, 0, as_stream(stream)>>>(in, out, nchans, nsamps, bpass,
                                                                 chanwts);
  return cuda_status(cudaGetLastError(), "zero_dm launch");
}

int spp_downsample_mean(const float* in, int64_t nrows, int64_t n, int64_t in_stride, int factor,
                        float* out, int64_t out_stride, void* stream) {
  if (!in || !out) return fail(SPP_ERR_ARG, "null pointer");
  if (factor <= 0) return fail(SPP_ERR_ARG, "Factor must be a positive integer.");
  if (nrows <= 0 || n < 0) return fail(SPP_ERR_ARG, "bad shape");
  if (factor > n) return fail(SPP_ERR_ARG, "Factor must be less than the size of the array.");
  if (nrows > 65535) return fail(SPP_ERR_UNSUPPORTED, "too many rows");
  const int64_t m = n / factor;
  dim3 grid((unsigned)std::min<int64_t>(ceil_div(m, 256), 4096), (unsigned)nrows);
  k_downsample<<<grid, 256, 0, as_stream(stream)>>>(in, n, in_stride, factor, out, out_stride);
  return cuda_status(cudaGetLastError(), "downsample launch");
}

int spp_downsample_2d_mean(const float* in, int64_t dim1, int64_t dim2, int factor1, int factor2,
                           float* out, void* stream) {
  if (!in || !out) return fail(SPP_ERR_ARG, "null pointer");
  if (factor1 <= 0 || factor2 <= 0) return fail(SPP_ERR_ARG, "factors must be positive");
  const int64_t total = (dim1 / factor1) * (dim2 / factor2);
  if (total == 0) return SPP_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(total, 256), 148 * 32);
  k_downsample_2d<float><<<blocks, 256, 0, as_stream(stream)>>>(in, dim1, dim2, factor1, factor2, out);
  return cuda_status(cudaGetLastError(), "downsample_2d launch");
}

int spp_downsample_2d_mean_u8(const uint8_t* in, int64_t dim1, int64_t dim2, int factor1,
                              int factor2, uint8_t* out, void* stream) {
  if (!in || !out) return fail(SPP_ERR_ARG, "null pointer");
  if (factor1 <= 0 || factor2 <= 0 || dim1 < 0 || dim2 < 0) return fail(SPP_ERR_ARG, "bad factors");
  const int64_t total = (dim1 / factor1) * (dim2 / factor2);
  if (total == 0) return SPP_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(total, 256), 148 * 32);
  k_downsample_2d<uint8_t><<<blocks, 256, 0, as_stream(stream)>>>(in, dim1, dim2, factor1, factor2,
                                                                  out);
  return cuda_status(cudaGetLastError(), "downsample_2d launch");
}

int spp_subband(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                const int32_t* delays, int32_t maxdelay, const int32_t* chan_to_sub, int64_t nsub,
                float* out, void* stream) {
  int rc = check_raw(in, nbits, bitorder, nchans, nsamps);
  if (rc) return rc;
  if (!delays || !chan_to_sub || !out || nsub <= 0) return fail(SPP_ERR_ARG, "bad arguments");
  const int64_t nout = nsamps - maxdelay;
  if (nout <= 0) return SPP_OK;
  cudaStream_t st = as_stream(stream);
  rc = cuda_status(cudaMemsetAsync(out, 0, sizeof(float) * nout * nsub, st), "subband memset");
  if (rc) return rc;
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(nout * nchans, 256), 148 * 64);
  rc = dispatch_nb(nbits, [&](auto nb) {
    k_subband<decltype(nb)::value><<<blocks, 256, 0, st>>>(in, nchans, nsamps, bitorder, delays,
                                                           chan_to_sub, nsub, nout, out);
  });
  if (rc) return rc;
  return cuda_status(cudaGetLastError(), "subband launch");
}

}  // extern "C"

// Samples per CTA of the chunk pass: the largest of 6144, 3072 and 1536 that
// still gives three CTAs per two SMs, so that few rows fill the chip too (one int32
// series of 20001, factors 1/2/4: 37 -> 12 us with the warp-wide final pass).
// Shorter chunks than that spend more on halos, barriers and the search of each
// width's first best than they gain (32 float32 rows x 100003, 9 widths / 24
// widths: 37 / 61 us in chunks of 6144, 58 / 110 us in chunks of 1536).
constexpr int64_t kSnrFill = 148 * 3 / 2;
static int snr_chunk(int64_t nrf, int64_t n) {
  for (int c = kSnrChunk; c > 1536; c /= 2)
    if (nrf * ceil_div(n, c) >= kSnrFill) return c;
  return 1536;
}

// Sizes the S/N workspace for `n` samples per row, and sets the chunks per series.
// The size is for any shorter series and any fewer of them too: scratch reserved
// for the largest call serves all.  Chunks shorter than kSnrChunk are taken while
// longer ones number below 148 * 8, so they number below twice that.
int64_t snr_ws(int64_t nrows, int64_t n, int nfactors, int nwidths, int64_t* nchunks) {
  const int64_t nrf = nrows * nfactors;
  n = std::max<int64_t>(n, 1);
  *nchunks = ceil_div(n, snr_chunk(nrf, n));
  const int64_t most = std::max(nrf * ceil_div(n, kSnrChunk),
                                std::min<int64_t>(nrf * ceil_div(n, 1536), 2 * kSnrFill));
  return kStatusBytes + round_up(most * nwidths * (int64_t)sizeof(SnrPart), 256) +
         round_up(most * 3 * (int64_t)sizeof(double), 256);
}

extern "C" {

int64_t spp_boxcar_snr_workspace_bytes(int64_t nrows, int64_t n, int nfactors, int nwidths) {
  int64_t nck;
  return snr_ws(nrows, n, nfactors, nwidths, &nck);
}

}  // extern "C"

// Robust z-score: loc and scale per (row, factor), and the selection's state, for
// any fewer series too (from kQSplitRows on they are not split and need none).
static int64_t robust_ws(int64_t nrf, int64_t n) {
  return round_up(nrf * 16, 256) + round_up(q_workspace(std::min<int64_t>(nrf, kQSplitRows - 1), n), 256);
}

static int boxcar_snr_impl(const void* in, int in_kind, int64_t nrows, int64_t n,
                           int64_t in_stride, const int32_t* factors, int nfactors,
                           const int32_t* widths, int nwidths, float* snr, int32_t* peak_index,
                           void* workspace, int64_t workspace_bytes, void* stream, bool robust) {
  if (!in || !factors || !widths || !snr || !workspace) return fail(SPP_ERR_ARG, "null pointer");
  if (in_kind != SPP_OUT_F32 && in_kind != SPP_OUT_I32) return fail(SPP_ERR_ARG, "bad in_kind");
  if (nrows <= 0 || n <= 0 || nfactors <= 0 || nfactors > 8 || nwidths <= 0 ||
      nwidths > kSnrMaxWidths)
    return fail(SPP_ERR_ARG, "bad sizes (nfactors <= 8, nwidths <= %d)", kSnrMaxWidths);
  if (nrows * nfactors > 65535) return fail(SPP_ERR_UNSUPPORTED, "rows*factors > 65535");
  SnrCfg cfg{};
  cfg.nf = nfactors;
  cfg.nw = nwidths;
  cfg.wmax = 1;
  for (int i = 0; i < nfactors; ++i) {
    if (factors[i] <= 0 || factors[i] > n) return fail(SPP_ERR_ARG, "invalid downsample factor %d", factors[i]);
    cfg.f[i] = factors[i];
  }
  for (int i = 0; i < nwidths; ++i) {
    if (widths[i] < 1 || widths[i] > kSnrMaxW) return fail(SPP_ERR_ARG, "invalid boxcar width: %d", widths[i]);
    cfg.w[i] = widths[i];
    cfg.wmax = std::max(cfg.wmax, (int)widths[i]);
  }
  int64_t nck;
  const int64_t base_need = snr_ws(nrows, n, nfactors, nwidths, &nck);
  const int64_t need = base_need + (robust ? robust_ws(nrows * nfactors, n) : 0);
  if (workspace_bytes < need)
    return fail(SPP_ERR_SIZE, "workspace %lld < %lld", (long long)workspace_bytes, (long long)need);
  cudaStream_t st = as_stream(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  SnrPart* parts = reinterpret_cast<SnrPart*>(ws + kStatusBytes);
  double* stats = reinterpret_cast<double*>(
      ws + kStatusBytes + round_up(nrows * nfactors * nwidths * nck * (int64_t)sizeof(SnrPart), 256));
  // chunks shorter than two halos would mostly load halo
  cfg.chunk = snr_chunk(nrows * nfactors, n);
  while (cfg.chunk < kSnrChunk && cfg.chunk < 2 * cfg.wmax) cfg.chunk *= 2;
  const bool ints = in_kind == SPP_OUT_I32;
  // float64 pieces of at least 512 starts fit beside the halo; whole runs of the
  // scan in registers
  const int most = cfg.chunk + cfg.wmax;
  const int runs = most <= 7 * kSnrThreads ? 7 : most <= 13 * kSnrThreads ? 13 : most <= 25 * kSnrThreads ? 25 : 0;
  cfg.smem_words = ints ? std::max({most + 2, 1 + runs * kSnrThreads, 2 * (cfg.wmax + 513)})
                        : 2 * (cfg.chunk + cfg.wmax + 1);
  const int64_t smem = (int64_t)cfg.smem_words * 4;
  // integer rows without a power-of-two factor have no use for the integer path
  const bool sums = ints && std::any_of(cfg.f, cfg.f + nfactors, [](int f) { return (f & (f - 1)) == 0; });
  auto fn = !ints ? k_snr_chunk<SPP_OUT_F32, false> : sums ? k_snr_chunk<SPP_OUT_I32, true> : k_snr_chunk<SPP_OUT_I32, false>;
  int rc = SPP_OK;
  if (smem > 48 * 1024) {
    rc = set_smem_attr(reinterpret_cast<const void*>(fn), smem);
    if (rc) return rc;
  }
  dim3 grid((unsigned)ceil_div(n, cfg.chunk), (unsigned)(nrows * nfactors));
  fn<<<grid, kSnrThreads, smem, st>>>(in, n, in_stride, cfg, nck, parts, stats);
  rc = cuda_status(cudaGetLastError(), "snr chunk launch");
  if (rc) return rc;
  double* locscale = nullptr;
  if (robust) {
    locscale = reinterpret_cast<double*>(ws + base_need);
    rc = launch_quantiles(in, in_kind, nrows * nfactors, n, in_stride, cfg, locscale,
                          ws + base_need + round_up(nrows * nfactors * 16, 256), st);
    if (rc) return rc;
  }
  const int64_t nout = nrows * nfactors * nwidths;
  int lanes = 1;
  while (lanes < 32 && lanes < ceil_div(n, cfg.chunk)) lanes *= 2;
  k_snr_final<<<(unsigned)ceil_div(nout * lanes, 256), 256, 0, st>>>(n, cfg, nrows, nck, lanes, parts, stats,
                                                                    snr, peak_index, locscale);
  return cuda_status(cudaGetLastError(), "snr final launch");
}

// ---------------------------------------------------------------------------
// Median absolute deviation of each row (stats._scale_mad, core/stats.py:
// 505-536, with estimate_loc's float32 median, core/stats.py:284-326).  One
// CTA per row: the two middle values by radix selection over order-preserving
// 32-bit float keys give the float32 median (averaged in float32) and the
// float64 one (averaged in float64, as np.median of the float64 copy); the
// two middle absolute deviations |f64(x) - median64| by radix selection over
// their 64-bit patterns (non-negative doubles order as unsigned integers) give
// the MAD, divided by Phi^-1(3/4); a MAD within 1e-8 of 0 is replaced by the
// mean absolute deviation over sqrt(2/pi) (a float64 sum in another order
// than numpy's pairwise one), and a scale within 1e-8 of 0 by 1.
// ---------------------------------------------------------------------------

// Ranks r0 <= r1 of n keys by radix selection in one CTA: digits of kQBits
// from the top; each pass histograms (warp-aggregated shared atomics) the
// keys that match a rank's fixed higher digits, then fixes that rank's next
// digit.  `out` (shared) receives the two keys.
template <typename K, class KeyF>
__device__ void select_pair(int64_t n, int64_t r0, int64_t r1, const KeyF& key, uint32_t* hist,
                            K* out) {
  constexpr int kBits = (int)sizeof(K) * 8;
  __shared__ K pre[2];
  __shared__ long long rk[2];
  if (threadIdx.x == 0) {
    pre[0] = pre[1] = K(0);
    rk[0] = r0;
    rk[1] = r1;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int hi = kBits; hi > 0; hi -= kQBits) {
    const int lo = hi > kQBits ? hi - kQBits : 0;
    const int wb = hi - lo;
    const K himask = hi >= kBits ? K(0) : ~((K(1) << hi) - K(1));
    const K dmask = (K(1) << wb) - K(1);
    for (int i = threadIdx.x; i < 2 * kQBins; i += blockDim.x) hist[i] = 0u;
    __syncthreads();
    const K p0 = pre[0], p1 = pre[1];
    const int64_t nr = (n + blockDim.x - 1) / blockDim.x * blockDim.x;  // whole warps iterate
    for (int64_t i = threadIdx.x; i < nr; i += blockDim.x) {
      int id0 = -1, id1 = -1;
      if (i < n) {
        const K k = key(i);
        const int dig = (int)((k >> lo) & dmask);
        if ((k & himask) == p0) id0 = dig;
        if ((k & himask) == p1) id1 = kQBins + dig;
      }
      unsigned peers = __match_any_sync(0xffffffffu, id0);
      if (id0 >= 0 && lane == __ffs(peers) - 1) atomicAdd(&hist[id0], (uint32_t)__popc(peers));
      peers = __match_any_sync(0xffffffffu, id1);
      if (id1 >= 0 && lane == __ffs(peers) - 1) atomicAdd(&hist[id1], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      const int r = threadIdx.x;
      const uint32_t* h = hist + r * kQBins;
      long long c = 0;
      int d = 0;
      for (; d < (1 << wb) - 1; ++d) {
        if (rk[r] < c + (long long)h[d]) break;
        c += h[d];
      }
      rk[r] -= c;
      pre[r] |= K(d) << lo;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = pre[0];
    out[1] = pre[1];
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kQThreads)
k_row_mad(const void* __restrict__ in, int kind, int64_t n, int64_t in_stride,
          double* __restrict__ locscale) {
  __shared__ uint32_t hist[2 * kQBins];
  __shared__ uint32_t k32[2];
  __shared__ unsigned long long k64[2];
  __shared__ double red[kQThreads / 32];
  const int64_t row = blockIdx.x;
  const char* base = static_cast<const char*>(in) + row * in_stride * 4;
  // the reference z-scores float32 data (integer rows converted exactly)
  auto xv = [&](int64_t i) -> float {
    return kind == SPP_OUT_I32 ? (float)reinterpret_cast<const int32_t*>(base)[i]
                               : reinterpret_cast<const float*>(base)[i];
  };
  const int64_t r0 = (n - 1) / 2, r1 = n / 2;
  select_pair<uint32_t>(n, r0, r1, [&](int64_t i) { return f32_key(xv(i)); }, hist, k32);
  const float a = key_f32(k32[0]), b = key_f32(k32[1]);
  const float med32 = (n & 1) ? a : __fmul_rn(__fadd_rn(a, b), 0.5f);
  const double med64 = (n & 1) ? (double)a : __dmul_rn(__dadd_rn((double)a, (double)b), 0.5);
  select_pair<unsigned long long>(
      n, r0, r1,
      [&](int64_t i) {
        return (unsigned long long)__double_as_longlong(fabs(__dsub_rn((double)xv(i), med64)));
      },
      hist, k64);
  const double da = __longlong_as_double((long long)k64[0]);
  const double db = __longlong_as_double((long long)k64[1]);
  const double medd = (n & 1) ? da : __dmul_rn(__dadd_rn(da, db), 0.5);
  double mad = __ddiv_rn(medd, 0.6744897501960817);  // scipy.stats.norm.ppf(0.75)
  if (fabs(mad) <= 1e-8) {  // np.isclose(mad, 0)
    double s = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) s += fabs(__dsub_rn((double)xv(i), med64));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < kQThreads / 32; ++w) t += red[w];
      mad = __ddiv_rn(__ddiv_rn(t, (double)n), __dsqrt_rn(__ddiv_rn(2.0, 3.141592653589793)));
    }
  }
  if (threadIdx.x == 0) {
    locscale[row * 2] = (double)med32;
    locscale[row * 2 + 1] = fabs(mad) <= 1e-8 ? 1.0 : mad;
  }
}

extern "C" {

int spp_boxcar_snr(const void* in, int in_kind, int64_t nrows, int64_t n, int64_t in_stride,
                   const int32_t* factors, int nfactors, const int32_t* widths, int nwidths,
                   float* snr, int32_t* peak_index, void* workspace, int64_t workspace_bytes,
                   void* stream) {
  return boxcar_snr_impl(in, in_kind, nrows, n, in_stride, factors, nfactors, widths, nwidths, snr,
                         peak_index, workspace, workspace_bytes, stream, false);
}

int spp_boxcar_filter(const float* in, int64_t n, int width, float* out, void* stream) {
  if (!in || !out) return fail(SPP_ERR_ARG, "spp_boxcar_filter: null pointer");
  if (width < 1) return fail(SPP_ERR_ARG, "invalid boxcar width: %d", width);
  if (n <= 0) return fail(SPP_ERR_ARG, "empty series");
  if (width > 8192) return fail(SPP_ERR_UNSUPPORTED, "boxcar width %d > 8192", width);
  if (in == out) return fail(SPP_ERR_ARG, "spp_boxcar_filter: in and out must differ");
  const int64_t pad_left = width / 2;
  // the reference's -width // 2 + 1 (odd) or -width // 2 (even), Python floor
  // division: -(width / 2) either way
  const int64_t ref_bin = -(int64_t)(width / 2);
  const int64_t smem = (int64_t)(kBoxT + width - 1) * 4;
  int rc = SPP_OK;
  if (smem > 48 * 1024) {
    rc = set_smem_attr(reinterpret_cast<const void*>(k_boxcar_filter), smem);
    if (rc) return rc;
  }
  k_boxcar_filter<<<(unsigned)ceil_div(n, kBoxT), kBoxThreads, smem, as_stream(stream)>>>(
      in, n, width, pad_left, ref_bin, out);
  return cuda_status(cudaGetLastError(), "boxcar filter launch");
}

int spp_row_loc_scale(const void* in, int in_kind, int64_t nrows, int64_t n, int64_t in_stride,
                      int method, double* loc_scale, void* stream) {
  if (!in || !loc_scale) return fail(SPP_ERR_ARG, "spp_row_loc_scale: null pointer");
  if (in_kind != SPP_OUT_F32 && in_kind != SPP_OUT_I32) return fail(SPP_ERR_ARG, "bad in_kind");
  if (nrows <= 0 || nrows > 65535 || n <= 0) return fail(SPP_ERR_ARG, "bad sizes");
  cudaStream_t st = as_stream(stream);
  if (method == 0) {
    k_row_mean_std<<<(unsigned)nrows, 256, 0, st>>>(in, in_kind, n, in_stride, loc_scale);
    return cuda_status(cudaGetLastError(), "mean/std launch");
  }
  if (method == 2) {
    k_row_mad<<<(unsigned)nrows, kQThreads, 0, st>>>(in, in_kind, n, in_stride, loc_scale);
    return cuda_status(cudaGetLastError(), "median/MAD launch");
  }
  if (method != 1)
    return fail(SPP_ERR_ARG, "method must be 0 (mean/std), 1 (median/iqr) or 2 (median/mad)");
  SnrCfg cfg{};
  cfg.nf = 1;
  cfg.f[0] = 1;
  return launch_quantiles(in, in_kind, nrows, n, in_stride, cfg, loc_scale, nullptr, st);
}

int spp_zscore(const float* in, int64_t n, const double* loc_scale, float* out, void* stream) {
  if (!in || !loc_scale || !out) return fail(SPP_ERR_ARG, "spp_zscore: null pointer");
  if (n <= 0) return fail(SPP_ERR_ARG, "empty series");
  const unsigned blocks = (unsigned)std::min<int64_t>(ceil_div(n, 256), 148 * 16);
  k_zscore<<<blocks, 256, 0, as_stream(stream)>>>(in, n, loc_scale, out);
  return cuda_status(cudaGetLastError(), "zscore launch");
}

int spp_matched_filter(const float* z, int64_t n, int64_t nfft, const double* temps,
                       const int32_t* temp_offsets, const int32_t* ref_bins,
                       const double* temp_stats, int ntemps, float* convs, void* workspace,
                       int64_t workspace_bytes, void* stream) {
  if (!z || !temps || !temp_offsets || !ref_bins || !temp_stats || !convs || !workspace)
    return fail(SPP_ERR_ARG, "spp_matched_filter: null pointer");
  if (n <= 0 || nfft < n) return fail(SPP_ERR_ARG, "need 0 < n <= nfft");
  if (ntemps <= 0 || ntemps > 65535) return fail(SPP_ERR_ARG, "bad template count");
  if (workspace_bytes < 16) return fail(SPP_ERR_SIZE, "workspace < 16 B");
  if ((int64_t)ntemps * n > 0xFFFFFFFFll) return fail(SPP_ERR_UNSUPPORTED, "ntemps * n >= 2^32");
  cudaStream_t st = as_stream(stream);
  double* spad = static_cast<double*>(workspace);
  unsigned long long* best = reinterpret_cast<unsigned long long*>(spad + 1);
  int rc = cuda_status(cudaMemsetAsync(best, 0, 8, st), "best clear");
  if (rc) return rc;
  k_padded_sum<<<1, 1024, 0, st>>>(z, n, nfft, spad);
  rc = cuda_status(cudaGetLastError(), "padded sum launch");
  if (rc) return rc;
  dim3 grid((unsigned)ceil_div(n, 256), (unsigned)ntemps);
  k_template_conv<<<grid, 256, 0, st>>>(z, n, nfft, temps, temp_offsets, ref_bins, temp_stats,
                                        spad, convs);
  rc = cuda_status(cudaGetLastError(), "template convolution launch");
  if (rc) return rc;
  const int64_t count = (int64_t)ntemps * n;
  k_argmax_first<<<(unsigned)std::min<int64_t>(ceil_div(count, 256), 148 * 8), 256, 0, st>>>(
      convs, count, best);
  return cuda_status(cudaGetLastError(), "argmax launch");
}

int64_t spp_boxcar_snr_robust_workspace_bytes(int64_t nrows, int64_t n, int nfactors,
                                              int nwidths) {
  int64_t nck;
  return snr_ws(nrows, n, nfactors, nwidths, &nck) + robust_ws(nrows * nfactors, n);
}

int spp_boxcar_snr_robust(const void* in, int in_kind, int64_t nrows, int64_t n,
                          int64_t in_stride, const int32_t* factors, int nfactors,
                          const int32_t* widths, int nwidths, float* snr, int32_t* peak_index,
                          void* workspace, int64_t workspace_bytes, void* stream) {
  return boxcar_snr_impl(in, in_kind, nrows, n, in_stride, factors, nfactors, widths, nwidths, snr,
                         peak_index, workspace, workspace_bytes, stream, true);
}

}  // extern "C"
