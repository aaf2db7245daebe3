// Single-pass single-DM dedispersion for 8-bit data (the Filterbank.dedisperse
// hot loop, kernels.dedisperse core/kernels.py:340-362): raw time-major bytes
// go straight from HBM into shared memory, no corner turn.
//
// CTA = 256 output samples [t0, t0 + 256) over all channels, walked in slabs
// of 32 channels (32 bytes of each raw row).  All warps first read the delays
// of every slab in parallel (one round trip) into shared tables.  Slabs are
// then staged in packs: as many consecutive slabs as fit the row budget, each
// slab's rows [t0 + dmin_s, t0 + 256 + dmax_s) copied with 4-byte cp.async
// into shared rows of 36 bytes (pitch 9 words: the 32 consecutive rows a warp
// reads for one channel fall in 32 different banks); rows outside the block
// wrap once (numba's negative-index wraparound) or read as zero.  Each thread
// accumulates one output sample over all channels (exact int32) and stores it
// once.
#include <algorithm>

#include "spp_common.cuh"

namespace spp {

constexpr int kS1T = 256;        // outputs per CTA
constexpr int kS1Slab = 32;      // channels per slab
constexpr int kS1Pitch = 36;     // bytes per staged row

__device__ __forceinline__ void cp_async4(void* dst, const void* src, bool valid) {
  const uint32_t d = smem_addr(dst);
  const int n = valid ? 4 : 0;  // src-size 0 fills zeros
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

struct S1Args {
  const uint8_t* raw;
  int64_t nchans, nsamps;
  const int32_t* delays;
  int32_t dlo, dhi;
  float* out;
  int64_t out_start, nvalid;
  uint32_t* status;
};

// Per-slab delay range (every warp computes it from the same 32 delays).
__device__ __forceinline__ void slab_range(const S1Args& a, int c0, int lane, int32_t& d_lane,
                                           int32_t& mn, int32_t& mx) {
  const int c = c0 + lane;
  int32_t d = 0;
  if (c < a.nchans) {
    d = __ldg(a.delays + c);
    if (d < a.dlo || d > a.dhi) {
      dev_flag(a.status, SPP_DEV_RANGE, (uint32_t)c);
      d = min(max(d, a.dlo), a.dhi);
    }
  }
  d_lane = d;
  mn = (c < a.nchans) ? d : INT32_MAX;
  mx = (c < a.nchans) ? d : INT32_MIN;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
}

// Stage rows [r0, r0 + nrows) of the slab starting at channel c0 into buf.
// Thread (row phase tid/8, word tid%8) walks rows 32 apart; rows inside the
// block use plain pointer increments, rows outside it wrap or read zero.
__device__ __forceinline__ void stage(const S1Args& a, uint8_t* buf, int64_t r0, int nrows, int c0) {
  const int64_t rowbytes = a.nchans;
  const int nw = min(kS1Slab, (int)(a.nchans - c0)) / 4;  // words per row (nchans % 4 == 0)
  const int w = threadIdx.x & 7;
  int r = threadIdx.x >> 3;
  constexpr int kStep = kS1T / 8;  // rows per pass
  if (w >= nw) return;
  if (r0 >= 0 && r0 + nrows <= a.nsamps) {
    const uint8_t* src = a.raw + (r0 + r) * rowbytes + c0 + 4 * w;
    uint8_t* dst = buf + r * kS1Pitch + 4 * w;
    const int64_t sstep = (int64_t)kStep * rowbytes;
    for (; r < nrows; r += kStep, src += sstep, dst += kStep * kS1Pitch) cp_async4(dst, src, true);
    return;
  }
  for (; r < nrows; r += kStep) {
    int64_t row = r0 + r;
    if (row < 0) row += a.nsamps;
    else if (row >= a.nsamps) row -= a.nsamps;
    const bool ok = row >= 0 && row < a.nsamps;
    const uint8_t* src = ok ? a.raw + row * rowbytes + c0 + 4 * w : a.raw;
    cp_async4(buf + r * kS1Pitch + 4 * w, src, ok);
  }
}

__global__ void __launch_bounds__(kS1T) k_dedisp_single8(const S1Args a, int32_t cap_rows) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int nslab = (int)((a.nchans + kS1Slab - 1) / kS1Slab);
  uint8_t* rowbuf = sm;
  int32_t* smn = reinterpret_cast<int32_t*>(sm + (int64_t)cap_rows * kS1Pitch);  // [nslab]
  int32_t* snr = smn + nslab;                                                    // [nslab] rows
  int32_t* sdo = snr + nslab;                                                    // [nslab][32]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t0 = (int64_t)blockIdx.x * kS1T;
  for (int sl = warp; sl < nslab; sl += kS1T / 32) {
    int32_t dl, mn, mx;
    slab_range(a, sl * kS1Slab, lane, dl, mn, mx);
    sdo[sl * 32 + lane] = (dl - mn) * kS1Pitch + lane;  // byte offset of channel lane
    if (lane == 0) {
      smn[sl] = mn;
      snr[sl] = kS1T + (mx - mn);
    }
  }
  __syncthreads();
  const int t = threadIdx.x;
  int32_t acc = 0;
  int s0 = 0;
  while (s0 < nslab) {
    // pack consecutive slabs into the row budget
    int s1 = s0, used = 0;
    while (s1 < nslab && used + snr[s1] <= cap_rows) used += snr[s1++];
    if (s1 == s0) {  // one slab larger than the budget: flag and stop
      if (t == 0) dev_flag(a.status, SPP_DEV_RANGE, (uint32_t)s0);
      return;
    }
    int off = 0;
    for (int sl = s0; sl < s1; ++sl) {
      stage(a, rowbuf + (int64_t)off * kS1Pitch, t0 + smn[sl], snr[sl], sl * kS1Slab);
      off += snr[sl];
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    off = 0;
    for (int sl = s0; sl < s1; ++sl) {
      const uint8_t* base = rowbuf + (int64_t)(off + t) * kS1Pitch;
      const int32_t* dd = sdo + sl * 32;
      const int64_t rem = a.nchans - (int64_t)sl * kS1Slab;
      int32_t sacc = 0;
      if (rem >= kS1Slab) {
#pragma unroll
        for (int c = 0; c < kS1Slab; ++c) sacc += base[dd[c]];
      } else {
        for (int c = 0; c < (int)rem; ++c) sacc += base[dd[c]];
      }
      acc += sacc;
      off += snr[sl];
    }
    __syncthreads();
    s0 = s1;
  }
  const int64_t tt = t0 + t;
  if (tt < a.nvalid) a.out[a.out_start + tt] = (float)acc;
}

// Launches the single-pass kernel when it applies (8-bit, nchans % 4 == 0,
// every slab's rows within the shared-memory budget); returns
// SPP_ERR_UNSUPPORTED to let the caller use the corner-turn path otherwise.
int launch_single8(const uint8_t* raw, int64_t nchans, int64_t nsamps, const int32_t* delays,
                   int32_t dlo, int32_t dhi, float* out, int64_t out_start, int64_t nvalid,
                   uint32_t* status, cudaStream_t st) {
  if (nchans % 4 != 0 || (reinterpret_cast<uintptr_t>(raw) & 3) != 0 || nchans > 8192)
    return SPP_ERR_UNSUPPORTED;
  const int64_t nslab = ceil_div(nchans, kS1Slab);
  // a slab never needs more than kS1T + (dhi - dlo) rows
  const int64_t cap = std::max<int64_t>(1600, kS1T + ((int64_t)dhi - dlo) + 1);
  const int64_t smem = cap * kS1Pitch + nslab * (2 + 32) * 4;
  if (smem > 110 * 1024) return SPP_ERR_UNSUPPORTED;
  int rc = set_smem_attr(reinterpret_cast<const void*>(k_dedisp_single8), smem);
  if (rc) return rc;
  S1Args a{raw, nchans, nsamps, delays, dlo, dhi, out, out_start, nvalid, status};
  const int64_t gx = ceil_div(nvalid, kS1T);
  if (gx > INT32_MAX) return SPP_ERR_UNSUPPORTED;
  k_dedisp_single8<<<(unsigned)gx, kS1T, smem, st>>>(a, (int32_t)cap);
  return cuda_status(cudaGetLastError(), "single-DM launch");
}

// ---------------------------------------------------------------------------
// Host-table variant (spp_dedisperse_hd): the delays are known on the host, so
// every per-slab row range and per-channel byte offset is computed there and
// passed in the kernel parameters.  A CTA issues the copies of all its slabs
// at once -- one cp.async group per slab, no delay round trip first -- and
// adds slab s as soon as group s has landed.
//
// Staged rows are the raw 32 bytes of a slab, dense (16-B cp.async.cg).  A warp
// covers 4 consecutive outputs x 8 channel words per load: lane (i = lane & 3,
// j = lane >> 2) reads channel 4j + k of output row t + i.  For any delays the
// 32 lanes hit 32 distinct banks (bank = 8 * (row mod 4) + j), so every load
// is one wavefront.  Each lane keeps G partial sums (outputs 4g + i of its
// warp's range, over its channels); three shuffles over j finish them.  A CTA
// of W warps covers T = 4 W G outputs; W is chosen per launch (up to 32) so
// that one CTA per SM covers the block.
// Used when nchans is a multiple of 32, at most 32 * NS, and all slabs of a CTA
// fit in shared memory together.

constexpr int kHdMaxWarps = 32;
constexpr int kHdMaxG = 8;                    // output groups of 4 per warp
constexpr int kHdPitch = 32;                  // bytes per staged row

template <int NS>
struct S2Args {
  const uint8_t* raw;
  int64_t nchans, nsamps;
  float* out;
  int64_t out_start, nvalid;
  int32_t nslab;
  int32_t tab_off;       // byte offset of the channel-offset table in shared memory
  int32_t mn[NS];        // per slab: min delay
  int32_t nrows[NS];     // per slab: T + max - min rows staged
  int32_t srow[NS];      // per slab: first staged row in shared memory
  int32_t off[NS * 32];  // per channel: (delay - slab min) * 32 + channel in slab
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const uint32_t d = smem_addr(dst);
  const int n = valid ? 16 : 0;  // src-size 0 fills zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n)
               : "memory");
}

// Stage rows [r0, r0 + nrows) of the 32-channel slab at c0 with cp.async: two
// 16-B chunks per row, chunk q = 2 * row + half, threads striding by the block
// size; rows outside the block wrap once (numba negative indices) or read 0.
__device__ __forceinline__ void stage_hd(const uint8_t* raw, int64_t rowbytes, int64_t nsamps,
                                         uint8_t* buf, int64_t r0, int nrows, int64_t c0) {
  const int nq = 2 * nrows;
  const int nt = blockDim.x;  // a multiple of 32: every thread keeps its half
  int q = threadIdx.x;
  const int h = q & 1;
  const int row_step = nt >> 1;
  if (r0 >= 0 && r0 + nrows <= nsamps) {
    const uint8_t* src = raw + (r0 + (q >> 1)) * rowbytes + c0 + 16 * h;
    uint8_t* dst = buf + (q >> 1) * kHdPitch + 16 * h;
    const int64_t sstep = (int64_t)row_step * rowbytes;
    for (; q < nq; q += nt, src += sstep, dst += row_step * kHdPitch) cp_async16(dst, src, true);
    return;
  }
  for (; q < nq; q += nt) {
    int64_t row = r0 + (q >> 1);
    if (row < 0) row += nsamps;
    else if (row >= nsamps) row -= nsamps;
    const bool ok = row >= 0 && row < nsamps;
    const uint8_t* src = ok ? raw + row * rowbytes + c0 + 16 * h : raw;
    cp_async16(buf + (q >> 1) * kHdPitch + 16 * h, src, ok);
  }
}

// cp.async.wait_group takes an immediate; with `n` known after unrolling the
// switch folds to the one instruction.
__device__ __forceinline__ void cp_async_wait_n(int n) {
  switch (n) {
#define SPP_WAIT_CASE(k) \
  case k:                \
    cp_async_wait<k>();  \
    break;
    SPP_WAIT_CASE(0) SPP_WAIT_CASE(1) SPP_WAIT_CASE(2) SPP_WAIT_CASE(3) SPP_WAIT_CASE(4)
    SPP_WAIT_CASE(5) SPP_WAIT_CASE(6) SPP_WAIT_CASE(7) SPP_WAIT_CASE(8) SPP_WAIT_CASE(9)
    SPP_WAIT_CASE(10) SPP_WAIT_CASE(11) SPP_WAIT_CASE(12) SPP_WAIT_CASE(13) SPP_WAIT_CASE(14)
    SPP_WAIT_CASE(15) SPP_WAIT_CASE(16) SPP_WAIT_CASE(17) SPP_WAIT_CASE(18) SPP_WAIT_CASE(19)
    SPP_WAIT_CASE(20) SPP_WAIT_CASE(21) SPP_WAIT_CASE(22) SPP_WAIT_CASE(23) SPP_WAIT_CASE(24)
    SPP_WAIT_CASE(25) SPP_WAIT_CASE(26) SPP_WAIT_CASE(27) SPP_WAIT_CASE(28) SPP_WAIT_CASE(29)
    SPP_WAIT_CASE(30) SPP_WAIT_CASE(31)
#undef SPP_WAIT_CASE
    default:
      cp_async_wait<0>();
  }
}

template <int NS, int G>
__global__ void __launch_bounds__(32 * kHdMaxWarps)
k_dedisp_single8_hd(const __grid_constant__ S2Args<NS> a) {
  extern __shared__ __align__(16) uint8_t sm[];
  const int T = 4 * G * (int)(blockDim.x >> 5);
  const int64_t t0 = (int64_t)blockIdx.x * T;
  // channel offsets into shared memory (each lane reads the four of its word);
  // kernel parameters only, so this runs before the wait below
  int32_t* tab = reinterpret_cast<int32_t*>(sm + a.tab_off);
  for (int c = threadIdx.x; c < 32 * a.nslab; c += blockDim.x) tab[c] = a.off[c];
  // Programmatic dependent launch: the previous kernel in the stream may still
  // be finishing (this grid was allowed to launch early); wait until its
  // memory operations are complete and visible before reading the input or
  // writing the output.  Without the launch attribute this returns at once.
  asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    if (s < a.nslab)
      stage_hd(a.raw, a.nchans, a.nsamps, sm + (int64_t)a.srow[s] * kHdPitch, t0 + a.mn[s],
               a.nrows[s], 32 * s);
    cp_async_commit();  // one group per slab (empty past nslab)
  }
  // the next kernel in the stream may start launching (it waits for this
  // grid's completion before touching memory)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = lane & 3, j = lane >> 2;
  const int obase = warp * 4 * G + i;  // this lane's first output row within the CTA
  int32_t acc[G];
#pragma unroll
  for (int g = 0; g < G; ++g) acc[g] = 0;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    cp_async_wait_n(NS - 1 - s);  // groups of slabs > s may still be in flight
    __syncthreads();
    if (s < a.nslab) {
      const int4 o4 = *reinterpret_cast<const int4*>(tab + 32 * s + 4 * j);
      const uint8_t* base = sm + (int64_t)(a.srow[s] + obase) * kHdPitch;
      const uint8_t* p0 = base + o4.x;
      const uint8_t* p1 = base + o4.y;
      const uint8_t* p2 = base + o4.z;
      const uint8_t* p3 = base + o4.w;
      uint32_t v[4][G];  // all 4 G loads of the slab issued before any add
#pragma unroll
      for (int g = 0; g < G; ++g) {
        v[0][g] = p0[g * 4 * kHdPitch];
        v[1][g] = p1[g * 4 * kHdPitch];
        v[2][g] = p2[g * 4 * kHdPitch];
        v[3][g] = p3[g * 4 * kHdPitch];
      }
#pragma unroll
      for (int g = 0; g < G; ++g) acc[g] += (int32_t)(v[0][g] + v[1][g] + v[2][g] + v[3][g]);
    }
  }
  // sum over the 8 channel words (lanes with equal i), then lane (i, j) writes group g = j
#pragma unroll
  for (int g = 0; g < G; ++g) {
    acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 4);
    acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 8);
    acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 16);
  }
  int32_t mine = 0;
#pragma unroll
  for (int g = 0; g < G; ++g)
    if (g == j) mine = acc[g];
  const int64_t tt = t0 + obase + 4 * j;
  if (j < G && tt < a.nvalid) a.out[a.out_start + tt] = (float)mine;
}

template <int NS>
static void (*hd_kernel(int G))(const S2Args<NS>) {
  switch (G) {
    case 1: return k_dedisp_single8_hd<NS, 1>;
    case 2: return k_dedisp_single8_hd<NS, 2>;
    case 3: return k_dedisp_single8_hd<NS, 3>;
    case 4: return k_dedisp_single8_hd<NS, 4>;
    case 5: return k_dedisp_single8_hd<NS, 5>;
    case 6: return k_dedisp_single8_hd<NS, 6>;
    case 7: return k_dedisp_single8_hd<NS, 7>;
    default: return k_dedisp_single8_hd<NS, 8>;
  }
}

template <int NS>
static int launch_hd(const uint8_t* raw, int64_t nchans, int64_t nsamps, const int32_t* d,
                     float* out, int64_t out_start, int64_t nvalid, cudaStream_t st) {
  S2Args<NS> a{};
  const int nslab = (int)(nchans / 32);
  int32_t mn[NS], mx[NS];
  for (int s = 0; s < nslab; ++s) {
    mn[s] = *std::min_element(d + 32 * s, d + 32 * s + 32);
    mx[s] = *std::max_element(d + 32 * s, d + 32 * s + 32);
  }
  // outputs per CTA T = 4 W G: one wave of CTAs covers the block, G up to 4
  // and as many warps W (up to 32) as that takes; shrink W until every slab's
  // rows are resident at once.  Blocks of more than 148 x 1024 outputs run two
  // CTAs per SM (half the shared memory each), so that one CTA's copies
  // overlap the other's adds (measured: 2^20 x 256 ch, 99 -> 90 us; at 65 536
  // samples one CTA per SM is faster).
  const int cps = nvalid > 148 * 1024 ? 2 : 1;
  const int64_t kMaxSmem = cps == 1 ? 227 * 1024 : 112 * 1024;
  const int64_t tab_bytes = 32 * 4 * (int64_t)nslab;
  const int64_t target = ceil_div(nvalid, 148 * cps);
  const int G = (int)std::min<int64_t>(kHdMaxG, std::max<int64_t>(1, ceil_div(target, 4 * kHdMaxWarps)));
  int W = (int)std::min<int64_t>(kHdMaxWarps, std::max<int64_t>(1, ceil_div(target, 4 * G)));
  int64_t rows = 0;
  for (; W >= 1; --W) {
    rows = 0;
    for (int s = 0; s < nslab; ++s) rows += 4 * W * G + (int64_t)(mx[s] - mn[s]);
    if (rows * kHdPitch + tab_bytes <= kMaxSmem) break;
  }
  if (W < 1) return SPP_ERR_UNSUPPORTED;
  const int T = 4 * W * G;
  int64_t r = 0;
  for (int s = 0; s < nslab; ++s) {
    a.mn[s] = mn[s];
    a.nrows[s] = T + (mx[s] - mn[s]);
    a.srow[s] = (int32_t)r;
    r += a.nrows[s];
    for (int c = 0; c < 32; ++c) a.off[32 * s + c] = (d[32 * s + c] - mn[s]) * kHdPitch + c;
  }
  a.raw = raw;
  a.nchans = nchans;
  a.nsamps = nsamps;
  a.out = out;
  a.out_start = out_start;
  a.nvalid = nvalid;
  a.nslab = nslab;
  a.tab_off = (int32_t)(rows * kHdPitch);
  const int64_t smem = rows * kHdPitch + tab_bytes;
  auto fn = hd_kernel<NS>(G);
  int rc = set_smem_attr(reinterpret_cast<const void*>(fn), smem);
  if (rc) return rc;
  const int64_t gx = ceil_div(nvalid, T);
  if (gx > INT32_MAX || nsamps > INT32_MAX) return SPP_ERR_UNSUPPORTED;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)gx);
  cfg.blockDim = dim3(32 * W);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cuda_status(cudaLaunchKernelEx(&cfg, fn, a), "single-DM (host table) launch");
}

// 8-bit, nchans a multiple of 32 up to 1024, delays in host memory; returns
// SPP_ERR_UNSUPPORTED when the shape is outside what the kernel covers.
int launch_single8_hd(const uint8_t* raw, int64_t nchans, int64_t nsamps, const int32_t* delays_host,
                      float* out, int64_t out_start, int64_t nvalid, cudaStream_t st) {
  if (nchans % 32 != 0 || nchans <= 0 || (reinterpret_cast<uintptr_t>(raw) & 15) != 0)
    return SPP_ERR_UNSUPPORTED;
  if (nchans <= 256)
    return launch_hd<8>(raw, nchans, nsamps, delays_host, out, out_start, nvalid, st);
  if (nchans <= 512)
    return launch_hd<16>(raw, nchans, nsamps, delays_host, out, out_start, nvalid, st);
  if (nchans <= 1024)
    return launch_hd<32>(raw, nchans, nsamps, delays_host, out, out_start, nvalid, st);
  return SPP_ERR_UNSUPPORTED;
}


// ---------------------------------------------------------------------------
// Streaming single-DM kernel, every sample width (spp_dedisperse_host): the
// block is read once, straight from its time-major rows, whatever its length,
// channel count and alignment.
//
// CTA = T outputs over all channels, walked in slabs of 32 bytes of each row
// (256 / NB channels; 64 bytes of float32).  Slab s needs rows [t0 + min delay, t0 + T + max delay)
// of its channels; a ring of them is filled ahead of the adds: 16-byte cp.async
// where rows are so aligned (up to six slabs), else aligned words shifted into
// place and stored.  Staged rows are dense 32-byte
// rows: lane (i = lane & 3, j = lane >> 2) reads a byte of word j in row
// t + i + delay, which hits 32 different banks for any delays; 1-, 2- and
// 4-bit fields are masked in place, summed per position within the byte and
// shifted once per word, so a channel costs a byte load and one and a half
// logic operations.  Float32 rows (16 channels, pitch 17 words) give each lane an
// output and are added in channel order in float64.
//
// Bound by the byte loads (32 adds per shared-memory wavefront) next to the row
// copies.  Against the planar path (corner turn, then the DM-time kernel on one
// row): 8-bit 1024 ch x 262144, DM 300: 392 -> 92 us (2.9 TB/s); 2-bit 1024 ch x
// 200000: 138 -> 46 us, 1020 ch (rows at odd addresses): 198 -> 78 us; 1-bit
// 1024 ch x 300000: 140 -> 55 us; float32 256 ch x 100000: 112 -> 53 us.
// ---------------------------------------------------------------------------
constexpr int kSdWarps = 16;
constexpr int kSdThreads = 32 * kSdWarps;
constexpr int kSdSeg = 32;  // bytes of a row per slab (integers)
// float32: 64 bytes (16 channels) at an odd word pitch
__host__ __device__ constexpr int sd_seg(int nb) { return nb == 32 ? 64 : kSdSeg; }
__host__ __device__ constexpr int sd_pitch(int nb) { return nb == 32 ? 68 : kSdSeg; }

template <int MAXC>
struct SdArgs {
  const uint8_t* raw;
  int64_t rowbytes, nsamps;
  float* out;           // output of sample 0
  int64_t nvalid;
  int32_t nslab, T, stages, stage_bytes;
  int32_t bitorder;
  int32_t align;        // of the rows: 16, 4 or 1 bytes
  int32_t mn[MAXC / 8];    // per slab: smallest delay (float32: 16 channels each)
  uint16_t rows[MAXC / 8]; // per slab: rows beyond T
  uint16_t off[MAXC];      // per channel: delay - the slab's smallest
};

// Aligned words of a row segment that starts at any byte: word k of the 32
// bytes from byte `seg` of row `row`, zero past the row's end.  Only words that
// hold a wanted byte are loaded.
__device__ __forceinline__ uint32_t row_word(const uint8_t* raw, int64_t rowbytes, int64_t row,
                                             int64_t seg, int k) {
  const int64_t left = rowbytes - seg - 4 * k;  // bytes of the row from this word on
  if (left <= 0) return 0u;
  const uint8_t* p = raw + row * rowbytes + seg + 4 * k;
  const int sh = (int)(reinterpret_cast<uintptr_t>(p) & 3);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(p - sh);
  const uint32_t lo = __ldg(w);
  const uint32_t hi = (sh && left > 4 - sh) ? __ldg(w + 1) : 0u;
  uint32_t v = __funnelshift_r(lo, hi, 8 * sh);
  if (left < 4) v &= (1u << (8 * left)) - 1u;
  return v;
}

template <int NB, int MAXC>
__device__ __forceinline__ void sd_stage(const SdArgs<MAXC>& a, uint8_t* buf, int64_t t0, int s) {
  const int64_t seg = (int64_t)s * sd_seg(NB);
  const int64_t r0 = t0 + a.mn[s];
  const int nrows = a.T + a.rows[s];
  auto wrap = [&](int64_t row) {  // rows outside the block wrap once or read zero
    if (row < 0) row += a.nsamps;
    else if (row >= a.nsamps) row -= a.nsamps;
    return (row >= 0 && row < a.nsamps) ? row : (int64_t)-1;
  };
  if (NB == 32) {
    // float rows keep an odd pitch for the adds, so they pass through registers:
    // 16-byte loads where rows allow, four in flight
    constexpr int PW = sd_pitch(NB) / 4;
    float* dst = reinterpret_cast<float*>(buf);
    if (a.align == 16) {
      constexpr int Q = sd_seg(NB) / 16;  // loads per row
      const int h = threadIdx.x % Q;
      const bool col = seg + 16 * h < a.rowbytes;
      for (int r = threadIdx.x / Q; r < nrows; r += 4 * (kSdThreads / Q)) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int rr = r + u * (kSdThreads / Q);
          const int64_t row = col && rr < nrows ? wrap(r0 + rr) : -1;
          v[u] = row >= 0 ? __ldg(reinterpret_cast<const float4*>(a.raw + row * a.rowbytes + seg) + h)
                          : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int rr = r + u * (kSdThreads / Q);
          if (rr >= nrows) break;
          float* q = dst + rr * PW + 4 * h;
          q[0] = v[u].x; q[1] = v[u].y; q[2] = v[u].z; q[3] = v[u].w;
        }
      }
    } else {
      constexpr int Q = sd_seg(NB) / 4;
      const int k = threadIdx.x % Q;
      const bool col = seg + 4 * k < a.rowbytes;
      for (int r = threadIdx.x / Q; r < nrows; r += 4 * (kSdThreads / Q)) {
        float v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int rr = r + u * (kSdThreads / Q);
          const int64_t row = col && rr < nrows ? wrap(r0 + rr) : -1;
          v[u] = row >= 0 ? __ldg(reinterpret_cast<const float*>(a.raw + row * a.rowbytes + seg) + k) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int rr = r + u * (kSdThreads / Q);
          if (rr < nrows) dst[rr * PW + k] = v[u];
        }
      }
    }
  } else if (a.align == 16) {
    const int h = threadIdx.x & 1;
    const bool col = seg + 16 * h < a.rowbytes;
    for (int r = threadIdx.x >> 1; r < nrows; r += kSdThreads / 2) {
      const int64_t row = col ? wrap(r0 + r) : -1;
      cp_async16(buf + r * kSdSeg + 16 * h, row >= 0 ? a.raw + row * a.rowbytes + seg + 16 * h : a.raw,
                 row >= 0);
    }
  } else {
    const int k = threadIdx.x & 7;
    const int left = (int)min(a.rowbytes - seg - 4 * k, (int64_t)4);  // bytes wanted of this word
    if (r0 >= 0 && r0 + nrows <= a.nsamps) {
      // whole rows of the block: the aligned words of four rows in flight
      const uint32_t keep = left >= 4 ? 0xFFFFFFFFu : left > 0 ? (1u << (8 * left)) - 1u : 0u;
      const uint8_t* p = a.raw + (r0 + (threadIdx.x >> 3)) * a.rowbytes + seg + 4 * k;
      const int64_t step = (int64_t)(kSdThreads / 8) * a.rowbytes;
      for (int r = threadIdx.x >> 3; r < nrows; r += kSdThreads / 2) {
        uint32_t lo[4], hi[4], sh[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          sh[u] = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3);
          const uint32_t* w = reinterpret_cast<const uint32_t*>(p - sh[u]);
          const bool on = left > 0 && r + u * (kSdThreads / 8) < nrows;
          lo[u] = on ? __ldg(w) : 0u;
          hi[u] = on && left + (int)sh[u] > 4 ? __ldg(w + 1) : 0u;
          p += step;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int row = r + u * (kSdThreads / 8);
          if (row < nrows)
            *reinterpret_cast<uint32_t*>(buf + row * kSdSeg + 4 * k) = __funnelshift_r(lo[u], hi[u], 8 * sh[u]) & keep;
        }
      }
    } else {
      for (int r = threadIdx.x >> 3; r < nrows; r += kSdThreads / 8) {
        const int64_t row = wrap(r0 + r);
        *reinterpret_cast<uint32_t*>(buf + r * kSdSeg + 4 * k) =
            row >= 0 ? row_word(a.raw, a.rowbytes, row, seg, k) : 0u;
      }
    }
  }
}

template <int NB, int G, int MAXC>
__global__ void __launch_bounds__(kSdThreads, 2)
k_dedisp_stream(const __grid_constant__ SdArgs<MAXC> a) {
  extern __shared__ __align__(16) uint8_t sm[];
  constexpr int CH = 8 * sd_seg(NB) / NB;  // channels per slab
  const int64_t t0 = (int64_t)blockIdx.x * a.T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // byte offset of every channel's first row and byte (float32: of its word)
  int32_t* tab = reinterpret_cast<int32_t*>(sm + (int64_t)a.stages * a.stage_bytes);
  for (int c = threadIdx.x; c < a.nslab * CH; c += kSdThreads)
    tab[c] = NB == 32 ? a.off[c] * sd_pitch(NB) + 4 * (c % CH) : a.off[c] * kSdSeg + (c % CH) * NB / 8;
  const int ahead = a.stages - 1;
  for (int s = 0; s < ahead; ++s) {
    if (s < a.nslab) sd_stage<NB, MAXC>(a, sm + (int64_t)s * a.stage_bytes, t0, s);
    cp_async_commit();
  }
  const int i = lane & 3, j = lane >> 2;
  const int obase = NB == 32 ? warp * 32 * G + lane : warp * 4 * G + i;  // first output row
  int32_t acc[G];
  double dacc[G];
#pragma unroll
  for (int g = 0; g < G; ++g) { acc[g] = 0; dacc[g] = 0.0; }
  int buf = 0, fill = ahead;
  for (int s = 0; s < a.nslab; ++s) {
    cp_async_wait_n(ahead - 1);  // slab s has landed
    __syncthreads();
    if (s + ahead < a.nslab) sd_stage<NB, MAXC>(a, sm + (int64_t)fill * a.stage_bytes, t0, s + ahead);
    cp_async_commit();
    const uint8_t* base = sm + (int64_t)buf * a.stage_bytes;
    if (++buf == a.stages) buf = 0;
    if (++fill == a.stages) fill = 0;
    if constexpr (NB == 32) {
      const uint8_t* p = base + obase * sd_pitch(NB);
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const uint8_t* q = p + tab[s * CH + c];
#pragma unroll
        for (int g = 0; g < G; ++g)
          dacc[g] += (double)*reinterpret_cast<const float*>(q + g * 32 * sd_pitch(NB));
      }
    } else {
      constexpr int CPW = 32 / NB;             // channels per 4-byte word
      constexpr int KG = CPW < 16 ? CPW : 16;  // taken at a time
      constexpr int PB = 8 / NB;               // channels per byte
      uint32_t mask[PB], sh[PB];
#pragma unroll
      for (int p = 0; p < PB; ++p) {
        sh[p] = (a.bitorder == SPP_BITORDER_BIG) ? 8 - (p + 1) * NB : p * NB;
        mask[p] = ((1u << NB) - 1u) << sh[p];
      }
      const uint8_t* p0 = base + obase * kSdSeg;
#pragma unroll
      for (int kg = 0; kg < CPW; kg += KG) {
        const uint8_t* q[KG];
#pragma unroll
        for (int k = 0; k < KG; k += 4) {
          const int4 o = *reinterpret_cast<const int4*>(tab + s * CH + j * CPW + kg + k);
          q[k] = p0 + o.x;
          q[k + 1] = p0 + o.y;
          q[k + 2] = p0 + o.z;
          q[k + 3] = p0 + o.w;
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
          uint32_t part[PB];
#pragma unroll
          for (int p = 0; p < PB; ++p) part[p] = 0u;
#pragma unroll
          for (int k = 0; k < KG; ++k) {
            const uint32_t b = q[k][g * 4 * kSdSeg];
            part[k % PB] += NB == 8 ? b : b & mask[k % PB];
          }
#pragma unroll
          for (int p = 0; p < PB; ++p) acc[g] += (int32_t)(NB == 8 ? part[p] : part[p] >> sh[p]);
        }
      }
    }
  }
  if constexpr (NB == 32) {
#pragma unroll
    for (int g = 0; g < G; ++g) {
      const int64_t t = t0 + obase + 32 * g;
      if (t < a.nvalid) a.out[t] = (float)dacc[g];
    }
  } else {
    // sum over the eight words (lanes with equal i); lane (i, j) writes groups j, j + 8
#pragma unroll
    for (int g = 0; g < G; ++g) {
      acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 4);
      acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 8);
      acc[g] += __shfl_xor_sync(0xffffffffu, acc[g], 16);
      const int64_t t = t0 + obase + 4 * g;
      if ((g & 7) == j && t < a.nvalid) a.out[t] = (float)acc[g];
    }
  }
}

template <int NB, int MAXC>
static void (*sd_kernel(int G))(const SdArgs<MAXC>) {
  if (NB == 32) return G <= 1 ? k_dedisp_stream<NB, 1, MAXC> : G <= 2 ? k_dedisp_stream<NB, 2, MAXC> : k_dedisp_stream<NB, 4, MAXC>;
  return G <= 2 ? k_dedisp_stream<NB, 2, MAXC> : G <= 4 ? k_dedisp_stream<NB, 4, MAXC>
         : G <= 8 ? k_dedisp_stream<NB, 8, MAXC> : G <= 12 ? k_dedisp_stream<NB, 12, MAXC>
                                                           : k_dedisp_stream<NB, 16, MAXC>;
}

template <int NB, int MAXC>
static int launch_stream(const uint8_t* raw, int bitorder, int64_t nchans, int64_t nsamps,
                         const int32_t* d, float* out, int64_t nvalid, double limit_us,
                         cudaStream_t st) {
  constexpr int CH = 8 * sd_seg(NB) / NB;
  constexpr int pitch = sd_pitch(NB);
  constexpr int unit = NB == 32 ? 32 * kSdWarps : 4 * kSdWarps;  // outputs per G
  static const int kG[] = {1, 2, 4, 8, 12, 16};
  SdArgs<MAXC> a{};
  a.nslab = (int32_t)ceil_div(nchans, CH);
  int32_t spread = 0;
  for (int s = 0; s < a.nslab; ++s) {
    const int64_t c0 = (int64_t)s * CH, c1 = std::min<int64_t>(nchans, c0 + CH);
    const int32_t mn = *std::min_element(d + c0, d + c1), mx = *std::max_element(d + c0, d + c1);
    if ((int64_t)mx - mn > 60000) return SPP_ERR_UNSUPPORTED;
    spread = std::max(spread, mx - mn);
    a.mn[s] = mn;
    a.rows[s] = (uint16_t)(mx - mn);
    // channels past the last read zeros: offset 0 of a zero-filled byte
    for (int64_t c = c0; c < c1; ++c) a.off[c] = (uint16_t)(d[c] - mn);
  }
  // outputs per CTA: two CTAs per SM where they fit, and the least estimated
  // time: waves x slabs x the longer of a slab's rows (2.7 ns each at two CTAs
  // per SM) and a copy's latency (1.5 us) over the slabs in flight, or both in
  // part where the copies go through registers
  const int64_t tab = (int64_t)a.nslab * CH * 4;
  a.rowbytes = NB == 32 ? nchans * 4 : nchans * NB / 8;
  const uintptr_t both = (uintptr_t)a.rowbytes | reinterpret_cast<uintptr_t>(raw);
  a.align = both % 16 == 0 ? 16 : both % 4 == 0 ? 4 : 1;
  const bool async = NB != 32 && a.align == 16;
  int G = 0;
  int64_t smem = 0;
  for (int cps = 2; cps >= 1 && G == 0; --cps) {
    const int64_t room = (cps == 2 ? 113 : 226) * 1024 - tab;
    double best = 0.0;
    for (int g : kG) {
      if (NB == 32 ? g > 4 : g < 2) continue;
      const int64_t T = (int64_t)unit * g;
      const int64_t stage = round_up((T + spread) * pitch, 16);
      if (2 * stage > room) break;
      const int64_t stages = std::min<int64_t>(async ? 6 : 2, room / stage);
      const double rows_us = 2.7e-3 * (double)(T + spread);
      const double slab_us = async ? std::max(rows_us, 1.5 / (double)(stages - 1)) : rows_us + 0.7;
      const double t = (double)ceil_div(ceil_div(nvalid, T), 148 * cps) * slab_us;
      if (G == 0 || t < best) {
        best = t;
        G = g;
        a.T = (int32_t)T;
        a.stage_bytes = (int32_t)stage;
        a.stages = (int32_t)stages;
        smem = stages * stage + tab;
      }
    }
  }
  if (G == 0) return SPP_ERR_UNSUPPORTED;
  // Estimated time: a launch, then slab after slab: a fixed part, its rows (a part
  // alone, a part shared with the other CTAs in flight) and its adds; where copies
  // go through registers nothing hides the first slab's.  Fitted to 850 blocks of
  // 16-4096 channels, 500-300000 outputs, cold caches: mostly within 20 %.
  const int64_t ctas = ceil_div(nvalid, a.T), full = 148 * (smem > 113 * 1024 ? 1 : 2);
  const double conc = std::max((double)std::min(ctas, full) / 148.0, 0.25);
  const double rows = 1e-3 * (double)(a.T + spread), add = G * std::max(conc, 1.0);
  const double slab = async       ? 0.30 + (0.38 + 0.11 * conc) * rows + 0.10 * add
                      : NB != 32  ? 0.87 + (0.87 + 0.42 * conc) * rows + 0.25 * add
                      : a.align == 16 ? 1.45 + (1.32 + 0.63 * conc) * rows
                                      : (2.93 + 0.41 * conc) * rows + 2.53 * add;
  const double first = async || (NB == 32 && a.align == 16) ? 0.0 : 3.2 * rows;
  if (6.0 + first + (double)ceil_div(ctas, full) * a.nslab * slab > limit_us) return SPP_ERR_UNSUPPORTED;
  a.raw = raw;
  a.nsamps = nsamps;
  a.out = out;
  a.nvalid = nvalid;
  a.bitorder = bitorder;
  const int64_t gx = ceil_div(nvalid, a.T);
  if (gx > INT32_MAX) return SPP_ERR_UNSUPPORTED;
  auto fn = sd_kernel<NB, MAXC>(G);
  int rc = set_smem_attr(reinterpret_cast<const void*>(fn), smem);
  if (rc) return rc;
  fn<<<(unsigned)gx, kSdThreads, smem, st>>>(a);
  return cuda_status(cudaGetLastError(), "single-DM stream launch");
}

// Any width, up to 4096 channels, delays in host memory; SPP_ERR_UNSUPPORTED
// (nothing launched) outside that, where a slab's delay spread does not fit, or
// where the estimated time is above `limit_us`.
int launch_single_stream(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                         const int32_t* delays_host, float* out, int64_t nvalid, double limit_us,
                         cudaStream_t st) {
  if (nchans > 4096 || (nbits == 32 && (reinterpret_cast<uintptr_t>(in) & 3) != 0))
    return SPP_ERR_UNSUPPORTED;
  const uint8_t* raw = static_cast<const uint8_t*>(in);
#define SPP_SD(NB)                                                                              \
  case NB:                                                                                      \
    return nchans <= 1024                                                                       \
               ? launch_stream<NB, 1024>(raw, bitorder, nchans, nsamps, delays_host, out, nvalid, limit_us, st) \
               : launch_stream<NB, 4096>(raw, bitorder, nchans, nsamps, delays_host, out, nvalid, limit_us, st)
  switch (nbits) {
    SPP_SD(1);
    SPP_SD(2);
    SPP_SD(4);
    SPP_SD(8);
    SPP_SD(32);
    default: return SPP_ERR_UNSUPPORTED;
  }
#undef SPP_SD
}

}  // namespace spp
