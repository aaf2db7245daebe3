// libsppgpu core: error state, unpack (R4), single-DM dedispersion (R2) and
// the DM-trial batch plan (R3).  Host code for the kernels in spp_dmt.cuh.
#include <algorithm>
#include <cmath>
#include <atomic>
#include <climits>
#include <cstring>
#include <limits>
#include <mutex>
#include <new>
#include <tuple>
#include <vector>

#include "spp_common.cuh"
#include "spp_dmt.cuh"
#include "spp_ilv.h"

namespace spp {

int launch_single8(const uint8_t* raw, int64_t nchans, int64_t nsamps, const int32_t* delays,
                   int32_t dlo, int32_t dhi, float* out, int64_t out_start, int64_t nvalid,
                   uint32_t* status, cudaStream_t st);
int launch_single8_hd(const uint8_t* raw, int64_t nchans, int64_t nsamps, const int32_t* delays_host,
                      float* out, int64_t out_start, int64_t nvalid, cudaStream_t st);
int launch_single_stream(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                         const int32_t* delays_host, float* out, int64_t nvalid, double limit_us,
                         cudaStream_t st);

static thread_local char g_err[1024] = "";

int fail(int code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

int cuda_status(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return SPP_OK;
  return fail(SPP_ERR_CUDA, "%s: %s (%s)", what, cudaGetErrorString(e), cudaGetErrorName(e));
}

static inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Raises a kernel's dynamic shared memory limit once per (device, kernel):
// later calls with a size at or below the recorded one issue no CUDA call, so
// launches stay legal inside CUDA-graph capture after one eager run.
int set_smem_attr(const void* fn, int64_t bytes) {
  static std::mutex mu;
  static std::vector<std::tuple<int, const void*, int64_t>> done;
  int dev = 0;
  int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(mu);
  for (auto& e : done)
    if (std::get<0>(e) == dev && std::get<1>(e) == fn && std::get<2>(e) >= bytes) return SPP_OK;
  rc = cuda_status(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes),
                   "cudaFuncSetAttribute");
  if (rc) return rc;
  done.emplace_back(dev, fn, bytes);
  return SPP_OK;
}

static inline bool valid_nbits(int nbits) {
  return nbits == 1 || nbits == 2 || nbits == 4 || nbits == 8 || nbits == 32;
}

// ---------------------------------------------------------------------------
// R4: standalone unpack (kernels.unpack{1,2,4}_8_{big,little})
// ---------------------------------------------------------------------------
template <int NB>
__global__ void k_unpack(const uint8_t* __restrict__ in, int64_t nbytes, int bitorder,
                         uint8_t* __restrict__ out) {
  constexpr int per = 8 / NB;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nbytes;
       i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t b = in[i];
#pragma unroll
    for (int k = 0; k < per; ++k) out[i * per + k] = (uint8_t)field_of<NB>(b, k, bitorder);
  }
}

// ---------------------------------------------------------------------------
// DMT kernel variants
// ---------------------------------------------------------------------------
// Estimated time (us) of a CTA's walk over the channels: alone, and per tile of those
// an SM runs beside one another.
struct WalkTime {
  double walk0, walk, tile, few;
};

struct Variant {
  int nb, acc, R, DW, TW, SLAB, STAGES;
  void (*fn)(const DmtArgs);
  int single;  // 1: meant for one DM (time-split warps)
  int planes;  // 1: bit-sliced kernel over bit-plane rows (R = words per thread)
  int slot;    // > 0: kernel compiled for exactly this slot width (words)
  WalkTime time = {};  // float64 sums
};

template <int NB, int R, int DW, int TW, int SLAB, int STAGES, int ACC>
static Variant mk(int single, WalkTime time = {}) {
  return Variant{NB, ACC, R, DW, TW, SLAB, STAGES, &k_dmt<NB, R, DW, TW, SLAB, STAGES, ACC>,
                 single, 0, 0, time};
}

// Bit-sliced counters hold sums below 2^bit_levels(nbits).
static int bit_levels(int nbits) {
  return nbits == 8 ? BitsLevels<8>::kLevels : nbits == 4 ? BitsLevels<4>::kLevels : BitsLevels<2>::kLevels;
}

template <int NB, int P, int DW, int TW, int STAGES, int SLAB = 64, int SLOT = 0, int MINB = 0>
static Variant mkb() {
  constexpr int L = BitsLevels<NB>::kLevels;
  void (*fn)(const DmtArgs) = &k_dmt_bits<NB, P, DW, TW, STAGES, L, SLAB, SLOT>;
  if constexpr (MINB > 0) fn = &k_dmt_bits_minb<NB, P, DW, TW, STAGES, L, SLAB, SLOT, MINB>;
  return Variant{NB, 0, P, DW, TW, SLAB, STAGES, fn, 0, 1, SLOT};
}

#define SPP_INT_VARIANTS(NB)                    \
  mk<NB, 2, 8, 1, 64, 3, 0>(0), mk<NB, 1, 8, 1, 64, 3, 0>(0), mk<NB, 2, 4, 2, 64, 3, 0>(0), \
      mk<NB, 2, 1, 4, 64, 3, 0>(1), mk<NB, 1, 1, 4, 64, 3, 0>(1)

static const std::vector<Variant>& variants() {
  static const std::vector<Variant> v = {
      // bit-sliced, 32 consecutive samples per word: blocks or tables that the
      // interleaved layout (spp_ilv.cu) does not take, fixed slot widths first
      mkb<2, 2, 8, 1, 2, 32, 80, 4>(), mkb<2, 2, 8, 1, 2, 32, 128>(), mkb<2, 2, 8, 1, 2, 32>(),
      mkb<2, 4, 8, 1, 2, 32>(),
      mkb<1, 2, 8, 1, 2, 32, 80>(), mkb<1, 2, 8, 1, 2, 32, 128>(), mkb<1, 2, 8, 1, 3, 32>(),
      // widest spreads of 1-bit rows (8 trials: up to 24000 samples, 14000 above)
      mkb<1, 4, 8, 1, 2, 32>(),
      SPP_INT_VARIANTS(1),
      SPP_INT_VARIANTS(2),
      // four plane rows per channel; 16-channel slabs keep a stage's planes
      // within a third of shared memory
      mkb<4, 2, 8, 1, 2, 16, 96, 3>(), mkb<4, 2, 8, 1, 2, 16>(),
      SPP_INT_VARIANTS(4),
      // byte lanes, eight words per thread: 1.2e13 channel-adds/s, also on wide
      // spreads; then eight plane rows per channel (1.0e13) for the widest
      mk<8, 8, 8, 1, 32, 2, 0>(0),
      mkb<8, 2, 8, 1, 2, 16, 96, 2>(), mkb<8, 2, 8, 1, 2, 16, 0, 2>(), mkb<8, 1, 8, 1, 2, 16>(),
      SPP_INT_VARIANTS(8),
      mk<8, 4, 1, 4, 16, 3, 0>(1),
      // float32 input, compensated fp32
      mk<32, 8, 8, 1, 32, 2, SPP_ACC_KAHAN32>(0),
      mk<32, 4, 8, 2, 32, 2, SPP_ACC_KAHAN32>(0),
      mk<32, 8, 16, 1, 32, 2, SPP_ACC_KAHAN32>(0),
      mk<32, 8, 4, 1, 16, 2, SPP_ACC_KAHAN32>(0),
      mk<32, 4, 1, 4, 32, 2, SPP_ACC_KAHAN32>(1),
      mk<32, 2, 1, 4, 32, 2, SPP_ACC_KAHAN32>(1),
      mk<32, 16, 4, 1, 16, 2, SPP_ACC_KAHAN32>(0),
      mk<32, 8, 2, 1, 16, 2, SPP_ACC_KAHAN32>(0),
      mk<32, 16, 2, 1, 16, 2, SPP_ACC_KAHAN32>(0),
      // float32 input, fp64 accumulator (channel-ordered sums: the reference's).
      // With the SMs full, 8 words x 8 trials x 2 warps were the fastest (1024
      // channels, 256 trials to DM 500, 57444 outputs: 2.98 ms; 16 words x 4 trials,
      // the choice before, 4.14 ms: three CTAs of four warps per SM leave the adders
      // waiting on slab hand-overs).  16 words per thread leave few registers for
      // loads in flight: 8 trials x 2 warps of them took 2.9 to 4.1 ms from one
      // compilation to the next and are not used.  Wide delay spreads fit only the
      // small tiles.  The arguments are fitted beside float64_us.
      mk<32, 8, 8, 2, 16, 2, SPP_ACC_F64>(0, {15.8, 0.147, 0.127, 1.9}),
      mk<32, 16, 5, 3, 16, 2, SPP_ACC_F64>(0, {17.8, 0.144, 0.213, 13.1}),
      mk<32, 8, 4, 1, 16, 2, SPP_ACC_F64>(0, {15.6, 0.0924, 0.0322, 1.28}),
      mk<32, 8, 4, 2, 16, 2, SPP_ACC_F64>(0, {15.5, 0.0968, 0.0624, 1.71}),
      mk<32, 16, 4, 1, 16, 2, SPP_ACC_F64>(0, {15.3, 0.111, 0.0589, 0.578}),
      mk<32, 16, 2, 1, 16, 2, SPP_ACC_F64>(0, {15.3, 0.123, 0.0289, 0.799}),
      mk<32, 8, 2, 1, 16, 2, SPP_ACC_F64>(0, {16.2, 0.0732, 0.0192, 0.785}),
      mk<32, 4, 1, 4, 32, 2, SPP_ACC_F64>(1),
      mk<32, 2, 1, 4, 32, 2, SPP_ACC_F64>(1),
  };
  return v;
}

static inline int spw_of(int nb) { return nb == 32 ? 1 : 32 / nb; }
static inline int spw_v(const Variant& v) { return v.planes ? 32 : spw_of(v.nb); }
static inline int64_t tile_T(const Variant& v) {
  return (int64_t)v.TW * 32 * v.R * spw_v(v);
}

static int slot_words(const Variant& v, int32_t span) {
  const int spw = spw_v(v);
  const int64_t w = tile_T(v) / spw + ceil_div(std::max<int32_t>(span, 0), spw) + 6 + v.R;
  const int need = (int)round_up(w, 4);
  if (v.slot > 0) return need <= v.slot ? v.slot : -1;  // fixed-width kernels
  return need;
}

static int64_t smem_bytes(const Variant& v, int slot_w) {
  if (v.planes) return v.STAGES * bits_stage_bytes(v.nb, v.SLAB, slot_w, v.DW) + 8 + 2 * v.STAGES * 8;
  return v.STAGES * dmt_stage_bytes(v.SLAB, slot_w, v.DW) + 8 + 2 * v.STAGES * 8;
}

static constexpr int64_t kMaxSmem = 227 * 1024;

// Planar geometry for one execution.
struct Geometry {
  int planes;
  int spw;
  int64_t halo;     // samples
  int64_t pitch_w;  // words per channel row
  int64_t bytes;    // nchans * pitch_w * 4
  int64_t ntiles_t;
  int64_t nvalid;
};

// omin/omax: range of the signed offsets applied to t (sign * delay).
static Geometry geometry(const Variant& v, int64_t nchans, int64_t nsamps, int64_t nvalid,
                         int32_t omin, int32_t omax, int slot_w) {
  Geometry g{};
  g.planes = v.planes;
  g.spw = spw_v(v);
  g.nvalid = nvalid;
  g.halo = round_up(std::max<int64_t>(0, -(int64_t)omin), 4 * g.spw);
  g.ntiles_t = ceil_div(std::max<int64_t>(nvalid, 1), tile_T(v));
  const int64_t last = g.ntiles_t * tile_T(v) + std::max<int64_t>(0, omax) + g.halo;
  g.pitch_w = round_up(ceil_div(last, g.spw) + slot_w + 8, 4);
  g.bytes = nchans * (v.planes ? v.nb : 1) * g.pitch_w * 4;
  (void)nsamps;
  return g;
}

static int ensure_smem(const Variant& v, int64_t bytes) {
  if (bytes > kMaxSmem)
    return fail(SPP_ERR_UNSUPPORTED, "DM tile needs %lld B of shared memory (> %lld)",
                (long long)bytes, (long long)kMaxSmem);
  if (bytes > 48 * 1024) return set_smem_attr(reinterpret_cast<const void*>(v.fn), bytes);
  return SPP_OK;
}

static int launch_corner_turn(int nb, const void* in, int bitorder, int64_t nchans,
                              int64_t nsamps, const Geometry& g, void* planar, cudaStream_t st,
                              const double* zdm = nullptr, const float* chanwts = nullptr,
                              const float* bpass = nullptr, uint32_t* special = nullptr) {
  if (g.planes) {
    dim3 grid((unsigned)ceil_div(nchans, planes_ct_chans(nb)),
              (unsigned)std::min<int64_t>(ceil_div(g.pitch_w, kPlaneWords), 65535));
    const uint8_t* raw = static_cast<const uint8_t*>(in);
    uint32_t* pl = static_cast<uint32_t*>(planar);
    if (nb == 1)
      k_corner_turn_planes<1><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w);
    else if (nb == 2)
      k_corner_turn_planes<2><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w);
    else if (nb == 4)
      k_corner_turn_planes<4><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w);
    else if (nb == 8)
      k_corner_turn_planes<8><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w);
    else
      return fail(SPP_ERR_UNSUPPORTED, "bit planes for nbits=%d", nb);
  } else if (nb == 32) {
    dim3 grid((unsigned)ceil_div(nchans, 32),
              (unsigned)std::min<int64_t>(ceil_div(g.pitch_w, 32), 65535));
    k_corner_turn_f32<<<grid, 256, 0, st>>>(static_cast<const float*>(in), nchans, nsamps,
                                            g.halo, static_cast<float*>(planar), g.pitch_w,
                                            zdm, chanwts, bpass, special);
  } else {
    dim3 grid((unsigned)ceil_div(nchans, kCtChans),
              (unsigned)std::min<int64_t>(ceil_div(g.pitch_w, kCtWords), 65535));
    const uint8_t* raw = static_cast<const uint8_t*>(in);
    uint32_t* pl = static_cast<uint32_t*>(planar);
    switch (nb) {
      case 1: k_corner_turn_int<1><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w); break;
      case 2: k_corner_turn_int<2><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w); break;
      case 4: k_corner_turn_int<4><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w); break;
      default: k_corner_turn_int<8><<<grid, 256, 0, st>>>(raw, nchans, nsamps, bitorder, g.halo, pl, g.pitch_w); break;
    }
  }
  return cuda_status(cudaGetLastError(), "corner turn launch");
}

static int launch_dmt(const Variant& v, const DmtArgs& a, int64_t ntiles_t, int64_t ndm,
                      cudaStream_t st) {
  const int64_t smem = smem_bytes(v, a.slot_w);
  int rc = ensure_smem(v, smem);
  if (rc) return rc;
  dim3 grid((unsigned)ceil_div(ndm, v.DW), (unsigned)ntiles_t);
  if (ntiles_t > 65535)
    return fail(SPP_ERR_UNSUPPORTED, "too many time tiles (%lld)", (long long)ntiles_t);
  const int threads = (v.DW * v.TW + 1) * 32;
  v.fn<<<grid, threads, smem, st>>>(a);
  return cuda_status(cudaGetLastError(), "dmt launch");
}

// Single-DM shape: the largest time tile that still yields >= 2 CTAs per SM
// (148 SMs), else the smallest tile.  Shapes are the same for both float
// accumulators, so the workspace size does not depend on `acc`.
static int pick_single_variant(int nb, int acc, int64_t nvalid) {
  const auto& vs = variants();
  int best_big = -1, best_small = -1;
  for (int i = 0; i < (int)vs.size(); ++i) {
    const Variant& v = vs[i];
    if (!v.single || v.nb != nb || (nb == 32 && v.acc != acc)) continue;
    if (smem_bytes(v, slot_words(v, 0)) > kMaxSmem) continue;
    const int64_t T = tile_T(v);
    if (ceil_div(nvalid, T) >= 296 && (best_big < 0 || T > tile_T(vs[best_big]))) best_big = i;
    if (best_small < 0 || T < tile_T(vs[best_small])) best_small = i;
  }
  return best_big >= 0 ? best_big : best_small;
}

}  // namespace spp

using namespace spp;

// ---------------------------------------------------------------------------
// extern "C" entry points
// ---------------------------------------------------------------------------
extern "C" {

const char* spp_last_error_string(void) { return g_err; }

int spp_version(void) { return 10000; }

int spp_status_read(const void* workspace, uint32_t* host_out, void* stream) {
  if (!workspace || !host_out) return fail(SPP_ERR_ARG, "spp_status_read: null pointer");
  cudaStream_t st = as_stream(stream);
  int rc = cuda_status(cudaMemcpyAsync(host_out, workspace, 16, cudaMemcpyDeviceToHost, st),
                       "status copy");
  if (rc) return rc;
  rc = cuda_status(cudaStreamSynchronize(st), "status sync");
  if (rc) return rc;
  if (host_out[0] != 0)
    return fail(SPP_ERR_DEVICE, "device status 0x%x (block %u, detail 0x%x)", host_out[0],
                host_out[1], host_out[2]);
  return SPP_OK;
}

int spp_status_clear(void* workspace, void* stream) {
  if (!workspace) return fail(SPP_ERR_ARG, "spp_status_clear: null pointer");
  return cuda_status(cudaMemsetAsync(workspace, 0, 16, as_stream(stream)), "status clear");
}

int spp_host_register(void* ptr, int64_t bytes) {
  if (!ptr || bytes <= 0) return fail(SPP_ERR_ARG, "spp_host_register: null pointer or size <= 0");
  const cudaError_t e = cudaHostRegister(ptr, (size_t)bytes, cudaHostRegisterPortable);
  if (e != cudaSuccess) {
    cudaGetLastError();  // a refused registration must not surface at the next launch check
    return fail(SPP_ERR_CUDA, "cudaHostRegister: %s", cudaGetErrorString(e));
  }
  return SPP_OK;
}

int spp_host_unregister(void* ptr) {
  if (!ptr) return fail(SPP_ERR_ARG, "spp_host_unregister: null pointer");
  const cudaError_t e = cudaHostUnregister(ptr);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(SPP_ERR_CUDA, "cudaHostUnregister: %s", cudaGetErrorString(e));
  }
  return SPP_OK;
}

int spp_unpack(const uint8_t* in, int64_t nbytes, int nbits, int bitorder, uint8_t* out,
               void* stream) {
  if (nbytes < 0) return fail(SPP_ERR_ARG, "nbytes < 0");
  if (nbytes == 0) return SPP_OK;
  if (!in || !out) return fail(SPP_ERR_ARG, "spp_unpack: null pointer");
  if (bitorder != SPP_BITORDER_BIG && bitorder != SPP_BITORDER_LITTLE)
    return fail(SPP_ERR_ARG, "bad bitorder %d", bitorder);
  cudaStream_t st = as_stream(stream);
  const int threads = 256;
  const int64_t blocks = std::min<int64_t>(ceil_div(nbytes, threads), 148 * 32);
  switch (nbits) {
    case 1: k_unpack<1><<<(unsigned)blocks, threads, 0, st>>>(in, nbytes, bitorder, out); break;
    case 2: k_unpack<2><<<(unsigned)blocks, threads, 0, st>>>(in, nbytes, bitorder, out); break;
    case 4: k_unpack<4><<<(unsigned)blocks, threads, 0, st>>>(in, nbytes, bitorder, out); break;
    default: return fail(SPP_ERR_ARG, "unpack: nbits must be 1, 2 or 4 (got %d)", nbits);
  }
  return cuda_status(cudaGetLastError(), "unpack launch");
}

// ---------------------------------------------------------------------------
// R2: single DM
// ---------------------------------------------------------------------------
static int single_setup(int nbits, int64_t nchans, int64_t nsamps, int32_t dmin, int32_t dmax,
                        int acc, const Variant** vout, Geometry* gout, int* slot_out) {
  if (!valid_nbits(nbits)) return fail(SPP_ERR_ARG, "nbits must be 1, 2, 4, 8 or 32 (got %d)", nbits);
  if (nchans <= 0 || nsamps < 0) return fail(SPP_ERR_ARG, "bad shape nchans=%lld nsamps=%lld", (long long)nchans, (long long)nsamps);
  if (nbits < 8 && (nchans * nbits) % 8 != 0)
    return fail(SPP_ERR_ARG, "nchans*nbits must be a multiple of 8");
  if (dmin > dmax) return fail(SPP_ERR_ARG, "delay_min > delay_max");
  if (nchans > INT32_MAX) return fail(SPP_ERR_ARG, "nchans too large");
  const int64_t maxabs = std::max<int64_t>(std::llabs(dmin), std::llabs(dmax));
  const int64_t nvalid = nsamps - maxabs;
  const int vi = pick_single_variant(nbits, acc, std::max<int64_t>(nvalid, 1));
  if (vi < 0) return fail(SPP_ERR_UNSUPPORTED, "no kernel for nbits=%d acc=%d", nbits, acc);
  const Variant& v = variants()[vi];
  const int slot = slot_words(v, 0);
  *vout = &v;
  *slot_out = slot;
  *gout = geometry(v, nchans, nsamps, nvalid, dmin, dmax, slot);
  return SPP_OK;
}

int64_t spp_dedisperse_workspace_bytes(int nbits, int64_t nchans, int64_t nsamps,
                                       int32_t delay_min, int32_t delay_max) {
  const Variant* v;
  Geometry g;
  int slot;
  if (single_setup(nbits, nchans, nsamps, delay_min, delay_max, SPP_ACC_F64, &v, &g, &slot))
    return -1;
  return kStatusBytes + g.bytes;
}

int spp_dedisperse(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                   const int32_t* delays, int32_t delay_min, int32_t delay_max, float* out,
                   int64_t out_len, int64_t out_start, int acc, void* workspace,
                   int64_t workspace_bytes, void* stream) {
  if (!in || !delays || !out || !workspace) return fail(SPP_ERR_ARG, "spp_dedisperse: null pointer");
  if (acc != SPP_ACC_F64 && acc != SPP_ACC_KAHAN32) return fail(SPP_ERR_ARG, "bad acc %d", acc);
  const Variant* v;
  Geometry g;
  int slot;
  int rc = single_setup(nbits, nchans, nsamps, delay_min, delay_max, acc, &v, &g, &slot);
  if (rc) return rc;
  if (g.nvalid <= 0) return SPP_OK;  // reference: prange over a non-positive count
  if (-(int64_t)delay_min > nsamps)
    return fail(SPP_ERR_DELAY, "negative delay %d reaches before the block", delay_min);
  if (out_start < 0 || out_start + g.nvalid > out_len)
    return fail(SPP_ERR_SIZE, "output too small: out_start %lld + %lld samples > out_len %lld",
                (long long)out_start, (long long)g.nvalid, (long long)out_len);
  if (workspace_bytes < kStatusBytes + g.bytes)
    return fail(SPP_ERR_SIZE, "workspace %lld B < required %lld B", (long long)workspace_bytes,
                (long long)(kStatusBytes + g.bytes));
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0)
    return fail(SPP_ERR_ALIGN, "workspace must be 256-B aligned");
  cudaStream_t st = as_stream(stream);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  if (nbits == 8) {
    // one pass over the raw block when the delay spread fits the staging buffer
    rc = launch_single8(static_cast<const uint8_t*>(in), nchans, nsamps, delays, delay_min,
                        delay_max, out, out_start, g.nvalid, reinterpret_cast<uint32_t*>(ws), st);
    if (rc != SPP_ERR_UNSUPPORTED) return rc;
  }
  void* planar = ws + kStatusBytes;
  rc = launch_corner_turn(nbits, in, bitorder, nchans, nsamps, g, planar, st);
  if (rc) return rc;
  DmtArgs a{};
  a.planar = planar;
  a.pitch_w = g.pitch_w;
  a.halo = g.halo;
  a.nchans = (int32_t)nchans;
  a.delays = delays;
  a.dpitch = nchans;
  a.ndm = 1;
  a.sign = 1;
  a.dlo = delay_min;
  a.dhi = delay_max;
  a.span_max = 0;
  a.slot_w = slot;
  a.out = out;
  a.out_kind = SPP_OUT_F32;
  a.out_stride = 0;
  a.out_start = out_start;
  a.nvalid = g.nvalid;
  a.status = reinterpret_cast<uint32_t*>(ws);
  return launch_dmt(*v, a, g.ntiles_t, 1, st);
}

int spp_dedisperse_hd(const void* in, int nbits, int64_t nchans, int64_t nsamps,
                      const int32_t* delays_host, float* out, int64_t out_len, int64_t out_start,
                      void* stream) {
  if (!in || !delays_host || !out) return fail(SPP_ERR_ARG, "spp_dedisperse_hd: null pointer");
  if (nbits != 8) return fail(SPP_ERR_UNSUPPORTED, "host-table path covers 8-bit data");
  if (nchans <= 0 || nsamps <= 0) return fail(SPP_ERR_ARG, "bad shape");
  const int32_t dmin = *std::min_element(delays_host, delays_host + nchans);
  const int32_t dmax = *std::max_element(delays_host, delays_host + nchans);
  const int64_t maxabs = std::max<int64_t>(std::llabs(dmin), std::llabs(dmax));
  const int64_t nvalid = nsamps - maxabs;
  if (nvalid <= 0) return SPP_OK;  // reference: prange over a non-positive count
  if (-(int64_t)dmin > nsamps)
    return fail(SPP_ERR_DELAY, "negative delay %d reaches before the block", dmin);
  if (out_start < 0 || out_start + nvalid > out_len)
    return fail(SPP_ERR_SIZE, "output too small: out_start %lld + %lld samples > out_len %lld",
                (long long)out_start, (long long)nvalid, (long long)out_len);
  const int rc = launch_single8_hd(static_cast<const uint8_t*>(in), nchans, nsamps, delays_host,
                                   out, out_start, nvalid, as_stream(stream));
  if (rc == SPP_ERR_UNSUPPORTED)
    return fail(rc, "host-table path needs nchans %% 32 == 0, nchans <= 1024, a 16-B aligned "
                "block and every slab resident in shared memory");
  return rc;
}

static int dedisperse_host(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                           const int32_t* delays_host, float* out, int64_t out_len,
                           int64_t out_start, double limit_us, void* stream) {
  if (!in || !delays_host || !out) return fail(SPP_ERR_ARG, "spp_dedisperse_host: null pointer");
  if (!valid_nbits(nbits)) return fail(SPP_ERR_ARG, "nbits must be 1, 2, 4, 8 or 32 (got %d)", nbits);
  if (bitorder != SPP_BITORDER_BIG && bitorder != SPP_BITORDER_LITTLE)
    return fail(SPP_ERR_ARG, "bad bitorder %d", bitorder);
  if (nchans <= 0 || nsamps <= 0) return fail(SPP_ERR_ARG, "bad shape");
  if (nbits < 8 && (nchans * nbits) % 8 != 0)
    return fail(SPP_ERR_ARG, "nchans*nbits must be a multiple of 8");
  const int32_t dmin = *std::min_element(delays_host, delays_host + nchans);
  const int32_t dmax = *std::max_element(delays_host, delays_host + nchans);
  const int64_t nvalid = nsamps - std::max<int64_t>(std::llabs(dmin), std::llabs(dmax));
  if (nvalid <= 0) return SPP_OK;  // reference: prange over a non-positive count
  if (-(int64_t)dmin > nsamps)
    return fail(SPP_ERR_DELAY, "negative delay %d reaches before the block", dmin);
  if (out_start < 0 || out_start + nvalid > out_len)
    return fail(SPP_ERR_SIZE, "output too small: out_start %lld + %lld samples > out_len %lld",
                (long long)out_start, (long long)nvalid, (long long)out_len);
  const int rc = launch_single_stream(in, nbits, bitorder, nchans, nsamps, delays_host,
                                      out + out_start, nvalid, limit_us, as_stream(stream));
  if (rc == SPP_ERR_UNSUPPORTED)
    return fail(rc, "streaming path needs nchans <= 4096 and every slab's delay spread in shared memory");
  return rc;
}

int spp_dedisperse_host(const void* in, int nbits, int bitorder, int64_t nchans, int64_t nsamps,
                        const int32_t* delays_host, float* out, int64_t out_len,
                        int64_t out_start, void* stream) {
  return dedisperse_host(in, nbits, bitorder, nchans, nsamps, delays_host, out, out_len, out_start,
                         std::numeric_limits<double>::infinity(), stream);
}

// What spp_dedisperse takes for a block, in us: launches, the DM-time kernel's walk
// over the channels, and both kernels' traffic, which bytes moved one at a time
// (rows at odd addresses) slow down.  Fitted with the estimate of
// launch_single_stream: mostly within 20 %.
static double planar_us(int nbits, int64_t nchans, int64_t nsamps, uintptr_t align) {
  const double mb = (double)nsamps * (double)(nchans * nbits) / 8e6;
  const bool a16 = align % 16 == 0, a4 = align % 4 == 0;
  if (nbits == 32) return 12.0 + 0.0455 * nchans + 0.94 * mb;
  if (nbits == 8)
    return a16 ? 8.0 + 0.032 * nchans + 0.57 * mb : 12.0 + 0.047 * nchans + (a4 ? 1.14 : 2.66) * mb;
  return 13.3 + 0.05 * nchans + (a16 ? 1.51 : a4 ? 1.57 : 2.93) * mb;
}

int64_t spp_dedisperse_block(const void* in, int nbits, int bitorder, int64_t nchans,
                             int64_t nsamps, const int32_t* delays_host, int acc, float* out,
                             int64_t out_len, int64_t out_start, void* stream) {
  if (!delays_host || nchans <= 0) return fail(SPP_ERR_ARG, "spp_dedisperse_block: bad delays");
  int32_t dmin = delays_host[0], dmax = delays_host[0];
  for (int64_t c = 1; c < nchans; ++c) {
    dmin = std::min(dmin, delays_host[c]);
    dmax = std::max(dmax, delays_host[c]);
  }
  const int64_t nvalid = nsamps - std::max<int64_t>(std::llabs(dmin), std::llabs(dmax));
  if (nvalid <= 0) return 0;
  int rc = SPP_ERR_UNSUPPORTED;
  if (nbits == 8)
    rc = spp_dedisperse_hd(in, nbits, nchans, nsamps, delays_host, out, out_len, out_start, stream);
  // 8-bit rows aligned to 4 bytes only, over a short delay range: the device-
  // table kernel copies them in one pass without touching registers (1020
  // channels x 100000 samples, DM 100: 91 us against 125 us; 336 channels at an
  // address that is 4 mod 16, 106670 samples: 33 against 54 us)
  const uintptr_t rows = reinterpret_cast<uintptr_t>(in) | (uintptr_t)(nchans * nbits / 8);
  const bool narrow = nbits == 8 && rows % 4 == 0 && rows % 16 != 0 && (int64_t)dmax - dmin <= 2600;
  // one CTA walks all channels of its outputs, so short blocks and wide delay
  // spreads can take longer than two passes over the whole block (float32, 2048
  // channels, 4147 outputs: 288 us against 149 us; 8-bit, 512 channels, 3148
  // samples within a slab, 97385 outputs: 277 against 112 us)
  if (rc == SPP_ERR_UNSUPPORTED && !narrow && bitorder >= 0 && (nbits != 32 || acc == SPP_ACC_F64))
    rc = dedisperse_host(in, nbits, bitorder, nchans, nsamps, delays_host, out, out_len, out_start,
                         planar_us(nbits, nchans, nsamps, rows), stream);
  return rc == SPP_OK ? nvalid : rc;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Single-DM dedispersion without allocation.
//
// For callers that must not allocate device memory once they are running --
// e.g. a real-time search pipeline that reserves its device memory at
// start-up and treats any later cudaMalloc (which can synchronise the device
// and can fail under memory pressure) as an error, or a host framework whose
// own allocator owns the device memory and hands out only input and output
// buffers.  The scratch that spp_dedisperse takes as `workspace` lives here
// in a fixed device array instead.
// ---------------------------------------------------------------------------
namespace {

constexpr int64_t kNoAllocScratchBytes = 32ll << 20;  // 32 MiB per device
static __device__ __align__(256) uint8_t g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kMaxDevices] = {};

// Device address of the scratch array for the current device, looked up
// once per device (the symbol name is only a host-side handle).
int noalloc_scratch(void** out) {
  int dev = 0;
  int rc = cuda_status(cudaGetDevice(&dev), "cudaGetDevice");
  if (rc) return rc;
  if (dev < 0 || dev >= kMaxDevices) return fail(SPP_ERR_UNSUPPORTED, "device index %d", dev);
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    rc = cuda_status(cudaGetSymbolAddress(&p, g_noalloc_scratch), "cudaGetSymbolAddress");
    if (rc) return rc;
    g_noalloc_ptr[dev] = p;
  }
  *out = g_noalloc_ptr[dev];
  return SPP_OK;
}

}  // namespace

extern "C" {

int64_t spp_dedisperse_noalloc_max_bytes(void) { return kNoAllocScratchBytes; }

int spp_dedisperse_noalloc(const void* in, int nbits, int bitorder, int64_t nchans,
                           int64_t nsamps, const int32_t* delays, int32_t delay_min,
                           int32_t delay_max, float* out, int64_t out_len, int64_t out_start,
                           int acc, void* stream) {
  if (!in || !delays || !out) return fail(SPP_ERR_ARG, "spp_dedisperse_noalloc: null pointer");
  if (acc != SPP_ACC_F64 && acc != SPP_ACC_KAHAN32) return fail(SPP_ERR_ARG, "bad acc %d", acc);
  const Variant* v;
  Geometry g;
  int slot;
  int rc = single_setup(nbits, nchans, nsamps, delay_min, delay_max, acc, &v, &g, &slot);
  if (rc) return rc;
  if (g.nvalid <= 0) return SPP_OK;
  if (out_start < 0 || out_start + g.nvalid > out_len)
    return fail(SPP_ERR_SIZE, "output too small: out_start %lld + %lld samples > out_len %lld",
                (long long)out_start, (long long)g.nvalid, (long long)out_len);
  const int64_t need = kStatusBytes + g.bytes;
  if (need > kNoAllocScratchBytes)
    return fail(SPP_ERR_SIZE,
                "block needs %lld B of scratch, above the fixed %lld B of the no-allocation "
                "entry point: use spp_dedisperse with a workspace, or smaller blocks",
                (long long)need, (long long)kNoAllocScratchBytes);
  void* base = nullptr;
  rc = noalloc_scratch(&base);
  if (rc) return rc;
  cudaStream_t st = as_stream(stream);
  uint8_t* ws = static_cast<uint8_t*>(base);
  // the status block must start at zero; the planar rows are fully rewritten
  rc = cuda_status(cudaMemsetAsync(ws, 0, kStatusBytes, st), "status clear");
  if (rc) return rc;
  void* planar = ws + kStatusBytes;
  rc = launch_corner_turn(nbits, in, bitorder, nchans, nsamps, g, planar, st);
  if (rc) return rc;
  DmtArgs a{};
  a.planar = planar;
  a.pitch_w = g.pitch_w;
  a.halo = g.halo;
  a.nchans = (int32_t)nchans;
  a.delays = delays;
  a.dpitch = nchans;
  a.ndm = 1;
  a.sign = 1;
  a.dlo = delay_min;
  a.dhi = delay_max;
  a.span_max = 0;
  a.slot_w = slot;
  a.out = out;
  a.out_kind = SPP_OUT_F32;
  a.out_stride = 0;
  a.out_start = out_start;
  a.nvalid = g.nvalid;
  a.status = reinterpret_cast<uint32_t*>(ws);
  return launch_dmt(*v, a, g.ntiles_t, 1, st);
}

// The status words of the last spp_dedisperse_noalloc call on the current
// device sit at the head of the fixed array, where the caller has no pointer
// to them; this copies them out (synchronising `stream`).
int spp_dedisperse_noalloc_status_read(uint32_t* host_out, void* stream) {
  if (!host_out) return fail(SPP_ERR_ARG, "spp_dedisperse_noalloc_status_read: null pointer");
  void* base = nullptr;
  const int rc = noalloc_scratch(&base);
  if (rc) return rc;
  return spp_status_read(base, host_out, stream);
}

}  // extern "C"

// ---------------------------------------------------------------------------
// R3: DM-trial batch plan
// ---------------------------------------------------------------------------
struct spp_dmt_plan {
  int nbits, bitorder, mode, out_kind, acc;
  int64_t nchans, nsamps_max, ndm;
  int32_t* d_delays = nullptr;  // device, ndm x dpitch (raw delays)
  int64_t dpitch;
  int32_t dmin, dmax;  // raw delay range
  int32_t omin, omax;  // range of sign * delay
  int32_t maxabs;
  std::vector<int> cands;      // candidate variant indices
  std::vector<int32_t> spans;  // span per candidate
  int cur = 0;                 // index into cands
  int packed[2] = {-1, -1};    // of these the packed shapes that estimates consider
  bool chosen = false;         // cur was set by the caller
  // interleaved bit-plane kernels: rows of channels and of channel pairs, and
  // per kernel shape the staging tables (sized at creation, built when first
  // selected)
  IlvRows ilv_rows[2];
  std::vector<IlvTables> ilv_tabs;
  void* room = nullptr;        // within the allocation of d_delays
  int64_t room_bytes = 0;
  // optional per-kernel timing: events (start, after corner turn, end) per execute
  bool timing = false;
  std::vector<cudaEvent_t> evpool;
  size_t evused = 0;
};

constexpr int64_t kMaxTimeTiles = 65535;  // gridDim.y

// Candidate codes at or above this name an interleaved bit-plane shape.
constexpr int kIlvCode = 1 << 20;
static int ilv_index(const spp_dmt_plan* p, int cand) {
  return p->cands[cand] >= kIlvCode ? p->cands[cand] - kIlvCode : -1;
}
static int plan_sign(const spp_dmt_plan* p) { return p->mode == SPP_MODE_ROLL ? -1 : 1; }
static IlvDelays ilv_delays(const spp_dmt_plan* p) {
  return IlvDelays{p->d_delays, p->ndm, p->nchans, plan_sign(p), p->nbits};
}

static cudaEvent_t plan_event(spp_dmt_plan* p) {
  if (p->evused == p->evpool.size()) {
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    p->evpool.push_back(e);
  }
  return p->evpool[p->evused++];
}

static int64_t plan_nvalid(const spp_dmt_plan* p, int64_t nsamps) {
  return p->mode == SPP_MODE_ROLL ? nsamps : nsamps - p->maxabs;
}

// Staging tables of candidate i, built the first time it is selected (plan
// creation for the initial choice, else set_variant).
static int ensure_tables(spp_dmt_plan* p, int i) {
  const int iv = ilv_index(p, i);
  if (iv < 0) return SPP_OK;
  const IlvCfg& c = ilv_cfgs()[iv];
  // the plan's room serves the first shape
  bool taken = false;
  for (const IlvTables& t : p->ilv_tabs) taken = taken || (t.d_off && !t.own);
  return ilv_build_tables(c, ilv_delays(p), p->ilv_rows[c.G - 1], p->room, taken ? 0 : p->room_bytes,
                          &p->ilv_tabs[iv]);
}

static void free_device(spp_dmt_plan* p) {
  for (IlvTables& t : p->ilv_tabs) ilv_free_tables(&t);
  if (p->d_delays) cudaFree(p->d_delays);
  p->d_delays = nullptr;
}

// Pair rows a plan may hold, per channel.
constexpr int64_t kPairRowsPerChan = 12;

// Device words of a plan: the delay table, then (for interleaved shapes) the words
// that make their rows, from a 256-byte boundary on: the range pass stores pairs of
// words there, whatever the table's size; then room for the staging tables of the
// shape that the plan starts from, of the most that they may need (some four times
// what they take).  The driver hands out chunks of 2 MB: a new chunk or a larger
// allocation takes 0.38 ms and its release 0.3, a part of a chunk 2 us.  So tables have
// room here where all of it is small or where words and tables would not share a
// chunk, unless they may be large; else they are allocated as they turn out (8-bit,
// beside other plans, 256 channels x 228 trials: creation 870 us with room of 1.4 MB,
// 450 us without; 1024 x 300: 920 us in two allocations, 560 us in one).
struct PlanWords {
  int64_t work, room, total;
};
static PlanWords plan_words(int nbits, int64_t nchans, int64_t ndm) {
  const int64_t table = ndm * nchans;
  if (ndm <= 1 || nbits > 8) return {table, table, table};
  const int64_t work = round_up(table, 64);
  const int64_t room = round_up(work + ilv_plan_words(nchans, kPairRowsPerChan * nchans), 64);
  const int64_t bytes = ilv_table_room(nbits, nchans, ndm);
  const bool one_chunk = 4 * room + bytes / 4 < 7ll << 18;  // 1.75 MB
  const bool here = one_chunk ? 4 * room + bytes <= 512ll << 10 : bytes <= 64ll << 20;
  return {work, room, room + (here ? bytes / 4 : 0)};
}

// Interleaved bit-plane shapes that channel count and sample width allow.
static std::vector<int> ilv_shapes(int nbits, int64_t nchans) {
  const auto& cfgs = ilv_cfgs();
  std::vector<int> which;
  for (int i = 0; i < (int)cfgs.size(); ++i) {
    const IlvCfg& c = cfgs[i];
    if (c.nb == nbits && nchans % c.G == 0 && nchans * ((1ll << c.nb) - 1) < (1ll << c.levels))
      which.push_back(i);
  }
  return which;
}

// Byte lanes, four trials x two warps: the packed shape with the shortest walk
// over the channels.
static bool short_walk(const Variant& v) { return !v.planes && v.R == 2 && v.DW == 4 && v.TW == 2; }

// Estimated times (us), fitted to 1573 plans measured with every shape they offer
// (16-4096 channels, 2-1024 trials, 1000-250000 outputs, trial grids from fine to
// thousands of samples apart; the logarithms' deviation is 0.08 to 0.2).

// A block by a packed kernel over 32 consecutive samples per word.  Few tiles: one
// CTA's walk over all channels, shorter where warps have no trial.  Many: tiles over
// 148 SMs, each slower the fewer CTAs an SM holds beside it.  Between the two the sum
// of fourth powers; then the corner turn, per MB of raw rows.
struct PackedTime {
  double walk0, walk, fill, full0, tile, few, mb;
};
static double packed_us(const spp_dmt_plan* p, int cand, int64_t nsamps, int64_t nvalid) {
  static const PackedTime first[] = {{15.7, 0.0909, 0.57, 20.6, 0.0543, 1.42, 2.69},
                                     {16.9, 0.126, 0.687, 24.0, 0.0716, 0.366, 1.98},
                                     {14.8, 0.25, 0.745, 23.6, 0.137, 2.01, 1.49},
                                     {14.4, 0.407, 0.819, 26.2, 0.0954, 3.79, 1.09}};
  static const PackedTime lanes8 = {10.3, 0.132, 0.95, 17.6, 0.0952, 0.59, 0.836};
  static const PackedTime brief[] = {{15.1, 0.106, 1.0, 24.4, 0.132, 0.173, 3.38},
                                     {11.7, 0.0686, 1.0, 20.5, 0.0595, 0.531, 2.3},
                                     {9.3, 0.0666, 1.0, 18.1, 0.0325, 1.89, 1.51},
                                     {6.43, 0.0649, 1.0, 18.1, 0.0299, 1.72, 0.649}};
  const Variant& v = variants()[p->cands[cand]];
  const int k = p->nbits == 1 ? 0 : p->nbits == 2 ? 1 : p->nbits == 4 ? 2 : 3;
  const PackedTime& c = short_walk(v) ? brief[k] : k == 3 && !v.planes ? lanes8 : first[k];
  const double fill = c.fill + (1.0 - c.fill) * std::min(1.0, (double)p->ndm / v.DW);
  const double ctas = (double)ceil_div(p->ndm, v.DW) * (double)ceil_div(nvalid, tile_T(v));
  const int64_t per_sm = std::max<int64_t>(1, (228 << 10) / (smem_bytes(v, slot_words(v, p->spans[cand])) + 1024));
  const double tile = c.tile * (1.0 + c.few * std::max(0.0, 1.0 / (double)per_sm - 0.25));
  const double walk = c.walk0 + c.walk * fill * (double)p->nchans;
  const double full = c.full0 + tile * fill * (double)p->nchans * ctas / 148.0;
  const double w2 = walk * walk, f2 = full * full;
  return std::sqrt(std::sqrt(w2 * w2 + f2 * f2)) +
         c.mb * (double)nsamps * (double)(p->nchans * p->nbits) / 8e6;
}

// The same by an interleaved shape: per wave of 148 CTAs a fixed part (start, first
// copies, stores) and a part per group of channels, both measured per shape
// (IlvCfg::us_wave, ns_group) and scaled; the corner turn per MB of raw rows and per
// byte of what its rows hold beyond the block; its further blocks of 32 runs; and the
// pair rows, by their bytes or, where those are many and short, their CTAs.  Raw rows
// that are no whole number of 16-byte units, and a last group of channels that is no
// whole 32 bytes, are turned byte by byte.
struct IlvTime {
  double us0, wave, group, mb, extra, odd_mb, odd0, block, row, pair_cta;
};
static double interleaved_us(const spp_dmt_plan* p, const IlvCfg& c, int64_t nsamps, const IlvGeom& g) {
  static const IlvTime chans[] = {{7.54, 0.847, 0.901, 1.77, 14e-7, 3.46, 5.32, 1.94, 0, 0},
                                  {6.87, 0.75, 0.904, 2.34, 9.14e-7, 2.88, 9.12, 1.93, 0, 0},
                                  {4.13, 0.75, 0.95, 1.56, 4.78e-7, 3.21, 6.82, 2.49, 0, 0},
                                  {6.25, 0.947, 0.974, 1.16, 1.59e-7, 3.08, 5.91, 3.24, 0, 0}};
  static const IlvTime pairs[] = {{},
                                  {8.0, 1.0, 1.0, 1.4, 7e-7, 3.41, 4.6, 2.01, 3.65e-7, 0.312e-3},
                                  {7.38, 0.75, 0.899, 1.53, 8.79e-7, 3.31, 8.73, 2.2, 2.1e-7, 0.814e-3},
                                  {9.84, 0.759, 0.937, 1.16, 0.06e-7, 3.29, 7.63, 1.54, 3.07e-7, 7.98e-3}};
  const int k = p->nbits == 1 ? 0 : p->nbits == 2 ? 1 : p->nbits == 4 ? 2 : 3;
  const IlvTime& e = c.G == 2 ? pairs[k] : chans[k];
  const int64_t ctas = ceil_div(p->ndm, c.DW) * ceil_div(g.M, c.words());
  const double ng = (double)round_up(p->nchans / c.G, 4 * c.nq);
  const int64_t rowbytes = p->nchans * c.nb / 8, odd = rowbytes % 16 ? rowbytes : rowbytes % 32;
  const double blocks = (double)(p->ilv_rows[0].max_group / (32 * g.M));
  double t = e.us0 + (double)ceil_div(ctas, 148) * (e.wave * c.us_wave + ng * e.group * c.ns_group * 1e-3);
  t += e.mb * (double)nsamps * (double)rowbytes * 1e-6;
  t += e.extra * (double)(g.chan_bytes - p->nchans * g.M * c.nb * 4);
  t += odd ? e.odd0 + e.odd_mb * 1e-6 * (double)nsamps * (double)odd + 4.0 * e.block * blocks : e.block * blocks;
  if (c.G == 2) {
    const double pair_ctas = (double)(p->nchans / 2) * (double)ceil_div(g.M + p->ilv_rows[0].max_ext, 512);
    t += std::max(e.row * (double)g.row_bytes, e.pair_cta * pair_ctas);
  }
  return t;
}

// Float64 sums of float32 rows, without the corner turn that all shapes share: one
// CTA's walk where few tiles run, else the SM's share of the tiles (whole ones: the
// fullest SM counts), slower below 12 adding warps per SM; the sum of fourth powers
// between.  Over 629 plans (16-4096 channels, 2-500 trials) the shape of least
// estimate takes 1.3 % longer than the fastest on average; a rate per shape over waves
// of full SMs, 5.1 %.
static double float64_us(const spp_dmt_plan* p, int cand, int64_t nvalid) {
  const Variant& v = variants()[p->cands[cand]];
  const int64_t smem = smem_bytes(v, slot_words(v, p->spans[cand])) + 1024;
  const int64_t per_sm = std::max<int64_t>(1, std::min<int64_t>((228 << 10) / smem, 64 / (v.DW * v.TW + 1)));
  const int64_t ctas = ceil_div(p->ndm, v.DW) * ceil_div(nvalid, tile_T(v));
  const double few = 1.0 + v.time.few * std::max(0.0, 12.0 / (double)(per_sm * v.DW * v.TW) - 1.0);
  const double walk = v.time.walk0 + v.time.walk * (double)p->nchans;
  const double full = v.time.tile * few * (double)p->nchans * (double)ceil_div(ctas, 148);
  const double w2 = walk * walk, f2 = full * full;
  return std::sqrt(std::sqrt(w2 * w2 + f2 * f2));
}

// The shape a plan starts from (without autotuning): the least estimated time
// at nsamps_max, over the interleaved shapes, the first packed one and the one of
// the shortest walk.  Over the 1573 plans that the estimates are fitted to the choice
// takes 3.3 % longer than the fastest shape on average, and some 20 take more than 8 %
// longer than before the interleaved shapes (2-bit plans of few tiles, where a kernel
// over channel pairs had been the fastest, and blocks of 20 to 40 us).  Rows and
// staging tables above kIlvDefaultBytes leave a shape to explicit choice: they grow
// with the block and the delay range, and with the trials.
// 2-bit grids so fine that a pair row serves 100 trials or more start from pairs
// from 4096 outputs on (a pair shape's shortest tile), so that the blocks of one
// observation run one kernel (4096 channels, 1024 trials to DM 2000: 45.9 ms
// against 52.6 ms without pairs at 1016174 outputs, 3.5 against 3.7 ms at 65536,
// 1.2 against 1.0 ms at 16384, 0.84 against 0.63 ms at 4096).
static int first_choice(spp_dmt_plan* p) {
  constexpr int64_t kIlvDefaultBytes = 16ll << 30;
  const int64_t nvalid = std::max<int64_t>(1, plan_nvalid(p, p->nsamps_max));
  // Time tiles are a grid's y extent: shapes of short tiles cannot run the
  // longest blocks (256-sample tiles: 16.8 million outputs).
  auto tiles_fit = [&](int i) {
    return ilv_index(p, i) >= 0 || ceil_div(nvalid, tile_T(variants()[p->cands[i]])) <= kMaxTimeTiles;
  };
  int first = 0;
  while (first + 1 < (int)p->cands.size() && !tiles_fit(first)) ++first;
  if (p->nbits == 32) {
    int pick = first;
    double best = 0.0;
    for (int i = 0; i < (int)p->cands.size(); ++i) {
      if (variants()[p->cands[i]].time.tile <= 0.0 || !tiles_fit(i)) continue;
      const double t = float64_us(p, i, nvalid);
      if (best == 0.0 || t < best) {
        best = t;
        pick = i;
      }
    }
    return pick;
  }
  for (int i = 0, n = 0; i < (int)p->cands.size() && n < 2; ++i)
    if (ilv_index(p, i) < 0 && tiles_fit(i) && (n == 0 ? i >= first : short_walk(variants()[p->cands[i]])))
      p->packed[n++] = i;
  const int64_t prows = p->ilv_rows[1].nrows;
  const bool shared_pairs = p->nbits == 2 && prows > 0 && nvalid >= 4096 &&
                            p->ndm * (p->nchans / 2) >= 100 * prows;
  int pick = first;
  bool any = false;
  bool paired = false;
  double best = 0.0;
  for (int i = 0; i < (int)p->cands.size(); ++i) {
    const int iv = ilv_index(p, i);
    double t;
    bool pairs = false;
    if (iv < 0) {
      if (i != p->packed[0] && i != p->packed[1]) continue;
      t = packed_us(p, i, p->nsamps_max, nvalid);
      if (i == p->packed[0]) t *= 0.92;  // near ties stay with the smaller workspace
    } else {
      const IlvCfg& c = ilv_cfgs()[iv];
      const IlvGeom g = ilv_geometry(c, p->ilv_rows[0], p->ilv_rows[c.G - 1], p->nchans, nvalid);
      const int64_t own = ilv_table_bytes(c, ilv_delays(p), p->ilv_tabs[iv]);
      if (g.chan_bytes + g.row_bytes + own > kIlvDefaultBytes && any) continue;
      t = interleaved_us(p, c, p->nsamps_max, g);
      pairs = c.G == 2;
    }
    if (paired && shared_pairs && !pairs) continue;
    if (t < best || !any || (shared_pairs && pairs && !paired)) {
      best = t;
      pick = i;
      any = true;
      paired = pairs;
    }
  }
  return pick;
}

// Range of a host table and the widest spread of a channel over tiles of two, four
// and eight trials, in one sweep (float32 plan of 1024 trials x 4096 channels: 7.1
// ms with a sweep per tile height and one for the range, 4.2 ms).
static void table_range(const int32_t* d, int64_t ndm, int64_t nchans, int32_t* dmin, int32_t* dmax,
                        int32_t (&span)[3]) {
  int32_t mn = INT32_MAX, mx = INT32_MIN, s2 = 0, s4 = 0, s8 = 0;
  for (int64_t t = 0; t < ndm; t += 8) {
    const int32_t* row[8];
    for (int i = 0; i < 8; ++i) row[i] = d + std::min(t + i, ndm - 1) * nchans;
    for (int64_t c = 0; c < nchans; ++c) {
      int32_t lo[4], hi[4];
      for (int i = 0; i < 4; ++i) {
        const int32_t x = row[2 * i][c], y = row[2 * i + 1][c];
        lo[i] = std::min(x, y);
        hi[i] = std::max(x, y);
        s2 = std::max(s2, hi[i] - lo[i]);
      }
      const int32_t la = std::min(lo[0], lo[1]), ha = std::max(hi[0], hi[1]);
      const int32_t lb = std::min(lo[2], lo[3]), hb = std::max(hi[2], hi[3]);
      const int32_t l8 = std::min(la, lb), h8 = std::max(ha, hb);
      s4 = std::max(s4, std::max(ha - la, hb - lb));
      s8 = std::max(s8, h8 - l8);
      mn = std::min(mn, l8);
      mx = std::max(mx, h8);
    }
  }
  *dmin = mn;
  *dmax = mx;
  span[0] = s2;
  span[1] = s4;
  span[2] = s8;
}

extern "C" {

int spp_dmt_plan_create(spp_dmt_plan** plan, int nbits, int bitorder, int64_t nchans,
                        int64_t nsamps_max, int64_t ndm, const int32_t* delays_host, int mode,
                        int out_kind, int acc) {
  if (!plan || !delays_host) return fail(SPP_ERR_ARG, "spp_dmt_plan_create: null pointer");
  *plan = nullptr;
  if (!valid_nbits(nbits)) return fail(SPP_ERR_ARG, "nbits must be 1, 2, 4, 8 or 32 (got %d)", nbits);
  if (nchans <= 0 || ndm <= 0 || nsamps_max <= 0 || nchans > INT32_MAX || ndm > INT32_MAX)
    return fail(SPP_ERR_ARG, "bad shape");
  if (nbits < 8 && (nchans * nbits) % 8 != 0)
    return fail(SPP_ERR_ARG, "nchans*nbits must be a multiple of 8");
  if (mode != SPP_MODE_DEDISPERSE && mode != SPP_MODE_ROLL) return fail(SPP_ERR_ARG, "bad mode");
  if (out_kind != SPP_OUT_F32 && out_kind != SPP_OUT_I32) return fail(SPP_ERR_ARG, "bad out_kind");
  if (out_kind == SPP_OUT_I32 && nbits == 32)
    return fail(SPP_ERR_ARG, "int32 output needs integer input");
  if (acc != SPP_ACC_F64 && acc != SPP_ACC_KAHAN32) return fail(SPP_ERR_ARG, "bad acc");
  if (bitorder != SPP_BITORDER_BIG && bitorder != SPP_BITORDER_LITTLE)
    return fail(SPP_ERR_ARG, "bad bitorder");
  spp_dmt_plan* p = new (std::nothrow) spp_dmt_plan();
  if (!p) return fail(SPP_ERR_ARG, "out of host memory");
  p->nbits = nbits; p->bitorder = bitorder; p->mode = mode; p->out_kind = out_kind; p->acc = acc;
  p->nchans = nchans; p->nsamps_max = nsamps_max; p->ndm = ndm;
  const bool ilv = ndm > 1 && nbits <= 8;
  const int sign = plan_sign(p);
  auto set_range = [&](int32_t omin, int32_t omax) {
    p->omin = omin; p->omax = omax;
    p->dmin = sign > 0 ? omin : -omax;
    p->dmax = sign > 0 ? omax : -omin;
    p->maxabs = (int32_t)std::max<int64_t>(std::llabs(omin), std::llabs(omax));
  };
  std::vector<std::pair<int, int32_t>> span_of_dw;  // widest spread of a channel over tiles of so many trials
  if (nbits == 32 && ndm > 1) {
    int32_t omin, omax, span[3];
    table_range(delays_host, ndm, nchans, &omin, &omax, span);
    set_range(sign > 0 ? omin : -omax, sign > 0 ? omax : -omin);
    span_of_dw = {{2, span[0]}, {4, span[1]}, {8, span[2]}};
  } else if (!ilv || mode == SPP_MODE_ROLL) {
    int32_t dmin = INT32_MAX, dmax = INT32_MIN;
    for (int64_t i = 0; i < ndm * nchans; ++i) {
      dmin = std::min(dmin, delays_host[i]);
      dmax = std::max(dmax, delays_host[i]);
    }
    set_range(sign > 0 ? dmin : -dmax, sign > 0 ? dmax : -dmin);
  }
  if (mode == SPP_MODE_ROLL && p->maxabs >= nsamps_max) {
    delete p;
    return fail(SPP_ERR_DELAY, "roll mode needs |delay| < nsamps");
  }
  p->dpitch = nchans;
  PlanWords words = plan_words(nbits, nchans, ndm);
  cudaError_t e = cudaMalloc(&p->d_delays, sizeof(int32_t) * words.total);
  if (e == cudaErrorMemoryAllocation && words.room < words.total) {  // the rest may still fit
    cudaGetLastError();
    words.total = words.room;
    e = cudaMalloc(&p->d_delays, sizeof(int32_t) * words.total);
  }
  if (e != cudaSuccess) { delete p; return cuda_status(e, "plan cudaMalloc"); }
  e = cudaMemcpy(p->d_delays, delays_host, sizeof(int32_t) * ndm * nchans, cudaMemcpyHostToDevice);
  int rc = cuda_status(e, "plan upload");
  p->room = p->d_delays + words.room;
  p->room_bytes = 4 * (words.total - words.room);
  // Ranges and the spreads of trial tiles, of four and eight trials for all packed
  // integer shapes: found on the device beside the interleaved rows (the host took
  // 0.14 ms per tile height and as much for the range over 512 trials x 1024
  // channels).
  IlvRange range{};
  const std::vector<int> shapes = ilv ? ilv_shapes(nbits, nchans) : std::vector<int>();
  if (rc == SPP_OK && ilv) {
    p->ilv_tabs.resize(ilv_cfgs().size());
    rc = ilv_find(shapes, ilv_delays(p), kPairRowsPerChan * nchans, p->d_delays + words.work, &range,
                  p->ilv_rows, &p->ilv_tabs);
    set_range(range.omin, range.omax);
  }
  // candidates; the delay spread of DM tiles is computed once per tile height
  const auto& vs = variants();
  if (ilv) span_of_dw = {{4, range.span4}, {8, range.span8}};
  auto tile_span = [&](int dw) -> int32_t {
    for (auto& e : span_of_dw)
      if (e.first == dw) return e.second;
    int32_t span = 0;
    std::vector<int32_t> mn(nchans), mx(nchans);
    for (int64_t d0 = 0; d0 < ndm; d0 += dw) {
      const int64_t d1 = std::min<int64_t>(ndm, d0 + dw);
      std::copy(delays_host + d0 * nchans, delays_host + (d0 + 1) * nchans, mn.begin());
      std::copy(mn.begin(), mn.end(), mx.begin());
      for (int64_t d = d0 + 1; d < d1; ++d) {
        const int32_t* row = delays_host + d * nchans;
        for (int64_t c = 0; c < nchans; ++c) {
          mn[c] = std::min(mn[c], row[c]);
          mx[c] = std::max(mx[c], row[c]);
        }
      }
      for (int64_t c = 0; c < nchans; ++c) span = std::max(span, mx[c] - mn[c]);
    }
    span_of_dw.emplace_back(dw, span);
    return span;
  };
  for (int i = 0; i < (int)vs.size(); ++i) {
    const Variant& v = vs[i];
    if (v.nb != nbits || (nbits == 32 && v.acc != acc)) continue;
    if (ndm == 1 ? !v.single : v.single) continue;
    if (v.planes && nchans * ((1 << nbits) - 1) >= (1 << bit_levels(nbits))) continue;
    const int32_t span = tile_span(v.DW);
    if (slot_words(v, span) < 0) continue;  // fixed slot too narrow for this table
    if (smem_bytes(v, slot_words(v, span)) > kMaxSmem) continue;
    p->cands.push_back(i);
    p->spans.push_back(span);
  }
  for (int i : shapes) {
    if (p->ilv_tabs.empty() || p->ilv_tabs[i].stages == 0) continue;
    p->cands.push_back(kIlvCode + i);
    p->spans.push_back(0);
  }
  if (rc == SPP_OK && p->cands.empty())
    rc = fail(SPP_ERR_UNSUPPORTED, "no kernel variant fits this delay table");
  if (rc == SPP_OK) {
    p->cur = first_choice(p);
    rc = ensure_tables(p, p->cur);
    // staging tables of a very fine grid may be larger than what is left of the
    // device memory; the packed shapes need none
    if (rc != SPP_OK && p->ilv_tabs[ilv_index(p, p->cur)].no_memory && p->packed[0] >= 0) {
      p->cur = p->packed[0];
      rc = SPP_OK;
    }
  }
  if (rc != SPP_OK) {
    free_device(p);
    delete p;
    return rc;
  }
  *plan = p;
  return SPP_OK;
}

int spp_dmt_plan_layout(int nbits, int64_t nchans, int64_t ndm, int64_t* work_offset,
                        int64_t* total_bytes) {
  if (!work_offset || !total_bytes) return fail(SPP_ERR_ARG, "spp_dmt_plan_layout: null pointer");
  if (!valid_nbits(nbits)) return fail(SPP_ERR_ARG, "nbits must be 1, 2, 4, 8 or 32 (got %d)", nbits);
  if (nchans <= 0 || ndm <= 0 || nchans > INT32_MAX || ndm > INT32_MAX)
    return fail(SPP_ERR_ARG, "bad shape");
  const PlanWords w = plan_words(nbits, nchans, ndm);
  *work_offset = 4 * w.work;
  *total_bytes = 4 * w.total;
  return SPP_OK;
}

int spp_dmt_plan_destroy(spp_dmt_plan* p) {
  if (!p) return SPP_OK;
  int rc = SPP_OK;
  for (cudaEvent_t e : p->evpool) cudaEventDestroy(e);
  if (p->d_delays) rc = cuda_status(cudaFree(p->d_delays), "plan cudaFree");
  p->d_delays = nullptr;
  free_device(p);
  delete p;
  return rc;
}

int64_t spp_dmt_plan_nvalid(const spp_dmt_plan* p, int64_t nsamps) {
  if (!p) return -1;
  return std::max<int64_t>(0, plan_nvalid(p, nsamps));
}

int spp_dmt_plan_num_variants(const spp_dmt_plan* p) { return p ? (int)p->cands.size() : 0; }

int spp_dmt_plan_set_variant(spp_dmt_plan* p, int variant) {
  if (!p) return fail(SPP_ERR_ARG, "null plan");
  if (variant < 0 || variant >= (int)p->cands.size()) return fail(SPP_ERR_ARG, "bad variant %d", variant);
  const int rc = ensure_tables(p, variant);
  if (rc != SPP_OK) return rc;
  p->cur = variant;
  p->chosen = true;
  return SPP_OK;
}

int spp_dmt_plan_describe(const spp_dmt_plan* p, int32_t* cfg) {
  if (!p || !cfg) return fail(SPP_ERR_ARG, "null pointer");
  const int iv = ilv_index(p, p->cur);
  if (iv >= 0) {
    const IlvCfg& c = ilv_cfgs()[iv];
    const IlvTables& t = p->ilv_tabs[iv];
    cfg[0] = c.nb | (1 << 8) | ((c.G == 2) << 9);
    cfg[1] = c.P; cfg[2] = c.DW; cfg[3] = c.TW; cfg[4] = 4 * c.nq; cfg[5] = t.stages;
    cfg[6] = 32 * c.words();
    cfg[7] = (int32_t)t.smem;
    return SPP_OK;
  }
  const Variant& v = variants()[p->cands[p->cur]];
  const int slot = slot_words(v, p->spans[p->cur]);
  cfg[0] = v.nb | (v.planes << 8); cfg[1] = v.R; cfg[2] = v.DW; cfg[3] = v.TW; cfg[4] = v.SLAB;
  cfg[5] = v.STAGES;
  cfg[6] = (int32_t)tile_T(v);
  cfg[7] = (int32_t)smem_bytes(v, slot);
  return SPP_OK;
}

static Geometry plan_geometry(const spp_dmt_plan* p, int cand, int64_t nsamps, int* slot) {
  const Variant& v = variants()[p->cands[cand]];
  *slot = slot_words(v, p->spans[cand]);
  return geometry(v, p->nchans, nsamps, plan_nvalid(p, nsamps), p->omin, p->omax, *slot);
}

static IlvGeom plan_ilv_geometry(const spp_dmt_plan* p, int iv, int64_t nsamps) {
  const IlvCfg& c = ilv_cfgs()[iv];
  return ilv_geometry(c, p->ilv_rows[0], p->ilv_rows[c.G - 1], p->nchans, plan_nvalid(p, nsamps));
}

int64_t spp_dmt_plan_workspace_bytes(const spp_dmt_plan* p, int64_t nsamps) {
  if (!p) return -1;
  const int iv = ilv_index(p, p->cur);
  if (iv >= 0) {
    const IlvGeom g = plan_ilv_geometry(p, iv, nsamps);
    return kStatusBytes + g.chan_bytes + g.row_bytes;
  }
  int slot;
  Geometry g = plan_geometry(p, p->cur, nsamps, &slot);
  return kStatusBytes + g.bytes;
}

// The transform by an interleaved bit-plane shape (arguments checked by dmt_run).
static int ilv_run(const spp_dmt_plan* p, int iv, const void* in, int64_t nsamps, void* out,
                   int64_t out_stride, int64_t out_start, uint8_t* ws, int64_t ws_bytes,
                   cudaStream_t st) {
  const int64_t nvalid = plan_nvalid(p, nsamps);
  const IlvCfg& c = ilv_cfgs()[iv];
  const IlvRows &chan = p->ilv_rows[0], &rows = p->ilv_rows[c.G - 1];
  const IlvGeom g = plan_ilv_geometry(p, iv, nsamps);
  const int64_t need = kStatusBytes + g.chan_bytes + g.row_bytes;
  if (ws_bytes < need)
    return fail(SPP_ERR_SIZE, "workspace %lld B < required %lld B", (long long)ws_bytes, (long long)need);
  spp_dmt_plan* pm = const_cast<spp_dmt_plan*>(p);
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  if (p->timing) {
    for (int i = 0; i < 3; ++i) {
      ev[i] = plan_event(pm);
      if (!ev[i]) return fail(SPP_ERR_CUDA, "cudaEventCreate failed");
    }
    cudaEventRecord(ev[0], st);
  }
  uint8_t* data = ws + kStatusBytes;
  int rc = ilv_corner_turn(c, chan, g, in, p->bitorder, p->nchans, nsamps, data, st);
  if (!rc) rc = ilv_group_rows(c, chan, rows, g, p->nchans, data, st);
  if (p->timing) cudaEventRecord(ev[1], st);
  if (!rc)
    rc = ilv_launch(c, p->ilv_tabs[iv], rows, g, p->nchans / c.G, p->ndm, data, out, p->out_kind,
                    out_stride, out_start, nvalid, reinterpret_cast<uint32_t*>(ws), st);
  if (p->timing) cudaEventRecord(ev[2], st);
  return rc;
}

// The shape that a block runs.  Interleaved rows carry the whole delay range
// whatever the block's length, so a block much shorter than the plan's longest (the
// last of a stream) goes to a packed shape where that is estimated to take less and
// the workspace, sized for the plan's own shape, holds its rows (1-bit, 336
// channels, 639 trials to DM 1877, 1012 of 16205 outputs: 501 us against 79 us).
// A shape that the caller set runs every block.
static int block_shape(const spp_dmt_plan* p, int64_t nsamps, int64_t ws_bytes) {
  const int iv = ilv_index(p, p->cur);
  const int64_t nvalid = plan_nvalid(p, nsamps);
  if (iv < 0 || p->chosen || 2 * nvalid > plan_nvalid(p, p->nsamps_max)) return p->cur;
  int pick = p->cur;
  double best = interleaved_us(p, ilv_cfgs()[iv], nsamps, plan_ilv_geometry(p, iv, nsamps));
  for (int i : p->packed) {
    if (i < 0) continue;
    int slot;
    const double t = packed_us(p, i, nsamps, nvalid);
    if (t < best && kStatusBytes + plan_geometry(p, i, nsamps, &slot).bytes <= ws_bytes) {
      best = t;
      pick = i;
    }
  }
  return pick;
}

static int dmt_run(const spp_dmt_plan* p, const void* in, int64_t nsamps, void* out,
                   int64_t out_stride, int64_t out_start, uint8_t* ws, int64_t ws_bytes,
                   cudaStream_t st, const float* zd_bpass = nullptr,
                   const float* zd_chanwts = nullptr, double* zd_rows = nullptr) {
  const int64_t nvalid = plan_nvalid(p, nsamps);
  if (nvalid <= 0) return SPP_OK;
  if (p->mode == SPP_MODE_ROLL && p->maxabs >= nsamps)
    return fail(SPP_ERR_DELAY, "roll mode needs |delay| < nsamps");
  if (-(int64_t)p->omin > nsamps)
    return fail(SPP_ERR_DELAY, "negative offset %d reaches before the block", p->omin);
  if (out_start < 0 || (p->ndm > 1 && out_stride < out_start + nvalid))
    return fail(SPP_ERR_SIZE, "out_stride %lld < out_start %lld + nvalid %lld",
                (long long)out_stride, (long long)out_start, (long long)nvalid);
  const int cand = block_shape(p, nsamps, ws_bytes);
  const int iv = ilv_index(p, cand);
  if (iv >= 0) return ilv_run(p, iv, in, nsamps, out, out_stride, out_start, ws, ws_bytes, st);
  int slot;
  Geometry g = plan_geometry(p, cand, nsamps, &slot);
  if (ws_bytes < kStatusBytes + g.bytes)
    return fail(SPP_ERR_SIZE, "workspace %lld B < required %lld B", (long long)ws_bytes,
                (long long)(kStatusBytes + g.bytes));
  if (g.ntiles_t > kMaxTimeTiles)
    return fail(SPP_ERR_UNSUPPORTED, "%lld time tiles exceed the grid limit", (long long)g.ntiles_t);
  const Variant& v = variants()[p->cands[cand]];
  void* planar = ws + kStatusBytes;
  spp_dmt_plan* pm = const_cast<spp_dmt_plan*>(p);
  cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
  if (p->timing) {
    for (int i = 0; i < 3; ++i) {
      ev[i] = plan_event(pm);
      if (!ev[i]) return fail(SPP_ERR_CUDA, "cudaEventCreate failed");
    }
    cudaEventRecord(ev[0], st);
  }
  int rc = SPP_OK;
  if (zd_rows) {
    const unsigned blocks = (unsigned)ceil_div(nsamps, 32 * kRowSumWarps);
    k_row_sum_f64<<<blocks, 32 * kRowSumWarps, 0, st>>>(static_cast<const float*>(in), p->nchans, nsamps, zd_rows);
    rc = cuda_status(cudaGetLastError(), "zero-DM row sums");
    if (rc) return rc;
  }
  // float64 sums of float32 rows: the corner turn flags samples that are not
  // finite floats (word kSpecialWord of the status block, cleared here)
  uint32_t* special = nullptr;
  if (p->nbits == 32 && v.acc == SPP_ACC_F64) {
    special = reinterpret_cast<uint32_t*>(ws) + kSpecialWord;
    rc = cuda_status(cudaMemsetAsync(special, 0, 4, st), "special-value flag clear");
    if (rc) return rc;
  }
  rc = launch_corner_turn(p->nbits, in, p->bitorder, p->nchans, nsamps, g, planar, st, zd_rows,
                          zd_chanwts, zd_bpass, special);
  if (rc) return rc;
  if (p->timing) cudaEventRecord(ev[1], st);
  DmtArgs a{};
  a.planar = planar;
  a.pitch_w = g.pitch_w;
  a.halo = g.halo;
  a.nchans = (int32_t)p->nchans;
  a.delays = p->d_delays;
  a.dpitch = p->dpitch;
  a.ndm = (int32_t)p->ndm;
  a.sign = plan_sign(p);
  a.dlo = p->omin;
  a.dhi = p->omax;
  a.span_max = p->spans[cand];
  a.slot_w = slot;
  a.out = out;
  a.out_kind = p->out_kind;
  a.out_stride = out_stride;
  a.out_start = out_start;
  a.nvalid = g.nvalid;
  a.status = reinterpret_cast<uint32_t*>(ws);
  a.special = special;
  rc = launch_dmt(v, a, g.ntiles_t, p->ndm, st);
  if (rc) return rc;
  if (p->timing) cudaEventRecord(ev[2], st);
  return SPP_OK;
}

int spp_dmt_plan_timing(spp_dmt_plan* p, int enable) {
  if (!p) return fail(SPP_ERR_ARG, "null plan");
  p->timing = enable != 0;
  p->evused = 0;
  return SPP_OK;
}

int spp_dmt_plan_timing_read(spp_dmt_plan* p, double* ms_corner_turn, double* ms_dmt,
                             int32_t* nexec) {
  if (!p || !ms_corner_turn || !ms_dmt || !nexec) return fail(SPP_ERR_ARG, "null pointer");
  double a = 0.0, b = 0.0;
  const size_t n = p->evused / 3;
  for (size_t i = 0; i < n; ++i) {
    float x = 0.f, y = 0.f;
    int rc = cuda_status(cudaEventSynchronize(p->evpool[3 * i + 2]), "event sync");
    if (rc) return rc;
    rc = cuda_status(cudaEventElapsedTime(&x, p->evpool[3 * i], p->evpool[3 * i + 1]), "elapsed");
    if (rc) return rc;
    rc = cuda_status(cudaEventElapsedTime(&y, p->evpool[3 * i + 1], p->evpool[3 * i + 2]), "elapsed");
    if (rc) return rc;
    a += x;
    b += y;
  }
  *ms_corner_turn = a;
  *ms_dmt = b;
  *nexec = (int32_t)n;
  return SPP_OK;
}

int spp_dmt_execute(const spp_dmt_plan* p, const void* in, int64_t nsamps, void* out,
                    int64_t out_stride, int64_t out_start, void* workspace,
                    int64_t workspace_bytes, void* stream) {
  if (!p || !in || !out || !workspace) return fail(SPP_ERR_ARG, "spp_dmt_execute: null pointer");
  if (nsamps <= 0 || nsamps > p->nsamps_max)
    return fail(SPP_ERR_SIZE, "nsamps %lld outside (0, %lld]", (long long)nsamps, (long long)p->nsamps_max);
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0)
    return fail(SPP_ERR_ALIGN, "workspace must be 256-B aligned");
  return dmt_run(p, in, nsamps, out, out_stride, out_start, static_cast<uint8_t*>(workspace),
                 workspace_bytes, as_stream(stream));
}

int64_t spp_dmt_plan_zero_dm_workspace_bytes(const spp_dmt_plan* p, int64_t nsamps) {
  if (!p) return -1;
  return spp_dmt_plan_workspace_bytes(p, nsamps) + round_up(nsamps * 8, 256);
}

int spp_dmt_execute_zero_dm(const spp_dmt_plan* p, const float* in, int64_t nsamps,
                            const float* bpass, const float* chanwts, void* out,
                            int64_t out_stride, int64_t out_start, void* workspace,
                            int64_t workspace_bytes, void* stream) {
  if (!p || !in || !bpass || !chanwts || !out || !workspace) return fail(SPP_ERR_ARG, "null pointer");
  if (p->nbits != 32) return fail(SPP_ERR_UNSUPPORTED, "zero-DM fusion needs float32 input");
  if (nsamps <= 0 || nsamps > p->nsamps_max) return fail(SPP_ERR_SIZE, "nsamps out of range");
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return fail(SPP_ERR_ALIGN, "workspace must be 256-B aligned");
  const int64_t need = spp_dmt_plan_zero_dm_workspace_bytes(p, nsamps);
  if (workspace_bytes < need) return fail(SPP_ERR_SIZE, "workspace %lld < %lld", (long long)workspace_bytes, (long long)need);
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  double* rows = reinterpret_cast<double*>(ws + spp_dmt_plan_workspace_bytes(p, nsamps));
  return dmt_run(p, in, nsamps, out, out_stride, out_start, ws, workspace_bytes, as_stream(stream),
                 bpass, chanwts, rows);
}

// --- end-to-end from host buffers ------------------------------------------------
static int64_t host_row_bytes(const spp_dmt_plan* p) {
  return p->nbits == 32 ? p->nchans * 4 : p->nchans * p->nbits / 8;
}

struct HostLayout {
  int64_t in_rows, in_bytes, out_bytes, run_bytes, set_bytes;
};

static HostLayout host_layout(const spp_dmt_plan* p, int64_t block) {
  HostLayout h{};
  h.in_rows = block + p->maxabs;
  h.in_bytes = round_up(h.in_rows * host_row_bytes(p), 256);
  h.out_bytes = round_up(p->ndm * block * 4, 256);
  h.run_bytes = round_up(spp_dmt_plan_workspace_bytes(p, h.in_rows), 256);
  h.set_bytes = h.in_bytes + h.out_bytes + h.run_bytes;
  return h;
}

// Host streaming keeps this many block buffer sets (and streams) in flight:
// copies in, DM kernel and copies out of consecutive blocks overlap.
constexpr int kHostSets = 3;

int64_t spp_dmt_host_workspace_bytes(const spp_dmt_plan* p, int64_t block_nsamps) {
  if (!p || block_nsamps <= 0) return -1;
  return kStatusBytes + kHostSets * host_layout(p, block_nsamps).set_bytes;
}

int spp_dmt_execute_host(const spp_dmt_plan* p, const void* in_host, int64_t nsamps,
                         void* out_host, int64_t out_stride, int64_t block_nsamps,
                         void* workspace, int64_t workspace_bytes) {
  if (!p || !in_host || !out_host || !workspace) return fail(SPP_ERR_ARG, "null pointer");
  if (p->mode != SPP_MODE_DEDISPERSE || p->omin < 0)
    return fail(SPP_ERR_UNSUPPORTED, "host streaming needs dedisperse mode and delays >= 0");
  if (block_nsamps <= 0) return fail(SPP_ERR_ARG, "block_nsamps <= 0");
  const int64_t nvalid = plan_nvalid(p, nsamps);
  if (nvalid <= 0) return SPP_OK;
  if (out_stride < nvalid) return fail(SPP_ERR_SIZE, "out_stride < nvalid");
  const HostLayout h = host_layout(p, block_nsamps);
  if (h.in_rows > p->nsamps_max)
    return fail(SPP_ERR_SIZE, "block + max delay (%lld) exceeds plan nsamps_max", (long long)h.in_rows);
  if (workspace_bytes < kStatusBytes + kHostSets * h.set_bytes)
    return fail(SPP_ERR_SIZE, "workspace too small");
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0) return fail(SPP_ERR_ALIGN, "workspace must be 256-B aligned");
  uint8_t* ws = static_cast<uint8_t*>(workspace);
  cudaStream_t s[kHostSets];
  int rc = SPP_OK;
  for (int i = 0; i < kHostSets; ++i) {
    rc = cuda_status(cudaStreamCreateWithFlags(&s[i], cudaStreamNonBlocking), "stream create");
    if (rc) {
      for (int j = 0; j < i; ++j) cudaStreamDestroy(s[j]);
      return rc;
    }
  }
  const int64_t rb = host_row_bytes(p);
  const int64_t es = 4;
  const int64_t nblocks = ceil_div(nvalid, block_nsamps);
  // each buffer set's run workspace starts with the device status words of
  // the kernels it hosts: cleared here, read back once everything finished
  for (int k = 0; k < kHostSets && rc == SPP_OK; ++k)
    rc = cuda_status(cudaMemsetAsync(ws + kStatusBytes + k * h.set_bytes + h.in_bytes + h.out_bytes,
                                     0, 16, s[k]),
                     "status clear");
  for (int64_t b = 0; b < nblocks && rc == SPP_OK; ++b) {
    const int k = (int)(b % kHostSets);
    uint8_t* set = ws + kStatusBytes + k * h.set_bytes;
    uint8_t* d_in = set;
    uint8_t* d_out = set + h.in_bytes;
    uint8_t* d_run = set + h.in_bytes + h.out_bytes;
    const int64_t t0 = b * block_nsamps;
    const int64_t nout = std::min(block_nsamps, nvalid - t0);
    const int64_t rows = nout + p->maxabs;
    rc = cuda_status(cudaMemcpyAsync(d_in, static_cast<const uint8_t*>(in_host) + t0 * rb,
                                     rows * rb, cudaMemcpyHostToDevice, s[k]), "H2D");
    if (rc) break;
    rc = dmt_run(p, d_in, rows, d_out, nout, 0, d_run, h.run_bytes, s[k]);
    if (rc) break;
    rc = cuda_status(cudaMemcpy2DAsync(static_cast<uint8_t*>(out_host) + t0 * es, out_stride * es,
                                       d_out, nout * es, nout * es, p->ndm,
                                       cudaMemcpyDeviceToHost, s[k]), "D2H");
  }
  for (int i = 0; i < kHostSets; ++i) {
    int r2 = cuda_status(cudaStreamSynchronize(s[i]), "stream sync");
    if (!rc) rc = r2;
    cudaStreamDestroy(s[i]);
  }
  for (int k = 0; k < kHostSets && rc == SPP_OK; ++k) {
    uint32_t words[4] = {0, 0, 0, 0};
    rc = cuda_status(cudaMemcpy(words, ws + kStatusBytes + k * h.set_bytes + h.in_bytes + h.out_bytes,
                                16, cudaMemcpyDeviceToHost),
                     "status copy");
    if (rc == SPP_OK && words[0] != 0)
      rc = fail(SPP_ERR_DEVICE, "device status 0x%x (block %u, detail 0x%x)", words[0], words[1],
                words[2]);
  }
  return rc;
}

}  // extern "C"
