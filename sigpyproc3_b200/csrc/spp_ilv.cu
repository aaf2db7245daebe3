// DM-time transform over interleaved bit planes (integer data, 1-8 bit).
//
// Layout.  An output row of nvalid samples is cut into 32 runs of M words:
// bit i of word w stands for sample i * M + w.  A channel's row holds, for
// every word w in [lo, lo + M + ext), the NB bit planes of samples
// i * M + w (i = 0..31), plane words next to each other.  A trial that shifts
// the channel by o samples then reads word w + o: the shift is an address
// offset, so the bit-sliced adders take the loaded words as they are.  (With
// 32 consecutive samples per word every plane word needs a funnel shift,
// which runs at half the rate of the logic that adds it and takes a second
// shared load for the neighbouring word.)  The price is that a row is longer
// than M words by the range of the channel's delays over the trials (ext).
//
// Rows may hold sums of two channels (2k, 2k+1) at one relative offset r:
// S[w] = x[2k][w] + x[2k+1][w + r], NB + 1 planes, shared by every trial whose
// delays differ by r there.
//
// k_ilv: one CTA = DW trials x W words (32 W samples).  A producer warp copies,
// per slab of 4 NQ groups, the distinct rows the tile's trials read (bulk
// copies, mbarrier ring); where each trial reads inside them does not depend
// on the word tile, so the plan tabulates it once.  Consumer warps (one trial,
// 32 P words each) run the carry-save network of spp_dmt.cuh and write 32
// samples per word as 32 coalesced stores.
#include <algorithm>
#include <climits>

#include "spp_dmt.cuh"
#include "spp_ilv.h"

namespace spp {

namespace {

constexpr int kIlvMaxEnt = 32;   // staged rows per slab: one producer lane each
constexpr int64_t kIlvMaxSmem = 227 * 1024;

struct IlvArgs {
  const uint32_t* rows;   // rows of NP-plane words
  const uint32_t* zero;   // W zero words (NP planes), for absent groups
  int64_t mp;             // words per row without its extra words
  int64_t M;              // output words
  const int32_t* off;
  const int4* ent;
  int32_t emax, nslab, stages, stage_bytes;
  int32_t ndt, njt, db;   // trial tiles, word tiles, trial tiles per block of the CTA order
  int32_t ndm;
  void* out;
  int32_t out_kind;
  int64_t out_stride, out_start, nvalid;
  uint32_t* status;
};

// Levels of the network: a quad of NP-plane rows leaves one carry of weight
// 2^ilv_quad(NP) (4 x (2^NP - 1) < 2^(NP + 2); two levels for one plane).
__host__ __device__ constexpr int ilv_quad(int np) { return np == 1 ? 2 : np + 2; }

// Where a thread reads one row: its word's address, and for NP = 8 that of the
// word's second 16 bytes.  Even plane counts use 8- or 16-byte loads; a warp's
// 32 consecutive words are conflict-free for every NP (for NP = 8 the two
// 16-byte halves of a word are swapped in every second group of four words,
// which keeps eight lanes on distinct banks).  The words 32 apart that a thread
// owns are reached by load immediates.
template <int NP>
struct IlvRow {
  static constexpr int kStep = NP == 8 ? 4 : NP;  // planes fetched at a time
  const unsigned char* p[NP == 8 ? 2 : 1];
  __device__ __forceinline__ void set(const unsigned char* stage, uint32_t a) {
    if constexpr (NP == 8) {
      const uint32_t z = a ^ ((a >> 3) & 16u);
      p[0] = stage + z;
      p[1] = stage + (z ^ 16u);
    } else {
      p[0] = stage + a;
    }
  }
  template <int H>
  __device__ __forceinline__ void load(int imm, uint32_t (&x)[kStep]) const {
    const unsigned char* q = p[H] + imm;
    if constexpr (NP % 4 == 0) {
      const uint4 v = *reinterpret_cast<const uint4*>(q);
      x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
    } else if constexpr (NP % 2 == 0) {
#pragma unroll
      for (int b = 0; b < NP; b += 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(q + 4 * b);
        x[b] = v.x; x[b + 1] = v.y;
      }
    } else {
#pragma unroll
      for (int b = 0; b < NP; ++b) x[b] = *reinterpret_cast<const uint32_t*>(q + 4 * b);
    }
  }
};

// Level B of a quad of rows: the four plane-B words and the carries of the
// level below, added into A[B] in pairs (an odd one through a half adder).
// Planes are fetched kStep at a time, when their first level is reached.
template <int NP, int B, int NCIN>
struct IlvLevel {
  template <int LR>
  __device__ __forceinline__ static void run(uint32_t (&A)[LR], const IlvRow<NP> (&r)[4], int imm,
                                             uint32_t (&x)[4][IlvRow<NP>::kStep],
                                             const uint32_t* cin, uint32_t& out) {
    constexpr int KS = IlvRow<NP>::kStep;
    if constexpr (B < NP && B % KS == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) r[q].template load<B / KS>(imm, x[q]);
    }
    constexpr int NPL = B < NP ? 4 : 0;
    constexpr int NIN = NPL + NCIN;
    constexpr int NOUT = (NIN + 1) / 2;
    uint32_t w[NIN], co[NOUT];
#pragma unroll
    for (int q = 0; q < NPL; ++q) w[q] = x[q][B % KS];
#pragma unroll
    for (int k = 0; k < NCIN; ++k) w[NPL + k] = cin[k];
#pragma unroll
    for (int k = 0; k < NIN / 2; ++k) csa(A[B], w[2 * k], w[2 * k + 1], co[k]);
    if constexpr (NIN & 1) half(A[B], w[NIN - 1], co[NOUT - 1]);
    if constexpr (NOUT == 1 && B + 1 >= NP) {
      static_assert(B + 1 == ilv_quad(NP), "quad carry level");
      out = co[0];
    } else {
      IlvLevel<NP, B + 1, NOUT>::run(A, r, imm, x, co, out);
    }
  }
};

// 16 x 16 bit transposes of both half-words at once: v[l] bit i -> v[i] bit l
// (i < 16, and i - 16 in the upper half).
__device__ __forceinline__ void transpose16x2(uint32_t (&v)[16]) {
#pragma unroll
  for (int s = 8; s >= 1; s >>= 1) {
    const uint32_t m = s == 8 ? 0x00FF00FFu : s == 4 ? 0x0F0F0F0Fu : s == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
    for (int l = 0; l < 16; ++l) {
      if (l & s) continue;
      const uint32_t a = v[l], b = v[l + s];
      v[l] = (a & m) | ((b & m) << s);
      v[l + s] = ((a >> s) & m) | (b & ~m);
    }
  }
}

template <int NP, int P, int DW, int TW, int NQ, int L, int LR>
__device__ __forceinline__ void ilv_body(const IlvArgs& a) {
  constexpr int NWC = DW * TW;
  constexpr int W = TW * 32 * P;
  constexpr int LQ = ilv_quad(NP);
  constexpr int LS = NQ == 1 ? 0 : NQ == 2 ? 1 : 2;  // folds within a slab
  constexpr int LF = LQ + LS;                        // level of a slab's one carry
  static_assert(LR <= L && LF + 2 <= LR, "register levels hold the folded carries");

  extern __shared__ __align__(256) unsigned char smem[];
  constexpr int nq4 = 4 * NQ;
  int32_t* soff = reinterpret_cast<int32_t*>(smem + (int64_t)a.stages * a.stage_bytes);
  uint32_t* shi = reinterpret_cast<uint32_t*>(soff + a.stages * DW * nq4);
  uint64_t* full = reinterpret_cast<uint64_t*>(shi + (L - LR) * P * NWC * 32);
  uint64_t* empty = full + a.stages;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // CTA order: blocks of db trial tiles sweep the word tiles together, so that
  // the windows of neighbouring trials overlap in L2
  const int blk = blockIdx.x / (a.db * a.njt);
  const int rem = blockIdx.x - blk * a.db * a.njt;
  const int dcnt = min(a.db, a.ndt - blk * a.db);
  const int jt = rem / dcnt;
  const int dt = blk * a.db + (rem - jt * dcnt);
  const int64_t j0 = (int64_t)jt * W;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], NWC);
    }
    fence_mbar_init();
  }
  __syncthreads();

  if (warp == NWC) {
    // producer: lane e copies row entry e of the slab
    const int32_t* toff = a.off + (int64_t)dt * a.nslab * DW * nq4;
    const int4* tent = a.ent + (int64_t)dt * a.nslab * a.emax;
    int s = 0;
    uint32_t ph = 1;  // parity of the phase before the first: passes at once
    for (int k = 0; k < a.nslab; ++k) {
      const int4 en = lane < a.emax ? __ldg(tent + (int64_t)k * a.emax + lane) : make_int4(-1, 0, 0, 0);
      const uint32_t bytes = en.x == -1 ? 0u : (uint32_t)en.z * (NP * 4);
      const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
      if (k >= a.stages && !mbar_wait(&empty[s], ph, a.status)) break;
      if (lane == 0) {
        mbar_arrive_expect_tx(&full[s], total + (uint32_t)(DW * nq4 * 4));
        bulk_g2s(soff + s * DW * nq4, toff + (int64_t)k * DW * nq4, DW * nq4 * 4, &full[s]);
      }
      __syncwarp();
      if (bytes) {
        const uint32_t* src = en.x < 0 ? a.zero : a.rows + ((int64_t)en.x * a.mp + en.y + j0) * NP;
        bulk_g2s(smem + (int64_t)s * a.stage_bytes + (int64_t)en.w * 4, src, bytes, &full[s]);
      }
      if (++s == a.stages) { s = 0; ph ^= 1; }
    }
    return;
  }

  // consumers: warp (trial dmw, word group tw); thread words 32 p + lane
  const int dmw = warp / TW, tw = warp % TW;
  const int dm = dt * DW + dmw;
  const int wl = tw * 32 * P + lane;
  const uint32_t wb = (uint32_t)wl * (NP * 4);
  const int ct = threadIdx.x;
  auto hi = [&](int l, int p) -> uint32_t& { return shi[((l - LR) * P + p) * (NWC * 32) + ct]; };
#pragma unroll
  for (int l = LR; l < L; ++l)
#pragma unroll
    for (int p = 0; p < P; ++p) hi(l, p) = 0u;
  uint32_t A[P][LR];
#pragma unroll
  for (int p = 0; p < P; ++p)
#pragma unroll
    for (int l = 0; l < LR; ++l) A[p][l] = 0u;
  auto ripple = [&](int p, int l0, uint32_t c) {
#pragma unroll
    for (int l = 0; l < LR; ++l) {
      if (l < l0) continue;
      uint32_t nc;
      half(A[p][l], c, nc);
      c = nc;
    }
#pragma unroll
    for (int l = LR; l < L; ++l) {
      if (c == 0u) break;
      uint32_t& h = hi(l, p);
      const uint32_t nc = h & c;
      h ^= c;
      c = nc;
    }
  };
  // quad carries are folded in pairs: log2(NQ) levels within a slab, two more
  // over slabs, then one ripple per four slabs
  uint32_t h0[P], h1[P];
  bool ok = true;
  int s = 0;
  uint32_t ph = 0;
  for (int k = 0; k < a.nslab; ++k) {
    if (!mbar_wait(&full[s], ph, a.status)) { ok = false; break; }
    const unsigned char* base = smem + s * a.stage_bytes;
    const int4* off = reinterpret_cast<const int4*>(soff + (s * DW + dmw) * nq4);
    int4 o[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) o[i] = off[i];
    uint32_t c0[P], c1[P];
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
      IlvRow<NP> r[4];
      r[0].set(base, (uint32_t)o[i].x + wb);
      r[1].set(base, (uint32_t)o[i].y + wb);
      r[2].set(base, (uint32_t)o[i].z + wb);
      r[3].set(base, (uint32_t)o[i].w + wb);
#pragma unroll
      for (int p = 0; p < P; ++p) {
        uint32_t x[4][IlvRow<NP>::kStep], cq;
        IlvLevel<NP, 0, 0>::run(A[p], r, p * 32 * NP * 4, x, nullptr, cq);
        if (i % 2 == 0) {
          c0[p] = cq;
        } else {
          csa(A[p][LQ], c0[p], cq, c0[p]);
          if (i == 1) c1[p] = c0[p];
          else if (i == 3) csa(A[p][LQ + 1], c1[p], c0[p], c0[p]);
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (++s == a.stages) { s = 0; ph ^= 1; }
    if (!(k & 1)) {
#pragma unroll
      for (int p = 0; p < P; ++p) h0[p] = c0[p];
    } else {
#pragma unroll
      for (int p = 0; p < P; ++p) csa(A[p][LF], h0[p], c0[p], c0[p]);
      if (!(k & 2)) {
#pragma unroll
        for (int p = 0; p < P; ++p) h1[p] = c0[p];
      } else {
#pragma unroll
        for (int p = 0; p < P; ++p) {
          uint32_t c2;
          csa(A[p][LF + 1], h1[p], c0[p], c2);
          ripple(p, LF + 2, c2);
        }
      }
    }
  }
  if (!ok || dm >= a.ndm) return;
#pragma unroll
  for (int p = 0; p < P; ++p) {
    if (a.nslab & 1) ripple(p, LF, h0[p]);
    if (a.nslab & 2) ripple(p, LF + 1, h1[p]);
  }
  // sample i * M + j of word j = bit i: 32 stores per word, each a warp's
  // consecutive samples
  const int64_t obase = (int64_t)dm * a.out_stride + a.out_start;
#pragma unroll 1
  for (int p = 0; p < P; ++p) {
    const int64_t j = j0 + wl + 32 * p;
    if (j >= a.M) break;
    uint32_t v[16], up[L > 16 ? L - 16 : 1];
#pragma unroll
    for (int pp = 0; pp < P; ++pp) {  // register arrays need a static index
      if (pp != p) continue;
#pragma unroll
      for (int l = 0; l < 16; ++l) v[l] = l < LR ? A[pp][l < LR ? l : 0] : l < L ? hi(l, pp) : 0u;
#pragma unroll
      for (int l = 16; l < L; ++l) up[l - 16] = l < LR ? A[pp][l < LR ? l : 0] : hi(l, pp);
    }
    transpose16x2(v);
    // the first `cnt` of the word's 32 samples lie inside the row
    const int cnt = j < a.nvalid ? (int)((a.nvalid - 1 - j) / a.M) + 1 : 0;
    auto emit = [&](auto* dst, auto conv) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        uint32_t c = i < 16 ? (v[i & 15] & 0xFFFFu) : (v[i & 15] >> 16);
#pragma unroll
        for (int l = 16; l < L; ++l) c |= ((up[l - 16] >> i) & 1u) << l;
        if (i < cnt) *dst = conv(c);
        dst += a.M;
      }
    };
    if (a.out_kind == SPP_OUT_I32)
      emit(static_cast<int32_t*>(a.out) + obase + j, [](uint32_t c) { return (int32_t)c; });
    else
      emit(static_cast<float*>(a.out) + obase + j, [](uint32_t c) { return (float)c; });
  }
}

template <int NP, int P, int DW, int TW, int NQ, int L, int LR, int MINB>
__global__ void __launch_bounds__((DW * TW + 1) * 32, MINB)
k_ilv(const IlvArgs a) {
  ilv_body<NP, P, DW, TW, NQ, L, LR>(a);
}

// ---------------------------------------------------------------------------
// Raw block -> channel rows.  A CTA owns 256 / NB channels (32 bytes of a raw
// row) and walks tiles of 8 words w in [lo, lo + M): it loads the raw rows
// i * M + w (whole 32-byte sectors, the next tile's loads in flight during this
// one) and bit-transposes 32 rows x 32 bits per warp step, which gives the
// words of i = 0..31 (block 0) and, where rows run past M words, of
// i = 32..63 (block 1) and so on.  Word w + q M is block q / 32 and the next
// one funnel-shifted by q mod 32, so every raw row is read and transposed once
// however long the rows are.  Each channel's 8 words x NB planes leave as one
// contiguous run.  Bound by the transposes (shuffles and logic) and the row
// stores.  LONG: rows of more than 32 M words beside the outputs', whose further
// blocks are loaded as the first two are, one ahead (2-bit, 4096 channels, delays
// to 32402: 128 words 232 -> 180 us, 32 words 699 -> 185 us when they were read
// byte by byte); a kernel of its own, since its registers cost the others a
// fifth of their rate.
// ---------------------------------------------------------------------------
template <int NB, bool LONG>
__global__ void __launch_bounds__(256)
k_ilv_turn(const uint8_t* __restrict__ raw, int64_t nchans, int64_t nsamps, int bitorder,
           int64_t M, int64_t mp, const int32_t* __restrict__ lo, const int32_t* __restrict__ ext,
           uint32_t* __restrict__ rows) {
  constexpr int CC = planes_ct_chans(NB);
  constexpr int RT = 256;
  constexpr int SBP = 36;
  constexpr int OP = 8 * NB + 4;  // words per channel in s_out
  __shared__ __align__(16) uint8_t s_raw[2][RT * SBP];
  __shared__ __align__(16) uint32_t s_out[2][CC * OP];
  __shared__ int s_rng[2];
  const int64_t c0 = (int64_t)blockIdx.x * CC;
  const int nc = (int)((nchans - c0) < CC ? (nchans - c0) : CC);
  const int seg = (nc * NB + 7) / 8;
  const int64_t rowbytes = nchans * NB / 8;
  const int64_t segstart = c0 * NB / 8;
  const bool vec16 = seg == 32 && (rowbytes & 15) == 0 && (reinterpret_cast<uintptr_t>(raw) & 15) == 0;
  if (threadIdx.x == 0) { s_rng[0] = INT_MAX; s_rng[1] = INT_MIN; }
  __syncthreads();
  for (int c = threadIdx.x; c < nc; c += blockDim.x) {
    const int l = lo[c0 + c];
    atomicMin(&s_rng[0], l);
    atomicMax(&s_rng[1], l + ext[c0 + c + 1] - ext[c0 + c]);
  }
  __syncthreads();
  const int64_t wlo = s_rng[0];
  const int64_t xw = s_rng[1] - wlo;  // words past M in the widest row of the group
  const int64_t ntile = M / 8;
  // each thread's two 16-byte output units: fixed channel, fixed place in the run
  int64_t odst[2];
  int64_t olo[2], ohi[2];
  int osrc[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int idx = threadIdx.x + u * 256;
    const int c = idx / (2 * NB), k = idx % (2 * NB);
    osrc[u] = c * OP + 4 * k;
    if (c < nc) {
      olo[u] = lo[c0 + c];
      ohi[u] = olo[u] + M + ext[c0 + c + 1] - ext[c0 + c];
      odst[u] = ((c0 + c) * mp + ext[c0 + c] - olo[u]) * NB + 4 * k;
    } else {
      olo[u] = INT_MAX; ohi[u] = INT_MIN; odst[u] = 0;
    }
  }
  const int lane = threadIdx.x & 31;
  const int bi = lane >> 3, bb = lane & 7;
  const int qc = (bitorder == SPP_BITORDER_BIG) ? (7 - bb) / NB : bb / NB;
  const int lc = bi * (8 / NB) + qc, lb = bb % NB;  // channel within the byte group, plane
  // tile row r = 32 w + i of block b holds raw row (32 b + i) * M + w; of block
  // b only the first `ni` rows are wanted
  auto fetch = [&](uint4 (&pre)[2], int64_t w0, int64_t b, int ni) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int idx = threadIdx.x + u * 256;
      const int r = idx >> 1, k = idx & 1;
      pre[u] = make_uint4(0u, 0u, 0u, 0u);
      if ((r & 31) >= ni) continue;
      const int64_t row = wrap_row((32 * b + (r & 31)) * M + w0 + (r >> 5), nsamps);
      if (row >= 0) pre[u] = __ldg(reinterpret_cast<const uint4*>(raw + row * rowbytes + segstart) + k);
    }
  };
  auto put = [&](const uint4 (&pre)[2], uint8_t* dst) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int idx = threadIdx.x + u * 256;
      uint32_t* d = reinterpret_cast<uint32_t*>(dst + (idx >> 1) * SBP + 16 * (idx & 1));
      d[0] = pre[u].x; d[1] = pre[u].y; d[2] = pre[u].z; d[3] = pre[u].w;
    }
  };
  auto fill = [&](uint8_t* dst, int64_t w0, int64_t b, int ni) {  // any alignment
    for (int idx = threadIdx.x; idx < RT * 32; idx += blockDim.x) {
      const int r = idx >> 5, k = idx & 31;
      uint8_t v = 0;
      if (k < seg && (r & 31) < ni) {
        const int64_t row = wrap_row((32 * b + (r & 31)) * M + w0 + (r >> 5), nsamps);
        if (row >= 0) v = __ldg(raw + row * rowbytes + segstart + k);
      }
      dst[r * SBP + k] = v;
    }
  };
  auto turn = [&](const uint8_t* src, uint32_t* dst) {  // warp = word, loop over 4-byte column groups
    const int w = threadIdx.x >> 5;
    // NB = 8: 16-byte halves swapped in every second group of four words
    const int b = NB == 8 ? lb ^ (w & 4) : lb;
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      uint32_t x = *reinterpret_cast<const uint32_t*>(src + (w * 32 + lane) * SBP + 4 * g);
      x = warp_transpose32(x, lane);
      dst[(4 * g * (8 / NB) + lc) * OP + w * NB + b] = x;
    }
  };
  // words past M of the tile at w0: q = 0..nq(w0), i.e. w0 + q M < wlo + M + xw
  const int m32 = (int)M, x32 = (int)xw;
  auto qmax = [&](int64_t w0) { return (m32 + x32 - 1 - (int)(w0 - wlo)) / m32; };
  auto rows_of = [&](int q, int b) {  // rows of block b that q <= qmax reaches
    return min(max(q - 32 * (b - 1), 0), 32);
  };
  uint4 pre0[2], pre1[2];
  if (vec16 && blockIdx.y < ntile) {
    const int64_t w0 = wlo + 8 * (int64_t)blockIdx.y;
    fetch(pre0, w0, 0, 32);
    fetch(pre1, w0, 1, rows_of(qmax(w0), 1));
  }
  for (int64_t tile = blockIdx.y; tile < ntile; tile += gridDim.y) {
    const int64_t w0 = wlo + 8 * tile;
    const int qm = qmax(w0);
    if (vec16) {
      put(pre0, s_raw[0]);
      if (qm > 0) put(pre1, s_raw[1]);
    } else {
      fill(s_raw[0], w0, 0, 32);
      if (qm > 0) fill(s_raw[1], w0, 1, rows_of(qm, 1));
    }
    __syncthreads();
    if (LONG && vec16 && qm >= 32) {
      fetch(pre0, w0, 2, rows_of(qm, 2));
    } else if (vec16 && tile + gridDim.y < ntile) {
      const int64_t w1 = w0 + 8 * (int64_t)gridDim.y;
      fetch(pre0, w1, 0, 32);
      fetch(pre1, w1, 1, rows_of(qmax(w1), 1));
    }
    turn(s_raw[0], s_out[0]);
    if (qm > 0) turn(s_raw[1], s_out[1]);
    __syncthreads();
    for (int b = 0;; ++b) {
      const uint32_t* sa = s_out[b & 1];
      const uint32_t* sb = s_out[(b + 1) & 1];
      const int q1 = min(qm, 32 * b + 31);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (olo[u] >= ohi[u]) continue;
        const uint4 x = *reinterpret_cast<const uint4*>(sa + osrc[u]);
        const uint4 y = *reinterpret_cast<const uint4*>(sb + osrc[u]);
        for (int q = 32 * b; q <= q1; ++q) {
          const int64_t w = w0 + q * M;
          if (w < olo[u] || w >= ohi[u]) continue;
          const int sh = q & 31;
          uint4 v;
          v.x = __funnelshift_r(x.x, y.x, sh);
          v.y = __funnelshift_r(x.y, y.y, sh);
          v.z = __funnelshift_r(x.z, y.z, sh);
          v.w = __funnelshift_r(x.w, y.w, sh);
          *reinterpret_cast<uint4*>(rows + odst[u] + w * NB) = v;
        }
      }
      if (qm < 32 * (b + 1)) break;
      // rows longer than 32 M words: the next block of 32 raw rows per word
      __syncthreads();
      if (LONG && vec16) {
        put(pre0, s_raw[0]);
        if (qm >= 32 * (b + 2)) {
          fetch(pre0, w0, b + 3, rows_of(qm, b + 3));
        } else if (tile + gridDim.y < ntile) {
          const int64_t w1 = w0 + 8 * (int64_t)gridDim.y;
          fetch(pre0, w1, 0, 32);
          fetch(pre1, w1, 1, rows_of(qmax(w1), 1));
        }
      } else {
        fill(s_raw[0], w0, b + 2, rows_of(qm, b + 2));
      }
      __syncthreads();
      turn(s_raw[0], s_out[b & 1]);
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// Pair rows: S[w] = x[2k][w] + x[2k+1][w + r] (ripple add of NB planes into
// NB + 1).  A CTA takes one pair and 512 words (1024 of 2-bit rows) and makes all of
// the pair's rows there: channel 2k's words stay in registers (two or four per
// thread), channel 2k+1's window in shared memory, so the channel rows are read
// once per pair and not once per row.  Each warp gathers its words in shared
// memory to store whole 16-byte units in order.  The rows' bounds are read into shared
// memory beside the window: read row by row they put a global load's latency
// into every step (4-bit, 1024 channels, 9553 rows of 1632 words: 138 -> 125 us;
// 2-bit, 4096 channels, 19038 rows of 31768 words: 1.98 -> 1.92 ms).  Bound by
// the row stores where rows are long; short blocks behind long delays are mostly
// CTAs that hold two rows or none, and twice the words per CTA of 2-bit rows takes
// 347 -> 270 us there (4096 outputs, delays to 32402; 262144 outputs: 750 -> 630).
// ---------------------------------------------------------------------------
template <int NB>
__device__ __forceinline__ void load_planes(const uint32_t* __restrict__ row, int64_t w, uint32_t (&x)[NB]) {
  if constexpr (NB == 8) {
    const uint4* p = reinterpret_cast<const uint4*>(row + w * 8);
    const int h = (int)(w >> 2) & 1;
    const uint4 a = __ldg(p + h), b = __ldg(p + (1 - h));
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  } else if constexpr (NB == 4) {
    const uint4 a = __ldg(reinterpret_cast<const uint4*>(row + w * 4));
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  } else {
    static_assert(NB == 2, "pair rows are sums of 2-, 4- and 8-bit channels");
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(row + w * 2));
    x[0] = a.x; x[1] = a.y;
  }
}

// words per thread: 4-bit and wider windows would leave fewer CTAs per SM
__host__ __device__ constexpr int pair_wpt(int nb) { return nb <= 2 ? 4 : 2; }
constexpr int kPairMaxOffsets = 512;  // distinct relative offsets of one pair, most
template <int NB>
__device__ __forceinline__ void load_planes_shared(const uint32_t* row, int w, uint32_t (&x)[NB]) {
  if constexpr (NB == 8) {
    const uint4* p = reinterpret_cast<const uint4*>(row + w * 8);
    const int h = (w >> 2) & 1;
    const uint4 a = p[h], b = p[1 - h];
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  } else if constexpr (NB == 4) {
    const uint4 a = *reinterpret_cast<const uint4*>(row + w * 4);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  } else {
    const uint2 a = *reinterpret_cast<const uint2*>(row + w * 2);
    x[0] = a.x; x[1] = a.y;
  }
}

template <int NB>
__global__ void __launch_bounds__(256)
k_ilv_pairs(const uint32_t* __restrict__ chan, int64_t mpc, const int32_t* __restrict__ clo,
            const int32_t* __restrict__ cext, int64_t M, const int32_t* __restrict__ rbase,
            const int32_t* __restrict__ roff, int64_t mpr, const int32_t* __restrict__ rlo,
            const int32_t* __restrict__ rext, int max_rows, uint32_t* __restrict__ rows) {
  constexpr int NP = NB + 1;
  constexpr int WPT = pair_wpt(NB), kPairWords = 256 * WPT, WW = 32 * WPT;  // words per thread, CTA, warp
  extern __shared__ __align__(16) uint32_t sm[];
  uint32_t* st = sm + (threadIdx.x >> 5) * WW * NP;  // this warp's words
  uint32_t* sy = sm + kPairWords * NP;               // channel 2k+1's window
  int3* srow = reinterpret_cast<int3*>(sy + (kPairWords + max_rows + 16) * NB);  // first word, end, extra words before
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = blockIdx.x, c = 2 * k;
  const int e0 = rbase[k], e1 = rbase[k + 1];
  const int r0 = roff[k];
  const int64_t alo = clo[c], alen = M + cext[c + 1] - cext[c];
  const int64_t blo = clo[c + 1], blen = M + cext[c + 2] - cext[c + 1];
  // words [w0, w0 + kPairWords) of channel 2k's grid; all offsets lie in its row
  const int64_t w0 = alo + (int64_t)blockIdx.y * kPairWords;
  if (w0 >= alo + alen) return;
  const uint32_t* a = chan + ((int64_t)c * mpc + cext[c]) * NB;
  const uint32_t* b = chan + ((int64_t)(c + 1) * mpc + cext[c + 1]) * NB;
  // window of channel 2k+1: from the 8-word group holding w0 + r0
  const int64_t y0 = (w0 + r0) & ~int64_t(7);
  const int yn = (int)((w0 + kPairWords + r0 + (e1 - e0) - y0 + 7) & ~int64_t(7));
  for (int e = e0 + threadIdx.x; e < e1; e += 256) {
    const int lo = rlo[e], x = rext[e];
    srow[e - e0] = make_int3(lo, lo + (int)M + rext[e + 1] - x, x);
  }
  for (int u = threadIdx.x; u < yn * NB / 4; u += 256) {
    const int64_t w = y0 - blo + u * 4 / NB;  // word of the unit's first value (in its row)
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (w >= 0 && w < blen) v = __ldg(reinterpret_cast<const uint4*>(b + (y0 - blo) * NB) + u);
    reinterpret_cast<uint4*>(sy)[u] = v;
  }
  uint32_t x[WPT][NB];
#pragma unroll
  for (int i = 0; i < WPT; ++i) {
    const int64_t w = w0 - alo + warp * WW + 32 * i + lane;
    if (w < alen) {
      load_planes<NB>(a, w, x[i]);
    } else {
#pragma unroll
      for (int q = 0; q < NB; ++q) x[i][q] = 0u;
    }
  }
  __syncthreads();
  const int64_t ww = w0 + warp * WW;  // this warp's first word
  for (int e = e0; e < e1; ++e) {
    const int3 row = srow[e - e0];
    const int64_t lo = row.x, hi = row.y;
    if (lo >= ww + WW || hi <= ww) continue;
    const int ys = (int)(ww + r0 + (e - e0) - y0);
#pragma unroll
    for (int i = 0; i < WPT; ++i) {
      uint32_t y[NB], o[NP];
      load_planes_shared<NB>(sy, ys + 32 * i + lane, y);
      uint32_t cy = 0u;
#pragma unroll
      for (int q = 0; q < NB; ++q) {
        o[q] = x[i][q] ^ y[q] ^ cy;
        cy = (x[i][q] & y[q]) | (x[i][q] & cy) | (y[q] & cy);
      }
      o[NB] = cy;
#pragma unroll
      for (int q = 0; q < NP; ++q) st[(lane + 32 * i) * NP + q] = o[q];
    }
    __syncwarp();
    // row bounds are multiples of 8 words = 2 NP units
    uint4* dst = reinterpret_cast<uint4*>(rows + (e * mpr + row.z + ww - lo) * NP);
    for (int u = lane; u < WW / 4 * NP; u += 32) {
      const int64_t w = ww + 8 * (u / (2 * NP));
      if (w >= lo && w < hi) dst[u] = reinterpret_cast<const uint4*>(st)[u];
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Plan tables, from the delay table on the device.
// ---------------------------------------------------------------------------
// One pass over the table: smallest and largest signed offset of every channel and
// relative offset of every pair, and the widest spread of a channel over tiles of
// four and of eight trials (per CTA).  A CTA takes 32 channels, its eight warps
// the tiles.
__global__ void __launch_bounds__(256)
k_ilv_scan(IlvDelays d, int2* __restrict__ chan, int2* __restrict__ pair, int2* __restrict__ spans) {
  __shared__ int2 red[8][32], redp[8][32], reds[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * 32 + lane;
  const bool on = c < d.nchans, two = !(lane & 1) && c + 1 < d.nchans;
  int mn = INT_MAX, mx = INT_MIN, pmn = INT_MAX, pmx = INT_MIN, s4 = 0, s8 = 0;
  for (int64_t t = warp; t * 8 < d.ndm; t += 8) {
    int o[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
      o[i] = on ? d.sign * __ldg(d.d_delays + min(t * 8 + i, d.ndm - 1) * d.nchans + c) : 0;
    int tn[2], tx[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      tn[h] = tx[h] = o[4 * h];
#pragma unroll
      for (int i = 1; i < 4; ++i) {
        tn[h] = min(tn[h], o[4 * h + i]);
        tx[h] = max(tx[h], o[4 * h + i]);
      }
      s4 = max(s4, tx[h] - tn[h]);
    }
    const int n8 = min(tn[0], tn[1]), x8 = max(tx[0], tx[1]);
    s8 = max(s8, x8 - n8);
    mn = min(mn, n8);
    mx = max(mx, x8);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = __shfl_down_sync(0xffffffffu, o[i], 1) - o[i];
      pmn = min(pmn, r);
      pmx = max(pmx, r);
    }
  }
  s4 = __reduce_max_sync(0xffffffffu, s4);
  s8 = __reduce_max_sync(0xffffffffu, s8);
  red[warp][lane] = make_int2(mn, mx);
  redp[warp][lane] = make_int2(pmn, pmx);
  if (lane == 0) reds[warp] = make_int2(s4, s8);
  __syncthreads();
  if (warp != 0) return;
  for (int w = 1; w < 8; ++w) {
    mn = min(mn, red[w][lane].x);
    mx = max(mx, red[w][lane].y);
    pmn = min(pmn, redp[w][lane].x);
    pmx = max(pmx, redp[w][lane].y);
    s4 = max(s4, reds[w].x);
    s8 = max(s8, reds[w].y);
  }
  if (on) chan[c] = make_int2(mn, mx);
  if (two) pair[c / 2] = make_int2(pmn, pmx);
  if (lane == 0) spans[blockIdx.x] = make_int2(s4, s8);
}

__device__ __forceinline__ int ilv_row_of(const IlvDelays& d, int G, const int32_t* rbase,
                                          const int32_t* rlo, int64_t dm, int64_t g, int* o) {
  const int32_t* row = d.d_delays + dm * d.nchans;
  if (G == 1) {
    *o = d.sign * row[g];
    return (int)g;
  }
  *o = d.sign * row[2 * g];
  return rbase[g] + (d.sign * row[2 * g + 1] - *o) - rlo[g];
}

// What plan creation reads back, in one copy.
constexpr int kIlvMaxShapes = 8;
struct IlvFoundRows {
  long long nrows, ext_total, max_ext, max_group;
  int max_offsets, ok;
};
struct IlvFound {
  IlvFoundRows rows[2];
  int omin, omax, span4, span8;
  int stats[2 * kIlvMaxShapes];  // per shape: most entries, most stage words
};

// Sum of the values of the threads before this one (1024 threads), and of all.
__device__ __forceinline__ long long block_before(long long v, long long* red, long long* all) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto scan = [&](long long x) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    return x;
  };
  const long long incl = scan(v);
  __syncthreads();
  if (lane == 31) red[warp] = incl;
  __syncthreads();
  const long long warps = scan(red[lane]);
  *all = __shfl_sync(0xffffffffu, warps, 31);
  const long long before = __shfl_sync(0xffffffffu, warps, warp - 1);
  return (warp ? before : 0) + incl - v;
}
// Largest value of the block in *to (shared, set before), once all threads pass a barrier.
__device__ __forceinline__ void block_largest(int v, int* to) {
  v = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) atomicMax(to, v);
}

// First word of a row of offsets mn..mx and its words beyond the common length.
__device__ __forceinline__ int row_first(int mn) { return mn & ~7; }
__device__ __forceinline__ long long row_extra(int mn, int mx) {
  return ((long long)mx - row_first(mn) + 8) & ~7ll;
}
constexpr long long kIlvMaxExtra = 1 << 30;  // of all rows of a grouping

// Words of a table's rows: where each part of a plan's words behind its delay
// table lies.
struct IlvWords {
  int2 *chan, *pair, *spans;  // k_ilv_scan's ranges
  int32_t *rmn, *rmx;         // offset ranges of pair rows
  IlvFound* found;
  int32_t *lo[2], *ext[2], *rbase, *rlo;
};

// One CTA of 1024 threads: channel rows, each pair's first row, and cleared ranges
// and sizes for the kernels that follow.  A thread takes a run of channels.  Row
// lengths are offsets' spreads plus up to 15 words: a spread above 2^30 counts as
// that, which is too many words in any case.
__global__ void __launch_bounds__(1024)
k_ilv_rows(int64_t nchans, int64_t nblk, int group, int64_t max_rows, int max_offsets, IlvWords w) {
  __shared__ long long red[32], redp[32];
  __shared__ int top[7];  // row words beyond the common length, -offset, offset, group span, spreads, pair rows
  const int tid = threadIdx.x;
  if (tid < 7) top[tid] = INT_MIN;
  __syncthreads();
  auto cap = [](long long v) { return (int)min(v, kIlvMaxExtra + 1); };
  const int64_t per = (nchans + 1023) / 1024;
  const int64_t a = min(tid * per, nchans), b = min(a + per, nchans);
  long long sum = 0;
  int most = 0, mn = INT_MAX, mx = INT_MIN;
  for (int64_t c = a; c < b; ++c) {
    const int2 r = w.chan[c];
    const long long x = row_extra(r.x, r.y);
    sum += x;
    most = max(most, cap(x));
    mn = min(mn, r.x);
    mx = max(mx, r.y);
  }
  long long total, run = block_before(sum, red, &total);
  for (int64_t c = a; c < b; ++c) {
    const int2 r = w.chan[c];
    w.lo[0][c] = row_first(r.x);
    w.ext[0][c] = (int32_t)run;
    run += row_extra(r.x, r.y);
  }
  int span = 0;  // words beside the common length that the rows of a turning CTA's channels cover
  for (int64_t g = tid; g * group < nchans; g += 1024) {
    long long first = LLONG_MAX, last = LLONG_MIN;
    for (int64_t c = g * group; c < min(nchans, (g + 1) * group); ++c) {
      const int2 r = w.chan[c];
      first = min(first, (long long)row_first(r.x));
      last = max(last, row_first(r.x) + row_extra(r.x, r.y));
    }
    span = max(span, cap(last - first));
  }
  int s4 = 0, s8 = 0;
  for (int64_t i = tid; i < nblk; i += 1024) {
    s4 = max(s4, w.spans[i].x);
    s8 = max(s8, w.spans[i].y);
  }
  // pairs: a row per relative offset
  const int64_t np = nchans % 2 ? 0 : nchans / 2;
  const int64_t pper = (np + 1023) / 1024;
  const int64_t pa = min(tid * pper, np), pb = min(pa + pper, np);
  long long rows = 0;
  int widest = 0;
  for (int64_t k = pa; k < pb; ++k) {
    const long long cnt = (long long)w.pair[k].y - w.pair[k].x + 1;
    rows += cnt;
    widest = max(widest, cap(cnt));
  }
  block_largest(most, top);
  block_largest(~mn, top + 1);
  block_largest(mx, top + 2);
  block_largest(span, top + 3);
  block_largest(s4, top + 4);
  block_largest(s8, top + 5);
  block_largest(widest, top + 6);
  long long nrows, first = block_before(rows, redp, &nrows);  // its barriers complete `top`
  const bool pairs = np > 0 && nrows <= max_rows && top[6] <= max_offsets;
  if (pairs) {
    for (int64_t k = pa; k < pb; ++k) {
      w.rbase[k] = (int32_t)first;
      w.rlo[k] = w.pair[k].x;
      first += (long long)w.pair[k].y - w.pair[k].x + 1;
    }
    for (int64_t i = tid; i < nrows; i += 1024) {
      w.rmn[i] = INT_MAX;
      w.rmx[i] = INT_MIN;
    }
  }
  if (tid < 2 * kIlvMaxShapes) w.found->stats[tid] = 0;
  if (tid != 0) return;
  w.ext[0][nchans] = (int32_t)total;
  if (pairs) w.rbase[np] = (int32_t)nrows;
  IlvFound* f = w.found;
  f->rows[0] = IlvFoundRows{nchans, total, top[0], top[3], 0, total <= kIlvMaxExtra};
  f->rows[1] = IlvFoundRows{pairs ? nrows : 0, 0, 0, 0, pairs ? top[6] : 0, pairs};
  f->omin = ~top[1];
  f->omax = top[2];
  f->span4 = top[4];
  f->span8 = top[5];
}

// Offset range of every pair row over the trials that read it.
__global__ void k_ilv_row_ranges(IlvDelays d, const int32_t* __restrict__ rbase,
                                 const int32_t* __restrict__ rlo, int32_t* __restrict__ mn,
                                 int32_t* __restrict__ mx, const IlvFound* __restrict__ found) {
  if (!found->rows[1].ok) return;
  const int64_t np = d.nchans / 2;
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= np) return;
  for (int64_t dm = blockIdx.y; dm < d.ndm; dm += gridDim.y) {
    int o;
    const int r = ilv_row_of(d, 2, rbase, rlo, dm, g, &o);
    atomicMin(mn + r, o);
    atomicMax(mx + r, o);
  }
}

// Pair rows from their offset ranges, as k_ilv_rows makes channel rows.
__global__ void __launch_bounds__(1024) k_ilv_pair_rows(IlvWords w) {
  __shared__ long long red[32];
  if (!w.found->rows[1].ok) return;
  const int tid = threadIdx.x;
  const int64_t n = w.found->rows[1].nrows, per = (n + 1023) / 1024;
  const int64_t a = min(tid * per, n), b = min(a + per, n);
  // an offset between two used ones that no trial has is never made
  auto extra = [](int mn, int mx) { return mn > mx ? 0ll : row_extra(mn, mx); };
  __shared__ int most;
  if (tid == 0) most = 0;
  long long sum = 0;
  int top = 0;
#pragma unroll 4
  for (int64_t i = a; i < b; ++i) {
    const long long x = extra(w.rmn[i], w.rmx[i]);
    sum += x;
    top = max(top, (int)min(x, kIlvMaxExtra + 1));
  }
  __syncthreads();
  block_largest(top, &most);
  long long total, run = block_before(sum, red, &total);  // its barriers complete `most`
#pragma unroll 4
  for (int64_t i = a; i < b; ++i) {
    const int mn = w.rmn[i], mx = w.rmx[i];
    w.lo[1][i] = mn > mx ? 1 << 30 : row_first(mn);
    w.ext[1][i] = (int32_t)run;
    run += extra(mn, mx);
  }
  if (tid != 0) return;
  w.ext[1][n] = (int32_t)total;
  w.found->rows[1].ext_total = total;
  w.found->rows[1].max_ext = most;
  w.found->rows[1].ok = total <= kIlvMaxExtra;
}

// Staging tables: a lane per group of a (trial tile, slab), whose 4 nq lanes sit in
// one warp and place their rows by a scan over it.  A thread per slab walked its
// groups one after the other: 15 to 37 us for the sizes of plans of any size, 17 to
// 30 us for the tables; 8 to 10 and 7 to 14 us.  Without `off` only the largest entry count and
// stage size are taken (stats[0], stats[1] in words).
struct IlvTableShape {
  int G, np, DW, W, nq;
  int64_t ntile, nslab;
  const int32_t *lo, *ext, *rbase, *rlo;
};
__device__ __forceinline__ void ilv_table(const IlvDelays& d, const IlvTableShape& sh, int64_t thread, int emax,
                                          int32_t* __restrict__ off, int4* __restrict__ ent,
                                          int* __restrict__ stats) {
  const int np = sh.np, DW = sh.DW, W = sh.W, nl = 4 * sh.nq;  // 4, 8 or 16 lanes
  const int32_t *lo = sh.lo, *ext = sh.ext;
  const int64_t id = thread / nl;
  if (id >= sh.ntile * sh.nslab) return;
  const int j = (int)(thread - id * nl), lane = threadIdx.x & 31;
  const uint32_t slab_lanes = ((1u << nl) - 1u) << (lane - j);
  const int64_t tile = id / sh.nslab, k = id - tile * sh.nslab;
  const int64_t ng = d.nchans / sh.G, g = k * nl + j;
  const bool on = g < ng, pad = !on && (j == 0 || g - 1 < ng);  // the slab's one zero row
  int o[16], rr[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    o[i] = rr[i] = 0;
    if (on && i < DW)
      rr[i] = ilv_row_of(d, sh.G, sh.rbase, sh.rlo, min(tile * DW + i, d.ndm - 1), g, &o[i]);
  }
  // rows of the group, in the order of their first trial: fn(trials, row, word, words)
  auto each_row = [&](auto&& fn) {
    uint32_t left = on ? (1u << DW) - 1u : 0u;
    while (left) {
      const int f = __ffs(left) - 1;
      const int r = rr[f];
      uint32_t same = 0;
      int mn = INT_MAX, mx = INT_MIN;
      for (int i = f; i < DW; ++i) {
        if (rr[i] != r) continue;
        same |= 1u << i;
        mn = min(mn, o[i]);
        mx = max(mx, o[i]);
      }
      left &= ~same;
      const int start = (mn - lo[r]) & ~7;  // words from the row's first, 8-word groups
      fn(same, r, start, (W + (mx - lo[r] - start) + 7) & ~7);
    }
  };
  // a spread that no stage can hold: the sum stays below overflow
  auto words_of = [&](int len) { return min(len, 1 << 20) * np; };
  int e = pad ? 1 : 0, pos = pad ? W * np : 0;
  each_row([&](uint32_t, int, int, int len) {
    ++e;
    pos = min(pos + words_of(len), 1 << 24);
  });
  const int own_e = e, own_pos = pos;
  for (int s = 1; s < nl; s <<= 1) {
    const int xe = __shfl_up_sync(slab_lanes, e, s, nl), xp = __shfl_up_sync(slab_lanes, pos, s, nl);
    if (j >= s) {
      e += xe;
      pos += xp;
    }
  }
  if (stats && j == nl - 1) {  // the values only grow: most slabs find theirs no larger
    if (e > __ldcg(&stats[0])) atomicMax(&stats[0], e);
    if (pos > __ldcg(&stats[1])) atomicMax(&stats[1], pos);
  }
  if (!off) return;
  const int all = __shfl_sync(slab_lanes, e, nl - 1, nl);
  e -= own_e;
  pos -= own_pos;
  int32_t* to = off + id * DW * nl + j;
  int4* en = ent + id * emax;
  if (!on) {
    const int zpos = pad ? pos : pos - W * np;
    if (pad && e < emax) en[e] = make_int4(-2, 0, W, zpos);
    for (int i = 0; i < DW; ++i) to[i * nl] = zpos * 4;
  }
  each_row([&](uint32_t same, int r, int start, int len) {
    if (e < emax) en[e] = make_int4(r, ext[r] + start, len, pos);
    for (int i = 0; i < DW; ++i)
      if (same >> i & 1) to[i * nl] = (pos + (o[i] - lo[r] - start) * np) * 4;
    ++e;
    pos += words_of(len);
  });
  for (int i = all + j; i < emax; i += nl) en[i] = make_int4(-1, 0, 0, 0);
}
constexpr int kIlvTableThreads = 128;
__global__ void __launch_bounds__(kIlvTableThreads)
k_ilv_tables(IlvDelays d, IlvTableShape sh, int emax, int32_t* __restrict__ off, int4* __restrict__ ent) {
  ilv_table(d, sh, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, emax, off, ent, nullptr);
}
// The sizes of several shapes at once (shape blockIdx.y).
struct IlvTableShapes {
  IlvTableShape s[kIlvMaxShapes];
};
__global__ void __launch_bounds__(kIlvTableThreads)
k_ilv_table_sizes(IlvDelays d, const __grid_constant__ IlvTableShapes sh, IlvFound* found) {
  const IlvTableShape& s = sh.s[blockIdx.y];
  if (!found->rows[0].ok || !found->rows[s.G - 1].ok) return;
  ilv_table(d, s, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, kIlvMaxEnt, nullptr, nullptr,
            found->stats + 2 * blockIdx.y);
}

template <int NB, int G, int P, int DW, int TW, int NQ, int LR, int MINB>
IlvCfg mki(double us_wave, double ns_group) {
  constexpr int NP = NB + (G == 2 ? 1 : 0);
  constexpr int L = NB == 8 ? 20 : NB == 4 ? 16 : 14;
  static_assert(DW <= 16, "trials per tile");
  static_assert((L - LR) * P * DW * TW * 32 * 4 % 8 == 0, "barriers follow the upper levels");
  IlvCfg c{};
  c.nb = NB; c.G = G; c.np = NP; c.P = P; c.DW = DW; c.TW = TW; c.nq = NQ;
  c.levels = L;
  c.threads = (DW * TW + 1) * 32;
  c.hi_bytes = (int64_t)(L - LR) * P * DW * TW * 32 * 4;
  c.us_wave = us_wave;
  c.ns_group = ns_group;
  c.fn = reinterpret_cast<const void*>(&k_ilv<NP, P, DW, TW, NQ, L, LR, MINB>);
  return c;
}

}  // namespace

const std::vector<IlvCfg>& ilv_cfgs() {
  static const std::vector<IlvCfg> v = {
      // <NB, G, P, DW, TW, NQ, register levels, CTAs per SM>(us per wave, ns per group).
      // One CTA per SM of 15 or 18 trial-warps (16 or 20 warps allocated: 128 or
      // 96 registers each): two thirds of the registers hold the counters, and
      // fewer, larger slabs of groups matter more than warps (2-bit pairs, 2^18 x
      // 1024 trials: slabs of 4 groups 14.4 ms, of 8 11.0 ms).  3 x 5 warps:
      // coarse trial grids, whose tiles of more trials would not fit the stages.
      mki<1, 1, 4, 11, 2, 4, 10, 1>(32, 97), mki<1, 1, 4, 9, 2, 4, 14, 1>(29, 86),
      mki<1, 1, 4, 15, 1, 4, 14, 1>(19, 81), mki<1, 1, 4, 3, 5, 4, 14, 1>(22, 83),
      mki<1, 1, 4, 3, 5, 2, 14, 1>(22, 95),
      mki<2, 2, 4, 9, 2, 2, 14, 1>(32, 190), mki<2, 2, 4, 15, 1, 2, 14, 1>(24, 160),
      mki<2, 2, 4, 7, 2, 2, 14, 1>(30, 150),
      mki<2, 1, 4, 15, 1, 4, 14, 1>(30, 101), mki<2, 1, 4, 9, 2, 4, 14, 1>(33, 141),
      mki<2, 1, 4, 3, 5, 4, 14, 1>(21, 103), mki<2, 1, 4, 3, 5, 2, 14, 1>(21, 115),
      mki<4, 2, 3, 7, 2, 2, 16, 1>(18, 174), mki<4, 2, 4, 9, 2, 1, 13, 1>(40, 312),
      mki<4, 2, 4, 15, 1, 1, 16, 1>(38, 254),
      mki<4, 1, 4, 15, 1, 2, 16, 1>(37, 174), mki<4, 1, 4, 7, 2, 2, 16, 1>(29, 181),
      mki<4, 1, 4, 3, 5, 2, 16, 1>(27, 184), mki<4, 1, 4, 3, 5, 1, 16, 1>(27, 200),
      mki<8, 2, 3, 7, 2, 1, 20, 1>(22, 307), mki<8, 2, 2, 9, 2, 1, 20, 1>(22, 273),
      mki<8, 2, 2, 3, 5, 1, 20, 1>(17, 247),
      mki<8, 1, 4, 15, 1, 1, 16, 1>(20, 363), mki<8, 1, 3, 7, 2, 2, 16, 1>(23, 258),
      mki<8, 1, 3, 15, 1, 1, 20, 1>(15, 279), mki<8, 1, 3, 3, 5, 1, 20, 1>(22, 284),
  };
  return v;
}

void ilv_free_tables(IlvTables* t) {
  if (t->own) cudaFree(t->d_off);
  t->d_off = nullptr;
  t->d_ent = nullptr;
  t->own = false;
}

// Device words a plan keeps behind its delay table: scratch of the passes that
// make its rows (ranges, sizes), and the rows of both groupings.
struct IlvWordOffsets {
  int64_t pair, spans, rmn, rmx, found, lo0, ext0, rbase, rlo, lo1, ext1, total;
  IlvWordOffsets(int64_t nchans, int64_t max_rows) {
    const int64_t np = nchans / 2;
    pair = 2 * nchans;
    spans = pair + 2 * np;
    rmn = spans + 2 * ceil_div(nchans, 32);
    rmx = rmn + max_rows;
    found = round_up(rmx + max_rows, 2);
    lo0 = found + (int64_t)(sizeof(IlvFound) / 4);
    ext0 = lo0 + nchans;
    rbase = ext0 + nchans + 1;
    rlo = rbase + np + 1;
    lo1 = rlo + np;
    ext1 = lo1 + max_rows;
    total = ext1 + max_rows + 1;
  }
};
int64_t ilv_plan_words(int64_t nchans, int64_t max_rows) { return IlvWordOffsets(nchans, max_rows).total; }

static IlvTableShape table_shape(const IlvCfg& c, const IlvDelays& d, const IlvRows& r) {
  return IlvTableShape{c.G, c.np, c.DW, c.words(), c.nq, ceil_div(d.ndm, c.DW),
                       ceil_div(d.nchans / c.G, 4 * c.nq), r.d_lo, r.d_ext, r.d_rbase, r.d_rlo};
}

static int64_t table_off_bytes(const IlvCfg& c, int64_t nchans, int64_t ndm) {
  return round_up(ceil_div(ndm, c.DW) * ceil_div(nchans / c.G, 4 * c.nq) * c.DW * 4 * c.nq * 4, 256);
}
static int64_t table_bytes(const IlvCfg& c, int64_t nchans, int64_t ndm, int emax) {
  return table_off_bytes(c, nchans, ndm) +
         ceil_div(ndm, c.DW) * ceil_div(nchans / c.G, 4 * c.nq) * emax * (int64_t)sizeof(int4);
}

int64_t ilv_table_bytes(const IlvCfg& c, const IlvDelays& d, const IlvTables& t) {
  return table_bytes(c, d.nchans, d.ndm, t.emax);
}

// Room for the staging tables of whichever shape a plan starts from: a slab's
// groups read a row each, pairs up to kIlvMaxEnt together.
int64_t ilv_table_room(int nb, int64_t nchans, int64_t ndm) {
  int64_t most = 0;
  for (const IlvCfg& c : ilv_cfgs())
    if (c.nb == nb && nchans % c.G == 0)
      most = std::max(most, table_bytes(c, nchans, ndm, c.G == 1 ? 4 * c.nq + 1 : kIlvMaxEnt));
  return most;
}

// Five kernels and one copy back: with the ranges on the host between them, plans
// of few channels and trials took 70 (8-bit) to 130 us (2-bit) longer than the
// allocation and the upload (256 channels x 64 trials: 480 us of 370 us, 441 us
// here; 1024 x 300: 640 -> 560 us).
int ilv_find(const std::vector<int>& which, const IlvDelays& d, int64_t max_rows, int32_t* words,
             IlvRange* range, IlvRows* rows, std::vector<IlvTables>* tabs) {
  if (reinterpret_cast<uintptr_t>(words) % sizeof(int2))  // ranges are stored as int2
    return fail(SPP_ERR_ARG, "interleaved rows: misaligned scratch");
  const int n = (int)which.size();
  if (n > kIlvMaxShapes) return fail(SPP_ERR_ARG, "more than %d interleaved shapes", kIlvMaxShapes);
  const int64_t np = d.nchans / 2, nblk = ceil_div(d.nchans, 32);
  const IlvWordOffsets at(d.nchans, max_rows);
  IlvWords w{};
  w.chan = reinterpret_cast<int2*>(words);
  w.pair = reinterpret_cast<int2*>(words + at.pair);
  w.spans = reinterpret_cast<int2*>(words + at.spans);
  w.rmn = words + at.rmn;
  w.rmx = words + at.rmx;
  w.found = reinterpret_cast<IlvFound*>(words + at.found);
  w.lo[0] = words + at.lo0;
  w.ext[0] = words + at.ext0;
  w.rbase = words + at.rbase;
  w.rlo = words + at.rlo;
  w.lo[1] = words + at.lo1;
  w.ext[1] = words + at.ext1;
  for (int g = 0; g < 2; ++g) {
    rows[g].G = g + 1;
    rows[g].d_lo = w.lo[g];
    rows[g].d_ext = w.ext[g];
  }
  rows[1].d_rbase = w.rbase;
  rows[1].d_rlo = w.rlo;
  k_ilv_scan<<<(unsigned)nblk, 256>>>(d, w.chan, w.pair, w.spans);
  k_ilv_rows<<<1, 1024>>>(d.nchans, nblk, planes_ct_chans(d.nb), max_rows, kPairMaxOffsets, w);
  bool pairs = false;
  IlvTableShapes sh{};
  int64_t most = 1;
  for (int i = 0; i < n; ++i) {
    const IlvCfg& c = ilv_cfgs()[which[i]];
    pairs = pairs || c.G == 2;
    sh.s[i] = table_shape(c, d, rows[c.G - 1]);
    most = std::max(most, sh.s[i].ntile * sh.s[i].nslab * 4 * c.nq);
  }
  if (pairs) {
    k_ilv_row_ranges<<<dim3((unsigned)ceil_div(np, 128), (unsigned)std::min<int64_t>(d.ndm, 64)), 128>>>(
        d, w.rbase, w.rlo, w.rmn, w.rmx, w.found);
    k_ilv_pair_rows<<<1, 1024>>>(w);
  }
  if (n > 0)
    k_ilv_table_sizes<<<dim3((unsigned)ceil_div(most, kIlvTableThreads), (unsigned)n), kIlvTableThreads>>>(d, sh, w.found);
  int rc = cuda_status(cudaGetLastError(), "row tables launch");
  IlvFound f{};
  if (!rc) rc = cuda_status(cudaMemcpy(&f, w.found, sizeof f, cudaMemcpyDeviceToHost), "row tables");
  if (rc) return rc;
  *range = IlvRange{f.omin, f.omax, f.span4, f.span8};
  for (int g = 0; g < (pairs ? 2 : 1); ++g) {
    if (!f.rows[g].ok) continue;  // no rows: shapes of this grouping are not offered
    rows[g].nrows = f.rows[g].nrows;
    rows[g].ext_total = f.rows[g].ext_total;
    rows[g].max_ext = f.rows[g].max_ext;
    rows[g].max_group = f.rows[g].max_group;
    rows[g].max_offsets = f.rows[g].max_offsets;
  }
  for (int i = 0; i < n; ++i) {
    const IlvCfg& c = ilv_cfgs()[which[i]];
    IlvTables& t = (*tabs)[which[i]];
    t.stages = 0;  // does not fit
    if (rows[0].nrows == 0 || rows[c.G - 1].nrows == 0) continue;
    if (f.stats[2 * i] > kIlvMaxEnt || f.stats[2 * i + 1] >= 1 << 18) continue;
    const int64_t stage = round_up((int64_t)f.stats[2 * i + 1] * 4, 256);
    const int64_t per = stage + (int64_t)c.DW * 4 * c.nq * 4 + 16;
    const int64_t avail = kIlvMaxSmem - c.hi_bytes - 16;
    const int64_t stages = std::min<int64_t>(4, avail / per);
    if (stages < 2) continue;
    t.emax = f.stats[2 * i];
    t.stage_bytes = stage;
    t.stages = (int)stages;
    t.smem = stages * per + c.hi_bytes + 16;
  }
  return SPP_OK;
}

int ilv_build_tables(const IlvCfg& c, const IlvDelays& d, const IlvRows& r, void* room, int64_t room_bytes,
                     IlvTables* t) {
  if (t->d_off) return SPP_OK;
  const int64_t bytes = table_bytes(c, d.nchans, d.ndm, t->emax);
  void* p = room;
  int rc = SPP_OK;
  if (bytes > room_bytes) {
    const cudaError_t e = cudaMalloc(&p, (size_t)bytes);
    t->no_memory = e == cudaErrorMemoryAllocation;
    if (t->no_memory) cudaGetLastError();  // left for no later launch to report
    rc = cuda_status(e, "plan table alloc");
    if (rc) return rc;
    t->own = true;
  }
  t->bytes = bytes;
  t->d_off = static_cast<int32_t*>(p);
  t->d_ent = reinterpret_cast<int4*>(static_cast<uint8_t*>(p) + table_off_bytes(c, d.nchans, d.ndm));
  const IlvTableShape sh = table_shape(c, d, r);
  k_ilv_tables<<<(unsigned)ceil_div(sh.ntile * sh.nslab * 4 * c.nq, kIlvTableThreads), kIlvTableThreads>>>(
      d, sh, t->emax, t->d_off, t->d_ent);
  rc = cuda_status(cudaGetLastError(), "staging tables");
  if (!rc) rc = cuda_status(cudaStreamSynchronize(nullptr), "staging tables");
  if (rc) ilv_free_tables(t);
  return rc;
}

IlvGeom ilv_geometry(const IlvCfg& c, const IlvRows& chan, const IlvRows& rows, int64_t nchans,
                     int64_t nvalid) {
  IlvGeom g{};
  g.M = round_up(ceil_div(std::max<int64_t>(nvalid, 1), 32), 8);
  g.mp = ceil_div(g.M, c.words()) * c.words() + 8;
  const int64_t zero = (int64_t)c.words() * c.np * 4;
  g.chan_bytes = round_up((nchans * g.mp + chan.ext_total) * c.nb * 4 + (c.G == 1 ? zero : 0), 256);
  g.row_bytes = c.G == 1 ? 0 : round_up((rows.nrows * g.mp + rows.ext_total) * c.np * 4 + zero, 256);
  return g;
}

int ilv_corner_turn(const IlvCfg& c, const IlvRows& chan, const IlvGeom& g, const void* in,
                    int bitorder, int64_t nchans, int64_t nsamps, void* ws, cudaStream_t st) {
  const int64_t nblk = ceil_div(nchans, planes_ct_chans(c.nb));
  dim3 grid((unsigned)nblk, (unsigned)std::min<int64_t>(std::max<int64_t>(1, ceil_div(148 * 8 * 4, nblk)),
                                                        ceil_div(g.M, 8)));
  const uint8_t* raw = static_cast<const uint8_t*>(in);
  uint32_t* rows = static_cast<uint32_t*>(ws);
  const bool lng = chan.max_group > 31 * g.M;  // (M + max_group - 1) / M >= 32
#define SPP_ILV_TURN(NB)                                                                            \
  (lng ? k_ilv_turn<NB, true> : k_ilv_turn<NB, false>)<<<grid, 256, 0, st>>>(                       \
      raw, nchans, nsamps, bitorder, g.M, g.mp, chan.d_lo, chan.d_ext, rows)
  switch (c.nb) {
    case 1: SPP_ILV_TURN(1); break;
    case 2: SPP_ILV_TURN(2); break;
    case 4: SPP_ILV_TURN(4); break;
    default: SPP_ILV_TURN(8); break;
  }
#undef SPP_ILV_TURN
  return cuda_status(cudaGetLastError(), "interleaved corner turn launch");
}

int ilv_group_rows(const IlvCfg& c, const IlvRows& chan, const IlvRows& rows, const IlvGeom& g,
                   int64_t nchans, void* ws, cudaStream_t st) {
  if (c.G == 1) return SPP_OK;
  const uint32_t* ch = static_cast<const uint32_t*>(ws);
  uint32_t* out = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(ws) + g.chan_bytes);
  const int pair_words = 256 * pair_wpt(c.nb);
  const int64_t gy = ceil_div(g.M + chan.max_ext, pair_words), ng = nchans / 2;
  if (gy > 65535) return fail(SPP_ERR_UNSUPPORTED, "pair rows of %lld words", (long long)g.M);
  dim3 grid((unsigned)ng, (unsigned)gy);
  const int64_t smem = (int64_t)pair_words * c.np * 4 + (int64_t)(pair_words + rows.max_offsets + 16) * c.nb * 4 +
                       (int64_t)rows.max_offsets * 12;
  int rc = SPP_OK;
#define SPP_ILV_PAIRS(NB)                                                                          \
  if (smem > 48 * 1024) rc = set_smem_attr(reinterpret_cast<const void*>(&k_ilv_pairs<NB>), smem); \
  if (rc) return rc;                                                                               \
  k_ilv_pairs<NB><<<grid, 256, smem, st>>>(ch, g.mp, chan.d_lo, chan.d_ext, g.M, rows.d_rbase,     \
                                           rows.d_rlo, g.mp, rows.d_lo, rows.d_ext, rows.max_offsets, out)
  switch (c.nb) {
    case 2: SPP_ILV_PAIRS(2); break;
    case 4: SPP_ILV_PAIRS(4); break;
    default: SPP_ILV_PAIRS(8); break;
  }
#undef SPP_ILV_PAIRS
  return cuda_status(cudaGetLastError(), "pair rows launch");
}

int ilv_launch(const IlvCfg& c, const IlvTables& t, const IlvRows& rows, const IlvGeom& g,
               int64_t ngroups, int64_t ndm, const void* ws, void* out, int out_kind,
               int64_t out_stride, int64_t out_start, int64_t nvalid, uint32_t* status,
               cudaStream_t st) {
  const uint8_t* base = static_cast<const uint8_t*>(ws) + (c.G == 1 ? 0 : g.chan_bytes);
  const int64_t nwords = rows.nrows * g.mp + rows.ext_total;
  IlvArgs a{};
  a.rows = reinterpret_cast<const uint32_t*>(base);
  a.zero = a.rows + nwords * c.np;
  if (ngroups % (4 * c.nq)) {
    const int rc = cuda_status(cudaMemsetAsync(const_cast<uint32_t*>(a.zero), 0,
                                               (size_t)c.words() * c.np * 4, st), "zero row");
    if (rc) return rc;
  }
  a.mp = g.mp;
  a.M = g.M;
  a.off = t.d_off;
  a.ent = t.d_ent;
  a.emax = t.emax;
  a.stages = t.stages;
  a.stage_bytes = (int32_t)t.stage_bytes;
  a.nslab = (int32_t)ceil_div(ngroups, 4 * c.nq);
  a.ndt = (int32_t)ceil_div(ndm, c.DW);
  a.njt = (int32_t)ceil_div(g.M, c.words());
  // 13 trial tiles per block: their windows of one row overlap, and the rows
  // the blocks in flight read stay near L2's size (2-bit, 4096 channels, 1024
  // trials, 2^20 samples: 46.0 ms; 2 per block 46.6, all 114: 46.9)
  a.db = std::min(a.ndt, 13);
  a.ndm = (int32_t)ndm;
  a.out = out;
  a.out_kind = out_kind;
  a.out_stride = out_stride;
  a.out_start = out_start;
  a.nvalid = nvalid;
  a.status = status;
  if (t.smem > 48 * 1024) {
    const int rc = set_smem_attr(c.fn, t.smem);
    if (rc) return rc;
  }
  const int64_t grid = (int64_t)a.ndt * a.njt;
  if (grid > INT32_MAX) return fail(SPP_ERR_UNSUPPORTED, "too many tiles");
  void* args[] = {&a};
  return cuda_status(cudaLaunchKernel(c.fn, dim3((unsigned)grid), dim3((unsigned)c.threads), args,
                                      (size_t)t.smem, st), "interleaved DM-time launch");
}

}  // namespace spp
