// Tensor-core assisted F-stage in FP32 accuracy for windows of 2-bit real data: 2048 and 4096 points with every channelised
// output type, 8192 to 32768 points with FP32 output.
//
// Four-step factorisation N = N1 x N2, n = n2 + N2 n1, k = k1 + N1 k2 (fxkernel's dofft,
// fxkernel/src/fxkernel.cpp:569-580, is the plain unnormalised forward DFT this restates); N2 = 128, at 32768 points 256:
//   X[k1 + N1 k2] = sum_n2 W_N2^(n2 k2) [ W_N^(n2 k1) sum_n1 W_N1^(n1 k1) x[n2 + N2 n1] ].
// Step 1, the N1-point DFTs of the raw 2-bit levels, is a GEMM on tcgen05 with FP32 accumulation in tensor memory:
// D1 (rows (window, k1), 64 of them; columns n2) = A1 B1^T per polarisation, real and imaginary part, K = (window,
// n1).  The fringe rotator of sample n is exp(-2 pi i (c0 + c1 n)): its n1 part is folded into A1 (rows k1 of
// window w: W_N1^(n1 k1) e^(-2 pi i 128 n1 c1), block-diagonal over the 64 / N1 windows of a group), its n2 part into
// the twiddles of step 2.  A1 is split into FP16 hi and lo halves (23 significand bits; the FP32 product that they hold is
// itself off by about a unit of the 24th).  B1 holds the levels as 1039 and 3466, FP16 values that stand for the FP32 levels
// to less than half a unit of their last bit (kUnit).  D1 = A_lo B + A_hi B, in this order: the small terms first, so that
// tensor memory's rounding toward zero acts on the large sum only once per K step of A_hi (one, two and four with terms at
// 2048, 4096 and 8192 points, eight beyond); what it takes away on average is in A1 (Plan::RZ).  An exact hi and lo pair of
// levels (3.3359375 - 628 x 2^-24) took half as many MMAs again and twice the decode's stores, 25.1 against 24.2 ms (16
// antennas, 62500 FFTs), and products of 48 bits in A1 24.5 -> 25.8 ms for 1 % less error.
//
// Error against FP64, FP32 sums of 32, 16, 8, 4 and 4 FFTs (2048 to 32768 points; 57 and 38 antennas, 256 MHz), with that of
// the register FFT as it was when this kernel took its place: power spectra 1.54, 1.39, 1.50, 2.05, 2.12e-7 rms (1.71, 1.65,
// 1.48, 2.46, 2.27e-7), of which the mean is 0.1e-7 (1.1, 1.1, 0.8, 1.5, 1.0e-7); cross products 2.5, 2.4, 2.4, 2.6, 2.7e-7
// (3.1, 3.1, 2.9, 3.2, 3.3e-7), and at 32 MHz, where the fringe turns further in a window, 2.6, 2.5, 2.5, 2.7, 2.7e-7 (3.3,
// 3.5, 4.5, 7.0, 13e-7).
// Step 2, the N2-point DFTs over n2, runs on the CUDA cores in FP32: a thread owns one row, so the transform needs no
// exchange between threads.  Radix 8 over j (n2 = i + (N2 / 8) j), back to tensor memory, radix N2 / 8 over i.  With
// theta = k1 / N + c1 both passes take their twiddles as powers of e^(-2 pi i theta) (the DFT at a shifted
// frequency costs what the plain one does); the products of at most four directly evaluated factors keep them at
// FP32 accuracy.
//
// One persistent CTA per SM, 28 warps: 16 transform warps (two teams on alternate groups), 8 decode warps (unpack,
// A1, tables), one that issues the MMAs (and three that idle).  Two operand slots and two 256-column tensor-memory
// slots are in flight, connected by mbarriers.
//
// What bounds it (16 antennas, 8192 points, FP32, 2048 FFTs, ncu): 40.5 instructions per sample and polarisation (53 for the
// packed register FFT) at 73 % issue active, FMA pipe 58 % (twiddles and butterflies), tensor pipe 29 %, DRAM 35 %.
// F-stage of the 16-antenna, nchan-4096 workload (62500 FFTs), FP32: 24.4 ms; 40.8 ms for the register FFT
// (fstage_pair_kernel); 6 antennas, nchan 1024, 15625 FFTs: 0.58 against 0.98 ms.
//
// From 16384 points on (N1 = 128) a group is one window; D1 is 128 rows of one polarisation, M = 128 MMAs over two K blocks,
// and A1 (128 KB) is single, shared by both polarisations and by all windows of the same slope.  At 16384 points team and
// slot s belong to polarisation s.  At 32768 points D1 takes all of tensor memory: eight transform warps of 144 registers
// (radix 32 holds 16 packed pairs) alternate with the MMAs (4,300 clocks of about 22,000 per window and polarisation).
// F-stage, 10 antennas, 32768 points, 3901 FFTs: 5.80 ms, 15.85 for the cluster kernel.
//
// Every wait is bounded; on expiry the kernel sets an error flag (read by gxc_sync as GXC_ERR_TIMEOUT), lets issued
// MMAs drain, frees tensor memory and returns.
#include "fstage_kernels.cuh"
#include "gxc_internal.h"
#include "tcgen05_util.cuh"

namespace gxc {

namespace f32tc {

constexpr int DW = 8, GT = DW * 32;          // decode warps and threads

template <int L>
struct Plan {
  static constexpr int N = 1 << L;
  static constexpr bool W1 = L >= 14;         // a group is one window, and D1 holds one polarisation in all lanes
  static constexpr int N1 = W1 ? 128 : N / 128, N2 = N / N1;
  static constexpr int ROWS = W1 ? 128 : 64, NW = ROWS / N1;  // rows of A1; windows per group
  static constexpr int NS = L == 15 ? 1 : 2;  // operand / tensor-memory slots
  static constexpr int FW = L == 15 ? 8 : 16, W_DEC = FW, W_MMA = FW + DW;  // transform warps; roles
  static constexpr int NT = (FW + DW + 4) * 32;  // + the MMA warp's warpgroup (three idle warps)
  static constexpr int REG = L == 15 ? 96 : 72, REG_FFT = L == 15 ? 144 : 80, REG_DEC = 72, REG_MMA = 40;
  static_assert(FW / 4 * REG_FFT + 2 * REG_DEC + REG_MMA <= NT / 128 * REG, "register shares");
  static constexpr int WPW = N / 8, NWORD = NW * WPW / GT;  // 32-bit words of one packed window (both pols); per thread
  static constexpr int NK2 = N2 / 2;          // kept k2 (real data)
  static constexpr int NP = N2 == 128 ? 7 : 8, ES = N2 == 128 ? 8 : 16;  // log2 N2; e entries of a window
  static constexpr int NPR = N2 / 16;         // pairs of samples i, i + 1
  static constexpr int NR = L == 15 ? 2 : 4;  // table ring
  // Tensor memory rounds its FP32 sums toward zero, which leaves D1 low by this much on average (a row has terms in one,
  // two, four or eight K steps); A1's lo half carries the inverse.  Measured on sampled noise: with it power spectra are
  // within 2e-8 of FP64 on average, at each length.
  static constexpr float RZ = L == 11 ? 1.04e-7f : L == 12 ? 1.13e-7f : L == 13 ? 1.39e-7f : L == 14 ? 2.0e-7f : 2.05e-7f;
  // ring entry (float2): fsub[(w, k1)], e[w][ES] (e^(-2 pi i 2^s c1), s < NP; e^(-2 pi i c0), or 0 for a flagged
  // window), fst[w][k2] = e^(2 pi i N1 k2 cf) * scale
  static constexpr int T_FSUB = 0, T_E = ROWS, T_FST = T_E + ES * NW, TAB = T_FST + NK2 * NW;
  // shared-memory image (byte offsets from a 1024-aligned base)
  static constexpr int APL = ROWS * 128 * (W1 ? 2 : 1), BPL = N2 * 128 * (W1 ? 2 : 1);  // planes of A1, of B1 (a pol)
  static constexpr int SLOT = 4 * APL + 2 * BPL;          // up to 8192 points: A1 [re, im][hi, lo], B1 [pol] per slot
  static constexpr int OFF_STAGE = W1 ? 4 * APL + NS * BPL : NS * SLOT;  // beyond: one A1, B1 of a pol per slot
  static constexpr int NSTG = L == 15 ? 1 : 2, STG = NW * WPW * 4;  // the packed windows, realigned
  static constexpr int OFF_TAB = OFF_STAGE + NSTG * STG;
  static constexpr int OFF_TST = OFF_TAB + NR * TAB * 8;  // tstep[(w, n1)], alternating
  static constexpr int OFF_WC = OFF_TST + 2 * ROWS * 8;   // W_N^(2^s k1) [NP][N1]
  static constexpr int NWR = ROWS, OFF_WR = OFF_WC + NP * N1 * 8;  // W_NWR^j [NWR]
  static constexpr int WKS = N2 == 128 ? 4 : 8, OFF_WK = OFF_WR + NWR * 8;  // W_N2^(2^s k) [8][WKS]
  static constexpr int OFF_GEOM = OFF_WK + 8 * WKS * 8;   // alternating: NW geometry records
  static constexpr int SMEM = OFF_GEOM + 2 * NW * 32 + 1024;
  static_assert(SMEM <= 227 * 1024, "shared memory");
  __host__ __device__ static constexpr int off_a(int slot) { return W1 ? 0 : slot * SLOT; }
  __host__ __device__ static constexpr int off_b(int slot) { return W1 ? 4 * APL + slot * BPL : slot * SLOT + 4 * APL; }
};

struct Params {
  Job job;
  int t0, nt, T;
  void *chan;
  float out_scale;
  const float *cscale;  // FP8 output: per-channel scale [nchan] (replaces out_scale), or null
  float2 *probe;        // decode probe (DBG kernels)
  int *err;
};

__device__ int g_f32tc_err;

// The operand levels 1039 and 3466 stand for 1039 kUnit and 3466 kUnit, which are 1 + 4.1e-8 and 3.3359f (1 - 0.8e-8): both
// round to the FP32 level.  (Their ratio is 4.9e-8 short of 3.3359f; the high level, which carries most of the power of
// sampled noise, is the nearer one.)
constexpr double kUnit = (1.0 + 4.1e-8) / 1039.0;
// A1 carries kUnit 2^14, so that its lo half stays in FP16's normal range; the frac-delay table carries 2^-14.  kScale holds
// it in FP32, kLevel the rest, which goes into the lo half.
constexpr float kScale = (float)(kUnit * 16384.0), kLevel = (float)(kUnit * 16384.0 / (double)kScale - 1.0);

// Tensor-memory column (= row of B1) of sample n2 = i + (N2 / 8) j (j < 8): 16 pr + 2 (j xor pr / 2) + (i mod 2) with
// pr = i / 2.  Samples i, i + 1 are adjacent columns, the lanes of packed FP32 pairs, and the eight j of a pair are 16
// consecutive columns; the exclusive or spreads the decode's stores over the swizzle positions.

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// Scaled FP16 levels of four 2-bit codes, one per byte of `codes` (the other bits are ignored): {-3466, -1039, 1039, 3466}.
// Their low bytes are one word, their high bytes another: code c picks bytes c and 4 + c.
__device__ __forceinline__ void level_quad(uint32_t codes, uint32_t (&v)[2]) {
  constexpr uint32_t kL = 0xC50F0FC5u, kH = 0x6A64E4EAu;  // 0xEAC5, 0xE40F, 0x640F, 0x6AC5
  const uint32_t sel = (codes & 0x03030303u) * 0x11u + 0x40404040u;
  v[0] = tc::prmt(kL, kH, sel);
  v[1] = tc::prmt(kL, kH, sel >> 16);
}

// Group of NW consecutive FFTs of one antenna; a CTA takes a contiguous run of groups, FFTs fastest, so that the
// rotator's slope (and with it A1) rarely changes from one group to the next.
struct Group {
  int ant, tg;
  __device__ __forceinline__ Group(int g, int ntg) : ant(g / ntg), tg(g % ntg) {}
  __device__ __forceinline__ void next(int ntg) {
    if (++tg == ntg) {
      tg = 0;
      ant++;
    }
  }
};

__device__ __forceinline__ void st16f(uint32_t a, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 "
      "[%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(a),
      "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
      "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
      : "memory");
}
__device__ __forceinline__ void ld2(uint32_t a, float2 &v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
}
__device__ __forceinline__ void wait_ld2(P2 *u) {  // eight
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(u[0].re.x), "+f"(u[0].re.y), "+f"(u[0].im.x), "+f"(u[0].im.y), "+f"(u[1].re.x), "+f"(u[1].re.y),
                 "+f"(u[1].im.x), "+f"(u[1].im.y), "+f"(u[2].re.x), "+f"(u[2].re.y), "+f"(u[2].im.x), "+f"(u[2].im.y),
                 "+f"(u[3].re.x), "+f"(u[3].re.y), "+f"(u[3].im.x), "+f"(u[3].im.y), "+f"(u[4].re.x), "+f"(u[4].re.y),
                 "+f"(u[4].im.x), "+f"(u[4].im.y), "+f"(u[5].re.x), "+f"(u[5].re.y), "+f"(u[5].im.x), "+f"(u[5].im.y)
               :
               : "memory");
  asm volatile("" : "+f"(u[6].re.x), "+f"(u[6].re.y), "+f"(u[6].im.x), "+f"(u[6].im.y), "+f"(u[7].re.x), "+f"(u[7].re.y),
                    "+f"(u[7].im.x), "+f"(u[7].im.y) : : "memory");
}

// both lanes times w, as scalar products (as many FMA-pipe cycles as packed ones, and no broadcast pairs to build)
__device__ __forceinline__ P2 pscale(const P2 &v, float2 w) {
  const float2 a = cmul(make_float2(v.re.x, v.im.x), w), b = cmul(make_float2(v.re.y, v.im.y), w);
  P2 r;
  r.re = make_float2(a.x, b.x);
  r.im = make_float2(a.y, b.y);
  return r;
}

// 8-point DFT of both lanes, natural order
__device__ __forceinline__ void dft8p(P2 (&u)[8]) {
  const float r = 0.70710678118654752440f;
  dft4p<false, false>(u[0], u[2], u[4], u[6]);
  dft4p<false, false>(u[1], u[3], u[5], u[7]);
  pcmul_c(u[3], r, -r);
  pcmul_c(u[7], -r, -r);
  P2 y[8];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const P2 a = u[2 * k], b = u[2 * k + 1];
    if (k == 2) {  // W8^2 = -i folded in
      y[k].re = cadd(a.re, b.im);
      y[k].im = csub(a.im, b.re);
      y[k + 4].re = csub(a.re, b.im);
      y[k + 4].im = cadd(a.im, b.re);
    } else {
      y[k].re = cadd(a.re, b.re);
      y[k].im = cadd(a.im, b.im);
      y[k + 4].re = csub(a.re, b.re);
      y[k + 4].im = csub(a.im, b.im);
    }
  }
#pragma unroll
  for (int k = 0; k < 8; k++) u[k] = y[k];
}

template <int L, typename OutT, bool DBG = false>
__global__ void __launch_bounds__(Plan<L>::NT, 1) fstage_tc32_kernel(Params p) {
  using namespace tc;
  using P = Plan<L>;
  constexpr int N = P::N, N1 = P::N1, N2 = P::N2, NW = P::NW, NR = P::NR, WPW = P::WPW, NS = P::NS, NT = P::NT, NP = P::NP;
  constexpr int ROWS = P::ROWS, FW = P::FW;
  constexpr bool W1 = P::W1;
  extern __shared__ unsigned char smem_raw[];
  // handshakes, one phase per use of a slot (up to 8192 points group i of the CTA uses slot i mod 2; pol p of group i uses
  // slot p at 16384 points, and the only slot at 32768) or of a ring entry (group i: i mod NR): ab_full
  // (decode -> MMA), ab_free (MMAs done -> decode), d_full (MMAs done -> transform), d_free (transform -> MMA),
  // tab_full (decode -> transform), tab_free (transform -> decode)
  __shared__ __align__(8) uint64_t ab_full[NS], ab_free[NS], d_full[NS], d_free[NS], tab_full[NR], tab_free[NR],
      bar_final;
  __shared__ uint32_t tmem_base_sh;
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = smem_u32(smem);
  const Job &job = p.job;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nant = job.nant, nstreams = 2 * nant;
  const size_t ctile_stride = (size_t)p.T * nstreams * CW;
  OutT *chan = reinterpret_cast<OutT *>(p.chan);
  float2 *const tab0 = reinterpret_cast<float2 *>(smem + P::OFF_TAB);
  float2 *const wc = reinterpret_cast<float2 *>(smem + P::OFF_WC), *const wr = reinterpret_cast<float2 *>(smem + P::OFF_WR);
  float2 *const wk = reinterpret_cast<float2 *>(smem + P::OFF_WK);

  // constant tables, and zeros (the off-diagonal blocks of A1 stay zero)
  auto root = [](int num, int den) {  // exp(-2 pi i num / den)
    float sn, cs;
    sincospif(-2.0f * (float)num / (float)den, &sn, &cs);
    return make_float2(cs, sn);
  };
  for (int i = tid; i < NP * N1; i += NT) wc[i] = root((i % N1) << (i / N1), N);
  for (int i = tid; i < P::NWR; i += NT) wr[i] = root(i, P::NWR);
  for (int i = tid; i < 8 * P::WKS; i += NT) wk[i] = root((i / P::WKS) << (i % P::WKS), N2);
  for (int s = 0; s < (W1 ? 1 : NS); s++)
    for (int i = tid; i < 4 * P::APL / 16; i += NT)
      *reinterpret_cast<uint4 *>(smem + P::off_a(s) + 16 * i) = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    for (int s = 0; s < NS; s++) {
      mbar_init(smem_u32(&ab_full[s]), DW);
      mbar_init(smem_u32(&ab_free[s]), 1);
      mbar_init(smem_u32(&d_full[s]), 1);
      mbar_init(smem_u32(&d_free[s]), 8);
    }
    for (int s = 0; s < NR; s++) {
      mbar_init(smem_u32(&tab_full[s]), 1);
      mbar_init(smem_u32(&tab_free[s]), L == 14 ? 16 : 8);
    }
    mbar_init(smem_u32(&bar_final), 1);
    fence_mbar_init();
  }
  if (warp == 0) {
    tmem_alloc(smem_u32(&tmem_base_sh), 512);
    tmem_relinquish();
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem0 = tmem_base_sh;  // slot s: D1 Re at columns 256 s, D1 Im N2 columns on
  const int ntg = (p.nt + NW - 1) / NW;
  const long long ngrp = (long long)ntg * nant;
  const int g0 = (int)(ngrp * blockIdx.x / gridDim.x), g1 = (int)(ngrp * (blockIdx.x + 1) / gridDim.x);
  const int ng = g1 - g0;

  if (warp < P::W_DEC) {
    // ------------------------------------------------------------ transform
    reg_inc<P::REG_FFT>();
    // Up to 8192 points row 16 q + lane mod 16 = (window, k1) of pol lane / 16, and two teams of eight warps take alternate
    // groups (team = slot), so that the four warps of an SM sub-partition are in two different phases.  At 16384 points
    // row 32 q + lane = k1, and team s takes pol s of every group; at 32768 one team takes both in turn.  Warps
    // h = 0, 1 of a team share a lane quarter.
    const int q = warp & 3, s = FW == 16 ? (warp >> 2) & 1 : 0, h = FW == 16 ? warp >> 3 : warp >> 2;
    const int row = W1 ? 32 * q + lane : 16 * q + (lane & 15), wn = row / N1, k1 = row % N1;
    const uint32_t tlane = tmem0 + ((uint32_t)(32 * q) << 16);
    // output address: channel k1 + N1 k2 of (window, pol)
    const uint32_t o1 = (uint32_t)(k1 >> 4) * (uint32_t)ctile_stride + (k1 & 15);
    const uint32_t step = (uint32_t)((N1 >= 16 ? N1 / 16 : 1) * ctile_stride * sizeof(OutT));  // (below 4 GB: launcher)
    Group grp(g0, ntg);
    if (!W1 && s) grp.next(ntg);
    bool ok = true;
    int v0 = W1 ? 0 : s;
    const int vn = L == 15 ? 2 * ng : ng;
    for (; v0 < vn; v0 += W1 ? 1 : 2) {
      const int i = L == 15 ? v0 >> 1 : v0, ri = i % NR;
      const int pol = !W1 ? lane >> 4 : L == 14 ? s : v0 & 1;
      const uint32_t ph = W1 ? v0 & 1 : (v0 >> 1) & 1;  // of this use of the slot
      if (!mbar_wait_warp(smem_u32(&tab_full[ri]), (i / NR) & 1, p.err)) break;
      const bool exists = grp.tg * NW + wn < p.nt;
      const float2 *tab = tab0 + ri * P::TAB;
      const float2 *fst = tab + P::T_FST + P::NK2 * wn;
      unsigned char *const o = reinterpret_cast<unsigned char *>(
          chan + o1 + ((size_t)(grp.tg * NW + wn) * nstreams + 2 * grp.ant + pol) * CW);
      auto put = [&](int k2, float2 v) {
        if (!exists) return;
        OutT *dst;
        if constexpr (N1 >= 16) dst = reinterpret_cast<OutT *>(o + (uint64_t)(uint32_t)k2 * step);
        else dst = reinterpret_cast<OutT *>(o + (uint64_t)(uint32_t)(k2 >> 1) * step) + 8 * (k2 & 1);
        *dst = to_out<OutT>(v, chan_scale<OutT>(p.cscale, k1 + N1 * k2, 1.0f));
      };
      {
        // powers of e^(-2 pi i theta), theta = k1 / N + c1, and the phase of sample 0 with the fine frac-delay (0 for a
        // flagged window, whose outputs are then zeros)
        const float2 *e = tab + P::T_E + P::ES * wn;
        const uint32_t tr = tlane + 256u * s;
        {
          float2 gj[8];
          {
            const float2 y1 = cmul(wc[(NP - 3) * N1 + k1], e[NP - 3]), y2 = cmul(wc[(NP - 2) * N1 + k1], e[NP - 2]);
            const float2 y4 = cmul(wc[(NP - 1) * N1 + k1], e[NP - 1]);
            gj[0] = cmul(e[NP], tab[P::T_FSUB + row]);
            gj[1] = cmul(gj[0], y1);
            gj[2] = cmul(gj[0], y2);
            gj[3] = cmul(gj[1], y2);
#pragma unroll
            for (int j = 0; j < 4; j++) gj[4 + j] = cmul(gj[j], y4);
          }
          ok = mbar_wait_warp(smem_u32(&d_full[s]), ph, p.err);
          if (!ok) break;
          tc_fence_after();
          // ---- radix 8 over j, for the pairs i = 2 pr, 2 pr + 1, pr = 2 pp + h; in place
#pragma unroll
          for (int pp = 0; pp < P::NPR / 2; pp++) {
            const uint32_t tp = tr + 16u * (2 * pp + h);
            float re[16], im[16];
            tmem_ld16_async(tp, re);
            tmem_ld16_async(tp + N2, im);
            tmem_wait_ld16(re);
            tmem_wait_ld16(im);
            P2 u[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const int x = 2 * (j ^ pp);  // column of j (pr / 2 = pp)
              P2 v;
              v.re = make_float2(re[x], re[x + 1]);
              v.im = make_float2(im[x], im[x + 1]);
              u[j] = pscale(v, gj[j]);
            }
            dft8p(u);
#pragma unroll
            for (int k = 0; k < 8; k++) {
              re[2 * k] = u[k].re.x;
              re[2 * k + 1] = u[k].re.y;
              im[2 * k] = u[k].im.x;
              im[2 * k + 1] = u[k].im.y;
            }
            st16f(tp, re);
            st16f(tp + N2, im);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        group_sync(2 + 4 * s + q, 64);
        tc_fence_after();
        // ---- radix 2 NPR over i: for each k, the pairs (i = 2 pr + b, lane b) through radix NPR over pr, then the lanes.
        //      Inputs carry z_k^i, z_k = e^(-2 pi i (k / N2 + theta)).
        constexpr int NPR = P::NPR;
        const float2 z1 = cmul(wc[0 * N1 + k1], e[0]), z2 = cmul(wc[1 * N1 + k1], e[1]), z4 = cmul(wc[2 * N1 + k1], e[2]);
        const float2 z8 = cmul(wc[3 * N1 + k1], e[3]), z16 = NPR == 16 ? cmul(wc[4 * N1 + k1], e[4]) : z8;
#pragma unroll 1
        for (int kk = 0; kk < 4; kk++) {
          const int k = 4 * h + kk;
          P2 u[NPR];
          // tensor memory is read by whole warps; put() branches by lane in a group whose last windows the block's end cuts off
          if constexpr (NW > 1) __syncwarp();
#pragma unroll
          for (int pr = 0; pr < NPR; pr++) {
            ld2(tr + 16 * pr + 2 * k, u[pr].re);
            ld2(tr + N2 + 16 * pr + 2 * k, u[pr].im);
          }
          const float2 *wkk = wk + P::WKS * k;
          const float4 wa = *reinterpret_cast<const float4 *>(wkk), wb = *reinterpret_cast<const float4 *>(wkk + 2);
          const float2 zk = cmul(z1, make_float2(wa.x, wa.y)), zk2 = cmul(z2, make_float2(wa.z, wa.w));
          const float2 zk4 = cmul(z4, make_float2(wb.x, wb.y)), zk8 = cmul(z8, make_float2(wb.z, wb.w));
          wait_ld2(u);
          if constexpr (NPR == 16) wait_ld2(u + 8);
          if (kk == 3) {  // D1 has been read: the MMAs of the slot's next group may overwrite it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&d_free[s]));
          }
          const float2 zk6 = cmul(zk4, zk2);
          u[1] = pscale(u[1], zk2);
          u[2] = pscale(u[2], zk4);
          u[3] = pscale(u[3], zk6);
#pragma unroll
          for (int b = 1; b < NPR / 4; b++) {
            float2 zb = zk8;
            if constexpr (NPR == 16) {
              const float2 zk16 = cmul(z16, wkk[4]);
              zb = b == 1 ? zk8 : b == 2 ? zk16 : cmul(zk16, zk8);
            }
            u[4 * b] = pscale(u[4 * b], zb);
            u[4 * b + 1] = pscale(u[4 * b + 1], cmul(zb, zk2));
            u[4 * b + 2] = pscale(u[4 * b + 2], cmul(zb, zk4));
            u[4 * b + 3] = pscale(u[4 * b + 3], cmul(zb, zk6));
          }
          if constexpr (NPR == 16) dft16p<false>(u);
          else dft8p(u);
          // output m: lane 0 + z_k W_(2 NPR)^m lane 1, then the frac-delay step of channel k1 + N1 (k + 8 m)
          constexpr float kC[8] = {1.0f, 0.98078528040323044913f, 0.92387953251128675613f, 0.83146961230254523708f,
                                   0.70710678118654752440f, 0.55557023301960222474f, 0.38268343236508977173f,
                                   0.19509032201612826785f};  // cos(pi m / 16); sin(pi m / 16) = kC[8 - m]
          constexpr int MS = 16 / NPR;
          float2 w[NPR / 2];
          w[0] = zk;
#pragma unroll
          for (int m = 1; m < NPR / 2; m++) w[m] = cmul(zk, make_float2(kC[MS * m], -kC[8 - MS * m]));
#pragma unroll
          for (int m = 0; m < NPR; m++) {
            const float2 wm = m < NPR / 2 ? w[m] : make_float2(w[m - NPR / 2].y, -w[m - NPR / 2].x);
            const float2 ev = make_float2(u[m].re.x, u[m].im.x), od = make_float2(u[m].re.y, u[m].im.y);
            const float2 v =
                make_float2(fmaf(od.x, wm.x, fmaf(-od.y, wm.y, ev.x)), fmaf(od.x, wm.y, fmaf(od.y, wm.x, ev.y)));
            put(k + 8 * m, cmul(v, fst[k + 8 * m]));
          }
        }
      }
      __syncwarp();
      if (lane == 0 && (L != 15 || pol == 1)) mbar_arrive(smem_u32(&tab_free[ri]));
      if constexpr (L == 15) {
        if (pol == 1) grp.next(ntg);
      } else {
        grp.next(ntg);
        if (!W1) grp.next(ntg);
      }
    }
    // a warp that gave up still meets the other warp of its lane quarter once per use
    for (; v0 < vn; v0 += W1 ? 1 : 2) group_sync(2 + 4 * s + q, 64);
  } else if (warp < P::W_MMA) {
    // ------------------------------------------------------------ decode
    // Group i + 1's samples load while B1 and A1 of group i are made; geometry records are two groups ahead.
    if constexpr (P::REG != P::REG_DEC) reg_dec<P::REG_DEC>();
    const int gt = tid - 32 * P::W_DEC;
    Geom *const sg = reinterpret_cast<Geom *>(smem + P::OFF_GEOM);  // records of group i at NW (i mod 2)
    const int myw = (gt & (ROWS - 1)) / N1;            // window of this thread's A1 rows
    float2 a1_slope[2] = {{1e30f, 0.f}, {1e30f, 0.f}};  // their rotator slope (and its rest) in the A1 of each slot
    constexpr int NWORD = P::NWORD;
    uint32_t pw[NWORD], pnext, greg = 0;
    Group grp(g0, ntg), nxt = grp;
    // this thread's word of the NW geometry records of group x (zeros past the block or the run: not valid)
    auto load_geom = [&](const Group &x, int i) -> uint32_t {
      const int t = x.tg * NW + (gt >> 3);
      if (gt >= 8 * NW || i >= ng || t >= p.nt) return 0u;
      return reinterpret_cast<const uint32_t *>(job.geom + (size_t)x.ant * job.nfft + p.t0 + t)[gt & 7];
    };
    auto set_geom = [&](uint32_t v, int i) {
      if (gt < 8 * NW) reinterpret_cast<uint32_t *>(sg + NW * (i & 1))[gt] = v;
    };
    // starts the loads of words gt + 256 j of the group's packed windows (window (gt + 256 j) / WPW, from the 4-byte
    // boundary before its first sample) and, in lane j, of the word after row j of this warp.  The buffer holds
    // (nfft+1)*F samples and offset <= (nfft-1)*F, so a window plus one word stays inside it.
    const uint8_t *in = nullptr;
    int in_ant = -1;
    auto prefetch = [&](const Group &x, const Geom *gg) {
      if (x.ant != in_ant) {
        in_ant = x.ant;
        in = job.inputs[x.ant];
      }
      auto word = [&](int wi, int first) -> uint32_t {  // word wi of the group; its window is that of word `first`
        const int w = first / WPW;
        if (!gg[w].valid) return 0u;
        return __ldg(reinterpret_cast<const uint32_t *>(in + (((long long)gg[w].offset >> 1) & ~3LL)) + (wi - w * WPW));
      };
#pragma unroll
      for (int j = 0; j < NWORD; j++) pw[j] = word(gt + GT * j, gt + GT * j);
      const int row = gt - lane + GT * (lane & (NWORD - 1));
      pnext = lane < NWORD ? word(row + 32, row) : 0u;
    };
    bool ok = true;
    if (ng > 0) {
      set_geom(load_geom(grp, 0), 0);
      group_sync(1, GT);
      prefetch(grp, sg);
      nxt.next(ntg);
      greg = load_geom(nxt, 1);
    }
    for (int i = 0; i < ng; i++) {
      const int ri = i % NR, s = W1 ? 0 : i & 1;  // ring entry, slot of A1
      float2 *const tab = tab0 + ri * P::TAB;
      unsigned char *const a1 = smem + P::off_a(s);
      unsigned char *const stage = smem + P::OFF_STAGE + (P::NSTG == 2 ? (i & 1) * P::STG : 0);
      float2 *const tst = reinterpret_cast<float2 *>(smem + P::OFF_TST) + ROWS * (i & 1);
      if (P::NSTG == 1 && i > 0) group_sync(1, GT);  // the last group's samples have been read
      const Geom *const gg = sg + NW * (i & 1);
      // samples, shifted so that each window's first one starts a word
#pragma unroll
      for (int j = 0; j < NWORD; j++) {
        const int off = gg[(gt + GT * j) / WPW].offset;
        const uint32_t up = __shfl_down_sync(0xffffffffu, pw[j], 1), last = __shfl_sync(0xffffffffu, pnext, j);
        reinterpret_cast<uint32_t *>(stage)[gt + GT * j] =
            __funnelshift_r(pw[j], lane < 31 ? up : last, ((off >> 1) & 3) * 8 + (off & 1) * 4);
      }
      // tables, one sincos each
      ok = i < NR || mbar_wait(smem_u32(&tab_free[ri]), ((i / NR) & 1) ^ 1, p.err);
#pragma unroll 1
      for (int x = gt; x < P::TAB; x += GT) {
        float arg, sc = 1.0f, lo = 0.0f;  // half turns; scale; small correction (radians)
        if (x < P::T_E) {
          arg = 2.0f * ((float)(x % N1) * gg[x / N1].cf);
        } else if (x < P::T_FST) {
          const Geom &gw = gg[(unsigned)(x - P::T_E) / P::ES];
          const int sft = (x - P::T_E) & (P::ES - 1);
          arg = -2.0f * (sft < NP ? (float)(1 << sft) * gw.c1 : gw.c0 - rintf(gw.c0));  // (the phase mod 1: exact)
          lo = -6.283185307f * (sft < NP ? (float)(1 << sft) * gw.c1_lo : gw.c0_lo);
          if (sft == NP) sc = gw.valid ? 1.0f : 0.0f;
        } else {
          const int y = x - P::T_FST;
          arg = 2.0f * ((float)(N1 * (y % P::NK2)) * gg[y / P::NK2].cf);
          sc = p.out_scale * 0x1p-14f;  // powers of two: exact
        }
        float sn, cs;
        sincospif(arg, &sn, &cs);
        tab[x] = make_float2(fmaf(-sn, lo, cs) * sc, fmaf(cs, lo, sn) * sc);
      }
      // A1 of this slot is rebuilt when the slope moved by more than 1.2e-8 turns over a window (half the last bit of a
      // slope of 0.4 turns per window): the phase error of keeping it stays below 7.5e-8 rad at the window's end
      const float smul = job.rotator == GXC_ROTATOR_FXKERNEL ? (float)job.stride : (float)N2;  // samples per n1 step
      const float2 slope = make_float2(gg[myw].c1, gg[myw].c1_lo), built = s ? a1_slope[1] : a1_slope[0];
      const bool rebuild = gg[myw].valid && !(fabsf((slope.x - built.x) + (slope.y - built.y)) * (float)N <= 1.2e-8f);
      if (rebuild) {
        if (s) a1_slope[1] = slope;
        else a1_slope[0] = slope;
        if (gt < ROWS) {  // row gt of tstep: (w, n1), with the levels' scale
          const float m = (float)(gt % N1) * smul, ph = m * slope.x;
          const float lo = -6.283185307f * fmaf(m, slope.y, fmaf(m, slope.x, -ph));
          float sn, cs;
          sincospif(-2.0f * ph, &sn, &cs);
          tst[gt] = make_float2(fmaf(-sn, lo, cs) * kScale, fmaf(cs, lo, sn) * kScale);
        }
      }
      uint32_t vm = 0;  // valid windows
      if constexpr (DBG) {
        for (int w = 0; w < NW; w++) vm |= gg[w].valid ? 1u << w : 0u;
      }
      set_geom(greg, i + 1);
      // the staged samples, tables and next records are complete (and the readers of the other staging buffer are done)
      if (!group_sync_and(1, GT, ok)) break;
      if (gt == 0) mbar_arrive(smem_u32(&tab_full[ri]));
      const Group cur = grp;
      grp = nxt;
      nxt.next(ntg);
      if (i + 1 < ng) prefetch(grp, sg + NW * ((i + 1) & 1));
      greg = load_geom(nxt, i + 2);
      // ---- B1 of one pol: samples n2 = 4 ln .. 4 ln + 3 of K rows (window, n1) = 8 o .. 8 o + 7.  In odd lanes (at 256
      //      samples per row, in lanes with bit 2 set) they are taken in the order 1 0 3 2, so that eight consecutive lanes
      //      store to eight swizzle positions.
      auto load_codes = [&](int o, int ln, uint32_t (&t)[2][2]) {  // [byte of the pair][K quad]: byte j = K row j
        const uint16_t *src = reinterpret_cast<const uint16_t *>(stage + N2 / 2 * 8 * o) + ln;
        uint32_t v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = src[N2 / 4 * j];
#pragma unroll
        for (int x = 0; x < 2; x++) {
          const uint32_t p01 = prmt(v[4 * x], v[4 * x + 1], 0x5410), p23 = prmt(v[4 * x + 2], v[4 * x + 3], 0x5410);
          t[0][x] = prmt(p01, p23, 0x6420);
          t[1][x] = prmt(p01, p23, 0x7531);
        }
      };
      auto store_b1 = [&](unsigned char *b1, int o, int ln, int pol, int r0, const uint32_t (&t)[2][2]) {
        const int odd = N2 == 128 ? ln & 1 : (ln >> 2) & 1, r = r0 ^ odd;  // n2 = 4 ln + r
        const int il = N2 == 128 ? ln & 3 : ln & 7, jl = N2 == 128 ? ln >> 2 : ln >> 3;
        const int col = 32 * il + 16 * (r0 >> 1) + 2 * (jl ^ il) + (r & 1);
        unsigned char *dst = b1 + (o >> 3) * (N2 * 128) + col * 128 + (((o & 7) ^ (col & 7)) << 4);
        const int sh = 4 * (r & 1) + 2 * pol;
        uint32_t h0[2], h1[2];
        level_quad(t[r0 >> 1][0] >> sh, h0);
        level_quad(t[r0 >> 1][1] >> sh, h1);
        *reinterpret_cast<uint4 *>(dst) = make_uint4(h0[0], h0[1], h1[0], h1[1]);
        if constexpr (DBG) {
          const int w = 8 * o / N1, tl = cur.tg * NW + w;
          if ((vm >> w) & 1u) {
            float2 *pr = p.probe + (((size_t)cur.ant * 2 + pol) * job.nfft + (p.t0 + tl)) * N + 4 * ln + r;
#pragma unroll
            for (int j = 0; j < 8; j++) {
              const uint32_t hb = j < 4 ? h0[j >> 1] : h1[(j - 4) >> 1];
              const float2 hf = __half22float2(*reinterpret_cast<const __half2 *>(&hb));
              pr[N2 * ((8 * o) % N1 + j)] = make_float2((float)((double)((j & 1) ? hf.y : hf.x) * kUnit), 0.f);
            }
          }
        }
      };
      // ---- A1: row (window, k1), K = (window, n1): W_N1^(n1 k1) tstep[n1], hi and lo halves, unless the slot holds it
      //      already
      auto make_a1 = [&]() {
#pragma unroll 1
        for (int x = gt; x < ROWS * N1 / 8; x += GT) {
          const int r = x & (ROWS - 1), cc = (unsigned)x / ROWS, w = r / N1, k1 = r % N1;
          const float2 *ts = tst + w * N1 + 8 * cc;
          uint32_t hr[4], hi[4], lr[4], li[4];
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int n1 = 8 * cc + 2 * e;
            const float2 a = cmul(ts[2 * e], wr[(n1 * k1 * (P::NWR / N1)) & (P::NWR - 1)]);
            const float2 b = cmul(ts[2 * e + 1], wr[((n1 + 1) * k1 * (P::NWR / N1)) & (P::NWR - 1)]);
            const __half2 xr = __floats2half2_rn(a.x, b.x), xi = __floats2half2_rn(a.y, b.y);
            const float2 fr = __half22float2(xr), fi = __half22float2(xi);
            hr[e] = *reinterpret_cast<const uint32_t *>(&xr);
            hi[e] = *reinterpret_cast<const uint32_t *>(&xi);
            constexpr float up = kLevel + P::RZ;
            lr[e] = pack_h2(fmaf(a.x, up, a.x - fr.x), fmaf(b.x, up, b.x - fr.y));
            li[e] = pack_h2(fmaf(a.y, up, a.y - fi.x), fmaf(b.y, up, b.y - fi.y));
          }
          const int ch = w * (N1 / 8) + cc;
          unsigned char *dst = a1 + (ch >> 3) * (ROWS * 128) + r * 128 + (((ch & 7) ^ (r & 7)) << 4);
          *reinterpret_cast<uint4 *>(dst) = make_uint4(hr[0], hr[1], hr[2], hr[3]);
          *reinterpret_cast<uint4 *>(dst + P::APL) = make_uint4(lr[0], lr[1], lr[2], lr[3]);
          *reinterpret_cast<uint4 *>(dst + 2 * P::APL) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4 *>(dst + 3 * P::APL) = make_uint4(li[0], li[1], li[2], li[3]);
        }
      };
      if constexpr (!W1) {
        ok = i < NS || mbar_wait(smem_u32(&ab_free[s]), ((i / NS) - 1) & 1, p.err);
        uint32_t t[2][2];
        load_codes(gt >> 5, lane, t);
#pragma unroll
        for (int r0 = 0; r0 < 4; r0++)
#pragma unroll
          for (int pol = 0; pol < 2; pol++) store_b1(smem + P::off_b(s) + pol * P::BPL, gt >> 5, lane, pol, r0, t);
        if (rebuild) make_a1();
        fence_proxy_async_smem();
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(smem_u32(&ab_full[s]));
      } else {
#pragma unroll 1
        for (int pol = 0; pol < 2; pol++) {
          const int sb = NS == 2 ? pol : 0, use = NS == 2 ? i : 2 * i + pol;  // slot of B1 and its use
          if (use > 0) ok = mbar_wait(smem_u32(&ab_free[sb]), (use - 1) & 1, p.err) && ok;
          if (pol == 0 && rebuild) {  // A1 belongs to both slots: the last group's MMAs are done with it
            if (NS == 2 && i > 0) ok = mbar_wait(smem_u32(&ab_free[1]), (i - 1) & 1, p.err) && ok;
            make_a1();
          }
#pragma unroll 1
          for (int x = gt; x < 4 * N2; x += GT) {
            uint32_t t[2][2];
            const int o = (unsigned)x / (N2 / 4), ln = x & (N2 / 4 - 1);
            load_codes(o, ln, t);
#pragma unroll
            for (int r0 = 0; r0 < 4; r0++) store_b1(smem + P::off_b(sb), o, ln, pol, r0, t);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (ok && lane == 0) mbar_arrive(smem_u32(&ab_full[sb]));
        }
      }
    }
  } else {
    reg_dec<P::REG_MMA>();
    if (lane == 0 && warp == P::W_MMA) {
      // ------------------------------------------------------------ step 1
      for (int v = 0; v < (W1 ? 2 * ng : ng); v++) {  // uses of the slots, in turn
        const int s = v % NS, use = v / NS;
        if (!mbar_wait(smem_u32(&ab_full[s]), use & 1, p.err)) break;
        if (use > 0 && !mbar_wait(smem_u32(&d_free[s]), (use - 1) & 1, p.err)) break;
        tc_fence_after();
        const uint32_t a1 = desc_lo(sbase + P::off_a(s)), b1 = desc_lo(sbase + P::off_b(s));
#pragma unroll
        for (int part = 0; part < 2; part++) {
          const uint32_t ah = a1 + 2 * part * P::APL / 16;
          if constexpr (W1) {  // a pol: A_lo B, A_hi B, eight K steps each
            const uint32_t d = tmem0 + 256u * s + N2 * part;
            constexpr uint32_t idesc = N2 == 256 ? IDESC_N256 : IDESC;
            mma_f16_lo<false>(d, ah + P::APL / 16, b1, idesc);
#pragma unroll
            for (int x = 1; x < 16; x++)
              mma_f16_lo<true>(d, ah + (x < 8 ? P::APL / 16 : 0) + ((x >> 2) & 1) * (ROWS * 128 / 16) + 2 * (x & 3),
                               b1 + ((x >> 2) & 1) * (N2 * 128 / 16) + 2 * (x & 3), idesc);
          } else {
#pragma unroll
            for (int pol = 0; pol < 2; pol++) {
              const uint32_t d = tmem0 + 256u * s + N2 * part + ((uint32_t)(16 * pol) << 16), bh = b1 + pol * P::BPL / 16;
              mma_f16_lo<false>(d, ah + P::APL / 16, bh, IDESC_M64);
#pragma unroll
              for (int x = 1; x < 8; x++)  // A_lo B, A_hi B, four K steps each
                mma_f16_lo<true>(d, ah + (x < 4 ? P::APL / 16 : 0) + 2 * (x & 3), bh + 2 * (x & 3), IDESC_M64);
            }
          }
        }
        mma_commit(smem_u32(&ab_free[s]));
        mma_commit(smem_u32(&d_full[s]));
      }
      mma_commit(smem_u32(&bar_final));
      mbar_wait_drain(smem_u32(&bar_final), 0);  // issued MMAs land before tensor memory is freed
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base_sh, 512);
}

template <int L, typename OutT, bool DBG>
static cudaError_t launch_l(const Params &p, cudaStream_t s) {
  using P = Plan<L>;
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const long long ngrp = (long long)((p.nt + P::NW - 1) / P::NW) * p.job.nant;
  const unsigned grid = (unsigned)(ngrp < nsm ? ngrp : nsm);
  auto kern = fstage_tc32_kernel<L, OutT, DBG>;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, P::SMEM);
  if (e != cudaSuccess) return e;
  kern<<<grid, P::NT, P::SMEM, s>>>(p);
  return cudaGetLastError();
}

template <typename OutT, bool DBG>
static cudaError_t launch_t(const Params &p, cudaStream_t s) {
  switch (p.job.log2F) {
    case 11: return launch_l<11, OutT, DBG>(p, s);
    case 12: return launch_l<12, OutT, DBG>(p, s);
    default: break;
  }
  if constexpr (sizeof(OutT) == 8) {
    if (p.job.log2F == 13) return launch_l<13, OutT, DBG>(p, s);
    if (p.job.log2F == 14) return launch_l<14, OutT, DBG>(p, s);
    if (p.job.log2F == 15) return launch_l<15, OutT, DBG>(p, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace f32tc

// 2048 and 4096 points of 2-bit real data, and 8192 to 32768 points with FP32 output (FP16 and FP8 spectra of 8192
// points have fstage_tc_kernel; those of 16384 and 32768 points keep fstage_h_kernel: without its FP16 roundings between
// passes their results would move).  At 1024 points, whose rows
// hold 8 channels, it measured no faster than the register FFT: 61.4 against 63.5 us for 12 groups per SM.  The
// rotator's phase must be linear over the samples n2 of a row and over the rows: always so in exact mode, in fxkernel
// mode when the table split is at N2 samples (8192 and 32768 points).  The output addresses use a 32-bit channel step.
int fstage_tc32_supported(const Job &job, int T, int chan_type) {
  const int n2 = job.log2F == 15 ? 256 : 128;
  return !job.is_complex && job.log2F >= 11 && (job.log2F <= 12 || (job.log2F <= 15 && chan_type == CHAN_F32)) &&
         (job.rotator == GXC_ROTATOR_EXACT || job.substride == n2) &&
         (unsigned long long)T * 2 * job.nant * CW * (job.log2F <= 13 ? 4 : 8) * sizeof(float2) <= 0xffffffffull;
}

// Three groups of 16384 samples per SM and block, or more: below that the persistent kernel's set-up shows.  FP32, F-stage
// with 2 / 3 / 4 / 12 groups per SM: 2048 points 22.6 / 22.5 / 28.7 / 57.3 us against 18.5 / 26.6 / 32.8 / 82.0 for the
// register FFT; 8192 points 18.4 / 22.6 / 26.6 / 59.4 against 20.4 / 26.7 / 32.8 / 81.9.  From 16384 points on, one
// window per SM: with 1 / 2 / 12 of them 20.1 / 30.3 / 129 us against 22.5 / 41.0 / 233 (16384 points), 34.4 / 59.0 / 282
// against 65.5 / 127 / 764 (32768 points, whose cluster kernel spreads fewer windows over more SMs).
int fstage_tc32_worth(const Job &job, int T, int chan_type) {
  int dev = 0, nsm = 0;
  if (!fstage_tc32_supported(job, T, chan_type) || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  const long long nw = job.F < 8192 ? 8192 / job.F : 1;  // windows per group
  return ((long long)T + nw - 1) / nw * job.nant >= (job.log2F >= 14 ? 1LL : 3LL) * nsm;
}

cudaError_t launch_fstage_tc32(const Job &job, int t0, int nt, int T, void *chan, int chan_type, float out_scale,
                               cudaStream_t s, const float *cscale, float2 *probe) {
  if (nt <= 0) return cudaSuccess;
  if (!fstage_tc32_supported(job, T, chan_type)) return cudaErrorInvalidValue;
  f32tc::Params p;
  p.job = job;
  p.t0 = t0;
  p.nt = nt;
  p.T = T;
  p.chan = chan;
  p.out_scale = out_scale;
  p.cscale = cscale;
  p.probe = probe;
  cudaError_t e = cudaGetSymbolAddress((void **)&p.err, f32tc::g_f32tc_err);
  if (e != cudaSuccess) return e;
  if (probe) {
    if (chan_type == CHAN_F32) return f32tc::launch_t<float2, true>(p, s);
    if (chan_type == CHAN_F8) return f32tc::launch_t<__nv_fp8x2_e4m3, true>(p, s);
    return f32tc::launch_t<__half2, true>(p, s);
  }
  if (chan_type == CHAN_F32) return f32tc::launch_t<float2, false>(p, s);
  if (chan_type == CHAN_F8) return f32tc::launch_t<__nv_fp8x2_e4m3, false>(p, s);
  return f32tc::launch_t<__half2, false>(p, s);
}

// Reads and clears the error flag (a bounded wait expired).
cudaError_t fstage_tc32_take_error(int *flag) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(flag, f32tc::g_f32tc_err, sizeof(int));
  if (e == cudaSuccess && *flag) e = cudaMemcpyToSymbol(f32tc::g_f32tc_err, &zero, sizeof(int));
  return e;
}

}  // namespace gxc
