// Tensor-core F-stage: 8192-point windows of 2-bit real data with FP16 or FP8
// channelised output, the FFT as two dense DFT products on tcgen05.
//
// Four-step factorisation N = 8192 = N1 x N2, N1 = 64, N2 = 128, n = n2 + 128 n1,
// k = k1 + 64 k2 (fxkernel's dofft, fxkernel/src/fxkernel.cpp:569-580, is the
// plain unnormalised forward DFT this restates):
//   X[k1 + 64 k2] = sum_n2 W128^(n2 k2) [ W8192^(n2 k1) sum_n1 W64^(n1 k1) x[n2 + 128 n1] ].
// Step 1 is a real GEMM, D1 = A1 B1_pol^T (M = 64 rows k1, N = 128 columns n2, K = n1) for the real and the
// imaginary part of each polarisation: A1 is Re / Im of DFT64, B1 the decoded window.  The M = 64 results of the two
// polarisations interleave by 16 tensor-memory lanes, so lane (pol, k1) holds Re and Im of Y[k1][n2] for every n2.
// The twiddle W8192^(n2 k1) and the fine part of the fractional-sample-delay correction, fsubt[k1], are applied on
// the CUDA cores; the product, rounded to FP16, goes back to tensor memory as the A operand of step 2, D3 = A3 B3^T
// (M = 128 rows (pol, k1), K = [Re, Im of Y' over n2], N = [Re, Im of X over k2 < 64]; real data keeps channels
// k < 4096).  B3 is the real form of the first 64 rows of DFT128.  The coarse frac-delay factor fstept[k2], the
// output scale and the cast are applied as D3 leaves tensor memory.
//
// Operands are FP16 (kind::f16) with FP32 accumulation in tensor memory.  The FFT then carries four FP16 roundings
// (the levels, both DFT matrices and the twiddled intermediate) on top of the FP16 / FP8 output rounding; it serves
// the FP16 and FP8 channelised paths only (the FP32 path keeps the CUDA-core FFT).
//
// The rotator and frac-delay tables of the fxkernel layout fall on the four-step indices: with stride 64 and
// substride 128 (fxkernel.cpp:57-64), sample n has rotator tsub[n2] * tstep[n1] and channel k frac-delay
// fsubt[k1] * fstept[k2].  tstep[n1] is folded into a per-window A1 (Re / Im of W64^(n1 k1) tstep[n1]), so B1 holds
// the real 2-bit levels and step 1 has K = 64; tsub[n2] joins the twiddle recurrence.
//
// One persistent CTA per SM (28 warps, about 175 KB of shared memory) runs the steps of neighbouring windows at the
// same time: 8 warps decode window i + 1 (and build its A1) while 8 warps twiddle window i and 8 warps write window
// i - 1 out; two more issue the MMAs of the two steps.  Mbarriers connect them; two operand slots and two 256-column
// tensor-memory slots are in flight.
//
// What bounds it (16 antennas, 2048 FFTs, ncu): 20 warp instructions per 32 samples at 56 % issue active, FMA pipe
// 40 %, tensor pipe 45 %, shared-memory data path 40 % + 28 % for MMA operands, DRAM 28 %; a window holds its
// tensor-memory slot for about 9,300 clocks (MMAs, 3,400 for the twiddle, 2,500 for the output), and two slots give
// one window per 4,850.  F-stage of the 16-antenna, nchan-4096 workload, FP16, 31250 FFTs: 7.4 ms; 15.5 ms for
// fstage_tc_cross_kernel (one 512-thread CTA that goes through the phases of a window together, the intermediate in shared
// memory written by 2-byte stores); 20.0 ms for the register FFT.
//
// Every mbarrier wait is bounded; on expiry the kernel sets an error flag (read by gxc_sync as GXC_ERR_TIMEOUT), lets
// issued MMAs drain, frees tensor memory and returns.
#include "fstage_kernels.cuh"
#include "gxc_internal.h"
#include "tcgen05_util.cuh"

#include <math.h>
#include <vector>

namespace gxc {

namespace ftc {

constexpr int N1 = 64, N2 = 128, F = N1 * N2, NCHAN = F / 2;
constexpr int SUB = 128, STRIDE = 64, FSUB = 64;  // rotator / frac-delay table split of nchan 4096
// warp roles: 8 twiddle warps, 8 output warps, 8 decode warps, one warp per MMA step (and two that idle: registers
// are shared out by warpgroups of four warps, out of 28 x 32 x 72)
constexpr int RW = 8, GT = RW * 32;
constexpr int W_OUT = RW, W_DEC = 2 * RW, W_MMA1 = 3 * RW, W_MMA2 = 3 * RW + 1;
constexpr int NT = (3 * RW + 4) * 32;
constexpr int REG_TWIDDLE = 88, REG_OUT = 64, REG_DEC = 80, REG_MMA = 40;
static_assert(2 * (REG_TWIDDLE + REG_OUT + REG_DEC) + REG_MMA <= 7 * 72, "register shares");
constexpr int NS = 2;                               // operand / tensor-memory slots (windows in flight)
constexpr int NR = 4;                               // table ring (windows between decode and output)
constexpr int KB = 128 * 128;                       // one 128-row SW128 K-block (64 FP16 K-elements)
constexpr int HB = KB / 2;                          // 64 rows of one
// shared-memory image (byte offsets from a 1024-aligned base)
constexpr int OFF_B3 = 0;                  // DFT128 rows k2 < 64, 4 K-blocks (constant)
constexpr int OFF_A1 = OFF_B3 + 4 * KB;     // per slot: A1 Re (64 rows k1, K = n1), A1 Im
constexpr int OFF_B1 = OFF_A1 + 2 * NS * HB;  // per slot: B1 of pol 0 (1 K-block), B1 of pol 1 (1)
constexpr int OFF_STAGE = OFF_B1 + 2 * NS * KB;     // two buffers: the packed window, realigned
constexpr int STAGE_BYTES = F / 2;
// per ring entry: frac-delay steps e^(2 pi i 64 k2 cf) * scale as pairs (re re' im im'), fsubt[64],
// tstep[8 c] (8), tstep[1], tsub[0..3], tsub steps of 4 and 8
constexpr int TAB_F2 = 64 + 64 + 16;
constexpr int TAB_BYTES = TAB_F2 * 8;
constexpr int T_FSTEP = 0, T_FSUB = 64, T_TSTEP8 = 128, T_TSTEP1 = 136, T_TSUB = 137, T_TSUB4 = 141, T_TSUB8 = 142;
constexpr int OFF_TAB = OFF_STAGE + 2 * STAGE_BYTES;
constexpr int SMEM_BYTES = OFF_TAB + NR * TAB_BYTES + 1024;  // + alignment slack
constexpr int CONST_BYTES = 4 * KB;
// global table image: B3 in its swizzled shared-memory layout
constexpr int TABLE_BYTES = CONST_BYTES;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

struct Params {
  Job job;
  const uint4 *tables;  // TABLE_BYTES image (make_fstage_tc_tables)
  int t0, nt, T;
  void *chan;
  float out_scale;
  const float *cscale;  // FP8 output: per-channel scale [nchan] (replaces out_scale), or null
  float2 *probe;        // decode probe (DBG kernels): [nant][2][nfft][F] decoded samples
  int *err;
};

__device__ int g_ftc_err;

// byte offset of FP16 element (row, k) in a SW128 K-major tile of 128-byte rows
__host__ __device__ inline int sw128_off(int row, int k) {
  return row * 128 + ((((k >> 3) ^ (row & 7)) & 7) << 4) + (k & 7) * 2;
}
// tensor-memory column (= row of B1) of sample n2: 32 (n2 mod 4) + n2 / 4.  A thread decodes the four samples of
// two neighbouring bytes; this order puts consecutive threads on consecutive rows, so their 16-byte stores hit all
// eight swizzle positions.
__host__ __device__ inline int col_of_n2(int n2) { return 32 * (n2 & 3) + (n2 >> 2); }

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  const __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t *>(&h);
}

// FP16 levels of four 2-bit codes, one per byte of `codes` (lowest two bits; the others are ignored): the level
// table of fxkernel.cpp:17-18 {-HiMag, -1, 1, HiMag} as FP16 bit patterns.  kLo holds the low bytes of the four
// levels, kHi the high bytes, so code c picks bytes c and 4 + c of {kHi:kLo}: the byte-permute selectors of all four
// codes come from one multiply-add.  HiMag = 3.3359 is 3.3359375 in FP16, the nearest half.
__device__ __forceinline__ void level_quad_h2(uint32_t codes, uint32_t &h01, uint32_t &h23) {
  constexpr uint32_t kLo = 0xAC0000ACu, kHi = 0x423CBCC2u;  // 0xC2AC, 0xBC00, 0x3C00, 0x42AC for codes 0..3
  const uint32_t sel = (codes & 0x03030303u) * 0x11u + 0x40404040u;
  h01 = tc::prmt(kLo, kHi, sel);
  h23 = tc::prmt(kLo, kHi, sel >> 16);
}

// The packed bytes of a window in flight: words gt + 256 j of the window and the one after each, counted from the
// 4-byte boundary before its first sample, `shift` bits before it.
struct Prefetch {
  uint32_t w[5];
  int shift;
};

// Starts the loads of this thread's words of a valid window (the buffer holds (nfft+1)*F samples and
// offset <= (nfft-1)*F, so the window plus one word stays inside it).
__device__ __forceinline__ void prefetch_window(const uint8_t *in, const Geom &g, int gt, Prefetch &pf) {
  const long long b0 = (long long)g.offset >> 1;
  const uint32_t *src = reinterpret_cast<const uint32_t *>(in + (b0 & ~3LL)) + gt;
  pf.shift = (int)(b0 & 3) * 8 + (g.offset & 1) * 4;
#pragma unroll
  for (int i = 0; i < 4; i++) pf.w[i] = __ldg(src + GT * i);
  // a warp's last word needs the first one after its row: lanes 0..3 fetch that of rows 0..3
  const int lane = gt & 31;
  pf.w[4] = lane < 4 ? __ldg(src - lane + GT * lane + 32) : 0u;
}

// Window w of the block, as (antenna, FFT); advanced by a fixed stride without a division.
struct Win {
  int ant, tl;
  __device__ __forceinline__ Win(int w, int nant) : ant(w % nant), tl(w / nant) {}
  __device__ __forceinline__ void advance(int da, int dt, int nant) {
    ant += da;
    tl += dt;
    if (ant >= nant) {
      ant -= nant;
      tl++;
    }
  }
};

// Writes the prefetched window, shifted so that its first sample starts word 0, and the window's tables (one
// sincos per thread).
__device__ __forceinline__ void stage_window(const Params &p, const Geom &g, const Prefetch &pf, unsigned char *stage,
                                             float2 *tab, int gt) {
  const int lane = gt & 31;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const uint32_t up = __shfl_down_sync(0xffffffffu, pf.w[i], 1), last = __shfl_sync(0xffffffffu, pf.w[4], i);
    reinterpret_cast<uint32_t *>(stage)[gt + GT * i] = __funnelshift_r(pf.w[i], lane < 31 ? up : last, pf.shift);
  }
  if (gt > T_TSUB8) return;
  float arg;  // half turns
  if (gt < T_FSUB) arg = 2.0f * ((float)(gt * FSUB) * g.cf);
  else if (gt < T_TSTEP8) arg = 2.0f * ((float)(gt - T_FSUB) * g.cf);
  else if (gt < T_TSTEP1) arg = -2.0f * ((float)(8 * (gt - T_TSTEP8)) * g.cstep);
  else if (gt == T_TSTEP1) arg = -2.0f * g.cstep;
  else if (gt < T_TSUB4) arg = -2.0f * fmaf((float)(gt - T_TSUB), g.c1, g.c0);
  else arg = -2.0f * ((gt == T_TSUB4 ? 4.0f : 8.0f) * g.c1);
  float sn, cs;
  sincospif(arg, &sn, &cs);
  if (gt < T_FSUB) {  // the output scale is a power of two: folding it in is exact
    float *f = reinterpret_cast<float *>(tab + T_FSTEP) + (gt >> 1) * 4 + (gt & 1);
    f[0] = cs * p.out_scale;
    f[2] = sn * p.out_scale;
  } else {
    tab[gt] = make_float2(cs, sn);
  }
}

// Decodes the staged window into B1 (both pols): row col_of_n2(n2), K = n1, the real 2-bit levels.
template <bool DBG>
__device__ __forceinline__ void decode_window(const Params &p, const Win &w, const unsigned char *stage,
                                              unsigned char *b1, int gt) {
  const int lane = gt & 31, o = gt >> 5;  // samples n2 = 4 lane .. 4 lane + 3 of rows n1 = 8 o .. 8 o + 7
  {
    const uint16_t *src = reinterpret_cast<const uint16_t *>(stage + 64 * 8 * o) + lane;
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = src[32 * i];
    uint32_t t[2][2];  // [byte of the pair][n1 quad]: byte i = n1 i, codes (A B A' B') of two samples
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const uint32_t p01 = tc::prmt(v[4 * q], v[4 * q + 1], 0x5410), p23 = tc::prmt(v[4 * q + 2], v[4 * q + 3], 0x5410);
      t[0][q] = tc::prmt(p01, p23, 0x6420);
      t[1][q] = tc::prmt(p01, p23, 0x7531);
    }
    unsigned char *dst = b1 + lane * 128 + ((o ^ (lane & 7)) << 4);
#pragma unroll
    for (int r = 0; r < 4; r++)  // sample n2 = 4 lane + r: row 32 r + lane
#pragma unroll
      for (int pol = 0; pol < 2; pol++) {
        const int sh = 4 * (r & 1) + 2 * pol;
        uint4 h;
        level_quad_h2(t[r >> 1][0] >> sh, h.x, h.y);
        level_quad_h2(t[r >> 1][1] >> sh, h.z, h.w);
        *reinterpret_cast<uint4 *>(dst + pol * KB + r * 32 * 128) = h;
        if constexpr (DBG) {
          const Job &job = p.job;
          float2 *pr = p.probe + (((size_t)w.ant * 2 + pol) * job.nfft + (p.t0 + w.tl)) * F + 4 * lane + r;
#pragma unroll
          for (int i = 0; i < 8; i++)
            pr[128 * (8 * o + i)] = make_float2(level2bit((int)((t[r >> 1][i >> 2] >> (8 * (i & 3) + sh)) & 3u)), 0.f);
        }
      }
  }
}

// Builds the window's A1.  The rotator of sample n = n2 + 128 n1 is tsub[n2] tstep[n1]: tstep[n1] goes into A1 (row k1,
// column n1: Re / Im of W64^(n1 k1) tstep[n1], one FP16 rounding), tsub[n2] into the twiddle.
//   wa = W64^k1, wc[j] = W64^(8 c k1) of this thread's two column chunks c = 2 (gt / 64) + j, k1 = gt mod 64.
__device__ __forceinline__ void build_a1(const float2 *tab, unsigned char *a1, int gt, float2 wa,
                                         const float2 (&wc)[2]) {
  // the thread's two column chunks are the two lanes of packed FP32 pairs, advanced along n1 by tstep[1] W64^k1
  const int k1 = gt & 63, c0 = 2 * (gt >> 6);
  const float2 st = cmul(tab[T_TSTEP1], wa);
  const float2 SR = make_float2(st.x, st.x), SI = make_float2(st.y, st.y), NSI = make_float2(-st.y, -st.y);
  const float2 e0 = cmul(tab[T_TSTEP8 + c0], wc[0]), e1 = cmul(tab[T_TSTEP8 + c0 + 1], wc[1]);
  float2 R = make_float2(e0.x, e1.x), I = make_float2(e0.y, e1.y);
  uint32_t hr[2][4], hi[2][4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const float2 R0 = R, I0 = I;
    R = pfma(R0, SR, pmul(I0, NSI));
    I = pfma(R0, SI, pmul(I0, SR));
    hr[0][e] = pack_h2(R0.x, R.x);
    hr[1][e] = pack_h2(R0.y, R.y);
    hi[0][e] = pack_h2(I0.x, I.x);
    hi[1][e] = pack_h2(I0.y, I.y);
    if (e < 3) {
      const float2 nr = pfma(R, SR, pmul(I, NSI));
      I = pfma(R, SI, pmul(I, SR));
      R = nr;
    }
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    unsigned char *dst = a1 + k1 * 128 + (((c0 + j) ^ (k1 & 7)) << 4);
    *reinterpret_cast<uint4 *>(dst) = make_uint4(hr[j][0], hr[j][1], hr[j][2], hr[j][3]);
    *reinterpret_cast<uint4 *>(dst + HB) = make_uint4(hi[j][0], hi[j][1], hi[j][2], hi[j][3]);
  }
}

// DBG = true (decode probe): every decoded sample is also written to p.probe before the rotation.
template <typename OutT, bool DBG = false>
__global__ void __launch_bounds__(NT, 1) fstage_tc_kernel(Params p) {
  using namespace tc;
  extern __shared__ unsigned char smem_raw[];
  // handshakes, one phase per valid window of a slot: ab_full (decode -> step 1), ab_free (step 1 done -> decode),
  // d1_full (step 1 -> twiddle), a3_full (twiddle -> step 2), d3_full (step 2 -> output), d_free (output -> step 1);
  // of a table ring entry, one phase per window: tab_full (decode -> all roles), tab_free (all roles -> decode)
  __shared__ __align__(8) uint64_t ab_full[NS], ab_free[NS], d1_full[NS], a3_full[NS], d3_full[NS], d_free[NS],
      tab_full[NR], tab_free[NR], bar_final[2];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int ring_valid[NR];
  unsigned char *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = smem_u32(smem);
  const Job &job = p.job;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nant = job.nant, nstreams = 2 * nant;
  const size_t ctile_stride = (size_t)p.T * nstreams * CW;
  OutT *chan = reinterpret_cast<OutT *>(p.chan);

  // constant operand B3, once per CTA
  for (int i = tid; i < CONST_BYTES / 16; i += NT)
    *reinterpret_cast<uint4 *>(smem + OFF_B3 + 16 * i) = __ldg(&p.tables[i]);
  if (tid == 0) {
    for (int s = 0; s < NS; s++) {
      mbar_init(smem_u32(&ab_full[s]), RW);
      mbar_init(smem_u32(&ab_free[s]), 1);
      mbar_init(smem_u32(&d1_full[s]), 1);
      mbar_init(smem_u32(&a3_full[s]), RW);
      mbar_init(smem_u32(&d3_full[s]), 1);
      mbar_init(smem_u32(&d_free[s]), RW);
    }
    for (int s = 0; s < NR; s++) {
      mbar_init(smem_u32(&tab_full[s]), 1);
      mbar_init(smem_u32(&tab_free[s]), 2 * RW + 2);
    }
    mbar_init(smem_u32(&bar_final[0]), 1);
    mbar_init(smem_u32(&bar_final[1]), 1);
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

  // slot s has 256 tensor-memory columns: D1 Re at [0, 128), D1 Im at [128, 256); the twiddled A3 takes the place
  // of D1 Im, the result D3 that of D1 Re
  const uint32_t tmem0 = tmem_base_sh;
  float2 *const tab0 = reinterpret_cast<float2 *>(smem + OFF_TAB);
  const int nwin = p.nt * nant, G = (int)gridDim.x;
  const int da = G % nant, dt = G / nant;
  auto root = [](int num, int den) {  // exp(-2 pi i num / den)
    float sn, cs;
    sincospif(-2.0f * (float)num / (float)den, &sn, &cs);
    return make_float2(cs, sn);
  };
  int c = 0;  // valid windows of this CTA so far (every role counts them alike)
  int i = 0;  // windows

  if (warp < W_OUT) {
    reg_inc<REG_TWIDDLE>();
    // ------------------------------------------------------------ twiddle
    // Fringe phase of n2, twiddle and fine frac-delay, FP16, into A3 (K order: 16 columns of Re, then 16 of Im).  Run
    // r of 32 columns holds n2 = 4 l + r: its factor W8192^(n2 k1) tsub[n2] fsubt[k1] is geometric in l (over 32
    // steps the recurrence's rounding stays near 3e-6, far below FP16's), and columns l, l + 1 are the two lanes of
    // packed FP32 pairs.  Warps w and w + 4 share a lane quarter, two runs each.
    const int q = warp & 3, h = warp >> 2;
    const int k1 = 16 * q + (lane & 15);  // lane 16 pol + k1 mod 16 of quarter k1 / 16
    const float2 wr0 = root(2 * h * k1, F), wr1 = root((2 * h + 1) * k1, F), w4 = root(4 * k1, F), w8 = root(8 * k1, F);
    for (int w = blockIdx.x; w < nwin; w += G, i++) {
      const int ri = i % NR, rp = (i / NR) & 1;
      if (!mbar_wait_warp(smem_u32(&tab_full[ri]), rp, p.err)) break;
      const float2 *tab = tab0 + ri * TAB_F2;
      const int valid = ring_valid[ri];
      const float2 s1 = cmul(w4, tab[T_TSUB4]), s2 = cmul(w8, tab[T_TSUB8]), fs = tab[T_FSUB + k1];
      const float2 ts0 = tab[T_TSUB + 2 * h], ts1 = tab[T_TSUB + 2 * h + 1];
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tab_free[ri]));
      if (!valid) continue;
      const int s = c % NS;
      const uint32_t trow = tmem0 + 256u * s + ((uint32_t)(32 * q) << 16) + 64u * h;
      const float2 SR = make_float2(s2.x, s2.x), SI = make_float2(s2.y, s2.y), NSI = make_float2(-s2.y, -s2.y);
      if (!mbar_wait_warp(smem_u32(&d1_full[s]), (c / NS) & 1, p.err)) break;
      tc_fence_after();
#pragma unroll 1
      for (int rr = 0; rr < 2; rr++) {
        const float2 w0 = cmul(cmul(rr ? wr1 : wr0, rr ? ts1 : ts0), fs), w1 = cmul(w0, s1);
        float2 WR = make_float2(w0.x, w1.x), WI = make_float2(w0.y, w1.y);
#pragma unroll
        for (int ch = 0; ch < 2; ch++) {
          float re[16], im[16];
          tmem_ld16_async(trow + 32 * rr + 16 * ch, re);
          tmem_ld16_async(trow + 128 + 32 * rr + 16 * ch, im);
          tmem_wait_ld16(re);
          tmem_wait_ld16(im);
          uint32_t a3[16];
#pragma unroll
          for (int e = 0; e < 8; e++) {
            const float2 VR = make_float2(re[2 * e], re[2 * e + 1]), VI = make_float2(im[2 * e], im[2 * e + 1]);
            const float2 yr = csub(pmul(VR, WR), pmul(VI, WI)), yi = pfma(VR, WI, pmul(VI, WR));
            a3[e] = pack_h2(yr.x, yr.y);
            a3[8 + e] = pack_h2(yi.x, yi.y);
            const float2 nr = pfma(WR, SR, pmul(WI, NSI));
            WI = pfma(WR, SI, pmul(WI, SR));
            WR = nr;
          }
          tmem_st16(trow + 128 + 32 * rr + 16 * ch, a3);
        }
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&a3_full[s]));
      c++;
    }
  } else if (warp < W_DEC) {
    reg_dec<REG_OUT>();
    // ------------------------------------------------------------ output
    // Frac-delay step, scale, cast, store: lane 16 pol + k1 mod 16 of quarter k1 / 16, columns 16 (k2 / 8) + 8 part +
    // k2 mod 8.  Warps w and w + 4 share a lane quarter, half of k2 each.  A warp's lanes are the 16 channels of a
    // tile for both pols, neighbouring rows of the channelised layout: each store is one contiguous 128-byte line
    // (FP16).
    const int q = warp & 3, h = (warp - W_OUT) >> 2;
    const int pol = lane >> 4, k1 = 16 * q + (lane & 15);
    const float *csc = p.cscale ? p.cscale + k1 + 64 * 32 * h : nullptr;
    const uint32_t step = (uint32_t)(4 * ctile_stride * sizeof(OutT));  // bytes from k2 to k2 + 1 (below 4 GB: launcher)
    OutT *const o0 = chan + (size_t)pol * CW + (k1 & 15) + (size_t)((k1 >> 4) + 4 * 32 * h) * ctile_stride;
    Win win(blockIdx.x, nant);
    for (int w = blockIdx.x; w < nwin; w += G, i++, win.advance(da, dt, nant)) {
      const int ri = i % NR, rp = (i / NR) & 1;
      if (!mbar_wait_warp(smem_u32(&tab_full[ri]), rp, p.err)) break;
      if (ring_valid[ri]) {
        const int s = c % NS;
        // FP8: the scales of eight channels, loaded one step ahead (before the wait for the first ones).  Loaded where they
        // were used they held this role up: 62500 FFTs of 16 antennas 17.4 ms, now 16.7 (FP16 without scales 14.8)
        constexpr bool SCALED = std::is_same<OutT, __nv_fp8x2_e4m3>::value;
        float scn[8];
        auto load_scales = [&](int jj) {
#pragma unroll
          for (int e = 0; e < 8; e++) scn[e] = chan_scale<OutT>(csc, 64 * (8 * jj + e), 1.0f);
        };
        if constexpr (SCALED) load_scales(0);
        if (!mbar_wait_warp(smem_u32(&d3_full[s]), (c / NS) & 1, p.err)) break;
        tc_fence_after();
        const uint32_t trow = tmem0 + 256u * s + ((uint32_t)(32 * q) << 16) + 64u * h;
        unsigned char *o = reinterpret_cast<unsigned char *>(o0 + ((size_t)win.tl * nstreams + 2 * win.ant) * CW);
        const float4 *ft = reinterpret_cast<const float4 *>(tab0 + ri * TAB_F2 + T_FSTEP) + 16 * h;
#pragma unroll
        for (int jj = 0; jj < 4; jj++) {
          float v[16];
          tmem_ld16_async(trow + 16 * jj, v);
          float sc[8];
#pragma unroll
          for (int e = 0; e < 8; e++) sc[e] = SCALED ? scn[e] : 1.0f;
          if constexpr (SCALED) {
            if (jj < 3) load_scales(jj + 1);
          }
          tmem_wait_ld16(v);
          if (jj == 3) {  // D3 has been read: step 1 of the slot's next window may overwrite it
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&d_free[s]));
          }
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float4 f = ft[4 * jj + e];
            const float2 FR = make_float2(f.x, f.y), FI = make_float2(f.z, f.w);
            const float2 VR = make_float2(v[2 * e], v[2 * e + 1]), VI = make_float2(v[8 + 2 * e], v[9 + 2 * e]);
            const float2 zr = csub(pmul(VR, FR), pmul(VI, FI)), zi = pfma(VR, FI, pmul(VI, FR));
            const uint32_t k2 = 8 * jj + 2 * e;
            *reinterpret_cast<OutT *>(o + (uint64_t)k2 * step) =
                to_out<OutT>(make_float2(zr.x, zi.x), sc[2 * e]);
            *reinterpret_cast<OutT *>(o + (uint64_t)(k2 + 1) * step) =
                to_out<OutT>(make_float2(zr.y, zi.y), sc[2 * e + 1]);
          }
        }
        c++;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tab_free[ri]));
    }
  } else if (warp < W_MMA1) {
    reg_inc<REG_DEC>();
    // ------------------------------------------------------------ decode
    // Window i + 1's geometry record loads while window i's samples are decoded, its bytes while A1 is built.
    const int gt = tid - 32 * W_DEC;
    const int ka = gt & 63, ca = 2 * (gt >> 6);
    const float2 wa = root(ka, 64);
    const float2 wc[2] = {root((8 * ca * ka) & 63, 64), root((8 * (ca + 1) * ka) & 63, 64)};
    Win win(blockIdx.x, nant);
    Geom g;
    Prefetch pf;
    if ((int)blockIdx.x < nwin) {
      g = job.geom[(size_t)win.ant * job.nfft + p.t0 + win.tl];
      if (g.valid) prefetch_window(job.inputs[win.ant], g, gt, pf);
    }
    bool ok = true;
    for (int w = blockIdx.x; w < nwin; w += G, i++) {
      const int ri = i % NR, rp = (i / NR) & 1;
      unsigned char *stage = smem + OFF_STAGE + (i & 1) * STAGE_BYTES;
      float2 *tab = tab0 + ri * TAB_F2;
      ok = i < NR || mbar_wait(smem_u32(&tab_free[ri]), rp ^ 1, p.err);
      const int valid = g.valid;
      if (valid) stage_window(p, g, pf, stage, tab, gt);
      if (gt == 0) ring_valid[ri] = valid;
      const Win cur = win;
      const bool more = w + G < nwin;
      win.advance(da, dt, nant);
      const uint8_t *in = nullptr;
      if (more) {
        g = job.geom[(size_t)win.ant * job.nfft + p.t0 + win.tl];
        in = job.inputs[win.ant];
      }
      // the staged window and tables are complete (and the other staging buffer's readers are done)
      if (!group_sync_and(1, GT, ok)) break;
      if (gt == 0) mbar_arrive(smem_u32(&tab_full[ri]));
      const int s = c % NS;
      unsigned char *const b1 = smem + OFF_B1 + 2 * s * KB, *const a1 = smem + OFF_A1 + 2 * s * HB;
      if (valid) {
        ok = c < NS || mbar_wait(smem_u32(&ab_free[s]), ((c / NS) - 1) & 1, p.err);
        decode_window<DBG>(p, cur, stage, b1, gt);
      }
      if (more && g.valid) prefetch_window(in, g, gt, pf);
      if (valid) {
        build_a1(tab, a1, gt, wa, wc);
        fence_proxy_async_smem();
        __syncwarp();
        if (ok && lane == 0) mbar_arrive(smem_u32(&ab_full[s]));
        c++;
      } else {
        // flagged: the X-stage sums zeros, the baseline counts exclude this FFT
        OutT *out0 = chan + ((size_t)cur.tl * nstreams + 2 * cur.ant) * CW;  // pol 0; pol 1 is CW further
        const OutT z = to_out<OutT>(make_float2(0.f, 0.f), 1.f);
        for (int j = gt; j < 2 * NCHAN; j += GT) {
          const int zp = j / NCHAN, ch = j - zp * NCHAN;
          out0[(size_t)zp * CW + (size_t)(ch >> 4) * ctile_stride + (ch & 15)] = z;
        }
      }
    }
  } else {
    reg_dec<REG_MMA>();
    if (lane == 0 && warp == W_MMA1) {
      // ------------------------------------------------------------ step 1
      // D1 (lane of (pol, k1), column of n2) = A1 x B1_pol^T, Re and Im: M = 64 (k1), the two pols interleaved by 16 lanes
      for (int w = blockIdx.x; w < nwin; w += G, i++) {
        const int ri = i % NR, rp = (i / NR) & 1;
        if (!mbar_wait(smem_u32(&tab_full[ri]), rp, p.err)) break;
        const int valid = ring_valid[ri];
        mbar_arrive(smem_u32(&tab_free[ri]));
        if (!valid) continue;
        const int s = c % NS;
        if (!mbar_wait(smem_u32(&ab_full[s]), (c / NS) & 1, p.err)) break;
        if (c >= NS && !mbar_wait(smem_u32(&d_free[s]), ((c / NS) - 1) & 1, p.err)) break;
        tc_fence_after();
        const uint32_t a1 = desc_lo(sbase + OFF_A1 + 2 * s * HB), b1 = desc_lo(sbase + OFF_B1 + 2 * s * KB);
#pragma unroll
        for (int part = 0; part < 2; part++)
#pragma unroll
          for (int pol = 0; pol < 2; pol++) {
            const uint32_t d = tmem0 + 256u * s + 128 * part + ((uint32_t)(16 * pol) << 16);
            const uint32_t a = a1 + part * HB / 16, b = b1 + pol * KB / 16;
            mma_f16_lo<false>(d, a, b, IDESC_M64);
#pragma unroll
            for (int kk = 1; kk < 4; kk++) mma_f16_lo<true>(d, a + 2 * kk, b + 2 * kk, IDESC_M64);
          }
        mma_commit(smem_u32(&ab_free[s]));
        mma_commit(smem_u32(&d1_full[s]));
        c++;
      }
      mma_commit(smem_u32(&bar_final[0]));
      mbar_wait_drain(smem_u32(&bar_final[0]), 0);  // issued MMAs land before tensor memory is freed
    } else if (lane == 0 && warp == W_MMA2) {
      // ------------------------------------------------------------ step 2
      // D3 = A3 B3^T, K = 256, A3 from tensor memory
      for (int w = blockIdx.x; w < nwin; w += G, i++) {
        const int ri = i % NR, rp = (i / NR) & 1;
        if (!mbar_wait(smem_u32(&tab_full[ri]), rp, p.err)) break;
        const int valid = ring_valid[ri];
        mbar_arrive(smem_u32(&tab_free[ri]));
        if (!valid) continue;
        const int s = c % NS;
        if (!mbar_wait(smem_u32(&a3_full[s]), (c / NS) & 1, p.err)) break;
        tc_fence_after();
        const uint32_t d = tmem0 + 256u * s, b3 = desc_lo(sbase + OFF_B3);
        mma_f16_ts_lo<false>(d, d + 128, b3, IDESC);
#pragma unroll
        for (int kk = 1; kk < 16; kk++)
          mma_f16_ts_lo<true>(d, d + 128 + 8 * kk, b3 + (kk >> 2) * KB / 16 + 2 * (kk & 3), IDESC);
        mma_commit(smem_u32(&d3_full[s]));
        c++;
      }
      mma_commit(smem_u32(&bar_final[1]));
      mbar_wait_drain(smem_u32(&bar_final[1]), 0);
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0) tmem_dealloc(tmem_base_sh, 512);
}

}  // namespace ftc

int fstage_tc_supported(const Job &job, int chan_type) {
  return chan_type != CHAN_F32 && !job.is_complex && job.F == ftc::F && job.nchan == ftc::NCHAN &&
         job.stride == ftc::STRIDE && job.substride == ftc::SUB && job.fsub == ftc::FSUB &&
         job.fstride == ftc::STRIDE;
}

// Table image: B3 = real form of DFT128 rows k2 < 64, FP16 rounded once from double, in its swizzled
// shared-memory layout.
cudaError_t make_fstage_tc_tables(void **out) {
  using namespace ftc;
  std::vector<unsigned char> img((size_t)TABLE_BYTES, 0);
  const double pi = 3.14159265358979323846;
  auto put = [&](int base, int kb, int row, int k, double v) {
    const __half h = __double2half(v);
    memcpy(&img[(size_t)base + (size_t)kb * KB + (size_t)sw128_off(row, k)], &h, 2);
  };
  // B3 row 16 (k2 / 8) + 8 part + k2 mod 8 (k2 < 64); K element 16 s + e: MMA step s holds, of the 16 columns
  // 16 (s / 2) + e of D1, the real parts (s even) or the imaginary parts (s odd)
  for (int k2 = 0; k2 < N2 / 2; k2++)
    for (int n2 = 0; n2 < N2; n2++) {
      const double ps = 2.0 * pi * (double)((n2 * k2) % N2) / (double)N2;
      const double cs = cos(ps), sn = sin(ps);
      const int row = 16 * (k2 >> 3) + (k2 & 7), col = col_of_n2(n2);
      const int kre = 32 * (col >> 4) + (col & 15), kim = kre + 16;
      put(0, kre >> 6, row, kre & 63, cs);
      put(0, kim >> 6, row, kim & 63, sn);
      put(0, kre >> 6, row + 8, kre & 63, -sn);
      put(0, kim >> 6, row + 8, kim & 63, cs);
    }
  cudaError_t e = cudaMalloc(out, img.size());
  if (e != cudaSuccess) return e;
  return cudaMemcpy(*out, img.data(), img.size(), cudaMemcpyHostToDevice);
}

cudaError_t launch_fstage_tc(const Job &job, const void *tables, int t0, int nt, int T, void *chan, int chan_type,
                             float out_scale, cudaStream_t s, const float *cscale, float2 *probe) {
  using namespace ftc;
  if (nt <= 0) return cudaSuccess;
  if (!fstage_tc_supported(job, chan_type) || !tables) return cudaErrorInvalidValue;
  Params p;
  p.job = job;
  p.tables = reinterpret_cast<const uint4 *>(tables);
  p.t0 = t0;
  p.nt = nt;
  p.T = T;
  p.chan = chan;
  p.out_scale = out_scale;
  p.cscale = cscale;
  p.probe = probe;
  cudaError_t e = cudaGetSymbolAddress((void **)&p.err, g_ftc_err);
  if (e != cudaSuccess) return e;
  int dev = 0, nsm = 0;
  e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  const long long nwin = (long long)nt * job.nant;
  const unsigned grid = (unsigned)(nwin < nsm ? nwin : nsm);
  if (!fstage_tc_addresses(job.nant, T, chan_type)) return cudaErrorInvalidValue;
  auto launch = [&](auto kern) -> cudaError_t {
    cudaError_t e2 = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e2 != cudaSuccess) return e2;
    kern<<<grid, NT, SMEM_BYTES, s>>>(p);
    return cudaGetLastError();
  };
  if (chan_type == CHAN_F8)
    return probe ? launch(fstage_tc_kernel<__nv_fp8x2_e4m3, true>) : launch(fstage_tc_kernel<__nv_fp8x2_e4m3>);
  return probe ? launch(fstage_tc_kernel<__half2, true>) : launch(fstage_tc_kernel<__half2>);
}

// Reads and clears the error flag of the tensor-core F-stage (a bounded wait expired).
cudaError_t fstage_tc_take_error(int *flag) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(flag, ftc::g_ftc_err, sizeof(int));
  if (e == cudaSuccess && *flag) e = cudaMemcpyToSymbol(ftc::g_ftc_err, &zero, sizeof(int));
  return e;
}

}  // namespace gxc
