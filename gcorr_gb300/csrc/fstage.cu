// F-stage of the FX correlator: per-(antenna, FFT) geometry, validity counts,
// twiddle tables, and the launcher of the fused channelising kernels
// (fstage_kernels.cuh: unpack -> fringe rotation -> FFT -> fractional-sample-delay
// correction -> cast -> write in the X-stage layout).
//
// Reference path restated: fxkernel/src/fxkernel.cpp:276-325 (station loop of
// process()), :425-440 getStationDelay, :443-487 unpack, :498-567 fringerotate,
// :569-580 dofft, :595-634 fracSampleCorrect.
#include <cooperative_groups.h>
#include <math.h>
#include <stdlib.h>
#include <type_traits>
#include <vector>

#include "fstage_kernels.cuh"
#include "gxc_internal.h"

namespace gxc {

// ----------------------------------------------------------------- geometry
// One thread per (antenna, FFT), antenna a0 + blockIdx.y.  FP64 with explicit round-to-nearest
// operations so the integer/fractional split matches the CPU reference bit
// for bit (no FMA contraction): fxkernel.cpp:432-439 and :289-309.
// The per-call parameters (input pointers, delay model) arrive as kernel parameters; the first block of an antenna
// writes its input pointer where the F-stage reads it.  Validity also goes out as one bit per FFT (vbits [nant][nw]).
// Bound by the FP64 pipe (two operations per clock and SM).
__global__ void geometry_kernel(Job job, const __grid_constant__ GeomParams u, int nw, uint32_t *__restrict__ vbits) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int al = blockIdx.y, ant = u.a0 + al;
  if (i == 0) job.inputs[ant] = u.ptrs[al];
  const bool in_range = i < job.nfft;
  const double *p = u.poly + 3 * al;
  const double fso = u.fso[al];
  const double fi = (double)i, fh = fi + 0.5, f1 = fi + 1.0;
  const double d0 = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(p[0], fi), fi), __dmul_rn(p[1], fi)), p[2]);
  const double d1 = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(p[0], fh), fh), __dmul_rn(p[1], fh)), p[2]);
  const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(p[0], f1), f1), __dmul_rn(p[1], f1)), p[2]);
  const double a = __dsub_rn(d2, d0);
  const double b = __dadd_rn(d0, __ddiv_rn(__dsub_rn(d1, __dadd_rn(__dmul_rn(a, 0.5), d0)), 3.0));
  const double mean = __dadd_rn(__dmul_rn(a, 0.5), b);
  const double ndf = __ddiv_rn(__dsub_rn(mean, fso), job.Ts);
  Geom g;
  g.c0 = g.c1 = g.cstep = g.cf = 0.0f;
  g.offset = 0;
  g.valid = 0;
  g.c0_lo = g.c1_lo = 0.0f;
  if (fabs(ndf) < 1.0e9) {  // false for NaN/Inf: flagged instead of undefined int()
    const int nd = __double2int_rz(__dadd_rn(ndf, 0.5));
    double frac = -__dmul_rn(__dsub_rn(ndf, (double)nd), job.Ts);
    long long off = (long long)i * job.F - nd;
    if (off == -1) { off++; frac = __dadd_rn(frac, job.Ts); }
    if (off == job.maxoffset + 1) { off--; frac = __dsub_rn(frac, job.Ts); }
    // Phase constants (fxkernel.cpp:503-535): phase(n) = LO*(b + a*n/F) turns, the
    // integer-sample part of b removed and the rest reduced mod 1 turn in FP64.
    const int intdelay = __double2int_rz(b);
    const double br = b - (double)intdelay;
    double c0 = br * job.lo_hz;
    if (job.fractional_lo) c0 += (job.lo_hz - trunc(job.lo_hz)) * (double)intdelay;
    c0 -= floor(c0);
    const double c1 = a * job.lo_hz * job.inv_F;  // turns per sample (F is a power of two)
    // coarse step: the reference advances its step table by `stride` samples per
    // entry (fxkernel.cpp:112) while applying it every `substride` samples;
    // FXKERNEL mode keeps that, EXACT uses the true step.
    const double stepmul = (job.rotator == GXC_ROTATOR_FXKERNEL) ? (double)job.stride : (double)job.substride;
    g.c0 = (float)c0;
    g.c0_lo = (float)(c0 - (double)g.c0);
    g.c1 = (float)c1;
    g.c1_lo = (float)(c1 - (double)g.c1);
    g.cstep = (float)(c1 * stepmul);
    // fractional-sample correction exp(+2 pi i c bw/nchan frac) (fxkernel.cpp:171-175,600-630)
    g.cf = (float)(job.bw_chan * frac);
    if (off >= 0 && off <= job.maxoffset) {
      g.offset = (int)off;
      g.valid = 1;
      const uint8_t *fv = u.fvalid[al];
      if (fv && in_range) {
        const long long f1 = (off + job.F - 1) / job.samples_per_frame;
        for (long long f = off / job.samples_per_frame; f <= f1; f++)
          if (!fv[f]) g.valid = 0;
      }
    }
  }
  if (in_range) job.geom[(size_t)ant * job.nfft + i] = g;
  const uint32_t bits = __ballot_sync(0xffffffffu, in_range && g.valid);
  if ((threadIdx.x & 31) == 0 && (i >> 5) < nw) vbits[(size_t)ant * nw + (i >> 5)] = bits;
}

cudaError_t launch_geometry(const Job &job, const GeomParams &u, int n, uint32_t *vbits, cudaStream_t s) {
  const int threads = 256, nw = (job.nfft + 31) / 32;
  dim3 grid((unsigned)((job.nfft + threads - 1) / threads), (unsigned)n);
  geometry_kernel<<<grid, threads, 0, s>>>(job, u, nw, vbits);
  return cudaGetLastError();
}

// ------------------------------------------------------------------- counts
// counts[bl] = number of FFTs where both antennas are valid (fxkernel.cpp:352), from the validity bits.  One CTA per
// baseline: 5 us for 16 antennas and 62500 FFTs (275 us when it read the geometry records and one CTA exported every
// flag).
__global__ void counts_kernel(const uint32_t *__restrict__ vbits, int nant, int nw, int32_t *counts) {
  const int bl = blockIdx.x;
  int j, k;
  baseline_antennas(bl, nant, &j, &k);
  int c = 0;
  for (int w = threadIdx.x; w < nw; w += blockDim.x)
    c += __popc(vbits[(size_t)j * nw + w] & vbits[(size_t)k * nw + w]);
  c = block_sum256(c);
  if (threadIdx.x == 0) counts[bl] = c;
}

cudaError_t launch_counts(const uint32_t *vbits, int nant, int nfft, int nbl, int32_t *counts, cudaStream_t s) {
  if (nbl == 0) return cudaSuccess;
  counts_kernel<<<nbl, 256, 0, s>>>(vbits, nant, (nfft + 31) / 32, counts);
  return cudaGetLastError();
}

// ----------------------------------------------------------------- twiddles
// tw[m] = exp(-2 pi i m / F), m < F, rounded once from double.  For F = 8192 the same
// allocation continues with the pass twiddles W_M^e (M = F/2) of the packed-pair kernel,
// laid out so that a warp reads consecutive entries:
//   pass 1, [r][k]  (256 entries):  e = 16 r k, k < 16
//   pass 2, [r][iv] (4096 entries): e = r iv,   iv < 256
cudaError_t make_twiddles(int F, float2 **out) {
  const size_t extra = F == 8192 ? (size_t)kPairTw1 + kPairTw2 : 0;
  std::vector<float2> h((size_t)F + extra);
  for (int m = 0; m < F; m++) {
    const double ang = -2.0 * 3.14159265358979323846 * (double)m / (double)F;
    h[(size_t)m] = make_float2((float)cos(ang), (float)sin(ang));
  }
  if (extra) {
    auto wm = [&](int e) { return h[(size_t)((2 * (long long)e) % F)]; };  // W_M^e = W_F^(2e)
    for (int r = 0; r < 16; r++)
      for (int k = 0; k < 16; k++) h[(size_t)F + (size_t)r * 16 + k] = wm(16 * r * k);
    for (int r = 0; r < 16; r++)
      for (int iv = 0; iv < 256; iv++) h[(size_t)F + kPairTw1 + (size_t)r * 256 + iv] = wm(r * iv);
  }
  cudaError_t e = cudaMalloc((void **)out, sizeof(float2) * h.size());
  if (e != cudaSuccess) return e;
  return cudaMemcpy(*out, h.data(), sizeof(float2) * h.size(), cudaMemcpyHostToDevice);
}

int fstage_supported(int F) { return F >= 256 && F <= 32768 && (F & (F - 1)) == 0; }

const char *fstage_kernel_name(int log2F, int chan_type) {  // as launch_fstage_l dispatches
  if (log2F == 13) return "fstage_pair_kernel";
  if (log2F >= 14 && chan_type != CHAN_F32) return "fstage_h_kernel";
  return log2F == 15 ? "fstage_cluster_kernel" : "fstage_kernel";
}

cudaError_t launch_fstage(const Job &job, const float2 *twiddles, int t0, int nt, int T, void *chan, int chan_type,
                          float out_scale, cudaStream_t s, const float *cscale) {
  if (nt <= 0) return cudaSuccess;
  const FParams prm = fstage_params(job, twiddles, t0, nt, T, chan, out_scale, nullptr, cscale);
  if (chan_type == CHAN_F32) {
    return job.is_complex ? launch_fstage_l<float2, true>(prm, nt, s) : launch_fstage_l<float2, false>(prm, nt, s);
  }
  if (chan_type == CHAN_F8) {
    return job.is_complex ? launch_fstage_l<__nv_fp8x2_e4m3, true>(prm, nt, s)
                          : launch_fstage_l<__nv_fp8x2_e4m3, false>(prm, nt, s);
  }
  return job.is_complex ? launch_fstage_l<__half2, true>(prm, nt, s) : launch_fstage_l<__half2, false>(prm, nt, s);
}

}  // namespace gxc
