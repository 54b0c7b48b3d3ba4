// A6: phase term and Z matrix.
//
// Reference: core/tau.py:30-31, 48-71 (exptau = exp(+i 2 pi nu / c * D . X), the
// sign the code uses), core/getz.py:52-105 (Z[a, f, x, s] = exptau[a, s] *
// sqrt_flux[s] * beam[beam_idx[a], f, x, s], rows a * nfeed + f, columns
// x * nsrc + s).
//
// Phase: t = (nu / c) (D . X) in cycles, evaluated in FP64 and reduced to
// r = t - rint(t) in [-1/2, 1/2] before an FP32 sincospi(2 r); at 1 km and
// 200 MHz |t| reaches 670 cycles, where an FP32 phase would carry 2.4e-4 rad of
// error.  Z columns are ordered k = s * nax + x (the source sum is the same).
//
// Split formats (the operand of the tensor-core Hermitian product):
//   bf16, P terms: t0 = bf16_rn(v), t1 = bf16_rn(v - t0), t2 = bf16_rn(v - t0 - t1)
//   tf32, 2 terms: t0 = tf32_rna(v), t1 = tf32_rna(v - t0)
//   fp16, 2 terms of s*v: t0 = fp16_rn(s v), t1 = fp16_rn(s v - t0), s = zscale
// each residual being exact in FP32.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace mvb {

constexpr double kInvC = 1.0 / 299792458.0;

// Nearest integer (ties to even) of |t| < 2^51 with two FP64 adds: adding and
// subtracting 1.5 * 2^52 leaves no fraction bits, so the first add rounds t to
// an integer in the current (round-to-nearest-even) mode -- the same value as
// rint(t), on the FP64 add pipe instead of the conversion unit.  |t| here is a
// path difference in wavelengths (< 2^40 for any physical array).
__device__ __forceinline__ double round_half_even(double t) {
  const double magic = 6755399441055744.0;  // 1.5 * 2^52
  return __dsub_rn(__dadd_rn(t, magic), magic);
}

__device__ __forceinline__ float tf32_rna(float v) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(v));
  return __uint_as_float(r);
}

// Vector stores of W consecutive 32-bit words (W = 1, 2, 4, 8: 4 to 32 bytes,
// aligned to min(size, 16) bytes by the callers).
template <int W>
__device__ __forceinline__ void store_words(void *p, const uint32_t *w) {
  static_assert(W == 1 || W == 2 || W == 4 || W == 8, "1, 2, 4 or 8 words");
  if constexpr (W == 8) {
    *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    *(reinterpret_cast<uint4 *>(p) + 1) = make_uint4(w[4], w[5], w[6], w[7]);
  } else if constexpr (W == 4)
    *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  else if constexpr (W == 2)
    *reinterpret_cast<uint2 *>(p) = make_uint2(w[0], w[1]);
  else
    *reinterpret_cast<uint32_t *>(p) = w[0];
}

// One 32-byte store of 8 words (p 32-byte aligned): a whole L2 sector in one
// instruction.
__device__ __forceinline__ void store_sector(void *p, const uint32_t *w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}

// Writes NV consecutive real values of one component (c = 0 real, 1 imaginary)
// as the P split terms into planes [2p + c] of a panel row, with vector stores:
// NV = 4 or 8 values: 8- or 16-byte stores of bf16 / fp16 (inside one 16-byte
// chunk of the swizzled row, at off), 16 bytes of float32 at off, or 2 x 16
// bytes of float32 at off (values 0..3) and off2 (values 4..7: the next chunk,
// which the swizzle may place anywhere in the row).
template <int MODE, int NV>
__device__ __forceinline__ void put_split(void *z, int64_t plane_stride, int64_t off, int64_t off2, int comp,
                                          const float *v, float zscale) {
  if constexpr (MODE == MVB_GEMM_F16_3) {
    // one paired conversion per two values for each term (cvt.rn.f16x2.f32)
    uint32_t whi[NV / 2], wlo[NV / 2];
#pragma unroll
    for (int i = 0; i < NV; i += 2) {
      const float r0 = v[i] * zscale, r1 = v[i + 1] * zscale;
      const __half2 hi = __floats2half2_rn(r0, r1);
      const float2 back = __half22float2(hi);
      const __half2 lo = __floats2half2_rn(r0 - back.x, r1 - back.y);
      whi[i / 2] = *reinterpret_cast<const uint32_t *>(&hi);
      wlo[i / 2] = *reinterpret_cast<const uint32_t *>(&lo);
    }
    __half *p0 = static_cast<__half *>(z) + off + (int64_t)(0 + comp) * plane_stride;
    __half *p1 = static_cast<__half *>(z) + off + (int64_t)(2 + comp) * plane_stride;
    store_words<NV / 2>(p0, whi);
    store_words<NV / 2>(p1, wlo);
  } else if constexpr (MODE == MVB_GEMM_TF32_3) {
    float hi[NV], lo[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      hi[i] = tf32_rna(v[i]);
      lo[i] = tf32_rna(v[i] - hi[i]);
    }
    float *p0 = static_cast<float *>(z) + off + (int64_t)(0 + comp) * plane_stride;
    float *p1 = static_cast<float *>(z) + off + (int64_t)(2 + comp) * plane_stride;
    uint32_t whi[NV], wlo[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      whi[i] = __float_as_uint(hi[i]);
      wlo[i] = __float_as_uint(lo[i]);
    }
    if constexpr (NV == 8) {
      // values 0..3 and 4..7 fill the two 16-byte chunks of one 32-byte sector
      // (the 64-byte swizzle keeps chunk pairs {0, 1} and {2, 3} together, in
      // either order): one sector store per plane
      const bool swapped = off2 < off;
      const int64_t base = swapped ? off2 : off;
      uint32_t shi[8], slo[8];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        shi[i] = swapped ? whi[4 + i] : whi[i];
        shi[4 + i] = swapped ? whi[i] : whi[4 + i];
        slo[i] = swapped ? wlo[4 + i] : wlo[i];
        slo[4 + i] = swapped ? wlo[i] : wlo[4 + i];
      }
      store_sector(static_cast<float *>(z) + base + (int64_t)(0 + comp) * plane_stride, shi);
      store_sector(static_cast<float *>(z) + base + (int64_t)(2 + comp) * plane_stride, slo);
    } else {
      store_words<NV>(p0, whi);
      store_words<NV>(p1, wlo);
    }
  } else {
    constexpr int P = MODE == MVB_GEMM_BF16_6 ? 3 : 2;
    float r[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) r[i] = v[i];
#pragma unroll
    for (int p = 0; p < P; ++p) {
      uint32_t w[NV / 2];
#pragma unroll
      for (int i = 0; i < NV; i += 2) {
        // one paired conversion per two values (cvt.rn.bf16x2.f32); bf16 -> f32 is exact
        const __nv_bfloat162 t = __floats2bfloat162_rn(r[i], r[i + 1]);
        const float2 back = __bfloat1622float2(t);
        r[i] -= back.x;
        r[i + 1] -= back.y;
        w[i / 2] = *reinterpret_cast<const uint32_t *>(&t);
      }
      __nv_bfloat16 *pp = static_cast<__nv_bfloat16 *>(z) + off + (int64_t)(2 * p + comp) * plane_stride;
      store_words<NV / 2>(pp, w);
    }
  }
}

// Single-value writer kept for the pack kernel (2 consecutive values).
template <int MODE>
struct PanelWriter {
  static constexpr int P = MODE == MVB_GEMM_BF16_6 ? 3 : 2;
  static __device__ __forceinline__ void put(void *z, int64_t plane_stride, int64_t off, int comp, const float *v,
                                             int X, float zscale) {
    if constexpr (MODE == MVB_GEMM_F16_3) {
      __half *zp = static_cast<__half *>(z) + off;
      for (int x = 0; x < X; ++x) {
        const float r = v[x] * zscale;
        const __half hi = __float2half_rn(r);
        zp[(2 * 0 + comp) * plane_stride + x] = hi;
        zp[(2 * 1 + comp) * plane_stride + x] = __float2half_rn(r - __half2float(hi));
      }
    } else if constexpr (MODE == MVB_GEMM_TF32_3) {
      float *zp = static_cast<float *>(z) + off;
      float hi[2], lo[2];
      for (int x = 0; x < X; ++x) {
        hi[x] = tf32_rna(v[x]);
        lo[x] = tf32_rna(v[x] - hi[x]);
      }
      float *p0 = zp + (2 * 0 + comp) * plane_stride;
      float *p1 = zp + (2 * 1 + comp) * plane_stride;
      if (X == 2) {
        *reinterpret_cast<float2 *>(p0) = make_float2(hi[0], hi[1]);
        *reinterpret_cast<float2 *>(p1) = make_float2(lo[0], lo[1]);
      } else {
        *p0 = hi[0];
        *p1 = lo[0];
      }
    } else {
      __nv_bfloat16 *zp = static_cast<__nv_bfloat16 *>(z) + off;
      __nv_bfloat16 t[3][2];
      for (int x = 0; x < X; ++x) {
        float r = v[x];
#pragma unroll
        for (int p = 0; p < P; ++p) {
          t[p][x] = __float2bfloat16_rn(r);
          r = r - __bfloat162float(t[p][x]);
        }
      }
#pragma unroll
      for (int p = 0; p < P; ++p) {
        __nv_bfloat16 *pp = zp + (2 * p + comp) * plane_stride;
        if (X == 2) {
          __nv_bfloat162 two;
          two.x = t[p][0];
          two.y = t[p][1];
          *reinterpret_cast<__nv_bfloat162 *>(pp) = two;
        } else {
          *pp = t[p][0];
        }
      }
    }
  }
};

// ---------------------------------------------------------------------------
// Fused writer.  CTA = 128 threads over 64 panel columns (32 sources at X = 2, 64
// at X = 1) x 64 antennas x `per_z` frequencies: thread bits 0..2 pick a group of 8
// consecutive columns (16-byte stores per plane at 16 bits), bits 3..6 one of 16
// antenna lanes, each lane taking every 16th antenna of the block (one frequency at
// X = 1: 32 columns, groups of 4).  A CTA writes 2
// or 4 k-blocks of 128 rows per frequency, so the Z lines it has open at any time
// fit, summed over the resident CTAs, well inside L2 (a wider k-range per CTA left
// partially written lines to be evicted); a warp's store writes 16 whole 32-byte
// sectors.
// What bounds it: instructions.  Per (antenna, source, frequency) it needs the
// phase reduction and sincos, F X complex products and their split and stores; the
// path difference, the beam values and the offsets depend on (antenna, source)
// only and stay in registers for the frequencies of the group, and what depends on
// (source, frequency) only -- the flux, or a polarised sky's Cholesky factor -- is
// staged once per CTA for its 16 antenna lanes.  fp16x3, 350 polarised antennas x
// 98,304 sources x 8 frequencies: 1,390 us, 6.3 TB/s written (0.97 of the copy
// rate), against 1,650 us with a frequency per CTA, which read the beam from shared
// memory and formed the path difference for each; 512 unpolarised antennas x 30,001
// sources x 8: 224 against 390 us (4.4 TB/s: instructions); 90 x 11,180 x 8: 23
// against 32 us; polarised sky, 350 x 24,576 x 4: 194 against 321 us (every antenna
// lane factored the coherency again).  The results are bit-identical.
// ---------------------------------------------------------------------------
constexpr int kTauZThreads = 128;
constexpr int kTauZCols = 8;                // consecutive columns per thread (tau_z_cols: 4 in one form)
constexpr int kTauZGroups = 8;              // column groups per CTA
constexpr int kTauZAntLanes = kTauZThreads / kTauZGroups;
constexpr int kTauZAnts = 64;               // antennas per CTA
constexpr int kTauZMaxBFX = 16;             // beam planes staged in shared memory, else read through L1
constexpr int kTauZMaxFreq = 8;             // frequencies per CTA
constexpr int kTauZCtasPerSm = 8;           // CTAs per SM that a small launch is cut into

// Columns per thread.  One frequency at one beam axis takes four: eight sources'
// paths and fluxes do not stay in registers, and nothing else of them is shared.
// 512 antennas x 60,000 sources, fp16x3: 82 us with four, 121 with eight (20 beams,
// read through L1: 91 and 176); 100 x 60,000 as a complex64 Z: 17 and 28.
__host__ __device__ constexpr int tau_z_cols(int X, bool group) { return X == 1 && !group ? 4 : kTauZCols; }

// CTAs per SM that a two-feed, two-axis tf32x3 or bf16x6 launch has to keep for
// frequencies to share them.  Those panels are 16 and 12 bytes a value and bound by
// their stores, and fewer, longer CTAs cost their last wave: tf32x3, 350 antennas x
// 6,000 slots x 12, half live, 141 us shared (15 CTAs per SM), 122 one by one; x 15,000 x
// 3 168 and 164 (19); x 40,000 x 3 438 and 455 (51); bf16x6, 512 x 9,000 x 12 437 and
// 408 (30); 350 x 40,000 x 6 620 and 658 (51).  A polarised sky's factors are shared
// too: bf16x6 always pays (x 40,000 x 6 635 and 733), tf32x3 never (x 40,000 x 3 263 and
// 245).
constexpr int kTauZWideCtasPerSm = 40;

// Resident CTAs per SM that the registers are held to (the best of 4, 5, 6, 8 and
// no bound, by form: the polarised group form keeps 32 beam values a thread).
constexpr int tau_z_min_blocks(int mode, int X, int F, bool group) {
  return X * F == 4 ? (!group ? 6 : (mode == MVB_GEMM_TF32_3 ? 5 : 4)) : (X == 1 && F == 2 ? 5 : 6);
}

struct TauZArgs {
  const double *antpos, *crd, *freqs;  // freqs: device array of the group, or null (f_over_c)
  double f_over_c;
  int64_t ld, nsrc, beam_ld, sflux_ld, coh_ld, zstride, Mpad, Kcap;
  const int32_t *n_dev, *sidx, *beam_idx;
  const float *sflux;
  const float2 *beam;
  const float4 *coh;
  const double2 *rot;
  void *z;
  int A, ants, nbeam, nfreq, per_z;  // ants: antennas per CTA
  float scale_beam, scale_flux;  // their product is the panel's power-of-two scale
  bool staged;                   // the beam planes fit the shared-memory stage
};

// Lower-triangular L of C' = R^T C R = L L^H (clamped at the PSD boundary), for
// the coherency c = (C00, C11, Re C01, Im C01) and R's (cos X, sin X).
__device__ __forceinline__ float4 coherency_factor(float4 c, double2 r) {
  const double cr = r.x, sr = r.y;
  const double a = c.x, d = c.y, br = c.z, bi = c.w;
  const double c00 = cr * cr * a + sr * sr * d - 2.0 * cr * sr * br;
  const double c11 = sr * sr * a + cr * cr * d + 2.0 * cr * sr * br;
  // C'_10 = conj(C'_01), C'_01 = cr sr (a - d) + cr^2 b - sr^2 conj(b)
  const double c10r = cr * sr * (a - d) + (cr * cr - sr * sr) * br;
  const double c10i = -(cr * cr + sr * sr) * bi;
  const double L00 = sqrt(fmax(c00, 0.0));
  const double L10r = L00 > 0.0 ? c10r / L00 : 0.0, L10i = L00 > 0.0 ? c10i / L00 : 0.0;
  return make_float4((float)L00, (float)L10r, (float)L10i,
                     (float)sqrt(fmax(c11 - L10r * L10r - L10i * L10i, 0.0)));
}

// POL: polarised sky.  Instead of sqrt(0.5 I) the source carries its coherency C
// (coh[sidx[s]] at this frequency) and frame rotation R (rot[s] = cos X, sin X);
// with C' = R^T C R = L L^H, Z[a, f, (s, y)] = exptau(a, s) sum_x beam[f, x, s]
// L[x, y, s], so that Z Z^H gives exptau_j conj(exptau_i) E_j C' E_i^H per source.
// grid.x: blocks of ROW columns, grid.y: blocks of kTauZAnts antennas, grid.z: per_z
// frequencies each, frequency g: fluxes sflux + g sflux_ld (coh + g coh_ld), panel
// z + g zstride bytes.  WIDE: every panel is aligned to the stores of eight columns
// (store_align); otherwise eight columns go out in two halves, the same bytes.
template <int MODE, int X, int F, bool POL, bool GROUP, bool WIDE>
__global__ void __launch_bounds__(kTauZThreads, tau_z_min_blocks(MODE, X, F, GROUP)) tau_z_kernel(const __grid_constant__ TauZArgs p) {
  static_assert(!POL || (X == 2 && F == 2), "the polarised sky needs two feeds and two beam axes");
  static_assert(!GROUP || WIDE, "narrow stores: one frequency per CTA");
  constexpr int COLS = tau_z_cols(X, GROUP);
  constexpr int ROW = COLS * kTauZGroups;  // columns of the CTA: staged values of one (beam, feed)
  constexpr int NS = COLS / X;             // sources per thread
  constexpr int BS = kTauZGroups * NS;     // sources per CTA
  pdl_wait();
  pdl_trigger();
  const int64_t n = p.n_dev ? min((int64_t)__ldcg(p.n_dev), p.nsrc) : p.nsrc;
  const int64_t s_end = round_up(n * X, kKAlign) / X;  // zero-fill up to here: a multiple of BS
  const int64_t sb = (int64_t)blockIdx.x * BS;
  if (sb >= s_end) return;  // uniform per CTA
  const int g0 = blockIdx.z * p.per_z, gn = min(p.per_z, p.nfreq - g0);

  __shared__ double crd_sm[3][BS], foc_sm[kTauZMaxFreq];
  extern __shared__ float4 dyn_sm[];
  // per (frequency, source): the flux, or the Cholesky factor; then the beam values
  // [(beam, feed)][column pair][group][2]: a thread's pair of columns is 16 bytes
  float *flux_sm = reinterpret_cast<float *>(dyn_sm);
  float4 *fac_sm = dyn_sm;
  float2 *beam_sm = reinterpret_cast<float2 *>(dyn_sm) + (POL ? 2 : 1) * (p.per_z * BS) / (POL ? 1 : 2);
  // every load of the prologue is issued before the first value is stored: the
  // CTA's start is one chain of loads (the flux behind its index), not four
  constexpr int PER = kTauZThreads / BS;  // (frequencies, coordinates, beam planes) the threads cover at a time
  const int sl = threadIdx.x % BS, lane0 = threadIdx.x / BS;
  const int64_t s = sb + sl;
  const bool live = s < n;
  const int64_t src = live && p.sidx ? __ldcg(p.sidx + s) : s;
  constexpr int NC = (3 + PER - 1) / PER, NB = kTauZMaxBFX / PER, NG = kTauZMaxFreq / PER;
  double c_in[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) c_in[i] = live && lane0 + i * PER < 3 ? __ldcg(p.crd + (lane0 + i * PER) * p.ld + s) : 0.0;
  const int nq = p.staged ? p.nbeam * F * X : 0;
  float2 b_in[NB];
#pragma unroll
  for (int i = 0; i < NB; ++i)
    b_in[i] = live && lane0 + i * PER < nq ? __ldcg(p.beam + (int64_t)(lane0 + i * PER) * p.beam_ld + s)
                                           : make_float2(0.f, 0.f);
  if (threadIdx.x < gn) foc_sm[threadIdx.x] = p.freqs ? __ldg(p.freqs + g0 + threadIdx.x) * kInvC : p.f_over_c;
  if constexpr (POL) {
    const double2 rot = live ? __ldcg(p.rot + s) : make_double2(0.0, 0.0);
    for (int g = lane0; g < gn; g += PER) {
      float4 l = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live) l = coherency_factor(__ldg(p.coh + (g0 + g) * p.coh_ld + src), rot);
      fac_sm[g * BS + sl] =
          make_float4(l.x * p.scale_flux, l.y * p.scale_flux, l.z * p.scale_flux, l.w * p.scale_flux);
    }
  } else {
    float f_in[NG];
#pragma unroll
    for (int i = 0; i < NG; ++i)
      f_in[i] = live && lane0 + i * PER < gn ? __ldg(p.sflux + (g0 + lane0 + i * PER) * p.sflux_ld + src) : 0.f;
#pragma unroll
    for (int i = 0; i < NG; ++i)
      if (lane0 + i * PER < gn) flux_sm[(lane0 + i * PER) * BS + sl] = f_in[i] * p.scale_flux;
  }
#pragma unroll
  for (int i = 0; i < NC; ++i)
    if (lane0 + i * PER < 3) crd_sm[lane0 + i * PER][sl] = c_in[i];
#pragma unroll
  for (int i = 0; i < NB; ++i) {
    const int q = lane0 + i * PER;
    if (q < nq) {
      const int k = (sl % NS) * X + q % X;  // the thread's column
      beam_sm[(q / X) * ROW + ((k >> 1) * kTauZGroups + sl / NS) * 2 + (k & 1)] =
          make_float2(b_in[i].x * p.scale_beam, b_in[i].y * p.scale_beam);
    }
  }
  __syncthreads();

  const int sg = threadIdx.x % kTauZGroups, alane = threadIdx.x / kTauZGroups;
  const int64_t k0 = (sb + sg * NS) * X;
  const int a0 = blockIdx.y * p.ants, a1 = min(a0 + p.ants, p.A);
  // one frequency: a thread's four sources' coordinates and fluxes stay in registers instead
  constexpr bool KEEP = !GROUP && NS <= 4;
  double cx[KEEP ? NS : 1], cy[KEEP ? NS : 1], cz[KEEP ? NS : 1];
  float sf1[KEEP ? NS : 1];
  if constexpr (KEEP) {
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      cx[j] = crd_sm[0][sg * NS + j];
      cy[j] = crd_sm[1][sg * NS + j];
      cz[j] = crd_sm[2][sg * NS + j];
      sf1[j] = POL ? 1.f : flux_sm[sg * NS + j];
    }
  }
  for (int a = a0 + alane; a < a1; a += kTauZAntLanes) {
    const int b = p.beam_idx ? __ldg(p.beam_idx + a) : 0;
    const double dx = __ldg(p.antpos + 3 * a), dy = __ldg(p.antpos + 3 * a + 1), dz = __ldg(p.antpos + 3 * a + 2);
    double path[NS];
#pragma unroll
    for (int j = 0; j < NS; ++j)
      path[j] = KEEP ? dx * cx[KEEP ? j : 0] + dy * cy[KEEP ? j : 0] + dz * cz[KEEP ? j : 0]
                     : dx * crd_sm[0][sg * NS + j] + dy * crd_sm[1][sg * NS + j] + dz * crd_sm[2][sg * NS + j];
    float2 bv[GROUP ? F : 1][COLS];
    auto load_beam = [&](int f, float2(&v)[COLS]) {
      if (p.staged) {
        const float4 *src = reinterpret_cast<const float4 *>(beam_sm + (b * F + f) * ROW) + sg;
#pragma unroll
        for (int k = 0; k < COLS; k += 2) {
          const float4 v2 = src[(k >> 1) * kTauZGroups];
          v[k] = make_float2(v2.x, v2.y);
          v[k + 1] = make_float2(v2.z, v2.w);
        }
      } else {
#pragma unroll
        for (int k = 0; k < COLS; ++k) {
          const int64_t s = sb + sg * NS + k / X;
          const float2 v1 = s < n ? __ldca(p.beam + (int64_t)((b * F + f) * X + k % X) * p.beam_ld + s)
                                  : make_float2(0.f, 0.f);
          v[k] = make_float2(v1.x * p.scale_beam, v1.y * p.scale_beam);
        }
      }
    };
    if constexpr (GROUP) {
#pragma unroll
      for (int f = 0; f < F; ++f) load_beam(f, bv[f]);
    }
#pragma unroll 1
    for (int g = 0; g < (GROUP ? gn : 1); ++g) {
      const double foc = foc_sm[g];
      float er[NS], ei[NS];
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const double t = path[j] * foc;
        const double r = t - round_half_even(t);
        float sn, cs;
        sincospif(2.f * (float)r, &sn, &cs);
        if constexpr (POL) {
          er[j] = cs;
          ei[j] = sn;
        } else {
          const float sf = KEEP ? sf1[KEEP ? j : 0] : flux_sm[g * BS + sg * NS + j];
          er[j] = cs * sf;
          ei[j] = sn * sf;
        }
      }
      uint8_t *zg = static_cast<uint8_t *>(p.z) + (g0 + g) * p.zstride;
#pragma unroll
      for (int f = 0; f < F; ++f) {
        float vr[COLS], vi[COLS];
        if constexpr (!GROUP) load_beam(f, bv[0]);
#pragma unroll
        for (int k = 0; k < COLS; ++k) {
          const float2 v = bv[GROUP ? f : 0][k];
          vr[k] = er[k / X] * v.x - ei[k / X] * v.y;
          vi[k] = er[k / X] * v.y + ei[k / X] * v.x;
        }
        if constexpr (POL) {
          // (g0, g1) = exptau * beam[f, 0:2]  ->  (g0 L00 + g1 L10, g1 L11)
#pragma unroll
          for (int j = 0; j < NS; ++j) {
            const float4 l = fac_sm[g * BS + sg * NS + j];
            const float g0r = vr[2 * j], g0i = vi[2 * j], g1r = vr[2 * j + 1], g1i = vi[2 * j + 1];
            vr[2 * j] = fmaf(-g1i, l.z, fmaf(g0r, l.x, g1r * l.y));
            vi[2 * j] = fmaf(g1i, l.y, fmaf(g1r, l.z, g0i * l.x));
            vr[2 * j + 1] = g1r * l.w;
            vi[2 * j + 1] = g1i * l.w;
          }
        }
        const int64_t m = (int64_t)a * F + f;
        if constexpr (MODE == MVB_Z_C64) {
          // the row's values start a multiple of 32 bytes into the panel (Kcap a
          // multiple of 64): whole 32-byte sectors, four values each
          float2 *zp = reinterpret_cast<float2 *>(zg) + m * p.Kcap + k0;
#pragma unroll
          for (int i = 0; i < COLS; i += 4) {
            const uint32_t w[8] = {__float_as_uint(vr[i]),     __float_as_uint(vi[i]),     __float_as_uint(vr[i + 1]),
                                   __float_as_uint(vi[i + 1]), __float_as_uint(vr[i + 2]), __float_as_uint(vi[i + 2]),
                                   __float_as_uint(vr[i + 3]), __float_as_uint(vi[i + 3])};
            if constexpr (WIDE)
              store_sector(zp + i, w);
            else
              store_words<8>(zp + i, w);
          }
        } else {
          // COLS consecutive k from a multiple of COLS: inside one k-block
          constexpr int KB = kKBlockBytes / (MODE == MVB_GEMM_TF32_3 ? 4 : 2);
          constexpr int NPL = MODE == MVB_GEMM_BF16_6 ? 6 : 4;
          const int64_t off = panel_off(m, k0, p.Mpad, KB, NPL);
          const int64_t off2 = panel_off(m, k0 + COLS / 2, p.Mpad, KB, NPL);
          if constexpr (WIDE || COLS == 4) {
            put_split<MODE, COLS>(zg, panel_plane_stride(KB), off, off2, 0, vr, 1.f);
            put_split<MODE, COLS>(zg, panel_plane_stride(KB), off, off2, 1, vi, 1.f);
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int64_t o = h ? off2 : off;
              put_split<MODE, 4>(zg, panel_plane_stride(KB), o, o, 0, vr + 4 * h, 1.f);
              put_split<MODE, 4>(zg, panel_plane_stride(KB), o, o, 1, vi + 4 * h, 1.f);
            }
          }
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Z from a caller's exptau (A, e_ld), complex64 (EXT = 1) or complex128 (EXT = 2):
// 32 sources x 64 antennas per CTA, four consecutive sources per thread.  The
// CTA's beam values are staged in shared memory for its 16 antenna lanes (or read
// through L1 beyond kTauZMaxBFX planes).
// ---------------------------------------------------------------------------
constexpr int kZExtSrc = 4;
constexpr int kZExtBlockSrc = kTauZGroups * kZExtSrc;
constexpr int kZExtRow = kZExtBlockSrc + 1;  // staged beam values per q, padded

template <int MODE, int X, int EXT, bool STAGED>
__global__ void __launch_bounds__(kTauZThreads)
    z_exptau_kernel(const void *__restrict__ ext, int64_t e_ld, int A, int64_t n, const float *__restrict__ sflux,
                    const float2 *__restrict__ beam, int64_t beam_ld, int nbeam, const int32_t *__restrict__ beam_idx,
                    int F, float zscale, void *__restrict__ z, int64_t Mpad, int64_t Kcap) {
  const int64_t s_end = round_up(n * X, kKAlign) / X;  // zero-fill up to here
  const int64_t s0 = (int64_t)blockIdx.x * kZExtBlockSrc + (threadIdx.x % kTauZGroups) * kZExtSrc;
  const int alane = threadIdx.x / kTauZGroups;
  if ((int64_t)blockIdx.x * kZExtBlockSrc >= s_end) return;  // uniform per CTA
  const bool write = s0 < s_end;  // s_end is a multiple of kZExtSrc (64 / X)
  float sf[kZExtSrc];
#pragma unroll
  for (int j = 0; j < kZExtSrc; ++j) sf[j] = s0 + j < n ? sflux[s0 + j] : 0.f;
  // staged as [q][j][group], rows of 33 values (q = (beam * F + f) * X + x): the 8
  // source groups of a warp read 8 consecutive values, and lanes with different
  // beams land on different banks
  extern __shared__ float2 bsm[];
  if constexpr (STAGED) {
    const int nq = nbeam * F * X;
    for (int e = threadIdx.x; e < nq * kZExtBlockSrc; e += kTauZThreads) {
      const int q = e / kZExtBlockSrc, sl = e % kZExtBlockSrc;  // sl = group * kZExtSrc + j
      const int64_t ss = (int64_t)blockIdx.x * kZExtBlockSrc + sl;
      bsm[q * kZExtRow + (sl % kZExtSrc) * kTauZGroups + sl / kZExtSrc] =
          ss < n ? __ldg(beam + (int64_t)q * beam_ld + ss) : make_float2(0.f, 0.f);
    }
    __syncthreads();
  }
  const int sg = threadIdx.x % kTauZGroups;
  const int a0 = blockIdx.y * kTauZAnts;
  const int a1 = min(a0 + kTauZAnts, A);
  for (int a = a0 + alane; a < a1; a += kTauZAntLanes) {
    const int b = beam_idx ? beam_idx[a] : 0;
    float er[kZExtSrc], ei[kZExtSrc];
#pragma unroll
    for (int j = 0; j < kZExtSrc; ++j) {
      er[j] = ei[j] = 0.f;
      if (s0 + j >= n) continue;
      if (EXT == 1) {
        const float2 e = static_cast<const float2 *>(ext)[(int64_t)a * e_ld + s0 + j];
        er[j] = e.x * sf[j];
        ei[j] = e.y * sf[j];
      } else {
        const double2 e = static_cast<const double2 *>(ext)[(int64_t)a * e_ld + s0 + j];
        er[j] = (float)(e.x * (double)sf[j]);
        ei[j] = (float)(e.y * (double)sf[j]);
      }
    }
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      if (f >= F) break;
      float vr[kZExtSrc * X], vi[kZExtSrc * X];
#pragma unroll
      for (int j = 0; j < kZExtSrc; ++j)
#pragma unroll
        for (int x = 0; x < X; ++x) {
          const int q = (b * F + f) * X + x;
          float2 bv;
          if constexpr (STAGED)
            bv = bsm[q * kZExtRow + j * kTauZGroups + sg];
          else
            bv = (s0 + j < n) ? __ldg(beam + (int64_t)q * beam_ld + s0 + j) : make_float2(0.f, 0.f);
          vr[j * X + x] = er[j] * bv.x - ei[j] * bv.y;
          vi[j * X + x] = er[j] * bv.y + ei[j] * bv.x;
        }
      if (!write) continue;
      const int64_t m = (int64_t)a * F + f;
      if constexpr (MODE == MVB_Z_C64) {
        // the row's kZExtSrc * X values start 32-byte aligned (Kcap a multiple
        // of 64, s0 X of 4): whole 32-byte sectors, four values each
        float2 *zp = static_cast<float2 *>(z) + m * Kcap + s0 * X;
#pragma unroll
        for (int i = 0; i < kZExtSrc * X; i += 4) {
          const uint32_t w[8] = {__float_as_uint(vr[i]),     __float_as_uint(vi[i]),     __float_as_uint(vr[i + 1]),
                                 __float_as_uint(vi[i + 1]), __float_as_uint(vr[i + 2]), __float_as_uint(vi[i + 2]),
                                 __float_as_uint(vr[i + 3]), __float_as_uint(vi[i + 3])};
          store_sector(zp + i, w);
        }
      } else {
        // kZExtSrc * X consecutive k from a multiple of kZExtSrc * X: inside one k-block
        constexpr int KB = kKBlockBytes / (MODE == MVB_GEMM_TF32_3 ? 4 : 2);
        constexpr int NPL = MODE == MVB_GEMM_BF16_6 ? 6 : 4;
        const int64_t off = panel_off(m, s0 * X, Mpad, KB, NPL);
        const int64_t off2 = panel_off(m, s0 * X + kZExtSrc * X / 2, Mpad, KB, NPL);
        put_split<MODE, kZExtSrc * X>(z, panel_plane_stride(KB), off, off2, 0, vr, zscale);
        put_split<MODE, kZExtSrc * X>(z, panel_plane_stride(KB), off, off2, 1, vi, zscale);
      }
    }
  }
}

__global__ void exptau_kernel(const double *__restrict__ antpos, int A, double f_over_c, const double *__restrict__ crd,
                              int64_t ld, int64_t nsrc, void *__restrict__ out, int out_c128) {
  const int64_t total = (int64_t)A * nsrc;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t a = i / nsrc, s = i % nsrc;
    const double t = (antpos[3 * a] * crd[s] + antpos[3 * a + 1] * crd[ld + s] + antpos[3 * a + 2] * crd[2 * ld + s]) *
                     f_over_c;
    const double r = t - rint(t);
    if (out_c128) {
      double sn, cs;
      sincospi(2.0 * r, &sn, &cs);
      static_cast<double2 *>(out)[i] = make_double2(cs, sn);
    } else {
      float sn, cs;
      sincospif((float)(2.0 * r), &sn, &cs);
      static_cast<float2 *>(out)[i] = make_float2(cs, sn);
    }
  }
}

// Power-of-two scale s with max |s Z| < 2^15 (the fp16 range) for a panel whose
// largest |Z| is `m` (with a margin of 2^-10); 1 for an empty or non-finite Z.
__device__ __forceinline__ float panel_scale(float m) {
  const double top = (double)m * (1.0 + 1.0 / 1024.0);
  if (!(top > 0.0) || isinf(top)) return 1.f;
  const int e = ilogb(16384.0 / top);
  return ldexpf(1.f, max(min(e, 100), -100));
}

// C values of a row from column k (zeros past K), whole 16-byte loads when vec.
template <int C, typename CT>
__device__ __forceinline__ void load_row(const CT *__restrict__ row, int64_t k, int64_t K, bool vec, float (&vr)[C],
                                         float (&vi)[C]) {
  if (vec && k + C <= K) {
    if constexpr (sizeof(CT) == 8) {
#pragma unroll
      for (int i = 0; i < C; i += 2) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(row + k + i));
        vr[i] = v.x, vi[i] = v.y, vr[i + 1] = v.z, vi[i + 1] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < C; ++i) {
        const double2 v = __ldg(reinterpret_cast<const double2 *>(row + k + i));
        vr[i] = (float)v.x, vi[i] = (float)v.y;
      }
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < C; ++i) {
    vr[i] = vi[i] = 0.f;
    if (k + i < K) {
      vr[i] = (float)row[k + i].x;
      vi[i] = (float)row[k + i].y;
    }
  }
}

// Packs a caller complex matrix (M, K) into a panel.  CTA = 256 threads: 16 groups
// of C columns (pack_cols) x 16 row lanes x `lane_rows` rows each, so
// stores fill 8 or 16 bytes of a plane row.  It is bound by HBM; the row blocks run
// last to first, so that those a maximum pass has just read come from L2.  With
// `absmax` the fp16 scale is formed here from that pass's result and written to
// scale_out.  700 rows x 49,152 columns, complex64 to fp16x3: 83 us (the copy rate),
// against 125 with two columns a thread (4-byte stores, 64-bit divisions per
// element); complex128: 118 against 157; to tf32x3: 136 against 197.
// vec: the source rows allow 16-byte loads; align: the panel's alignment (2: 32
// bytes, 1: 16, 0: less).
constexpr int kPackThreads = 256;
constexpr int kPackGroups = 16;

// Columns per thread: 8 of complex64 and 4 of complex128, 64 bytes, beyond which a load
// instruction touches a line per lane.  Rows of an odd pitch are loaded value by value,
// for which 64 bytes a lane are too far apart: 4 of complex64 (fp16x3 writes more per
// value than it loads and keeps 8).  700 x 50,001 complex64 to a plain Z: 92 us with 4,
// 100 with 8; 90 x 50,001 from L2: 11.7 and 16.3; 700 x 50,001 to fp16x3: 106 and 104.
constexpr int pack_cols(int mode, int value_bytes, bool vec) {
  return value_bytes == 16 || (!vec && mode != MVB_GEMM_F16_3) ? 4 : 8;
}

template <int MODE, typename CT, int C>
__global__ void __launch_bounds__(kPackThreads)
    z_pack_kernel(const CT *__restrict__ zs, int64_t M, int64_t K, int64_t ldz, float zscale,
                  const float *__restrict__ absmax, float *__restrict__ scale_out, void *__restrict__ z, int64_t Mpad,
                  int64_t Kcap, int lane_rows, bool vec, int align) {
  constexpr int LANES = kPackThreads / kPackGroups;
  if (absmax) {
    zscale = panel_scale(*absmax);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *scale_out = zscale;
  }
  const int64_t k = ((int64_t)blockIdx.x * kPackGroups + threadIdx.x % kPackGroups) * C;
  if (k >= round_up(K, kKAlign)) return;
  const int64_t nrb = ceil_div(M, (int64_t)LANES * lane_rows);
  for (int64_t rb = blockIdx.y; rb < nrb; rb += gridDim.y) {
    int64_t m = (nrb - 1 - rb) * LANES * lane_rows + threadIdx.x / kPackGroups;
#pragma unroll 2
    for (int i = 0; i < lane_rows; ++i, m += LANES) {
      if (m >= M) break;
      float vr[C], vi[C];
      load_row<C>(zs + m * ldz, k, K, vec, vr, vi);
      if constexpr (MODE == MVB_Z_C64) {
        float2 *p = static_cast<float2 *>(z) + m * Kcap + k;
#pragma unroll
        for (int j = 0; j < C; j += 4) {
          const uint32_t w[8] = {__float_as_uint(vr[j]),     __float_as_uint(vi[j]),     __float_as_uint(vr[j + 1]),
                                 __float_as_uint(vi[j + 1]), __float_as_uint(vr[j + 2]), __float_as_uint(vi[j + 2]),
                                 __float_as_uint(vr[j + 3]), __float_as_uint(vi[j + 3])};
          if (align == 2)
            store_sector(p + j, w);
          else
            store_words<8>(p + j, w);
        }
      } else {
        constexpr int KB = kKBlockBytes / (MODE == MVB_GEMM_TF32_3 ? 4 : 2);
        constexpr int NPL = MODE == MVB_GEMM_BF16_6 ? 6 : 4;
        const int64_t off = panel_off(m, k, Mpad, KB, NPL);
        if (align == 2 || (align == 1 && MODE != MVB_GEMM_TF32_3)) {
          const int64_t off2 = panel_off(m, k + C / 2, Mpad, KB, NPL);
          put_split<MODE, C>(z, panel_plane_stride(KB), off, off2, 0, vr, zscale);
          put_split<MODE, C>(z, panel_plane_stride(KB), off, off2, 1, vi, zscale);
        } else {
#pragma unroll
          for (int j = 0; j < C; j += 2) {
            const int64_t o = panel_off(m, k + j, Mpad, KB, NPL);
            PanelWriter<MODE>::put(z, panel_plane_stride(KB), o, 0, vr + j, 2, zscale);
            PanelWriter<MODE>::put(z, panel_plane_stride(KB), o, 1, vi + j, 2, zscale);
          }
        }
      }
    }
  }
}

// Largest |z|: the squares in FP64 (exact for complex64), one square root per
// thread -- it is monotonic, so the result is that of a root per element, which
// bounded this pass.  Two elements per load where the source allows (vec), and one
// atomic per CTA: one per warp, 9,472 on one word, took 8 us whatever the size.
// 275 MB: 53 us, against 78; 1 M elements: 3.9 against 8.7.
constexpr int kAbsmaxThreads = 256;

template <typename CT>
__global__ void __launch_bounds__(kAbsmaxThreads) absmax_kernel(const CT *__restrict__ z, int64_t n, float *__restrict__ out, bool vec) {
  double m2 = 0.0;
  auto take = [&](double x, double y) { m2 = fmax(m2, x * x + y * y); };
  const int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  if (sizeof(CT) == 8 && vec) {
    const float4 *z4 = reinterpret_cast<const float4 *>(z);
    const int64_t n4 = n / 2;
    int64_t i = i0;
    for (; i + 3 * step < n4; i += 4 * step) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __ldg(z4 + i + u * step);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        take(v[u].x, v[u].y);
        take(v[u].z, v[u].w);
      }
    }
    for (; i < n4; i += step) {
      const float4 v = __ldg(z4 + i);
      take(v.x, v.y);
      take(v.z, v.w);
    }
    if ((n & 1) && i0 == 0) take(z[n - 1].x, z[n - 1].y);
  } else {
    for (int64_t i = i0; i < n; i += step) {
      const CT v = z[i];
      take(v.x, v.y);
    }
  }
  float m = (float)sqrt(m2);
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float warp_m[kAbsmaxThreads / 32];
  if ((threadIdx.x & 31) == 0) warp_m[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kAbsmaxThreads / 32; ++w) m = fmaxf(m, warp_m[w]);
    // non-negative floats order like their bit patterns
    atomicMax(reinterpret_cast<int *>(out), __float_as_int(m));
  }
}

}  // namespace mvb

using namespace mvb;

static int launch_absmax(const void *z, int z_c128, int64_t n, float *out, cudaStream_t s) {
  if (n == 0) return MVB_OK;
  const int threads = kAbsmaxThreads;
  const int64_t blocks = std::min<int64_t>(ceil_div(n, threads * 4), (int64_t)num_sms() * 8);
  const bool vec = reinterpret_cast<uintptr_t>(z) % 16 == 0;
  if (z_c128)
    absmax_kernel<double2><<<(unsigned)blocks, threads, 0, s>>>(static_cast<const double2 *>(z), n, out, vec);
  else
    absmax_kernel<float2><<<(unsigned)blocks, threads, 0, s>>>(static_cast<const float2 *>(z), n, out, vec);
  return check_launch("absmax_kernel");
}

extern "C" int mvb_absmax(const void *z, int z_c128, int64_t n, float *out, void *stream) {
  if (!out || n < 0 || (n > 0 && !z)) return fail(MVB_ERR_ARG, "mvb_absmax: bad arguments");
  return launch_absmax(z, z_c128, n, out, as_stream(stream));
}

extern "C" size_t mvb_zpanel_bytes(int mode, int64_t Mpad, int64_t Kcap) {
  if (mode == MVB_Z_C64) return (size_t)Mpad * Kcap * 8;
  return (size_t)2 * mode_terms(mode) * Mpad * Kcap * mode_elem_bytes(mode);
}

static int check_panel(int mode, int64_t M, int64_t Mpad, int64_t Kcap, const char *who) {
  if (mode < MVB_GEMM_BF16_3 || mode > MVB_GEMM_F16_3) return fail(MVB_ERR_ARG, "%s: unknown mode %d", who, mode);
  if (Kcap % kKAlign) return fail(MVB_ERR_ARG, "%s: Kcap must be a multiple of %d", who, kKAlign);
  if (Mpad < M) return fail(MVB_ERR_ARG, "%s: Mpad < M", who);
  if (mode != MVB_Z_C64 && Mpad % kTile) return fail(MVB_ERR_ARG, "%s: Mpad must be a multiple of %d", who, kTile);
  return MVB_OK;
}

extern "C" int mvb_exptau(const double *antpos, int A, double freq, const double *crd, int64_t ld, int64_t nsrc,
                          void *exptau, int out_c128, void *stream) {
  if (A < 0 || nsrc < 0 || ((int64_t)A * nsrc > 0 && (!antpos || !crd || !exptau)))
    return fail(MVB_ERR_ARG, "mvb_exptau: bad arguments");
  const int64_t total = (int64_t)A * nsrc;
  if (total == 0) return MVB_OK;
  const int threads = 256;
  const int64_t blocks = std::min<int64_t>(ceil_div(total, threads), (int64_t)num_sms() * 16);
  exptau_kernel<<<(unsigned)blocks, threads, 0, as_stream(stream)>>>(antpos, A, freq * kInvC, crd, ld, nsrc, exptau,
                                                                     out_c128);
  return check_launch("exptau_kernel");
}

template <int MODE, bool POL, bool GROUP, bool WIDE>
static int launch_tau_z_form(const TauZArgs &p, int F, int X, dim3 grid, size_t smem, cudaStream_t s) {
  auto launch = [&](auto kernel) { return launch_chained("tau_z_kernel", kernel, grid, kTauZThreads, smem, s, p); };
  if constexpr (POL) {
    return launch(tau_z_kernel<MODE, 2, 2, true, GROUP && MODE != MVB_GEMM_TF32_3, WIDE>);
  } else if (X == 2) {
    return F == 2 ? launch(tau_z_kernel<MODE, 2, 2, false, GROUP, WIDE>)
                  : launch(tau_z_kernel<MODE, 2, 1, false, GROUP, WIDE>);
  } else {
    return F == 2 ? launch(tau_z_kernel<MODE, 1, 2, false, GROUP, WIDE>)
                  : launch(tau_z_kernel<MODE, 1, 1, false, GROUP, WIDE>);
  }
}

template <int MODE, bool POL>
static int launch_tau_z_mode(const TauZArgs &p, bool wide, int F, int X, dim3 grid, size_t smem, cudaStream_t s) {
  if (!wide) return launch_tau_z_form<MODE, POL, false, false>(p, F, X, grid, smem, s);
  // (tau_z_cols: the launch's shape goes with this choice)
  if (p.per_z > 1) return launch_tau_z_form<MODE, POL, true, true>(p, F, X, grid, smem, s);
  return launch_tau_z_form<MODE, POL, false, true>(p, F, X, grid, smem, s);
}

// Alignment of a panel that the stores of `cols` consecutive columns of a mode need:
// 8 columns are 16 bytes at 16 bits and whole sectors at 32 and in a complex64 Z; 4
// are 8 bytes, 16, and a sector again (which the fused writer halves).
static int store_align(int mode, int cols) {
  if (mode == MVB_Z_C64) return 32;
  return cols * (mode == MVB_GEMM_TF32_3 ? 4 : 2);
}

static int check_align(const char *who, const void *z, int bytes) {
  if (reinterpret_cast<uintptr_t>(z) % bytes) return fail(MVB_ERR_ARG, "%s: panel not %d-byte aligned", who, bytes);
  return MVB_OK;
}

// The launch of both fused writers (arguments checked by the callers).
template <bool POL>
static int launch_tau_z(const char *who, TauZArgs p, const double *antpos, int A, double freq, const double *freqs_dev, int nfreq,
                        const double *crd, int64_t ld, const int32_t *n_dev, int64_t nsrc, const int32_t *sidx,
                        const void *beam, int64_t beam_ld, int nbeam, const int32_t *beam_idx, int F, int X, int mode,
                        float zscale, void *z, int64_t z_stride, int64_t Mpad, int64_t Kcap, void *stream) {
  const int64_t cols = round_up(nsrc * X, kKAlign);
  if (cols == 0) return MVB_OK;
  // The package's own panels are aligned to the wide stores; a C caller's may lie on
  // (or be spaced by) less, and then go out a frequency per CTA in half-wide stores.
  const int align = store_align(mode, kTauZCols);
  const bool wide = reinterpret_cast<uintptr_t>(z) % align == 0 && (nfreq == 1 || z_stride % align == 0);
  if (int rc = wide ? MVB_OK : check_align(who, z, mode == MVB_Z_C64 ? 16 : store_align(mode, kTauZCols / 2))) return rc;
  p.antpos = antpos;
  p.crd = crd;
  p.freqs = freqs_dev;
  p.f_over_c = freq * kInvC;
  p.ld = ld;
  p.nsrc = nsrc;
  p.beam_ld = beam_ld;
  p.zstride = z_stride;
  p.Mpad = Mpad;
  p.Kcap = Kcap;
  p.n_dev = n_dev;
  p.sidx = sidx;
  p.beam_idx = beam_idx;
  p.beam = static_cast<const float2 *>(beam);
  p.z = z;
  p.A = A;
  p.nbeam = nbeam;
  p.nfreq = nfreq;
  // the fp16 panel's power-of-two scale, half of its exponent on the beam and half
  // on the flux (exact, and neither leaves the range of FP32)
  p.scale_beam = p.scale_flux = 1.f;
  if (mode == MVB_GEMM_F16_3) {
    int e;
    const bool pow2 = std::isfinite(zscale) && std::frexp(zscale, &e) == 0.5f;
    p.scale_beam = !pow2 ? zscale : std::ldexp(1.f, (e - 1) / 2);
    p.scale_flux = !pow2 ? 1.f : std::ldexp(1.f, (e - 1) - (e - 1) / 2);
  }
  const int nq = nbeam * F * X;
  p.staged = nq <= kTauZMaxBFX;
  // A CTA's share in units of (16 antennas x one frequency of its columns): all 8
  // frequencies of 64 antennas in a large launch, less where that leaves fewer than 8
  // CTAs per SM (about half of a sky's slots are below the horizon), frequencies
  // before antennas, since they share more.  Measured with 4 / 8 / 12 / 16 CTAs per
  // SM: 90 unpolarised antennas x 11,180 sources x 8 frequencies 25.8 / 22.7 / 22.6 /
  // 25.4 us, 37 polarised x 2,501 x 7 7.8 / 8.5 / 9.9 / 9.8, 256 unpolarised x 3,000 x
  // 8 22.4 / 17.7 / 20.3 / 20.2; larger ones within 1 %.
  const int64_t xblocks = cols / (kTauZCols * kTauZGroups);
  const int64_t units = xblocks * ceil_div(A, kTauZAntLanes) * nfreq;
  const int64_t share = std::max<int64_t>(1, units / ((int64_t)num_sms() * kTauZCtasPerSm));
  const int64_t parts = ceil_div(nfreq, std::min<int64_t>({share, (int64_t)kTauZMaxFreq, (int64_t)nfreq}));
  const int per = (int)ceil_div(nfreq, parts);
  // At one beam axis two frequencies do not repay the eight-column form (tau_z_cols):
  // 350 antennas x 15,000 slots x 2, half live, tf32x3: 20.6 us one by one, 27.0 together.
  bool group = wide && !(X == 1 && per == 2);
  if (POL && mode == MVB_GEMM_TF32_3) group = false;
  if (!POL && X * F == 4 && (mode == MVB_GEMM_TF32_3 || mode == MVB_GEMM_BF16_6))
    group = group && xblocks * ceil_div(A, kTauZAnts) * ceil_div(nfreq, per) >= (int64_t)num_sms() * kTauZWideCtasPerSm;
  p.per_z = group ? per : 1;
  const int tcols = tau_z_cols(X, p.per_z > 1);  // (a launch of one frequency per CTA: the form that is not GROUP)
  const int64_t lanes =
      std::min<int64_t>(std::max<int64_t>(share * (kTauZCols / tcols) / p.per_z, 1), kTauZAnts / kTauZAntLanes);
  const int64_t ablocks = ceil_div(A, lanes * kTauZAntLanes);
  p.ants = (int)round_up(ceil_div(A, ablocks), kTauZAntLanes);  // even shares, whole lanes
  const dim3 grid((unsigned)(cols / (tcols * kTauZGroups)), (unsigned)ceil_div(A, p.ants),
                  (unsigned)ceil_div(nfreq, p.per_z));
  const int bs = tcols / X * kTauZGroups;
  const size_t smem = (size_t)p.per_z * bs * (POL ? sizeof(float4) : sizeof(float)) +
                      (p.staged ? (size_t)nbeam * F * tcols * kTauZGroups * sizeof(float2) : 0);
  cudaStream_t s = as_stream(stream);
  switch (mode) {
    case MVB_GEMM_BF16_3: return launch_tau_z_mode<MVB_GEMM_BF16_3, POL>(p, wide, F, X, grid, smem, s);
    case MVB_GEMM_BF16_6: return launch_tau_z_mode<MVB_GEMM_BF16_6, POL>(p, wide, F, X, grid, smem, s);
    case MVB_GEMM_TF32_3: return launch_tau_z_mode<MVB_GEMM_TF32_3, POL>(p, wide, F, X, grid, smem, s);
    case MVB_GEMM_F16_3: return launch_tau_z_mode<MVB_GEMM_F16_3, POL>(p, wide, F, X, grid, smem, s);
    default: return launch_tau_z_mode<MVB_Z_C64, POL>(p, wide, F, X, grid, smem, s);
  }
}

// Fused phase + Z writer for nfreq frequencies: freqs_dev == nullptr means one
// frequency, freq; otherwise freqs_dev[0 .. nfreq) on the device, with the
// fluxes sflux_ld floats and the panels z_stride bytes apart.
static int tau_z_impl(const char *who, const double *antpos, int A, double freq, const double *freqs_dev, int nfreq,
                      const double *crd, int64_t ld, const int32_t *n_dev, int64_t nsrc, const float *sflux,
                      int64_t sflux_ld, const int32_t *sidx, const void *beam, int64_t beam_ld, int nbeam,
                      const int32_t *beam_idx, int F, int X, int mode, float zscale, void *z, int64_t z_stride,
                      int64_t Mpad, int64_t Kcap, void *stream) {
  if (A <= 0 || nsrc < 0 || !antpos || !z || !beam || !sflux || (nsrc > 0 && !crd) || (F != 1 && F != 2) ||
      (X != 1 && X != 2) || nbeam <= 0 || beam_ld < nsrc || nfreq <= 0 || nfreq > 65535)
    return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  int rc = check_panel(mode, (int64_t)A * F, Mpad, Kcap, who);
  if (rc) return rc;
  if (round_up(nsrc * X, kKAlign) > Kcap) return fail(MVB_ERR_ARG, "%s: Kcap too small for nsrc * nax", who);
  if (nfreq > 1 && (sflux_ld < nsrc || z_stride < (int64_t)mvb_zpanel_bytes(mode, Mpad, Kcap) || z_stride % 16))
    return fail(MVB_ERR_ARG, "%s: flux rows or panels overlap", who);
  TauZArgs p{};
  p.sflux = sflux;
  p.sflux_ld = sflux_ld;
  return launch_tau_z<false>(who, p, antpos, A, freq, freqs_dev, nfreq, crd, ld, n_dev, nsrc, sidx, beam, beam_ld, nbeam,
                             beam_idx, F, X, mode, zscale, z, z_stride, Mpad, Kcap, stream);
}

extern "C" int mvb_tau_z(const double *antpos, int A, double freq, const double *crd, int64_t ld, const int32_t *n_dev,
                         int64_t nsrc, const float *sflux, const int32_t *sidx, const void *beam, int64_t beam_ld,
                         int nbeam, const int32_t *beam_idx, int F, int X, int mode, float zscale, void *z,
                         int64_t Mpad, int64_t Kcap, void *stream) {
  return tau_z_impl("mvb_tau_z", antpos, A, freq, nullptr, 1, crd, ld, n_dev, nsrc, sflux, 0, sidx, beam, beam_ld,
                    nbeam, beam_idx, F, X, mode, zscale, z, 0, Mpad, Kcap, stream);
}

extern "C" int mvb_tau_z_grouped(const double *antpos, int A, const double *freqs, int nfreq, const double *crd,
                                 int64_t ld, const int32_t *n_dev, int64_t nsrc, const float *sflux, int64_t sflux_ld,
                                 const int32_t *sidx, const void *beam, int64_t beam_ld, int nbeam,
                                 const int32_t *beam_idx, int F, int X, int mode, float zscale, void *z,
                                 size_t z_stride, int64_t Mpad, int64_t Kcap, void *stream) {
  if (!freqs || z_stride > (size_t)INT64_MAX) return fail(MVB_ERR_ARG, "mvb_tau_z_grouped: bad arguments");
  return tau_z_impl("mvb_tau_z_grouped", antpos, A, 0.0, freqs, nfreq, crd, ld, n_dev, nsrc, sflux, sflux_ld, sidx,
                    beam, beam_ld, nbeam, beam_idx, F, X, mode, zscale, z, (int64_t)z_stride, Mpad, Kcap, stream);
}

static int z_pack_impl(const char *who, const void *zsrc, int z_c128, int64_t M, int64_t K, int64_t ldz, int mode,
                       float zscale, const float *absmax, float *scale_out, void *z, int64_t Mpad, int64_t Kcap,
                       cudaStream_t s) {
  const int64_t cols = round_up(K, kKAlign);
  if (M == 0 || cols == 0) return MVB_OK;
  // the narrowest stores: 16 bytes of a complex64 Z, pairs of float32 or bf16, single fp16
  int rc = check_align(who, z, mode == MVB_Z_C64 ? 16 : mode == MVB_GEMM_TF32_3 ? 8 : mode == MVB_GEMM_F16_3 ? 2 : 4);
  if (rc) return rc;
  const bool vec = reinterpret_cast<uintptr_t>(zsrc) % 16 == 0 && (z_c128 || ldz % 2 == 0);
  const int64_t xblocks = ceil_div(cols, kPackGroups * pack_cols(mode, z_c128 ? 16 : 8, vec));
  // four rows a lane (a 64-row block) where that still leaves eight CTAs per SM
  constexpr int lanes = kPackThreads / kPackGroups;
  const int lane_rows = xblocks * ceil_div(M, 4 * lanes) >= (int64_t)num_sms() * 8 ? 4 : 1;
  const dim3 grid((unsigned)xblocks, (unsigned)std::min<int64_t>(ceil_div(M, (int64_t)lane_rows * lanes), 65535));
  const int align = reinterpret_cast<uintptr_t>(z) % 32 == 0 ? 2 : (reinterpret_cast<uintptr_t>(z) % 16 == 0 ? 1 : 0);
#define MVB_PACK(M_, CT, VEC)                                                                                       \
  z_pack_kernel<M_, CT, pack_cols(M_, sizeof(CT), VEC)><<<grid, kPackThreads, 0, s>>>(static_cast<const CT *>(zsrc), M, K, ldz, zscale, absmax,     \
                                                      scale_out, z, Mpad, Kcap, lane_rows, vec, align)
#define MVB_PACK2(M_) \
  if (z_c128)         \
    MVB_PACK(M_, double2, true); \
  else if (vec)       \
    MVB_PACK(M_, float2, true); \
  else                \
    MVB_PACK(M_, float2, false)
  switch (mode) {
    case MVB_GEMM_BF16_3: MVB_PACK2(MVB_GEMM_BF16_3); break;
    case MVB_GEMM_BF16_6: MVB_PACK2(MVB_GEMM_BF16_6); break;
    case MVB_GEMM_TF32_3: MVB_PACK2(MVB_GEMM_TF32_3); break;
    case MVB_GEMM_F16_3: MVB_PACK2(MVB_GEMM_F16_3); break;
    default: MVB_PACK2(MVB_Z_C64); break;
  }
#undef MVB_PACK2
#undef MVB_PACK
  return check_launch("z_pack_kernel");
}

static int check_pack(const char *who, const void *zsrc, int64_t M, int64_t K, int64_t ldz, int mode, const void *z,
                      int64_t Mpad, int64_t Kcap) {
  if (M < 0 || K < 0 || ldz < K || !z || (M * K > 0 && !zsrc)) return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  int rc = check_panel(mode, M, Mpad, Kcap, who);
  if (rc) return rc;
  if (round_up(K, kKAlign) > Kcap) return fail(MVB_ERR_ARG, "%s: Kcap too small", who);
  return MVB_OK;
}

extern "C" int mvb_z_pack(const void *zsrc, int z_c128, int64_t M, int64_t K, int64_t ldz, int mode, float zscale,
                          void *z, int64_t Mpad, int64_t Kcap, void *stream) {
  int rc = check_pack("mvb_z_pack", zsrc, M, K, ldz, mode, z, Mpad, Kcap);
  if (rc) return rc;
  return z_pack_impl("mvb_z_pack", zsrc, z_c128, M, K, ldz, mode, zscale, nullptr, nullptr, z, Mpad, Kcap,
                     as_stream(stream));
}

extern "C" int mvb_z_pack_scaled(const void *zsrc, int z_c128, int64_t M, int64_t K, int64_t ldz, int mode,
                                 float *scale, void *z, int64_t Mpad, int64_t Kcap, void *stream) {
  const char *who = "mvb_z_pack_scaled";
  int rc = check_pack(who, zsrc, M, K, ldz, mode, z, Mpad, Kcap);
  if (rc) return rc;
  if (!scale || ldz != K || M * K == 0) return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  cudaStream_t s = as_stream(stream);
  cudaError_t e = cudaMemsetAsync(scale, 0, sizeof(float), s);
  if (e != cudaSuccess) return fail(MVB_ERR_CUDA, "%s: %s", who, cudaGetErrorString(e));
  rc = launch_absmax(zsrc, z_c128, M * K, scale, s);
  if (rc) return rc;
  return z_pack_impl(who, zsrc, z_c128, M, K, ldz, mode, 1.f, scale, scale + 1, z, Mpad, Kcap, s);
}

static int tau_z_pol_impl(const char *who, const double *antpos, int A, double freq, const double *freqs_dev,
                          int nfreq, const double *crd, int64_t ld, const int32_t *n_dev, int64_t nsrc,
                          const float *coh, int64_t coh_ld, const int32_t *sidx, const double *rot, const void *beam,
                          int64_t beam_ld, int nbeam, const int32_t *beam_idx, int mode, float zscale, void *z,
                          int64_t z_stride, int64_t Mpad, int64_t Kcap, void *stream) {
  const int F = 2, X = 2;
  if (A <= 0 || nsrc < 0 || !antpos || !z || !beam || !coh || !rot || (nsrc > 0 && !crd) || nbeam <= 0 ||
      beam_ld < nsrc || nfreq <= 0 || nfreq > 65535)
    return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  int rc = check_panel(mode, (int64_t)A * F, Mpad, Kcap, who);
  if (rc) return rc;
  if (round_up(nsrc * X, kKAlign) > Kcap) return fail(MVB_ERR_ARG, "%s: Kcap too small for nsrc * nax", who);
  if (reinterpret_cast<uintptr_t>(coh) % 16 || reinterpret_cast<uintptr_t>(rot) % 16)
    return fail(MVB_ERR_ARG, "%s: coh and rot must be 16-byte aligned", who);
  if (nfreq > 1 && (coh_ld < nsrc || z_stride < (int64_t)mvb_zpanel_bytes(mode, Mpad, Kcap) || z_stride % 16))
    return fail(MVB_ERR_ARG, "%s: coherency rows or panels overlap", who);
  TauZArgs p{};
  p.coh = reinterpret_cast<const float4 *>(coh);
  p.coh_ld = coh_ld;
  p.rot = reinterpret_cast<const double2 *>(rot);
  return launch_tau_z<true>(who, p, antpos, A, freq, freqs_dev, nfreq, crd, ld, n_dev, nsrc, sidx, beam, beam_ld, nbeam,
                            beam_idx, F, X, mode, zscale, z, z_stride, Mpad, Kcap, stream);
}

extern "C" int mvb_tau_z_pol(const double *antpos, int A, double freq, const double *crd, int64_t ld,
                             const int32_t *n_dev, int64_t nsrc, const float *coh, const int32_t *sidx,
                             const double *rot, const void *beam, int64_t beam_ld, int nbeam,
                             const int32_t *beam_idx, int mode, float zscale, void *z, int64_t Mpad, int64_t Kcap,
                             void *stream) {
  return tau_z_pol_impl("mvb_tau_z_pol", antpos, A, freq, nullptr, 1, crd, ld, n_dev, nsrc, coh, 0, sidx, rot, beam,
                        beam_ld, nbeam, beam_idx, mode, zscale, z, 0, Mpad, Kcap, stream);
}

extern "C" int mvb_tau_z_pol_grouped(const double *antpos, int A, const double *freqs, int nfreq, const double *crd,
                                     int64_t ld, const int32_t *n_dev, int64_t nsrc, const float *coh, int64_t coh_ld,
                                     const int32_t *sidx, const double *rot, const void *beam, int64_t beam_ld,
                                     int nbeam, const int32_t *beam_idx, int mode, float zscale, void *z,
                                     size_t z_stride, int64_t Mpad, int64_t Kcap, void *stream) {
  if (!freqs || z_stride > (size_t)INT64_MAX) return fail(MVB_ERR_ARG, "mvb_tau_z_pol_grouped: bad arguments");
  return tau_z_pol_impl("mvb_tau_z_pol_grouped", antpos, A, 0.0, freqs, nfreq, crd, ld, n_dev, nsrc, coh, coh_ld,
                        sidx, rot, beam, beam_ld, nbeam, beam_idx, mode, zscale, z, (int64_t)z_stride, Mpad, Kcap,
                        stream);
}

extern "C" int mvb_z_from_exptau(const void *exptau, int e_c128, int64_t e_ld, int A, int64_t nsrc, const float *sflux,
                                 const void *beam, int64_t beam_ld, int nbeam, const int32_t *beam_idx, int F, int X,
                                 int mode, float zscale, void *z, int64_t Mpad, int64_t Kcap, void *stream) {
  if (A <= 0 || nsrc < 0 || !exptau || !z || !beam || !sflux || (F != 1 && F != 2) || (X != 1 && X != 2) ||
      nbeam <= 0 || beam_ld < nsrc || e_ld < nsrc)
    return fail(MVB_ERR_ARG, "mvb_z_from_exptau: bad arguments");
  int rc = check_panel(mode, (int64_t)A * F, Mpad, Kcap, "mvb_z_from_exptau");
  if (rc) return rc;
  if (round_up(nsrc * X, kKAlign) > Kcap) return fail(MVB_ERR_ARG, "mvb_z_from_exptau: Kcap too small");
  const int64_t s_max = round_up(nsrc * X, kKAlign) / X;
  if (s_max == 0) return MVB_OK;
  rc = check_align("mvb_z_from_exptau", z, store_align(mode, kZExtSrc * X));
  if (rc) return rc;
  dim3 grid((unsigned)ceil_div(s_max, kZExtBlockSrc), (unsigned)ceil_div(A, kTauZAnts));
  const bool staged = nbeam * F * X <= kTauZMaxBFX;
  const size_t smem = staged ? (size_t)nbeam * F * X * kZExtRow * sizeof(float2) : 0;
  const float2 *bm = static_cast<const float2 *>(beam);
  cudaStream_t s = as_stream(stream);
#define MVB_ZX(M, XX, E)                                                                                            \
  do {                                                                                                              \
    if (staged)                                                                                                     \
      z_exptau_kernel<M, XX, E, true><<<grid, kTauZThreads, smem, s>>>(exptau, e_ld, A, nsrc, sflux, bm, beam_ld,    \
                                                                       nbeam, beam_idx, F, zscale, z, Mpad, Kcap);  \
    else                                                                                                            \
      z_exptau_kernel<M, XX, E, false><<<grid, kTauZThreads, 0, s>>>(exptau, e_ld, A, nsrc, sflux, bm, beam_ld,     \
                                                                     nbeam, beam_idx, F, zscale, z, Mpad, Kcap);    \
  } while (0)
#define MVB_ZX3(M, E) \
  if (X == 2)         \
    MVB_ZX(M, 2, E);  \
  else                \
    MVB_ZX(M, 1, E)
#define MVB_ZX2(M)    \
  if (e_c128)         \
    MVB_ZX3(M, 2);    \
  else                \
    MVB_ZX3(M, 1)
  switch (mode) {
    case MVB_GEMM_BF16_3: MVB_ZX2(MVB_GEMM_BF16_3); break;
    case MVB_GEMM_BF16_6: MVB_ZX2(MVB_GEMM_BF16_6); break;
    case MVB_GEMM_TF32_3: MVB_ZX2(MVB_GEMM_TF32_3); break;
    case MVB_GEMM_F16_3: MVB_ZX2(MVB_GEMM_F16_3); break;
    default: MVB_ZX2(MVB_Z_C64); break;
  }
#undef MVB_ZX2
#undef MVB_ZX3
#undef MVB_ZX
  return check_launch("z_exptau_kernel");
}

// sqrt(0.5 I) per source and frequency (cpu/cpu.py:188), transposed from the
// caller's (N, Nf) float64 Stokes I to the (Nf, N) float32 rows the Z writers
// read; 32 x 32 tiles through shared memory so both sides are coalesced.
namespace mvb {
__global__ void flux_sqrt_half_kernel(const double *__restrict__ flux, int64_t N, int nf, float *__restrict__ out) {
  __shared__ float tile[32][33];
  const int64_t s0 = (int64_t)blockIdx.x * 32;
  const int f0 = blockIdx.y * 32;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int64_t s = s0 + r;
    const int f = f0 + threadIdx.x;
    if (s < N && f < nf) tile[r][threadIdx.x] = (float)sqrt(0.5 * flux[s * nf + f]);
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += blockDim.y) {
    const int f = f0 + r;
    const int64_t s = s0 + threadIdx.x;
    if (s < N && f < nf) out[(int64_t)f * N + s] = tile[threadIdx.x][r];
  }
}
}  // namespace mvb

extern "C" int mvb_flux_sqrt_half(const double *flux, int64_t N, int nf, float *sflux, void *stream) {
  if (N < 0 || nf <= 0 || (N > 0 && (!flux || !sflux))) return fail(MVB_ERR_ARG, "mvb_flux_sqrt_half: bad arguments");
  if (N == 0) return MVB_OK;
  if (ceil_div(N, 32) > 0x7fffffff || ceil_div(nf, 32) > 65535)
    return fail(MVB_ERR_ARG, "mvb_flux_sqrt_half: too many sources or frequencies");
  dim3 grid((unsigned)ceil_div(N, 32), (unsigned)ceil_div(nf, 32));
  flux_sqrt_half_kernel<<<grid, dim3(32, 8), 0, as_stream(stream)>>>(flux, N, nf, sflux);
  return check_launch("flux_sqrt_half_kernel");
}
