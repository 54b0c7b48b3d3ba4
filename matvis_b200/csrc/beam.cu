// A5: beam interpolation at the above-horizon sources.
//
// Reference: gpu/beams.py:127-200 (gpu_beam_interpolation: order-1
// map_coordinates per (beam, feed, axis) at row = za / dza, col = (az - azmin) /
// daz, sqrt after interpolating a power beam), gpu/beams.py:103-124 and
// coordinates.py:31-88 (enu_to_az_za with orientation="uvbeam").
//
// Edge rule (scipy / cupyx map_coordinates, mode='constant', order=1): a point
// whose row or column coordinate lies outside [0, n-1] gives 0; inside, the
// 2x2 neighbours are blended with FP64 weights (a neighbour index of n carries
// weight 0).
//
// Layout: grids (nbeam, nax, nfeed, nza, naz), complex64 or float32 power;
// output (nbeam, nfeed, nax, nout) complex.  One thread per source: the FP64
// (az, za) and each beam's grid coordinates are computed once and serve all its
// planes, whose 2 x 2 neighbours are gathered through L1 / L2 (a beam's grids are
// about 1 MB: they stay in L2).  What bounds it is the gathers' sectors: four
// planes of a complex beam stored apart take 2.6 sectors per (plane, source) for
// scattered sources; with the four values of a grid point side by side
// (beam_pack_kernel, into the caller's workspace) one neighbour is one 32-byte
// sector for all of them.  Measured, 91 x 361 grids: 98,304 map sources x 4
// polarised beams 16.5 us, 500,000 scattered sources x 4 70 us, 2,500 sources x 1
// 6.2 us.  The form this replaces staged one real 131 KB plane per CTA in shared
// memory (one CTA of 8 warps per SM, each plane reading the coordinates that a pass
// before it had written): 95, 521 and 16.5 us.
#include <math_constants.h>

#include "common.cuh"

namespace mvb {

constexpr int kBeamThreads = 128;
constexpr int64_t kBeamPackMin = 300000;  // (source slots - 2 grid points) x beams from which packing pays

struct BeamParams {
  double daz, dza, azmin;
};

// numpy.mod(a, b) for b > 0: result in [0, b).
__device__ __forceinline__ double py_mod(double a, double b) {
  double m = fmod(a, b);
  if (m != 0.0 && m < 0.0) m += b;
  return m;
}

// enu_to_az_za(orientation="uvbeam", periodic_azimuth=True), FP64.
__device__ __forceinline__ void az_za_uvbeam(double e, double n, double &az, double &za) {
  const double lsqr = n * n + e * e;
  const double zeta = lsqr < 1.0 ? sqrt(1.0 - lsqr) : 0.0;
  const double a = atan2(e, n);
  za = 0.5 * CUDART_PI - asin(zeta);
  az = py_mod(0.5 * CUDART_PI - a, 2.0 * CUDART_PI);
}

// Order-1 neighbours of one grid position: offsets (in grid points) and weights;
// in = false outside [0, n - 1] on either axis (the sample is then 0).
struct Cell {
  int64_t o00, o01, o10, o11;
  double fr, fc;
  bool in;
};

__device__ __forceinline__ Cell grid_cell(int nza, int naz, double row, double col) {
  Cell c{0, 0, 0, 0, 0.0, 0.0, false};
  if (!(row >= 0.0 && row <= (double)(nza - 1) && col >= 0.0 && col <= (double)(naz - 1))) return c;
  const int r0 = min((int)floor(row), nza - 1);
  const int c0 = min((int)floor(col), naz - 1);
  c.fr = row - r0;
  c.fc = col - c0;
  const int r1 = min(r0 + 1, nza - 1), c1 = min(c0 + 1, naz - 1);
  c.o00 = (int64_t)r0 * naz + c0;
  c.o01 = (int64_t)r0 * naz + c1;
  c.o10 = (int64_t)r1 * naz + c0;
  c.o11 = (int64_t)r1 * naz + c1;
  c.in = true;
  return c;
}

__device__ __forceinline__ double blend(const Cell &c, double v00, double v01, double v10, double v11) {
  return (1.0 - c.fr) * ((1.0 - c.fc) * v00 + c.fc * v01) + c.fr * ((1.0 - c.fc) * v10 + c.fc * v11);
}

// kind 0: complex64, 1: complex128 (one store); 2, 3: the same for an output that is
// not aligned to its complex elements (a C caller's), one store per component.
__device__ __forceinline__ void store_beam(void *out, int kind, int64_t idx, double re, double im) {
  if (kind == 0) {
    static_cast<float2 *>(out)[idx] = make_float2((float)re, (float)im);
  } else if (kind == 1) {
    static_cast<double2 *>(out)[idx] = make_double2(re, im);
  } else if (kind == 2) {
    static_cast<float *>(out)[2 * idx] = (float)re;
    static_cast<float *>(out)[2 * idx + 1] = (float)im;
  } else {
    static_cast<double *>(out)[2 * idx] = re;
    static_cast<double *>(out)[2 * idx + 1] = im;
  }
}

// A complex value of a grid; `whole`: the grids are 8-byte aligned.
__device__ __forceinline__ float2 load_grid(const float *g, int64_t o, bool whole) {
  return whole ? __ldg(reinterpret_cast<const float2 *>(g) + o) : make_float2(__ldg(g + 2 * o), __ldg(g + 2 * o + 1));
}

// The four complex planes of every beam, (nbeam, 4, points) -> (nbeam, points, 4).
__global__ void beam_pack_kernel(const float2 *__restrict__ grids, int64_t points, int nbeam,
                                 float4 *__restrict__ packed) {
  pdl_wait();
  pdl_trigger();
  const int64_t total = (int64_t)nbeam * points;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = i / points, p = i % points;
    const float2 *g = grids + 4 * b * points + p;
    const float2 v0 = g[0], v1 = g[points], v2 = g[2 * points], v3 = g[3 * points];
    packed[2 * i] = make_float4(v0.x, v0.y, v1.x, v1.y);
    packed[2 * i + 1] = make_float4(v2.x, v2.y, v3.x, v3.y);
  }
}

// One thread per source; blockIdx.y = a slice of `per_y` beams.  KIND 0: complex64
// planes, 1: float32 power planes, 2: packed complex64 (4 values per grid point,
// nax = nfeed = 2).  AZZA: crd holds (az, za) rows instead of ENU (e, n).
template <int KIND, bool AZZA>
__global__ void __launch_bounds__(kBeamThreads)
    beam_gather_kernel(const float *__restrict__ grids, int nbeam, int per_y, int nax, int nfeed, int nza, int naz,
                       const BeamParams *__restrict__ params, const double *__restrict__ crd, int64_t ld,
                       const int32_t *__restrict__ n_dev, int64_t nsrc, void *__restrict__ out, int out_kind,
                       int64_t nout, int32_t *__restrict__ status) {
  pdl_wait();
  pdl_trigger();
  const int64_t n = n_dev ? min((int64_t)__ldcg(n_dev), nsrc) : nsrc;
  const bool whole = reinterpret_cast<uintptr_t>(grids) % 8 == 0;
  const int b0 = blockIdx.y * per_y, b1 = min(b0 + per_y, nbeam);
  const int64_t points = (int64_t)nza * naz;
  const int ngrid = nax * nfeed;
  for (int64_t i = blockIdx.x * (int64_t)kBeamThreads + threadIdx.x; i < nout; i += (int64_t)gridDim.x * kBeamThreads) {
    if (i >= n) {  // slots past the count hold zeros
      for (int64_t q = (int64_t)b0 * ngrid; q < (int64_t)b1 * ngrid; ++q) store_beam(out, out_kind, q * nout + i, 0.0, 0.0);
      continue;
    }
    double az, za;
    if constexpr (AZZA) {
      az = __ldcg(crd + i);
      za = __ldcg(crd + ld + i);
    } else {
      az_za_uvbeam(__ldcg(crd + i), __ldcg(crd + ld + i), az, za);
    }
    bool finite = true;
    for (int b = b0; b < b1; ++b) {
      const BeamParams bp = params[b];
      const Cell c = grid_cell(nza, naz, za / bp.dza, (az - bp.azmin) / bp.daz);
      const int64_t row0 = (int64_t)b * ngrid * nout + i;  // output (b, feed, axis, i), rows nout apart
      if constexpr (KIND == 2) {
        const float4 *g = reinterpret_cast<const float4 *>(grids) + 2 * (int64_t)b * points;
        // values of a point: (ax 0, feed 0), (ax 0, feed 1), (ax 1, feed 0), (ax 1, feed 1)
        double v[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
          // packed by the kernel before
          const float4 v00 = c.in ? __ldca(g + 2 * c.o00 + h) : z4, v01 = c.in ? __ldca(g + 2 * c.o01 + h) : z4;
          const float4 v10 = c.in ? __ldca(g + 2 * c.o10 + h) : z4, v11 = c.in ? __ldca(g + 2 * c.o11 + h) : z4;
          v[4 * h + 0] = blend(c, v00.x, v01.x, v10.x, v11.x);
          v[4 * h + 1] = blend(c, v00.y, v01.y, v10.y, v11.y);
          v[4 * h + 2] = blend(c, v00.z, v01.z, v10.z, v11.z);
          v[4 * h + 3] = blend(c, v00.w, v01.w, v10.w, v11.w);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // q = 2 ax + feed -> output row 2 feed + ax
          const double re = v[2 * q], im = v[2 * q + 1];
          finite = finite && isfinite(re) && isfinite(im);
          store_beam(out, out_kind, row0 + (int64_t)(2 * (q & 1) + (q >> 1)) * nout, re, im);
        }
      } else {
#pragma unroll 2
        for (int q = 0; q < ngrid; ++q) {
          const int ax = q / nfeed, fd = q % nfeed;
          double re = 0.0, im = 0.0;
          if (KIND == 0) {
            if (c.in) {
              const float *g = grids + 2 * ((int64_t)b * ngrid + q) * points;
              const float2 v00 = load_grid(g, c.o00, whole), v01 = load_grid(g, c.o01, whole),
                           v10 = load_grid(g, c.o10, whole), v11 = load_grid(g, c.o11, whole);
              re = blend(c, v00.x, v01.x, v10.x, v11.x);
              im = blend(c, v00.y, v01.y, v10.y, v11.y);
            }
          } else {
            if (c.in) {
              const float *g = grids + ((int64_t)b * ngrid + q) * points;
              re = blend(c, __ldg(g + c.o00), __ldg(g + c.o01), __ldg(g + c.o10), __ldg(g + c.o11));
            }
            re = sqrt(re);
          }
          finite = finite && isfinite(re) && isfinite(im);
          store_beam(out, out_kind, row0 + (int64_t)(fd * nax + ax) * nout, re, im);
        }
      }
    }
    if (status && !finite) atomicOr(status, MVB_DEV_NONFINITE);
  }
}

__global__ void beam_gaussian_kernel(const double *__restrict__ sigmas, int nbeam, const double *__restrict__ crd,
                                     int64_t ld, const int32_t *__restrict__ n_dev, int64_t nsrc, void *__restrict__ out,
                                     int out_c128, int64_t nout) {
  pdl_wait();
  pdl_trigger();
  const int64_t n = n_dev ? min((int64_t)__ldcg(n_dev), nsrc) : nsrc;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nout; i += (int64_t)gridDim.x * blockDim.x) {
    double za = 0.0;
    if (i < n) {
      double az;
      az_za_uvbeam(__ldcg(crd + i), __ldcg(crd + ld + i), az, za);
    }
    for (int b = 0; b < nbeam; ++b) {
      const double s = sigmas[b];
      // sqrt of the power exp(-za^2 / s^2)
      const double v = i < n ? exp(-(za * za) / (2.0 * s * s)) : 0.0;
      if (out_c128) {
        double *o = static_cast<double *>(out) + 2 * ((int64_t)b * nout + i);
        o[0] = v;
        o[1] = 0.0;
      } else {
        float *o = static_cast<float *>(out) + 2 * ((int64_t)b * nout + i);
        o[0] = (float)v;
        o[1] = 0.0f;
      }
    }
  }
}

}  // namespace mvb

using namespace mvb;

static int beam_interp_impl(bool azza, const void *grids, int grid_kind, int nbeam, int nax, int nfeed, int nza,
                            int naz, const double *params, const double *crd, int64_t ld, const int32_t *n_dev,
                            int64_t nsrc, void *out, int out_c128, int64_t nout, int32_t *status, void *ws,
                            size_t ws_bytes, void *stream) {
  const char *who = azza ? "mvb_beam_interp_azza" : "mvb_beam_interp";
  if (!grids || !params || !out || (nsrc > 0 && !crd) || nbeam <= 0 || nax <= 0 || nfeed <= 0 || nza < 1 || naz < 1 ||
      (grid_kind != 0 && grid_kind != 1) || nout < nsrc || nsrc < 0)
    return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  if (ws && (ws_bytes < (size_t)2 * nbeam * nout * sizeof(double) || reinterpret_cast<uintptr_t>(ws) % 8))
    return fail(MVB_ERR_ARG, "%s: workspace too small", who);
  if (nout == 0) return MVB_OK;
  const int nsm = num_sms();
  const int64_t points = (int64_t)nza * naz;
  const BeamParams *bp = reinterpret_cast<const BeamParams *>(params);
  const float *g = static_cast<const float *>(grids);
  cudaStream_t s = as_stream(stream);
  // Packing costs a launch (about 2 us) and one read and write of the grids, and
  // saves the gathers sectors: 91 x 361 grids, half of the slots occupied by
  // scattered sources: 4 beams, 66,000 slots 14.0 us packed, 12.4 not; 120,000 slots
  // 18.5 both; 196,608 slots 22.7 and 28.7; 1 beam, 500,000 slots 17.7 and 17.6.
  const bool pack = !azza && ws && grid_kind == 0 && nax == 2 && nfeed == 2 && nbeam * (nout - 2 * points) >= kBeamPackMin &&
                    ws_bytes >= (size_t)nbeam * points * 32 && reinterpret_cast<uintptr_t>(ws) % 16 == 0 &&
                    reinterpret_cast<uintptr_t>(grids) % 8 == 0;
  const int out_kind = (out_c128 ? 1 : 0) + (reinterpret_cast<uintptr_t>(out) % (out_c128 ? 16 : 8) ? 2 : 0);
  if (pack) {
    const int64_t blocks = std::min<int64_t>(ceil_div(nbeam * points, 256), (int64_t)nsm * 8);
    int rc = launch_chained("beam_pack_kernel", beam_pack_kernel, (unsigned)blocks, 256, 0, s,
                            static_cast<const float2 *>(grids), points, nbeam, static_cast<float4 *>(ws));
    if (rc) return rc;
    g = static_cast<const float *>(ws);
  }
  // few sources: the beams are sliced over CTAs, each of which repeats the source's
  // az/za in FP64, so no more slices than fill the GPU four times over (200 power beams,
  // 50,000 sources: 165 us in two slices, 185 with a CTA per beam; 20 beams: 20.1)
  const int64_t xblocks = std::min<int64_t>(ceil_div(nout, kBeamThreads), (int64_t)nsm * 64);
  const int64_t slices = std::min<int64_t>(nbeam, ceil_div((int64_t)nsm * 4, xblocks));
  const dim3 grid((unsigned)xblocks, (unsigned)std::min<int64_t>(slices, 65535));
  const int per = (int)ceil_div(nbeam, grid.y);
#define MVB_BEAM(KIND, AZZA)                                                                                          \
  launch_chained("beam_gather_kernel", beam_gather_kernel<KIND, AZZA>, grid, kBeamThreads, 0, s, g, nbeam, per, nax,  \
                 nfeed, nza, naz, bp, crd, ld, n_dev, nsrc, out, out_kind, nout, status)
  if (pack) return MVB_BEAM(2, false);
  if (grid_kind == 0) return azza ? MVB_BEAM(0, true) : MVB_BEAM(0, false);
  return azza ? MVB_BEAM(1, true) : MVB_BEAM(1, false);
#undef MVB_BEAM
}

extern "C" size_t mvb_beam_interp_ws_bytes(int nbeam, int64_t nout) {
  if (nbeam <= 0 || nout <= 0) return 8;
  return (size_t)2 * nbeam * nout * sizeof(double);
}

extern "C" int mvb_beam_interp(const void *grids, int grid_kind, int nbeam, int nax, int nfeed, int nza, int naz,
                               const double *params, const double *crd, int64_t ld, const int32_t *n_dev, int64_t nsrc,
                               void *out, int out_c128, int64_t nout, int32_t *status, void *ws, size_t ws_bytes,
                               void *stream) {
  return beam_interp_impl(false, grids, grid_kind, nbeam, nax, nfeed, nza, naz, params, crd, ld, n_dev, nsrc, out,
                          out_c128, nout, status, ws, ws_bytes, stream);
}

extern "C" int mvb_beam_interp_azza(const void *grids, int grid_kind, int nbeam, int nax, int nfeed, int nza, int naz,
                                    const double *params, const double *azza, int64_t ld, int64_t nsrc, void *out,
                                    int out_c128, void *stream) {
  return beam_interp_impl(true, grids, grid_kind, nbeam, nax, nfeed, nza, naz, params, azza, ld, nullptr, nsrc, out,
                          out_c128, nsrc, nullptr, nullptr, 0, stream);
}

extern "C" int mvb_beam_gaussian(const double *sigmas, int nbeam, const double *crd, int64_t ld, const int32_t *n_dev,
                                 int64_t nsrc, void *out, int out_c128, int64_t nout, void *stream) {
  if (!sigmas || !out || nbeam <= 0 || nsrc < 0 || nout < nsrc || (nsrc > 0 && !crd))
    return fail(MVB_ERR_ARG, "mvb_beam_gaussian: bad arguments");
  if (nout == 0) return MVB_OK;
  const int threads = 256;
  const int64_t blocks = std::min<int64_t>(ceil_div(nout, threads), (int64_t)num_sms() * 8);
  return launch_chained("beam_gaussian_kernel", beam_gaussian_kernel, (unsigned)blocks, threads, 0, as_stream(stream),
                        sigmas, nbeam, crd, ld, n_dev, nsrc, out, out_c128, nout);
}
