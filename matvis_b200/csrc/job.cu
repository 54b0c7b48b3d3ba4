// The launch sequence of a batched visibility job, on the host.
//
// Reference: wrapper.py:180-199 (the frequency loop), cpu/cpu.py:247-272 and
// gpu/gpu.py:197-254 (the time and chunk loops): rotation, horizon selection, beam,
// tau, Z, product, sum over chunks.
//
// Every call below is one of the library's own entry points.  A small job is a few
// hundred launches of 2 to 20 us; made one by one through the Python binding they
// cost 10 to 16 us of host time each (37 antennas x 5,003 sources x 7 frequencies x
// 5 times: 478 us a run for 290 us of kernels; 361 us from here, one call a run, and
// 290 us with the kernels launched as a chain: launch_chained).
#include <algorithm>

#include "common.cuh"

using namespace mvb;

static int job_prologue(const mvb_job &j, int t, int c, void *stream) {
  int rc;
  if (c == 0) {
    const double *src = j.eci;
    if (j.bcrs) {
      if (j.refresh[t] && (rc = mvb_bcrs(j.eci, j.nsrc, j.astrom + 18 * (int64_t)t, j.bcrs, stream))) return rc;
      src = j.bcrs;
    }
    if (j.nchunks == 1)
      return rotate_select(src, j.nsrc, j.rot + 9 * (int64_t)t, j.topo, j.crd, j.kept, j.n_above, j.cap, j.status,
                           j.select_ws, j.select_ws_bytes, stream);
    if ((rc = mvb_rotate(src, j.nsrc, j.rot + 9 * (int64_t)t, j.topo, stream))) return rc;
  }
  const int64_t c0 = std::min<int64_t>(c * j.chunk_size, j.nsrc), c1 = std::min<int64_t>((c + 1) * j.chunk_size, j.nsrc);
  if ((rc = mvb_horizon_compact(j.topo, j.nsrc, c0, c1, nullptr, j.crd, j.kept, nullptr, j.n_above, j.cap, j.status,
                                j.select_ws, j.select_ws_bytes, stream)))
    return rc;
  return MVB_OK;
}

// The beam of frequency index f (an achromatic one has a single entry).
static int job_beam(const mvb_job &j, int f, void *stream) {
  if (j.sigmas)
    return mvb_beam_gaussian(j.sigmas, j.nbeam, j.crd, j.cap, j.n_above, j.cap, j.beam, 0, j.cap, stream);
  return mvb_beam_interp(j.grids[f], j.grid_kind, j.nbeam, j.nfeed, j.nfeed, j.nza, j.naz, j.grid_params[f], j.crd,
                         j.cap, j.n_above, j.cap, j.beam, 0, j.cap, j.status, j.beam_ws, j.beam_ws_bytes, stream);
}

// Frequencies f0 .. f0 + g - 1 of one chunk, g > 1 only for a group of panels.
static int job_group(const mvb_job &j, int t, int f0, int g, int accumulate, void *stream) {
  int rc;
  const int F = j.nfeed;
  uint8_t *out = static_cast<uint8_t *>(j.vis) + f0 * j.vis_f_stride + t * j.vis_t_stride;
  if (j.freq_group > 1) {
    if (j.coh)
      rc = mvb_tau_z_pol_grouped(j.antpos, j.nant, j.freqs_dev + f0, g, j.crd, j.cap, j.n_above, j.cap,
                                 j.coh + 4 * f0 * j.flux_ld, j.flux_ld, j.kept, j.frame_rot, j.beam, j.cap, j.nbeam,
                                 j.beam_idx, j.mode, j.zscale, j.z, j.z_stride, j.Mpad, j.Kcap, stream);
    else
      rc = mvb_tau_z_grouped(j.antpos, j.nant, j.freqs_dev + f0, g, j.crd, j.cap, j.n_above, j.cap,
                             j.sflux + f0 * j.flux_ld, j.flux_ld, j.kept, j.beam, j.cap, j.nbeam, j.beam_idx, F, F,
                             j.mode, j.zscale, j.z, j.z_stride, j.Mpad, j.Kcap, stream);
  } else if (j.coh) {
    rc = mvb_tau_z_pol(j.antpos, j.nant, j.freqs[f0], j.crd, j.cap, j.n_above, j.cap, j.coh + 4 * f0 * j.flux_ld,
                       j.kept, j.frame_rot, j.beam, j.cap, j.nbeam, j.beam_idx, j.mode, j.zscale, j.z, j.Mpad, j.Kcap,
                       stream);
  } else {
    rc = mvb_tau_z(j.antpos, j.nant, j.freqs[f0], j.crd, j.cap, j.n_above, j.cap, j.sflux + f0 * j.flux_ld, j.kept,
                   j.beam, j.cap, j.nbeam, j.beam_idx, F, F, j.mode, j.zscale, j.z, j.Mpad, j.Kcap, stream);
  }
  if (rc) return rc;
  if (j.mode == MVB_Z_C64) {
    if (j.plan)
      return mvb_vecdot_staged(j.z, j.Kcap, j.n_above, j.cap, F, F, j.nant, j.plan, j.nbundles, j.npairs, j.k_chunk,
                               j.ws, j.ws_bytes, out, j.out_c128, accumulate, j.status, stream);
    return mvb_vecdot(j.z, j.Kcap, j.n_above, j.cap, F, F, j.pairs, j.npairs, j.k_chunk, j.ws, j.ws_bytes, out,
                      j.out_c128, accumulate, stream);
  }
  if ((rc = herk_grouped_chained(j.z, j.z_stride, g, j.mode, j.Mpad, (int64_t)j.nant * F, j.Kcap, j.n_above, j.cap, F,
                             j.k_chunk, j.drain_ksteps, j.ws, j.ws_bytes, j.status, stream)))
    return rc;
  return herk_reduce_grouped_chained(j.ws, j.ws_bytes, g, j.Mpad, j.Kcap, j.n_above, j.cap, F, j.k_chunk, j.nant, F,
                                 j.pairs, j.npairs, out, (size_t)j.vis_f_stride, j.out_c128,
                                 1.0 / ((double)j.zscale * j.zscale), accumulate, stream);
}

extern "C" int mvb_job_enqueue(const mvb_job *job, int t0, int t1, int c0, int c1, int f0, int f1, void *stream) {
  const char *who = "mvb_job_enqueue";
  if (!job) return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  const mvb_job &j = *job;
  if (t0 < 0 || t1 > j.ntime || c0 < 0 || c1 > j.nchunks || f0 < 0 || f1 > j.nfreq || j.freq_group < 1 ||
      (f0 > 0 && f0 % j.freq_group) || j.chunk_size <= 0 || !j.rot || (j.bcrs && (!j.refresh || !j.astrom)) ||
      (!j.sigmas && (!j.grids || !j.grid_params)) || (j.coh && !j.frame_average) || (!j.coh && !j.sflux && j.nfreq) ||
      (t0 < t1 && f0 < f1 && (!j.freqs || !j.freqs_dev || !j.vis)) || (j.chromatic && (j.freq_group != 1 || j.sigmas)) ||
      (j.mode == MVB_Z_C64 && (j.freq_group != 1 || (!j.plan && !j.pairs && j.npairs))))
    return fail(MVB_ERR_ARG, "%s: bad arguments", who);
  // Frequencies after the first group continue one (time, chunk), chunks after the first
  // one time: more than one would take the sky or the rotation the last call left.
  const int nt = std::max(t1 - t0, 0), nc = std::max(c1 - c0, 0);
  if ((f0 > 0 && f0 < f1 && (int64_t)nt * nc > 1) || (c0 > 0 && nt > 1 && nc > 0))
    return fail(MVB_ERR_ARG, "%s: a later frequency or chunk of more than one time or chunk", who);
  int rc;
  // the products' work-unit counter: cleared here, then by each reduction
  if (t0 < t1 && c0 < c1 && f0 < f1 && j.mode != MVB_Z_C64 && (rc = clear_unit_counter(j.ws, j.ws_bytes, stream))) return rc;
  for (int t = t0; t < t1; ++t)
    for (int c = c0; c < c1; ++c) {
      if (f0 == 0) {
        if ((rc = job_prologue(j, t, c, stream))) return rc;
        if (!j.chromatic && (rc = job_beam(j, 0, stream))) return rc;
        if (j.coh && (rc = mvb_coherency_rotation(j.radec, j.nsrc, j.kept, j.crd, j.cap, j.n_above, j.cap,
                                                  j.frame_average + 9 * (int64_t)t, j.frame_rot, stream)))
          return rc;
      }
      for (int f = f0; f < f1; f += j.freq_group) {
        if (j.chromatic && (rc = job_beam(j, f, stream))) return rc;
        if ((rc = job_group(j, t, f, std::min(j.freq_group, f1 - f), c > 0, stream))) return rc;
      }
    }
  return MVB_OK;
}
