// sm_100a kernels of the moving-mesh finite-volume step.
//
// One RK substep is eight launches in a CUDA graph:
//   k_merge    per annulus pair : the r-face list of pair (i, i+1) (face_create
//                                 / build_jloop) as a checked parallel merge of
//                                 the two sorted phi-edge lists, cell_set_w
//                                 and the frame terms of a moving frame
//                                 (k_ring_mean per annulus: cell_set_w of a
//                                 rigidly rotating mesh)
//   k_cellprep per cell         : cell_clean_pi, cell_plm_p, GravMass copy /
//                                 clean_pi
//   k_rslope   per r face       : the face slope S and the wrapped offsets of
//                                 cell_plm_rz / riemann_setup_rz
//   k_plm_r    per cell         : cell_plm_rz (face-weighted slope + limiter)
//                                 and, in substep 1, the CFL minimum
//                                 (cell_mindt), from which dt is formed
//                                 (timestep_set_dt: step_dt)
//   k_source   per cell         : the increments of cell_add_src and
//                                 cell_add_visc_src; per-annulus constants
//   k_flux_phi per phi face     : riemann_setup_p + riemann_AddFlux
//   k_flux_r   per r face       : riemann_setup_rz + riemann_AddFlux; both
//                                 flux kernels store dt*dA*F per face
//   k_update   per cell         : gathers the increments in the reference's
//                                 accumulation order, cell_add_split_fictitious,
//                                 cell_update_phi/_dphi, cell_calc_prim, the
//                                 fixed radial boundary, cell_bc_damp and
//                                 cell_calc_cons; its first block advances the
//                                 GravMass state
// and, for disks with the outflow radial boundary, k_outflow, eight lanes per
// boundary cell (cell_boundary_outflow_r).  k_merge runs beside k_cellprep on a
// second stream, and k_source beside k_flux_r; k_flux_phi runs on a third
// stream up to two waves of cells, behind k_source above that (dctx_substep).
//
// Built with -fmad=false: every expression keeps the reference's operation
// order and rounding (double '/' and sqrt are IEEE-rounded on the GPU), so
// paths without transcendentals reproduce the reference bit for bit.
#include <cuda_runtime.h>
#include <climits>
#include <math.h>
#include <stdint.h>

#include "dgpu_step.cuh"

// minimum resident blocks per SM requested from the register allocator
// (measured on B200, circumbinary disk: these kernels are latency-bound, so
// occupancy beats the extra spills)
#ifndef DGPU_MINB_FACE
#define DGPU_MINB_FACE 5
#endif
#ifndef DGPU_MINB_CELLPREP
#define DGPU_MINB_CELLPREP 5
#endif
#ifndef DGPU_MINB_PLM
#define DGPU_MINB_PLM 4
#endif
#ifndef DGPU_MINB_FLUX
#define DGPU_MINB_FLUX 4
#endif
#ifndef DGPU_MINB_FLUXR
#define DGPU_MINB_FLUXR 3
#endif
#ifndef DGPU_MINB_SOURCE
#define DGPU_MINB_SOURCE 3
#endif
#ifndef DGPU_MINB_UPDATE
#define DGPU_MINB_UPDATE 4
#endif
#ifndef DGPU_MINB_PREP
#define DGPU_MINB_PREP 4
#endif
#ifndef DGPU_MINB_SWEEP
#define DGPU_MINB_SWEEP 3
#endif

// Threads per block of k_plm_r, k_flux_phi, k_flux_r and k_update: half of BLK
// at the same registers per thread.  A block's registers are given back when
// its slowest warp is done, so smaller blocks leave fewer of them idle (a step
// of 16 disks, 4 M cells: 4.43 ms at 256, 4.37 at 128, 4.38-4.44 at 64; one
// 258,078-cell disk 0.353, 0.351 and 0.353-0.367).
#define TBLK 128

namespace {


// ---------------------------------------------------------------------------
// r-face list of one annulus pair (build_jloop, face_create_destroy.c:22-128)
// ---------------------------------------------------------------------------
struct FaceCtx {
  const double *tin, *din, *tout, *dout;
  int Nin, Nout;
  int *fL, *fR;
  double *fdphi, *fcm;
  int *runs;
  int *sruns;   // copy of runs the rr pass reads (shared memory when staged)
  int *fstart;  // fstart of the inner annulus cells (indexed by j)
  int cap, rcap;
  int *err;
  int offL, offR;  // global cell numbers of inner/outer cell 0 (face records hold global cells)
};

// The body of the reference's j loop for inner cell j starting at outer cell
// jp: emits its faces and advances jp.  n = running face number, s = running
// count of jp advances (the run index of the next face).  FILL writes.
template <bool FILL>
__device__ void face_cell(const FaceCtx &c, int j, int &jp, int &n, int &s) {
  int jm = j - 1;
  if (jm < 0) jm = c.Nin - 1;
  bool mark = false;
  auto emit = [&](double dphi, double tp) {
    if (FILL) {
      if (n < c.cap) {
        c.fL[n] = c.offL + j;
        c.fR[n] = c.offR + jp;
        c.fdphi[n] = dphi;
        c.fcm[n] = tp - .5 * dphi;
      }
      if (mark && s < c.rcap) c.runs[s] = c.sruns[s] = n;
    }
    mark = false;
    ++n;
  };
  auto advance = [&]() {
    ++jp;
    if (jp == c.Nout) jp = 0;
    ++s;
    mark = true;
  };
  if (FILL) c.fstart[j] = n;
  double dp = c.tout[jp] - c.tin[jm];
  dp = wrap_pos(dp, c.err);
  if (c.din[j] < dp) {
    emit(c.din[j], c.tin[j]);
    return;
  }
  emit(dp, c.tout[jp]);
  advance();
  dp = c.tin[j] - c.tout[jp];
  dp = wrap_pm(dp, c.err);
  int guard = 0;
  while (dp > 0.0) {
    emit(c.dout[jp], c.tout[jp]);
    advance();
    dp = c.tin[j] - c.tout[jp];
    dp = wrap_pm(dp, c.err);
    if (++guard > c.Nout + 2) {
      set_err(c.err, DGPU_EF_FACE_OVERFLOW);
      break;
    }
  }
  dp = c.dout[jp] + dp;
  emit(dp, c.tin[j]);
}

// Exclusive scan of one value per thread over the block (blockDim.x a multiple
// of 32, at most 1024); sh needs blockDim.x / 32 entries.
template <typename T>
__device__ T block_excl_scan(T v, T *sh, T &total) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(full, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  if (w == 0) {
    T t = lane < nw ? sh[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(full, t, o);
      if (lane >= o) t += y;
    }
    if (lane < nw) sh[lane] = t;
  }
  __syncthreads();
  T pre = w > 0 ? sh[w - 1] : T(0);
  total = sh[nw - 1];
  __syncthreads();
  return pre + x - v;
}

// Per cell, once per substep: cell_clean_pi of the phi edge
// (src/Cell/cell_misc.c:12-26) and cell_plm_p (src/Cell/cell_plm.c:116-161).
template <typename T, bool PS, int NV = 5>
__device__ __forceinline__ void cellprep_cell(const DevPtrs &d, const TanPtrs &tp, int g, int substep) {
  const Pl QS = {PS ? d.qs : 5};
  const double *traw = substep == 1 ? d.tiph0 : d.tiph1;
  pf_planes(d.prim, NV, QS, g);
  pf(d.dphi + g);
  pf(traw + g);
  const int a = d.cell_ann[g];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  const int np = A.np, off = A.cell_off, j = g - off;
  d.tiphw[g] = wrap_pos(traw[g], d.err);
  const int gl = off + (j == 0 ? np - 1 : j - 1);
  const int gr = off + (j == np - 1 ? 0 : j + 1);
  const double dc = d.dphi[g];
  const double dpL = .5 * (dc + d.dphi[gl]);
  const double dpR = .5 * (dc + d.dphi[gr]);
  const double plm = P.plm;
  // two planes at a time: all five at once spill at this kernel's registers
  auto slopes = [&](auto K, int q) {
    T pc[2], pl[2], pr[2];
    ldk<K.value, T, true>(d.prim, tp.prim, q, QS, g, pc);
    ldk<K.value, T, true>(d.prim, tp.prim, q, QS, gl, pl);
    ldk<K.value, T, true>(d.prim, tp.prim, q, QS, gr, pr);
#pragma unroll
    for (int k = 0; k < K.value; ++k) pc[k] = plm_p_slope(pl[k], pc[k], pr[k], dpL, dpR, plm);
    stk<K.value, T>(d.gradp, tp.gradp, q, QS, g, pc);
  };
  slopes(std::integral_constant<int, 2>(), 0);
  slopes(std::integral_constant<int, 2>(), 2);
  if constexpr (NV == 5) slopes(std::integral_constant<int, 1>(), 4);
  for (int q = 5; q < 5 + (PS ? P.num_n : 0); ++q)
    d.gradp[ix(q, QS, g)] =
        plm_p_slope(ld(d.prim, q, QS, gl), ld(d.prim, q, QS, g), ld(d.prim, q, QS, gr), dpL, dpR, P.plm);
}

// Instances that carry the four-plane form (no_vz) beside the five: the plain
// forward ones.  Each also exists without it (V4 = false), for contexts that
// can never take it (3-D disks) and for the reverse sweep's replays: the two
// forms in one kernel share its register budget, which cost the 3-D torus 5%
// of its step.
template <typename T, bool PS>
constexpr bool forward_v4 = std::is_same<T, double>::value && !PS;

// cellprep_cell for every cell and, for the first cell of each disk,
// gravMass_copy at the start of a step (GravMass_misc.c:20-28) and
// gravMass_clean_pi (GravMass_misc.c:9-17).  Runs concurrently with k_merge.
template <typename T, bool PS = false, bool V4 = forward_v4<T, PS>>
__global__ void __launch_bounds__(BLK, DGPU_MINB_CELLPREP) k_cellprep(DevPtrs d, TanPtrs tp, int substep) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.n_cells) return;
  if (V4 && no_vz(d)) cellprep_cell<T, PS, V4 ? 4 : 5>(d, tp, g, substep);
  else cellprep_cell<T, PS>(d, tp, g, substep);
  const Annulus &A = d.ann[d.cell_ann[g]];
  const DiskParams &P = d.par[A.inst];
  if (g == P.cell_base) {
    InstState &S = d.ist[A.inst];
    if (substep == 1) {
      for (int p = 0; p < 2; ++p) {
        S.grk_r[p] = S.gr[p];
        S.grk_phi[p] = S.gphi[p];
        S.grk_M[p] = S.gM[p];
        S.grk_om[p] = S.gom[p];
        // gravMass_dist of the step-start positions (the CFL's viscosity)
        S.rkx[p] = S.gr[p] * cos(S.gphi[p]);
        S.rky[p] = S.gr[p] * sin(S.gphi[p]);
      }
      S.dtkey = (unsigned long long)__double_as_longlong(1.e100);
    }
    for (int p = 0; p < 2; ++p) S.gphi[p] = wrap_pos(S.gphi[p], d.err);  // 2.*M_PI == PHIMAX
  }
}

// The frame terms of annulus a that depend on the binary's separation
// (A_MILOS) into d.frame, one lane each: sim_rOm_a, sim_rdrOm_a and sim_dtOm_a
// at the annulus centre and sim_rdrOm_a at the radius of pair (i, i+1).
__device__ __forceinline__ void milos_frame(const DevPtrs &d, const DiskParams &P, const Annulus &A, int a,
                                            int lane) {
  if (lane >= DGPU_FR_N) return;
  const InstState &S = d.ist[A.inst];
  const double a_sep = S.gr[0] + S.gr[1];
  const double r = lane == DGPU_FR_FRDROM ? A.f_r : .5 * (A.rp + A.rm);
  double v;
  if (lane == DGPU_FR_ROM) v = milos_rom(r, a_sep);
  else if (lane == DGPU_FR_DTOM) v = milos_dtom(r, a_sep, P.orb_tscale);
  else v = milos_rdrom(r, a_sep);
  d.frame[(size_t)lane * d.n_ann + a] = v;
}

// C_RIGID (cell_set_w.c:41-49): the mass-weighted mean v_phi of annulus a,
// summed in j order like the reference, by one warp.  Its two sums are chains
// of dependent additions (8.2 cycles each on B200), so all else is kept out of
// them: the warp loads 128 cells ahead, puts the terms in shared memory, and
// even lanes add those of one sum while odd lanes add the other's.  (With a
// lane loading and adding cell by cell 32 us for 96 annuli of up to 660 cells;
// with 32 cells ahead and the terms shuffled to every lane 24.)
#define RING_CHUNK 128
__device__ __forceinline__ void ring_mean(const DevPtrs &d, int a, int lane, double (&sh)[2][RING_CHUNK]) {
  constexpr int K = RING_CHUNK / 32;
  const unsigned full = 0xffffffffu;
  const Annulus &A = d.ann[a];
  const Pl QS = {d.qs};
  const int np = A.np, off = A.cell_off;
  const double r = A.r;
  double u[K], m[K], sum = 0.0;
  auto fetch = [&](int j) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      const int c = off + min(j + 32 * i + lane, np - 1);
      u[i] = ldr(d.prim, D_UPP, QS, c);
      m[i] = ldr(d.cons, D_DDD, QS, c);
    }
  };
  fetch(0);
  for (int j = 0; j < np; j += RING_CHUNK) {
#pragma unroll
    for (int i = 0; i < K; ++i) {
      sh[0][32 * i + lane] = r * u[i] * m[i];
      sh[1][32 * i + lane] = m[i];
    }
    __syncwarp();
    if (j + RING_CHUNK < np) fetch(j + RING_CHUNK);
    const double *t = sh[lane & 1];
    if (np - j >= RING_CHUNK) {
#pragma unroll 16
      for (int k = 0; k < RING_CHUNK; ++k) sum += t[k];
    } else {
#pragma unroll 4
      for (int k = 0; k < np - j; ++k) sum += t[k];
    }
    __syncwarp();
  }
  const double w = __shfl_sync(full, sum, 0), Mring = __shfl_sync(full, sum, 1);
  if (lane == 0) d.w_ann[a] = w / Mring;
}

// The ring means of the rigidly rotating disks, a warp per annulus, beside
// k_merge and k_cellprep (only k_plm_r's CFL and later kernels read them; at
// the end of the merge's blocks they stood in the step's chain: Gresho vortex,
// 96 annuli, 0.105 -> 0.090 ms a step).
#define RING_BLK 64
__global__ void __launch_bounds__(RING_BLK) k_ring_mean(DevPtrs d) {
  __shared__ double sh[RING_BLK / 32][2][RING_CHUNK];
  const int a = (blockIdx.x * RING_BLK + threadIdx.x) / 32;
  if (a < d.n_ann && d.par[d.ann[a].inst].w_numeric == DC_RIGID)
    ring_mean(d, a, threadIdx.x & 31, sh[threadIdx.x / 32]);
}

// Per annulus pair (i, i+1) of a disk, one block: the r-face list of
// face_create/build_jloop (src/Face/face_create_destroy.c:22-193) as a checked
// parallel merge, and cell_set_w (src/Cell/cell_set_w.c:12-102) of annulus i.
// Z: the z pair (ring a, ring a+NR) of a 3-D disk (build_jloop with zDir:
// both rings have N_p cells of annulus i) into the z-face arrays; no
// cell_set_w then.
template <bool Z>
__device__ __forceinline__ void merge_pair(const DevPtrs &d, int a, int substep) {
  __shared__ int sh_i[BLK / 32];
  __shared__ int sh_j[BLK];
  __shared__ double sh_v[BLK / 32];
  __shared__ int sh_flag, sh_nf, sh_T;
  // staged phi edges and widths of the pair, then the runs
  extern __shared__ double sm[];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  const double *traw = substep == 1 ? d.tiph0 : d.tiph1;
  const int tid = threadIdx.x, nt = blockDim.x;
  const int np = A.np, off = A.cell_off;
  if (!Z && tid == 0 && P.w_numeric != DC_RIGID) d.w_ann[a] = A.wnum;
  if (!Z && tid >= nt - 32 && P.w_analytic == DA_MILOS) milos_frame(d, P, A, a, tid & 31);
  // the pair's arrays: r faces of (a, a+1), or z faces of (a, a+NR)
  int *const pfL = Z ? d.zfL : d.fL, *const pfR = Z ? d.zfR : d.fR;
  double *const pfdphi = Z ? d.zfdphi : d.fdphi, *const pfcm = Z ? d.zfcm : d.fcm;
  int *const pruns = Z ? d.zruns : d.runs, *const pfstart = Z ? d.zfstart : d.fstart;
  int *const prr = Z ? d.zrr : d.rr;
  int *const p_nf = Z ? d.zpair_nf : d.pair_nf, *const p_jpmin = Z ? d.zpair_jpmin : d.pair_jpmin;
  int *const p_T = Z ? d.zpair_T : d.pair_T, *const p_seq = Z ? d.zpair_seq : d.pair_seq;
  const int fbase = Z ? A.zface_base : A.face_base, fcap = Z ? A.zface_cap : A.face_cap;
  const int rbase = Z ? A.zrun_base : A.run_base;
  const int partner = Z ? a + P.NR : a + 1;
  if (Z ? A.k < P.NZ - 1 : A.i < P.NR - 1) {
    const int npo = d.ann[partner].np;
    const int offo = d.ann[partner].cell_off;
    const int rcap = Z ? A.zrun_cap : A.run_cap;
    const bool staged = d.smem_face >= (int)sizeof(double) * 2 * (np + npo) + (int)sizeof(int) * rcap;
    const double *tin = traw + off, *din = d.dphi + off;
    const double *tout = traw + offo, *dout = d.dphi + offo;
    if (staged) {
      double *s_tin = sm, *s_din = sm + np, *s_tout = sm + 2 * np, *s_dout = sm + 2 * np + npo;
      for (int j = tid; j < np; j += nt) {
        s_tin[j] = tin[j];
        s_din[j] = din[j];
      }
      for (int j = tid; j < npo; j += nt) {
        s_tout[j] = tout[j];
        s_dout[j] = dout[j];
      }
      __syncthreads();
      tin = s_tin;
      din = s_din;
      tout = s_tout;
      dout = s_dout;
    }
    FaceCtx c;
    c.tin = tin;
    c.din = din;
    c.tout = tout;
    c.dout = dout;
    c.Nin = np;
    c.Nout = npo;
    c.fL = pfL + fbase;
    c.fR = pfR + fbase;
    c.fdphi = pfdphi + fbase;
    c.fcm = pfcm + fbase;
    c.runs = pruns + rbase;
    c.sruns = staged ? reinterpret_cast<int *>(sm + 2 * (np + npo)) : c.runs;
    c.fstart = pfstart + off;
    c.cap = fcap;
    c.rcap = rcap;
    c.err = d.err;
    c.offL = off;
    c.offR = offo;
    const double p0 = c.tin[np - 1];

    // jpmin: first outer cell with the smallest wrap(tiph - p0), start (PHIMAX, 0)
    double bv = PHIMAX;
    int bi = 0;
    {
      for (int jp = tid; jp < c.Nout; jp += nt) {
        double dp = wrap_pos(c.tout[jp] - p0, d.err);
        if (dp < bv || (dp == bv && jp < bi)) {
          bv = dp;
          bi = jp;
        }
      }
      // the (value, index) minimum is the same in any order of combination:
      // per warp by shuffles, then over the warps
      const unsigned full = 0xffffffffu;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        double v2 = __shfl_down_sync(full, bv, o);
        int i2 = __shfl_down_sync(full, bi, o);
        if (v2 < bv || (v2 == bv && i2 < bi)) {
          bv = v2;
          bi = i2;
        }
      }
      if ((tid & 31) == 0) {
        sh_v[tid >> 5] = bv;
        sh_i[tid >> 5] = bi;
      }
      __syncthreads();
      bv = sh_v[0];
      bi = sh_i[0];
      for (int w = 1; w < (nt >> 5); ++w) {
        const double v2 = sh_v[w];
        const int i2 = sh_i[w];
        if (v2 < bv || (v2 == bv && i2 < bi)) {
          bv = v2;
          bi = i2;
        }
      }
    }
    const int jpmin = bi;

    // A contiguous chunk of inner cells per thread, from a guessed start: the
    // outer cells that end before the chunk's left edge, counted from jpmin
    // with both measured as wrap(edge - p0).  Every inner cell gives one face
    // and every advance of the outer pointer one more, so that count is also
    // the number of advances before the chunk and, with the chunk's first
    // inner cell, the number of its first face: no counting pass and no scan.
    // The guesses are verified below.  The cells of an annulus are usually of
    // one width, so the search starts where the count would then be and
    // brackets from there.  (258,078-cell disk: 25 -> 21 us; 59,746 cells: 16.3 ->
    // 12.6, its step 0.104 -> 0.099 ms.)
    const int chunk = (np + nt - 1) / nt;
    const int j0 = min(np, tid * chunk), j1 = min(np, j0 + chunk);
    int lo = 0;
    if (j0 > 0 && j0 < np) {
      const double L = wrap_pos(c.tin[j0 - 1] - p0, d.err);
      auto before = [&](int m) {
        int k = jpmin + m;
        if (k >= c.Nout) k -= c.Nout;
        return wrap_pos(c.tout[k] - p0, d.err) < L;
      };
      int hi = c.Nout, m = min(max((int)(L * (c.Nout / PHIMAX)), 0), c.Nout - 1), step = 1;
      if (before(m)) {
        lo = m + 1;
        while (lo < hi) {
          m = min(lo + step - 1, hi - 1);
          step *= 2;
          if (before(m)) {
            lo = m + 1;
          } else {
            hi = m;
            break;
          }
        }
      } else {
        hi = m;
        while (lo < hi) {
          m = max(hi - step, lo);
          step *= 2;
          if (before(m)) {
            lo = m + 1;
            break;
          }
          hi = m;
        }
      }
      while (lo < hi) {
        m = (lo + hi) >> 1;
        if (before(m)) lo = m + 1;
        else hi = m;
      }
    }
    sh_j[tid] = j0 < j1 ? lo : -1;
    if (tid == 0) sh_flag = 0;
    __syncthreads();
    if (j0 < j1) {
      int n = j0 + lo, sv = lo, jp = jpmin + lo;
      if (jp >= c.Nout) jp -= c.Nout;
      for (int j = j0; j < j1; ++j) face_cell<true>(c, j, jp, n, sv);
      if (j1 < np) {
        // the next chunk must start where this one ended: its advances (which
        // also fix its outer cell), and with them its first face
        int next = jpmin + sh_j[tid + 1];
        if (next >= c.Nout) next -= c.Nout;
        if (sh_j[tid + 1] != sv || next != jp) sh_flag = 1;
      } else {
        sh_nf = n;
        sh_T = sv;
      }
    }
    __syncthreads();
    if (sh_flag) {
      // a guess was wrong (coinciding edges): the exact sequential replay of
      // build_jloop from jpmin, over whatever the chunks wrote
      if (tid == 0) {
        int n = 0, sv = 0, jp = jpmin;
        for (int j = 0; j < np; ++j) face_cell<true>(c, j, jp, n, sv);
        sh_nf = n;
        sh_T = sv;
      }
      __syncthreads();
    }
    if (tid == 0) {
      const int ntot = sh_nf, stot = sh_T;
      if (ntot > c.cap || stot + 2 > c.rcap) {
        set_err(d.err, DGPU_EF_FACE_OVERFLOW);
        p_nf[a] = 0;
        p_T[a] = 0;
        sh_nf = 0;
        sh_T = 0;
      } else {
        c.runs[0] = c.sruns[0] = 0;
        c.runs[stot + 1] = c.sruns[stot + 1] = ntot;
        p_nf[a] = ntot;
        p_jpmin[a] = jpmin;
        p_T[a] = stot;
        p_seq[a] = sh_flag;
      }
    }
    __syncthreads();
    // per outer cell, the face ranges of its runs s = jp - jpmin (mod Nout) and
    // s + Nout (the cell at the wrap point); z = INT_MIN flags a third run
    {
      const int nf = sh_nf, T = sh_T;
      for (int jq = tid; jq < npo; jq += nt) {
        int4 rr = make_int4(0, 0, 0, 0);
        if (nf > 0) {
          int s0 = jq - jpmin;
          if (s0 < 0) s0 += npo;
          if (s0 <= T) rr.x = c.sruns[s0], rr.y = c.sruns[s0 + 1];
          if (s0 + npo <= T) rr.z = c.sruns[s0 + npo], rr.w = c.sruns[s0 + npo + 1];
          if (s0 + 2 * npo <= T) rr.z = INT_MIN;
        }
        reinterpret_cast<int4 *>(prr)[offo + jq] = rr;
      }
      // slab slots past the list hold no face
      for (int n = nf + tid; n < c.cap; n += nt) c.fL[n] = -1;
    }
  }
}

__global__ void __launch_bounds__(BLK, DGPU_MINB_FACE) k_merge(DevPtrs d, int substep) {
  merge_pair<false>(d, blockIdx.x, substep);
}

// The z-face lists of a 3-D disk: one block per ring a with k < NZ-1.
__global__ void __launch_bounds__(BLK, DGPU_MINB_FACE) k_zmerge(DevPtrs d, int substep) {
  merge_pair<true>(d, blockIdx.x, substep);
}

// ---------------------------------------------------------------------------
// cell_plm_rz (src/Cell/cell_plm.c:13-114) per cell + CFL (cell_mindt.c:32-100)
// ---------------------------------------------------------------------------
// r-face slope and reconstruction offsets, once per face: the S of
// cell_plm_rz (src/Cell/cell_plm.c:31-53) and the wrapped dpL, dpR that
// cell_plm_rz, riemann_setup_rz (Riemann_setup.c:18-25) and riemann_visc_flux
// (Riemann_routines.c:220-228) all form the same way.
template <typename T, bool PS, int NV = 5>
__device__ __forceinline__ void rslope_face(const DevPtrs &d, const TanPtrs &tp, int slot) {
  const int cL = rd(d.fL + slot);
  if (cL < 0) return;  // slot past the face list of its pair
  const int cR = rd(d.fR + slot);
  const Pl QS = {PS ? d.qs : 5};
  pf_planes(d.prim, NV, QS, cL);
  pf_planes(d.prim, NV, QS, cR);
  pf_planes(d.gradp, NV, QS, cL);
  pf_planes(d.gradp, NV, QS, cR);
  const int a = rd(d.slot_ann + slot);
  const Annulus &A = d.ann[a];
  const double cm = rd(d.fcm + slot);
  double pL = rd(d.tiphw + cL) - .5 * rd(d.dphi + cL);
  double pR = rd(d.tiphw + cR) - .5 * rd(d.dphi + cR);
  double dpL = cm - pL;
  dpL = wrap_pm(dpL, d.err);
  double dpR = pR - cm;
  dpR = wrap_pm(dpR, d.err);
  const double dp[2] = {dpL, dpR};
  stk<2>(d.fdp, 0, P2, slot, dp);
  const double den = A.f_dr + A.f_dl;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    const T WL = ldqr<T>(d.prim, tp.prim, q, QS, cL) + dpL * ldqr<T>(d.gradp, tp.gradp, q, QS, cL);
    const T WR = ldqr<T>(d.prim, tp.prim, q, QS, cR) - dpR * ldqr<T>(d.gradp, tp.gradp, q, QS, cR);
    stq<T>(d.fS, tp.fS, q, QS, slot, (WR - WL) / den);
  }
  for (int q = 5; q < 5 + (PS ? d.par[A.inst].num_n : 0); ++q) {
    const double WL = ldr(d.prim, q, QS, cL) + dpL * ldr(d.gradp, q, QS, cL);
    const double WR = ldr(d.prim, q, QS, cR) - dpR * ldr(d.gradp, q, QS, cR);
    d.fS[ix(q, QS, slot)] = (WR - WL) / den;
  }
}

template <typename T, bool PS = false, bool V4 = forward_v4<T, PS>>
__global__ void __launch_bounds__(BLK) k_rslope(DevPtrs d, TanPtrs tp) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= d.n_slots) return;
  if (V4 && no_vz(d)) rslope_face<T, PS, V4 ? 4 : 5>(d, tp, slot);
  else rslope_face<T, PS>(d, tp, slot);
}

// cell_plm_rz's limiter of plane q (src/Cell/cell_plm.c:81-113) as the
// reference runs it: face after face against the running slope, from the mean
// that grad holds to the limited slope in its place.
template <typename T>
__device__ __noinline__ void limit_seq(const DevPtrs &d, const TanPtrs &tp, int g, int q) {
  const int a = d.cell_ann[g];
  const DiskParams &P = d.par[d.ann[a].inst];
  const Pl QS = {d.qs};
  T gq = ldq<T>(d.grad, tp.grad, q, QS, g);
  for_cell_rface_ranges(d, d.ann[a], a, g, P.NR, [&](int s, int e, int) {
    for (int n = s; n < e; ++n) {
      const T S = ldq<T>(d.fS, tp.fS, q, QS, n);
      if (S * gq < 0.0) gq = 0.0;
      else if (fabs(P.plm * S) < fabs(gq)) gq = P.plm * S;
    }
  });
  stq<T>(d.grad, tp.grad, q, QS, g, gq);
}

// cell_plm_rz's r slope of cell g (src/Cell/cell_plm.c:56-114): the
// face-area-weighted mean of the face slopes S, then the theta limiter against
// each face's S.  One walk over the faces keeps the sum and what the limiter
// needs: the plm * S nearest zero (the first of equals) and whether any S was
// negative or positive.  The limiter then gives 0 if some S opposes the mean,
// else the nearer of the mean and that plm * S, which is where the reference's
// face-by-face loop ends.  It would not where the product of an opposing S and
// the loop's running slope, which an earlier face may have clipped, underflows
// to -0 (or an S is 0), so that its test S * slope < 0 fails: planes where that
// could be (limit_left) run the loop itself (limit_seq).  Two walks, one for the sum and
// one for the limiter, took 229 us in substep 2 of 16 disks (4 M cells) and
// 23.5 us of one 258,078-cell disk against 191 and 19.3 here.  Forming each S
// here from the cell across the face, with no slopes stored, took 495 us for
// the 191 and k_rslope's 200: the walk is as long as the longest lane's, and a
// face-parallel kernel has no such waste.
template <typename T, bool PS, int NV = 5>
__device__ __forceinline__ void plm_r_grad(const DevPtrs &d, const TanPtrs &tp, int g) {
  const Pl QS = {PS ? d.qs : 5};
  pf(d.rr + 4 * (size_t)g);
  pf(d.fstart + g);
  pf(d.dphi + g);
  const int a = d.cell_ann[g];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  const double plm = P.plm;
  T gq[5], lim[5];
  int neg = plm < 0.0 ? 31 : 0, pos = neg;  // (a negative PLM: always the loop)
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    gq[q] = 0.0;
    lim[q] = HUGE_VAL;
  }
  for_cell_rface_ranges(d, A, a, g, P.NR, [&](int s, int e, int outer) {
    const Annulus &Q = outer ? d.ann[a - 1] : A;
    const double fr = Q.f_r, fperp = Q.f_dperp;
    for (int n = s; n < e; ++n) {
      const double dA = fr * rd(d.fdphi + n) * fperp;
      T Sf[5];
      ldk<NV, T>(d.fS, tp.fS, 0, QS, n, Sf);
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const T S = Sf[q];
        gq[q] += S * dA;
        const T ps = plm * S;
        if (fabs(ps) < fabs(lim[q])) lim[q] = ps;
        neg |= (S < 0.0) << q;
        pos |= (S > 0.0) << q;
      }
    }
  });
  double dAtot;
  {
    double dz = A.dz, dp = d.dphi[g];
    if (A.i == 0) dAtot = dz * A.rp * dp;
    else if (A.i == P.NR - 1) dAtot = dz * A.rm * dp;
    else dAtot = dz * (A.rp + A.rm) * dp;
  }
  const double floor = limit_floor(plm);
  int seq = 0;  // planes that run the loop itself
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    T m = gq[q] / dAtot;
    const bool opposed = (m < 0.0 && (pos >> q & 1)) || (m > 0.0 && (neg >> q & 1));
    seq |= limit_left(m, lim[q], opposed, floor) << q;
    gq[q] = m;
  }
  stk<NV, T>(d.grad, tp.grad, 0, QS, g, gq);
  for (; seq; seq &= seq - 1) limit_seq<T>(d, tp, g, __ffs(seq) - 1);
  // passive scalars: the same face-weighted slope and limiter
  for (int q = 5; q < 5 + (PS ? P.num_n : 0); ++q) {
    double gs = 0.0;
    for_cell_rfaces(d, A, a, g, P.NR, [&](const RFace &F, int slot, int) {
      double dA = F.r * F.dphi * F.dperp;
      gs += ld(d.fS, q, QS, slot) * dA;
    });
    d.grad[ix(q, QS, g)] = gs / dAtot;
    limit_seq<double>(d, tp, g, q);
  }
}

// The CFL step of non-ghost cell g (cell_mindt, src/Cell/cell_mindt.c:10-100)
// as the bit pattern of the positive double (~0: no candidate, also for a NaN,
// which is reported).  rkx/rky/rkM: the step-start GravMass positions and
// masses (the viscous limit's nu); wa = wiph of the annulus.
__device__ __forceinline__ unsigned long long cfl_key(const DevPtrs &d, const Annulus &A, const DiskParams &P,
                                                      int g, double wa, const double *rkx, const double *rky,
                                                      const double *rkM) {
  const Pl QS = {d.qs};
  const double *traw = d.tiph0;
  double w = .5 * (wa + wa);
  double dr = A.rp - A.rm;
  double r = .5 * (A.rp + A.rm);
  double dx = dr;
  double rdphi = .5 * (A.rp + A.rm) * d.dphi[g];
  if (rdphi < dr) dx = rdphi;
  if (dx > A.dz) dx = A.dz;
  double Pp = ld(d.prim, D_PPP, QS, g), rho = ld(d.prim, D_RHO, QS, g);
  double vp = ld(d.prim, D_UPP, QS, g) * r - w;
  double vr = ld(d.prim, D_URR, QS, g), vz = ld(d.prim, D_UZZ, QS, g);
  double cs = sqrt(P.gamma * Pp / rho);
  double cf2 = cs * cs;
  double maxv = sqrt(cf2) + sqrt(vr * vr + vp * vp + vz * vz);
  double dt = P.cfl * dx / maxv;
  if (P.has_visc) {
    double nu;
    if (P.visc_const == 1) {
      nu = P.visc;
    } else {
      double tc = traw[g] - 0.5 * d.dphi[g];
      if (P.init_type == DI_SHEAR) {
        nu = P.visc * P.gamma * Pp / rho * dpow(fabs(r * cos(tc)), 2.0);
        if (r * cos(tc) > 20.) nu = 0.000000001;
      } else {
        double sc, cc;
        sincos(tc, &sc, &cc);
        const double x = r * cc, y = r * sc;
        double d0 = gm_dist_xy(x, y, rkx[0], rky[0]);
        double d1 = gm_dist_xy(x, y, rkx[1], rky[1]);
        double eps = P.g_eps;
        nu = P.visc * Pp / rho /
             sqrt(dpow(d0 * d0 + eps * eps, -1.5) * rkM[0] + dpow(d1 * d1 + eps * eps, -1.5) * rkM[1]);
      }
    }
    double dt_visc = .25 * dx * dx / nu;
    dt = dt / (1. + dt / dt_visc);
  }
  unsigned long long key = (unsigned long long)__double_as_longlong(dt);
  if (__longlong_as_double((long long)key) < 0.0 || dt != dt) key = ~0ull;
  // the reference's minimum skips such a cell too (cell_mindt.c); here it
  // is also reported
  if (dt != dt) set_err(d.err, DGPU_EF_NONFINITE);
  return key;
}

template <typename T, int MB = DGPU_MINB_PLM, bool PS = false, bool V4 = forward_v4<T, PS>>
__global__ void __launch_bounds__(TBLK, MB * (BLK / TBLK)) k_plm_r(const __grid_constant__ DevPtrs d, const __grid_constant__ TanPtrs tp,
                                                                        int substep) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = d.n_cells;
  unsigned long long key = ~0ull;
  int inst = -1;
  if (g < d.n_inst) {
    // GravMass positions of this substep (gravMass_dist, cell_source.c:103-107)
    InstState &S = d.ist[g];
    for (int p = 0; p < 2; ++p) {
      S.gc[p] = cos(S.gphi[p]);
      S.gs[p] = sin(S.gphi[p]);
      S.gx[p] = S.gr[p] * S.gc[p];
      S.gy[p] = S.gr[p] * S.gs[p];
    }
  }
  if (g < N) {
    if (V4 && no_vz(d)) plm_r_grad<T, PS, V4 ? 4 : 5>(d, tp, g);
    else plm_r_grad<T, PS>(d, tp, g);
    const int a = d.cell_ann[g];
    const Annulus &A = d.ann[a];
    inst = A.inst;
    // CFL candidate (cell_mindt), substep 1 only, non-ghost annuli
    if (substep == 1 && (A.kind & DGPU_AK_CFL)) {
      const InstState &S = d.ist[A.inst];
      key = cfl_key(d, A, d.par[A.inst], g, d.w_ann[a], S.rkx, S.rky, S.grk_M);
    }
  }
  if (substep != 1) return;

  // minimum per disk: warp reduction when the warp holds one disk
  const unsigned full = 0xffffffffu;
  int inst0 = __shfl_sync(full, inst, 0);
  bool uniform = __all_sync(full, inst == inst0);
  if (uniform) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long k2 = __shfl_down_sync(full, key, o);
      key = k2 < key ? k2 : key;
    }
    if ((threadIdx.x & 31) == 0 && inst0 >= 0 && key != ~0ull) atomicMin(&d.ist[inst0].dtkey, key);
  } else if (inst >= 0 && key != ~0ull) {
    atomicMin(&d.ist[inst].dtkey, key);
  }
}

// Stores each disk's dt of substep 1, for readers of InstState.dt that run
// before k_update does.
__global__ void k_dt(DevPtrs d) {
  for (int k = threadIdx.x; k < d.n_inst; k += blockDim.x) {
    InstState &S = d.ist[k];
    S.dt = cfl_dt(S, d.par[k]);
  }
}

// ---------------------------------------------------------------------------
// Face increments: one thread per phi face (at its left cell) and per r-face slot
// ---------------------------------------------------------------------------
// phi faces: thread per cell j, face (j, j+1) (riemann_setup_p, Riemann_setup.c:46-80)
// ist: the disks' states with this substep's GravMass positions (NULL: d.ist).
template <typename T, bool PS, int NV = 5>
__device__ __forceinline__ void flux_phi_cell(const DevPtrs &d, const TanPtrs &tp, int g, const InstState *ist,
                                              int substep) {
  const Pl QS = {PS ? d.qs : 5}, QF = {PS ? d.qf : 8};
  // the cell's own planes (its right neighbour's share the lines) ahead of
  // the annulus lookups
  pf_planes(d.prim, NV, QS, g);
  pf_planes(d.gradp, NV, QS, g);
  pf_planes(d.grad, NV, QS, g);
  pf(d.tiphw + g);
  pf(d.dphi + g);
  const int a = d.cell_ann[g];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  const int j = g - A.cell_off;
  const int cL = g, cR = (j == A.np - 1) ? A.cell_off : g + 1;
  const double dpL = d.dphi[cL], dpR = d.dphi[cR];
  const double dz = A.dz;
  const double dr = A.rp - A.rm;
  const double r = .5 * (A.rp + A.rm);
  const double dA = dr * dz;
  T pL[5], pR[5];
  {
    T gL[5], gR[5];
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cL, pL);
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cR, pR);
    ldk<NV, T>(d.gradp, tp.gradp, 0, QS, cL, gL);
    ldk<NV, T>(d.gradp, tp.gradp, 0, QS, cR, gR);
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      pL[q] = pL[q] + 0.5 * gL[q] * dpL;
      pR[q] = pR[q] - 0.5 * gR[q] * dpR;
    }
  }
  const double w = d.w_ann[a];
  T F[5];
  double qL[DGPU_MAX_PASSIVE], qR[DGPU_MAX_PASSIVE], Fq[DGPU_MAX_PASSIVE];
  const int np = PS ? P.num_n : 0;
  for (int s = 0; s < np; ++s) {
    qL[s] = ld(d.prim, 5 + s, QS, cL) + 0.5 * ld(d.gradp, 5 + s, QS, cL) * dpL;
    qR[s] = ld(d.prim, 5 + s, QS, cR) - 0.5 * ld(d.gradp, 5 + s, QS, cR) * dpR;
  }
  riemann_flux<NV>(pL, pR, r, 1, w, P.gamma, P.riemann, F, np, qL, qR, Fq);
  const InstState &S = ist ? *ist : d.ist[A.inst];
  const double k = (substep == 1 ? 1.0 : 0.5) * step_dt(d, S, P, substep) * dA;
#pragma unroll
  for (int q = 0; q < NV; ++q) F[q] = k * F[q];
  stk<NV, T>(d.fphi, tp.fphi, 0, QF, g, F);
  for (int s = 0; s < np; ++s) d.fphi[ix(8 + s, QF, g)] = k * Fq[s];
  if (P.has_visc) {
    ViscIn<T> v;
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cL, v.cL);
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cR, v.cR);
    ldk<4, T>(d.grad, tp.grad, 0, QS, cL, v.grL);
    ldk<4, T>(d.grad, tp.grad, 0, QS, cR, v.grR);
    v.tL = d.tiphw[cL];
    v.tR = d.tiphw[cR];
    v.dpL = v.dpR = 0.0;
    v.r = r;
    v.cm = d.tiphw[cL];
    v.r_cell_L = r;
    v.r_cell_R = r;
    v.rdr_om = frame_val(d, P, A.rdrom, a, DGPU_FR_RDROM);
    GravT<T> G;
    grav_t(G, S, P, tp, A.inst);
    T Fv[3], u[4];
    visc_flux<NV>(v, 1, P, G, Fv, d.err);
#pragma unroll
    for (int q = 0; q < 3; ++q) u[1 + q] = k * Fv[q];
    stk<3, T>(d.fphi, tp.fphi, 5, QF, g, u + 1);
  }
}

template <typename T, int MB = DGPU_MINB_FLUX, bool PS = false, bool V4 = forward_v4<T, PS>>
__global__ void __launch_bounds__(TBLK, MB * (BLK / TBLK)) k_flux_phi(DevPtrs d, TanPtrs tp, int substep) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.n_cells) return;
  if (V4 && no_vz(d)) flux_phi_cell<T, PS, V4 ? 4 : 5>(d, tp, g, nullptr, substep);
  else flux_phi_cell<T, PS>(d, tp, g, nullptr, substep);
}

// r faces: thread per face slot (riemann_setup_rz, Riemann_setup.c:11-44)
template <typename T, bool PS, int NV = 5>
__device__ __forceinline__ void flux_r_face(const DevPtrs &d, const TanPtrs &tp, int slot, const InstState *ist,
                                            int substep) {
  const Pl QS = {PS ? d.qs : 5}, QF = {PS ? d.qf : 8};
  const int cL = d.fL[slot];
  if (cL < 0) return;  // slot past the face list of its pair
  const int cR = d.fR[slot];
  const int a = d.slot_ann[slot];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  const double fdphi = d.fdphi[slot], cm = d.fcm[slot];
  const double deltaL = A.f_dl, deltaR = A.f_dr;
  double dp[2];
  ldk<2, false>(d.fdp, 0, P2, slot, dp);
  const double dpL = dp[0], dpR = dp[1];
  const double r = A.f_r;
  const double dA = r * fdphi * A.f_dperp;
  const double r_cell_L = r - deltaL;
  const double r_cell_R = r + deltaR;
  T pL[5], pR[5];
  {
    T u[5], w[5];
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cL, pL);
    ldk<NV, T>(d.grad, tp.grad, 0, QS, cL, u);
    ldk<NV, T>(d.gradp, tp.gradp, 0, QS, cL, w);
#pragma unroll
    for (int q = 0; q < NV; ++q) pL[q] = pL[q] + u[q] * deltaL + w[q] * dpL;
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cR, pR);
    ldk<NV, T>(d.grad, tp.grad, 0, QS, cR, u);
    ldk<NV, T>(d.gradp, tp.gradp, 0, QS, cR, w);
#pragma unroll
    for (int q = 0; q < NV; ++q) pR[q] = pR[q] - u[q] * deltaR - w[q] * dpR;
  }
  T F[5];
  double qL[DGPU_MAX_PASSIVE], qR[DGPU_MAX_PASSIVE], Fq[DGPU_MAX_PASSIVE];
  const int np = PS ? P.num_n : 0;
  for (int s = 0; s < np; ++s) {
    qL[s] = ld(d.prim, 5 + s, QS, cL) + ld(d.grad, 5 + s, QS, cL) * deltaL + ld(d.gradp, 5 + s, QS, cL) * dpL;
    qR[s] = ld(d.prim, 5 + s, QS, cR) - ld(d.grad, 5 + s, QS, cR) * deltaR - ld(d.gradp, 5 + s, QS, cR) * dpR;
  }
  riemann_flux<NV>(pL, pR, r, 0, 0.0, P.gamma, P.riemann, F, np, qL, qR, Fq);
  const InstState &S = ist ? *ist : d.ist[A.inst];
  const double k = (substep == 1 ? 1.0 : 0.5) * step_dt(d, S, P, substep) * dA;
#pragma unroll
  for (int q = 0; q < NV; ++q) F[q] = k * F[q];
  stk<NV, T>(d.frf, tp.frf, 0, QF, slot, F);
  for (int s = 0; s < np; ++s) d.frf[ix(8 + s, QF, slot)] = k * Fq[s];
  if (P.has_visc) {
    ViscIn<T> v;
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cL, v.cL);
    ldk<NV, T>(d.prim, tp.prim, 0, QS, cR, v.cR);
    ldk<NV, T>(d.gradp, tp.gradp, 0, QS, cL, v.gpL);
    ldk<NV, T>(d.gradp, tp.gradp, 0, QS, cR, v.gpR);
    v.tL = d.tiphw[cL];
    v.tR = d.tiphw[cR];
    v.dpL = dpL;
    v.dpR = dpR;
    v.r = r;
    v.cm = cm;
    v.r_cell_L = r_cell_L;
    v.r_cell_R = r_cell_R;
    v.rdr_om = frame_val(d, P, A.f_rdrom, a, DGPU_FR_FRDROM);
    GravT<T> G;
    grav_t(G, S, P, tp, A.inst);
    T Fv[3], u[4];
    visc_flux<NV>(v, 0, P, G, Fv, d.err);
#pragma unroll
    for (int q = 0; q < 3; ++q) u[1 + q] = k * Fv[q];
    stk<3, T>(d.frf, tp.frf, 5, QF, slot, u + 1);
  }
}

template <typename T, int MB = DGPU_MINB_FLUXR, bool PS = false, bool V4 = forward_v4<T, PS>>
__global__ void __launch_bounds__(TBLK, MB * (BLK / TBLK)) k_flux_r(DevPtrs d, TanPtrs tp, int substep) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= d.n_slots) return;
  if (V4 && no_vz(d)) flux_r_face<T, PS, V4 ? 4 : 5>(d, tp, slot, nullptr, substep);
  else flux_r_face<T, PS>(d, tp, slot, nullptr, substep);
}

// ---------------------------------------------------------------------------
// z faces of 3-D disks (face_create with direction 1, cell_plm_rz with
// Z_DIR, the z-face riemann_setup_rz + riemann_AddFlux of
// src/TimeStep/timestep_routines.c:63-71)
// ---------------------------------------------------------------------------
// z-face slope and reconstruction offsets, once per face: as k_rslope, with
// the half heights of the two layers in place of the radial half widths.
__global__ void __launch_bounds__(BLK) k_zslope(DevPtrs d) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= d.n_zslots) return;
  const int cL = rd(d.zfL + slot);
  if (cL < 0) return;  // slot past the face list of its pair
  const int cR = rd(d.zfR + slot);
  const int a = rd(d.zslot_ann + slot);
  const Annulus &A = d.ann[a];
  const double cm = rd(d.zfcm + slot);
  double pL = rd(d.tiphw + cL) - .5 * rd(d.dphi + cL);
  double pR = rd(d.tiphw + cR) - .5 * rd(d.dphi + cR);
  double dpL = cm - pL;
  dpL = wrap_pm(dpL, d.err);
  double dpR = pR - cm;
  dpR = wrap_pm(dpR, d.err);
  const double dp[2] = {dpL, dpR};
  stk<2>(d.zfdp, 0, P2, slot, dp);
  const double den = A.zf_dr + A.zf_dl;
  const Pl QS = {d.qs};
  double wL[5], wR[5], gL[5], gR[5];
  ldk<5, true>(d.prim, 0, QS, cL, wL);
  ldk<5, true>(d.prim, 0, QS, cR, wR);
  ldk<5, true>(d.gradp, 0, QS, cL, gL);
  ldk<5, true>(d.gradp, 0, QS, cR, gR);
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const double WL = wL[q] + dpL * gL[q];
    const double WR = wR[q] - dpR * gR[q];
    wL[q] = (WR - WL) / den;
  }
  stk<5>(d.zfS, 0, P5, slot, wL);
}

// cell_plm_rz's limiter of plane q with Z_DIR as the reference runs it, from
// the mean that gradz holds to the limited slope in its place (see limit_seq).
__device__ __noinline__ void limit_seq_z(const DevPtrs &d, int g, int q) {
  const int a = d.cell_ann[g];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  double gq = ld(d.gradz, q, P5, g);
  for_cell_zface_ranges(d, A, a, g, P.NR, P.NZ, [&](int s, int e, int) {
    for (int n = s; n < e; ++n) {
      const double S = ld(d.zfS, q, P5, n);
      if (S * gq < 0.0) gq = 0.0;
      else if (fabs(P.plm * S) < fabs(gq)) gq = P.plm * S;
    }
  });
  d.gradz[ix(q, P5, g)] = gq;
}

// cell_plm_rz with Z_DIR (src/Cell/cell_plm.c:13-114) per cell of a 3-D disk:
// the face-area-weighted mean of the z-face slopes over
// dAtot = 2*.5*(rp^2 - rm^2)*dphi, then the limiter, in one walk over the
// cell's faces as plm_r_grad (15.4 -> 11.3 us for torus.par's 139,440 cells).
// The reference overwrites grad with it; here it goes to gradz, which the z
// fluxes and (in 3-D) the viscous source read.
__global__ void __launch_bounds__(BLK) k_plm_z(const __grid_constant__ DevPtrs d) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.n_cells) return;
  const int a = d.cell_ann[g];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  if (P.NZ == 1) return;
  const double rm = A.rm, rp = A.rp, plm = P.plm;
  const double zr = .5 * (rp + rm), zperp = rp - rm;  // build_jloop's r and deltaPerp of a z face
  double gq[5], lim[5];
  int neg = plm < 0.0 ? 31 : 0, pos = neg;  // (a negative PLM: always the loop)
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    gq[q] = 0.0;
    lim[q] = HUGE_VAL;
  }
  for_cell_zface_ranges(d, A, a, g, P.NR, P.NZ, [&](int s, int e, int) {
    for (int n = s; n < e; ++n) {
      const double dA = zr * rd(d.zfdphi + n) * zperp;
      double S[5];
      ldk<5, true>(d.zfS, 0, P5, n, S);
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        gq[q] += S[q] * dA;
        const double ps = plm * S[q];
        if (fabs(ps) < fabs(lim[q])) lim[q] = ps;
        neg |= (S[q] < 0.0) << q;
        pos |= (S[q] > 0.0) << q;
      }
    }
  });
  const double dp = d.dphi[g];
  const double dAtot = 2. * .5 * (rp * rp - rm * rm) * dp;
  const double floor = limit_floor(plm);
  int seq = 0;  // planes that run the loop itself
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    double m = gq[q] / dAtot;
    const bool opposed = (m < 0.0 && (pos >> q & 1)) || (m > 0.0 && (neg >> q & 1));
    seq |= limit_left(m, lim[q], opposed, floor) << q;
    gq[q] = m;
  }
  stk<5>(d.gradz, 0, P5, g, gq);
  for (; seq; seq &= seq - 1) limit_seq_z(d, g, __ffs(seq) - 1);
}

// z faces: thread per face slot (riemann_setup_rz with ZDIRECTION,
// Riemann_setup.c:11-44, and riemann_AddFlux with w = 0): the states are
// reconstructed with the z slopes; the viscous flux of a z face is zero, and
// only the reference's v_z check remains.
__global__ void __launch_bounds__(BLK) k_flux_z(DevPtrs d, int substep) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= d.n_zslots) return;
  const int cL = d.zfL[slot];
  if (cL < 0) return;
  const int cR = d.zfR[slot];
  const int a = d.zslot_ann[slot];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  const InstState &S = d.ist[A.inst];
  const double fac = substep == 1 ? 1.0 : 0.5;
  const double deltaL = A.zf_dl, deltaR = A.zf_dr;
  double dp[2];
  ldk<2, true>(d.zfdp, 0, P2, slot, dp);
  const double dpL = dp[0], dpR = dp[1];
  const double r = A.zf_r;
  const double dA = r * d.zfdphi[slot] * A.zf_dperp;
  double pL[5], pR[5], F[5];
  {
    const Pl QS = {d.qs};
    double u[5], w[5];
    ldk<5, true>(d.prim, 0, QS, cL, pL);
    ldk<5, true>(d.gradz, 0, P5, cL, u);
    ldk<5, true>(d.gradp, 0, QS, cL, w);
#pragma unroll
    for (int q = 0; q < 5; ++q) pL[q] = pL[q] + u[q] * deltaL + w[q] * dpL;
    ldk<5, true>(d.prim, 0, QS, cR, pR);
    ldk<5, true>(d.gradz, 0, P5, cR, u);
    ldk<5, true>(d.gradp, 0, QS, cR, w);
#pragma unroll
    for (int q = 0; q < 5; ++q) pR[q] = pR[q] - u[q] * deltaR - w[q] * dpR;
  }
  riemann_flux(pL, pR, r, 2, 0.0, P.gamma, P.riemann, F);
  const double k = fac * step_dt(d, S, P, substep) * dA;
#pragma unroll
  for (int q = 0; q < 5; ++q) F[q] = k * F[q];
  stk<5>(d.zfrf, 0, P5, slot, F);
  if (P.has_visc) {
    // riemann_visc_flux averages the reconstructed states on a z face and
    // exits on a nonzero v_z (Riemann_routines.c:271-274)
    const double vz = .5 * (pL[D_UZZ] + pR[D_UZZ]);
    if (fabs(vz) > 1.e-12) set_err(d.err, DGPU_EF_VISC_VZ);
  }
}

// The single-rank cell_syncproc_z (src/Cell/cell_sync.c:156-205) at the end
// of a substep of a 3-D disk, then cell_calc_cons of the cells it wrote: the
// ng lowest layers take prim, RKcons and tiph of layers NZ-2ng .. NZ-ng-1, the
// ng highest those of layers ng .. 2ng-1 (dphi stays the cell's own).  Runs
// after k_update and the radial boundary, which have finished every layer.
__global__ void __launch_bounds__(BLK) k_zsync(DevPtrs d, int substep) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = d.n_cells, zg = d.zghost;
  // zghost > 0: threads cover the ng lowest layers' cells, then the ng highest
  const int g = zg > 0 ? (t < zg ? t : N - 2 * zg + t) : t;
  if (zg > 0 ? t >= 2 * zg : g >= N) return;
  const int a = d.cell_ann[g];
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  if (P.NZ == 1) return;
  const int ng = P.ngz, shift = P.NZ - 2 * ng;
  int ks;
  if (A.k < ng) ks = A.k + shift;
  else if (A.k >= P.NZ - ng) ks = A.k - shift;
  else return;
  const Annulus &Sr = d.ann[a + (ks - A.k) * P.NR];
  const int gs = Sr.cell_off + (g - A.cell_off);
  double *tout = substep == 1 ? d.tiph1 : d.tiph0;
  const Pl QS = {d.qs};  // (a 3-D disk itself carries no passive scalars)
  double pr[5], c[5];
  ldk<5, false>(d.prim, 0, QS, gs, pr);
  stk<5>(d.prim, 0, QS, g, pr);
  ldk<5, false>(d.rkcons, 0, QS, gs, c);
  stk<5>(d.rkcons, 0, QS, g, c);
  tout[g] = tout[gs];
  const double r = .5 * (A.rm + A.rp);
  const double dV = A.dv_half * d.dphi[g] * A.dz;
  prim2cons(pr, c, r, dV, P.gamma);
  stk<5>(d.cons, 0, QS, g, c);
}

// ---------------------------------------------------------------------------
// Per-cell update: flux gather + sources + mesh motion + prim/cons + BC + damping
// ---------------------------------------------------------------------------

// Source increments of cell_add_src (src/Cell/cell_source.c:73-214) and
// cell_add_visc_src (cell_source.c:216-277), per cell, for k_update to add in
// the reference's order: src[0..4] = S_r (pressure/centrifugal), S_r (gravity
// + frame), L, S_z, tau; src[5] = viscous heating; src[6+p] = sink mass of mass
// p.  They read only the substep's primitives, slopes and GravMass positions,
// so this kernel runs concurrently with k_flux_r.  Its first n_ann threads also
// form the per-annulus constants of the substep (epicyclic rotation of
// cell_add_split_fictitious.c:26-38, relaxation factor of cell_misc.c:121).
// Per-annulus constants of the substep for the update of annulus t: the
// epicyclic rotation of cell_add_split_fictitious
// (cell_add_split_fictitious.c:26-38) and the relaxation factor of
// cell_bc_damp (cell_misc.c:121), identical for every cell of the annulus.
__device__ __forceinline__ void ann_consts(const DevPtrs &d, int t, const InstState &S, double dt) {
  const Annulus &A = d.ann[t];
  const DiskParams &P = d.par[A.inst];
  const double r = 0.5 * (A.rm + A.rp);
  const double rom = frame_val(d, P, A.rom, t, DGPU_FR_ROM);
  const double Omega = rom / r;
  const double dr_r2Om = 2. * rom + r * frame_val(d, P, A.rdrom, t, DGPU_FR_RDROM);
  const double kappa2 = 2. * Omega / r * dr_r2Om;
  double kappa = 0.0, ck = 1.0, sk = 0.0;
  if (kappa2 > 0.) {
    kappa = sqrt(kappa2);
    ck = cos(kappa * dt);
    sk = sin(kappa * dt);
  }
  const int NA = d.n_ann;
  d.ann_c[t] = kappa;
  d.ann_c[NA + t] = ck;
  d.ann_c[2 * NA + t] = sk;
  d.ann_c[3 * NA + t] = (A.kind & DGPU_AK_DAMP) ? (1. - exp(-A.damp_rate * dt)) : 0.0;
}

// The source increments of cell g (see k_source); the sink masses of the
// cells counted in Mdot are added to md0 / md1.
template <typename T, bool PS, int NV = 5>
__device__ __forceinline__ void source_cell_k(const DevPtrs &d, const TanPtrs &tp, int g, const InstState &S,
                                              double dt, double &md0, double &md1) {
  const Pl QS = {PS ? d.qs : 5};
  {
    pf_planes(d.prim, NV, QS, g);
    pf(d.grad + ix(D_UPP, QS, g));
    pf(d.gradp + ix(D_URR, QS, g));
    pf(d.tiphw + g);
    pf(d.dphi + g);
    const int a = d.cell_ann[g];
    const Annulus &A = d.ann[a];
    const DiskParams &P = d.par[A.inst];
    const double dphi = d.dphi[g];
    const double rm = A.rm, rp = A.rp;
    double phi = d.tiphw[g] - .5 * dphi;
    double r = .5 * (rp + rm);
    T pm[5];
    ldk<NV, T>(d.prim, tp.prim, 0, QS, g, pm);
    SrcGeom sg;
    sg.r = r;
    sg.dt = dt;
    sg.dV = dphi * .5 * A.dv_diff * A.dz;
    sincos(phi, &sg.sinp, &sg.cosp);
    sg.xpos = r * sg.cosp;
    sg.ypos = r * sg.sinp;
    {
      double z = A.z;
      double R = sqrt(r * r + z * z);
      if (P.grav2d == 1) {
        sg.sint = 1.0;
        sg.cost = 0.0;
        sg.gravdist = r;
      } else {
        sg.sint = r / R;
        sg.cost = z / R;
        sg.gravdist = R;
      }
    }
    double w_a = frame_val(d, P, A.rom, a, DGPU_FR_ROM);
    sg.rdrOm = frame_val(d, P, A.rdrom, a, DGPU_FR_RDROM);
    sg.Fc = w_a * w_a / r;
    sg.dtOm = frame_val(d, P, A.dtom, a, DGPU_FR_DTOM);
    GravT<T> G;
    grav_t(G, S, P, tp, A.inst);
    T gu = 0.0, gpu = 0.0;
    if (P.has_visc) {
      // in 3-D cell_plm_rz(Z_DIR) has overwritten grad with the z slopes by the
      // time cell_add_visc_src reads it (timestep_routines.c:63-81)
      gu = (d.has_z && P.NZ > 1) ? T(ld(d.gradz, D_UPP, P5, g)) : ldq<T>(d.grad, tp.grad, D_UPP, QS, g);
      gpu = ldq<T>(d.gradp, tp.gradp, D_URR, QS, g);
    }
    T sv[6];
    source_cell<NV>(sg, P, pm, gu, gpu, G, sv);
    stk<3, T>(d.src, tp.src, 0, P8, g, sv);
    if constexpr (NV == 5) stq<T>(d.src, tp.src, 3, P8, g, sv[3]);
    stk<2, T>(d.src, tp.src, 4, P8, g, sv + 4);
    const double xpos = sg.xpos, ypos = sg.ypos, dV = sg.dV;
    const T rho = pm[D_RHO], Pp = pm[D_PPP];
    if (P.rho_sink_on == 1) {
      // get_rho_sink (src/Cell/cell_source.c:15-47); no tangent (refused by the
      // differentiated runs)
      const double rhov = val(rho), Pv = val(Pp);
      double r0 = sqrt((xpos - S.gx[0]) * (xpos - S.gx[0]) + (ypos - S.gy[0]) * (ypos - S.gy[0]));
      double r1 = sqrt((xpos - S.gx[1]) * (xpos - S.gx[1]) + (ypos - S.gy[1]) * (ypos - S.gy[1]));
      double M0 = S.gM[0], M1 = S.gM[1];
      double Mtotal = M0 + M1;
      double alpha = P.visc;
      double one_o_nu = 1.0 / (alpha * Pv / rhov) * sqrt(pow(r0, -3) * M0 / Mtotal + pow(r1, -3) * M1 / Mtotal);
      double t_visc0 = 1.0 * 2. / 3. * r0 * r0 * one_o_nu;
      double t_visc1 = 1.0 * 2. / 3. * r1 * r1 * one_o_nu;
      if (t_visc0 < 10. * dt) t_visc0 = 10. * dt;
      if (t_visc1 < 10. * dt) t_visc1 = 10. * dt;
      double sink_size = 0.5;
      for (int p = 0; p < P.num_sinks && p < 2; ++p) {
        double drho = 0.0;
        if (p == 0) { if (r0 < sink_size) drho = rhov / t_visc0; }
        else { if (r1 < sink_size) drho = rhov / t_visc1; }
        stq<T>(d.src, tp.src, 6 + p, P8, g, T(drho * dt * dV));
        if (A.kind & DGPU_AK_SINK_SUM) {
          if (p == 0) md0 += drho * dV;
          else md1 += drho * dV;
        }
      }
    }
  }
}

// The place in mdot_part of disk k's sink sums over the cells of block b: one
// apart from block to block and from disk to disk, so no two of them share one
// (at most n_inst more than there are blocks).
__device__ __forceinline__ size_t mdot_slot(int b, int k) { return (size_t)b + (size_t)k; }

template <typename T, int MB = DGPU_MINB_SOURCE, bool PS = false, bool V4 = forward_v4<T, PS>>
__global__ void __launch_bounds__(BLK, MB) k_source(DevPtrs d, TanPtrs tp, int substep, int cells) {
  __shared__ double sh_md[2][BLK / 32];
  __shared__ int sh_k[2];  // the first and the last cell's disk
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int N = d.n_cells;
  const double fac = substep == 1 ? 1.0 : 0.5;
  if (t < d.n_ann) {
    const int inst = d.ann[t].inst;
    const InstState &S = d.ist[inst];
    ann_consts(d, t, S, fac * step_dt(d, S, d.par[inst], substep));
  }
  double md0 = 0.0, md1 = 0.0;
  int inst = 0;
  if (t < N && cells) {
    inst = d.ann[d.cell_ann[t]].inst;
    const InstState &S = d.ist[inst];
    const double dt = fac * step_dt(d, S, d.par[inst], substep);
    if (V4 && no_vz(d)) source_cell_k<T, PS, V4 ? 4 : 5>(d, tp, t, S, dt, md0, md1);
    else source_cell_k<T, PS>(d, tp, t, S, dt, md0, md1);
  }
  // deterministic Mdot partial sums, one per block and disk in it (mdot_slot;
  // reduced in block order by k_update).  The sums over the whole block first,
  // which are the disk's where the block holds one; else disk after disk.
  auto partial = [&](double m0, double m1) {
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      m0 += __shfl_down_sync(full, m0, o);
      m1 += __shfl_down_sync(full, m1, o);
    }
    if ((threadIdx.x & 31) == 0) {
      sh_md[0][threadIdx.x >> 5] = m0;
      sh_md[1][threadIdx.x >> 5] = m1;
    }
    __syncthreads();
  };
  auto store = [&](int k) {
    if (threadIdx.x == 0) {
      double s0 = 0.0, s1 = 0.0;
      for (int w = 0; w < BLK / 32; ++w) {
        s0 += sh_md[0][w];
        s1 += sh_md[1][w];
      }
      double *p = d.mdot_part + 2 * mdot_slot(blockIdx.x, k);
      p[0] = s0;
      p[1] = s1;
    }
  };
  if ((size_t)blockIdx.x * BLK >= (size_t)N) return;
  if (threadIdx.x == 0) sh_k[0] = inst;
  if (t == min((int)(blockIdx.x + 1) * BLK, N) - 1) sh_k[1] = inst;
  partial(md0, md1);
  const int k0 = sh_k[0], k1 = sh_k[1];
  if (k0 == k1) {
    store(k0);
    return;
  }
  for (int k = k0; k <= k1; ++k) {
    __syncthreads();
    const bool mine = t < N && inst == k;
    partial(mine ? md0 : 0.0, mine ? md1 : 0.0);
    store(k);
  }
}

// The update of cell g after its face and source increments are in place:
// the conserved sum in the reference's order (update_sum),
// cell_update_phi/_dphi, cell_calc_prim, the fixed radial boundary,
// cell_bc_damp and cell_calc_cons.  ist: the disk's state (NULL: d.ist).  XC: the
// increments were written by other blocks of the running kernel (plain loads,
// not the read-only path).  rec (the adjoint's segment replay, else NULL): the
// conserved sum before cons2prim and the new width of each cell go to slot
// 2 * (*rec_idx) + substep - 1 of rec (per slot 6 planes over n_pad cells).
template <typename T, bool PS, bool XC = false, int NV = 5>
__device__ __forceinline__ void update_cell(const DevPtrs &d, const TanPtrs &tp, int g, int substep, int stop,
                                            const InstState *ist, double *rec, const int *rec_idx) {
  const Pl QS = {PS ? d.qs : 5}, QF = {PS ? d.qf : 8};
  {
    // the cell's own planes, before the annulus lookups they do not depend on
    pf_planes(d.cons, NV, QS, g);
    if (substep == 2) {
      pf_planes(d.rkcons, NV, QS, g);
      pf(d.rktiph + g);
    }
    pf_planes(d.fphi, 8, QF, g);
    pf_planes(d.src, 6, P8, g);
    pf(d.tiphw + g);
    pf((substep == 1 ? d.tiph0 : d.tiph1) + g);
    // and its r-face run ranges and first face, which k_merge just wrote
    pf(d.rr + 4 * (size_t)g);
    pf(d.fstart + g);
    const int a = d.cell_ann[g];
    const Annulus &A = d.ann[a];
    const DiskParams &P = d.par[A.inst];
    const double dt = (substep == 1 ? 1.0 : 0.5) * step_dt(d, ist ? *ist : d.ist[A.inst], P, substep);
    T c[5];
    double cp[DGPU_MAX_PASSIVE], pp[DGPU_MAX_PASSIVE];
    const int np = PS ? P.num_n : 0;
    if (np > 0) passive_sum(d, A, a, g, substep, stop, np, cp);
    if (!update_sum<T, !XC, PS, NV>(d, tp, A, a, g, substep, stop, dt, true, c)) {
      stk<NV, T>(d.cons, tp.cons, 0, QS, g, c);
      for (int k = 0; k < np; ++k) d.cons[ix(5 + k, QS, g)] = cp[k];
    } else {
      double tn, rk;
      const double dphi_n = mesh_advance(d, A, a, g, substep, dt, tn, rk);
      if (substep == 1) d.rktiph[g] = rk;
      (substep == 1 ? d.tiph1 : d.tiph0)[g] = tn;
      d.dphi[g] = dphi_n;
      if (rec) {
        double *rs = rec + (size_t)(2 * (*rec_idx) + substep - 1) * 6 * d.n_pad;
        double u[6];
        u[D_SZZ] = 0.0;
#pragma unroll
        for (int q = 0; q < NV; ++q) u[q] = val(c[q]);
        u[5] = dphi_n;
        stk<6>(rs, 0, P6, g, u);
      }
      // cell_calc_prim -> cell_cons2prim (src/Cell/cell_conversion.c:57-122)
      const double r = .5 * (A.rm + A.rp);
      const double dV = A.dv_half * dphi_n * A.dz;
      T pr[5];
      cons2prim<NV>(c, dV, r, P, pr);
      // v_z of a cell without the v_z planes that is not finite (nan_vz); the
      // annuli that the outflow boundary rewrites take it from obuf
      if (NV == 4 && nan_vz(val(c[D_DDD]), val(c[D_SRR])) && !(A.kind & DGPU_AK_OUT_DST))
        d.prim[ix(D_UZZ, QS, g)] = d.cons[ix(D_SZZ, QS, g)] =
            (A.kind & DGPU_AK_BC_FIXED) && (A.kind & DGPU_AK_IC) ? 0.0 : NAN;
      // passive scalars: prim = cons / cons[DDD] (cell_conversion.c:98-101)
      for (int k = 0; k < np; ++k) pp[k] = cp[k] / val(c[D_DDD]);
      // the outflow boundary reads these prims before any damping; the
      // annuli it rewrites are damped and converted by k_outflow
      if (A.ob_off >= 0 && stop >= 6) {
#pragma unroll
        for (int q = 0; q < 5; ++q)
          d.obuf[(size_t)q * d.n_ob + A.ob_off + (g - A.cell_off)] =
              q < NV ? val(pr[q]) : nan_vz(val(c[D_DDD]), val(c[D_SRR])) ? NAN : 0.0;
        for (int k = 0; k < np; ++k) d.obuf[(size_t)(5 + k) * d.n_ob + A.ob_off + (g - A.cell_off)] = pp[k];
      }
      const bool own = !(A.kind & DGPU_AK_OUT_DST);
      if (stop >= 6 && own) {
        bc_damp<NV>(d, A, a, pr);
        // cell_single_init_vortex's dye at the cell's new phi, in the fixed
        // boundary (cell_init_vortex.c:22-35); no other family sets one
        if (np > 0 && P.init_type == DI_VORTEX && (A.kind & DGPU_AK_BC_FIXED) && (A.kind & DGPU_AK_IC))
          pp[0] = cos(tn - .5 * dphi_n) < 0.0 ? 0.0 : 1.0;
      }
      // cell_calc_cons (src/Cell/cell_conversion.c:35-55)
      if (stop >= 7 && own) {
        prim2cons<NV>(pr, c, r, dV, P.gamma);
        for (int k = 0; k < np; ++k) cp[k] = pp[k] * val(c[D_DDD]);
      }
      stk<NV, T>(d.prim, tp.prim, 0, QS, g, pr);
      stk<NV, T>(d.cons, tp.cons, 0, QS, g, c);
      for (int k = 0; k < np; ++k) {
        d.prim[ix(5 + k, QS, g)] = pp[k];
        d.cons[ix(5 + k, QS, g)] = cp[k];
      }
    }
  }
}

// GravMass after the substep for disk k: gravMass_update_RK
// (GravMass_misc.c:66-77), then gravMass_move(t, fac*dt) (GravMass_misc.c:31-64);
// after substep 2 also t += dt and Macc += Mdot*dt (timestep_algorithm.c:27-39).
// S.gphi holds the substep's wrapped phases (gravMass_clean_pi) and S.mdot
// the substep's sink rates.
__device__ __forceinline__ void gm_tail(const DevPtrs &d, InstState &S, const DiskParams &P, int substep,
                                        int tail) {
  const double RK = substep == 1 ? 0.0 : 0.5;
  const double fac = substep == 1 ? 1.0 : 0.5;
  for (int p = 0; p < 2; ++p) {
    S.grk_phi[p] = adjust_toward(S.gphi[p], S.grk_phi[p], M_PI, 2. * M_PI, d.err);
    S.gr[p] = (1.0 - RK) * S.gr[p] + RK * S.grk_r[p];
    S.gphi[p] = (1.0 - RK) * S.gphi[p] + RK * S.grk_phi[p];
    S.gM[p] = (1.0 - RK) * S.gM[p] + RK * S.grk_M[p];
    S.gom[p] = (1.0 - RK) * S.gom[p] + RK * S.grk_om[p];
  }
  if (tail >= 2) {
    double t = S.t, dtm = fac * S.dt;
    double m0 = S.gM[0], m1 = S.gM[1];
    double M = m0 + m1;
    double a_0 = 1.0, tau_0 = P.orb_tscale, T0 = P.orb_t0;
    double asep, omega;
    if ((t - T0) / tau_0 < 1.) {
      asep = a_0 * pow((1.0 - (t - T0) / tau_0), 0.25);
      omega = pow(asep / M, -1.5);
    } else {
      asep = 0.0;
      omega = 0.0;
    }
    double r0, r1;
    if (M < 1.e-12) {
      r0 = 0.0;
      r1 = 0.0;
    } else {
      r0 = m1 / M * asep;
      r1 = m0 / M * asep;
    }
    S.gphi[0] += omega * dtm;
    S.gphi[1] += omega * dtm;
    S.gr[0] = r0;
    S.gr[1] = r1;
    S.gom[0] = omega;
    S.gom[1] = omega;
    if (substep == 2) {
      S.t += S.dt;
      for (int p = 0; p < 2; ++p) S.macc[p] = S.macc[p] + S.mdot[p] * S.dt;
    }
  }
}

// Every block updates cells; with tail > 0 block 0 moves the GravMass of every
// disk instead, while the others work: no cell of this kernel reads what it
// writes.  (A last block elected by a counter did it after all the others, a
// chain of two pow at the end of every substep.)
template <typename T, int MB = DGPU_MINB_UPDATE, bool PS = false, bool V4 = forward_v4<T, PS>>
__global__ void __launch_bounds__(TBLK, MB * (BLK / TBLK)) k_update(DevPtrs d, TanPtrs tp, int substep, int stop,
                                                                  int tail, double *rec, const int *rec_idx) {
  int b = blockIdx.x;
  if (tail > 0 && b-- == 0) {
    if (threadIdx.x == 0) d.counters[DGPU_CT_NO_VZ] = V4 && no_vz(d);
    for (int k = threadIdx.x; k < d.n_inst; k += blockDim.x) {
      InstState &S = d.ist[k];
      const DiskParams &P = d.par[k];
      if (substep == 1 && d.form_dt) S.dt = cfl_dt(S, P);
      // Mdot of this disk: its partials in block order
      const int c0 = P.cell_base, c1 = P.cell_base + P.n_cells;
      const int b0 = c0 / BLK, b1 = (c1 + BLK - 1) / BLK;
      double s0 = 0.0, s1 = 0.0;
      if (P.rho_sink_on == 1) {
        for (int m = b0; m < b1; ++m) {
          s0 += d.mdot_part[2 * mdot_slot(m, k)];
          s1 += d.mdot_part[2 * mdot_slot(m, k) + 1];
        }
      }
      S.mdot[0] = s0;
      S.mdot[1] = s1;
      gm_tail(d, S, P, substep, tail);
    }
    return;
  }
  const int g = b * TBLK + threadIdx.x;
  if (g >= d.n_cells) return;
  if (V4 && no_vz(d)) update_cell<T, PS, false, V4 ? 4 : 5>(d, tp, g, substep, stop, nullptr, rec, rec_idx);
  else update_cell<T, PS>(d, tp, g, substep, stop, nullptr, rec, rec_idx);
}

// ---------------------------------------------------------------------------
// The fused substep: k_prep then k_sweep
// ---------------------------------------------------------------------------
// k_prep: one block per annulus a of every disk.  The face list of pair
// (a, a+1) and cell_set_w (merge_pair), cell_clean_pi and cell_plm_p of the
// annulus's cells and, in substep 1, gravMass_copy and the annulus's CFL
// minimum (cell_mindt, src/Cell/cell_mindt.c:10-100), from which every block of
// k_sweep forms the disk's dt (timestep_set_dt).  It also clears the sweep's
// progress flags and work counters.
template <int MB>
__global__ void __launch_bounds__(BLK, MB) k_prep(DevPtrs d, int substep) {
  __shared__ unsigned long long sh_k[BLK / 32];
  __shared__ double sh_rk[6], sh_ring[2][RING_CHUNK];
  const int a = blockIdx.x;
  const TanPtrs tp = {};
  merge_pair<false>(d, a, substep);
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  if (P.w_numeric == DC_RIGID && threadIdx.x >= BLK - 32) ring_mean(d, a, threadIdx.x & 31, sh_ring);
  __syncthreads();  // w_ann[a] (one lane) before the CFL
  for (int j = threadIdx.x; j < A.np; j += BLK) cellprep_cell<double, false>(d, tp, A.cell_off + j, substep);
  if (threadIdx.x == 0) {
    d.sweep_flag[a] = 0;
    if (a == 0) {
      d.counters[3] = 0;
      d.counters[4] = 0;
      d.counters[DGPU_CT_NO_VZ] = 0;
    }
  }
  if (substep != 1) return;
  if (threadIdx.x == 0) {
    InstState &S = d.ist[A.inst];
    // gravMass_dist of the step-start positions, for the CFL's viscosity
    for (int p = 0; p < 2; ++p) {
      sh_rk[p] = S.gr[p] * cos(S.gphi[p]);
      sh_rk[2 + p] = S.gr[p] * sin(S.gphi[p]);
      sh_rk[4 + p] = S.gM[p];
    }
    if (A.i == 0) {
      // gravMass_copy (GravMass_misc.c:20-28); no block of this kernel reads
      // these copies
      for (int p = 0; p < 2; ++p) {
        S.grk_r[p] = S.gr[p];
        S.grk_phi[p] = S.gphi[p];
        S.grk_M[p] = S.gM[p];
        S.grk_om[p] = S.gom[p];
      }
    }
  }
  __syncthreads();
  unsigned long long key = ~0ull;
  if (A.kind & DGPU_AK_CFL) {
    const double wa = d.w_ann[a];
    for (int j = threadIdx.x; j < A.np; j += BLK) {
      const unsigned long long k = cfl_key(d, A, P, A.cell_off + j, wa, sh_rk, sh_rk + 2, sh_rk + 4);
      key = k < key ? k : key;
    }
  }
  const unsigned full = 0xffffffffu;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long k2 = __shfl_down_sync(full, key, o);
    key = k2 < key ? k2 : key;
  }
  if ((threadIdx.x & 31) == 0) sh_k[threadIdx.x >> 5] = key;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < BLK / 32; ++w) key = sh_k[w] < key ? sh_k[w] : key;
    d.cfl_ann[a] = key;
  }
}

// dt of a disk from k_prep's per-annulus CFL minima: the minimum (1e100 when
// no cell has a candidate), clipped to Time_Max (timestep_set_dt,
// src/TimeStep/timestep_set.c:16-21).  The same value as cfl_dt forms from dtkey.
__device__ __forceinline__ double sweep_dt(const DevPtrs &d, const DiskParams &P, double t) {
  unsigned long long key = (unsigned long long)__double_as_longlong(1.e100);
  for (int k = P.ann_base; k < P.ann_base + P.NR; ++k) {
    const unsigned long long v = d.cfl_ann[k];
    key = v < key ? v : key;
  }
  double dt = __longlong_as_double((long long)key);
  if (t + dt > P.t_max) dt = P.t_max - t;
  return dt;
}

// Progress flags of k_sweep: after a __syncthreads, thread 0 publishes that
// this block's phase v of annulus a is done (its stores ordered before the
// flag), or waits until the block of annulus a has published v (the block's
// later loads ordered after the flag).  A wait gives up after
// DGPU_SWEEP_SPIN_LIMIT polls, reports DGPU_EF_SWEEP_WAIT and returns.
#define DGPU_SWEEP_SPIN_LIMIT (1 << 18)
__device__ __forceinline__ void sweep_publish(const DevPtrs &d, int a, int v) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(d.sweep_flag + a), "r"(v) : "memory");
  }
}
__device__ __forceinline__ void sweep_wait(const DevPtrs &d, int a, int v) {
  if (threadIdx.x == 0) {
    int it = 0, f;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(f) : "l"(d.sweep_flag + a) : "memory");
      if (f >= v) break;
      if (++it > DGPU_SWEEP_SPIN_LIMIT) {
        set_err(d.err, DGPU_EF_SWEEP_WAIT);
        break;
      }
      __nanosleep(100);
    }
  }
  __syncthreads();
}

// The phases of k_sweep for the block's annulus (the block's threads stride
// over the annulus's faces or cells).  Inlined: as separate calls they spill
// more across the call boundaries and run slower (measured).
#define SWEEP_FN __device__ __forceinline__
SWEEP_FN void sweep_slopes(const DevPtrs &d, int a) {
  const TanPtrs tp = {};
  const Annulus &A = d.ann[a];
  const int nf = d.pair_nf[a];
  for (int n = threadIdx.x; n < nf; n += BLK) rslope_face<double, false>(d, tp, A.face_base + n);
}
SWEEP_FN void sweep_grad(const DevPtrs &d, int a) {
  const TanPtrs tp = {};
  const Annulus &A = d.ann[a];
  for (int j = threadIdx.x; j < A.np; j += BLK) plm_r_grad<double, false>(d, tp, A.cell_off + j);
}
SWEEP_FN void sweep_flux_r(const DevPtrs &d, int b, const InstState &S, int substep) {
  const TanPtrs tp = {};
  const Annulus &Q = d.ann[b];
  const int nf = d.pair_nf[b];
  for (int n = threadIdx.x; n < nf; n += BLK) flux_r_face<double, false>(d, tp, Q.face_base + n, &S, substep);
}
SWEEP_FN void sweep_cells(const DevPtrs &d, int a, const InstState &S, int substep, double dt) {
  const TanPtrs tp = {};
  const Annulus &A = d.ann[a];
  double md0 = 0.0, md1 = 0.0;
  for (int j = threadIdx.x; j < A.np; j += BLK) {
    const int g = A.cell_off + j;
    flux_phi_cell<double, false>(d, tp, g, &S, substep);
    source_cell_k<double, false>(d, tp, g, S, dt, md0, md1);
  }
}
SWEEP_FN void sweep_update_cells(const DevPtrs &d, int b, int substep, const InstState &S) {
  const TanPtrs tp = {};
  const Annulus &B = d.ann[b];
  for (int j = threadIdx.x; j < B.np; j += BLK)
    update_cell<double, false, true>(d, tp, B.cell_off + j, substep, 7, &S, nullptr, nullptr);
}

// The update of annulus b's cells (update_cell) once its increments are in
// place, with the annulus's constants of the substep.
__device__ __forceinline__ void sweep_update(const DevPtrs &d, int b, int substep, const InstState &S, double dt) {
  if (threadIdx.x == 0) ann_consts(d, b, S, dt);
  __syncthreads();
  sweep_update_cells(d, b, substep, S);
}

// k_sweep: the rest of the substep as one wavefront over the annuli.  Each
// block takes the next annulus a in order (a work counter, so every earlier
// annulus is held by a block that is already running) and does, waiting only
// on the block of annulus a-1 of the same disk:
//   1. the face slopes S and offsets of the faces of pair (a, a+1) (k_rslope);
//   2. the r slopes of annulus a (cell_plm_rz) -- needs 1. of a-1;
//   3. the fluxes of the faces of pair (a-1, a) (riemann_setup_rz +
//      riemann_AddFlux) -- needs 2. of a-1 -- and the phi faces and source
//      increments of annulus a;
//   4. the update of annulus a-1 (and of a itself when it is the disk's last),
//      whose increments are then all in place -- needs 3. of a-1.
// A block never waits for a later annulus, so the wavefront always advances.
// The last block to finish advances the GravMass state (gm_tail).  The
// increments pass between neighbouring annuli through L2 instead of HBM round
// trips between eight kernels, and phases of different annuli overlap on the
// SMs.
template <int MB>
__global__ void __launch_bounds__(BLK, MB) k_sweep(const __grid_constant__ DevPtrs d, int substep) {
  __shared__ int s_a;
  __shared__ InstState s_S;
  __shared__ bool s_last;
  if (threadIdx.x == 0) s_a = (int)atomicAdd(&d.counters[3], 1u);
  __syncthreads();
  const int a = s_a;
  const Annulus &A = d.ann[a];
  const DiskParams &P = d.par[A.inst];
  if (threadIdx.x == 0) {
    // the disk's state with the substep's GravMass positions (gravMass_clean_pi,
    // then gravMass_dist's r cos(phi), r sin(phi)) and, in substep 1, its dt
    s_S = d.ist[A.inst];
    for (int p = 0; p < 2; ++p) {
      const double ph = wrap_pos(s_S.gphi[p], d.err);
      s_S.gphi[p] = ph;
      s_S.gc[p] = cos(ph);
      s_S.gs[p] = sin(ph);
      s_S.gx[p] = s_S.gr[p] * s_S.gc[p];
      s_S.gy[p] = s_S.gr[p] * s_S.gs[p];
    }
    if (substep == 1) s_S.dt = sweep_dt(d, P, s_S.t);
  }
  __syncthreads();
  const double dt = (substep == 1 ? 1.0 : 0.5) * s_S.dt;
  const int first = A.i == 0, last = A.i == P.NR - 1;
  // 1. face slopes of pair (a, a+1)
  if (!last) sweep_slopes(d, a);
  sweep_publish(d, a, 1);
  // 2. r slopes of annulus a
  if (!first) sweep_wait(d, a - 1, 1);
  sweep_grad(d, a);
  sweep_publish(d, a, 2);
  // 3. fluxes of pair (a-1, a); phi faces and sources of annulus a
  if (!first) {
    sweep_wait(d, a - 1, 2);
    sweep_flux_r(d, a - 1, s_S, substep);
  }
  sweep_cells(d, a, s_S, substep, dt);
  sweep_publish(d, a, 3);
  // 4. update of annulus a-1, then of the disk's last annulus
  if (!first) {
    sweep_wait(d, a - 1, 3);
    sweep_update(d, a - 1, substep, s_S, dt);
  }
  if (last) {
    __syncthreads();
    sweep_update(d, a, substep, s_S, dt);
  }
  // the last block: the GravMass of every disk.  It reads nothing that
  // another block of this kernel writes.
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&d.counters[4], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  for (int k = threadIdx.x; k < d.n_inst; k += BLK) {
    InstState &S = d.ist[k];
    const DiskParams &Pk = d.par[k];
    if (substep == 1) S.dt = sweep_dt(d, Pk, S.t);
    for (int p = 0; p < 2; ++p) S.gphi[p] = wrap_pos(S.gphi[p], d.err);
    S.mdot[0] = 0.0;  // no sink on this path
    S.mdot[1] = 0.0;
    gm_tail(d, S, Pk, substep, 2);
  }
  if (threadIdx.x == 0) {
    d.counters[3] = 0;
    d.counters[4] = 0;
  }
}

// cell_calc_cons over all cells (set-up and state upload)
template <typename T, bool PS = false>
__global__ void __launch_bounds__(BLK) k_calc_cons(DevPtrs d, TanPtrs tp) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  const Pl QS = {PS ? d.qs : 5};
  if (g >= d.n_cells) return;
  const Annulus &A = d.ann[d.cell_ann[g]];
  const DiskParams &P = d.par[A.inst];
  double r = .5 * (A.rp + A.rm);
  double dV = A.dv_half * d.dphi[g] * A.dz;
  T p[5], c[5];
  ldk<5, T>(d.prim, tp.prim, 0, QS, g, p);
  prim2cons(p, c, r, dV, P.gamma);
  stk<5, T>(d.cons, tp.cons, 0, QS, g, c);
  for (int q = 5; q < 5 + (PS ? P.num_n : 0); ++q) d.cons[ix(q, QS, g)] = ld(d.prim, q, QS, g) * val(c[D_DDD]);
}

// cell_boundary_outflow_r (src/Cell/cell_boundary.c:14-139) runs three passes
// over the substep's r faces, each reading the one before: annulus 0 from
// annulus 1 (unless NoInnerBC == 1), NR-2 from NR-3, NR-1 from the new NR-2.
// A pass gives every cell the sum, in face order, of prim * dA of the cells
// across its faces, divided by dz * FacePos(i) * dphi.  The reference's build
// constants EXTRAP_BC, SS_BCS, diode and KEP_BNDRY are 0 (header.h); its inner
// term (prim - 0 * grad * (...) / 2.) * dA is prim * dA for a finite slope.  A
// cell with no face keeps its own value, divided (the reference zeroes only the
// cells its face loop visits).
//
// Every pass is formed here from the prims k_update left in obuf, which nothing
// writes any more: a cell of NR-1 forms the two or three NR-2 values it reads
// again itself.  So the passes need no barrier, and the work is spread over
// the chip: OB_LANES lanes per boundary cell, a face each, whose terms are
// added in face order by shuffles.  It is a chain of dependent loads (ranges,
// face, cell) that bounds this kernel, not its few thousand cells.
#define OB_LANES 8

// The value of cell g of annulus a after its pass, formed by one thread from
// the prims of the annulus read, four faces' loads in flight at a time.  PASS
// 1: annulus 0 from 1; 2: NR-2 from NR-3.  NQ: 5, or 5 + DGPU_MAX_PASSIVE
// (planes past nq are skipped).
template <int PASS, int NQ>
__device__ __forceinline__ void outflow_value(const DevPtrs &d, const DiskParams &P, int a, int g, int nq,
                                              double *v) {
  const Annulus &A = d.ann[a];
  constexpr int outer = PASS != 1;
  const Annulus &Q = d.ann[a - outer];              // the pair (i, i+1) walked
  const Annulus &S = d.ann[outer ? a - 1 : a + 1];  // the annulus read
  const size_t NB = d.n_ob;
  const int off = S.ob_off - S.cell_off;
  const double fr = Q.f_r, fperp = Q.f_dperp;
  double s[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) s[q] = 0.0;
  int nface = 0;
  for_cell_rface_ranges(d, A, a, g, P.NR, [&](int n0, int n1, int side) {
    if (side != outer) return;
    for (int n = n0; n < n1; n += 4) {
      int c[4];
      double dA[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int f = min(n + k, n1 - 1);
        c[k] = off + rd((outer ? d.fL : d.fR) + f);
        dA[k] = fr * rd(d.fdphi + f) * fperp;
      }
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        if (NQ > 5 && q >= nq) break;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double u = rd(d.obuf + q * NB + c[k]);
          if (n + k < n1) s[q] += u * dA[k];
        }
      }
      nface += min(4, n1 - n);
    }
  });
  const double dA = A.dz * fr * d.dphi[g];
  const size_t self = (size_t)A.ob_off + (g - A.cell_off);
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    if (NQ == 5 || q < nq) v[q] = (nface ? s[q] : rd(d.obuf + q * NB + self)) / dA;
}

// The outflow radial boundary, OB_LANES threads per cell of the annuli it
// reads or writes (ob_cell): the value after the cell's pass, then, for the
// rewritten annuli, cell_bc_damp and, for stop 7, cell_calc_cons.  PS: some
// disk carries passive scalars.  THREE: some disk has three annuli, where NR-2
// is annulus 1 and reads the new annulus 0.
#define OUTFLOW_BLK 64
template <bool PS, bool THREE>
__global__ void __launch_bounds__(OUTFLOW_BLK) k_outflow(DevPtrs d, int stop) {
  constexpr int NQ = PS ? 5 + DGPU_MAX_PASSIVE : 5;
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) / OB_LANES;
  const int lane = threadIdx.x & 31, sub = lane % OB_LANES, first = lane - sub;
  const unsigned group = ((1u << OB_LANES) - 1u) << first;
  if (t >= d.n_ob) return;
  const int g = rd(d.ob_cell + t);
  const Pl QS = {PS ? d.qs : 5};
  const int a = rd(d.cell_ann + g);
  const Annulus &A = d.ann[a];
  if (!(A.kind & DGPU_AK_OUT_DST)) return;
  const DiskParams &P = d.par[A.inst];
  const size_t NB = d.n_ob;
  const int nq = PS ? 5 + P.num_n : 5;
  const int pass = A.i == P.NR - 1 ? 3 : A.i == P.NR - 2 ? 2 : 1;
  const bool chain1 = THREE && P.NR == 3 && (P.outflow & 2);
  const int outer = pass != 1;
  const Annulus &Q = d.ann[a - outer];
  const Annulus &S = d.ann[outer ? a - 1 : a + 1];
  double s[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) s[q] = 0.0;
  int nface = 0;
  for_cell_rface_ranges(d, A, a, g, P.NR, [&](int n0, int n1, int side) {
    if (side != outer) return;
    for (int n = n0; n < n1; n += OB_LANES) {
      const int nk = min(OB_LANES, n1 - n);
      double u[NQ], dA = 0.0;
#pragma unroll
      for (int q = 0; q < NQ; ++q) u[q] = 0.0;
      if (sub < nk) {
        const int f = n + sub;
        const int c = rd((outer ? d.fL : d.fR) + f);
        dA = Q.f_r * rd(d.fdphi + f) * Q.f_dperp;
        if (THREE && pass == 3 && chain1) {
          const Annulus &S1 = d.ann[a - 1], &Q1 = d.ann[a - 2];
          int nf1 = 0;
          for_cell_rface_ranges(d, S1, a - 1, c, P.NR, [&](int m0, int m1, int side1) {
            if (side1 != 1) return;
            for (int m = m0; m < m1; ++m) {
              double v[NQ];
              outflow_value<1, NQ>(d, P, a - 2, rd(d.fL + m), nq, v);
              const double dA1 = Q1.f_r * rd(d.fdphi + m) * Q1.f_dperp;
              for (int q = 0; q < nq; ++q) u[q] += v[q] * dA1;
              ++nf1;
            }
          });
          const double dA1 = S1.dz * Q1.f_r * d.dphi[c];
          for (int q = 0; q < nq; ++q)
            u[q] = (nf1 ? u[q] : rd(d.obuf + q * NB + (S1.ob_off + (c - S1.cell_off)))) / dA1;
        } else if (pass == 3) {
          outflow_value<2, NQ>(d, P, a - 1, c, nq, u);
        } else if (THREE && pass == 2 && chain1) {
          outflow_value<1, NQ>(d, P, a - 1, c, nq, u);
        } else {
#pragma unroll
          for (int q = 0; q < NQ; ++q)
            if (!PS || q < nq) u[q] = rd(d.obuf + q * NB + (S.ob_off + (c - S.cell_off)));
        }
      }
      // the terms of these faces in face order
#pragma unroll
      for (int q = 0; q < NQ; ++q) u[q] *= dA;
      for (int k = 0; k < nk; ++k)
#pragma unroll
        for (int q = 0; q < NQ; ++q) s[q] += __shfl_sync(group, u[q], first + k);
      nface += nk;
    }
  });
  if (sub != 0) return;
  const double dphi = d.dphi[g];
  const double dA = A.dz * Q.f_r * dphi;
  const size_t self = (size_t)A.ob_off + (g - A.cell_off);
  double pr[NQ], c[5];
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    if (!PS || q < nq) pr[q] = (nface ? s[q] : rd(d.obuf + q * NB + self)) / dA;
  bc_damp(d, A, a, pr);
#pragma unroll
  for (int q = 0; q < NQ; ++q)
    if (!PS || q < nq) d.prim[ix(q, QS, g)] = pr[q];
  if (stop >= 7) {
    const double r = .5 * (A.rm + A.rp);
    const double dV = A.dv_half * dphi * A.dz;
    prim2cons(pr, c, r, dV, P.gamma);
#pragma unroll
    for (int q = 0; q < 5; ++q) d.cons[ix(q, QS, g)] = c[q];
#pragma unroll
    for (int q = 5; q < NQ; ++q)
      if (q < nq) d.cons[ix(q, QS, g)] = pr[q] * c[D_DDD];
  }
}

// Torque on the binary: -sum over non-ghost cells of r*rho*dV*F_phi, with the
// gas state's cell-centre phi and F_phi from gravMassForce; per-block partial
// sums, reduced in block order by the last block.
__global__ void __launch_bounds__(BLK) k_torque(DevPtrs d, int inst, double *part, double *out) {
  __shared__ double sh[BLK / 32];
  __shared__ bool last;
  const DiskParams &P = d.par[inst];
  const InstState &S = d.ist[inst];
  const int g = P.cell_base + blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (g < P.cell_base + P.n_cells) {
    const Annulus &A = d.ann[d.cell_ann[g]];
    if (A.kind & DGPU_AK_CFL) {
      double dphi = d.dphi[g];
      double phi = d.tiph0[g] - .5 * dphi;
      double r = .5 * (A.rp + A.rm);
      double rho = ld(d.prim, D_RHO, Pl{d.qs}, g);
      double dV = dphi * .5 * A.dv_diff * P.dz;
      double cosp = cos(phi), sinp = sin(phi);
      double Fp = 0.0;
      for (int p = 0; p < 2; ++p) {
        double dx = r * cosp - S.gr[p] * cos(S.gphi[p]);
        double dy = r * sinp - S.gr[p] * sin(S.gphi[p]);
        double script_r = sqrt(dx * dx + dy * dy);
        double cosa = dx / script_r, sina = dy / script_r;
        double sinap = sina * cosp - cosa * sinp;
        Fp += sinap * -fgrav(S.gM[p], script_r, P.g_eps, P.phi_order);
      }
      v = -(r * rho * dV * Fp);
    }
  }
  const unsigned full = 0xffffffffu;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(full, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < BLK / 32; ++w) s += sh[w];
    part[blockIdx.x] = s;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&d.counters[2], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  double s = 0.0;
  for (int b = 0; b < (int)gridDim.x; ++b) s += ((volatile double *)part)[b];
  *out = s;
  d.counters[2] = 0;
}

// AoS rows [n][nq] (the boundary format) <-> cells base .. base + n of an
// array of `planes` planes
// vz (may be NULL): set when a row has a v_z
__global__ void k_aos_to_soa(double *soa, int nq, Pl planes, int base, const double *aos, int n, int *vz) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  if (vz && aos[(size_t)c * nq + D_UZZ] != 0.0) *vz = 1;
  for (int q = 0; q < nq; ++q) soa[ix(q, planes, base + c)] = aos[(size_t)c * nq + q];
}
// The context's v_z flag vz[0] from the disks' vz[1 + k].
__global__ void k_any_vz(int *vz, int n_inst) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < n_inst; k += blockDim.x)
    if (vz[1 + k]) any = 1;
  __syncthreads();
  if (threadIdx.x == 0) vz[0] = any;
}
__global__ void __launch_bounds__(BLK) k_clear_vz(DevPtrs d) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= d.n_cells || d.counters[DGPU_CT_NO_VZ] == 0) return;
  const Pl QS = {d.qs};
  d.grad[ix(D_UZZ, QS, g)] = d.gradp[ix(D_UZZ, QS, g)] = 0.0;
  d.rkcons[ix(D_SZZ, QS, g)] = 0.0;
}
__global__ void k_soa_to_aos(double *aos, int nq, Pl planes, int base, const double *soa, int n) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  for (int q = 0; q < nq; ++q) aos[(size_t)c * nq + q] = soa[ix(q, planes, base + c)];
}

}  // namespace

extern "C" {

int dgk_aos_to_soa(double *soa, int nq, int planes, int base, const double *aos, int n, int *vz, void *stream) {
  if (n <= 0) return 0;
  k_aos_to_soa<<<(n + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(soa, nq, Pl{planes}, base, aos, n, vz);
  return (int)cudaGetLastError();
}
int dgk_any_vz(int *vz, int n_inst, void *stream) {
  k_any_vz<<<1, BLK, 0, (cudaStream_t)stream>>>(vz, n_inst);
  return (int)cudaGetLastError();
}
int dgk_clear_vz(const DevPtrs *d, void *stream) {
  k_clear_vz<<<(d->n_cells + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d);
  return (int)cudaGetLastError();
}
int dgk_soa_to_aos(double *aos, int nq, int planes, int base, const double *soa, int n, void *stream) {
  if (n <= 0) return 0;
  k_soa_to_aos<<<(n + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(aos, nq, Pl{planes}, base, soa, n);
  return (int)cudaGetLastError();
}

int dgk_update_blocks(int n_cells) { return (n_cells + BLK - 1) / BLK; }
int dgk_block_size(void) { return BLK; }

// Whether the context's disks can be without a v_z at all.
static bool may_v4(const DevPtrs *d) { return d->vz && !d->has_z; }

// t == NULL: the forward kernels; otherwise their tangent instances.
// Contexts with passive scalars take the instances that carry them (PS).
#define DGK_LAUNCH(kern, grid, smem, stream, ...)                                                  \
  do {                                                                                            \
    static const TanPtrs none_ = {};                                                              \
    if (t) kern<Dual><<<(grid), BLK, (smem), (cudaStream_t)(stream)>>>(*d, *t, __VA_ARGS__);       \
    else if (d->n_pass > 0)                                                                       \
      kern<double, true><<<(grid), BLK, (smem), (cudaStream_t)(stream)>>>(*d, none_, __VA_ARGS__); \
    else if (!may_v4(d))                                                                          \
      kern<double, false, false><<<(grid), BLK, (smem), (cudaStream_t)(stream)>>>(*d, none_, __VA_ARGS__); \
    else kern<double><<<(grid), BLK, (smem), (cudaStream_t)(stream)>>>(*d, none_, __VA_ARGS__);    \
  } while (0)
// The same for the kernels the autotuner sizes, in blocks of blk threads: the
// forward instance with d->tune[which] resident blocks of BLK threads per SM
// (0: the built-in choice).
#define DGK_TUNE_SWITCH(kern, which, mbdef, v4, grid, blk, s_, ...)                              \
  switch (d->tune[which]) {                                                                     \
    case 2: kern<double, 2, false, v4><<<(grid), blk, 0, s_>>>(*d, none_, __VA_ARGS__); break;   \
    case 3: kern<double, 3, false, v4><<<(grid), blk, 0, s_>>>(*d, none_, __VA_ARGS__); break;   \
    case 4: kern<double, 4, false, v4><<<(grid), blk, 0, s_>>>(*d, none_, __VA_ARGS__); break;   \
    case 5: kern<double, 5, false, v4><<<(grid), blk, 0, s_>>>(*d, none_, __VA_ARGS__); break;   \
    default: kern<double, mbdef, false, v4><<<(grid), blk, 0, s_>>>(*d, none_, __VA_ARGS__);    \
  }
#define DGK_LAUNCH_TUNED(kern, which, mbdef, grid, blk, stream, ...)                      \
  do {                                                                                   \
    static const TanPtrs none_ = {};                                                     \
    cudaStream_t s_ = (cudaStream_t)(stream);                                            \
    if (t) {                                                                             \
      kern<Dual><<<(grid), blk, 0, s_>>>(*d, *t, __VA_ARGS__);                            \
    } else if (d->n_pass > 0) {                                                          \
      kern<double, mbdef, true><<<(grid), blk, 0, s_>>>(*d, none_, __VA_ARGS__);          \
    } else if (may_v4(d)) {                                                              \
      DGK_TUNE_SWITCH(kern, which, mbdef, true, grid, blk, s_, __VA_ARGS__)              \
    } else {                                                                             \
      DGK_TUNE_SWITCH(kern, which, mbdef, false, grid, blk, s_, __VA_ARGS__)             \
    }                                                                                    \
  } while (0)

int dgk_cellprep(const DevPtrs *d, const TanPtrs *t, int substep, void *stream) {
  DGK_LAUNCH(k_cellprep, (d->n_cells + BLK - 1) / BLK, 0, stream, substep);
  return (int)cudaGetLastError();
}
int dgk_merge(const DevPtrs *d, int substep, void *stream) {
  k_merge<<<d->n_ann, d->merge_nt > 0 ? d->merge_nt : BLK, d->smem_face, (cudaStream_t)stream>>>(*d, substep);
  return (int)cudaGetLastError();
}
int dgk_ring_mean(const DevPtrs *d, void *stream) {
  if (!d->has_rigid) return 0;
  k_ring_mean<<<(d->n_ann + RING_BLK / 32 - 1) / (RING_BLK / 32), RING_BLK, 0, (cudaStream_t)stream>>>(*d);
  return (int)cudaGetLastError();
}
int dgk_rslope(const DevPtrs *d, const TanPtrs *t, void *stream) {
  if (d->n_slots <= 0) return 0;
  static const TanPtrs none = {};
  if (t) k_rslope<Dual><<<(d->n_slots + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, *t);
  else if (d->n_pass > 0) k_rslope<double, true><<<(d->n_slots + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, none);
  else if (!may_v4(d)) k_rslope<double, false, false><<<(d->n_slots + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, none);
  else k_rslope<double><<<(d->n_slots + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, none);
  return (int)cudaGetLastError();
}
int dgk_plm_r(const DevPtrs *d, const TanPtrs *t, int substep, void *stream) {
  DGK_LAUNCH_TUNED(k_plm_r, DGPU_TUNE_PLM, DGPU_MINB_PLM, (d->n_cells + TBLK - 1) / TBLK, TBLK, stream, substep);
  return (int)cudaGetLastError();
}
int dgk_dt(const DevPtrs *d, void *stream) {
  k_dt<<<1, BLK, 0, (cudaStream_t)stream>>>(*d);
  return (int)cudaGetLastError();
}
int dgk_flux_phi(const DevPtrs *d, const TanPtrs *t, int substep, void *stream) {
  DGK_LAUNCH_TUNED(k_flux_phi, DGPU_TUNE_FLUXPHI, DGPU_MINB_FLUX, (d->n_cells + TBLK - 1) / TBLK, TBLK, stream,
                   substep);
  return (int)cudaGetLastError();
}
int dgk_flux_r(const DevPtrs *d, const TanPtrs *t, int substep, void *stream) {
  if (d->n_slots <= 0) return 0;
  DGK_LAUNCH_TUNED(k_flux_r, DGPU_TUNE_FLUXR, DGPU_MINB_FLUXR, (d->n_slots + TBLK - 1) / TBLK, TBLK, stream,
                   substep);
  return (int)cudaGetLastError();
}
int dgk_source(const DevPtrs *d, const TanPtrs *t, int substep, void *stream) {
  int n = d->n_cells > d->n_ann ? d->n_cells : d->n_ann;
  DGK_LAUNCH_TUNED(k_source, DGPU_TUNE_SOURCE, DGPU_MINB_SOURCE, (n + BLK - 1) / BLK, BLK, stream, substep, 1);
  return (int)cudaGetLastError();
}
// k_update's blocks: the cells', and the GravMass block with tail > 0
static int update_grid(const DevPtrs *d, int tail) { return (d->n_cells + TBLK - 1) / TBLK + (tail > 0); }
// k_update's resident blocks of BLK threads per SM where none was tuned: the
// built-in 4 (64 registers, spills), or 3 (80) when the cells take as many
// waves of the 148 SMs either way: 199,428 cells 30.7 -> 28.8 us (0.233 ->
// 0.2275 ms a step), 59,746 cells 16.4 -> 15, 36,962 cells 0.112 -> 0.108 ms a
// step; with a wave more 258,078 cells go from 35.5 to 39 us.  No other sizes
// were measured.  The instances with passive scalars and the tangents exist for
// the built-in budget alone.
static int update_blocks_per_sm(const DevPtrs *d) {
  const long long c3 = 148LL * 3 * BLK, c4 = 148LL * 4 * BLK, n = d->n_cells;
  return (n + c3 - 1) / c3 == (n + c4 - 1) / c4 ? 3 : DGPU_MINB_UPDATE;
}
int dgk_update(const DevPtrs *d0, const TanPtrs *t, int substep, int stop, void *stream) {
  int tail = stop >= 7 ? 2 : (stop >= 5 ? 1 : 0);
  DevPtrs h = *d0;
  const DevPtrs *d = &h;
  if (!h.tune[DGPU_TUNE_UPDATE]) h.tune[DGPU_TUNE_UPDATE] = update_blocks_per_sm(d0);
  DGK_LAUNCH_TUNED(k_update, DGPU_TUNE_UPDATE, DGPU_MINB_UPDATE, update_grid(d, tail), TBLK, stream, substep, stop, tail,
                   (double *)NULL, (const int *)NULL);
  return (int)cudaGetLastError();
}
int dgk_update_rec(const DevPtrs *d, int substep, double *rec, const int *rec_idx, void *stream) {
  static const TanPtrs none = {};
  k_update<double, DGPU_MINB_UPDATE, false, false><<<update_grid(d, 2), TBLK, 0, (cudaStream_t)stream>>>(*d, none, substep, 7, 2, rec, rec_idx);
  return (int)cudaGetLastError();
}
int dgk_ann_consts(const DevPtrs *d, int substep, void *stream) {
  static const TanPtrs none = {};
  k_source<double, DGPU_MINB_SOURCE, false, false><<<(d->n_ann + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, none, substep, 0);
  return (int)cudaGetLastError();
}
int dgk_update_stage(const DevPtrs *d, int substep, int stop, void *stream) {
  int tail = stop >= 5 ? 1 : 0;
  static const TanPtrs none = {};
  const int nb = update_grid(d, tail);
  if (d->n_pass > 0)
    k_update<double, DGPU_MINB_UPDATE, true><<<nb, TBLK, 0, (cudaStream_t)stream>>>(
        *d, none, substep, stop, tail, nullptr, nullptr);
  else
    k_update<double, DGPU_MINB_UPDATE, false, false><<<nb, TBLK, 0, (cudaStream_t)stream>>>(*d, none, substep, stop, tail, nullptr, nullptr);
  return (int)cudaGetLastError();
}
int dgk_zmerge(const DevPtrs *d, int substep, void *stream) {
  if (!d->has_z) return 0;
  k_zmerge<<<d->n_ann, d->merge_nt > 0 ? d->merge_nt : BLK, d->smem_face, (cudaStream_t)stream>>>(*d, substep);
  return (int)cudaGetLastError();
}
int dgk_zslope(const DevPtrs *d, void *stream) {
  if (!d->has_z || d->n_zslots <= 0) return 0;
  k_zslope<<<(d->n_zslots + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d);
  return (int)cudaGetLastError();
}
int dgk_plm_z(const DevPtrs *d, void *stream) {
  if (!d->has_z) return 0;
  k_plm_z<<<(d->n_cells + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d);
  return (int)cudaGetLastError();
}
int dgk_flux_z(const DevPtrs *d, int substep, void *stream) {
  if (!d->has_z || d->n_zslots <= 0) return 0;
  k_flux_z<<<(d->n_zslots + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, substep);
  return (int)cudaGetLastError();
}
int dgk_zsync(const DevPtrs *d, int substep, void *stream) {
  if (!d->has_z) return 0;
  const int n = d->zghost > 0 ? 2 * d->zghost : d->n_cells;
  k_zsync<<<(n + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, substep);
  return (int)cudaGetLastError();
}
int dgk_prep(const DevPtrs *d, int substep, void *stream) {
  k_prep<DGPU_MINB_PREP><<<d->n_ann, BLK, d->smem_face, (cudaStream_t)stream>>>(*d, substep);
  return (int)cudaGetLastError();
}
int dgk_sweep(const DevPtrs *d, int substep, void *stream) {
  cudaStream_t s_ = (cudaStream_t)stream;
  DevPtrs h = *d;
  h.form_dt = 0;  // its blocks hold the dt they form themselves (sweep_dt)
  switch (d->tune[DGPU_TUNE_SWEEP]) {
    case 2: k_sweep<2><<<d->n_ann, BLK, 0, s_>>>(h, substep); break;
    case 4: k_sweep<4><<<d->n_ann, BLK, 0, s_>>>(h, substep); break;
    default: k_sweep<DGPU_MINB_SWEEP><<<d->n_ann, BLK, 0, s_>>>(h, substep);
  }
  return (int)cudaGetLastError();
}
int dgk_outflow(const DevPtrs *d, int stop, void *stream) {
  if (d->n_ob <= 0 || stop < 6) return 0;
  const int grid = (int)(((long long)d->n_ob * OB_LANES + OUTFLOW_BLK - 1) / OUTFLOW_BLK);
  cudaStream_t s_ = (cudaStream_t)stream;
  if (d->n_pass > 0) k_outflow<true, true><<<grid, OUTFLOW_BLK, 0, s_>>>(*d, stop);
  else if (d->ob_three) k_outflow<false, true><<<grid, OUTFLOW_BLK, 0, s_>>>(*d, stop);
  else k_outflow<false, false><<<grid, OUTFLOW_BLK, 0, s_>>>(*d, stop);
  return (int)cudaGetLastError();
}
int dgk_calc_cons(const DevPtrs *d, const TanPtrs *t, void *stream) {
  static const TanPtrs none = {};
  if (t) k_calc_cons<Dual><<<(d->n_cells + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, *t);
  else if (d->n_pass > 0) k_calc_cons<double, true><<<(d->n_cells + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, none);
  else k_calc_cons<double><<<(d->n_cells + BLK - 1) / BLK, BLK, 0, (cudaStream_t)stream>>>(*d, none);
  return (int)cudaGetLastError();
}
int dgk_torque(const DevPtrs *d, int inst, double *part, double *out, int n_inst_cells, void *stream) {
  int nb = (n_inst_cells + BLK - 1) / BLK;
  k_torque<<<nb, BLK, 0, (cudaStream_t)stream>>>(*d, inst, part, out);
  return (int)cudaGetLastError();
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Face list without allocation (dgpu_face_list_noalloc).
//
// For callers that cannot allocate device memory: the face list of one disk is
// built from the caller's device arrays into the caller's device arrays, and
// the only working memory is g_noalloc_scratch below, a fixed static array
// that every GPU loading this library holds until the process exits.  Per
// annulus pair it keeps only counts and offsets, so its size is set by the
// number of annuli (DGPU_NOALLOC_MAX_ANNULI), not by the number of cells.
// ---------------------------------------------------------------------------
extern "C" {
#include "dgpu_sim.h"
}

#define NOALLOC_MAXA DGPU_NOALLOC_MAX_ANNULI

struct NoallocScratch {
  int np[NOALLOC_MAXA];        // N_p per annulus
  int off[NOALLOC_MAXA];       // first cell of each annulus
  int cnt[NOALLOC_MAXA];       // faces per pair
  int base[NOALLOC_MAXA + 1];  // first face of each pair; base[NR-1] = total
  double rface[NOALLOC_MAXA + 1];
  double dperp;
  int err;                     // DGPU_EF_* flags of this call
  int total;
  int fill_ok;                 // written only by k_noalloc_offsets: 1 when total <= cap
};
static_assert(sizeof(NoallocScratch) <= DGPU_NOALLOC_SCRATCH_BYTES, "scratch too small");

static __device__ __align__(256) unsigned char g_noalloc_scratch[DGPU_NOALLOC_SCRATCH_BYTES];

namespace {

__global__ void k_noalloc_setup(NoallocScratch *S, int NR) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int o = 0;
  for (int i = 0; i < NR; ++i) {
    S->off[i] = o;
    o += S->np[i];
  }
  S->err = 0;
  S->total = 0;
  S->fill_ok = 0;
}

// Chunk start, count and verification of one pair; the same decisions as k_merge.
struct PairPlan {
  int jpmin, jp_start, j0, j1, cnt, sequential;
};

__device__ PairPlan noalloc_plan(const FaceCtx &c, int *sh_i, int *sh_j, double *sh_v, int *sh_flag) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int np = c.Nin;
  const double p0 = c.tin[np - 1];
  PairPlan pl;
  double bv = PHIMAX;
  int bi = 0;
  for (int jp = tid; jp < c.Nout; jp += nt) {
    double dp = wrap_pos(c.tout[jp] - p0, c.err);
    if (dp < bv || (dp == bv && jp < bi)) {
      bv = dp;
      bi = jp;
    }
  }
  sh_v[tid] = bv;
  sh_i[tid] = bi;
  __syncthreads();
  for (int o = nt / 2; o > 0; o >>= 1) {
    if (tid < o) {
      double v2 = sh_v[tid + o];
      int i2 = sh_i[tid + o];
      if (v2 < sh_v[tid] || (v2 == sh_v[tid] && i2 < sh_i[tid])) {
        sh_v[tid] = v2;
        sh_i[tid] = i2;
      }
    }
    __syncthreads();
  }
  pl.jpmin = sh_i[0];
  __syncthreads();
  const int chunk = (np + nt - 1) / nt;
  pl.j0 = min(np, tid * chunk);
  pl.j1 = min(np, pl.j0 + chunk);
  pl.jp_start = pl.jpmin;
  if (pl.j0 > 0 && pl.j0 < np) {
    double L = wrap_pos(c.tin[pl.j0 - 1] - p0, c.err);
    int lo = 0, hi = c.Nout;
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      int k = pl.jpmin + mid;
      if (k >= c.Nout) k -= c.Nout;
      double e = wrap_pos(c.tout[k] - p0, c.err);
      if (e < L) lo = mid + 1;
      else hi = mid;
    }
    pl.jp_start = pl.jpmin + lo;
    if (pl.jp_start >= c.Nout) pl.jp_start -= c.Nout;
  }
  int jp = pl.jp_start, n = 0, s = 0;
  for (int j = pl.j0; j < pl.j1; ++j) face_cell<false>(c, j, jp, n, s);
  pl.cnt = n;
  if (tid == 0) *sh_flag = 0;
  sh_j[tid] = (pl.j0 < pl.j1) ? pl.jp_start : -1;
  __syncthreads();
  if (pl.j0 < pl.j1 && tid + 1 < nt && sh_j[tid + 1] >= 0 && sh_j[tid + 1] != jp) *sh_flag = 1;
  __syncthreads();
  pl.sequential = *sh_flag;
  __syncthreads();
  return pl;
}

__device__ FaceCtx noalloc_ctx(const NoallocScratch *S, int i, const double *tiph, const double *dphi,
                               int *err) {
  FaceCtx c;
  c.tin = tiph + S->off[i];
  c.din = dphi + S->off[i];
  c.tout = tiph + S->off[i + 1];
  c.dout = dphi + S->off[i + 1];
  c.Nin = S->np[i];
  c.Nout = S->np[i + 1];
  c.fL = c.fR = nullptr;
  c.fdphi = c.fcm = nullptr;
  c.runs = c.sruns = c.fstart = nullptr;
  c.cap = c.rcap = 0;
  c.err = err;
  c.offL = c.offR = 0;
  return c;
}

__global__ void __launch_bounds__(BLK) k_noalloc_count(NoallocScratch *S, const double *tiph,
                                                       const double *dphi) {
  __shared__ int sh_i[BLK];
  __shared__ int sh_j[BLK];
  __shared__ double sh_v[BLK];
  __shared__ int sh_flag;
  const int i = blockIdx.x;
  FaceCtx c = noalloc_ctx(S, i, tiph, dphi, &S->err);
  PairPlan pl = noalloc_plan(c, sh_i, sh_j, sh_v, &sh_flag);
  if (!pl.sequential) {
    int tot;
    block_excl_scan<int>(pl.cnt, sh_i, tot);
    if (threadIdx.x == 0) S->cnt[i] = tot;
  } else if (threadIdx.x == 0) {
    int jp = pl.jpmin, n = 0, s = 0;
    for (int j = 0; j < c.Nin; ++j) face_cell<false>(c, j, jp, n, s);
    S->cnt[i] = n;
  }
}

__global__ void k_noalloc_offsets(NoallocScratch *S, int NR, int cap, int *nri) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int o = 0;
  for (int i = 0; i < NR - 1; ++i) {
    S->base[i] = o;
    nri[i] = o;
    o += S->cnt[i];
  }
  S->base[NR - 1] = o;
  nri[NR - 1] = o;
  S->total = o;
  S->fill_ok = o <= cap ? 1 : 0;
  if (o > cap) S->err |= DGPU_EF_FACE_OVERFLOW;
}

// One inner cell of build_jloop writing the reference's face records
// (addFace, face_create_destroy.c:11-20) straight into the caller's arrays.
struct NoallocOut {
  int *L, *R;
  double *dphi, *dA, *cm;
  int offL, offR;
  int limit;                   // faces this pair may write (its count)
  double r, dperp;
  int *err;
};

__device__ void noalloc_cell(const FaceCtx &c, const NoallocOut &o, int j, int &jp, int &n) {
  int jm = j - 1;
  if (jm < 0) jm = c.Nin - 1;
  auto emit = [&](double dphi, double tp) {
    if (n >= 0 && n < o.limit) {
      o.L[n] = o.offL + j;
      o.R[n] = o.offR + jp;
      o.dphi[n] = dphi;
      o.dA[n] = o.r * dphi * o.dperp;
      o.cm[n] = tp - .5 * dphi;
    } else {
      set_err(o.err, DGPU_EF_FACE_OVERFLOW);
    }
    ++n;
  };
  double dp = c.tout[jp] - c.tin[jm];
  dp = wrap_pos(dp, c.err);
  if (c.din[j] < dp) {
    emit(c.din[j], c.tin[j]);
    return;
  }
  emit(dp, c.tout[jp]);
  ++jp;
  if (jp == c.Nout) jp = 0;
  dp = c.tin[j] - c.tout[jp];
  dp = wrap_pm(dp, c.err);
  int guard = 0;
  while (dp > 0.0) {
    emit(c.dout[jp], c.tout[jp]);
    ++jp;
    if (jp == c.Nout) jp = 0;
    dp = c.tin[j] - c.tout[jp];
    dp = wrap_pm(dp, c.err);
    if (++guard > c.Nout + 2) {
      set_err(c.err, DGPU_EF_FACE_OVERFLOW);
      break;
    }
  }
  dp = c.dout[jp] + dp;
  emit(dp, c.tin[j]);
}

__global__ void __launch_bounds__(BLK) k_noalloc_fill(NoallocScratch *S, const double *tiph, const double *dphi,
                                                      int *L, int *R, double *fdphi, double *fdA,
                                                      double *fcm) {
  __shared__ int sh_i[BLK];
  __shared__ int sh_j[BLK];
  __shared__ double sh_v[BLK];
  __shared__ int sh_flag;
  // fill_ok, base, cnt and total were written by the earlier kernels and are
  // only read here, so these early exits are uniform across the block
  if (!S->fill_ok) return;
  const int i = blockIdx.x;
  const int b = S->base[i];
  if (b < 0 || S->cnt[i] < 0 || b + S->cnt[i] > S->total) return;
  FaceCtx c = noalloc_ctx(S, i, tiph, dphi, &S->err);
  PairPlan pl = noalloc_plan(c, sh_i, sh_j, sh_v, &sh_flag);
  NoallocOut o;
  o.L = L + b;
  o.R = R + b;
  o.dphi = fdphi + b;
  o.dA = fdA + b;
  o.cm = fcm + b;
  o.offL = S->off[i];
  o.offR = S->off[i + 1];
  o.limit = S->cnt[i];
  o.r = S->rface[i + 1];
  o.dperp = S->dperp;
  o.err = &S->err;
  if (!pl.sequential) {
    int tot;
    int fo = block_excl_scan<int>(pl.cnt, sh_i, tot);
    if (tot != S->cnt[i]) {
      if (threadIdx.x == 0) set_err(&S->err, DGPU_EF_FACE_OVERFLOW);
      return;
    }
    int jp = pl.jp_start, n = fo;
    for (int j = pl.j0; j < pl.j1; ++j) noalloc_cell(c, o, j, jp, n);
  } else if (threadIdx.x == 0) {
    int jp = pl.jpmin, n = 0;
    for (int j = 0; j < c.Nin; ++j) noalloc_cell(c, o, j, jp, n);
  }
}

}  // namespace

// The device address of the scratch array is looked up on every call, in the
// calling thread's current context, so it stays valid after a device reset or
// from another context on the same device.  Every pointer argument must be
// memory of that current device.

extern "C" __attribute__((visibility("default"))) int dgpu_face_list_noalloc(const dgpu_sim *sim, const double *tiph, const double *dphi, int cap,
                                      int *nri, int *L, int *R, double *fdphi, double *fdA, double *fcm,
                                      int *nf, void *stream) {
  int dev = -1;
  cudaStream_t st = (cudaStream_t)stream;
  if (!sim || !tiph || !dphi || !nri || !L || !R || !fdphi || !fdA || !fcm || !nf || cap < 0)
    return DGPU_ERR_ARG;
  const int NR = sim->NR;
  if (NR > NOALLOC_MAXA || NR < 3) return DGPU_ERR_ARG;  // more annuli than the static scratch holds
  if (sim->NumZ != 1) return DGPU_ERR_UNSUPPORTED;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return DGPU_ERR_CUDA;
  void *sp = nullptr;
  if (cudaGetSymbolAddress(&sp, g_noalloc_scratch) != cudaSuccess || !sp) return DGPU_ERR_CUDA;
  NoallocScratch *S = (NoallocScratch *)sp;
  const double dperp = dsim_zface(sim, 0) - dsim_zface(sim, -1);
  if (cudaMemcpyAsync(S->np, sim->N_p, sizeof(int) * (size_t)NR, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(S->rface, sim->r_faces, sizeof(double) * (size_t)(NR + 1), cudaMemcpyHostToDevice, st) !=
          cudaSuccess ||
      cudaMemcpyAsync(&S->dperp, &dperp, sizeof(double), cudaMemcpyHostToDevice, st) != cudaSuccess)
    return DGPU_ERR_CUDA;
  k_noalloc_setup<<<1, 1, 0, st>>>(S, NR);
  k_noalloc_count<<<NR - 1, BLK, 0, st>>>(S, tiph, dphi);
  k_noalloc_offsets<<<1, 1, 0, st>>>(S, NR, cap, nri);
  k_noalloc_fill<<<NR - 1, BLK, 0, st>>>(S, tiph, dphi, L, R, fdphi, fdA, fcm);
  if (cudaGetLastError() != cudaSuccess) return DGPU_ERR_CUDA;
  int res[2] = {0, 0};
  if (cudaMemcpyAsync(&res[0], &S->err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaMemcpyAsync(&res[1], &S->total, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return DGPU_ERR_CUDA;
  *nf = res[1];
  if (res[0] & DGPU_EF_FACE_OVERFLOW) return res[1] > cap ? DGPU_ERR_ARG : DGPU_ERR_FACE_OVERFLOW;
  if (res[0]) return DGPU_ERR_NUMERIC;
  return DGPU_OK;
}
