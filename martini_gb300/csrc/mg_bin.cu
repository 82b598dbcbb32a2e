// Footprint binning: per-particle records, tile histograms, work-item plan and
// the tile-major particle list.
//
// The footprint of particle p is the reference's Chebyshev-box mask
// |i - x_p| <= r_p, |j - y_p| <= r_p (martini/martini.py:272-274) with
// r_p = ceil(sm_length * size_in_fwhm) (martini/sph_kernels.py:257-262).
// Its integer bounds are found here once per particle with the same FP64
// predicate, so the set of (pixel, particle) pairs equals the reference's.
#include <cmath>

#include "mg_internal.cuh"

namespace mg {

// ---------------------------------------------------------------------------
// The galaxy table: kernel parameters into the workspace (no host copy, so
// the insertion can be captured in a CUDA graph).
// ---------------------------------------------------------------------------

constexpr int GALS_PER_SET = 16;
struct GalChunk {
  Gal g[GALS_PER_SET];
};
static_assert(sizeof(GalChunk) <= 3584, "galaxy chunk must fit the 4 KB parameter space");

__global__ void k_set_gals(GalChunk c, int first, int count, Geo g, Ws w) {
  const int k = threadIdx.x;
  if (k < count) {
    const Gal& G = c.g[k];
    const int gi = first + k;
    w.gal[gi] = G;
    w.gp0[gi] = G.p0;
    w.gt0[gi] = G.tile0;
    w.gs0[gi] = G.seg0;
    w.ge0[gi] = G.edge0;
    w.gr0[gi] = G.row0;
  }
  if (k == 0 && first + count == g.ngal) {
    w.gp0[g.ngal] = g.n;
    w.gt0[g.ngal] = g.ntiles;
    w.gs0[g.ngal] = g.nseg;
    w.ge0[g.ngal] = (int)g.nedge;
    w.gr0[g.ngal] = g.nrows;
  }
}

void launch_set_gals(const Gal* gals, const Geo& g, const Ws& w, cudaStream_t s) {
  for (int first = 0; first < g.ngal; first += GALS_PER_SET) {
    GalChunk c;
    const int count = g.ngal - first < GALS_PER_SET ? g.ngal - first : GALS_PER_SET;
    for (int k = 0; k < count; ++k) c.g[k] = gals[first + k];
    k_set_gals<<<1, 32, 0, s>>>(c, first, count, g, w);
  }
}

// ---------------------------------------------------------------------------
// Records and tile coverage
// ---------------------------------------------------------------------------

// One thread per particle of the batch: exact footprint, Dirac pixel,
// spectral support, packed record.  Tile coverage goes into the cube's 2D
// difference array over its tile grid, (ntx + 1) x (nty + 1): +1 at the
// corners (tx0, ty0) and (tx1 + 1, ty1 + 1), -1 at (tx0, ty1 + 1) and
// (tx1 + 1, ty0), so four integer atomics per particle whatever its
// footprint; k_diff_prefix turns them into exact per-tile counts.  A block
// takes one contiguous run of particles, cube by cube: a cube's array that
// fits (PREP_SMEM_DIFF) lives in shared memory meanwhile and is added to the
// global one once per block and cube, and the cube's maxima are reduced in
// registers first.  (Small cubes have few counters, and 7 million particles of
// a 48-galaxy batch met on them in global memory: 1.77 ms with all counters there,
// 0.81 ms with the arrays in shared memory.)  The FP64 pipe bounds it (83 % busy
// with about 70 instructions a particle), so the comparisons of FP64 values are
// made on their bits and starting points and guesses come from FP32: 4M particles
// in 1024^2 x 512 0.58 ms before and 0.34 ms with both, 1M particles 0.14 and 0.09,
// the batch 0.81 and 0.44.

// The tiles a particle is listed for: those of its footprint box that hold a
// pixel within the kernel's support radius, so the tiles in the corners of a
// wide box, where every weight is exactly zero, make no pairs: 17 % fewer
// of them on 1M particles in 512^2 x 256 (20.8M to 17.3M, contraction 6.5 to
// 5.7 ms), 20 % on 500k wide ones in 1024^2 x 256 (30.4 to 25.8 ms).  `reach2`
// is the squared radius in px with a margin far above the rounding of the FP32
// weights (2e-5 relative and 2e-4 px); a kernel without a radius (Dirac: its box
// is one pixel) or with one past 1e8 px keeps the whole box.  So does a particle
// whose line or weights may not be finite: zero weights make NaN of an infinite
// line, and a length of zero makes NaN of every weight, all over the box.
// Rounded operations only, so that the counts and the list agree whatever the
// compiler fuses.
__device__ __forceinline__ float reach2(const PRec& r, const KSpec& k) {
  if (k.type == MG_KERNEL_DIRAC || !(fabsf(r.amp) < 1e30f) || !(r.inv_h2 < 1e30f)) return 1e30f;
  const float rad = k.type == MG_KERNEL_GAUSSIAN
                        ? __fmul_rn(k.truncate, __fmul_rn(r.h, 0.42466090014400953f))
                        : r.h;
  const float m = __fadd_rn(__fmul_rn(fabsf(rad), 1.00002f), 2e-4f);
  return __fmul_rn(m, m);
}

// Tile columns [t0, t1] of tile row tx (empty: t0 > t1).
__device__ __forceinline__ void row_tiles(int xi, float xf, int yi, float yf, int ilo, int ihi,
                                          int jlo, int jhi, float reach2, int tx, int& t0,
                                          int& t1) {
  if (reach2 < 1e16f) {
    const int a = max(tx * TILE_I, ilo), b = min(tx * TILE_I + TILE_I - 1, ihi);
    const float d = fmaxf(
        fmaxf(__fsub_rn((float)(a - xi), xf), __fadd_rn((float)(xi - b), xf)), 0.f);
    const float rem = __fsub_rn(reach2, __fmul_rn(d, d));
    const float half = __fsqrt_rn(fmaxf(rem, 0.f));
    jlo = max(jlo, yi + (int)ceilf(__fsub_rn(yf, half)));
    jhi = rem < 0.f ? jlo - 1 : min(jhi, yi + (int)floorf(__fadd_rn(yf, half)));
    if (jhi < jlo) {
      t0 = 1;
      t1 = 0;
      return;
    }
  }
  t0 = jlo / TILE_J;
  t1 = jhi / TILE_J;
}

// An FP64 value in FP32 by its bits, toward zero (2^-20 of it), without the few
// FP64 units; NaN from 2^60 on.
__device__ __forceinline__ float coarse_float(double v) {
  const int hi = __double2hiint(v), m = hi & 0x7fffffff;
  if (m >= (1023 + 60) << 20) return __int_as_float(0x7fffffff);
  if (m < (1023 - 60) << 20) return 0.f;
  return __int_as_float((hi & (int)0x80000000) | (m - ((1023 - 127) << 20)) << 3);
}

// Whether [x - r, x + r] certainly misses the pixels [0, n); false for NaN.
__device__ __forceinline__ bool certainly_off(double x, double r, int n) {
  const float xf = coarse_float(x), rf = coarse_float(r);
  const float reach = rf + 1.f + 1e-5f * (fabsf(xf) + fabsf(rf));
  return xf < -reach || xf - (float)n > reach;
}

// Whether a particle's tabulated spectrum holds a value that reach2 takes for
// not finite, into the pair counts (which the records kernel reads and
// overwrites).  One more pass over the table, bound by HBM where it is long:
// a warp takes `group` particles, whose rows are contiguous, and streams them
// from the first to the last whose box may reach the cube (the others have no
// pairs).  bf16x6 insertions without the pass and with it: 500k spectra of 128
// channels on 200 x 200 962 and 1025 us, nearly all of them off the cube 264 and
// 275; 2M of 16 channels on 300 x 300 1853 and 1908, with a warp per row 2016.
__global__ void k_table_finite(Geo g, Ws w, int group) {
  const int lane = threadIdx.x & 31;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long base = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * group;
       base < g.n; base += nwarps * group) {
    const long long P = base + lane;
    bool on = false;
    if (lane < group && P < g.n) {
      const Gal& G = w.gal[find_gal(w.gp0, g.ngal, P)];
      const long long p = P - G.p0;
      on = !certainly_off(G.x[p], G.r[p], G.nx) && !certainly_off(G.y[p], G.r[p], G.ny);
    }
    unsigned bad = 0u;  // bit k: particle base + k
    for (unsigned m = __ballot_sync(0xffffffffu, on); m;) {
      // rows k0 .. k1 - 1: those of the first wanted one's cube
      const int k0 = __ffs(m) - 1;
      const int gk = find_gal(w.gp0, g.ngal, base + k0);
      const Gal& G = w.gal[gk];
      const int k1 = (int)min((long long)(32 - __clz(m)), w.gp0[gk + 1] - base);
      m = k1 < 32 ? m >> k1 << k1 : 0u;
      const int nc = G.nc;
      const float* const s = G.spectra + (base + k0 - G.p0) * nc;
      const long long total = (long long)(k1 - k0) * nc;
      for (long long e = lane; e < total; e += 256) {
        float v[8];
        bool any = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = e + 32 * j < total ? __ldg(s + e + 32 * j) : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) any |= !(fabsf(v[j]) < 1e30f);
        if (any) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (!(fabsf(v[j]) < 1e30f)) bad |= 1u << (k0 + (int)((e + 32 * j) / nc));
        }
      }
    }
    bad = __reduce_or_sync(0xffffffffu, bad);
    if (lane < group && P < g.n) w.npairs[P] = (bad >> lane) & 1u;
  }
}

constexpr int PREP_THREADS = 256;
constexpr int PREP_SMEM_DIFF = 11776;  // 46 KB: static and dynamic within 48 KB

// RUNS: a block takes its run cube by cube, as above.  Batches of cubes with few
// particles (at most PREP_FEW on average) are taken without: a cube's turn costs a
// block about 4 us whatever its particles, and a run has many such cubes, while
// few particles meet on a counter.  Binning of 3000 cubes with one particle each:
// 3.08 ms with runs, 1.83 now (1.7 ms of both sets the cubes' table up); 1000 cubes
// of 32^3 with 64 particles each 782 us without runs, with 65 each 802 us with.
constexpr long long PREP_FEW = 64;

template <bool RUNS>
__global__ void __launch_bounds__(PREP_THREADS) k_prep(Geo g, Ws w, long long per) {
  extern __shared__ int s_diff[];  // the difference array of the cube when it fits
  __shared__ unsigned long long s_spec;
  if (threadIdx.x == 0) s_spec = 0ull;
  unsigned my_spec = 0u;  // support channels of this thread's particles
  const int lane = threadIdx.x & 31;
  const long long run1 = min((long long)(blockIdx.x + 1) * per, g.n);
  for (long long run0 = (long long)blockIdx.x * per; run0 < run1;) {
    // the run's particles of one cube
    const int run_gk = find_gal(w.gp0, g.ngal, run0);
    const long long run_hi = RUNS ? min(run1, w.gp0[run_gk + 1]) : run1;
    const int nd = (w.gal[run_gk].ntx + 1) * (w.gal[run_gk].nty + 1);
    const bool smem_hist = RUNS && nd <= PREP_SMEM_DIFF;
    if (smem_hist)
      for (int t = threadIdx.x; t < nd; t += blockDim.x) s_diff[t] = 0;
    __syncthreads();
    int wmax_v = 0;
    unsigned wb_v = 0u, sb_v = 0u;
    const ChanGrid run_grid(w.gal[run_gk].edges, w.gal[run_gk].nc, w.gst[run_gk].dec);
    for (long long P = run0 + threadIdx.x; P < run_hi; P += PREP_THREADS) {
      const int gk = RUNS ? run_gk : find_gal(w.gp0, g.ngal, P);
      const Gal& G = w.gal[gk];
      const long long p = P - G.p0;
      const int dec = w.gst[gk].dec;
      const ChanGrid grid = RUNS ? run_grid : ChanGrid(G.edges, G.nc, dec);
      const double* edges = G.edges;
      PRec rec;
      rec.ilo = 0; rec.ihi = -1; rec.jlo = 0; rec.jhi = -1;
      rec.clo = 1; rec.chi = 0;
      rec.xi = rec.yi = 0;
      rec.xf = rec.yf = 0.f;
      rec.h = 1.f; rec.inv_h2 = 1.f;
      rec.vhi = rec.vlo = 0.f; rec.inv_s = 0.f; rec.amp = 0.f; rec.flags = 0;
      int ks = G.kidx ? (int)G.kidx[p] : 0;
      if (ks < 0 || ks >= g.n_kernels) ks = 0;  // -1: kernels[0] (sph_kernels.py:1360)
      rec.kslot = ks;
      double x = G.x[p], y = G.y[p], r = G.r[p];
      // |coordinate| > 2^30 px cannot reach the cube (and would overflow int)
      // (2^30 as the high word of an FP64 value; infinities and NaN are past it)
      bool ok = (__double2hiint(x) & 0x7fffffff) < 0x41d00000 &&
                (__double2hiint(y) & 0x7fffffff) < 0x41d00000;
      if (ok) {
        box_bounds(x, r, G.nx, rec.ilo, rec.ihi);
        box_bounds(y, r, G.ny, rec.jlo, rec.jhi);
        ok = rec.ilo <= rec.ihi && rec.jlo <= rec.jhi;
      }
      if (ok && g.ks[ks].type == MG_KERNEL_DIRAC) {
        // weight 1 iff |x - i| < 0.5 and |y - j| < 0.5 (sph_kernels.py:1165):
        // at most one pixel per axis, tested in FP64.
        int di = -1, dj = -1;
        double fx = floor(x), fy = floor(y);
        if (fabs(x - fx) < 0.5) di = (int)fx; else if (fabs(x - (fx + 1.0)) < 0.5) di = (int)fx + 1;
        if (fabs(y - fy) < 0.5) dj = (int)fy; else if (fabs(y - (fy + 1.0)) < 0.5) dj = (int)fy + 1;
        if (di < rec.ilo || di > rec.ihi || dj < rec.jlo || dj > rec.jhi) {
          ok = false;
        } else {
          rec.ilo = rec.ihi = di;
          rec.jlo = rec.jhi = dj;
        }
      }
      if (ok) {
        double fx = floor(x), fy = floor(y);
        rec.xi = (int)fx;
        rec.yi = (int)fy;
        rec.xf = (float)(x - fx);
        rec.yf = (float)(y - fy);
        float h = G.h ? G.h[p] : 1.f;
        rec.h = h;
        rec.inv_h2 = 1.f / (h * h);
        if (g.ks[ks].type <= MG_KERNEL_QUARTIC_SPLINE) {
          // every table kernel reaches h px; rows outside the cube are never
          // stored.  Tested in FP32 with a margin well above its rounding
          // (coordinates below 2^30 px): a flag missed near the edge only
          // keeps the per-row box test
          const float xf32 = (float)x;
          const float reach = h * (1.f + 0x1p-18f) + 1e-6f * (fabsf(xf32) + 1.f);
          const bool lo_in = rec.ilo == 0 || xf32 - (float)(rec.ilo - 1) >= reach;
          const bool hi_in = rec.ihi == G.nx - 1 || (float)(rec.ihi + 1) - xf32 >= reach;
          if (lo_in && hi_in) rec.flags |= PREC_ROWS_COVER;
          const float yf32 = (float)y;
          const float reach_y = h * (1.f + 0x1p-18f) + 1e-6f * (fabsf(yf32) + 1.f);
          const bool lo_jn = rec.jlo == 0 || yf32 - (float)(rec.jlo - 1) >= reach_y;
          const bool hi_jn = rec.jhi == G.ny - 1 || (float)(rec.jhi + 1) - yf32 >= reach_y;
          if (lo_jn && hi_jn) rec.flags |= PREC_COLS_COVER;
        }
        if (g.spectral_model == MG_SPECTRUM_TABLE) {
          rec.clo = 0;
          rec.chi = G.nc - 1;
          rec.amp = w.npairs[P] ? __int_as_float(0x7f800000) : 1.f;  // k_table_finite
        } else {
          double v = G.v[p];
          double am = G.amp[p];
          rec.amp = (float)am;
          double vh = (double)(float)v;
          rec.vhi = (float)vh;
          rec.vlo = (float)(v - vh);
          if (g.spectral_model == MG_SPECTRUM_GAUSSIAN) {
            double sg = G.sigma ? (double)G.sigma[p] : (double)G.sigma_const;
            rec.inv_s = 1.f / (float)(1.4142135623730951 * sg);  // FP32 division
            // |u| <= 4.5: beyond it each wing holds erfc(4.5) / 2 = 1e-10 of
            // the line's flux
            double half = 4.5 * 1.4142135623730951 * sg;
            const float half_f = 4.5f / rec.inv_s;
            channel_range(edges, G.nc, dec, grid, v - half, v + half, rec.vhi - half_f,
                          rec.vhi + half_f, rec.clo, rec.chi);
          } else {
            channel_range(edges, G.nc, dec, grid, v, v, rec.vhi, rec.vhi, rec.clo, rec.chi);
          }
          if (am == 0.0 || !isfinite(v)) {
            rec.clo = 1;
            rec.chi = 0;
          }
        }
        ok = rec.clo <= rec.chi;
      }
      if (!ok) {
        rec.ilo = 0; rec.ihi = -1; rec.jlo = 0; rec.jhi = -1;
      }
      w.rec[P] = rec;
      int np = 0;
      if (ok) {
        const int tx0 = rec.ilo / TILE_I, tx1 = rec.ihi / TILE_I;
        const int ty0 = rec.jlo / TILE_J, ty1 = rec.jhi / TILE_J;
        // one pair per (tile, channel block) the line meets
        const int nb = G.ncb > 1 ? rec.chi / G.width - rec.clo / G.width + 1 : 1;
        const float r2 = reach2(rec, g.ks[ks]);
        for (int tx = tx0; tx <= tx1; ++tx) {
          int t0, t1;
          row_tiles(rec.xi, rec.xf, rec.yi, rec.yf, rec.ilo, rec.ihi, rec.jlo, rec.jhi, r2, tx, t0,
                    t1);
          np += t1 - t0 + 1;
        }
        np *= nb;
        const int dw = G.nty + 1;
        int* const diff = smem_hist ? s_diff : w.tile_diff + G.diff0;
        atomicAdd(&diff[tx0 * dw + ty0], 1);
        atomicAdd(&diff[tx0 * dw + ty1 + 1], -1);
        atomicAdd(&diff[(tx1 + 1) * dw + ty0], -1);
        atomicAdd(&diff[(tx1 + 1) * dw + ty1 + 1], 1);
        wmax_v = max(wmax_v, rec.chi - rec.clo);
        my_spec += (unsigned)(rec.chi - rec.clo + 1);
        if (g.form == MG_FORM_F16X3) {
          // magnitude bounds for the scaled FP16 split (non-negative floats
          // order like their bit patterns)
          const KSpec k = g.ks[ks];
          wb_v = max(wb_v, __float_as_uint(weight_bound(k.type, rec.inv_h2, k.gnorm)));
          float sb = rec.amp;
          if (g.spectral_model == MG_SPECTRUM_TABLE) {
            sb = 0.f;
            for (int c = 0; c < G.nc; ++c) sb = fmaxf(sb, fabsf(G.spectra[p * G.nc + c]));
          }
          sb_v = max(sb_v, __float_as_uint(sb));
        }
      }
      w.npairs[P] = np;
      if (!RUNS) {
        if (wmax_v) atomicMax(&w.gst[gk].wmax, wmax_v);
        if (wb_v) atomicMax(&w.gst[gk].wbound_bits, wb_v);
        if (sb_v) atomicMax(&w.gst[gk].sbound_bits, sb_v);
        wmax_v = 0;
        wb_v = sb_v = 0u;
      }
    }
    if (!RUNS) break;
    const int gk = run_gk;
    wmax_v = __reduce_max_sync(0xffffffffu, wmax_v);
    wb_v = __reduce_max_sync(0xffffffffu, wb_v);
    sb_v = __reduce_max_sync(0xffffffffu, sb_v);
    if (lane == 0) {
      if (wmax_v) atomicMax(&w.gst[gk].wmax, wmax_v);
      if (wb_v) atomicMax(&w.gst[gk].wbound_bits, wb_v);
      if (sb_v) atomicMax(&w.gst[gk].sbound_bits, sb_v);
    }
    __syncthreads();
    if (smem_hist) {
      for (int t = threadIdx.x; t < nd; t += blockDim.x)
        if (s_diff[t]) atomicAdd(&w.tile_diff[w.gal[gk].diff0 + t], s_diff[t]);
      __syncthreads();
    }
    run0 = run_hi;
  }
  my_spec = __reduce_add_sync(0xffffffffu, my_spec);
  __syncthreads();
  if (lane == 0) atomicAdd(&s_spec, (unsigned long long)my_spec);
  __syncthreads();
  if (threadIdx.x == 0 && stored_lines(g.spectral_model))
    atomicAdd(reinterpret_cast<unsigned long long*>(&w.hdr->spec_bound), s_spec);
}

__global__ void k_tile_init(Geo g, Ws w, long long cap_pairs, long long cap_partial) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < g.ndiff; t += stride)
    w.tile_diff[t] = 0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < g.ngal; k += stride) {
    GalState z;
    z.dec = 0;
    z.wmax = 0;
    z.wbound_bits = z.sbound_bits = z.invw_bits = 0u;
    z.pad_[0] = z.pad_[1] = z.pad_[2] = 0;
    w.gst[k] = z;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    WsHeader* h = w.hdr;
    h->status = 0;
    h->item_counter = 0;
    h->n_pairs = h->n_items = h->n_partial_items = h->partial_bound = 0;
    h->cap_pairs = cap_pairs;
    h->cap_partial_items = cap_partial;
    h->spec_bound = 0;
    h->n_spec = 0;
    h->spec_ready = 0;
    h->kch = KCH_MIN;
    h->plan_key = 0;
  }
}

// Channel edges of every cube as double-float pairs, inverse channel widths,
// edge direction and the strict-monotonicity check of
// spectral_models.py:180-187.  Batch-wide edge index e = edge0 + k.
__global__ void k_edges(Geo g, Ws w) {
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < g.nedge;
       e += (long long)gridDim.x * blockDim.x) {
    const int gk = find_gal(w.ge0, g.ngal, (int)e);
    const Gal& G = w.gal[gk];
    const int k = (int)e - G.edge0;
    const double* ed = G.edges;
    const int dec = ed[G.nc] < ed[0];
    if (k == 0) w.gst[gk].dec = dec;
    const double v = ed[k];
    const float hi = (float)v;
    w.ehi[e] = hi;
    w.elo[e] = (float)(v - (double)hi);
    if (k < G.nc) {
      const float iw = (float)(1.0 / fabs(ed[k + 1] - ed[k]));
      w.inv_w[e] = iw;
      atomicMax(&w.gst[gk].invw_bits, __float_as_uint(iw));
      const bool mono = dec ? (ed[k + 1] < ed[k]) : (ed[k + 1] > ed[k]);
      if (!mono) atomicOr(&w.hdr->status, ST_EDGES);
    } else {
      w.inv_w[e] = 0.f;
    }
  }
}

// One block per cube: exact per-tile counts from the cube's difference array
// (prefix sums along ty, then along tx; in shared memory when it fits in
// `smem_cap` ints, else in place).
__global__ void k_diff_prefix(Geo g, Ws w, int smem_cap) {
  extern __shared__ int s_d[];
  const Gal& G = w.gal[blockIdx.x];
  const int dw = G.nty + 1, dh = G.ntx + 1;
  const int nd = dw * dh;
  const bool in_smem = nd <= smem_cap;
  int* const d = in_smem ? s_d : w.tile_diff + G.diff0;
  const int* src = w.tile_diff + G.diff0;
  if (in_smem)
    for (int e = threadIdx.x; e < nd; e += blockDim.x) s_d[e] = src[e];
  __syncthreads();
  for (int r = threadIdx.x; r < dh; r += blockDim.x) {
    int acc = 0;
    for (int c = 0; c < dw; ++c) {
      acc += d[r * dw + c];
      d[r * dw + c] = acc;
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < dw; c += blockDim.x) {
    int acc = 0;
    for (int r = 0; r < dh; ++r) {
      acc += d[r * dw + c];
      d[r * dw + c] = acc;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < G.ntiles; t += blockDim.x) {
    const int tx = t / G.nty, ty = t - tx * G.nty;
    w.tile_count[G.tile0 + t] = d[tx * dw + ty];
  }
}

// After the scans of the pair counts (total in hdr->n_pairs) and the tile
// counts: the work item size from the total pairs, the split-K bound with it
// (every segment of a tile lists at most the tile's particles, each once)
// and the pair-capacity check.
__global__ void k_plan_finish(Geo g, Ws w, int num_sms, unsigned long long plan_key) {
  __shared__ long long red[256];
  const long long total = w.hdr->n_pairs;
  const int kch = item_particles(total, num_sms, g.items_per_sm);
  long long sb = 0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < g.ntiles; t += gridDim.x * blockDim.x) {
    const long long cnt = w.tile_off[t + 1] - w.tile_off[t];
    const long long nk = (cnt + kch - 1) / kch;
    if (nk > 1) sb += nk * w.gal[find_gal(w.gt0, g.ngal, t)].ncb;
  }
  red[threadIdx.x] = sb;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0 && red[0])
    atomicAdd(reinterpret_cast<unsigned long long*>(&w.hdr->partial_bound),
              (unsigned long long)red[0]);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    WsHeader* h = w.hdr;
    h->kch = kch;
    h->plan_key = plan_key;
    if (total > h->cap_pairs) atomicOr(&h->status, ST_PAIRS);
  }
}

// Continue from the plan that this workspace holds: its records and counts
// stand, the header takes the capacities and the launch shape of this run.
// The later stages overwrite the counts, so a plan serves one run.  A binning
// pass less in a call that plans first: 1M particles 6.01 to 5.80 ms, 5k particles
// 0.42 to 0.38 ms.  For an engine's later calls only: where the workspace grows
// after the plan, as in the first call, the run bins again.
__global__ void k_resume(Geo g, Ws w, int num_sms, long long cap_pairs, long long cap_partial,
                         unsigned long long plan_key) {
  WsHeader* h = w.hdr;
  const bool ok = h->plan_key == plan_key;
  const long long total = ok ? h->n_pairs : 0;
  // bad channel edges stay an error of the run, as they were of the plan; the
  // plan's pair status does not (it ran without room for pairs)
  h->status = ok ? (h->status & ST_EDGES) | (total > cap_pairs ? ST_PAIRS : 0u)
                 : (ST_NO_PLAN | ST_PAIRS);
  h->item_counter = 0;
  h->n_pairs = total;
  h->n_items = h->n_partial_items = 0;
  h->n_valid = 0;
  h->cap_pairs = cap_pairs;
  h->cap_partial_items = cap_partial;
  h->n_spec = 0;
  h->spec_ready = 0;
  h->kch = item_particles(total, num_sms, g.items_per_sm);
  h->plan_key = 0;
}

void launch_resume(const Geo& g, const Ws& w, int num_sms, cudaStream_t s, long long cap_pairs,
                   long long cap_partial, unsigned long long plan_key) {
  k_resume<<<1, 1, 0, s>>>(g, w, num_sms, cap_pairs, cap_partial, plan_key);
}

// a / b for 0 <= a < 2^24, b >= 1, from a reciprocal estimate corrected to
// the exact quotient.
__device__ __forceinline__ int div_exact(int a, int b, float rb) {
  int q = (int)(((float)a + 0.5f) * rb);
  int r = a - q * b;
  while (r < 0) {
    --q;
    r += b;
  }
  while (r >= b) {
    ++q;
    r -= b;
  }
  return q;
}

// Exclusive sum over the warp's lanes; total in every lane.
__device__ __forceinline__ int warp_exclusive(int v, int lane, int& total) {
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  total = __shfl_sync(0xffffffffu, x, 31);
  return x - v;
}

// Last lane whose value is <= f (values ascend over the lanes; an empty one
// shares its value with the next).
__device__ __forceinline__ int lane_of(int first, int f) {
  int src = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1) {
    const int v = __shfl_sync(0xffffffffu, first, src + step);
    if (v <= f) src += step;
  }
  return src;
}

// Pairs in the order of `order` (particles by kernel class and first channel):
// key = global segment, value = particle, one pair per tile (row_tiles) and
// channel block the particle's line meets.  A warp takes 32 particles, whose
// pairs are one contiguous range of the output (pair_off is the exclusive scan
// of the counts in this order).  Their tile rows are dealt to the lanes, 32 at a
// time, and the pairs of those rows again, so that every lane has work whatever
// the footprints and every store of the warp is contiguous.  The pairs of a
// particle run row-major over its tiles, then over its channel blocks.
__global__ void k_emit(Geo g, Ws w, const int* __restrict__ order, unsigned* __restrict__ keys,
                       int* __restrict__ vals) {
  if (w.hdr->status & (ST_PAIRS | ST_EDGES)) return;
  const int lane = threadIdx.x & 31;
  const long long nwarps = (long long)gridDim.x * (blockDim.x >> 5);
  const long long nv = w.hdr->n_valid;
  for (long long base = ((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5) * 32;
       base < nv; base += nwarps * 32) {
    const long long K = base + lane;
    PRec rec;
    rec.xi = rec.yi = rec.ilo = rec.ihi = rec.jlo = rec.jhi = 0;
    rec.xf = rec.yf = 0.f;
    float r2 = 0.f;
    int P = 0, nr = 0, tx0 = 0, cb0 = 0, nb = 1, seg0 = 0, nty = 1, ncb = 1;
    if (K < nv) {
      P = order[K];
      rec = w.rec[P];
      const Gal& G = w.gal[find_gal(w.gp0, g.ngal, (long long)P)];
      tx0 = rec.ilo / TILE_I;
      nr = rec.ihi / TILE_I - tx0 + 1;
      cb0 = G.ncb > 1 ? rec.clo / G.width : 0;
      nb = G.ncb > 1 ? rec.chi / G.width - cb0 + 1 : 1;
      seg0 = G.seg0;
      nty = G.nty;
      ncb = G.ncb;
      r2 = reach2(rec, g.ks[rec.kslot]);
    }
    long long out = __shfl_sync(0xffffffffu, K < nv ? w.pair_off[K] : 0ll, 0);
    int nrows;
    const int row0 = warp_exclusive(nr, lane, nrows);
    for (int q0 = 0; q0 < nrows; q0 += 32) {  // warp-uniform
      // this lane's tile row
      const int src = lane_of(row0, q0 + lane);
      const int tx = __shfl_sync(0xffffffffu, tx0, src) + (q0 + lane) -
                     __shfl_sync(0xffffffffu, row0, src);
      const int xi = __shfl_sync(0xffffffffu, rec.xi, src);
      const int yi = __shfl_sync(0xffffffffu, rec.yi, src);
      const float xf = __shfl_sync(0xffffffffu, rec.xf, src);
      const float yf = __shfl_sync(0xffffffffu, rec.yf, src);
      const int ilo = __shfl_sync(0xffffffffu, rec.ilo, src);
      const int ihi = __shfl_sync(0xffffffffu, rec.ihi, src);
      const int jlo = __shfl_sync(0xffffffffu, rec.jlo, src);
      const int jhi = __shfl_sync(0xffffffffu, rec.jhi, src);
      const float rr = __shfl_sync(0xffffffffu, r2, src);
      const int rnb = __shfl_sync(0xffffffffu, nb, src);
      const int rncb = __shfl_sync(0xffffffffu, ncb, src);
      const int rP = __shfl_sync(0xffffffffu, P, src);
      int t0 = 1, t1 = 0;
      if (q0 + lane < nrows) row_tiles(xi, xf, yi, yf, ilo, ihi, jlo, jhi, rr, tx, t0, t1);
      // the row's first segment: its first tile's first block
      const int sg = __shfl_sync(0xffffffffu, seg0, src) +
                     (tx * __shfl_sync(0xffffffffu, nty, src) + t0) * rncb +
                     __shfl_sync(0xffffffffu, cb0, src);
      int total;
      const int first = warp_exclusive((t1 - t0 + 1) * rnb, lane, total);
      for (int f0 = 0; f0 < total; f0 += 32) {  // warp-uniform
        const int f = f0 + lane;
        const int rs = lane_of(first, f);
        const int e = f - __shfl_sync(0xffffffffu, first, rs);
        const int b = __shfl_sync(0xffffffffu, rnb, rs);
        const int sncb = __shfl_sync(0xffffffffu, rncb, rs);
        const int ssg = __shfl_sync(0xffffffffu, sg, rs);
        const int sP = __shfl_sync(0xffffffffu, rP, rs);
        if (f < total) {
          const int t = b > 1 ? div_exact(e, b, __frcp_rn((float)b)) : e;
          keys[out + f] = (unsigned)(ssg + t * sncb + (e - t * b));
          vals[out + f] = sP;
        }
      }
      out += total;
    }
  }
}

// First index in [lo, hi) of sorted keys with key >= k, by a warp: 32 probes a
// round (a thread's bisection is 15 to 27 dependent reads, which took 15 us
// even for a list of 30,000 pairs).
__device__ __forceinline__ long long lower_bound_keys(const unsigned* keys, long long lo,
                                                      long long hi, unsigned k, int lane) {
  while (lo < hi) {
    const long long step = (hi - lo + 31) / 32;
    const long long m = lo + lane * step;  // probes in ascending order
    const bool less = m < hi && keys[m] < k;
    const int n = __popc(__ballot_sync(0xffffffffu, less));  // the first n probes are less
    if (n == 0) return lo;
    const long long last = lo + (long long)(n - 1) * step;  // the last one that is
    hi = min(hi, last + step);
    lo = last + 1;
  }
  return lo;
}

// One warp per segment (tile, channel block): its range of the sorted list,
// its K chunks and its split-K partial items.
__global__ void k_segments(Geo g, Ws w) {
  const bool bad = (w.hdr->status & (ST_PAIRS | ST_EDGES)) != 0;
  const int kch = w.hdr->kch;
  const long long n = w.hdr->n_pairs;
  const int lane = threadIdx.x & 31;
  const int sg = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  if (sg >= g.nseg) return;
  long long lo = 0, hi = 0;
  int items = 0, part = 0;
  if (!bad && n > 0) {
    lo = lower_bound_keys(w.keys, 0, n, (unsigned)sg, lane);
    hi = sg + 1 == g.nseg ? n : lower_bound_keys(w.keys, lo, n, (unsigned)sg + 1u, lane);
    const long long cnt = hi - lo;
    if (cnt > 0) {
      items = (int)((cnt + kch - 1) / kch);
      part = items > 1 ? items : 0;
    }
  }
  if (lane == 0) {
    w.seg_lo[sg] = lo;
    w.seg_hi[sg] = hi;
    w.seg_items[sg] = items;
    w.seg_part[sg] = part;
  }
}

// Work-queue keys: one thread per segment writes the keys of its items
// (item k of a segment holds min(kch, cnt - k kch) particles).  Estimated
// cost = particles x (2 TILE_PX + width): the kernel weights at the tile's
// pixels and the spectra and products over the segment's channel block.
// Key = top - cost scaled to RS_BITS bits, so that one stable distribution
// pass puts the largest items first and keeps segment order among equal ones:
// the persistent contraction then ends on the small items instead of leaving
// one large item to a single SM at the end.
__global__ void k_item_keys(Geo g, Ws w) {
  if (w.hdr->status & (ST_PAIRS | ST_EDGES)) return;
  const int kch = w.hdr->kch;
  const double top = (double)((1 << RS_BITS) - 1);
  const double cmax = (double)kch * (2.0 * TILE_PX + (double)g.max_width);
  for (int sg = blockIdx.x * blockDim.x + threadIdx.x; sg < g.nseg; sg += gridDim.x * blockDim.x) {
    const int n_it = w.seg_items[sg];
    if (n_it == 0) continue;
    const long long base = w.item_off[sg];
    const long long cnt = w.seg_hi[sg] - w.seg_lo[sg];
    const int width = w.gal[find_gal(w.gs0, g.ngal, sg)].width;
    for (int k = 0; k < n_it && base + k < w.cap_items; ++k) {
      const long long left = cnt - (long long)k * kch;
      const double lc = (double)(left < kch ? left : kch);
      double q = lc * (2.0 * TILE_PX + (double)width) / cmax * top + 0.5;
      if (q > top) q = top;
      // all keys equal: the stable sort keeps segment order
      w.item_key_tmp[base + k] = g.cost_order ? (unsigned)top - (unsigned)q : 0u;
      w.item_order_tmp[base + k] = (int)(base + k);
      w.item_seg[base + k] = sg;
    }
  }
}

__global__ void k_check_partials(Ws w) {
  WsHeader* h = w.hdr;
  if (h->n_partial_items > h->cap_partial_items) h->status |= ST_PARTIALS;
}

static unsigned grid_for(long long n, int num_sms) {
  long long blocks = (n + 255) / 256;
  if (blocks > (long long)num_sms * 32) blocks = (long long)num_sms * 32;
  return (unsigned)(blocks > 0 ? blocks : 1);
}

// Records, tile histograms, per-particle pair offsets and the tile plan.
void launch_prep(const Geo& g, const Ws& w, int num_sms, cudaStream_t s, long long cap_pairs,
                 long long cap_partial, unsigned long long plan_key) {
  long long init_n = g.ndiff > g.ntiles ? g.ndiff : g.ntiles;
  if (g.ngal > init_n) init_n = g.ngal;
  k_tile_init<<<grid_for(init_n, num_sms), 256, 0, s>>>(g, w, cap_pairs, cap_partial);
  k_edges<<<grid_for(g.nedge, num_sms), 256, 0, s>>>(g, w);
  if (g.n > 0) {
    if (g.spectral_model == MG_SPECTRUM_TABLE) {
      // 32 particles a warp, fewer while that leaves SMs with few warps
      const int group = (int)std::min<long long>(32, 1 + g.n / (num_sms * 32ll));
      k_table_finite<<<grid_for((g.n + group - 1) / group * 32, num_sms), 256, 0, s>>>(g, w, group);
    }
    // every block adds its arrays to the global ones: fewer, longer runs where
    // the arrays are large
    const bool runs = g.ngal == 1 || g.n > PREP_FEW * g.ngal;
    const int nd = !runs                          ? 0
                   : g.max_diff <= PREP_SMEM_DIFF ? g.max_diff
                   : g.ngal > 1                   ? PREP_SMEM_DIFF
                                                  : 0;
    const size_t hist_bytes = sizeof(int) * (size_t)nd;
    long long blocks = grid_for(g.n, num_sms);
    const long long most = (hist_bytes <= 16384 ? 8ll : 4ll) * num_sms;
    if (blocks > most) blocks = most;
    const long long per =
        ((g.n + blocks - 1) / blocks + PREP_THREADS - 1) / PREP_THREADS * PREP_THREADS;
    (runs ? k_prep<true> : k_prep<false>)<<<(unsigned)((g.n + per - 1) / per), PREP_THREADS,
                                            hist_bytes, s>>>(g, w, per);
  }
  launch_scan(w.npairs, g.n, w.pair_off, w.scan_sums, &w.hdr->n_pairs, s);
  // per-cube prefix sums of the difference arrays, in up to 200 KB of
  // dynamic shared memory (the attribute is per device: set on every launch)
  constexpr int kPlanSmemCap = 50 * 1024;
  int cap = g.max_diff <= kPlanSmemCap ? g.max_diff : 0;
  if (cap > 12 * 1024 &&
      cudaFuncSetAttribute(k_diff_prefix, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)(sizeof(int) * kPlanSmemCap)) != cudaSuccess) {
    cudaGetLastError();  // fall back to the in-place prefix sums
    cap = 0;
  }
  k_diff_prefix<<<g.ngal, 256, sizeof(int) * (size_t)cap, s>>>(g, w, cap);
  launch_scan(w.tile_count, g.ntiles, w.tile_off, w.scan_sums, w.tile_off + g.ntiles, s);
  k_plan_finish<<<grid_for(g.ntiles, num_sms), 256, 0, s>>>(g, w, num_sms, plan_key);
}

int seg_bits(const Geo& g) {
  int b = 0;
  while ((1LL << b) < (long long)g.nseg) ++b;
  return b;
}

// Bits of a key of segment, kernel class and first channel.  Problems past 32 are
// refused: the list's keys held all three once.  They hold the segment alone now;
// the limit stands as part of the interface.
int sort_bits(const Geo& g) { return seg_bits(g) + g.cbits; }

// The list sorted by segment, then class and first channel, then the segments
// with their work-item and partial offsets.  Pairs are emitted into the buffer
// from which an even/odd number of passes ends in w.keys / w.list; the
// particle order lies in the other buffer's keys until the first pass.
void launch_sort_segments(const Geo& g, const Ws& w, long long cap_pairs, int num_sms,
                          cudaStream_t s) {
  const int bits = seg_bits(g);
  const bool odd = (radix_passes(bits) & 1) != 0;
  unsigned* k0 = odd ? w.keys_tmp : w.keys;
  int* v0 = odd ? w.list_tmp : w.list;
  unsigned* k1 = odd ? w.keys : w.keys_tmp;
  int* v1 = odd ? w.list : w.list_tmp;
  if (g.n > 0) {
    int* const order = reinterpret_cast<int*>(k1);  // n_valid <= pairs <= cap_pairs
    // The particle pass's chunk counts lie in the pair offsets, which the scan
    // after it writes: 6 KB a chunk of 8192 particles against 64 KB.  The pairs'
    // scratch would hold few chunks where most particles miss the cube (10M
    // particles, 15k pairs on 64 x 64 x 32: two, binning 4.96 ms; now 0.70).
    const long long chunks = radix_chunks(g.n);
    long long* const off = w.pair_off;
    launch_order_particles(g, w, order, reinterpret_cast<int*>(off + (chunks << RS_BITS)), off, s);
    launch_scan_gather(w.npairs, order, &w.hdr->n_valid, g.n, w.pair_off, w.scan_sums, s);
    k_emit<<<grid_for(g.n, num_sms), 256, 0, s>>>(g, w, order, k0, v0);
  }
  launch_radix_sort(k0, v0, k1, v1, &w.hdr->n_pairs, cap_pairs, bits, w.rs_hist, w.rs_off,
                    w.scan_sums, s);
  k_segments<<<(unsigned)((g.nseg + 7) / 8), 256, 0, s>>>(g, w);
  launch_scan(w.seg_items, g.nseg, w.item_off, w.scan_sums, &w.hdr->n_items, s);
  launch_scan(w.seg_part, g.nseg, w.part_off, w.scan_sums, &w.hdr->n_partial_items, s);
  // the work queue: items by estimated cost, largest first (one pass, into
  // item_key / item_order)
  k_item_keys<<<(unsigned)((g.nseg + 255) / 256), 256, 0, s>>>(g, w);
  launch_radix_sort(w.item_key_tmp, w.item_order_tmp, w.item_key, w.item_order, &w.hdr->n_items,
                    w.cap_items, RS_BITS, w.rs_hist, w.rs_off, w.scan_sums, s);
  k_check_partials<<<1, 1, 0, s>>>(w);
}

}  // namespace mg
