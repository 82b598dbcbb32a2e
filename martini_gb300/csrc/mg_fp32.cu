// Plain FP32 contraction: for each work item (tile, particle chunk, channel
// block) the CTA builds W[32 particles][128 pixels] and S[32][64 channels] in
// shared memory and accumulates out[128][64] += W^T S on CUDA cores.
//
// This is the per-pixel sum of martini/martini.py:243-283 reorganised around
// output tiles: a pixel's spectrum is the sum over the particles whose
// footprint box contains it of weight * spectrum.
//
// Bound by latency: 51 % of issue slots used with three blocks on an SM, warps
// waiting for shared memory and the table's cells most.  A chunk's records
// and spectrum-store rows are copied while the chunk before is multiplied, the
// lines come from the store (once per particle instead of once per tile), the
// weights are taken by whole warps with what a particle's pixels share computed
// once, and the FMAs work on pairs of pixels; three blocks fit on an SM.  100k
// quartic-spline particles on 187 x 211 x 75 (1.44M pairs): 2.09 ms before (1058
// warp instructions a pair, of which 256 multiply), 1.12 ms now (464).
#include "mg_internal.cuh"

namespace mg {

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

constexpr int F32_THREADS = 256;
constexpr int F32_BLOCKS_PER_SM = 3;
constexpr int F32_KC = 32;  // particles per shared-memory chunk
// Floats per particle row of S: every value twice (the FMAs work on pairs of
// pixels and take a channel's value in both halves), the first two channels of
// each thread's four in one half of the row and the others in the other, so
// that a warp's 16-byte reads are contiguous; rows 16 apart in the banks.
constexpr int F32_SROW = 2 * CBLK + 16;
__device__ __forceinline__ int f32_scol(int c) {
  return (c & 2) * (CBLK / 2) + (c >> 2) * 4 + (c & 1) * 2;
}
constexpr int F32_MASTER_BYTES = 32 * F32_THREADS * 4;  // master accumulators (dynamic)

struct ItemInfo {
  int seg, gal, tile, tx, ty, kc, nk;  // tile: within the cube
  int c0;            // first channel of this item's block
  long long lbeg;    // particle list range
  int lcount;
};

__device__ __forceinline__ ItemInfo decode_item(const Geo& g, const Ws& w, long long item,
                                                int kch) {
  ItemInfo it;
  const int sg = w.item_seg[item];
  it.seg = sg;
  it.gal = find_gal(w.gs0, g.ngal, sg);
  const Gal& G = w.gal[it.gal];
  const int ls = sg - G.seg0;
  it.tile = ls / G.ncb;
  const int cb = ls - it.tile * G.ncb;
  it.tx = it.tile / G.nty;
  it.ty = it.tile - it.tx * G.nty;
  it.nk = w.seg_items[sg];
  it.kc = (int)(item - w.item_off[sg]);
  it.c0 = cb * G.width;
  it.lbeg = w.seg_lo[sg] + (long long)it.kc * kch;
  const long long left = w.seg_hi[sg] - it.lbeg;
  it.lcount = (int)(left < kch ? left : kch);
  return it;
}

__global__ void __launch_bounds__(F32_THREADS, F32_BLOCKS_PER_SM)
k_contract_fp32(Geo g, Ws w) {
  __shared__ __align__(16) float Ws_[F32_KC][TILE_PX];
  __shared__ __align__(16) float Ss_[F32_KC][F32_SROW];
  // Master accumulator: each F32_KC-particle chunk is summed from zero in
  // registers and added here (round to nearest).  One running FP32 sum over
  // an item's particles (up to ~10^6 on a dense tile) drops every product
  // below half an ulp of the sum, a loss that only grows with the count; a
  // chunk sum of 32 products meets the master far less often.  Laid out
  // [value][thread] in dynamic shared memory (F32_MASTER_BYTES): each
  // thread's slots are conflict-free.
  extern __shared__ float Ms_dyn[];
  f2(*Ms_)[F32_THREADS] = reinterpret_cast<f2(*)[F32_THREADS]>(Ms_dyn);
  // records of this chunk and, copied meanwhile, of the next
  __shared__ __align__(16) PRec recs2[2][F32_KC];
  __shared__ int s_pid2[2][F32_KC];
  __shared__ long long s_off2[2][F32_KC];  // spectrum-store rows
  __shared__ KSpec s_ks[MG_MAX_KERNELS];
  __shared__ long long s_item;
  __shared__ unsigned s_rank;
  __shared__ int s_next;  // where this block takes its items from (take)

  const int tid = threadIdx.x;
  if (tid < MG_MAX_KERNELS) s_ks[tid] = g.ks[tid];
  const WsHeader* hdr = w.hdr;
  if (hdr->status) return;
  const long long n_items = hdr->n_items;
  // Items fewer than the resident blocks go to as few blocks of an SM as they
  // need: all blocks start at once, and without this some SMs would take three
  // items and others none.  (A rule on blockIdx does not do: consecutive blocks
  // share SMs.)  The first block that starts on an SM always stays.  200k particles
  // on 128 x 128 x 64 (128 items, 239k pairs): contraction 635 us, 444 now; 500k with
  // Dirac kernels and lines (256 items) 592 us, 466 now.
  if (tid == 0) {
    unsigned id;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(id));
    id %= SM_BUCKETS;
    const unsigned sh = 8u * (id & 3u);
    s_rank = (atomicAdd(&w.hdr->sm_blocks[id >> 2], 1u << sh) >> sh) & 255u;
  }
  __syncthreads();
  const int nsm = gridDim.x / F32_BLOCKS_PER_SM;
  if ((long long)s_rank * nsm >= n_items) return;
  // The queue's items in cost order, largest first.  The first nsm of them go to
  // the blocks that are the first of their SM, the next nsm to the second blocks
  // (smallest first) and so on, so that an SM does not start on three large ones
  // while another has three small; then whichever block is free takes the next, and
  // in the end what is left of the first ones.  305k particles with Dirac lines on
  // 98 x 9 x 2406 (items of 1 to 2048 particles): contraction 835 us with one
  // cursor, 700 now.
  auto first_item = [&](int r) -> long long {  // of the blocks that are the r-th of their SM
    const long long m = min((long long)nsm, n_items - (long long)r * nsm);
    const int sh = 21 * r;
    const long long c = (atomicAdd(&w.hdr->first_items, 1ull << sh) >> sh) & 0x1fffffull;
    return c < m ? (long long)r * nsm + (r == 1 ? m - 1 - c : c) : -1;
  };
  auto take = [&]() -> long long {  // by one thread; n_items: none left
    if (s_next < 0) {
      s_next = 0;
      const long long f = s_rank < F32_BLOCKS_PER_SM ? first_item((int)s_rank) : -1;
      if (f >= 0) return f;
    }
    if (s_next == 0) {
      const long long q = (long long)F32_BLOCKS_PER_SM * nsm +
                          (long long)atomicAdd(&w.hdr->item_counter, 1u);
      if (q < n_items) return q;
      s_next = 1;
    }
    for (; s_next <= F32_BLOCKS_PER_SM; ++s_next) {
      const long long f = first_item(s_next - 1);
      if (f >= 0) return f;
    }
    return n_items;
  };
  if (tid == 0) s_next = -1;
  const int kch = hdr->kch;
  const unsigned* spec = stored_lines(g.spectral_model) && w.cap_spec > 0 && hdr->spec_ready
                             ? w.spec
                             : nullptr;
  const int warp = tid >> 5, lane = tid & 31;
  const int tr = tid >> 4;  // pixel group: pixels tr*8 .. tr*8+7
  const int tc = tid & 15;  // channel group: channels tc*4 .. tc*4+3

  for (;;) {
    if (tid == 0) s_item = take();
    __syncthreads();
    const long long item = s_item;
    __syncthreads();
    if (item >= n_items) break;
    // the queue runs over the items in cost order, largest first
    const ItemInfo it = decode_item(g, w, (long long)w.item_order[item], kch);
    const Gal& G = w.gal[it.gal];
    const int dec = w.gst[it.gal].dec;
    const int nc = G.nc;
    const float* ehi = w.ehi + G.edge0;
    const float* elo = w.elo + G.edge0;
    const float* inv_w = w.inv_w + G.edge0;
    const int i0 = it.tx * TILE_I, j0 = it.ty * TILE_J;

    f2 acc2[4][4];  // pixel pairs x channels
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc2[a][b] = 0ull;
#pragma unroll
    for (int v = 0; v < 16; ++v) Ms_[v][tid] = 0ull;

    // The records of the chunk at kb, whose list entries lie in s_pid2[b], into
    // buffer b by asynchronous copies of 8 bytes, the last piece the particle's
    // spectrum-store row; an empty box past the list's end.
    auto recs_in = [&](int kb, int b) {
      constexpr int PIECES = sizeof(PRec) / 8 + 1;
      static_assert(sizeof(PRec) % 8 == 0, "record copy");
      for (int e = tid; e < F32_KC * PIECES; e += F32_THREADS) {
        const int q = e / PIECES, piece = e - q * PIECES;
        if (kb + q < it.lcount) {
          const int pid = s_pid2[b][q];
          if (piece + 1 < PIECES)
            cp_async8(reinterpret_cast<char*>(&recs2[b][q]) + 8 * piece,
                      reinterpret_cast<const char*>(w.rec + pid) + 8 * piece);
          else
            cp_async8(&s_off2[b][q], w.pair_off + pid);
        } else if (piece == 0) {
          PRec& z = recs2[b][q];
          z.ilo = 0; z.ihi = -1; z.jlo = 0; z.jhi = -1; z.clo = 0; z.chi = -1;  // hits no block
          z.xi = z.yi = 0; z.xf = z.yf = 0.f; z.h = 1.f; z.inv_h2 = 1.f;
          z.kslot = 0; z.flags = 0;
        }
      }
    };
    if (tid < 2 * F32_KC && tid < it.lcount)
      s_pid2[tid / F32_KC][tid % F32_KC] = w.list[it.lbeg + tid];
    __syncthreads();
    recs_in(0, 0);
    cp_async_wait();
    for (int k0 = 0, b = 0; k0 < it.lcount; k0 += F32_KC, b ^= 1) {
      const int kn = min(F32_KC, it.lcount - k0);
      const PRec* recs = recs2[b];
      const int* s_pid = s_pid2[b];
      const long long* s_off = s_off2[b];
      __syncthreads();
      recs_in(k0 + F32_KC, b ^ 1);
      // the list entries of the chunk after next, stored at this chunk's end
      const int ahead = k0 + 2 * F32_KC + tid;
      const int next_pid = tid < F32_KC && ahead < it.lcount ? w.list[it.lbeg + ahead] : 0;
      {
        // W: four particles a warp, two tile rows (32 pixels) at a time, so
        // that a warp's stores are contiguous and rows past a particle's box
        // cost nothing
#pragma unroll 1
        for (int e = 0; e < F32_KC / 8; ++e) {
          const int q = warp * (F32_KC / 8) + e;
          const PRec& r = recs[q];
          // a particle listed for this block whose line misses it (the list
          // bound is conservative) contributes nothing: no weights
          const bool hit = r.chi >= it.c0 && r.clo < it.c0 + CBLK;
          const int kt = s_ks[r.kslot].type;
          const int i = i0 + (lane >> 4), j = j0 + (lane & 15);
          if (hit && kt <= MG_KERNEL_QUARTIC_SPLINE && kt != MG_KERNEL_CUBIC_SPLINE) {
            // kernels with cells in s: pixel_weight's arithmetic with what the
            // four pixels share (column, table, box test) taken once
            const KTableInfo& inf = kt_info[kt];
            const float cpu = inf.reg[0].cells_per_unit, cap = (float)inf.reg[0].ncell;
            const float4* tab = reinterpret_cast<const float4*>(kt_coef) + inf.reg[0].first;
            const float scale = inf.scale, inv_h2 = r.inv_h2;
            const float dy = (float)(r.yi - j) + r.yf;
            const float xi = (float)(r.xi - i);  // exact, as are the steps of 2 below
            const int ilo = r.jlo <= j && j <= r.jhi ? r.ilo : 0x7fffffff, ihi = r.ihi;
#pragma unroll
            for (int h = 0; h < TILE_I / 2; ++h) {
              const float dx = (xi - (float)(2 * h)) + r.xf;
              const float r2 = dx * dx + dy * dy;
              const float u = fminf(r2 * inv_h2 * cpu, cap);
              float t;
              const int c = kt_floor(u, t);
              const float4 cf = __ldg(tab + c);
              const float f = fmaf(fmaf(fmaf(cf.w, t, cf.z), t, cf.y), t, cf.x);
              Ws_[q][h * 32 + lane] =
                  i + 2 * h >= ilo && i + 2 * h <= ihi ? f * scale * inv_h2 : 0.f;
            }
          } else if (hit && kt == MG_KERNEL_GAUSSIAN) {
            // w_gaussian's arithmetic; its row factors (lane l computes that of
            // row l mod 8) and column factors are shared by the 128 pixels: 8
            // error functions a lane instead of 20
            const float trunc = s_ks[r.kslot].truncate, ign = 1.f / s_ks[r.kslot].gnorm;
            const float inv_hs = 1.f / (r.h * 0.42466090014400953f);
            const float sg = inv_hs * 0.70710678118654752f;
            const float dy = (float)(r.yi - j) + r.yf;
            const float ey = erff((dy + 0.5f) * sg) - erff((dy - 0.5f) * sg);
            const float dxr = (float)(r.xi - (i0 + (lane & 7))) + r.xf;
            const float exr = erff((dxr + 0.5f) * sg) - erff((dxr - 0.5f) * sg);
            const bool in_j = r.jlo <= j && j <= r.jhi;
#pragma unroll
            for (int h = 0; h < TILE_I / 2; ++h) {
              const int row = 2 * h + (lane >> 4);
              const float ex = __shfl_sync(0xffffffffu, exr, row);
              const float dx = (float)(r.xi - (i0 + row)) + r.xf;
              const float dr = sqrtf(dx * dx + dy * dy);
              const float q = dr * inv_hs;
              const float zmax = trunc > q ? sqrtf(trunc * trunc - q * q) : 0.f;
              const float f = 0.25f * erff(zmax * 0.70710678118654752f) * ex * ey * ign;
              const bool in = in_j && i0 + row >= r.ilo && i0 + row <= r.ihi &&
                              !((dr - 0.70710678118654752f) * inv_hs > trunc);
              Ws_[warp * (F32_KC / 8) + e][h * 32 + lane] = in ? f : 0.f;
            }
          } else {
#pragma unroll
            for (int h = 0; h < TILE_I / 2; ++h) {
              float v = 0.f;
              if (hit && r.ilo <= i0 + 2 * h + 1 && r.ihi >= i0 + 2 * h)
                v = pixel_weight(r, s_ks, i + 2 * h, j);
              Ws_[q][h * 32 + lane] = v;
            }
          }
        }
        // S: particle q, every eighth channel of the block
        const int q = tid >> 3, ii = tid & 7;
        const PRec& r = recs[q];
        const unsigned* row = spec && q < kn ? spec + s_off[q] - r.clo : nullptr;
        if (g.spectral_model == MG_SPECTRUM_TABLE) {
          // all loads in flight at once: rows of a table far larger than the
          // caches are not fetched ahead (Dirac kernels, 162k spectra on 30 x 19 x
          // 616: contraction 1252 us with a load at a time, 862 now)
          const float* tab = G.spectra + ((long long)s_pid[q] - G.p0) * nc + it.c0 + ii;
          const int left = q < kn ? nc - it.c0 - ii : 0;
          float v[CBLK / 8];
#pragma unroll
          for (int k = 0; k < CBLK / 8; ++k) v[k] = 8 * k < left ? tab[8 * k] : 0.f;
#pragma unroll
          for (int k = 0; k < CBLK / 8; ++k)
            *reinterpret_cast<float2*>(&Ss_[q][f32_scol(ii + 8 * k)]) = make_float2(v[k], v[k]);
        } else {
          for (int cc = ii; cc < CBLK; cc += 8) {
            const int c = it.c0 + cc;
            float s = 0.f;
            if (c < nc && q < kn) {
              if (spec) {
                if (c >= r.clo && c <= r.chi) s = __uint_as_float(__ldg(row + c));
              } else {
                s = channel_spectrum(r, g.spectral_model, c, dec, ehi, elo, inv_w);
              }
            }
            *reinterpret_cast<float2*>(&Ss_[q][f32_scol(cc)]) = make_float2(s, s);
          }
        }
      }
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < F32_KC; ++k) {
        const ulonglong2 wa = *reinterpret_cast<const ulonglong2*>(&Ws_[k][tr * 8]);
        const ulonglong2 wb = *reinterpret_cast<const ulonglong2*>(&Ws_[k][tr * 8 + 4]);
        const ulonglong2 sa = *reinterpret_cast<const ulonglong2*>(&Ss_[k][tc * 4]);
        const ulonglong2 sb = *reinterpret_cast<const ulonglong2*>(&Ss_[k][CBLK + tc * 4]);
        const f2 wv[4] = {wa.x, wa.y, wb.x, wb.y};
        const f2 sv[4] = {sa.x, sa.y, sb.x, sb.y};
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc2[a][b] = f2_fma(wv[a], sv[b], acc2[a][b]);
      }
      // chunk sum into the master, registers back to zero
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          Ms_[a * 4 + b][tid] = f2_add(Ms_[a * 4 + b][tid], acc2[a][b]);
          acc2[a][b] = 0ull;
        }
      if (tid < F32_KC) s_pid2[b][tid] = next_pid;
      cp_async_wait();
    }
    __syncthreads();
    float acc[8][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const float2 m = f2_split(Ms_[a * 4 + b][tid]);
        acc[2 * a][b] = m.x;
        acc[2 * a + 1][b] = m.y;
      }

    // epilogue: direct cube write (single K chunk) or split-K partial
    if (it.nk == 1) {
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const int px = tr * 8 + a;
        const int i = i0 + px / TILE_J, j = j0 + px % TILE_J;
        if (i >= G.nx || j >= G.ny) continue;
        float* dst = G.cube + ((long long)i * G.ny + j) * nc;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int c = it.c0 + tc * 4 + b;
          if (c < nc) dst[c] = g.accumulate ? dst[c] + acc[a][b] : acc[a][b];
        }
      }
    } else {
      const long long slot = w.part_off[it.seg] + it.kc;
      float* dst = w.partial + slot * (long long)(TILE_PX * g.max_width);
      if (tid == 0) w.item_key[w.item_order[item]] = part_window(0, CBLK);
#pragma unroll
      for (int a = 0; a < 8; ++a) {
        const int px = tr * 8 + a;
        *reinterpret_cast<float4*>(&dst[px * CBLK + tc * 4]) =
            make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
      }
    }
  }
}

// Split-K reduction, shared by every form: a segment with nk > 1 work items
// left nk partial rows of TILE_PX x seg_width floats (pixel-major), of which
// an item wrote the channels of its window only (item_key, part_window).  A
// block takes one chunk of RED_CHUNK floats of the split segments among
// RED_SEGS: its lanes look them up at once, because few segments are split
// and a block that visited every (segment, chunk) alone spent its time on
// the lookups (4M particles in 1024^2 x 512: 0.45 ms, 0.04 ms now).  The RED_SEGS
// lie a grid's length apart, so that dense neighbouring tiles go to different
// blocks.  Each thread sums four channels of one pixel over the rows in
// ascending row order, so the result does not depend on scheduling, with
// RED_ROWS float4 loads in flight.
constexpr int RED_THREADS = 256;
constexpr int RED_CHUNK = RED_THREADS * 4;
constexpr int RED_ROWS = 8;
constexpr int RED_SEGS = 32;

__device__ __forceinline__ void reduce_chunk(const Geo& g, const Ws& w, int sg, int nk,
                                             int chunk) {
  const long long slot = (long long)TILE_PX * g.max_width;  // floats per partial row
  const int gk = find_gal(w.gs0, g.ngal, sg);
  const Gal& G = w.gal[gk];
  const int width = G.width;  // a multiple of 16 channels
  const int e = chunk * RED_CHUNK + threadIdx.x * 4;
  if (e >= TILE_PX * width) return;
  const int px = e / width, cl = e - px * width;
  const unsigned* win = w.item_key + w.item_off[sg];
  const float4* src = reinterpret_cast<const float4*>(w.partial + w.part_off[sg] * slot + e);
  const long long row4 = slot / 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < nk; k0 += RED_ROWS) {
    float4 v[RED_ROWS];
#pragma unroll
    for (int q = 0; q < RED_ROWS; ++q)
      if (k0 + q < nk) {
        const unsigned pw = win[k0 + q];  // the row's channels [low half, high half)
        v[q] = (unsigned)cl - (pw & 0xFFFFu) < (pw >> 16) - (pw & 0xFFFFu)
                   ? __ldcs(src + (long long)(k0 + q) * row4)
                   : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
    for (int q = 0; q < RED_ROWS; ++q)
      if (k0 + q < nk) {
        acc.x += v[q].x;
        acc.y += v[q].y;
        acc.z += v[q].z;
        acc.w += v[q].w;
      }
  }
  const int ls = sg - G.seg0;
  const int t = ls / G.ncb;
  const int cb = ls - t * G.ncb;
  const int tx = t / G.nty, ty = t - tx * G.nty;
  const int c = cb * width + cl;
  const int i = tx * TILE_I + px / TILE_J, j = ty * TILE_J + px % TILE_J;
  if (i >= G.nx || j >= G.ny) return;
  const int nc = G.nc;
  float* dst = G.cube + ((long long)i * G.ny + j) * nc + c;
  if (g.accumulate) {
    if (c < nc) acc.x += dst[0];
    if (c + 1 < nc) acc.y += dst[1];
    if (c + 2 < nc) acc.z += dst[2];
    if (c + 3 < nc) acc.w += dst[3];
  }
  if (c < nc) dst[0] = acc.x;
  if (c + 1 < nc) dst[1] = acc.y;
  if (c + 2 < nc) dst[2] = acc.z;
  if (c + 3 < nc) dst[3] = acc.w;
}

__global__ void __launch_bounds__(RED_THREADS) k_reduce_partials(Geo g, Ws w) {
  if (w.hdr->status) return;
  const int nchunk = (TILE_PX * g.max_width + RED_CHUNK - 1) / RED_CHUNK;
  const int ngrp = (g.nseg + RED_SEGS - 1) / RED_SEGS;
  const long long units = (long long)ngrp * nchunk;
  const int lane = threadIdx.x & 31;
  for (long long u = blockIdx.x; u < units; u += gridDim.x) {
    const int grp = (int)(u / nchunk), chunk = (int)(u - (long long)grp * nchunk);
    const long long mine = grp + (long long)lane * ngrp;
    const int nk = mine < g.nseg ? w.seg_part[mine] : 0;
    for (unsigned m = __ballot_sync(0xffffffffu, nk > 0); m; m &= m - 1) {
      const int l = __ffs(m) - 1;
      const int n = __shfl_sync(0xffffffffu, nk, l);
      reduce_chunk(g, w, grp + l * ngrp, n, chunk);
      __syncwarp();
    }
  }
}

void launch_reduce_partials(const Geo& g, const Ws& w, int num_sms, cudaStream_t s) {
  k_reduce_partials<<<num_sms * 8, RED_THREADS, 0, s>>>(g, w);
}

// Flux sums over the unpadded region (martini/martini.py:367-392), in a
// fixed order: per pixel row (one block per row of the unpadded region, a
// thread per channel) in double-float, then the row sums in FP64 in row
// order.
constexpr int FLUX_ROWS = 1;  // pixel rows (axis 0) per chunk

// Double-float running sum (Knuth's TwoSum): hi carries the FP32 sum and lo
// the rounding errors of its additions, so hi + lo is the sum to ~n eps^2
// without FP64 arithmetic (FP64 units are few on this part).
struct DFloat {
  float hi, lo;
};

__device__ __forceinline__ void df_add(DFloat& a, float x) {
  const float t = __fadd_rn(a.hi, x);
  const float bp = __fadd_rn(t, -a.hi);
  const float e = __fadd_rn(__fadd_rn(a.hi, -__fadd_rn(t, -bp)), __fadd_rn(x, -bp));
  a.hi = t;
  a.lo = __fadd_rn(a.lo, e);
}

// Sum of one pixel row's voxels of channel c (stride nc), j in [j0, j1), in
// a fixed order: four interleaved double-float sums combined in FP64.
__device__ __forceinline__ double row_sum(const float* row, int j0, int j1, int nc) {
  DFloat a[4] = {{0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}, {0.f, 0.f}};
  int j = j0;
  for (; j + 4 <= j1; j += 4) {
    float x[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) x[u] = __ldcs(row + (long long)(j + u) * nc);
#pragma unroll
    for (int u = 0; u < 4; ++u) df_add(a[u], x[u]);
  }
  for (; j < j1; ++j) df_add(a[0], __ldcs(row + (long long)j * nc));
  double acc = 0.0;
#pragma unroll
  for (int u = 0; u < 4; ++u) acc += (double)a[u].hi + (double)a[u].lo;
  return acc;
}

__global__ void k_flux_partial(const float* __restrict__ cube, int nx, int ny, int nc, int padx,
                               int pady, double* __restrict__ part) {
  const int chunk = blockIdx.x;
  const int i0 = padx + chunk * FLUX_ROWS;
  const int i1 = min(nx - padx, i0 + FLUX_ROWS);
  for (int c = threadIdx.x; c < nc; c += blockDim.x) {
    double acc = 0.0;
    for (int i = i0; i < i1; ++i) acc += row_sum(cube + ((long long)i * ny) * nc + c, pady, ny - pady, nc);
    part[(long long)chunk * nc + c] = acc;
  }
}

__global__ void k_flux_final(const double* __restrict__ part, int nchunks, int nc,
                             double* __restrict__ flux) {
  __shared__ double red[1024];
  double tot = 0.0;
  for (int c = threadIdx.x; c < nc; c += blockDim.x) {
    double s = 0.0;
    for (int k = 0; k < nchunks; ++k) s += part[(long long)k * nc + c];
    flux[1 + c] = s;
    tot += s;
  }
  red[threadIdx.x] = tot;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) flux[0] = red[0];
}

int flux_chunks(int nx, int padx) {
  int rows = nx - 2 * padx;
  if (rows < 1) rows = 1;
  return (rows + FLUX_ROWS - 1) / FLUX_ROWS;
}

void launch_flux(const float* cube, int nx, int ny, int nc, int padx, int pady, double* part,
                 double* flux, cudaStream_t s) {
  const int nch = flux_chunks(nx, padx);
  const int thr = nc < 256 ? ((nc + 31) / 32) * 32 : 256;
  k_flux_partial<<<nch, thr, 0, s>>>(cube, nx, ny, nc, padx, pady, part);
  k_flux_final<<<1, 1024, 0, s>>>(part, nch, nc, flux);
}

int launch_contract_fp32(const Geo& g, const Ws& w, int num_sms, cudaStream_t s) {
  // the dynamic shared-memory attribute is per device: set once on each
  // (host-side, before a graph capture by the first insertion on a device)
  constexpr int kMaxDev = 64;
  static bool attr_set[kMaxDev] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDev) return MG_ERR_CUDA;
  if (!attr_set[dev]) {
    if (cudaFuncSetAttribute(k_contract_fp32, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             F32_MASTER_BYTES) != cudaSuccess)
      return MG_ERR_CUDA;
    attr_set[dev] = true;
  }
  k_contract_fp32<<<num_sms * F32_BLOCKS_PER_SM, F32_THREADS, F32_MASTER_BYTES, s>>>(g, w);
  launch_reduce_partials(g, w, num_sms, s);
  return MG_OK;
}

// Flux sums of every cube of a batch: one block per unpadded pixel row of
// all cubes, a thread per channel adding the row's voxels in a fixed order
// (four interleaved double-float sums, combined in FP64), then per cube and
// channel eight row groups (rows r = g mod 8) summed in FP64 and combined in
// group order, and one block per cube adding the channels.
__global__ void k_flux_rows(Geo g, Ws w) {
  const int gk = find_gal(w.gr0, g.ngal, (int)blockIdx.x);
  const Gal& G = w.gal[gk];
  if (!G.flux) return;
  const int r = blockIdx.x - G.row0;
  const int i = G.padx + r;
  const int nc = G.nc;
  const int j1 = G.ny - G.pady;
  for (int c = threadIdx.x; c < nc; c += blockDim.x)
    w.flux_part[G.fpart0 + (long long)r * nc + c] =
        row_sum(G.cube + ((long long)i * G.ny) * nc + c, G.pady, j1, nc);
}

constexpr int FLUX_CH = 32;  // channels per block of k_flux_channels
constexpr int FLUX_RG = 8;   // row groups per block: rows r = g (mod FLUX_RG)

__global__ void __launch_bounds__(FLUX_CH * FLUX_RG) k_flux_channels(Geo g, Ws w) {
  __shared__ double part[FLUX_RG][FLUX_CH];
  const Gal& G = w.gal[blockIdx.y];
  if (!G.flux) return;
  const int cl = threadIdx.x % FLUX_CH, rg = threadIdx.x / FLUX_CH;
  const int c = blockIdx.x * FLUX_CH + cl;
  const int rows = G.nx - 2 * G.padx;
  double s = 0.0;
  if (c < G.nc)
    for (int r = rg; r < rows; r += FLUX_RG) s += w.flux_part[G.fpart0 + (long long)r * G.nc + c];
  part[rg][cl] = s;
  __syncthreads();
  if (rg == 0 && c < G.nc) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < FLUX_RG; ++k) t += part[k][cl];
    G.flux[1 + c] = t;
  }
}

__global__ void k_flux_cubes(Geo g, Ws w) {
  __shared__ double red[256];
  const Gal& G = w.gal[blockIdx.x];
  if (!G.flux) return;
  double tot = 0.0;
  for (int c = threadIdx.x; c < G.nc; c += blockDim.x) tot += G.flux[1 + c];
  red[threadIdx.x] = tot;
  __syncthreads();
  for (int off = blockDim.x / 2; off > 0; off >>= 1) {
    if (threadIdx.x < off) red[threadIdx.x] += red[threadIdx.x + off];
    __syncthreads();
  }
  if (threadIdx.x == 0) G.flux[0] = red[0];
}

void launch_flux_batch(const Geo& g, const Ws& w, cudaStream_t s) {
  if (g.nrows <= 0) return;
  const int thr = g.max_nc < 256 ? ((g.max_nc + 31) / 32) * 32 : 256;
  k_flux_rows<<<g.nrows, thr, 0, s>>>(g, w);
  k_flux_channels<<<dim3((unsigned)((g.max_nc + FLUX_CH - 1) / FLUX_CH), (unsigned)g.ngal),
                    FLUX_CH * FLUX_RG, 0, s>>>(g, w);
  k_flux_cubes<<<g.ngal, 256, 0, s>>>(g, w);
}

}  // namespace mg
