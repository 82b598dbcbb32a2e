// Global profile: the spatially integrated spectrum of a source
// (GlobalProfile.insert_source_in_spectrum, martini/martini.py:1551-1596).
//
// The reference inserts every particle that survives spectral and mass
// pruning into a one-pixel cube with a DiracDeltaKernel of infinite range at
// pixel (0, 0), so each particle's weight is 1 and the spectrum in Jy is
// spectrum[c] = sum_p S_p(c).  Here that sum is formed directly.  A warp takes
// 32 particles at a time: each lane finds one particle's line (channel support
// by the same FP64 search as the cube path), then the lanes evaluate the lines
// one after the other over their supports only and add them, in FP64 and in
// particle order, to the warp's own spectrum in shared memory.  Channel c
// belongs to lane c mod 32, so no two lanes meet.  The warps' spectra are added
// in warp order, the blocks' in a fixed order, so the result is deterministic.
// Bound by the FP64 pipe (75 % busy: a conversion and an addition for each
// particle and channel; 67 % of issue slots, the error functions among them).
// Before, a thread per channel walked every particle of its block, and 1,000,000
// particles on 256 channels took 1.01 ms; now 0.36 ms a call, 0.27 ms in the sum.
// A warp's lines are one chain, so where there are few particles they are dealt
// to more blocks and all warps, and the band to blocks of channels (which also
// keeps eight warps' spectra in shared memory whatever the band).  With whole
// bands and 1024 particles a block, 400 lines across 8192 channels took 15.5 ms a
// call and 32 across 256 143 us (1.9 ms and 81 us with a thread per channel);
// 130 and 67 us now, 20k lines of 28 channels 118 and 74 us.
#include <algorithm>
#include <string>

#include "mg_internal.cuh"

namespace mg {
void set_last_error(const std::string& msg);  // mg_api.cu
}

namespace {

using namespace mg;

constexpr int PROF_WARPS = 8;          // warps per block
constexpr int PROF_PER_BLOCK = 1024;   // most particles per block, while the blocks suffice
constexpr int PROF_MAX_BLOCKS = 2048;
constexpr int PROF_FILL = 152;         // blocks that fill the chip's SMs
constexpr long long PROF_PART = 1 << 22;  // partial sums (32 MB) that more blocks may take
constexpr int PROF_CHUNK = 1536;       // most channels per block: 96 KB of the warps' spectra
constexpr int PROF_MIN_CHUNK = 64;
constexpr int PROF_CH = 32, PROF_GROUPS = 16;  // channels, block groups of k_profile_final

struct ProfWs {
  WsHeader* hdr;
  float* ehi;
  float* elo;
  float* inv_w;
  int* dec;
  double* part;  // [blocks][nc]
};

size_t al(size_t x) { return (x + 255) & ~size_t(255); }

// Particle ranges, a block (or one per channel chunk) each: PROF_PER_BLOCK
// particles, fewer while that leaves SMs idle, but one for each warp.
int prof_blocks(long long n, int nc) {
  const long long full = (n + PROF_PER_BLOCK - 1) / PROF_PER_BLOCK;
  long long b = std::min<long long>((n + PROF_WARPS - 1) / PROF_WARPS, 2 * PROF_FILL);
  b = std::max(std::min(b, PROF_PART / nc), full);
  b = std::min<long long>(b, PROF_MAX_BLOCKS);
  return (int)(b > 0 ? b : 1);
}

// Channels of a block's chunk: the band in equal chunks of at most PROF_CHUNK,
// smaller while the blocks do not fill the chip.
int prof_chunk(int nc, int blocks) {
  long long k = (nc + PROF_CHUNK - 1) / PROF_CHUNK;
  const long long fill = (PROF_FILL + blocks - 1) / blocks;
  k = std::max<long long>(k, std::min<long long>(fill, (nc + PROF_MIN_CHUNK - 1) / PROF_MIN_CHUNK));
  return (int)(((nc + k - 1) / k + 31) / 32 * 32);
}

size_t prof_layout(long long n, int nc, size_t* off) {
  size_t o = 0;
  off[0] = o; o += al(sizeof(WsHeader));
  off[1] = o; o += al(sizeof(float) * (size_t)(nc + 1));
  off[2] = o; o += al(sizeof(float) * (size_t)(nc + 1));
  off[3] = o; o += al(sizeof(float) * (size_t)(nc + 1));
  off[4] = o; o += al(sizeof(int));
  off[5] = o; o += al(sizeof(double) * (size_t)prof_blocks(n, nc) * nc);
  return o;
}

__global__ void k_profile_edges(const double* __restrict__ e, int nc, ProfWs w) {
  const int dec = e[nc] < e[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    w.hdr->status = 0;
    *w.dec = dec;
  }
  __syncthreads();
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k <= nc; k += gridDim.x * blockDim.x) {
    const double v = e[k];
    const float hi = (float)v;
    w.ehi[k] = hi;
    w.elo[k] = (float)(v - (double)hi);
    if (k < nc) {
      w.inv_w[k] = (float)(1.0 / fabs(e[k + 1] - e[k]));
      const bool mono = dec ? (e[k + 1] < e[k]) : (e[k + 1] > e[k]);
      if (!mono) atomicOr(&w.hdr->status, ST_EDGES);
    }
  }
}

// erfc(|u|) and the sign of u at edge e of a Gaussian line.
__device__ __forceinline__ float profile_edge(float vhi, float vlo, float inv_s, int e,
                                              const ProfWs& w, bool& pos) {
  const float u = ((w.ehi[e] - vhi) + (w.elo[e] - vlo)) * inv_s;
  pos = u >= 0.f;
  return erfcf(fabsf(u));
}

// Block (x, y): particle range x, channels [y chunk, (y + 1) chunk).
__global__ void __launch_bounds__(PROF_WARPS * 32)
k_profile_sum(long long n, int nc, int chunk, int model, const double* __restrict__ v,
              const float* __restrict__ sigma, float sigma_const,
              const double* __restrict__ amp, const double* __restrict__ edges, ProfWs w) {
  extern __shared__ double s_acc[];  // [warp][chunk]
  if (w.hdr->status) return;
  const int dec = *w.dec;
  const ChanGrid grid(edges, nc, dec);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int c0 = blockIdx.y * chunk, c1 = min(c0 + chunk, nc);
  double* const acc = s_acc + (size_t)warp * chunk - c0;  // this warp's, by channel
  for (int c = c0 + lane; c < c1; c += 32) acc[c] = 0.0;
  const long long per = (n + gridDim.x - 1) / gridDim.x;
  const long long p1 = min((long long)(blockIdx.x + 1) * per, n);
  // particles a warp takes at a time: all warps' shares where the range is short
  const int at = (int)min(32ll, (per + nw - 1) / nw);
  // a lane only ever touches its own channels (c0 is a multiple of 32): no
  // barrier between particles
  for (long long p0 = (long long)blockIdx.x * per + warp * at; p0 < p1; p0 += at * nw) {
    const long long p = p0 + lane;
    float vhi = 0.f, vlo = 0.f, inv_s = 0.f, am = 0.f;
    int clo = 1, chi = 0;
    if (lane < at && p < p1) {
      const double vp = v[p], a = amp[p];
      const double vh = (double)(float)vp;
      vhi = (float)vh;
      vlo = (float)(vp - vh);
      am = (float)a;
      if (model == MG_SPECTRUM_GAUSSIAN) {
        const double s = sigma ? (double)sigma[p] : (double)sigma_const;
        inv_s = (float)(1.0 / (1.4142135623730951 * s));
        const double half = 4.5 * 1.4142135623730951 * s;
        const float half_f = (float)half;
        channel_range(edges, nc, dec, grid, vp - half, vp + half, vhi - half_f, vhi + half_f, clo,
                      chi);
      } else {
        channel_range(edges, nc, dec, grid, vp, vp, vhi, vhi, clo, chi);
      }
      if (a == 0.0 || !isfinite(vp)) {  // mass pruning (martini.py:168-241)
        clo = 1;
        chi = 0;
      }
      clo = max(clo, c0);
      chi = min(chi, c1 - 1);
    }
    const int m = (int)min((long long)at, p1 - p0);
    for (int k = 0; k < m; ++k) {
      const int a = __shfl_sync(0xffffffffu, clo, k), b = __shfl_sync(0xffffffffu, chi, k);
      if (a > b) continue;
      const float qa = __shfl_sync(0xffffffffu, am, k);
      if (model == MG_SPECTRUM_DIRAC) {
        for (int c = a + ((lane - a) & 31); c <= b; c += 32)
          acc[c] += (double)(qa * w.inv_w[c]);
        continue;
      }
      const float qh = __shfl_sync(0xffffffffu, vhi, k), ql = __shfl_sync(0xffffffffu, vlo, k);
      const float qs = __shfl_sync(0xffffffffu, inv_s, k);
      // 31 channels at a time: a lane evaluates its channel's edge and takes
      // the next edge from the next lane
      for (int base = a; base <= b; base += 31) {
        const int c = base + ((lane - base) & 31);
        bool pa;
        const float ca = profile_edge(qh, ql, qs, min(c, nc), w, pa);
        const float cb = __shfl_sync(0xffffffffu, ca, (lane + 1) & 31);
        const bool pb = __shfl_sync(0xffffffffu, (int)pa, (lane + 1) & 31) != 0;
        if (c < base + 31 && c <= b) {
          // 0.5 [erf(upper) - erf(lower)]; edge c is the lower one for
          // increasing edges
          const float x = dec ? cb : ca, y = dec ? ca : cb;
          const bool px = dec ? pb : pa, py = dec ? pa : pb;
          const float phi =
              (px || !py) ? 0.5f * (px ? x - y : y - x) : fmaf(-0.5f, x + y, 1.f);
          acc[c] += (double)(qa * phi * w.inv_w[c]);
        }
      }
    }
  }
  __syncthreads();
  for (int c = c0 + threadIdx.x; c < c1; c += blockDim.x) {
    double t = 0.0;
    for (int k = 0; k < nw; ++k) t += s_acc[(size_t)k * chunk + (c - c0)];
    w.part[(size_t)blockIdx.x * nc + c] = t;
  }
}

// Block partials: PROF_CH channels a block, the partial rows over PROF_GROUPS
// groups (rows r = g mod PROF_GROUPS), then the groups in order.
__global__ void __launch_bounds__(PROF_CH * PROF_GROUPS)
k_profile_final(int nblocks, int nc, ProfWs w, double* __restrict__ spectrum) {
  __shared__ double part[PROF_GROUPS][PROF_CH];
  if (w.hdr->status) return;
  const int cl = threadIdx.x % PROF_CH, g = threadIdx.x / PROF_CH;
  const int c = blockIdx.x * PROF_CH + cl;
  double s = 0.0;
  if (c < nc)
    for (int b = g; b < nblocks; b += PROF_GROUPS) s += w.part[(long long)b * nc + c];
  part[g][cl] = s;
  __syncthreads();
  if (g == 0 && c < nc) {
    double t = 0.0;
#pragma unroll
    for (int k = 0; k < PROF_GROUPS; ++k) t += part[k][cl];
    spectrum[c] = t;
  }
}

}  // namespace

extern "C" size_t mg_global_profile_workspace_size(int64_t n, int32_t nc) {
  size_t off[6];
  return prof_layout(n, nc > 0 ? nc : 1, off);
}

extern "C" int mg_global_profile(const mg_problem* p, double* spectrum, void* workspace,
                                 size_t workspace_bytes, void* stream) {
  if (!p || !spectrum || !p->edges || p->nc <= 0 || p->n < 0) {
    mg::set_last_error("mg_global_profile: invalid arguments");
    return MG_ERR_INVALID_ARGUMENT;
  }
  if (p->spectral_model != MG_SPECTRUM_GAUSSIAN && p->spectral_model != MG_SPECTRUM_DIRAC) {
    mg::set_last_error("mg_global_profile: GAUSSIAN or DIRAC spectral model");
    return MG_ERR_INVALID_ARGUMENT;
  }
  if (p->n > 0 && (!p->v || !p->amp ||
                   (p->spectral_model == MG_SPECTRUM_GAUSSIAN && !p->sigma &&
                    !(p->sigma_const > 0.f)))) {
    mg::set_last_error("mg_global_profile: v, amp and (Gaussian) sigma are required");
    return MG_ERR_INVALID_ARGUMENT;
  }
  size_t off[6];
  const size_t need = prof_layout(p->n, p->nc, off);
  if (!workspace || workspace_bytes < need) {
    mg::set_last_error("mg_global_profile: workspace too small: need " + std::to_string(need));
    return MG_ERR_WORKSPACE;
  }
  char* b = static_cast<char*>(workspace);
  ProfWs w;
  w.hdr = reinterpret_cast<WsHeader*>(b + off[0]);
  w.ehi = reinterpret_cast<float*>(b + off[1]);
  w.elo = reinterpret_cast<float*>(b + off[2]);
  w.inv_w = reinterpret_cast<float*>(b + off[3]);
  w.dec = reinterpret_cast<int*>(b + off[4]);
  w.part = reinterpret_cast<double*>(b + off[5]);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(w.hdr, 0, sizeof(WsHeader), s);
  if (e != cudaSuccess) {
    mg::set_last_error(std::string("mg_global_profile: ") + cudaGetErrorString(e));
    return MG_ERR_CUDA;
  }
  // one block, so the edge direction is known before the range checks
  k_profile_edges<<<1, 256, 0, s>>>(p->edges, p->nc, w);
  const int nb = prof_blocks(p->n, p->nc);
  if (p->n > 0) {
    const int chunk = prof_chunk(p->nc, nb);
    const size_t smem = sizeof(double) * (size_t)PROF_WARPS * chunk;
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(k_profile_sum, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(sizeof(double) * PROF_WARPS * PROF_CHUNK)) != cudaSuccess) {
      mg::set_last_error("mg_global_profile: shared memory attribute");
      return MG_ERR_CUDA;
    }
    k_profile_sum<<<dim3((unsigned)nb, (unsigned)((p->nc + chunk - 1) / chunk)), PROF_WARPS * 32,
                    smem, s>>>(p->n, p->nc, chunk, p->spectral_model, p->v, p->sigma,
                               p->sigma_const, p->amp, p->edges, w);
  } else {
    cudaMemsetAsync(w.part, 0, sizeof(double) * (size_t)nb * p->nc, s);
  }
  k_profile_final<<<(p->nc + PROF_CH - 1) / PROF_CH, PROF_CH * PROF_GROUPS, 0, s>>>(nb, p->nc, w,
                                                                                    spectrum);
  e = cudaGetLastError();
  if (e != cudaSuccess) {
    mg::set_last_error(std::string("mg_global_profile launch: ") + cudaGetErrorString(e));
    return MG_ERR_CUDA;
  }
  return MG_OK;
}
