// Beam convolution of the inserted cube (Martini.convolve_beam,
// martini/martini.py:863-901): every channel of the padded cube convolved
// with the beam image in "same" mode, the pad dropped, and the result scaled
// from Jy/arcsec^2 to Jy/beam by the beam area.
//
// The reference convolves each spatial slice with scipy's fftconvolve; the
// direct form here gives the same sums in FP32:
//   out[i][j] = scale * sum_{a,b} in[i + hx - a][j + hy - b] * K[a][b],
// hx = (kx - 1) / 2, hy = (ky - 1) / 2, zero outside the padded cube, for the
// unpadded pixels only.
//
// k_beam_conv: a block computes 16 x 16 output pixels of 32 channels (the
// cube's channel axis is the fastest, so a lane is a channel); each of its 8
// warps holds two output rows, 32 sums a lane.  The work is bound by FP32 FMAs
// (729 a voxel for a 27 px beam), so an input value must be read from shared
// memory once for many of them: a lane loads a window of 16 + T - 1 pixels and
// applies T = 8 taps of two kernel rows to it, 128 paired FMAs for 23 loads (one
// load per FMA before: 9.70 ms on 512 x 512 x 256 with a 27 px beam; now
// 2.21 ms, 1.23 ms of it at the FP32 FMA rate).  Input rows stream through a ring
// in shared memory (cp.async, BR_AHEAD rows ahead): at step s warp w takes input row 2 w + s, so that every
// warp works on kernel rows kx - 1 - s and kx - s and only 15 rows are live.
// That leaves room for two blocks on an SM, and the ring's size depends on ky
// mostly, so beams up to 71 px take this path whole (27 px before).  Wider ones
// (also beams of few rows, 5 x 101 px say) are taken as column chunks, one after
// the other into the same totals.  Each kernel row of a chunk is summed from zero
// and added to the voxel's total, which keeps the FP32 error below that of one
// running sum over all taps.
// k_beam_conv_direct: beams of so many rows that not even a chunk's taps fit,
// through the cache.
#include <string>

#include "mg_internal.cuh"

namespace mg {
void set_last_error(const std::string& msg);  // mg_api.cu
}

namespace {

using mg::f2;
using mg::f2_add;
using mg::f2_fma;
using mg::f2_make;
using mg::f2_split;

constexpr int BT_I = 16;    // output rows per block, two per warp
constexpr int BT_J = 16;    // output columns per thread
constexpr int BC = 32;      // channels per block (one per lane)
constexpr int BR_LIVE = BT_I - 1;  // input rows in use at a step
constexpr int BR_AHEAD = 2;        // input rows in flight
constexpr int BR_RING = BR_LIVE + BR_AHEAD;
constexpr int BEAM_THREADS = BT_I / 2 * 32;
constexpr size_t kBeamSmemMax = 226 * 1024;
constexpr size_t kBeamSmemTwo = 113 * 1024;  // two blocks on an SM

__host__ __device__ inline int beam_kstride(int ky) { return (ky + 3) & ~3; }
size_t beam_smem(int kx, int ky) {
  return sizeof(float) *
         ((size_t)BR_RING * (BT_J + ky - 1) * BC + 2 * (size_t)(kx + 1) * beam_kstride(ky));
}

// Columns per chunk of a beam: all of them where they fit; else the widest
// chunk of 40 columns or fewer with which two blocks fit on an SM, or one where
// the beam has too many rows for two; 0 if none fits.  256 x 256 x 64, 5 x 101 px:
// 172 us in chunks, 1461 us through the cache, 433 us with the whole halo
// staged.
int beam_chunk(int kx, int ky) {
  if (beam_smem(kx, ky) <= kBeamSmemMax) return ky;
  for (const size_t room : {kBeamSmemTwo, kBeamSmemMax})
    for (int kc = 40; kc >= 16; kc -= 8)
      if (beam_smem(kx, kc) <= room) return kc;
  return 0;
}

// Taps b0 .. b0 + T - 1 of a step's kernel-row pair kp[b] = (row of output row
// 0, row of output row 1) on the input row at `in` (this lane's channel):
// acc[u] += in[u + ky - 1 - b] kp[b].
template <int T>
__device__ __forceinline__ void beam_taps(const float* in, const f2* kp, int b0, int ky,
                                          f2 (&acc)[BT_J]) {
  const float* col = in + (size_t)(ky - b0 - T) * BC;
  float v[BT_J + T - 1];
#pragma unroll
  for (int q = 0; q < BT_J + T - 1; ++q) v[q] = col[q * BC];
  f2 k[T];
  if constexpr (T % 2 == 0) {
#pragma unroll
    for (int e = 0; e < T; e += 2) {
      const ulonglong2 t = *reinterpret_cast<const ulonglong2*>(kp + b0 + e);
      k[e] = t.x;
      k[e + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int e = 0; e < T; ++e) k[e] = kp[b0 + e];
  }
#pragma unroll
  for (int q = 0; q < BT_J + T - 1; ++q) {
    const f2 x = f2_make(v[q], v[q]);
#pragma unroll
    for (int e = 0; e < T; ++e) {
      const int u = q - (T - 1) + e;
      if (u >= 0 && u < BT_J) acc[u] = f2_fma(x, k[e], acc[u]);
    }
  }
}

// One input row: the row sums of both output rows, added to their totals.
__device__ __forceinline__ void beam_row(const float* in, const f2* kp, int ky, f2 (&tot)[BT_J]) {
  f2 acc[BT_J];
#pragma unroll
  for (int u = 0; u < BT_J; ++u) acc[u] = 0ull;
  int b = 0;
#pragma unroll 1
  for (; b + 8 <= ky; b += 8) beam_taps<8>(in, kp, b, ky, acc);
  if (ky - b >= 4) {
    beam_taps<4>(in, kp, b, ky, acc);
    b += 4;
  }
#pragma unroll 1
  for (; b < ky; ++b) beam_taps<1>(in, kp, b, ky, acc);
#pragma unroll
  for (int u = 0; u < BT_J; ++u) tot[u] = f2_add(tot[u], acc[u]);
}

// The first and last steps, where one of the two output rows (H) has no
// kernel row: the other's sums only (no product of an input with a zero that
// is not a tap).
template <int H>
__device__ __forceinline__ void beam_row1(const float* in, const f2* kp, int ky, f2 (&tot)[BT_J]) {
  float acc[BT_J];
#pragma unroll
  for (int u = 0; u < BT_J; ++u) acc[u] = 0.f;
#pragma unroll 1
  for (int b = 0; b < ky; ++b) {
    const float2 k = f2_split(kp[b]);
#pragma unroll
    for (int u = 0; u < BT_J; ++u)
      acc[u] = fmaf(in[(size_t)(u + ky - 1 - b) * BC], H ? k.x : k.y, acc[u]);
  }
#pragma unroll
  for (int u = 0; u < BT_J; ++u) {
    const float2 t = f2_split(tot[u]);
    tot[u] = H ? f2_make(t.x + acc[u], t.y) : f2_make(t.x, t.y + acc[u]);
  }
}

// VEC: 16-byte copies (nc a multiple of 4 and the cube 16-byte aligned).
// CHUNKS: the beam's kyt columns are taken ky at a time (else kyt = ky).
template <bool VEC, bool CHUNKS>
__global__ void __launch_bounds__(BEAM_THREADS, 2)
k_beam_conv(const float* __restrict__ in, int nx, int ny, int nc, int px, int py,
            const float* __restrict__ kern, int kx, int kyt, int kyc, float scale,
            float* __restrict__ out) {
  extern __shared__ __align__(16) float sm[];
  float* const ring = sm;
  f2* const s_k = reinterpret_cast<f2*>(sm + (size_t)BR_RING * (BT_J + kyc - 1) * BC);
  const int i0 = px + blockIdx.y * BT_I, j0 = py + blockIdx.x * BT_J, c0 = blockIdx.z * BC;
  const int rb = i0 - (kx - 1) / 2;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int nrows = BT_I + kx - 1;
  f2 tot[BT_J];
#pragma unroll
  for (int u = 0; u < BT_J; ++u) tot[u] = 0ull;
#pragma unroll 1
  for (int b0 = 0; b0 < (CHUNKS ? kyt : 1); b0 += kyc) {
    const int ky = CHUNKS ? min(kyc, kyt - b0) : kyt;  // beam columns b0 .. b0 + ky - 1
    const int hj = BT_J + ky - 1, ks = beam_kstride(ky);
    const int cb = j0 + (kyt - 1) / 2 - (b0 + ky - 1);  // input column of ring column 0
    // a thread copies the same channels of every QS-th pixel of a row: what does
    // not depend on the row is taken out of the copy, whose instructions bound
    // small beams (3 px on 48 x 48 x 33, copied a channel at a time: 12.6 us, 8.9 now;
    // 10.9 us with the whole halo staged before the sums)
    constexpr int V = VEC ? 4 : 1, LPP = BC / V, QS = BEAM_THREADS / LPP;
    const int q0 = tid / LPP, cc = (tid % LPP) * V;
    const int qlo = c0 + cc < nc ? max(-cb, 0) : hj, qhi = min(hj, ny - cb);  // in the cube
    const long long qoff = (long long)(cb + q0) * nc + c0 + cc, qstep = (long long)QS * nc;
    const unsigned dst0 = (unsigned)__cvta_generic_to_shared(ring + q0 * BC + cc);
    auto load_row = [&](int r) {  // input row r of the block into its ring slot
      if (r < nrows) {
        const int gi = rb + r;
        const bool row_in = gi >= 0 && gi < nx;
        const float* src = in + (long long)gi * ny * nc + qoff;
        unsigned d = dst0 + (unsigned)(r % BR_RING) * (unsigned)(hj * BC * 4);
        for (int q = q0; q < hj; q += QS, src += qstep, d += QS * BC * 4) {
          const bool ok = row_in && q >= qlo && q < qhi;
          const float* const g = ok ? src : in;
          if (VEC)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(g),
                         "r"(ok ? 16 : 0)
                         : "memory");
          else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(g),
                         "r"(ok ? 4 : 0)
                         : "memory");
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (CHUNKS) __syncthreads();  // every warp is done with the chunk before
    for (int r = 0; r < BR_LIVE - 1; ++r) load_row(r);
    for (int r = 0; r < BR_AHEAD; ++r) load_row(BR_LIVE - 1 + r);
    // s_k[s][b]: the kernel rows of step s, kx - 1 - s and kx - s, as pairs
    const float* const kb = kern + (CHUNKS ? b0 : 0);
    for (int t = tid; t < (kx + 1) * ks; t += BEAM_THREADS) {
      const int st = t / ks, b = t - st * ks;
      const int a0 = kx - 1 - st;
      s_k[t] = f2_make(b < ky && a0 >= 0 ? kb[a0 * kyt + b] : 0.f,
                       b < ky && a0 + 1 < kx ? kb[(a0 + 1) * kyt + b] : 0.f);
    }
    for (int s = 0; s <= kx; ++s) {
      // row s + BR_LIVE - 1 has arrived; every warp is done with row s - 1,
      // whose slot the next row takes
      asm volatile("cp.async.wait_group %0;" ::"n"(BR_AHEAD - 1) : "memory");
      __syncthreads();
      load_row(s + BR_LIVE - 1 + BR_AHEAD);
      const float* row = ring + (size_t)((2 * w + s) % BR_RING) * hj * BC + lane;
      const f2* kp = s_k + (size_t)s * ks;
      if (s == 0)
        beam_row1<1>(row, kp, ky, tot);
      else if (s == kx)
        beam_row1<0>(row, kp, ky, tot);
      else
        beam_row(row, kp, ky, tot);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  }
  const int c = c0 + lane;
  if (c >= nc) return;
  const int nyo = ny - 2 * py;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int i = i0 + 2 * w + h;
    if (i >= nx - px) continue;
#pragma unroll
    for (int u = 0; u < BT_J; ++u) {
      const int j = j0 + u;
      const float2 t = f2_split(tot[u]);
      if (j < ny - py)
        out[((long long)(i - px) * nyo + (j - py)) * nc + c] = (h ? t.y : t.x) * scale;
    }
  }
}

// Beams of very many rows: one output voxel per thread, input through the cache.
__global__ void k_beam_conv_direct(const float* __restrict__ in, int nx, int ny, int nc, int px,
                                   int py, const float* __restrict__ kern, int kx, int ky,
                                   float scale, float* __restrict__ out) {
  const int nxo = nx - 2 * px, nyo = ny - 2 * py;
  const long long total = (long long)nxo * nyo * nc;
  const int hx = (kx - 1) / 2, hy = (ky - 1) / 2;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(e % nc);
    const long long pix = e / nc;
    const int i = px + (int)(pix / nyo), j = py + (int)(pix % nyo);
    float acc = 0.f;
    for (int a = 0; a < kx; ++a) {
      const int gi = i + hx - a;
      if (gi < 0 || gi >= nx) continue;
      for (int b = 0; b < ky; ++b) {
        const int gj = j + hy - b;
        if (gj < 0 || gj >= ny) continue;
        acc = fmaf(__ldg(in + ((long long)gi * ny + gj) * nc + c), __ldg(kern + a * ky + b), acc);
      }
    }
    out[e] = acc * scale;
  }
}

}  // namespace

extern "C" int mg_convolve_beam(const float* cube, int32_t nx, int32_t ny, int32_t nc,
                                int32_t padx, int32_t pady, const float* kernel, int32_t kx,
                                int32_t ky, float scale, float* out, void* stream) {
  if (!cube || !kernel || !out || nx <= 0 || ny <= 0 || nc <= 0 || kx <= 0 || ky <= 0 ||
      (kx % 2) == 0 || (ky % 2) == 0 || padx < 0 || pady < 0 || 2 * padx >= nx ||
      2 * pady >= ny) {
    mg::set_last_error("mg_convolve_beam: invalid arguments (odd kernel sizes, pads < half size)");
    return MG_ERR_INVALID_ARGUMENT;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int kyc = beam_chunk(kx, ky);
  if (kyc > 0) {
    const size_t smem = beam_smem(kx, kyc);
    const bool vec = (nc & 3) == 0 && (reinterpret_cast<uintptr_t>(cube) & 15) == 0;
    const auto kernel_fn = kyc < ky ? (vec ? k_beam_conv<true, true> : k_beam_conv<false, true>)
                                    : (vec ? k_beam_conv<true, false> : k_beam_conv<false, false>);
    if (smem > 48 * 1024 &&
        cudaFuncSetAttribute(kernel_fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kBeamSmemMax) != cudaSuccess) {
      mg::set_last_error("mg_convolve_beam: shared memory attribute");
      return MG_ERR_CUDA;
    }
    const dim3 grid((unsigned)((ny - 2 * pady + BT_J - 1) / BT_J),
                    (unsigned)((nx - 2 * padx + BT_I - 1) / BT_I), (unsigned)((nc + BC - 1) / BC));
    kernel_fn<<<grid, BEAM_THREADS, smem, s>>>(cube, nx, ny, nc, padx, pady, kernel, kx, ky, kyc,
                                               scale, out);
  } else {
    k_beam_conv_direct<<<4096, 256, 0, s>>>(cube, nx, ny, nc, padx, pady, kernel, kx, ky, scale,
                                            out);
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    mg::set_last_error(std::string("mg_convolve_beam launch: ") + cudaGetErrorString(e));
    return MG_ERR_CUDA;
  }
  return MG_OK;
}
