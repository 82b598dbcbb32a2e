// Device-wide exclusive scan and stable one-digit distribution passes (an LSD
// radix sort with digits of up to 9 bits).
//
// The footprint binning orders (segment, particle) pairs by segment, then
// kernel class, then first channel.  The particles that reach the cube are
// ordered by class and channel first -- one pass over particles -- and their
// pairs are emitted in that order, so the pairs themselves only need to be
// distributed by segment: one pass up to 512 segments, two up to 2^18.  Every
// pass is stable, so equal particles keep their index order and the binning is
// deterministic.
#include "mg_internal.cuh"

namespace mg {

constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;  // 2048

// Block-wide exclusive scan of one value per thread (returns the block total).
template <typename T>
__device__ __forceinline__ T block_exclusive_scan(T v, T* smem, T& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) smem[warp] = x;
  __syncthreads();
  if (warp == 0) {
    T w = lane < (int)(blockDim.x >> 5) ? smem[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    smem[lane] = w;
  }
  __syncthreads();
  const T warp_base = warp > 0 ? smem[warp - 1] : T(0);
  total = smem[(blockDim.x >> 5) - 1];
  __syncthreads();
  return warp_base + x - v;
}

// Input of a scan: counts, or counts[idx[k]] for k < *m (0 beyond).
struct ScanIn {
  const int* in;
  const int* idx;
  const long long* m;
  long long n;
  __device__ __forceinline__ long long size() const { return m ? min(*m, n) : n; }
  __device__ __forceinline__ int at(long long i, long long sz) const {
    return i < sz ? in[idx ? idx[i] : i] : 0;
  }
};

// Phase 1: per-block sums of int32 counts.
__global__ void k_scan_reduce(ScanIn in, long long* __restrict__ sums) {
  __shared__ long long sm[32];
  const long long n = in.size();
  long long base = (long long)blockIdx.x * SCAN_TILE;
  long long s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) s += in.at(base + (long long)k * SCAN_THREADS + threadIdx.x, n);
  long long tot;
  block_exclusive_scan<long long>(s, sm, tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// Phase 2: exclusive scan of the block sums in one block (any count).
__global__ void k_scan_top(long long* __restrict__ sums, long long nblocks, long long* __restrict__ total) {
  __shared__ long long sm[32];
  long long carry = 0;
  for (long long b0 = 0; b0 < nblocks; b0 += blockDim.x) {
    long long i = b0 + threadIdx.x;
    long long v = i < nblocks ? sums[i] : 0;
    long long tot;
    long long ex = block_exclusive_scan<long long>(v, sm, tot);
    if (i < nblocks) sums[i] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

// Phase 3: scan within each block plus the block's offset.
__global__ void k_scan_apply(ScanIn in, const long long* __restrict__ sums,
                             long long* __restrict__ out) {
  __shared__ long long sm[32];
  const long long n = in.size();
  long long base = (long long)blockIdx.x * SCAN_TILE + (long long)threadIdx.x * SCAN_ITEMS;
  long long v[SCAN_ITEMS];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    v[k] = in.at(base + k, n);
    s += v[k];
  }
  long long tot;
  long long run = sums[blockIdx.x] + block_exclusive_scan<long long>(s, sm, tot);
#pragma unroll
  for (int k = 0; k < SCAN_ITEMS; ++k) {
    if (base + k < in.n) out[base + k] = run;
    run += v[k];
  }
}

// The whole scan in one block: the three phases' launches cost more than the
// work up to SCAN_ONE_MAX entries (6.6 us of launches against 3 us).
constexpr int SCAN_ONE_THREADS = 1024;
constexpr int SCAN_ONE_MAX = 8192;
__global__ void __launch_bounds__(SCAN_ONE_THREADS)
k_scan_one(ScanIn in, long long* __restrict__ out, long long* __restrict__ total) {
  __shared__ long long sm[32];
  const long long n = in.size();
  constexpr int PER = SCAN_ONE_MAX / SCAN_ONE_THREADS;
  const long long base = (long long)threadIdx.x * PER;
  int v[PER];
  long long s = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    v[k] = in.at(base + k, n);
    s += v[k];
  }
  long long tot;
  long long run = block_exclusive_scan<long long>(s, sm, tot);
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    if (base + k < in.n) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 0 && total) *total = tot;
}

long long scan_blocks(long long n) { return (n + SCAN_TILE - 1) / SCAN_TILE; }

static void scan_launch(const ScanIn& in, long long* out, long long* sums, long long* total,
                        cudaStream_t s) {
  if (in.n <= SCAN_ONE_MAX) {
    k_scan_one<<<1, SCAN_ONE_THREADS, 0, s>>>(in, out, total);
    return;
  }
  const long long nb = scan_blocks(in.n);
  k_scan_reduce<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, sums);
  k_scan_top<<<1, 1024, 0, s>>>(sums, nb, total);
  k_scan_apply<<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, sums, out);
}

// Exclusive scan of n int32 counts into out (int64); total into *total.
// sums needs scan_blocks(n) entries.
void launch_scan(const int* in, long long n, long long* out, long long* sums, long long* total,
                 cudaStream_t s) {
  scan_launch(ScanIn{in, nullptr, nullptr, n}, out, sums, total, s);
}

// The same of in[idx[k]], k < *m <= n.
void launch_scan_gather(const int* in, const int* idx, const long long* m, long long n,
                        long long* out, long long* sums, cudaStream_t s) {
  scan_launch(ScanIn{in, idx, m, n}, out, sums, nullptr, s);
}

// ---------------------------------------------------------------------------
// One stable distribution pass.  The elements are split into `chunks` runs of
// whole tiles, a block each.  A block ranks a tile's elements by digit (each
// warp counts its own slice, 32 elements at a time by match_any), moves them
// into digit order in shared memory and writes each digit's run to its place:
// the stores are contiguous runs of tile / bins elements instead of single
// elements, which is what bounds a pass on lists far larger than L2 (94.7M
// pairs: 1.40 ms a pass with single-element stores, 0.92 ms now; and two
// passes instead of three).
// With one chunk (up to two tiles) the block counts its own digits, so a small
// sort is a single launch; otherwise a histogram and a scan come first.
// ---------------------------------------------------------------------------

constexpr int RS_THREADS = 512;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;  // 8192
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_MAX_CHUNKS = 1216;  // four waves of two blocks on each of 152 SMs

// chunks of a pass over at most n elements
long long radix_chunks(long long n) {
  long long t = (n + RS_TILE - 1) / RS_TILE;
  if (t <= 2) t = 1;
  return t < RS_MAX_CHUNKS ? t : RS_MAX_CHUNKS;
}

// Elements of a pass over (key, value) pairs: digit (key >> shift) & mask.
struct RsPairs {
  const unsigned* kin;
  const int* vin;
  unsigned* kout;
  int* vout;
  const long long* np;
  long long cap;
  int shift;
  unsigned mask;
  __device__ __forceinline__ long long size() const { return min(*np, cap); }
  __device__ __forceinline__ bool get(long long i, unsigned& key, int& val) const {
    key = kin[i];
    val = vin[i];
    return true;
  }
  __device__ __forceinline__ unsigned key_only(long long i, bool& ok) const {
    ok = true;
    return kin[i];
  }
  __device__ __forceinline__ unsigned digit(unsigned key) const { return (key >> shift) & mask; }
  __device__ __forceinline__ void put(long long o, unsigned key, int val) const {
    kout[o] = key;
    vout[o] = val;
  }
  __device__ __forceinline__ bool skip() const { return false; }
};

// Elements of the particle pass: the particles with pairs, digit = kernel
// class << 7 | first channel >> cshift (class 0 for the table kernels, 1 for
// the Dirac kernel, 2 for the Gaussian and cubic-spline kernels: each class's
// particles then form stages of their own, which the tensor-core producers
// take on the class's own path).  Channels are ordered to 1/128 of the band,
// finer than the 16-channel windows they serve.
struct RsParticles {
  const PRec* rec;
  const int* npairs;
  const WsHeader* hdr;
  int* vout;
  long long n;
  int cshift;
  unsigned char cls[MG_MAX_KERNELS];
  __device__ __forceinline__ long long size() const { return n; }
  __device__ __forceinline__ unsigned key_only(long long i, bool& ok) const {
    ok = npairs[i] > 0;
    if (!ok) return 0u;
    const int clo = rec[i].clo, ks = rec[i].kslot;
    return (unsigned)cls[ks] << 7 | (unsigned)(clo >> cshift);
  }
  __device__ __forceinline__ bool get(long long i, unsigned& key, int& val) const {
    bool ok;
    key = key_only(i, ok);
    val = (int)i;
    return ok;
  }
  __device__ __forceinline__ unsigned digit(unsigned key) const { return key; }
  __device__ __forceinline__ void put(long long o, unsigned, int val) const { vout[o] = val; }
  __device__ __forceinline__ bool skip() const {
    return (hdr->status & (ST_PAIRS | ST_EDGES)) != 0;  // no room for the particles
  }
};

__device__ __forceinline__ void rs_range(long long n, long long chunks, long long& lo,
                                         long long& hi) {
  const long long tiles = (n + RS_TILE - 1) / RS_TILE;
  const long long per = (tiles + chunks - 1) / chunks * RS_TILE;
  lo = min((long long)blockIdx.x * per, n);
  hi = min(lo + per, n);
}

// Digit counts of every chunk, digit-major.
template <class E>
__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(E el, int bins, int* __restrict__ hist) {
  __shared__ int h[RS_THREADS];
  h[threadIdx.x] = 0;
  __syncthreads();
  long long lo, hi;
  rs_range(el.skip() ? 0 : el.size(), gridDim.x, lo, hi);
  for (long long i = lo + threadIdx.x; i < hi; i += RS_THREADS) {
    bool ok;
    const unsigned key = el.key_only(i, ok);
    if (ok) atomicAdd(&h[el.digit(key)], 1);
  }
  __syncthreads();
  if (threadIdx.x < bins) hist[(long long)threadIdx.x * gridDim.x + blockIdx.x] = h[threadIdx.x];
}

template <class E>
__global__ void __launch_bounds__(RS_THREADS) k_radix_scatter(E el, int bins,
                                                              const long long* __restrict__ off,
                                                              long long* __restrict__ total) {
  extern __shared__ __align__(16) unsigned char rs_smem[];
  unsigned* const s_key = reinterpret_cast<unsigned*>(rs_smem);              // [RS_TILE]
  int* const s_val = reinterpret_cast<int*>(s_key + RS_TILE);                // [RS_TILE]
  unsigned short* const wh = reinterpret_cast<unsigned short*>(s_val + RS_TILE);  // [warp][bin]
  __shared__ long long goff[RS_THREADS];  // next place of each digit
  __shared__ int dstart[RS_THREADS];      // its first element in the tile
  __shared__ int wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  long long lo, hi;
  rs_range(el.skip() ? 0 : el.size(), gridDim.x, lo, hi);
  if (off) {
    goff[tid] = tid < bins ? off[(long long)tid * gridDim.x + blockIdx.x] : 0;
  } else {
    // the only chunk: its digit counts and their scan
    dstart[tid] = 0;
    __syncthreads();
    for (long long i = lo + tid; i < hi; i += RS_THREADS) {
      bool ok;
      const unsigned key = el.key_only(i, ok);
      if (ok) atomicAdd(&dstart[el.digit(key)], 1);
    }
    __syncthreads();
    int tot;
    const int ex = block_exclusive_scan<int>(dstart[tid], wsum, tot);
    goff[tid] = ex;
    if (tid == 0 && total) *total = tot;
  }
  for (long long base = lo; base < hi; base += RS_TILE) {
    for (int k = tid; k < RS_WARPS * bins / 2; k += RS_THREADS) reinterpret_cast<int*>(wh)[k] = 0;
    __syncthreads();
    unsigned key[RS_ITEMS];
    int val[RS_ITEMS];
    unsigned short rank[RS_ITEMS];
    unsigned okm = 0u;
    unsigned short* const mine = wh + warp * bins;
    const long long wbase = base + warp * (32 * RS_ITEMS) + lane;
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
      const long long i = wbase + r * 32;
      key[r] = 0u;
      val[r] = 0;
      if (i < hi && el.get(i, key[r], val[r])) okm |= 1u << r;
    }
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
      const bool ok = (okm >> r) & 1u;
      const unsigned d = ok ? el.digit(key[r]) : 0xFFFFu;
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      unsigned old = 0u;
      if (ok) old = mine[d];
      rank[r] = (unsigned short)(old + __popc(peers & lt));
      __syncwarp();
      if (ok && (peers & lt) == 0u) mine[d] = (unsigned short)(old + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    // per digit: the warps' first ranks, the tile's count
    int cnt = 0;
    if (tid < bins)
      for (int w = 0; w < RS_WARPS; ++w) {
        const int t = wh[w * bins + tid];
        wh[w * bins + tid] = (unsigned short)cnt;
        cnt += t;
      }
    int tot;
    const int ex = block_exclusive_scan<int>(cnt, wsum, tot);
    dstart[tid] = ex;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r)
      if ((okm >> r) & 1u) {
        const unsigned d = el.digit(key[r]);
        const int pos = dstart[d] + mine[d] + rank[r];
        s_key[pos] = key[r];
        s_val[pos] = val[r];
      }
    __syncthreads();
    for (int k = tid; k < tot; k += RS_THREADS) {
      const unsigned kk = s_key[k];
      const unsigned d = el.digit(kk);
      el.put(goff[d] + (k - dstart[d]), kk, s_val[k]);
    }
    __syncthreads();
    goff[tid] += cnt;
  }
}

template <class E>
static void rs_pass(const E& el, int bits, long long chunks, int* hist, long long* off,
                    long long* sums, long long* total, cudaStream_t s) {
  const int bins = bits < 1 ? 2 : 1 << bits;
  const int smem = RS_TILE * 8 + RS_WARPS * bins * 2;
  // the attribute is per device: set on every launch (host-side only)
  cudaFuncSetAttribute(k_radix_scatter<E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       RS_TILE * 8 + RS_WARPS * RS_THREADS * 2);
  if (chunks <= 1) {
    k_radix_scatter<E><<<1, RS_THREADS, smem, s>>>(el, bins, nullptr, total);
    return;
  }
  k_radix_hist<E><<<(unsigned)chunks, RS_THREADS, 0, s>>>(el, bins, hist);
  launch_scan(hist, (long long)bins * chunks, off, sums, total, s);
  k_radix_scatter<E><<<(unsigned)chunks, RS_THREADS, smem, s>>>(el, bins, off, nullptr);
}

int radix_passes(int bits) { return bits < 1 ? 1 : (bits + RS_BITS - 1) / RS_BITS; }

// Sort the pairs (keys, vals), *np <= cap of them, by the low `bits` bits of
// the key; kt / vt are the second buffer, in which the result lands after an
// odd number of radix_passes(bits).  hist and off need 2^RS_BITS *
// radix_chunks(cap) entries, sums scan_blocks of that.
void launch_radix_sort(unsigned* keys, int* vals, unsigned* kt, int* vt, const long long* np,
                       long long cap, int bits, int* hist, long long* off, long long* sums,
                       cudaStream_t s) {
  const int passes = radix_passes(bits);
  const int width = (bits + passes - 1) / passes;
  const long long chunks = radix_chunks(cap);
  for (int p = 0; p < passes; ++p) {
    const RsPairs el{keys, vals, kt, vt, np, cap, p * width, (1u << width) - 1u};
    rs_pass(el, width, chunks, hist, off, sums, nullptr, s);
    unsigned* tk = keys; keys = kt; kt = tk;
    int* tv = vals; vals = vt; vt = tv;
  }
}

// The particles with pairs in order of kernel class and first channel:
// their indices into `out`, their number into hdr->n_valid.  hist and off
// need 2^RS_BITS * radix_chunks(g.n) entries where there are several chunks
// (g.n > 2 RS_TILE, so that scan_sums, which has room for g.n, has room for
// those too).
void launch_order_particles(const Geo& g, const Ws& w, int* out, int* hist, long long* off,
                            cudaStream_t s) {
  RsParticles el{w.rec, w.npairs, w.hdr, out, g.n, 0, {}};
  while (((g.max_nc - 1) >> el.cshift) > 127) ++el.cshift;
  for (int k = 0; k < g.n_kernels; ++k) {
    const int t = g.ks[k].type;
    el.cls[k] = (t == MG_KERNEL_GAUSSIAN || t == MG_KERNEL_CUBIC_SPLINE) ? 2
                : t == MG_KERNEL_DIRAC                                     ? 1
                                                                            : 0;
  }
  rs_pass(el, RS_BITS, radix_chunks(g.n), hist, off, w.scan_sums, &w.hdr->n_valid, s);
}

}  // namespace mg
