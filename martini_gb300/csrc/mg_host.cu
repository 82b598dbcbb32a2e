// Host side of an insertion: the inserted FP32 cube into the caller's FP64
// array, its unit conversion and the summary's sums, in one pass.
//
// Bound by host memory (20 bytes a voxel: the array read and written, the
// cube read) and by the FP64 divisions.  As whole-array operations (convert,
// add, divide, multiply, sum twice) the same work made six passes and three
// temporaries.  A call on a 128^3 cube and 100k particles (0.9 ms of it on the GPU),
// with the particle amplitudes' power as a division too: the first of a new object
// 10.6 ms before and 4.7 ms now, in a new process 19 and 6.3, repeated on one
// object 9.0 and 4.4.
// Pixel rows go to a few threads; each row's per-channel sums are kept apart
// and added in row order, so the result does not depend on the thread count.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <exception>
#include <string>
#include <thread>
#include <vector>

#include "martini_gb300.h"

namespace mg {
void set_last_error(const std::string& msg);  // mg_api.cu
}

namespace {

constexpr int HOST_THREADS = 8;
constexpr long long HOST_CELLS_PER_THREAD = 1 << 17;  // starting a thread costs about 30 us
constexpr long long HOST_RUN_CELLS = 1 << 18;         // 2 MB of the array: a huge page
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14
#endif

struct CubeAdd {
  double* array;
  const float* add;
  long long nx, ny, nc, padx, pady;
  double px2;
  bool divide_all;
  double* row_sums;  // [nx][nc]
};

void add_row(const CubeAdd& q, long long i) {
  double* sums = q.row_sums + i * q.nc;
  std::fill(sums, sums + q.nc, 0.0);
  const bool in_i = i >= q.padx && i < q.nx - q.padx;
  for (long long j = 0; j < q.ny; ++j) {
    double* a = q.array + (i * q.ny + j) * q.nc;
    const float* b = q.add + (i * q.ny + j) * q.nc;
    if (q.divide_all)
      for (long long c = 0; c < q.nc; ++c) a[c] = (a[c] + (double)b[c]) / q.px2;
    else
      for (long long c = 0; c < q.nc; ++c) a[c] += (double)b[c] / q.px2;
    if (in_i && j >= q.pady && j < q.ny - q.pady)
      for (long long c = 0; c < q.nc; ++c) sums[c] += a[c] * q.px2;
  }
}

// Map the pages of a run of the array for writing, contents kept.  A first
// insertion meets an array that nothing has touched, and the pass reads each
// page before it writes it: two faults a page, which threads on neighbouring
// rows serialise.  A hint only: where the kernel does not know it, the pass
// takes those faults.  Not for a run whose middle is mapped already (90 ns a page).
void map_for_writing(double* a, long long cells) {
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  const uintptr_t lo = (uintptr_t)a & ~(page - 1);
  const uintptr_t hi = ((uintptr_t)(a + cells) + page - 1) & ~(page - 1);
  const uintptr_t mid = (uintptr_t)(a + cells / 2) & ~(page - 1);
  unsigned char there = 0;
  if (mincore(reinterpret_cast<void*>(mid), page, &there) == 0 && (there & 1)) return;
  madvise(reinterpret_cast<void*>(lo), hi - lo, MADV_POPULATE_WRITE);
}

}  // namespace

extern "C" int mg_cube_add(double* array, const float* add, int64_t nx, int64_t ny, int64_t nc,
                           int64_t padx, int64_t pady, double px2, int32_t divide_all,
                           double* per_channel) {
  if (!array || !add || !per_channel || nx <= 0 || ny <= 0 || nc <= 0 || padx < 0 || pady < 0) {
    mg::set_last_error("mg_cube_add: invalid argument");
    return MG_ERR_INVALID_ARGUMENT;
  }
  try {
    std::vector<double> rows((size_t)(nx * nc));
    const CubeAdd q{array, add, nx, ny, nc, padx, pady, px2, divide_all != 0, rows.data()};
    const long long want =
        std::min<long long>({HOST_THREADS, (long long)std::thread::hardware_concurrency(),
                             nx * ny * nc / HOST_CELLS_PER_THREAD, nx});
    // a thread takes a run of whole rows at a time: a huge page or so, less
    // where the threads would not all get one
    const long long share = want > 1 ? (nx + want - 1) / want : nx;
    const long long run =
        std::max<long long>(1, std::min<long long>(share, HOST_RUN_CELLS / (ny * nc)));
    std::atomic<long long> next{0};
    auto work = [&]() {
      for (long long i0; (i0 = next.fetch_add(run)) < nx;) {
        const long long i1 = std::min<long long>(i0 + run, nx);
        map_for_writing(array + i0 * ny * nc, (i1 - i0) * ny * nc);
        for (long long i = i0; i < i1; ++i) add_row(q, i);
      }
    };
    std::vector<std::thread> pool;
    pool.reserve(HOST_THREADS);
    try {
      for (long long t = 1; t < want; ++t) pool.emplace_back(work);
    } catch (const std::exception&) {
      // no more threads (or memory for one) to be had: the ones there and this
      // one do the work; they must be joined before the pool goes
    }
    work();
    for (std::thread& t : pool) t.join();
    std::fill(per_channel, per_channel + nc, 0.0);
    for (long long i = 0; i < nx; ++i)
      for (long long c = 0; c < nc; ++c) per_channel[c] += rows[(size_t)(i * nc + c)];
  } catch (const std::exception& e) {
    mg::set_last_error(std::string("mg_cube_add: ") + e.what());
    return MG_ERR_WORKSPACE;
  }
  return MG_OK;
}
