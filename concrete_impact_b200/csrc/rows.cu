// Gather and scatter of the rows of several arrays in one launch: a phase's points out of, and
// back into, the arrays of all points (src/concrete_impact's phased.py does one fancy index per
// array).  Up to CIB_ROW_COPIES arrays of any width share the list of points.
//
// Bound by its launch: a two-phase RVE of 20,480 points moves 8 MB per phase; one launch per
// array took some 50 launches and 26 fills per update, 0.5 ms of host time.
#include <cuda_runtime.h>
#include <stdint.h>

#include "cib_common.cuh"

namespace cib {
namespace {

constexpr int ROW_THREADS = 256;

struct RowCopies {
  cib_row_copy a[CIB_ROW_COPIES];
};

// blockIdx.y: the array.  Consecutive threads take consecutive elements of a row.
__global__ void __launch_bounds__(ROW_THREADS) copy_rows_kernel(int64_t count, const int64_t* __restrict__ ids,
                                                                const __grid_constant__ RowCopies copies, int scatter) {
  const cib_row_copy& c = copies.a[blockIdx.y];
  const int64_t total = count * c.width, stride = (int64_t)gridDim.x * ROW_THREADS;
  for (int64_t e = (int64_t)blockIdx.x * ROW_THREADS + threadIdx.x; e < total; e += stride) {
    const int64_t row = c.width == 1 ? e : e / c.width, k = e - row * c.width;
    const int64_t far = ids[row] * c.width + k;
    if (scatter)
      c.dst[far] = c.src ? c.src[e] : c.fill;
    else
      c.dst[e] = c.src[far];
  }
}

}  // namespace
}  // namespace cib

using namespace cib;

extern "C" int cib_copy_rows(int64_t count, const int64_t* ids, int32_t arrays, const cib_row_copy* copies,
                             int32_t scatter, void* stream) {
  if (count < 0 || arrays < 0 || arrays > CIB_ROW_COPIES || (arrays > 0 && !copies) || (count > 0 && !ids))
    return CIB_EINVAL;
  RowCopies args{};
  int64_t widest = 0;
  for (int i = 0; i < arrays; ++i) {
    if (copies[i].width < 1 || !copies[i].dst || (!scatter && !copies[i].src)) return CIB_EINVAL;
    args.a[i] = copies[i];
    widest = copies[i].width > widest ? copies[i].width : widest;
  }
  if (count == 0 || arrays == 0) return CIB_OK;
  const int64_t blocks = (count * widest + ROW_THREADS - 1) / ROW_THREADS, cap = 8 * (int64_t)sm_count();
  copy_rows_kernel<<<dim3((unsigned)(blocks < cap ? blocks : cap), (unsigned)arrays), ROW_THREADS, 0,
                     reinterpret_cast<cudaStream_t>(stream)>>>(count, ids, args, scatter);
  return check_launch();
}
