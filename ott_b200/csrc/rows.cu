// Kernels of the FP32 row-owner engine (engine_rows.cuh), one per padded
// dimension, and the table the solve's host side launches them from.
#include "rows.h"

#include "engine_rows.cuh"

namespace ottb {

namespace {

template <int D>
RowsKernel entry() {
  RowsKernel k;
  k.D = D;
  k.grid = (const void*)&sinkhorn_rows_kernel<D, true>;
  k.cluster = (const void*)&sinkhorn_rows_kernel<D, false>;
  return k;
}

}  // namespace

RowsKernel rows_kernel(int d) {
  if (d <= 2) return entry<2>();
  if (d <= 3) return entry<3>();
  if (d <= 4) return entry<4>();
  if (d <= 5) return entry<5>();
  if (d <= 6) return entry<6>();
  if (d <= 8) return entry<8>();
  if (d <= 10) return entry<10>();
  if (d <= 12) return entry<12>();
  if (d <= 16) return entry<16>();
  return RowsKernel{};
}

static_assert(sizeof(RowsShared) + 64 + kRowsSmemMax <= 227 * 1024, "a CTA's shared memory");

size_t rows_static_smem() { return sizeof(RowsShared); }

}  // namespace ottb
