// mp_row.cuh - how the half-step and adjoint kernels deal the cells of a plane to
// threads, and vector accesses along a row.
#ifndef MPB_MP_ROW_CUH
#define MPB_MP_ROW_CUH

#include "mp_checked.cuh"

namespace mpb {

// Rows (warps) per block: with one row the y neighbours come from other blocks
// through L2 and the 256 x 256 x 512 E half takes 824 instead of 737 us; 2 and 8
// rows 1% and 7% slower than 4.
constexpr int kRowTile = 4;
constexpr int kRowThreads = 32 * kRowTile;

__device__ __forceinline__ void prefetch_l2(const void *a) { asm volatile("prefetch.global.L2 [%0];" ::"l"(a)); }

// V consecutive elements of a row.
template <typename T, int V>
struct alignas(sizeof(T) * V <= 16 ? sizeof(T) * V : 16) RowV {
  T v[V];
};

// The accesses at column c of the plane at element `base` of an array of n
// elements (aligned to a row of V), checked like ld_c / st_c.  Plain loads, not
// the read-only path: a kernel launched early must not have them moved ahead
// of its wait.
template <typename T, int V>
__device__ __forceinline__ bool row_in(long long i, long long n, int *st) {
  return in_bounds(i, n, st) && (V == 1 || in_bounds(i + V - 1, n, st));
}
template <int V, typename T>
__device__ __forceinline__ RowV<T, V> ldp(const T *a, long long base, unsigned c, long long n, int *st) {
  RowV<T, V> r = {};
  if (row_in<T, V>(base + c, n, st)) r = *reinterpret_cast<const RowV<T, V> *>(a + base + c);
  return r;
}
template <int V, typename T>
__device__ __forceinline__ void stp(T *a, long long base, unsigned c, long long n, int *st, const RowV<T, V> &r) {
  if (row_in<T, V>(base + c, n, st)) *reinterpret_cast<RowV<T, V> *>(a + base + c) = r;
}

// The columns of a thread, row j, columns i0 .. i0 + V - 1 of the plane: rows
// are taken in groups of kRowTile, warp w of a block holds row w of a group, and
// its 32 lanes run along the row and on into the same row of the next group, so
// that a block covers kRowTile neighbouring rows (their y neighbours meet in
// L1) and no lane is idle on narrow or odd rows.
struct RowMap {
  unsigned nrow, nvec;  // threads per row (nx / V), and per warp over all groups
  unsigned mul, shift;  // t / nrow = (t * mul) >> (32 + shift) for t < 2^31
};

template <int V>
__device__ __forceinline__ bool row_cells(const RowMap &g, unsigned block, int ny, int &i0, int &j) {
  const unsigned t = block * 32 + (threadIdx.x & 31);
  const unsigned grp = __umulhi(t, g.mul) >> g.shift;
  i0 = int(t - grp * g.nrow) * V;
  j = int(grp * kRowTile + (threadIdx.x >> 5));
  return t < g.nvec && j < ny;
}

// nx / V >= 2.
static inline RowMap row_map(int nx, int ny, int V) {
  RowMap r;
  r.nrow = unsigned(nx / V);
  r.nvec = r.nrow * unsigned((ny + kRowTile - 1) / kRowTile);
  // exact for every t < 2^31 with shift = ceil(log2(nrow)) - 1 and mul =
  // ceil(2^(32 + shift) / nrow) (Granlund and Montgomery, PLDI 1994)
  int l = 0;
  while ((1ULL << l) < r.nrow) ++l;
  r.shift = unsigned(l - 1);
  r.mul = unsigned(((1ULL << (32 + r.shift)) + r.nrow - 1) / r.nrow);
  return r;
}

}  // namespace mpb

#endif
