// rad_split.h -- where a CTA of the radiation transfer lists the wall-corner splits
// of one slab's columns (rad.cu): columns 1 .. DA one after the other.  An interior
// column has room for kMaxSplits (more are reported as unsupported) or its rows'
// number, if that is less; the first and the last, which every box splits, for as
// many as they can have, one a row of the cells' positions (Dv).
#pragma once
#ifdef __CUDACC__
#define GFM_HD_SPLIT __host__ __device__ __forceinline__
#else
#define GFM_HD_SPLIT inline
#endif

namespace gfm {

constexpr int kMaxSplits = 64;

GFM_HD_SPLIT int split_room(int DA, int Dv, int column) {
    return column == 1 || column == DA || Dv < kMaxSplits ? Dv : kMaxSplits;
}
// entries before a column's, and of all columns (column DA + 1)
GFM_HD_SPLIT int split_first(int DA, int Dv, int column) {
    if (column <= 1) return 0;
    const int inner = column - 2 < DA - 2 ? column - 2 : DA - 2;
    return Dv + (inner > 0 ? inner * split_room(DA, Dv, 0) : 0) + (column > DA && DA > 1 ? Dv : 0);
}

}  // namespace gfm
