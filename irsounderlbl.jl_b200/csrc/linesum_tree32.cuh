// linesum_tree32.cuh -- what the FP32 line sums (forward and Jacobian) share: an index of
// the lines by grid cell, and a binary tree of blocks on which distant lines are summed at
// Chebyshev nodes.
//
// A line's far wing is smooth over a block of half-width h that its centre is 2 h or more
// away from, so there it is evaluated at 16 Chebyshev nodes of the block and interpolated
// (error of one line's term below 1.6e-8 of its largest value on the block).  Blocks of
// 4096, 2048, ..., 128 points (a leaf: one warp's points): a line is summed at the widest
// block that it is far from and whose points it covers wholly, and node values go down from
// a block to its halves through two fixed 16 x 16 matrices (in FP64, so that the levels add
// no rounding).  Summing at factor-two levels makes every level cost a warp about the same
// (2 R lines for a block of R/128 warps); with two levels (1024 or 2048 points, then 128) most
// of a warp's time went to lines in between, staged and evaluated once per warp.
#pragma once
#include "linesum.cuh"

namespace irs {

constexpr int kTrNodes = 16;
constexpr int kTrLevels = 6;                         // 4096, 2048, 1024, 512, 256, 128 points
constexpr int kTrLeaf = 128;
constexpr int kTrStrip = kTrLeaf << (kTrLevels - 1);  // 4096
constexpr int kTrLeaves = kTrStrip / kTrLeaf;         // 32

// built on the host in extended precision (tree32_tables, irs_host.cpp)
struct TreeTables {
    double M[2][kTrNodes][kTrNodes];  // [half][k][j]: L_k at node j of the left / right half
    float L[kTrNodes][kTrLeaf];       // [k][i]: L_k at point i of a leaf
};

// node k on [-1, 1], cos((2k+1) pi / 32), rounded to FP32
__device__ __forceinline__ float tree_node_f(int k) {
    const int a = k < 8 ? k : 15 - k;
    const float v = a == 0 ? 9.951847196e-01f : a == 1 ? 9.569403529e-01f : a == 2 ? 8.819212914e-01f
                  : a == 3 ? 7.730104327e-01f : a == 4 ? 6.343932748e-01f : a == 5 ? 4.713967443e-01f
                  : a == 6 ? 2.902846634e-01f : 9.801714122e-02f;
    return k < 8 ? v : -v;
}

// Index by cells of `cell` grid points, from V = -half cell offset: idx[j] = first line with
// (V + 0.5 + off) / cell >= j, V the sorted (unshifted) centres; off covers the cutoff and
// the margins.  Thresholds are rounded to cells, which only moves a line from one list of
// the sum to another, so every bound is one load instead of a search.
struct CellIndex {
    const int* idx;     // [rows][n]
    int n;              // cells + 1 per row
    float inv_cell, off;
};
__device__ __forceinline__ int cell_floor(const CellIndex& ci, const int* row, float v) {  // first line of the cell holding v
    return row[min(max((int)floorf((v + 0.5f + ci.off) * ci.inv_cell), 0), ci.n - 1)];
}
__device__ __forceinline__ int cell_ceil(const CellIndex& ci, const int* row, float v) {
    return row[min(max((int)ceilf((v + 0.5f + ci.off) * ci.inv_cell), 0), ci.n - 1)];
}
__global__ void __launch_bounds__(256) cell_index_kernel(const double* __restrict__ V, const long long* __restrict__ offs,
                                                         const int* __restrict__ counts, int n, double cell,
                                                         double off, int* __restrict__ idx) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const double* v = V + offs[blockIdx.y];
    idx[(size_t)blockIdx.y * n + j] = (int)lower_bound0(v, (double)j * cell - off - 0.5, counts[blockIdx.y]);
}

// The far lines of the block of points [cb, cb + 2 h): index ranges [x, y) and [z, w)
// (empty at the centre when the cutoff or the core leaves none).  R = max(2 h, core reach + h)
// + m keeps every core off the block; m, the segment's largest shift and two points, covers U
// against V (the keys are unshifted, so their order is exact) and the rounding of the bounds.
__device__ __forceinline__ int4 tree_ranges(const CellIndex& ci, const int* row, float cb, float h, float cut, float m,
                                            float reach) {
    const float c = cb + h - 0.5f, R = fmaxf(2.f * h, reach + h) + m;
    if (!(cut - h - m > R)) {
        const int j = cell_floor(ci, row, c);
        return make_int4(j, j, j, j);
    }
    int4 r;
    r.x = cell_ceil(ci, row, c + h - cut + m);
    r.y = max(r.x, cell_floor(ci, row, c - R));
    r.z = max(r.y, cell_ceil(ci, row, c + R));
    r.w = max(r.z, cell_floor(ci, row, c - h + cut - m));
    return r;
}
// a block's ranges contain those of the block above (by the thresholds; rounding apart)
__device__ __forceinline__ int4 tree_inside(int4 s, int4 up) {
    if (up.y > up.x) { s.x = min(s.x, up.x); s.y = max(s.y, up.y); }
    if (up.w > up.z) { s.z = min(s.z, up.z); s.w = max(s.w, up.w); }
    s.y = max(s.x, s.y);
    s.z = max(s.y, s.z);
    s.w = max(s.z, s.w);
    return s;
}
// a block's own far lines without those of the block above (up.x == up.y: it has none on
// that side): four pieces, walked as one list t = 0 .. n - 1
struct TreeList {
    int4 a;       // first lines of the pieces
    int n1, n2, n3, n;  // ends of the pieces in t
};
__device__ __forceinline__ TreeList tree_list(int4 own, int4 up) {
    TreeList L;
    const int l1 = up.y > up.x ? up.x : own.y, l2 = up.y > up.x ? up.y : own.y;
    const int r1 = up.w > up.z ? up.z : own.w, r2 = up.w > up.z ? up.w : own.w;
    L.a = make_int4(own.x, l2, own.z, r2);
    L.n1 = max(l1 - own.x, 0);
    L.n2 = L.n1 + max(own.y - l2, 0);
    L.n3 = L.n2 + max(r1 - own.z, 0);
    L.n = L.n3 + max(own.w - r2, 0);
    return L;
}
__device__ __forceinline__ int tree_line(const TreeList& L, int t) {
    return t < L.n1 ? L.a.x + t : t < L.n2 ? L.a.y + (t - L.n1) : t < L.n3 ? L.a.z + (t - L.n2) : L.a.w + (t - L.n3);
}

}  // namespace irs
