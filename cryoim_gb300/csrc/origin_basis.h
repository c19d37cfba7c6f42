// origin_basis.h — the small set of functions that carries a correlation's origin grid.
#pragma once
#include <vector>

namespace cryoim {

// Rows of a particle with fixed places: functions (m, k) with m, k < nb and m + k <= cut,
// m-major, then second rows (see below) for the functions with m + k < second, m-major.  The first
// fourteen are of grids of few origins, whose rows an exhaustive search packs several particles to a unit
// (64 particles of box 256 on the 1-degree grid, 1, 25 and 49 origins: 21 ms with 96 rows each, now 3.5, 7.2
// and 12.5; a row per origin took 4.2, 8.8 and 15.2).
struct OriginLayout {
    int nb, cut, second, rows;
    constexpr bool in(int m, int k) const { return m < nb && k < nb && m + k <= cut; }
    constexpr bool twice(int m, int k) const { return in(m, k) && m + k < second; }
};
constexpr OriginLayout OB_LAYOUT[] = {{1, 0, 1, 2},     {3, 3, 2, 11},    {4, 3, 2, 13},   {3, 4, 3, 15},
                                      {3, 4, 5, 18},    {4, 4, 3, 19},    {5, 4, 3, 21},   {5, 6, 4, 32},
                                      {5, 8, 5, 40},    {6, 7, 5, 45},    {7, 8, 5, 54},   {8, 9, 5, 64},
                                      {7, 12, 5, 64},   {8, 11, 5, 73},   {9, 16, 5, 96},  {10, 14, 3, 96},
                                      {11, 15, 6, 128}, {12, 17, 7, 160}, {13, 19, 3, 160}};
constexpr int OB_LAYOUTS = 19, OB_FEW = 14;
// grids of up to OB_WHOLE origins an axis keep all their functions, unless their step is at most a quarter of
// the band's sampling distance n / 2R (most of such a grid's functions are below the tail)
constexpr int OB_WHOLE = 8;
constexpr int OB_UNIT = 160;  // rows come in units of this many where no layout is enough

// The cross-correlation of one (particle, orientation) as a function of the origin is
// band-limited: sum_h c_h exp(2 pi i h.x / n) with |h| <= maxR.  On an origin grid finer
// than n / (2 maxR) pixels its values are far from independent (+-6 px at 0.5 px, maxR
// 64 of 256: 625 values, ~130 of them), so the contraction runs over an orthonormal basis
// of the grid instead of over the grid: row b of operand A is sum_o Q[o][b] A_o, and
// C[o] = sum_b Q[o][b] (A'_b B^T) in FP32 afterwards.  Q is a product of 1D functions per
// axis: eigenvectors of the Dirichlet kernel of the band on the axis (discrete prolate
// sequences: the energies of the ones left out fall off faster than exponentially),
// split into even and odd ones, so every transform is real or imaginary.
// Measured (GB300, 1-degree grid, a particle against 239,040 orientations): 625 origin rows 2.45
// ms; 160 basis rows against the half turn of omegas 0.29 ms + 0.09 ms for the expansion
// (box 256, BF16).  Root mean square error of the correlations of the 32 best candidates
// against FP64: 1.25e-4 (BF16) where one row per origin gave 1.67e-4, 1.75e-3 against 2.6e-3 (e4m3,
// box 192, +-6 px).  With fewer functions than origin_basis.cpp asks for it was 2.4e-4 and 6.8e-3.
struct OriginBasis {
    int n1 = 0;        // origins per axis: origin_i = mid + step (i - (n1 - 1) / 2)
    int nb = 0;        // functions per axis, even and odd ones alternating
    int slots = 0;     // rows of A per particle, in units of equal size (a multiple of 32)
    int used = 0;      // the first of them that hold something
    int units = 1;
    int layout = -1;   // the fixed places above, -1: rows by worth, any number of units
    int R = 0;
    float mid = 0.0f;  // centre of the grid on each axis, pixels
    // [nb][n1], orthonormal but for the scale 2^-ge[m]; q[m][n1-1-i] = (-1)^m q[m][i]; zero
    // for m >= n1
    std::vector<float> q;
    std::vector<float> f;    // [nb][2 R + 1]: even m: sum_i q cos(2 pi h u_i / n), odd: sum_i q sin, times 2^ge[m]
    std::vector<int> ge;     // [nb] powers of two (FP8 operands: the largest |f| in 0.5 .. 1; 0 for BF16)
    // row b holds function (m of x, k of y), part 0: the value rounded to the operand type,
    // part 1: what part 0's rounding left (times 16 for FP8); -1: an empty row
    std::vector<int> mx, my, part;
    std::vector<int> slot;   // [nb * nb][2]: row of part 0, of part 1 of function mx * nb + my, -1: none
    // the functions four at a time: entry i of ent_off[a] .. ent_off[a + 1] has (2a, 2b), (2a, 2b + 1),
    // (2a + 1, 2b), (2a + 1, 2b + 1) with b = i - ent_off[a]: row of part 0, of part 1 of each, -1: none;
    // an even number for each a
    std::vector<int> ent, ent_off;
    // q at the upper half of the origins, hi(j) = n1/2 + j, by couples of functions, zero beyond: qy
    // [hn][h rounded up to even][2] = q_2a(hi j), q_2a+1(hi j); qx [hn / 2 rounded up, and 8 more][h][4] =
    // the couple at j = 2i, then at 2i + 1 (h = (nb + 1) / 2, hn = (n1 + 1) / 2)
    std::vector<float> qx, qy;
};

// Origins i = 0 .. n1-1 at -omax + step i on both axes, frequencies |h| <= R (minR <= |h|)
// of an n-pixel transform.  f8: the operands are e4m3 (else BF16).
OriginBasis make_origin_basis(int n, int min_r, int R, float omax, float step, int n1, bool f8);

}  // namespace cryoim
