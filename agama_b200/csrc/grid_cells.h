// The cell of a grid that holds a value: a table of guesses by even bins, then the next cell or a bisection.
#pragma once
#include "common.cuh"
#include <algorithm>
#include <vector>

namespace agb {

/** device view of one grid of the 2-D splines, for the search of the cell that holds a value: cell
    k < n - 1 is (node k, 1 / (node k+1 - node k)) and entry n - 1 the last node, so that two
    neighbouring 16-byte loads give both nodes of a cell and its reciprocal width.  lut[b] is the
    last cell that begins at or before the left edge of bin b of an even division of the grid into
    nlut bins, at most half as wide as the narrowest cell: a value of the bin is in that cell or the
    next one.  An uneven grid that would need more bins than 4096 and four times its nodes has no
    such table (nlut = 0). */
struct alignas(16) GridNode { double x, invH; };
struct GridView {
    const GridNode* cell;
    const int* lut;
    double x0, xEnd, lutScale;      // first and last node, nlut / (xEnd - x0)
    int n, nlut;
};
constexpr int GRID_LUT_MAX = 4096;

/// the tables of a grid of two or more ascending nodes (the view's pointers are left to the caller)
inline void makeGridTables(const std::vector<double>& g, std::vector<GridNode>* cell, std::vector<int>* lut, GridView* v)
{
    const int n = static_cast<int>(g.size());
    cell->resize(n);
    double narrowest = INFINITY;
    for(int k = 0; k < n; k++) {
        (*cell)[k].x = g[k];
        (*cell)[k].invH = k + 1 < n ? 1 / (g[k + 1] - g[k]) : 0;
        if(k + 1 < n) narrowest = std::min(narrowest, g[k + 1] - g[k]);
    }
    v->n = n;
    v->x0 = g.front();
    v->xEnd = g.back();
    const double bins = 2 * (v->xEnd - v->x0) / narrowest;
    v->nlut = bins < std::max(GRID_LUT_MAX, 4 * n) ? std::max(1, static_cast<int>(bins) + 1) : 0;
    v->lutScale = v->nlut / (v->xEnd - v->x0);
    // the edge is moved down by a millionth of a bin: a value just below it may be put into this bin by
    // the rounding of (x - x0) * lutScale
    lut->resize(v->nlut);
    for(int b = 0, k = 0; b < v->nlut; b++) {
        const double edge = v->x0 + (b - 1e-6) / v->lutScale;
        while(k < n - 2 && g[k + 1] <= edge) k++;
        (*lut)[b] = k;
    }
}

/// truncation to an integer, saturated; NaN gives the smallest one
AGB_HD int saturatedInt(double x)
{
#ifdef __CUDA_ARCH__
    return __double2int_rz(x);
#else
    return x >= 2147483647. ? 2147483647 : x > -2147483648. ? static_cast<int>(x) : -2147483647 - 1;
#endif
}

/** The cell of a grid that holds x (x0 <= x <= xEnd; the last node belongs to the last cell): its index
    and the entries of its two nodes.  For x outside or NaN the result is some cell of the grid.
    node(k) and guess(b) load an entry of either table.  An uneven grid is bisected (steps to the next cell from a
    guess took 107 ms instead of 5.4 for 2e4 orbits on a grid with 3000 nodes within 3e-5 of its radius,
    0.58 ms instead of 0.05 for 2e5 forces); the choice is the grid's, so that it costs the others one
    uniform branch (a bisection after the guess has failed cost 4 % of 6e4 galaxy orbits). */
template<class Node, class Guess>
AGB_HD int findCell(const GridView& g, double x, GridNode* lo, GridNode* hi, const Node& node, const Guess& guess)
{
    int k = 0;
    if(g.nlut) {
        const int b = saturatedInt((x - g.x0) * g.lutScale);
        k = guess(b < 0 ? 0 : b < g.nlut ? b : g.nlut - 1);
    } else {
        int end = g.n - 1;
        while(end - k > 1) {
            const int mid = (k + end) / 2;
            if(x >= node(mid).x) k = mid; else end = mid;
        }
    }
    *lo = node(k);
    *hi = node(k + 1);
    if(x >= hi->x && k < g.n - 2) {
        k++;
        *lo = *hi;
        *hi = node(k + 1);
    }
    return k;
}

}  // namespace agb
