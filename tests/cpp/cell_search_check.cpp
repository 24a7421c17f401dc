// Host build of the cell search of the spline grids (agama_b200/csrc/grid_cells.h): the cell that findCell
// gives is that of binSearch for every point within the grid, a cell of the grid for every other point, and
// the number of loads is bounded by that of a bisection on any grid.  Grids: uniform, geometric,
// random spacing, two nodes, and clusters of up to 3000 nodes within 1e-9 to 1e-4 of the grid's length;
// points: nodes, their two floating-point neighbours, random points over, around and inside the
// clusters, NaN and the infinities.  Prints "checked N mismatches M most loads over the bound L".
#include "grid_cells.h"
#include <cmath>
#include <cstdio>
#include <random>

using namespace agb;

int main()
{
    std::mt19937_64 rng(7);
    std::uniform_real_distribution<double> U(0, 1);
    std::vector<std::vector<double>> grids{ { -1, 1 }, { 0, 1, 1.000001 }, { 0, 1e-12, 1 } };
    for(int g = 0; g < 300; g++) {
        std::vector<double> a;
        const int n = 2 + static_cast<int>(rng() % 90);
        double acc = -1;
        for(int i = 0; i < n; i++)
            a.push_back(g % 3 == 0 ? -1 + 2.0 * i / (n - 1) : g % 3 == 1 ? acc += 0.05 + U(rng) : std::log(1e-3) + std::log(1e6) * i / (n - 1));
        if(g % 4 == 3) {        // a cluster (or two)
            const double width = (a.back() - a.front()) * std::pow(10., -4 - 5 * U(rng));
            for(int c = 0; c < 1 + g % 2; c++) {
                const int m = 10 + static_cast<int>(rng() % 3000);
                const double at = a.front() + (a.back() - a.front()) * U(rng);
                for(int i = 0; i < m; i++) a.push_back(at + width * i / m);
            }
            std::sort(a.begin(), a.end());
            a.erase(std::unique(a.begin(), a.end()), a.end());
        }
        grids.push_back(a);
    }
    long total = 0, bad = 0, over = -1000;
    for(const std::vector<double>& a : grids) {
        const int n = static_cast<int>(a.size());
        std::vector<GridNode> cell;
        std::vector<int> lut;
        GridView v;
        makeGridTables(a, &cell, &lut, &v);
        std::vector<double> xs{ NAN, INFINITY, -INFINITY };
        for(double x : a) for(double y : { x, std::nextafter(x, -INFINITY), std::nextafter(x, INFINITY) }) xs.push_back(y);
        const double span = a[n - 1] - a[0];
        for(int k = 0; k < 400; k++) xs.push_back(a[0] - 0.1 * span + 1.2 * span * U(rng));
        for(int k = 0; k < 400; k++) { const size_t i = rng() % (n - 1); xs.push_back(a[i] + (a[i + 1] - a[i]) * U(rng)); }
        const long bound = 5 + static_cast<long>(std::ceil(std::log2(n)));
        for(double x : xs) {
            long loads = 0;
            GridNode lo, hi;
            const int k = findCell(v, x, &lo, &hi, [&](int i) { loads++; return cell.at(i); }, [&](int b) { loads++; return lut.at(b); });
            total++;
            const bool inside = x >= a[0] && x <= a[n - 1];
            if(k < 0 || k > n - 2 || lo.x != a[k] || hi.x != a[k + 1] || (inside && k != binSearch(x, a.data(), n))) bad++;
            over = std::max(over, loads - bound);
        }
    }
    std::printf("checked %ld mismatches %ld most loads over the bound %ld\n", total, bad, over);
    return bad != 0 || over > 0;
}
