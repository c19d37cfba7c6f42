// origin_basis.cpp — the origin grid's basis (origin_basis.h), on the host in FP64.
#include "origin_basis.h"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <numeric>

namespace cryoim {
namespace {

// Eigenvectors of the symmetric m x m matrix a (destroyed), by cyclic Jacobi rotations;
// columns of v in descending order of eigenvalue.
void eigenvectors(std::vector<double>& a, int m, std::vector<double>& v) {
    v.assign((size_t)m * m, 0.0);
    for (int i = 0; i < m; ++i) v[(size_t)i * m + i] = 1.0;
    for (int sweep = 0; sweep < 60; ++sweep) {
        double off = 0.0, dia = 0.0;
        for (int i = 0; i < m; ++i)
            for (int j = 0; j < m; ++j) (i == j ? dia : off) += a[(size_t)i * m + j] * a[(size_t)i * m + j];
        if (off <= 1e-28 * (dia + off)) break;
        for (int p = 0; p < m; ++p)
            for (int q = p + 1; q < m; ++q) {
                const double apq = a[(size_t)p * m + q];
                if (apq == 0.0) continue;
                const double th = 0.5 * (a[(size_t)q * m + q] - a[(size_t)p * m + p]) / apq;
                const double t = (th >= 0 ? 1.0 : -1.0) / (std::fabs(th) + std::sqrt(th * th + 1.0));
                const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
                for (int k = 0; k < m; ++k) {
                    const double x = a[(size_t)k * m + p], y = a[(size_t)k * m + q];
                    a[(size_t)k * m + p] = c * x - s * y;
                    a[(size_t)k * m + q] = s * x + c * y;
                }
                for (int k = 0; k < m; ++k) {
                    const double x = a[(size_t)p * m + k], y = a[(size_t)q * m + k];
                    a[(size_t)p * m + k] = c * x - s * y;
                    a[(size_t)q * m + k] = s * x + c * y;
                }
                for (int k = 0; k < m; ++k) {
                    const double x = v[(size_t)k * m + p], y = v[(size_t)k * m + q];
                    v[(size_t)k * m + p] = c * x - s * y;
                    v[(size_t)k * m + q] = s * x + c * y;
                }
            }
    }
    std::vector<int> ord(m);
    std::iota(ord.begin(), ord.end(), 0);
    std::sort(ord.begin(), ord.end(), [&](int x, int y) { return a[(size_t)x * m + x] > a[(size_t)y * m + y]; });
    std::vector<double> w((size_t)m * m);
    for (int j = 0; j < m; ++j)
        for (int i = 0; i < m; ++i) w[(size_t)i * m + j] = v[(size_t)i * m + ord[j]];
    v.swap(w);
}

}  // namespace

OriginBasis make_origin_basis(int n, int min_r, int R, float omax, float step, int n1, bool f8) {
    OriginBasis ob;
    ob.n1 = n1;
    ob.R = R;
    ob.mid = (float)(-(double)omax + 0.5 * (double)step * (n1 - 1));
    const double w0 = 2.0 * 3.14159265358979323846 / n;
    std::vector<double> u(n1);
    for (int i = 0; i < n1; ++i) u[i] = (double)step * (i - 0.5 * (n1 - 1));
    // cos and sin of w0 h u_i for h = 0 .. R, [h][i] (u_{n1-1-i} = -u_i)
    std::vector<double> cs((size_t)(R + 1) * n1), sn((size_t)(R + 1) * n1);
    const int he = (n1 + 1) / 2, ho = n1 / 2;
    for (int h = 0; h <= R; ++h)
        for (int i = 0; i < he; ++i) {
            const size_t q = (size_t)h * n1 + i, r = (size_t)h * n1 + n1 - 1 - i;
            cs[q] = cs[r] = std::cos(w0 * h * u[i]);
            sn[q] = std::sin(w0 * h * u[i]);
            if (r != q) sn[r] = -sn[q];
        }
    // even and odd eigenvectors apart: v(i) = +- v(n1 - 1 - i)
    std::vector<std::vector<double>> fun;  // [function][n1], even and odd alternating
    std::vector<double> vec[2];
    for (int odd = 0; odd < 2; ++odd) {
        const int m = odd ? ho : he;
        const std::vector<double>& t = odd ? sn : cs;
        std::vector<double> a((size_t)m * m, 0.0);
        for (int h = -R; h <= R; ++h) {
            const double* th = t.data() + (size_t)std::abs(h) * n1;  // (the signs of a negative h cancel)
            for (int i = 0; i < m; ++i)
                for (int j = 0; j <= i; ++j) a[(size_t)i * m + j] += th[i] * th[j];
        }
        // orthonormal half-grid vectors (e_i +- e_mirror) / sqrt 2 (the middle one alone)
        auto norm = [&](int i) { return (!odd && (n1 & 1) && i == m - 1) ? 1.0 : std::sqrt(2.0); };
        for (int i = 0; i < m; ++i)
            for (int j = 0; j <= i; ++j) {
                const double s = a[(size_t)i * m + j];
                a[(size_t)i * m + j] = s * norm(i) * norm(j);
                a[(size_t)j * m + i] = s * norm(j) * norm(i);
            }
        eigenvectors(a, m, vec[odd]);
    }
    for (int k = 0; k < n1; ++k) {
        const int odd = k & 1, m = odd ? ho : he, col = k / 2;
        std::vector<double> g(n1, 0.0);
        for (int i = 0; i < m; ++i) {
            const bool middle = !odd && (n1 & 1) && i == m - 1;
            const double x = vec[odd][(size_t)i * m + col] * (middle ? 1.0 : std::sqrt(0.5));
            g[i] = x;
            if (!middle) g[n1 - 1 - i] = odd ? -x : x;
        }
        fun.push_back(g);
    }
    // their transforms over the band, even or odd in h as the function is
    const int H = 2 * R + 1;
    std::vector<double> f((size_t)n1 * H), sq((size_t)(R + 1) * n1);  // sq: their squares, [h][function]
    for (int k = 0; k < n1; ++k) {
        const std::vector<double>& t = (k & 1) ? sn : cs;
        for (int h = 0; h <= R; ++h) {
            const double* th = t.data() + (size_t)h * n1;
            double s = 0.0;
            for (int i = 0; i < n1; ++i) s += fun[k][i] * th[i];
            f[(size_t)k * H + R + h] = s;
            f[(size_t)k * H + R - h] = (k & 1) ? -s : s;
            sq[(size_t)h * n1 + k] = s * s;
        }
    }
    // energy of each product over the half-plane band samples (hx > 0, or hx = 0 and ky > 0): row by
    // row of hx, whose samples are minR^2 <= hx^2 + ky^2 <= R^2
    std::vector<double> e((size_t)n1 * n1, 0.0), row(n1);
    double total = 0.0;
    for (int hx = 0; hx <= R; ++hx) {
        std::fill(row.begin(), row.end(), 0.0);
        long samples = 0;
        for (int ky = 0; ky <= R; ++ky) {
            const int d2 = hx * hx + ky * ky;
            if ((hx == 0 && ky == 0) || d2 < min_r * min_r || d2 > R * R) continue;
            const int both = hx > 0 && ky > 0 ? 2 : 1;  // ky and -ky
            samples += both;
            const double* sk = sq.data() + (size_t)ky * n1;
            for (int k = 0; k < n1; ++k) row[k] += both * sk[k];
        }
        total += (double)samples * n1 * n1;
        const double* sm = sq.data() + (size_t)hx * n1;
        for (int m = 0; m < n1; ++m)
            for (int k = 0; k < n1; ++k) e[(size_t)m * n1 + k] += sm[m] * row[k];
    }
    // What is left out (tail, of total) acts on the score like a change of the particle's phases,
    // the same for every sample that carries the signal, so it adds up where rounding averages
    // out: its root mean square stays 5e-5 (BF16) or 4e-4 (e4m3), far below the operands' rounding
    // (1e-3, 2e-2) and, in the score, below what thousands of rounded samples leave of that.
    const double most = f8 ? 1.6e-7 : 2.5e-9;
    auto at = [&](int m, int k) { return m < n1 && k < n1 ? e[(size_t)m * n1 + k] : 0.0; };
    auto place = [&](int b, int m, int k, int part) {
        ob.mx[b] = m;
        ob.my[b] = k;
        ob.part[b] = part;
        ob.slot[((size_t)m * ob.nb + k) * 2 + part] = b;
    };
    auto clear = [&](int nb, int slots) {
        ob.nb = nb;
        ob.slots = slots;
        ob.mx.assign(slots, -1);
        ob.my.assign(slots, -1);
        ob.part.assign(slots, 0);
        ob.slot.assign(2 * (size_t)nb * nb, -1);
    };
    for (int l = 0; l < OB_LAYOUTS && ob.layout < 0; ++l) {
        const OriginLayout& L = OB_LAYOUT[l];
        // (summed from what is out: the difference of two nearly equal sums would not do)
        // likewise the functions that the layouts of few rows leave without the second row that the others
        // give them: 5e-4 of total, 2 % of the rounding of A as it would be with none
        double tail = 0.0, single = 0.0;
        bool whole = true;
        for (int m = 0; m < n1; ++m)
            for (int k = 0; k < n1; ++k)
                if (!L.in(m, k)) {
                    tail += at(m, k);
                    whole = false;
                } else if (l < OB_FEW && !L.twice(m, k) && m + k < 5) {
                    single += at(m, k);
                }
        if (tail > most * total || single > 5e-4 * total) continue;
        if (n1 <= OB_WHOLE && !whole && 8.0 * R * (double)step > n) continue;
        ob.layout = l;
        clear(L.nb, (L.rows + 31) / 32 * 32);
        ob.used = L.rows;
        int b = 0;
        for (int part = 0; part < 2; ++part)
            for (int m = 0; m < L.nb; ++m)
                for (int k = 0; k < L.nb; ++k)
                    if (part ? L.twice(m, k) : L.in(m, k)) {
                        if (m < n1 && k < n1) place(b, m, k, part);
                        ++b;
                    }
    }
    if (ob.layout < 0) {
        // more functions: in the order of their energy, in as many units as it takes, and second
        // rows (worth the energy of their function's rounding, the same order) in the rest
        std::vector<int> ord((size_t)n1 * n1);
        std::iota(ord.begin(), ord.end(), 0);
        std::stable_sort(ord.begin(), ord.end(), [&](int x, int y) { return e[x] > e[y]; });
        size_t cnt = ord.size();
        double tail = 0.0;
        while (cnt > 1 && tail + e[ord[cnt - 1]] <= most * total) tail += e[ord[--cnt]];
        ob.units = (int)((cnt + OB_UNIT - 1) / OB_UNIT);
        int top = 0;
        for (size_t b = 0; b < cnt; ++b) top = std::max(top, std::max(ord[b] / n1, ord[b] % n1) + 1);
        clear(top, ob.units * OB_UNIT);
        ob.used = ob.slots;
        for (size_t b = 0; b < cnt; ++b) place((int)b, ord[b] / n1, ord[b] % n1, 0);
        for (size_t b = cnt; b < (size_t)ob.slots && b < 2 * cnt; ++b)
            place((int)b, ord[b - cnt] / n1, ord[b - cnt] % n1, 1);
    }
    for (int a = 0; 2 * a < ob.nb; ++a) {
        ob.ent_off.push_back((int)ob.ent.size() / 8);
        size_t used = ob.ent.size();
        for (int b = 0; 2 * b < ob.nb; ++b) {
            bool any = false;
            for (int i = 0; i < 4; ++i) {
                const int m = 2 * a + i / 2, k = 2 * b + i % 2;
                const bool in = m < ob.nb && k < ob.nb;
                for (int part = 0; part < 2; ++part) {
                    const int v = in ? ob.slot[((size_t)m * ob.nb + k) * 2 + part] : -1;
                    any = any || v >= 0;
                    ob.ent.push_back(v);
                }
            }
            if (any) used = ob.ent.size();
        }
        ob.ent.resize(used);
        if ((used / 8 - ob.ent_off.back()) & 1) ob.ent.resize(used + 8, -1);
    }
    ob.ent_off.push_back((int)ob.ent.size() / 8);
    ob.q.assign((size_t)ob.nb * n1, 0.0f);
    ob.f.assign((size_t)ob.nb * H, 0.0f);
    ob.ge.assign(ob.nb, 0);
    for (int k = 0; k < std::min(ob.nb, n1); ++k) {
        double fm = 0.0;
        for (int h = 0; h < H; ++h) fm = std::max(fm, std::fabs(f[(size_t)k * H + h]));
        if (f8 && fm > 0.0) ob.ge[k] = std::max(-60, std::min(60, -(int)std::ceil(std::log2(fm))));
        for (int i = 0; i < n1; ++i) ob.q[(size_t)k * n1 + i] = (float)std::ldexp(fun[k][i], -ob.ge[k]);
        for (int h = 0; h < H; ++h) ob.f[(size_t)k * H + h] = (float)std::ldexp(f[(size_t)k * H + h], ob.ge[k]);
    }
    auto hi = [&](int m, int j) { return m < ob.nb && j < he ? ob.q[(size_t)m * n1 + n1 / 2 + j] : 0.0f; };
    const int couples = (ob.nb + 1) / 2;
    for (int j = 0; j < he + 16; j += 2)
        for (int a = 0; a < couples; ++a)
            for (int i = 0; i < 4; ++i) ob.qx.push_back(hi(2 * a + i % 2, j + i / 2));
    for (int j = 0; j < he; ++j)
        for (int m = 0; m < 2 * ((couples + 1) / 2 * 2); ++m) ob.qy.push_back(hi(m, j));
    return ob;
}

}  // namespace cryoim
