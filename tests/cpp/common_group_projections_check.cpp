// Checks common_stabilizers.hpp over many projections, gates and removed qubits,
// against dense vectors: the generators stay independent (no more than qubits),
// stabilize the vector, and hold the projected Z's; a projection on the outcome
// that the generators exclude is reported.  A register of 64 qubits projected
// twice keeps following gates.
#include <complex>
#include <cstdio>
#include <random>

#include "common_stabilizers.hpp"

using namespace nsg;
using C = std::complex<double>;
using V = std::vector<C>;

static V apply(const HPauli& p, const V& v) {
    static const C ph[4] = {1, C(0, 1), -1, C(0, -1)};
    V o(v.size());
    for (size_t x = 0; x < v.size(); x++) o[x ^ p.x] += ph[p.k & 3] * (parity64(x & p.z) ? -1.0 : 1.0) * v[x];
    return o;
}

static void gate(V& v, uint32_t c) {
    const uint32_t op = c & 255, a = (c >> 8) & 255, b = (c >> 16) & 255;
    V o(v.size());
    for (size_t x = 0; x < v.size(); x++) {
        const bool xa = (x >> a) & 1;
        if (op == P_H) {
            o[x] += (xa ? -1.0 : 1.0) * M_SQRT1_2 * v[x];
            o[x ^ (1u << a)] += M_SQRT1_2 * v[x];
        } else if (op == P_S) {
            o[x] = (xa ? C(0, 1) : C(1, 0)) * v[x];
        } else if (op == P_X) {
            o[x ^ (1u << a)] = v[x];
        } else {
            o[xa ? x ^ (1u << b) : x] = v[x];
        }
    }
    v = o;
}

static bool stabilized(const CommonGroup& g, const V& v) {
    for (const HPauli& p : g.gens) {
        const V w = apply(p, v);
        for (size_t i = 0; i < v.size(); i++)
            if (std::abs(w[i] - v[i]) > 1e-9) return false;
    }
    return true;
}

static size_t rank_of(std::vector<HPauli> g) {
    const size_t nx = reduce_rows(g, 0, ~0ull, true).size();
    return nx + reduce_rows(g, nx, ~0ull, false).size();
}

int main() {
    std::mt19937 r(2);
    int bad = 0, refused = 0;
    for (int it = 0; it < 400; it++) {
        const int n = 2 + (int)(r() % 5);
        const int s = (int)(r() % (n + 1));
        V v((size_t)1 << n);
        for (size_t x = 0; x < v.size(); x += (size_t)1 << s) v[x] = C((int)(r() % 2001) - 1000, (int)(r() % 2001) - 1000);
        CommonGroup g;
        for (int i = 0; i < s; i++) g.gens.push_back({0, 1ull << i, 0});
        for (int step = 0; step < 30; step++) {
            std::vector<uint32_t> ops;
            for (int i = (int)(r() % 4); i > 0; i--) {
                const uint32_t kinds[] = {P_H, P_S, P_X, P_CX}, op = kinds[r() % 4], a = r() % n, b = (a + 1 + r() % (n - 1)) % n;
                ops.push_back(enc_op(op, a, op == P_CX ? b : 0));
            }
            for (uint32_t c : ops) gate(v, c);
            bad += !g.apply(ops);
            const int q = (int)(r() % n);
            const bool one = r() % 2;
            V w = v;
            double left = 0, all = 0;
            for (size_t x = 0; x < v.size(); x++) {
                all += std::norm(v[x]);
                if ((bool)((x >> q) & 1) != one) w[x] = 0;
                left += std::norm(w[x]);
            }
            CommonGroup h = g;
            const bool ok = h.project(q, one);
            if (left < 1e-9 * all) {  // no state is left; the generators may not know
                refused += !ok;
                continue;
            }
            bad += !ok;
            for (C& x : w) x /= std::sqrt(left);
            v = w;
            g = h;
            bad += !stabilized(g, v) || g.gens.size() > (size_t)n || rank_of(g.gens) != g.gens.size();
            std::vector<HPauli> more = g.gens;
            more.push_back({0, 1ull << q, 0});
            bad += rank_of(more) != g.gens.size();
        }
    }
    CommonGroup g;  // every qubit, twice
    for (int pass = 0; pass < 2; pass++)
        for (int q = 0; q < 64; q++) bad += !g.project(q, q & 1);
    bad += g.gens.size() != 64 || !g.apply({enc_op(P_H, 5)});
    bool x5 = false;
    for (const HPauli& p : g.gens) x5 = x5 || (p.x == 1ull << 5 && p.z == 0 && p.k == 2);
    bad += !x5;
    std::printf("bad %d refused %d\n", bad, refused);
    return bad == 0 && refused > 50 ? 0 : 1;
}
