// common_stabilizers.hpp — host side of the reduction of a state by the
// stabilizers that all of its terms share.
//
// If every term satisfies g|s_k⟩ = |s_k⟩ for each g of a commuting set of r
// independent Paulis, then |s_k⟩ = C (|+…+⟩ ⊗ |0…0⟩ ⊗ |t_k⟩) with one control-
// type Clifford C for all k (C fixes ⟨0^n|), so the pair values of the terms are
// those of the t_k on n − r qubits: ⟨s_a|P|s_b⟩ = ⟨t_a|P'|t_b⟩, or 0 for a P
// that anticommutes with some g.  A compiled state of t T gates shares at least
// n − t of them.  Nothing here needs C itself: the logical X operators X'_q,
// q = 1 … n − r, that read the amplitudes ⟨x|t_k⟩ = 2^{r_X/2}·⟨0^n|X'(x)|s_k⟩
// off the terms, and the map P ↦ P' follow from the reduced generators.
#pragma once

#include <cstdint>
#include <utility>
#include <vector>

#include "device_state.hpp"

namespace nsg {

inline int parity64(uint64_t x) { return __builtin_popcountll(x) & 1; }

// i^k X(x) Z(z).
struct HPauli {
    uint64_t x = 0, z = 0;
    int k = 0;
    HPauli operator*(const HPauli& o) const { return {x ^ o.x, z ^ o.z, (k + o.k + 2 * parity64(z & o.x)) & 3}; }
    bool anticommutes(const HPauli& o) const { return parity64((x & o.z)) != parity64((z & o.x)); }
};

// 64×64 bit-matrix transpose in place (row i = word i), by recursive block swaps
// (H. S. Warren, Hacker's Delight, section 7-3).
inline void transpose64(uint64_t (&a)[64]) {
    uint64_t m = 0x00000000ffffffffull;
    for (int j = 32; j; j >>= 1, m ^= m << j)
        for (int k = 0; k < 64; k = (k + j + 1) & ~j) {
            const uint64_t t = ((a[k] >> j) ^ a[k + j]) & m;
            a[k] ^= t << j;
            a[k + j] ^= t;
        }
}

// Independent generators of a group of stabilizers common to all terms of a
// state: at most as many as qubits.
struct CommonGroup {
    std::vector<HPauli> gens;
    // Mean |v| of sampled terms, for a choice of kernels only, and the H gates and
    // projections since they were sampled: each changes a term's |v| by one at most.
    double mean_v = -1.0;
    int v_changes = 0;
    void v_changed() { v_changes = v_changes < 128 ? v_changes + 1 : v_changes; }

    // Conjugation by Clifford gates, all generators at once: bit i of X[q], Z[q]
    // is generator i's at qubit q, of R its sign as a product of I, X, Y, Z
    // (i^k X(x) Z(z) has k = #Y + 2·sign).  False: more generators than a word has
    // bits, which stay as they are (nothing is known then).
    bool apply(const std::vector<uint32_t>& ops) {
        for (uint32_t c : ops)
            if ((c & 0xff) == P_H) v_changed();
        if (gens.empty()) return true;
        if (gens.size() > 64) return false;
        uint64_t X[64] = {}, Z[64] = {}, R = 0;
        for (size_t i = 0; i < gens.size(); i++) {
            X[i] = gens[i].x;
            Z[i] = gens[i].z;
            const int y = __builtin_popcountll(gens[i].x & gens[i].z);
            R |= (uint64_t)(((gens[i].k - y) >> 1) & 1) << i;
        }
        transpose64(X);
        transpose64(Z);
        for (uint32_t c : ops) {
            const uint32_t op = c & 0xff, a = (c >> 8) & 0xff, b = (c >> 16) & 0xff;
            switch (op) {
                case P_H:  // the only gate that changes v
                    R ^= X[a] & Z[a];
                    std::swap(X[a], Z[a]);
                    break;
                case P_S:
                    R ^= X[a] & Z[a];
                    Z[a] ^= X[a];
                    break;
                case P_SDG:
                    R ^= X[a] & ~Z[a];
                    Z[a] ^= X[a];
                    break;
                case P_X: R ^= Z[a]; break;
                case P_Y: R ^= X[a] ^ Z[a]; break;
                case P_Z: R ^= X[a]; break;
                case P_CX:
                    R ^= X[a] & Z[b] & ~(X[b] ^ Z[a]);
                    X[b] ^= X[a];
                    Z[a] ^= Z[b];
                    break;
                case P_CZ:
                    R ^= X[a] & X[b] & (Z[a] ^ Z[b]);
                    Z[a] ^= X[b];
                    Z[b] ^= X[a];
                    break;
                default: break;
            }
        }
        transpose64(X);
        transpose64(Z);
        for (size_t i = 0; i < gens.size(); i++) {
            gens[i].x = X[i];
            gens[i].z = Z[i];
            gens[i].k = (__builtin_popcountll(X[i] & Z[i]) + 2 * (int)((R >> i) & 1)) & 3;
        }
        return true;
    }
    // The group after every term was projected on Z_q = (-1)^outcome (terms that
    // it annihilates left the state): the elements that commute with Z_q, and Z_q.
    // False if -Z_q is one of them: no term is left, and nothing is known.
    bool project(int q, bool outcome);
    // The group after qubit q (in |0⟩ in every term) was removed; false if Z_q
    // is not among the elements (then nothing is known).
    bool discard(int q);
};

// The reduction by a group: kept qubits and the operators that read them.
struct Reduction {
    int n = 0, n2 = 0, rx = 0;     // width, reduced width, X-type generators
    std::vector<HPauli> gx;        // i^k X(a_i) Z(z_i), a_i reduced: pivot bit px[i] in row i only
    std::vector<int> px;
    std::vector<uint64_t> gz;      // Z(h_j), pivot bit pz[j] in row j only, off the X pivots
    std::vector<int> pz;
    uint64_t x0 = 0;               // X(x0) turns every generator's sign to + (applied to the terms first)
    std::vector<int> kept;         // q: the reduced qubits' bits
    std::vector<uint64_t> ax, bz;  // X'_q = X(ax) Z(bz)

    // False when the generators contradict one another (no state has them all).
    bool build(int width, std::vector<HPauli> g);
    // P ↦ P'; false: P anticommutes with a generator, every pair value is 0.
    bool map(const DevPauli& p, DevPauli& out) const;
};

// Rows of i^k X(x) Z(z) reduced on the bits `cols` of x (or z): returns the
// pivot bits of the first rows; the other rows are zero there.
inline std::vector<int> reduce_rows(std::vector<HPauli>& g, size_t from, uint64_t cols, bool on_x) {
    std::vector<int> piv;
    size_t row = from;
    for (int c = 0; c < 64 && row < g.size(); c++) {
        if (!((cols >> c) & 1)) continue;
        size_t r = row;
        while (r < g.size() && !(((on_x ? g[r].x : g[r].z) >> c) & 1)) r++;
        if (r == g.size()) continue;
        std::swap(g[r], g[row]);
        for (size_t k = from; k < g.size(); k++)
            if (k != row && (((on_x ? g[k].x : g[k].z) >> c) & 1)) g[k] = g[k] * g[row];
        piv.push_back(c);
        row++;
    }
    return piv;
}

inline bool Reduction::build(int width, std::vector<HPauli> g) {
    *this = Reduction();
    n = width;
    const uint64_t all = n >= 64 ? ~0ull : (1ull << n) - 1;
    px = reduce_rows(g, 0, all, true);
    const size_t nx = px.size();
    uint64_t pmask = 0;
    for (int p : px) pmask |= 1ull << p;
    // Z-type rows commute with the X-type ones, so none is supported on X pivots alone.
    pz = reduce_rows(g, nx, all & ~pmask, false);
    for (size_t r = nx + pz.size(); r < g.size(); r++)
        if (g[r].k & 2) return false;  // -1 in the group
    while (nx + pz.size() >= (size_t)n && n > 0) {  // keep one qubit at least: the last generator is not used
        if (!pz.empty()) pz.pop_back();
        else px.pop_back();
        if (nx > px.size()) break;
    }
    rx = (int)px.size();
    uint64_t used = 0;
    for (size_t j = 0; j < pz.size(); j++) {
        gz.push_back(g[nx + j].z);
        if (g[nx + j].k & 2) x0 |= 1ull << pz[j];
        used |= 1ull << pz[j];
    }
    for (int i = 0; i < rx; i++) {
        HPauli p = g[i];
        p.k = (p.k + 2 * parity64(x0 & p.z)) & 3;
        gx.push_back(p);
        used |= 1ull << px[i];
    }
    for (int q = 0; q < n; q++) {
        if ((used >> q) & 1) continue;
        uint64_t a = 1ull << q, b = 0;
        for (size_t j = 0; j < pz.size(); j++)
            if ((gz[j] >> q) & 1) a |= 1ull << pz[j];
        for (int i = 0; i < rx; i++)
            if (parity64(a & gx[i].z)) b |= 1ull << px[i];
        kept.push_back(q);
        ax.push_back(a);
        bz.push_back(b);
    }
    n2 = (int)kept.size();
    return true;
}

inline bool Reduction::map(const DevPauli& p, DevPauli& out) const {
    for (uint64_t h : gz)
        if (parity64(h & p.px)) return false;
    HPauli g;  // Π g_i^{α_i}: the pivot bits of P's X part
    for (int i = 0; i < rx; i++) {
        if (parity64(gx[i].z & p.px) != parity64(gx[i].x & p.pz)) return false;
        if ((p.px >> px[i]) & 1) g = g * gx[i];
    }
    uint64_t beta = 0;
    HPauli r;  // X'(β)·Π g_i^{α_i}: P's X part
    for (int q = 0; q < n2; q++)
        if (((p.px ^ g.x) >> kept[q]) & 1) {
            beta |= 1ull << q;
            r = r * HPauli{ax[q], bz[q], 0};
        }
    r = r * g;
    // P = i^{ny'} X'(β) Z(z) Π g_i^{α_i}; Z(z) acts on the reduced qubits as Π Z_q^{z·a_q}
    const uint64_t z = r.z ^ p.pz;
    out.px = beta;
    out.pz = 0;
    for (int q = 0; q < n2; q++)
        if (parity64(z & ax[q])) out.pz |= 1ull << q;
    out.ny = (p.ny + 2 * parity64(x0 & p.pz) - r.k + 2 * parity64(z & g.x)) & 3;
    out.pad = 0;
    return true;
}

// Whether X(x) Z(z) is a product of the rows up to a power of i.  On bits alone, since
// every projection asks: 33 projections of 33 qubits take 13 us on the host, 35 where
// each eliminates with signs.
inline bool depends(const std::vector<HPauli>& g, uint64_t x, uint64_t z) {
    std::vector<std::pair<uint64_t, uint64_t>> rows;
    for (const HPauli& p : g) rows.push_back({p.x, p.z});
    for (size_t i = 0; i < rows.size(); i++) {
        const auto [px, pz] = rows[i];
        const uint64_t bx = px & (0 - px), bz = px ? 0 : pz & (0 - pz);  // the row's lowest bit
        if (!(bx | bz)) continue;
        for (size_t k = i + 1; k < rows.size(); k++) {
            const uint64_t has = 0 - (uint64_t)(((rows[k].first & bx) | (rows[k].second & bz)) != 0);
            rows[k].first ^= px & has;
            rows[k].second ^= pz & has;
        }
        if ((x & bx) | (z & bz)) {
            x ^= px;
            z ^= pz;
        }
    }
    return !(x | z);
}

inline bool CommonGroup::project(int q, bool outcome) {
    v_changed();
    const HPauli zq{0, 1ull << q, outcome ? 2 : 0};
    std::vector<HPauli> out;
    const HPauli* pivot = nullptr;
    for (const HPauli& g : gens) {
        if (!((g.x >> q) & 1)) out.push_back(g);
        else if (!pivot) pivot = &g;
        else out.push_back(g * *pivot);
    }
    if (!pivot && depends(gens, 0, 1ull << q)) {  // Z_q or -Z_q is an element: its sign
        std::vector<HPauli> rows = gens;
        const size_t nx = reduce_rows(rows, 0, ~0ull, true).size();
        const std::vector<int> pz = reduce_rows(rows, nx, ~0ull, false);
        HPauli rest = zq;
        for (size_t j = 0; j < pz.size(); j++)
            if ((rest.z >> pz[j]) & 1) rest = rest * rows[nx + j];
        return !(rest.k & 2);
    }
    out.push_back(zq);
    gens = std::move(out);
    return true;
}

inline bool CommonGroup::discard(int q) {
    v_changed();
    const uint64_t bit = 1ull << q;
    // bring Z_q to a row of its own: reduce on z with column q last, over the Z-type rows
    std::vector<HPauli> g = gens;
    const std::vector<int> px = reduce_rows(g, 0, ~0ull, true);
    const size_t nx = px.size();
    reduce_rows(g, nx, ~0ull & ~bit, false);
    size_t at = g.size();
    for (size_t r = nx; r < g.size(); r++)
        if (g[r].x == 0 && g[r].z == bit && !(g[r].k & 2)) at = r;
    if (at == g.size()) return false;
    std::vector<HPauli> out;
    const uint64_t low = bit - 1;
    for (size_t r = 0; r < g.size(); r++) {
        if (r == at || (g[r].x == 0 && g[r].z == 0)) continue;
        HPauli p = (g[r].z & bit) ? g[r] * HPauli{0, bit, 0} : g[r];
        if (p.x & bit) return false;
        p.x = (p.x & low) | ((p.x >> 1) & ~low);
        p.z = (p.z & low) | ((p.z >> 1) & ~low);
        out.push_back(p);
    }
    gens = std::move(out);
    return true;
}

}  // namespace nsg
