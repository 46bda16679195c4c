// kernels_reduce.cu — the stabilizers shared by all terms of a state, and the
// terms on the qubits that those leave.
//
// The χ² pair sums (kernels_pairs.cu) cost about n² word operations a pair, and
// the terms of one state mostly agree on a large part of their stabilizers (a
// compiled state of t T gates on n - t of them at least).  Two kernels find that
// part and divide it out; the host side between them is common_stabilizers.hpp.
#include <cuda_runtime.h>

#include <climits>

#include "device_state.hpp"
#include "warp_chform.cuh"

namespace nsg {
namespace {

using dev::FULL;
using dev::shfl;

// The rows of one term in shared memory (n ≤ 64).
struct TermRows {
    uint64_t F[64], M[64], G[64];
};

__device__ __forceinline__ void load_rows(TermRows& s, const TermsView& tv, int64_t term, int lane) {
    for (int r = lane; r < 64; r += 32) {
        const size_t idx = ((size_t)term * tv.R + r) * tv.W;  // word 0 (n ≤ 64)
        s.F[r] = tv.F[idx];
        s.M[r] = tv.M[idx];
        s.G[r] = tv.G[idx];
    }
}

// U_C^{-1} (i^k X(x) Z(z)) U_C = i^{k'} X(a) Z(b) for the Paulis of one lane.
template <int NP>
__device__ __forceinline__ void conj_by_term(const TermRows& s, int n, uint64_t gl, uint64_t gh,
                                             const uint64_t (&x)[NP], const uint64_t (&z)[NP], const int (&k)[NP],
                                             uint64_t (&a)[NP], uint64_t (&b)[NP], int (&kk)[NP]) {
    uint64_t m[NP];
    int cnt[NP];
#pragma unroll
    for (int t = 0; t < NP; t++) {
        a[t] = b[t] = m[t] = 0;
        cnt[t] = 0;
    }
#pragma unroll 4
    for (int q = 0; q < n; q++) {
        const uint64_t f = s.F[q], mm = s.M[q], g = s.G[q];
#pragma unroll
        for (int t = 0; t < NP; t++) {
            if ((x[t] >> q) & 1) {
                cnt[t] += __popcll(m[t] & f);
                m[t] ^= mm;
                a[t] ^= f;
            }
            if ((z[t] >> q) & 1) b[t] ^= g;
        }
    }
#pragma unroll
    for (int t = 0; t < NP; t++) {
        b[t] ^= m[t];
        kk[t] = (k[t] + __popcll(x[t] & gl) + 2 * __popcll(x[t] & gh) + 2 * cnt[t]) & 3;
    }
}

// ---- common stabilizers --------------------------------------------------------
// One block of 32 warps per state; warp w holds one term's rows.  Every warp
// holds the same ≤ 64 Paulis (two per lane), generators of term 0's stabilizer
// group to begin with, and how far each is from stabilizing the warp's own term:
// the bits of U_C^{-1} Q U_C that are no Z on ¬v or no X on v, linear in Q.  One
// elimination over the 32 terms keeps the products without such bits, a second
// over their 32 signs those with eigenvalue +1 on every term.  Then 32 more
// terms.  What is left stabilizes up to 64 sampled terms; the reduction kernel
// checks every term (a term it fails on is sampled first the next time).
// Latency-bound: 64 steps over shared rows and a few syncs per eliminated
// generator, 80-100 us whatever χ is (n = 50 and 64), once per state: gates,
// projections and discards carry the group on the host.
constexpr int CWARPS = 32;

struct CommonShared {
    TermRows rows[CWARPS];
    uint64_t gx[64], gz[64];
    int gk[64];
    uint64_t mask[2];
    uint32_t sign_lo[CWARPS], sign_hi[CWARPS];
    int key[2], vsum;
};

__device__ __forceinline__ int64_t sampled_term(const CommonDesc& d, int i) {
    const int64_t chi = d.tv.chi;
    if (i < d.nextra) return d.extra[i];
    if (chi <= 2 * CWARPS) return i - d.nextra;  // every term, in turn
    if (i == d.nextra) return 0;
    // scattered over all the digits of the term index
    return (int64_t)(((uint64_t)i * 0x9E3779B97F4A7C15ull >> 20) % (uint64_t)chi);
}

__global__ void __launch_bounds__(CWARPS * 32) common_kernel(const CommonDesc* __restrict__ descs,
                                                             CommonOut* __restrict__ outs) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    CommonShared& sh = *(CommonShared*)smem_raw;
    const CommonDesc& d = descs[blockIdx.x];
    const TermsView tv = d.tv;
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = tv.n;
    uint64_t x[2], z[2], viol[2] = {0, 0}, a[2], b[2];
    int k[2], kk[2];
    uint64_t alive = n >= 64 ? ~0ull : (1ull << n) - 1;  // the same in every warp

    // Generators of term 0: U_C Z_j U_C^{-1} (v_j = 0) or U_C X_j U_C^{-1} (v_j = 1), times (-1)^{s_j}.
    if (wid == 0) load_rows(sh.rows[0], tv, 0, lane);
    if (threadIdx.x == 0) {
        sh.key[0] = sh.key[1] = INT_MAX;
        sh.vsum = 0;
    }
    __syncthreads();
    if (threadIdx.x < 64) {
        const int j = threadIdx.x;
        const TermRows& s = sh.rows[0];
        uint64_t xx = 0, zz = 0;
        int ph = 0;
        if (j < n) {
            const uint64_t v = tv.V[0], sv = tv.S[0];
            if ((v >> j) & 1) {  // i^{γ_V} X(F_V) Z(M_V), the inverse tableau (see frames_kernel)
                uint64_t y = 0;
                int cnt = 0;
                for (int q = 0; q < n; q++)
                    if ((s.G[q] >> j) & 1) {
                        xx |= 1ull << q;
                        cnt += __popcll(y & s.F[q]);
                        y ^= s.M[q];
                    }
                for (int c = 0; c < n; c++) zz |= (uint64_t)(__popcll(y & s.F[c]) & 1) << c;
                ph = -(__popcll(xx & tv.GL[0]) + 2 * __popcll(xx & tv.GH[0])) + 2 * cnt;
            } else {
                for (int q = 0; q < n; q++) zz |= ((s.F[q] >> j) & 1) << q;
            }
            ph += 2 * (int)((sv >> j) & 1);
        }
        sh.gx[j] = xx;
        sh.gz[j] = zz;
        sh.gk[j] = ph & 3;
    }
    __syncthreads();
#pragma unroll
    for (int t = 0; t < 2; t++) {
        x[t] = sh.gx[32 * t + lane];
        z[t] = sh.gz[32 * t + lane];
        k[t] = sh.gk[32 * t + lane];
    }
    const int total = d.tv.chi <= 2 * CWARPS ? (int)d.tv.chi + d.nextra : 2 * CWARPS;
    // multiply element e into the elements of m (e ∉ m) and drop it
    auto eliminate = [&](int e, uint64_t m) {
        const int es = e >> 5, el = e & 31;
        const uint64_t px = shfl<uint64_t>(es ? x[1] : x[0], el), pz = shfl<uint64_t>(es ? z[1] : z[0], el),
                       pv = shfl<uint64_t>(es ? viol[1] : viol[0], el);
        const int pk = __shfl_sync(FULL, es ? k[1] : k[0], el);
#pragma unroll
        for (int t = 0; t < 2; t++)
            if ((m >> (32 * t + lane)) & 1) {
                k[t] = (k[t] + pk + 2 * __popcll(z[t] & px)) & 3;
                x[t] ^= px;
                z[t] ^= pz;
                viol[t] ^= pv;
            }
        alive &= ~(1ull << e);
    };
    for (int batch = 0; batch * CWARPS < total; batch++) {
        const bool active = batch * CWARPS + wid < total;
        uint64_t v = 0, sv = 0, gl = 0, gh = 0;
        __syncthreads();  // rows of the last batch are read
        if (active) {
            const int64_t term = sampled_term(d, batch * CWARPS + wid);
            load_rows(sh.rows[wid], tv, term, lane);
            v = tv.V[term * tv.W];
            sv = tv.S[term * tv.W];
            gl = tv.GL[term * tv.W];
            gh = tv.GH[term * tv.W];
            if (lane == 0) atomicAdd(&sh.vsum, __popcll(v));
        }
        __syncwarp();
        auto evaluate = [&]() {  // viol, and the sign of elements without any (bit 1 of kk)
            if (active) {
                conj_by_term<2>(sh.rows[wid], n, gl, gh, x, z, k, a, b, kk);
#pragma unroll
                for (int t = 0; t < 2; t++) {
                    viol[t] = (a[t] & ~v) | (b[t] & v);
                    kk[t] = (kk[t] + 2 * __popcll((a[t] ^ b[t]) & sv)) & 3;
                }
            } else {
                viol[0] = viol[1] = 0;
                kk[0] = kk[1] = 0;
            }
        };
        evaluate();
        bool changed = false;
        int par = 0;
        while (true) {
            const uint64_t bad = ((uint64_t)__ballot_sync(FULL, viol[0] != 0) |
                                  ((uint64_t)__ballot_sync(FULL, viol[1] != 0) << 32)) & alive;
            if (bad && lane == 0) atomicMin(&sh.key[par], wid * 64 + (__ffsll((long long)bad) - 1));
            __syncthreads();
            const int key = sh.key[par];
            if (key == INT_MAX) break;
            const int e = key & 63;
            if (wid == key >> 6) {  // the elements that share the pivot bit
                const uint64_t ve = shfl<uint64_t>((e >> 5) ? viol[1] : viol[0], e & 31);
                const uint64_t bit = ve & (~ve + 1);
                const uint64_t m = ((uint64_t)__ballot_sync(FULL, (viol[0] & bit) != 0) |
                                    ((uint64_t)__ballot_sync(FULL, (viol[1] & bit) != 0) << 32)) & alive;
                if (lane == 0) {
                    sh.mask[par] = m & ~(1ull << e);
                    sh.key[par ^ 1] = INT_MAX;
                }
            }
            __syncthreads();
            eliminate(e, sh.mask[par]);
            changed = true;
            par ^= 1;
        }
        __syncthreads();  // everyone has read the last key
        if (threadIdx.x == 0) sh.key[0] = sh.key[1] = INT_MAX;
        if (changed) evaluate();
        const uint32_t s0 = __ballot_sync(FULL, kk[0] & 2), s1 = __ballot_sync(FULL, kk[1] & 2);
        if (lane == 0) {
            sh.sign_lo[wid] = s0;
            sh.sign_hi[wid] = s1;
        }
        __syncthreads();
        // lane w: the signs on warp w's term; every warp runs the same elimination
        uint64_t sg = (uint64_t)sh.sign_lo[lane] | ((uint64_t)sh.sign_hi[lane] << 32);
        while (true) {
            const uint32_t some = __ballot_sync(FULL, (sg & alive) != 0);
            if (!some) break;
            const uint64_t m = shfl<uint64_t>(sg, __ffs(some) - 1) & alive;
            const int e = __ffsll((long long)m) - 1;
            const uint64_t rest = m & ~(1ull << e);
            if ((sg >> e) & 1) sg ^= rest;
            eliminate(e, rest);
        }
    }
    if (wid == 0) {
        CommonOut& o = outs[blockIdx.x];
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int e = 32 * t + lane;
            if ((alive >> e) & 1) {
                const int at = __popcll(alive & ((1ull << e) - 1));
                o.x[at] = x[t];
                o.z[at] = z[t];
                o.k[at] = (uint8_t)k[t];
            }
        }
        if (lane == 0) {
            o.count = __popcll(alive);
            o.sampled = total;
            o.vsum = sh.vsum;
        }
    }
}

// ---- reduced terms ---------------------------------------------------------------
// One warp per term.  The amplitudes of the reduced term, ⟨x|t⟩ =
// 2^{r_X/2}·⟨0|X'(x)|s⟩, are read off the images of the logical operators X'_q:
// with i^{γ_q} X(F_q) Z(M_q) = U_C^{-1} X'_q U_C they are
//   ω^phase·2^{-|v'|/2}·i^{L·x}·(-1)^{Σ_{p<r} J_pr x_p x_r}·[(xF ⊕ s) ∧ ¬v = 0],
// J_pr = M_max·F_min, L_p = γ_p + 2(M_p·F_p + F_p·(v ∧ s)).  The constraints are
// reduced (z_p = rhs_p ⊕ R_p·z for a pivot p, the other variables free), which
// gives a CH-form of n2 qubits: D = Π S^{L_p} Π CZ^{J_pr} after the linear map
// u ↦ x, x_p = u_p ⊕ R_p·u on pivots; v' the free variables, s' = rhs.
// The generators are evaluated too: each has to stabilize the term.  Bound by
// integer work: 10 us for 486 terms of n = 50, 14 us for 1,458 of n = 64, about
// two pairs' work a term, against half a χ of pairs that get shorter: the pair
// launch of n = 60, χ = 8,748, 256 observables went from 478 to 68 ms, that of
// n = 40, χ = 972, 64 observables from 1.18 to 0.45 ms.
constexpr int RWARPS = 4;

__global__ void __launch_bounds__(RWARPS * 32) reduce_terms_kernel(const ReduceDesc* __restrict__ descs, int num,
                                                                   int64_t total) {
    __shared__ TermRows rows[RWARPS];
    __shared__ uint64_t sA[RWARPS][64], sB[RWARPS][64];
    const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t gterm = (int64_t)blockIdx.x * RWARPS + wid;
    if (gterm >= total) return;
    int lo = 0, hi = num;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (descs[mid].term0 <= gterm) lo = mid;
        else hi = mid;
    }
    const ReduceDesc& d = descs[lo];
    const TermsView tv = d.in, o = d.out;
    const int64_t term = gterm - d.term0;
    const int n = tv.n, n2 = o.n;
    TermRows& s = rows[wid];
    load_rows(s, tv, term, lane);
    __syncwarp();
    const uint64_t v = tv.V[term * tv.W], gl = tv.GL[term * tv.W], gh = tv.GH[term * tv.W];
    uint64_t sv = tv.S[term * tv.W];
    int phase = tv.phase[term];
    uint64_t x[2], z[2], a[2], b[2];
    int k[2], kk[2];
    if (d.x0) {  // X(x0) first: i^g X(a) Z(b) in the term's frame, on U_H|s⟩
        const uint64_t x1[1] = {d.x0}, z1[1] = {0};
        const int k1[1] = {0};
        uint64_t a1[1], b1[1];
        int g1[1];
        conj_by_term<1>(s, n, gl, gh, x1, z1, k1, a1, b1, g1);
        const uint64_t bv = b1[0] & v;
        phase += 2 * g1[0] + 4 * __popcll((b1[0] & ~v & sv) ^ (a1[0] & v & (sv ^ bv)));
        sv ^= (a1[0] & ~v) ^ bv;
    }
    // rows 0 .. n2-1: the logical X; then the n - n2 generators
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int r = 32 * t + lane;
        x[t] = r < n ? d.rows[r].x : 0;
        z[t] = r < n ? d.rows[r].z : 0;
        k[t] = r < n ? d.rows[r].k : 0;
    }
    conj_by_term<2>(s, n, gl, gh, x, z, k, a, b, kk);
    bool bad = false;
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int r = 32 * t + lane;
        if (r >= n2 && r < n)
            bad |= (((a[t] & ~v) | (b[t] & v)) != 0) || ((kk[t] + 2 * __popcll((a[t] ^ b[t]) & sv)) & 3);
    }
    __syncwarp();
    uint64_t* sF = sA[wid];
    uint64_t* sM = sB[wid];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int r = 32 * t + lane;
        sF[r] = r < n2 ? a[t] : 0;
        sM[r] = r < n2 ? b[t] : 0;
    }
    __syncwarp();
    // J with L's odd bits on its diagonal, and L
    uint64_t J[2];
    int L[2];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int p = 32 * t + lane;
        uint64_t j = 0;
        if (p < n2) {
            for (int r = 0; r < n2; r++) {
                const uint64_t m = r <= p ? b[t] : sM[r], f = r <= p ? sF[r] : a[t];
                j |= (uint64_t)(__popcll(m & f) & 1) << r;
            }
            L[t] = (kk[t] + 2 * (int)((j >> p) & 1) + 2 * __popcll(a[t] & v & sv)) & 3;
            j = (j & ~(1ull << p)) | ((uint64_t)(L[t] & 1) << p);
        } else {
            L[t] = 0;
        }
        J[t] = j;
    }
    // constraints (xF)_c = s_c for c ∉ v, solved for pivots: z_p = rr_p ⊕ R_p·z
    uint64_t Fc[2] = {lane < n2 ? a[0] : 0, lane + 32 < n2 ? a[1] : 0};
    uint64_t R[2] = {0, 0}, piv = 0;
    bool rr[2] = {false, false};
    uint64_t cons = ~v & (n >= 64 ? ~0ull : (1ull << n) - 1), rs = sv;
    while (cons) {
        const uint64_t c = cons & (~cons + 1);
        cons ^= c;
        const uint64_t l = (uint64_t)__ballot_sync(FULL, (Fc[0] & c) != 0) |
                           ((uint64_t)__ballot_sync(FULL, (Fc[1] & c) != 0) << 32);
        const bool rb = (rs & c) != 0;
        if (!l) {
            bad |= rb;  // no amplitude at all: the generators do not fit this term
            continue;
        }
        const int p = __ffsll((long long)l) - 1;
        const uint64_t lp = l & (l - 1);
        const uint64_t Fp = shfl<uint64_t>(p < 32 ? Fc[0] : Fc[1], p & 31);
        if (rb) rs ^= Fp;
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int q = 32 * t + lane;
            if ((lp >> q) & 1) Fc[t] ^= Fp;
            if ((R[t] >> p) & 1) {  // an earlier pivot's solution used z_p
                R[t] = (R[t] & ~(1ull << p)) ^ lp;
                rr[t] ^= rb;
            }
            if (q == p) {
                Fc[t] = 0;
                R[t] = lp;
                rr[t] = rb;
            }
        }
        piv |= 1ull << p;
    }
    const uint64_t full2 = n2 >= 64 ? ~0ull : (1ull << n2) - 1;
    const uint64_t v2 = full2 & ~piv;
    bad |= __popcll(v) - d.rx != __popcll(v2);  // the amplitudes' norm
    // G_p = e_p (⊕ R_p on pivots), F = G^{-T}, M = (J ⊕ diag(L mod 2))·G, γ = -L
    uint64_t Fo[2], Mo[2];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int q = 32 * t + lane;
        Fo[t] = q < n2 ? 1ull << q : 0;
        Mo[t] = J[t];
    }
    uint64_t pm = piv;
    while (pm) {
        const int p = __ffsll((long long)pm) - 1;
        pm &= pm - 1;
        const uint64_t Rp = shfl<uint64_t>(p < 32 ? R[0] : R[1], p & 31);
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int q = 32 * t + lane;
            if ((Rp >> q) & 1) Fo[t] |= 1ull << p;
            if ((J[t] >> p) & 1) Mo[t] ^= Rp;
        }
    }
    uint64_t gl2 = 0, gh2 = 0, s2 = 0;
#pragma unroll
    for (int t = 0; t < 2; t++) {
        const int q = 32 * t + lane;
        const size_t idx = (size_t)term * 64 + q;
        o.G[idx] = q < n2 ? (1ull << q) ^ R[t] : 0;
        o.F[idx] = Fo[t];
        o.M[idx] = q < n2 ? Mo[t] : 0;
        const int g = -L[t] & 3;
        gl2 |= (uint64_t)__ballot_sync(FULL, q < n2 && (g & 1)) << (32 * t);
        gh2 |= (uint64_t)__ballot_sync(FULL, q < n2 && (g & 2)) << (32 * t);
        s2 |= (uint64_t)__ballot_sync(FULL, rr[t]) << (32 * t);
    }
    // the term as a quadratic form, for the form pair kernel
    unsigned char* fp = d.forms + (size_t)term * (sizeof(FormHeader) + (n2 <= 32 ? 256 : 1024));  // form_bytes(n2)
    const uint64_t l0 = (uint64_t)__ballot_sync(FULL, L[0] & 1) | ((uint64_t)__ballot_sync(FULL, L[1] & 1) << 32);
    const uint64_t l1 = (uint64_t)__ballot_sync(FULL, L[0] & 2) | ((uint64_t)__ballot_sync(FULL, L[1] & 2) << 32);
    if (n2 <= 32) {
        uint32_t* rw = (uint32_t*)(fp + sizeof(FormHeader));
        rw[lane] = (uint32_t)(J[0] & ~(1ull << lane));
        rw[32 + lane] = (uint32_t)R[0];
    } else {
        uint64_t* rw = (uint64_t*)(fp + sizeof(FormHeader));
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int q = 32 * t + lane;
            rw[q] = J[t] & ~(1ull << q);
            rw[64 + q] = R[t];
        }
    }
    const bool any_bad = __any_sync(FULL, bad);
    if (lane == 0) {
        FormHeader h;
        h.L0 = l0;
        h.L1 = l1;
        h.piv = piv;
        h.rhs = s2;
        h.r = __popcll(v2);
        h.coef_r = tv.coef_r[term];
        h.phase = (uint8_t)(phase & 7);
        h.coef_k = tv.coef_k[term];
        for (int t = 0; t < 6; t++) h.pad[t] = 0;
        *(FormHeader*)fp = h;
        o.V[term] = v2;
        o.S[term] = s2;
        o.GL[term] = gl2;
        o.GH[term] = gh2;
        o.phase[term] = (uint8_t)(phase & 7);
        o.coef_k[term] = tv.coef_k[term];
        o.coef_r[term] = tv.coef_r[term];
        if ((uint32_t)term % d.v_stride == 0) atomicAdd(&d.flag[kReduceFlags - 1], __popcll(v2));
        if (any_bad) {
            const int at = atomicAdd(&d.flag[0], 1);
            if (at < kMaxBadTerms) d.flag[1 + at] = (int)term;
        }
    }
}

}  // namespace

cudaError_t launch_common(const CommonDesc* descs, CommonOut* outs, int num, cudaStream_t st) {
    if (num == 0) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(common_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(CommonShared));
    if (e != cudaSuccess) return e;
    common_kernel<<<num, CWARPS * 32, sizeof(CommonShared), st>>>(descs, outs);
    return cudaGetLastError();
}

cudaError_t launch_reduce_terms(const ReduceDesc* descs, int num, int64_t total, cudaStream_t st) {
    if (num == 0 || total == 0) return cudaSuccess;
    reduce_terms_kernel<<<(unsigned)((total + RWARPS - 1) / RWARPS), RWARPS * 32, 0, st>>>(descs, num, total);
    return cudaGetLastError();
}

}  // namespace nsg
