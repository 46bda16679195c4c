// kernels_dense.cu — the amplitudes of a decomposed state as exact integers,
// and what is summed from them: ⟨P⟩, outcome weights, the state vector.
//
// Every amplitude is Σ_k ω^{k0}·i^{Q_k(x)}·2^{-r_k/2} over the terms whose
// support holds x, so ψ(x)·2^{R/2} (R the largest r_k) is an integer combination
// c0 + c1 ω + c2 ω² + c3 ω³ of the eighth roots of unity, and every ⟨P⟩ is
// 2^{-R}·(X + Y/√2) with integers X, Y: nothing is rounded before the end, and
// a value that is zero comes out as zero.  With few qubits and many terms this
// is far less work than the χ² pairs: 2^n·χ amplitudes of 0.13 ps each (below)
// against χ²/2 pairs of 0.3 to 1.4 ns.
#include <cuda_runtime.h>

#include <climits>

#include "device_state.hpp"
#include "warp_chform.cuh"

namespace nsg {
namespace {

using dev::FULL;

constexpr int DWARPS = 4;
// Exponents of restored terms are any 32-bit numbers: beyond ±kMaxExponent the
// integers are refused, and twice that is where they are cut off, so that no sum or
// difference of them overflows (the weights index shared memory).
constexpr int kMaxExponent = 1 << 20;

template <typename Desc>
__device__ __forceinline__ const Desc& owner_of(const Desc* descs, int num, int64_t i, int64_t Desc::*begin) {
    int lo = 0, hi = num;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (descs[mid].*begin <= i) lo = mid;
        else hi = mid;
    }
    return descs[lo];
}

// ---- terms as quadratic forms ----------------------------------------------------
// One warp per term, lane p its row p (n ≤ 32).  ⟨x|term⟩ = ω^{k0}·2^{-r/2}·
// i^{Q(x)} on the points with c_j·x = rhs_j, Q(x) = Σ L_p x_p + 2Σ_{p<q} J_pq x_p x_q
// (the form of reduce_terms_kernel).  The constraints are an echelon whose pivot
// is the lowest bit of its row.  For the amplitude kernel, which splits x into
// eight bits of the thread, five of the bit within a word and the block's, the
// term's Q over the word bits (two planes of 32) and, for every thread value, Q
// and the coupling to the word bits (one byte) are tabulated.
__global__ void __launch_bounds__(DWARPS * 32) dense_terms_kernel(const DenseDesc* __restrict__ descs, int num,
                                                                  int64_t total) {
    const int lane = threadIdx.x & 31;
    const int64_t gterm = (int64_t)blockIdx.x * DWARPS + (threadIdx.x >> 5);
    if (gterm >= total) return;
    const DenseDesc& d = owner_of(descs, num, gterm, &DenseDesc::term0);
    const TermsView& tv = d.tv;
    const int64_t term = gterm - d.term0;
    const int n = tv.n;
    const size_t idx = ((size_t)term * tv.R + lane) * tv.W;
    const uint32_t F = lane < n ? (uint32_t)tv.F[idx] : 0u, M = lane < n ? (uint32_t)tv.M[idx] : 0u;
    const uint32_t v = (uint32_t)tv.V[term * tv.W], s = (uint32_t)tv.S[term * tv.W];
    const uint32_t gl = (uint32_t)tv.GL[term * tv.W], gh = (uint32_t)tv.GH[term * tv.W];
    uint32_t J = 0;
    for (int r = 0; r < n; r++) {
        const uint32_t f = __shfl_sync(FULL, F, r), m = __shfl_sync(FULL, M, r);
        J |= (uint32_t)(__popc((r <= lane ? M : m) & (r <= lane ? f : F)) & 1) << r;
    }
    int L = (int)((gl >> lane) & 1) + 2 * (int)((gh >> lane) & 1) + 2 * (int)((J >> lane) & 1) +
            2 * __popc(F & v & s);
    L = lane < n ? L & 3 : 0;
    J = lane < n ? J & ~(1u << lane) : 0u;
    DenseTerm* o = d.terms + term;
    // constraints (xF)_c = s_c, c ∉ v
    uint32_t Fc = F, R = 0, piv = 0, cons = ~v & (n >= 32 ? ~0u : (1u << n) - 1), rs = s;
    bool rr = false, empty = false;
    while (cons) {
        const uint32_t c = cons & (~cons + 1);
        cons ^= c;
        const uint32_t l = __ballot_sync(FULL, (Fc & c) != 0);
        const bool rb = (rs & c) != 0;
        if (!l) {
            empty |= rb;
            continue;
        }
        const int p = __ffs(l) - 1;
        const uint32_t lp = l & (l - 1);
        const uint32_t Fp = __shfl_sync(FULL, Fc, p);
        if (rb) rs ^= Fp;
        if ((lp >> lane) & 1) Fc ^= Fp;
        if ((R >> p) & 1) {
            R = (R & ~(1u << p)) ^ lp;
            rr ^= rb;
        }
        if (lane == p) {
            Fc = 0;
            R = lp;
            rr = rb;
        }
        piv |= 1u << p;
    }
    const uint32_t rhs = __ballot_sync(FULL, rr);
    // tables over the thread bits 0-7 and the word bits 8-12
    uint32_t jw[13];
    int lw[13];
#pragma unroll
    for (int p = 0; p < 13; p++) {
        jw[p] = __shfl_sync(FULL, J, p);
        lw[p] = __shfl_sync(FULL, L, p);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int th = lane + 32 * i;
        uint32_t w = 0;
        int q = 0;
#pragma unroll
        for (int p = 0; p < 8; p++)
            if ((th >> p) & 1) {
                q += lw[p] + 2 * (int)((w >> p) & 1);
                w ^= jw[p];
            }
        o->tab[th] = (uint8_t)((q & 3) | (((w >> 8) & 31) << 2));
    }
    {
        uint32_t w = 0;
        int q = 0;
#pragma unroll
        for (int p = 8; p < 13; p++)
            if ((lane >> (p - 8)) & 1) {
                q += lw[p] + 2 * (int)((w >> p) & 1);
                w ^= jw[p];
            }
        const uint32_t q0 = __ballot_sync(FULL, q & 1), q1 = __ballot_sync(FULL, q & 2);
        const uint32_t l0 = __ballot_sync(FULL, L & 1), l1 = __ballot_sync(FULL, L & 2);
        o->J[lane] = J;
        o->cons[lane] = ((piv >> lane) & 1) ? R | (1u << lane) : 0u;
        if (lane == 0) {
            o->q0 = q0;
            o->q1 = q1;
            o->L0 = l0;
            o->L1 = l1;
            o->piv = piv;
            o->rhs = rhs;
            o->k0 = (tv.phase[term] + tv.coef_k[term]) & 7;
            d.kr[term] = make_int2(o->k0, empty ? INT_MIN
                                                : __popc(v) + min(max(tv.coef_r[term], -2 * kMaxExponent), 2 * kMaxExponent));
        }
    }
}

// ---- order -------------------------------------------------------------------------
// One block per state: the terms sorted by (group, weight), group = (k0 mod 2,
// (R - r) mod 2) and weight 2^e, e = (R - r)/2, largest first; and whether the
// integers fit: Σ 2^⌈(R-r)/2⌉ below 2^23, so that a coordinate fits the 24 bit
// planes of the amplitude kernel and the sums of products 64 bits per thread.
// Bound by latency: the terms of a state share a few keys, so a warp counts its
// lanes of one key with one shared atomic (an atomic per term took 18 us for 1,000
// terms, 3.4 us now).
constexpr int OTHREADS = 512;

__global__ void __launch_bounds__(OTHREADS) dense_order_kernel(const DenseDesc* __restrict__ descs) {
    __shared__ int cnt[kDenseKeys + 1];
    __shared__ int rmax;
    __shared__ unsigned bound;
    __shared__ int wide;
    const DenseDesc& d = descs[blockIdx.x];
    const int chi = (int)d.tv.chi, lane = threadIdx.x & 31;
    constexpr unsigned kTooMany = 1u << kDensePlanes;  // where the bound is cut off: 2^24, over the limit
    for (int k = threadIdx.x; k <= kDenseKeys; k += OTHREADS) cnt[k] = 0;
    if (threadIdx.x == 0) {
        rmax = INT_MIN;
        bound = 0;
        wide = 0;
    }
    __syncthreads();
    int m = INT_MIN;
    for (int i = threadIdx.x; i < chi; i += OTHREADS) m = max(m, d.kr[i].y);
    m = __reduce_max_sync(FULL, m);
    if (lane == 0) atomicMax(&rmax, m);
    __syncthreads();
    // key of a term, or -1: no amplitudes, or an exponent that is too far off
    auto key_of = [&](int i, int& w) {
        const int2 kr = i < chi ? d.kr[i] : make_int2(0, INT_MIN);
        if (kr.y == INT_MIN) return -1;
        w = rmax - kr.y;
        return w > 46 || abs(kr.y) > kMaxExponent ? -2 : ((kr.x & 1) * 2 + (w & 1)) * 32 + (31 - (w >> 1));
    };
    unsigned mine = 0;
    const int rounds = (chi + OTHREADS - 1) / OTHREADS;
    for (int r = 0; r < rounds; r++) {
        int w = 0;
        const int key = key_of(r * OTHREADS + (int)threadIdx.x, w);
        if (key == -2) wide = 1;
        if (key >= 0) mine = min(mine + (1u << ((w + 1) >> 1)), kTooMany);
        const unsigned same = __match_any_sync(FULL, key);
        if (key >= 0 && lane == __ffs(same) - 1) atomicAdd(&cnt[key], __popc(same));
    }
    mine = __reduce_add_sync(FULL, mine);
    if (lane == 0) atomicAdd(&bound, min(mine, kTooMany));
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive prefix over the keys, four per lane
        int c[kDenseKeys / 32], sum = 0;
#pragma unroll
        for (int k = 0; k < kDenseKeys / 32; k++) {
            c[k] = cnt[threadIdx.x * (kDenseKeys / 32) + k];
            sum += c[k];
        }
        int at = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, at, o);
            if (lane >= o) at += y;
        }
        if (lane == 31) {
            d.info->start[kDenseKeys] = at;
            d.info->rmax = rmax == INT_MIN ? 0 : rmax;
            d.info->ok = !wide && bound < (1u << (kDensePlanes - 1));
        }
        at -= sum;
#pragma unroll
        for (int k = 0; k < kDenseKeys / 32; k++) {
            d.info->start[threadIdx.x * (kDenseKeys / 32) + k] = at;
            cnt[threadIdx.x * (kDenseKeys / 32) + k] = at;
            at += c[k];
        }
    }
    __syncthreads();
    if (wide) return;
    for (int r = 0; r < rounds; r++) {
        int w = 0;
        const int i = r * OTHREADS + (int)threadIdx.x, key = key_of(i, w);
        const unsigned same = __match_any_sync(FULL, key);
        int at = 0;
        if (key >= 0 && lane == __ffs(same) - 1) at = atomicAdd(&cnt[key], __popc(same));
        at = __shfl_sync(FULL, at, __ffs(same) - 1);
        if (key >= 0) d.order[at + __popc(same & ((1u << lane) - 1))] = i;  // any order within a key: the sums are exact
    }
}

// ---- amplitudes ----------------------------------------------------------------------
// A thread owns 32 points x that differ in bits 8-12, one per bit of a word, and
// adds the terms' i^Q into bit-sliced counters: four (Re, Im) × (+, -) counters,
// eight terms at a time through carry-save adders (two three-input logic
// operations add two words into a counter bit).  At the end of a weight class
// the differences are added to bit-sliced signed accumulators that double from
// one class to the next, and a 32×32 bit transpose (recursive block swaps: H. S.
// Warren, Hacker's Delight, section 7-3) turns them into integers.
// About 50 integer instructions per term and 32 points, and as much again per
// weight class and block for folding and writing back.  No pipe is full: 36 % of
// the issue slots at n = 22 (24 T gates), a block waits for the loads and barriers
// of its staging, with four warps per scheduler to cover them.  0.13-0.16 ps per
// amplitude: 1.27 ms for the 8.2·10^9 of n = 23, χ = 972; 0.84 ms for n = 23, χ =
// 3,159 of a shallow circuit, where most blocks hold no point of a term (χ²/2
// pairs take 5.9 ms there; chunks of terms that end at each class took 1.08 ms).
constexpr int ATHREADS = 256;
constexpr int CHUNK = 96;  // terms staged at a time
constexpr int WBITS = 13;  // bits of x below the block's

struct AmpShared {
    uint8_t tab[CHUNK][256];
    uint4 info[CHUNK];  // q0, q1, Q(block) | w5 << 2 | w8 << 8, constraints: count | first << 8
    uint2 cons[CHUNK * WBITS];
    int term[CHUNK];    // of `order`
    uint8_t key[CHUNK], run[CHUNK];
    uint32_t walsh[32];
    int warp_count[CHUNK / 32], ncons;
};

__device__ __forceinline__ uint32_t maj3(uint32_t a, uint32_t b, uint32_t c) { return (a & b) | (c & (a | b)); }

// acc += x over NB planes from plane 0 on, both bit-sliced two's complement.
template <int NB>
__device__ __forceinline__ void add_planes(uint32_t (&acc)[kDensePlanes], const uint32_t (&x)[NB]) {
    uint32_t c = 0;
#pragma unroll
    for (int p = 0; p < kDensePlanes; p++) {
        const uint32_t b = x[p < NB ? p : NB - 1], a = acc[p];  // sign extension
        acc[p] = a ^ b ^ c;
        c = maj3(a, b, c);
    }
}

constexpr int CPLANES = 7;                              // counter planes above the carry-save levels (8, 16, ...)
constexpr int kFold = (1 << (CPLANES + 3)) - 8;         // terms after which a counter is folded

struct Counter {
    uint32_t one, two, four, hi[CPLANES];
    __device__ __forceinline__ void clear() {
        one = two = four = 0;
#pragma unroll
        for (int p = 0; p < CPLANES; p++) hi[p] = 0;
    }
};

__global__ void __launch_bounds__(ATHREADS, 2) dense_amp_kernel(const DenseDesc* __restrict__ descs, int num) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    AmpShared& sh = *(AmpShared*)smem_raw;
    const DenseDesc& d = owner_of(descs, num, (int64_t)blockIdx.x, &DenseDesc::block0);
    if (!d.info->ok) return;
    const int tid = threadIdx.x;
    const int n = d.tv.n;
    const int64_t lb = (int64_t)blockIdx.x - d.block0;
    const uint32_t tile = (uint32_t)(lb / d.splits);  // block bits of x
    const int split = (int)(lb % d.splits);
    const int total = d.info->start[kDenseKeys];
    const int t0 = (int)((int64_t)total * split / d.splits), t1 = (int)((int64_t)total * (split + 1) / d.splits);
    if (tid < 32) {  // bit j of walsh[w]: parity of w & j
        uint32_t m = 0;
        for (int j = 0; j < 32; j++) m |= (uint32_t)(__popc(tid & j) & 1) << j;
        sh.walsh[tid] = m;
    }
    Counter ct[4];  // Re+, Re-, Im+, Im-
    const uint32_t hi = n > WBITS ? tile << WBITS : 0u;
    for (int group = 0; group < 4; group++) {
        const int a = max(d.info->start[group * 32], t0), b = min(d.info->start[group * 32 + 32], t1);
        if (a >= b) continue;
        uint32_t re[kDensePlanes], im[kDensePlanes];
#pragma unroll
        for (int p = 0; p < kDensePlanes; p++) re[p] = im[p] = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) ct[q].clear();
        int counted = 0, cur = -1;  // terms counted, exponent of their weight (none yet)
        auto fold = [&]() {  // the counters' differences into the accumulators
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const Counter &u = ct[2 * h], &w = ct[2 * h + 1];
                uint32_t x[CPLANES + 4];
                uint32_t c = ~0u;  // u - w = u + ~w + 1
#pragma unroll
                for (int p = 0; p < CPLANES + 3; p++) {
                    const uint32_t ub = p == 0 ? u.one : p == 1 ? u.two : p == 2 ? u.four : u.hi[p >= 3 ? p - 3 : 0];
                    const uint32_t wb = ~(p == 0 ? w.one : p == 1 ? w.two : p == 2 ? w.four : w.hi[p >= 3 ? p - 3 : 0]);
                    x[p] = ub ^ wb ^ c;
                    c = maj3(ub, wb, c);
                }
                x[CPLANES + 3] = ~c;  // sign
                if (h == 0) add_planes<CPLANES + 4>(re, x);
                else add_planes<CPLANES + 4>(im, x);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) ct[q].clear();
            counted = 0;
        };
        auto weigh = [&](int e) {  // down to terms of weight 2^e: what was counted so far doubles for each step
            if (counted) fold();
            if (cur < 0) cur = e;
            for (; cur > e; cur--) {
#pragma unroll
                for (int p = kDensePlanes - 1; p > 0; p--) {
                    re[p] = re[p - 1];
                    im[p] = im[p - 1];
                }
                re[0] = im[0] = 0;
            }
        };
        for (int base = a; base < b; base += CHUNK) {
            const int m = min(CHUNK, b - base);
            __syncthreads();  // the last chunk is read
            if (tid == 0) sh.ncons = 0;
            __syncthreads();
            // One thread per term: the block's part of Q and of the constraints;
            // terms without a point in the block are left out.  All of a term's
            // loads are issued together (they are the latency of this part).
            bool on = false;
            uint32_t q = 0, w = 0, lowp = 0, rhs = 0, q0 = 0, q1 = 0;
            int term = 0, key = 0;
            if (tid < CHUNK) {
                if (tid < m) {
                    term = d.order[base + tid];
                    const DenseTerm& t = d.terms[term];
                    uint32_t jr[kDenseMaxQubits - WBITS];
#pragma unroll
                    for (int p = 0; p < kDenseMaxQubits - WBITS; p++) jr[p] = t.J[WBITS + p];
                    const uint32_t l0 = t.L0, l1 = t.L1, piv = t.piv;
                    rhs = t.rhs;
                    q0 = t.q0;
                    q1 = t.q1;
                    q = (uint32_t)(t.k0 >> 1);  // ω^{k0} = ω^{k0 mod 2}·i^{k0/2}
                    on = true;
                    for (uint32_t pm = piv >> WBITS; pm; pm &= pm - 1) {
                        const int p = WBITS + __ffs(pm) - 1;
                        on &= (uint32_t)(__popc(t.cons[p] & hi) & 1) == ((rhs >> p) & 1);
                    }
#pragma unroll
                    for (int p = 0; p < kDenseMaxQubits - WBITS; p++)
                        if ((hi >> (WBITS + p)) & 1) {
                            q += ((l0 >> (WBITS + p)) & 1) + 2 * ((l1 >> (WBITS + p)) & 1) + 2 * ((w >> (WBITS + p)) & 1);
                            w ^= jr[p];
                        }
                    lowp = piv & ((1u << WBITS) - 1);
                    const int2 kr = d.kr[term];
                    key = (d.info->rmax - kr.y) >> 1;
                }
                const uint32_t bal = __ballot_sync(FULL, on);
                if ((tid & 31) == 0) sh.warp_count[tid >> 5] = __popc(bal);
                q = (q & 3) | (((w >> 8) & 31) << 2) | ((w & 255) << 8);
                w = bal;
            }
            __syncthreads();
            int cnt = 0, at = 0;
#pragma unroll
            for (int k = 0; k < CHUNK / 32; k++) {
                if (k == tid >> 5) at = cnt;
                cnt += sh.warp_count[k];
            }
            if (on) {
                at += __popc(w & ((1u << (tid & 31)) - 1));
                const DenseTerm& t = d.terms[term];
                const int nc = __popc(lowp);
                int c = nc ? atomicAdd(&sh.ncons, nc) : 0;
                sh.info[at] = make_uint4(q0, q1, q, (uint32_t)nc | ((uint32_t)c << 8));
                sh.term[at] = term;
                sh.key[at] = (uint8_t)key;
                for (uint32_t pm = lowp; pm; pm &= pm - 1) {
                    const int p = __ffs(pm) - 1;
                    const uint32_t cm = t.cons[p];
                    const uint32_t rb = ((rhs >> p) & 1) ^ (__popc(cm & hi) & 1);
                    // allowed points of the word for even thread parity
                    sh.cons[c++] = make_uint2(~(sh.walsh[(cm >> 8) & 31] ^ (0u - rb)), cm & 255);
                }
            }
            __syncthreads();
            // the tables of the terms that are left, 16 bytes per thread at a time
            for (int e = tid; e < cnt * 16; e += ATHREADS)
                ((uint4*)sh.tab[e >> 4])[e & 15] = ((const uint4*)d.terms[sh.term[e >> 4]].tab)[e & 15];
            if (tid < cnt) {  // terms of the same weight from here on, eight at most
                int r = 1;
                while (r < 8 && tid + r < cnt && sh.key[tid + r] == sh.key[tid]) r++;
                sh.run[tid] = (uint8_t)r;
            }
            __syncthreads();
            int g = 0;
            while (g < cnt) {
                const int run = sh.run[g];
                if (sh.key[g] != cur) weigh(sh.key[g]);
                uint32_t in[4], c2[4], c4[4];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    uint32_t msk[4] = {0, 0, 0, 0};
                    if (u < run) {
                        const uint4 f = sh.info[g + u];
                        const uint32_t e = sh.tab[g + u][tid];
                        const uint32_t w5 = ((e ^ f.z) >> 2) & 31;
                        const uint32_t qq = e + f.z + 2 * (uint32_t)__popc((f.z >> 8) & tid);  // bits 0, 1
                        const uint32_t a0 = 0u - (qq & 1), a1 = 0u - ((qq >> 1) & 1);
                        const uint32_t m0 = f.x ^ a0;
                        const uint32_t m1 = f.y ^ a1 ^ (a0 & f.x) ^ sh.walsh[w5];
                        uint32_t sup = ~0u;
                        const uint32_t nc = f.w & 255;
                        for (uint32_t c = 0; c < nc; c++) {
                            const uint2 k = sh.cons[(f.w >> 8) + c];
                            sup &= k.x ^ (0u - (__popc(k.y & tid) & 1));
                        }
                        msk[0] = sup & ~m0 & ~m1;
                        msk[1] = sup & ~m0 & m1;
                        msk[2] = sup & m0 & ~m1;
                        msk[3] = sup & m0 & m1;
                    }
#pragma unroll
                    for (int k4 = 0; k4 < 4; k4++) {
                        Counter& k = ct[k4];
                        if ((u & 1) == 0) {
                            in[k4] = msk[k4];
                            continue;
                        }
                        const uint32_t t2 = maj3(k.one, in[k4], msk[k4]);
                        k.one ^= in[k4] ^ msk[k4];
                        if ((u & 2) == 0) {
                            c2[k4] = t2;
                            continue;
                        }
                        const uint32_t t4 = maj3(k.two, c2[k4], t2);
                        k.two ^= c2[k4] ^ t2;
                        if ((u & 4) == 0) {
                            c4[k4] = t4;
                            continue;
                        }
                        uint32_t c = maj3(k.four, c4[k4], t4);
                        k.four ^= c4[k4] ^ t4;
#pragma unroll
                        for (int p = 0; p < CPLANES; p++) {
                            const uint32_t h = k.hi[p];
                            k.hi[p] = h ^ c;
                            c &= h;
                        }
                    }
                }
                counted += 8;
                if (counted > kFold - 8) fold();
                g += run;
            }
        }
        weigh(0);
        // Integers: plane p of lane-local word j -> bit p of integer j.
        const bool odd = group & 1, up = group >= 2;
        // ω^κ·√2^odd·(S0 + i S1): (κ, odd) = (0,0): c0, c2; (1,0): c1, c3; (0,1): c1 += S0+S1, c3 += S1-S0;
        // (1,1): c0 += S0-S1, c2 += S0+S1.  ψ is stored as (c0, c2, c1, c3).
        const int half = (odd ? !up : up) ? 1 : 0;
        uint32_t A[32], B[32];
#pragma unroll
        for (int p = 0; p < 32; p++) {
            A[p] = re[p < kDensePlanes ? p : kDensePlanes - 1];
            B[p] = im[p < kDensePlanes ? p : kDensePlanes - 1];
        }
#pragma unroll
        for (int t = 0; t < 5; t++) {
            const int j = 16 >> t;
            const uint32_t mk = t == 0 ? 0x0000ffffu : t == 1 ? 0x00ff00ffu : t == 2 ? 0x0f0f0f0fu : t == 3 ? 0x33333333u : 0x55555555u;
#pragma unroll
            for (int k = 0; k < 32; k++) {
                if (k & j) continue;
                uint32_t x = ((A[k] >> j) ^ A[k + j]) & mk;
                A[k] ^= x << j;
                A[k + j] ^= x;
                x = ((B[k] >> j) ^ B[k + j]) & mk;
                B[k] ^= x << j;
                B[k + j] ^= x;
            }
        }
        const uint32_t npts = n >= WBITS ? 1u << WBITS : 1u << n;
#pragma unroll
        for (int j = 0; j < 32; j++) {
            const uint32_t lo = (uint32_t)tid | ((uint32_t)j << 8);
            if (lo >= npts) continue;
            const int S0 = (int)A[j], S1 = (int)B[j];
            int2 add;
            if (!odd) add = make_int2(S0, S1);
            else if (!up) add = make_int2(S0 + S1, S1 - S0);
            else add = make_int2(S0 - S1, S0 + S1);
            int* at = (int*)(d.psi + (((size_t)tile << WBITS) | lo)) + 2 * half;
            if (d.splits > 1) {
                if (add.x) atomicAdd(at, add.x);
                if (add.y) atomicAdd(at + 1, add.y);
            } else {
                int2 old = *(int2*)at;
                *(int2*)at = make_int2(old.x + add.x, old.y + add.y);
            }
        }
    }
}

// ---- ⟨P⟩ ---------------------------------------------------------------------------------
// One block per (observable, slice of the points): X and Y of 2^{-R}(X + Y/√2) =
// i^{ny}·Σ_x (-1)^{pz·x}·conj(ψ(x ⊕ px))·ψ(x).  The terms of x and x ⊕ px are
// complex conjugates of one another, so half of the points are summed, twice.
// Each point's sums fit 50 bits, a thread's (at most 2^9 points) 62; the block's
// go to the result as two 64-bit sums of 32-bit halves.  Bound by the two reads
// of ψ (16 bytes a point each; from L2 while ψ is below its 126 MB).
constexpr int VTHREADS = 256;

__device__ __forceinline__ void pair_product(const int4& dv, const int4& fv, long long& X, long long& Y) {
    // stored as (c0, c2, c1, c3)
    const long long f0 = fv.x, f2 = fv.y, f1 = fv.z, f3 = fv.w;
    X += (long long)dv.x * f0 + (long long)dv.z * f1 + (long long)dv.y * f2 + (long long)dv.w * f3;
    Y += (long long)dv.x * (f1 - f3) + (long long)dv.z * (f0 + f2) + (long long)dv.y * (f1 + f3) +
         (long long)dv.w * (f2 - f0);
}

__device__ __forceinline__ int4 times_i(int4 c, int k) {  // i^k·(c0, c2, c1, c3): (c0, c1, c2, c3) -> (-c2, -c3, c0, c1)
    for (; k > 0; k--) c = make_int4(-c.y, c.x, -c.w, c.z);
    return c;
}

__device__ __forceinline__ void block_sum_to(long long X, long long Y, unsigned long long* out) {
    // 32-bit halves: their sums over the block and over all blocks fit 64 bits
    long long v[4] = {X & 0xffffffffll, X >> 32, Y & 0xffffffffll, Y >> 32};
    __shared__ long long sh[4][VTHREADS / 32];
#pragma unroll
    for (int t = 0; t < 4; t++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[t] += __shfl_down_sync(FULL, v[t], o);
        if ((threadIdx.x & 31) == 0) sh[t][threadIdx.x >> 5] = v[t];
    }
    __syncthreads();
    if (threadIdx.x < 4) {
        long long a = 0;
#pragma unroll
        for (int w = 0; w < VTHREADS / 32; w++) a += sh[threadIdx.x][w];
        if (a) atomicAdd(out + threadIdx.x, (unsigned long long)a);
    }
}

__global__ void __launch_bounds__(VTHREADS) dense_values_kernel(const DenseDesc* __restrict__ descs, int num) {
    const DenseDesc& d = owner_of(descs, num, (int64_t)blockIdx.x, &DenseDesc::vblock0);
    if (!d.info->ok) return;
    const int64_t lb = (int64_t)blockIdx.x - d.vblock0;
    const int o = (int)(lb / d.vslices);
    const uint32_t slice = (uint32_t)(lb % d.vslices);
    const DevPauli P = d.paulis[o];
    const uint32_t px = (uint32_t)P.px, pz = (uint32_t)P.pz;
    const int n = d.tv.n;
    const uint32_t half = px ? 1u << (31 - __clz(px)) : 0u;  // points with this bit clear are summed
    const uint64_t pts = (uint64_t)1 << (px ? n - 1 : n);
    const uint64_t per = (pts + d.vslices - 1) / d.vslices;
    const uint64_t p0 = slice * per, p1 = min(p0 + per, pts);
    long long X = 0, Y = 0;
    for (uint64_t i = p0 + threadIdx.x; i < p1; i += VTHREADS) {
        const uint32_t x = px ? (uint32_t)((i & (half - 1)) | ((i & ~(uint64_t)(half - 1)) << 1)) : (uint32_t)i;
        const int4 f = d.psi[x];
        const int4 g = px ? d.psi[x ^ px] : f;
        long long a = 0, b = 0;
        pair_product(g, times_i(f, P.ny), a, b);
        if (__popc(x & pz) & 1) {
            X -= a;
            Y -= b;
        } else {
            X += a;
            Y += b;
        }
    }
    if (px) {
        X *= 2;
        Y *= 2;
    }
    block_sum_to(X, Y, d.sums + 4 * (size_t)o);
}

// ---- weights of outcomes -----------------------------------------------------------------
// |ψ(x)|² summed over the points with the same outcome y (bit i of y the bit
// bits[i] of x): integers X, Y of 2^{-R}(X + Y/√2) per outcome.
__global__ void __launch_bounds__(VTHREADS) dense_weights_kernel(const int4* __restrict__ psi, const DenseInfo* info, int n,
                                                                 DenseBits bits, unsigned long long* __restrict__ out) {
    if (!info->ok) return;
    const uint64_t pts = (uint64_t)1 << n;
    const bool whole = bits.count == n;  // one point per outcome
    for (uint64_t x = (uint64_t)blockIdx.x * VTHREADS + threadIdx.x; x < pts; x += (uint64_t)gridDim.x * VTHREADS) {
        const int4 f = psi[x];
        long long X = 0, Y = 0;
        pair_product(f, f, X, Y);
        uint32_t y = 0;
        for (int i = 0; i < bits.count; i++) y |= (uint32_t)((x >> bits.bit[i]) & 1) << i;
        if (whole) {
            out[2 * (size_t)y] = (unsigned long long)X;
            out[2 * (size_t)y + 1] = (unsigned long long)Y;
        } else {
            if (X) atomicAdd(out + 2 * (size_t)y, (unsigned long long)X);
            if (Y) atomicAdd(out + 2 * (size_t)y + 1, (unsigned long long)Y);
        }
    }
}

// ---- state vector --------------------------------------------------------------------------
__global__ void __launch_bounds__(VTHREADS) dense_vector_kernel(const int4* __restrict__ psi, const DenseInfo* info, int n,
                                                                double gf_re, double gf_im, double2* __restrict__ out) {
    if (!info->ok) return;
    const dev::AmplitudeScale amplitude(info->rmax, gf_re, gf_im);
    const uint64_t pts = (uint64_t)1 << n;
    for (uint64_t x = (uint64_t)blockIdx.x * VTHREADS + threadIdx.x; x < pts; x += (uint64_t)gridDim.x * VTHREADS) {
        const int4 c = psi[x];  // (c0, c2, c1, c3)
        out[x] = amplitude(c.x, c.z, c.y, c.w);
    }
}

}  // namespace

cudaError_t launch_dense_amplitudes(const DenseDesc* descs, int num, int64_t terms, int64_t blocks, cudaStream_t st) {
    if (num == 0) return cudaSuccess;
    dense_terms_kernel<<<(unsigned)((terms + DWARPS - 1) / DWARPS), DWARPS * 32, 0, st>>>(descs, num, terms);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    dense_order_kernel<<<num, OTHREADS, 0, st>>>(descs);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    dense_amp_kernel<<<(unsigned)blocks, ATHREADS, sizeof(AmpShared), st>>>(descs, num);
    return cudaGetLastError();
}

cudaError_t launch_dense_values(const DenseDesc* descs, int num, int64_t blocks, cudaStream_t st) {
    if (num == 0 || blocks == 0) return cudaSuccess;
    dense_values_kernel<<<(unsigned)blocks, VTHREADS, 0, st>>>(descs, num);
    return cudaGetLastError();
}

cudaError_t launch_dense_weights(const int4* psi, const DenseInfo* info, int n, const DenseBits& bits,
                                 unsigned long long* out, cudaStream_t st) {
    const uint64_t want = (((uint64_t)1 << n) + VTHREADS - 1) / VTHREADS;
    const unsigned blocks = (unsigned)(want < 65536 ? want : 65536);
    dense_weights_kernel<<<blocks, VTHREADS, 0, st>>>(psi, info, n, bits, out);
    return cudaGetLastError();
}

cudaError_t launch_dense_vector(const int4* psi, const DenseInfo* info, int n, double gf_re, double gf_im, double* out,
                                cudaStream_t st) {
    const uint64_t want = (((uint64_t)1 << n) + VTHREADS - 1) / VTHREADS;
    const unsigned blocks = (unsigned)(want < 65536 ? want : 65536);
    dense_vector_kernel<<<blocks, VTHREADS, 0, st>>>(psi, info, n, gf_re, gf_im, (double2*)out);
    return cudaGetLastError();
}

}  // namespace nsg
