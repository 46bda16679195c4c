// warp_chform.cuh — one CH-form term held by one warp.
//
// Layout: row r of G, F, M lives in lane (r & 31), slot (r >> 5); a row is W
// words of `Word` (u32 or u64), bit c of the row is column c.  γ_r (an
// exponent of i, mod 4) is kept by the row's lane as 2 bits per slot.  The
// vectors v, s and the Z8 phase are warp-uniform.  Row operations move a row
// between lanes with one shuffle per word; column operations (the right
// multiplications inside _resolve_superposition) are lane-local, so an H gate
// costs O(W) instructions per lane instead of the reference's O(w²) byte loop.
//
// Every rule reproduces the reference's update exactly (same pivots, same
// order), so the tableau bits match crates/stabilizer-ch-form-rust/src/form/.
// Where the reference applies a sequence of column operations that commute
// (resolve_superposition.rs:155-176, discard.rs:152-158, :174-178) they are
// applied as one masked update; each such batch is annotated with why the
// result is identical.
//
// Invariant violations that the reference turns into panics
// (resolve_superposition.rs:121, discard.rs:140,155) set `err` instead.
#pragma once

#include <cstdint>

namespace nsg {
namespace dev {

constexpr unsigned FULL = 0xffffffffu;

template <typename Word>
__device__ __forceinline__ Word shfl(Word x, int src) {
    return __shfl_sync(FULL, x, src);
}

template <typename Word>
__device__ __forceinline__ int popc(Word x);
template <>
__device__ __forceinline__ int popc<uint32_t>(uint32_t x) { return __popc(x); }
template <>
__device__ __forceinline__ int popc<uint64_t>(uint64_t x) { return __popcll(x); }

template <typename Word>
__device__ __forceinline__ int ffs0(Word x);  // index of lowest set bit, -1 if none
template <>
__device__ __forceinline__ int ffs0<uint32_t>(uint32_t x) { return __ffs(x) - 1; }
template <>
__device__ __forceinline__ int ffs0<uint64_t>(uint64_t x) { return __ffsll((long long)x) - 1; }

__device__ __forceinline__ int parity_of(uint32_t x) { return __popc(x) & 1; }
__device__ __forceinline__ int parity_of(uint64_t x) { return __popc((uint32_t)x ^ (uint32_t)(x >> 32)) & 1; }

// ---- W-word bit vectors (uniform or per lane) -----------------------------
template <typename Word, int W>
struct BV {
    static constexpr int B = 8 * sizeof(Word);
    Word w[W];

    __device__ __forceinline__ static BV zero() {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) r.w[k] = 0;
        return r;
    }
    // Word selection by a run-time bit index is written with masks over every
    // word (never a guarded or indexed access), so the vector stays in registers.
    __device__ __forceinline__ bool bit(int q) const {
        Word x = 0;
#pragma unroll
        for (int k = 0; k < W; k++) x |= w[k] & ((q / B) == k ? ~(Word)0 : (Word)0);
        return (x >> (q & (B - 1))) & 1;
    }
    __device__ __forceinline__ void flip(int q) {
        const Word m = (Word)1 << (q & (B - 1));
#pragma unroll
        for (int k = 0; k < W; k++) w[k] ^= ((q / B) == k) ? m : (Word)0;
    }
    __device__ __forceinline__ void set(int q, bool b) {
#pragma unroll
        for (int k = 0; k < W; k++) {
            const Word m = ((q / B) == k) ? ((Word)1 << (q & (B - 1))) : (Word)0;
            w[k] = b ? (w[k] | m) : (w[k] & ~m);
        }
    }
    __device__ __forceinline__ bool any() const {
        Word a = 0;
#pragma unroll
        for (int k = 0; k < W; k++) a |= w[k];
        return a != 0;
    }
    __device__ __forceinline__ Word folded() const {
        Word x = 0;
#pragma unroll
        for (int k = 0; k < W; k++) x ^= w[k];
        return x;
    }
    // One count: they run at a quarter of the rate of an XOR.
    __device__ __forceinline__ int parity() const { return parity_of(folded()); }
    // this ^= m where c is not zero.
    __device__ __forceinline__ void xor_if(uint32_t c, const BV& m) {
        if constexpr (sizeof(Word) == 4 && W == 2) {
            asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p xor.b32 %0, %0, %3;\n\t@p xor.b32 %1, %1, %4;\n\t}"
                : "+r"(w[0]), "+r"(w[1])
                : "r"(c), "r"(m.w[0]), "r"(m.w[1]));
        } else if constexpr (sizeof(Word) == 4 && W == 3) {
            asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p xor.b32 %0, %0, %4;\n\t@p xor.b32 %1, %1, %5;\n\t"
                "@p xor.b32 %2, %2, %6;\n\t}"
                : "+r"(w[0]), "+r"(w[1]), "+r"(w[2])
                : "r"(c), "r"(m.w[0]), "r"(m.w[1]), "r"(m.w[2]));
        } else if constexpr (sizeof(Word) == 4) {
#pragma unroll
            for (int k = 0; k < W; k++)
                asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p xor.b32 %0, %0, %2;\n\t}"
                    : "+r"(w[k])
                    : "r"(c), "r"(m.w[k]));
        } else {
            *this ^= select(c != 0, m);
        }
    }
    // Not zero where this and m share a bit.
    __device__ __forceinline__ uint32_t meets(const BV& m) const {
        Word x = 0;
#pragma unroll
        for (int k = 0; k < W; k++) x |= w[k] & m.w[k];
        return sizeof(Word) == 4 ? (uint32_t)x : (uint32_t)(x != 0);
    }
    // The lowest set bit alone (zero if there is none).
    __device__ __forceinline__ BV lowest() const {
        BV r;
        bool found = false;
#pragma unroll
        for (int k = 0; k < W; k++) {
            r.w[k] = found ? (Word)0 : (w[k] & (~w[k] + 1));
            found = found || w[k] != 0;
        }
        return r;
    }
    __device__ __forceinline__ int first() const {  // lowest set bit or -1
        int r = -1;
#pragma unroll
        for (int k = W - 1; k >= 0; k--) {
            int f = ffs0<Word>(w[k]);
            if (f >= 0) r = f + k * B;
        }
        return r;
    }
    __device__ __forceinline__ bool operator==(const BV& o) const {
        bool e = true;
#pragma unroll
        for (int k = 0; k < W; k++) e &= (w[k] == o.w[k]);
        return e;
    }
    __device__ __forceinline__ BV operator^(const BV& o) const {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) r.w[k] = w[k] ^ o.w[k];
        return r;
    }
    __device__ __forceinline__ BV operator&(const BV& o) const {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) r.w[k] = w[k] & o.w[k];
        return r;
    }
    __device__ __forceinline__ BV operator|(const BV& o) const {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) r.w[k] = w[k] | o.w[k];
        return r;
    }
    __device__ __forceinline__ BV operator~() const {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) r.w[k] = ~w[k];
        return r;
    }
    __device__ __forceinline__ BV& operator^=(const BV& o) {
#pragma unroll
        for (int k = 0; k < W; k++) w[k] ^= o.w[k];
        return *this;
    }
    // r = cond ? mask : 0
    __device__ __forceinline__ static BV select(bool cond, const BV& m) {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) r.w[k] = cond ? m.w[k] : (Word)0;
        return r;
    }
    // Mask of the first n bits.
    __device__ __forceinline__ static BV low(int n) {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) {
            int lo = k * B;
            if (n >= lo + B) r.w[k] = ~(Word)0;
            else if (n <= lo) r.w[k] = 0;
            else r.w[k] = ((Word)1 << (n - lo)) - 1;
        }
        return r;
    }
    __device__ __forceinline__ BV shfl_from(int src) const {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) r.w[k] = shfl<Word>(w[k], src);
        return r;
    }
    // Remove bit q: bits above q move down by one.
    __device__ __forceinline__ BV drop_bit(int q) const {
        BV r;
#pragma unroll
        for (int k = 0; k < W; k++) {
            Word x = w[k];
            Word carry_in = (k + 1 < W) ? (w[(k + 1 < W) ? k + 1 : k] & 1) : 0;
            int lo = k * B;
            Word res;
            if (q >= lo + B) {
                res = x;  // q above this word: unchanged
            } else if (q < lo) {
                res = (x >> 1);  // whole word shifts down
            } else {
                int b = q - lo;
                Word below = (b == 0) ? (Word)0 : (x & (((Word)1 << b) - 1));
                Word above = (b == B - 1) ? (Word)0 : ((x >> (b + 1)) << b);
                res = below | above;
            }
            if (q < lo + B) res |= carry_in << (B - 1);
            r.w[k] = res;
        }
        return r;
    }
};

// g·2^{-R/2}·(c0 + c1 ω + c2 ω² + c3 ω³), ω = e^{iπ/4}, of exact integers: what both
// state vector kernels end with.
struct AmplitudeScale {
    double re, im;  // g·2^{-R/2}
    __device__ __forceinline__ AmplitudeScale(int R, double gf_re, double gf_im) {
        // an exact power of two, times 1/√2 for odd R
        const double p = ldexp((R & 1) ? 0.70710678118654752440 : 1.0, -((R - (R & 1)) / 2));
        re = gf_re * p;
        im = gf_im * p;
    }
    template <typename Int>
    __device__ __forceinline__ double2 operator()(Int c0, Int c1, Int c2, Int c3) const {
        const double r2 = 0.70710678118654752440;
        const double a = (double)c0 + (double)(c1 - c3) * r2, b = (double)c2 + (double)(c1 + c3) * r2;
        return make_double2(a * re - b * im, a * im + b * re);
    }
};

// A row slot known when the code is compiled.
template <int K>
struct Slot {
    __device__ constexpr operator int() const { return K; }
};

// ---- the warp-held term ----------------------------------------------------
template <typename Word, int W, int RPL>
struct WarpCH {
    using V = BV<Word, W>;
    static constexpr int B = 8 * sizeof(Word);
    static constexpr int MAXW = (32 * RPL < W * B) ? 32 * RPL : W * B;

    V G[RPL], F[RPL], M[RPL];  // this lane's rows
    uint32_t gam;              // 2 bits per slot
    V v, s;                    // uniform
    int phase;                 // uniform Z8
    int n;                     // uniform width
    int lane;
    int err;                   // uniform: 0 ok, else invariant id

    // ---- per-lane row access (slot index must be warp-uniform)
    __device__ __forceinline__ int gam_of(int sl) const { return (gam >> (2 * sl)) & 3; }
    __device__ __forceinline__ void gam_set(int sl, int g) {
        gam = (gam & ~(3u << (2 * sl))) | ((uint32_t)(g & 3) << (2 * sl));
    }
    __device__ __forceinline__ V pick(const V (&X)[RPL], int sl) const {
        V r = V::zero();
#pragma unroll
        for (int k = 0; k < RPL; k++) r = r | V::select(sl == k, X[k]);
        return r;
    }
    __device__ __forceinline__ V row(const V (&X)[RPL], int q) const {
        return pick(X, q >> 5).shfl_from(q & 31);
    }
    __device__ __forceinline__ bool owns(int q) const { return lane == (q & 31); }
    // f(slot) with the slot of row q known where it is used: one branch of the warp
    // instead of a selection for every word of every slot (n = 60, 36 T gates 11.2 ->
    // 7.4 ms).  The updates in it are predicated XORs (xor_if); a guarded assignment
    // would be merged over the slots into an indexed one, which moves the term to
    // local memory.
    template <typename Fn>
    __device__ __forceinline__ void at_slot(int q, Fn&& f) {
        const int sl = q >> 5;
        if (RPL == 1 || sl == 0) f(Slot<0>());
        else if (RPL == 2 || sl == 1) f(Slot<(RPL > 1 ? 1 : 0)>());
        else if (RPL == 3 || sl == 2) f(Slot<(RPL > 2 ? 2 : 0)>());
        else f(Slot<(RPL > 3 ? 3 : 0)>());
    }
    __device__ __forceinline__ bool on_row(int q, int k) const { return owns(q) && (q >> 5) == k; }

    __device__ __forceinline__ void init_zero(int width) {  // StabilizerCHForm::new
        n = width;
        err = 0;
        phase = 0;
        gam = 0;
        v = V::zero();
        s = V::zero();
#pragma unroll
        for (int k = 0; k < RPL; k++) {
            int r = k * 32 + lane;
            G[k] = V::zero();
            F[k] = V::zero();
            M[k] = V::zero();
            if (r < width) {
                G[k].set(r, true);
                F[k].set(r, true);
            }
        }
    }

    // ---- left multiplications (form/left_multiplication/*.rs) --------------
    __device__ __forceinline__ void left_cx(int c, int t) {  // cx.rs:13-51
        V Gc = V::zero(), Ft, Mt;
        int gt = 0;
        at_slot(c, [&](auto k) { Gc = G[k].shfl_from(c & 31); });
        at_slot(t, [&](auto k) {
            Ft = F[k].shfl_from(t & 31);
            Mt = M[k].shfl_from(t & 31);
            gt = gam_of(k);
            G[k].xor_if(owns(t), Gc);
        });
        gt = shfl<uint32_t>((uint32_t)gt, t & 31);
        at_slot(c, [&](auto k) {
            const uint32_t on = owns(c);
            const int sum = (int)(gam >> (2 * k)) + gt + 2 * (M[k] & Ft).parity();
            F[k].xor_if(on, Ft);
            M[k].xor_if(on, Mt);
            if (on) gam_set(k, sum);
        });
    }
    __device__ __forceinline__ void left_cz(int a, int b) {  // cz.rs:12-35
        V Ga, Gb;
        at_slot(a, [&](auto k) { Ga = G[k].shfl_from(a & 31); });
        at_slot(b, [&](auto k) {
            Gb = G[k].shfl_from(b & 31);
            M[k].xor_if(owns(b), Ga);
        });
        at_slot(a, [&](auto k) { M[k].xor_if(owns(a), Gb); });
    }
    __device__ __forceinline__ void left_s_like(int q, int dg) {  // s.rs:13-33 (dg = 3 S, 1 Sdg)
        at_slot(q, [&](auto k) { M[k].xor_if(owns(q), G[k]); });
        const uint32_t z = owns(q) ? 1u << (2 * (q >> 5)) : 0u;
        gam ^= z | (((dg == 3 ? ~gam : gam) & z) << 1);
    }
    __device__ __forceinline__ void left_s(int q) { left_s_like(q, 3); }
    __device__ __forceinline__ void left_sdg(int q) { left_s_like(q, 1); }
    __device__ __forceinline__ void left_z(int q) {  // z.rs:7-14
        gam ^= owns(q) ? 2u << (2 * (q >> 5)) : 0u;
    }
    __device__ __forceinline__ int beta_of(const V& Fq, const V& Mq) const {  // x.rs:20-29
        V b = (Mq & ~v & s) ^ (Fq & v & (Mq ^ s));
        return b.parity();
    }
    __device__ __forceinline__ void left_x(int q) {  // x.rs:12-48
        V Fq, Mq;
        int gq = 0;
        at_slot(q, [&](auto k) {
            Fq = F[k].shfl_from(q & 31);
            Mq = M[k].shfl_from(q & 31);
            gq = shfl<uint32_t>((uint32_t)gam_of(k), q & 31);
        });
        if (beta_of(Fq, Mq)) phase = (phase + 4) & 7;
        s ^= (Fq & ~v) ^ (Mq & v);
        phase = (phase + 2 * gq) & 7;
    }
    __device__ __forceinline__ void left_y(int q) {  // y.rs:4-11
        left_z(q);
        left_x(q);
        phase = (phase + 2) & 7;
    }

    // ---- right multiplications, lane-local (form/right_multiplication/*.rs)
    // right_cx(c, t): G[:,c] ^= G[:,t]; F[:,t] ^= F[:,c]; M[:,c] ^= M[:,t]
    __device__ __forceinline__ void right_cx(int c, int t) {
#pragma unroll
        for (int k = 0; k < RPL; k++) {
            if (G[k].bit(t)) G[k].flip(c);
            if (F[k].bit(c)) F[k].flip(t);
            if (M[k].bit(t)) M[k].flip(c);
        }
    }
    // right_s (s.rs:8-24) on the column of mask P: M[:,q] ^= F[:,q]; γ_p -= 1 where F[p,q].
    __device__ __forceinline__ void right_s(const V& P) {
        uint32_t z = 0;
#pragma unroll
        for (int k = 0; k < RPL; k++) {
            const uint32_t f = F[k].meets(P);
            M[k].xor_if(f, P);
            z |= f ? 1u << (2 * k) : 0u;
        }
        gam ^= z | ((~gam & z) << 1);
    }

    // _resolve_superposition (resolve_superposition.rs:6-176); delta is Z8.
    __device__ __forceinline__ void resolve(const V& t, const V& u, int delta) {
        if (t == u) {  // handle_same_vecs_case :115-133
            if (delta == 4) {
                err = 1;
                return;
            }
            s = t;
            if (delta == 2) phase = (phase + 1) & 7;
            if (delta == 6) phase = (phase + 7) & 7;
            return;
        }
        // The pivot is held as a mask P of one bit, so that neither its index nor a
        // word selected by it is needed.
        const V diff = t ^ u, d0 = diff & ~v, d1 = diff & v;
        V P;
        uint32_t gam2 = 0;  // γ += 2, by slot
        if (!d0.any()) {
            // pivot = D1[0]; right_cx(i, pivot) for i in D1[1:].  Each step
            // changes only column i of G/M (from column pivot, never changed)
            // and column pivot of F (from column i, never changed), so the
            // sequence equals one masked update.
            P = d1.lowest();
            const V rest = d1 ^ P;
#pragma unroll
            for (int k = 0; k < RPL; k++) {
                G[k].xor_if(G[k].meets(P), rest);
                F[k].xor_if((F[k] & rest).parity(), P);
                M[k].xor_if(M[k].meets(P), rest);
            }
        } else {
            // pivot = D0[0]; right_cx(pivot, i) for i in D0[1:]: column pivot
            // of G/M accumulates columns i (unchanged), columns i of F take
            // column pivot (unchanged).  Then right_cz(pivot, i) for i in D1:
            // F is not modified by CZ, columns i ∉ {pivot} ∪ D0.
            P = d0.lowest();
            const V rest = d0 ^ P;
#pragma unroll
            for (int k = 0; k < RPL; k++) {
                const uint32_t fp = F[k].meets(P);
                const Word d1f = (F[k] & d1).folded();  // right_cz(pivot, i), i ∈ D1 (cz.rs:8-35)
                G[k].xor_if((G[k] & rest).parity(), P);
                M[k].xor_if(parity_of((M[k] & rest).folded() ^ d1f), P);
                M[k].xor_if(fp, d1);
                F[k].xor_if(fp, rest);
                if (fp && parity_of(d1f)) gam2 |= 2u << (2 * k);
            }
        }
        gam ^= gam2;
        const bool vp = (v & P).any(), odd = (delta & 2) != 0, hi = (delta & 4) != 0;
        const bool tp = (t & P).any();
        // δ = 2, 6: right_s, v = 1 at the pivot, s from t, v and δ; δ = 0, 4: v flipped
        const bool sp = odd ? (hi != (vp != tp)) : hi;
        int dph = 0;
        if (odd) dph = vp ? (hi ? 7 : 1) : (tp ? (hi ? 6 : 2) : 0);
        else if (tp && hi) dph = 4;
        s = ((tp ? u : t) & ~P) | V::select(sp, P);
        v = (v & ~P) | V::select(odd || !vp, P);
        phase = (phase + dph) & 7;
        if (odd) right_s(P);
    }

    __device__ __forceinline__ void left_h(int q) {  // h.rs:13-65
        V Gq, Fq, Mq;
        int gq = 0;
        at_slot(q, [&](auto k) {
            Gq = G[k].shfl_from(q & 31);
            Fq = F[k].shfl_from(q & 31);
            Mq = M[k].shfl_from(q & 31);
            gq = shfl<uint32_t>((uint32_t)gam_of(k), q & 31);
        });
        V t = s ^ (Gq & v);
        V u = s ^ (Fq & ~v) ^ (Mq & v);
        int alpha = (Gq & ~v & s).parity();
        int beta = beta_of(Fq, Mq);
        int delta = (2 * gq + ((alpha ^ beta) ? 4 : 0)) & 7;
        if (alpha) phase = (phase + 4) & 7;
        resolve(t, u, delta);
    }

    // project (project.rs:33-76): returns 1 deterministic, 0 random, -1 impossible.
    __device__ __forceinline__ int project(int q, bool outcome) {
        V Gq;
        at_slot(q, [&](auto k) { Gq = G[k].shfl_from(q & 31); });
        V gv = Gq & v;
        if (!gv.any()) {
            int val = (Gq & s).parity();
            return (val == (int)outcome) ? 1 : -1;
        }
        V t = gv ^ s;
        int alpha = (Gq & ~v & s).parity();
        int delta = (alpha ^ (int)outcome) ? 4 : 0;
        V scopy = s;
        resolve(scopy, t, delta);
        return 0;
    }

    // discard (discard.rs:21-181): q must already be projected onto |0⟩.
    __device__ void discard(int q) {
        V valid = V::low(n);
        if (v.bit(q) || s.bit(q)) {  // set_s_v_to_false :98-132
            V cleanm = ~v & ~s & valid;
            cleanm.set(q, false);
            int clean = cleanm.first();
            if (clean < 0) {
                V cand = ~v & s & valid;
                int f = cand.first();
                if (f >= 0) {
                    cand.flip(f);
                    int sc = cand.first();
                    if (sc >= 0) {
                        right_cx(f, sc);
                        s.set(sc, false);
                        clean = sc;
                    }
                }
            }
            if (clean < 0) {
                err = 2;  // CannotDiscardQubit
                return;
            }
            if (clean != q) {
                right_cx(clean, q);
                right_cx(q, clean);
                right_cx(clean, q);
                bool vq = v.bit(q), vc = v.bit(clean), sq = s.bit(q), sc2 = s.bit(clean);
                v.set(q, vc);
                v.set(clean, vq);
                s.set(q, sc2);
                s.set(clean, sq);
            }
        }
        // transform_g :135-161
        {
            V Gq = row(G, q);
            if (!Gq.bit(q)) {
                V m = Gq & valid;
                m.set(q, false);
                int pivot = m.first();
                if (pivot < 0) {
                    err = 3;
                    return;
                }
                right_cx(q, pivot);
            }
            // left_cx(q, i) for i ≠ q with G[i][q]: each step changes row i of G (by
            // row q, which stays) and row q of F, M, γ, which is removed below.
            Gq = row(G, q);
#pragma unroll
            for (int k = 0; k < RPL; k++) G[k] ^= V::select(G[k].bit(q) && !on_row(q, k), Gq);
            // right_cx(i, q) for i ≠ q with G[q][i]: column i of G/M takes column
            // q (unchanged), column q of F accumulates columns i (unchanged).  Of G
            // only row q changes now, of F only column q: both are removed.
            V mask = Gq & valid;
            mask.set(q, false);
            if ((mask & v).any()) {
                err = 4;
                return;
            }
#pragma unroll
            for (int k = 0; k < RPL; k++) M[k] ^= V::select(M[k].bit(q), mask);
        }
        // transform_m :164-181 leaves every other row and column as it is: now
        // G[i][q] = G[q][i] = 0 for i ≠ q, so F = G^{-T} has F[i][q] = 0 too; the
        // left_cx(q, i) change column q of G and row q of the rest, the left_sdg(q)
        // row q, and the right_cz(q, i) only column q of M where F[·][q] = 0.
        remove_qubit(q);
    }

    // Removes row and column q (n -> n-1).
    __device__ __forceinline__ void remove_qubit(int q) {
        if (q == n - 1) {  // the last one, as in a compile: nothing moves
            const V keep = V::low(q);
#pragma unroll
            for (int k = 0; k < RPL; k++) {
                const bool row = 32 * k + lane < q;
                G[k] = V::select(row, G[k] & keep);
                F[k] = V::select(row, F[k] & keep);
                M[k] = V::select(row, M[k] & keep);
                if (!row) gam_set(k, 0);
            }
            v = v & keep;
            s = s & keep;
            n--;
            return;
        }
#pragma unroll
        for (int k = 0; k < RPL; k++) {
            G[k] = G[k].drop_bit(q);
            F[k] = F[k].drop_bit(q);
            M[k] = M[k].drop_bit(q);
        }
        v = v.drop_bit(q);
        s = s.drop_bit(q);
        // rows r >= q take row r+1
        V nG[RPL], nF[RPL], nM[RPL];
        uint32_t ngam = gam;
#pragma unroll
        for (int k = 0; k < RPL; k++) {
            int src = (lane + 1) & 31;
            int ks = (lane == 31) ? k + 1 : k;  // slot of row r+1
            V g1 = G[k].shfl_from(src), f1 = F[k].shfl_from(src), m1 = M[k].shfl_from(src);
            uint32_t gm1 = shfl<uint32_t>((uint32_t)gam_of(k), src);
            V g2 = V::zero(), f2 = V::zero(), m2 = V::zero();
            uint32_t gm2 = 0;
            if (k + 1 < RPL) {
                g2 = G[(k + 1 < RPL) ? k + 1 : k].shfl_from(0);
                f2 = F[(k + 1 < RPL) ? k + 1 : k].shfl_from(0);
                m2 = M[(k + 1 < RPL) ? k + 1 : k].shfl_from(0);
                gm2 = shfl<uint32_t>((uint32_t)gam_of((k + 1 < RPL) ? k + 1 : k), 0);
            }
            int r = k * 32 + lane;
            bool moved = r >= q;
            bool from_next_slot = (ks != k);
            V gn = from_next_slot ? g2 : g1, fn = from_next_slot ? f2 : f1, mn = from_next_slot ? m2 : m1;
            uint32_t gmn = from_next_slot ? gm2 : gm1;
            if (r >= n - 1) {
                gn = V::zero();
                fn = V::zero();
                mn = V::zero();
                gmn = 0;
            }
            nG[k] = moved ? gn : G[k];
            nF[k] = moved ? fn : F[k];
            nM[k] = moved ? mn : M[k];
            if (moved) ngam = (ngam & ~(3u << (2 * k))) | ((gmn & 3) << (2 * k));
        }
#pragma unroll
        for (int k = 0; k < RPL; k++) {
            G[k] = nG[k];
            F[k] = nF[k];
            M[k] = nM[k];
        }
        gam = ngam;
        n -= 1;
    }
};

}  // namespace dev
}  // namespace nsg
