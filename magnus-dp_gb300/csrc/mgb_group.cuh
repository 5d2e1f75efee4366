// The block rules on groups of four samples: as chains for a rule fixed at
// compile time, and as weights chosen at run time (one kernel serves all four
// rules).
#pragma once

#include "mgb_common.cuh"

namespace mgb {
namespace {

// Prefix sums of one element over a group of four samples, from the group's
// start: s[l - 1] = lo + (rule's weights of f0..f_l), so that the prefix at
// sample l is base + s[l - 1] (the block rules of mgb_common.cuh's fwd_step).
// all = false: s[3] only.  The terms of a block enter by the size of their
// weights, smallest first: the partial sums, and so their roundings, stay small
// (2 x 2 trajectories of nine samples, n = 2, Boole in FP32: 3.2e-7, and 4.3e-7 in
// the samples' order).
template <class T, int RULE>
__device__ __forceinline__ void group_sums(T lo, T f0, T f1, T f2, T f3, T f4, const RuleCoef<T>& k, bool all, T (&s)[4]) {
    if (RULE == R_BOOLE) {
        if (all) {
            s[0] = fma(f1, k.h, fma(f0, k.h, lo));
            s[1] = fma(f1, k.c4_3, fma(f2, k.t3, fma(f0, k.t3, lo)));
            s[2] = fma(f2, k.c98, fma(f1, k.c98, fma(f3, k.c38, fma(f0, k.c38, lo))));
        }
        s[3] = fma(f3, k.b64, fma(f1, k.b64, fma(f2, k.b24, fma(f4, k.b14, fma(f0, k.b14, lo)))));
    } else if (RULE == R_SIMPSON) {
        const T t43 = T(4) * k.t3;
        if (all) s[0] = fma(f1, k.h, fma(f0, k.h, lo));
        s[1] = fma(f1, t43, fma(f2, k.t3, fma(f0, k.t3, lo)));
        if (all) s[2] = fma(f3, k.h, fma(f2, k.h, s[1]));
        s[3] = fma(f3, t43, fma(f4, k.t3, fma(f2, k.t3, s[1])));
    } else if (RULE == R_TRAP) {
        s[0] = fma(f1, k.h, fma(f0, k.h, lo));
        s[1] = fma(f2, k.h, fma(f1, k.h, s[0]));
        s[2] = fma(f3, k.h, fma(f2, k.h, s[1]));
        s[3] = fma(f4, k.h, fma(f3, k.h, s[2]));
    } else {
        s[0] = fma(f1, k.dt, lo);
        s[1] = fma(f2, k.dt, s[0]);
        s[2] = fma(f3, k.dt, s[1]);
        s[3] = fma(f4, k.dt, s[2]);
    }
}
// base + lo += the group's total s4 (which starts from lo)
__device__ __forceinline__ void group_end(float& base, float& lo, float s4) {
    float v, e;
    two_sum(base, s4, v, e);
    base = v;
    lo = e;
}
__device__ __forceinline__ void group_end(double& base, double&, double s4) { base += s4; }

// Prefix P of one element at the samples of a full group (f0: the input at its
// anchor, f1..f4 at its samples) from the running value base + lo, which is
// advanced.  all = false: the running value is all that is wanted.  Boole in
// FP32 compensates the group's total, Simpson each pair's (2 x 2 trajectories of
// nine samples, n = 2: 2.5e-7, and 4.2e-7 with the group's alone; 4096 curves of
// 65537 samples, n = 6: 2.09 ms for 1.85).  (Trapezoid and Riemann in FP32 go sample by sample,
// fwd_step.)
template <class T, int RULE>
__device__ __forceinline__ void group_prefix(T& base, T& lo, T f0, T f1, T f2, T f3, T f4, const RuleCoef<T>& k, bool all, T (&P)[4]) {
    if (sizeof(T) == 4 && RULE == R_SIMPSON) {
        const T t43 = T(4) * k.t3;
        if (all) P[0] = base + fma(f1, k.h, fma(f0, k.h, lo));
        group_end(base, lo, fma(f1, t43, fma(f2, k.t3, fma(f0, k.t3, lo))));
        if (all) {
            P[1] = base + lo;
            P[2] = base + fma(f3, k.h, fma(f2, k.h, lo));
        }
        group_end(base, lo, fma(f3, t43, fma(f4, k.t3, fma(f2, k.t3, lo))));
        P[3] = base + lo;
        return;
    }
    T s[4];
    group_sums<T, RULE>(lo, f0, f1, f2, f3, f4, k, all, s);
    if (all)
#pragma unroll
        for (int l = 0; l < 3; ++l) P[l] = base + s[l];
    group_end(base, lo, s[3]);
    P[3] = base + lo;
}

// Weights of the block rules on a group: the prefix at sample l of the group
// is the anchor's plus sum_{i <= l} w[l - 1][i] f_i (mgb_common.cuh's rules).
template <class T>
struct GroupW {
    T w[4][5];
    // each: FP32 rules compensated by sample (Simpson: by pair), which go by
    // forward<true> and adjoint<true>; the caller branches around its whole loop
    // over elements, so that a rule's code is all it runs through
    bool each, simpson, riemann;
    __device__ __forceinline__ GroupW(int rule, const RuleCoef<T>& k)
        : each(sizeof(T) == 4 && rule != R_BOOLE), simpson(rule == R_SIMPSON), riemann(rule == R_RIEMANN) {
#pragma unroll
        for (int l = 0; l < 4; ++l)
#pragma unroll
            for (int i = 0; i < 5; ++i) w[l][i] = T(0);
        if (rule == R_BOOLE) {
            w[0][0] = w[0][1] = k.h;
            w[1][0] = w[1][2] = k.t3; w[1][1] = k.c4_3;
            w[2][0] = w[2][3] = k.c38; w[2][1] = w[2][2] = k.c98;
            w[3][0] = w[3][4] = k.b14; w[3][1] = w[3][3] = k.b64; w[3][2] = k.b24;
        } else if (rule == R_SIMPSON) {
            const T t43 = T(4) * k.t3;
            w[0][0] = w[0][1] = k.h;
            w[1][0] = w[1][2] = k.t3; w[1][1] = t43;
            w[2][0] = k.t3; w[2][1] = t43; w[2][2] = k.t3 + k.h; w[2][3] = k.h;
            w[3][0] = w[3][4] = k.t3; w[3][1] = w[3][3] = t43; w[3][2] = k.t3 + k.t3;
        } else if (rule == R_TRAP) {
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                w[l][0] = w[l][l + 1] = k.h;
#pragma unroll
                for (int i = 1; i <= l; ++i) w[l][i] = k.h + k.h;
            }
        } else {
#pragma unroll
            for (int l = 0; l < 4; ++l)
#pragma unroll
                for (int i = 1; i <= l + 1; ++i) w[l][i] = k.dt;
        }
    }
    // Prefix of one element over a group of cnt samples: v the rule's inputs
    // in, the prefix at the samples out (carry cy added if with_cy); base + lo
    // its running local value, f0 the input at the group's anchor.  FP32
    // Trapezoid and Riemann compensate every sample's increment, Simpson every
    // pair's.  all = false:
    // the running value is all that is wanted.
    template <bool EACH>
    __device__ __forceinline__ void forward(T (&v)[4], int cnt, T& base, T& lo, T f0, bool with_cy, const Carry<T>& cy,
                                            bool all = true) const {
        auto out = [&](T x) { return with_cy ? add_carry(x, cy) : x; };
        if constexpr (EACH) {
            T fp = f0, f1 = T(0);
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const T fl = v[l];
                if (simpson && l % 2 == 0) {
                    v[l] = out((fma(fl, w[0][1], fp * w[0][0]) + lo) + base);
                    f1 = fl;
                } else {
                    const T inc = simpson ? fma(f1, w[1][1], fma(fp, w[1][0], fl * w[1][2])) : fma(fl, w[0][1], fp * w[0][0]);
                    if (l < cnt) acc_add(base, lo, inc);
                    v[l] = out(base + lo);
                    fp = fl;
                }
            }
            return;
        }
        if (!all && cnt == 4) {
            group_end(base, lo, fma(v[2], w[3][3], fma(v[0], w[3][1], fma(v[1], w[3][2], fma(v[3], w[3][4], fma(f0, w[3][0], lo))))));
            return;
        }
        // (smallest weights first, as in group_sums)
        const T s1 = fma(v[0], w[0][1], fma(f0, w[0][0], lo));
        const T s2 = fma(v[0], w[1][1], fma(v[1], w[1][2], fma(f0, w[1][0], lo)));
        const T s3 = fma(v[1], w[2][2], fma(v[0], w[2][1], fma(v[2], w[2][3], fma(f0, w[2][0], lo))));
        T s4 = fma(v[2], w[3][3], fma(v[0], w[3][1], fma(v[1], w[3][2], fma(v[3], w[3][4], fma(f0, w[3][0], lo)))));
        if (cnt < 4) s4 = cnt == 1 ? s1 : cnt == 2 ? s2 : s3;
        v[0] = out(base + s1);
        v[1] = out(base + s2);
        v[2] = out(base + s3);
        group_end(base, lo, s4);
        v[3] = out(base + lo);
    }
    // Its adjoint, groups backwards: v the cotangents on the prefix at the
    // group's samples in (local), on the rule's inputs there out; Rb + rlo the
    // cotangent on the anchor from later samples (cy: from beyond the chunk),
    // pend in: on the last input from the later group, out: on the anchor's.
    // FP32 Trapezoid and Riemann compensate every sample's cotangent (Simpson:
    // every pair's), as the forward pass does its increment: with the group's plain sum the gradient of
    // 3 x 3 trajectories of nine samples, n = 4, was off by 1.08e-7 (Riemann) and
    // 9.1e-8 (Trapezoid) instead of 9.6e-8 and 8.2e-8.
    template <bool EACH>
    __device__ __forceinline__ void adjoint(T (&v)[4], int cnt, T& Rb, T& rlo, T& pend, bool with_cy, const Carry<T>& cy) const {
        if constexpr (EACH) {
            auto total = [&](T x) { return with_cy ? add_carry(x, cy) : x; };
            T R = T(0), he = T(0);  // a pair's end: the cotangent on its prefix, and the local part
#pragma unroll
            for (int l = 3; l >= 0; --l) {
                const T h = v[l];
                if (l >= cnt) continue;
                if (simpson && l % 2 == 1) {
                    he = h;
                    R = total((h + rlo) + Rb);
                    v[l] = fma(R, w[1][0], pend);
                } else if (simpson) {
                    v[l] = fma(R, w[1][1], h * w[0][1]);
                    pend = fma(R, w[1][0], h * w[0][0]);
                    acc_add(Rb, rlo, h + he);
                } else {
                    acc_add(Rb, rlo, h);
                    R = total(Rb + rlo);
                    v[l] = fma(R, w[0][1], pend);
                    pend = riemann ? T(0) : R * w[0][0];  // (no weight on the anchor: infinities stay out)
                }
            }
            return;
        }
        T H[4];
#pragma unroll
        for (int l = 0; l < 4; ++l) H[l] = l < cnt ? v[l] : T(0);
        const T Hend = cnt == 4 ? H[3] : cnt == 3 ? H[2] : cnt == 2 ? H[1] : H[0];
        T R = (Hend + rlo) + Rb;
        if (with_cy) R = add_carry(R, cy);
        acc_add(Rb, rlo, H[0] + H[1] + H[2] + H[3]);
        // the group end's cotangent stands in for its sample's; later ones are absent
#pragma unroll
        for (int l = 0; l < 4; ++l) H[l] = l + 1 == cnt ? R : H[l];
        T g[5];
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            // the group end's term, by far the largest, last: one rounding at its size
            g[i] = T(0);
#pragma unroll
            for (int l = 0; l < 4; ++l)
                if (l + 1 >= i) g[i] = fma(H[l], w[l][i], g[i]);
        }
#pragma unroll
        for (int l = 0; l < 4; ++l) v[l] = l + 1 == cnt ? g[l + 1] + pend : g[l + 1];
        pend = g[0];
    }
};

}  // namespace
}  // namespace mgb
