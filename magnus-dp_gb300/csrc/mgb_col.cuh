// Chunk kernel for small matrices (d = 3..8), both precision forms, with one
// thread per matrix column: variant 0 of the generic kernel at these
// dimensions.
//
// In W_{j+1} = A P_j and H_j = A^T G_{j+1} the columns of the right factor are
// independent, so a team of d lanes runs a whole chunk with the column's
// values in registers and only A shared: its rows come from shared memory as
// broadcasts, one 16-byte load per four (FP64: two) multiply-adds.  dA += G
// P^T mixes the columns: the team puts G into shared memory and lane c forms
// column c of dA from it and row c of P.  Samples go four at a time, all
// levels per group; the prefix state of every level lives in shared memory
// (per lane, free of bank conflicts), so that the level loop stays rolled and
// any order runs the same code.  The block rules enter as their weights on a
// group's samples.  The VJP replays its run into a tape of P_j (global, row
// major) and walks the groups backwards.
//
// The level-major kernel (mgb_generic.cu) reads both factors of every
// multiply-add from global level buffers.  256 trajectories of 8193 samples,
// n = 4, FP32, forward local pass / VJP, level-major -> here: d = 8: 7.46 ->
// 0.73 / 18.7 -> 2.70 ms, d = 4: 1.96 -> 0.22 / 4.81 -> 0.76; FP64, 64
// trajectories, d = 8: 4.33 -> 3.05 / 10.2 -> 8.11 ms (73 % of the FP64 pipe's
// two multiply-adds a clock).  The FP32 VJP holds eight warps an SM (registers)
// and waits for its tape rows and carries: asking for them ahead of the
// products took it from 3.24 to 2.70 ms.
//
// Small calls: LPC teams of a CTA share a chunk, each taking a run of groups;
// their totals meet in shared memory, where one team carries the state from
// run to run in FP64 (Chen's identity) and another the cotangent backwards.
#pragma once

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <type_traits>
#include <vector>

#include "mgb_common.cuh"
#include "mgb_group.cuh"
#include "mgb_tuned.h"

namespace mgb {
namespace {

constexpr size_t kColSmem = 200 * 1024;

// CNT threads per CTA: 64 (shared memory per CTA bounds the resident warps), and
// 128 for FP64 calls so small that sixteen runs share a chunk.
template <class T, int D, int CNT_ = 64>
struct ColGeo {
    static constexpr int CNT = CNT_;
    static constexpr int m = D * D;
    static constexpr int TPW = 32 / D;               // teams per warp
    static constexpr int TC = TPW * (CNT / 32);      // teams per CTA
    static constexpr int PADT = 16 / (int)sizeof(T);
    // a team's buffer of four samples; 16-byte aligned, teams on different banks
    static constexpr int BUF = (4 * m + PADT - 1) / PADT * PADT + PADT;
    static constexpr bool F32 = sizeof(T) == 4;
    static constexpr int NS = F32 ? 3 : 2;           // state values per element and level
    static size_t team_bytes(int mode, int nmax, int lpc) {
        const size_t bufs = (size_t)(mode == MODE_LOCAL ? 2 : 3) * BUF * sizeof(T);
        const size_t lam = lpc > 1 ? (size_t)nmax * m * sizeof(double) : 0;
        return (std::max(bufs, lam) + 15) / 16 * 16;
    }
    static size_t smem(int mode, int nmax, int lpc) {
        return (size_t)TC * team_bytes(mode, nmax, lpc) + (size_t)nmax * NS * D * CNT * sizeof(T);
    }
    // team slot (VJP): start state and end cotangent (FP32: hi and lo), tape
    static int64_t slot(int nmax, int64_t kmax, int lpc) {
        const int64_t run = 4 * (((kmax + 3) / 4 + lpc - 1) / lpc);
        return (int64_t)nmax * m * (F32 ? 4 : 2) + (run + 1) * std::max(nmax - 1, 0) * m;
    }
};

// row of D values (a multiple of D from a 16-byte boundary), in 16-byte loads where D allows
template <int D>
__device__ __forceinline__ void load_row(const float* p, float (&v)[D]) {
    if constexpr (D % 4 == 0) {
#pragma unroll
        for (int i = 0; i < D / 4; ++i) {
            const float4 x = reinterpret_cast<const float4*>(p)[i];
            v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
        }
    } else if constexpr (D % 2 == 0) {
#pragma unroll
        for (int i = 0; i < D / 2; ++i) {
            const float2 x = reinterpret_cast<const float2*>(p)[i];
            v[2 * i] = x.x; v[2 * i + 1] = x.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < D; ++i) v[i] = p[i];
    }
}
template <int D>
__device__ __forceinline__ void load_row(const double* p, double (&v)[D]) {
    if constexpr (D % 2 == 0) {
#pragma unroll
        for (int i = 0; i < D / 2; ++i) {
            const double2 x = reinterpret_cast<const double2*>(p)[i];
            v[2 * i] = x.x; v[2 * i + 1] = x.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < D; ++i) v[i] = p[i];
    }
}

// y = A x (A row-major in shared memory)
template <class T, int D>
__device__ __forceinline__ void mat_vec(const T* A, const T (&x)[D], T (&y)[D]) {
#pragma unroll
    for (int r = 0; r < D; ++r) {
        T a[D];
        load_row<D>(A + r * D, a);
        T s = a[0] * x[0];
#pragma unroll
        for (int k = 1; k < D; ++k) s = fma(a[k], x[k], s);
        y[r] = s;
    }
}
// y = A^T x
template <class T, int D>
__device__ __forceinline__ void mat_t_vec(const T* A, const T (&x)[D], T (&y)[D]) {
#pragma unroll
    for (int k = 0; k < D; ++k) {
        T a[D];
        load_row<D>(A + k * D, a);
#pragma unroll
        for (int r = 0; r < D; ++r) y[r] = k == 0 ? a[r] * x[k] : fma(a[r], x[k], y[r]);
    }
}

template <class T, int D, int MODE, int CNT>
__global__ void __launch_bounds__(CNT)
    k_col(const InstDev* __restrict__ insts, const ChunkRef* __restrict__ work, int64_t nwork, T* __restrict__ scratch,
          int64_t slot_elems, int lpc, int rule, int f64io, int team_bytes) {
    using Geo = ColGeo<T, D, CNT>;
    constexpr int m = Geo::m, TPW = Geo::TPW, TC = Geo::TC, BUF = Geo::BUF, NS = Geo::NS;
    constexpr bool F32 = Geo::F32;
    extern __shared__ __align__(16) uint8_t shb[];
    const bool f64 = f64io != 0;
    const int tid = threadIdx.x, lane = tid & 31, tw = lane / D, c = lane - tw * D;
    const bool lane_on = tw < TPW;
    const int tix = (tid >> 5) * TPW + (lane_on ? tw : 0);  // team of the CTA
    const unsigned tmask = ((1u << D) - 1u) << ((lane_on ? tw : 0) * D);
    T* const buf = reinterpret_cast<T*>(shb + (size_t)tix * team_bytes);  // A x 2, then G
    double* const lamS = reinterpret_cast<double*>(buf);                  // (between phases) the run's totals
    T* const state = reinterpret_cast<T*>(shb + (size_t)TC * team_bytes) + tid;
    double* const dstate = reinterpret_cast<double*>(shb + (size_t)TC * team_bytes) + tid;
    auto st = [&](int j, int v, int r) -> T& { return state[((j * NS + v) * D + r) * CNT]; };
    // per CTA: TC / lpc chunks, team tix works on chunk tix / lpc as run tix % lpc
    const int cpb = TC / lpc, mych = tix / lpc, sub = tix - mych * lpc;
    T* const slot = scratch + ((int64_t)blockIdx.x * TC + tix) * slot_elems;

    for (int64_t w0 = (int64_t)blockIdx.x * cpb; w0 < nwork; w0 += (int64_t)gridDim.x * cpb) {
        const bool on = lane_on && mych < cpb && w0 + mych < nwork;
        const ChunkRef wk = work[on ? w0 + mych : 0];
        const InstDev& I = insts[wk.inst];
        const int ch = wk.chunk, n = I.n;
        const int64_t b = (int64_t)ch * I.K;
        const int64_t e = (b + I.K < I.S - 1) ? b + I.K : I.S - 1;
        const int Kp = (int)(e - b);
        const int span = 4 * (((Kp + 3) / 4 + lpc - 1) / lpc);
        const int l0 = min(sub * span, Kp), l1 = min(l0 + span, Kp);  // samples (l0, l1]
        const bool riem0 = rule == R_RIEMANN && ch == 0 && sub == 0;  // Riemann's first sample counts
        const bool riem = rule == R_RIEMANN;  // (its anchor sample has no weight: kept out, infinities and all)
        const RuleCoef<T> kc = rule_coef<T>(I);
        const GroupW<T> gw(rule, kc);
        const int64_t nm = (int64_t)n * m;
        T* const sPI = slot;                              // [n][m] (+ [n][m] lo)
        T* const sRHO = sPI + nm * (F32 ? 2 : 1);         // likewise
        T* const tape = sRHO + nm * (F32 ? 2 : 1);        // [run + 1][n - 1][m]

        // samples li .. li + 3 of A into the team's buffer q (zeros past the
        // run's end), asynchronously when no conversion is needed
        auto stage = [&](int li, int q) {
            T* dst = buf + q * BUF;
            const int cnt = (min(l1, li + 3) - li + 1) * m;
            const int64_t at = (b + li) * m;
            if (f64 == !F32) {
                const T* src = static_cast<const T*>(I.A) + at;
#pragma unroll
                for (int i = 0; i < 4 * D; ++i) {
                    const int x = c + i * D;
                    if (x < cnt)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + x)),
                                     "l"(src + x), "n"((int)sizeof(T))
                                     : "memory");
                    else dst[x] = T(0);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 4 * D; ++i) {
                    const int x = c + i * D;
                    dst[x] = x < cnt ? load_in<T>(I.A, at + x, f64) : T(0);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto landed = [&]() {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp(tmask);
        };
        // the run's groups: first sample and count (Riemann's sample 0 is a group of one)
        const int g0 = riem0 ? 0 : l0 + 1;
        auto next_of = [&](int li) { return (riem0 && li == 0) ? 1 : li + 4; };
        auto prev_of = [&](int li) { return (riem0 && li == 1) ? 0 : li - 4; };
        auto count_of = [&](int li) { return (riem0 && li == 0) ? 1 : min(4, l1 - li + 1); };
        const int glast = l1 > l0 ? l0 + 1 + ((l1 - l0 - 1) & ~3) : (riem0 ? 0 : l1 + 1);

        // One pass forward over the run: NL levels from the lane's state;
        // carry: the start state is added to emitted values, which go to the
        // tape; emit_top: the last level's values are wanted too
        auto forward = [&](int NL, bool carry, bool emit_top) {
            if (g0 > l1 || NL == 0) return;
            int q = 0;
            stage(g0, 0);
            for (int li = g0; li <= l1; li = next_of(li), q ^= 1) {
                landed();
                if (next_of(li) <= l1) stage(next_of(li), q ^ 1);
                const T* A = buf + q * BUF;
                const int cnt = count_of(li);
                T f[4][D];
#pragma unroll
                for (int l = 0; l < 4; ++l)
#pragma unroll
                    for (int r = 0; r < D; ++r) f[l][r] = A[l * m + r * D + c];
                // a level's carries are asked for ahead of the products before it
                T chi[D], clo[D];
                auto load_carry = [&](int j) {
                    if (carry) {
#pragma unroll
                        for (int r = 0; r < D; ++r) {
                            chi[r] = sPI[j * m + r * D + c];
                            clo[r] = F32 ? sPI[nm + j * m + r * D + c] : T(0);
                        }
                    }
                };
                load_carry(0);
                for (int j = 0; j < NL; ++j) {
                    const bool emit = emit_top || j + 1 < NL;
                    auto prefix = [&](auto eachc) {
#pragma unroll
                        for (int r = 0; r < D; ++r) {
                            T base = st(j, 0, r), f0 = st(j, 1, r), lo = F32 ? st(j, NS - 1, r) : T(0);
                            Carry<T> cy{T(0), T(0)};
                            if (carry) cy = Carry<T>{chi[r], clo[r]};
                            T v[4] = {f[0][r], f[1][r], f[2][r], f[3][r]};
                            const T fl = cnt == 4 ? v[3] : cnt == 3 ? v[2] : cnt == 2 ? v[1] : v[0];
                            gw.template forward<decltype(eachc)::value>(v, cnt, base, lo, f0, carry, cy, emit);
#pragma unroll
                            for (int l = 0; l < 4; ++l) f[l][r] = v[l];
                            st(j, 0, r) = base;
                            if (F32) st(j, NS - 1, r) = lo;
                            st(j, 1, r) = riem ? T(0) : fl;
                        }
                    };
                    if (F32 && gw.each) prefix(std::integral_constant<bool, F32>{});
                    else prefix(std::false_type{});
                    if (!emit) break;
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        if (l >= cnt) break;
                        if (carry) {
                            T* tp = tape + ((int64_t)(li + l - l0) * (n - 1) + j) * m + c;
#pragma unroll
                            for (int r = 0; r < D; ++r) tp[r * D] = f[l][r];
                        }
                    }
                    if (j + 1 < NL) {
                        load_carry(j + 1);
#pragma unroll
                        for (int l = 0; l < 4; ++l) {
                            T y[D];
                            mat_vec<T, D>(A + l * m, f[l], y);
#pragma unroll
                            for (int r = 0; r < D; ++r) f[l][r] = y[r];
                        }
                    }
                }
                __syncwarp(tmask);  // the buffer is free
            }
        };
        // state of a zero-carry pass at sample l0
        auto local_start = [&]() {
            for (int j = 0; j < n; ++j)
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    st(j, 0, r) = T(0);
                    if (F32) st(j, NS - 1, r) = T(0);
                    st(j, 1, r) = j == 0 && !riem ? load_in<T>(I.A, (b + l0) * m + r * D + c, f64) : T(0);
                }
        };
        // the run's totals (local prefix at its end) into shared memory
        auto publish = [&]() {
            for (int j = 0; j < n; ++j)
#pragma unroll
                for (int r = 0; r < D; ++r)
                    lamS[j * m + r * D + c] = (double)st(j, 0, r) + (F32 ? (double)st(j, NS - 1, r) : 0.0);
        };
        auto run_lam = [&](int s) {  // totals of run s of this chunk
            return reinterpret_cast<const double*>(shb + (size_t)(mych * lpc + s) * team_bytes);
        };
        // column c of the state, FP64, in the lane's state memory
        auto ds = [&](int j, int r) -> double& { return dstate[(j * D + r) * CNT]; };
        // state <- Chen(totals of run s, state)
        auto chen = [&](const double* L) {
            for (int j = n - 1; j >= 0; --j) {
                double v[D];
#pragma unroll
                for (int r = 0; r < D; ++r) v[r] = ds(j, r) + L[j * m + r * D + c];
                for (int mm = 0; mm < j; ++mm) {
                    double x[D], y[D];
#pragma unroll
                    for (int r = 0; r < D; ++r) x[r] = ds(mm, r);
                    mat_vec<double, D>(L + (j - mm - 1) * m, x, y);
#pragma unroll
                    for (int r = 0; r < D; ++r) v[r] += y[r];
                }
#pragma unroll
                for (int r = 0; r < D; ++r) ds(j, r) = v[r];
            }
        };

        if (MODE == MODE_LOCAL) {
            if (on) {
                local_start();
                forward(n, false, false);
                if (lpc == 1) {
                    for (int j = 0; j < n; ++j)
#pragma unroll
                        for (int r = 0; r < D; ++r)
                            I.lam[(int64_t)ch * nm + j * m + r * D + c] =
                                (double)st(j, 0, r) + (F32 ? (double)st(j, NS - 1, r) : 0.0);
                } else {
                    publish();
                }
            }
            if (lpc > 1) {
                __syncthreads();
                if (on && sub == 0) {
                    for (int j = 0; j < n; ++j)
#pragma unroll
                        for (int r = 0; r < D; ++r) ds(j, r) = lamS[j * m + r * D + c];
                    for (int s = 1; s < lpc; ++s) chen(run_lam(s));
                    for (int j = 0; j < n; ++j)
#pragma unroll
                        for (int r = 0; r < D; ++r) I.lam[(int64_t)ch * nm + j * m + r * D + c] = ds(j, r);
                }
                __syncthreads();
            }
            continue;
        }

        // ================================ VJP ================================
        const double* pic = I.pi + (int64_t)ch * nm;
        const double* rcc = I.rho + (int64_t)ch * nm;
        const bool riem_c0 = rule == R_RIEMANN && ch == 0;
        // FP64 column -> a run's slot (hi, and lo in FP32)
        auto put = [&](T* dst, int j, int r, double v) {
            const Carry<T> s = split_carry<T>(v);
            dst[j * m + r * D + c] = s.hi;
            if (F32) dst[nm + j * m + r * D + c] = s.lo;
        };
        if (lpc > 1) {
            if (on) {
                local_start();
                forward(n, false, false);
                __syncwarp(tmask);
                publish();
            }
            __syncthreads();
            auto slot_of = [&](int s) { return scratch + ((int64_t)blockIdx.x * TC + mych * lpc + s) * slot_elems; };
            if (on && sub == 0) {
                // start states of the runs
                for (int j = 0; j < n; ++j)
#pragma unroll
                    for (int r = 0; r < D; ++r) ds(j, r) = riem_c0 ? 0.0 : pic[j * m + r * D + c];
                for (int s = 0; s < lpc; ++s) {
                    T* dst = slot_of(s);
                    for (int j = 0; j < n; ++j)
#pragma unroll
                        for (int r = 0; r < D; ++r) put(dst, j, r, ds(j, r));
                    if (s + 1 < lpc) chen(run_lam(s));
                }
            }
            if (on && sub == 1) {
                // end cotangents of the runs: rho_m += sum_{j>m} Lambda_{j-m}^T rho_j
                for (int j = 0; j < n; ++j)
#pragma unroll
                    for (int r = 0; r < D; ++r) ds(j, r) = rcc[j * m + r * D + c];
                for (int s = lpc - 1; s >= 0; --s) {
                    T* dst = slot_of(s) + nm * (F32 ? 2 : 1);
                    for (int j = 0; j < n; ++j)
#pragma unroll
                        for (int r = 0; r < D; ++r) put(dst, j, r, ds(j, r));
                    const double* L = run_lam(s);
                    for (int mm = 0; s > 0 && mm < n; ++mm) {
                        double v[D];
#pragma unroll
                        for (int r = 0; r < D; ++r) v[r] = ds(mm, r);
                        for (int j = mm + 1; j < n; ++j) {
                            double x[D], y[D];
#pragma unroll
                            for (int r = 0; r < D; ++r) x[r] = ds(j, r);
                            mat_t_vec<double, D>(L + (j - mm - 1) * m, x, y);
#pragma unroll
                            for (int r = 0; r < D; ++r) v[r] += y[r];
                        }
#pragma unroll
                        for (int r = 0; r < D; ++r) ds(mm, r) = v[r];
                    }
                }
            }
            __syncthreads();
        } else if (on) {
            for (int j = 0; j < n; ++j)
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    put(sPI, j, r, riem_c0 ? 0.0 : pic[j * m + r * D + c]);
                    put(sRHO, j, r, rcc[j * m + r * D + c]);
                }
            __syncwarp(tmask);
        }

        T dlast[D];
#pragma unroll
        for (int r = 0; r < D; ++r) dlast[r] = T(0);
        const bool next = sub + 1 < lpc && l1 < Kp;  // another run continues at l1
        if (on) {
            // replay from the start state
            stage(l0, 0);
            landed();
            for (int j = 0; j < n - 1; ++j) {
                T x[D], y[D];
                if (j > 0) {
#pragma unroll
                    for (int r = 0; r < D; ++r) x[r] = sPI[(j - 1) * m + r * D + c];
                    mat_vec<T, D>(buf, x, y);
                } else {
#pragma unroll
                    for (int r = 0; r < D; ++r) y[r] = buf[r * D + c];
                }
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    st(j, 0, r) = T(0);
                    if (F32) st(j, NS - 1, r) = T(0);
                    st(j, 1, r) = riem ? T(0) : y[r];
                }
            }
            __syncwarp(tmask);
            forward(n - 1, true, true);

            // ---- adjoint: Rb, pend, (FP32) rlo
            for (int j = 0; j < n; ++j)
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    st(j, 0, r) = T(0);
                    if (F32) st(j, NS - 1, r) = T(0);
                    st(j, 1, r) = T(0);
                }
            __syncwarp(tmask);
            T* const Gs = buf + 2 * BUF;
            if (g0 <= l1) {
                int q = 0;
                stage(glast, 0);
                for (int li = glast; li >= g0; li = prev_of(li), q ^= 1) {
                    landed();
                    if (prev_of(li) >= g0) stage(prev_of(li), q ^ 1);
                    const T* A = buf + q * BUF;
                    const int cnt = count_of(li);
                    T G[4][D], dA[4][D];
#pragma unroll
                    for (int l = 0; l < 4; ++l)
#pragma unroll
                        for (int r = 0; r < D; ++r) G[l][r] = dA[l][r] = T(0);
                    for (int j = n - 1; j >= 0; --j) {
                        // the level's global operands are asked for ahead of the
                        // products: the carry, and each sample's row of P one
                        // sample early (waiting for them took half of the cycles)
                        T rh[D], rl[D], p[D];
#pragma unroll
                        for (int r = 0; r < D; ++r) {
                            rh[r] = sRHO[j * m + r * D + c];
                            rl[r] = F32 ? sRHO[nm + j * m + r * D + c] : T(0);
                        }
                        const T* const tp = tape + ((int64_t)(li - l0) * (n - 1) + j) * m + c * D;
                        if (j + 1 < n) {
                            load_row<D>(tp, p);
                            // G_{j+1} to shared memory; dA += G_{j+1} P_j^T, H_j = A^T G_{j+1}
#pragma unroll
                            for (int l = 0; l < 4; ++l)
#pragma unroll
                                for (int r = 0; r < D; ++r) Gs[l * m + r * D + c] = G[l][r];
                            __syncwarp(tmask);
#pragma unroll
                            for (int l = 0; l < 4; ++l) {
                                if (l >= cnt) break;
                                T pn[D];
                                if (l + 1 < 4 && l + 1 < cnt) load_row<D>(tp + (int64_t)(l + 1) * (n - 1) * m, pn);
#pragma unroll
                                for (int r = 0; r < D; ++r) {
                                    T g[D];
                                    load_row<D>(Gs + l * m + r * D, g);
                                    T s = g[0] * p[0];
#pragma unroll
                                    for (int k = 1; k < D; ++k) s = fma(g[k], p[k], s);
                                    dA[l][r] += s;  // (one running sum over the levels too rounds more)
                                }
                                T h[D];
                                mat_t_vec<T, D>(A + l * m, G[l], h);
#pragma unroll
                                for (int k = 0; k < D; ++k) p[k] = pn[k];
#pragma unroll
                                for (int r = 0; r < D; ++r) G[l][r] = h[r];
                            }
                            __syncwarp(tmask);
                        }
                        auto reverse = [&](auto eachc) {
#pragma unroll
                            for (int r = 0; r < D; ++r) {
                                T Rb = st(j, 0, r), pend = st(j, 1, r), rlo = F32 ? st(j, NS - 1, r) : T(0);
                                Carry<T> cy{T(0), T(0)};
                                cy = Carry<T>{rh[r], rl[r]};
                                T v[4] = {G[0][r], G[1][r], G[2][r], G[3][r]};
                                gw.template adjoint<decltype(eachc)::value>(v, cnt, Rb, rlo, pend, true, cy);
#pragma unroll
                                for (int l = 0; l < 4; ++l) G[l][r] = v[l];
                                st(j, 0, r) = Rb;
                                st(j, 1, r) = riem ? T(0) : pend;
                                if (F32) st(j, NS - 1, r) = rlo;
                            }
                        };
                        if (F32 && gw.each) reverse(std::integral_constant<bool, F32>{});
                        else reverse(std::false_type{});
                    }
#pragma unroll
                    for (int l = 0; l < 4; ++l) {
                        if (l >= cnt) break;
                        const int lis = li + l;
                        if (next && lis == l1) {
                            // completed below by the next run's share
#pragma unroll
                            for (int r = 0; r < D; ++r) dlast[r] = dA[l][r] + G[l][r];
                        } else {
                            const bool shared = lis == Kp && ch < I.C - 1;
#pragma unroll
                            for (int r = 0; r < D; ++r) {
                                const T v = dA[l][r] + G[l][r];
                                const int64_t at = (b + lis) * m + r * D + c;
                                if (shared) atomic_add_out<T>(I.dA, at, v, f64);
                                else store_out<T>(I.dA, at, v, f64);
                            }
                        }
                    }
                    __syncwarp(tmask);
                }
            }
            // this run's copy of W_j at sample l0: dA[l0] += pend_1 + sum_{j<n} pend_{j+1} pi_j^T
            if (rule != R_RIEMANN && (sub == 0 || l0 < l1)) {
                T v[D];
#pragma unroll
                for (int r = 0; r < D; ++r) v[r] = st(0, 1, r);
                for (int j = 1; j < n; ++j) {
                    __syncwarp(tmask);
#pragma unroll
                    for (int r = 0; r < D; ++r) Gs[r * D + c] = st(j, 1, r);
                    __syncwarp(tmask);
                    T p[D];
                    load_row<D>(sPI + (j - 1) * m + c * D, p);
#pragma unroll
                    for (int r = 0; r < D; ++r) {
                        T g[D];
                        load_row<D>(Gs + r * D, g);
#pragma unroll
                        for (int k = 0; k < D; ++k) v[r] = fma(g[k], p[k], v[r]);
                    }
                }
                __syncwarp(tmask);
                if (sub == 0) {
#pragma unroll
                    for (int r = 0; r < D; ++r) {
                        const int64_t at = b * m + r * D + c;
                        if (ch > 0) atomic_add_out<T>(I.dA, at, v[r], f64);
                        else store_out<T>(I.dA, at, v[r], f64);
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < D; ++r) Gs[r * D + c] = v[r];
                }
            } else if (sub > 0) {
#pragma unroll
                for (int r = 0; r < D; ++r) Gs[r * D + c] = T(0);
            }
        }
        if (lpc > 1) {
            __syncthreads();
            if (on && next) {
                const T* nv = reinterpret_cast<const T*>(shb + (size_t)(tix + 1) * team_bytes) + 2 * BUF;
#pragma unroll
                for (int r = 0; r < D; ++r)
                    store_out<T>(I.dA, (b + l1) * m + r * D + c, dlast[r] + nv[r * D + c], f64);
            }
            __syncthreads();
        }
    }
}

template <class T, int D, int MODE, int CNT>
cudaError_t col_go(int rule, const LaunchArgs& a, int nmax, bool prepare_only) {
    using Geo = ColGeo<T, D, CNT>;
    static std::mutex mu;
    static std::vector<bool> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(mu);
        if ((int)done.size() <= dev) done.resize(dev + 1, false);
        if (!done[dev]) {
            e = cudaFuncSetAttribute(k_col<T, D, MODE, CNT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kColSmem);
            if (e != cudaSuccess) return e;
            done[dev] = true;
        }
    }
    if (prepare_only) return cudaSuccess;
    if (a.lpc < 1 || a.lpc > Geo::TC) return cudaErrorInvalidValue;  // a chunk's runs must fit in one CTA
    const int cpb = Geo::TC / a.lpc;
    int64_t blocks = (a.nwork + cpb - 1) / cpb;
    int64_t slot = 0;
    if (MODE == MODE_VJP) {
        // one slot per team of a resident CTA, cut from the segment's scratch
        slot = Geo::slot(nmax, a.kmax, a.lpc);
        blocks = std::min<int64_t>(blocks, a.grid * a.slot_elems / (slot * Geo::TC));
        if (blocks < 1) return cudaErrorInvalidValue;
    }
    k_col<T, D, MODE, CNT><<<(unsigned)std::max<int64_t>(1, blocks), Geo::CNT, Geo::smem(MODE, nmax, a.lpc), a.stream>>>(
        a.insts, a.work, a.nwork, static_cast<T*>(a.scratch), slot, a.lpc, rule, a.f64io,
        (int)Geo::team_bytes(MODE, nmax, a.lpc));
    return cudaGetLastError();
}

template <class T, int D>
cudaError_t col_m(int rule, int mode, const LaunchArgs& a, int nmax, bool prepare_only) {
    if constexpr (sizeof(T) == 8) {
        if (prepare_only || a.lpc == 16) {
            const cudaError_t e = mode == MODE_LOCAL ? col_go<T, D, MODE_LOCAL, 128>(rule, a, nmax, prepare_only)
                                                     : col_go<T, D, MODE_VJP, 128>(rule, a, nmax, prepare_only);
            if (e != cudaSuccess || !prepare_only) return e;
        }
    }
    return mode == MODE_LOCAL ? col_go<T, D, MODE_LOCAL, 64>(rule, a, nmax, prepare_only)
                              : col_go<T, D, MODE_VJP, 64>(rule, a, nmax, prepare_only);
}

template <class T>
cudaError_t col_d(int D, int rule, int mode, const LaunchArgs& a, int nmax, bool prepare_only) {
    switch (D) {
        case 3: return col_m<T, 3>(rule, mode, a, nmax, prepare_only);
        case 4: return col_m<T, 4>(rule, mode, a, nmax, prepare_only);
        case 5: return col_m<T, 5>(rule, mode, a, nmax, prepare_only);
        case 6: return col_m<T, 6>(rule, mode, a, nmax, prepare_only);
        case 7: return col_m<T, 7>(rule, mode, a, nmax, prepare_only);
        default: return col_m<T, 8>(rule, mode, a, nmax, prepare_only);
    }
}

}  // namespace
}  // namespace mgb
