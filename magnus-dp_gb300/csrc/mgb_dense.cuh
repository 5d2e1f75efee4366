// Chunk kernel for d = 9..32 where no tensor-core kernel serves (the plain
// form from d = 16, and in the mixed form float64 data and other dimensions):
// one of the generic kernel's variants there (dense_variant in mgb_tuned.cu).
//
// One CTA per chunk, four samples at a time, all levels per group.  A thread
// owns a 1 x 4 tile of the matrices at all four samples, so that W = A P
// leaves the values its prefix pass needs in its own registers and only P (G,
// in the VJP) goes through shared memory; the prefix state of every level is
// kept in shared memory, per thread.  The VJP replays the chunk into a tape of
// P_j (global memory), and walks the groups backwards with dA in registers.
// In FP64 a multiply-add holds the pipe for 16 clocks a warp, and the three
// shared loads per four of them hide behind it: the kernel is bound by the
// FP64 pipe.  The level-major kernel (mgb_generic.cu), whose operands come
// from global level buffers, ran at a third of it.
// Forward local pass / VJP, level-major -> here: FP64, 4 trajectories of d = 32,
// S = 8193, n = 4: 17.2 -> 8.1 / 53.7 -> 22.3 ms (one chunk per SM on 128 of
// them: the pipe's own time is 7.6 ms forward); d = 16, 16 trajectories: 5.7 ->
// 4.6 / 16.8 -> 12.3.  FP32, 64 trajectories of d = 24, n = 6: 25.6 -> 8.4 / 88.6
// -> 43.5 ms.  Where half of a CTA's threads have no tile or there is one
// warp of them (d = 9..12) the level-major kernel is the faster one for small calls,
// and in FP64 for all below d = 16.
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

constexpr size_t kDenseSmem = 220 * 1024;

// Threads, row pitch (elements; rows start on 16 bytes) and shared memory
__host__ __device__ inline int dense_tiles(int d) { return (d + 3) / 4; }
__host__ __device__ inline int dense_threads(int d) { return (d * dense_tiles(d) + 31) / 32 * 32; }
template <class T>
__host__ __device__ inline int dense_pitch(int d) { return 4 * dense_tiles(d) + 16 / (int)sizeof(T); }
template <class T>
inline size_t dense_smem(int mode, int d, int nmax) {
    const size_t mats = (size_t)(mode == MODE_LOCAL ? 2 : 3) * 4 * 4 * dense_tiles(d) * dense_pitch<T>(d);
    const size_t state = (size_t)nmax * (sizeof(T) == 4 ? 3 : 2) * 4 * dense_threads(d);
    return (mats + state) * sizeof(T);
}

__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}
__device__ __forceinline__ void load4(const double* p, double (&v)[4]) {
    const double2 x = reinterpret_cast<const double2*>(p)[0], y = reinterpret_cast<const double2*>(p)[1];
    v[0] = x.x; v[1] = x.y; v[2] = y.x; v[3] = y.y;
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void store4(double* p, const double (&v)[4]) {
    reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}

template <class T, int MODE>
__global__ void __launch_bounds__(256)
    k_dense(const InstDev* __restrict__ insts, const ChunkRef* __restrict__ work, int64_t nwork, T* __restrict__ scratch,
            int64_t slot_elems, int d, int rule, int f64io) {
    constexpr bool F32 = sizeof(T) == 4;
    constexpr int NS = F32 ? 3 : 2;
    extern __shared__ __align__(16) uint8_t shd[];
    const bool f64 = f64io != 0;
    const int tiles = dense_tiles(d), NT = dense_threads(d), pit = dense_pitch<T>(d), mat = 4 * tiles * pit, m = d * d;
    const int tid = threadIdx.x, r = tid / tiles, c0 = 4 * (tid - r * tiles);
    const bool mine = r < d;             // spare threads only help with the copies
    const int nc = mine ? min(4, d - c0) : 0;  // valid columns of the tile
    T* const sA = reinterpret_cast<T*>(shd);   // [4][rows][pit], zero-padded
    T* const sP = sA + 4 * mat;                // P (forward) / G (adjoint)
    T* const sQ = sP + 4 * mat;                // P in the adjoint (VJP)
    T* const state = (MODE == MODE_LOCAL ? sQ : sQ + 4 * mat) + tid;
    auto st = [&](int j, int v, int u) -> T& { return state[((j * NS + v) * 4 + u) * NT]; };
    T* const slot = scratch + (int64_t)blockIdx.x * slot_elems;

    // the padding columns and rows are never written again
    for (int i = tid; i < (MODE == MODE_LOCAL ? 8 : 12) * mat; i += NT) sA[i] = T(0);
    __syncthreads();

    for (int64_t w = blockIdx.x; w < nwork; w += gridDim.x) {
        const ChunkRef wk = work[w];
        const InstDev& I = insts[wk.inst];
        const int ch = wk.chunk, n = I.n;
        const int64_t b = (int64_t)ch * I.K;
        const int64_t e = (b + I.K < I.S - 1) ? b + I.K : I.S - 1;
        const int Kp = (int)(e - b);
        const bool riem = rule == R_RIEMANN, riem0 = riem && ch == 0;  // Riemann's first sample counts
        const RuleCoef<T> kc = rule_coef<T>(I);
        const GroupW<T> gw(rule, kc);
        const int64_t nm = (int64_t)n * m;
        T* const sPI = slot;                       // FP32: carries hi [n][m], lo [n][m]
        T* const sRHO = sPI + (F32 ? 2 * nm : 0);  // likewise
        T* const tape = sRHO + (F32 ? 2 * nm : 0); // [Kp + 1][n - 1][m]
        const double* pic = I.pi + (int64_t)ch * nm;
        const double* rcc = I.rho + (int64_t)ch * nm;

        // samples li .. li + cnt - 1 of A (zeros after them)
        auto stage = [&](int li, int cnt) {
            for (int x = tid; x < 4 * m; x += NT) {
                const int l = x / m, el = x - l * m, row = el / d;
                sA[l * mat + row * pit + el - row * d] = l < cnt ? load_in<T>(I.A, (b + li + l) * m + el, f64) : T(0);
            }
        };
        // out = X Y for the thread's tile of sample l (X from shared memory by
        // rows, Y likewise), or X^T Y
        auto product = [&](const T* X, const T* Y, bool trans, T (&o)[4]) {
#pragma unroll
            for (int u = 0; u < 4; ++u) o[u] = T(0);
            const T* x = trans ? X + r : X + r * pit;
            const int sx = trans ? pit : 1;
#pragma unroll 4
            for (int k = 0; k < d; ++k) {
                T y[4];
                load4(Y + k * pit + c0, y);
                const T a = x[k * sx];
#pragma unroll
                for (int u = 0; u < 4; ++u) o[u] = fma(a, y[u], o[u]);
            }
        };
        auto next_of = [&](int li) { return (riem0 && li == 0) ? 1 : li + 4; };
        auto prev_of = [&](int li) { return (riem0 && li == 1) ? 0 : li - 4; };
        auto count_of = [&](int li) { return (riem0 && li == 0) ? 1 : min(4, Kp - li + 1); };
        const int g0 = riem0 ? 0 : 1, glast = 1 + ((Kp - 1) & ~3);

        // forward over the chunk: NL levels; carry: values go to the tape with
        // the chunk's start state added
        auto forward = [&](int NL, bool carry, bool emit_top) {
            if (NL == 0) return;
            for (int li = g0; li <= Kp; li = next_of(li)) {
                const int cnt = count_of(li);
                stage(li, cnt);
                __syncthreads();
                T f[4][4];
#pragma unroll
                for (int l = 0; l < 4; ++l)
#pragma unroll
                    for (int u = 0; u < 4; ++u) f[l][u] = mine ? sA[l * mat + r * pit + c0 + u] : T(0);
                for (int j = 0; j < NL; ++j) {
                    const bool emit = emit_top || j + 1 < NL;
                    if (mine) {
                        auto prefix = [&](auto eachc) {
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                T base = st(j, 0, u), f0 = st(j, 1, u), lo = F32 ? st(j, NS - 1, u) : T(0);
                                Carry<T> cy{T(0), T(0)};
                                if (carry && u < nc) {
                                    const int64_t el = (int64_t)j * m + r * d + c0 + u;
                                    cy = F32 ? Carry<T>{sPI[el], sPI[nm + el]} : Carry<T>{(T)(riem0 ? 0.0 : pic[el]), T(0)};
                                }
                                T v[4] = {f[0][u], f[1][u], f[2][u], f[3][u]};
                                const T fl = cnt == 4 ? v[3] : cnt == 3 ? v[2] : cnt == 2 ? v[1] : v[0];
                                gw.template forward<decltype(eachc)::value>(v, cnt, base, lo, f0, carry, cy, emit);
#pragma unroll
                                for (int l = 0; l < 4; ++l) f[l][u] = u < nc ? v[l] : T(0);
                                st(j, 0, u) = base;
                                if (F32) st(j, NS - 1, u) = lo;
                                st(j, 1, u) = riem ? T(0) : fl;
                            }
                        };
                        if (F32 && gw.each) prefix(std::integral_constant<bool, F32>{});
                        else prefix(std::false_type{});
                        if (emit) {
#pragma unroll
                            for (int l = 0; l < 4; ++l) {
                                store4(sP + l * mat + r * pit + c0, f[l]);
                                if (carry && l < cnt) {
                                    T* tp = tape + ((int64_t)(li + l) * (n - 1) + j) * m + r * d + c0;
#pragma unroll
                                    for (int u = 0; u < 4; ++u)
                                        if (u < nc) tp[u] = f[l][u];
                                }
                            }
                        }
                    }
                    if (j + 1 == NL) break;
                    __syncthreads();
                    if (mine) {
#pragma unroll
                        for (int l = 0; l < 4; ++l) product(sA + l * mat, sP + l * mat, false, f[l]);
                    }
                    __syncthreads();
                }
                __syncthreads();
            }
        };

        if (MODE == MODE_LOCAL) {
            if (mine)
                for (int j = 0; j < n; ++j)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        st(j, 0, u) = T(0);
                        if (F32) st(j, NS - 1, u) = T(0);
                        st(j, 1, u) = j == 0 && !riem && u < nc ? load_in<T>(I.A, b * m + r * d + c0 + u, f64) : T(0);
                    }
            forward(n, false, false);
            if (mine)
                for (int j = 0; j < n; ++j)
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (u < nc)
                            store_lam(I, (int64_t)ch * nm + j * m + r * d + c0 + u, st(j, 0, u), F32 ? st(j, NS - 1, u) : T(0));
            __syncthreads();
            continue;
        }

        // ================================ VJP ================================
        // start state into sP (level by level) and f0_j = A[b] pi_{j-1}
        stage(0, 1);
        if (F32 && mine)
            for (int j = 0; j < n; ++j)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (u < nc) {
                        const int64_t el = (int64_t)j * m + r * d + c0 + u;
                        const Carry<T> p = split_carry<T>(riem0 ? 0.0 : pic[el]), q = split_carry<T>(rcc[el]);
                        sPI[el] = p.hi;
                        sPI[nm + el] = p.lo;
                        sRHO[el] = q.hi;
                        sRHO[nm + el] = q.lo;
                    }
        for (int j = 0; j + 1 < n; ++j) {
            __syncthreads();
            if (j > 0 && mine) {
                T v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = u < nc && !riem0 ? (T)pic[(int64_t)(j - 1) * m + r * d + c0 + u] : T(0);
                store4(sP + r * pit + c0, v);
            }
            __syncthreads();
            if (mine) {
                T y[4];
                if (j > 0) {
                    product(sA, sP, false, y);
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) y[u] = sA[r * pit + c0 + u];
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    st(j, 0, u) = T(0);
                    if (F32) st(j, NS - 1, u) = T(0);
                    st(j, 1, u) = riem ? T(0) : y[u];
                }
            }
        }
        __syncthreads();
        forward(n - 1, true, true);

        if (mine)
            for (int j = 0; j < n; ++j)
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    st(j, 0, u) = T(0);
                    if (F32) st(j, NS - 1, u) = T(0);
                    st(j, 1, u) = T(0);
                }
        for (int li = glast; li >= g0; li = prev_of(li)) {
            const int cnt = count_of(li);
            stage(li, cnt);
            T G[4][4], dA[4][4];
#pragma unroll
            for (int l = 0; l < 4; ++l)
#pragma unroll
                for (int u = 0; u < 4; ++u) G[l][u] = dA[l][u] = T(0);
            for (int j = n - 1; j >= 0; --j) {
                if (j + 1 < n) {
                    // G_{j+1} and P_j of the group to shared memory
                    if (mine)
#pragma unroll
                        for (int l = 0; l < 4; ++l) store4(sP + l * mat + r * pit + c0, G[l]);
                    for (int x = tid; x < cnt * m; x += NT) {
                        const int l = x / m, el = x - l * m, row = el / d;
                        sQ[l * mat + row * pit + el - row * d] = tape[((int64_t)(li + l) * (n - 1) + j) * m + el];
                    }
                    __syncthreads();
                    if (mine) {
#pragma unroll
                        for (int l = 0; l < 4; ++l) {
                            if (l >= cnt) break;
                            // dA += G_{j+1} P_j^T
                            T o[4] = {T(0), T(0), T(0), T(0)};
                            const T* g = sP + l * mat + r * pit;
                            const T* q = sQ + l * mat + c0 * pit;
#pragma unroll 4
                            for (int k = 0; k < d; ++k) {
                                const T a = g[k];
#pragma unroll
                                for (int u = 0; u < 4; ++u) o[u] = fma(a, q[u * pit + k], o[u]);
                            }
#pragma unroll
                            for (int u = 0; u < 4; ++u) dA[l][u] += o[u];
                            product(sA + l * mat, sP + l * mat, true, G[l]);  // H_j = A^T G_{j+1}
                        }
                    }
                    __syncthreads();
                }
                if (mine) {
                    auto reverse = [&](auto eachc) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            T Rb = st(j, 0, u), pend = st(j, 1, u), rlo = F32 ? st(j, NS - 1, u) : T(0);
                            Carry<T> cy{T(0), T(0)};
                            if (u < nc) {
                                const int64_t el = (int64_t)j * m + r * d + c0 + u;
                                cy = F32 ? Carry<T>{sRHO[el], sRHO[nm + el]} : Carry<T>{(T)rcc[el], T(0)};
                            }
                            T v[4] = {G[0][u], G[1][u], G[2][u], G[3][u]};
                            gw.template adjoint<decltype(eachc)::value>(v, cnt, Rb, rlo, pend, true, cy);
#pragma unroll
                            for (int l = 0; l < 4; ++l) G[l][u] = u < nc ? v[l] : T(0);
                            st(j, 0, u) = Rb;
                            st(j, 1, u) = riem ? T(0) : pend;
                            if (F32) st(j, NS - 1, u) = rlo;
                        }
                    };
                    if (F32 && gw.each) reverse(std::integral_constant<bool, F32>{});
                    else reverse(std::false_type{});
                }
                if (n == 1) __syncthreads();
            }
            if (mine) {
#pragma unroll
                for (int l = 0; l < 4; ++l) {
                    if (l >= cnt) break;
                    const int lis = li + l;
                    const bool shared = lis == Kp && ch < I.C - 1;
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (u >= nc) break;
                        const int64_t at = (b + lis) * m + r * d + c0 + u;
                        const T v = dA[l][u] + G[l][u];
                        if (shared) atomic_add_out<T>(I.dA, at, v, f64);
                        else store_out<T>(I.dA, at, v, f64);
                    }
                }
            }
        }
        // this chunk's copy of W_j[b]: dA[b] += pend_1 + sum_{j<n} pend_{j+1} pi_j^T
        if (!riem) {
            T v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = mine ? st(0, 1, u) : T(0);
            for (int j = 1; j < n; ++j) {
                __syncthreads();
                if (mine) {
                    T p[4], q[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        p[u] = st(j, 1, u);
                        q[u] = u < nc ? (T)pic[(int64_t)(j - 1) * m + r * d + c0 + u] : T(0);
                    }
                    store4(sP + r * pit + c0, p);
                    store4(sQ + r * pit + c0, q);
                }
                __syncthreads();
                if (mine) {
                    const T* g = sP + r * pit;
                    const T* q = sQ + c0 * pit;
#pragma unroll 4
                    for (int k = 0; k < d; ++k) {
                        const T a = g[k];
#pragma unroll
                        for (int u = 0; u < 4; ++u) v[u] = fma(a, q[u * pit + k], v[u]);
                    }
                }
            }
            if (mine)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (u < nc) {
                        const int64_t at = b * m + r * d + c0 + u;
                        if (ch > 0) atomic_add_out<T>(I.dA, at, v[u], f64);
                        else store_out<T>(I.dA, at, v[u], f64);
                    }
        }
        __syncthreads();
    }
}

template <class T, int MODE>
cudaError_t dense_go(int d, int rule, const LaunchArgs& a, int nmax, bool prepare_only) {
    static std::mutex mu;
    static std::vector<bool> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    {
        std::lock_guard<std::mutex> lock(mu);
        if ((int)done.size() <= dev) done.resize(dev + 1, false);
        if (!done[dev]) {
            e = cudaFuncSetAttribute(k_dense<T, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDenseSmem);
            if (e != cudaSuccess) return e;
            done[dev] = true;
        }
    }
    if (prepare_only) return cudaSuccess;
    // the forward pass has no slot; the VJP's grid is the slots it was given
    const int64_t blocks = MODE == MODE_LOCAL ? a.nwork : std::min<int64_t>(a.nwork, a.grid);
    k_dense<T, MODE><<<(unsigned)std::max<int64_t>(1, blocks), dense_threads(d), dense_smem<T>(MODE, d, nmax), a.stream>>>(
        a.insts, a.work, a.nwork, static_cast<T*>(a.scratch), a.slot_elems, d, rule, a.f64io);
    return cudaGetLastError();
}

template <class T>
cudaError_t dense_T(int d, int rule, int mode, const LaunchArgs& a, int nmax, bool prepare_only) {
    return mode == MODE_LOCAL ? dense_go<T, MODE_LOCAL>(d, rule, a, nmax, prepare_only)
                              : dense_go<T, MODE_VJP>(d, rule, a, nmax, prepare_only);
}

}  // namespace
}  // namespace mgb
