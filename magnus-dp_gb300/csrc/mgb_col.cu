// The small-matrix chunk kernel (mgb_col.cuh) of the plain form, and the
// family's launch geometry.
#include "mgb_col.cuh"

namespace mgb {

cudaError_t launch_col_f32(int D, int rule, int mode, const LaunchArgs& a, int nmax, bool prepare_only);

namespace {
// f(ColGeo) for the form, dimension and teams per chunk
template <class T, int CNT, class F>
auto col_geo(int D, F&& f) {
    switch (D) {
        case 3: return f(ColGeo<T, 3, CNT>{});
        case 4: return f(ColGeo<T, 4, CNT>{});
        case 5: return f(ColGeo<T, 5, CNT>{});
        case 6: return f(ColGeo<T, 6, CNT>{});
        case 7: return f(ColGeo<T, 7, CNT>{});
        default: return f(ColGeo<T, 8, CNT>{});
    }
}
template <class F>
auto col_geo_t(bool plain, int D, int lpc, F&& f) {
    if (!plain) return col_geo<float, 64>(D, f);
    return lpc == 16 ? col_geo<double, 128>(D, f) : col_geo<double, 64>(D, f);
}
}  // namespace

bool col_ok(bool plain, int D, int nmax) {
    if (D < 3 || D > 8) return false;
    return col_geo_t(plain, D, 16, [&](auto g) { return g.smem(MODE_VJP, nmax, 2) <= kColSmem; });
}

// Teams (runs) per chunk: doubled while the call has fewer than 128 (FP64: 64)
// threads per SM, every run keeps two groups, and a chunk's chain gets shorter by it:
// a run's groups at 4 (n - 1) d^2 + 18 n d operations each (a clock apart four
// in FP32, sixteen in FP64), then the FP64 composition of the runs one after
// the other, n (n - 1) / 2 (d^2 + d) operations each (16 clocks apart, and as
// long again where FP32 runs wait for it).
int col_lanes(bool plain, int D, int nmax, int64_t nwork, int64_t kmax, int sms) {
    const int64_t groups = (kmax + 3) / 4, want = (int64_t)sms * (plain ? 64 : 128);
    // A chunk's runs share one CTA, so the geometry that a count selects must hold
    // that count (d = 3, 4: 32 runs would select 64 threads, 20 or 16 teams).
    auto fit = [&](int runs) { return runs <= col_geo_t(plain, D, runs, [](auto g) { return g.TC; }); };
    const double group = (4.0 * (nmax - 1) * D * D + 18.0 * nmax * D) * (plain ? 16 : 4);
    const double join = 0.5 * nmax * (nmax - 1) * (D * D + D) * (plain ? 16 : 32);
    // The line: FP32, d = 8, 64 trajectories, n = 4, forward / VJP at 128, 256, 512:
    // 0.21 / 1.09, 0.36 / 1.51, 0.56 / 2.26 ms; FP64 at 64, 128, 256: 3.13 / 8.24,
    // 3.51 / 11.4, 3.03 / 11.9 ms.
    int lpc = 1;
    while (fit(2 * lpc) && nwork * lpc * D < want && groups >= 4 * lpc &&
           groups / (2.0 * lpc) * group > lpc * join)
        lpc *= 2;
    return lpc;
}

// Scratch elements for a VJP over nwork chunks: the CTAs an SM holds by shared
// memory, six at most (registers), or all teams of a smaller call.
int64_t col_scratch(bool plain, int D, int nmax, int64_t nwork, int64_t kmax, int lpc, int sms) {
    return col_geo_t(plain, D, lpc, [&](auto g) {
        const int64_t cpb = g.TC / lpc, per_sm = std::max<int64_t>(1, std::min<int64_t>(6, 222 * 1024 / (int64_t)(g.smem(MODE_VJP, nmax, lpc) + 1024))),
                      blocks = std::min<int64_t>((nwork + cpb - 1) / cpb, sms * per_sm);
        return blocks * g.TC * g.slot(nmax, kmax, lpc);
    });
}
int64_t col_scratch_min(bool plain, int D, int nmax, int64_t kmax, int lpc) {
    return col_geo_t(plain, D, lpc, [&](auto g) { return (int64_t)g.TC * g.slot(nmax, kmax, lpc); });
}

cudaError_t launch_col(bool plain, int D, int rule, int mode, const LaunchArgs& a, int nmax, bool prepare_only) {
    return plain ? col_d<double>(D, rule, mode, a, nmax, prepare_only) : launch_col_f32(D, rule, mode, a, nmax, prepare_only);
}

}  // namespace mgb
