// Host staging of a batch: input checks, the copy into page-locked buffers,
// and each structure's centre and impact-disk radius, in one native call
// (as per-structure numpy expressions this was 35 us a structure; 200
// structures of 1500 atoms took 7 ms).  Large batches are spread over a few
// threads.  Compiled with -ffp-contract=off: every operation rounds once, as
// numpy's and the device builder's do.
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <thread>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif
#include "../../include/ehss_b200.h"

namespace ehss {

void set_error(const char* fmt, ...);

// Row-order column sums divided by n (numpy's mean(axis=0), ehss_state.py:46), and
// max(|c - centre| + r) * (1 + 1e-9) (ehss_state.py:47; norm as
// sqrt((x*x + y*y) + z*z)); NaN when a distance is.
void enclosing_sphere(int64_t n, const double* xyz, const double* radii, double* center, double* radius) {
    double a = 0., b = 0., c = 0.;
    for (int64_t i = 0; i < n; ++i) { a += xyz[3 * i]; b += xyz[3 * i + 1]; c += xyz[3 * i + 2]; }
    center[0] = a / (double)n; center[1] = b / (double)n; center[2] = c / (double)n;
    double most = 0.;
    bool nan = false;
    for (int64_t i = 0; i < n; ++i) {
        const double x = xyz[3 * i] - center[0], y = xyz[3 * i + 1] - center[1], z = xyz[3 * i + 2] - center[2];
        const double len = std::sqrt((x * x + y * y) + z * z) + radii[i];
        nan |= len != len;
        most = len > most ? len : most;
    }
    *radius = nan ? NAN : most * 1.000000001;
}

// Copy into a page-locked buffer, past the caches: lines that several cores hold modified slow the upload that reads
// them next (40 structures of 5000 atoms staged by several threads: 130 us of upload became 170 to 300).
static void copy_out(double* dst, const double* src, int64_t n) {
#if defined(__x86_64__)
    int64_t i = 0;
    if (n > 0 && ((uintptr_t)dst & 15u)) { dst[0] = src[0]; i = 1; }
    for (; i + 2 <= n; i += 2) _mm_stream_pd(dst + i, _mm_loadu_pd(src + i));
    if (i < n) dst[i] = src[i];
    _mm_sfence();
#else
    std::memcpy(dst, src, sizeof(double) * (size_t)n);
#endif
}

// Runs f(0) .. f(count - 1), on up to `threads` threads; a thread that cannot be started is done without.
template <typename F>
static void spread(int count, int threads, F f) {
    std::atomic<int> next{0};
    auto work = [&] { for (int i; (i = next.fetch_add(1)) < count;) f(i); };
    std::thread pool[8];
    int started = 0;
    for (; started < threads - 1 && started < 8; ++started) {
        try { pool[started] = std::thread(work); } catch (...) { break; }
    }
    work();
    for (int t = 0; t < started; ++t) pool[t].join();
}

}  // namespace ehss

using namespace ehss;

extern "C" int ehss_stage_structures(int n_structures, const double* const* xyz, const double* const* radii,
                                     const int64_t* n_atoms, double* xyz_out, double* radii_out, double* centers_out,
                                     double* enclosing_out) {
    if (n_structures < 1 || !xyz || !radii || !n_atoms || !xyz_out || !radii_out || !centers_out || !enclosing_out) {
        set_error("invalid arguments");
        return EHSS_ERR_VALUE;
    }
    int64_t total = 0;
    for (int s = 0; s < n_structures; ++s) {
        if (n_atoms[s] < 1 || !xyz[s] || !radii[s]) { set_error("structure %d: no atoms", s); return EHSS_ERR_VALUE; }
        total += n_atoms[s];
    }
    // a thread is worth starting for about 40,000 atoms (0.3 ms of this work)
    const int cores = (int)std::thread::hardware_concurrency();
    const int64_t want = 1 + total / 40000;
    const int threads = (int)(want < 8 ? want : 8) < (cores > 1 ? cores : 1) ? (int)(want < 8 ? want : 8) : (cores > 1 ? cores : 1);
    std::atomic<int> bad{-1};
    spread(n_structures, threads, [&](int s) {
        const int64_t n = n_atoms[s];
        const double *c = xyz[s], *r = radii[s];
        bool ok = true;
        for (int64_t i = 0; i < 3 * n; ++i) ok &= std::isfinite(c[i]);
        for (int64_t i = 0; i < n; ++i) ok &= std::isfinite(r[i]) && r[i] > 0.;
        if (!ok) { bad = s; return; }
        enclosing_sphere(n, c, r, centers_out + 3 * s, enclosing_out + s);
    });
    if (bad >= 0) {                                          // nothing is staged unless everything is valid
        set_error("structure %d: Finite centers (N,3) and positive finite radii required.", bad.load());
        return EHSS_ERR_VALUE;
    }
    // copies in the order of the structures
    const int blocks = threads;
    spread(blocks, threads, [&](int b) {
        const int first = (int)((int64_t)n_structures * b / blocks), end = (int)((int64_t)n_structures * (b + 1) / blocks);
        int64_t at = 0;
        for (int s = 0; s < first; ++s) at += n_atoms[s];
        for (int s = first; s < end; ++s) {
            copy_out(xyz_out + 3 * at, xyz[s], 3 * n_atoms[s]);
            copy_out(radii_out + at, radii[s], n_atoms[s]);
            at += n_atoms[s];
        }
    });
    return EHSS_OK;
}
