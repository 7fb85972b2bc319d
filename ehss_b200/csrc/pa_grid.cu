// Adaptive finite-grid PA on the device.
//
// Replaces ccs_cli.adaptive_pa (src/support_exchange_transport/ccs_cli.py:142-160):
// for each of n_dirs directions drawn from Sobol(2, seed) through unit_sphere
// (inside_out_pa.py:45-49), project the atom centres on the plane normal to
// the direction (project_grid, pa_walsh_geometry.py:171-180), lay an n x n
// grid of pixel midpoints over the enclosing square and count the pixels that
// lie in the union of the atom disks -- the quantity the reference's sparse
// quadtree (block_disks / block_count, pa_sparse_blocks.py:134-166) counts
// with the exact row inequality of row_span (pa_dyadic_bitmask.py:50-61).
//
// k_grid_project, then one of the two others:
//   k_grid_project  one CTA per (direction, 1024 atoms): direction frame,
//                   projected centres (FP64, leaf order), the CTA's extent
//   k_grid_cover    one CTA per (direction, band of rows), one warp per 32
//                   rows and one lane per row: the rows' pixels as a bit mask
//                   in shared memory, counted in place
//   k_grid_scatter  one thread per atom, where a disk spans few rows
// Where directions are few, the CTAs of a cluster share a direction's atoms, each
// with a mask of its own, and count the union of their masks.
// Counts are integers, so a direction's count equals the reference's count
// whenever the projected coordinates are the same.
//
// What bounds k_grid_cover: instruction issue and the latency of each warp's
// own chain (masks, staged disks and lists live in shared memory, the
// projected centres in L2).  What keeps both down:
//   * A row's two ends come from FP32 arithmetic in pixel units relative to
//     the atom's own pixel, with an error bound; only an end that lies within
//     its bound of a pixel centre is decided by the reference's FP64
//     predicate, so the pixel set is the reference's.
//   * A lane owns its row, so its words are updated without atomics, and warps
//     meet only where the next atoms are staged.
//   * The pixels of a protein are covered many times over (145 times for
//     20,000 atoms on a 1024 grid).  Atoms are visited in a strided order
//     (leaf order is spatial, so a stride samples the whole structure), each
//     warp keeps the columns that are full in all of its rows, and an atom
//     whose columns are full is dropped before its rows are formed.
//   * An exterior scene's buried atoms (behind n_active in leaf order) are not
//     visited: their whole surface lies inside other spheres with a margin
//     far above FP64 rounding, so every pixel of theirs is another atom's.
// Measured (64 directions, device time of both kernels under ncu): 34 us for 650
// atoms on a 512 grid and 179 us for 20,000 on a 1024 grid; one thread per
// (atom, direction) with FP64 row ends and global atomics took 121 and 1005 us.
#include <cooperative_groups.h>
#include <algorithm>
#include <cstdio>
#include "ehss_internal.cuh"

namespace ehss {

struct Sobol2Params { uint32_t sv[2][30]; uint32_t shift[2]; };

__device__ __forceinline__ double dot3(const double* a, const double* b) {
    return dadd(dadd(dmul(a[0], b[0]), dmul(a[1], b[1])), dmul(a[2], b[2]));
}

// Atoms of one k_grid_project CTA; 256 threads.
constexpr int kProjectAtoms = 1024;

// Atoms that a direction's pixels need: every atom, or the exposed ones of an
// exterior scene (all of them where the caller asks for the projections).
__device__ __forceinline__ int grid_atoms(const SceneHeader* H, int m_max, bool all) {
    const int m = H->exterior && !all ? H->n_active : H->n_atoms;
    return min(m, m_max);
}

__global__ void __launch_bounds__(256) k_grid_project(const void* scene, Sobol2Params sob, int m_max, int chunks,
                                                      double* extents, double2* xy, unsigned long long* counts,
                                                      double* xy_out) {
    const int dir = blockIdx.x / chunks, chunk = blockIdx.x % chunks;
    SceneView S = scene_view(scene);
    const int m = grid_atoms(S.h, m_max, xy_out != nullptr);
    __shared__ double frame[6];
    __shared__ double partial[8];
    if (threadIdx.x == 0) {
        if (chunk == 0) counts[dir] = 0;
        // unit_sphere of Sobol(2) point `dir` (the reference's direction list order)
        uint32_t g = (uint32_t)dir ^ ((uint32_t)dir >> 1);
        uint32_t q0 = sob.shift[0], q1 = sob.shift[1];
        while (g) {
            int k = __ffs(g) - 1;
            g &= g - 1;
            q0 ^= sob.sv[0][k];
            q1 ^= sob.sv[1][k];
        }
        double u0 = q0 * 0x1p-30, u1 = q1 * 0x1p-30;
        double z = dsub(1.0, dmul(2.0, u0));
        double phi = dmul(2.0 * 3.141592653589793, u1);
        double rho = dsqrt(dmax0(dsub(1.0, dmul(z, z))));
        double sp, cp;
        sincos(phi, &sp, &cp);
        double d[3] = {dmul(rho, cp), dmul(rho, sp), z};
        // project_grid: normalise, frame axis e_z unless |d_z| >= 0.9 (then e_x)
        double nd = dsqrt(dot3(d, d));
        for (int c = 0; c < 3; ++c) d[c] = ddiv(d[c], nd);
        double a[3] = {0., 0., 1.};
        if (!(fabs(d[2]) < .9)) { a[0] = 1.; a[2] = 0.; }
        double u[3] = {dsub(dmul(a[1], d[2]), dmul(a[2], d[1])), dsub(dmul(a[2], d[0]), dmul(a[0], d[2])),
                       dsub(dmul(a[0], d[1]), dmul(a[1], d[0]))};
        double nu = dsqrt(dot3(u, u));
        for (int c = 0; c < 3; ++c) u[c] = ddiv(u[c], nu);
        double v[3] = {dsub(dmul(d[1], u[2]), dmul(d[2], u[1])), dsub(dmul(d[2], u[0]), dmul(d[0], u[2])),
                       dsub(dmul(d[0], u[1]), dmul(d[1], u[0]))};
        for (int c = 0; c < 3; ++c) { frame[c] = u[c]; frame[3 + c] = v[c]; }
    }
    __syncthreads();
    const double u[3] = {frame[0], frame[1], frame[2]}, v[3] = {frame[3], frame[4], frame[5]};
    double ext = 0.;
    for (int j = chunk * kProjectAtoms + threadIdx.x; j < min(m, (chunk + 1) * kProjectAtoms); j += blockDim.x) {
        const double4 a = S.atoms64[j];
        double c[3] = {dsub(a.x, S.h->center[0]), dsub(a.y, S.h->center[1]), dsub(a.z, S.h->center[2])};
        const double x = dot3(c, u), y = dot3(c, v);
        xy[(int64_t)dir * m_max + j] = make_double2(x, y);
        if (xy_out) {                                   // the caller's copy is in input order
            double* o = xy_out + 2 * ((int64_t)dir * m_max + S.ids[j]);
            o[0] = x;
            o[1] = y;
        }
        ext = fmax(ext, fmax(dadd(fabs(x), a.w), dadd(fabs(y), a.w)));
    }
    for (int off = 16; off > 0; off >>= 1) ext = fmax(ext, __shfl_xor_sync(0xffffffffu, ext, off));
    if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = ext;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) ext = fmax(ext, partial[w]);
        extents[blockIdx.x] = ext;
    }
}

// row_span (pa_dyadic_bitmask.py:50-61) in FP64 without contraction.
__device__ __noinline__ void row_span(double cx, double cy, double r, double lower, double spacing, int y, int n,
                                         int& lo_out, int& hi_out) {
    lo_out = hi_out = 0;
    double dy = dsub(dadd(lower, dmul((double)y + .5, spacing)), cy);
    double rem = dsub(dmul(r, r), dmul(dy, dy));
    if (rem < 0) return;
    double half = dsqrt(rem);
    double a = ceil(dsub(ddiv(dsub(dsub(cx, half), lower), spacing), .5));
    double b = floor(dsub(ddiv(dsub(dadd(cx, half), lower), spacing), .5));
    long long lo = (long long)a, hi = (long long)b + 1;
    lo = lo < n ? lo : n; lo = lo > 0 ? lo : 0;
    hi = hi < n ? hi : n; hi = hi > 0 ? hi : 0;
    for (int it = 0; it < 4 && lo > 0; ++it) {
        double t = dsub(dadd(lower, dmul((double)lo - .5, spacing)), cx);
        if (dmul(t, t) <= rem) --lo; else break;
    }
    for (int it = 0; it < 4 && lo < hi; ++it) {
        double t = dsub(dadd(lower, dmul((double)lo + .5, spacing)), cx);
        if (dmul(t, t) > rem) ++lo; else break;
    }
    for (int it = 0; it < 4 && hi < n; ++it) {
        double t = dsub(dadd(lower, dmul((double)hi + .5, spacing)), cx);
        if (dmul(t, t) <= rem) ++hi; else break;
    }
    for (int it = 0; it < 4 && hi > lo; ++it) {
        double t = dsub(dadd(lower, dmul((double)hi - .5, spacing)), cx);
        if (dmul(t, t) > rem) --hi; else break;
    }
    lo_out = (int)lo;
    hi_out = (int)hi;
}

// One atom's disk in pixel units of its direction's grid: pixel k's centre lies
// at lower + (k + .5) spacing, so the disk's centre sits at x0 + fx (x0 the
// pixel below it, 0 <= fx < 1) and row y covers the pixels k with
// |k - (x0 + fx)| <= sqrt(r^2 - (y - y0 - fy)^2).
//
// Error bounds of the FP32 row ends (u = 2^-24, r the radius in pixels).
// fx, fy and r2 are rounded once from FP64, y - y0 is an exact integer below
// r + 2 in magnitude and dy = (y - y0) - fy is off by at most u (r + 1), so
// rem = r2 - dy^2 is off by at most u (4 r^2 + 3 r + 1); tol is u (8 r^2 + 6 r + 4).
// rem >= 4 tol bounds the error of sqrt(rem) by tol / sqrt(rem); rsqrtf's
// 2 ulp, the product and fx -/+ half add less than 2^-21 (half + 1), of which
// the bound takes twice.  FP64's own roundings are below 1e-9 pixel.
__device__ __forceinline__ float pixel_tol(float r) { return 0x1p-23f * (4.f * r * r + 3.f * r + 2.f); }

constexpr int kStage = 1024;            // atoms staged at a time
constexpr int kStageLoads = 2;
constexpr int kDraw = 4;

// Visiting order of the leaf order's runs of 8 atoms: the runs are cut into
// 2^bits strata of `width`, taken in bit-reversed order, one run of each, then
// the next of each, so that every stretch samples the whole structure.
// Positions are 0 .. width 2^bits - 1; up to a quarter name no run.
__device__ __forceinline__ int spread_run(int i, int bits, int width) {
    const int stratum = bits ? (int)(__brev((unsigned)i) >> (32 - bits)) : 0;
    return stratum * width + (i >> bits);
}

// row_span's predicate: is pixel k's centre within the row's half width?
__device__ __forceinline__ bool pixel_in(double cx, double rem, double lower, double spacing, int k) {
    const double t = dsub(dadd(lower, dmul((double)k + .5, spacing)), cx);
    return dmul(t, t) <= rem;
}

// Integers below 2^22 in magnitude as floats and back, and rounding to them, by
// adding 1.5 2^23 (the conversion unit works at a quarter of the rate).
constexpr float kRound = 12582912.f;

// Ends of row y of a staged disk: the pixel centre nearest to each (kl, kr), the
// end's distance from it (fl, fr), its error bound e.  Straight-line code, so
// that several atoms' chains overlap.
struct RowEnds {
    int kl, kr;
    float fl, fr, e, rem, tol;
};

__device__ __forceinline__ RowEnds row_ends(float4 d, int2 o, int y) {
    RowEnds R;
    R.tol = pixel_tol(d.w);
    const float dy = (__int_as_float(__float_as_int(kRound) + y - o.y) - kRound) - d.y;
    R.rem = fmaf(-dy, dy, d.z);
    float q;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(fmaxf(R.rem, R.tol)));
    const float half = R.rem * q;
    R.e = fmaf(R.tol, q, fmaf(half, 0x1p-20f, 0x1p-20f));
    const float xl = d.x - half, xr = d.x + half, nl = xl + kRound, nr = xr + kRound;
    R.kl = o.x + __float_as_int(nl) - __float_as_int(kRound);
    R.kr = o.x + __float_as_int(nr) - __float_as_int(kRound);
    R.fl = xl - (nl - kRound);
    R.fr = xr - (nr - kRound);
    return R;
}

// Pixels [lo, hi) of a row whose ends FP32 does not decide.
__device__ __noinline__ int2 exact_ends(double2 c, double r, float4 d, int2 o, int y, int n, double lower, double spacing) {
    const RowEnds R = row_ends(d, o, y);
    int lo, hi;
    if (R.rem < 4.f * R.tol || R.e > .25f) {
        row_span(c.x, c.y, r, lower, spacing, y, n, lo, hi);
    } else {
        // a true end within e of pixel k's centre: on one side of it or the other
        const double dy64 = dsub(dadd(lower, dmul((double)y + .5, spacing)), c.y);
        const double rem64 = dsub(dmul(r, r), dmul(dy64, dy64));
        lo = R.kl + (R.fl > 0.f);
        hi = R.kr + (R.fr >= 0.f);
        if (fabsf(R.fl) <= R.e) lo = pixel_in(c.x, rem64, lower, spacing, R.kl) ? R.kl : R.kl + 1;
        if (fabsf(R.fr) <= R.e) hi = pixel_in(c.x, rem64, lower, spacing, R.kr) ? R.kr + 1 : R.kr;
    }
    return make_int2(lo, hi);
}

// Columns a .. b that a disk reaches in rows row0 .. row0 + 31: those of its
// widest row there, one pixel wider on each side.
__device__ __forceinline__ void disk_columns(float4 d, int2 o, int row0, int n, int& a, int& b) {
    const float dy = fmaxf(0.f, fmaxf((float)(row0 - o.y - 1), (float)(o.y - row0 - 31)));
    float half;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(half) : "f"(fmaxf(0.f, (d.w + 1.f) * (d.w + 1.f) - dy * dy)));
    const int h = (int)half + 1;
    a = max(0, o.x - h);
    b = min(n - 1, o.x + h + 1);
}

// Whether columns a .. b are full (bits of full).
__device__ __forceinline__ bool columns_full(const unsigned* full, int a, int b) {
    for (int w = a >> 5; w <= b >> 5; ++w) {
        unsigned need = ~0u;
        if (w == a >> 5) need = ~0u << (a & 31);
        if (w == b >> 5) need &= ~0u >> (31 - (b & 31));
        if ((full[w] & need) != need) return false;
    }
    return true;
}

// Adds the pixels of a CTA's mask, or of the union of the masks of a cluster of
// `parts` CTAs that share their rows, to a direction's count.
__device__ __forceinline__ void add_covered(unsigned* masks, int size, int parts, int part, unsigned long long* counts) {
    int count = 0;
    if (parts == 1) {
        __syncthreads();
        for (int w = threadIdx.x; w < size; w += blockDim.x) count += __popc(masks[w]);
    } else {
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        cluster.sync();
        for (int w = part * blockDim.x + threadIdx.x; w < size; w += parts * blockDim.x) {
            unsigned v = 0u;
            for (int q = 0; q < parts; ++q) v |= cluster.map_shared_rank(masks, q)[w];
            count += __popc(v);
        }
        cluster.sync();                                      // no CTA ends while another reads its mask
    }
    count = __reduce_add_sync(0xffffffffu, count);
    if ((threadIdx.x & 31) == 0 && count) atomicAdd(counts, (unsigned long long)count);
}

__global__ void __launch_bounds__(512) k_grid_cover(const void* scene, int m_max, int all_atoms, int n, int bands, int words,
                                                    int pitch, int parts, int chunks, const double* extents, const double2* xy_all,
                                                    unsigned long long* counts, double* spacing_out) {
    extern __shared__ __align__(16) unsigned char cover_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    float4* const disk = reinterpret_cast<float4*>(cover_smem);                 // [kStage] fx, fy, r^2, r
    int2* const cell = reinterpret_cast<int2*>(disk + kStage);                  // [kStage] x0, y0
    unsigned short* const lists = reinterpret_cast<unsigned short*>(cell + kStage);   // [nwarps][kStage]
    short2* const span = reinterpret_cast<short2*>(lists + nwarps * kStage);    // [kStage] first and last row
    int* const atom = reinterpret_cast<int*>(span + kStage);                    // [kStage] leaf-order index
    int* const n_staged = atom + kStage;
    unsigned* const fulls = reinterpret_cast<unsigned*>(n_staged + 1);          // [nwarps][words]
    unsigned* const masks = fulls + nwarps * words;                             // [32 nwarps][pitch]
    const int part = blockIdx.x % parts, band = blockIdx.x / parts % bands, dir = blockIdx.x / (parts * bands);
    const SceneView S = scene_view(scene);
    const int m = grid_atoms(S.h, m_max, all_atoms != 0);
    const double2* xy = xy_all + (int64_t)dir * m_max;
    double extent = 0.;
    for (int k = 0; k < chunks; ++k) extent = fmax(extent, extents[(int64_t)dir * chunks + k]);
    extent = dmul(extent, 1.0000000001);
    const double lower = -extent, spacing = ddiv(dmul(2.0, extent), (double)n), inv = 1.0 / spacing;
    if (spacing_out && band == 0 && part == 0 && threadIdx.x == 0) spacing_out[dir] = spacing;
    const int band0 = band * 32 * nwarps, row0 = band0 + 32 * warp, y = row0 + lane;
    unsigned* const row = masks + threadIdx.x * pitch;
    unsigned* const full = fulls + warp * words;             // bit c: column c is covered in all of the warp's rows
    unsigned short* const list = lists + warp * kStage;
    for (int w = 0; w < pitch; ++w) row[w] = 0u;             // the pad too: it is counted
    for (int w = lane; w < words; w += 32) full[w] = 0u;
    // Rounds take runs of 8 atoms spread over the leaf order: a first round of kStage atoms, then twice as many as
    // before while the band's full columns drop enough of them that the rest fit the stage.
    const int runs = (m + 7) >> 3, bits = max(0, 29 - __clz(runs)), width = (runs + (1 << bits) - 1) >> bits;
    const int places = (width << bits) / parts + (part < (width << bits) % parts);
    int drawn = 0, next = 8;                                 // atoms drawn; the full columns are formed at 8 and every quarter more
    int size = kStage / 8;
    for (int begin = 0; begin < places;) {
        if (threadIdx.x == 0) *n_staged = 0;
        __syncthreads();                                     // the masks are zero, the full columns current
        // stage the atoms that the band's rows still need, kStageLoads of a thread's at a time so that their loads and
        // FP64 chains overlap
        const int end = min(places, begin + size), cnt = 8 * (end - begin);
        for (int k0 = threadIdx.x; k0 < ((cnt + 31) & ~31); k0 += kStageLoads * blockDim.x) {
            double2 c[kStageLoads];
            double r[kStageLoads];
            int j[kStageLoads];
#pragma unroll
            for (int i = 0; i < kStageLoads; ++i) {
                const int k = k0 + i * (int)blockDim.x;
                j[i] = k < cnt ? 8 * spread_run((begin + (k >> 3)) * parts + part, bits, width) + (k & 7) : m;
                c[i] = xy[min(j[i], m - 1)];
                r[i] = S.atoms64[min(j[i], m - 1)].w;
            }
#pragma unroll
            for (int i = 0; i < kStageLoads; ++i) {
                const double cx = (c[i].x - lower) * inv - .5, cy = (c[i].y - lower) * inv - .5, rp = r[i] * inv;
                const double flx = floor(cx), fly = floor(cy);
                const float4 d = make_float4((float)(cx - flx), (float)(cy - fly), (float)(rp * rp), (float)rp);
                const int2 o = make_int2((int)flx, (int)fly);
                const int ya = o.y - (int)d.w - 1, yb = o.y + (int)d.w + 2;
                bool open = false;
                if (j[i] < m) {
                    const int ga = max(0, (ya - band0) >> 5), gb = min(nwarps - 1, (yb - band0) >> 5);
                    open = ga <= gb && begin == 0;
                    for (int g = ga; g <= gb && !open; ++g) {
                        int a, b;
                        disk_columns(d, o, band0 + 32 * g, n, a, b);
                        open = !columns_full(fulls + g * words, a, b);
                    }
                }
                const unsigned b = __ballot_sync(0xffffffffu, open);
                if (!b) continue;
                int at = 0;
                if (lane == 0) at = atomicAdd(n_staged, __popc(b));
                at = __shfl_sync(0xffffffffu, at, 0) + __popc(b & ((1u << lane) - 1u));
                if (open && at < kStage) {
                    disk[at] = d;
                    cell[at] = o;
                    span[at] = make_short2((short)ya, (short)yb);
                    atom[at] = j[i];
                }
            }
        }
        __syncthreads();
        // list the atoms that meet this warp's rows, then take them 32 spread over the list at a time
        const int found = *n_staged, staged = min(found, kStage);
        int L = 0;
#pragma unroll 4
        for (int k0 = 0; k0 < staged; k0 += 32) {
            const int k = k0 + lane;
            const short2 v = span[min(k, staged - 1)];
            const bool in = k < staged && v.x < row0 + 32 && v.y >= row0;
            const unsigned b = __ballot_sync(0xffffffffu, in);
            if (in) list[L + __popc(b & ((1u << lane) - 1u))] = (unsigned short)k;
            L += __popc(b);
        }
        __syncwarp();
        const int per = (L + 31) >> 5;
        for (int s = 0; s < per; ++s) {
            const int t = lane * per + s;
            bool draw = t < L;
            int k = 0;
            if (draw) {
                k = list[t];
                int a, b;
                disk_columns(disk[k], cell[k], row0, n, a, b);
                draw = !columns_full(full, a, b);
            }
            unsigned todo = __ballot_sync(0xffffffffu, draw);
            drawn += __popc(todo);
            while (todo) {
                // kDraw atoms at a time: their chains to the row ends overlap, then the words are updated in turn
                int lo[kDraw], hi[kDraw], which[kDraw];
                unsigned open_ends = 0;
#pragma unroll
                for (int i = 0; i < kDraw; ++i) {
                    const bool any = todo != 0;
                    const int at = __shfl_sync(0xffffffffu, k, any ? __ffs(todo) - 1 : 0);
                    todo &= todo - 1;
                    which[i] = at;
                    const RowEnds R = row_ends(disk[at], cell[at], y);
                    const bool some = any && R.rem >= -R.tol && y < n;
                    lo[i] = R.kl + (R.fl > 0.f);
                    hi[i] = some ? R.kr + (R.fr >= 0.f) : -1;
                    if (some && (fminf(fabsf(R.fl), fabsf(R.fr)) <= R.e || R.rem < 4.f * R.tol)) open_ends |= 1u << i;
                }
                if (open_ends) {
#pragma unroll
                    for (int i = 0; i < kDraw; ++i) {
                        if (!((open_ends >> i) & 1u)) continue;
                        const int j = atom[which[i]];
                        const int2 v = exact_ends(xy[j], S.atoms64[j].w, disk[which[i]], cell[which[i]], y, n, lower, spacing);
                        lo[i] = v.x;
                        hi[i] = v.y;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < kDraw; ++i) {
                    // four words without a branch, which is every word of most rows
                    const int a = max(lo[i], 0), b = min(hi[i], n) - 1, wa = a >> 5, wb = a <= b ? b >> 5 : -1;
                    const unsigned first = ~0u << (a & 31), last = ~0u >> (31 - (b & 31));
                    unsigned v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = wa + q <= wb ? row[wa + q] : 0u;
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (wa + q <= wb) row[wa + q] = v[q] | ((q == 0 ? first : ~0u) & (wa + q == wb ? last : ~0u));
                    for (int w = wa + 4; w <= wb; ++w) row[w] = w == wb ? row[w] | last : ~0u;
                }
            }
            if (drawn >= next) {
                next = drawn + max(8, drawn >> 2);
                __syncwarp();
#pragma unroll 8
                for (int w = 0; w < words; ++w) {
                    const unsigned all = __reduce_and_sync(0xffffffffu, y < n ? row[w] : ~0u);
                    if (lane == (w & 31)) full[w] = all;
                }
                __syncwarp();
            }
        }
        __syncthreads();
        if (found > kStage) {
            size = max(kStage / 8, size / 2);               // some were left out: this round again, smaller (drawing is idempotent)
        } else {
            begin = end;
            if (2 * found <= kStage) size *= 2;
        }
    }
    add_covered(masks, 32 * nwarps * pitch, parts, part, counts + dir);
}

// The same count with a thread for each atom: the atom's rows in turn, their
// words set by shared-memory atomics, and one direction's atoms shared among
// the `parts` CTAs of a cluster, which read one another's masks to count.
__global__ void __launch_bounds__(512) k_grid_scatter(const void* scene, int m_max, int all_atoms, int n, int bands, int rows,
                                                      int pitch, int parts, int chunks, const double* extents,
                                                      const double2* xy_all, unsigned long long* counts, double* spacing_out) {
    extern __shared__ __align__(16) unsigned char cover_smem[];
    unsigned* const masks = reinterpret_cast<unsigned*>(cover_smem);            // [rows][pitch]
    const int part = blockIdx.x % parts, band = blockIdx.x / parts % bands, dir = blockIdx.x / (parts * bands);
    const SceneView S = scene_view(scene);
    const int m = grid_atoms(S.h, m_max, all_atoms != 0), band0 = band * rows, size = rows * pitch;
    const double2* xy = xy_all + (int64_t)dir * m_max;
    for (int w = threadIdx.x; w < size; w += blockDim.x) masks[w] = 0u;
    double extent = 0.;
    for (int k = 0; k < chunks; ++k) extent = fmax(extent, extents[(int64_t)dir * chunks + k]);
    extent = dmul(extent, 1.0000000001);
    const double lower = -extent, spacing = ddiv(dmul(2.0, extent), (double)n), inv = 1.0 / spacing;
    if (spacing_out && band == 0 && part == 0 && threadIdx.x == 0) spacing_out[dir] = spacing;
    __syncthreads();
    const int runs = (m + 7) >> 3, bits = max(0, 29 - __clz(runs)), width = (runs + (1 << bits) - 1) >> bits;
    const int places = 8 * (width << bits);
    for (int k = part * blockDim.x + threadIdx.x; k < places; k += parts * blockDim.x) {
        const int j = 8 * spread_run(k >> 3, bits, width) + (k & 7);
        if (j >= m) continue;
        const double2 c = xy[j];
        const double r = S.atoms64[j].w;
        const double cx = (c.x - lower) * inv - .5, cy = (c.y - lower) * inv - .5, rp = r * inv;
        const double flx = floor(cx), fly = floor(cy);
        const float4 d = make_float4((float)(cx - flx), (float)(cy - fly), (float)(rp * rp), (float)rp);
        const int2 o = make_int2((int)flx, (int)fly);
        const int ya = max(o.y - (int)d.w - 1, band0), yb = min(o.y + (int)d.w + 2, min(band0 + rows, n) - 1);
        for (int y = ya; y <= yb; ++y) {
            const RowEnds R = row_ends(d, o, y);
            if (R.rem < -R.tol) continue;
            int2 v = make_int2(R.kl + (R.fl > 0.f), R.kr + (R.fr >= 0.f));
            if (fminf(fabsf(R.fl), fabsf(R.fr)) <= R.e || R.rem < 4.f * R.tol) v = exact_ends(c, r, d, o, y, n, lower, spacing);
            const int a = max(v.x, 0), b = min(v.y, n) - 1;
            if (a > b) continue;
            unsigned* const row = masks + (y - band0) * pitch;
            for (int w = a >> 5; w <= b >> 5; ++w) {
                unsigned need = ~0u;
                if (w == a >> 5) need = ~0u << (a & 31);
                if (w == b >> 5) need &= ~0u >> (31 - (b & 31));
                if (need & ~row[w]) atomicOr(row + w, need);     // most pixels are covered already
            }
        }
    }
    add_covered(masks, size, parts, part, counts + dir);
}

// Most shared memory that a CTA of k_grid_cover or k_grid_scatter is given.
constexpr int kGridSmem = 160 * 1024;

static int64_t project_chunks(int64_t n_atoms) { return (n_atoms + kProjectAtoms - 1) / kProjectAtoms; }

uint64_t grid_workspace_bytes(int64_t n_atoms, int n_dirs, int n) {
    (void)n;
    return align256(8ull * n_dirs * project_chunks(n_atoms)) + align256(16ull * n_atoms * n_dirs) + 256;
}

int launch_grid_pa(const void* scene, int64_t n_atoms, int n_dirs, uint64_t seed, int n, unsigned long long* counts,
                   double* spacing_out, double* xy_out, void* workspace, uint64_t ws_bytes, cudaStream_t stream) {
    uint64_t need = grid_workspace_bytes(n_atoms, n_dirs, n);
    if (ws_bytes < need) {
        set_error("adaptive PA workspace holds %llu bytes, %llu required", (unsigned long long)ws_bytes,
                  (unsigned long long)need);
        return EHSS_ERR_CAPACITY;
    }
    char* p = (char*)(((uintptr_t)workspace + 255u) & ~(uintptr_t)255u);
    const int chunks = (int)project_chunks(n_atoms);
    double* extents = (double*)p; p += align256(8ull * n_dirs * chunks);
    double2* xy = (double2*)p;
    Sobol2Params sob;
    uint32_t sv[2 * 30], shift[2];
    sobol_scramble(2, seed, sv, shift);
    for (int j = 0; j < 2; ++j) {
        for (int k = 0; k < 30; ++k) sob.sv[j][k] = sv[j * 30 + k];
        sob.shift[j] = shift[j];
    }
    const int words = (n + 31) / 32, pitch = words | 1;                  // odd pitch: the rows' words spread over all banks
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    cudaLaunchConfig_t cfg = {};
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto launch = [&](auto kernel, int bands, int parts, int threads, unsigned smem, auto... geometry) {
        if (smem > 48u * 1024u) {
            // a limit, not an allocation, held per function and device: the same one on every call, so that calls on
            // other threads never lower it ahead of this launch
            const int rc = cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGridSmem),
                                       "grid shared memory");
            if (rc) return rc;
        }
        cfg.gridDim = dim3((unsigned)(bands * parts * n_dirs));
        cfg.blockDim = dim3((unsigned)threads);
        cfg.dynamicSmemBytes = smem;
        attr[0].val.clusterDim.x = (unsigned)parts;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        return cuda_status(cudaLaunchKernelEx(&cfg, kernel, scene, (int)n_atoms, (int)(xy_out != nullptr), n, bands, geometry...,
                                              parts, chunks, (const double*)extents, (const double2*)xy, counts, spacing_out),
                           "adaptive PA launch");
    };
    k_grid_project<<<(unsigned)chunks * n_dirs, 256, 0, stream>>>(scene, sob, (int)n_atoms, chunks, extents, xy, counts, xy_out);
    int parts = 1;
    // A disk of a compact structure spans about 2 n / atoms^(1/3) rows. Where that is fewer than a warp has lanes
    // (n < 16 atoms^(1/3)), most lanes of k_grid_cover have no row and its warps, one for 32 rows, are few. Device times,
    // cover / scatter, 1 and 64 directions: 2000 atoms on a 64 grid 206 / 20 and 218 / 24 us, 6000 on 256: 66 / 42 and
    // 124 / 81; on the line's other side 20,000 on 512: 91 / 114 and 239 / 335, 650 on 256: 27 / 36 and 36 / 42.
    if ((long long)n * n * n < 4096ll * n_atoms) {
        int rows = n;
        while (rows > 1 && 4ll * rows * pitch > 136ll * 1024) rows /= 2;      // at most kGridSmem: a row is 1 KB
        const int bands = n / rows;
        // CTAs that share a direction's atoms: up to two an SM, 128 atoms each (20,000 atoms, one direction, 256 grid:
        // 527 us with one, 69 with eight)
        while (parts < 8 && n_atoms > 128ll * parts && (long long)n_dirs * bands * parts <= sm_count()) parts *= 2;
        const int threads = (int)std::min<int64_t>(512, (n_atoms + 32 * parts - 1) / (32 * parts) * 32);
        return launch(k_grid_scatter, bands, parts, threads, 4u * rows * pitch, rows, pitch);
    }
    // Warps of a CTA (32 rows each): every CTA stages every atom of its part of the direction, so as many as leave a CTA
    // for five SMs (20,000 atoms on a 1024 grid, 64 directions: 179 us with 16 warps, 240 with fewer), down to two; fewer
    // where the masks (33 KB a warp on an 8192 grid) would not fit. What SMs are left then share a direction's atoms,
    // 256 at least to a CTA (16 directions: 228 -> 97 us; one: 279 -> 73).
    const int groups = (n + 31) / 32;
    auto bytes = [&](int warps) {
        return (unsigned)(kStage * (sizeof(float4) + sizeof(int2) + sizeof(short2) + 4) + 4 + warps * (kStage * 2 + 4 * words + 128 * pitch));
    };
    int warps = groups < 16 ? groups : 16;
    while (warps > 2 && (bytes(warps) > (unsigned)kGridSmem || 5ll * n_dirs * (groups / warps) < sm_count())) warps /= 2;
    const int bands = groups / warps;
    while (parts < 8 && n_atoms > 256ll * parts && 2ll * n_dirs * bands * parts <= sm_count()) parts *= 2;
    return launch(k_grid_cover, bands, parts, 32 * warps, bytes(warps), words, pitch);
}

}  // namespace ehss
