// EHSS and PA kernels: nearest-entry query over the device LBVH, specular
// bounce loop, any-hit PA, and the fused Sobol -> trace -> reduction blocks.
//
// Reference behaviour restated (paths relative to the reference project):
//   nearest_scalar        src/support_exchange_transport/ehss_cpu.py:43-63
//   _trace_loop           ehss_cpu.py:66-100, src/native/ehss_cpu.cpp:54-78
//   entry_scalar/reflect  ehss_cpu.py:12-40 (see ehss_internal.cuh)
//   tree_blocked / _one   pa_spatial.py:114-142 with sphere_hit inside_out_pa.py:93-101
//   readout               ehss_state.py:84-103, ccs_cli.py:209-219
//
// Query design.  The reference walks a median-split tree in pre-order and
// keeps the lexicographic (distance, atom id) minimum of the FP64 entry
// distances.  Here the 4-wide LBVH is walked near-child-first with a
// per-thread stack; node boxes are FP32, rounded outward and expanded by eps_box, so a
// box is culled only when it provably holds no entry at or before the
// current bound U.  Two sphere-test precisions share the walk:
//   EXACT (EHSS_PREC_FP64): every reached sphere is tested in FP64, with the
//     reference's formula unless an FP64 discriminant shows a certain miss;
//     U is the running best distance rounded up.
//   FILTER (EHSS_PREC_FP32): spheres are tested in FP32 with a discriminant
//     formed from the ray's point nearest the structure's centre (seven
//     operations a sphere, sphere_disc below) and error bounds
//     (Ep on projections, Edisc on the discriminant).  Certain misses are dropped;
//     certain hits give an interval [t - Et, t + Et] and lower U to t + Et;
//     every sphere whose lower bound is <= U (certain or near-tangent) is
//     kept in a 2-entry candidate list, re-tested in FP64 at the end with the
//     reference formula and the (distance, id) rule.  The reached candidates
//     always contain the FP64 winner, so outcomes equal EXACT's; a full list
//     re-runs the query in EXACT mode.
// Ray origins farther than 3 S from the structure centre (never produced by
// the impact-disk source) use an FP64 all-atom search instead.
#include <algorithm>
#include <cstdio>
#include "ehss_internal.cuh"

namespace ehss {

constexpr float kU32 = 5.9604645e-08f;   // 2^-24
// Candidate slots per query.  A slot whose lower bound exceeds the current U is
// reused, so two slots overflow only when three spheres are within the error
// band of each other (275 of 125 M queries on the mixed 256-globule batch).  Each
// slot is two registers of the fused kernel, which runs at its 64-register
// bound: before the shorter sphere test 2 slots traced that batch in 27.9 ms, 3 in 28.8, 4 in 29.7, while 1
// slot sent every grazing query to the FP64 search (1e5 fallbacks, 29.0 ms).
constexpr int kCand = 2;
constexpr int kSmemBins = 16;

struct LocalStats {
    uint32_t box, sphere, queries, grazing, fallback, fp64, errors;
    __device__ LocalStats() : box(0), sphere(0), queries(0), grazing(0), fallback(0), fp64(0), errors(0) {}
};

// FP32 copy of a ray in the scene frame (centre at the origin): the line's point
// o nearest the centre, d / sqrt 2, the inverse direction, and the two
// thresholds of the sphere test.  With x(tau) = o + tau d the ray starts at
// tau0, and t = tau - tau0.
//   thr  = (|o|^2 - Edisc) / 2
//   bmin = (tau0 - Ep) / sqrt 2
struct RayF {
    float ox, oy, oz, dx, dy, dz, ix, iy, iz, thr, bmin;
};

constexpr float kSqrt2 = 1.41421356f, kHalfSqrt2 = 0.707106781f;

// Inverse direction component for the box tests, from the fast quotient
// (within 2 ulp for these arguments, whose magnitude lies in [1e-20, 1]).  A
// relative error e in inv moves a slab crossing along the ray by |t| e; with
// t below 6 S (origins within 3 S, boxes within S) that is under 1.5e-6 S
// even with the slab's own roundings, well inside the 2^-14 S (6.1e-5 S) by
// which every node box is widened, and the sign, which picks the near plane,
// is exact.  The start's distance along the line enters a crossing with d inv in
// place of 1 (3u |tau0|) and less Ep: another 3.5e-6 S.
__device__ __forceinline__ float safe_rcp(float x) {
    float a = fabsf(x) < 1e-20f ? copysignf(1e-20f, x) : x;
    return __fdividef(1.0f, a);
}

// Error bounds of the FP32 sphere test, from the scene's scale S alone
// (|c| + r <= S for every atom; |o| <= S (1 + 1e-5), since a line farther out
// meets none; u = 2^-24).  In exact arithmetic, with o.d = 0 and |d| = 1,
//     disc = r^2 - |c - o|^2 + (c.d)^2 = 2 (D - |o|^2 / 2),
//     D = (c.d / sqrt 2)^2 + c.o + k,   k = (r^2 - |c|^2) / 2 per atom.
// 2 D is off by at most: k rounded once, u S^2; c and o rounded, 2u S |o| each;
// b = c.d / sqrt 2 from rounded c and d (twice) and three roundings, 6u S, so
// 12u S^2 on its square; the three sums of c.o + k, 3u (S^2 + 2 S |o|); the last
// fma, 2u S (S + |o|); the threshold's own rounding, 2u |o|^2: together at most
// 18u S^2 + 12u S |o| + 2u |o|^2 <= 33u S^2.  Edisc = 48u S^2.
// t-units: b sqrt 2 - tau0 is off by 9u S from b, and |tau0|, |t| <= 4 S round
// by u each at most three times: 21u S.  Ep = 48u S.
constexpr float kEdisc = 48.0f * kU32, kEp = 48.0f * kU32;

__device__ __forceinline__ float ray_edisc(const SceneHeader* H) { const float S = __ldg(&H->scale_f); return kEdisc * S * S; }
__device__ __forceinline__ float ray_ep(const SceneHeader* H) { return kEp * __ldg(&H->scale_f); }

constexpr int kRayFar = 0, kRayOk = 1, kRayNotUnit = 2;

// |d|^2 off by at most this counts as unit.  Other directions take the walk from
// kShortest to kLongest of |d|^2, where the entry formula's margins, which are in
// units of |d|, stay far below the filter's.
constexpr double kUnitError = 1e-11, kShortest = 0x1p-40, kLongest = 0x1p40;

// FP32 copy of an FP64 ray.  kRayFar: the origin is beyond 3 S from the centre
// (or not finite), where node boxes are not widened enough.
// Directions that are not unit (UNIT: there are none, the caller's are unit to
// rounding): FILTER classifies along the normalised ray, whose spheres and order
// of entries are the same, and FP64 decides with the caller's direction.  For
// EXACT the boxes hold as they are, with o the ray's own origin and distances in
// units of |d|, so none is taken off them (Ep in such units exceeds the boxes'
// widening from |d| = 20 on); the sphere test's identity does not hold.
// kRayNotUnit: such a ray, or one outside the range above.
template <bool EXACT, bool UNIT>
__device__ __forceinline__ int setup_ray(const SceneHeader* H, const double* o, const double* d, RayF& r) {
    const double x = o[0] - H->center[0], y = o[1] - H->center[1], z = o[2] - H->center[2];
    const float S = H->scale_f;
    const float fx = (float)x, fy = (float)y, fz = (float)z;
    if (!(sqrtf(fmaf(fx, fx, fmaf(fy, fy, fz * fz))) <= 3.0f * S)) return kRayFar;
    const double aa = fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2]));
    bool unit = fabs(aa - 1.0) <= kUnitError;
    double d0 = d[0], d1 = d[1], d2 = d[2];
    if (!EXACT && !UNIT && !unit && aa >= kShortest && aa <= kLongest) {
        const double inv = 1.0 / sqrt(aa);
        d0 *= inv; d1 *= inv; d2 *= inv;
        unit = true;
    }
    const double tau0 = unit ? fma(x, d0, fma(y, d1, z * d2)) : 0.0;
    r.ox = (float)fma(-tau0, d0, x);
    r.oy = (float)fma(-tau0, d1, y);
    r.oz = (float)fma(-tau0, d2, z);
    const float dx = (float)d0, dy = (float)d1, dz = (float)d2;
    r.ix = safe_rcp(dx); r.iy = safe_rcp(dy); r.iz = safe_rcp(dz);
    r.dx = dx * kHalfSqrt2; r.dy = dy * kHalfSqrt2; r.dz = dz * kHalfSqrt2;
    const float q = fmaf(r.ox, r.ox, fmaf(r.oy, r.oy, r.oz * r.oz));
    // a line beyond S passes every sphere by 1e-5 S: all tests miss
    r.thr = q > 1.00002f * S * S ? CUDART_INF_F : 0.5f * (q - kEdisc * S * S);
    r.bmin = UNIT || unit ? ((float)tau0 - kEp * S) * kHalfSqrt2 : 0.0f;
    return unit ? kRayOk : kRayNotUnit;
}

// D (above) of atom a = (c, k) and b = c.d / sqrt 2.
__device__ __forceinline__ float sphere_disc(const RayF& r, const float4& a, float& b) {
    b = fmaf(a.x, r.dx, fmaf(a.y, r.dy, a.z * r.dz));
    return fmaf(b, b, fmaf(a.x, r.ox, fmaf(a.y, r.oy, fmaf(a.z, r.oz, a.w))));
}

// sqrt(disc) of a certain hit (computed disc >= 2 Edisc) and the error bound Et
// of its entry and exit distances bt -/+ sqrt(disc), from one reciprocal square
// root: s = disc * y and Edisc / s = Edisc * y.  rsqrtf is within 2 ulp of 1/sqrt(disc) (the CUDA
// math library's stated bound; at most 2.09 u measured over every float in
// [2^-14, 2^8)), so s is within 5.01 u of sqrt(disc) and Edisc * y within
// 5.01 u of Edisc / sqrt(disc).  With the roundings of disc from D (2u), of s
// and of bt -/+ s the distance error stays below Ep + Edisc / sqrt(disc) +
// 8.1 u (|bt| + s), which Et covers with a factor-2 margin on its first two
// terms.
__device__ __forceinline__ float certain_sqrt(float bt, float disc, float Ep, float Edisc, float& Et) {
    const float y = rsqrtf(disc);
    const float s = disc * y;
    Et = 2.0f * (Ep + Edisc * y) + 12.0f * kU32 * (fabsf(bt) + s);
    return s;
}

__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Slab test of one child box against [0, U]; returns entry distance or +inf.
// The planes come as near (n*) and far (f*) per axis: with inv >= 0 the low
// plane is met first, and fma(lo, inv, -oi) <= fma(hi, inv, -oi) because
// rounding is monotone, so the near plane's distance is the slab minimum the
// textbook test forms with fminf, bit for bit.  An unused slot holds the box
// lo = +inf, hi = -inf, whose near distance is +inf on every axis, so it
// misses without a check of its reference.  oi = o * inv + tau0 per axis
// (distances from the ray's start), formed once per node visit (held per lane
// it would cost three registers of the fused kernel).
template <bool WIDE>
__device__ __forceinline__ float box_enter(const RayF& r, float oix, float oiy, float oiz, float nx, float fx, float ny,
                                           float fy, float nz, float fz, float U, float wx, float wy, float wz) {
    float tnx = fmaf(nx, r.ix, -oix), tfx = fmaf(fx, r.ix, -oix);
    float tny = fmaf(ny, r.iy, -oiy), tfy = fmaf(fy, r.iy, -oiy);
    float tnz = fmaf(nz, r.iz, -oiz), tfz = fmaf(fz, r.iz, -oiz);
    if (WIDE) { tnx -= wx; tfx += wx; tny -= wy; tfy += wy; tnz -= wz; tfz += wz; }
    float tmin = max3f(tnx, tny, fmaxf(tnz, 0.0f));
    float tmax = min3f(tfx, tfy, fminf(tfz, U));
    return tmin <= tmax ? tmin : CUDART_INF_F;
}

// One 4-wide node: entry distances of the children that the ray meets within
// [0, U], sorted ascending (misses and empty slots last, at +inf).
struct Hits4 {
    int ref[4];
    float t[4];
    int n;
};

__device__ __forceinline__ void cswap(Hits4& h, int a, int b) {
    bool s = h.t[b] < h.t[a];
    float ta = s ? h.t[b] : h.t[a], tb = s ? h.t[a] : h.t[b];
    int ra = s ? h.ref[b] : h.ref[a], rb = s ? h.ref[a] : h.ref[b];
    h.t[a] = ta; h.t[b] = tb; h.ref[a] = ra; h.ref[b] = rb;
}

// WIDE: the planes of axis x (y, z) are moved wx (wy, wz) along the ray apart.
template <bool WIDE = false>
__device__ __forceinline__ Hits4 visit4(const float4* nodes, int node, const RayF& r, float U, float wx = 0.f, float wy = 0.f,
                                        float wz = 0.f) {
    const float4* nd = nodes + 8 * (int64_t)node;
    // near and far plane rows by the direction's sign per axis (the node stores lo, hi)
    const int sx = __float_as_uint(r.ix) >> 31, sy = __float_as_uint(r.iy) >> 31, sz = __float_as_uint(r.iz) >> 31;
    float4 nx = __ldg(nd + sx), fx = __ldg(nd + (1 - sx)), ny = __ldg(nd + (2 + sy)), fy = __ldg(nd + (3 - sy));
    float4 nz = __ldg(nd + (4 + sz)), fz = __ldg(nd + (5 - sz)), rf = __ldg(nd + 6);
    Hits4 h;
    h.ref[0] = __float_as_int(rf.x); h.ref[1] = __float_as_int(rf.y);
    h.ref[2] = __float_as_int(rf.z); h.ref[3] = __float_as_int(rf.w);
    // distances from the ray's start (less Ep, which the boxes' widening absorbs)
    const float tau0 = r.bmin * kSqrt2;
    const float oix = fmaf(r.ox, r.ix, tau0), oiy = fmaf(r.oy, r.iy, tau0), oiz = fmaf(r.oz, r.iz, tau0);
    h.t[0] = box_enter<WIDE>(r, oix, oiy, oiz, nx.x, fx.x, ny.x, fy.x, nz.x, fz.x, U, wx, wy, wz);
    h.t[1] = box_enter<WIDE>(r, oix, oiy, oiz, nx.y, fx.y, ny.y, fy.y, nz.y, fz.y, U, wx, wy, wz);
    h.t[2] = box_enter<WIDE>(r, oix, oiy, oiz, nx.z, fx.z, ny.z, fy.z, nz.z, fz.z, U, wx, wy, wz);
    h.t[3] = box_enter<WIDE>(r, oix, oiy, oiz, nx.w, fx.w, ny.w, fy.w, nz.w, fz.w, U, wx, wy, wz);
    cswap(h, 0, 1); cswap(h, 2, 3); cswap(h, 0, 2); cswap(h, 1, 3); cswap(h, 1, 2);
    h.n = (h.t[0] != CUDART_INF_F) + (h.t[1] != CUDART_INF_F) + (h.t[2] != CUDART_INF_F) + (h.t[3] != CUDART_INF_F);
    return h;
}

// Reference rule of nearest_scalar (ehss_cpu.py:60): strictly nearer, or
// equally near with a smaller input atom id.
__device__ __forceinline__ bool better(double dist, int id, double best, int best_id) {
    return dist < best || (dist == best && isfinite(dist) && (best_id < 0 || id < best_id));
}

// FP64 all-atom nearest search (origins far from the structure).
__device__ __forceinline__ int nearest_flat(const SceneView& S, const double* o, const double* d, int last_rank, double& best_out,
                            LocalStats& st) {
    int n = S.h->n_atoms;
    double best = CUDART_INF;
    int best_rank = -1, best_id = -1;
    for (int k = 0; k < n; ++k) {
        if (k == last_rank) continue;
        double4 a = S.atoms64[k];
        double t = entry64(o[0], o[1], o[2], d[0], d[1], d[2], a.x, a.y, a.z, a.w);
        ++st.sphere; ++st.fp64;
        int id = S.ids[k];
        if (better(t, id, best, best_id)) { best = t; best_rank = k; best_id = id; }
    }
    best_out = best;
    return best_rank;
}

// Nearest entry: returns the leaf-order rank of the collider (or -1) and its
// FP64 entry distance, identical to the reference's choice.  Parked rays
// (rest_of_path, EXACT) and the cap extension use it.
template <bool EXACT, bool UNIT = false>
__device__ __forceinline__ int nearest(const SceneView& S, const double* o, const double* d, int last_rank,
                                    double& best_out, LocalStats& st) {
    ++st.queries;
    RayF r;
    const int kind = setup_ray<EXACT, UNIT>(S.h, o, d, r);
    if (kind == kRayFar) return nearest_flat(S, o, d, last_rank, best_out, st);
    if (!EXACT && kind == kRayNotUnit) { --st.queries; return nearest<true, UNIT>(S, o, d, last_rank, best_out, st); }
    const float Edisc = ray_edisc(S.h), Ep = ray_ep(S.h);
    float U = CUDART_INF_F;
    double best = CUDART_INF;
    int best_rank = -1, best_id = -1;
    int cand_rank[kCand];
    float cand_lo[kCand];
#pragma unroll
    for (int e = 0; e < kCand; ++e) { cand_rank[e] = -1; cand_lo[e] = CUDART_INF_F; }
    bool overflow = false, grazing = false;

    int stack_ref[kStackDepth];
    float stack_t[kStackDepth];
    int sp = 0;
    int cur = 0;
    const int n_nodes = S.h->n_nodes, n_atoms = S.h->n_atoms;
    // each node and leaf is entered at most once per query; more steps mean a malformed tree
    for (int steps = 0;; ++steps) {
        if (cur >= n_nodes || steps > 2 * n_nodes + 2) { ++st.errors; break; }
        if (cur >= 0) {
            Hits4 h = visit4(S.nodes, cur, r, U);
            st.box += 4;
            if (h.n > 0) {
                for (int k = h.n - 1; k >= 1; --k) {
                    if (sp < kStackDepth) { stack_ref[sp] = h.ref[k]; stack_t[sp] = h.t[k]; ++sp; }
                    else { ++st.errors; }
                }
                cur = h.ref[0];
                continue;
            }
        } else {
            int code = ~cur;
            int first = code >> kLeafBits, cnt = (code & (kMaxLeaf - 1)) + 1;
            if (first + cnt > n_atoms) { ++st.errors; cnt = 0; }
            for (int k = first; k < first + cnt; ++k) {
                if (k == last_rank) continue;
                ++st.sphere;
                if (EXACT) {
                    double4 a = S.atoms64[k];
                    double t = entry64(o[0], o[1], o[2], d[0], d[1], d[2], a.x, a.y, a.z, a.w);
                    ++st.fp64;
                    int id = __ldg(S.ids + k);
                    if (better(t, id, best, best_id)) {
                        best = t; best_rank = k; best_id = id;
                        U = __double2float_ru(best);
                    }
                } else {
                    const float4 a = __ldg(S.atoms + k);
                    float b;
                    const float D = sphere_disc(r, a, b);
                    if (D < r.thr || b < r.bmin) continue;               // certain miss
                    const float disc = fmaf(2.0f, D - r.thr, -Edisc), bt = fmaf(b - r.bmin, kSqrt2, -Ep);
                    float lo;
                    bool certain = false;
                    if (disc >= 2.0f * Edisc) {
                        float Et;
                        const float t = bt - certain_sqrt(bt, disc, Ep, Edisc, Et);
                        if (t < -2.0f * Et) continue;                    // origin inside: no entry ahead
                        if (t > Et) {
                            certain = true;
                            lo = t - Et;
                            float up = t + Et;
                            if (up < U) U = up;
                        }
                    }
                    if (!certain) {
                        lo = fmaxf(0.0f, (bt - Ep - sqrtf(fmaxf(disc, 0.0f) + Edisc)) * (1.0f - 8.0f * kU32));
                        grazing = true;
                    }
                    if (lo <= U) {
                        bool placed = false;
#pragma unroll
                        for (int e = 0; e < kCand; ++e) {
                            bool free_slot = cand_rank[e] < 0 || cand_lo[e] > U;
                            if (!placed && free_slot) { cand_rank[e] = k; cand_lo[e] = lo; placed = true; }
                        }
                        if (!placed) overflow = true;
                    }
                }
            }
        }
        // pop the nearest pending subtree that can still hold an entry <= U
        bool found = false;
        while (sp > 0) {
            --sp;
            if (stack_t[sp] <= U) { cur = stack_ref[sp]; found = true; break; }
        }
        if (!found) break;
    }
    if (!EXACT) {
        if (grazing) ++st.grazing;
        if (overflow) {
            ++st.fallback;
            --st.queries;
            return nearest<true, UNIT>(S, o, d, last_rank, best_out, st);
        }
#pragma unroll
        for (int e = 0; e < kCand; ++e) {
            if (cand_rank[e] >= 0 && cand_lo[e] <= U) {
                int k = cand_rank[e];
                double4 a = S.atoms64[k];
                double t = entry64(o[0], o[1], o[2], d[0], d[1], d[2], a.x, a.y, a.z, a.w);
                ++st.fp64;
                int id = __ldg(S.ids + k);
                if (better(t, id, best, best_id)) { best = t; best_rank = k; best_id = id; }
            }
        }
    }
    best_out = best;
    return best_rank;
}

// The same out of line, for kernels that are not bound by their registers.
template <bool EXACT>
__device__ __noinline__ int nearest_call(const SceneView& S, const double* o, const double* d, int last_rank,
                                         double& best_out, LocalStats& st) {
    return nearest<EXACT>(S, o, d, last_rank, best_out, st);
}

// Direction off unit length, for the any-hit query: sphere_hit takes |d| = 1, so
// with e = |d|^2 - 1 and b the distance along the line of its point nearest the
// centre, its discriminant is the normalised ray's plus e b^2, |b| <= |o| + S.
// Certain misses and hits keep that much more distance (more, less), and boxes
// are moved sqrt(more) apart, at most 8 S, where every box holds the origin: the
// ray meets nothing farther than that from a sphere.
struct OffUnit {
    float more, less, wx, wy, wz;
};

// Any-hit walk (pa_spatial._one with sphere_hit): true when the ray meets any
// sphere other than owner_rank.
template <bool UNIT>
__device__ __forceinline__ bool anyhit_walk(const SceneView& S, const RayF& r, const double* o, const double* d, int owner_rank,
                                            const OffUnit& f, LocalStats& st) {
    const float Edisc = ray_edisc(S.h), Ep = ray_ep(S.h);
    const float miss = UNIT ? r.thr : r.thr - 0.5f * f.more, hit = UNIT ? 2.0f * Edisc : fmaf(2.0f, Edisc, f.less);
    int stack_ref[kStackDepth];
    int sp = 0;
    int cur = 0;
    const float U = CUDART_INF_F;
    const int n_nodes = S.h->n_nodes, n_atoms = S.h->n_atoms;
    for (int steps = 0;; ++steps) {
        if (cur >= n_nodes || steps > 2 * n_nodes + 2) { ++st.errors; break; }
        if (cur >= 0) {
            Hits4 h = visit4<!UNIT>(S.nodes, cur, r, U, f.wx, f.wy, f.wz);
            st.box += 4;
            if (h.n > 0) {
                for (int k = h.n - 1; k >= 1; --k) {
                    if (sp < kStackDepth) stack_ref[sp++] = h.ref[k]; else ++st.errors;
                }
                cur = h.ref[0];
                continue;
            }
        } else {
            int code = ~cur;
            int first = code >> kLeafBits, cnt = (code & (kMaxLeaf - 1)) + 1;
            if (first + cnt > n_atoms) { ++st.errors; cnt = 0; }
            for (int k = first; k < first + cnt; ++k) {
                if (k == owner_rank) continue;
                ++st.sphere;
                const float4 a = __ldg(S.atoms + k);
                float b;
                const float D = sphere_disc(r, a, b);
                if (D < miss) continue;
                const float disc = fmaf(2.0f, D - r.thr, -Edisc), bt = fmaf(b - r.bmin, kSqrt2, -Ep);
                if (disc >= hit) {
                    float Et;
                    // far root: the reference's -b + sqrt(disc) with b = x.d = -(v.d)
                    const float exitp = bt + certain_sqrt(bt, disc, Ep, Edisc, Et);
                    if (exitp > Et) return true;
                    if (exitp < -2.0f * Et) continue;
                } else if (bt + sqrtf(fmaxf(disc, 0.0f) + Edisc) < -2.0f * Ep) {
                    continue;
                }
                double4 a64 = S.atoms64[k];
                ++st.fp64;
                if (sphere_hit64(o[0], o[1], o[2], d[0], d[1], d[2], a64.x, a64.y, a64.z, a64.w)) return true;
            }
        }
        if (sp == 0) break;
        cur = stack_ref[--sp];
    }
    return false;
}

// Any-hit PA query of a ray.  UNIT: the caller's directions are unit to rounding.
template <bool UNIT>
__device__ __noinline__ bool anyhit(const SceneView& S, const double* o, const double* d, int owner_rank,
                                    LocalStats& st) {
    ++st.queries;
    RayF r;
    if (setup_ray<false, UNIT>(S.h, o, d, r) == kRayOk) {
        OffUnit f = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (UNIT) return anyhit_walk<true>(S, r, o, d, owner_rank, f, st);
        const double e = fma(d[0], d[0], fma(d[1], d[1], d[2] * d[2])) - 1.0;
        if (fabs(e) > kUnitError) {
            const float scale = S.h->scale_f;
            const double x = o[0] - S.h->center[0], y = o[1] - S.h->center[1], z = o[2] - S.h->center[2];
            const float reach = sqrtf((float)fma(x, x, fma(y, y, z * z))) + scale, change = 1.001f * (float)fabs(e) * reach * reach;
            // lines beyond S meet such spheres too: the bound of the FP32 test for |o| up to 3 S, 72u S^2, takes 24u more
            const float error = 32.0f * kU32 * scale * scale;
            r.thr = 0.5f * (fmaf(r.ox, r.ox, fmaf(r.oy, r.oy, r.oz * r.oz)) - kEdisc * scale * scale);
            f.more = e > 0.0 ? change + error : error;
            f.less = e > 0.0 ? error : change + error;
            const float wide = fminf(1.001f * sqrtf(f.more), 8.0f * scale);
            f.wx = wide * fabsf(r.ix); f.wy = wide * fabsf(r.iy); f.wz = wide * fabsf(r.iz);
        }
        return anyhit_walk<false>(S, r, o, d, owner_rank, f, st);
    }
    const int n = S.h->n_atoms;
    for (int k = 0; k < n; ++k) {
        if (k == owner_rank) continue;
        const double4 a = S.atoms64[k];
        ++st.sphere; ++st.fp64;
        if (sphere_hit64(o[0], o[1], o[2], d[0], d[1], d[2], a.x, a.y, a.z, a.w)) return true;
    }
    return false;
}

__device__ __forceinline__ void flush_stats(const LocalStats& st, uint64_t* stats) {
    if (!stats) return;
    unsigned v[7] = {st.box, st.sphere, st.queries, st.grazing, st.fallback, st.fp64, st.errors};
    const int slot[7] = {EHSS_STAT_BOX_TESTS, EHSS_STAT_SPHERE_TESTS, EHSS_STAT_QUERIES, EHSS_STAT_GRAZING,
                         EHSS_STAT_FALLBACK, EHSS_STAT_FP64_TESTS, EHSS_STAT_ERRORS};
    unsigned lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        // 64-bit warp sum (per-thread counts can exceed 2^32 / 32 on long runs)
        unsigned long long x = v[i];
        for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
        if (lane == 0 && x) atomicAdd((unsigned long long*)&stats[slot[i]], x);
    }
}

// --------------------------------------------------------------------------
// Explicit-ray kernels (EHSS: k_rays, after the Walker it shares with k_blocks)
// --------------------------------------------------------------------------
// Rays [base, base + k) of a caller's [n, 3] array into this lane's a[3] (lane
// q < k gets ray base + q): the array is read with consecutive lanes on
// consecutive doubles, so that a page-locked host array crosses PCIe in whole
// 128-byte reads.  buf: 96 doubles of shared memory of this warp.
__device__ __forceinline__ void load_rays(const double* src, int64_t base, int k, int q, double* buf, double* a) {
    const unsigned lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const int w = lane + 32 * t;
        if (w < 3 * k) buf[w] = src[3 * base + w];
    }
    __syncwarp();
    if (q < k) {
#pragma unroll
        for (int c = 0; c < 3; ++c) a[c] = buf[3 * q + c];
    }
}

// One thread per ray.  origins and directions may lie in page-locked host
// memory; the kernel then runs at the rate at which they cross PCIe.
__global__ void __launch_bounds__(128) k_pa_rays(const void* scene, int64_t n, const double* P, const double* D,
                                                 const int64_t* owners, uint8_t* blocked, uint64_t* stats) {
    __shared__ double buf[4][96];
    SceneView S = scene_view(scene);
    LocalStats st;
    const unsigned lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    // exterior scenes hold only the atoms reachable from outside the union: not for arbitrary rays
    bool ok = S.h->magic == kSceneMagic && S.h->status == 0 && S.h->exterior == 0;
    for (int64_t base = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; base < n; base += stride) {
        const int k = (int)min((int64_t)32, n - base);
        double o[3], d[3];
        load_rays(P, base, k, lane, buf[threadIdx.x >> 5], o);
        load_rays(D, base, k, lane, buf[threadIdx.x >> 5], d);
        const int64_t i = base + lane;
        if (i >= n) continue;
        int64_t owner = owners ? owners[i] : -1;
        if (!ok || owner < -1 || owner >= S.h->n_atoms) { ++st.errors; blocked[i] = 0; continue; }
        blocked[i] = anyhit<false>(S, o, d, owner >= 0 ? S.rank[owner] : -1, st);
    }
    __syncwarp();
    flush_stats(st, stats);
}

__global__ void k_sobol_points(int dim, SobolParams p, int64_t first, int64_t n, uint32_t* q) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t idx = (uint32_t)(first + i);
    uint32_t g = idx ^ (idx >> 1);
    for (int j = 0; j < dim; ++j) {
        uint32_t v = p.shift[j];
        uint32_t gg = g;
        while (gg) {
            int k = __ffs(gg) - 1;
            gg &= gg - 1;
            v ^= p.sv[j * 30 + k];
        }
        q[i * dim + j] = v;
    }
}

__global__ void k_source_rays(const void* scene, Sobol4Params p, int64_t first, int64_t n, double* O, double* Dd) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    SceneView S = scene_view(scene);
    uint4 q = sobol4(p.sv, p.shift, (uint32_t)(first + i));
    Ray64 ray = impact_ray(q, S.h->center, S.h->radius);
    for (int c = 0; c < 3; ++c) { O[3 * i + c] = ray.o[c]; Dd[3 * i + c] = ray.d[c]; }
}

// --------------------------------------------------------------------------
// Fused blocks (persistent): Sobol -> impact disk -> EHSS / PA -> reduction
//
// One warp takes one chunk (chunk_rays consecutive positions of one block's
// coherent Sobol enumeration) at a time.  Lanes are refilled with the chunk's
// next rays, kNewRayBatch or more at a time.  Each warp alternates two phases:
//   traverse  while-while walk for every lane whose query is open: inner
//             nodes until each lane holds a leaf (a lane holding one walks on
//             to its next), then one leaf per lane, all lanes together;
//             repeated until at least `resolve_batch` lanes have finished
//             their query or wait for a new ray, or none is left traversing;
//   resolve   for all finished lanes together: FP64 candidate re-test,
//             escape / cap / reflection, and new rays once enough lanes
//             wait for one.
// Batching the FP64 work keeps most lanes of the warp busy in both phases.
// The FP64 ray state (position, direction, incoming direction) waits in
// shared memory while the lane traverses in FP32.
// --------------------------------------------------------------------------
// Per-warp accumulators of the chunk in shared memory (updated once per ray
// or per query, so registers stay free for the traversal).
struct WarpAcc {
    unsigned count[kSmemBins];
    unsigned long long ledger[kSmemBins];
    unsigned long long angle_fx;
    unsigned hits, unresolved, escaped, pa;
    unsigned queries, grazing, fallback, fp64, errors, pad;
    unsigned long long box, sphere;
    unsigned long long hits_fx, unres_fx, pa_fx;   // weighted sums of ray blocks
    uint4 q0;
};

struct LaneRay {
    double o[3], d[3], din[3];
};

// The fused kernel's dynamic shared memory: per-warp accumulators, per-lane
// FP64 ray state, then the lanes' traversal-stack columns (and, for ray
// blocks, the lanes' ray weights).
extern __shared__ __align__(16) unsigned char smem_raw[];

// Byte offset of the stack columns.  Recomputed from blockDim wherever a
// stack entry is addressed, so no lane keeps a pointer to its column in
// registers (the fused kernel runs at its 64-register bound: holding the
// pointer and the column stride cost 24 bytes of spills per thread and 1.8 %
// of trace time on the mixed 256-globule batch).
__device__ __forceinline__ unsigned stack_off() {
    return (unsigned)(sizeof(WarpAcc) * (blockDim.x >> 5) + sizeof(LaneRay) * blockDim.x);
}

__device__ __forceinline__ unsigned long long warp_sum64(unsigned long long x) {
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    return x;
}

// Point at position p of a block's coherent enumeration.
__device__ __forceinline__ uint4 block_point(const uint4* basis, uint4 base, uint32_t p) {
    uint4 q = base;
    while (p) {
        int e = __ffs(p) - 1;
        p &= p - 1;
        uint4 v = __ldg(basis + e);
        q.x ^= v.x; q.y ^= v.y; q.z ^= v.z; q.w ^= v.w;
    }
    return q;
}

constexpr int kIdle = 0, kTraverse = 1, kDone = 2, kNeedRay = 3, kParked = 4;
// Lanes whose ray has finished wait for a new one until this many of a warp
// do (16 of 32: the 256-globule batch traces in 23.9 ms against 24.6 with a
// new ray at once, 24.2 with 8 and 24.2 with 24).
constexpr int kNewRayBatch = 16;
constexpr int kSentinel = INT32_MAX - 1;   // stack exhausted
constexpr int kNoLeaf = INT32_MAX;

// Traversal stack: the top kSmemStack entries of each lane live in shared
// memory (entry i of lane t at smem_stack[i * blockDim + t], conflict-free);
// deeper entries, rare for an LBVH walked near-child first, go to a
// per-lane local array.
constexpr int kSmemStackMax = 32;

// UNIT: every ray's direction is unit to rounding (disk rays).
template <bool EXACT, bool COUNT, bool UNIT>
struct Walker {
    RayF r;
    float U;
    int cur, leaf, sp, steps;
    int cand_rank[kCand];
    float cand_lo[kCand];
    bool overflow, grazing, error;
    double best;
    int best_rank, best_id;
    unsigned box, sphere;
    // shared-memory stack entry i of this lane
    __device__ __forceinline__ int2* slot(int i) const {
        return reinterpret_cast<int2*>(smem_raw + stack_off()) + i * blockDim.x + threadIdx.x;
    }
    int deep_ref[kStackDepth];
    float deep_t[kStackDepth];

    __device__ __forceinline__ void push(int ref, float t, int sdepth) {
        if (sp < sdepth) *slot(sp) = make_int2(ref, __float_as_int(t));
        else if (sp < kStackDepth) { deep_ref[sp - sdepth] = ref; deep_t[sp - sdepth] = t; }
        else { error = true; return; }
        ++sp;
    }

    __device__ __forceinline__ void reset() {
        U = CUDART_INF_F;
        cur = 0; leaf = kNoLeaf; sp = 0; steps = 0;
#pragma unroll
        for (int e = 0; e < kCand; ++e) { cand_rank[e] = -1; cand_lo[e] = CUDART_INF_F; }
        overflow = grazing = error = false;
        if (EXACT) { best = CUDART_INF; best_rank = -1; best_id = -1; }
    }
    __device__ __forceinline__ int pop(int sdepth) {
        while (sp > 0) {
            --sp;
            int ref;
            float t;
            if (sp < sdepth) { int2 e = *slot(sp); ref = e.x; t = __int_as_float(e.y); }
            else { ref = deep_ref[sp - sdepth]; t = deep_t[sp - sdepth]; }
            if (t <= U) return ref;
        }
        return kSentinel;
    }
    __device__ __forceinline__ int visit(const float4* nodes, int node, int sdepth) {
        Hits4 h = visit4(nodes, node, r, U);
        if (COUNT) box += 4;
        // the distances are sorted with misses at +inf
        if (h.t[0] == CUDART_INF_F) return pop(sdepth);
        if (h.t[3] != CUDART_INF_F) push(h.ref[3], h.t[3], sdepth);
        if (h.t[2] != CUDART_INF_F) push(h.ref[2], h.t[2], sdepth);
        if (h.t[1] != CUDART_INF_F) push(h.ref[1], h.t[1], sdepth);
        return h.ref[0];
    }
    // One step of a lane: inner nodes until it holds a leaf (the first leaf reached is
    // held while the lane walks on), then that leaf's tests; the lane's next leaf joins the
    // next step.  The query is finished when cur == kSentinel and leaf == kNoLeaf.
    __device__ __forceinline__ void advance(const SceneView& S, int sdepth, int last_rank, const LaneRay& L) {
        while (cur >= 0 && cur != kSentinel) {
            const int n_nodes = __ldg(&S.h->n_nodes);
            if (cur >= n_nodes || ++steps > 2 * n_nodes + 2) { error = true; cur = kSentinel; break; }
            cur = visit(S.nodes, cur, sdepth);
            if (cur < 0 && leaf == kNoLeaf) {
                leaf = cur;
                cur = pop(sdepth);
            }
            if (!__any_sync(__activemask(), leaf == kNoLeaf)) break;
        }
        if (leaf != kNoLeaf) {
            leaf_tests(S, leaf, last_rank, L);
            next_leaf(sdepth);
        }
    }
    __device__ __forceinline__ void next_leaf(int sdepth) {
        leaf = kNoLeaf;
        if (cur < 0) {
            leaf = cur;
            cur = pop(sdepth);
        }
    }
    __device__ __forceinline__ bool finished() const { return cur == kSentinel && leaf == kNoLeaf; }
    __device__ __forceinline__ void add_candidate(int k, float lo) {
        if (lo > U) return;
        bool placed = false;
#pragma unroll
        for (int e = 0; e < kCand; ++e) {
            bool free_slot = cand_rank[e] < 0 || cand_lo[e] > U;
            if (!placed && free_slot) { cand_rank[e] = k; cand_lo[e] = lo; placed = true; }
        }
        if (!placed) overflow = true;
    }
    __device__ __forceinline__ void leaf_tests(const SceneView& S, int ref, int last_rank, const LaneRay& L) {
        int code = ~ref;
        int first = code >> kLeafBits, cnt = (code & (kMaxLeaf - 1)) + 1;
        if (first + cnt > S.h->n_atoms) { error = true; return; }
        if (COUNT) sphere += cnt - ((unsigned)(last_rank - first) < (unsigned)cnt ? 1 : 0);
        // EXACT: the FP64 reject takes |d| = 1 and is off (infinite bounds) for other directions
        const double slack = EXACT ? (!UNIT && r.thr == CUDART_INF_F ? CUDART_INF : 1.0) : 0.;
        const double Edisc = EXACT ? ray_edisc(S.h) * slack : 0., Ep = EXACT ? ray_ep(S.h) * slack : 0.;
        for (int k = first; k < first + cnt; ++k) {
            if (EXACT) {
                // FP64 reject before the reference's formula (two divisions and a square root; 650 atoms,
                // 20 x 65,536 rays with PA: 1.55 -> 1.09 ms together with PA from the first query):
                // q = x.d, w = |x|^2 - r^2 and disc = q^2 - w are within 1e-13 A^2 of their true
                // values for unit d, far inside the FP32 filter's bounds
                const double4 a = S.atoms64[k];
                const double x0 = L.o[0] - a.x, x1 = L.o[1] - a.y, x2 = L.o[2] - a.z;
                const double q = fma(x0, L.d[0], fma(x1, L.d[1], x2 * L.d[2]));
                const double w = fma(x0, x0, fma(x1, x1, fma(x2, x2, -a.w * a.w)));
                const double disc = fma(q, q, -w);
                if (disc < -Edisc || q > Ep) continue;                 // certain miss
                if (k == last_rank) continue;
                bool certain = false;
                if (disc >= 2.0 * Edisc) {
                    float Et;
                    const float b = (float)-q, t = b - certain_sqrt(b, (float)disc, (float)Ep, (float)Edisc, Et);
                    if (t < -2.0f * Et || t - Et > U) continue;        // no entry ahead, or behind the best one
                    certain = t > Et;
                }
                if (!certain) grazing = true;
                const double t = entry64<UNIT>(L.o[0], L.o[1], L.o[2], L.d[0], L.d[1], L.d[2], a.x, a.y, a.z, a.w);
                const int id = __ldg(S.ids + k);
                if (better(t, id, best, best_id)) {
                    best = t; best_rank = k; best_id = id;
                    U = __double2float_ru(best);
                }
            } else {
                const float4 a = __ldg(S.atoms + k);
                float b;
                const float D = sphere_disc(r, a, b);
                if (D < r.thr || b < r.bmin) continue;
                // the start atom is excluded after the cheap reject, which a ray leaving that
                // atom's surface (moving away from its centre) nearly always takes
                if (k == last_rank) continue;
                const float Edisc = ray_edisc(S.h), Ep = ray_ep(S.h);
                const float disc = fmaf(2.0f, D - r.thr, -Edisc), bt = fmaf(b - r.bmin, kSqrt2, -Ep);
                if (disc >= 2.0f * Edisc) {
                    float Et;
                    const float t = bt - certain_sqrt(bt, disc, Ep, Edisc, Et);
                    if (t < -2.0f * Et) continue;
                    if (t > Et) {
                        const float up = t + Et;
                        if (up < U) U = up;
                        add_candidate(k, t - Et);
                        continue;
                    }
                }
                grazing = true;
                add_candidate(k, fmaxf(0.0f, (bt - Ep - sqrtf(fmaxf(disc, 0.0f) + Edisc)) * (1.0f - 8.0f * kU32)));
            }
        }
    }
    // The ray of a new query.  Not kRayOk: a query for the out-of-line search (an origin beyond the walk's bounds, or
    // for FILTER a direction that is not unit).
    __device__ __forceinline__ int start(const SceneHeader* H, const LaneRay& L) {
        reset();
        const int kind = setup_ray<EXACT, UNIT>(H, L.o, L.d, r);
        if (!EXACT || kind == kRayFar) return kind;
        r.thr = kind == kRayOk ? 0.0f : CUDART_INF_F;
        return kRayOk;
    }
    // No lane of the warp is in a query: nothing of it has to be kept across a call.
    __device__ __forceinline__ void forget() {
        reset();
        r = RayF{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        best = 0.; best_rank = best_id = -1;
    }
};

// FP64 resolution of a finished FILTER query: re-test the candidates with the
// reference formula and the (distance, id) rule.
template <bool COUNT, bool UNIT>
__device__ __forceinline__ int resolve_candidates(const SceneView& S, const Walker<false, COUNT, UNIT>& W, const LaneRay& L,
                                                  double& best, unsigned& fp64) {
    best = CUDART_INF;
    int k = -1, best_id = -1;
#pragma unroll
    for (int e = 0; e < kCand; ++e) {
        if (W.cand_rank[e] >= 0 && W.cand_lo[e] <= W.U) {
            int kk = W.cand_rank[e];
            double4 a = S.atoms64[kk];
            double t = entry64<UNIT>(L.o[0], L.o[1], L.o[2], L.d[0], L.d[1], L.d[2], a.x, a.y, a.z, a.w);
            ++fp64;
            int id = __ldg(S.ids + kk);
            if (better(t, id, best, best_id)) { best = t; k = kk; best_id = id; }
        }
    }
    return k;
}

// The rest of a parked ray's path, from its current query on, in FP64.  A lane parks its ray when the query overflows its candidate slots
// (one in 450,000 on the mixed 256-globule batch) or cannot be walked in FP32,
// and the warp takes the parked rays when no lane is in a query: as a call in the
// resolve phase, every value that a lane holds across it was stored and
// reloaded on the hot path (10 % of the batched trace).  Inlined here, where no value of a query is live; as a call it still
// cost 4 %.  Returns whether the ray escaped.
template <bool UNIT>
__device__ __forceinline__ bool rest_of_path(const void* scene, LaneRay& L, int cap, int& bounces, int& last_rank,
                                          int32_t* history, LocalStats& st) {
    const SceneView S = scene_view(scene);
    bool first = true;
    while (true) {
        double best;
        const int k = nearest<true, UNIT>(S, L.o, L.d, last_rank, best, st);
        if (first) --st.queries;                          // counted when the query began
        first = false;
        if (k < 0) return true;
        if (bounces >= cap) return false;
        const double4 a = S.atoms64[k];
        reflect64(L.o[0], L.o[1], L.o[2], L.d[0], L.d[1], L.d[2], a.x, a.y, a.z, a.w, best);
        if (history) history[bounces] = S.ids[k];
        ++bounces;
        last_rank = k;
    }
}

// Rare path of k_blocks, kept out of line so that it costs the hot loop no registers.
__device__ __noinline__ void save_residual(ehss_residual* residual, long long capacity, unsigned long long* count,
                                           const LaneRay& L, int block, int last_rank, int bounces) {
    unsigned long long at = atomicAdd(count, 1ull);
    if (at >= (unsigned long long)capacity) return;
    ehss_residual& R = residual[at];
    for (int i = 0; i < 3; ++i) { R.o[i] = L.o[i]; R.d[i] = L.d[i]; R.din[i] = L.din[i]; }
    R.block = block;
    R.last_rank = last_rank;
    R.bounces = bounces;
    R.reserved = 0;
}

// Work distribution: the chunk list is cut into one contiguous range per SM
// (partition = %smid mod n_parts) so that the warps of an SM trace the same
// structure, and neighbouring regions of its ray space, at the same time and
// share their L1.  A warp whose range is used up takes chunks from the next
// ranges in turn.  counters[p] counts the chunks handed out from range p.
// Only the window [first, first + total) of the chunk list is traced (the
// whole list, or one GPU's share of it).
__device__ __forceinline__ bool next_chunk(unsigned long long* counters, int n_parts, int& scan, int64_t first,
                                           int64_t total, long long& chunk) {
    for (; scan < n_parts; ++scan) {
        unsigned smid;
        asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
        int p = (int)((smid + (unsigned)scan) % (unsigned)n_parts);
        int64_t begin = total * p / n_parts, end = total * (p + 1) / n_parts;
        if (begin >= end) continue;
        unsigned long long t = atomicAdd(counters + p, 1ull);
        if (begin + (int64_t)t < end) { chunk = first + begin + (int64_t)t; return true; }
    }
    return false;
}

// RAYS: the instance for blocks with EHSS_BLOCK_RAYS (caller-made weighted rays);
// each instance skips the other kind's chunks, like the precision instances.
// PA: the instance that serves EHSS_BLOCK_PA; the caller says with
// EHSS_LAUNCH_NO_PA that no block has it (such a block is then an error), which
// keeps the any-hit query's registers out of the kernel (spill stores / loads a
// thread 174 / 230 -> 116 / 156 B; the 256-globule batch 2 % faster).
template <bool EXACT, bool COUNT, bool RAYS, bool PA>
__global__ void __launch_bounds__(128, 8) k_blocks(const ehss_block* blocks, int nb, int64_t chunk_first,
                                                   int64_t total_chunks, int chunk_rays, int resolve_batch,
                                                   ehss_block_result* results,
                                                   uint64_t* hist, uint64_t* ledger, unsigned long long* work,
                                                   int n_parts, int smem_stack, ehss_residual* residual,
                                                   long long residual_capacity, unsigned long long* residual_count) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    WarpAcc& A = reinterpret_cast<WarpAcc*>(smem_raw)[warp];
    LaneRay& L = reinterpret_cast<LaneRay*>(smem_raw + sizeof(WarpAcc) * nwarps)[threadIdx.x];
    int2* stack_base = reinterpret_cast<int2*>(smem_raw + sizeof(WarpAcc) * nwarps + sizeof(LaneRay) * blockDim.x);
    // RAYS: each lane's ray weight relative to the block's largest, after the stack
    double* rho_lane = reinterpret_cast<double*>(stack_base + smem_stack * blockDim.x) + threadIdx.x;
    const unsigned lt_mask = (1u << lane) - 1u;
    Walker<EXACT, COUNT, !RAYS> W;
    int scan = 0;
    while (true) {
        long long c = 0;
        int have = 0;
        if (lane == 0) have = next_chunk(work, n_parts, scan, chunk_first, total_chunks, c);
        have = __shfl_sync(0xffffffffu, have, 0);
        if (!have) break;
        c = __shfl_sync(0xffffffffu, c, 0);
        int bi = 0, hi = nb - 1;
        while (bi < hi) {
            int mid = (bi + hi + 1) >> 1;
            if (blocks[mid].chunk_begin <= c) bi = mid; else hi = mid - 1;
        }
        const ehss_block* B = blocks + bi;
        if ((B->precision == EHSS_PREC_FP64) != EXACT) continue;     // the other instantiation's chunk
        if (((B->flags & EHSS_BLOCK_RAYS) != 0) != RAYS) continue;
        const int64_t ray0 = (c - B->chunk_begin) * (int64_t)chunk_rays;
        const int cnt = (int)min((long long)chunk_rays, (long long)((1ll << B->log2_rays) - ray0));
        // only the scene's base stays live across the phases; each phase rebuilds the view
        // it needs from the (L1-resident) header, which keeps the traversal's registers free
        const void* const sbase = B->scene;
        const bool ok = scene_view(sbase).h->magic == kSceneMagic && scene_view(sbase).h->status == 0 &&
                        (PA || !(B->flags & EHSS_BLOCK_PA));
        if (lane < kSmemBins) { A.count[lane] = 0; A.ledger[lane] = 0; }
        if (lane == 0) {
            const uint4 b0 = make_uint4(B->base[0], B->base[1], B->base[2], B->base[3]);
            A.q0 = block_point(reinterpret_cast<const uint4*>(B->basis), b0, (uint32_t)ray0);
            A.angle_fx = 0; A.hits = A.unresolved = A.escaped = A.pa = 0;
            A.queries = A.grazing = A.fallback = A.fp64 = 0;
            A.errors = ok ? 0 : 1;
            A.box = A.sphere = 0;
            A.hits_fx = A.unres_fx = A.pa_fx = 0;
        }
        __syncwarp();
        if (COUNT) { W.box = 0; W.sphere = 0; }
        int status = ok ? kNeedRay : kIdle;
        int pool = 0, bounces = 0, last_rank = -1;
        while (true) {
            // ---- resolve finished queries (FP64) ----
            if (PA && !RAYS && status == kDone && bounces == 0 && (W.grazing || W.overflow) &&
                (__ldg(&B->flags) & EHSS_BLOCK_PA)) {
                // a near-tangent first query leaves PA (below) to the any-hit query
                LocalStats pst;
                if (anyhit<!RAYS>(scene_view(sbase), L.o, L.d, -1, pst)) atomicAdd(&A.pa, 1u);
                if (COUNT) { W.box += pst.box; W.sphere += pst.sphere; }
            }
            if (!EXACT && status == kDone && W.overflow && !W.error) {
                if (W.grazing) atomicAdd(&A.grazing, 1u);
                atomicAdd(&A.fallback, 1u);
                status = kParked;                         // rest_of_path
            }
            if (status == kDone) {
                const SceneView S = scene_view(sbase);
                int k;
                double best;
                if (W.error) {
                    atomicAdd(&A.errors, 1u);
                    k = -1; best = CUDART_INF;
                } else if (EXACT) {
                    k = W.best_rank; best = W.best;
                    atomicAdd(&A.fp64, 1u);
                } else {
                    if (W.grazing) atomicAdd(&A.grazing, 1u);
                    unsigned f = 0;
                    k = resolve_candidates(S, reinterpret_cast<const Walker<false, COUNT, !RAYS>&>(W), L, best, f);
                    atomicAdd(&A.fp64, f);
                }
                // PA of a ray that is traced too: its first query has met a sphere for certain or missed every one
                // for certain, unless a test was near-tangent.  Disk rays start outside every sphere, where "meets"
                // and "enters" agree.
                if (PA && !RAYS && bounces == 0 && k >= 0 && !W.grazing && (__ldg(&B->flags) & EHSS_BLOCK_PA))
                    atomicAdd(&A.pa, 1u);
                if (k < 0 || bounces >= __ldg(&B->cap)) {
                    bool escaped = k < 0;
                    unsigned long long fx = 0;
                    if (escaped) {
                        double a = scatter_angle(L.din[0], L.din[1], L.din[2], L.d[0], L.d[1], L.d[2]);
                        fx = __double2ull_rn((RAYS ? a * *rho_lane : a) * kFxScale);
                        atomicAdd(&A.escaped, 1u);
                        if (fx) atomicAdd(&A.angle_fx, fx);
                    } else {
                        atomicAdd(&A.unresolved, 1u);
                        if (RAYS) atomicAdd(&A.unres_fx, __double2ull_rn(*rho_lane * kFxScale));
                        // save the state for a later cap extension
                        if (residual) save_residual(residual, residual_capacity, residual_count, L, bi, last_rank, bounces);
                    }
                    if (bounces > 0 || !escaped) {
                        atomicAdd(&A.hits, 1u);
                        if (RAYS) atomicAdd(&A.hits_fx, __double2ull_rn(*rho_lane * kFxScale));
                    }
                    if (bounces < kSmemBins) {
                        atomicAdd(&A.count[bounces], 1u);
                        if (fx) atomicAdd(&A.ledger[bounces], fx);
                    } else {
                        atomicAdd((unsigned long long*)&hist[B->hist_offset + bounces], 1ull);
                        if (fx) atomicAdd((unsigned long long*)&ledger[B->hist_offset + bounces], fx);
                    }
                    status = kNeedRay;
                } else {
                    double4 a = S.atoms64[k];
                    reflect64<!RAYS>(L.o[0], L.o[1], L.o[2], L.d[0], L.d[1], L.d[2], a.x, a.y, a.z, a.w, best);
                    ++bounces;
                    last_rank = k;
                    W.error = W.start(S.h, L) != kRayOk;     // bounce points lie within S, directions are unit
                    atomicAdd(&A.queries, 1u);
                    status = kTraverse;
                }
            }
            // ---- new rays for lanes whose ray finished ----
            // made once kNewRayBatch lanes wait for one (or the chunk is used up, or no
            // lane traverses), so that the FP64 impact-disk work runs at warp width
            unsigned need = __ballot_sync(0xffffffffu, status == kNeedRay);
            if (need && (__popc(need) >= kNewRayBatch || pool >= cnt || !__any_sync(0xffffffffu, status == kTraverse))) {
                const SceneView S = scene_view(sbase);
                if (status == kNeedRay) {
                    int p = pool + __popc(need & lt_mask);
                    if (p < cnt) {
                        if (RAYS) {
                            // caller-made rays: origins [3n], directions [3n], weights [n]
                            const int64_t n = 1ll << B->log2_rays, r = ray0 + p;
                            const double* R = B->rays;
#pragma unroll
                            for (int i = 0; i < 3; ++i) {
                                L.o[i] = R[3 * r + i];
                                L.d[i] = L.din[i] = R[3 * n + 3 * r + i];
                            }
                            *rho_lane = R[6 * n + r] * B->ray_scale;
                        } else {
                            // ray0 is a multiple of the chunk size, so point(ray0 + p) = point(ray0) ^ B(p)
                            uint4 q = block_point(reinterpret_cast<const uint4*>(B->basis), A.q0, (uint32_t)p);
                            Ray64 ray = impact_ray(q, S.h->center, S.h->radius);
#pragma unroll
                            for (int i = 0; i < 3; ++i) { L.o[i] = ray.o[i]; L.d[i] = ray.d[i]; L.din[i] = ray.d[i]; }
                        }
                        if (PA && (__ldg(&B->flags) & EHSS_BLOCK_PA) && (RAYS || !(__ldg(&B->flags) & EHSS_BLOCK_EHSS))) {
                            LocalStats pst;
                            if (anyhit<!RAYS>(S, L.o, L.d, -1, pst)) {
                                atomicAdd(&A.pa, 1u);
                                if (RAYS) atomicAdd(&A.pa_fx, __double2ull_rn(*rho_lane * kFxScale));
                            }
                            // the counting instance adds the any-hit tests to the block's counters
                            if (COUNT) { W.box += pst.box; W.sphere += pst.sphere; }
                        }
                        bounces = 0;
                        last_rank = -1;
                        if (__ldg(&B->flags) & EHSS_BLOCK_EHSS) {
                            const int kind = W.start(S.h, L);
                            W.error = kind == kRayFar;
                            atomicAdd(&A.queries, 1u);
                            status = kTraverse;
                            if (!EXACT && kind == kRayNotUnit) { atomicAdd(&A.fallback, 1u); status = kParked; }
                        }
                    } else {
                        status = kIdle;
                    }
                }
                pool += __popc(need);
                if (__any_sync(0xffffffffu, status == kNeedRay)) continue;   // PA-only lanes refill again
            }
            if (!__any_sync(0xffffffffu, status == kTraverse)) {
                if (EXACT || !__any_sync(0xffffffffu, status == kParked)) break;
                // ---- parked rays ----
                if (status == kParked) {
                    LocalStats st;
                    int count = bounces, last = last_rank;      // copies: the variables stay in registers
                    const bool escaped = rest_of_path<!RAYS>(sbase, L, __ldg(&B->cap), count, last, nullptr, st);
                    bounces = count;
                    last_rank = last;
                    atomicAdd(&A.queries, st.queries);
                    atomicAdd(&A.grazing, st.grazing);
                    atomicAdd(&A.fallback, st.fallback);
                    atomicAdd(&A.fp64, st.fp64);
                    atomicAdd(&A.errors, st.errors);
                    if (COUNT) { W.box += st.box; W.sphere += st.sphere; }
                    status = kDone;                       // without candidates: escaped
                    if (!escaped) {
                        atomicAdd(&A.unresolved, 1u);
                        atomicAdd(&A.hits, 1u);
                        if (RAYS) {
                            atomicAdd(&A.unres_fx, __double2ull_rn(*rho_lane * kFxScale));
                            atomicAdd(&A.hits_fx, __double2ull_rn(*rho_lane * kFxScale));
                        }
                        if (residual) save_residual(residual, residual_capacity, residual_count, L, bi, last_rank, bounces);
                        if (bounces < kSmemBins) atomicAdd(&A.count[bounces], 1u);
                        else atomicAdd((unsigned long long*)&hist[B->hist_offset + bounces], 1ull);
                        status = kNeedRay;
                    }
                }
                W.forget();
                continue;
            }
            // ---- traverse until enough queries are finished ----
            const SceneView S = scene_view(sbase);
            while (true) {
                if (status == kTraverse) {
                    // Walker::advance, written out: as a call it costs this kernel 8 bytes of spills and 1 % of its time
                    while (W.cur >= 0 && W.cur != kSentinel) {
                        const int n_nodes = __ldg(&S.h->n_nodes);
                        if (W.cur >= n_nodes || ++W.steps > 2 * n_nodes + 2) { W.error = true; W.cur = kSentinel; break; }
                        W.cur = W.visit(S.nodes, W.cur, smem_stack);
                        if (W.cur < 0 && W.leaf == kNoLeaf) {
                            W.leaf = W.cur;
                            W.cur = W.pop(smem_stack);
                        }
                        if (!__any_sync(__activemask(), W.leaf == kNoLeaf)) break;
                    }
                    if (W.leaf != kNoLeaf) {
                        W.leaf_tests(S, W.leaf, last_rank, L);
                        W.next_leaf(smem_stack);
                    }
                    if (W.finished()) status = kDone;
                }
                // lanes waiting for a new ray count towards the resolve batch
                unsigned done = __ballot_sync(0xffffffffu, status == kDone || status == kNeedRay);
                unsigned trav = __ballot_sync(0xffffffffu, status == kTraverse);
                if (!trav || __popc(done) >= resolve_batch) break;
            }
        }
        if (COUNT) {
            unsigned long long b = warp_sum64(W.box), sp = warp_sum64(W.sphere);
            if (lane == 0) { A.box = b; A.sphere = sp; }
        }
        __syncwarp();
        // one atomic per field into the block result
        ehss_block_result* R = results + bi;
        if (lane == 0) {
            if (A.angle_fx) atomicAdd((unsigned long long*)&R->angle_fx, A.angle_fx);
            if (A.hits) atomicAdd((unsigned long long*)&R->hits, (unsigned long long)A.hits);
            if (A.unresolved) atomicAdd((unsigned long long*)&R->unresolved, (unsigned long long)A.unresolved);
            if (A.escaped) atomicAdd((unsigned long long*)&R->escaped, (unsigned long long)A.escaped);
            if (A.pa) atomicAdd((unsigned long long*)&R->pa_blocked, (unsigned long long)A.pa);
            if (A.hits_fx) atomicAdd((unsigned long long*)&R->hits_fx, A.hits_fx);
            if (A.unres_fx) atomicAdd((unsigned long long*)&R->unresolved_fx, A.unres_fx);
            if (A.pa_fx) atomicAdd((unsigned long long*)&R->pa_fx, A.pa_fx);
            unsigned long long v[7] = {A.box, A.sphere, A.queries, A.grazing, A.fallback, A.fp64, A.errors};
            const int slot[7] = {EHSS_STAT_BOX_TESTS, EHSS_STAT_SPHERE_TESTS, EHSS_STAT_QUERIES, EHSS_STAT_GRAZING,
                                 EHSS_STAT_FALLBACK, EHSS_STAT_FP64_TESTS, EHSS_STAT_ERRORS};
            for (int i = 0; i < 7; ++i)
                if (v[i]) atomicAdd((unsigned long long*)&R->stats[slot[i]], v[i]);
        }
        if (lane < kSmemBins && lane <= B->cap) {
            if (A.count[lane])
                atomicAdd((unsigned long long*)&hist[B->hist_offset + lane], (unsigned long long)A.count[lane]);
            if (A.ledger[lane]) atomicAdd((unsigned long long*)&ledger[B->hist_offset + lane], A.ledger[lane]);
        }
        __syncwarp();
    }
}

// --------------------------------------------------------------------------
// Explicit rays (EHSS), the Walker and phases of k_blocks with per-ray inputs
// and outputs.  A lane whose ray has finished takes the next ray of the whole
// call (a shared counter), so a warp's lanes stay busy until the call's rays
// are used up; one thread per ray left a warp running until its longest path.
// Rays are read where they lie: device memory, or page-locked host memory
// (whole 128-byte PCIe reads, load_rays).  Results go to device arrays; when
// the caller wants them in page-locked host memory too, the lane whose ray
// completes a run of kExportRays consecutive rays has its warp copy the run's
// results there (whole lines again), so reading, tracing and writing back
// overlap in one launch.  Nothing waits: a run is copied by whoever finishes it.
// Bound by latency: long-scoreboard stalls (nodes, atoms and, at the ends, the
// host's memory) take 12 of 20 cycles an instruction.  2000 atoms, 262,144 rays,
// FP32: 412 us on device arrays (one thread per ray: 620 us) and 660 us with
// rays and results in host memory (35 copies on two streams around four
// launches: 1500 us); runs of 32 rays leave sooner than runs of 256 (700 us),
// and 6 CTAs of 80 registers beat 8 of 64 there (713 us).
// --------------------------------------------------------------------------
constexpr int kRayCtas = 6, kRayResolve = 28;     // CTAs per SM; finished lanes that start a resolve phase

struct RayCall {
    const void* scene;
    int64_t n;
    int cap;
    const double *P, *D;               // source rays; may equal Po, Do
    const int64_t *last, *bounces;     // NULL: -1 and 0 for every ray
    double *Po, *Do;                   // results (device)
    int64_t* bounces_out;
    uint8_t *escaped, *unresolved;
    int32_t* history;
    uint64_t* stats;
    unsigned long long* next;          // rays handed out; NULL: warps take fixed runs of `lanes` in turn
    unsigned* finished;                // per run of kExportRays rays; NULL: results stay on the device
    int lanes;                         // lanes of a warp that take rays
    double *hP, *hD;                   // page-locked copies of the results
    int64_t* hb;
    uint8_t *he, *hu;
};

struct RayAcc {
    unsigned queries, grazing, fallback, fp64, errors, pad;
    double buf[96];
};

// Copies bytes [begin, end) of a result array to its host copy, 16 bytes a lane where both are aligned.
__device__ __forceinline__ void export_bytes(void* dst, const void* src, int64_t begin, int64_t end) {
    const unsigned lane = threadIdx.x & 31;
    char* d = (char*)dst;
    const char* s = (const char*)src;
    if (!(((uintptr_t)(d + begin) | (uintptr_t)(s + begin)) & 15u)) {
        for (int64_t i = begin + 16 * lane; i + 16 <= end; i += 512) *(uint4*)(d + i) = __ldcg((const uint4*)(s + i));
        begin += (end - begin) & ~(int64_t)15;
    }
    for (int64_t i = begin + lane; i < end; i += 32) d[i] = __ldcg(s + i);
}

__device__ __forceinline__ void store_result(const RayCall& C, const LaneRay& L, int64_t ray, int bounces, bool escaped) {
#pragma unroll
    for (int c = 0; c < 3; ++c) { C.Po[3 * ray + c] = L.o[c]; C.Do[3 * ray + c] = L.d[c]; }
    C.bounces_out[ray] = bounces;
    C.escaped[ray] = escaped;
    C.unresolved[ray] = !escaped;
}

// Counts the warp's finished rays; runs that are complete with them go to the host.
// The results of a run come from several warps.  Each lane's are ordered before
// its count by the fence ahead of it; the lane whose count completes the run
// orders them before what follows by the fence behind it, and the warp barrier
// (a ballot or shuffle orders no memory) passes that on to the lanes that copy.
__device__ __forceinline__ void export_runs(const RayCall& C, bool fin, int64_t ray) {
    bool last_of_run = false;
    if (fin) {
        const int64_t g = ray / kExportRays;
        const unsigned size = (unsigned)min((int64_t)kExportRays, C.n - g * kExportRays);
        __threadfence();
        last_of_run = atomicAdd(C.finished + g, 1u) + 1u == size;
        if (last_of_run) __threadfence();
    }
    __syncwarp();
    for (unsigned todo = __ballot_sync(0xffffffffu, last_of_run); todo; todo &= todo - 1) {
        const int64_t b = __shfl_sync(0xffffffffu, ray, __ffs(todo) - 1) / kExportRays * kExportRays;
        const int64_t e = min(b + kExportRays, C.n);
        export_bytes(C.hP, C.Po, 24 * b, 24 * e);
        export_bytes(C.hD, C.Do, 24 * b, 24 * e);
        export_bytes(C.hb, C.bounces_out, 8 * b, 8 * e);
        export_bytes(C.he, C.escaped, b, e);
        export_bytes(C.hu, C.unresolved, b, e);
    }
}

template <bool EXACT>
__global__ void __launch_bounds__(128, kRayCtas) k_rays(const __grid_constant__ RayCall C, int resolve_batch, int smem_stack) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5, full = 0xffffffffu;
    LaneRay& L = reinterpret_cast<LaneRay*>(smem_raw + sizeof(WarpAcc) * nwarps)[threadIdx.x];
    RayAcc& A = *reinterpret_cast<RayAcc*>(smem_raw + sizeof(WarpAcc) * nwarps + sizeof(LaneRay) * blockDim.x +
                                           sizeof(int2) * smem_stack * blockDim.x + sizeof(RayAcc) * warp);
    const unsigned lt_mask = (1u << lane) - 1u;
    const SceneHeader* const H = reinterpret_cast<const SceneHeader*>(C.scene);
    // exterior scenes hold only the atoms reachable from outside the union: not for arbitrary rays
    const bool ok = H->magic == kSceneMagic && H->status == 0 && H->exterior == 0;
    if (lane == 0) A.queries = A.grazing = A.fallback = A.fp64 = A.errors = 0;
    __syncwarp();
    Walker<EXACT, true, false> W;
    W.box = W.sphere = 0;
    int status = lane < C.lanes ? kNeedRay : kIdle, bounces = 0, last_rank = -1;
    const int refill_at = min(kNewRayBatch, (C.lanes + 1) / 2);
    int64_t ray = 0;
    // fixed runs (no counter): this warp's current run [pool, pool_end) and its next one
    int64_t run = C.lanes * (blockIdx.x * (int64_t)nwarps + warp), pool = run, pool_end = min(run + C.lanes, C.n);
    bool more = true;
    while (true) {
        // ---- resolve finished queries (FP64) ----
        bool fin = false;
        if (!EXACT && status == kDone && W.overflow && !W.error) {
            if (W.grazing) atomicAdd(&A.grazing, 1u);
            atomicAdd(&A.fallback, 1u);
            status = kParked;                             // rest_of_path
        }
        if (status == kDone) {
            const SceneView S = scene_view(C.scene);
            int k;
            double best;
            if (W.error) {
                atomicAdd(&A.errors, 1u);
                k = -1; best = CUDART_INF;
            } else if (EXACT) {
                k = W.best_rank; best = W.best;
            } else {
                if (W.grazing) atomicAdd(&A.grazing, 1u);
                unsigned f = 0;
                k = resolve_candidates(S, reinterpret_cast<const Walker<false, true, false>&>(W), L, best, f);
                atomicAdd(&A.fp64, f);
            }
            if (k < 0 || bounces >= C.cap) {
                store_result(C, L, ray, bounces, k < 0);
                fin = true;
                status = kNeedRay;
            } else {
                const double4 a = S.atoms64[k];
                reflect64(L.o[0], L.o[1], L.o[2], L.d[0], L.d[1], L.d[2], a.x, a.y, a.z, a.w, best);
                if (C.history) C.history[ray * (int64_t)C.cap + bounces] = S.ids[k];
                ++bounces;
                last_rank = k;
                status = W.start(S.h, L) == kRayOk ? kTraverse : kParked;
                atomicAdd(&A.queries, 1u);
            }
        }
        if (C.finished && __any_sync(full, fin)) export_runs(C, fin, ray);
        // ---- new rays for lanes whose ray finished ----
        bool bad = false;
        const unsigned need = __ballot_sync(full, status == kNeedRay);
        const bool refill = need && (__popc(need) >= refill_at || !more || !__any_sync(full, status == kTraverse));
        int64_t base = 0;
        int got = 0;
        if (refill && more) {
            const int want = __popc(need);
            if (C.next) {
                unsigned long long t = 0;
                if (lane == 0) t = atomicAdd(C.next, (unsigned long long)want);
                base = (int64_t)__shfl_sync(full, t, 0);
                got = (int)max((int64_t)0, min((int64_t)want, C.n - base));
                more = base + want < C.n;
            } else {
                if (pool >= pool_end) {
                    run += C.lanes * (int64_t)gridDim.x * nwarps;
                    pool = run;
                    pool_end = min(run + C.lanes, C.n);
                }
                base = pool;
                got = (int)max((int64_t)0, min((int64_t)want, pool_end - pool));
                pool += got;
                more = got > 0;
            }
        }
        if (refill) {
            const int q = status == kNeedRay ? __popc(need & lt_mask) : 32;
            if (got > 0) {
                double o[3], d[3];
                load_rays(C.P, base, got, q, A.buf, o);
                load_rays(C.D, base, got, q, A.buf, d);
                if (q < got) {
                    const SceneView S = scene_view(C.scene);
                    ray = base + q;
                    const int64_t count = C.bounces ? C.bounces[ray] : 0, last_id = C.last ? C.last[ray] : -1;
#pragma unroll
                    for (int c = 0; c < 3; ++c) { L.o[c] = o[c]; L.d[c] = d[c]; }
                    if (!ok || last_id < -1 || last_id >= S.h->n_atoms || count < 0 || count > 1 || (count == 1 && last_id < 0)) {
                        atomicAdd(&A.errors, 1u);
                        if (C.Po != C.P) {
#pragma unroll
                            for (int c = 0; c < 3; ++c) { C.Po[3 * ray + c] = o[c]; C.Do[3 * ray + c] = d[c]; }
                            C.bounces_out[ray] = count;
                        }
                        C.escaped[ray] = 0;
                        C.unresolved[ray] = 0;
                        bad = true;                       // stays kNeedRay
                    } else {
                        if (C.history && count == 1) C.history[ray * (int64_t)C.cap] = (int32_t)last_id;
                        bounces = (int)count;
                        last_rank = last_id >= 0 ? S.rank[last_id] : -1;
                        status = W.start(S.h, L) == kRayOk ? kTraverse : kParked;
                        atomicAdd(&A.queries, 1u);
                    }
                }
            }
            if (!more && status == kNeedRay && !(q < got)) status = kIdle;
        }
        if (C.finished && __any_sync(full, bad)) export_runs(C, bad, ray);
        if (!__any_sync(full, status == kTraverse)) {
            if (__any_sync(full, status == kParked)) {
                // ---- parked rays ----
                const bool parked = status == kParked;
                if (parked) {
                    LocalStats st;
                    int count = bounces, last = last_rank;      // copies: the variables stay in registers
                    const bool out = rest_of_path<false>(C.scene, L, C.cap, count, last,
                                                         C.history ? C.history + ray * (int64_t)C.cap : nullptr, st);
                    bounces = count;
                    last_rank = last;
                    atomicAdd(&A.queries, st.queries);
                    atomicAdd(&A.grazing, st.grazing);
                    atomicAdd(&A.fallback, st.fallback);
                    if (!EXACT) atomicAdd(&A.fp64, st.fp64);
                    atomicAdd(&A.errors, st.errors);
                    W.box += st.box;
                    W.sphere += st.sphere;
                    store_result(C, L, ray, bounces, out);
                    status = kNeedRay;
                }
                W.forget();
                if (C.finished) export_runs(C, parked, ray);
                continue;
            }
            if (!__any_sync(full, status == kNeedRay)) break;
            continue;
        }
        // ---- traverse until enough queries are finished ----
        const SceneView S = scene_view(C.scene);
        while (true) {
            if (status == kTraverse) {
                W.advance(S, smem_stack, last_rank, L);
                if (W.finished()) status = kDone;
            }
            // lanes without a ray count towards the batch: the call's last rays do not wait for one another
            const unsigned trav = __ballot_sync(full, status == kTraverse);
            if (32 - __popc(trav) >= resolve_batch) break;
        }
    }
    if (!C.stats) return;
    const unsigned long long box = warp_sum64(W.box), sphere = warp_sum64(W.sphere);
    __syncwarp();
    if (lane == 0) {
        const unsigned long long v[7] = {box, sphere, A.queries, A.grazing, A.fallback, EXACT ? sphere : A.fp64, A.errors};
        const int slot[7] = {EHSS_STAT_BOX_TESTS, EHSS_STAT_SPHERE_TESTS, EHSS_STAT_QUERIES, EHSS_STAT_GRAZING,
                             EHSS_STAT_FALLBACK, EHSS_STAT_FP64_TESTS, EHSS_STAT_ERRORS};
        for (int i = 0; i < 7; ++i)
            if (v[i]) atomicAdd((unsigned long long*)&C.stats[slot[i]], v[i]);
    }
}

// --------------------------------------------------------------------------
// Host launchers
// --------------------------------------------------------------------------
static unsigned grid_for(int64_t n, int threads) {
    int64_t want = (n + threads - 1) / threads;
    int64_t cap = (int64_t)sm_count() * 16;
    if (want > cap) want = cap;
    return (unsigned)(want > 0 ? want : 1);
}

int launch_trace_rays(const RayBuffers& B, int precision, cudaStream_t stream) {
    if (B.n == 0) return EHSS_OK;
    RayCall C;
    C.scene = B.scene; C.n = B.n; C.cap = B.cap;
    C.P = B.origins; C.D = B.directions; C.last = B.last; C.bounces = B.bounces;
    C.Po = B.positions; C.Do = B.outgoing; C.bounces_out = B.bounces_out; C.escaped = B.escaped; C.unresolved = B.unresolved;
    C.history = B.history; C.stats = B.stats;
    C.next = B.next; C.finished = B.finished;
    C.hP = B.host_positions; C.hD = B.host_outgoing; C.hb = B.host_bounces; C.he = B.host_escaped; C.hu = B.host_unresolved;
    // Few rays take few lanes of a warp, up to one warp a scheduler: a warp's lanes diverge, so fewer of them finish
    // sooner (2000 atoms, 4096 rays: 125 us against 165; with more warps than that, 32,768 rays: 218 against 205).
    // At least four a warp, in one-warp CTAs where warps are few.
    const int64_t slots = (int64_t)sm_count() * 4;
    C.lanes = (int)std::min<int64_t>(32, std::max<int64_t>(4, (B.n + slots - 1) / slots));
    const int64_t warps = (B.n + C.lanes - 1) / C.lanes;
    const int threads = warps < 4ll * sm_count() ? 32 : 128;
    const int64_t want = (warps * 32 + threads - 1) / threads, most = (int64_t)sm_count() * kRayCtas;
    const int sdepth = 5;
    const size_t smem = sizeof(WarpAcc) * (size_t)(threads / 32) + sizeof(LaneRay) * (size_t)threads +
                        sizeof(int2) * sdepth * (size_t)threads + sizeof(RayAcc) * (size_t)(threads / 32);
    const unsigned grid = (unsigned)(want < most ? want : most);
    if (precision == EHSS_PREC_FP64) k_rays<true><<<grid, threads, smem, stream>>>(C, kRayResolve, sdepth);
    else k_rays<false><<<grid, threads, smem, stream>>>(C, kRayResolve, sdepth);
    return cuda_status(cudaGetLastError(), "trace launch");
}

int launch_pa_rays(const void* scene, int64_t n, const double* P, const double* D, const int64_t* owners,
                   uint8_t* blocked, uint64_t* stats, cudaStream_t stream) {
    if (n == 0) return EHSS_OK;
    k_pa_rays<<<grid_for(n, 128), 128, 0, stream>>>(scene, n, P, D, owners, blocked, stats);
    return cuda_status(cudaGetLastError(), "PA launch");
}

int launch_sobol_points(int dim, const SobolParams& p, int64_t first, int64_t n, uint32_t* q, cudaStream_t stream) {
    if (n == 0) return EHSS_OK;
    k_sobol_points<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(dim, p, first, n, q);
    return cuda_status(cudaGetLastError(), "Sobol launch");
}

int launch_source_rays(const void* scene, const Sobol4Params& p, int64_t first, int64_t n, double* O, double* D,
                       cudaStream_t stream) {
    if (n == 0) return EHSS_OK;
    k_source_rays<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(scene, p, first, n, O, D);
    return cuda_status(cudaGetLastError(), "source launch");
}

int launch_blocks(const ehss_block* blocks, int nb, int64_t chunk_first, int64_t total_chunks, const ehss_launch& L,
                  ehss_block_result* results, uint64_t* hist, uint64_t* ledger, unsigned long long* work,
                  cudaStream_t stream, ehss_residual* residual, int64_t residual_capacity,
                  unsigned long long* residual_count) {
    int warps = L.block_threads / 32;
    const int sdepth = L.smem_stack > 0 ? L.smem_stack : 16;
    const size_t smem = sizeof(WarpAcc) * (size_t)warps + sizeof(LaneRay) * (size_t)L.block_threads +
                        sizeof(int2) * sdepth * (size_t)L.block_threads;
    const size_t smem_rays = smem + sizeof(double) * (size_t)L.block_threads;
    unsigned grid = (unsigned)(sm_count() * L.ctas_per_sm);
    int batch = L.resolve_batch > 0 ? L.resolve_batch : 1;
    const bool count = (L.options & EHSS_LAUNCH_COUNT_TESTS) != 0, pa = (L.options & EHSS_LAUNCH_NO_PA) == 0;
    // one launch per precision and ray kind present; each skips the other blocks' chunks
    const int mask = L.precisions ? L.precisions : 3;
    const int kinds = (L.options & EHSS_LAUNCH_RAY_BLOCKS) ? ((L.options & EHSS_LAUNCH_NO_DISK_BLOCKS) ? 2 : 3) : 1;
    bool first = true;
    for (int exact = 1; exact >= 0; --exact) {
        if (!((mask >> (exact ? EHSS_PREC_FP64 : EHSS_PREC_FP32)) & 1)) continue;
        for (int rays = 0; rays <= 1; ++rays) {
            if (!((kinds >> rays) & 1)) continue;
            if (!first) {
                int rc = cuda_status(cudaMemsetAsync(work, 0, sizeof(unsigned long long) * kMaxWorkParts, stream),
                                     "work counter reset");
                if (rc) return rc;
            }
            first = false;
            const int n_parts = sm_count() < kMaxWorkParts ? sm_count() : kMaxWorkParts;
#define EHSS_LAUNCH_BLOCKS(E, C, R, P) \
            k_blocks<E, C, R, P><<<grid, L.block_threads, R ? smem_rays : smem, stream>>>( \
                blocks, nb, chunk_first, total_chunks, L.chunk_rays, batch, results, hist, ledger, work, n_parts, sdepth, \
                residual, residual_capacity, residual_count)
#define EHSS_PICK_PA(E, C, R) if (pa) EHSS_LAUNCH_BLOCKS(E, C, R, true); else EHSS_LAUNCH_BLOCKS(E, C, R, false)
#define EHSS_PICK_COUNT(E, R) if (count) { EHSS_PICK_PA(E, true, R); } else { EHSS_PICK_PA(E, false, R); }
            if (exact) {
                if (rays) { EHSS_PICK_COUNT(true, true) } else { EHSS_PICK_COUNT(true, false) }
            } else {
                if (rays) { EHSS_PICK_COUNT(false, true) } else { EHSS_PICK_COUNT(false, false) }
            }
#undef EHSS_PICK_COUNT
#undef EHSS_PICK_PA
#undef EHSS_LAUNCH_BLOCKS
            int rc = cuda_status(cudaGetLastError(), "blocks launch");
            if (rc) return rc;
        }
    }
    return EHSS_OK;
}

// --------------------------------------------------------------------------
// Cap extension: continue saved unresolved rays (one thread per ray) from
// their exact state, so each follows the path it would have followed with
// the larger cap from the start.  Sums are the same integers k_blocks uses.
// --------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_extend(const ehss_block* blocks, int nb, const int32_t* row_of, int rows,
                                                const ehss_residual* in, int64_t n_in, int new_cap,
                                                ehss_extension* ext, uint64_t* hist, uint64_t* ledger,
                                                ehss_residual* out, int64_t out_capacity,
                                                unsigned long long* out_count, uint64_t* stats) {
    LocalStats st;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_in; i += stride) {
        const ehss_residual R = in[i];
        if (R.block < 0 || R.block >= nb) { ++st.errors; continue; }
        const int row = row_of[R.block];
        if (row < 0) continue;
        if (row >= rows) { ++st.errors; continue; }
        const ehss_block* B = blocks + R.block;
        const SceneView S = scene_view(B->scene);
        if ((B->flags & EHSS_BLOCK_RAYS) || S.h->magic != kSceneMagic || S.h->status != 0 || R.bounces >= new_cap || R.last_rank < -1 ||
            R.last_rank >= S.h->n_atoms) {
            ++st.errors;
            continue;
        }
        const bool exact = B->precision == EHSS_PREC_FP64;
        double o[3] = {R.o[0], R.o[1], R.o[2]}, d[3] = {R.d[0], R.d[1], R.d[2]};
        int last_rank = R.last_rank, count = R.bounces;
        bool escaped = false;
        double so[3], sd[3];
        int s_last = last_rank;
        while (true) {
            double best;
            const int k = exact ? nearest_call<true>(S, o, d, last_rank, best, st)
                                : nearest_call<false>(S, o, d, last_rank, best, st);
            if (k < 0) { escaped = true; break; }
            if (count >= new_cap) {
                for (int c = 0; c < 3; ++c) { so[c] = o[c]; sd[c] = d[c]; }
                s_last = last_rank;
                break;
            }
            const double4 a = S.atoms64[k];
            reflect64(o[0], o[1], o[2], d[0], d[1], d[2], a.x, a.y, a.z, a.w, best);
            ++count;
            last_rank = k;
        }
        ehss_extension& E = ext[row];
        uint64_t* h = hist + (int64_t)row * (new_cap + 1);
        uint64_t* l = ledger + (int64_t)row * (new_cap + 1);
        atomicAdd((unsigned long long*)&E.continued, 1ull);
        atomicAdd((unsigned long long*)&h[count], 1ull);
        if (escaped) {
            const double ang = scatter_angle(R.din[0], R.din[1], R.din[2], d[0], d[1], d[2]);
            const unsigned long long fx = __double2ull_rn(ang * kFxScale);
            atomicAdd((unsigned long long*)&E.escaped, 1ull);
            if (fx) {
                atomicAdd((unsigned long long*)&E.angle_fx, fx);
                atomicAdd((unsigned long long*)&l[count], fx);
            }
        } else {
            atomicAdd((unsigned long long*)&E.unresolved, 1ull);
            const unsigned long long at = atomicAdd(out_count, 1ull);
            if (at < (unsigned long long)out_capacity) {
                ehss_residual& Q = out[at];
                for (int c = 0; c < 3; ++c) { Q.o[c] = so[c]; Q.d[c] = sd[c]; Q.din[c] = R.din[c]; }
                Q.block = R.block;
                Q.last_rank = s_last;
                Q.bounces = count;
                Q.reserved = 0;
            }
        }
    }
    flush_stats(st, stats);
}

int launch_extend(const ehss_block* blocks, int nb, const int32_t* row, int rows, const ehss_residual* in,
                  int64_t n_in, int new_cap, ehss_extension* ext, uint64_t* hist, uint64_t* ledger,
                  ehss_residual* out, int64_t out_capacity, unsigned long long* out_count, uint64_t* stats,
                  cudaStream_t stream) {
    if (n_in == 0) return EHSS_OK;
    k_extend<<<grid_for(n_in, 128), 128, 0, stream>>>(blocks, nb, row, rows, in, n_in, new_cap, ext, hist, ledger,
                                                      out, out_capacity, out_count, stats);
    return cuda_status(cudaGetLastError(), "cap extension launch");
}

}  // namespace ehss
