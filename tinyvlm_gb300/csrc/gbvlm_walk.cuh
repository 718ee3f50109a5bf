// Ring and strip walkers of the Biot-Savart vortex-ring law, templated on
// the arithmetic type T (float, double, or the float pair Fe of
// gbvlm_math.cuh): the per-operator kernels, the batched assembly and its
// extended-precision correction evaluate the same walk.
#pragma once
#include "gbvlm_math.cuh"

namespace gbvlm {

template <class T>
__device__ __forceinline__ T inv_four_pi();
template <>
__device__ __forceinline__ float inv_four_pi<float>() { return 1.0f / (4.0f * PI_F); }
template <>
__device__ __forceinline__ double inv_four_pi<double>() { return 1.0 / (double)(4.0f * PI_F); }

// value of one full ring (4 vertices given) at point (px,py,pz) + mirror, dotted with normal (unscaled by 1/4pi)
template <class T, bool SIGMA, bool DCUT = false>
__device__ __forceinline__ T ring_normal_full(T px, T py, T pz, T nx, T ny, T nz, const V3<T>* q, T sigma2) {
    Rel<T> a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        a[k] = make_rel<T>(px - q[k].x, py - q[k].y, pz - q[k].z);
        b[k] = make_rel<T>(px - q[k].x, -py - q[k].y, pz - q[k].z);
    }
    T v = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int e = (k + 1) & 3;
        const T rx = q[e].x - q[k].x, ry = q[e].y - q[k].y, rz = q[e].z - q[k].z;
        v += seg_normal<T, SIGMA, DCUT>(a[k], a[e], rx, ry, rz, nx, ny, nz, sigma2);
        v += seg_normal<T, SIGMA, DCUT>(b[k], b[e], rx, ry, rz, nx, -ny, nz, sigma2);
    }
    return v;
}

// Walk the rings of one strip whose vertex lines sit in shared memory
// (top/bot: 3 planes W apart), local vertices 0..nvs-1; calls
// f(ring_index, 4*pi*(v.n + v_mirror.n_mirror)) for rings 0..nvs-2.
// SEG: the segment vectors come precomputed in seg[t * W + k] (shared by all
// evaluation points of a tile): t = 0 the chordwise segment top(k) -> bot(k),
// t = 1 the top segment top(k-1) -> top(k), t = 2 the bottom segment
// bot(k) -> bot(k-1); otherwise each walk forms them.
template <class T, bool SIGMA, bool DCUT = false, bool SEG = false, class F>
__device__ __forceinline__ void strip_normal(const T* top, const T* bot, int W, int nvs, T px, T py, T pz, T nx, T ny,
                                             T nz, T sg, F&& f, const V3<T>* seg = nullptr) {
    auto V = [&](const T* line, int sl) { return V3<T>{line[sl], line[W + sl], line[2 * W + sl]}; };
    V3<T> v0 = V(top, 0), v3 = V(bot, 0);
    Rel<T> A0 = make_rel<T>(px - v0.x, py - v0.y, pz - v0.z), A3 = make_rel<T>(px - v3.x, py - v3.y, pz - v3.z);
    Rel<T> B0 = make_rel<T>(px - v0.x, -py - v0.y, pz - v0.z), B3 = make_rel<T>(px - v3.x, -py - v3.y, pz - v3.z);
    const V3<T> l0 = SEG ? seg[0] : V3<T>{v3.x - v0.x, v3.y - v0.y, v3.z - v0.z};
    T Ca = seg_normal<T, SIGMA, DCUT>(A0, A3, l0.x, l0.y, l0.z, nx, ny, nz, sg);
    T Cb = seg_normal<T, SIGMA, DCUT>(B0, B3, l0.x, l0.y, l0.z, nx, -ny, nz, sg);
    for (int k = 1; k < nvs; k++) {
        const V3<T> v1 = V(top, k), v2 = V(bot, k);
        const Rel<T> A1 = make_rel<T>(px - v1.x, py - v1.y, pz - v1.z), A2 = make_rel<T>(px - v2.x, py - v2.y, pz - v2.z);
        const Rel<T> B1 = make_rel<T>(px - v1.x, -py - v1.y, pz - v1.z), B2 = make_rel<T>(px - v2.x, -py - v2.y, pz - v2.z);
        const V3<T> c3 = SEG ? seg[k] : V3<T>{v2.x - v1.x, v2.y - v1.y, v2.z - v1.z};          // right chordwise segment
        const V3<T> t3 = SEG ? seg[W + k] : V3<T>{v1.x - v0.x, v1.y - v0.y, v1.z - v0.z};      // top segment v0->v1
        const V3<T> b3 = SEG ? seg[2 * W + k] : V3<T>{v3.x - v2.x, v3.y - v2.y, v3.z - v2.z};  // bottom segment v2->v3
        const T cx = c3.x, cy = c3.y, cz = c3.z;
        const T tx = t3.x, ty = t3.y, tz = t3.z;
        const T bx = b3.x, by = b3.y, bz = b3.z;
        const T Cra = seg_normal<T, SIGMA, DCUT>(A1, A2, cx, cy, cz, nx, ny, nz, sg);
        const T Crb = seg_normal<T, SIGMA, DCUT>(B1, B2, cx, cy, cz, nx, -ny, nz, sg);
        T val = seg_normal<T, SIGMA, DCUT>(A0, A1, tx, ty, tz, nx, ny, nz, sg) + Cra +
                seg_normal<T, SIGMA, DCUT>(A2, A3, bx, by, bz, nx, ny, nz, sg) - Ca;
        val += seg_normal<T, SIGMA, DCUT>(B0, B1, tx, ty, tz, nx, -ny, nz, sg) + Crb +
               seg_normal<T, SIGMA, DCUT>(B2, B3, bx, by, bz, nx, -ny, nz, sg) - Cb;
        f(k - 1, val);
        A0 = A1; A3 = A2; B0 = B1; B3 = B2; Ca = Cra; Cb = Crb; v0 = v1; v3 = v2;
    }
}

// ---------------------------------------------------------------------------
// Sums over a whole lattice with given ring strengths.  A segment belongs to
// two rings, so the sum needs each segment once, with the difference of their
// strengths: per ring one spanwise and one chordwise segment and one vertex,
// where the ring-by-ring walk evaluates three segments and two vertices.  A
// point and its image in y = 0 share every product without a y in it.
// ---------------------------------------------------------------------------

// Square root and reciprocal of the double walk: the hardware's 20-bit
// approximation and one step of Householder's third-order iteration (its
// relative error e becomes about e^3), to within two units in the last place
// (2^-52 relative); the pair of quotients below, with one reciprocal and three
// more roundings, to within four.
// Five and three fp64 instructions where sqrt() and 1 / x take about twice
// that, on the pipe that bounds the walk.  The sums are as exact as with sqrt()
// and a / b: against quadruple precision, relative rms errors over six wakes of
// 135 to 420 rings 4.2e-16 before and 3.9e-16 now, of AIC entries 1.8e-16 and
// 1.6e-16 (fewer segments, each once).
__device__ __forceinline__ float length_of(float n2) { return fast_len<float>(n2); }
__device__ __forceinline__ double length_of(double n2) {
    double y;
    const double m = n2 + 1e-290;  // a zero length stays (almost) zero
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(m));
    const double t = m * y, e = fma(-t, y, 1.0);
    return fma(t * e, fma(e, 0.375, 0.5), t);
}
__device__ __forceinline__ double reciprocal(double d) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// a vertex seen from the point (y0, n0) and from its image (y1, n1)
template <class T> struct RelPair { T x, z, y0, y1, n0, n1; };

template <class T>
__device__ __forceinline__ RelPair<T> make_rel_pair(T px, T py, T pz, T vx, T vy, T vz) {
    RelPair<T> r;
    r.x = px - vx;
    r.z = pz - vz;
    r.y0 = py - vy;
    r.y1 = -py - vy;
    const T s = r.x * r.x + r.z * r.z;
    r.n0 = length_of(r.y0 * r.y0 + s);
    r.n1 = length_of(r.y1 * r.y1 + s);
    return r;
}

// x < c for x a sum of squares or a length (not negative, possibly NaN) and
// c > 0: in double by the bits, which order like the values, since the fp64
// pipe is the bound there (a NaN is not below, whatever its sign)
__device__ __forceinline__ bool below(float x, float c) { return x < c; }
__device__ __forceinline__ bool below(double x, double c) {
    return (unsigned long long)__double_as_longlong(x) < (unsigned long long)__double_as_longlong(c);
}
__device__ __forceinline__ bool not_negative(float x) { return x >= 0.f; }
__device__ __forceinline__ bool not_negative(double x) { return __double2hiint(x) >= 0; }

// the quotients n0 / d0 and n1 / d1; in double with one division (a cut
// quotient is zero whatever its operands)
__device__ __forceinline__ void two_quotients(float n0, float d0, bool cut0, float n1, float d1, bool cut1, float& q0,
                                              float& q1) {
    q0 = fast_div<float>(n0, d0);
    q1 = fast_div<float>(n1, d1);
    if (cut0) q0 = 0.f;
    if (cut1) q1 = 0.f;
}
__device__ __forceinline__ void two_quotients(double n0, double d0, bool cut0, double n1, double d1, bool cut1,
                                              double& q0, double& q1) {
    if (cut0) d0 = 1.0;
    if (cut1) d1 = 1.0;
    const double inv = reciprocal(d0 * d1);
    q0 = cut0 ? 0.0 : n0 * (d1 * inv);
    q1 = cut1 ? 0.0 : n1 * (d0 * inv);
}

// seg_coeff for a point and its image: k and r0 x a of both (the y component
// of the cross product is common)
template <class T, bool SIGMA>
__device__ __forceinline__ void seg_pair(const RelPair<T>& a, const RelPair<T>& b, T rx, T ry, T rz, T sigma2, T& k0,
                                         T& k1, T& cy, T& cx0, T& cx1, T& cz0, T& cz1) {
    const T px = ry * a.z, pz = ry * a.x;
    cy = rz * a.x - rx * a.z;
    cx0 = px - rz * a.y0;
    cx1 = px - rz * a.y1;
    cz0 = rx * a.y0 - pz;
    cz1 = rx * a.y1 - pz;
    const T cyy = cy * cy;
    const T sq0 = cz0 * cz0 + (cx0 * cx0 + cyy), sq1 = cz1 * cz1 + (cx1 * cx1 + cyy);
    const T abxz = a.x * b.x + a.z * b.z;
    const T ab0 = a.y0 * b.y0 + abxz, ab1 = a.y1 * b.y1 + abxz;
    const T nab0 = a.n0 * b.n0, nab1 = a.n1 * b.n1;
    const T s0 = a.n0 + b.n0, s1 = a.n1 + b.n1;
    constexpr T rcut = Prec<T>::rcut_norm;
    const bool cut0 = below(sq0, (T)RCUT_SQ) | below(a.n0, rcut) | below(b.n0, rcut);
    const bool cut1 = below(sq1, (T)RCUT_SQ) | below(a.n1, rcut) | below(b.n1, rcut);
    const bool pos0 = not_negative(ab0), pos1 = not_negative(ab1);
    T num0, num1, den0, den1;
    if constexpr (sizeof(T) == 8) {
        // nab + |ab| serves both signs of ab: two fp64 additions less
        const T e0 = nab0 + fabs(ab0), e1 = nab1 + fabs(ab1);
        num0 = s0 * (pos0 ? (T)1 : e0), num1 = s1 * (pos1 ? (T)1 : e1);
        den0 = nab0 * (pos0 ? e0 : sq0), den1 = nab1 * (pos1 ? e1 : sq1);
    } else {
        num0 = pos0 ? s0 : s0 * (nab0 - ab0), num1 = pos1 ? s1 : s1 * (nab1 - ab1);
        den0 = nab0 * (pos0 ? nab0 + ab0 : sq0), den1 = nab1 * (pos1 ? nab1 + ab1 : sq1);
    }
    if (SIGMA) {
        const T sm = sigma2 * (rx * rx + ry * ry + rz * rz);
        num0 *= sq0;
        num1 *= sq1;
        den0 *= dsqrt<T>(sq0 * sq0 + sm * sm);
        den1 *= dsqrt<T>(sq1 * sq1 + sm * sm);
    }
    two_quotients(num0, den0, cut0, num1, den1, cut1, k0, k1);
}

// four consecutive values in one or two 16-byte loads
template <class T> struct alignas(16) Quad { T x, y, z, w; };

// A piece of a lattice in shared memory: nl <= LR vertex lines of nk + 1
// vertices, line l's vertex k at [l * W + k].
//   v: position, and the net strength of the spanwise segment k-1 -> k
//   s: that segment's vector, and the net strength of the chordwise segment
//      from this line to the next at k
//   c: the chordwise segment's vector
// Calls add(g, k0, k1, cy, cx0, cx1, cz0, cz1) for every segment of strength
// g.  The spanwise segments of the last line belong to the next piece unless
// `last`, the chordwise ones of vertex 0 to the piece before unless `first`.
// FULL: nl == LR, known to the compiler, so a vertex column is straight code.
template <class T, bool SIGMA, int LR, bool FULL, class F>
__device__ __forceinline__ void lattice_walk(const Quad<T>* v, const Quad<T>* s, const Quad<T>* c, int W, int nl, int nk,
                                             bool first, bool last, T px, T py, T pz, T sg, F&& add) {
    RelPair<T> prev[LR];
    T k0, k1, cy, cx0, cx1, cz0, cz1;
#pragma unroll
    for (int l = 0; l < LR; l++)
        if (FULL || l < nl) {
            const Quad<T> q = v[l * W];
            prev[l] = make_rel_pair<T>(px, py, pz, q.x, q.y, q.z);
            if (l > 0 && first) {
                const Quad<T> e = c[(l - 1) * W];
                seg_pair<T, SIGMA>(prev[l > 0 ? l - 1 : 0], prev[l], e.x, e.y, e.z, sg, k0, k1, cy, cx0, cx1, cz0, cz1);
                add(s[(l - 1) * W].w, k0, k1, cy, cx0, cx1, cz0, cz1);
            }
        }
#pragma unroll 1
    for (int k = 1; k <= nk; k++) {
        RelPair<T> up = prev[0];
        T gup = 0;
#pragma unroll
        for (int l = 0; l < LR; l++)
            if (FULL || l < nl) {
                const Quad<T> q = v[l * W + k], e = s[l * W + k];
                const RelPair<T> cur = make_rel_pair<T>(px, py, pz, q.x, q.y, q.z);
                if ((FULL ? l + 1 < LR : l + 1 < nl) || last) {
                    seg_pair<T, SIGMA>(prev[l], cur, e.x, e.y, e.z, sg, k0, k1, cy, cx0, cx1, cz0, cz1);
                    add(q.w, k0, k1, cy, cx0, cx1, cz0, cz1);
                }
                if (l > 0) {
                    const Quad<T> d = c[(l - 1) * W + k];
                    seg_pair<T, SIGMA>(up, cur, d.x, d.y, d.z, sg, k0, k1, cy, cx0, cx1, cz0, cz1);
                    add(gup, k0, k1, cy, cx0, cx1, cz0, cz1);
                }
                up = cur;
                gup = e.w;
                prev[l] = cur;
            }
    }
}

// Every ring of a lattice piece (laid out as for lattice_walk, at most LR - 1
// ring rows) at unit strength: calls emit(row, ring, 4 pi (v . n + v_image .
// n_image)).  A segment is evaluated once, forward, for the two rings it bounds,
// so a ring's value does not depend on how the lattice was cut into pieces.
template <class T, bool SIGMA, int LR, class F>
__device__ __forceinline__ void lattice_rings(const Quad<T>* v, const Quad<T>* s, const Quad<T>* c, int W, int nl, int nk,
                                              T px, T py, T pz, T nx, T ny, T nz, T sg, F&& emit) {
    RelPair<T> prev[LR];
    T left[LR - 1];  // the chordwise segments of the vertex before
    auto seg = [&](const RelPair<T>& a, const RelPair<T>& b, const Quad<T>& e) {
        T k0, k1, cy, cx0, cx1, cz0, cz1;
        seg_pair<T, SIGMA>(a, b, e.x, e.y, e.z, sg, k0, k1, cy, cx0, cx1, cz0, cz1);
        const T tn = cy * ny;
        return k0 * (cx0 * nx + tn + cz0 * nz) + k1 * (cx1 * nx - tn + cz1 * nz);
    };
#pragma unroll
    for (int l = 0; l < LR; l++)
        if (l < nl) {
            const Quad<T> q = v[l * W];
            prev[l] = make_rel_pair<T>(px, py, pz, q.x, q.y, q.z);
            if (l > 0) left[l - 1] = seg(prev[l > 0 ? l - 1 : 0], prev[l], c[(l - 1) * W]);
        }
#pragma unroll 1
    for (int k = 1; k <= nk; k++) {
        RelPair<T> up = prev[0];
        T above = 0;
#pragma unroll
        for (int l = 0; l < LR; l++)
            if (l < nl) {
                const Quad<T> q = v[l * W + k];
                const RelPair<T> cur = make_rel_pair<T>(px, py, pz, q.x, q.y, q.z);
                const T span = seg(prev[l], cur, s[l * W + k]);
                if (l > 0) {
                    const T right = seg(up, cur, c[(l - 1) * W + k]);
                    emit(l - 1, k - 1, (above - span) + (right - left[l - 1]));
                    left[l - 1] = right;
                }
                up = cur;
                above = span;
                prev[l] = cur;
            }
    }
}

}  // namespace gbvlm
