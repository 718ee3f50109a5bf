// Host drivers above the operator C ABI: the steady VLM simulation
// (vlm/src/vlm.cpp:17-151), the nonlinear VLM (vlm.cpp:153-295) and the
// plot3d reader (vlm/src/vlm_mesh.cpp).
// These are the per-solve paths, in float (the reference's semantics) or double:
// AIC assembly, factorisation and solve are the operators of the C ABI, and what
// lies around them is one launch before the assembly (wake, pose, metrics), one
// before the solve (right-hand side) and one after it (circulation, forces and
// every sum), read back together.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <fstream>
#include <string>
#include <vector>

#include "gbvlm_internal.h"
#include "gbvlm_loads.cuh"

namespace gbvlm {

template <class T>
struct SteadyArgs {
    int32_t n = 0;
    int64_t ns[GBVLM_MAX_SURFACES], nc[GBVLM_MAX_SURFACES];
    int64_t poff[GBVLM_MAX_SURFACES + 1], soff[GBVLM_MAX_SURFACES + 1];  // first panel, first strip
    const T* vinit[GBVLM_MAX_SURFACES];
    T *verts[GBVLM_MAX_SURFACES], *wake[GBVLM_MAX_SURFACES], *colloc[GBVLM_MAX_SURFACES],
        *normals[GBVLM_MAX_SURFACES], *areas[GBVLM_MAX_SURFACES];
    T* rhs = nullptr;          // right-hand side, then the solution
    T* strip = nullptr;        // angles of the strips (nonlinear)
    double* part = nullptr;    // [blocks][LOAD_PART]
    double* out = nullptr;     // [n][7]: lift, area, moment x, y, z, chord numerator, drag sum
    unsigned* done = nullptr;  // blocks finished, zero between launches
    T tr[16];                  // pose of every surface
    T factor = 0;              // collocation point's share of the chord
    T V[3], la[3], ref[3];     // panel velocity, lift axis, moment point
    T sigma = 0;

    __device__ __forceinline__ int surf(int64_t g) const {
        int m = 0;
        while (m + 1 < n && g >= poff[m + 1]) m++;
        return m;
    }
};

// the wake row from the trailing edge at rest to that of the moved wing, the
// moved wing and its metrics (wake_shed, displace, wake_shed, mesh_metrics)
template <class T>
__global__ void __launch_bounds__(LOAD_THREADS) k_vlm_place(SteadyArgs<T> a) {
    const int64_t g = blockIdx.x * (int64_t)LOAD_THREADS + threadIdx.x;
    if (g < a.poff[a.n]) {
        const int m = a.surf(g);
        move_panel(a.vinit[m], a.verts[m], a.tr, a.ns[m], a.nc[m], g - a.poff[m], a.factor, a.colloc[m], a.normals[m],
                   a.areas[m]);
        return;
    }
    int64_t r = g - a.poff[a.n];
    for (int m = 0; m < a.n; m++) {
        const int64_t nv = a.ns[m] + 1;
        if (r < nv) {
            const int64_t vld = nv * (a.nc[m] + 1), q = r + a.nc[m] * nv;
            T y[4];
            move_vertex(a.vinit[m], vld, q, a.tr, y);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                a.wake[m][2 * k * nv + r] = y[k];
                a.wake[m][2 * k * nv + nv + r] = a.vinit[m][k * vld + q];
            }
            return;
        }
        r -= nv;
    }
}

// right-hand side -V . n: V the free stream, or with strip angles theirs
// (vlm.cpp:186-196: freestream(u_inf, alpha_strip, 0))
template <class T>
__global__ void __launch_bounds__(LOAD_THREADS) k_vlm_rhs(SteadyArgs<T> a, bool strips, T u) {
    const int64_t g = blockIdx.x * (int64_t)LOAD_THREADS + threadIdx.x;
    if (g >= a.poff[a.n]) return;
    const int m = a.surf(g);
    const int64_t p = g - a.poff[m], np = a.ns[m] * a.nc[m];
    const T* n = a.normals[m];
    T V[3] = {a.V[0], a.V[1], a.V[2]};
    if (strips) {
        const T al = a.strip[a.soff[m] + p % a.ns[m]];
        V[0] = u * cos(al);
        V[1] = 0;
        V[2] = u * sin(al);
    }
    a.rhs[g] = (T)0 + -(V[0] * n[p] + V[1] * n[np + p] + V[2] * n[2 * np + p]);
}

// the steady force on the bound segment of panel (i, j) (vlm_backend_cpu.cpp:276-297), rho = 1
template <class T>
__device__ __forceinline__ V3<T> steady_force(const T* x, const T* v, int64_t ns, int64_t nc, int64_t i, int64_t j,
                                              V3<T> V, V3<T>& v0, V3<T>& v1) {
    const int64_t p = i + j * ns, ia = i + j * (ns + 1), ib = ia + 1, vld = (ns + 1) * (nc + 1);
    const T g = x[p], gd = (j > 0) ? g - x[p - ns] : g, rho = 1;
    v0 = V3<T>{v[ia], v[vld + ia], v[2 * vld + ia]};
    v1 = V3<T>{v[ib], v[vld + ib], v[2 * vld + ib]};
    return (rho * gd) * cross(V, v1 - v0);
}

// The sums that the coefficients are made of (vlm_backend.cpp:72-139,
// ispc:273-323) from the solution, one launch: panel blocks, chord blocks, a
// block per wake ring.  all: with the chords and the drag.  alpha: the panel
// velocity u (cos, 0, sin) of it instead of V.  Four sums and the drag by a
// launch and a read-back each took 90 us of a 256-panel case.
template <class T>
__global__ void __launch_bounds__(LOAD_THREADS) k_vlm_loads(SteadyArgs<T> a, bool all, bool from_alpha, T u, T alpha) {
    __shared__ LoadShared sh;
    __shared__ double red[32];
    const int t = threadIdx.x;
    int64_t blk = blockIdx.x;
    int m = 0, kind = 0;
    for (; m < a.n; m++) {
        const int64_t cnt[3] = {(a.ns[m] * a.nc[m] + LOAD_THREADS - 1) / LOAD_THREADS,
                                all ? (a.ns[m] + LOAD_CHORDS - 1) / LOAD_CHORDS : 0, all ? a.ns[m] : 0};
        for (kind = 0; kind < 3; kind++) {
            if (blk < cnt[kind]) break;
            blk -= cnt[kind];
        }
        if (kind < 3) break;
    }
    const int64_t ns = a.ns[m], nc = a.nc[m], np = ns * nc;
    const T *x = a.rhs + a.poff[m], *v = a.verts[m];
    double* part = a.part + LOAD_PART * (int64_t)blockIdx.x;
    if (kind == 0) {
        const int64_t p = blk * LOAD_THREADS + t;
        double s[LOAD_SUMS] = {0, 0, 0, 0, 0};
        if (p < np) {
            V3<T> V{a.V[0], a.V[1], a.V[2]}, v0, v1;
            if (from_alpha) V = V3<T>{u * cos(alpha), (T)0, u * sin(alpha)};
            const int64_t j = p / ns, i = p - j * ns;
            const V3<T> F = steady_force(x, v, ns, nc, i, j, V, v0, v1);
            const double Fx = F.x, Fy = F.y, Fz = F.z;
            s[0] = Fx * a.la[0] + Fy * a.la[1] + Fz * a.la[2];
            s[1] = a.areas[m][p];
            if (all) {
                const double ex = 0.5 * ((double)v0.x + v1.x) - a.ref[0];
                const double ey = 0.5 * ((double)v0.y + v1.y) - a.ref[1];
                const double ez = 0.5 * ((double)v0.z + v1.z) - a.ref[2];
                s[2] = ey * Fz - ez * Fy;
                s[3] = ez * Fx - ex * Fz;
                s[4] = ex * Fy - ey * Fx;
            }
        }
#pragma unroll
        for (int q = 0; q < LOAD_SUMS; q++) sh.s[q][t] = s[q];
        block_sums(sh, LOAD_SUMS, part);
    } else if (kind == 1) {
        chord_terms(sh, v, ns, nc, blk);
        block_sums(sh, 1, part);
    } else {
        const double d = trefftz_ring(ns + 1, (int64_t)2, (const T*)a.wake[m], x + (nc - 1) * ns, a.sigma, blk, red);
        if (t == 0) part[0] = d;
    }
    if (!last_block(sh, a.done)) return;
    int64_t b0 = 0;
    for (int k = 0; k < a.n; k++) {
        const int64_t pb = (a.ns[k] * a.nc[k] + LOAD_THREADS - 1) / LOAD_THREADS;
        const int64_t cb = all ? (a.ns[k] + LOAD_CHORDS - 1) / LOAD_CHORDS : 0, rb = all ? a.ns[k] : 0;
        add_parts(sh, a.part, b0, pb, cb, rb);
        if (t < 7) a.out[7 * k + t] = sh.tot[t];
        b0 += pb + cb + rb;
    }
}

template <class T>
__global__ void k_cast(const float* in, T* out, int64_t n) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = (T)in[i];
}

template <class T>
struct Ops;
#define OPS(T, sfx)                                                                                                  \
    template <>                                                                                                      \
    struct Ops<T> {                                                                                                  \
        static int lhs(T* a, int64_t ld, int32_t ns, const gbvlm_dims* d, const T* const* c, const T* const* n,      \
                       const T* const* vw, const T* const* vk, int32_t it, T sg, gbvlm_stream s) {                    \
            return gbvlm_lhs_assemble_##sfx(a, ld, ns, d, c, n, vw, vk, it, sg, s);                                  \
        }                                                                                                            \
        static int factor(gbvlm_lu h, T* a, int64_t n, gbvlm_stream s) { return gbvlm_lu_factor_##sfx(h, a, n, n, s); } \
        static int solve(gbvlm_lu h, const T* a, int64_t n, T* x, gbvlm_stream s) {                                  \
            return gbvlm_lu_solve_##sfx(h, a, n, n, x, n, 1, s);                                                     \
        }                                                                                                            \
    };
OPS(float, f32)
OPS(double, f64)

// Per-precision simulation state of a steady VLM (vlm/src/vlm.cpp:60-95).
struct VlmBase {
    virtual ~VlmBase() = default;
    virtual int run(double alpha, double beta, double u_inf, double rho, const double* ref_pt, gbvlm_coeffs* out,
                    double* gamma_out, cudaStream_t st) = 0;
    virtual int run_shared(int32_t nalpha, const double* alphas, double u_inf, double rho, const double* ref_pt,
                           gbvlm_coeffs* out, double* gamma_out, cudaStream_t st) = 0;
};

template <class T>
struct VlmState : VlmBase {
    int32_t nsurf = 0;
    std::vector<gbvlm_dims> dims;
    int64_t n = 0;
    void* mem = nullptr;
    std::vector<T*> verts_init, verts, wake, colloc, normals, areas;
    SteadyArgs<T> sa;
    int64_t loads_blocks = 0, lift_blocks = 0;  // of k_vlm_loads with and without the chords and the drag
    T* lhs = nullptr;
    T* rhs = nullptr;
    gbvlm_lu lu = nullptr;
    T sigma = 0;

    ~VlmState() override {
        if (lu) gbvlm_lu_destroy(lu);
        if (mem) cudaFree(mem);
    }

    int init(int32_t ns_, const gbvlm_dims* d, const float* const* vinit_host) {
        nsurf = ns_;
        dims.assign(d, d + ns_);
        size_t bytes = 0;
        n = 0;
        for (auto& x : dims) {
            x.nwv = 2;  // single row of wake panels (vlm.cpp:73)
            int64_t np = x.ns * x.nc, nv = (x.ns + 1) * (x.nc + 1);
            n += np;
            bytes += sizeof(T) * (2 * 4 * nv + 4 * (x.ns + 1) * 2 + 7 * np);
            lift_blocks += cdiv(np, LOAD_THREADS);
            loads_blocks += cdiv(np, LOAD_THREADS) + cdiv(x.ns, LOAD_CHORDS) + x.ns;
        }
        bytes += sizeof(T) * (n * n + n) + 256 * (6 * ns_ + 5) + sizeof(double) * (LOAD_PART * loads_blocks + 7 * ns_);
        GB_CUDA(cudaMalloc(&mem, bytes));
        GB_CUDA(cudaMemset(mem, 0, bytes));
        char* p = (char*)mem;
        auto take = [&](int64_t cnt) {
            T* r = (T*)p;
            p += ((sizeof(T) * cnt + 255) / 256) * 256;
            return r;
        };
        lhs = take(n * n);
        rhs = take(n);
        for (auto& x : dims) {
            int64_t np = x.ns * x.nc, nv = (x.ns + 1) * (x.nc + 1);
            verts_init.push_back(take(4 * nv));
            verts.push_back(take(4 * nv));
            wake.push_back(take(4 * (x.ns + 1) * 2));
            colloc.push_back(take(3 * np));
            normals.push_back(take(3 * np));
            areas.push_back(take(np));
        }
        // upload initial vertices (float host) and set wake w = 1
        for (int m = 0; m < nsurf; m++) {
            int64_t nv = (dims[m].ns + 1) * (dims[m].nc + 1);
            float* tmp = nullptr;
            GB_CUDA(cudaMalloc(&tmp, sizeof(float) * 4 * nv));
            GB_CUDA(cudaMemcpy(tmp, vinit_host[m], sizeof(float) * 4 * nv, cudaMemcpyHostToDevice));
            k_cast<T><<<(unsigned)cdiv(4 * nv, 256), 256>>>(tmp, verts_init[m], 4 * nv);
            GB_LAUNCH_CHECK();
            GB_CUDA(cudaDeviceSynchronize());
            cudaFree(tmp);
            std::vector<T> ones(2 * (dims[m].ns + 1), (T)1);
            GB_CUDA(cudaMemcpy(wake[m] + 3 * 2 * (dims[m].ns + 1), ones.data(), sizeof(T) * ones.size(),
                               cudaMemcpyHostToDevice));
        }
        sa.n = nsurf;
        sa.poff[0] = sa.soff[0] = 0;
        for (int m = 0; m < nsurf; m++) {
            sa.ns[m] = dims[m].ns;
            sa.nc[m] = dims[m].nc;
            sa.poff[m + 1] = sa.poff[m] + dims[m].ns * dims[m].nc;
            sa.soff[m + 1] = sa.soff[m] + dims[m].ns;
            sa.vinit[m] = verts_init[m];
            sa.verts[m] = verts[m];
            sa.wake[m] = wake[m];
            sa.colloc[m] = colloc[m];
            sa.normals[m] = normals[m];
            sa.areas[m] = areas[m];
        }
        sa.rhs = rhs;
        auto take_bytes = [&](size_t b) {
            void* r = p;
            p += (b + 255) / 256 * 256;
            return r;
        };
        sa.part = (double*)take_bytes(sizeof(double) * LOAD_PART * loads_blocks);
        sa.out = (double*)take_bytes(sizeof(double) * 7 * nsurf);
        sa.done = (unsigned*)take_bytes(sizeof(unsigned));
        int rc = gbvlm_lu_create(&lu);
        if (rc) return rc;
        return gbvlm_lu_init(lu, n);
    }

    // FlowData (vlm_utils.cpp:5-19): free stream and lift axis
    static void flow(T alpha, T beta, T u, T* fs, T* la) {
        fs[0] = u * (T)cos(alpha) * (T)cos(beta);
        fs[1] = -(u * (T)cos(alpha) * (T)sin(beta));
        fs[2] = u * (T)sin(alpha);
        la[0] = -fs[2];
        la[1] = (T)0;
        la[2] = fs[0];
        T ll = (T)sqrt(la[0] * la[0] + la[1] * la[1] + la[2] * la[2]);
        la[0] /= ll; la[1] /= ll; la[2] /= ll;
    }

    // Geometry, AIC and its factorisation for the angle alpha (vlm.cpp:97-126):
    // the 100-chord wake row along the free stream, collocation points with the
    // high-AoA factor of alpha; `tr` receives the wake translation.
    int assemble(T alpha, T u, T* tr, gbvlm_stream s, cudaStream_t st) {
        GB_CUDA(cudaMemsetAsync(lhs, 0, sizeof(T) * n * n, st));
        // 100-chord wake (vlm.cpp:104-114)
        const T t16[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, (T)-100 * u * (T)cos(alpha), 0,
                           (T)-100 * u * (T)sin(alpha), 1};
        for (int k = 0; k < 16; k++) tr[k] = t16[k];
        for (int k = 0; k < 16; k++) sa.tr[k] = t16[k];
        sa.factor = aoa_factor(alpha);
        std::vector<const T*> cverts(verts.begin(), verts.end()), ccol(colloc.begin(), colloc.end()),
            cnor(normals.begin(), normals.end()), cwake(wake.begin(), wake.end());
        int64_t cnt = n;
        for (auto& x : dims) cnt += x.ns + 1;
        k_vlm_place<T><<<(unsigned)cdiv(cnt, LOAD_THREADS), LOAD_THREADS, 0, st>>>(sa);
        GB_LAUNCH_CHECK();
        int rc;
        if ((rc = Ops<T>::lhs(lhs, n, nsurf, dims.data(), ccol.data(), cnor.data(), cverts.data(), cwake.data(), 1, sigma, s)))
            return rc;
        return Ops<T>::factor(lu, lhs, n, s);
    }

    // Right-hand side for the free stream fs, the solve, the circulation
    // update and the loads (vlm.cpp:115-151) on the factored AIC.
    int solve_loads(const T* fs, const T* la, T rho, const T* tr, const double* ref_pt, gbvlm_coeffs* out,
                    double* gamma_out, gbvlm_stream s, cudaStream_t st) {
        for (int k = 0; k < 3; k++) {
            sa.V[k] = fs[k];
            sa.la[k] = la[k];
        }
        sa.sigma = (T)sqrt((double)(sigma * sigma));
        k_vlm_rhs<T><<<(unsigned)cdiv(n, LOAD_THREADS), LOAD_THREADS, 0, st>>>(sa, false, (T)0);
        GB_LAUNCH_CHECK();
        int rc;
        if ((rc = Ops<T>::solve(lu, lhs, n, rhs, s))) return rc;
        // coefficient reductions (vlm_backend.cpp:72-139) + Trefftz drag
        // the wing sits displaced by the wake translation; move the moment
        // reference with it so CM is the body-frame moment about ref_pt
        T ref[3] = {(T)(ref_pt ? ref_pt[0] : 0) + tr[12], (T)(ref_pt ? ref_pt[1] : 0) + tr[13],
                    (T)(ref_pt ? ref_pt[2] : 0) + tr[14]};
        for (int k = 0; k < 3; k++) sa.ref[k] = ref[k];
        k_vlm_loads<T><<<(unsigned)loads_blocks, LOAD_THREADS, 0, st>>>(sa, true, false, (T)0, (T)0);
        GB_LAUNCH_CHECK();
        // the sums, the circulations and the solve's error words in one wait
        const size_t sums = sizeof(double) * 7 * nsurf;
        char* h = (char*)host_scratch(16 + sums + sizeof(T) * n);
        GB_REQUIRE(h != nullptr, "pinned host allocation failed");
        const double* r = (const double*)(h + 16);
        const T* g = (const T*)(h + 16 + sums);
        if ((rc = lu_solve_words(lu, (int*)h, st))) return rc;
        GB_CUDA(cudaMemcpyAsync(h + 16, sa.out, sums, cudaMemcpyDeviceToHost, st));
        if (gamma_out) GB_CUDA(cudaMemcpyAsync(h + 16 + sums, rhs, sizeof(T) * n, cudaMemcpyDeviceToHost, st));
        GB_CUDA(cudaStreamSynchronize(st));
        const T v2 = fs[0] * fs[0] + fs[1] * fs[1] + fs[2] * fs[2];
        const double v2d = (double)fs[0] * fs[0] + (double)fs[1] * fs[1] + (double)fs[2] * fs[2];
        T cl = 0, ta = 0, tm = 0, cdn = 0;
        T cm[3] = {0, 0, 0};
        for (int m = 0; m < nsurf; m++, r += 7) {
            const T area = (T)r[1], mac = (T)(r[5] / r[1]);
            const T clm = (T)(r[0] / ((double)((T)0.5 * rho * v2 * area)));
            const double d = (double)((T)0.5 * rho * v2 * area * mac);
            const T cdm = (T)(r[6] / (v2d * (double)area));
            cl += clm * area;
            cdn += cdm * area;
            for (int k = 0; k < 3; k++) cm[k] += (T)(r[2 + k] / d) * area * mac;
            ta += area;
            tm += mac;
        }
        out->cl = (double)(cl / ta);
        out->cdi = (double)(cdn / ta);
        for (int k = 0; k < 3; k++) out->cm[k] = (double)(cm[k] / (ta * tm));
        if (gamma_out)
            for (int64_t i = 0; i < n; i++) gamma_out[i] = (double)g[i];
        return lu_solve_verdict(lu, (const int*)h, st);  // the solve finished its bounded waits
    }

    int run(double alpha_d, double beta_d, double u_inf_d, double rho_d, const double* ref_pt, gbvlm_coeffs* out,
            double* gamma_out, cudaStream_t st) override {
        gbvlm_stream s = (gbvlm_stream)st;
        const T alpha = (T)alpha_d, beta = (T)beta_d, u = (T)u_inf_d, rho = (T)rho_d;
        T fs[3], la[3], tr[16];
        flow(alpha, beta, u, fs, la);
        int rc = assemble(alpha, u, tr, s, st);
        if (rc) return rc;
        return solve_loads(fs, la, rho, tr, ref_pt, out, gamma_out, s, st);
    }

    int run_shared(int32_t nalpha, const double* alphas, double u_inf_d, double rho_d, const double* ref_pt,
                   gbvlm_coeffs* out, double* gamma_out, cudaStream_t st) override {
        gbvlm_stream s = (gbvlm_stream)st;
        const T u = (T)u_inf_d, rho = (T)rho_d;
        T tr[16];
        int rc = assemble((T)0, u, tr, s, st);
        if (rc) return rc;
        for (int32_t k = 0; k < nalpha; k++) {
            T fs[3], la[3];
            flow((T)alphas[k], (T)0, u, fs, la);
            rc = solve_loads(fs, la, rho, tr, ref_pt, out + k, gamma_out ? gamma_out + (int64_t)k * n : nullptr, s, st);
            if (rc) return rc;
        }
        return GBVLM_OK;
    }
};

// ---------------------------------------------------------------------------
// Nonlinear VLM (vlm/src/vlm.cpp:153-295): strip-wise correction of the
// angle of attack toward a 2D lift polar (van Dam's method).  The AIC of the
// wing with its 100-chord wake row is factored once; each iteration runs on
// the device (panel velocities from the strip angles, RHS, solve, gamma
// deltas, forces, strip correction) and the host reads one error per
// surface to decide whether to continue, as the reference's loop does.
// ---------------------------------------------------------------------------

// Akima interpolant (headeronly/tinyinterpolate.hpp:26-73): lower_bound on
// x, the cubic of that interval, the end segment's line outside the table
template <class T>
__device__ T akima_at(const T* x, const T* y, const T* m, const T* s, int n, T xq) {
    int lo = 0, hi = n;  // first index with x[i] >= xq
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (x[mid] < xq) lo = mid + 1;
        else hi = mid;
    }
    if (lo == 0) return y[0] - m[0] * (x[0] - xq);
    if (lo == n) return y[n - 1] + m[n - 2] * (xq - x[n - 1]);
    const int i = lo - 1;
    const T dx = x[i + 1] - x[i], dxx = xq - x[i];
    const T c = ((T)3 * m[i] - (T)2 * s[i] - s[i + 1]) / dx;
    const T d = (s[i] + s[i + 1] - (T)2 * m[i]) / (dx * dx);
    return y[i] + s[i] * dxx + c * dxx * dxx + d * dxx * dxx * dxx;
}

// a strip per thread: its circulation differences and forces, its CL about its
// own lift axis, the effective angle and the correction toward the polar
// (vlm.cpp:257-276); *err = the sum of |correction| over all surfaces
constexpr int STRIP_THREADS = 32;

template <class T>
__global__ void __launch_bounds__(STRIP_THREADS) k_strip_correct(SteadyArgs<T> a, T alpha, T beta, T u, T rho,
                                                                 const T* tx, const T* ty, const T* tm, const T* ts,
                                                                 int ntab, double* err) {
    __shared__ bool last;
    const T two_pi = (T)(2.0f * 3.141593f);  // 2 PI_f with the reference's float pi (vlm_types.hpp:22)
    const int64_t q = blockIdx.x * (int64_t)STRIP_THREADS + threadIdx.x;
    double e = 0;
    if (q < a.soff[a.n]) {
        int m = 0;
        while (m + 1 < a.n && q >= a.soff[m + 1]) m++;
        const int64_t i = q - a.soff[m], ns = a.ns[m], nc = a.nc[m];
        const T* x = a.rhs + a.poff[m];
        const T al = a.strip[q];
        // FlowData of the strip (vlm_utils.cpp:5-19): freestream and lift axis
        const T fx = u * cos(al) * cos(beta), fy = -(u * cos(al) * sin(beta)), fz = u * sin(al);
        T lx = -fz, lz = fx;
        const T ll = sqrt(lx * lx + lz * lz);
        lx /= ll;
        lz /= ll;
        const V3<T> V{u * cos(al), (T)0, u * sin(al)};
        T fl = 0, area = 0;
        for (int64_t j = 0; j < nc; j++) {
            V3<T> v0, v1;
            const V3<T> F = steady_force(x, (const T*)a.verts[m], ns, nc, i, j, V, v0, v1);
            fl += F.x * lx + F.z * lz;  // the lift axis has no y component
            area += a.areas[m][i + j * ns];
        }
        const T cl = fl / ((T)0.5 * rho * (fx * fx + fy * fy + fz * fz) * area);
        const T eff = cl / two_pi - al + alpha;
        const T corr = (akima_at<T>(tx, ty, tm, ts, ntab, eff) - cl) / two_pi;
        a.strip[q] = al + corr;
        e = fabs((double)corr);
    }
    auto lanes = [&](double y) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) y += __shfl_xor_sync(0xffffffffu, y, d);
        return y;
    };
    e = lanes(e);
    if (threadIdx.x == 0) {
        a.part[blockIdx.x] = e;
        __threadfence();
        last = atomicInc(a.done, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    CSum s;
    for (int64_t b = threadIdx.x; b < gridDim.x; b += STRIP_THREADS) s.add(__ldcg(a.part + b));
    e = lanes(s.value());
    if (threadIdx.x == 0) *err = e;
}

template <class T>
__global__ void k_fill(T* v, int64_t n, T x) {
    const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p < n) v[p] = x;
}

struct NlvlmBase {
    virtual ~NlvlmBase() = default;
    virtual int run(double alpha, double beta, double u_inf, double rho, const float* db_alpha, const float* db_cl,
                    int32_t ndb, double tol, int32_t max_iter, double* cl, int32_t* iters, double* err,
                    float* strip_out, cudaStream_t st) = 0;
    virtual gbvlm_lu solver() = 0;
};

template <class T>
struct NlvlmState : NlvlmBase {
    VlmState<T> w;  // wing, wake, AIC and per-panel buffers of the steady simulation
    gbvlm_lu solver() override { return w.lu; }
    void* mem = nullptr;
    T* strip = nullptr;  // angles, all surfaces' strips
    int64_t strips = 0;
    double* d_err = nullptr;
    T* tab = nullptr;  // x, y, m, s of the polar
    int32_t tab_cap = 0;

    ~NlvlmState() override {
        if (mem) cudaFree(mem);
        if (tab) cudaFree(tab);
    }

    int init(int32_t ns_, const gbvlm_dims* d, const float* const* vinit) {
        int rc = w.init(ns_, d, vinit);
        if (rc) return rc;
        for (auto& x : w.dims) strips += x.ns;
        GB_CUDA(cudaMalloc(&mem, 256 + sizeof(T) * strips));
        d_err = (double*)mem;
        strip = (T*)((char*)mem + 256);
        w.sa.strip = strip;
        return GBVLM_OK;
    }

    int run(double alpha_d, double beta_d, double u_inf_d, double rho_d, const float* db_alpha, const float* db_cl,
            int32_t ndb, double tol, int32_t max_iter, double* cl_out, int32_t* iters_out, double* err_out,
            float* strip_out, cudaStream_t st) override {
        gbvlm_stream s = (gbvlm_stream)st;
        const int32_t nsurf = w.nsurf;
        const T alpha = (T)alpha_d, beta = (T)beta_d, u = (T)u_inf_d, rho = (T)rho_d;
        // the polar's Akima coefficients (tinyinterpolate.hpp:29-54), as the reference builds them on the host
        std::vector<T> table(4 * ndb);  // x, y, m, s as in `tab`
        T *tx = table.data(), *ty = tx + ndb, *tm = ty + ndb, *ts = tm + ndb;
        for (int i = 0; i < ndb; i++) {
            tx[i] = (T)db_alpha[i];
            ty[i] = (T)db_cl[i];
            GB_REQUIRE(i == 0 || tx[i] > tx[i - 1], "NLVLM: polar angles must increase");
        }
        for (int i = 0; i + 1 < ndb; i++) tm[i] = (ty[i + 1] - ty[i]) / (tx[i + 1] - tx[i]);
        ts[0] = tm[0];
        ts[1] = (T)0.5 * (tm[0] + tm[1]);
        for (int i = 2; i < ndb - 2; i++) {
            const T d1 = std::abs(tm[i + 1] - tm[i]), d2 = std::abs(tm[i - 1] - tm[i - 2]);
            ts[i] = d1 + d2 > (T)0 ? (d1 * tm[i - 1] + d2 * tm[i]) / (d1 + d2) : (T)0.5 * (tm[i] + tm[i - 1]);
        }
        ts[ndb - 2] = (T)0.5 * (tm[ndb - 3] + tm[ndb - 2]);
        ts[ndb - 1] = tm[ndb - 2];
        if (tab_cap < ndb) {
            if (tab) cudaFree(tab);
            tab = nullptr;
            GB_CUDA(cudaMalloc(&tab, sizeof(T) * 4 * ndb));
            tab_cap = ndb;
        }
        T* dx = tab;
        T* dy = tab + ndb;
        T* dm = tab + 2 * ndb;
        T* dsp = tab + 3 * ndb;
        GB_CUDA(cudaMemcpyAsync(tab, tx, sizeof(T) * 4 * ndb, cudaMemcpyHostToDevice, st));  // (pageable: staged at return)
        // the wing with its 100-chord wake row and the factored AIC (vlm.cpp:201-217)
        T tr[16];
        int rc;
        if ((rc = w.assemble(alpha, u, tr, s, st))) return rc;
        k_fill<T><<<(unsigned)cdiv(strips, 128), 128, 0, st>>>(strip, strips, alpha);
        GB_LAUNCH_CHECK();
        // the corrections' sum, the load sums, the solves' error words, the strips
        double* herr = (double*)host_scratch(sizeof(double) * (2 + 7 * nsurf) + sizeof(T) * strips);
        GB_REQUIRE(herr != nullptr, "pinned host allocation failed");
        double err = 1.0;
        int32_t it = 0;
        for (; it < max_iter && err > tol; it++) {
            k_vlm_rhs<T><<<(unsigned)cdiv(w.n, LOAD_THREADS), LOAD_THREADS, 0, st>>>(w.sa, true, u);
            GB_LAUNCH_CHECK();
            if ((rc = Ops<T>::solve(w.lu, w.lhs, w.n, w.rhs, s))) return rc;
            k_strip_correct<T><<<(unsigned)cdiv(strips, STRIP_THREADS), STRIP_THREADS, 0, st>>>(
                w.sa, alpha, beta, u, rho, dx, dy, dm, dsp, ndb, d_err);
            GB_LAUNCH_CHECK();
            GB_CUDA(cudaMemcpyAsync(herr, d_err, sizeof(double), cudaMemcpyDeviceToHost, st));
            GB_CUDA(cudaStreamSynchronize(st));
            err = *herr;
            err /= (double)w.n;  // per panel, as the reference normalises
        }
        int* words = (int*)(herr + 1 + 7 * nsurf);
        T* hs = (T*)(herr + 2 + 7 * nsurf);
        if (strip_out) GB_CUDA(cudaMemcpyAsync(hs, strip, sizeof(T) * strips, cudaMemcpyDeviceToHost, st));
        // final loads with the strips back at alpha (vlm.cpp:281-291)
        T fs[3] = {u * (T)cos(alpha) * (T)cos(beta), -(u * (T)cos(alpha) * (T)sin(beta)), u * (T)sin(alpha)};
        T la[3] = {-fs[2], (T)0, fs[0]};
        const T ll = (T)sqrt(la[0] * la[0] + la[2] * la[2]);
        la[0] /= ll;
        la[2] /= ll;
        for (int k = 0; k < 3; k++) w.sa.la[k] = la[k];
        k_vlm_loads<T><<<(unsigned)w.lift_blocks, LOAD_THREADS, 0, st>>>(w.sa, false, true, u, alpha);
        GB_LAUNCH_CHECK();
        GB_CUDA(cudaMemcpyAsync(herr + 1, w.sa.out, sizeof(double) * 7 * nsurf, cudaMemcpyDeviceToHost, st));
        if ((rc = lu_solve_words(w.lu, words, st))) return rc;
        GB_CUDA(cudaStreamSynchronize(st));
        if (strip_out)
            for (int64_t i = 0; i < strips; i++) strip_out[i] = (float)hs[i];
        const T v2 = fs[0] * fs[0] + fs[1] * fs[1] + fs[2] * fs[2];
        T cl = 0, ta = 0;
        for (int m = 0; m < nsurf; m++) {
            const double* r = herr + 1 + 7 * m;
            const T area = (T)r[1];
            cl += (T)(r[0] / ((double)((T)0.5 * rho * v2 * area))) * area;
            ta += area;
        }
        *cl_out = (double)(cl / ta);
        if (iters_out) *iters_out = it;
        if (err_out) *err_out = err;
        return lu_solve_verdict(w.lu, words, st);  // the solves finished their bounded waits
    }
};

}  // namespace gbvlm

using namespace gbvlm;

struct gbvlm_vlm_s {
    VlmBase* impl = nullptr;
};

struct gbvlm_nlvlm_s {
    NlvlmBase* impl = nullptr;
};

extern "C" {

int gbvlm_vlm_create(gbvlm_vlm* out, int32_t nsurf, const gbvlm_dims* dims, const float* const* verts_init,
                     int32_t precision) {
    GB_REQUIRE(out && dims && verts_init, "null argument");
    GB_REQUIRE(nsurf >= 1 && nsurf <= GBVLM_MAX_SURFACES, "nsurf=%d outside [1, %d]", nsurf, GBVLM_MAX_SURFACES);
    GB_REQUIRE(precision == 32 || precision == 64, "precision must be 32 or 64");
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(verts_init[m], "verts_init[%d] is null", m);
        GB_REQUIRE(dims[m].ns >= 1 && dims[m].nc >= 1, "surface %d has bad sizes", m);
    }
    auto* h = new gbvlm_vlm_s();
    int rc;
    if (precision == 32) {
        auto* s = new VlmState<float>();
        h->impl = s;
        rc = s->init(nsurf, dims, verts_init);
    } else {
        auto* s = new VlmState<double>();
        h->impl = s;
        rc = s->init(nsurf, dims, verts_init);
    }
    if (rc) {
        delete h->impl;
        delete h;
        return rc;
    }
    *out = h;
    return GBVLM_OK;
}

int gbvlm_vlm_destroy(gbvlm_vlm h) {
    if (!h) return GBVLM_OK;
    delete h->impl;
    delete h;
    return GBVLM_OK;
}

int gbvlm_vlm_run(gbvlm_vlm h, double alpha, double beta, double u_inf, double rho, const double* ref_pt,
                  gbvlm_coeffs* out, double* gamma_out, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl && out, "null argument");
    return h->impl->run(alpha, beta, u_inf, rho, ref_pt, out, gamma_out, to_cuda(stream));
}

int gbvlm_vlm_run_shared(gbvlm_vlm h, int32_t nalpha, const double* alphas, double u_inf, double rho,
                         const double* ref_pt, gbvlm_coeffs* out, double* gamma_out, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl && out && alphas, "null argument");
    GB_REQUIRE(nalpha >= 1, "nalpha=%d < 1", nalpha);
    return h->impl->run_shared(nalpha, alphas, u_inf, rho, ref_pt, out, gamma_out, to_cuda(stream));
}

int gbvlm_nlvlm_create(gbvlm_nlvlm* out, int32_t nsurf, const gbvlm_dims* dims, const float* const* verts_init,
                       int32_t precision) {
    GB_REQUIRE(out && dims && verts_init, "null argument");
    GB_REQUIRE(nsurf >= 1 && nsurf <= GBVLM_MAX_SURFACES, "nsurf=%d outside [1, %d]", nsurf, GBVLM_MAX_SURFACES);
    GB_REQUIRE(precision == 32 || precision == 64, "precision must be 32 or 64");
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(verts_init[m], "verts_init[%d] is null", m);
        GB_REQUIRE(dims[m].ns >= 1 && dims[m].nc >= 1, "surface %d has bad sizes", m);
    }
    auto* h = new gbvlm_nlvlm_s();
    int rc;
    if (precision == 32) {
        auto* st = new NlvlmState<float>();
        h->impl = st;
        rc = st->init(nsurf, dims, verts_init);
    } else {
        auto* st = new NlvlmState<double>();
        h->impl = st;
        rc = st->init(nsurf, dims, verts_init);
    }
    if (rc) {
        delete h->impl;
        delete h;
        return rc;
    }
    *out = h;
    return GBVLM_OK;
}

int gbvlm_nlvlm_destroy(gbvlm_nlvlm h) {
    if (!h) return GBVLM_OK;
    delete h->impl;
    delete h;
    return GBVLM_OK;
}

int gbvlm_nlvlm_run(gbvlm_nlvlm h, double alpha, double beta, double u_inf, double rho, const float* db_alpha,
                    const float* db_cl, int32_t n_db, double tol, int32_t max_iter, double* cl, int32_t* iters,
                    double* err, float* strip_alpha, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl && db_alpha && db_cl && cl, "null argument");
    GB_REQUIRE(n_db >= 4, "NLVLM: the polar needs at least 4 points (Akima), got %d", n_db);
    GB_REQUIRE(max_iter >= 0, "NLVLM: max_iter must be non-negative");
    return h->impl->run(alpha, beta, u_inf, rho, db_alpha, db_cl, n_db, tol, max_iter, cl, iters, err, strip_alpha,
                        to_cuda(stream));
}

int gbvlm_test_nlvlm_withhold(gbvlm_nlvlm h, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl, "null argument");
    return gbvlm_test_lu_withhold(h->impl->solver(), stream);
}

int gbvlm_read_plot3d(const char* path, int32_t quarter_chord, gbvlm_dims* dims, float* verts) {
    GB_REQUIRE(path && dims, "null argument");
    std::ifstream f(path);
    if (!f.is_open()) {
        set_error("Failed to open mesh file %s", path);
        return GBVLM_ERR_IO;
    }
    long long blocks = 0, ni = 0, nj = 0, nk = 0;
    f >> blocks;
    if (blocks != 1) {
        set_error("Only single block plot3d mesh is supported");
        return GBVLM_ERR_IO;
    }
    f >> ni >> nj >> nk;
    if (nk != 1 || ni < 2 || nj < 2 || !f) {
        set_error("Only 2D plot3d mesh is supported");
        return GBVLM_ERR_IO;
    }
    dims->nc = ni - 1;
    dims->ns = nj - 1;
    dims->nwv = 0;
    if (!verts) return GBVLM_OK;
    // reference tensor (nj, ni, 4): span index fastest (vlm_mesh.cpp:61-78)
    const int64_t nv = ni * nj;
    for (int k = 0; k < 3; k++) {
        for (long long j = 0; j < nj; j++) {
            for (long long i = 0; i < ni; i++) {
                double x;
                if (!(f >> x)) {
                    set_error("plot3d file %s ended early", path);
                    return GBVLM_ERR_IO;
                }
                verts[k * nv + j + i * nj] = (float)x;
            }
        }
    }
    for (int64_t q = 0; q < nv; q++) verts[3 * nv + q] = 1.0f;
    const float first_y = verts[nv];
    for (long long i = 1; i < ni; i++) {
        if (verts[nv + i * nj] != first_y) {
            set_error("Mesh vertices should be ordered in chordwise direction");
            return GBVLM_ERR_IO;
        }
    }
    if (quarter_chord) {
        // vlm_mesh.cpp:16-32
        for (long long i = 0; i + 1 < ni; i++)
            for (long long j = 0; j < nj; j++)
                for (int k = 0; k < 3; k++) {
                    float* a = &verts[k * nv + j + i * nj];
                    a[0] = 0.75f * a[0] + 0.25f * a[nj];
                }
        const long long i = ni - 2;
        for (long long j = 0; j < nj; j++)
            for (int k = 0; k < 3; k++) {
                float* a = &verts[k * nv + j + i * nj];
                a[nj] = (4.f / 3.f) * a[nj] - (1.f / 3.f) * a[0];
            }
    }
    return GBVLM_OK;
}

}  // extern "C"
