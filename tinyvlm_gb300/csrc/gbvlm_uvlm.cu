// Unsteady VLM driver (vlm/src/vlm.cpp:297-509) with the whole time loop on
// the device.  The caller evaluates each surface's kinematic transform and
// its time derivative at t_i = i dt (the reference does this on the host
// with forward-mode dual numbers, vlm/include/vlm_kinematics.hpp:215-239)
// and uploads all steps at once; the loop then runs without host
// round-trips: CL(t) and CM(t) land in device arrays read at the end.
//
// Per step i (t = i dt), as UVLM::run:
//   wake_shed(i); V_p = -dT(t)/dt [c0_p, 1] at the t = 0 collocation points;
//   rhs = -V.n - wake influence (i rows); LU solve (AIC factored once at
//   t = 0 without wake); gamma, gamma_delta, dgamma/dt, TE gamma shed to the
//   wake; for i > 0 unsteady forces, CL and CM about ref(t); optional free-
//   wake roll-up (the reference's kernel_rollup, whose caller it disables);
//   move to t + dt and recompute the panel metrics.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <atomic>
#include <chrono>
#include <mutex>
#include <thread>
#include <type_traits>
#include <vector>

#include "gbvlm_internal.h"
#include "gbvlm_loads.cuh"
#include "gbvlm_math.cuh"

namespace gbvlm {

// ---------------------------------------------------------------------------
// The elementwise parts of a time step, three launches per step whatever the
// number of surfaces (they were about ten, each of one or two microseconds of
// work and as much again of launch):
//   k_step_start  wake shed, panel velocities, the kinematic right-hand side;
//   k_step_loads  circulation, forces, CL and CM of the solution;
//   k_step_move   wing to its next pose, panel metrics.
// The step index is `step`, or idx[0] when idx is set (graphs replayed for any
// step).  by_step: the transforms, free streams, moment points and records are
// indexed by the step; otherwise they are the caller's current ones.
// ---------------------------------------------------------------------------
template <class T>
struct StepArgs {
    int32_t n = 0;
    int64_t ns[GBVLM_MAX_SURFACES], nc[GBVLM_MAX_SURFACES];
    int64_t poff[GBVLM_MAX_SURFACES + 1];  // first panel of each surface
    const T* vpos[GBVLM_MAX_SURFACES];     // vertices that the transforms move
    const T* colloc0[GBVLM_MAX_SURFACES];  // collocation points that the velocities belong to
    T *verts[GBVLM_MAX_SURFACES], *wake[GBVLM_MAX_SURFACES], *vel[GBVLM_MAX_SURFACES], *colloc[GBVLM_MAX_SURFACES],
        *normals[GBVLM_MAX_SURFACES], *areas[GBVLM_MAX_SURFACES], *gamma[GBVLM_MAX_SURFACES],
        *gprev[GBVLM_MAX_SURFACES], *gwake[GBVLM_MAX_SURFACES];
    int64_t nwv = 0;                        // wake vertex rows
    T* rhs = nullptr;                       // right-hand side
    const T* sol = nullptr;                 // solution (rhs itself after a solve in place)
    const T *Tm = nullptr, *Tdm = nullptr;  // [step][surface][16] column-major
    const T *fs = nullptr, *ref = nullptr;  // [step][3]
    double* out = nullptr;                  // [step][4]: CL, CM
    T inv_dt = 0;
    double rho = 1;
    double* part = nullptr;    // [step_load_blocks][LOAD_PART]
    unsigned* done = nullptr;  // blocks finished, zero between launches
    const int64_t* idx = nullptr;
    bool by_step = true;
    bool keep = true;   // gprev = gamma after use
    bool flap = false;  // the second surface's leading row carries the first's trailing-edge circulation off

    __device__ __forceinline__ int64_t at(int64_t step) const { return idx ? idx[0] : step; }
    __device__ __forceinline__ int surf(int64_t g) const {
        int m = 0;
        while (m + 1 < n && g >= poff[m + 1]) m++;
        return m;
    }
};

constexpr int STEP_THREADS = LOAD_THREADS;

template <class T>
static void step_dims(StepArgs<T>& a, const std::vector<gbvlm_dims>& dims) {
    a.n = (int32_t)dims.size();
    a.poff[0] = 0;
    for (int m = 0; m < a.n; m++) {
        a.ns[m] = dims[m].ns;
        a.nc[m] = dims[m].nc;
        a.poff[m + 1] = a.poff[m] + dims[m].ns * dims[m].nc;
    }
}

static int64_t step_load_blocks(const std::vector<gbvlm_dims>& dims) {
    int64_t b = 0;
    for (auto& d : dims) b += cdiv(d.ns * d.nc, STEP_THREADS) + cdiv(d.ns, LOAD_CHORDS);
    return b;
}

template <class T>
__global__ void __launch_bounds__(STEP_THREADS) k_step_start(StepArgs<T> a, int64_t step) {
    const int64_t i = a.at(step), g = blockIdx.x * (int64_t)STEP_THREADS + threadIdx.x;
    const T* Tdm = a.Tdm + (a.by_step ? 16 * a.n * i : 0);
    if (g < a.poff[a.n]) {
        const int m = a.surf(g);
        const int64_t p = g - a.poff[m], np = a.ns[m] * a.nc[m];
        const T *c0 = a.colloc0[m], *n = a.normals[m], *Td = Tdm + 16 * m;
        T* vel = a.vel[m];
        const T x = c0[p], y = c0[np + p], z = c0[2 * np + p];
        T v[3];
        // -(dT/dt) [x y z 1]
#pragma unroll
        for (int r = 0; r < 3; r++) {
            v[r] = -(Td[r] * x + Td[r + 4] * y + Td[r + 8] * z + Td[r + 12]);
            vel[r * np + p] = v[r];
        }
        a.rhs[g] = (T)0 + -(v[0] * n[p] + v[1] * n[np + p] + v[2] * n[2 * np + p]);
        return;
    }
    // trailing edge to wake row i
    int64_t r = g - a.poff[a.n];
    for (int m = 0; m < a.n; m++) {
        const int64_t nv = a.ns[m] + 1;
        if (r < 4 * nv) {
            const int64_t k = r / nv, q = r - k * nv;
            if (i >= 0 && i < a.nwv)
                a.wake[m][k * nv * a.nwv + q + (a.nwv - 1 - i) * nv] =
                    a.verts[m][k * nv * (a.nc[m] + 1) + q + a.nc[m] * nv];
            return;
        }
        r -= 4 * nv;
    }
}

// verts = T vpos and the metrics of the moved panels, the collocation point at 3/4 chord
template <class T>
__global__ void __launch_bounds__(STEP_THREADS) k_step_move(StepArgs<T> a, int64_t step) {
    const int64_t g = blockIdx.x * (int64_t)STEP_THREADS + threadIdx.x;
    if (g >= a.poff[a.n]) return;
    const int m = a.surf(g);
    const T* tr = a.Tm + (a.by_step ? 16 * a.n * (a.at(step) + 1) : 0) + 16 * m;
    move_panel(a.vpos[m], a.verts[m], tr, a.ns[m], a.nc[m], g - a.poff[m], (T)0.5, a.colloc[m], a.normals[m],
               a.areas[m]);
}

// Circulation of the solution (gamma, the trailing edge's into the wake), with
// `loads` the unsteady forces (vlm_backend_cpu.cpp:276-321) and the multibody
// CL and CM about ref (vlm/src/vlm_backend.cpp:72-139): the sums in double,
// out[0] cl and out[1..3] cm.  The sums over all panels in a single block took
// 70 us a step for 1600 panels.
template <class T>
__global__ void __launch_bounds__(STEP_THREADS) k_step_loads(StepArgs<T> a, int64_t step, bool loads) {
    __shared__ LoadShared sh;
    const int64_t it = a.at(step), o = a.by_step ? it : 0;
    const int t = threadIdx.x;
    const T *fsp = a.fs + 3 * o, *rp = a.ref + 3 * o;
    int64_t blk = blockIdx.x;
    int m = 0;
    bool chords = false;
    for (; m < a.n; m++) {
        const int64_t pb = (a.ns[m] * a.nc[m] + STEP_THREADS - 1) / STEP_THREADS;
        const int64_t cb = loads ? (a.ns[m] + LOAD_CHORDS - 1) / LOAD_CHORDS : 0;
        if (blk < pb) break;
        blk -= pb;
        if (blk < cb) {
            chords = true;
            break;
        }
        blk -= cb;
    }
    const int64_t ns = a.ns[m], nc = a.nc[m], np = ns * nc, vld = (ns + 1) * (nc + 1);
    const T* v = a.verts[m];
    if (!chords) {
        const int64_t p = blk * STEP_THREADS + t;
        double s[LOAD_SUMS] = {0, 0, 0, 0, 0};
        if (p < np) {
            const int64_t j = p / ns, i = p - j * ns;
            const T* x = a.sol + a.poff[m];
            const T g = x[p];
            a.gamma[m][p] = g;
            const int64_t wcol = a.nwv - 2 - it;
            if (j == nc - 1 && wcol >= 0 && wcol < a.nwv - 1) a.gwake[m][i + wcol * ns] = g;
            if (loads) {
                T gd = (j > 0) ? g - x[p - ns] : g;
                // the reference's wing-flap coupling (uvlm_2dof.cpp:578-584)
                if (a.flap && m == 1 && j == 0) gd -= a.sol[a.poff[0] + i + (a.nc[0] - 1) * a.ns[0]];
                const T dg = (g - a.gprev[m][p]) * a.inv_dt;
                const T *vel = a.vel[m], *nor = a.normals[m];
                const T area = a.areas[m][p], rho = 1;
                const int64_t ia = i + j * (ns + 1), ib = ia + 1;
                const V3<T> V{vel[p], vel[np + p], vel[2 * np + p]}, n{nor[p], nor[np + p], nor[2 * np + p]};
                const V3<T> v0{v[ia], v[vld + ia], v[2 * vld + ia]}, v1{v[ib], v[vld + ib], v[2 * vld + ib]};
                V3<T> F = (rho * gd) * cross(V, v1 - v0);
                F = F + (rho * dg * area) * n;
                const double Fx = F.x, Fy = F.y, Fz = F.z;
                const double ex = 0.5 * ((double)v0.x + v1.x) - rp[0];
                const double ey = 0.5 * ((double)v0.y + v1.y) - rp[1];
                const double ez = 0.5 * ((double)v0.z + v1.z) - rp[2];
                s[0] = Fz * fsp[0] - Fx * fsp[2];  // lift times the length of (-fz, fx)
                s[1] = area;
                s[2] = ey * Fz - ez * Fy;
                s[3] = ez * Fx - ex * Fz;
                s[4] = ex * Fy - ey * Fx;
            }
            if (a.keep) a.gprev[m][p] = g;
        }
#pragma unroll
        for (int q = 0; q < LOAD_SUMS; q++) sh.s[q][t] = s[q];
    } else {
        chord_terms(sh, v, ns, nc, blk);
    }
    if (!loads) return;
    block_sums(sh, chords ? 1 : LOAD_SUMS, a.part + LOAD_PART * (int64_t)blockIdx.x);
    if (!last_block(sh, a.done)) return;
    double cl = 0, ta = 0, tm = 0;  // of thread t < 4: CL, CM x, y, z
    const double fx = fsp[0], fy = fsp[1], fz = fsp[2];
    const double qd = 0.5 * a.rho * (fx * fx + fy * fy + fz * fz), ll = sqrt(fz * fz + fx * fx);
    int64_t b0 = 0;
    for (int k = 0; k < a.n; k++) {
        const int64_t pb = (a.ns[k] * a.nc[k] + STEP_THREADS - 1) / STEP_THREADS;
        const int64_t cb = (a.ns[k] + LOAD_CHORDS - 1) / LOAD_CHORDS;
        add_parts(sh, a.part, b0, pb, cb, 0);
        if (t < 4) {
            const double S = sh.tot[1], mac = sh.tot[5] / S;
            cl += t == 0 ? sh.tot[0] / ll / (qd * S) * S : sh.tot[1 + t] / (qd * S * mac) * S * mac;
            ta += S;
            tm += mac;
        }
        b0 += pb + cb;
    }
    if (t < 4) a.out[4 * o + t] = t == 0 ? cl / ta : cl / (ta * tm);
}

template <class T>
static int step_start(const StepArgs<T>& a, int64_t step, cudaStream_t st) {
    int64_t n = a.poff[a.n];
    for (int m = 0; m < a.n; m++) n += 4 * (a.ns[m] + 1);
    k_step_start<T><<<(unsigned)cdiv(n, STEP_THREADS), STEP_THREADS, 0, st>>>(a, step);
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}
template <class T>
static int step_move(const StepArgs<T>& a, int64_t step, cudaStream_t st) {
    k_step_move<T><<<(unsigned)cdiv(a.poff[a.n], STEP_THREADS), STEP_THREADS, 0, st>>>(a, step);
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}
template <class T>
static int step_loads(const StepArgs<T>& a, int64_t step, bool loads, cudaStream_t st) {
    int64_t blocks = 0;
    for (int m = 0; m < a.n; m++)
        blocks += cdiv(a.ns[m] * a.nc[m], STEP_THREADS) + (loads ? cdiv(a.ns[m], LOAD_CHORDS) : 0);
    k_step_loads<T><<<(unsigned)blocks, STEP_THREADS, 0, st>>>(a, step, loads);
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}

// ---------------------------------------------------------------------------
// The AIC is factored once and solved for at every step, a chain of n / 128
// (n / 64 in double) dependent blocks twice over.  A run of many steps forms
// the inverse instead, as the solution for the identity, and a step's solve is
// a product with it: every row by a warp of its own, no chain, the matrix read
// from L2.  1600 panels in float: a solve 71 us, the product 6, the inverse
// once 0.52 ms (500 steps 126 -> 97 ms); 576 in double: 147, 5 and 1.15 ms (160
// steps 140 -> 120 ms).
// Its error beside the solve's: float circulations after 500 steps of 1600 panels
// 0.92 to 1.26 times, 1.05 on average over ten motions; double ones against
// quadruple precision the same (1.22e-15 and 1.21e-15, 1.43e-15 and 1.46e-15).
// inv_steps: the number of steps from which the inverse is formed.  It costs
// as much as 3 to 13 solves up to 2304 unknowns and 36 at 4096 (double: 1 to 12
// up to 1024, 50 at 2304, beyond that the solve for many columns is out of
// shared memory and slow), with about as many again kept in hand.
// ---------------------------------------------------------------------------
template <class T>
static int64_t inv_steps(int64_t n) {
    if (n > (sizeof(T) == 4 ? 4096 : 2304)) return INT64_MAX;
    return 16 + n / (sizeof(T) == 4 ? 64 : 32);
}
constexpr int INV_WARPS = 4;       // rows of a block

template <class T>
static int64_t inv_ld(int64_t n) {
    constexpr int64_t V = 16 / sizeof(T);
    return (n + V - 1) / V * V;
}

template <class T>
__global__ void k_set_diagonal(T* m, int64_t n, int64_t ld) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r < n) m[r * (ld + 1)] = (T)1;
}

// m = m^T in place, a pair of 32 x 32 tiles per block (grid: tiles x tiles, the lower ones at work)
template <class T>
__global__ void __launch_bounds__(256) k_transpose(T* m, int64_t n, int64_t ld) {
    __shared__ T s0[32][33], s1[32][33];
    const int64_t i0 = 32 * (int64_t)blockIdx.x, j0 = 32 * (int64_t)blockIdx.y;
    if (j0 > i0) return;
    const int x = threadIdx.x & 31;
    for (int y = threadIdx.x >> 5; y < 32; y += 8) {
        if (j0 + y < n && i0 + x < n) s0[y][x] = m[(j0 + y) * ld + i0 + x];
        if (i0 + y < n && j0 + x < n) s1[y][x] = m[(i0 + y) * ld + j0 + x];
    }
    __syncthreads();
    for (int y = threadIdx.x >> 5; y < 32; y += 8) {
        if (j0 + y < n && i0 + x < n) m[(j0 + y) * ld + i0 + x] = s1[x][y];
        if (i0 + y < n && j0 + x < n) m[(i0 + y) * ld + j0 + x] = s0[x][y];
    }
}

// x = M b, M by rows with a leading dimension of whole 16-byte vectors (M and b
// zero from n to there)
template <class T>
__global__ void __launch_bounds__(32 * INV_WARPS) k_inverse_apply(const T* M, int64_t n, int64_t ld, const T* b, T* x) {
    constexpr int V = 16 / sizeof(T);
    struct alignas(16) Vec {
        T v[V];
    };
    const int64_t r = blockIdx.x * (int64_t)INV_WARPS + (threadIdx.x >> 5);
    if (r >= n) return;
    const Vec *mv = reinterpret_cast<const Vec*>(M + r * ld), *bv = reinterpret_cast<const Vec*>(b);
    T acc[V];
#pragma unroll
    for (int e = 0; e < V; e++) acc[e] = 0;
#pragma unroll 4
    for (int64_t k = threadIdx.x & 31; k < ld / V; k += 32) {
        const Vec p = mv[k], q = bv[k];
#pragma unroll
        for (int e = 0; e < V; e++) acc[e] += p.v[e] * q.v[e];
    }
    T s = acc[0] + acc[1];
    if constexpr (V == 4) s += acc[2] + acc[3];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if ((threadIdx.x & 31) == 0) x[r] = s;
}

template <class T>
struct Ops2;
#define OPS2(T, sfx)                                                                                                \
    template <>                                                                                                     \
    struct Ops2<T> {                                                                                                \
        static int metrics(int32_t ns, const gbvlm_dims* d, const T* const* v, T* const* c, T* const* n,            \
                           T* const* ar, gbvlm_stream s) {                                                          \
            return gbvlm_mesh_metrics_##sfx((T)0, ns, d, v, c, n, ar, s);                                          \
        }                                                                                                           \
        static int lhs(T* a, int64_t ld, int32_t ns, const gbvlm_dims* d, const T* const* c, const T* const* n,     \
                       const T* const* vw, T sg, gbvlm_stream s) {                                                   \
            return gbvlm_lhs_assemble_##sfx(a, ld, ns, d, c, n, vw, nullptr, 0, sg, s);                             \
        }                                                                                                           \
        static int displace(int32_t ns, const gbvlm_dims* d, const T* const* t, T* const* v, const T* const* vi,    \
                            gbvlm_stream s) {                                                                       \
            return gbvlm_displace_wing_##sfx(ns, d, t, v, vi, s);                                                  \
        }                                                                                                           \
        static int wake(T* r, int32_t ns, const gbvlm_dims* d, const T* const* g, const T* const* c,                \
                        const T* const* n, const T* const* k, const int32_t* lf, int32_t it, T sg, gbvlm_stream s) { \
            return gbvlm_rhs_assemble_wake_influence_##sfx(r, ns, d, g, c, n, k, lf, it, sg, s);                   \
        }                                                                                                           \
        static int rollup(int32_t ns, const gbvlm_dims* d, T* const* k, const T* const* v, const T* const* g,       \
                          const T* const* gw, const int32_t* lf, T sg, T dt, int32_t it, gbvlm_stream s) {           \
            return gbvlm_wake_rollup_##sfx(ns, d, k, v, g, gw, lf, sg, dt, it, s);                                 \
        }                                                                                                           \
        static int factor(gbvlm_lu h, T* a, int64_t n, gbvlm_stream s) { return gbvlm_lu_factor_##sfx(h, a, n, n, s); } \
        static int solve(gbvlm_lu h, const T* a, int64_t n, T* x, gbvlm_stream s) {                                 \
            return gbvlm_lu_solve_##sfx(h, a, n, n, x, n, 1, s);                                                    \
        }                                                                                                           \
        static int solve_many(gbvlm_lu h, const T* a, int64_t n, T* x, int64_t ldx, int64_t nrhs, gbvlm_stream s) {  \
            return gbvlm_lu_solve_##sfx(h, a, n, n, x, ldx, nrhs, s);                                               \
        }                                                                                                           \
    };
OPS2(float, f32)
OPS2(double, f64)

// Device-indexed UVLM step (float, no roll-up): the step index i lives in
// idx[0] on the device, so one captured graph advances the case any number of
// times.  Its last launch: i -> i + 1.
__global__ void k_uvlm_dev_end(int64_t* idx) { idx[0] += 1; }

struct UvlmBase {
    virtual ~UvlmBase() = default;
    virtual int set_kinematics(const double* T, const double* Td, const double* fs, const double* ref) = 0;
    virtual int run(double dt, int32_t rollup, double sigma, cudaStream_t st) = 0;
    virtual int begin(double dt, int32_t rollup, double sigma, cudaStream_t st) = 0;
    virtual int step(cudaStream_t st) = 0;
    virtual int step_graph(cudaStream_t st) = 0;
    virtual int step_result(int64_t i, double* cl, double* cm, cudaStream_t st) = 0;
    virtual int64_t last_step() const = 0;
    virtual int results(double* cl, double* cm, double* gamma_last, cudaStream_t st) = 0;
    int64_t t_steps = 0, n = 0;
    bool looping = false;  // a request loop (gbvlm_uvlm_loop_*) owns the steps
};

template <class T>
struct UvlmState : UvlmBase {
    int32_t nsurf = 0;
    std::vector<gbvlm_dims> dims;
    std::vector<int32_t> lifting;
    void* mem = nullptr;
    std::vector<T*> vinit, vpos, verts, wake, colloc, colloc0, normals, areas, gamma, gprev, gwake, vel;
    T *lhs = nullptr, *rhs = nullptr, *Tm = nullptr, *Tdm = nullptr, *fs = nullptr, *ref = nullptr;
    double* res = nullptr;  // [t_steps][4]
    T *inv = nullptr, *sol = nullptr;  // the AIC's inverse by rows and its product, where the run pays for it
    int64_t ldi = 0;
    gbvlm_lu lu = nullptr;

    // device-indexed step (step_graph): counter, wake scratch, the staged LU
    // solve and the captured graph
    int64_t* d_idx = nullptr;
    float* wsc = nullptr;
    void* dmem = nullptr;
    void* lut = nullptr;
    int64_t dev_idx = -1;  // the value idx[0] holds on the device (-1: unknown)
    cudaStream_t scap = nullptr;
    cudaGraph_t sgraph = nullptr;
    cudaGraphExec_t sexec = nullptr;

    ~UvlmState() override {
        if (sexec) cudaGraphExecDestroy(sexec);
        if (sgraph) cudaGraphDestroy(sgraph);
        if (scap) cudaStreamDestroy(scap);
        if (lut) lu_solve_tables_free(lut);
        if (dmem) cudaFree(dmem);
        if (lu) gbvlm_lu_destroy(lu);
        if (mem) cudaFree(mem);
    }

    int init(int32_t ns_, const gbvlm_dims* d, const float* const* vh, const int32_t* lift, int64_t steps) {
        nsurf = ns_;
        t_steps = steps;
        dims.assign(d, d + ns_);
        lifting.assign(lift, lift + ns_);
        size_t bytes = 0;
        n = 0;
        auto al = [](size_t b) { return (b + 255) / 256 * 256; };
        for (auto& x : dims) {
            x.nwv = t_steps;  // wake (ns+1, t_steps, 4) (vlm.cpp:388-399)
            const int64_t np = x.ns * x.nc, nv = (x.ns + 1) * (x.nc + 1);
            n += np;
            bytes += al(sizeof(T) * 4 * nv) * 3 + al(sizeof(T) * 4 * (x.ns + 1) * t_steps) + al(sizeof(T) * 3 * np) * 4 +
                     al(sizeof(T) * np) * 3 + al(sizeof(T) * x.ns * (t_steps - 1));
        }
        bytes += al(sizeof(T) * n * n) + al(sizeof(T) * n) + 2 * al(sizeof(T) * 16 * nsurf * (t_steps + 1)) +
                 2 * al(sizeof(T) * 3 * (t_steps + 1)) + al(sizeof(double) * 4 * t_steps) +
                 al(sizeof(double) * LOAD_PART * step_load_blocks(dims)) + al(sizeof(unsigned));
        ldi = t_steps - 1 >= inv_steps<T>(n) ? inv_ld<T>(n) : 0;
        bytes += al(sizeof(T) * n * ldi) + al(sizeof(T) * ldi);
        GB_CUDA(cudaMalloc(&mem, bytes));
        GB_CUDA(cudaMemset(mem, 0, bytes));
        char* p = (char*)mem;
        auto take = [&](size_t cnt) {
            T* r = (T*)p;
            p += al(sizeof(T) * cnt);
            return r;
        };
        lhs = take(n * n);
        rhs = take(n);  // (to a multiple of 256 bytes, zero past n)
        if (ldi) {
            inv = take(n * ldi);
            sol = take(ldi);
        }
        Tm = take(16 * nsurf * (t_steps + 1));
        Tdm = take(16 * nsurf * (t_steps + 1));
        fs = take(3 * (t_steps + 1));
        ref = take(3 * (t_steps + 1));
        res = (double*)p;
        p += al(sizeof(double) * 4 * t_steps);
        sa.part = (double*)p;
        p += al(sizeof(double) * LOAD_PART * step_load_blocks(dims));
        sa.done = (unsigned*)p;
        p += al(sizeof(unsigned));
        for (auto& x : dims) {
            const int64_t np = x.ns * x.nc, nv = (x.ns + 1) * (x.nc + 1);
            vinit.push_back(take(4 * nv));
            vpos.push_back(take(4 * nv));
            verts.push_back(take(4 * nv));
            wake.push_back(take(4 * (x.ns + 1) * t_steps));
            colloc.push_back(take(3 * np));
            colloc0.push_back(take(3 * np));
            normals.push_back(take(3 * np));
            vel.push_back(take(3 * np));
            areas.push_back(take(np));
            gamma.push_back(take(np));
            gprev.push_back(take(np));
            gwake.push_back(take(x.ns * (t_steps - 1)));
        }
        for (int m = 0; m < nsurf; m++) {
            const int64_t nv = (dims[m].ns + 1) * (dims[m].nc + 1);
            std::vector<T> h(4 * nv);
            for (int64_t q = 0; q < 4 * nv; q++) h[q] = (T)vh[m][q];
            GB_CUDA(cudaMemcpy(vinit[m], h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice));
            std::vector<T> ones((dims[m].ns + 1) * t_steps, (T)1);  // wake w plane
            GB_CUDA(cudaMemcpy(wake[m] + 3 * (dims[m].ns + 1) * t_steps, ones.data(), sizeof(T) * ones.size(),
                               cudaMemcpyHostToDevice));
        }
        step_dims(sa, dims);
        for (int m = 0; m < nsurf; m++) {
            sa.vpos[m] = vpos[m];
            sa.colloc0[m] = colloc0[m];
            sa.verts[m] = verts[m];
            sa.wake[m] = wake[m];
            sa.vel[m] = vel[m];
            sa.colloc[m] = colloc[m];
            sa.normals[m] = normals[m];
            sa.areas[m] = areas[m];
            sa.gamma[m] = gamma[m];
            sa.gprev[m] = gprev[m];
            sa.gwake[m] = gwake[m];
        }
        sa.nwv = t_steps;
        sa.rhs = rhs;
        sa.sol = inv ? sol : rhs;
        sa.Tm = Tm;
        sa.Tdm = Tdm;
        sa.fs = fs;
        sa.ref = ref;
        sa.out = res;
        int rc = gbvlm_lu_create(&lu);
        if (rc) return rc;
        return gbvlm_lu_init(lu, n);
    }

    int set_kinematics(const double* Th, const double* Tdh, const double* fsh, const double* refh) override {
        const size_t nt = (size_t)16 * nsurf * (t_steps + 1);
        std::vector<T> a(nt), b(nt), c(3 * (t_steps + 1)), d(3 * (t_steps + 1));
        for (size_t i = 0; i < nt; i++) {
            a[i] = (T)Th[i];
            b[i] = (T)Tdh[i];
        }
        for (size_t i = 0; i < c.size(); i++) {
            c[i] = (T)fsh[i];
            d[i] = refh ? (T)refh[i] : (T)0;
        }
        GB_CUDA(cudaMemcpy(Tm, a.data(), sizeof(T) * nt, cudaMemcpyHostToDevice));
        GB_CUDA(cudaMemcpy(Tdm, b.data(), sizeof(T) * nt, cudaMemcpyHostToDevice));
        GB_CUDA(cudaMemcpy(fs, c.data(), sizeof(T) * c.size(), cudaMemcpyHostToDevice));
        GB_CUDA(cudaMemcpy(ref, d.data(), sizeof(T) * d.size(), cudaMemcpyHostToDevice));
        return GBVLM_OK;
    }

    std::vector<const T*> tr_at(const T* base, int64_t i) {
        std::vector<const T*> out;
        for (int m = 0; m < nsurf; m++) out.push_back(base + 16 * ((size_t)i * nsurf + m));
        return out;
    }

    StepArgs<T> sa;
    T dt_ = 0, sigma_ = 0;
    int32_t roll_ = 0;
    int64_t next_step = 0;

    static std::vector<const T*> C(const std::vector<T*>& v) { return std::vector<const T*>(v.begin(), v.end()); }

    int run(double dt_d, int32_t roll, double sigma_d, cudaStream_t st) override {
        int rc = begin(dt_d, roll, sigma_d, st);
        if (rc) return rc;
        for (int64_t i = 0; i + 1 < t_steps; i++)
            if ((rc = step(st))) return rc;
        return GBVLM_OK;
    }

    int begin(double dt_d, int32_t roll, double sigma_d, cudaStream_t st) override {
        gbvlm_stream s = (gbvlm_stream)st;
        const T dt = (T)dt_d, sigma = (T)sigma_d;
        dt_ = dt;
        sigma_ = sigma;
        roll_ = roll;
        next_step = 0;
        GB_REQUIRE(!looping, "UVLM: a request loop advances this case (destroy it first)");
        int rc;
        // a new run refactors the AIC: the staged solve and the step graph are rebuilt on first use
        if (sexec) cudaGraphExecDestroy(sexec);
        if (sgraph) cudaGraphDestroy(sgraph);
        sexec = nullptr;
        sgraph = nullptr;
        if (lut) lu_solve_tables_free(lut);
        lut = nullptr;
        dev_idx = -1;
        // t = 0 placement (vlm.cpp:368-376): verts_pos = T(0) verts_init; metrics; colloc at t = 0 kept
        auto t0 = tr_at(Tm, 0);
        if ((rc = Ops2<T>::displace(nsurf, dims.data(), t0.data(), vpos.data(), C(vinit).data(), s))) return rc;
        for (int m = 0; m < nsurf; m++) {
            const int64_t nv = (dims[m].ns + 1) * (dims[m].nc + 1);
            GB_CUDA(cudaMemcpyAsync(verts[m], vpos[m], sizeof(T) * 4 * nv, cudaMemcpyDeviceToDevice, st));
        }
        if ((rc = Ops2<T>::metrics(nsurf, dims.data(), C(verts).data(), colloc.data(), normals.data(), areas.data(), s)))
            return rc;
        for (int m = 0; m < nsurf; m++) {
            const int64_t np = dims[m].ns * dims[m].nc;
            GB_CUDA(cudaMemcpyAsync(colloc0[m], colloc[m], sizeof(T) * 3 * np, cudaMemcpyDeviceToDevice, st));
        }
        // AIC without wake, factored once (vlm.cpp:401-403)
        GB_CUDA(cudaMemsetAsync(lhs, 0, sizeof(T) * n * n, st));
        if ((rc = Ops2<T>::lhs(lhs, n, nsurf, dims.data(), C(colloc).data(), C(normals).data(), C(verts).data(), sigma, s)))
            return rc;
        if ((rc = Ops2<T>::factor(lu, lhs, n, s))) return rc;
        if (inv) {
            GB_CUDA(cudaMemsetAsync(inv, 0, sizeof(T) * n * ldi, st));
            k_set_diagonal<T><<<(unsigned)cdiv(n, 256), 256, 0, st>>>(inv, n, ldi);
            GB_LAUNCH_CHECK();
            if ((rc = Ops2<T>::solve_many(lu, lhs, n, inv, ldi, n, s))) return rc;
            const dim3 g((unsigned)cdiv(n, 32), (unsigned)cdiv(n, 32));
            k_transpose<T><<<g, 256, 0, st>>>(inv, n, ldi);
            GB_LAUNCH_CHECK();
        }
        sa.inv_dt = (T)1 / dt;
        GB_CUDA(cudaMemsetAsync(res, 0, sizeof(double) * 4 * t_steps, st));
        return GBVLM_OK;
    }

    int apply_inverse(cudaStream_t st) {
        k_inverse_apply<T><<<(unsigned)cdiv(n, INV_WARPS), 32 * INV_WARPS, 0, st>>>(inv, n, ldi, rhs, sol);
        GB_LAUNCH_CHECK();
        return GBVLM_OK;
    }

    // one time step (vlm.cpp:410-508); steps run in order 0, 1, ..., t_steps-2
    int step(cudaStream_t st) override {
        gbvlm_stream s = (gbvlm_stream)st;
        GB_REQUIRE(!looping, "UVLM: a request loop advances this case (destroy it first)");
        GB_REQUIRE(next_step + 1 < t_steps, "UVLM: all %lld steps done (wake capacity)", (long long)t_steps);
        const int64_t i = next_step++;
        const T dt = dt_, sigma = sigma_;
        const int32_t roll = roll_;
        int rc;
        {
            if ((rc = step_start(sa, i, st))) return rc;
            if ((rc = Ops2<T>::wake(rhs, nsurf, dims.data(), C(gwake).data(), C(colloc).data(), C(normals).data(),
                                    C(wake).data(), lifting.data(), (int32_t)i, sigma, s)))
                return rc;
            if ((rc = inv ? apply_inverse(st) : Ops2<T>::solve(lu, lhs, n, rhs, s))) return rc;
            if ((rc = step_loads(sa, i, i > 0, st))) return rc;
            if (roll && i > 0) {
                if ((rc = Ops2<T>::rollup(nsurf, dims.data(), wake.data(), C(verts).data(), C(gamma).data(),
                                          C(gwake).data(), lifting.data(), sigma, dt, (int32_t)i, s)))
                    return rc;
            }
            if ((rc = step_move(sa, i, st))) return rc;
        }
        return GBVLM_OK;
    }

    // The step of step() with every step-dependent argument read from the
    // device (float, no roll-up, from step 1 on): captured into one graph on
    // first use and replayed, one launch per step.  Results equal step()'s
    // within float rounding (the wake sums are sliced for the run's last row
    // count, not the step's).
    int step_graph(cudaStream_t st) override {
        if constexpr (!std::is_same<T, float>::value) {
            set_error("UVLM graph step: float runs only");
            return GBVLM_ERR_ARG;
        } else {
            GB_REQUIRE(!looping, "UVLM: a request loop advances this case (destroy it first)");
            GB_REQUIRE(!roll_, "UVLM graph step: roll-up runs step on the host");
            GB_REQUIRE(next_step >= 1, "UVLM graph step: take the first step with gbvlm_uvlm_step");
            GB_REQUIRE(next_step + 1 < t_steps, "UVLM: all %lld steps done (wake capacity)", (long long)t_steps);
            int rc;
            if (!sexec && (rc = build_step_graph(st))) return rc;
            if (dev_idx != next_step) {
                GB_CUDA(cudaMemcpyAsync(d_idx, &next_step, sizeof(int64_t), cudaMemcpyHostToDevice, st));
                GB_CUDA(cudaStreamSynchronize(st));  // next_step is host memory that changes below
            }
            GB_CUDA(cudaGraphLaunch(sexec, st));
            next_step++;
            dev_idx = next_step;
            return GBVLM_OK;
        }
    }

    // the device-indexed step on stream c (captured by step_graph and by the
    // request loop of gbvlm_uvlm_loop_*)
    int enqueue_dev_step(cudaStream_t c) {
        StepArgs<T> a = sa;
        a.idx = d_idx;
        int r;
        if ((r = step_start(a, 0, c))) return r;
        if ((r = wake_influence_dev_f32(rhs, nsurf, dims.data(), C(gwake).data(), C(colloc).data(),
                                        C(normals).data(), C(wake).data(), lifting.data(), d_idx,
                                        (int32_t)(t_steps - 2), wsc, c)))
            return r;
        if ((r = inv ? apply_inverse(c) : lu_solve_prepared_f32(lu, lut, n, c))) return r;
        if ((r = step_loads(a, 0, true, c))) return r;
        if ((r = step_move(a, 0, c))) return r;
        k_uvlm_dev_end<<<1, 1, 0, c>>>(d_idx);
        GB_LAUNCH_CHECK();
        return GBVLM_OK;
    }

    // device buffers of the device-indexed step and the staged LU solve
    int prepare_dev(cudaStream_t st) {
        if (!dmem) {
            GB_CUDA(cudaMalloc(&dmem, 256 + sizeof(float) * WAKE_DEV_MAX_SLICES * n));
            d_idx = (int64_t*)dmem;
            wsc = (float*)((char*)dmem + 256);
        }
        if constexpr (std::is_same<T, float>::value) {
            if (!lut && !inv) {
                int rc = lu_solve_prepare_f32(lu, lhs, n, rhs, &lut, st);
                if (rc) return rc;
            }
        }
        return GBVLM_OK;
    }

    int build_step_graph(cudaStream_t st) {
        if constexpr (std::is_same<T, float>::value) {
            int rc = prepare_dev(st);
            if (rc) return rc;
            if (!scap) GB_CUDA(cudaStreamCreateWithFlags(&scap, cudaStreamNonBlocking));
            GB_CUDA(cudaStreamSynchronize(st));
            GB_CUDA(cudaStreamBeginCapture(scap, cudaStreamCaptureModeThreadLocal));
            rc = enqueue_dev_step(scap);
            cudaGraph_t g = nullptr;
            const cudaError_t e = cudaStreamEndCapture(scap, &g);
            if (rc) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            GB_CUDA(e);
            sgraph = g;
            GB_CUDA(cudaGraphInstantiate(&sexec, sgraph, 0));
            dev_idx = -1;
            return GBVLM_OK;
        } else {
            (void)st;
            return GBVLM_ERR_ARG;
        }
    }

    int64_t last_step() const override { return next_step - 1; }

    int step_result(int64_t i, double* cl, double* cm, cudaStream_t st) override {
        GB_REQUIRE(i >= 0 && i < t_steps, "step index outside the run");
        double h[4];
        GB_CUDA(cudaMemcpyAsync(h, res + 4 * i, sizeof(h), cudaMemcpyDeviceToHost, st));
        GB_CUDA(cudaStreamSynchronize(st));
        if (cl) *cl = h[0];
        if (cm) for (int k = 0; k < 3; k++) cm[k] = h[1 + k];
        return lu_solve_check(lu, st);  // the steps' solves finished their bounded waits
    }

    int results(double* cl, double* cm, double* gamma_last, cudaStream_t st) override {
        std::vector<double> h(4 * t_steps);
        GB_CUDA(cudaMemcpyAsync(h.data(), res, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, st));
        std::vector<T> g(n);
        if (gamma_last) {
            int64_t off = 0;
            for (int m = 0; m < nsurf; m++) {
                const int64_t np = dims[m].ns * dims[m].nc;
                GB_CUDA(cudaMemcpyAsync(g.data() + off, gamma[m], sizeof(T) * np, cudaMemcpyDeviceToHost, st));
                off += np;
            }
        }
        GB_CUDA(cudaStreamSynchronize(st));
        for (int64_t i = 0; i < t_steps; i++) {
            if (cl) cl[i] = h[4 * i];
            if (cm)
                for (int k = 0; k < 3; k++) cm[3 * i + k] = h[4 * i + 1 + k];
        }
        if (gamma_last)
            for (int64_t q = 0; q < n; q++) gamma_last[q] = (double)g[q];
        return lu_solve_check(lu, st);  // the steps' solves finished their bounded waits
    }
};

// ===========================================================================
// Coupled aeroelastic 2-DOF (pitch-plunge) UVLM, tests/uvlm_2dof.cpp:437-808
// (COUPLED branch).  Aerodynamics in float as the reference; structure in
// double on the device (Newmark-beta, gbvlm_struct.cu).  Per time step i a
// Newton loop on the load increment: Newmark step -> state at i+1 -> pose
// fs(t+dt).heave.pitch (value and time derivative) -> displaced wing,
// metrics, wake shed, panel velocities, RHS with the wake, solve with the
// AIC factored at t = 0 -> gamma, wing-flap delta coupling, forces, CL/CM ->
// loads F(i+1) and their increment -> converged when |du_prev - du| <= eps.
// Each iteration is a fixed chain of launches; the host reads one flag per
// iteration to end the loop.
// ===========================================================================
struct A2Dev {
    double M[4], C[4], K[4];
    double du[2], dv[2], da[2], dF[2], du_prev[2];
    double coef[4];  // CL, CM x, y, z of the iterate
    float T[16], dT[16], ref[3], fs[3];
    int converged;
    int32_t iter, max_iter;  // Newton iterations of the current step, and their limit
    int64_t step;            // the step being advanced: state i -> i + 1
    int64_t wit;             // wake rows of that step's solve (step + 1)
};

// state at i+1 from the Newmark increments, the pose and the moment point
__global__ void k_a2_pose(A2Dev* d, double* u, double* v, double* a, float dtf, double a_h, int32_t nsurf,
                          float* T_all, float* dT_all) {
    if (threadIdx.x != 0) return;
    const int64_t i = d->step;
    const double t_next = (double)((float)i * dtf + dtf);
    double* u1 = u + 2 * (i + 1);
    double* v1 = v + 2 * (i + 1);
    double* a1 = a + 2 * (i + 1);
    for (int k = 0; k < 2; k++) {
        u1[k] = u[2 * i + k] + d->du[k];
        v1[k] = v[2 * i + k] + d->dv[k];
        a1[k] = a[2 * i + k] + d->da[k];
    }
    const double h = u1[0], al = u1[1], hd = v1[0], ad = v1[1];
    const double px = 1.0 + a_h;
    // pitch: rotation about y through (px, 0, 0) (vlm_kinematics.hpp:184-201), and d/dt = dR/dalpha * alpha'
    const double c = cos(al), sn = sin(al);
    double P[16] = {c, 0, -sn, 0, 0, 1, 0, 0, sn, 0, c, 0, px - c * px, 0, sn * px, 1};   // column-major
    double dP[16] = {-sn * ad, 0, -c * ad, 0, 0, 0, 0, 0, c * ad, 0, -sn * ad, 0, sn * px * ad, 0, c * px * ad, 0};
    // heave: translation (0, 0, -h), d/dt (0, 0, -h'); freestream: translation (-t, 0, 0), d/dt (-1, 0, 0)
    double H[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, 0, 0, -h, 1};
    double dH[16] = {0};
    dH[14] = -hd;
    double Fm[16] = {1, 0, 0, 0, 0, 1, 0, 0, 0, 0, 1, 0, -t_next, 0, 0, 1};
    double dFm[16] = {0};
    dFm[12] = -1.0;
    auto mul = [](const double* A, const double* B, double* R) {
        for (int cc = 0; cc < 4; cc++)
            for (int r = 0; r < 4; r++) {
                double s_ = 0;
                for (int k = 0; k < 4; k++) s_ += A[r + 4 * k] * B[k + 4 * cc];
                R[r + 4 * cc] = s_;
            }
    };
    double HP[16], dHP[16], t1[16], t2[16], TT[16], dTT[16];
    mul(H, P, HP);
    mul(dH, P, t1);
    mul(H, dP, t2);
    for (int q = 0; q < 16; q++) dHP[q] = t1[q] + t2[q];
    mul(Fm, HP, TT);
    mul(dFm, HP, t1);
    mul(Fm, dHP, t2);
    for (int q = 0; q < 16; q++) dTT[q] = t1[q] + t2[q];
    for (int q = 0; q < 16; q++) {
        d->T[q] = (float)TT[q];
        d->dT[q] = (float)dTT[q];
    }
    for (int r = 0; r < 3; r++) d->ref[r] = (float)(TT[r] * px + TT[r + 12]);
    for (int m = 0; m < nsurf; m++)
        for (int q = 0; q < 16; q++) {
            T_all[16 * m + q] = (float)TT[q];
            dT_all[16 * m + q] = (float)dTT[q];
        }
}

__host__ __device__ inline double torsional_cubic(double al) { return 0.1 * al + 40.0 * al * al * al; }

// loads of the iterate (uvlm_2dof.cpp:728-744) and the Newton test; the
// loop of the time step's graph continues while the test fails and at most
// max_iter iterations have run (the reference's loop, :639-807)
__global__ void k_a2_loads(A2Dev* d, double* u, double* F, double mu, double r_a, double om, double Ua, double eps,
                           cudaGraphConditionalHandle loop) {
    if (threadIdx.x != 0) return;
    const int64_t i = d->step;
    const double pi_f = (double)3.141593f;
    F[2 * (i + 1)] = -d->coef[0] / (pi_f * mu);
    F[2 * (i + 1) + 1] = (2.0 * d->coef[2]) / (pi_f * mu * r_a * r_a);
    d->dF[0] = F[2 * (i + 1)] - F[2 * i] - (om / Ua) * (om / Ua) * d->du[0];
    d->dF[1] = F[2 * (i + 1) + 1] - F[2 * i + 1] -
               1.0 / (Ua * Ua) * (torsional_cubic(u[2 * (i + 1) + 1]) - torsional_cubic(u[2 * i + 1]));
    const double k0 = d->du_prev[0] - d->du[0], k1 = d->du_prev[1] - d->du[1];
    d->converged = sqrt(k0 * k0 + k1 * k1) <= eps ? 1 : 0;
    d->iter += 1;
    cudaGraphSetConditional(loop, (!d->converged && d->iter <= d->max_iter) ? 1u : 0u);
}

// start of a time step: the previous circulation kept, increments and the
// iteration count cleared
struct A2Copy {
    int32_t n;
    const float* src[GBVLM_MAX_SURFACES];
    float* dst[GBVLM_MAX_SURFACES];
    int64_t cnt[GBVLM_MAX_SURFACES];
};
__global__ void k_a2_step_begin(A2Dev* d, A2Copy c) {
    for (int m = 0; m < c.n; m++)
        for (int64_t e = threadIdx.x; e < c.cnt[m]; e += blockDim.x) c.dst[m][e] = c.src[m][e];
    if (threadIdx.x == 0) {
        d->dF[0] = d->dF[1] = 0.0;
        d->du[0] = d->du[1] = 0.0;
        d->iter = 0;
    }
}
// end of a time step: its iteration count recorded, the next step's indices
__global__ void k_a2_step_end(A2Dev* d, int32_t* iters) {
    if (threadIdx.x != 0) return;
    iters[d->step] = d->iter;
    d->step += 1;
    d->wit = d->step + 1;
}
__global__ void k_a2_set(A2Dev* d, int64_t step, int32_t max_iter) {
    if (threadIdx.x != 0) return;
    d->step = step;
    d->wit = step + 1;
    d->max_iter = max_iter;
}

struct Aero2Dof {
    int32_t nsurf = 0;
    std::vector<gbvlm_dims> dims;
    std::vector<int32_t> lifting;
    gbvlm_2dof_vars vars{};
    double dt = 0;
    int64_t t_steps = 0, n = 0, done = 0;  // steps advanced
    void* mem = nullptr;
    std::vector<float*> vinit, verts, wake, colloc, colloch, normals, areas, gamma, gprev, gwake, vel;
    float *lhs = nullptr, *rhs = nullptr, *T_all = nullptr, *dT_all = nullptr;
    double *u = nullptr, *v = nullptr, *a = nullptr, *F = nullptr;
    A2Dev* dev = nullptr;
    gbvlm_lu lu = nullptr;
    gbvlm_newmark nm = nullptr;
    std::vector<int32_t> iters;
    StepArgs<float> sa;
    // one time step as a CUDA graph: the Newton iterations in a conditional
    // while node, replayed step after step without host round trips
    void* aux = nullptr;             // iteration counts per step, wake-influence scratch
    int32_t* iters_dev = nullptr;
    float* wscratch = nullptr;
    void* lut = nullptr;             // the staged LU solve of the factored AIC
    cudaStream_t cap = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;

    ~Aero2Dof() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (cap) cudaStreamDestroy(cap);
        if (lut) lu_solve_tables_free(lut);
        if (aux) cudaFree(aux);
        if (lu) gbvlm_lu_destroy(lu);
        if (nm) gbvlm_newmark_destroy(nm);
        if (mem) cudaFree(mem);
    }

    static std::vector<const float*> C(const std::vector<float*>& x) { return std::vector<const float*>(x.begin(), x.end()); }

    int init(int32_t ns_, const gbvlm_dims* d, const float* const* vh, const int32_t* lift, const gbvlm_2dof_vars& vr,
             double t_final, cudaStream_t st) {
        nsurf = ns_;
        vars = vr;
        dims.assign(d, d + ns_);
        lifting.assign(lift, lift + ns_);
        // nondimensional vertices (uvlm_2dof.cpp:428-435) and the time step: the chord of the last
        // chordwise panel of the last surface at the first spanwise station (:473-480), in float
        std::vector<std::vector<float>> vnd(nsurf);
        for (int m = 0; m < nsurf; m++) {
            const int64_t nv = (dims[m].ns + 1) * (dims[m].nc + 1);
            vnd[m].assign(vh[m], vh[m] + 4 * nv);
            for (int64_t q = 0; q < 3 * nv; q++) vnd[m][q] = (float)(vnd[m][q] / (float)vars.b);
        }
        {
            const gbvlm_dims& L = dims[nsurf - 1];
            const int64_t nv = (L.ns + 1) * (L.nc + 1), lastj = L.nc * (L.ns + 1), prevj = (L.nc - 1) * (L.ns + 1);
            const std::vector<float>& w = vnd[nsurf - 1];
            const float dx = w[lastj] - w[prevj], dy = w[nv + lastj] - w[nv + prevj];
            const float dz = w[2 * nv + lastj] - w[2 * nv + prevj];
            const float dtf = sqrtf(dx * dx + dy * dy + dz * dz);
            dt = (double)dtf;
            t_steps = (int64_t)((float)t_final / dtf);
        }
        GB_REQUIRE(t_steps >= 3, "aeroelastic 2-DOF: t_final %.3g gives %lld steps of %.3g", t_final,
                   (long long)t_steps, dt);
        size_t bytes = 0;
        auto al = [](size_t b) { return (b + 255) / 256 * 256; };
        n = 0;
        for (auto& x : dims) {
            x.nwv = t_steps;
            const int64_t np = x.ns * x.nc, nv = (x.ns + 1) * (x.nc + 1);
            n += np;
            bytes += al(4 * 4 * nv) * 2 + al(4 * 4 * (x.ns + 1) * t_steps) + al(4 * 3 * np) * 4 + al(4 * np) * 3 +
                     al(4 * x.ns * (t_steps - 1));
        }
        bytes += al(4 * n * n) + al(4 * n) + 2 * al(4 * 16 * nsurf) + 4 * al(8 * 2 * t_steps) + al(sizeof(A2Dev)) +
                 al(sizeof(double) * LOAD_PART * step_load_blocks(dims)) + al(sizeof(unsigned));
        GB_CUDA(cudaMalloc(&mem, bytes));
        GB_CUDA(cudaMemset(mem, 0, bytes));
        char* p = (char*)mem;
        auto take = [&](size_t b) {
            void* r = p;
            p += al(b);
            return r;
        };
        lhs = (float*)take(4 * n * n);
        rhs = (float*)take(4 * n);
        T_all = (float*)take(4 * 16 * nsurf);
        dT_all = (float*)take(4 * 16 * nsurf);
        u = (double*)take(8 * 2 * t_steps);
        v = (double*)take(8 * 2 * t_steps);
        a = (double*)take(8 * 2 * t_steps);
        F = (double*)take(8 * 2 * t_steps);
        dev = (A2Dev*)take(sizeof(A2Dev));
        sa.part = (double*)take(sizeof(double) * LOAD_PART * step_load_blocks(dims));
        sa.done = (unsigned*)take(sizeof(unsigned));
        {
            const size_t ib = (sizeof(int32_t) * t_steps + 255) / 256 * 256;
            GB_CUDA(cudaMalloc(&aux, ib + sizeof(float) * WAKE_DEV_MAX_SLICES * n));
            iters_dev = (int32_t*)aux;
            wscratch = (float*)((char*)aux + ib);
        }
        for (auto& x : dims) {
            const int64_t np = x.ns * x.nc, nv = (x.ns + 1) * (x.nc + 1);
            vinit.push_back((float*)take(4 * 4 * nv));
            verts.push_back((float*)take(4 * 4 * nv));
            wake.push_back((float*)take(4 * 4 * (x.ns + 1) * t_steps));
            colloc.push_back((float*)take(4 * 3 * np));
            colloch.push_back((float*)take(4 * 3 * np));
            normals.push_back((float*)take(4 * 3 * np));
            vel.push_back((float*)take(4 * 3 * np));
            areas.push_back((float*)take(4 * np));
            gamma.push_back((float*)take(4 * np));
            gprev.push_back((float*)take(4 * np));
            gwake.push_back((float*)take(4 * x.ns * (t_steps - 1)));
        }
        for (int m = 0; m < nsurf; m++) {
            GB_CUDA(cudaMemcpy(vinit[m], vnd[m].data(), 4 * vnd[m].size(), cudaMemcpyHostToDevice));
            std::vector<float> ones((dims[m].ns + 1) * t_steps, 1.f);  // wake w plane
            GB_CUDA(cudaMemcpy(wake[m] + 3 * (dims[m].ns + 1) * t_steps, ones.data(), 4 * ones.size(),
                               cudaMemcpyHostToDevice));
        }
        // structure (uvlm_2dof.cpp:352-416): K = 0, the linear stiffness is in the load
        A2Dev h{};
        const double xa = vars.x_a, ra = vars.r_a, om = vars.omega, Ua = vars.U_a;
        h.M[0] = 1.0;
        h.M[1] = xa / (ra * ra);
        h.M[2] = xa;
        h.M[3] = 1.0;
        h.C[0] = 2.0 * vars.zeta_h * (om / Ua);
        h.C[3] = 2.0 * vars.zeta_a / Ua;
        h.fs[0] = 1.f;  // -d/dt of the freestream translation (-t, 0, 0)
        GB_CUDA(cudaMemcpy(dev, &h, sizeof(h), cudaMemcpyHostToDevice));
        {
            const double u0[2] = {0.0, 3.0 * M_PI / 180.0}, v0[2] = {0.0, 0.0};
            const double r0[2] = {-(om / Ua) * (om / Ua) * u0[0], -1.0 / (Ua * Ua) * torsional_cubic(u0[1])};
            // M a0 = r0 - C v0 - K u0 (2 x 2, column-major M)
            const double det = h.M[0] * h.M[3] - h.M[2] * h.M[1];
            const double a0[2] = {(h.M[3] * r0[0] - h.M[2] * r0[1]) / det, (-h.M[1] * r0[0] + h.M[0] * r0[1]) / det};
            GB_CUDA(cudaMemcpy(u, u0, sizeof(u0), cudaMemcpyHostToDevice));
            GB_CUDA(cudaMemcpy(v, v0, sizeof(v0), cudaMemcpyHostToDevice));
            GB_CUDA(cudaMemcpy(a, a0, sizeof(a0), cudaMemcpyHostToDevice));
        }
        int rc = gbvlm_newmark_create(&nm, 0.25, 0.5);
        if (rc) return rc;
        if ((rc = gbvlm_newmark_init(nm, 2, dev->M, dev->C, dev->K, dt, (gbvlm_stream)st))) return rc;
        if ((rc = gbvlm_lu_create(&lu))) return rc;
        if ((rc = gbvlm_lu_init(lu, n))) return rc;
        step_dims(sa, dims);
        for (int m = 0; m < nsurf; m++) {
            sa.vpos[m] = vinit[m];
            sa.colloc0[m] = colloch[m];
            sa.verts[m] = verts[m];
            sa.wake[m] = wake[m];
            sa.vel[m] = vel[m];
            sa.colloc[m] = colloc[m];
            sa.normals[m] = normals[m];
            sa.areas[m] = areas[m];
            sa.gamma[m] = gamma[m];
            sa.gprev[m] = gprev[m];
            sa.gwake[m] = gwake[m];
        }
        sa.nwv = t_steps;
        sa.rhs = rhs;
        sa.sol = rhs;
        sa.Tm = T_all;
        sa.Tdm = dT_all;
        sa.fs = dev->fs;
        sa.ref = dev->ref;
        sa.out = dev->coef;
        sa.inv_dt = 1.f / (float)dt;
        sa.rho = vars.rho;
        sa.by_step = sa.keep = false;  // the pose and loads of the iterate; gprev stays the step's
        sa.flap = nsurf > 1 && dims[1].ns == dims[0].ns;
        return start(st);
    }

    // initial pose, AIC factored once, the t = 0 solve (uvlm_2dof.cpp:453-515)
    int start(cudaStream_t st) {
        gbvlm_stream s = (gbvlm_stream)st;
        const double px = 1.0 + vars.a_h, th = 3.0 * M_PI / 180.0, c = cos(th), sn = sin(th);
        float T0[16] = {(float)c, 0, (float)-sn, 0, 0, 1, 0, 0, (float)sn, 0, (float)c, 0,
                        (float)(px - c * px), 0, (float)(sn * px), 1};
        float dT0[16] = {0};
        dT0[12] = -1.f;
        std::vector<float> ta(16 * nsurf), tb(16 * nsurf);
        for (int m = 0; m < nsurf; m++)
            for (int q = 0; q < 16; q++) {
                ta[16 * m + q] = T0[q];
                tb[16 * m + q] = dT0[q];
            }
        GB_CUDA(cudaMemcpyAsync(T_all, ta.data(), 4 * ta.size(), cudaMemcpyHostToDevice, st));
        GB_CUDA(cudaMemcpyAsync(dT_all, tb.data(), 4 * tb.size(), cudaMemcpyHostToDevice, st));
        std::vector<const float*> tr(nsurf);
        for (int m = 0; m < nsurf; m++) tr[m] = T_all + 16 * m;
        int rc;
        if ((rc = Ops2<float>::displace(nsurf, dims.data(), tr.data(), verts.data(), C(vinit).data(), s))) return rc;
        if ((rc = Ops2<float>::metrics(nsurf, dims.data(), C(verts).data(), colloc.data(), normals.data(),
                                       areas.data(), s)))
            return rc;
        for (int m = 0; m < nsurf; m++)
            GB_CUDA(cudaMemcpyAsync(colloch[m], colloc[m], 4 * 3 * dims[m].ns * dims[m].nc, cudaMemcpyDeviceToDevice,
                                    st));
        GB_CUDA(cudaMemsetAsync(lhs, 0, 4 * n * n, st));
        if ((rc = Ops2<float>::lhs(lhs, n, nsurf, dims.data(), C(colloc).data(), C(normals).data(), C(verts).data(),
                                   0.f, s)))
            return rc;
        if ((rc = Ops2<float>::factor(lu, lhs, n, s))) return rc;
        if (!lut && (rc = lu_solve_prepare_f32(lu, lhs, n, rhs, &lut, st))) return rc;
        if ((rc = aero_solve(0, st))) return rc;
        done = 0;
        iters.clear();
        return GBVLM_OK;
    }

    // wake shed, velocities, RHS, solve and circulation of the current pose (wake rows 0..it)
    int aero_solve(int64_t it, cudaStream_t st) {
        gbvlm_stream s = (gbvlm_stream)st;
        int rc;
        if ((rc = step_start(sa, it, st))) return rc;
        if ((rc = Ops2<float>::wake(rhs, nsurf, dims.data(), C(gwake).data(), C(colloc).data(), C(normals).data(),
                                    C(wake).data(), lifting.data(), (int32_t)it, 0.f, s)))
            return rc;
        if ((rc = Ops2<float>::solve(lu, lhs, n, rhs, s))) return rc;
        return step_loads(sa, it, false, st);
    }

    // one Newton iteration of the step dev->step (uvlm_2dof.cpp:639-751), with
    // every step-dependent index read on the device: captured into the body
    // of the step graph's while node
    int iterate_dev(cudaStream_t st, cudaGraphConditionalHandle loop) {
        int rc;
        GB_CUDA(cudaMemcpyAsync(dev->du_prev, dev->du, sizeof(double) * 2, cudaMemcpyDeviceToDevice, st));
        if ((rc = newmark_step_dev(nm, dev->M, dev->C, v, a, &dev->step, dev->du, dev->dv, dev->da, dev->dF, dt, st)))
            return rc;
        k_a2_pose<<<1, 32, 0, st>>>(dev, u, v, a, (float)dt, vars.a_h, nsurf, T_all, dT_all);
        GB_LAUNCH_CHECK();
        StepArgs<float> d = sa;
        d.idx = &dev->wit;
        if ((rc = step_move(d, 0, st))) return rc;
        // wake shed, velocities, RHS, solve and loads of the pose (wake rows 0..step+1)
        if ((rc = step_start(d, 0, st))) return rc;
        if ((rc = wake_influence_dev_f32(rhs, nsurf, dims.data(), C(gwake).data(), C(colloc).data(),
                                         C(normals).data(), C(wake).data(), lifting.data(), &dev->wit,
                                         (int32_t)(t_steps - 2), wscratch, st)))
            return rc;
        if ((rc = lu_solve_prepared_f32(lu, lut, n, st))) return rc;
        if ((rc = step_loads(d, 0, true, st))) return rc;
        k_a2_loads<<<1, 32, 0, st>>>(dev, u, F, vars.mu, vars.r_a, vars.omega, vars.U_a,
                                     (double)1.1920928955078125e-07, loop);
        GB_LAUNCH_CHECK();
        return GBVLM_OK;
    }

    // the step graph: begin (previous circulation, cleared increments) ->
    // while (Newton test fails and iterations <= max_iter) { iteration } -> end
    int build_graph() {
        if (exec) return GBVLM_OK;
        GB_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        GB_CUDA(cudaGraphCreate(&graph, 0));
        cudaGraphConditionalHandle loop;
        GB_CUDA(cudaGraphConditionalHandleCreate(&loop, graph, 1, cudaGraphCondAssignDefault));
        A2Copy cp{};
        cp.n = nsurf;
        for (int m = 0; m < nsurf; m++) {
            cp.src[m] = gamma[m];
            cp.dst[m] = gprev[m];
            cp.cnt[m] = dims[m].ns * dims[m].nc;
        }
        cudaGraphNode_t nb, nw, ne;
        {
            void* args[] = {&dev, &cp};
            cudaKernelNodeParams kp = {};
            kp.func = (void*)k_a2_step_begin;
            kp.gridDim = dim3(1);
            kp.blockDim = dim3(256);
            kp.kernelParams = args;
            GB_CUDA(cudaGraphAddKernelNode(&nb, graph, nullptr, 0, &kp));
        }
        cudaGraphNodeParams wp = {};
        wp.type = cudaGraphNodeTypeConditional;
        wp.conditional.handle = loop;
        wp.conditional.type = cudaGraphCondTypeWhile;
        wp.conditional.size = 1;
        GB_CUDA(cudaGraphAddNode(&nw, graph, &nb, nullptr, 1, &wp));
        cudaGraph_t body = wp.conditional.phGraph_out[0];
        GB_CUDA(cudaStreamBeginCaptureToGraph(cap, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
        int rc = iterate_dev(cap, loop);
        cudaGraph_t got = nullptr;
        const cudaError_t e = cudaStreamEndCapture(cap, &got);
        if (rc) return rc;
        GB_CUDA(e);
        {
            void* args[] = {&dev, &iters_dev};
            cudaKernelNodeParams kp = {};
            kp.func = (void*)k_a2_step_end;
            kp.gridDim = dim3(1);
            kp.blockDim = dim3(32);
            kp.kernelParams = args;
            GB_CUDA(cudaGraphAddKernelNode(&ne, graph, &nw, 1, &kp));
        }
        GB_CUDA(cudaGraphInstantiate(&exec, graph, 0));
        return GBVLM_OK;
    }

    int run(int64_t steps, int32_t max_iter, cudaStream_t st) {
        GB_REQUIRE(done + steps <= t_steps - 2, "aeroelastic 2-DOF: %lld steps requested, %lld left",
                   (long long)steps, (long long)(t_steps - 2 - done));
        GB_REQUIRE(max_iter >= 0, "aeroelastic 2-DOF: max_iter must be non-negative");
        if (steps <= 0) return GBVLM_OK;
        int rc = build_graph();
        if (rc) return rc;
        k_a2_set<<<1, 32, 0, st>>>(dev, done, max_iter);
        GB_LAUNCH_CHECK();
        for (int64_t k = 0; k < steps; k++) GB_CUDA(cudaGraphLaunch(exec, st));
        std::vector<int32_t> h(steps);
        int* words = (int*)host_scratch(2 * sizeof(int));
        GB_REQUIRE(words != nullptr, "pinned host allocation failed");
        GB_CUDA(cudaMemcpyAsync(h.data(), iters_dev + done, sizeof(int32_t) * steps, cudaMemcpyDeviceToHost, st));
        if ((rc = lu_solve_words(lu, words, st))) return rc;
        GB_CUDA(cudaStreamSynchronize(st));
        iters.insert(iters.end(), h.begin(), h.end());
        done += steps;
        return lu_solve_verdict(lu, words, st);  // the steps' solves finished their bounded waits
    }
};

}  // namespace gbvlm

using namespace gbvlm;

struct gbvlm_uvlm_s {
    UvlmBase* impl = nullptr;
};

// ===========================================================================
// Device-resident request loop over a resident UVLM case.  One CUDA graph: a
// while node whose body is the device-indexed step followed by
// k_uvlm_loop_next.  The host submits a request by raising a counter in
// mapped host memory; the running graph takes one step per request, writes
// each step's coefficients into a mapped record and raises the done
// counter, then waits (bounded) for the next request.  After poll_ns
// without one it marks itself stopped and ends; the next submit launches
// the graph again.  Between requests no CUDA call is made.
// ===========================================================================
namespace gbvlm {

struct LoopCtl {
    int64_t enq;    // requests submitted (host)
    int64_t done;   // requests completed (device)
    int32_t state;  // 0: no graph running or about to run, 1: running (both sides, system-scope atomics)
    int32_t stop;   // host: end the loop
    int32_t error;  // device: 1 = the wake is full
    int32_t pad;
};
struct LoopRec {
    int64_t step;
    double c[4];     // CL, CM x, y, z
    int64_t failed;  // a solve's bounded wait ran out
};

__device__ __forceinline__ uint64_t loop_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// last_idx: the largest step index the wake holds; err0, err1: the error words of the solves (or null)
__global__ void k_uvlm_loop_next(LoopCtl* ctl, LoopRec* rec, const int64_t* idx, const double* res, int64_t last_idx,
                                 const int* err0, const int* err1, uint64_t poll_ns, cudaGraphConditionalHandle loop) {
    if (threadIdx.x != 0) return;
    volatile LoopCtl* vc = ctl;
    const int64_t i = idx[0] - 1;  // the step this iteration took
    const int64_t t = vc->done;
    rec[t].step = i;
    for (int k = 0; k < 4; k++) rec[t].c[k] = res[4 * i + k];
    rec[t].failed = (err0 && *err0) || (err1 && *err1);
    __threadfence_system();
    vc->done = t + 1;
    __threadfence_system();
    unsigned cont = 0;
    bool released = false;
    if (idx[0] > last_idx) {
        vc->error = 1;
    } else {
        const uint64_t t0 = loop_ns();
        while (true) {
            if (vc->stop) break;
            if (vc->enq > t + 1) {
                cont = 1;
                break;
            }
            if (loop_ns() - t0 > poll_ns) {
                // stop, unless a request came in meanwhile and the host has
                // not already taken the running state to launch a new graph
                atomicExch_system(&ctl->state, 0);
                released = true;
                __threadfence_system();
                if (vc->enq > t + 1 && atomicCAS_system(&ctl->state, 0, 1) == 0) {
                    cont = 1;
                    released = false;
                }
                break;
            }
            __nanosleep(2000);
        }
    }
    if (!cont && !released) atomicExch_system(&ctl->state, 0);
    cudaGraphSetConditional(loop, cont);
}

}  // namespace gbvlm

struct gbvlm_uvlm_loop_s {
    gbvlm_uvlm owner = nullptr;
    UvlmState<float>* u = nullptr;
    LoopCtl* ctl = nullptr;  // mapped host memory
    LoopRec* rec = nullptr;
    LoopCtl* ctl_d = nullptr;
    LoopRec* rec_d = nullptr;
    int64_t cap = 0, base_step = 0, enq = 0, launches = 0;
    cudaStream_t st = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::mutex mu;
    ~gbvlm_uvlm_loop_s() {
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        if (st) cudaStreamDestroy(st);
        if (ctl) cudaFreeHost(ctl);
        if (rec) cudaFreeHost(rec);
    }
};

extern "C" {

int gbvlm_uvlm_create(gbvlm_uvlm* out, int32_t nsurf, const gbvlm_dims* dims, const float* const* verts_init,
                      const int32_t* lifting, int64_t t_steps, int32_t precision) {
    GB_REQUIRE(out && dims && verts_init && lifting, "null argument");
    GB_REQUIRE(nsurf >= 1 && nsurf <= GBVLM_MAX_SURFACES, "nsurf=%d outside [1, %d]", nsurf, GBVLM_MAX_SURFACES);
    GB_REQUIRE(t_steps >= 2, "t_steps must be at least 2");
    GB_REQUIRE(precision == 32 || precision == 64, "precision must be 32 or 64");
    for (int m = 0; m < nsurf; m++) GB_REQUIRE(verts_init[m] && dims[m].ns >= 1 && dims[m].nc >= 1, "surface %d", m);
    auto* h = new gbvlm_uvlm_s();
    int rc;
    if (precision == 32) {
        auto* s = new UvlmState<float>();
        h->impl = s;
        rc = s->init(nsurf, dims, verts_init, lifting, t_steps);
    } else {
        auto* s = new UvlmState<double>();
        h->impl = s;
        rc = s->init(nsurf, dims, verts_init, lifting, t_steps);
    }
    if (rc) {
        delete h->impl;
        delete h;
        return rc;
    }
    *out = h;
    return GBVLM_OK;
}

int gbvlm_uvlm_destroy(gbvlm_uvlm h) {
    if (!h) return GBVLM_OK;
    GB_REQUIRE(!h->impl || !h->impl->looping, "UVLM: destroy its request loop first");
    delete h->impl;
    delete h;
    return GBVLM_OK;
}

int gbvlm_uvlm_set_kinematics(gbvlm_uvlm h, const double* transforms, const double* dtransforms,
                              const double* freestream, const double* ref_pt) {
    GB_REQUIRE(h && h->impl && transforms && dtransforms && freestream, "null argument");
    return h->impl->set_kinematics(transforms, dtransforms, freestream, ref_pt);
}

int gbvlm_uvlm_run(gbvlm_uvlm h, double dt, int32_t rollup, double sigma, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl && dt > 0, "bad arguments");
    return h->impl->run(dt, rollup, sigma, to_cuda(stream));
}

int gbvlm_uvlm_begin(gbvlm_uvlm h, double dt, int32_t rollup, double sigma, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl && dt > 0, "bad arguments");
    return h->impl->begin(dt, rollup, sigma, to_cuda(stream));
}

int gbvlm_uvlm_step(gbvlm_uvlm h, int64_t* step_index, double* cl, double* cm, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl, "null argument");
    int rc = h->impl->step(to_cuda(stream));
    if (rc) return rc;
    auto* u = h->impl;
    const int64_t i = u->last_step();
    if (step_index) *step_index = i;
    if (cl || cm) return u->step_result(i, cl, cm, to_cuda(stream));
    return GBVLM_OK;
}

int gbvlm_uvlm_step_graph(gbvlm_uvlm h, int64_t* step_index, double* cl, double* cm, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl, "null argument");
    int rc = h->impl->step_graph(to_cuda(stream));
    if (rc) return rc;
    auto* u = h->impl;
    const int64_t i = u->last_step();
    if (step_index) *step_index = i;
    if (cl || cm) return u->step_result(i, cl, cm, to_cuda(stream));
    return GBVLM_OK;
}

int gbvlm_uvlm_loop_create(gbvlm_uvlm_loop* out, gbvlm_uvlm h, double poll_s) {
    GB_REQUIRE(out && h && h->impl, "null argument");
    GB_REQUIRE(poll_s > 0 && poll_s <= 1.0, "poll_s=%g outside (0, 1] s", poll_s);
    auto* u = dynamic_cast<UvlmState<float>*>(h->impl);
    GB_REQUIRE(u, "UVLM request loop: float runs only");
    GB_REQUIRE(!u->looping, "UVLM request loop: this case already has one");
    GB_REQUIRE(!u->roll_, "UVLM request loop: roll-up runs step on the host");
    GB_REQUIRE(u->next_step >= 1, "UVLM request loop: take the first step with gbvlm_uvlm_step");
    GB_REQUIRE(u->next_step + 1 < u->t_steps, "UVLM: all %lld steps done (wake capacity)", (long long)u->t_steps);
    int dev = 0, native = 0;
    GB_CUDA(cudaGetDevice(&dev));
    GB_CUDA(cudaDeviceGetAttribute(&native, cudaDevAttrHostNativeAtomicSupported, dev));
    GB_REQUIRE(native, "UVLM request loop: the device has no native atomics on host memory");
    auto* l = new gbvlm_uvlm_loop_s();
    l->owner = h;
    l->u = u;
    l->base_step = u->next_step;
    l->cap = u->t_steps - 1 - u->next_step;
    auto fail = [&](int rc) {
        delete l;
        return rc;
    };
    int rc = u->prepare_dev(0);
    if (rc) return fail(rc);
    cudaError_t e = cudaStreamCreateWithFlags(&l->st, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaHostAlloc((void**)&l->ctl, sizeof(LoopCtl), cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostAlloc((void**)&l->rec, sizeof(LoopRec) * (size_t)l->cap, cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void**)&l->ctl_d, l->ctl, 0);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void**)&l->rec_d, l->rec, 0);
    if (e != cudaSuccess) return fail(cuda_fail(e, "UVLM request loop set-up", __FILE__, __LINE__));
    memset(l->ctl, 0, sizeof(LoopCtl));
    memset(l->rec, 0, sizeof(LoopRec) * (size_t)l->cap);
    // the device step counter at the case's next step
    e = cudaMemcpy(u->d_idx, &u->next_step, sizeof(int64_t), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail(cuda_fail(e, "UVLM request loop set-up", __FILE__, __LINE__));
    u->dev_idx = u->next_step;
    // graph: while (cond) { device-indexed step; next }
    cudaGraphConditionalHandle cond;
    cudaGraphNode_t nw;
    cudaGraphNodeParams wp = {};
    e = cudaGraphCreate(&l->graph, 0);
    if (e == cudaSuccess) e = cudaGraphConditionalHandleCreate(&cond, l->graph, 1, cudaGraphCondAssignDefault);
    if (e == cudaSuccess) {
        wp.type = cudaGraphNodeTypeConditional;
        wp.conditional.handle = cond;
        wp.conditional.type = cudaGraphCondTypeWhile;
        wp.conditional.size = 1;
        e = cudaGraphAddNode(&nw, l->graph, nullptr, nullptr, 0, &wp);
    }
    if (e == cudaSuccess)
        e = cudaStreamBeginCaptureToGraph(l->st, wp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                          cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return fail(cuda_fail(e, "UVLM request loop graph", __FILE__, __LINE__));
    rc = u->enqueue_dev_step(l->st);
    if (rc == GBVLM_OK) {
        const uint64_t poll_ns = (uint64_t)(poll_s * 1e9);
        const int* words[2];
        lu_solve_word_addresses(u->lu, words);
        k_uvlm_loop_next<<<1, 32, 0, l->st>>>(l->ctl_d, l->rec_d, u->d_idx, u->res, u->t_steps - 2, words[0], words[1],
                                              poll_ns, cond);
        const cudaError_t le = cudaGetLastError();
        if (le != cudaSuccess) rc = cuda_fail(le, "k_uvlm_loop_next", __FILE__, __LINE__);
    }
    cudaGraph_t got = nullptr;
    e = cudaStreamEndCapture(l->st, &got);
    if (rc) return fail(rc);
    if (e == cudaSuccess) e = cudaGraphInstantiate(&l->exec, l->graph, 0);
    if (e != cudaSuccess) return fail(cuda_fail(e, "UVLM request loop graph", __FILE__, __LINE__));
    u->looping = true;
    *out = l;
    return GBVLM_OK;
}

int gbvlm_uvlm_loop_submit(gbvlm_uvlm_loop l, int64_t* ticket) {
    GB_REQUIRE(l && ticket, "null argument");
    std::lock_guard<std::mutex> g(l->mu);
    GB_REQUIRE(l->enq < l->cap, "UVLM request loop: the wake holds %lld more steps", (long long)l->cap);
    GB_REQUIRE(!__atomic_load_n(&l->ctl->stop, __ATOMIC_SEQ_CST), "UVLM request loop: stopped");
    const int64_t t = ++l->enq;
    __atomic_store_n(&l->ctl->enq, t, __ATOMIC_SEQ_CST);
    std::atomic_thread_fence(std::memory_order_seq_cst);
    int32_t idle = 0;
    if (__atomic_load_n(&l->ctl->state, __ATOMIC_SEQ_CST) == 0 &&
        __atomic_compare_exchange_n(&l->ctl->state, &idle, 1, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {
        GB_CUDA(cudaGraphLaunch(l->exec, l->st));
        l->launches++;
    }
    *ticket = t;
    return GBVLM_OK;
}

int gbvlm_uvlm_loop_wait(gbvlm_uvlm_loop l, int64_t ticket, double timeout_s, int64_t* step_index, double* cl,
                         double* cm) {
    GB_REQUIRE(l && ticket >= 1 && timeout_s >= 0, "bad arguments");
    GB_REQUIRE(ticket <= l->enq, "UVLM request loop: ticket %lld not submitted", (long long)ticket);
    const auto deadline = std::chrono::steady_clock::now() + std::chrono::duration<double>(timeout_s);
    while (__atomic_load_n(&l->ctl->done, __ATOMIC_ACQUIRE) < ticket) {
        if (__atomic_load_n(&l->ctl->error, __ATOMIC_ACQUIRE)) {
            set_error("UVLM request loop: the wake is full");
            return GBVLM_ERR_ARG;
        }
        const cudaError_t q = cudaStreamQuery(l->st);
        if (q != cudaSuccess && q != cudaErrorNotReady) return cuda_fail(q, "UVLM request loop", __FILE__, __LINE__);
        if (std::chrono::steady_clock::now() > deadline) {
            set_error("UVLM request loop: ticket %lld not done within %g s", (long long)ticket, timeout_s);
            return GBVLM_ERR_CUDA;
        }
        std::this_thread::sleep_for(std::chrono::microseconds(20));
    }
    const LoopRec& r = l->rec[ticket - 1];
    if (step_index) *step_index = r.step;
    if (cl) *cl = r.c[0];
    if (cm)
        for (int k = 0; k < 3; k++) cm[k] = r.c[1 + k];
    if (r.failed) {
        set_error("UVLM request loop: step %lld: a triangular solve's block timed out waiting for the blocks it depends on",
                  (long long)r.step);
        return GBVLM_ERR_CUDA;
    }
    return GBVLM_OK;
}

int gbvlm_uvlm_loop_stats(gbvlm_uvlm_loop l, int64_t* submitted, int64_t* completed, int64_t* launches) {
    GB_REQUIRE(l, "null argument");
    std::lock_guard<std::mutex> g(l->mu);
    if (submitted) *submitted = l->enq;
    if (completed) *completed = __atomic_load_n(&l->ctl->done, __ATOMIC_ACQUIRE);
    if (launches) *launches = l->launches;
    return GBVLM_OK;
}

int gbvlm_uvlm_loop_destroy(gbvlm_uvlm_loop l) {
    if (!l) return GBVLM_OK;
    int rc = GBVLM_OK;
    {
        std::lock_guard<std::mutex> g(l->mu);
        __atomic_store_n(&l->ctl->stop, 1, __ATOMIC_SEQ_CST);
    }
    // a running graph sees the stop flag within its poll wait and ends
    cudaError_t e = cudaStreamSynchronize(l->st);
    if (e != cudaSuccess) rc = cuda_fail(e, "UVLM request loop", __FILE__, __LINE__);
    // the case continues host-stepped from where the loop left it
    const int64_t done = __atomic_load_n(&l->ctl->done, __ATOMIC_ACQUIRE);
    l->u->next_step = l->base_step + done;
    l->u->dev_idx = l->u->next_step;
    l->u->looping = false;
    delete l;
    return rc;
}

int gbvlm_uvlm_results(gbvlm_uvlm h, double* cl, double* cm, double* gamma_last, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl, "null argument");
    return h->impl->results(cl, cm, gamma_last, to_cuda(stream));
}

int gbvlm_aero2dof_create(gbvlm_aero2dof* out, int32_t nsurf, const gbvlm_dims* dims, const float* const* verts_init,
                          const int32_t* lifting, const gbvlm_2dof_vars* vars, double t_final, int64_t* t_steps,
                          double* dt, gbvlm_stream stream) {
    GB_REQUIRE(out && dims && verts_init && lifting && vars, "null argument");
    GB_REQUIRE(nsurf >= 1 && nsurf <= GBVLM_MAX_SURFACES, "nsurf=%d outside [1, %d]", nsurf, GBVLM_MAX_SURFACES);
    GB_REQUIRE(vars->b > 0 && vars->mu > 0 && vars->r_a > 0 && vars->U_a > 0, "aeroelastic 2-DOF: bad parameters");
    for (int m = 0; m < nsurf; m++) GB_REQUIRE(verts_init[m] && dims[m].ns >= 1 && dims[m].nc >= 1, "surface %d", m);
    GB_REQUIRE(dims[nsurf - 1].nc >= 2, "aeroelastic 2-DOF: the last surface needs two chordwise panels (time step)");
    auto* h = new Aero2Dof();
    int rc = h->init(nsurf, dims, verts_init, lifting, *vars, t_final, to_cuda(stream));
    if (rc) {
        delete h;
        return rc;
    }
    if (t_steps) *t_steps = h->t_steps;
    if (dt) *dt = h->dt;
    *out = (gbvlm_aero2dof)h;
    return GBVLM_OK;
}

int gbvlm_aero2dof_destroy(gbvlm_aero2dof h) {
    delete (Aero2Dof*)h;
    return GBVLM_OK;
}

int gbvlm_aero2dof_run(gbvlm_aero2dof h, int64_t steps, int32_t max_iter, gbvlm_stream stream) {
    GB_REQUIRE(h && steps >= 0 && max_iter >= 1, "bad arguments");
    return ((Aero2Dof*)h)->run(steps, max_iter, to_cuda(stream));
}

int gbvlm_test_aero2dof_withhold(gbvlm_aero2dof h, gbvlm_stream stream) {
    GB_REQUIRE(h, "null argument");
    return gbvlm_test_lu_withhold(((Aero2Dof*)h)->lu, stream);
}

int gbvlm_test_uvlm_withhold(gbvlm_uvlm h, gbvlm_stream stream) {
    GB_REQUIRE(h && h->impl, "null argument");
    auto* u = dynamic_cast<UvlmState<float>*>(h->impl);
    GB_REQUIRE(u, "float runs only");
    return gbvlm_test_lu_withhold(u->lu, stream);
}

int gbvlm_aero2dof_results(gbvlm_aero2dof h, int64_t* steps_done, double* u, double* v, double* a, double* F,
                           int32_t* iters, gbvlm_stream stream) {
    GB_REQUIRE(h, "null argument");
    Aero2Dof* s = (Aero2Dof*)h;
    cudaStream_t st = to_cuda(stream);
    const size_t nb = sizeof(double) * 2 * (size_t)(s->done + 1);
    if (u) GB_CUDA(cudaMemcpyAsync(u, s->u, nb, cudaMemcpyDeviceToHost, st));
    if (v) GB_CUDA(cudaMemcpyAsync(v, s->v, nb, cudaMemcpyDeviceToHost, st));
    if (a) GB_CUDA(cudaMemcpyAsync(a, s->a, nb, cudaMemcpyDeviceToHost, st));
    if (F) GB_CUDA(cudaMemcpyAsync(F, s->F, nb, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    if (steps_done) *steps_done = s->done;
    if (iters)
        for (int64_t k = 0; k < s->done; k++) iters[k] = s->iters[k];
    return GBVLM_OK;
}

}  // extern "C"
