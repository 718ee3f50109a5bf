// Per-operator kernels of the vortex-lattice hot path (the vlm::Backend
// operator set) in float and double, and their C-ABI entry points.
//
// Layout contract: see include/gbvlm.h.  Kernels are templated on the
// precision T; the float instantiation keeps the reference's float
// semantics (cut-offs, 5000-row wake window), the double one the reference's
// double kernels (vlm_backend_cpu_kernels.ispc:383-502).
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <mutex>
#include <type_traits>
#include <vector>

#include "gbvlm_internal.h"
#include "gbvlm_loads.cuh"
#include "gbvlm_math.cuh"
#include "gbvlm_walk.cuh"

namespace gbvlm {

// ---------------------------------------------------------------------------
// error state
// ---------------------------------------------------------------------------
static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
    set_error("CUDA error %s (%s) in %s at %s:%d", cudaGetErrorName(e), cudaGetErrorString(e), what, file, line);
    return e == cudaErrorMemoryAllocation ? GBVLM_ERR_NOMEM : GBVLM_ERR_CUDA;
}

void* host_scratch(size_t bytes) {
    static thread_local void* p = nullptr;
    static thread_local size_t cap = 0;
    if (bytes > cap) {
        if (p) cudaFreeHost(p);
        cap = bytes < 4096 ? 4096 : bytes;
        if (cudaMallocHost(&p, cap) != cudaSuccess) {
            p = nullptr;
            cap = 0;
        }
    }
    return p;
}

// Scratch for partial sums and small reductions, one buffer per (thread,
// device): calls from different host threads (each with its own stream) never
// share one, and a grow only has to wait for the calling thread's stream.  It
// starts at the partial sums' limit (LT_SCRATCH doubles), so that only sums over
// more points than that let it grow: a captured call that follows any other call
// of the thread, with fewer wake rows, finds it large enough.
int device_scratch(size_t bytes, void** out, cudaStream_t s) {
    static thread_local std::vector<std::pair<void*, size_t>> per_dev(64, {nullptr, 0});
    int dev = 0;
    GB_CUDA(cudaGetDevice(&dev));
    GB_REQUIRE(dev >= 0 && dev < 64, "device index %d out of range", dev);
    auto& slot = per_dev[dev];
    if (bytes > slot.second) {
        if (slot.first) {
            GB_CUDA(cudaStreamSynchronize(s));
            GB_CUDA(cudaFree(slot.first));
        }
        constexpr size_t least = sizeof(double) * (1 << 20);
        const size_t cap = bytes < least ? least : bytes;
        GB_CUDA(cudaMalloc(&slot.first, cap));
        slot.second = cap;
    }
    *out = slot.first;
    return GBVLM_OK;
}

// ---------------------------------------------------------------------------
// multi-surface argument table passed by value
// ---------------------------------------------------------------------------
template <class T>
struct Surfs {
    int32_t n;
    int64_t ns[GBVLM_MAX_SURFACES], nc[GBVLM_MAX_SURFACES], nwv[GBVLM_MAX_SURFACES];
    int64_t poff[GBVLM_MAX_SURFACES + 1];  // packed panel offsets
    const T* a[GBVLM_MAX_SURFACES];
    const T* b[GBVLM_MAX_SURFACES];
    const T* c[GBVLM_MAX_SURFACES];
    const T* d[GBVLM_MAX_SURFACES];
    T* o0[GBVLM_MAX_SURFACES];
    T* o1[GBVLM_MAX_SURFACES];
    T* o2[GBVLM_MAX_SURFACES];
    int32_t flag[GBVLM_MAX_SURFACES];
};

template <class T>
static int make_surfs(Surfs<T>& s, int32_t nsurf, const gbvlm_dims* dims) {
    GB_REQUIRE(nsurf >= 1 && nsurf <= GBVLM_MAX_SURFACES, "nsurf=%d outside [1, %d]", nsurf, GBVLM_MAX_SURFACES);
    GB_REQUIRE(dims != nullptr, "dims is null");
    memset(&s, 0, sizeof(s));
    s.n = nsurf;
    s.poff[0] = 0;
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(dims[m].ns >= 1 && dims[m].nc >= 1, "surface %d has ns=%lld nc=%lld", m, (long long)dims[m].ns,
                   (long long)dims[m].nc);
        s.ns[m] = dims[m].ns;
        s.nc[m] = dims[m].nc;
        s.nwv[m] = dims[m].nwv;
        s.poff[m + 1] = s.poff[m] + dims[m].ns * dims[m].nc;
    }
    return GBVLM_OK;
}

template <class T>
__device__ __forceinline__ int find_surf(const Surfs<T>& s, int64_t p) {
    int m = 0;
    while (m + 1 < s.n && p >= s.poff[m + 1]) m++;
    return m;
}

// ---------------------------------------------------------------------------
// a6: mesh metrics (vlm_backend_cpu.cpp:391-433)
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_mesh_metrics(Surfs<T> s, T factor) {
    int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g >= s.poff[s.n]) return;
    int m = find_surf(s, g);
    int64_t p = g - s.poff[m], ns = s.ns[m], nc = s.nc[m];
    int64_t i = p % ns, j = p / ns;
    const T* v = s.a[m];
    int64_t vld = (ns + 1) * (nc + 1), np = ns * nc;
    int64_t a = i + j * (ns + 1), b = a + 1, c = b + (ns + 1), d = a + (ns + 1);
    V3<T> v0{v[a], v[vld + a], v[2 * vld + a]}, v1{v[b], v[vld + b], v[2 * vld + b]};
    V3<T> v2{v[c], v[vld + c], v[2 * vld + c]}, v3_{v[d], v[vld + d], v[2 * vld + d]};
    V3<T> nn = cross(v3_ - v1, v2 - v0);
    T l = dsqrt(len2(nn));
    T* col = s.o0[m];
    T* nor = s.o1[m];
    T* ar = s.o2[m];
    nor[p] = nn.x / l;
    nor[np + p] = nn.y / l;
    nor[2 * np + p] = nn.z / l;
    V3<T> f = v3_ - v0, bb = v2 - v0, e = v1 - v0;
    ar[p] = (T)0.5 * (dsqrt(len2(cross(f, bb))) + dsqrt(len2(cross(bb, e))));
    V3<T> ch = (T)0.5 * (((v2 + v3_) - v0) - v1);
    V3<T> cp = (T)0.5 * (v0 + v1) + factor * ch;
    col[p] = cp.x;
    col[np + p] = cp.y;
    col[2 * np + p] = cp.z;
}

float aoa_factor(float alpha) {
    return (alpha < EPS_F) ? 0.5f : 0.5f * (alpha / (sinf(alpha) + EPS_F));
}
double aoa_factor(double alpha) {
    return (alpha < (double)EPS_F) ? 0.5 : 0.5 * (alpha / (sin(alpha) + (double)EPS_F));
}

template <class T>
static int mesh_metrics(T alpha, int32_t nsurf, const gbvlm_dims* dims, const T* const* verts, T* const* colloc,
                        T* const* normals, T* const* areas, cudaStream_t st) {
    Surfs<T> s;
    int rc = make_surfs(s, nsurf, dims);
    if (rc) return rc;
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(verts[m] && colloc[m] && normals[m] && areas[m], "null pointer for surface %d", m);
        s.a[m] = verts[m];
        s.o0[m] = colloc[m];
        s.o1[m] = normals[m];
        s.o2[m] = areas[m];
    }
    int64_t n = s.poff[nsurf];
    k_mesh_metrics<T><<<(unsigned)cdiv(n, 256), 256, 0, st>>>(s, aoa_factor(alpha));
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}

// ---------------------------------------------------------------------------
// a1: AIC assembly, one launch per (influenced, influencing) surface pair
// (vlm_backend_cpu.cpp:84-148).  Block = LHS_THREADS collocation points (one per
// thread, each with its y-mirror) x a piece of the influencing surface, ROWS
// ring rows x `span` rings, staged in shared memory with its segment vectors;
// lattice_rings evaluates each segment once for the two rings it bounds, 2.25
// to 2.5 segments and 1.25 to 1.5 vertices per ring and point where the
// ring-by-ring walk took three and two.  The block of the last ring row adds
// the wake rows to the trailing-edge columns.
// Bound: the fp32 (fp64) pipe; small surfaces, the number of blocks, so the
// pieces shrink until the launch covers the SMs twice (a ring's value does not
// depend on the cut).
// ---------------------------------------------------------------------------
constexpr int LHS_THREADS = 64;
constexpr int LHS_SPAN = 32;  // rings of a piece at most

template <class T>
struct LhsPair {
    T* lhs;
    int64_t ld;
    const T* colloc;
    const T* normals;
    int64_t np_i;
    const T* vw;
    int64_t ns, nc;
    const T* vk;
    int64_t nwv;
    int32_t iteration;
    T sigma2;
    int64_t row_off, col_off;
};

// lines [r0, r0 + nl) and vertices [k0, k0 + nk] of the lattice v (n vertices per line) into shared memory
template <class T>
__device__ __forceinline__ void stage_piece(const T* v, int64_t n, int64_t vld, int64_t r0, int64_t k0, int nl, int nk,
                                            int W, Quad<T>* sv, Quad<T>* ss, Quad<T>* sc) {
    for (int e = threadIdx.x; e < nl * (nk + 1); e += blockDim.x) {
        const int li = e / (nk + 1), k = e - li * (nk + 1);
        const int64_t vi = k0 + k + (r0 + li) * n;
        const T x = v[vi], y = v[vld + vi], z = v[2 * vld + vi];
        sv[li * W + k] = Quad<T>{x, y, z, 0};
        if (k > 0) ss[li * W + k] = Quad<T>{x - v[vi - 1], y - v[vld + vi - 1], z - v[2 * vld + vi - 1], 0};
        if (li + 1 < nl) sc[li * W + k] = Quad<T>{v[vi + n] - x, v[vld + vi + n] - y, v[2 * vld + vi + n] - z, 0};
    }
}

template <class T, bool SIGMA, int ROWS>
__global__ void __launch_bounds__(LHS_THREADS) k_lhs_pair(LhsPair<T> a) {
    constexpr int LR = ROWS + 1, W = LHS_SPAN + 1;
    __shared__ Quad<T> sv[LR * W], ss[LR * W], sc[LR * W];
    const int64_t c0 = (int64_t)blockIdx.y * ROWS;
    const int64_t s0 = (int64_t)blockIdx.z * a.ns / gridDim.z, s1 = (int64_t)(blockIdx.z + 1) * a.ns / gridDim.z;
    const int nr = (int)min((int64_t)ROWS, a.nc - c0), nk = (int)(s1 - s0);
    const int64_t n = a.ns + 1;
    stage_piece<T>(a.vw, n, n * (a.nc + 1), c0, s0, nr + 1, nk, W, sv, ss, sc);
    const int64_t i = (int64_t)blockIdx.x * LHS_THREADS + threadIdx.x;
    const bool active = i < a.np_i;
    const int64_t ip = active ? i : 0;
    const T px = a.colloc[ip], py = a.colloc[a.np_i + ip], pz = a.colloc[2 * a.np_i + ip];
    const T nx = a.normals[ip], ny = a.normals[a.np_i + ip], nz = a.normals[2 * a.np_i + ip];
    T* out = a.lhs + (a.row_off + ip) + (a.col_off + c0 * a.ns + s0) * a.ld;
    __syncthreads();
    lattice_rings<T, SIGMA, LR>(sv, ss, sc, W, nr + 1, nk, px, py, pz, nx, ny, nz, a.sigma2, [&](int r, int k, T val) {
        if (active) out[(r * a.ns + k) * a.ld] += val * inv_four_pi<T>();
    });
    if (c0 + nr < a.nc) return;
    out += (int64_t)(nr - 1) * a.ns * a.ld;
    for (int32_t it = 0; it < a.iteration; it++) {
        __syncthreads();
        stage_piece<T>(a.vk, n, n * a.nwv, a.nwv - 2 - it, s0, 2, nk, W, sv, ss, sc);
        __syncthreads();
        lattice_rings<T, SIGMA, 2>(sv, ss, sc, W, 2, nk, px, py, pz, nx, ny, nz, a.sigma2, [&](int, int k, T val) {
            if (active) out[k * a.ld] += val * inv_four_pi<T>();
        });
    }
}

template <class T>
static int lhs_assemble(T* lhs, int64_t ld, int32_t nsurf, const gbvlm_dims* dims, const T* const* colloc,
                        const T* const* normals, const T* const* verts_wing, const T* const* verts_wake,
                        int32_t iteration, T sigma, cudaStream_t st) {
    Surfs<T> s;
    int rc = make_surfs(s, nsurf, dims);
    if (rc) return rc;
    GB_REQUIRE(lhs != nullptr, "lhs is null");
    GB_REQUIRE(iteration >= 0, "iteration < 0");
    const int64_t n = s.poff[nsurf];
    GB_REQUIRE(ld >= n, "ld=%lld < n=%lld", (long long)ld, (long long)n);
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(colloc[m] && normals[m] && verts_wing[m], "null pointer for surface %d", m);
        if (iteration > 0) {
            GB_REQUIRE(verts_wake && verts_wake[m], "wake of surface %d is null", m);
            GB_REQUIRE(dims[m].nwv >= iteration + 1, "surface %d: nwv=%lld < iteration+1", m, (long long)dims[m].nwv);
        }
    }
    for (int mj = 0; mj < nsurf; mj++) {
        for (int mi = 0; mi < nsurf; mi++) {
            LhsPair<T> a;
            a.lhs = lhs;
            a.ld = ld;
            a.colloc = colloc[mi];
            a.normals = normals[mi];
            a.np_i = s.ns[mi] * s.nc[mi];
            a.vw = verts_wing[mj];
            a.ns = s.ns[mj];
            a.nc = s.nc[mj];
            a.vk = iteration > 0 ? verts_wake[mj] : nullptr;
            a.nwv = dims[mj].nwv;
            a.iteration = iteration;
            a.sigma2 = sigma * sigma;
            a.row_off = s.poff[mi];
            a.col_off = s.poff[mj];
            // four ring rows x 32 rings per piece, fewer until the blocks cover the SMs twice
            int rows = 4;
            int64_t span = LHS_SPAN;
            auto blocks = [&]() { return cdiv(a.np_i, (int64_t)LHS_THREADS) * cdiv(a.nc, (int64_t)rows) * cdiv(a.ns, span); };
            if (blocks() < 2 * sm_count()) rows = 2;
            while (span > 8 && blocks() < 2 * sm_count()) span /= 2;
            dim3 grid((unsigned)cdiv(a.np_i, (int64_t)LHS_THREADS), (unsigned)cdiv(a.nc, (int64_t)rows),
                      (unsigned)cdiv(a.ns, span));
            auto launch = [&](auto SIGMA) {
                constexpr bool sg = decltype(SIGMA)::value;
                if (rows == 4) k_lhs_pair<T, sg, 4><<<grid, LHS_THREADS, 0, st>>>(a);
                else k_lhs_pair<T, sg, 2><<<grid, LHS_THREADS, 0, st>>>(a);
            };
            if (sigma != (T)0) launch(std::true_type{});
            else launch(std::false_type{});
            GB_LAUNCH_CHECK();
        }
    }
    return GBVLM_OK;
}

// The same AIC ring by ring, for the harmonic-balance solver
// (gbvlm_internal.h): block = 128 collocation points x one ring row in chunks of
// 256 rings; along the span a thread keeps the left vertex terms and the left
// chordwise segment of the previous ring.
constexpr int LHR_THREADS = 128, LHR_SPAN = 256;

__global__ void __launch_bounds__(LHR_THREADS) k_lhs_rings(LhsPair<double> a) {
    constexpr int W = LHR_SPAN + 1;
    __shared__ double sv[6 * W];
    const int64_t c = blockIdx.y, s0 = (int64_t)blockIdx.z * LHR_SPAN;
    const int nv = (int)(min(s0 + (int64_t)LHR_SPAN, a.ns) - s0 + 1);
    const int64_t vld = (a.ns + 1) * (a.nc + 1);
    for (int t = threadIdx.x; t < 2 * nv; t += LHR_THREADS) {
        const int r = t / nv, sl = t - r * nv;
        const int64_t vi = (s0 + sl) + (c + r) * (a.ns + 1);
        for (int k = 0; k < 3; k++) sv[(r * 3 + k) * W + sl] = a.vw[k * vld + vi];
    }
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * LHR_THREADS + threadIdx.x;
    if (i >= a.np_i) return;
    const double px = a.colloc[i], py = a.colloc[a.np_i + i], pz = a.colloc[2 * a.np_i + i];
    const double nx = a.normals[i], ny = a.normals[a.np_i + i], nz = a.normals[2 * a.np_i + i];
    double* out = a.lhs + (a.row_off + i) + (a.col_off + c * a.ns) * a.ld;
    strip_normal<double, false>(sv, sv + 3 * W, W, nv, px, py, pz, nx, ny, nz, 0.0, [&](int k, double val) {
        out[(s0 + k) * a.ld] += val * inv_four_pi<double>();
    });
}

int lhs_assemble_rings_f64(double* lhs, int64_t ld, int32_t nsurf, const gbvlm_dims* dims,
                           const double* const* colloc, const double* const* normals,
                           const double* const* verts_wing, cudaStream_t st) {
    Surfs<double> s;
    int rc = make_surfs(s, nsurf, dims);
    if (rc) return rc;
    GB_REQUIRE(lhs && ld >= s.poff[nsurf], "bad lhs");
    for (int mj = 0; mj < nsurf; mj++)
        for (int mi = 0; mi < nsurf; mi++) {
            LhsPair<double> a = {};
            a.lhs = lhs;
            a.ld = ld;
            a.colloc = colloc[mi];
            a.normals = normals[mi];
            a.np_i = s.ns[mi] * s.nc[mi];
            a.vw = verts_wing[mj];
            a.ns = s.ns[mj];
            a.nc = s.nc[mj];
            a.row_off = s.poff[mi];
            a.col_off = s.poff[mj];
            k_lhs_rings<<<dim3((unsigned)cdiv(a.np_i, (int64_t)LHR_THREADS), (unsigned)a.nc,
                               (unsigned)cdiv(a.ns, (int64_t)LHR_SPAN)),
                          LHR_THREADS, 0, st>>>(a);
            GB_LAUNCH_CHECK();
        }
    return GBVLM_OK;
}

// ---------------------------------------------------------------------------
// a2: rhs += -(V . n) (vlm_backend_cpu.cpp:156-179)
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_rhs_velocities(Surfs<T> s, T* rhs) {
    int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g >= s.poff[s.n]) return;
    int m = find_surf(s, g);
    int64_t p = g - s.poff[m], np = s.ns[m] * s.nc[m];
    const T* n = s.a[m];
    const T* v = s.b[m];
    rhs[g] += -(v[p] * n[p] + v[np + p] * n[np + p] + v[2 * np + p] * n[2 * np + p]);
}

template <class T>
static int rhs_velocities(T* rhs, int32_t nsurf, const gbvlm_dims* dims, const T* const* normals,
                          const T* const* velocities, cudaStream_t st) {
    Surfs<T> s;
    int rc = make_surfs(s, nsurf, dims);
    if (rc) return rc;
    GB_REQUIRE(rhs != nullptr, "rhs is null");
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(normals[m] && velocities[m], "null pointer for surface %d", m);
        s.a[m] = normals[m];
        s.b[m] = velocities[m];
    }
    int64_t n = s.poff[nsurf];
    k_rhs_velocities<T><<<(unsigned)cdiv(n, 256), 256, 0, st>>>(s, rhs);
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}

// ---------------------------------------------------------------------------
// Lattice sums: a3, the wake influence on the RHS (vlm_backend_cpu.cpp:181-224),
// and a17, the free-wake roll-up (ispc:215-271).
//
// Grid x: blocks of LT_THREADS evaluation points, one per thread; grid y:
// slices of the sources (split-K).  The sources are cut into pieces of at most
// LatticeRows ring rows x LT_SPAN rings; a slice takes a run of consecutive
// pieces.  A piece is staged in shared memory as vertices, segment vectors and
// net segment strengths (lattice_walk), so each segment is evaluated once for
// the two rings it bounds.  Each slice writes its sums to a scratch table and
// a second kernel adds them in a fixed order, so results do not depend on
// scheduling.
//
// Bound: issue slots and the fp32 pipe (float), the fp64 pipe (double, 89 % busy).
// Per point and ring two segments and 1.25 vertices, each with its image: 150
// instructions, where the ring-by-ring walk spent 370.
// LatticeRows: a piece's last vertex line is formed again by the next piece, so
// (rows + 1) / rows vertices per ring; a line's relative vectors are 6
// registers in float, 12 in double, where three rows leave room for a third
// block per SM (1600 points x 8000 rings 3.81 ms with four rows, 3.01 with
// three).  LT_SPAN: short, so that a wake of a few rows still gives every SM
// work; each piece repeats one vertex column.  Full pieces of float are
// straight code without tests of the line count (370 -> 308 us below); the same
// in double costs registers (3.01 -> 3.31 ms).
// Measured (before -> after): 1600 points x 40,000 rings in float 595 -> 308 us,
// 8000 rings in double 7.0 -> 2.90 ms; roll-up of 12,150 vertices (95 blocks
// before, one per 128 points, which left SMs idle) 3417 -> 763 us.
// Not kept: the point and its image as the two halves of packed fp32
// instructions (a fifth fewer issue slots per ring, but 128 registers: 320 us),
// and the cut-offs left out of a first walk that a second one repeats where a
// lane met one (298 us, but the roll-up 763 -> 819).
// ---------------------------------------------------------------------------
constexpr int LT_THREADS = 128;
template <class T> struct LatticeRows { static constexpr int value = 4; };
template <> struct LatticeRows<double> { static constexpr int value = 3; };
constexpr int LT_SPAN = 32;
constexpr int LT_MIN_BLOCKS_F32 = 5;

template <class T>
struct LatticeArgs {
    // RHS: a = colloc, b = normals; roll-up: a = verts_wing, b = gamma_wing;
    // c = verts_wake, d = gamma_wake, flag = lifting; o0 = verts_wake (roll-up, written by the reduction)
    Surfs<T> s;
    int32_t iteration;
    int32_t window;  // 0 = no window
    T sigma2;
    T* partial;             // [slices][n_points], roll-up: [slices][3][n_points]
    const int64_t* it_dev;  // if set: the iteration, read on the device (the grid covers up to `iteration`)
    int64_t voff[GBVLM_MAX_SURFACES + 1];  // roll-up: packed moving-vertex offsets
    int64_t npts;
};

// one source lattice: vertex lines of n vertices, ring rows [first, first + rows)
template <class T>
struct Lattice {
    const T* v;
    const T* g;
    int64_t n, vld, first, rows, groups, chunks;
};

template <class T, bool ROLL>
__device__ __forceinline__ Lattice<T> lattice_of(const LatticeArgs<T>& w, int l, int64_t it) {
    const int m = ROLL ? l >> 1 : l;
    Lattice<T> L;
    L.n = w.s.ns[m] + 1;
    if (ROLL && !(l & 1)) {
        L.v = w.s.a[m];
        L.g = w.s.b[m];
        L.vld = L.n * (w.s.nc[m] + 1);
        L.first = 0;
        L.rows = w.s.nc[m];
    } else {
        L.v = w.s.c[m];
        L.g = w.s.d[m];
        L.vld = L.n * w.s.nwv[m];
        L.first = w.s.nwv[m] - it - 1;
        int64_t end = w.s.nwv[m] - 1;
        if (!ROLL && w.window > 0 && it > w.window) end = L.first + w.window;
        L.rows = w.s.flag[m] ? max(end - L.first, (int64_t)0) : 0;
    }
    L.groups = (L.rows + LatticeRows<T>::value - 1) / LatticeRows<T>::value;
    L.chunks = (L.n - 1 + LT_SPAN - 1) / LT_SPAN;
    return L;
}

template <class T, bool SIGMA, bool ROLL>
__global__ void __launch_bounds__(LT_THREADS, sizeof(T) == 4 ? LT_MIN_BLOCKS_F32 : 1) k_lattice_sum(LatticeArgs<T> w) {
    constexpr int ROWS = LatticeRows<T>::value, LR = ROWS + 1, W = LT_SPAN + 1;
    constexpr bool FAST = sizeof(T) == 4 && !SIGMA;  // full pieces as straight code
    __shared__ Quad<T> sv[LR * W], ss[LR * W], sc[LR * W];
    const int64_t g = (int64_t)blockIdx.x * LT_THREADS + threadIdx.x;
    const bool active = g < w.npts;
    T px = 0, py = 0, pz = 0, nx = 0, ny = 0, nz = 0;
    if (active) {
        if constexpr (ROLL) {
            int m = 0;
            while (m + 1 < w.s.n && g >= w.voff[m + 1]) m++;
            const int64_t n = w.s.ns[m] + 1, vld = n * w.s.nwv[m];
            const int64_t vi = (w.s.nwv[m] - w.iteration) * n + (g - w.voff[m]);
            px = w.s.c[m][vi]; py = w.s.c[m][vld + vi]; pz = w.s.c[m][2 * vld + vi];
        } else {
            const int m = find_surf(w.s, g);
            const int64_t p = g - w.s.poff[m], np = w.s.ns[m] * w.s.nc[m];
            px = w.s.a[m][p]; py = w.s.a[m][np + p]; pz = w.s.a[m][2 * np + p];
            nx = w.s.b[m][p]; ny = w.s.b[m][np + p]; nz = w.s.b[m][2 * np + p];
        }
    }
    const int64_t it = w.it_dev ? *w.it_dev : (int64_t)w.iteration;
    const int nlat = ROLL ? 2 * w.s.n : w.s.n;
    int64_t pieces = 0;
    for (int l = 0; l < nlat; l++) {
        const Lattice<T> L = lattice_of<T, ROLL>(w, l, it);
        pieces += L.groups * L.chunks;
    }
    // slices past the pieces of the current iteration contribute zero
    const int64_t per = (pieces + gridDim.y - 1) / gridDim.y;
    const int64_t u0 = (int64_t)blockIdx.y * per, u1 = min(u0 + per, pieces);
    T ax = 0, ay = 0, az = 0;  // RHS: the sum in ax
    int64_t base = 0;
    for (int l = 0; l < nlat && base < u1; l++) {
        const Lattice<T> L = lattice_of<T, ROLL>(w, l, it);
        const int64_t cnt = L.groups * L.chunks;
        for (int64_t u = max(u0, base); u < min(u1, base + cnt); u++) {
            const int64_t grp = (u - base) / L.chunks, ch = (u - base) - grp * L.chunks;
            const int64_t r0 = L.first + grp * ROWS, rend = L.first + L.rows;
            const int nr = (int)min((int64_t)ROWS, rend - r0);
            const int64_t k0 = ch * (L.n - 1) / L.chunks, k1 = (ch + 1) * (L.n - 1) / L.chunks;
            const int nk = (int)(k1 - k0), nl = nr + 1;
            __syncthreads();  // the previous piece has been read
            for (int e = threadIdx.x; e < nl * (nk + 1); e += LT_THREADS) {
                const int li = e / (nk + 1), k = e - li * (nk + 1);
                const int64_t row = r0 + li, col = k0 + k, vi = col + row * L.n;
                // strengths of the four rings around the vertex that the two segments bound; none outside the lattice
                const int64_t gi = row * (L.n - 1) + col;
                const bool here = row < rend, left = col > 0, right = col < L.n - 1, above = row > L.first;
                const T g_l = here && left ? L.g[gi - 1] : (T)0;
                const T g_r = here && right ? L.g[gi] : (T)0;
                const T g_al = above && left ? L.g[gi - 1 - (L.n - 1)] : (T)0;
                const T x = L.v[vi], y = L.v[L.vld + vi], z = L.v[2 * L.vld + vi];
                Quad<T> q{x, y, z, g_l - g_al};
                sv[li * W + k] = q;
                q = Quad<T>{0, 0, 0, g_l - g_r};
                if (k > 0) {
                    q.x = x - L.v[vi - 1];
                    q.y = y - L.v[L.vld + vi - 1];
                    q.z = z - L.v[2 * L.vld + vi - 1];
                }
                ss[li * W + k] = q;
                if (li < nr) sc[li * W + k] = Quad<T>{L.v[vi + L.n] - x, L.v[L.vld + vi + L.n] - y,
                                                      L.v[2 * L.vld + vi + L.n] - z, 0};
            }
            __syncthreads();
            T bx = 0, by = 0, bz = 0;  // the piece's own sums: fewer roundings of the running ones
            auto walk = [&](auto FULL) {
                lattice_walk<T, SIGMA, LR, decltype(FULL)::value>(
                    sv, ss, sc, W, nl, nk, k0 == 0, r0 + nr == rend, px, py, pz, w.sigma2,
                    [&](T gm, T q0, T q1, T cy, T cx0, T cx1, T cz0, T cz1) {
                        if constexpr (ROLL) {
                            q0 *= gm;
                            q1 *= gm;
                            bx += q0 * cx0 + q1 * cx1;
                            by += (q0 - q1) * cy;
                            bz += q0 * cz0 + q1 * cz1;
                        } else {
                            const T tn = cy * ny;
                            bx += gm * (q0 * (cx0 * nx + tn + cz0 * nz) + q1 * (cx1 * nx - tn + cz1 * nz));
                        }
                    });
            };
            if (FAST && nl == LR) walk(std::integral_constant<bool, FAST>{});
            else walk(std::false_type{});
            ax += bx;
            ay += by;
            az += bz;
        }
        base += cnt;
    }
    if (active) {
        const int64_t np = w.npts;
        if constexpr (ROLL) {
            T* o = w.partial + (int64_t)blockIdx.y * 3 * np + g;
            o[0] = ax;
            o[np] = ay;
            o[2 * np] = az;
        } else {
            w.partial[(int64_t)blockIdx.y * np + g] = ax;
        }
    }
}

// The slices' sums of a point, in order: LT_RED threads per point take every
// LT_RED-th slice, then the point's partial sums are added.
constexpr int LT_RED = 8;

template <class T>
__device__ __forceinline__ T slice_sum(const T* partial, int64_t slices, int64_t stride, int64_t at, bool active,
                                       T (*sh)[32]) {
    const int p = threadIdx.x & 31, q = threadIdx.x >> 5;
    T s = 0;
    if (active)
#pragma unroll 4
        for (int64_t k = q; k < slices; k += LT_RED) s += partial[k * stride + at];
    __syncthreads();  // the previous sum's use of sh
    sh[q][p] = s;
    __syncthreads();
    s = sh[0][p];
#pragma unroll
    for (int j = 1; j < LT_RED; j++) s += sh[j][p];
    return s;
}

template <class T>
__global__ void __launch_bounds__(32 * LT_RED) k_wake_reduce(const T* partial, int64_t slices, int64_t ntg, T* rhs) {
    __shared__ T sh[LT_RED][32];
    const int64_t g = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    const T s = slice_sum<T>(partial, slices, ntg, g, g < ntg, sh);
    if (g < ntg && threadIdx.x < 32) rhs[g] -= s * inv_four_pi<T>();
}

// moves the wake's vertices in place: every old position has been read
template <class T>
__global__ void __launch_bounds__(32 * LT_RED) k_roll_reduce(LatticeArgs<T> w, int64_t slices, T dt) {
    __shared__ T sh[LT_RED][32];
    const int64_t g = (int64_t)blockIdx.x * 32 + (threadIdx.x & 31);
    const bool on = g < w.npts;
    T v[3];
#pragma unroll
    for (int k = 0; k < 3; k++) v[k] = slice_sum<T>(w.partial, slices, 3 * w.npts, k * w.npts + g, on, sh);
    if (!on || threadIdx.x >= 32) return;
    int m = 0;
    while (m + 1 < w.s.n && g >= w.voff[m + 1]) m++;
    const int64_t n = w.s.ns[m] + 1, vld = n * w.s.nwv[m];
    const int64_t vi = (w.s.nwv[m] - w.iteration) * n + (g - w.voff[m]);
    const T sc = dt * inv_four_pi<T>();
#pragma unroll
    for (int k = 0; k < 3; k++) w.s.o0[m][k * vld + vi] += v[k] * sc;
}

template <class T>
static int64_t lattice_pieces(int64_t rows, int64_t ns) {
    return cdiv(rows, (int64_t)LatticeRows<T>::value) * cdiv(ns, (int64_t)LT_SPAN);
}

// Slices of `pieces` pieces for `npts` points: about 4 x `wake.waves` x SMs
// CTAs (tuned per shape; a CTA of one or two pieces is short, so the last
// wave's idle part is too), one piece each at least.  `cap`: values that the
// scratch holds, `vals` per point and slice.
static int64_t lattice_slices(int64_t pieces, int64_t npts, int64_t vals, int64_t cap) {
    int64_t want = cdiv(4 * tune().wake_waves * sm_count(), cdiv(npts, LT_THREADS));
    want = std::min<int64_t>(want, cap / (npts * vals));
    if (want < 1) want = 1;
    return cdiv(pieces, cdiv(pieces, want));
}

// partial sums of a launch are at most this many values (4 MiB of floats: the
// allocation-free entry point's array, so that it and the regular one cut the
// sums alike)
constexpr int64_t LT_SCRATCH = 1 << 20;

template <class T>
static int wake_influence(T* rhs, int32_t nsurf, const gbvlm_dims* dims, const T* const* gamma_wake,
                          const T* const* colloc, const T* const* normals, const T* const* verts_wake,
                          const int32_t* lifting, int32_t iteration, T sigma, int32_t window, T* scratch,
                          size_t scratch_elems, cudaStream_t st, const int64_t* it_dev = nullptr) {
    LatticeArgs<T> w;
    int rc = make_surfs(w.s, nsurf, dims);
    if (rc) return rc;
    GB_REQUIRE(rhs != nullptr, "rhs is null");
    GB_REQUIRE(lifting != nullptr, "lifting is null");
    GB_REQUIRE(iteration >= 0, "iteration < 0");
    w.it_dev = it_dev;
    w.iteration = iteration;
    w.window = window;
    w.sigma2 = sigma * sigma;
    int64_t pieces = 0;
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(colloc[m] && normals[m], "null pointer for surface %d", m);
        w.s.a[m] = colloc[m];
        w.s.b[m] = normals[m];
        w.s.flag[m] = lifting[m] ? 1 : 0;
        if (lifting[m] && iteration > 0) {
            GB_REQUIRE(verts_wake && verts_wake[m] && gamma_wake && gamma_wake[m], "wake of surface %d is null", m);
            GB_REQUIRE(dims[m].nwv >= iteration + 1, "surface %d: nwv=%lld < iteration+1", m, (long long)dims[m].nwv);
            w.s.c[m] = verts_wake[m];
            w.s.d[m] = gamma_wake[m];
            pieces += lattice_pieces<T>(window > 0 && iteration > window ? window : iteration, dims[m].ns);
        } else {
            w.s.flag[m] = 0;
        }
    }
    if (pieces == 0) return GBVLM_OK;
    const int64_t ntg = w.s.poff[nsurf];
    w.npts = ntg;
    const int64_t cap = scratch ? std::min<int64_t>((int64_t)scratch_elems, LT_SCRATCH) : LT_SCRATCH;
    const int64_t slices = lattice_slices(pieces, ntg, 1, cap);
    if (scratch == nullptr) {
        GB_REQUIRE(it_dev == nullptr, "the device-iteration form needs its own scratch");
        void* p = nullptr;
        rc = device_scratch(sizeof(T) * slices * ntg, &p, st);
        if (rc) return rc;
        scratch = (T*)p;
    } else {
        GB_REQUIRE((size_t)(slices * ntg) <= scratch_elems, "scratch too small: need %lld elements",
                   (long long)(slices * ntg));
    }
    w.partial = scratch;
    dim3 grid((unsigned)cdiv(ntg, LT_THREADS), (unsigned)slices);
    if (sigma != (T)0)
        k_lattice_sum<T, true, false><<<grid, LT_THREADS, 0, st>>>(w);
    else
        k_lattice_sum<T, false, false><<<grid, LT_THREADS, 0, st>>>(w);
    GB_LAUNCH_CHECK();
    k_wake_reduce<T><<<(unsigned)cdiv(ntg, 32), 32 * LT_RED, 0, st>>>(scratch, slices, ntg, rhs);
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}

template <class T>
static int wake_rollup(int32_t nsurf, const gbvlm_dims* dims, T* const* verts_wake, const T* const* verts_wing,
                       const T* const* gamma_wing, const T* const* gamma_wake, const int32_t* lifting, T sigma, T dt,
                       int32_t iteration, cudaStream_t st) {
    LatticeArgs<T> w;
    int rc = make_surfs(w.s, nsurf, dims);
    if (rc) return rc;
    GB_REQUIRE(lifting != nullptr, "lifting is null");
    GB_REQUIRE(iteration >= 0, "iteration < 0");
    if (iteration == 0) return GBVLM_OK;
    w.voff[0] = 0;
    int64_t pieces = 0;
    for (int m = 0; m < nsurf; m++) {
        GB_REQUIRE(verts_wake[m] && verts_wing[m] && gamma_wing[m], "null pointer for surface %d", m);
        GB_REQUIRE(dims[m].nwv >= iteration + 1, "surface %d: nwv=%lld < iteration+1", m, (long long)dims[m].nwv);
        w.s.a[m] = verts_wing[m];
        w.s.b[m] = gamma_wing[m];
        w.s.c[m] = verts_wake[m];
        w.s.d[m] = gamma_wake ? gamma_wake[m] : nullptr;
        w.s.o0[m] = verts_wake[m];
        w.s.flag[m] = lifting[m] ? 1 : 0;
        if (lifting[m]) GB_REQUIRE(gamma_wake && gamma_wake[m], "gamma_wake of surface %d is null", m);
        w.voff[m + 1] = w.voff[m] + (int64_t)iteration * (dims[m].ns + 1);
        pieces += lattice_pieces<T>(dims[m].nc, dims[m].ns) + (lifting[m] ? lattice_pieces<T>(iteration, dims[m].ns) : 0);
    }
    w.npts = w.voff[nsurf];
    w.iteration = iteration;
    w.window = 0;
    w.it_dev = nullptr;
    w.sigma2 = sigma * sigma;
    const int64_t slices = lattice_slices(pieces, w.npts, 3, LT_SCRATCH);
    void* scratch = nullptr;
    int64_t whole = 0;  // the wakes' vertices: the size does not depend on the iteration
    for (int m = 0; m < nsurf; m++) whole += dims[m].nwv * (dims[m].ns + 1);
    rc = device_scratch(sizeof(T) * std::max(3 * slices * w.npts, 3 * whole), &scratch, st);
    if (rc) return rc;
    w.partial = (T*)scratch;
    dim3 grid((unsigned)cdiv(w.npts, LT_THREADS), (unsigned)slices);
    if (sigma != (T)0)
        k_lattice_sum<T, true, true><<<grid, LT_THREADS, 0, st>>>(w);
    else
        k_lattice_sum<T, false, true><<<grid, LT_THREADS, 0, st>>>(w);
    GB_LAUNCH_CHECK();
    k_roll_reduce<T><<<(unsigned)cdiv(w.npts, 32), 32 * LT_RED, 0, st>>>(w, slices, dt);
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}

// ---------------------------------------------------------------------------
// a9: panel forces (vlm_backend_cpu.cpp:276-321), rho = 1
// ---------------------------------------------------------------------------
template <class T, bool UNSTEADY>
__global__ void k_forces(int64_t ns, int64_t nc, const T* vw, const T* gd, const T* dg, const T* vel, const T* ar,
                         const T* nor, T* f) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int64_t np = ns * nc;
    if (p >= np) return;
    int64_t i = p % ns, j = p / ns, vld = (ns + 1) * (nc + 1);
    int64_t a = i + j * (ns + 1), b = a + 1;
    const T rho = 1;
    V3<T> V{vel[p], vel[np + p], vel[2 * np + p]};
    V3<T> v0{vw[a], vw[vld + a], vw[2 * vld + a]}, v1{vw[b], vw[vld + b], vw[2 * vld + b]};
    V3<T> F = (rho * gd[p]) * cross(V, v1 - v0);
    if (UNSTEADY) {
        V3<T> n{nor[p], nor[np + p], nor[2 * np + p]};
        F = F + (rho * dg[p] * ar[p]) * n;
    }
    f[p] = F.x;
    f[np + p] = F.y;
    f[2 * np + p] = F.z;
}

// ---------------------------------------------------------------------------
// a10/a11/a12: reductions in double with compensation, one block
// ---------------------------------------------------------------------------
constexpr int RED_THREADS = 512;

// kind 0: cl = sum F.L ; kind 1: cm = sum (0.5(v0+v1) - ref) x F ; kind 2: sum x ; kind 3: mac numerator
template <class T>
__global__ void __launch_bounds__(RED_THREADS) k_reduce(int kind, int64_t ns, int64_t nc, const T* x, const T* vw,
                                                        double ax, double ay, double az, double* out) {
    __shared__ double sh[32];
    CSum s0, s1, s2;
    const int64_t np = ns * nc, vld = (ns + 1) * (nc + 1);
    if (kind == 0) {
        for (int64_t p = threadIdx.x; p < np; p += blockDim.x)
            s0.add((double)x[p] * ax + (double)x[np + p] * ay + (double)x[2 * np + p] * az);
    } else if (kind == 1) {
        for (int64_t p = threadIdx.x; p < np; p += blockDim.x) {
            int64_t i = p % ns, j = p / ns, a = i + j * (ns + 1), b = a + 1;
            double lx = 0.5 * ((double)vw[a] + (double)vw[b]) - ax;
            double ly = 0.5 * ((double)vw[vld + a] + (double)vw[vld + b]) - ay;
            double lz = 0.5 * ((double)vw[2 * vld + a] + (double)vw[2 * vld + b]) - az;
            double fx = x[p], fy = x[np + p], fz = x[2 * np + p];
            s0.add(ly * fz - lz * fy);
            s1.add(lz * fx - lx * fz);
            s2.add(lx * fy - ly * fx);
        }
    } else if (kind == 2) {
        for (int64_t p = threadIdx.x; p < ns; p += blockDim.x) s0.add((double)x[p]);
    } else {
        const int64_t last = nc * (ns + 1);
        for (int64_t i = threadIdx.x; i < ns; i += blockDim.x) {
            double dx0 = (double)vw[i] - vw[last + i], dy0 = (double)vw[vld + i] - vw[vld + last + i];
            double dz0 = (double)vw[2 * vld + i] - vw[2 * vld + last + i];
            double dx1 = (double)vw[i + 1] - vw[last + i + 1], dy1 = (double)vw[vld + i + 1] - vw[vld + last + i + 1];
            double dz1 = (double)vw[2 * vld + i + 1] - vw[2 * vld + last + i + 1];
            double c0 = sqrt(dx0 * dx0 + dy0 * dy0 + dz0 * dz0), c1 = sqrt(dx1 * dx1 + dy1 * dy1 + dz1 * dz1);
            double dx3 = (double)vw[i + 1] - vw[i], dy3 = (double)vw[vld + i + 1] - vw[vld + i];
            double dz3 = (double)vw[2 * vld + i + 1] - vw[2 * vld + i];
            s0.add(0.5 * (c0 * c0 + c1 * c1) * sqrt(dx3 * dx3 + dy3 * dy3 + dz3 * dz3));
        }
        // areas sum in s1 (x = areas)
        for (int64_t p = threadIdx.x; p < np; p += blockDim.x) s1.add((double)x[p]);
    }
    double r0 = block_sum(s0.value(), sh), r1 = block_sum(s1.value(), sh), r2 = block_sum(s2.value(), sh);
    if (threadIdx.x == 0) {
        out[0] = r0;
        out[1] = r1;
        out[2] = r2;
    }
}

template <class T>
static int reduce_sync(int kind, int64_t ns, int64_t nc, const T* x, const T* vw, double ax, double ay, double az,
                       double* host_out, cudaStream_t st) {
    void* d = nullptr;
    int rc = device_scratch(4 * sizeof(double), &d, st);
    if (rc) return rc;
    k_reduce<T><<<1, RED_THREADS, 0, st>>>(kind, ns, nc, x, vw, ax, ay, az, (double*)d);
    GB_LAUNCH_CHECK();
    double* h = (double*)host_scratch(4 * sizeof(double));
    GB_REQUIRE(h != nullptr, "pinned host allocation failed");
    GB_CUDA(cudaMemcpyAsync(h, d, 3 * sizeof(double), cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    host_out[0] = h[0];
    host_out[1] = h[1];
    host_out[2] = h[2];
    return GBVLM_OK;
}

// ---------------------------------------------------------------------------
// a13: wake gamma from trailing-edge Fourier coefficients (cpu.cpp:470-503)
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_gamma_wake(T* gw, int64_t ns, int64_t ncols, const T* co, int32_t H, T tn, T omega, T dt, int64_t it) {
    int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (g >= ns * it) return;
    const int64_t start = ncols - it;
    int64_t i = g % ns, j = start + g / ns;
    const int32_t U = 2 * H + 1;
    const T s0 = (T)1 / dsqrt((T)U), s2 = dsqrt((T)2 / (T)U);
    T v = co[i] * s0;
    for (int32_t h = 0; h < H; h++) {
        const T wk = omega * (T)(h + 1);
        T ph = wk * (tn - (T)(j - start + 1) * dt);
        T sn, cs;
        if constexpr (sizeof(T) == 4) {
            sincosf(ph, &sn, &cs);
        } else {
            sincos(ph, &sn, &cs);
        }
        v += co[i + (2 * h + 1) * ns] * cs * s2;
        v += co[i + (2 * h + 2) * ns] * sn * s2;
    }
    gw[i + j * ns] = v;
}

// ---------------------------------------------------------------------------
// a5 / a4: displacement and wake shedding
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_displace(Surfs<T> s) {
    int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    // vertex offsets in poff-like packing: reuse nwv as vertex counts
    int m = 0;
    int64_t base = 0;
    while (m < s.n) {
        int64_t nv = (s.ns[m] + 1) * (s.nc[m] + 1);
        if (g < base + nv) break;
        base += nv;
        m++;
    }
    if (m >= s.n) return;
    int64_t r = g - base, nv = (s.ns[m] + 1) * (s.nc[m] + 1);
    const T* tr = s.a[m];
    const T* in = s.b[m];
    T* out = s.o0[m];
    T x[4] = {in[r], in[nv + r], in[2 * nv + r], in[3 * nv + r]};
#pragma unroll
    for (int c = 0; c < 4; c++) {
        T acc = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) acc += x[k] * tr[c + 4 * k];
        out[c * nv + r] = acc;
    }
}

template <class T>
__global__ void k_wake_shed(Surfs<T> s, int32_t it) {
    int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int m = 0;
    int64_t base = 0;
    while (m < s.n) {
        int64_t cnt = 4 * (s.ns[m] + 1);
        if (g < base + cnt) break;
        base += cnt;
        m++;
    }
    if (m >= s.n) return;
    int64_t r = g - base, n = s.ns[m] + 1;
    int64_t k = r / n, i = r % n;
    const T* vw = s.a[m];
    T* vk = s.o0[m];
    int64_t vld = n * (s.nc[m] + 1), kld = n * s.nwv[m];
    vk[k * kld + i + (s.nwv[m] - 1 - it) * n] = vw[k * vld + i + s.nc[m] * n];
}

// ---------------------------------------------------------------------------
// a8: fused circulation update (vlm.cpp:442-458)
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_gamma_update(int64_t ns, int64_t nc, const T* x, T* g, T* gd, T* gw, int64_t wcol, const T* gp,
                               T* dgdt, T inv_dt) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= ns * nc) return;
    int64_t i = p % ns, j = p / ns;
    T v = x[p];
    g[p] = v;
    gd[p] = (j > 0) ? v - x[p - ns] : v;
    if (gw && j == nc - 1) gw[i + wcol * ns] = v;
    if (dgdt) dgdt[p] = (v - gp[p]) * inv_dt;
}

// ---------------------------------------------------------------------------
// Trefftz-plane drag (ispc:273-323): one block per spanwise ring
// ---------------------------------------------------------------------------
template <class T>
__global__ void k_trefftz(int64_t nv, int64_t nwv, const T* v, const T* gam, T sigma, double* partial) {
    __shared__ double sh[32];
    const double d = trefftz_ring(nv, nwv, v, gam, sigma, (int64_t)blockIdx.x, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = d;
}

__global__ void k_sum_partials(const double* p, int64_t n, double* out) {
    __shared__ double sh[32];
    CSum s;
    for (int64_t k = threadIdx.x; k < n; k += blockDim.x) s.add(p[k]);
    double r = block_sum(s.value(), sh);
    if (threadIdx.x == 0) out[0] = r;
}

template <class T>
static int trefftz(int64_t ns, int64_t nwv, const T* vk, const T* gw, const T* fs, T area, T sigma, T* out,
                   cudaStream_t st) {
    GB_REQUIRE(ns >= 1 && nwv >= 2, "trefftz needs ns>=1 and nwv>=2");
    GB_REQUIRE(vk && gw && fs && out, "null pointer");
    void* d = nullptr;
    int rc = device_scratch(sizeof(double) * (ns + 2), &d, st);
    if (rc) return rc;
    double* part = (double*)d;
    k_trefftz<T><<<(unsigned)ns, 128, 0, st>>>(ns + 1, nwv, vk, gw, (T)sqrt((double)(sigma * sigma)), part);
    GB_LAUNCH_CHECK();
    k_sum_partials<<<1, 256, 0, st>>>(part, ns, part + ns);
    GB_LAUNCH_CHECK();
    double* h = (double*)host_scratch(sizeof(double));
    GB_CUDA(cudaMemcpyAsync(h, part + ns, sizeof(double), cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    double v2 = (double)fs[0] * fs[0] + (double)fs[1] * fs[1] + (double)fs[2] * fs[2];
    *out = (T)(h[0] / (v2 * (double)area));
    return GBVLM_OK;
}

}  // namespace gbvlm

using namespace gbvlm;

// ===========================================================================
// C ABI
// ===========================================================================
namespace gbvlm {
// out[i] = length_of(a[i]) (kind 0), reciprocal(a[i]) (1); kind 2: out[2 i], out[2 i + 1] = the two quotients of
// a[2 i] / b[2 i] and a[2 i + 1] / b[2 i + 1]
__global__ void k_test_walk_math(int kind, int64_t n, const double* a, const double* b, double* out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (kind == 0) out[i] = length_of(a[i]);
    else if (kind == 1) out[i] = reciprocal(a[i]);
    else two_quotients(a[2 * i], b[2 * i], false, a[2 * i + 1], b[2 * i + 1], false, out[2 * i], out[2 * i + 1]);
}
}  // namespace gbvlm

extern "C" {
int gbvlm_test_walk_math(int32_t kind, int64_t n, const double* a, const double* b, double* out, gbvlm_stream stream) {
    GB_REQUIRE(kind >= 0 && kind <= 2 && n >= 1 && a && out && (kind != 2 || b), "bad arguments");
    k_test_walk_math<<<(unsigned)cdiv(n, 256), 256, 0, to_cuda(stream)>>>(kind, n, a, b, out);
    GB_LAUNCH_CHECK();
    return GBVLM_OK;
}


const char* gbvlm_last_error(void) { return g_err; }
int gbvlm_version(void) { return 10000; }

#define GB_BOTH(MACRO) MACRO(f32, float) MACRO(f64, double)

#define DEF_LHS(sfx, T)                                                                                       \
    int gbvlm_lhs_assemble_##sfx(T* lhs, int64_t ld, int32_t nsurf, const gbvlm_dims* dims,                 \
                                 const T* const* colloc, const T* const* normals, const T* const* verts_wing, \
                                 const T* const* verts_wake, int32_t iteration, T sigma, gbvlm_stream stream) { \
        GB_REQUIRE(colloc && normals && verts_wing, "null surface array");                                   \
        return lhs_assemble<T>(lhs, ld, nsurf, dims, colloc, normals, verts_wing, verts_wake, iteration, sigma, \
                               to_cuda(stream));                                                              \
    }
GB_BOTH(DEF_LHS)

#define DEF_RHSV(sfx, T)                                                                                  \
    int gbvlm_rhs_assemble_velocities_##sfx(T* rhs, int32_t nsurf, const gbvlm_dims* dims,               \
                                            const T* const* normals, const T* const* velocities,         \
                                            gbvlm_stream stream) {                                       \
        GB_REQUIRE(normals && velocities, "null surface array");                                         \
        return rhs_velocities<T>(rhs, nsurf, dims, normals, velocities, to_cuda(stream));                \
    }
GB_BOTH(DEF_RHSV)

int gbvlm_rhs_assemble_wake_influence_f32(float* rhs, int32_t nsurf, const gbvlm_dims* dims,
                                          const float* const* gamma_wake, const float* const* colloc,
                                          const float* const* normals, const float* const* verts_wake,
                                          const int32_t* lifting, int32_t iteration, float sigma,
                                          gbvlm_stream stream) {
    GB_REQUIRE(colloc && normals, "null surface array");
    return wake_influence<float>(rhs, nsurf, dims, gamma_wake, colloc, normals, verts_wake, lifting, iteration, sigma,
                                 5000, nullptr, 0, to_cuda(stream));
}
}  // extern "C"

namespace gbvlm {

int wake_influence_dev_f32(float* rhs, int32_t nsurf, const gbvlm_dims* dims, const float* const* gamma_wake,
                           const float* const* colloc, const float* const* normals, const float* const* verts_wake,
                           const int32_t* lifting, const int64_t* it_dev, int32_t it_max, float* scratch,
                           cudaStream_t st) {
    GB_REQUIRE(colloc && normals && it_dev && scratch, "null argument");
    int64_t ntg = 0;
    for (int m = 0; m < nsurf; m++) ntg += dims[m].ns * dims[m].nc;
    return wake_influence<float>(rhs, nsurf, dims, gamma_wake, colloc, normals, verts_wake, lifting, it_max, 0.f, 5000,
                                 scratch, (size_t)(WAKE_DEV_MAX_SLICES * ntg), st, it_dev);
}

}  // namespace gbvlm

extern "C" {

int gbvlm_rhs_assemble_wake_influence_f64(double* rhs, int32_t nsurf, const gbvlm_dims* dims,
                                          const double* const* gamma_wake, const double* const* colloc,
                                          const double* const* normals, const double* const* verts_wake,
                                          const int32_t* lifting, int32_t iteration, double sigma,
                                          gbvlm_stream stream) {
    GB_REQUIRE(colloc && normals, "null surface array");
    return wake_influence<double>(rhs, nsurf, dims, gamma_wake, colloc, normals, verts_wake, lifting, iteration,
                                  sigma, 0, nullptr, 0, to_cuda(stream));
}

#define DEF_FORCES(sfx, T)                                                                                    \
    int gbvlm_forces_steady_##sfx(int64_t ns, int64_t nc, const T* verts_wing, const T* gamma_delta,         \
                                  const T* velocities, T* forces, gbvlm_stream stream) {                     \
        GB_REQUIRE(ns >= 1 && nc >= 1, "bad sizes");                                                         \
        GB_REQUIRE(verts_wing && gamma_delta && velocities && forces, "null pointer");                       \
        k_forces<T, false><<<(unsigned)cdiv(ns * nc, 256), 256, 0, to_cuda(stream)>>>(                        \
            ns, nc, verts_wing, gamma_delta, nullptr, velocities, nullptr, nullptr, forces);                 \
        GB_LAUNCH_CHECK();                                                                                   \
        return GBVLM_OK;                                                                                     \
    }                                                                                                        \
    int gbvlm_forces_unsteady_##sfx(int64_t ns, int64_t nc, const T* verts_wing, const T* gamma_delta,       \
                                    const T* dgamma_dt, const T* velocities, const T* areas, const T* normals, \
                                    T* forces, gbvlm_stream stream) {                                        \
        GB_REQUIRE(ns >= 1 && nc >= 1, "bad sizes");                                                         \
        GB_REQUIRE(verts_wing && gamma_delta && dgamma_dt && velocities && areas && normals && forces,       \
                   "null pointer");                                                                          \
        k_forces<T, true><<<(unsigned)cdiv(ns * nc, 256), 256, 0, to_cuda(stream)>>>(                         \
            ns, nc, verts_wing, gamma_delta, dgamma_dt, velocities, areas, normals, forces);                 \
        GB_LAUNCH_CHECK();                                                                                   \
        return GBVLM_OK;                                                                                     \
    }
GB_BOTH(DEF_FORCES)

#define DEF_COEFF(sfx, T)                                                                                     \
    int gbvlm_coeff_cl_##sfx(int64_t ns, int64_t nc, const T* forces, const T* lift_axis, const T* freestream, \
                             T rho, T area, T* out, gbvlm_stream stream) {                                    \
        GB_REQUIRE(ns >= 1 && nc >= 1 && forces && lift_axis && freestream && out, "bad arguments");          \
        double r[3];                                                                                          \
        int rc = reduce_sync<T>(0, ns, nc, forces, nullptr, lift_axis[0], lift_axis[1], lift_axis[2], r,      \
                                to_cuda(stream));                                                            \
        if (rc) return rc;                                                                                    \
        T v2 = freestream[0] * freestream[0] + freestream[1] * freestream[1] + freestream[2] * freestream[2];   \
        *out = (T)(r[0] / ((double)((T)0.5 * rho * v2 * area)));                                              \
        return GBVLM_OK;                                                                                      \
    }                                                                                                         \
    int gbvlm_coeff_cm_##sfx(int64_t ns, int64_t nc, const T* forces, const T* verts_wing, const T* ref_pt,   \
                             const T* freestream, T rho, T area, T mac, T* out, gbvlm_stream stream) {        \
        GB_REQUIRE(ns >= 1 && nc >= 1 && forces && verts_wing && ref_pt && freestream && out, "bad arguments"); \
        double r[3];                                                                                          \
        int rc = reduce_sync<T>(1, ns, nc, forces, verts_wing, ref_pt[0], ref_pt[1], ref_pt[2], r,            \
                                to_cuda(stream));                                                            \
        if (rc) return rc;                                                                                    \
        T v2 = freestream[0] * freestream[0] + freestream[1] * freestream[1] + freestream[2] * freestream[2];   \
        double d = (double)((T)0.5 * rho * v2 * area * mac);                                                  \
        out[0] = (T)(r[0] / d);                                                                               \
        out[1] = (T)(r[1] / d);                                                                               \
        out[2] = (T)(r[2] / d);                                                                               \
        return GBVLM_OK;                                                                                      \
    }                                                                                                         \
    int gbvlm_mesh_mac_##sfx(int64_t ns, int64_t nc, const T* verts_wing, const T* areas, T* out,            \
                             gbvlm_stream stream) {                                                           \
        GB_REQUIRE(ns >= 1 && nc >= 1 && verts_wing && areas && out, "bad arguments");                       \
        double r[3];                                                                                          \
        int rc = reduce_sync<T>(3, ns, nc, areas, verts_wing, 0, 0, 0, r, to_cuda(stream));                  \
        if (rc) return rc;                                                                                    \
        *out = (T)(r[0] / r[1]);                                                                              \
        return GBVLM_OK;                                                                                      \
    }                                                                                                         \
    int gbvlm_sum_##sfx(const T* x, int64_t n, T* out, gbvlm_stream stream) {                                 \
        GB_REQUIRE(x && out && n >= 0, "bad arguments");                                                     \
        double r[3];                                                                                          \
        int rc = reduce_sync<T>(2, n, 1, x, nullptr, 0, 0, 0, r, to_cuda(stream));                           \
        if (rc) return rc;                                                                                    \
        *out = (T)r[0];                                                                                       \
        return GBVLM_OK;                                                                                      \
    }
GB_BOTH(DEF_COEFF)

#define DEF_METRICS(sfx, T)                                                                                   \
    int gbvlm_mesh_metrics_##sfx(T alpha_rad, int32_t nsurf, const gbvlm_dims* dims, const T* const* verts_wing, \
                                 T* const* colloc, T* const* normals, T* const* areas, gbvlm_stream stream) {  \
        GB_REQUIRE(verts_wing && colloc && normals && areas, "null surface array");                          \
        return mesh_metrics<T>(alpha_rad, nsurf, dims, verts_wing, colloc, normals, areas, to_cuda(stream));  \
    }
GB_BOTH(DEF_METRICS)

#define DEF_GWAKE(sfx, T)                                                                                     \
    int gbvlm_gamma_wake_from_coeffs_##sfx(T* gamma_wake, int64_t ns, int64_t ncols, const T* coeffs,        \
                                           int32_t harmonics, T tn, T omega, T dt, int64_t iteration,         \
                                           gbvlm_stream stream) {                                             \
        GB_REQUIRE(gamma_wake && coeffs && ns >= 1 && harmonics >= 0, "bad arguments");                      \
        GB_REQUIRE(iteration >= 0 && iteration <= ncols, "iteration=%lld outside [0, ncols]", (long long)iteration); \
        if (iteration == 0) return GBVLM_OK;                                                                  \
        k_gamma_wake<T><<<(unsigned)cdiv(ns * iteration, 256), 256, 0, to_cuda(stream)>>>(                   \
            gamma_wake, ns, ncols, coeffs, harmonics, tn, omega, dt, iteration);                             \
        GB_LAUNCH_CHECK();                                                                                   \
        return GBVLM_OK;                                                                                      \
    }
GB_BOTH(DEF_GWAKE)

#define DEF_DISPLACE(sfx, T)                                                                                  \
    int gbvlm_displace_wing_##sfx(int32_t nsurf, const gbvlm_dims* dims, const T* const* transforms,         \
                                  T* const* verts_wing, const T* const* verts_wing_init, gbvlm_stream stream) { \
        Surfs<T> s;                                                                                          \
        int rc = make_surfs(s, nsurf, dims);                                                                  \
        if (rc) return rc;                                                                                    \
        GB_REQUIRE(transforms && verts_wing && verts_wing_init, "null surface array");                       \
        int64_t total = 0;                                                                                    \
        for (int m = 0; m < nsurf; m++) {                                                                     \
            GB_REQUIRE(transforms[m] && verts_wing[m] && verts_wing_init[m], "null pointer surface %d", m);   \
            s.a[m] = transforms[m];                                                                           \
            s.b[m] = verts_wing_init[m];                                                                      \
            s.o0[m] = verts_wing[m];                                                                          \
            total += (dims[m].ns + 1) * (dims[m].nc + 1);                                                     \
        }                                                                                                     \
        k_displace<T><<<(unsigned)cdiv(total, 256), 256, 0, to_cuda(stream)>>>(s);                            \
        GB_LAUNCH_CHECK();                                                                                   \
        return GBVLM_OK;                                                                                      \
    }                                                                                                         \
    int gbvlm_wake_shed_##sfx(int32_t nsurf, const gbvlm_dims* dims, const T* const* verts_wing,             \
                              T* const* verts_wake, int32_t iteration, gbvlm_stream stream) {                 \
        Surfs<T> s;                                                                                          \
        int rc = make_surfs(s, nsurf, dims);                                                                  \
        if (rc) return rc;                                                                                    \
        GB_REQUIRE(verts_wing && verts_wake, "null surface array");                                          \
        int64_t total = 0;                                                                                    \
        for (int m = 0; m < nsurf; m++) {                                                                     \
            GB_REQUIRE(verts_wing[m] && verts_wake[m], "null pointer surface %d", m);                        \
            GB_REQUIRE(iteration >= 0 && iteration < dims[m].nwv, "iteration %d outside wake of surface %d",   \
                       iteration, m);                                                                        \
            s.a[m] = verts_wing[m];                                                                           \
            s.o0[m] = verts_wake[m];                                                                          \
            total += 4 * (dims[m].ns + 1);                                                                    \
        }                                                                                                     \
        k_wake_shed<T><<<(unsigned)cdiv(total, 256), 256, 0, to_cuda(stream)>>>(s, iteration);                \
        GB_LAUNCH_CHECK();                                                                                   \
        return GBVLM_OK;                                                                                      \
    }
GB_BOTH(DEF_DISPLACE)

#define DEF_ROLLUP(sfx, T)                                                                                    \
    int gbvlm_wake_rollup_##sfx(int32_t nsurf, const gbvlm_dims* dims, T* const* verts_wake,                 \
                                const T* const* verts_wing, const T* const* gamma_wing,                      \
                                const T* const* gamma_wake, const int32_t* lifting, T sigma, T dt,           \
                                int32_t iteration, gbvlm_stream stream) {                                    \
        GB_REQUIRE(verts_wake && verts_wing && gamma_wing, "null surface array");                            \
        return wake_rollup<T>(nsurf, dims, verts_wake, verts_wing, gamma_wing, gamma_wake, lifting, sigma, dt, \
                              iteration, to_cuda(stream));                                                    \
    }
GB_BOTH(DEF_ROLLUP)

#define DEF_TREFFTZ(sfx, T)                                                                                   \
    int gbvlm_trefftz_cd_##sfx(int64_t ns, int64_t nwv, const T* verts_wake, const T* gamma_wake,            \
                               const T* freestream, T area, T sigma, T* out, gbvlm_stream stream) {          \
        return trefftz<T>(ns, nwv, verts_wake, gamma_wake, freestream, area, sigma, out, to_cuda(stream));    \
    }
GB_BOTH(DEF_TREFFTZ)

#define DEF_GUPDATE(sfx, T)                                                                                   \
    int gbvlm_gamma_update_##sfx(int64_t ns, int64_t nc, const T* x, T* gamma, T* gamma_delta, T* gamma_wake, \
                                 int64_t wake_col, const T* gamma_prev, T* dgamma_dt, T dt, gbvlm_stream stream) { \
        GB_REQUIRE(ns >= 1 && nc >= 1 && x && gamma && gamma_delta, "bad arguments");                        \
        GB_REQUIRE(!dgamma_dt || (gamma_prev && dt != (T)0), "dgamma_dt needs gamma_prev and dt != 0");      \
        k_gamma_update<T><<<(unsigned)cdiv(ns * nc, 256), 256, 0, to_cuda(stream)>>>(                         \
            ns, nc, x, gamma, gamma_delta, gamma_wake, wake_col, gamma_prev, dgamma_dt,                      \
            dgamma_dt ? (T)1 / dt : (T)0);                                                                   \
        GB_LAUNCH_CHECK();                                                                                   \
        return GBVLM_OK;                                                                                      \
    }
GB_BOTH(DEF_GUPDATE)

}  // extern "C"

// ===========================================================================
// Allocation-free variant of the float wake-influence entry point.
//
// Some callers cannot call cudaMalloc: a host application whose device
// memory is all owned by its own allocator or pool, a serving loop that
// admits work by a fixed device-memory budget and must not grow it behind
// the budget's back, and latency paths that must keep cudaMalloc's
// device-wide synchronisation out of every step.  For them the split-K
// partial sums of gbvlm_rhs_assemble_wake_influence_f32 live in the fixed
// array below instead of the library's grown-on-demand scratch buffer.
//
// The array is GBVLM_WAKE_SCRATCH_FLOATS floats (4 MiB) in this library's
// device image, so every GPU that loads the library holds it until the
// process exits.  Host code cannot hand the array's name to a kernel (on the
// host it is only a stand-in symbol), so the first call on each device looks
// up its device address with cudaGetSymbolAddress while that device is
// current and caches it with the context it belongs to; a later call from a
// different context (the primary context released and created again) looks
// it up again.
// All calls share the one array and every call overwrites the part it uses
// (each partial is written before it is read), so no contents carry over;
// calls whose kernels overlap on the GPU (different streams, no ordering
// between them) race on the array and must not be issued.
// ===========================================================================
#define GBVLM_WAKE_SCRATCH_FLOATS (1 << 20)

static __device__ __align__(256) float g_wake_scratch[GBVLM_WAKE_SCRATCH_FLOATS];

// cuCtxGetCurrent, resolved through the runtime so that loading the library
// needs no driver library (hosts without a GPU load it to check its exports)
typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
static CtxGetCurrentFn ctx_get_current() {
    static CtxGetCurrentFn fn = []() -> CtxGetCurrentFn {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return nullptr;
        return (CtxGetCurrentFn)p;
    }();
    return fn;
}

static float* wake_scratch_address(int* rc) {
    static std::mutex mu;
    static float* addr[64] = {nullptr};
    static CUcontext owner[64] = {nullptr};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) {
        *rc = cuda_fail(e, "cudaGetDevice", __FILE__, __LINE__);
        return nullptr;
    }
    if (dev < 0 || dev >= 64) {
        set_error("device index %d out of range", dev);
        *rc = GBVLM_ERR_ARG;
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(mu);
    CtxGetCurrentFn get_ctx = ctx_get_current();
    CUcontext cur = nullptr;
    if (addr[dev] && (!get_ctx || get_ctx(&cur) != CUDA_SUCCESS || cur != owner[dev])) addr[dev] = nullptr;
    if (!addr[dev]) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_wake_scratch);
        if (e != cudaSuccess) {
            *rc = cuda_fail(e, "cudaGetSymbolAddress(g_wake_scratch)", __FILE__, __LINE__);
            return nullptr;
        }
        if (!get_ctx || get_ctx(&cur) != CUDA_SUCCESS || cur == nullptr) {
            set_error("no current CUDA context after cudaGetSymbolAddress (cuCtxGetCurrent %s)",
                      get_ctx ? "failed" : "unavailable");
            *rc = GBVLM_ERR_CUDA;
            return nullptr;
        }
        addr[dev] = (float*)p;
        owner[dev] = cur;
    }
    *rc = GBVLM_OK;
    return addr[dev];
}

extern "C" int gbvlm_rhs_assemble_wake_influence_f32_noalloc(
    float* rhs, int32_t nsurf, const gbvlm_dims* dims, const float* const* gamma_wake, const float* const* colloc,
    const float* const* normals, const float* const* verts_wake, const int32_t* lifting, int32_t iteration,
    float sigma, gbvlm_stream stream) {
    GB_REQUIRE(colloc && normals && dims, "null surface array");
    GB_REQUIRE(nsurf >= 1 && nsurf <= GBVLM_MAX_SURFACES, "nsurf=%d outside [1, %d]", nsurf, GBVLM_MAX_SURFACES);
    int64_t ntg = 0;
    for (int m = 0; m < nsurf; m++) ntg += dims[m].ns * dims[m].nc;
    GB_REQUIRE(ntg <= GBVLM_WAKE_SCRATCH_FLOATS,
               "%lld collocation points exceed the %d-float fixed scratch of the allocation-free entry point",
               (long long)ntg, GBVLM_WAKE_SCRATCH_FLOATS);
    int rc = GBVLM_OK;
    float* scratch = wake_scratch_address(&rc);
    if (!scratch) return rc;
    // wake_influence() sizes its split-K slices from the problem and rejects a
    // partial-sum table larger than the scratch it is given
    return wake_influence<float>(rhs, nsurf, dims, gamma_wake, colloc, normals, verts_wake, lifting, iteration, sigma,
                                 5000, scratch, GBVLM_WAKE_SCRATCH_FLOATS, to_cuda(stream));
}
