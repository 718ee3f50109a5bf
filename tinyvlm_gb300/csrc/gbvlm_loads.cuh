// Pieces that the drivers' fused kernels share: a panel moved with its metrics,
// the Trefftz-plane drag of a ring, and load sums in double over many blocks.
#pragma once
#include "gbvlm_math.cuh"

namespace gbvlm {

__device__ __forceinline__ double block_sum(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) sh[wid] = v;
    __syncthreads();
    double r = 0;
    if (threadIdx.x == 0) {
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) r += sh[k];
    }
    __syncthreads();
    return r;
}

// vertex q of `in` (4 planes of vld) moved by the column-major transform tr
template <class T>
__device__ __forceinline__ void move_vertex(const T* in, int64_t vld, int64_t q, const T* tr, T (&y)[4]) {
    const T x[4] = {in[q], in[vld + q], in[2 * vld + q], in[3 * vld + q]};
#pragma unroll
    for (int c = 0; c < 4; c++) {
        T acc = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) acc += x[k] * tr[c + 4 * k];
        y[c] = acc;
    }
}

// Panel p of out = tr in with its metrics (k_displace, then k_mesh_metrics): a
// panel's thread moves its four corners and writes the one at its origin, the
// last strip and row those beyond.
template <class T>
__device__ __forceinline__ void move_panel(const T* in, T* out, const T* tr, int64_t ns, int64_t nc, int64_t p, T factor,
                                           T* col, T* nor, T* area) {
    const int64_t np = ns * nc, vld = (ns + 1) * (nc + 1), j = p / ns, i = p - j * ns, v = i + j * (ns + 1);
    auto move = [&](int64_t q, bool write) {
        T y[4];
        move_vertex(in, vld, q, tr, y);
        if (write) {
#pragma unroll
            for (int c = 0; c < 4; c++) out[c * vld + q] = y[c];
        }
        return V3<T>{y[0], y[1], y[2]};
    };
    const bool lc = i == ns - 1, lr = j == nc - 1;
    const V3<T> v0 = move(v, true), v1 = move(v + 1, lc), v2 = move(v + ns + 2, lc && lr), v3_ = move(v + ns + 1, lr);
    const V3<T> nn = cross(v3_ - v1, v2 - v0);
    const T l = dsqrt(len2(nn));
    nor[p] = nn.x / l;
    nor[np + p] = nn.y / l;
    nor[2 * np + p] = nn.z / l;
    const V3<T> f = v3_ - v0, bb = v2 - v0, e = v1 - v0;
    area[p] = (T)0.5 * (dsqrt(len2(cross(f, bb))) + dsqrt(len2(cross(bb, e))));
    const V3<T> ch = (T)0.5 * (((v2 + v3_) - v0) - v1);
    const V3<T> cp = (T)0.5 * (v0 + v1) + factor * ch;
    col[p] = cp.x;
    col[np + p] = cp.y;
    col[2 * np + p] = cp.z;
}

// Trefftz-plane drag of wake ring j (ispc:273-323), one block: minus its
// circulation times the velocity that the row's trailing legs induce at its
// centre, along its normal, times its span.  Thread 0 returns it.
template <class T>
__device__ __forceinline__ double trefftz_ring(int64_t nv, int64_t nwv, const T* v, const T* gam, T sigma, int64_t j,
                                               double* sh) {
    const int64_t i = nwv - 2, ld = nv * nwv;
    auto P = [&](int64_t idx) { return V3<T>{v[idx], v[ld + idx], v[2 * ld + idx]}; };
    const V3<T> a = P(i * nv + j), b = P(i * nv + j + 1), d = P((i + 1) * nv + j + 1), e = P((i + 1) * nv + j);
    const V3<T> c = (T)0.25 * (((a + b) + d) + e);
    const V3<T> nn = cross(e - b, d - a);
    const T l = dsqrt(len2(nn));
    const V3<T> n{nn.x / l, nn.y / l, nn.z / l};
    double acc = 0;
    for (int64_t jj = threadIdx.x; jj < nv - 1; jj += blockDim.x) {
        const V3<T> w0 = P(i * nv + jj), w1 = P(i * nv + jj + 1);
        const V3<T> w2 = P((i + 1) * nv + jj + 1), w3 = P((i + 1) * nv + jj);
        V3<T> inf2{0, 0, 0};
        symmetry_ref(inf2, c, w1, w2, sigma);
        symmetry_ref(inf2, c, w3, w0, sigma);
        acc += (double)gam[i * (nv - 1) + jj] * (double)dot(inf2, n);
    }
    const double iv = block_sum(acc, sh);
    return -(double)gam[i * (nv - 1) + j] * iv * sqrt((double)len2(b - a));
}

// ---------------------------------------------------------------------------
// Load sums in double, blocks of LOAD_THREADS.
// Bound: latency.  A warp's double instruction takes about 100 cycles on this
// device, so what a block does in double is kept short: one panel per thread,
// the sums of a block's panels through shared memory (8 additions and 4
// exchanges where warp-wide trees of five sums take 25), blocks of their own
// for the chords (three square roots a strip), and the block that finishes last
// adds the blocks' sums in a fixed order.  Five sums over 1600 panels in a
// single block took 70 us.
// ---------------------------------------------------------------------------
constexpr int LOAD_THREADS = 128;
constexpr int LOAD_CHORDS = LOAD_THREADS - 1;  // strips of a chord block (a strip needs two chords)
constexpr int LOAD_SUMS = 5;                   // a panel block's: lift, area, moment x, y, z
constexpr int LOAD_PART = 6;                   // doubles a block leaves

struct LoadShared {
    double s[LOAD_SUMS][LOAD_THREADS];
    double tot[8];
    bool last;
};

__device__ __forceinline__ double lanes16(double x) {
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
    return x;
}

// the numerator of the mean aerodynamic chord over the strips of chord block blk, into S.s[0]
template <class T>
__device__ __forceinline__ void chord_terms(LoadShared& S, const T* v, int64_t ns, int64_t nc, int64_t blk) {
    const int t = threadIdx.x;
    const int64_t i = blk * LOAD_CHORDS + t, end = nc * (ns + 1), vld = (ns + 1) * (nc + 1);
    auto dist = [&](int64_t a, int64_t b) {
        const double dx = (double)v[a] - v[b], dy = (double)v[vld + a] - v[vld + b];
        const double dz = (double)v[2 * vld + a] - v[2 * vld + b];
        return sqrt(dx * dx + dy * dy + dz * dz);
    };
    S.s[1][t] = i <= ns ? dist(i, end + i) : 0.0;
    __syncthreads();
    double x = 0;
    if (t < LOAD_CHORDS && i < ns) {
        const double c0 = S.s[1][t], c1 = S.s[1][t + 1];
        x = 0.5 * (c0 * c0 + c1 * c1) * dist(i + 1, i);
    }
    S.s[0][t] = x;
}

// the block's sums 0 .. nq-1 (nq <= LOAD_SUMS) of S.s to part
__device__ __forceinline__ void block_sums(LoadShared& S, int nq, double* part) {
    __syncthreads();
    const int q = threadIdx.x >> 4, l = threadIdx.x & 15;
    if (threadIdx.x < 96) {  // whole warps
        double x = 0;
        if (q < nq) {
#pragma unroll
            for (int k = 0; k < LOAD_THREADS / 16; k++) x += S.s[q][l + 16 * k];
        }
        x = lanes16(x);
        if (l == 0 && q < nq) part[q] = x;
    }
}

// true in every thread of the block that finishes last; done is zero between launches
__device__ __forceinline__ bool last_block(LoadShared& S, unsigned* done) {
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) S.last = atomicInc(done, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!S.last) return false;
    __threadfence();
    return true;
}

// S.tot[0..4]: the panel blocks' sums, tot[5]: the chord blocks', tot[6]: the rings' (blocks in that order from b0)
__device__ __forceinline__ void add_parts(LoadShared& S, const double* part, int64_t b0, int64_t panels, int64_t chords,
                                          int64_t rings) {
    const int q = threadIdx.x >> 4, l = threadIdx.x & 15;
    const int64_t first = b0 + (q < 5 ? 0 : q == 5 ? panels : panels + chords);
    const int64_t cnt = q < 5 ? panels : q == 5 ? chords : q == 6 ? rings : 0;
    CSum s;
    for (int64_t e = l; e < cnt; e += 16) s.add(__ldcg(part + LOAD_PART * (first + e) + (q < 5 ? q : 0)));
    const double x = lanes16(s.value());
    __syncthreads();
    if (l == 0) S.tot[q] = x;
    __syncthreads();
}

}  // namespace gbvlm
