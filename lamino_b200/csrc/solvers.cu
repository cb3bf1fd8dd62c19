// Solver kernels and loops for the laminography reconstructions (sm_100a).
//
// Arithmetic follows the reference's float expressions element by element
// (including where it promotes to double); reductions use FP64 accumulation
// with warp-shuffle trees instead of the reference's serial float sums.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "fft_engine.cuh"
#include "solvers.cuh"

namespace lamino {

namespace {
std::mutex g_pool_mu;
std::map<int, cudaMemPool_t> g_pools;
}  // namespace

cudaMemPool_t call_pool() {
    int dev = 0, has = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&has, cudaDevAttrMemoryPoolsSupported, dev) != cudaSuccess || !has) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(g_pool_mu);
    cudaMemPool_t &p = g_pools[dev];
    uint64_t keep = kCallPoolKeep;
    // (the attribute call also tells a pool that a device reset took away)
    if (p && cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) == cudaSuccess) return p;
    cudaGetLastError();
    p = nullptr;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    if (cudaMemPoolCreate(&p, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();
        p = nullptr;
    }
    return p;
}
void trim_call_pool() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    auto it = g_pools.find(dev);
    if (it != g_pools.end() && it->second && cudaMemPoolTrimTo(it->second, 0) != cudaSuccess) cudaGetLastError();
}

// ---------------------------------------------------------------------------
// reductions
// ---------------------------------------------------------------------------

namespace {
// Pinned host blocks of the calling thread, kept for reuse until it exits.
struct PinnedCache {
    std::vector<std::pair<double *, int>> free_;
    double *take(int n) {
        for (size_t i = 0; i < free_.size(); ++i)
            if (free_[i].second >= n) {
                double *p = free_[i].first;
                free_.erase(free_.begin() + (long)i);
                return p;
            }
        double *p = nullptr;
        LAMINO_CUDA(cudaMallocHost((void **)&p, sizeof(double) * std::max(n, 64)));
        return p;
    }
    void give(double *p, int n) { free_.emplace_back(p, std::max(n, 64)); }
    ~PinnedCache() {
        for (auto &b : free_) cudaFreeHost(b.first);
    }
};
PinnedCache &pinned_cache() {
    static thread_local PinnedCache c;
    return c;
}
}  // namespace

Reducer::Reducer(int n) : cap(n) {
    dbuf.alloc((size_t)n);
    d = dbuf.p;
    h = pinned_cache().take(n);
}
Reducer::~Reducer() {
    if (h) pinned_cache().give(h, cap);
}
void Reducer::zero(int n, cudaStream_t s) { LAMINO_CUDA(cudaMemsetAsync(d, 0, sizeof(double) * n, s)); }
void Reducer::fetch(int n, cudaStream_t s) {
    LAMINO_CUDA(cudaMemcpyAsync(h, d, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    LAMINO_CUDA(cudaStreamSynchronize(s));
}

__device__ __forceinline__ double block_sum(double v) {
    __shared__ double ws[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) ws[wid] = v;
    __syncthreads();
    int nw = (blockDim.x + 31) >> 5;
    v = (threadIdx.x < nw) ? ws[threadIdx.x] : 0.0;
    if (wid == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    return v;
}

__global__ void k_dot(const float *__restrict__ x, const float *__restrict__ y, int64_t n, double *out) {
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s += (double)x[i] * (double)y[i];
    s = block_sum(s);
    if (threadIdx.x == 0) atomicAdd(out, s);
}

__global__ void k_sqdist3(const float *__restrict__ x, const float *__restrict__ y, int64_t V, double *out3) {
    const int c = blockIdx.y;
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < V; i += (int64_t)gridDim.x * blockDim.x) {
        float v = y ? (x[c * V + i] - y[c * V + i]) : x[c * V + i];
        s += (double)v * (double)v;
    }
    s = block_sum(s);
    if (threadIdx.x == 0) atomicAdd(out3 + c, s);
}

__device__ __forceinline__ int float_key(float f) {
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7fffffff;
}

__global__ void k_max(const float *__restrict__ x, int64_t n, int *out) {
    int m = INT_MIN;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = max(m, float_key(x[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

__global__ void k_key_to_double(const int *key, double *out) {
    int k = *key;
    int i = k >= 0 ? k : k ^ 0x7fffffff;
    *out = (double)__int_as_float(i);
}

void vec_dot(const float *x, const float *y, int64_t n, double *out, cudaStream_t s) {
    k_dot<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(x, y, n, out);
    LAMINO_LAUNCH("k_dot");
}
void vec_sqdist3(const float *x, const float *y, int64_t V, double *out3, cudaStream_t s) {
    dim3 g(grid_for(V, 256, 148 * 4), 3);
    k_sqdist3<<<g, 256, 0, s>>>(x, y, V, out3);
    LAMINO_LAUNCH("k_sqdist3");
}
void vec_max(const float *x, int64_t n, double *out, cudaStream_t s) {
    static_assert(sizeof(double) >= sizeof(int), "slot size");
    int *key = reinterpret_cast<int *>(out);  // use the slot's storage for the int key
    int init = INT_MIN;
    LAMINO_CUDA(cudaMemcpyAsync(key, &init, sizeof(int), cudaMemcpyHostToDevice, s));
    k_max<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(x, n, key);
    LAMINO_LAUNCH("k_max");
    k_key_to_double<<<1, 1, 0, s>>>(key, out);
    LAMINO_LAUNCH("k_key_to_double");
    LAMINO_CUDA(cudaStreamSynchronize(s));  // `init` lives on this stack frame
}

__global__ void k_lin2(float *__restrict__ out, float a, const float *__restrict__ x, float b,
                       const float *__restrict__ y, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = a * x[i] + (y ? b * y[i] : 0.f);
}
void vec_lin2(float *out, float a, const float *x, float b, const float *y, int64_t n, cudaStream_t s) {
    k_lin2<<<grid_for(n, 256), 256, 0, s>>>(out, a, x, b, y, n);
    LAMINO_LAUNCH("k_lin2");
}
void vec_scale(float *out, float a, const float *x, int64_t n, cudaStream_t s) { vec_lin2(out, a, x, 0.f, nullptr, n, s); }

// One thread per (k, j) column of voxels (and component): k = blockIdx.x * kVoxX +
// threadIdx.x, j = blockIdx.y, and a contiguous run of the planes z = comp * n1 + i
// for blockIdx.z (PlaneRun), so no thread divides its index.  About 148 x 64 CTAs in all.
struct Idx3 {
    int i, j, k;
};
constexpr int kVoxX = 128;
// this CTA's contiguous run of planes [z0, z1) of nz: neighbouring planes follow
// each other in one thread, so their shared rows are still in L1
struct PlaneRun {
    int z0, z1;
    __device__ PlaneRun(int nz) {
        const int per = (nz + (int)gridDim.z - 1) / (int)gridDim.z;
        z0 = (int)blockIdx.z * per;
        z1 = min(nz, z0 + per);
    }
};
static dim3 vox_grid(Dims3 d, int ncomp) {
    if (d.n2 > 65535) throw Error(ERR_ARG, "n2 above 65535 is not supported by the voxel kernels");
    const int64_t gx = (d.n3 + kVoxX - 1) / kVoxX, gy = d.n2;
    const int64_t gz = std::max<int64_t>(1, std::min<int64_t>({d.n1 * ncomp, 65535, 148LL * 64 / (gx * gy) + 1}));
    return dim3((unsigned)gx, (unsigned)gy, (unsigned)gz);
}

// ---------------------------------------------------------------------------
// qGGMRF (src/qggmrf.cpp:25-95)
// ---------------------------------------------------------------------------

__constant__ float c_qggmrf_w[27] = {0.0302f, 0.037f, 0.0302f, 0.037f, 0.0523f, 0.037f, 0.0302f, 0.037f, 0.0302f,
                                     0.037f,  0.0523f, 0.037f, 0.0532f, 0.f,     0.0523f, 0.037f, 0.0523f, 0.037f,
                                     0.0302f, 0.037f, 0.0302f, 0.037f, 0.0523f, 0.037f, 0.0302f, 0.037f, 0.0302f};

// rho'(delta) with q = 2, C = 0.001, evaluated with the reference's float/double mix
// Derivative of the qGGMRF potential (src/qggmrf.cpp:42-57), q = 2, C = 0.001,
// in float (powf for |delta|^(q-p)); the reference evaluates parts of it in
// double, which moves the result by ~1e-7 relative.
struct QgConst {
    float qmp;         // q - p
    float inv_sqp;     // 1 / sigma^(q-p)
    float inv_sq;      // 1 / sigma^q
    float at_zero;     // q / (sigma^q C)
};
// x^q for x > 0 as 2^(q log2 x): x = 2^e m with m in [1/sqrt 2, sqrt 2),
// log2 m = f P(f), f = m - 1, and 2^z = Q(z) on [-1/2, 1/2], P and Q polynomials of
// degree 8 and 6 fitted to the functions in the largest error (4e-8 and 2e-9;
// Lawson's reweighted least squares); the product q e is kept to twice float
// precision, so the result's error is that of a float: 2.9e-8 rms and at most
// 1.1e-7 relative over x in [1e-9, 1e4], q in [-0.3, 0.9] (against double;
// rounding alone has 2.5e-8 rms).  powf takes x that is not a normal number and
// results near the ends of the float range.
__device__ __forceinline__ float pow_pos(float x, float q) {
    const int b = __float_as_int(x);
    const int e = (b - 0x3f3504f3) >> 23;
    const float f = __int_as_float(b - (e << 23)) - 1.0f;
    float p = 0.12926264f;
    p = fmaf(p, f, -0.20893306f);
    p = fmaf(p, f, 0.21521251f);
    p = fmaf(p, f, -0.2386758f);
    p = fmaf(p, f, 0.28793907f);
    p = fmaf(p, f, -0.36071625f);
    p = fmaf(p, f, 0.48091027f);
    p = fmaf(p, f, -0.7213472f);
    p = fmaf(p, f, 1.442695f);
    const float ef = (float)e, ph = q * ef, low = fmaf(q, f * p, fmaf(q, ef, -ph));
    const float t = ph + low, rm = t + 12582912.0f;  // 1.5 * 2^23: the sum's low bits are rint(t)
    const float z = (ph - (rm - 12582912.0f)) + low;
    float v = 0.00015478018f;
    v = fmaf(v, z, 0.0013400431f);
    v = fmaf(v, z, 0.009617995f);
    v = fmaf(v, z, 0.05550327f);
    v = fmaf(v, z, 0.24022652f);
    v = fmaf(v, z, 0.6931472f);
    v = fmaf(v, z, 1.0f);
    if ((unsigned)b - 0x00800000u < 0x7f000000u && fabsf(t) < 120.0f)
        return __int_as_float(__float_as_int(v) + (__float_as_int(rm) << 23));
    return powf(x, q);
}
// 1 / (C + t1): __fdividef gives 0 for divisors above 2^126, which a quarter of any
// float is not; the scaling by 4 is exact.  (An IEEE reciprocal takes 305 us instead of
// 246 at 362 x 44 x 362, at the same error, 2.5e-8 against double.)
__device__ __forceinline__ float d_potential(float delta, const QgConst &k) {
    const float C = 0.001f;
    const float ad = fabsf(delta);
    if (!(ad > 0.f)) return k.at_zero;
    const float t1 = pow_pos(ad, k.qmp) * k.inv_sqp;
    const float r = 0.25f * __fdividef(1.0f, fmaf(0.25f, t1, 0.25f * C));
    const float a = delta * r * k.inv_sq;
    return a * (2.0f - k.qmp * t1 * r);
}

// d_potential of two differences at once, operation by operation the same with the
// arithmetic packed in pairs.  Differences outside pow_pos's range go one by one.
__device__ __forceinline__ float2 d_potential2(float2 delta, const QgConst &k) {
    auto both = [](float v) { return make_float2(v, v); };
    const float ax = fabsf(delta.x), ay = fabsf(delta.y);
    const int bx = __float_as_int(ax), by = __float_as_int(ay);
    const int ex = (bx - 0x3f3504f3) >> 23, ey = (by - 0x3f3504f3) >> 23;
    const float2 f = __fadd2_rn(make_float2(__int_as_float(bx - (ex << 23)), __int_as_float(by - (ey << 23))), both(-1.0f));
    float2 p = both(0.12926264f);
    p = __ffma2_rn(p, f, both(-0.20893306f));
    p = __ffma2_rn(p, f, both(0.21521251f));
    p = __ffma2_rn(p, f, both(-0.2386758f));
    p = __ffma2_rn(p, f, both(0.28793907f));
    p = __ffma2_rn(p, f, both(-0.36071625f));
    p = __ffma2_rn(p, f, both(0.48091027f));
    p = __ffma2_rn(p, f, both(-0.7213472f));
    p = __ffma2_rn(p, f, both(1.442695f));
    const float2 q = both(k.qmp), ef = make_float2((float)ex, (float)ey);
    const float2 nph = __fmul2_rn(both(-k.qmp), ef);  // -q e
    const float2 low = __ffma2_rn(q, __fmul2_rn(f, p), __ffma2_rn(q, ef, nph));
    const float2 t = __ffma2_rn(nph, both(-1.0f), low), rm = __fadd2_rn(t, both(12582912.0f));
    const float2 z = __ffma2_rn(__fadd2_rn(nph, __fadd2_rn(rm, both(-12582912.0f))), both(-1.0f), low);
    float2 v = both(0.00015478018f);
    v = __ffma2_rn(v, z, both(0.0013400431f));
    v = __ffma2_rn(v, z, both(0.009617995f));
    v = __ffma2_rn(v, z, both(0.05550327f));
    v = __ffma2_rn(v, z, both(0.24022652f));
    v = __ffma2_rn(v, z, both(0.6931472f));
    v = __ffma2_rn(v, z, both(1.0f));
    const bool zx = !(ax > 0.f), zy = !(ay > 0.f);
    if ((zx || ((unsigned)bx - 0x00800000u < 0x7f000000u && fabsf(t.x) < 120.0f)) &&
        (zy || ((unsigned)by - 0x00800000u < 0x7f000000u && fabsf(t.y) < 120.0f))) {
        const float2 w = make_float2(__int_as_float(__float_as_int(v.x) + (__float_as_int(rm.x) << 23)),
                                     __int_as_float(__float_as_int(v.y) + (__float_as_int(rm.y) << 23)));
        const float2 t1 = __fmul2_rn(w, both(k.inv_sqp)), t3 = __ffma2_rn(both(0.25f), t1, both(0.25f * 0.001f));
        const float2 r = __fmul2_rn(both(0.25f), make_float2(__fdividef(1.0f, t3.x), __fdividef(1.0f, t3.y)));
        const float2 a = __fmul2_rn(__fmul2_rn(delta, r), both(k.inv_sq));
        const float2 o = __fmul2_rn(a, __ffma2_rn(__fmul2_rn(both(-k.qmp), t1), r, both(2.0f)));
        return make_float2(zx ? k.at_zero : o.x, zy ? k.at_zero : o.y);
    }
    return make_float2(d_potential(delta.x, k), d_potential(delta.y, k));
}

// qGGMRF gradient: g[interior] += sum over the 26 neighbours of w_d rho'(x[c+d] -
// x[c]) (src/qggmrf.cpp:60-95), with each neighbour pair's derivative evaluated
// once.  rho'(-delta) = -rho'(delta) exactly in float for delta != 0 (the sign only
// flips a product), and both sides take rho'(0) = q / (sigma^q C) at delta = 0,
// so the 13 "forward" directions (dx = +1, and dx = 0 with (dy, dz) after
// (0, 0)) give every pair: the owner c keeps rho'(x[c+d] - x[c]) for its own
// sum and leaves the other side's term in shared memory.  A CTA owns a tile of
// TJ x QG_TK columns (j, k) and marches through a run of planes i; its
// threads cover the tile plus a one-column halo, whose pairs reach into the
// tile.  The 26 terms of every voxel are added in the reference's order (dx,
// dy, dz from -1 to 1), as a direct 26-neighbour loop would add them.
// Tiles start at the first interior column, and their height divides the interior
// rows with the least halo (TJ: 14 rows for 44 thick, 10 for 22 and 32, 8 for 10).
// Bound by instruction issue (13 powers per voxel), so pairs are evaluated two at a
// time with packed arithmetic.  Measured at 362 x 44 x 362, sigma 1000, p 1.2:
// 246 us; 262 one pair at a time; 424 with powf, IEEE division and tiles of 12 from
// the border in two waves of CTAs.  The registers of the packed form cost the tiles of 8
// and 12 rows a resident CTA (without that, spills: 90 x 10 x 90 16.5 against 14.5 us).
constexpr int QG_TK = 32, QG_HK = QG_TK + 2;
__host__ __device__ constexpr int qg_threads(int TJ) { return (TJ + 2) * QG_HK; }  // 340, 408, 476, 544 threads
__host__ __device__ constexpr int qg_ctas(int TJ) { return TJ <= 10 ? 3 : 2; }  // resident per SM

template <int TJ>
__global__ void __launch_bounds__(qg_threads(TJ), qg_ctas(TJ)) k_qggmrf_pairs(float *__restrict__ g, const float *__restrict__ x,
                                                             int n1, int n2, int n3, int ncomp, QgConst kq) {
    constexpr int QG_THREADS = qg_threads(TJ);
    __shared__ float q9[2][9][QG_THREADS];  // other-side terms of the dx = +1 pairs, planes i - 1 and i
    __shared__ float q4[4][QG_THREADS];     // other-side terms of the dx = 0 forward pairs, plane i
    const int t = threadIdx.x;
    const int tx = t % QG_HK, ty = t / QG_HK;
    const int k = blockIdx.x * QG_TK + tx, j = blockIdx.y * TJ + ty;
    const bool col = j < n2 && k < n3;
    const bool fin = tx >= 1 && tx <= QG_TK && ty >= 1 && ty <= TJ && j <= n2 - 2 && k <= n3 - 2;
    const int64_t sj = n3, si = (int64_t)n2 * n3;
    // the components' runs of planes follow one another along z
    const int runs = (int)gridDim.z / ncomp, comp = (int)blockIdx.z / runs, run = (int)blockIdx.z - comp * runs;
    const int per = (n1 + runs - 1) / runs, z0 = run * per, z1 = min(n1, z0 + per);
    x += comp * si * n1;
    g += comp * si * n1;
    float p9[9], p4[4];
    // own derivatives of plane i's forward pairs; other sides into shared memory
    // (neighbours beyond the volume are read at the border instead: no interior
    // voxel uses their pairs)
    const int ym = j > 0 ? -(int)sj : 0, yp = j < n2 - 1 ? (int)sj : 0, zm = k > 0 ? -1 : 0, zp = k < n3 - 1 ? 1 : 0;
    auto pairs = [&](int i, int buf, bool with4) {
        if (!col || i < 0 || i >= n1) return;
        const float *xc = x + (i * si + j * sj + k);
        const float u = xc[0];
        if (i + 1 < n1) {
            const float *xn = xc + si;
            auto diff = [&](int e) {
                return xn[(e / 3 == 0 ? ym : e / 3 == 1 ? 0 : yp) + (e % 3 == 0 ? zm : e % 3 == 1 ? 0 : zp)] - u;
            };
            auto keep = [&](int e, float delta, float pv) {
                p9[e] = pv;
                q9[buf][e][t] = !(fabsf(delta) > 0.f) ? kq.at_zero : -pv;
            };
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const float2 delta = make_float2(diff(e), diff(e + 1)), pv = d_potential2(delta, kq);
                keep(e, delta.x, pv.x);
                keep(e + 1, delta.y, pv.y);
            }
            const float delta = diff(8);
            keep(8, delta, d_potential(delta, kq));
        }
        if (with4) {
            const int off[4] = {zp, yp + zm, yp, yp + zp};
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                const float2 delta = make_float2(xc[off[e]] - u, xc[off[e + 1]] - u), pv = d_potential2(delta, kq);
                p4[e] = pv.x;
                p4[e + 1] = pv.y;
                q4[e][t] = !(fabsf(delta.x) > 0.f) ? kq.at_zero : -pv.x;
                q4[e + 1][t] = !(fabsf(delta.y) > 0.f) ? kq.at_zero : -pv.y;
            }
        }
    };
    int buf = 0;
    pairs(z0 - 1, buf, false);  // plane z0 - 1's dx = +1 pairs feed plane z0
    for (int i = z0; i < z1; ++i) {
        buf ^= 1;
        pairs(i, buf, true);
        __syncthreads();
        if (fin && i >= 1 && i <= n1 - 2) {
            const int pb = buf ^ 1;
            float sum = 0.f;
            // dx = -1: pairs owned by plane i - 1, at column (j + dy, k + dz), direction (1, -dy, -dz)
#pragma unroll
            for (int dy = -1; dy < 2; ++dy)
#pragma unroll
                for (int dz = -1; dz < 2; ++dz)
                    sum += c_qggmrf_w[(dy + 1) * 3 + (dz + 1)] *
                           q9[pb][(1 - dy) * 3 + (1 - dz)][t + dy * QG_HK + dz];
            // dx = 0, dy = -1: owned by (j - 1, k + dz), direction (0, 1, -dz)
            sum += c_qggmrf_w[9] * q4[3][t - QG_HK - 1];
            sum += c_qggmrf_w[10] * q4[2][t - QG_HK];
            sum += c_qggmrf_w[11] * q4[1][t - QG_HK + 1];
            // dx = 0, dy = 0: (0, 0, -1) owned by (j, k - 1); (0, 0, 1) own
            sum += c_qggmrf_w[12] * q4[0][t - 1];
            sum += c_qggmrf_w[14] * p4[0];
            // dx = 0, dy = 1: own
            sum += c_qggmrf_w[15] * p4[1];
            sum += c_qggmrf_w[16] * p4[2];
            sum += c_qggmrf_w[17] * p4[3];
            // dx = +1: own
#pragma unroll
            for (int e = 0; e < 9; ++e) sum += c_qggmrf_w[18 + e] * p9[e];
            g[i * si + j * sj + k] += sum;
        }
        __syncthreads();
    }
}

void qggmrf_add(float *g, const float *x, Dims3 d, int ncomp, float sigma, float p, cudaStream_t s) {
    if (d.n1 < 3 || d.n2 < 3 || d.n3 < 3) return;  // no interior voxels
    float sigma_q = std::pow(sigma, 2.0f);
    float sigma_qp = std::pow(sigma, 2.0f - p);
    QgConst kq;
    kq.qmp = 2.0f - p;
    kq.inv_sqp = (float)(1.0 / (double)sigma_qp);
    kq.inv_sq = (float)(1.0 / (double)sigma_q);
    kq.at_zero = (float)(2.0 / ((double)sigma_q * 0.001));
    // tile height: the fewest rows formed, halos included
    int TJ = 8;
    for (int t : {10, 12, 14})
        if ((d.n2 - 2 + t - 1) / t * (t + 2) <= (d.n2 - 2 + TJ - 1) / TJ * (TJ + 2)) TJ = t;
    if (d.n2 - 2 > (int64_t)65535 * TJ) throw Error(ERR_ARG, "n2 too large for the qGGMRF kernel");
    const int64_t gx = (d.n3 - 2 + QG_TK - 1) / QG_TK, gy = (d.n2 - 2 + TJ - 1) / TJ;
    // runs of planes: six waves of CTAs (with two, the CTAs at the border leave
    // the last one uneven: 316 against 274 us), a run not shorter than 4 planes,
    // as its first plane's pairs are also formed by the run before
    const int64_t cols = gx * gy * ncomp, resident = 148LL * qg_ctas(TJ);
    const int64_t runs = std::max<int64_t>(1, std::min<int64_t>({(d.n1 + 3) / 4, 65535 / ncomp, 6 * resident / cols}));
    auto kern = TJ == 8 ? k_qggmrf_pairs<8> : TJ == 10 ? k_qggmrf_pairs<10> : TJ == 12 ? k_qggmrf_pairs<12> : k_qggmrf_pairs<14>;
    kern<<<dim3((unsigned)gx, (unsigned)gy, (unsigned)(runs * ncomp)), qg_threads(TJ), 0, s>>>(
        g, x, (int)d.n1, (int)d.n2, (int)d.n3, ncomp, kq);
    LAMINO_LAUNCH("k_qggmrf_pairs");
}

// ---------------------------------------------------------------------------
// finite differences (src/finitediff.cpp:8-71, include/bregman.h:34-36)
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool interior(int i, int j, int k, int n1, int n2, int n3) {
    return i >= 1 && i < n1 - 1 && j >= 1 && j < n2 - 1 && k >= 1 && k < n3 - 1;
}

// grad along dim `dim` at (i,j,k): (u[+] - u[-]) / 2.0 on interior, else 0 (float result)
__device__ __forceinline__ float gdir(const float *__restrict__ u, int i, int j, int k, int n1, int n2, int n3,
                                      int dim) {
    if (!interior(i, j, k, n1, n2, n3)) return 0.f;
    int64_t c = ((int64_t)i * n2 + j) * n3 + k;
    int64_t st = dim == 0 ? (int64_t)n2 * n3 : (dim == 1 ? n3 : 1);
    return (u[c + st] - u[c - st]) * 0.5f;  // the reference's (float diff) / 2.0: halving is exact
}

__global__ void __launch_bounds__(kVoxX) k_grad_u(const float *__restrict__ u, int n1, int n2, int n3,
                                                  float *__restrict__ out3) {
    const int k = blockIdx.x * kVoxX + threadIdx.x, j = blockIdx.y;
    if (k >= n3) return;
    const int64_t V = (int64_t)n1 * n2 * n3;
    const PlaneRun pr(n1);
    for (int i = pr.z0; i < pr.z1; ++i) {
        const int64_t t = ((int64_t)i * n2 + j) * n3 + k;
        for (int dim = 0; dim < 3; ++dim) out3[dim * V + t] = gdir(u, i, j, k, n1, n2, n3, dim);
    }
}

// negative divergence of a 3-field given by an accessor
template <class F>
__device__ __forceinline__ float neg_div(const F &f, int i, int j, int k, int n1, int n2, int n3) {
    if (!interior(i, j, k, n1, n2, n3)) return 0.f;
    double a = -(double)(f(0, i + 1, j, k) - f(0, i - 1, j, k)) / 2.0;
    double b = (double)(f(1, i, j + 1, k) - f(1, i, j - 1, k)) / 2.0;
    double c = (double)(f(2, i, j, k + 1) - f(2, i, j, k - 1)) / 2.0;
    return (float)(a - b - c);
}

__global__ void __launch_bounds__(kVoxX) k_divergence(const float *__restrict__ du3, int n1, int n2, int n3,
                                                      float *__restrict__ out) {
    const int k = blockIdx.x * kVoxX + threadIdx.x, j = blockIdx.y;
    if (k >= n3) return;
    const int64_t V = (int64_t)n1 * n2 * n3;
    auto f = [&](int dim, int i, int j, int k) { return du3[dim * V + ((int64_t)i * n2 + j) * n3 + k]; };
    const PlaneRun pr(n1);
    for (int i = pr.z0; i < pr.z1; ++i) out[((int64_t)i * n2 + j) * n3 + k] = neg_div(f, i, j, k, n1, n2, n3);
}

// y += mu * divergence(grad_u(u)) for the 3 contiguous components.  The stencil
// reaches the centre and +-2 along each axis; a thread marches along i through a
// run of planes of one component (blockIdx.z = comp * runs + run) with
// u[i-2 .. i+2] of its (j, k) column in registers, so each voxel loads u[i+3]
// and the j and k neighbours only.  Same arithmetic as gdir / neg_div: float
// differences halved in float, combined in double.
__global__ void __launch_bounds__(kVoxX) k_laplacian_axpy(float *__restrict__ y, float mu, const float *__restrict__ u,
                                                          int n1, int n2, int n3) {
    const int k = blockIdx.x * kVoxX + threadIdx.x, j = blockIdx.y;
    if (k >= n3) return;
    const int runs = (int)gridDim.z / 3;
    const int comp = (int)blockIdx.z / runs, run = (int)blockIdx.z - comp * runs;
    const int per = (n1 + runs - 1) / runs;
    const int i0 = run * per, i1 = min(n1, i0 + per);
    if (i0 >= i1) return;
    const int64_t V = (int64_t)n1 * n2 * n3, s1 = (int64_t)n2 * n3;
    const bool jk_in = j >= 1 && j <= n2 - 2 && k >= 1 && k <= n3 - 2;
    const int64_t col = (int64_t)j * n3 + k;
    const float *uc = u + comp * V + col;
    float *yc = y + comp * V + col;
    auto ld = [&](int ii) { return (ii >= 0 && ii < n1) ? uc[ii * s1] : 0.f; };
    float w0 = ld(i0 - 2), w1 = ld(i0 - 1), w2 = ld(i0), w3 = ld(i0 + 1), w4 = ld(i0 + 2);
    for (int i = i0; i < i1; ++i) {
        float l = 0.f;
        if (jk_in && i >= 1 && i <= n1 - 2) {
            const float *pc = uc + (int64_t)i * s1;
            const float g0p = i + 1 <= n1 - 2 ? (w4 - w2) * 0.5f : 0.f;
            const float g0m = i - 1 >= 1 ? (w2 - w0) * 0.5f : 0.f;
            const float g1p = j + 1 <= n2 - 2 ? (pc[2 * n3] - w2) * 0.5f : 0.f;
            const float g1m = j - 1 >= 1 ? (w2 - pc[-2 * n3]) * 0.5f : 0.f;
            const float g2p = k + 1 <= n3 - 2 ? (pc[2] - w2) * 0.5f : 0.f;
            const float g2m = k - 1 >= 1 ? (w2 - pc[-2]) * 0.5f : 0.f;
            const double a = -(double)(g0p - g0m) / 2.0;
            const double b = (double)(g1p - g1m) / 2.0;
            const double c = (double)(g2p - g2m) / 2.0;
            l = (float)(a - b - c);
        }
        yc[(int64_t)i * s1] += l * mu;
        w0 = w1;
        w1 = w2;
        w2 = w3;
        w3 = w4;
        w4 = ld(i + 3);
    }
}

__global__ void __launch_bounds__(kVoxX) k_sb_rhs(const float *__restrict__ yT, const float *__restrict__ d9,
                                                  const float *__restrict__ b9, float mu, int n1, int n2, int n3,
                                                  float *__restrict__ rhs) {
    const int k = blockIdx.x * kVoxX + threadIdx.x, j = blockIdx.y;
    if (k >= n3) return;
    const int64_t V = (int64_t)n1 * n2 * n3;
    const PlaneRun pr(3 * n1);
    for (int z = pr.z0; z < pr.z1; ++z) {
        const int comp = z / n1, i = z - comp * n1;
        const float *dc = d9 + 3 * comp * V, *bc = b9 + 3 * comp * V;
        auto f = [&](int dim, int ii, int jj, int kk) {
            int64_t c = dim * V + ((int64_t)ii * n2 + jj) * n3 + kk;
            return dc[c] - bc[c];
        };
        const int64_t t = ((int64_t)i * n2 + j) * n3 + k;
        const float dv = neg_div(f, i, j, k, n1, n2, n3);
        rhs[comp * V + t] = yT[comp * V + t] + dv * mu;
    }
}

__global__ void __launch_bounds__(kVoxX) k_sb_shrink(const float *__restrict__ x3, float *__restrict__ d9,
                                                     float *__restrict__ b9, float lam, float mu, int n1, int n2,
                                                     int n3) {
    const int k = blockIdx.x * kVoxX + threadIdx.x, jj = blockIdx.y;
    if (k >= n3) return;
    const int64_t V = (int64_t)n1 * n2 * n3;
    const float eps = 1e-8f;
    const float thr = lam / mu;
    const PlaneRun prn(n1);
    for (int ii = prn.z0; ii < prn.z1; ++ii) {
        const int64_t t = ((int64_t)ii * n2 + jj) * n3 + k;
        const Idx3 p{ii, jj, k};
        float gx[9], tb[9];
        float sk = 1.0f * eps;
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                gx[i * 3 + j] = gdir(x3 + i * V, p.i, p.j, p.k, n1, n2, n3, j);
                tb[i * 3 + j] = gx[i * 3 + j] + b9[(i * 3 + j) * V + t];
                sk += tb[i * 3 + j] * tb[i * 3 + j];
            }
        sk = sqrtf(sk);
        float m = fmaxf(sk - thr, 0.f);
#pragma unroll
        for (int q = 0; q < 9; ++q) {
            float dv = m * (tb[q] / sk);
            d9[q * V + t] = dv;
            b9[q * V + t] += gx[q] - dv;
        }
    }
}

void grad_u(const float *u, Dims3 d, float *out3, cudaStream_t s) {
    k_grad_u<<<vox_grid(d, 1), kVoxX, 0, s>>>(u, (int)d.n1, (int)d.n2, (int)d.n3, out3);
    LAMINO_LAUNCH("k_grad_u");
}
void divergence(const float *du3, Dims3 d, float *out, cudaStream_t s) {
    k_divergence<<<vox_grid(d, 1), kVoxX, 0, s>>>(du3, (int)d.n1, (int)d.n2, (int)d.n3, out);
    LAMINO_LAUNCH("k_divergence");
}
void laplacian_axpy(float *y, float mu, const float *u, Dims3 d, cudaStream_t s) {
    dim3 g = vox_grid(d, 1);  // runs of planes per component, 3 components
    g.z = (unsigned)std::max<int64_t>(1, std::min<int64_t>(g.z, 65535 / 3)) * 3;
    k_laplacian_axpy<<<g, kVoxX, 0, s>>>(y, mu, u, (int)d.n1, (int)d.n2, (int)d.n3);
    LAMINO_LAUNCH("k_laplacian_axpy");
}
void sb_rhs(const float *yT3, const float *d9, const float *b9, float mu, Dims3 dims, float *rhs3, cudaStream_t s) {
    k_sb_rhs<<<vox_grid(dims, 3), kVoxX, 0, s>>>(yT3, d9, b9, mu, (int)dims.n1, (int)dims.n2, (int)dims.n3, rhs3);
    LAMINO_LAUNCH("k_sb_rhs");
}
void sb_shrink(const float *x3, float *d9, float *b9, float lam, float mu, Dims3 dims, cudaStream_t s) {
    k_sb_shrink<<<vox_grid(dims, 1), kVoxX, 0, s>>>(x3, d9, b9, lam, mu, (int)dims.n1, (int)dims.n2,
                                                    (int)dims.n3);
    LAMINO_LAUNCH("k_sb_shrink");
}

// ---------------------------------------------------------------------------
// ramp preconditioner (include/precond.h:33-87)
// ---------------------------------------------------------------------------

__global__ void k_filter_mul(float2 *__restrict__ S, const float *__restrict__ f, int64_t plane, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float w = f[i % plane];
        S[i].x *= w;
        S[i].y *= w;
    }
}

// Along n2 the filter step (forward DFT, multiply by the ramp, inverse DFT) is a
// circulant convolution for each k3 column, z(:, k3) = G_k3 (*) x(:, k3), with
// G_k3[d] = sum_k2 f(k2, k3) cos(2 pi k2 d / n2): f is real and even in k2, so G_k3
// is real (and even).  One CTA per (n1 slice, RC_KB consecutive k3 columns): the
// column tile twice over in shared memory (so m - d + n2 needs no wrap), lanes on
// columns, warps on output rows, taps summed in order d = 0 .. n2-1.
constexpr int RC_KB = 32;
constexpr int RC_WARPS = 8;
constexpr int RC_ROWS = 9;  // output rows per thread: 8 warps x 9 rows cover n2 <= 72 in one pass
constexpr int kRampConvMaxN2 = 128;

__global__ void __launch_bounds__(RC_WARPS * 32) k_ramp_cols(float2 *__restrict__ S, const float *__restrict__ G,
                                                             int n2, int h3) {
    extern __shared__ float2 xs[];                                // [2 n2][RC_KB]
    float *gs = reinterpret_cast<float *>(xs + 2 * n2 * RC_KB);   // [n2][RC_KB]
    const int k3b = blockIdx.x * RC_KB;
    const int nk = min(RC_KB, h3 - k3b);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float2 *Sp = S + (int64_t)blockIdx.y * n2 * h3 + k3b;
    // load: the column tile (twice) and the kernels, 8 independent loads in flight per thread
    constexpr int LB = 8;
    const int total = n2 * RC_KB;
    for (int t0 = threadIdx.x; t0 < total; t0 += LB * RC_WARPS * 32) {
        float2 v[LB];
        float gv[LB];
#pragma unroll
        for (int u = 0; u < LB; ++u) {
            const int t = t0 + u * RC_WARPS * 32;
            const int j = t / RC_KB, kk = t - j * RC_KB;
            const bool ok = t < total && kk < nk;
            v[u] = ok ? Sp[(int64_t)j * h3 + kk] : make_float2(0.f, 0.f);
            gv[u] = ok ? __ldg(G + (int64_t)j * h3 + k3b + kk) : 0.f;
        }
#pragma unroll
        for (int u = 0; u < LB; ++u) {
            const int t = t0 + u * RC_WARPS * 32;
            if (t < total) {
                const int j = t / RC_KB, kk = t - j * RC_KB;
                xs[j * RC_KB + kk] = v[u];
                xs[(j + n2) * RC_KB + kk] = v[u];
                gs[j * RC_KB + kk] = gv[u];
            }
        }
    }
    __syncthreads();
    // rows m0 .. m0 + 8 of a thread need x[m0 + r - dd]: as dd grows the window
    // shifts by one, so it lives in a rotating register buffer, slot (r - dd) mod 9,
    // and each tap loads one new x (smem tile index m - dd + n2 stays in [1, 2 n2))
    for (int m0 = warp * RC_ROWS; m0 < n2; m0 += RC_ROWS * RC_WARPS) {
        float2 acc[RC_ROWS], buf[RC_ROWS];
#pragma unroll
        for (int r = 0; r < RC_ROWS; ++r) {
            acc[r] = make_float2(0.f, 0.f);
            // rows past n2 - 1 start from row n2 - 1 (inside the tile) and are never stored
            buf[r] = xs[(min(m0 + r, n2 - 1) + n2) * RC_KB + lane];
        }
        for (int d0 = 0; d0 < n2; d0 += RC_ROWS) {
#pragma unroll
            for (int u = 0; u < RC_ROWS; ++u) {
                const int dd = d0 + u;
                if (dd < n2) {
                    if (dd > 0) buf[(RC_ROWS - u) % RC_ROWS] = xs[(m0 - dd + n2) * RC_KB + lane];
                    const float g = gs[dd * RC_KB + lane];
#pragma unroll
                    for (int r = 0; r < RC_ROWS; ++r) {
                        const float2 x = buf[(r - u + RC_ROWS) % RC_ROWS];
                        acc[r] = __ffma2_rn(make_float2(g, g), x, acc[r]);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < RC_ROWS; ++r) {
            const int m = m0 + r;
            if (m < n2 && lane < nk) Sp[(int64_t)m * h3 + lane] = acc[r];
        }
    }
}

// Real transforms along n3 = N as Bluestein convolutions through the pencil's FFT
// pipeline: X[k] = sum_n x[n] e^{-2 pi i k n / N}
// = conj(w_k) sum_n (x_n conj(w_n)) w_{k-n} with w_m = e^{i pi m^2 / N}, a circular
// convolution of length M >= 2N - 1, taken as undo(FWD(u) . V) with V the
// transform of v (v_m = w_m for m < N, v_{M-m} = w_m for 0 < m < N, zero between),
// divided by M and stored in DIF position order.  The inverse uses conj(w) in
// place of w.  M = 1458 (the compile-time pipeline, fused outer stages) for
// 365 <= N <= 729; otherwise M = the next 2,3,5-smooth even length >= 2N - 1 on
// the runtime pipeline (same fused outer stages, FIXED = false), used for N >= 128
// with a prime factor above 7, where cuFFT slows down.  Two real rows travel as one
// complex row (a + i b), three complex rows per CTA; the spectra keep the R2C
// layout [row][N/2 + 1].
constexpr int kBlueM = 1458;
constexpr int kBlueHalf = 729;
constexpr int kBlueMaxM = 4096;

struct BlueR2CRows {
    const float *x;
    int64_t nrows, q0;
    int N, hm;  // hm: M / 2, the stride of zb
    const float2 *chirp;
    float2 *zb;  // 3 x M/2 results in shared memory
    __device__ __forceinline__ float2 get(int c, int i) const {
        const int64_t r = 2 * (q0 + c);
        if (i >= N || r >= nrows) return make_float2(0.f, 0.f);
        const float a = x[r * N + i], b = r + 1 < nrows ? x[(r + 1) * N + i] : 0.f;
        return c_mulc(make_float2(a, b), __ldg(chirp + i));
    }
    __device__ __forceinline__ bool want(int i) const { return i < N; }
    __device__ __forceinline__ void put(int c, int i, float2 v) const {
        zb[c * hm + i] = c_mulc(v, __ldg(chirp + i));
    }
};

// FWD(u), the pointwise product with V, undo: rows loaded and stored by `rows`
template <bool FIXED, class Rows>
__device__ __forceinline__ void blue_convolve(const Rows &rows, const FftLen &F, const float2 *__restrict__ V,
                                              const float2 *__restrict__ tw, float2 *sm, int M) {
    if constexpr (FIXED) {
        fft1458_load(rows, tw, sm, threadIdx.x);
        __syncthreads();
        ct_forward<kBlueM, 2>(sm, 3, kBlueM, tw, threadIdx.x, blockDim.x);
    } else {
        fftlead_any<false>(rows, F, sm, M, threadIdx.x, blockDim.x);
        __syncthreads();
        fft_forward(sm, 3, M, F, 2, threadIdx.x, blockDim.x);
    }
    for (int p = threadIdx.x; p < M; p += blockDim.x) {
        const float2 v = __ldg(V + p);
#pragma unroll
        for (int c = 0; c < 3; ++c) sm[c * M + p] = c_mul(sm[c * M + p], v);
    }
    __syncthreads();
    if constexpr (FIXED) {
        ct_inverse<kBlueM, 3, 2>(sm, 3, kBlueM, tw, threadIdx.x, blockDim.x);
        fft1458_store(rows, tw, sm, threadIdx.x);
    } else {
        fft_inverse(sm, 3, M, F, 2, threadIdx.x, blockDim.x);
        fftlead_any<true>(rows, F, sm, M, threadIdx.x, blockDim.x);
    }
}

template <bool FIXED>
__global__ void __launch_bounds__(256, 4) k_blue_r2c(const float *__restrict__ x, int64_t nrows, int N,
                                                     const float2 *__restrict__ chirp,
                                                     const float2 *__restrict__ V,
                                                     const float2 *__restrict__ tw, FftLen F,
                                                     float2 *__restrict__ S) {
    extern __shared__ float2 sm[];  // 3 transform rows of M, then 3 x M/2 results
    const int M = FIXED ? kBlueM : F.n, hm = M / 2;
    const int h = N / 2 + 1;
    const int64_t q0 = (int64_t)blockIdx.x * 3;
    const BlueR2CRows rows{x, nrows, q0, N, hm, chirp, sm + 3 * M};
    blue_convolve<FIXED>(rows, F, V, tw, sm, M);
    __syncthreads();
    // A = (Z_k + conj Z_{N-k}) / 2, B = (Z_k - conj Z_{N-k}) / 2i
    const float2 *zb = sm + 3 * M;
    for (int t = threadIdx.x; t < 3 * h; t += blockDim.x) {
        const int c = t / h, k = t - c * h;
        const int64_t r = 2 * (q0 + c);
        if (r >= nrows) continue;
        const float2 zk = zb[c * hm + k];
        const float2 zm = zb[c * hm + (k == 0 ? 0 : N - k)];
        S[r * h + k] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        if (r + 1 < nrows) S[(r + 1) * h + k] = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
    }
}

struct BlueC2RRows {
    const float2 *S;
    float *y;
    int64_t nrows, q0;
    int N, h;
    const float2 *chirp;
    __device__ __forceinline__ float2 get(int c, int i) const {
        const int64_t r = 2 * (q0 + c);
        if (i >= N || r >= nrows) return make_float2(0.f, 0.f);
        const bool lo = i < h;
        const int k = lo ? i : N - i;
        float2 A = S[r * h + k];
        float2 B = r + 1 < nrows ? S[(r + 1) * h + k] : make_float2(0.f, 0.f);
        if (k == 0 || 2 * k == N) A.y = B.y = 0.f;  // as a C2R reads them: real
        if (!lo) {
            A.y = -A.y;
            B.y = -B.y;
        }
        return c_mul(make_float2(A.x - B.y, A.y + B.x), __ldg(chirp + i));  // (A + i B) w
    }
    __device__ __forceinline__ bool want(int i) const { return i < N; }
    __device__ __forceinline__ void put(int c, int i, float2 v) const {
        const int64_t r = 2 * (q0 + c);
        if (r >= nrows) return;
        const float2 z = c_mul(v, __ldg(chirp + i));
        y[r * N + i] = z.x;
        if (r + 1 < nrows) y[(r + 1) * N + i] = z.y;
    }
};

template <bool FIXED>
__global__ void __launch_bounds__(256, FIXED ? 5 : 4) k_blue_c2r(const float2 *__restrict__ S, int64_t nrows, int N,
                                                     const float2 *__restrict__ chirp,
                                                     const float2 *__restrict__ V,
                                                     const float2 *__restrict__ tw, FftLen F,
                                                     float *__restrict__ y) {
    extern __shared__ float2 sm[];  // 3 transform rows of M
    const int M = FIXED ? kBlueM : F.n;
    const BlueC2RRows rows{S, y, nrows, (int64_t)blockIdx.x * 3, N, N / 2 + 1, chirp};
    blue_convolve<FIXED>(rows, F, V, tw, sm, M);
}

// The tables of a size, built on the device in FP64 (on the host their sums, M^2
// and n2^2 n3 / 2 terms, took 11 ms at 721 x 71 x 721, five times the apply).

// filter value f(k2, k3), in the reference's float operations, with the
// 1 / (n2 n3) of the c2r folded in
__device__ __forceinline__ float ramp_filter(int j, int i, int n2, int n3, float scale) {
    const float x = __fdiv_rn((float)i, (float)n3);
    const float y = __fdiv_rn((float)(j <= n2 / 2 ? j : j - n2), (float)n2);
    return __fmul_rn(__fsqrt_rn(__fadd_rn(__fmul_rn(x, x), __fmul_rn(y, y))), scale);
}
// conv: G[d][k3] = sum_k2 f(k2, k3) cos(2 pi k2 d / n2) (n2 <= kRampConvMaxN2), else f itself
__global__ void __launch_bounds__(128) k_ramp_table(int n2, int n3, int h3, float scale, bool conv,
                                                    float *__restrict__ out) {
    __shared__ double cs[kRampConvMaxN2];
    if (conv) {
        for (int t = threadIdx.x; t < n2; t += blockDim.x) cs[t] = cospi(2.0 * t / n2);
        __syncthreads();
    }
    const int64_t n = (int64_t)n2 * h3;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int d = (int)(e / h3), i = (int)(e - (int64_t)d * h3);
        if (!conv) {
            out[e] = ramp_filter(d, i, n2, n3, scale);
            continue;
        }
        double acc = 0.0;
        for (int j = 0, t = 0; j < n2; ++j) {
            acc += (double)ramp_filter(j, i, n2, n3, scale) * cs[t];
            t += d;
            if (t >= n2) t -= n2;
        }
        out[e] = (float)acc;
    }
}
// chirp w_n = e^{i pi n^2 / N}, the M-point twiddles and, in double for
// k_blue_spectra, w and cos(2 pi e / M)
__global__ void k_blue_tables(int N, int M, float2 *__restrict__ chirp, float2 *__restrict__ tw, double2 *__restrict__ w,
                              double *__restrict__ cs) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    double s, c;
    if (i < N) {
        sincospi((double)(((long long)i * i) % (2LL * N)) / N, &s, &c);
        w[i] = make_double2(c, s);
        chirp[i] = make_float2((float)c, (float)s);
    }
    if (i < M) {
        sincospi(2.0 * i / M, &s, &c);
        cs[i] = c;
        tw[i] = make_float2((float)c, (float)-s);
    }
}
// the convolution kernel's spectrum, V_k = w_0 + 2 sum_{0 < m < N} w_m cos(2 pi k m / M)
// (v is even, so V is), over M, in DIF position order, and its conjugate (the
// spectrum of conj v); one warp per k
__global__ void __launch_bounds__(256) k_blue_spectra(int N, int M, const double2 *__restrict__ w,
                                                      const double *__restrict__ cs, const int *__restrict__ pos,
                                                      float2 *__restrict__ vf, float2 *__restrict__ vi) {
    const int k = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (k >= M) return;
    double re = 0.0, im = 0.0;
    for (int m = 1 + lane; m < N; m += 32) {
        const double c = cs[(int)(((long long)k * m) % M)];
        re += w[m].x * c;
        im += w[m].y * c;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        re += __shfl_down_sync(0xffffffffu, re, o);
        im += __shfl_down_sync(0xffffffffu, im, o);
    }
    if (lane) return;
    re = (w[0].x + 2.0 * re) / M;
    im = (w[0].y + 2.0 * im) / M;
    vf[pos[k]] = make_float2((float)re, (float)im);
    vi[pos[k]] = make_float2((float)re, (float)-im);
}

// largest prime factor of n
static int64_t largest_prime_factor(int64_t n) {
    int64_t p = 1;
    for (int64_t q = 2; q * q <= n; ++q)
        while (n % q == 0) {
            p = q;
            n /= q;
        }
    return n > 1 ? std::max(p, n) : p;
}

// schedule of the runtime Bluestein length M (lead 2) over the device twiddles
static FftLen blue_len(int M, const float2 *tw_dev) {
    const std::vector<int> r = fft_schedule(M, true);
    FftLen F{};
    F.n = M;
    F.ns = (int)r.size();
    int b = M;
    for (int s = 0; s < F.ns; ++s) {
        F.radix[s] = r[s];
        F.bsz[s] = b;
        F.dm[s] = FastDiv::make((uint32_t)(b / r[s]));
        F.dnb[s] = FastDiv::make((uint32_t)(M / r[s]));
        F.dblk[s] = FastDiv::make((uint32_t)(M / b));
        b /= r[s];
    }
    F.tw = tw_dev;
    return F;
}

RampPrecond::RampPrecond(Dims3 dd, cudaStream_t s) : d(dd) {
    const int64_t n2 = d.n2, n3 = d.n3, h3 = n3 / 2 + 1;
    cols = n2 <= kRampConvMaxN2 && 3 * d.n1 <= 65535;
    const bool fixed = n3 >= 365 && n3 <= kBlueHalf;
    const int64_t mrt = next_smooth_even(2 * n3 - 1);
    blue_fixed = cols && fixed;
    blue = cols && (fixed || (n3 >= 128 && largest_prime_factor(n3) > 7 && mrt <= kBlueMaxM));
    const int M = !blue ? 0 : (fixed ? kBlueM : (int)mrt), N = blue ? (int)n3 : 0;
    // one allocation for the tables and the spectra
    size_t bytes = 0;
    auto room = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t of = room(n2 * h3 * sizeof(float)), oc = room(N * sizeof(float2)), ot = room(M * sizeof(float2)),
                 ovf = room(M * sizeof(float2)), ovi = room(M * sizeof(float2)), ow = room(N * sizeof(double2)),
                 ocs = room(M * sizeof(double)), op = room(M * sizeof(int)),
                 os = room(3 * d.n1 * n2 * h3 * sizeof(float2));
    mem.alloc(bytes);
    char *m0 = mem.p;
    spec = reinterpret_cast<float2 *>(m0 + os);
    filt = reinterpret_cast<float *>(m0 + of);
    chirp = reinterpret_cast<float2 *>(m0 + oc);
    tw = reinterpret_cast<float2 *>(m0 + ot);
    vfwd = reinterpret_cast<float2 *>(m0 + ovf);
    vinv = reinterpret_cast<float2 *>(m0 + ovi);
    const float scale = (float)(1.0 / (double)(n2 * n3));
    k_ramp_table<<<grid_for(n2 * h3, 128), 128, 0, s>>>((int)n2, (int)n3, (int)h3, scale, cols, filt);
    LAMINO_LAUNCH("k_ramp_table");
    if (blue) {
        const std::vector<int> hpos = fft_positions(M, fft_schedule(M, true));
        int *pos = reinterpret_cast<int *>(m0 + op);
        LAMINO_CUDA(cudaMemcpyAsync(pos, hpos.data(), M * sizeof(int), cudaMemcpyHostToDevice, s));
        double2 *w = reinterpret_cast<double2 *>(m0 + ow);
        double *cs = reinterpret_cast<double *>(m0 + ocs);
        k_blue_tables<<<(unsigned)((std::max(M, N) + 127) / 128), 128, 0, s>>>(N, M, chirp, tw, w, cs);
        LAMINO_LAUNCH("k_blue_tables");
        k_blue_spectra<<<(unsigned)((M + 7) / 8), 256, 0, s>>>(N, M, w, cs, pos, vfwd, vinv);
        LAMINO_LAUNCH("k_blue_spectra");
        LAMINO_CUDA(cudaStreamSynchronize(s));  // hpos goes out of scope
        blue_f = blue_len(M, tw);
        raise_smem_limit((const void *)k_blue_r2c<true>, (int)(3 * (kBlueM + kBlueHalf) * sizeof(float2)));
        raise_smem_limit((const void *)k_blue_c2r<true>, (int)(3 * kBlueM * sizeof(float2)));
        raise_smem_limit((const void *)k_blue_r2c<false>, (int)(3 * (M + M / 2) * sizeof(float2)));
        raise_smem_limit((const void *)k_blue_c2r<false>, (int)(3 * M * sizeof(float2)));
    } else if (cols) {
        int n[1] = {(int)n3};
        r2c.make(1, n, CUFFT_R2C, (int)(3 * d.n1 * n2));
        c2r.make(1, n, CUFFT_C2R, (int)(3 * d.n1 * n2));
    } else {
        int n[2] = {(int)n2, (int)n3};
        r2c.make(2, n, CUFFT_R2C, (int)(3 * d.n1));
        c2r.make(2, n, CUFFT_C2R, (int)(3 * d.n1));
    }
    if (cols) raise_smem_limit((const void *)k_ramp_cols, (int)(n2 * RC_KB * (2 * sizeof(float2) + sizeof(float))));
}

void RampPrecond::apply3(const float *r3, float *z3, cudaStream_t s) {
    int64_t h3 = d.n3 / 2 + 1, plane = d.n2 * h3;
    const int64_t nrows = 3 * d.n1 * d.n2;
    const unsigned gblue = (unsigned)(((nrows + 1) / 2 + 2) / 3);
    const int M = blue_f.n;
    if (blue && blue_fixed) {
        k_blue_r2c<true><<<gblue, 256, 3 * (kBlueM + kBlueHalf) * sizeof(float2), s>>>(
            r3, nrows, (int)d.n3, chirp, vfwd, tw, blue_f, spec);
        LAMINO_LAUNCH("k_blue_r2c");
    } else if (blue) {
        k_blue_r2c<false><<<gblue, 256, 3 * (M + M / 2) * sizeof(float2), s>>>(r3, nrows, (int)d.n3, chirp,
                                                                              vfwd, tw, blue_f, spec);
        LAMINO_LAUNCH("k_blue_r2c");
    } else {
        LAMINO_CUFFT(cufftSetStream(r2c.h, s));
        LAMINO_CUFFT(cufftExecR2C(r2c.h, const_cast<float *>(r3), (cufftComplex *)spec));
    }
    if (cols) {
        const dim3 grid((unsigned)((h3 + RC_KB - 1) / RC_KB), (unsigned)(3 * d.n1));
        const int smem = (int)(d.n2 * RC_KB * (2 * sizeof(float2) + sizeof(float)));
        k_ramp_cols<<<grid, RC_WARPS * 32, smem, s>>>(spec, filt, (int)d.n2, (int)h3);
        LAMINO_LAUNCH("k_ramp_cols");
    } else {
        k_filter_mul<<<grid_for(3 * d.n1 * plane, 256), 256, 0, s>>>(spec, filt, plane, 3 * d.n1 * plane);
        LAMINO_LAUNCH("k_filter_mul");
    }
    if (blue && blue_fixed) {
        k_blue_c2r<true><<<gblue, 256, 3 * kBlueM * sizeof(float2), s>>>(spec, nrows, (int)d.n3, chirp,
                                                                         vinv, tw, blue_f, z3);
        LAMINO_LAUNCH("k_blue_c2r");
    } else if (blue) {
        k_blue_c2r<false><<<gblue, 256, 3 * M * sizeof(float2), s>>>(spec, nrows, (int)d.n3, chirp, vinv,
                                                                     tw, blue_f, z3);
        LAMINO_LAUNCH("k_blue_c2r");
    } else {
        LAMINO_CUFFT(cufftSetStream(c2r.h, s));
        LAMINO_CUFFT(cufftExecC2R(c2r.h, (cufftComplex *)spec, z3));
    }
}

// ---------------------------------------------------------------------------
// CG (src/conjgrad.cpp:37-117)
// ---------------------------------------------------------------------------

__global__ void k_cg_update(float *__restrict__ x, float *__restrict__ r, const float *__restrict__ p,
                            const float *__restrict__ Ap, float alpha, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        x[i] += p[i] * alpha;
        r[i] -= Ap[i] * alpha;
    }
}
__global__ void k_cg_dir(float *__restrict__ p, const float *__restrict__ z, float beta, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        p[i] = z[i] + p[i] * beta;
}

CgStats cgsolver(const OpFn &A, const float *y3, float *x3, Dims3 d, int max_iter, float tol, cudaStream_t s) {
    CgWork w(d, s);
    CgStats st = cgsolver(A, y3, x3, w, max_iter, tol, s);
    LAMINO_CUDA(cudaStreamSynchronize(s));
    return st;
}

CgStats cgsolver(const OpFn &A, const float *y3, float *x3, CgWork &w, int max_iter, float tol, cudaStream_t s) {
    const Dims3 d = w.d;
    const int64_t n = 3 * d.size();
    DevBuf<float> &r = w.r, &p = w.p, &z = w.z, &Ap = w.Ap;
    RampPrecond &M = w.M;
    Reducer &red = w.red;
    CgStats st;
    A(x3, Ap.p, s);
    vec_lin2(r.p, 1.f, y3, -1.f, Ap.p, n, s);
    M.apply3(r.p, z.p, s);
    LAMINO_CUDA(cudaMemcpyAsync(p.p, z.p, n * 4, cudaMemcpyDeviceToDevice, s));
    red.zero(1, s);
    vec_dot(z.p, r.p, n, red.d, s);
    red.fetch(1, s);
    double rs_old = red.h[0];
    for (int it = 0; it < max_iter; ++it) {
        A(p.p, Ap.p, s);
        red.zero(2, s);
        vec_dot(p.p, Ap.p, n, red.d, s);
        red.fetch(1, s);
        double pAp = red.h[0];
        if (std::fabs(pAp) < 1e-10) break;
        float alpha = (float)(rs_old / pAp);
        k_cg_update<<<grid_for(n, 256), 256, 0, s>>>(x3, r.p, p.p, Ap.p, alpha, n);
        LAMINO_LAUNCH("k_cg_update");
        M.apply3(r.p, z.p, s);
        red.zero(1, s);
        vec_dot(z.p, r.p, n, red.d, s);
        red.fetch(1, s);
        double rs_new = red.h[0];
        st.iters = it + 1;
        st.last_res = std::sqrt(std::fabs(rs_new));
        if (std::sqrt(std::fabs(rs_new)) < tol) break;
        float beta = (float)(rs_new / rs_old);
        k_cg_dir<<<grid_for(n, 256), 256, 0, s>>>(p.p, z.p, beta, n);
        LAMINO_LAUNCH("k_cg_dir");
        rs_old = rs_new;
    }
    return st;
}

CgStats cgsolver_refined(const OpFn &A_hi, const OpFn &A_lo, const float *y3, float *x3, Dims3 d, int inner,
                         int refinements, float tol, cudaStream_t s) {
    CgWork w(d, s);
    CgStats st = cgsolver_refined(A_hi, A_lo, y3, x3, w, inner, refinements, tol, s);
    LAMINO_CUDA(cudaStreamSynchronize(s));
    return st;
}

CgStats cgsolver_refined(const OpFn &A_hi, const OpFn &A_lo, const float *y3, float *x3, CgWork &w, int inner,
                         int refinements, float tol, cudaStream_t s) {
    const int64_t n = 3 * w.d.size();
    if (w.e1.n != (size_t)n) w.e1.alloc(n);
    if (w.e2.n != (size_t)n) w.e2.alloc(n);
    DevBuf<float> &r = w.e1, &dx = w.e2;
    Reducer &red = w.red;
    CgStats st;
    for (int k = 0; k < refinements; ++k) {
        A_hi(x3, r.p, s);
        vec_lin2(r.p, 1.f, y3, -1.f, r.p, n, s);  // r = y - A_hi x
        red.zero(1, s);
        vec_dot(r.p, r.p, n, red.d, s);
        red.fetch(1, s);
        st.last_res = std::sqrt(red.h[0]);
        if (st.last_res < tol) break;
        LAMINO_CUDA(cudaMemsetAsync(dx.p, 0, dx.bytes(), s));
        CgStats in = cgsolver(A_lo, r.p, dx.p, w, inner, tol, s);
        st.iters += in.iters;
        vec_lin2(x3, 1.f, x3, 1.f, dx.p, n, s);
    }
    return st;
}

// ---------------------------------------------------------------------------
// split Bregman (src/bregman.cpp:39-134)
// ---------------------------------------------------------------------------

int split_bregman(const OpFn &A, const float *yT3, float *x3, Dims3 d, float lam, float mu, int outer_max,
                  int inner_max, float tol, float xtol, cudaStream_t s) {
    return split_bregman_refined(A, OpFn(), 0, yT3, x3, d, lam, mu, outer_max, inner_max, tol, xtol, s);
}

int split_bregman_refined(const OpFn &A, const OpFn &A_lo, int refinements, const float *yT3, float *x3, Dims3 d,
                          float lam, float mu, int outer_max, int inner_max, float tol, float xtol, cudaStream_t s) {
    const int64_t V = d.size(), n = 3 * V;
    DevBuf<float> xold(n), dd(9 * V), bb(9 * V), rhs(n);
    LAMINO_CUDA(cudaMemcpyAsync(xold.p, x3, n * 4, cudaMemcpyDeviceToDevice, s));
    LAMINO_CUDA(cudaMemsetAsync(dd.p, 0, dd.bytes(), s));
    LAMINO_CUDA(cudaMemsetAsync(bb.p, 0, bb.bytes(), s));
    OpFn Ap = [&](const float *u, float *out, cudaStream_t st) {
        A(u, out, st);
        laplacian_axpy(out, mu, u, d, st);
    };
    OpFn Ap_lo = [&](const float *u, float *out, cudaStream_t st) {
        A_lo(u, out, st);
        laplacian_axpy(out, mu, u, d, st);
    };
    Reducer red(8);
    CgWork work(d, s);
    int it = 0;
    for (; it < outer_max; ++it) {
        sb_rhs(yT3, dd.p, bb.p, mu, d, rhs.p, s);
        // x = cgsolver(Ap, rhs, x_old, ...)
        LAMINO_CUDA(cudaMemcpyAsync(x3, xold.p, n * 4, cudaMemcpyDeviceToDevice, s));
        if (A_lo && refinements > 0)
            cgsolver_refined(Ap, Ap_lo, rhs.p, x3, work, inner_max, refinements, tol, s);
        else
            cgsolver(Ap, rhs.p, x3, work, inner_max, tol, s);
        sb_shrink(x3, dd.p, bb.p, lam, mu, d, s);
        red.zero(6, s);
        vec_sqdist3(x3, xold.p, V, red.d, s);
        vec_sqdist3(xold.p, nullptr, V, red.d + 3, s);
        red.fetch(6, s);
        double nd = 0.0;
        for (int i = 0; i < 3; ++i) nd += std::sqrt(red.h[i]) / (std::sqrt(red.h[3 + i]) + 1e-8);
        LAMINO_CUDA(cudaMemcpyAsync(xold.p, x3, n * 4, cudaMemcpyDeviceToDevice, s));
        if (nd < xtol) { ++it; break; }
    }
    LAMINO_CUDA(cudaStreamSynchronize(s));
    return it;
}

// ---------------------------------------------------------------------------
// Nesterov (src/nagopt.cpp:116-209)
// ---------------------------------------------------------------------------

__global__ void k_extrap(float *__restrict__ y, const float *__restrict__ x, const float *__restrict__ xo, float beta,
                         int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = x[i] + (x[i] - xo[i]) * beta;
}

// One host read per line-search step: the losses of x and y, |g| and the
// x-change norms (used when the step is accepted) are reduced on the device
// into one buffer and fetched together, where the reference reads each as it
// goes; the values and the decisions are the same.  The reference evaluates
// loss(x) once more after each line search (src/nagopt.cpp); x has not changed
// since the line search's last evaluation, so that value is reused.
NagSolve::NagSolve(GradFn grad, LossTerms loss, float *x3, Dims3 d, int max_iters, float lipschitz, float tol,
                   float xtol, int max_inner, cudaStream_t s)
    : grad_(std::move(grad)), loss_(std::move(loss)), x_(x3), d_(d), max_iters_(max_iters), max_inner_(max_inner),
      tol_(tol), xtol_(xtol), s_(s), xold_(3 * d.size()), y_(3 * d.size()), g_(3 * d.size()),
      red_(2 * loss_.nterms + 9) {
    step_ = step_prev_ = (float)(0.1 / lipschitz);
    LAMINO_CUDA(cudaMemcpyAsync(xold_.p, x_, 3 * d.size() * 4, cudaMemcpyDeviceToDevice, s_));
    done_ = max_iters_ <= 0 || max_inner_ <= 0;
}

// slots: [loss terms of x][loss terms of y][|g_c|^2][|x_c - xold_c|^2][|x_c|^2]
void NagSolve::enqueue() {
    const int64_t V = d_.size(), n = 3 * V;
    const int M = loss_.nterms;
    double *const gsl = red_.d + 2 * M;
    const float beta = (float)(tnew_ * (1.0 / t_ - 1.0));
    tnew_ = 0.5 * (std::sqrt(std::pow(t_, 4) + 4 * std::pow(t_, 2)) - std::pow(t_, 2));
    k_extrap<<<grid_for(n, 256), 256, 0, s_>>>(y_.p, x_, xold_.p, beta, n);
    LAMINO_LAUNCH("k_extrap");
    red_.zero(2 * M + 9, s_);
    grad_(y_.p, g_.p, red_.d + M, s_);
    vec_lin2(x_, 1.f, y_.p, -step_, g_.p, n, s_);
    loss_.enqueue(x_, red_.d, s_);
    vec_sqdist3(g_.p, nullptr, V, gsl, s_);
    vec_sqdist3(x_, xold_.p, V, gsl + 3, s_);
    vec_sqdist3(x_, nullptr, V, gsl + 6, s_);
    LAMINO_CUDA(cudaMemcpyAsync(red_.h, red_.d, sizeof(double) * (2 * M + 9), cudaMemcpyDeviceToHost, s_));
}

bool NagSolve::finish() {
    const int M = loss_.nterms;
    const double *h = red_.h;
    const double ex = loss_.value(h), ey = loss_.value(h + M);
    double gy = 0.0;
    for (int i = 0; i < 3; ++i) gy += std::sqrt(h[2 * M + i]);
    gy *= 0.5 * step_;
    bool line_search_over = false;
    if (ex > ey + gy) {
        step_ *= 0.9f;
    } else {
        step_ = step_prev_;
        t_ = tnew_;
        double xe = 0, xn = 0;
        for (int i = 0; i < 3; ++i) {
            xe += std::sqrt(h[2 * M + 3 + i]);
            xn += std::sqrt(h[2 * M + 6 + i]);
        }
        xerr_ = xe / xn;
        if (xerr_ < xtol_) {
            ++it_;
            done_ = true;
            return true;
        }
        LAMINO_CUDA(cudaMemcpyAsync(xold_.p, x_, 3 * d_.size() * 4, cudaMemcpyDeviceToDevice, s_));
        line_search_over = true;
    }
    if (!line_search_over && ++inner_ < max_inner_) return false;
    // end of an outer iteration: its loss is ex (x unchanged since)
    inner_ = 0;
    ++it_;
    if (ex < tol_ || it_ >= max_iters_) done_ = true;
    return done_;
}

int nagopt(const GradFn &grad, const LossTerms &loss, float *x, Dims3 d, int max_iters, float lipschitz, float tol,
           float xtol, int max_inner, cudaStream_t s) {
    NagSolve nag(grad, loss, x, d, max_iters, lipschitz, tol, xtol, max_inner, s);
    while (!nag.done()) {
        nag.enqueue();
        LAMINO_CUDA(cudaStreamSynchronize(s));
        nag.finish();
    }
    LAMINO_CUDA(cudaStreamSynchronize(s));
    return nag.iterations();
}

// ---------------------------------------------------------------------------
// power iteration
// ---------------------------------------------------------------------------

__global__ void k_uniform(float *__restrict__ x, int64_t n, unsigned long long seed) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        x[i] = (float)((z >> 40) * (1.0 / 16777216.0));
    }
}

// x = Ax / sqrt(*sq) with the factor formed in double and rounded to float, as
// the host does in the loop below
__global__ void k_scale_inv_norm(float *__restrict__ out, const float *__restrict__ x, const double *sq, int64_t n) {
    const float a = (float)(1.0 / sqrt(*sq));
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = a * x[i] + 0.f;
}

double lipschitz(const OpFn &A, Dims3 d, int max_iters, double tol, unsigned long long seed, cudaStream_t s) {
    const int64_t n = 3 * d.size();
    DevBuf<float> x(n), Ax(n);
    if (tol == 0.0 && max_iters > 0) {
        // no early stop: the whole iteration stays on the device (the norms into
        // one slot each, the normalisation read from the slot) and the norms are
        // fetched once; same arithmetic as the loop below
        Reducer red(max_iters + 1);
        red.zero(max_iters + 1, s);
        k_uniform<<<grid_for(n, 256), 256, 0, s>>>(x.p, n, seed);
        LAMINO_LAUNCH("k_uniform");
        vec_dot(x.p, x.p, n, red.d, s);
        k_scale_inv_norm<<<grid_for(n, 256), 256, 0, s>>>(x.p, x.p, red.d, n);
        LAMINO_LAUNCH("k_scale_inv_norm");
        for (int i = 0; i < max_iters; ++i) {
            A(x.p, Ax.p, s);
            vec_dot(Ax.p, Ax.p, n, red.d + 1 + i, s);
            k_scale_inv_norm<<<grid_for(n, 256), 256, 0, s>>>(x.p, Ax.p, red.d + 1 + i, n);
            LAMINO_LAUNCH("k_scale_inv_norm");
        }
        red.fetch(max_iters + 1, s);
        double L = 0.0;
        for (int i = 0; i < max_iters; ++i) {
            const double nA = std::sqrt(red.h[1 + i]);
            if (nA < 1e-12) return 0.0;
            L = nA;
        }
        return L;
    }
    Reducer red(2);
    k_uniform<<<grid_for(n, 256), 256, 0, s>>>(x.p, n, seed);
    LAMINO_LAUNCH("k_uniform");
    red.zero(1, s);
    vec_dot(x.p, x.p, n, red.d, s);
    red.fetch(1, s);
    vec_scale(x.p, (float)(1.0 / std::sqrt(red.h[0])), x.p, n, s);
    double L = 0.0;
    for (int i = 0; i < max_iters; ++i) {
        A(x.p, Ax.p, s);
        red.zero(1, s);
        vec_dot(Ax.p, Ax.p, n, red.d, s);
        red.fetch(1, s);
        double nA = std::sqrt(red.h[0]);
        if (nA < 1e-12) return 0.0;
        vec_scale(x.p, (float)(1.0 / nA), Ax.p, n, s);
        if (std::fabs(nA - L) < tol) { L = nA; break; }
        L = nA;
    }
    LAMINO_CUDA(cudaStreamSynchronize(s));
    return L;
}

}  // namespace lamino
