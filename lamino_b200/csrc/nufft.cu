// ES-kernel NUFFT for the laminography operator (sm_100a).
//
// Reference behaviour replaced: include/nufft.h:37-64 (FINUFFT 3-D type 1 with
// iflag +1 and type 2 with iflag -1, n_modes = {ncols, nrows, nslices},
// upsampfac 2, tol 1.2e-6 in float), src/projection.cpp:42-126 (forward /
// adjoint) and src/gradient.cpp:34-89 (sysmat).
//
// Design.  The points of one geometry are a lattice, and the transform is
// factorised over it.  With the detector axis a = (cos g, 0, -sin g) and
// b(theta) = (cos th sin g, -sin th, cos th cos g) in (x, y, z), point
// (p, j, k) is q = X_k a + Y_j b(theta_p); a is the same for every angle, and
// b's part outside y lies along the fixed axis t = (sin g, 0, cos g).  So
//     q = X_k a + T t + y e_y,   T = Y_j cos(th_p),   y = -Y_j sin(th_p):
// one regular axis X shared by all detector rows of all angles, and a 2-D
// scattered set of (T, y) positions, one per detector row.  Interpolation from
// the fine grid (type 2) then takes two 2-D steps instead of one 3-D step of
// w^3 taps per point:
//   1. (z, x) -> (T, X): the values at the nodes of a regular (T, X) grid, for
//      every fine-grid y (k_nodes_gather: w^2 taps per node, lanes along y);
//   2. (T, y) -> detector rows: w^2 taps per row, the same taps for all columns
//      (k_rows_gather: lanes along X).
// The T axis is oversampled by 2 with respect to the volume's extent along t,
// n3 |sin g| + n1 |cos g|, and deconvolved per mode (its frequency along t is
// k3 sin g + k1 cos g, not an integer).  Type 1 is the transpose.  At the
// padded README size (721 x 71 x 721, 361 x 1233^2 points) that is 49 taps for
// 3.0e8 node values and 49 for 5.5e8 points, all of it contiguous along y or X,
// in place of 343 taps per point from scattered tiles.
// Measured on B200 against antipodal point pairs spread through 3-D tiles (the
// form before): adjoint at that size 333.5 -> 26.6 ms, forward of 181 x 362^2
// points from 362 x 44 x 362 19.5 -> 2.45 ms, sysmat of 2 x 91 x 309^2 points on
// 180 x 16 x 180 19.9 -> 1.29 ms, and no sort of the points on the first call
// (adjoint of a new geometry 351 -> 31 ms).
//
// The three components need one complex transform, not three.  The beam vector
// (sin g sin th, cos th, cos g sin th) spans two dimensions:
//   S = sin g m0 + cos g m2 and C = m1 are projected with weights sin th, cos th.
// S and C are real, so W = S + i C has V_S(q) = (F(q) + conj F(-q)) / 2 and
// V_C(q) = (F(q) - conj F(-q)) / 2i, F the transform of W.  With
// a_p = (sin th - i cos th) / 2 the projection spectrum is
//   P(q) = a_p F(q) + conj(a_p F(-q)),
// and -q is the lattice point (p, nrows-1-j, ncols-1-k).  The second term is
// folded into the 2-D transform over the detector as a real factor and a phase
// (twist below), so only F(q) is evaluated.  The adjoint runs the same steps
// transposed.  This needs a lattice that is symmetric under q -> -q to more than
// float rounding.  The reference's float frequencies are not (their grid is off
// centre by up to 3e-7, which alone would move a 721-wide result by 2e-5), so
// these operators take the antisymmetric part of the float frequencies, with
// products and sums in double; the raw transforms, whose data have no such
// symmetry, keep the float positions.
#include <array>
#include <cmath>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "nufft.cuh"

namespace lamino {

int64_t next_smooth_even(int64_t n) {
    if (n < 2) n = 2;
    if (n % 2) ++n;
    for (;; n += 2) {
        int64_t m = n;
        for (int p : {2, 3, 5})
            while (m % p == 0) m /= p;
        if (m == 1) return n;
    }
}

// Gauss-Legendre nodes on (0, 1) of an even rule on [-1, 1] (Newton iteration on
// P_n), with the weights times the ES kernel: the transform of the kernel at
// frequency k of a grid of nf cells is p(k) = w sum_q wphi_q cos(k pi w x_q / nf).
static constexpr int kQuad = 100;
static std::vector<double2> es_quadrature(double beta) {
    const int nq = 2 * kQuad;
    std::vector<double2> out(kQuad);
    for (int i = 0; i < kQuad; ++i) {
        double x = std::cos(M_PI * (i + 0.75) / (nq + 0.5)), wt = 0.0;
        for (int it = 0; it < 100; ++it) {
            double p0 = 1.0, p1 = x;
            for (int k = 2; k <= nq; ++k) {
                double p2 = ((2.0 * k - 1.0) * x * p1 - (k - 1.0) * p0) / k;
                p0 = p1;
                p1 = p2;
            }
            double dp = nq * (x * p1 - p0) / (x * x - 1.0);
            double dx = p1 / dp;
            x -= dx;
            wt = 2.0 / ((1.0 - x * x) * dp * dp);
            if (std::fabs(dx) < 1e-16) break;
        }
        out[i] = make_double2(x, wt * std::exp(beta * (std::sqrt(1.0 - x * x) - 1.0)));
    }
    return out;
}

NufftPlan::NufftPlan(Dims3 d, double eps_) : vol(d), eps(eps_) {
    if (d.n1 <= 0 || d.n2 <= 0 || d.n3 <= 0) throw Error(ERR_ARG, "volume dims must be positive");
    w = es_width(eps);
    if (w < 4 || w > 8) throw Error(ERR_ARG, "NUFFT tolerance must give kernel width 4..8 (eps 1e-3..1e-7)");
    beta = (float)(2.30 * w);
    nf1 = next_smooth_even(std::max<int64_t>(2 * d.n1, 2 * w));
    nf2 = next_smooth_even(std::max<int64_t>(2 * d.n2, 2 * w));
    nf3 = next_smooth_even(std::max<int64_t>(2 * d.n3, 2 * w));
    if (nf() > (int64_t)INT32_MAX) throw Error(ERR_ARG, "fine grid too large");
    const std::vector<double2> q = es_quadrature(beta);
    quad.alloc(kQuad);
    upload(quad.p, q.data(), (size_t)kQuad);
    auto up = [&](DevBuf<float> &buf, int64_t nf_, int64_t N) {
        std::vector<float> ip(N);
        for (int64_t i = 0; i < N; ++i) {
            const double k = (double)(i - N / 2);
            double p = 0.0;
            for (int t = 0; t < kQuad; ++t) p += q[t].y * std::cos(k * M_PI * w * q[t].x / (double)nf_);
            ip[i] = (float)(1.0 / (w * p));
        }
        buf.alloc(N);
        upload(buf.p, ip.data(), (size_t)N);
    };
    up(ip1, nf1, d.n1);
    up(ip2, nf2, d.n2);
    up(ip3, nf3, d.n3);
    grid.alloc(nf());
    // node grids are 0.9 to 1.2 fine grids for the detectors and volumes that the
    // MBIR drivers pad together
    work.alloc(nf() + nf() / 4);
    // Modes fill the n1 planes [0, (n1 + 1) / 2) and the last n1 / 2 of the fine
    // grid: with the transform along n1 last (type 2) or first (type 1) the other
    // planes skip their 2-D transforms, half the passes along n3 and n2 (1458 x 1458
    // x 144: 6.1 -> 4.5 ms).  Grids below 64 MB stay with one 3-D transform: they are
    // bound by launches.
    split3 = nf() >= (8 << 20);
    int n[3] = {(int)nf1, (int)nf3, (int)nf2};
    if (split3) {
        fft3.make(2, n + 1, CUFFT_C2C, (int)(d.n1 - d.n1 / 2));
        fft3n1.make(1, n, CUFFT_C2C, (int)(nf3 * nf2), (int)(nf3 * nf2));
    } else {
        fft3.make(3, n, CUFFT_C2C, 1);
    }
}

// ---------------------------------------------------------------------------
// the ES kernel on the fine grid
// ---------------------------------------------------------------------------

struct Fine {
    int nf1, nf2, nf3;
    double s1, s2, s3;  // nf / (2 pi)
    float beta;
};

// first tap of a coordinate xc on a grid of s cells per unit (not wrapped), and
// its offset d0 in [-W/2, -W/2 + 1) from the coordinate, in grid units
template <int W>
__device__ __forceinline__ int es_first(double xc, double s, float &d0) {
    const double u = xc * s;
    const double l0 = ceil(u - 0.5 * W);
    d0 = (float)(l0 - u);
    return (int)l0;
}
__device__ __forceinline__ int wrap(int l, int nf) {
    l %= nf;
    return l < 0 ? l + nf : l;
}
// kernel value at tap t of a footprint with offset d0; 0 outside the footprint
template <int W>
__device__ __forceinline__ float es_weight(float d0, int t, float beta) {
    const float a = (d0 + (float)t) * (2.0f / W);
    const float q = 1.0f - a * a;
    return q > 0.f ? expf(beta * (sqrtf(q) - 1.0f)) : 0.f;
}
template <int W>
__device__ __forceinline__ float es_tap(float d0, int t, float beta) {
    return (unsigned)t < (unsigned)W ? es_weight<W>(d0, t, beta) : 0.f;
}

// ---------------------------------------------------------------------------
// volume <-> fine grid
// ---------------------------------------------------------------------------

// CTA -> (i1, first i2, first i3) of its 32 x 32 tile
__device__ __forceinline__ void volume_tile(int n2, int n3, int &i1, int &b2, int &b3) {
    const unsigned t3 = (n3 + 31) / 32, t2 = (n2 + 31) / 32, r = blockIdx.x / t3;
    b3 = (int)(blockIdx.x - r * t3) * 32;
    i1 = (int)(r / t2);
    b2 = (int)(r - i1 * t2) * 32;
}
// Volumes have n3 fastest, the fine grid n2: both sides transpose 32 x 32 tiles
// of (i3, i2) through shared memory so that reads and writes are contiguous.
// W = S + i C (real volume, gamma's sines) or the complex modes, deconvolved.
template <bool CPLX>
__global__ void __launch_bounds__(256) k_pad(const float *__restrict__ x, const float2 *__restrict__ modes, int n1,
                                             int n2, int n3, float sg, float cg, float2 *__restrict__ g, Fine F,
                                             const float *__restrict__ ip1, const float *__restrict__ ip2,
                                             const float *__restrict__ ip3, const float *__restrict__ ipT) {
    __shared__ float2 tile[32][33];
    int i1, b2, b3;
    volume_tile(n2, n3, i1, b2, b3);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t V = (int64_t)n1 * n2 * n3;
    int l1 = i1 - n1 / 2; if (l1 < 0) l1 += F.nf1;
    const float c1 = __ldg(ip1 + i1);
    const int i3 = b3 + tx;
    if (i3 < n3) {
        float c = c1 * __ldg(ip3 + i3);
        if (ipT) c *= __ldg(ipT + (int64_t)i1 * n3 + i3);
        for (int r = ty; r < 32 && b2 + r < n2; r += 8) {
            const int64_t idx = ((int64_t)i1 * n2 + b2 + r) * n3 + i3;
            const float d = c * __ldg(ip2 + b2 + r);
            if (CPLX) {
                const float2 v = modes[idx];
                tile[r][tx] = make_float2(v.x * d, v.y * d);
            } else {
                tile[r][tx] = make_float2((sg * x[idx] + cg * x[2 * V + idx]) * d, x[V + idx] * d);
            }
        }
    }
    __syncthreads();
    const int i2 = b2 + tx;
    if (i2 >= n2) return;
    int l2 = i2 - n2 / 2; if (l2 < 0) l2 += F.nf2;
    for (int r = ty; r < 32 && b3 + r < n3; r += 8) {
        int l3 = b3 + r - n3 / 2; if (l3 < 0) l3 += F.nf3;
        g[((int64_t)l1 * F.nf3 + l3) * F.nf2 + l2] = tile[tx][r];
    }
}

// fine grid -> modes: y_i (+)= the beam components of U = S + i C, or the complex modes
template <bool CPLX>
__global__ void __launch_bounds__(256) k_extract(const float2 *__restrict__ g, int n1, int n2, int n3, float sg,
                                                 float cg, float *__restrict__ y, float2 *__restrict__ modes, Fine F,
                                                 const float *__restrict__ ip1, const float *__restrict__ ip2,
                                                 const float *__restrict__ ip3, const float *__restrict__ ipT,
                                                 float scale, int accumulate) {
    __shared__ float2 tile[32][33];
    int i1, b2, b3;
    volume_tile(n2, n3, i1, b2, b3);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t V = (int64_t)n1 * n2 * n3;
    int l1 = i1 - n1 / 2; if (l1 < 0) l1 += F.nf1;
    const int i2 = b2 + tx;
    if (i2 < n2) {
        int l2 = i2 - n2 / 2; if (l2 < 0) l2 += F.nf2;
        for (int r = ty; r < 32 && b3 + r < n3; r += 8) {
            int l3 = b3 + r - n3 / 2; if (l3 < 0) l3 += F.nf3;
            tile[tx][r] = g[((int64_t)l1 * F.nf3 + l3) * F.nf2 + l2];
        }
    }
    __syncthreads();
    const int i3 = b3 + tx;
    if (i3 >= n3) return;
    float c = __ldg(ip1 + i1) * __ldg(ip3 + i3) * scale;
    if (ipT) c *= __ldg(ipT + (int64_t)i1 * n3 + i3);
    for (int r = ty; r < 32 && b2 + r < n2; r += 8) {
        const int64_t idx = ((int64_t)i1 * n2 + b2 + r) * n3 + i3;
        const float d = c * __ldg(ip2 + b2 + r);
        const float2 v = tile[r][tx];
        const float re = v.x * d, im = v.y * d;
        if (CPLX) {
            modes[idx] = make_float2(re, im);
        } else if (accumulate) {
            y[idx] += sg * re;
            y[V + idx] += im;
            y[2 * V + idx] += cg * re;
        } else {
            y[idx] = sg * re;
            y[V + idx] = im;
            y[2 * V + idx] = cg * re;
        }
    }
}

// ---------------------------------------------------------------------------
// building a lattice
// ---------------------------------------------------------------------------

// column frequencies, beam factors and the twist factors: for detector-space
// index m of a dimension of n, d = n / 2,
//   (cos, sin)(pi m (2 d + 1) / n + off u) and (cos, sin)(pi m / n),
// u the centred index of m and off the mean of the dimension's float
// frequencies: a spectrum sampled off centre is an image times e^{-i off u}, of
// which the operators take the real part
__device__ __forceinline__ double odd_part(const float *q, int i, int n) {
    return 0.5 * ((double)__ldg(q + i) - (double)__ldg(q + n - 1 - i));
}
__global__ void k_lat_tables(GeomView g, bool raw, double offX, double offY, double *__restrict__ X, float2 *__restrict__ a,
                             float4 *__restrict__ trow, float4 *__restrict__ tcol) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g.ncols) X[i] = raw ? (double)g.qX[i] : odd_part(g.qX, i, g.ncols);
    if (i < g.nproj) a[i] = make_float2(0.5f * g.st[i], -0.5f * g.ct[i]);
    for (int d = 0; d < 2; ++d) {
        const int n = d ? g.ncols : g.nrows;
        if (i >= n) continue;
        double s0, c0, s1, c1;
        const long long r = ((long long)i * (2 * (n / 2) + 1)) % (2LL * n);
        const int u = i < (n + 1) / 2 ? i : i - n;
        sincos(r * (M_PI / n) + u * (d ? offX : offY), &s0, &c0);
        sincospi((double)i / n, &s1, &c1);
        (d ? tcol : trow)[i] = make_float4((float)c0, (float)s0, (float)c1, (float)s1);
    }
}

// 1 / p_T at every mode's frequency along t, from the plan's quadrature
__global__ void k_lat_deconv(const double2 *__restrict__ quad, int n1, int n3, double sg, double cg, int w, int nTf,
                             float *__restrict__ ipT) {
    __shared__ double2 q[kQuad];
    for (int i = threadIdx.x; i < kQuad; i += blockDim.x) q[i] = quad[i];
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n1 * n3) return;
    const int i1 = i / n3, i3 = i - i1 * n3;
    const double k = (i3 - n3 / 2) * sg + (i1 - n1 / 2) * cg;
    double p = 0.0;
    for (int t = 0; t < kQuad; ++t) p += q[t].y * cospi(k * w * q[t].x / nTf);
    ipT[i] = (float)(1.0 / (w * p));
}

// place of a detector row where first halves are stored first (Lattice::half)
__device__ __forceinline__ int64_t half_row(int p, int j, int np, int nr) {
    const int jh = (nr + 1) / 2;
    return j < jh ? (int64_t)p * jh + j : (int64_t)np * jh + (int64_t)p * (nr - jh) + (j - jh);
}
// the (T, y) position of detector row `id` = p nrows + j and its footprint; a row
// of an angle that is not a number gets some cell of the lattice and a footprint
// whose weights are all zero
struct RowPos {
    int p, j, lT, ly;
    float dT, dy;
};
template <int W>
__device__ __forceinline__ RowPos row_pos(const GeomView &g, bool raw, double invh, int T0, int nstart,
                                          const Fine &F, int id) {
    RowPos r;
    r.p = id / g.nrows;
    r.j = id - r.p * g.nrows;
    double T, y;
    if (raw) {
        const float qy = __ldg(g.qY + r.j);
        T = (double)__fmul_rn(qy, __ldg(g.ct + r.p));
        y = (double)__fmul_rn(-qy, __ldg(g.st + r.p));
    } else {
        const double qy = odd_part(g.qY, r.j, g.nrows);
        T = qy * (double)__ldg(g.ct + r.p);
        y = -qy * (double)__ldg(g.st + r.p);
    }
    r.lT = max(0, min(es_first<W>(T, invh, r.dT) - T0, nstart - 1));
    r.ly = wrap(es_first<W>(y, F.s2, r.dy), F.nf2);
    return r;
}
template <int W>
__global__ void __launch_bounds__(256) k_rows_count(GeomView g, bool raw, double invh,
                                                    int T0, int nstart, Fine F, uint32_t *__restrict__ cnt) {
    const int n = g.nproj * g.nrows;
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < n; id += gridDim.x * blockDim.x) {
        const RowPos r = row_pos<W>(g, raw, invh, T0, nstart, F, id);
        atomicAdd(cnt + (int64_t)r.ly * nstart + r.lT, 1u);
    }
}
template <int W>
__global__ void __launch_bounds__(256) k_rows_place(GeomView g, bool raw, double invh,
                                                    bool half, int T0, int nstart, Fine F, uint32_t *__restrict__ cursor,
                                                    int4 *__restrict__ pt, float2 *__restrict__ pd) {
    const int n = g.nproj * g.nrows;
    for (int id = blockIdx.x * blockDim.x + threadIdx.x; id < n; id += gridDim.x * blockDim.x) {
        const RowPos r = row_pos<W>(g, raw, invh, T0, nstart, F, id);
        const uint32_t at = atomicAdd(cursor + (int64_t)r.ly * nstart + r.lT, 1u);
        pt[at] = make_int4(half ? (int)half_row(r.p, r.j, g.nproj, g.nrows) : id, r.lT, r.ly, id);
        pd[at] = make_float2(r.dT, r.dy);
    }
}


// ---------------------------------------------------------------------------
// (z, x) <-> (T, X)
// ---------------------------------------------------------------------------

// the lattice's columns first .. first + nc - 1 of ncols (Lattice::ncc at a time)
struct LatView {
    const double *X;
    double cg, sg, h;
    int nc, nT, T0;
    int first, ncols;
    double p1, p3, kX, kT;  // position per z and x cell, columns and T lines per position
};
// footprint of node (line t, column k) in the (z, x) plane
template <int W>
__device__ __forceinline__ void node_pos(const LatView &L, const Fine &F, int t, int k, int &l1, int &l3, float &d1,
                                         float &d3) {
    const double X = L.X[k], T = (L.T0 + t) * L.h;
    l3 = es_first<W>(X * L.cg + T * L.sg, F.s3, d3);
    l1 = es_first<W>(T * L.cg - X * L.sg, F.s1, d1);
}

// Fine grid -> nodes.  A CTA owns 128 nodes (16 columns x 8 T lines, or 8 x 16).
// Per chunk of up to 16 y it stages the (z, x) box of cells that the nodes'
// footprints cover in shared memory; a thread then takes two nodes, one T line
// apart, and two y: the lattice keeps T lines at most one cell apart (see lattice()), so both
// footprints lie in (W + 1)^2 cells, each read once (16 bytes) and weighted for
// both nodes with the weights padded by zeros.  A tile with a pair that starts
// further apart, which rounding alone could bring about, goes tap by tap.  Results go through shared memory
// to the node grid [T][y][X], X fastest.  Bound by shared-memory wavefronts:
// 64 16-byte reads per four values where one node and one y at a time takes 196
// of 8 bytes.  A box that does not fit (a detector far coarser than the fine
// grid) is read from global memory tap by tap.
// Measured (before: every tap from global memory, one node and one y per lane,
// five wavefronts per tap where runs straddle lines): 362 x 1020 nodes x 90 y
// 1314 -> 857 us; staging through registers instead of asynchronous copies 1267 us.
constexpr int kNodes = 128, kNodeY = 16;
__device__ __forceinline__ void copy16_async(void *smem, const void *global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(global) : "memory");
}
template <int W, int kNodeK>
__global__ void __launch_bounds__(256, 2) k_nodes_gather(LatView L, Fine F, const float2 *__restrict__ g,
                                                         float2 *__restrict__ G, int pitch, int ktiles, int ychunk,
                                                         uint32_t ydiv, int nchunk, int boxcap) {
    constexpr int kNodeT = kNodes / kNodeK, kPairs = kNodes / 2;
    extern __shared__ __align__(16) float2 box[];  // [cell][ychunk]; then the results [y][node], kNodes + 1 apart
    __shared__ float w1[W + 2][kNodes], w3[W + 2][kNodes];  // weights between two zeros
    __shared__ int n1[kNodes], n3[kNodes];
    __shared__ int lo1, hi1, lo3, hi3;
    const int t0 = blockIdx.x / ktiles, k0 = (blockIdx.x - t0 * ktiles) * kNodeK;
    const int tid = threadIdx.x;
    if (tid == 0) {
        lo1 = lo3 = 0x7fffffff;
        hi1 = hi3 = -0x7fffffff;
    }
    __syncthreads();
    {
        // threads 0..127 the z side of a node, 128..255 the x side
        const int n = tid & (kNodes - 1);
        const int k = min(k0 + n % kNodeK, L.nc - 1), t = min(t0 * kNodeT + n / kNodeK, L.nT - 1);
        int l1, l3;
        float d1, d3;
        node_pos<W>(L, F, t, k, l1, l3, d1, d3);
        const bool z = tid < kNodes;
        const int l = z ? l1 : l3;
        (z ? n1 : n3)[n] = l;
        atomicMin(z ? &lo1 : &lo3, __reduce_min_sync(0xffffffffu, l));
        atomicMax(z ? &hi1 : &hi3, __reduce_max_sync(0xffffffffu, l));
        float(*wt)[kNodes] = z ? w1 : w3;
        wt[0][n] = wt[W + 1][n] = 0.f;
#pragma unroll
        for (int r = 0; r < W; ++r) wt[r + 1][n] = es_weight<W>(z ? d1 : d3, r, F.beta);
    }
    __syncthreads();
    bool far = false;
    if (tid < kPairs) {
        const int a = tid / kNodeK * 2 * kNodeK + tid % kNodeK, b = a + kNodeK;
        far = abs(n1[a] - n1[b]) > 1 || abs(n3[a] - n3[b]) > 1;
    }
    const int B1 = hi1 - lo1 + W + 1, B3 = hi3 - lo3 + W + 1;
    const int base1 = wrap(lo1, F.nf1), base3 = wrap(lo3, F.nf3);
    const bool staged = !__syncthreads_or(far) && (int64_t)B1 * B3 <= boxcap;
    const int half = ychunk / 2;
    for (int c = blockIdx.y; c < nchunk; c += gridDim.y) {
        const int y0 = c * ychunk, ny = min(ychunk, F.nf2 - y0);
        if (staged) {
            // eight lanes per cell, two y per load (y0 and nf2 are even); 32 cells a pass
            const int y = 2 * (tid & 7);
            int r1 = 0, r3 = tid >> 3;
            while (r3 >= B3) { r3 -= B3; ++r1; }
            while (r1 < B1) {
                int i1 = base1 + r1, i3 = base3 + r3;
                while (i1 >= F.nf1) i1 -= F.nf1;
                while (i3 >= F.nf3) i3 -= F.nf3;
                if (y < ny) copy16_async(box + (r1 * B3 + r3) * ychunk + y, g + ((int64_t)i1 * F.nf3 + i3) * F.nf2 + y0 + y);
                r3 += 32;
                while (r3 >= B3) { r3 -= B3; ++r1; }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        // (pair, y pair) items, at most two per thread; kept until the box is free
        float4 va[2], vb[2];
        int where[2];
#pragma unroll
        for (int it = 0; it < 2; ++it) {
            const int e = tid + 256 * it;
            const int q = (int)__umulhi((uint32_t)e, ydiv), y = 2 * (e - q * half);
            where[it] = -1;
            if (q >= kPairs || y >= ny) continue;
            const int a = q / kNodeK * 2 * kNodeK + q % kNodeK, b = a + kNodeK;  // nodes of the pair
            where[it] = y * (kNodes + 1) + a;
            float2 a0 = make_float2(0.f, 0.f), a1 = a0, b0 = a0, b1 = a0;
            if (staged) {
                const int s1 = min(n1[a], n1[b]), s3 = min(n3[a], n3[b]);
                const float *wa1 = &w1[1 - (n1[a] - s1)][a], *wb1 = &w1[1 - (n1[b] - s1)][b];
                const float *wa3 = &w3[1 - (n3[a] - s3)][a], *wb3 = &w3[1 - (n3[b] - s3)][b];
                const float2 *p = box + ((s1 - lo1) * B3 + s3 - lo3) * ychunk + y;
                float ua[W + 1], ub[W + 1];
#pragma unroll
                for (int r = 0; r <= W; ++r) {
                    ua[r] = wa3[r * kNodes];
                    ub[r] = wb3[r * kNodes];
                }
#pragma unroll
                for (int r1 = 0; r1 <= W; ++r1) {
                    const float2 *row = p + r1 * B3 * ychunk;
                    float2 sa0 = make_float2(0.f, 0.f), sa1 = sa0, sb0 = sa0, sb1 = sa0;
#pragma unroll
                    for (int r3 = 0; r3 <= W; ++r3) {
                        const float4 v = *reinterpret_cast<const float4 *>(row + r3 * ychunk);
                        const float2 x = make_float2(v.x, v.y), z = make_float2(v.z, v.w);
                        const float2 wa = make_float2(ua[r3], ua[r3]), wb = make_float2(ub[r3], ub[r3]);
                        sa0 = __ffma2_rn(wa, x, sa0);
                        sa1 = __ffma2_rn(wa, z, sa1);
                        sb0 = __ffma2_rn(wb, x, sb0);
                        sb1 = __ffma2_rn(wb, z, sb1);
                    }
                    const float fa = wa1[r1 * kNodes], fb = wb1[r1 * kNodes];
                    a0 = __ffma2_rn(make_float2(fa, fa), sa0, a0);
                    a1 = __ffma2_rn(make_float2(fa, fa), sa1, a1);
                    b0 = __ffma2_rn(make_float2(fb, fb), sb0, b0);
                    b1 = __ffma2_rn(make_float2(fb, fb), sb1, b1);
                }
            } else {
                for (int m = 0; m < 2; ++m) {
                    const int n = m ? b : a, l1 = wrap(n1[n], F.nf1), l3 = wrap(n3[n], F.nf3);
                    float2 c0 = make_float2(0.f, 0.f), c1 = c0;
                    for (int r1 = 0; r1 < W; ++r1) {
                        int i1 = l1 + r1; if (i1 >= F.nf1) i1 -= F.nf1;
                        const float2 *row = g + (int64_t)i1 * F.nf3 * F.nf2 + y0 + y;
                        for (int r3 = 0; r3 < W; ++r3) {
                            int i3 = l3 + r3; if (i3 >= F.nf3) i3 -= F.nf3;
                            const float t = w1[r1 + 1][n] * w3[r3 + 1][n];
                            const float4 v = __ldg(reinterpret_cast<const float4 *>(row + (int64_t)i3 * F.nf2));
                            c0 = __ffma2_rn(make_float2(t, t), make_float2(v.x, v.y), c0);
                            c1 = __ffma2_rn(make_float2(t, t), make_float2(v.z, v.w), c1);
                        }
                    }
                    if (m) { b0 = c0; b1 = c1; } else { a0 = c0; a1 = c1; }
                }
            }
            va[it] = make_float4(a0.x, a0.y, a1.x, a1.y);
            vb[it] = make_float4(b0.x, b0.y, b1.x, b1.y);
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < 2; ++it)
            if (where[it] >= 0) {
                float2 *o = box + where[it];
                o[0] = make_float2(va[it].x, va[it].y);
                o[kNodeK] = make_float2(vb[it].x, vb[it].y);
                o[kNodes + 1] = make_float2(va[it].z, va[it].w);
                o[kNodes + 1 + kNodeK] = make_float2(vb[it].z, vb[it].w);
            }
        __syncthreads();
        for (int e = tid; e < kNodes * ny; e += 256) {
            const int n = e & (kNodes - 1), y = e / kNodes;
            const int k = k0 + n % kNodeK, t = t0 * kNodeT + n / kNodeK;
            if (k < L.nc && t < L.nT) G[((int64_t)t * F.nf2 + y0 + y) * pitch + k] = box[y * (kNodes + 1) + n];
        }
        __syncthreads();
    }
}

// 2-D tiles in strips of 8 along x, y within a strip: the source values that a
// tile shares with its neighbours in both directions are then still in L2 (in
// row order the README-size detector rows between two rows of tiles are 60 MB).
constexpr int kStrip = 8;
__host__ __device__ __forceinline__ int64_t strip_count(int64_t nx, int64_t ny) { return (nx + kStrip - 1) / kStrip * kStrip * ny; }
__device__ __forceinline__ bool strip_order(int i, int nx, int ny, int &x, int &y) {
    const int s = i / (kStrip * ny), r = i - s * (kStrip * ny);
    y = r / kStrip;
    x = s * kStrip + r - y * kStrip;
    return x < nx && y < ny;
}

// Nodes -> fine grid (the transpose).  A CTA owns 4 x 4 (z, x) cells for all y,
// a thread one y: it walks the nodes whose footprint meets the cells and adds
// each into its 16 complex sums, held in registers, so no cell is written
// twice and the order of the sum is fixed.  The nodes are found from the
// lattice: the cells' box of footprint starts, turned into (X, T), bounds a
// range of columns and lines; candidates are tested in parallel and the
// accepted ones listed, with their 16 weights, in shared memory.  The box is
// tried at every period of the fine grid that the lattice reaches.  The first list
// needs the lattice only, so it is built while the row kernel's last blocks still
// run (type 1 of 180 x 22 x 180 / 80 x 24 x 180: 148 -> 141 us with the row
// kernel's own list over the zeroing before it).
constexpr int kCell = 4;
template <int W>
__global__ void __launch_bounds__(256, 3) k_nodes_spread(LatView L, Fine F, int reach1, int reach3, int xtiles,
                                                      const float2 *Gt, float2 *g) {
    extern __shared__ __align__(16) unsigned char nsm[];
    allow_next();
    const int cap = 2 * blockDim.x;
    float4 *lw = reinterpret_cast<float4 *>(nsm);  // [cap][kCell]
    int *ln = reinterpret_cast<int *>(lw + cap * kCell);
    __shared__ int wsum[9];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    int xt, zt;
    if (!strip_order(blockIdx.x, xtiles, (F.nf1 + kCell - 1) / kCell, xt, zt)) return;
    const int c1 = zt * kCell, c3 = xt * kCell;
    const int y = blockIdx.y * blockDim.x + tid;
    const float2 *src = Gt + min(y, F.nf2 - 1);
    float2 re[kCell][2], im[kCell][2];
#pragma unroll
    for (int i = 0; i < kCell; ++i) re[i][0] = re[i][1] = im[i][0] = im[i][1] = make_float2(0.f, 0.f);
    int n = 0;  // listed nodes (the same in every thread)
    auto flush = [&]() {
        wait_previous();
        __syncthreads();
#pragma unroll 4
        for (int q = 0; q < n; ++q) {
            const float2 v = src[(int64_t)ln[q] * F.nf2];
            const float2 vr = make_float2(v.x, v.x), vi = make_float2(v.y, v.y);
#pragma unroll
            for (int i = 0; i < kCell; ++i) {
                const float4 t = lw[q * kCell + i];
                re[i][0] = __ffma2_rn(make_float2(t.x, t.y), vr, re[i][0]);
                re[i][1] = __ffma2_rn(make_float2(t.z, t.w), vr, re[i][1]);
                im[i][0] = __ffma2_rn(make_float2(t.x, t.y), vi, im[i][0]);
                im[i][1] = __ffma2_rn(make_float2(t.z, t.w), vi, im[i][1]);
            }
        }
        __syncthreads();
        n = 0;
    };
    // copies of the cells, one period apart, that the lattice reaches: the
    // footprints lie in [-reach, reach] along each axis
    const int m1 = (reach1 + c1 + kCell) / F.nf1, m3 = (reach3 + c3 + kCell) / F.nf3;
    for (int b1 = c1 - m1 * F.nf1; b1 <= reach1; b1 += F.nf1)
        for (int b3 = c3 - m3 * F.nf3; b3 <= reach3; b3 += F.nf3) {
            // positions whose footprint starts in [b - W + 1, b + kCell - 1]
            const double zlo = (b1 - W + 0.5 * W) * L.p1, zhi = (b1 + kCell - 1 + 0.5 * W) * L.p1;
            const double xlo = (b3 - W + 0.5 * W) * L.p3, xhi = (b3 + kCell - 1 + 0.5 * W) * L.p3;
            const double xm = 0.5 * (xlo + xhi), zm = 0.5 * (zlo + zhi), xr = 0.5 * (xhi - xlo), zr = 0.5 * (zhi - zlo);
            const double Xm = xm * L.cg - zm * L.sg, Xr = xr * fabs(L.cg) + zr * fabs(L.sg);
            const double Tm = xm * L.sg + zm * L.cg, Tr = xr * fabs(L.sg) + zr * fabs(L.cg);
            // one column / line of margin for the rounding of the positions
            const int ka = max(0, (int)floor((Xm - Xr + M_PI) * L.kX - 0.5) - 1 - L.first);
            const int kb = min(L.nc - 1, (int)ceil((Xm + Xr + M_PI) * L.kX - 0.5) + 1 - L.first);
            const int ta = max(0, (int)floor((Tm - Tr) * L.kT) - L.T0 - 1);
            const int tb = min(L.nT - 1, (int)ceil((Tm + Tr) * L.kT) - L.T0 + 1);
            if (ka > kb || ta > tb) continue;
            const int nk = kb - ka + 1, cnt = nk * (tb - ta + 1);
            for (int base = 0; base < cnt; base += blockDim.x) {
                const int id = base + tid;
                bool ok = false;
                int e1 = 0, e3 = 0, node = 0;
                float d1 = 0.f, d3 = 0.f;
                if (id < cnt) {
                    const int t = ta + id / nk, k = ka + id % nk;
                    node_pos<W>(L, F, t, k, e1, e3, d1, d3);
                    e1 = b1 - e1;  // tap of the box's first cell
                    e3 = b3 - e3;
                    ok = e1 > -kCell && e1 < W && e3 > -kCell && e3 < W;
                    node = t * L.nc + k;
                }
                const unsigned m = __ballot_sync(0xffffffffu, ok);
                if (lane == 0) wsum[warp] = __popc(m);
                __syncthreads();
                int at = n + __popc(m & ((1u << lane) - 1u)), tot = 0;
                for (int v = 0; v < nwarps; ++v) {
                    if (v == warp) at += tot;
                    tot += wsum[v];
                }
                if (ok) {
                    float u[kCell];
#pragma unroll
                    for (int i = 0; i < kCell; ++i) u[i] = es_tap<W>(d3, e3 + i, F.beta);
#pragma unroll
                    for (int i = 0; i < kCell; ++i) {
                        const float s = es_tap<W>(d1, e1 + i, F.beta);
                        lw[at * kCell + i] = make_float4(s * u[0], s * u[1], s * u[2], s * u[3]);
                    }
                    ln[at] = node;
                }
                n += tot;
                __syncthreads();
                if (n > cap - (int)blockDim.x) flush();
            }
        }
    flush();
    if (y >= F.nf2) return;
#pragma unroll
    for (int i = 0; i < kCell; ++i) {
        if (c1 + i >= F.nf1) break;
        float2 *o = g + ((int64_t)(c1 + i) * F.nf3 + c3) * F.nf2 + y;
#pragma unroll
        for (int r = 0; r < kCell; ++r) {
            if (c3 + r >= F.nf3) break;
            const float2 a = re[i][r / 2], b = im[i][r / 2];
            float2 v = r & 1 ? make_float2(a.y, b.y) : make_float2(a.x, b.x);
            if (L.first) v = make_float2(v.x + o[r * F.nf2].x, v.y + o[r * F.nf2].y);
            o[r * F.nf2] = v;
        }
    }
}

// ---------------------------------------------------------------------------
// (T, y) <-> detector rows
// ---------------------------------------------------------------------------

// Nodes -> rows.  A CTA takes 32 rows, consecutive in cell order, and 64
// columns; a warp two rows at a time, two columns per lane, 16-byte loads
// of contiguous columns.  Rows of neighbouring cells share most of their taps,
// which stay in L1, whose bandwidth is the bound.  There are 0.7 to 1.7 rows per
// cell, so the next row mostly starts in the same T line or the next one: w + 1
// lines then hold the taps of both, with the weights padded by zeros, and each value
// is read once for the two (the weights in registers, at three CTAs per SM).
// Measured (before: one row at a time): 2 x 91 x 309^2 270 -> 212 us, 181 x 362^2
// 398 -> 340 us, 90 x 200 x 181 58.8 -> 50.9 us.
constexpr int kRowGroup = 32;
template <int W>
__global__ void __launch_bounds__(256, 3) k_rows_gather(const int4 *__restrict__ pt, const float2 *__restrict__ pd, int nrow,
                                                     const float2 *__restrict__ G, int nf2, int pitch, int nc, int ncols,
                                                     int groups, float beta, float2 *__restrict__ out) {
    __shared__ float wT[kRowGroup][W + 2], wy[kRowGroup][W];  // wT between two zeros
    __shared__ int4 info[kRowGroup];
    const int kb = blockIdx.x / groups, base = (blockIdx.x - kb * groups) * kRowGroup, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 2 * kRowGroup) {
        const int r = threadIdx.x & (kRowGroup - 1), q = base + r;
        if (q < nrow) {
            const float2 d = pd[q];
            if (threadIdx.x < kRowGroup) {
                info[r] = pt[q];
#pragma unroll
                for (int t = 0; t < W; ++t) wT[r][t + 1] = es_weight<W>(d.x, t, beta);
                wT[r][0] = wT[r][W + 1] = 0.f;
            } else {
#pragma unroll
                for (int t = 0; t < W; ++t) wy[r][t] = es_weight<W>(d.y, t, beta);
            }
        }
    }
    __syncthreads();
    const int k = kb * 64 + 2 * lane;
    if (k >= nc) return;
    const int64_t line = (int64_t)nf2 * pitch;
    auto store = [&](int id, float2 a0, float2 a1) {
        float2 *o = out + (int64_t)id * ncols + k;
        o[0] = a0;
        if (k + 1 < nc) o[1] = a1;
    };
    auto tap = [](float u, float4 v, float2 &s0, float2 &s1) {
        s0 = __ffma2_rn(make_float2(u, u), make_float2(v.x, v.y), s0);
        s1 = __ffma2_rn(make_float2(u, u), make_float2(v.z, v.w), s1);
    };
    for (int r = 2 * warp; r < kRowGroup && base + r < nrow; r += 16) {
        const int4 I = info[r], J = info[r + 1];
        const bool two = base + r + 1 < nrow;
        const int d = J.y - I.y;
        if (two && J.z == I.z && (unsigned)d <= 1u) {  // W + 1 lines hold the taps of both
            const float2 *p = G + I.y * line + k;
            float wa[W + 1], wb[W + 1];
#pragma unroll
            for (int t = 0; t <= W; ++t) {
                wa[t] = wT[r][t + 1];
                wb[t] = wT[r + 1][t + 1 - d];
            }
            float2 a0 = make_float2(0.f, 0.f), a1 = a0, b0 = a0, b1 = a0;
#pragma unroll
            for (int t2 = 0; t2 < W; ++t2) {
                int yy = I.z + t2; if (yy >= nf2) yy -= nf2;
                const float2 *q = p + (int64_t)yy * pitch;
                float2 s0 = make_float2(0.f, 0.f), s1 = s0, u0 = s0, u1 = s0;
#pragma unroll
                for (int t1 = 0; t1 <= W; ++t1) {
                    // (with d = 0 the line after the last one may not exist; its weights are zero)
                    const float4 v = __ldg(reinterpret_cast<const float4 *>(q + (t1 < W ? t1 : W - 1 + d) * line));
                    tap(wa[t1], v, s0, s1);
                    tap(wb[t1], v, u0, u1);
                }
                const float fa = wy[r][t2], fb = wy[r + 1][t2];
                a0 = __ffma2_rn(make_float2(fa, fa), s0, a0);
                a1 = __ffma2_rn(make_float2(fa, fa), s1, a1);
                b0 = __ffma2_rn(make_float2(fb, fb), u0, b0);
                b1 = __ffma2_rn(make_float2(fb, fb), u1, b1);
            }
            store(I.x, a0, a1);
            store(J.x, b0, b1);
            continue;
        }
        for (int e = 0; e < 1 + two; ++e) {
            const int4 R = e ? J : I;
            const float2 *p = G + R.y * line + k;
            float2 a0 = make_float2(0.f, 0.f), a1 = a0;
#pragma unroll
            for (int t2 = 0; t2 < W; ++t2) {
                int yy = R.z + t2; if (yy >= nf2) yy -= nf2;
                const float2 *q = p + (int64_t)yy * pitch;
                float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
                for (int t1 = 0; t1 < W; ++t1)
                    tap(wT[r + e][t1 + 1], __ldg(reinterpret_cast<const float4 *>(q + t1 * line)), s0, s1);
                const float u = wy[r + e][t2];
                a0 = __ffma2_rn(make_float2(u, u), s0, a0);
                a1 = __ffma2_rn(make_float2(u, u), s1, a1);
            }
            store(R.x, a0, a1);
        }
    }
}

// the run of rows (first, count) that start in y cell c2 - (W - 1) + r, if the
// tile's y cells (the last tile has fewer than kCell where nf2 is no multiple of it) lie
// in the footprint, and whose footprint meets T cells [c1, c1 + kCell)
template <int W>
__device__ __forceinline__ int2 tile_run(const uint32_t *__restrict__ start, int nstart, int nf2, int c1, int c2, int r) {
    if (r - (W - 1) >= nf2 - c2) return make_int2(0, 0);
    const int lo = max(0, c1 - (W - 1)), hi = min(nstart - 1, c1 + kCell - 1);
    const uint32_t *o = start + (int64_t)wrap(c2 - (W - 1) + r, nf2) * nstart;
    return make_int2((int)o[lo], (int)(o[hi + 1] - o[lo]));
}
// work items of k_rows_spread: (tile, first row of the segment, sign bit set if
// the tile has several segments); empty tiles get one item, which stores zeros.
// Tiles are taken in strips (strip_order).
template <int W>
__global__ void __launch_bounds__(128) k_tile_items(const uint32_t *__restrict__ start, int nstart, int nf2, int ntile,
                                                    int ntiles, int seg, int *__restrict__ nitem, int2 *__restrict__ items) {
    int tx, ty;
    if (!strip_order(blockIdx.x * blockDim.x + threadIdx.x, ntile, ntiles / ntile, tx, ty)) return;
    const int t = ty * ntile + tx, c1 = tx * kCell, c2 = ty * kCell;
    int n = 0;
    for (int r = 0; r < W + kCell - 1; ++r) n += tile_run<W>(start, nstart, nf2, c1, c2, r).y;
    const int m = max(1, (n + seg - 1) / seg), at = atomicAdd(nitem, m);
    for (int i = 0; i < m; ++i) items[at + i] = make_int2(t, (i * seg) | (m > 1 ? (int)0x80000000 : 0));
}
__global__ void __launch_bounds__(256) k_tiles_zero(const int *__restrict__ nitem, const int2 *__restrict__ items, int nT,
                                                    int ntile, int nf2, int nc, float2 *__restrict__ Gt) {
    allow_next();
    const int n = __ldg(nitem);
    for (int q = blockIdx.x; q < n; q += gridDim.x) {
        const int2 item = __ldg(items + q);
        if (item.y != (int)0x80000000) continue;  // first segment of several
        const int ty = item.x / ntile, c1 = (item.x - ty * ntile) * kCell, c2 = ty * kCell;
        for (int e = threadIdx.x; e < 2 * kCell * nc; e += blockDim.x) {
            const int h = e & 1, i = (e >> 1) & (kCell - 1), k = e >> 3;
            if (c1 + i < nT && c2 + 2 * h < nf2)
                *reinterpret_cast<float4 *>(Gt + ((int64_t)(c1 + i) * nc + k) * nf2 + c2 + 2 * h) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
}

// Rows -> nodes (the transpose).  A CTA owns 4 x 4 (T, y) cells, a thread one
// column: 16 complex sums in registers over the rows whose footprint meets the
// cells, which the cell order gives as W + 3 runs (one per y start).  Writes
// the node grid as [T][X][y], y fastest, four y at a time.  With SYM a row's
// value is the projection spectrum of sysmat, formed from F at q and at -q:
// the strength conj(a) 2 P / N = (F(q) / 2 + 2 conj(a)^2 conj F(-q)) / N.  With
// HALF the source holds P of the first half of the rows (Lattice::half).
//
// Every projection passes through the origin, so the tiles there meet many
// times the average of about 200 rows (all angles x 8 rows), and the walk over
// a tile's rows is serial in its CTA.  The rows of a tile are therefore cut into
// segments (k_tile_items, once per lattice); tiles of one segment are stored,
// the others zeroed first and added to with vector atomics.
// Measured (before: one CTA per tile, 256 threads of one column, tiles in row
// order): 60 x 154^2 rows 186 -> 31 us, 2 x 91 x 309^2 (SYM) 1090 -> 340 us,
// 361 x 1233^2 8.1 -> 6.9 ms.
constexpr int kCols = 2;   // columns per thread
constexpr int kAhead = 4;  // rows in flight per thread
template <int W, int SRC>
__global__ void __launch_bounds__(128, 4) k_rows_spread(const int *__restrict__ nitem, const int2 *__restrict__ items,
                                                     int seg, const uint32_t *__restrict__ start,
                                                     const int4 *__restrict__ pt, const float2 *__restrict__ pd, int nstart,
                                                     int nT, int ntile, int nf2,
                                                     const float2 *src, int nr, int nc, int kfirst, int ncols, float beta,
                                                     const float2 *__restrict__ beam, int np, bool half, float scale,
                                                     float2 *__restrict__ Gt) {
    constexpr bool SYM = SRC == NufftPlan::ROWS_SYSMAT, HALF = SRC == NufftPlan::ROWS_HALF;
    extern __shared__ __align__(16) unsigned char rsm[];
    const int cap = blockDim.x;  // rows listed at a time
    float4 *lw = reinterpret_cast<float4 *>(rsm);            // [row][kCell] weights, T by y
    uint2 *lr = reinterpret_cast<uint2 *>(lw + (cap + 2 * kAhead) * kCell);  // row's first value, mirrored row's last
    float4 *lb = reinterpret_cast<float4 *>(lr + cap + 2 * kAhead);          // factors of the row's value
    constexpr int NR = W + kCell - 1;
    __shared__ int beg[NR], pre[NR + 1];
    allow_next();
    if ((int)blockIdx.x >= __ldg(nitem)) return;
    const int2 item = __ldg(items + blockIdx.x);
    const int tid = threadIdx.x, ty = item.x / ntile;
    const int c1 = (item.x - ty * ntile) * kCell, c2 = ty * kCell;
    const int first = item.y & 0x7fffffff;
    const bool shared_tile = item.y < 0;
    const int k0 = blockIdx.y * kCols * blockDim.x + tid;
    int kc[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) kc[c] = min(k0 + c * (int)blockDim.x, nc - 1);
    if (tid < NR) {
        const int2 r = tile_run<W>(start, nstart, nf2, c1, c2, tid);
        beg[tid] = r.x;
        pre[tid + 1] = r.y;
    }
    __syncthreads();
    if (tid == 0) {
        pre[0] = 0;
        for (int r = 0; r < NR; ++r) pre[r + 1] += pre[r];
    }
    __syncthreads();
    const int total = min(pre[NR], first + seg);
    float2 re[kCols][kCell][2], im[kCols][kCell][2];
#pragma unroll
    for (int c = 0; c < kCols; ++c)
#pragma unroll
        for (int i = 0; i < kCell; ++i) re[c][i][0] = re[c][i][1] = im[c][i][0] = im[c][i][1] = make_float2(0.f, 0.f);
    for (int base = first; base < total; base += cap) {
        const int n = min(cap, total - base);
        // the last row is listed again, with weights of zero, up to 2 kAhead times:
        // the loop below takes kAhead rows at a time and fetches as many beyond
        for (int e = tid; e < n + 2 * kAhead; e += cap) {
            const int q = min(e, n - 1);
            int r = 0;
            while (base + q >= pre[r + 1]) ++r;
            const int at = beg[r] + base + q - pre[r];
            const int4 I = pt[at];
            const float2 d = pd[at];
            const float on = e < n ? 1.f : 0.f;
            float u[kCell];
#pragma unroll
            for (int i = 0; i < kCell; ++i) u[i] = on * es_tap<W>(d.y, i + W - 1 - r, beta);
#pragma unroll
            for (int i = 0; i < kCell; ++i) {
                const float s = es_tap<W>(d.x, c1 + i - I.y, beta);
                lw[e * kCell + i] = make_float4(s * u[0], s * u[1], s * u[2], s * u[3]);
            }
            const int p = I.w / nr, j = I.w - p * nr;
            const uint32_t mirror = (uint32_t)(half ? half_row(p, nr - 1 - j, np, nr) : p * nr + nr - 1 - j) * ncols + ncols - 1 - kfirst;
            lr[e] = make_uint2((uint32_t)I.x * ncols + kfirst, mirror);
            if (SYM) {  // conj(a)^2 = (ax^2 - ay^2) - 2 i ax ay
                const float2 a = beam[p];
                lb[e] = make_float4(2 * scale * (a.x * a.x - a.y * a.y), -4 * scale * a.x * a.y, 0.f, 0.f);
            }
            if (HALF) {  // conj(a) v, or conj(a) conj(v) of the mirrored value for a second-half row
                const float2 a = beam[p];
                const bool second = j >= (nr + 1) / 2;
                lb[e] = second ? make_float4(a.x, -a.y, -a.y, -a.x) : make_float4(a.x, a.y, -a.y, a.x);
                if (second) lr[e].x = mirror | 0x80000000u;
            }
        }
        __syncthreads();
        if (base == first) wait_previous();  // the lattice's tables are older than the kernel before
        // values of the next kAhead rows are in flight while a row is added
        float2 v[kAhead][kCols], m[kAhead][kCols];
        auto fetch = [&](int q, float2 (&a)[kCols], float2 (&b)[kCols]) {
            const uint2 row = lr[q];
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                if (HALF) a[c] = src[(int64_t)(row.x & 0x7fffffffu) + ((int)row.x < 0 ? -kc[c] : kc[c])];
                else a[c] = src[(int64_t)row.x + kc[c]];
                if (SYM) b[c] = src[(int64_t)row.y - kc[c]];
            }
        };
#pragma unroll
        for (int u = 0; u < kAhead; ++u) fetch(u, v[u], m[u]);
        for (int q0 = 0; q0 < n; q0 += kAhead) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) {
                const int q = q0 + u;
                float2 x[kCols];
#pragma unroll
                for (int c = 0; c < kCols; ++c) {
                    x[c] = v[u][c];
                    if (HALF) {
                        const float4 b = lb[q];
                        x[c] = make_float2(b.x * x[c].x + b.y * x[c].y, b.z * x[c].x + b.w * x[c].y);
                    }
                    if (SYM) {
                        const float4 b = lb[q];
                        x[c] = make_float2(fmaf(b.x, m[u][c].x, fmaf(b.y, m[u][c].y, 0.5f * scale * x[c].x)),
                                           fmaf(b.y, m[u][c].x, fmaf(-b.x, m[u][c].y, 0.5f * scale * x[c].y)));
                    }
                }
                fetch(q + kAhead, v[u], m[u]);
#pragma unroll
                for (int i = 0; i < kCell; ++i) {
                    const float4 t = lw[q * kCell + i];
#pragma unroll
                    for (int c = 0; c < kCols; ++c) {
                        const float2 vr = make_float2(x[c].x, x[c].x), vi = make_float2(x[c].y, x[c].y);
                        re[c][i][0] = __ffma2_rn(make_float2(t.x, t.y), vr, re[c][i][0]);
                        re[c][i][1] = __ffma2_rn(make_float2(t.z, t.w), vr, re[c][i][1]);
                        im[c][i][0] = __ffma2_rn(make_float2(t.x, t.y), vi, im[c][i][0]);
                        im[c][i][1] = __ffma2_rn(make_float2(t.z, t.w), vi, im[c][i][1]);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (total <= first) wait_previous();
#pragma unroll
    for (int c = 0; c < kCols; ++c) {
        const int k = k0 + c * (int)blockDim.x;
        if (k >= nc) break;
#pragma unroll
        for (int i = 0; i < kCell; ++i) {
            if (c1 + i >= nT) break;
            float4 *o = reinterpret_cast<float4 *>(Gt + ((int64_t)(c1 + i) * nc + k) * nf2 + c2);
            const float2(&r)[2] = re[c][i], (&m)[2] = im[c][i];
            const float4 v0 = make_float4(r[0].x, m[0].x, r[0].y, m[0].y);  // nf2 is even: pairs are whole
            const float4 v1 = make_float4(r[1].x, m[1].x, r[1].y, m[1].y);
            if (shared_tile) {
                atomicAdd(o, v0);
                if (c2 + 2 < nf2) atomicAdd(o + 1, v1);
            } else {
                o[0] = v0;
                if (c2 + 2 < nf2) o[1] = v1;
            }
        }
    }
}

// ---------------------------------------------------------------------------
// projection space: fftshift2 / ifftshift2, the beam factor and the mirrored
// half of the spectrum, as one factor per detector pixel:
//   proj = scale Re(c a t), spectrum input = proj conj(a t),
//   t(m1, m2) = 2 cos(b1 + b2) e^{i pi (m1 / nr + m2 / nc)}, b from k_lat_tables
// ---------------------------------------------------------------------------

__device__ __forceinline__ float2 twist(float4 r, float4 c, float2 a) {
    const float f = 2.f * (r.x * c.x - r.y * c.y);
    const float tr = r.z * c.z - r.w * c.w, ti = r.z * c.w + r.w * c.z;
    return make_float2(f * (tr * a.x - ti * a.y), f * (tr * a.y + ti * a.x));
}
// one CTA row of blocks per detector row (blockIdx.y = projection * nr + row)
__global__ void __launch_bounds__(256) k_proj_post(const float2 *__restrict__ P, int64_t nrow, int nr, int nc,
                                                   const float4 *__restrict__ trow, const float4 *__restrict__ tcol,
                                                   const float2 *__restrict__ beam, float scale, float *__restrict__ proj) {
    const int e1 = (nr + 1) / 2, e2 = (nc + 1) / 2;
    for (int64_t row = blockIdx.x; row < nrow; row += gridDim.x) {
        const int p = (int)(row / nr), j = (int)(row - (int64_t)p * nr);
        int js = j + e1; if (js >= nr) js -= nr;
        const float2 a = __ldg(beam + p);
        const float4 tr = __ldg(trow + js);
        const float2 *src = P + ((int64_t)p * nr + js) * nc;
        for (int k = threadIdx.x; k < nc; k += blockDim.x) {
            int ks = k + e2; if (ks >= nc) ks -= nc;
            const float2 t = twist(tr, __ldg(tcol + ks), a), c = src[ks];
            proj[row * nc + k] = (c.x * t.x - c.y * t.y) * scale;
        }
    }
}
__global__ void __launch_bounds__(256) k_proj_pre(const float *__restrict__ proj, int64_t nrow, int nr, int nc,
                                                  const float4 *__restrict__ trow, const float4 *__restrict__ tcol,
                                                  const float2 *__restrict__ beam, float2 *__restrict__ P) {
    const int d1 = nr / 2, d2 = nc / 2;
    for (int64_t row = blockIdx.x; row < nrow; row += gridDim.x) {
        const int p = (int)(row / nr), j = (int)(row - (int64_t)p * nr);
        int js = j + d1; if (js >= nr) js -= nr;
        const float2 a = __ldg(beam + p);
        const float4 tr = __ldg(trow + j);
        const float *src = proj + ((int64_t)p * nr + js) * nc;
        for (int k = threadIdx.x; k < nc; k += blockDim.x) {
            int ks = k + d2; if (ks >= nc) ks -= nc;
            const float2 t = twist(tr, __ldg(tcol + k), a);
            const float v = src[ks];
            P[row * nc + k] = make_float2(v * t.x, -v * t.y);
        }
    }
}

// The same with half the transforms (Lattice::half).  With the phases e^{-i pi m / n}
// of a half-sample frequency offset, P(j, k) is the transform of a real array g, so
// P(nr-1-j, nc-1-k) = conj P(j, k): along the rows' index two real columns are
// transformed as one complex one, the half j < jh of the rows is separated from the
// pairs, and only those rows are transformed along the columns.
// g = 2 cos(b1 + b2) proj.  Pairs are stored z[projection, pair][m1], so that both
// transforms are of contiguous data (the library's strided one took 1.5 times as
// long); the kernels between transpose 32 x 32 tiles through shared memory.
__device__ __forceinline__ float2 cmul(float2 a, float cr, float ci) {
    return make_float2(a.x * cr - a.y * ci, a.x * ci + a.y * cr);
}
// CTA -> projection, first row and first pair of its tile
__device__ __forceinline__ void half_tile(int rows, int nch, int64_t t, int &p, int &r0, int &c0) {
    const int tc = (nch + 31) / 32, tr = (rows + 31) / 32;
    const int64_t q = t / tc;
    c0 = (int)(t - q * tc) * 32;
    p = (int)(q / tr);
    r0 = (int)(q - (int64_t)p * tr) * 32;
}
__global__ void __launch_bounds__(256) k_half_pre(const float *__restrict__ proj, int nr, int nc,
                                                  const float4 *__restrict__ trow, const float4 *__restrict__ tcol,
                                                  float2 *__restrict__ z) {
    __shared__ float2 tile[32][33];
    const int d1 = nr / 2, d2 = nc / 2, nch = (nc + 1) / 2;
    int p, r0, c0;
    half_tile(nr, nch, blockIdx.x, p, r0, c0);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c = c0 + tx;
    if (c < nch)
        for (int r = ty; r < 32 && r0 + r < nr; r += 8) {
            const int m1 = r0 + r;
            int js = m1 + d1; if (js >= nr) js -= nr;
            const float4 tr = __ldg(trow + m1);
            const float *src = proj + ((int64_t)p * nr + js) * nc;
            float f[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m2 = 2 * c + h;
                int ks = m2 + d2; if (ks >= nc) ks -= nc;
                const float4 tc = __ldg(tcol + min(m2, nc - 1));
                f[h] = m2 < nc ? src[ks] * 2.f * (tr.x * tc.x - tr.y * tc.y) : 0.f;
            }
            tile[r][tx] = cmul(make_float2(f[0], f[1]), tr.z, -tr.w);
        }
    __syncthreads();
    const int m1 = r0 + tx;
    if (m1 < nr)
        for (int q = ty; q < 32 && c0 + q < nch; q += 8) z[((int64_t)p * nch + c0 + q) * nr + m1] = tile[tx][q];
}
__global__ void __launch_bounds__(256) k_half_unpack(const float2 *__restrict__ z, int nr, int nc,
                                                     const float4 *__restrict__ tcol, float2 *__restrict__ S) {
    __shared__ float2 tile[2][32][33];
    const int nch = (nc + 1) / 2, jh = (nr + 1) / 2;
    int p, r0, c0;
    half_tile(jh, nch, blockIdx.x, p, r0, c0);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (r0 + tx < jh)
        for (int q = ty; q < 32 && c0 + q < nch; q += 8) {
            const float2 *row = z + ((int64_t)p * nch + c0 + q) * nr;
            tile[0][q][tx] = row[r0 + tx];
            tile[1][q][tx] = row[nr - 1 - r0 - tx];
        }
    __syncthreads();
    const int c = c0 + tx;
    if (c >= nch) return;
    const float4 t0 = __ldg(tcol + 2 * c), t1 = __ldg(tcol + min(2 * c + 1, nc - 1));
    for (int r = ty; r < 32 && r0 + r < jh; r += 8) {
        const float2 a = tile[0][tx][r], b = tile[1][tx][r];
        float2 *o = S + ((int64_t)p * jh + r0 + r) * nc + 2 * c;
        o[0] = cmul(make_float2(0.5f * (a.x + b.x), 0.5f * (a.y - b.y)), t0.z, -t0.w);
        if (2 * c + 1 < nc) o[1] = cmul(make_float2(0.5f * (a.y + b.y), -0.5f * (a.x - b.x)), t1.z, -t1.w);
    }
}
// first-half rows P = a F(j, k) + conj(a F(nr-1-j, nc-1-k)), in place: a thread takes
// columns k and nc-1-k of a row, the only ones that read what it overwrites
__global__ void __launch_bounds__(256) k_half_combine(float2 *__restrict__ F, int np, int nr, int nc,
                                                      const float2 *__restrict__ beam) {
    const int jh = (nr + 1) / 2;
    for (int64_t row = blockIdx.x; row < (int64_t)np * jh; row += gridDim.x) {
        const int p = (int)(row / jh), j = (int)(row - (int64_t)p * jh);
        const float2 a = __ldg(beam + p);
        float2 *f = F + row * nc;
        const float2 *m = F + half_row(p, nr - 1 - j, np, nr) * nc;
        for (int k = threadIdx.x; k < (nc + 1) / 2; k += blockDim.x) {
            const int k2 = nc - 1 - k;
            const float2 u = cmul(f[k], a.x, a.y), u2 = cmul(f[k2], a.x, a.y), v = cmul(m[k], a.x, a.y),
                         v2 = cmul(m[k2], a.x, a.y);
            f[k] = make_float2(u.x + v2.x, u.y - v2.y);
            f[k2] = make_float2(u2.x + v.x, u2.y - v.y);
        }
    }
}
__global__ void __launch_bounds__(256) k_half_pack(const float2 *__restrict__ S, int nr, int nc,
                                                   const float4 *__restrict__ tcol, float2 *__restrict__ z) {
    __shared__ float2 tile[2][32][33];
    const int nch = (nc + 1) / 2, jh = (nr + 1) / 2;
    int p, r0, c0;
    half_tile(jh, nch, blockIdx.x, p, r0, c0);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int c = c0 + tx;
    if (c < nch) {
        const float4 t0 = __ldg(tcol + 2 * c), t1 = __ldg(tcol + min(2 * c + 1, nc - 1));
        for (int r = ty; r < 32 && r0 + r < jh; r += 8) {
            const float2 *s = S + ((int64_t)p * jh + r0 + r) * nc + 2 * c;
            const float2 a = cmul(s[0], t0.z, t0.w);
            const float2 b = 2 * c + 1 < nc ? cmul(s[1], t1.z, t1.w) : make_float2(0.f, 0.f);
            tile[0][r][tx] = make_float2(a.x - b.y, a.y + b.x);  // a + i b
            tile[1][r][tx] = make_float2(a.x + b.y, b.x - a.y);  // conj a + i conj b
        }
    }
    __syncthreads();
    const int j = r0 + tx;
    if (j < jh)
        for (int q = ty; q < 32 && c0 + q < nch; q += 8) {
            float2 *row = z + ((int64_t)p * nch + c0 + q) * nr;
            row[j] = tile[0][tx][q];
            if (nr - 1 - j != j) row[nr - 1 - j] = tile[1][tx][q];
        }
}
__global__ void __launch_bounds__(256) k_half_post(const float2 *__restrict__ z, int nr, int nc,
                                                   const float4 *__restrict__ trow, const float4 *__restrict__ tcol,
                                                   float scale, float *__restrict__ proj) {
    __shared__ float2 tile[32][33];
    const int d1 = nr / 2, d2 = nc / 2, nch = (nc + 1) / 2;
    int p, r0, c0;
    half_tile(nr, nch, blockIdx.x, p, r0, c0);
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    if (r0 + tx < nr) {
        const float4 tr = __ldg(trow + r0 + tx);
        for (int q = ty; q < 32 && c0 + q < nch; q += 8)
            tile[q][tx] = cmul(z[((int64_t)p * nch + c0 + q) * nr + r0 + tx], tr.z, tr.w);
    }
    __syncthreads();
    const int c = c0 + tx;
    if (c >= nch) return;
    for (int r = ty; r < 32 && r0 + r < nr; r += 8) {
        const int m1 = r0 + r;
        int js = m1 + d1; if (js >= nr) js -= nr;
        const float4 tr = __ldg(trow + m1);
        const float2 v = tile[tx][r];
        float *o = proj + ((int64_t)p * nr + js) * nc;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m2 = 2 * c + h;
            if (m2 >= nc) break;
            int ks = m2 + d2; if (ks >= nc) ks -= nc;
            const float4 tc = __ldg(tcol + m2);
            o[ks] = (h ? v.y : v.x) * (tr.x * tc.x - tr.y * tc.y) * scale;
        }
    }
}

// ---------------------------------------------------------------------------
// direct sysmat per point, for calls that may not allocate a lattice: w^3 taps
// per point from the fine grid of W and atomics into the fine grid of U, at q
// and at -q.  The points are the lattice's (the antisymmetric part of the float
// frequencies, products and sums in double), so that the result does not depend on
// whether an earlier call has built one.
// ---------------------------------------------------------------------------

template <int W>
struct Taps {
    float w1[W], w2[W], w3[W];
    int l1, l2, l3;
    __device__ __forceinline__ Taps(const Fine &F, double x, double y, double z) {
        float d1, d2, d3;
        l3 = wrap(es_first<W>(x, F.s3, d3), F.nf3);
        l2 = wrap(es_first<W>(y, F.s2, d2), F.nf2);
        l1 = wrap(es_first<W>(z, F.s1, d1), F.nf1);
#pragma unroll
        for (int t = 0; t < W; ++t) {
            w1[t] = es_weight<W>(d1, t, F.beta);
            w2[t] = es_weight<W>(d2, t, F.beta);
            w3[t] = es_weight<W>(d3, t, F.beta);
        }
    }
    template <class Fn>
    __device__ __forceinline__ void each(const Fine &F, Fn &&fn) const {
        for (int a = 0; a < W; ++a) {
            int i1 = l1 + a; if (i1 >= F.nf1) i1 -= F.nf1;
            for (int b = 0; b < W; ++b) {
                int i3 = l3 + b; if (i3 >= F.nf3) i3 -= F.nf3;
                const int64_t row = ((int64_t)i1 * F.nf3 + i3) * F.nf2;
                const float u = w1[a] * w3[b];
#pragma unroll
                for (int c = 0; c < W; ++c) {
                    int i2 = l2 + c; if (i2 >= F.nf2) i2 -= F.nf2;
                    fn(row + i2, u * w2[c]);
                }
            }
        }
    }
};
template <int W>
__global__ void __launch_bounds__(256) k_sysmat_points(GeomView g, const float2 *__restrict__ G, float2 *__restrict__ H,
                                                       Fine F, float inv_scale) {
    const uint32_t plane = (uint32_t)g.nrows * g.ncols, M = (uint32_t)g.nproj * plane;
    for (uint32_t pid = blockIdx.x * blockDim.x + threadIdx.x; pid < M; pid += gridDim.x * blockDim.x) {
        const int p = (int)(pid / plane);
        const uint32_t r = pid - (uint32_t)p * plane;
        const int j = (int)(r / (uint32_t)g.ncols), k = (int)(r - (uint32_t)j * g.ncols);
        const double X = odd_part(g.qX, k, g.ncols), Y = odd_part(g.qY, j, g.nrows), T = Y * (double)__ldg(g.ct + p);
        const double x = X * g.cg + T * g.sg, y = -Y * (double)__ldg(g.st + p), z = T * g.cg - X * g.sg;
        const float ax = 0.5f * __ldg(g.st + p), ay = -0.5f * __ldg(g.ct + p);
        const Taps<W> tq(F, x, y, z), tm(F, -x, -y, -z);
        float2 f = make_float2(0.f, 0.f), h = f;
        tq.each(F, [&](int64_t i, float u) { const float2 v = __ldg(G + i); f.x = fmaf(u, v.x, f.x); f.y = fmaf(u, v.y, f.y); });
        tm.each(F, [&](int64_t i, float u) { const float2 v = __ldg(G + i); h.x = fmaf(u, v.x, h.x); h.y = fmaf(u, v.y, h.y); });
        // P = a F(q) + conj(a F(-q)); strengths conj(a) P at q, conj(a) conj(P) at -q
        const float pr = (ax * f.x - ay * f.y + ax * h.x - ay * h.y) * inv_scale;
        const float pi = (ax * f.y + ay * f.x - ax * h.y - ay * h.x) * inv_scale;
        const float2 s = make_float2(ax * pr + ay * pi, ax * pi - ay * pr);
        const float2 m = make_float2(ax * pr - ay * pi, -ax * pi - ay * pr);
        tq.each(F, [&](int64_t i, float u) { atomicAdd(H + i, make_float2(u * s.x, u * s.y)); });
        tm.each(F, [&](int64_t i, float u) { atomicAdd(H + i, make_float2(u * m.x, u * m.y)); });
    }
}

// ---------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------

constexpr int64_t kHalfPrime = 13;  // see halved()

// tiles of kCell cells along y that a footprint of w cells meets, at most: one
// that wraps past the end of the fine grid may meet the short last tile besides
static int64_t y_tiles_met(int w, int nf2) {
    int most = (w + kCell - 2) / kCell + 1;
    for (int s = nf2 - w + 1; s < nf2; ++s)  // first cell; last cell s + w - 1 - nf2 (nf2 >= 2 w)
        most = std::max(most, (nf2 - 1) / kCell - s / kCell + 1 + (s + w - 1 - nf2) / kCell + 1);
    return most;
}

static Fine fine_of(const NufftPlan &pl) {
    Fine F;
    F.nf1 = (int)pl.nf1; F.nf2 = (int)pl.nf2; F.nf3 = (int)pl.nf3;
    F.s1 = (double)pl.nf1 / (2 * M_PI);
    F.s2 = (double)pl.nf2 / (2 * M_PI);
    F.s3 = (double)pl.nf3 / (2 * M_PI);
    F.beta = pl.beta;
    return F;
}
static unsigned volume_tiles(const Dims3 &v) { return (unsigned)(v.n1 * ((v.n2 + 31) / 32) * ((v.n3 + 31) / 32)); }
static LatView lat_view(const Lattice &l, const Geom &g, const Fine &F, int64_t first) {
    return LatView{l.X + first, l.cg, l.sg, l.h, (int)std::min<int64_t>(l.ncc, g.ncols - first), l.nT, l.T0, (int)first,
                   (int)g.ncols, 1.0 / F.s1, 1.0 / F.s3, g.ncols * (0.5 / M_PI), 1.0 / l.h};
}
static void check_points(const Geom &g) {
    if (g.npts() > (int64_t)UINT32_MAX / 2) throw Error(ERR_ARG, "too many points in one geometry");
}

// width as a compile-time constant for a generic lambda
template <class Fn>
static void with_width(int w, Fn &&fn) {
    switch (w) {
        case 4: fn(std::integral_constant<int, 4>{}); break;
        case 5: fn(std::integral_constant<int, 5>{}); break;
        case 6: fn(std::integral_constant<int, 6>{}); break;
        case 7: fn(std::integral_constant<int, 7>{}); break;
        case 8: fn(std::integral_constant<int, 8>{}); break;
        default: throw Error(ERR_ARG, "unsupported kernel width");
    }
}

void NufftPlan::pad_real(const float *x3, double sg, double cg, const float *ipT, cudaStream_t s) {
    LAMINO_CUDA(cudaMemsetAsync(grid.p, 0, nf() * sizeof(float2), s));
    const unsigned b = volume_tiles(vol);
    k_pad<false><<<b, 256, 0, s>>>(x3, nullptr, (int)vol.n1, (int)vol.n2, (int)vol.n3, (float)sg, (float)cg, grid.p,
                                   fine_of(*this), ip1.p, ip2.p, ip3.p, ipT);
    LAMINO_LAUNCH("k_pad");
}

void NufftPlan::extract_real(float *y3, double sg, double cg, const float *ipT, float scale, bool accumulate,
                             cudaStream_t s) {
    const unsigned b = volume_tiles(vol);
    k_extract<false><<<b, 256, 0, s>>>(grid.p, (int)vol.n1, (int)vol.n2, (int)vol.n3, (float)sg, (float)cg, y3, nullptr,
                                       fine_of(*this), ip1.p, ip2.p, ip3.p, ipT, scale, accumulate ? 1 : 0);
    LAMINO_LAUNCH("k_extract");
}

static void exec_c2c(const FftPlan &p, float2 *a, int sign, cudaStream_t s) {
    LAMINO_CUFFT(cufftSetStream(p.h, s));
    LAMINO_CUFFT(cufftExecC2C(p.h, (cufftComplex *)a, (cufftComplex *)a, sign < 0 ? CUFFT_FORWARD : CUFFT_INVERSE));
}

void NufftPlan::fft_fine(float2 *g, int sign, cudaStream_t s) {
    if (!split3) {
        exec_c2c(fft3, g, sign, s);
        return;
    }
    const int64_t plane = nf3 * nf2, keep = vol.n1 - vol.n1 / 2;
    if (sign > 0) exec_c2c(fft3n1, g, sign, s);
    exec_c2c(fft3, g, sign, s);
    exec_c2c(fft3, g + (nf1 - keep) * plane, sign, s);
    if (sign < 0) exec_c2c(fft3n1, g, sign, s);
}

// the larger of the primes of n
static int64_t largest_prime(int64_t n) {
    int64_t p = 1;
    for (int64_t q = 2; q * q <= n; ++q)
        while (n % q == 0) {
            p = q;
            n /= q;
        }
    return n > 1 ? std::max(p, n) : p;
}
// Whether a geometry's detector transforms are halved: where a side has a large
// prime the transforms are convolutions of twice the length and bound by
// arithmetic, and half of them pay for the extra pass over memory.  Measured,
// adjoint / forward of 60 projections, 2-D transform against halved: 618^2 2.15 / 2.05
// against 1.48 / 1.44 ms, 724^2 1.96 / 1.91 against 1.42 / 1.46; 433^2 0.94 / 0.84
// against 0.77 / 0.67.  With primes up to 13 only it is within 5 % either way (154^2
// 0.305 / 0.315 against 0.320 / 0.332, 480^2 0.767 / 0.700 against 0.754 / 0.680), and the
// 2-D transform has three launches fewer.
static bool halved(const Geom &g) { return std::max(largest_prime(g.nrows), largest_prime(g.ncols)) > kHalfPrime; }

void NufftPlan::ensure_proj(const Geom &g) {
    check_points(g);
    const bool half = halved(g);
    const int64_t need = half ? g.nproj * ((g.nrows + 1) / 2 * g.ncols + (g.ncols + 1) / 2 * g.nrows) : g.npts();
    if ((int64_t)pbuf.n < need) pbuf.alloc(need);
    if (f2_np != g.nproj || f2_nr != g.nrows || f2_nc != g.ncols) {
        int n[2] = {(int)g.nrows, (int)g.ncols};
        f2_np = -1;
        if (half) {
            const int pairs = (int)(g.nproj * ((g.ncols + 1) / 2));
            fft2.make(1, n + 1, CUFFT_C2C, (int)(g.nproj * ((g.nrows + 1) / 2)));
            fft2n.make(1, n, CUFFT_C2C, pairs);
        } else {
            fft2n.reset();
            fft2.make(2, n, CUFFT_C2C, (int)g.nproj);
        }
        f2_np = g.nproj; f2_nr = g.nrows; f2_nc = g.ncols;
    }
}

static unsigned half_tiles(const Geom &g, int rows) {
    return (unsigned)(g.nproj * ((rows + 31) / 32) * (((g.ncols + 1) / 2 + 31) / 32));
}

// rows (pbuf) -> projections: the beam factors, the detector transform, real part
void NufftPlan::rows_to_proj(const Lattice &l, const Geom &g, float *proj, cudaStream_t s) {
    const int64_t nrow = g.nproj * g.nrows;
    const int nr = (int)g.nrows, nc = (int)g.ncols;
    const float scale = 1.0f / (float)(g.nrows * g.ncols);
    const unsigned grid = (unsigned)std::min<int64_t>(nrow, 148 * 64);
    if (!l.half) {
        exec_c2c(fft2, pbuf.p, +1, s);
        k_proj_post<<<grid, 256, 0, s>>>(pbuf.p, nrow, nr, nc, l.trow, l.tcol, l.a, scale, proj);
        LAMINO_LAUNCH("k_proj_post");
        return;
    }
    const int jh = (nr + 1) / 2, np = (int)g.nproj;
    float2 *z = pbuf.p + (int64_t)np * jh * nc;
    k_half_combine<<<grid, 256, 0, s>>>(pbuf.p, np, nr, nc, l.a);
    LAMINO_LAUNCH("k_half_combine");
    exec_c2c(fft2, pbuf.p, +1, s);
    k_half_pack<<<half_tiles(g, jh), 256, 0, s>>>(pbuf.p, nr, nc, l.tcol, z);
    LAMINO_LAUNCH("k_half_pack");
    exec_c2c(fft2n, z, +1, s);
    k_half_post<<<half_tiles(g, nr), 256, 0, s>>>(z, nr, nc, l.trow, l.tcol, scale, proj);
    LAMINO_LAUNCH("k_half_post");
}

// projections -> rows (pbuf), the transpose
void NufftPlan::proj_to_rows(const Lattice &l, const Geom &g, const float *proj, cudaStream_t s) {
    const int64_t nrow = g.nproj * g.nrows;
    const int nr = (int)g.nrows, nc = (int)g.ncols;
    const unsigned grid = (unsigned)std::min<int64_t>(nrow, 148 * 64);
    if (!l.half) {
        k_proj_pre<<<grid, 256, 0, s>>>(proj, nrow, nr, nc, l.trow, l.tcol, l.a, pbuf.p);
        LAMINO_LAUNCH("k_proj_pre");
        exec_c2c(fft2, pbuf.p, -1, s);
        return;
    }
    const int jh = (nr + 1) / 2, np = (int)g.nproj;
    float2 *z = pbuf.p + (int64_t)np * jh * nc;
    k_half_pre<<<half_tiles(g, nr), 256, 0, s>>>(proj, nr, nc, l.trow, l.tcol, z);
    LAMINO_LAUNCH("k_half_pre");
    exec_c2c(fft2n, z, -1, s);
    k_half_unpack<<<half_tiles(g, jh), 256, 0, s>>>(z, nr, nc, l.tcol, pbuf.p);
    LAMINO_LAUNCH("k_half_unpack");
    exec_c2c(fft2, pbuf.p, -1, s);
}

// Bin layouts were the tiles of a point-by-point spread; the limits on them
// (that kernel's tile, two sets of three components and its staged points, in
// 227 KB of shared memory) still define which layouts the entry point takes.
void NufftPlan::set_bins(int c1, int c2, int c3) {
    if (c1 <= 0 || c2 <= 0 || c3 <= 0) throw Error(ERR_ARG, "bin sizes must be positive");
    if (c1 > 16) throw Error(ERR_ARG, "bin extent along n1 must be at most 16");
    if (c2 > 4095 || c3 > 4095) throw Error(ERR_ARG, "bin extents along n2 and n3 must be below 4096");
    const int64_t cells = (int64_t)(c1 + w - 1) * (c2 + w - 1) * (c3 + w - 1);
    const int64_t rec = (16 * 3 + 24 * w + 4 + 15) / 16 * 16, tables = 4 * (8 * 16 + 17);
    if ((48 * cells + 15) / 16 * 16 + 256 * rec > 227 * 1024 - tables)
        throw Error(ERR_ARG, "bin tile too large for shared memory");
    b1 = c1; b2 = c2; b3 = c3;
}

// exclusive scan of the cell counts (one CTA of 1024 threads, 4096 cells per pass)
__global__ void __launch_bounds__(1024) k_scan_offsets(const uint32_t *__restrict__ cnt, int n,
                                                       uint32_t *__restrict__ start, uint32_t *__restrict__ cursor) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t carry_s;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry_s = 0;
    __syncthreads();
    for (int base = 0; base < n; base += 4096) {
        const int i0 = base + threadIdx.x * 4;
        uint32_t v[4], sum = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = i0 + q < n ? cnt[i0 + q] : 0u;
            sum += v[q];
        }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[wid] = x;
        __syncthreads();
        if (wid == 0) {
            uint32_t w = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            wsum[lane] = w;
        }
        __syncthreads();
        uint32_t e = carry_s + (wid ? wsum[wid - 1] : 0u) + x - sum;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (i0 + q < n) {
                start[i0 + q] = e;
                cursor[i0 + q] = e;
            }
            e += v[q];
        }
        __syncthreads();
        if (threadIdx.x == 0) carry_s += wsum[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) start[n] = carry_s;
}

const Lattice *NufftPlan::find_lattice(const Geom &g, bool raw) const {
    for (const auto &l : lats)
        if (l->uid == g.uid && l->raw == raw) return l.get();
    return nullptr;
}

void NufftPlan::need_work(int64_t n) {
    if ((int64_t)work.n >= n) return;
    const size_t had = std::max<size_t>(work.n, (size_t)(nf() + nf() / 4));
    try {
        work.alloc((size_t)n);
    } catch (...) {  // the other geometries still work with what there was
        try {
            work.alloc(had);
        } catch (const Error &) {
        }
        throw;
    }
}

const Lattice &NufftPlan::lattice(const Geom &g, bool raw, cudaStream_t s) {
    for (auto &l : lats)
        if (l->uid == g.uid && l->raw == raw) {
            need_work(node_values(*l));
            l->last_use = ++use_clock;
            return *l;
        }
    check_points(g);
    if (lats.size() >= keep_lattices) {
        size_t lru = 0;
        for (size_t i = 1; i < lats.size(); ++i)
            if (lats[i]->last_use < lats[lru]->last_use) lru = i;
        lats.erase(lats.begin() + (long)lru);
    }
    auto l = std::make_unique<Lattice>();
    l->uid = g.uid;
    l->raw = raw;
    l->half = !raw && halved(g);
    l->cg = g.cg;
    l->sg = g.sg;
    // twice the volume's extent along t, in cells over the period 2 pi
    const double band = vol.n3 * std::fabs(l->sg) + vol.n1 * std::fabs(l->cg);
    int nTf = band > w ? 2 * (int)std::ceil(band - 1e-9) : 2 * w;  // (also for a NaN tilt)
    // and no T line more than one cell of the fine grid from the next (k_nodes_gather).
    // Lines exactly one cell apart (no tilt, or a quarter turn) lie at the cells: the
    // footprints of odd widths then start half a cell from an integer, those of even widths
    // at an integer up to rounding, which puts some lines' first taps two cells
    // apart.  Even widths take their lines closer than one cell.
    const double near = std::max(nf1 * std::fabs(l->cg), nf3 * std::fabs(l->sg)) + (w % 2 ? 0 : 1);
    if (near > nTf) nTf = 2 * (int)std::ceil(0.5 * near);
    l->h = 2 * M_PI / nTf;
    // |T| <= pi up to float rounding: footprints start in [-nTf/2 - w/2, nTf/2 - w/2 + 1)
    l->T0 = -nTf / 2 - (w + 1) / 2 - 1;
    l->nT = nTf + w + 4;
    l->nstart = l->nT - w + 1;
    const int64_t np = g.nproj, nrow = np * g.nrows, cells = (int64_t)l->nstart * nf2;
    if (cells > (int64_t)INT32_MAX - 1) throw Error(ERR_ARG, "node grid too large");
    l->ncc = (int)node_columns(l->nT, nf2, g.ncols);
    // Segments of k_rows_spread: 256 rows, fewer where that would leave less than
    // about 16 CTAs per SM (a row meets 6 to 9 tiles).
    l->ntile = (l->nT + kCell - 1) / kCell;
    const int64_t ntiles = (int64_t)l->ntile * ((nf2 + kCell - 1) / kCell);
    l->seg = (int)std::min<int64_t>(256, std::max<int64_t>(32, nrow * 6 * ((g.ncols + 255) / 256) / (148 * 16) / 32 * 32));
    const int64_t meet = (w + kCell - 2) / kCell + 1;  // tiles a footprint meets along T, at most
    const int64_t max_items = ntiles + nrow * meet * y_tiles_met(w, (int)nf2) / l->seg + 1;
    l->max_items = (int)max_items;
    // one allocation for all tables
    size_t bytes = 0;
    auto room = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t oX = room(g.ncols * sizeof(double)), oa = room(np * sizeof(float2)), otr = room(g.nrows * sizeof(float4)),
                 otc = room(g.ncols * sizeof(float4)), oip = room(vol.n1 * vol.n3 * sizeof(float)),
                 opt = room(nrow * sizeof(int4)), opd = room(nrow * sizeof(float2)),
                 ost = room((cells + 1) * sizeof(uint32_t)), ocnt = room(cells * sizeof(uint32_t)),
                 oni = room(sizeof(int)), oit = room(l->max_items * sizeof(int2));
    l->mem.alloc(bytes);
    char *m0 = l->mem.p;
    l->X = reinterpret_cast<double *>(m0 + oX);
    l->a = reinterpret_cast<float2 *>(m0 + oa);
    l->trow = reinterpret_cast<float4 *>(m0 + otr);
    l->tcol = reinterpret_cast<float4 *>(m0 + otc);
    l->ipT = reinterpret_cast<float *>(m0 + oip);
    l->pt = reinterpret_cast<int4 *>(m0 + opt);
    l->pd = reinterpret_cast<float2 *>(m0 + opd);
    l->start = reinterpret_cast<uint32_t *>(m0 + ost);
    l->nitem = reinterpret_cast<int *>(m0 + oni);
    l->items = reinterpret_cast<int2 *>(m0 + oit);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(m0 + ocnt);  // counts, then placement cursors
    need_work(node_values(*l));
    LAMINO_CUDA(cudaMemsetAsync(cnt, 0, (size_t)(reinterpret_cast<char *>(l->items) - reinterpret_cast<char *>(cnt)), s));
    const Fine F = fine_of(*this);
    const GeomView gv = g.view();
    const int64_t m = std::max(std::max(g.ncols, g.nrows), np);
    k_lat_tables<<<(unsigned)((m + 127) / 128), 128, 0, s>>>(gv, raw, g.offX, g.offY, l->X, l->a, l->trow, l->tcol);
    LAMINO_LAUNCH("k_lat_tables");
    const int64_t modes = vol.n1 * vol.n3;
    k_lat_deconv<<<(unsigned)((modes + 127) / 128), 128, 0, s>>>(quad.p, (int)vol.n1, (int)vol.n3, l->sg, l->cg, w, nTf,
                                                                 l->ipT);
    LAMINO_LAUNCH("k_lat_deconv");
    const double invh = nTf / (2 * M_PI);
    const unsigned grid_n = grid_for(nrow, 256);
    with_width(w, [&](auto WC) {
        constexpr int W = decltype(WC)::value;
        k_rows_count<W><<<grid_n, 256, 0, s>>>(gv, raw, invh, l->T0, l->nstart, F, cnt);
        LAMINO_LAUNCH("k_rows_count");
        k_scan_offsets<<<1, 1024, 0, s>>>(cnt, (int)cells, l->start, cnt);
        LAMINO_LAUNCH("k_scan_offsets");
        k_rows_place<W><<<grid_n, 256, 0, s>>>(gv, raw, invh, l->half, l->T0, l->nstart, F, cnt, l->pt, l->pd);
        LAMINO_LAUNCH("k_rows_place");
        k_tile_items<W><<<(unsigned)((strip_count(l->ntile, ntiles / l->ntile) + 127) / 128), 128, 0, s>>>(l->start, l->nstart, (int)nf2, l->ntile, (int)ntiles,
                                                                         l->seg, l->nitem, l->items);
        LAMINO_LAUNCH("k_tile_items");
    });
    l->last_use = ++use_clock;
    lats.push_back(std::move(l));
    return *lats.back();
}

void NufftPlan::nodes_to_rows(const Lattice &l, const Geom &g, float2 *rows, cudaStream_t s) {
    const Fine F = fine_of(*this);
    const int pitch = (int)node_pitch(l.ncc);
    // The box of cells under a tile of nodes, one cell of slack on either side, for
    // 16 x 8 and 8 x 16 tiles (columns are 1.2 to 2 cells apart, T lines 0.7 to 1):
    // the smaller box is staged, with 16 y where two CTAs then fit an SM, else with
    // fewer.
    auto box_cells = [&](int K) {
        const double ek = (double)(std::min<int64_t>(K, g.ncols) - 1) * 2 * M_PI / g.ncols, et = (kNodes / K - 1) * l.h;
        return std::ceil(F.s1 * (ek * std::fabs(l.sg) + et * std::fabs(l.cg)) + w + 3) *
               std::ceil(F.s3 * (ek * std::fabs(l.cg) + et * std::fabs(l.sg)) + w + 3);
    };
    const int K = box_cells(16) <= box_cells(8) ? 16 : 8;
    const double cells = box_cells(K);
    constexpr double kBoxBytes = 100 * 1024;
    // y in even chunks of at most 16; small node grids spread the chunks over CTAs
    int nchunk = (int)((nf2 + kNodeY - 1) / kNodeY), ychunk = (int)((nf2 + nchunk - 1) / nchunk + 1) / 2 * 2;
    if (cells * 4 * sizeof(float2) <= kBoxBytes)
        while (cells * ychunk * sizeof(float2) > kBoxBytes) ychunk -= 2;
    nchunk = (int)((nf2 + ychunk - 1) / ychunk);
    const int boxcap = cells * ychunk * sizeof(float2) <= kBoxBytes ? (int)cells : 0;
    const int smem = (int)(std::max(boxcap, kNodes + 1) * ychunk * sizeof(float2));
    const int ktiles = (l.ncc + K - 1) / K;
    dim3 b1((unsigned)(ktiles * ((l.nT + kNodes / K - 1) / (kNodes / K))));
    b1.y = (unsigned)std::min<int64_t>(nchunk, std::max<int64_t>(1, 148LL * 12 / b1.x));
    const uint32_t ydiv = (uint32_t)((0x100000000ULL + ychunk / 2 - 1) / (ychunk / 2));
    const int64_t nrow = g.nproj * g.nrows;
    const int groups = (int)((nrow + kRowGroup - 1) / kRowGroup);
    with_width(w, [&](auto WC) {
        constexpr int W = decltype(WC)::value;
        auto ng = K == 16 ? k_nodes_gather<W, 16> : k_nodes_gather<W, 8>;
        raise_smem_limit((const void *)ng, smem);
        for (int64_t k0 = 0; k0 < g.ncols; k0 += l.ncc) {
            const LatView L = lat_view(l, g, F, k0);
            ng<<<b1, 256, smem, s>>>(L, F, grid.p, work.p, pitch, ktiles, ychunk, ydiv, nchunk, boxcap);
            LAMINO_LAUNCH("k_nodes_gather");
            k_rows_gather<W><<<(unsigned)groups * ((L.nc + 63) / 64), 256, 0, s>>>(
                l.pt, l.pd, (int)nrow, work.p, (int)nf2, pitch, L.nc, L.ncols, groups, beta, rows + k0);
            LAMINO_LAUNCH("k_rows_gather");
        }
    });
}

void NufftPlan::rows_to_nodes(const Lattice &l, const Geom &g, const float2 *rows, RowSource from, cudaStream_t s) {
    const Fine F = fine_of(*this);
    const int nc = l.ncc;
    // 32 to 128 threads of two columns each: the width that pads the columns least
    int bt = 128;
    for (int b : {96, 64, 32})
        if ((nc + kCols * b - 1) / (kCols * b) * b < (nc + kCols * bt - 1) / (kCols * bt) * bt) bt = b;
    const dim3 b1((unsigned)l.max_items, (unsigned)((nc + kCols * bt - 1) / (kCols * bt)));
    const int smem1 = (bt + 2 * kAhead) * (int)(kCell * sizeof(float4) + sizeof(uint2) + sizeof(float4));
    const int yb = (int)std::min<int64_t>(256, (nf2 + 31) / 32 * 32);
    const int xtiles = (int)((nf3 + kCell - 1) / kCell);
    const dim3 b2((unsigned)strip_count(xtiles, (nf1 + kCell - 1) / kCell), (unsigned)((nf2 + yb - 1) / yb));
    // largest |footprint cell| of the nodes along z and x (a NaN tilt has none)
    const double Tmax = std::max(-l.T0, l.T0 + l.nT) * l.h;
    auto reach = [&](double c, double t, double sc) {
        const double r = sc * (3.1416 * std::fabs(c) + Tmax * std::fabs(t)) + w + 1;
        return r < 1e9 ? (int)r : 0;
    };
    const int reach1 = reach(l.sg, l.cg, F.s1), reach3 = reach(l.cg, l.sg, F.s3);
    const int smem2 = 2 * yb * (int)(kCell * sizeof(float4) + sizeof(int));
    const float scale = 1.0f / (float)(g.nrows * g.ncols);
    with_width(w, [&](auto WC) {
        constexpr int W = decltype(WC)::value;
        auto rs = from == ROWS_SYSMAT ? k_rows_spread<W, ROWS_SYSMAT>
                  : from == ROWS_HALF ? k_rows_spread<W, ROWS_HALF> : k_rows_spread<W, ROWS_PLAIN>;
        for (int64_t k0 = 0; k0 < g.ncols; k0 += l.ncc) {
            const LatView L = lat_view(l, g, F, k0);
            k_tiles_zero<<<(unsigned)std::min(l.max_items, 148 * 8), 256, 0, s>>>(l.nitem, l.items, l.nT, l.ntile, (int)nf2,
                                                                                  L.nc, work.p);
            LAMINO_LAUNCH("k_tiles_zero");
            launch_after(rs, b1, bt, smem1, s, l.nitem, l.items, l.seg, l.start, l.pt, l.pd, l.nstart, l.nT, l.ntile,
                         (int)nf2, rows, (int)g.nrows, L.nc, L.first, L.ncols, beta, l.a, (int)g.nproj, l.half, scale,
                         work.p);
            LAMINO_LAUNCH("k_rows_spread");
            launch_after(k_nodes_spread<W>, b2, yb, smem2, s, L, F, reach1, reach3, xtiles, work.p, grid.p);
            LAMINO_LAUNCH("k_nodes_spread");
        }
    });
}

namespace {
std::mutex g_bins_mu;
std::map<std::array<int64_t, 6>, std::array<int, 3>> g_bins_cache;

__global__ void k_fill(float *__restrict__ a, int64_t n, float v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        a[i] = v;
}
}  // namespace

double NufftPlan::autotune_bins(const std::vector<const Geom *> &gs, int objective, cudaStream_t s) {
    if (gs.empty()) throw Error(ERR_ARG, "autotune needs at least one geometry");
    if (objective != 0 && objective != 1) throw Error(ERR_ARG, "objective must be 0 (adjoint) or 1 (normal)");
    int64_t pts = 0;
    for (const Geom *g : gs) pts += g->npts();
    const std::array<int64_t, 6> key{nf1, nf2, nf3, (int64_t)w, (int64_t)objective, pts};
    {
        std::lock_guard<std::mutex> lk(g_bins_mu);
        auto it = g_bins_cache.find(key);
        if (it != g_bins_cache.end()) {
            b1 = it->second[0]; b2 = it->second[1]; b3 = it->second[2];
            return 0.0;
        }
    }
    const int64_t nv = 3 * vol.size();
    DevBuf<float> x((size_t)nv), y((size_t)nv), proj;
    k_fill<<<grid_for(nv, 256), 256, 0, s>>>(x.p, nv, 1.0f);
    LAMINO_LAUNCH("k_fill");
    if (objective == 0) {
        proj.alloc((size_t)gs[0]->npts());
        k_fill<<<grid_for(gs[0]->npts(), 256), 256, 0, s>>>(proj.p, gs[0]->npts(), 1.0f);
        LAMINO_LAUNCH("k_fill");
    }
    if (objective == 1) normal(gs, x.p, y.p, s);  // builds the lattices
    cudaEvent_t e0, e1;
    LAMINO_CUDA(cudaEventCreate(&e0));
    LAMINO_CUDA(cudaEventCreate(&e1));
    float ms = 0.f;
    LAMINO_CUDA(cudaEventRecord(e0, s));
    if (objective == 0) adjoint(*gs[0], proj.p, y.p, false, s);
    else normal(gs, x.p, y.p, s);
    LAMINO_CUDA(cudaEventRecord(e1, s));
    LAMINO_CUDA(cudaEventSynchronize(e1));
    LAMINO_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    std::lock_guard<std::mutex> lk(g_bins_mu);
    g_bins_cache[key] = {b1, b2, b3};
    return ms;
}

void NufftPlan::forward(const Geom &g, const float *m3, float *proj, cudaStream_t s) {
    ensure_proj(g);
    const Lattice &l = lattice(g, false, s);
    pad_real(m3, l.sg, l.cg, l.ipT, s);
    fft_fine(grid.p, -1, s);
    nodes_to_rows(l, g, pbuf.p, s);
    rows_to_proj(l, g, proj, s);
}

void NufftPlan::adjoint(const Geom &g, const float *proj, float *m3, bool accumulate, cudaStream_t s) {
    ensure_proj(g);
    const Lattice &l = lattice(g, false, s);
    proj_to_rows(l, g, proj, s);
    rows_to_nodes(l, g, pbuf.p, l.half ? ROWS_HALF : ROWS_PLAIN, s);
    fft_fine(grid.p, +1, s);
    extract_real(m3, l.sg, l.cg, l.ipT, 1.0f / (float)(g.nrows * g.ncols), accumulate, s);
}

// one geometry's sysmat, (+)= into y3: over its lattice, or point by point without one
void NufftPlan::normal_one(const Geom &g, const Lattice *l, const float *x3, float *y3, bool accumulate,
                           cudaStream_t s) {
    const double sg = l ? l->sg : (double)g.sg, cg = l ? l->cg : (double)g.cg;
    const float *ipT = l ? l->ipT : nullptr;
    pad_real(x3, sg, cg, ipT, s);
    fft_fine(grid.p, -1, s);
    if (l) {
        nodes_to_rows(*l, g, pbuf.p, s);
        rows_to_nodes(*l, g, pbuf.p, ROWS_SYSMAT, s);
        fft_fine(grid.p, +1, s);
        extract_real(y3, sg, cg, ipT, 1.0f, accumulate, s);
        return;
    }
    LAMINO_CUDA(cudaMemsetAsync(work.p, 0, nf() * sizeof(float2), s));
    const Fine F = fine_of(*this);
    with_width(w, [&](auto WC) {
        constexpr int W = decltype(WC)::value;
        k_sysmat_points<W><<<grid_for(g.npts(), 256, 148LL * 16 * 8), 256, 0, s>>>(
            g.view(), grid.p, work.p, F, 1.0f / (float)(g.nrows * g.ncols));
        LAMINO_LAUNCH("k_sysmat_points");
    });
    LAMINO_CUDA(cudaMemcpyAsync(grid.p, work.p, nf() * sizeof(float2), cudaMemcpyDeviceToDevice, s));
    fft_fine(grid.p, +1, s);
    extract_real(y3, sg, cg, nullptr, 1.0f, accumulate, s);
}

void NufftPlan::normal(const std::vector<const Geom *> &gs, const float *x3, float *y3, cudaStream_t s) {
    if (gs.empty()) throw Error(ERR_ARG, "normal operator needs at least one geometry");
    for (const Geom *g : gs) {
        if (!g) throw Error(ERR_ARG, "bad geometry");
        check_points(*g);
        if ((int64_t)pbuf.n < g->npts()) pbuf.alloc(g->npts());
    }
    keep_lattices = std::max(keep_lattices, gs.size());
    for (const Geom *g : gs) lattice(*g, false, s);
    for (size_t i = 0; i < gs.size(); ++i) normal_one(*gs[i], &lattice(*gs[i], false, s), x3, y3, i > 0, s);
}

void NufftPlan::normal_ptrs(const Geom *const *gs, int ng, const float *x3, float *y3, cudaStream_t s) {
    if (!gs || ng <= 0) throw Error(ERR_ARG, "normal operator needs at least one geometry");
    for (int i = 0; i < ng; ++i)
        if (!gs[i] || gs[i]->npts() > (int64_t)UINT32_MAX / 2) throw Error(ERR_ARG, "bad geometry");
    for (int i = 0; i < ng; ++i) {
        const Lattice *l = find_lattice(*gs[i], false);
        if (l && ((int64_t)pbuf.n < gs[i]->npts() || (int64_t)work.n < node_values(*l)))
            l = nullptr;  // no row buffer or node grid from an earlier call
        if ((int64_t)work.n < nf()) throw Error(ERR_OOM, "the plan lost its scratch to a failed allocation");
        normal_one(*gs[i], l, x3, y3, i > 0, s);
    }
}

void NufftPlan::type2(const Geom &g, const float2 *modes, float2 *c, cudaStream_t s) {
    const Lattice &l = lattice(g, true, s);
    LAMINO_CUDA(cudaMemsetAsync(grid.p, 0, nf() * sizeof(float2), s));
    const unsigned b = volume_tiles(vol);
    k_pad<true><<<b, 256, 0, s>>>(nullptr, modes, (int)vol.n1, (int)vol.n2, (int)vol.n3, 0.f, 0.f, grid.p, fine_of(*this),
                                  ip1.p, ip2.p, ip3.p, l.ipT);
    LAMINO_LAUNCH("k_pad");
    fft_fine(grid.p, -1, s);
    nodes_to_rows(l, g, c, s);
}

void NufftPlan::type1(const Geom &g, const float2 *c, float2 *modes, cudaStream_t s) {
    const Lattice &l = lattice(g, true, s);
    rows_to_nodes(l, g, c, ROWS_PLAIN, s);
    fft_fine(grid.p, +1, s);
    const unsigned b = volume_tiles(vol);
    k_extract<true><<<b, 256, 0, s>>>(grid.p, (int)vol.n1, (int)vol.n2, (int)vol.n3, 0.f, 0.f, nullptr, modes,
                                      fine_of(*this), ip1.p, ip2.p, ip3.p, l.ipT, 1.0f, 0);
    LAMINO_LAUNCH("k_extract");
}

}  // namespace lamino
