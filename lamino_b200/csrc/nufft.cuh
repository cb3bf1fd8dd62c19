// ES-kernel 3-D NUFFT on the laminography planes (type 1 / type 2), plus the
// projection-space stages of the forward and adjoint operators.
#pragma once

#include <memory>
#include <vector>

#include "common.cuh"
#include "geometry.cuh"

namespace lamino {

// Width / shape of the exponential-of-semicircle kernel for a tolerance at
// oversampling 2 (Barnett, Magland, af Klinteberg, SIAM J. Sci. Comput. 2019).
inline int es_width(double eps) {
    int w = (int)std::ceil(std::log10(10.0 / eps));
    return w < 2 ? 2 : w;
}
int64_t next_smooth_even(int64_t n);

// The points of one geometry as a lattice (see nufft.cu): every point is
// X a(gamma) + (T, y)(theta, Y), X a column frequency, T = Y cos(theta) the
// coordinate along the tilted axis normal to a and y.  The plane of columns and
// T lines is a regular grid of nodes (nT lines, spacing h, first line T0); the
// (T, y) positions of the detector rows are kept sorted by the grid cell their
// kernel footprint starts in.
struct Lattice {
    uint64_t uid = 0;
    bool raw = false;        // the float frequencies as they are (raw transforms), else
                             // their antisymmetric part (forward, adjoint, sysmat)
    uint64_t last_use = 0;
    // The projection spectra of real images are symmetric, so the detector transform
    // needs only the first half of the rows: two real columns travel as one
    // complex one.  Rows are then stored first halves of all projections first,
    // and the second halves are read as mirrored conjugates.
    bool half = false;
    double cg = 1, sg = 0, h = 0;
    int nT = 0, T0 = 0;
    int nstart = 0;          // footprint starts along T: nT - w + 1
    int ncc = 0;             // columns of the node grid at a time
    DevBuf<char> mem;        // holds the tables below
    double *X = nullptr;     // column frequencies
    float *ipT = nullptr;    // 1 / p_T of every mode (k1, k3): deconvolution along T
    float2 *a = nullptr;     // (sin - i cos) / 2 of every angle
    float4 *trow = nullptr, *tcol = nullptr;  // twist factors of the projection-space transform
    int4 *pt = nullptr;      // rows sorted by cell: place among the stored rows, T start, y start, id (angle, row)
    float2 *pd = nullptr;    // offsets of the T and y footprints from the row's position
    uint32_t *start = nullptr;  // first row of each (y start, T start) cell
    int ntile = 0, seg = 0, max_items = 0;  // rows -> nodes: tiles along T, rows per work item, bound on the items
    int *nitem = nullptr;    // number of work items
    int2 *items = nullptr;
};

struct NufftPlan {
    Dims3 vol;                // recon volume (n1, n2, n3), n3 fastest
    int64_t nf1, nf2, nf3;    // fine grid paired with n1 (z), n2 (y), n3 (x)
    int w = 7;
    float beta = 16.1f;
    double eps = 1.2e-6;
    DevBuf<float> ip1, ip2, ip3;   // 1 / p(k) per mode index along each dim
    DevBuf<double2> quad;          // quadrature of the kernel's transform (node, weight x kernel)
    DevBuf<float2> grid;           // fine grid [nf1][nf3][nf2] (n2 fastest)
    DevBuf<float2> work;           // node grid, or the direct form's second fine grid
    FftPlan fft3;                  // C2C 3-D on the fine grid; or, split, its planes of n1 ...
    FftPlan fft3n1;                // ... and the transform along n1
    bool split3 = false;           // only the planes that hold modes run their 2-D transforms
    // projection-space workspace (largest geometry seen), with its 2-D plan
    DevBuf<float2> pbuf;
    FftPlan fft2;                  // 2-D; or, halved (Lattice::half), along the detector rows ...
    FftPlan fft2n;                 // ... and along the columns, two real ones at a time
    int64_t f2_np = -1, f2_nr = -1, f2_nc = -1;
    // lattices of the geometries used with this plan (least recently used goes first)
    std::vector<std::unique_ptr<Lattice>> lats;
    uint64_t use_clock = 0;
    // how many: 16, or the geometries of the largest sum so far.  A sum with more than are
    // kept would build them anew in every call, also in one that is being captured,
    // where their memory would become the graph's.
    size_t keep_lattices = 16;
    int b1 = 4, b2 = 8, b3 = 16;   // bin layout of lamino_plan_set_bins (a hint, see set_bins)

    NufftPlan(Dims3 d, double eps);
    int64_t nf() const { return nf1 * nf2 * nf3; }
    // values of a lattice's node grid, and at least n values in `work`: if there is no
    // memory for them, `work` keeps its size and the error goes on to the caller
    int64_t node_values(const Lattice &l) const { return (int64_t)l.nT * nf2 * node_pitch(l.ncc); }
    void need_work(int64_t n);
    void ensure_proj(const Geom &g);
    // projection space <-> rows (see Lattice::half): proj is read / written
    void rows_to_proj(const Lattice &lat, const Geom &g, float *proj, cudaStream_t s);
    void proj_to_rows(const Lattice &lat, const Geom &g, const float *proj, cudaStream_t s);
    // accepts the layouts that a tile of (b + w - 1)^3 cells in shared memory
    // allows; the lattice transforms choose their own tiles
    void set_bins(int b1, int b2, int b3);
    // the geometry's lattice (built on first use, then cached) with the node grid allocated
    const Lattice &lattice(const Geom &g, bool raw, cudaStream_t s);
    const Lattice *find_lattice(const Geom &g, bool raw) const;
    // one pass of the adjoint (objective 0, with the building of its lattice: a setup
    // pass) or of the sum over the geometries of sysmat (objective 1, without) timed;
    // cached per (fine grid, width, objective, points) for the process.  Returns its
    // time in ms (0 when taken from the cache).
    double autotune_bins(const std::vector<const Geom *> &gs, int objective, cudaStream_t s);

    // --- operators (device pointers; volumes are 3 contiguous components) ---
    // forward projection (src/projection.cpp:42-77)
    void forward(const Geom &g, const float *m3, float *proj, cudaStream_t s);
    // adjoint (src/projection.cpp:90-126); accumulate adds into m3
    void adjoint(const Geom &g, const float *proj, float *m3, bool accumulate, cudaStream_t s);
    // sum over geometries of sysmat (src/gradient.cpp:34-89), NUFFT form
    void normal(const std::vector<const Geom *> &gs, const float *x3, float *y3, cudaStream_t s);
    // same sum over geometries given as a pointer array, without any allocation
    // (geometries whose lattice is not cached take the direct point kernel)
    void normal_ptrs(const Geom *const *gs, int ng, const float *x3, float *y3, cudaStream_t s);
    // raw transforms on one geometry (FINUFFT-level boundary, complex data)
    void type2(const Geom &g, const float2 *modes, float2 *c, cudaStream_t s);
    void type1(const Geom &g, const float2 *c, float2 *modes, cudaStream_t s);

    // internals
    void normal_one(const Geom &g, const Lattice *lat, const float *x3, float *y3, bool accumulate, cudaStream_t s);
    void pad_real(const float *x3, double sg, double cg, const float *ipT, cudaStream_t s);
    void extract_real(float *y3, double sg, double cg, const float *ipT, float scale, bool accumulate, cudaStream_t s);
    void fft_fine(float2 *g, int sign, cudaStream_t s);
    void nodes_to_rows(const Lattice &lat, const Geom &g, float2 *rows, cudaStream_t s);   // grid -> nodes -> rows
    enum RowSource { ROWS_PLAIN, ROWS_SYSMAT, ROWS_HALF };  // see k_rows_spread
    void rows_to_nodes(const Lattice &lat, const Geom &g, const float2 *rows, RowSource from, cudaStream_t s);
    // whole 128-byte lines, so that a run of columns never straddles one
    static int64_t node_pitch(int64_t ncols) { return (ncols + 15) / 16 * 16; }
    // columns of the node grid at a time (Lattice::ncc), and the bytes they take.  A wide
    // detector over a thin volume has far more nodes than fine-grid cells (2400 T
    // lines x 4096 y x 2048 columns for 16 x 2048 x 2048 at 35 degrees: 161 GB), and the
    // columns don't meet before the fine grid.  The largest usual case (721 x 71 x 721, 1233
    // columns) takes 2.9 GB, in one piece.
    static int64_t node_columns(int64_t lines, int64_t nf2, int64_t ncols) {
        constexpr int64_t kBytes = 4LL << 30;
        return std::min(ncols, std::max<int64_t>(64, kBytes / (lines * nf2 * (int64_t)sizeof(float2)) / 64 * 64));
    }
    static int64_t node_bytes(int64_t lines, int64_t nf2, int64_t ncols) {
        return lines * nf2 * node_pitch(node_columns(lines, nf2, ncols)) * (int64_t)sizeof(float2);
    }
};

}  // namespace lamino
