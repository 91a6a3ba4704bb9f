// Node form of the FP32 split-phase sum (sm_103a): tile fields on a few
// Chebyshev nodes of the detector, interpolated to its pixels.
//
// The field of a compact group of atoms relative to its own centre o,
//   F(P) = sum_a E_a exp(2 pi i [w(P, o).D_a + the |d|^2 term]),
// is a smooth function of the pixel position: along one detector axis its
// phase runs over +-phi, phi = k r (half the patch's extent) / |P|, so on
// n Chebyshev nodes per axis it is interpolated with a relative error of at
// most 4 J_n(phi) <= 4 (phi/2)^n / n!. A 512-atom tile (r ~ 2.5 nm) of the
// 8.19M-atom exposure needs 12 nodes per axis for all of its 512 x 512
// pixels: 144 terms an atom instead of 262,144. The steps are
//   leaf    V0[tile][node] = F of every tile on its patch's nodes (the terms
//           of the split kernel, phase and sin/cos in FP32),
//   merge   V1[group][fine node]: the tiles of a group (consecutive on the
//           Hilbert curve) interpolated from the coarse patch's nodes to the
//           nodes of finer patches, each times exp(2 pi i phase of its origin
//           relative to the group's), added; in two steps by way of runs of
//           a few tiles on middle patches where that is cheaper,
//   pixels  every group's field interpolated from the fine patch's nodes to
//           the pixels, times exp(2 pi i phase of the group's origin), added
//           (Kahan), times the species' factor (mk_factor_table); slices of
//           groups are reduced in FP64 in fixed order.
// Tiles wider than the tile radius of the plan skip the merge (their fine
// nodes are evaluated directly), and tiles wider than the group radius are
// left to the split kernel. With no groups every tile goes from the leaf
// straight to the pixels.
//
// A phase q.d (q = k/2pi (b - u), up to 1e4 cycles) is formed in two-float
// FP32 arithmetic (q = qh + ql, d = dh + dl, the product qh dh with its
// rounding error from an FMA), mod 1 per component: good to ~1e-7 cycles at
// 1/20 of the FP64 pipe's cost (2 FP64 operations per clock and SM).
//
// Measured against the split kernel on every (atom, pixel), through the entry
// point: 8.19M atoms x 512^2 354 -> 7.6 ms, 5.3M x 1024^2 at 0.5 m 1042 ->
// 9.6 ms, 2M x 256^2 29.1 -> 5.3 ms, 32k x 128^2 1.43 -> 0.91 ms; a staged scan
// of 16 frames x 500k atoms 103 -> 1.0 ms. Error against FP64 at 64 pixels
// spread over the detector: peak-relative intensity 4 to 6e-7 (split kernel
// 8.5e-7) on the first, 1.6 to 1.8e-6 (1.6 to 2.0e-6) on the second.
//
// Interpolation weights are FP64 Lagrange products rounded once; the pixel
// coordinates they are taken at are the pixels' own (projected on the
// detector's axes), so an uneven pitch is interpolated exactly; a detector
// off its plane or off the (column, row) product grid is not admitted.
#include <vector>

#include "mk_split.cuh"

#define MK_NODE_MAX 20       // nodes per axis at most (fine nodes: 16)
#define MK_NODE_SB(n) ((n) > 16 ? 4 : (n) == 16 ? 6 : 8)   // sources staged per step, within 48 KB
#define MK_MERGE_NT 128      // threads of a merge block
#define MK_PIX_COLS 32       // pixel block: 32 columns x 16 rows, 4 rows a thread
#define MK_PIX_ROWS 16
#define MK_NODE_PAD 0.25     // half pixel pitches the node interval exceeds the pixel centres

// exp(i phase) by __sincosf is 7.3e-8 short of unit length on average (2^24
// phases over a turn, against FP64). A leaf's term, a merged tile and a pixel's
// source each carry one such factor, the same for all, so that without this a
// sum of three or four levels came out 2 to 4e-7 small.
#define MK_SINCOS_SHORT 7.3e-8f
__device__ __forceinline__ float mk_unshort(float v) { return fmaf(v, MK_SINCOS_SHORT, v); }

// Levels of patches: tiles' coarse ones, the middle ones of runs of a few tiles
// (only in plans with two merges), the fine ones of groups. Patches of one
// level are ratio_y x ratio_z of the next finer one.
enum { MK_COARSE = 0, MK_MIDDLE = 1, MK_FINE = 2 };

// A merge step of a frame: into the middle patches (0), into the fine ones (1).
struct MkNodeMerge {
    int ratio_y, ratio_z;               // finer patches per patch
    int strip, strips;                  // finer patches per strip, strips per patch
    int rowg, chunks;                   // row groups of a block, blocks per strip
    long long w_off, item_off;
};

// One frame of a plan: py[L] x pz[L] patches of ly[L] x lz[L] pixels.
struct MkNodeFrame {
    double p0[3], ey[3], ez[3], b[3];
    int ny, nz;
    int ly[3], lz[3], py[3], pz[3];
    int bpy, bpz;                       // pixel blocks per fine patch
    MkNodeMerge mg[2];
    long long off[3];                   // patches of each level before this frame
    long long pix_off, pblk_off, part_off, w_off;
};

// A source of the pixel step: a group of `count` tiles (or runs) from `first`
// on, or a single tile (count 0). A run of tiles on middle nodes is one too.
struct MkNodeSrc {
    float dh[3];
    int species;
    float dl[3];
    int count;
    double o[3];
    long long first;
};

struct MkNodeRec {       // one node's direction: 64 bytes
    float4 w;            // b - u, 1/|P|
    float4 u;            // u, b.x
    float4 qh;           // k/2pi (b - u), high parts, b.y
    float4 ql;           // low parts, b.z
};

// ------------------------------------------------------------- plane fit
// Per frame: first pixel, mean column and row steps, and how far the pixels
// are from the product grid p0 + y_col ey + z_row ez of their own projected
// coordinates (fit[9], m), the smallest |P| (fit[10]) and the largest
// departure of y_col, z_row from column and row number (fit[11], pixels). The
// three are gathered as squares; ~35 operations of the FP64 pipe a pixel.

// Coordinate of a first-row (first-column) pixel along its axis, in steps;
// inv = 1 / |e|^2, 0 for an axis of one pixel.
__device__ __forceinline__ double mk_axis_coord(const double *p, const double *p0, const double *e, double inv)
{
    return ((p[0] - p0[0]) * e[0] + (p[1] - p0[1]) * e[1] + (p[2] - p0[2]) * e[2]) * inv;
}
__device__ __forceinline__ double mk_axis_inv(const double *e)
{
    const double n2 = e[0] * e[0] + e[1] * e[1] + e[2] * e[2];
    return n2 > 0.0 ? 1.0 / n2 : 0.0;
}

__global__ void mk_fit_init_kernel(int n_frames, const long long *__restrict__ shapes,
                                   const double *__restrict__ xyz, double *__restrict__ fit)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_frames) return;
    const double *p = xyz + 3 * shapes[3 * f];
    const long long ny = shapes[3 * f + 1], nz = shapes[3 * f + 2];
    double *o = fit + 12 * (long long)f;
    for (int c = 0; c < 3; ++c) {
        o[c] = p[c];
        o[3 + c] = ny > 1 ? (p[3 * (ny - 1) + c] - p[c]) / (ny - 1) : 0.0;
        o[6 + c] = nz > 1 ? (p[3 * (nz - 1) * ny + c] - p[c]) / (nz - 1) : 0.0;
    }
    o[9] = 0.0;
    o[10] = 1e300;
    o[11] = 0.0;
}

__global__ void mk_fit_kernel(const long long *__restrict__ shapes, const double *__restrict__ xyz,
                              double *__restrict__ fit)
{
    const int f = blockIdx.x;
    const long long off = shapes[3 * f];
    const int ny = (int)shapes[3 * f + 1], nz = (int)shapes[3 * f + 2];
    const double *P = xyz + 3 * off;
    double *o = fit + 12 * (long long)f;
    const double p0[3] = {o[0], o[1], o[2]}, ey[3] = {o[3], o[4], o[5]}, ez[3] = {o[6], o[7], o[8]};
    const double iy = mk_axis_inv(ey), iz = mk_axis_inv(ez);
    double dev = 0.0, rmin = 1e300, skew = 0.0;
    const long long n = (long long)ny * nz;
    for (long long i = (long long)blockIdx.y * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.y * blockDim.x) {
        const int row = (int)(i / ny), col = (int)(i - (long long)row * ny);
        const double y = mk_axis_coord(P + 3ll * col, p0, ey, iy);
        const double z = mk_axis_coord(P + 3ll * row * ny, p0, ez, iz);
        double d2 = 0.0, r2 = 0.0;
        for (int c = 0; c < 3; ++c) {
            const double v = P[3 * i + c], m = p0[c] + y * ey[c] + z * ez[c];
            d2 += (v - m) * (v - m);
            r2 += v * v;
        }
        const double s = fmax(fabs(y - (ny > 1 ? col : 0)), fabs(z - (nz > 1 ? row : 0)));
        dev = fmax(dev, d2 <= 1e300 ? d2 : INFINITY);       // a NaN counts as infinite
        skew = fmax(skew, s <= 1e300 ? s : INFINITY);
        rmin = fmin(rmin, r2 >= 0.0 ? r2 : 0.0);
    }
    for (int w = 16; w > 0; w >>= 1) {
        dev = fmax(dev, __shfl_xor_sync(0xffffffffu, dev, w));
        skew = fmax(skew, __shfl_xor_sync(0xffffffffu, skew, w));
        rmin = fmin(rmin, __shfl_xor_sync(0xffffffffu, rmin, w));
    }
    if ((threadIdx.x & 31) == 0) {      // non-negative doubles order as their bits
        dev = sqrt(dev);
        rmin = sqrt(rmin);
        atomicMax(reinterpret_cast<unsigned long long *>(o + 9), (unsigned long long)__double_as_longlong(dev));
        atomicMin(reinterpret_cast<unsigned long long *>(o + 10), (unsigned long long)__double_as_longlong(rmin));
        atomicMax(reinterpret_cast<unsigned long long *>(o + 11), (unsigned long long)__double_as_longlong(skew));
    }
}

extern "C" int mk_plane_fit(int n_frames, const long long *shapes, long long max_pix, const double *xyz,
                            double *fit, void *stream)
{
    MK_REQUIRE(n_frames >= 1 && shapes && xyz && fit && max_pix >= 1, "mk_plane_fit: bad arguments");
    cudaStream_t st = mk_stream(stream);
    mk_fit_init_kernel<<<(n_frames + 127) / 128, 128, 0, st>>>(n_frames, shapes, xyz, fit);
    const int gy = (int)std::max<long long>(1, std::min<long long>((max_pix + 1023) / 1024, 512));
    mk_fit_kernel<<<dim3(n_frames, gy), 256, 0, st>>>(shapes, xyz, fit);
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

// ------------------------------------------------------------------ plan
#define MK_SUM_PARTS 64      // chunks a frame's intensity sum is added in
namespace {

const int kNodeCounts[] = {6, 8, 10, 12, 16, 20};

// Largest phase half-range phi [rad] n Chebyshev nodes interpolate to
// 4 (phi/2)^n / n! <= 3e-8.
double phi_of(int n)
{
    double f = 7.5e-9;
    for (int i = 2; i <= n; ++i) f *= i;
    return 2.0 * std::pow(f, 1.0 / n);
}
struct PhiTable {
    double v[MK_NODE_MAX + 1];
    PhiTable() { for (int n = 1; n <= MK_NODE_MAX; ++n) v[n] = phi_of(n); }
};
const PhiTable kPhi;
double phi_max(int n) { return kPhi.v[n]; }

// Largest patch (pixels) whose phase half-range stays within `phi` for atoms
// up to k r = kr [rad] off the centre, a rad of direction per pixel.
double patch_limit(double phi, double kr, double a)
{
    const double half = phi / std::max(1.05 * kr * a, 1e-300);   // pixels, pad included
    return std::min(2.0 * (half - MK_NODE_PAD) + 1.0, 1e9);
}

// Even cut of n pixels into patches of at most `most`, a multiple of `unit`
// unless one patch holds all; false when even `unit` pixels are too many.
bool cut(int n, double most, int unit, int *len, int *count)
{
    if (most >= n) { *len = n; *count = 1; return true; }
    const int lim = (int)(most / unit) * unit;
    if (lim < unit) return false;
    const int c = (n + lim - 1) / lim;
    *len = ((n + c - 1) / c + unit - 1) / unit * unit;
    *count = (n + *len - 1) / *len;
    return true;
}

// One ROI shape: the widest angular steps of its frames, and how many there are.
struct Geo { double ay, az; int ny, nz, frames; };

// A level's patches of one ROI shape: py x pz of ly x lz pixels, each ry x rz of
// the finer level's.
struct Cut { int ly, lz, py, pz, ry, rz; };

// Fine patches of every ROI shape for sources of radius r on n nodes; the nodes
// of all frames.
bool fine_cut(const std::vector<Geo> &g, double k, double r, int n, std::vector<Cut> *out, double *nodes)
{
    *nodes = 0.0;
    for (size_t f = 0; f < g.size(); ++f) {
        Cut &C = (*out)[f];
        if (!cut(g[f].ny, patch_limit(phi_max(n), k * r, g[f].ay), MK_PIX_COLS, &C.ly, &C.py) ||
            !cut(g[f].nz, patch_limit(phi_max(n), k * r, g[f].az), MK_PIX_ROWS, &C.lz, &C.pz))
            return false;
        C.ry = C.rz = 1;
        *nodes += (double)g[f].frames * C.py * C.pz * n * n;
    }
    return true;
}

// Even blocks of at most `most` of p patches: how many patches a block, how many blocks.
void blocks_of(int p, int most, int *ratio, int *count)
{
    *count = (p + most - 1) / most;
    *ratio = (p + *count - 1) / *count;
    *count = (p + *ratio - 1) / *ratio;
}

// Patches of sources of radius r on n nodes, each a block of the finer level's.
bool parent_cut(const std::vector<Geo> &g, double k, double r, int n, const std::vector<Cut> &finer,
                std::vector<Cut> *out, double *nodes)
{
    *nodes = 0.0;
    for (size_t f = 0; f < g.size(); ++f) {
        const Cut &S = finer[f];
        Cut &C = (*out)[f];
        const int ry = (int)std::min<double>(S.py, std::floor(patch_limit(phi_max(n), k * r, g[f].ay) / S.ly));
        const int rz = (int)std::min<double>(S.pz, std::floor(patch_limit(phi_max(n), k * r, g[f].az) / S.lz));
        if (ry < 1 || rz < 1) return false;
        blocks_of(S.py, ry, &C.ry, &C.py);
        blocks_of(S.pz, rz, &C.rz, &C.pz);
        C.ly = S.ly * C.ry;
        C.lz = S.lz * C.rz;
        *nodes += (double)g[f].frames * C.py * C.pz * n * n;
    }
    return true;
}

// A run of tiles being gathered: the box of their origins and their widest
// radius bound its radius about the box's centre.
struct Run {
    double lo[3], hi[3], rmax;
    int count, species;
    bool single;                         // one tile, too wide for the coarse nodes
    long long first;
    void start(const double *o, int sp)
    {
        for (int c = 0; c < 3; ++c) lo[c] = hi[c] = o[c];
        rmax = o[3];
        count = 1;
        species = sp;
        single = false;
    }
    // Takes in a box of origins and their widest radius if the run's radius
    // stays within r2.
    bool add(const double *bl, const double *bh, double br, double r2)
    {
        double l[3], h[3], d2 = 0.0;
        for (int c = 0; c < 3; ++c) {
            l[c] = std::min(lo[c], bl[c]);
            h[c] = std::max(hi[c], bh[c]);
            d2 += (h[c] - l[c]) * (h[c] - l[c]);
        }
        const double r = std::max(rmax, br);
        if (!(0.5 * std::sqrt(d2) + r <= r2)) return false;
        for (int c = 0; c < 3; ++c) { lo[c] = l[c]; hi[c] = h[c]; }
        rmax = r;
        ++count;
        return true;
    }
};

// Cuts the narrow tiles (radius <= r1) of [a, b), in order, into runs of one
// species, radius <= r2 and at most `most` tiles: done(run) for each.
template <class Done>
void cut_runs(const double *org, const int *tsp, int a, int b, double r1, double r2, int most, Done done)
{
    Run R;
    R.count = 0;
    for (int t = a; t < b; ++t) {
        const double *o = org + 4ll * t;
        if (!(o[3] <= r1)) continue;
        if (R.count && tsp[t] == R.species && R.count < most && R.add(o, o, o[3], r2)) continue;
        if (R.count) done(R);
        R.start(o, tsp[t]);
    }
    if (R.count) done(R);
}

// Rows a thread of the merge holds, a divisor of n1.
int merge_rows(int n1) { return n1 == 10 ? 5 : n1 == 6 || n1 == 12 ? 3 : 4; }

// Cuts a patch's row of finer patches (n1 nodes) into strips of at most 128 node
// columns for the merge's blocks, the strip length that keeps most of their
// 128 threads busy.
void lay_strips(MkNodeMerge *M, int n1)
{
    const int rows = merge_rows(n1), most = std::min(M->ratio_y, MK_MERGE_NT / n1);
    double best = -1.0;
    for (int sp = 1; sp <= most; ++sp) {
        const int strips = (M->ratio_y + sp - 1) / sp;
        const int rowg = std::min(MK_MERGE_NT / (sp * n1), n1 / rows);
        const int chunks = (n1 / rows + rowg - 1) / rowg;
        const double use = (double)M->ratio_y * n1 * n1 / ((double)strips * chunks * MK_MERGE_NT * rows) + 1e-3 * sp;
        if (use > best) { best = use; M->strip = sp; M->strips = strips; M->rowg = rowg; M->chunks = chunks; }
    }
}

size_t up256(size_t b) { return (b + 255) & ~(size_t)255; }

// Costs [s], measured: one leaf term (2.1e12 a second), one (source, pixel) and
// one (tile, fine node) of the merge, both times 0.4 + 0.05 n for n nodes per
// axis, what a launch costs, and a term and the set-up of the split kernel where
// it takes a few wide tiles (its bounds, its plan, its own reduction).
const double kLeaf = 0.48e-12, kPix = 4.1e-12, kMerge = 3.8e-12, kLaunch = 4e-6;
const double kWide = 0.3e-12, kWideSetup = 150e-6;
double per_node(int n) { return 0.4 + 0.05 * n; }

// Nodes per axis an eighth of a tile is evaluated on before it is interpolated
// to the tile's n0, in two classes (0: evaluated whole): on the Hilbert curve an
// eighth has about half the tile's radius, and most tiles are much narrower than
// the widest one, r1. The phase that fewer nodes take is 0.49 (14 of 20), 0.34 (12
// of 20), 0.53 (12 of 16), 0.33 (10 of 16), 0.63 (10 of 12), 0.33 (8 of 12), 0.52
// (8 of 10) and 0.37 (6 of 8) of the tile's.
int sub_nodes(int n0, int tile_atoms, bool narrow)
{
    if (tile_atoms < 512) return 0;
    switch (n0) {
    case 20: return narrow ? 12 : 14;
    case 16: return narrow ? 10 : 12;
    case 12: return narrow ? 8 : 10;
    case 10: return narrow ? 8 : 0;
    case 8: return narrow ? 6 : 0;
    }
    return 0;
}

// Widest tile that goes with the narrow class, for tiles up to r1 on n0 nodes: an
// eighth is half of it where tiles are whole cubes (at 0.55 of it 1.48 + 1.03 ms
// went on the 5.3M-atom exposure, at 0.51 and 0.47 2.3 ms).
double narrow_radius(int n0, int nt, double r1) { return r1 * phi_max(nt) / phi_max(n0) / 0.50; }

// Leaf terms per coarse patch of an atom of the two classes, interpolation of
// the eighths and the wide ones among them included.
double leaf_terms(int n0, int tile_atoms, bool narrow)
{
    const int ns = sub_nodes(n0, tile_atoms, narrow);
    return ns ? 1.2 * ns * ns : (double)n0 * n0;
}

// Radii and nodes of tiles (r1, n0), runs (rm, nm; nm 0: no middle level) and
// groups (r2, n1; G 0: none).
struct Choice {
    double cost = 1e300, r1 = 0.0, rm = 0.0, r2 = 0.0;
    int n0 = 0, nm = 0, n1 = 0, G = 0;
};

// Node records of a plan: coarse, middle, fine, and the eighths' on the coarse patches.
long long records(const mk_node_plan &P)
{
    return P.patches0 * (P.n0 * P.n0 + P.ns[0] * P.ns[0] + P.ns[1] * P.ns[1]) + P.patchesm * P.nm * P.nm + P.patches1 * P.n1 * P.n1;
}

// Whole frames from f on whose node fields and partials fit `budget` bytes (one
// at least), and their launches fit a grid: their patches of each level, pixels,
// pixel blocks, merge blocks per source and bytes. Returns the frame after them.
struct Pass {
    long long patches[3], pix, pblk, items[2];
    size_t bytes, field[3];
};
int next_pass(const mk_node_plan &plan, const MkNodeFrame *fr, int f, size_t budget, Pass *out)
{
    const int n[3] = {plan.n0, plan.nm, plan.n1};
    const double rows[3] = {(double)plan.n_members, (double)plan.n_msrc, (double)plan.n_src};
    Pass P{};
    for (int g = f; g < plan.n_frames; ++g) {
        const MkNodeFrame &F = fr[g];
        Pass Q = P;
        bool too_many = false;
        for (int l = 0; l < 3; ++l) {
            Q.patches[l] += (long long)F.py[l] * F.pz[l];
            const double nodes = (double)Q.patches[l] * n[l] * n[l];
            too_many |= nodes > 256.0 * 60000;
            Q.field[l] = up256((size_t)(8.0 * nodes * rows[l]));
        }
        Q.pix += (long long)F.ny * F.nz;
        Q.pblk += (long long)F.py[MK_FINE] * F.pz[MK_FINE] * F.bpy * F.bpz;
        for (int m = 0; m < 2; ++m) {
            const int in = m == 0 || !plan.nm ? MK_COARSE : MK_MIDDLE, to = m == 0 ? MK_MIDDLE : MK_FINE;
            Q.items[m] += (long long)F.pz[to] * F.py[in] * F.mg[m].strips * F.mg[m].chunks;
            too_many |= Q.items[m] * std::max(m == 0 ? plan.n_msrc : plan.n_groups, 1) > (1ll << 30);
        }
        Q.bytes = Q.field[0] + Q.field[1] + Q.field[2] + up256(16 * (size_t)Q.pix * plan.slices);
        if (g > f && (Q.bytes > budget || too_many)) {
            *out = P;
            return g;
        }
        P = Q;
    }
    *out = P;
    return plan.n_frames;
}

}  // namespace

extern "C" size_t mk_nodes_plan_bytes(int n_frames, int n_tiles)
{
    if (n_frames < 1 || n_tiles < 0) return 0;
    return up256(sizeof(MkNodeFrame) * (size_t)n_frames) + 2 * up256(sizeof(MkNodeSrc) * (size_t)n_tiles) +
           up256(sizeof(double4) * (size_t)n_tiles) + 7 * up256(sizeof(int) * (size_t)n_tiles);
}

extern "C" int mk_nodes_plan(int n_tiles, int tile_atoms, int n_species, const int64_t *counts,
                             const double *origins, int n_frames, const long long *shapes,
                             const double *fit, const double *beam_dirs, double k, double phase_tol,
                             double direct_s_per_term, int group_tiles, mk_node_plan *plan,
                             void *host_buf, size_t host_bytes)
{
    MK_REQUIRE(n_tiles >= 1 && n_frames >= 1 && counts && origins && shapes && fit && beam_dirs && plan &&
                   host_buf && n_species >= 1 && n_species <= MK_MAX_SPECIES && tile_atoms >= 1,
               "mk_nodes_plan: bad arguments");
    MK_REQUIRE(host_bytes >= mk_nodes_plan_bytes(n_frames, n_tiles), "mk_nodes_plan: buffer too small");
    memset(plan, 0, sizeof(*plan));
    std::vector<Geo> geo;
    std::vector<int> shape_of(n_frames);
    double n_pix = 0.0, rmin = 1e300, dev = 0.0;
    for (int f = 0; f < n_frames; ++f) {
        const double *t = fit + 12ll * f;
        // the fit's own sanity: on the grid, within a quarter pixel of it
        if (!(t[9] <= 1e300) || !(t[11] <= 0.25) || !(t[10] > 0.0)) {
            mk_set_error("mk_nodes_plan: frame %d is not a plane grid of pixels", f);
            return MK_EDECLINE;
        }
        const int ny = (int)shapes[3 * f + 1], nz = (int)shapes[3 * f + 2];
        size_t i = 0;
        while (i < geo.size() && (geo[i].ny != ny || geo[i].nz != nz)) ++i;
        if (i == geo.size()) geo.push_back(Geo{0.0, 0.0, ny, nz, 0});
        shape_of[f] = (int)i;
        geo[i].ay = std::max(geo[i].ay, std::sqrt(t[3] * t[3] + t[4] * t[4] + t[5] * t[5]) / t[10]);
        geo[i].az = std::max(geo[i].az, std::sqrt(t[6] * t[6] + t[7] * t[7] + t[8] * t[8]) / t[10]);
        ++geo[i].frames;
        n_pix += (double)ny * nz;
        rmin = std::min(rmin, t[10]);
        dev = std::max(dev, t[9] / t[10]);
    }
    std::vector<int> tsp(n_tiles);
    {
        int t = 0;
        for (int s = 0; s < n_species; ++s)
            for (int64_t i = 0; i < (counts[s] + tile_atoms - 1) / tile_atoms; ++i)
                if (t < n_tiles) tsp[t++] = s;
        MK_REQUIRE(t == n_tiles, "mk_nodes_plan: %d tiles, the species counts give %d", n_tiles, t);
    }
    std::vector<double> rad(n_tiles);
    double rmax = 0.0, omax = 0.0;
    for (int t = 0; t < n_tiles; ++t) {
        const double *o = origins + 4ll * t;
        rad[t] = o[3];
        const double on = std::sqrt(o[0] * o[0] + o[1] * o[1] + o[2] * o[2]);
        if (!(o[3] < 1.0) || !(on < 1.0)) {
            mk_set_error("mk_nodes_plan: tile %d has no finite extent", t);
            return MK_EDECLINE;
        }
        rmax = std::max(rmax, o[3]);
        omax = std::max(omax, on);
    }
    // the factor is taken at the pixels' own directions (as the split
    // kernel's factor table), and third-order terms are dropped
    auto admitted = [&](double r) {
        const double third = k * (r * r * r + omax * omax * omax + 3.0 * omax * omax * r) / (rmin * rmin);
        return third + k * r * dev <= phase_tol && 2.0 * (omax + r) / rmin < 1e-6;
    };
    const double T = tile_atoms;
    plan->direct_s = n_tiles * T * n_pix * direct_s_per_term + 2.0 * kLaunch;
    auto split = [&](double n) { return n > 0.0 ? n * T * n_pix * kWide + n_pix * 30e-12 + kWideSetup : 0.0; };

    // Search on a sample: at most 2048 tiles, in 4 stretches of the curve.
    const int stretch = n_tiles <= 2048 ? n_tiles : 512, stretches = n_tiles <= 2048 ? 1 : 4;
    std::vector<double> some;
    std::vector<int> starts;
    for (int i = 0; i < stretches; ++i) {
        const int a = (int)((long long)(n_tiles - stretch) * i / std::max(stretches - 1, 1));
        starts.push_back(a);
        some.insert(some.end(), rad.begin() + a, rad.begin() + a + stretch);
    }
    std::sort(some.begin(), some.end());
    const double up = (double)n_tiles / some.size();
    auto q = [&](double x) { return some[(size_t)std::floor(x * (some.size() - 1) + 0.5)]; };
    std::vector<double> tail;               // the widest tiles, all of them: few, but dear
    for (double r : rad)
        if (r > q(0.9)) tail.push_back(r);
    std::sort(tail.begin(), tail.end());
    Choice best;
    std::vector<Cut> c1(geo.size()), cm(geo.size()), c0(geo.size());
    const double q1[] = {rmax, q(0.99), q(0.95), q(0.8)};
    const double f2[] = {1.0, 1.5, 2.2, 3.2, 4.5, 6.5, 9.0};
    const int nf2 = sizeof(f2) / sizeof(f2[0]);
    const int G = group_tiles > 0 ? group_tiles : 4096;
    const bool groups = group_tiles != 0 && (group_tiles > 0 || n_tiles >= 32);
    double run_count[nf2];                  // runs of all tiles within every radius
    for (int i = 0; groups && i < nf2; ++i) {
        run_count[i] = 0.0;
        for (int a : starts)
            cut_runs(origins, tsp.data(), a, a + stretch, q(0.95), std::max(f2[i] * q(0.5), q(0.95)), G,
                     [&](const Run &) { run_count[i] += up / 0.95; });
    }
    for (int i1 = 0; i1 < 4; ++i1) {
        const double r1 = q1[i1];
        if (i1 > 0 && r1 == q1[i1 - 1]) continue;
        auto above = [&](double r) {            // tiles wider than r (few: exactly)
            if (r >= q(0.9)) return (double)(tail.end() - std::upper_bound(tail.begin(), tail.end(), r));
            return up * (double)(some.end() - std::upper_bound(some.begin(), some.end(), r));
        };
        const double n_nar = n_tiles - above(r1);
        if (n_nar < 1.0) continue;
        // no groups: every tile within r1 straight from its nodes
        if (admitted(r1) && group_tiles <= 0)
            for (int n1 : kNodeCounts) {
                double N1;
                if (n1 > 16 || !fine_cut(geo, k, r1, n1, &c1, &N1)) continue;
                const double c = n_nar * T * N1 * kLeaf + n_nar * n_pix * kPix * per_node(n1) +
                                 split(n_tiles - n_nar) + 4.0 * kLaunch;
                if (c < best.cost) { best = Choice(); best.cost = c; best.r1 = best.r2 = r1; best.n1 = n1; }
            }
        if (!groups) continue;
        double rads[nf2], runs[nf2], wider[nf2];     // radii, runs within them, single tiles beyond them
        int nr = 0;
        for (int i = 0; i < nf2; ++i) {
            const double r = f2[i] * q(0.5);
            if (r < r1 || !admitted(r)) continue;
            rads[nr] = r;
            runs[nr] = run_count[i] * n_nar / n_tiles;
            wider[nr++] = above(r);
        }
        for (int i2 = 0; i2 < nr; ++i2)
            for (int n1 : kNodeCounts) {
                double N1, Nm, N0;
                if (n1 > 12 || !fine_cut(geo, k, rads[i2], n1, &c1, &N1)) continue;
                const double pixel = runs[i2] * n_pix * kPix * per_node(n1) + split(wider[i2]) + 6.0 * kLaunch;
                const double one = T * N1 * kLeaf + n_pix * kPix * per_node(n1);     // a single tile
                for (int im = -1; im < i2; ++im) {
                    // im < 0: tiles straight into groups; else by runs of radius rads[im]
                    const double single = (im < 0 ? above(r1) : wider[im]) - wider[i2];
                    const double rest = pixel + single * one;
                    if (rest >= best.cost) continue;
                    for (int nm : kNodeCounts) {
                        double part = rest, Nt = N1;
                        if (im < 0) {
                            if (nm != kNodeCounts[0]) break;
                        } else {
                            if (nm < 8 || nm > 16 || !parent_cut(geo, k, rads[im], nm, c1, &cm, &Nm)) continue;
                            const double own = above(r1) - wider[im];
                            part += own * T * Nm * kLeaf + (runs[im] + own) * N1 * kMerge * per_node(nm) + 2.0 * kLaunch;
                            Nt = Nm;
                        }
                        if (part >= best.cost) continue;
                        for (int n0 : kNodeCounts) {
                            if (n0 < 8 || !parent_cut(geo, k, r1, n0, im < 0 ? c1 : cm, &c0, &N0)) continue;
                            const int nt = sub_nodes(n0, tile_atoms, true);
                            const double narrow = nt ? std::min(n_tiles - above(narrow_radius(n0, nt, r1)), n_nar) : 0.0;
                            const double leaf = narrow * leaf_terms(n0, tile_atoms, true) +
                                                (n_nar - narrow) * leaf_terms(n0, tile_atoms, false);
                            const double c = part + T * N0 / (n0 * n0) * leaf * kLeaf + n_nar * Nt * kMerge * per_node(n0);
                            if (c >= best.cost) continue;
                            best.cost = c;
                            best.r1 = r1;
                            best.rm = im < 0 ? 0.0 : rads[im];
                            best.r2 = rads[i2];
                            best.n0 = n0;
                            best.nm = im < 0 ? 0 : nm;
                            best.n1 = n1;
                            best.G = G;
                        }
                    }
                }
            }
    }
    plan->form_s = best.cost;
    if (!(best.cost < plan->direct_s)) {
        mk_set_error("mk_nodes_plan: the direct sum is as fast (%.3g s against %.3g s) or the geometry "
                     "leaves the error budget", plan->direct_s, best.cost);
        return MK_EDECLINE;
    }
    // lay the chosen plan out
    std::vector<MkNodeFrame> fr(n_frames);
    double nodes;
    fine_cut(geo, k, best.r2, best.n1, &c1, &nodes);
    if (best.nm) parent_cut(geo, k, best.rm, best.nm, c1, &cm, &nodes);
    if (best.G) parent_cut(geo, k, best.r1, best.n0, best.nm ? cm : c1, &c0, &nodes);
    auto level = [&](MkNodeFrame *F, int l, const Cut &C) {
        F->ly[l] = C.ly;
        F->lz[l] = C.lz;
        F->py[l] = C.py;
        F->pz[l] = C.pz;
    };
    auto merge = [&](MkNodeMerge *M, const Cut &C, int n_out) {     // patches of C from the finer level's
        M->ratio_y = C.ry;
        M->ratio_z = C.rz;
        lay_strips(M, n_out);
    };
    for (int f = 0; f < n_frames; ++f) {
        MkNodeFrame &F = fr[f];
        const int g = shape_of[f];
        F = MkNodeFrame{};
        F.ny = geo[g].ny;
        F.nz = geo[g].nz;
        level(&F, MK_FINE, c1[g]);
        F.bpy = (c1[g].ly + MK_PIX_COLS - 1) / MK_PIX_COLS;
        F.bpz = (c1[g].lz + MK_PIX_ROWS - 1) / MK_PIX_ROWS;
        if (best.G) {
            level(&F, MK_COARSE, c0[g]);
            merge(&F.mg[1], best.nm ? cm[g] : c0[g], best.n1);
        }
        if (best.nm) {
            level(&F, MK_MIDDLE, cm[g]);
            merge(&F.mg[0], c0[g], best.nm);
        }
    }
    std::vector<MkNodeSrc> src, msrc;
    std::vector<double4> morg;
    std::vector<int> members, mid, wide, msingle, mrow;
    auto source = [&](const double *c, int species, int count, long long first) {
        MkNodeSrc S{};
        for (int i = 0; i < 3; ++i) {
            S.o[i] = c[i];
            S.dh[i] = (float)c[i];
            S.dl[i] = (float)(c[i] - (double)S.dh[i]);
        }
        S.species = species;
        S.count = count;
        S.first = first;
        return S;
    };
    auto centre = [&](const Run &R, double *c) {
        for (int i = 0; i < 3; ++i) c[i] = 0.5 * (R.lo[i] + R.hi[i]);
    };
    const double reach = best.nm ? best.rm : best.r1;       // widest tile of a group
    for (int t = 0; t < n_tiles; ++t) {
        if (rad[t] > best.r2) wide.push_back(t);
        else if (best.G == 0 || rad[t] > reach) mid.push_back(t);
        else if (rad[t] <= best.r1) members.push_back(t);
    }
    if (best.nm) {
        // runs of tiles within rm, and the tiles between r1 and rm by themselves, in
        // the order of the curve; then groups of those
        std::vector<Run> list;
        long long first = 0;
        Run R;
        R.count = 0;
        auto close = [&]() {
            if (!R.count) return;
            R.first = first;
            first += R.count;
            list.push_back(R);
            R.count = 0;
        };
        for (int t = 0; t < n_tiles; ++t) {
            const double *o = origins + 4ll * t;
            if (o[3] > best.rm) continue;
            if (o[3] > best.r1) {
                Run S;
                S.start(o, tsp[t]);
                S.single = true;
                S.first = t;
                list.push_back(S);
                continue;
            }
            if (R.count && tsp[t] == R.species && R.count < best.G && R.add(o, o, o[3], best.rm)) continue;
            close();
            R.start(o, tsp[t]);
        }
        close();
        std::stable_sort(list.begin(), list.end(), [](const Run &a, const Run &b) { return a.species < b.species; });
        Run Q;
        int tiles_in = 0;
        Q.count = 0;
        auto emit = [&]() {
            double c[3];
            if (!Q.count) return;
            centre(Q, c);
            src.push_back(source(c, Q.species, Q.count, (long long)msrc.size() - Q.count));
            Q.count = 0;
        };
        for (const Run &L : list) {
            const int n = L.single ? 1 : L.count;
            if (!(Q.count && L.species == Q.species && tiles_in + n <= best.G && Q.add(L.lo, L.hi, L.rmax, best.r2))) {
                emit();
                Q = L;
                Q.count = 1;
                tiles_in = 0;
            }
            tiles_in += n;
            double c[3];
            centre(L, c);
            msrc.push_back(source(c, L.species, L.single ? 0 : L.count, L.single ? 0 : L.first));
            morg.push_back(double4{c[0], c[1], c[2], 0.0});
            if (L.single) {
                msingle.push_back((int)L.first);
                mrow.push_back((int)msrc.size() - 1);
            }
        }
        emit();
    } else if (best.G) {
        long long first = 0;
        cut_runs(origins, tsp.data(), 0, n_tiles, best.r1, best.r2, best.G, [&](const Run &R) {
            double c[3];
            centre(R, c);
            src.push_back(source(c, R.species, R.count, first));
            first += R.count;
        });
    }
    plan->n_groups = (int)src.size();
    for (int t : mid) src.push_back(source(origins + 4ll * t, tsp[t], 0, 0));
    plan->n_src = (int)src.size();
    plan->n_members = (int)members.size();
    plan->n_mid = (int)mid.size();
    plan->n_wide = (int)wide.size();
    plan->n0 = best.G ? best.n0 : 0;
    plan->nm = best.nm;
    plan->n_msrc = (int)msrc.size();
    plan->n_msingle = (int)msingle.size();
    plan->n1 = best.n1;
    plan->n_frames = n_frames;
    plan->n_tiles = n_tiles;
    plan->group_tiles = best.G;
    plan->radius1_m = best.r1;
    plan->radiusm_m = best.rm;
    plan->radius2_m = best.r2;
    plan->n_pix = (long long)n_pix;
    if (plan->n_src < 1) {
        mk_set_error("mk_nodes_plan: every tile is wider than the plan's radius");
        return MK_EDECLINE;
    }
    const int n[3] = {plan->n0, plan->nm, plan->n1};
    long long pblk = 0, wf = 0, patches[3] = {0, 0, 0}, item[2] = {0, 0};
    for (int f = 0; f < n_frames; ++f) {
        MkNodeFrame &F = fr[f];
        const double *t = fit + 12ll * f;
        for (int c = 0; c < 3; ++c) {
            F.p0[c] = t[c];
            F.ey[c] = t[3 + c];
            F.ez[c] = t[6 + c];
            F.b[c] = beam_dirs[3ll * f + c];
        }
        F.pix_off = shapes[3 * f];
        F.pblk_off = pblk;
        F.w_off = wf;
        pblk += (long long)F.py[MK_FINE] * F.pz[MK_FINE] * F.bpy * F.bpz;
        wf += (long long)best.n1 * (F.ny + F.nz);
        for (int l = 0; l < 3; ++l) {
            F.off[l] = patches[l];
            patches[l] += (long long)F.py[l] * F.pz[l];
        }
        for (int m = 0; m < 2; ++m) {
            MkNodeMerge &M = F.mg[m];
            const int in = m == 0 || !best.nm ? MK_COARSE : MK_MIDDLE, to = m == 0 ? MK_MIDDLE : MK_FINE;
            M.w_off = wf;
            M.item_off = item[m];
            wf += (long long)(M.ratio_y + M.ratio_z) * n[to] * n[in];
            item[m] += (long long)F.pz[to] * F.py[in] * M.strips * M.chunks;
        }
    }
    int sms = 152, devid = 0;               // 152: planned without a device
    if (cudaGetDevice(&devid) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, devid);
    plan->sms = sms;
    const long long patch = patches[MK_FINE];
    plan->patches0 = patches[MK_COARSE];
    plan->patchesm = patches[MK_MIDDLE];
    // leaves by eighths: the narrow class's tiles first, and the rows of their fields
    std::vector<int> leaf, leaf_row;
    for (int c = 0; c < 2 && best.G; ++c) {
        const int ns = sub_nodes(best.n0, tile_atoms, c == 0);
        if (!sub_nodes(best.n0, tile_atoms, true)) break;
        // a second launch pays where both fill the chip: eight blocks an SM
        const bool two = (long long)members.size() * plan->patches0 >= 8ll * sms;
        const double split_at = two ? narrow_radius(best.n0, sub_nodes(best.n0, tile_atoms, true), best.r1) : -1.0;
        for (size_t i = 0; i < members.size(); ++i)
            if ((rad[members[i]] <= split_at) == (c == 0)) {
                leaf.push_back(members[i]);
                leaf_row.push_back((int)i);
            }
        if (c == 0) plan->n_narrow = (int)leaf.size();
        plan->ns[c] = ns;
        plan->sub_radius_m[c] = ns ? best.r1 * phi_max(ns) / phi_max(best.n0) : 0.0;
        plan->sub_w_off[c] = wf;
        wf += best.n0 * ns;
    }
    plan->patches1 = patch;
    plan->weights = wf;
    // slices of sources: enough blocks for every SM several times over, at
    // least eight sources a slice
    const long long want = (12ll * sms + pblk - 1) / pblk;
    plan->slices = (int)std::max<long long>(1, std::min<long long>(std::min<long long>(want, 256),
                                                                   plan->n_src / 8));
    plan->src_per_slice = (plan->n_src + plan->slices - 1) / plan->slices;
    plan->slices = (plan->n_src + plan->src_per_slice - 1) / plan->src_per_slice;
    for (int f = 0; f < n_frames; ++f) fr[f].part_off = fr[f].pix_off * plan->slices;
    // frames per pass: as many as a few GB of node fields and partials hold
    size_t need = 0;
    int passes = 0;
    for (int f = 0; f < n_frames; ++passes) {
        Pass P;
        f = next_pass(*plan, fr.data(), f, (size_t)4 << 30, &P);
        need = std::max(need, P.bytes);
        for (int l = 0; l < 3; ++l)
            if (P.patches[l] * n[l] * n[l] > 256ll * 65535) {
                mk_set_error("mk_nodes_plan: too many nodes in one frame");
                return MK_EDECLINE;
            }
    }
    plan->passes = passes;
    if (need > ((size_t)16 << 30)) {
        mk_set_error("mk_nodes_plan: %zu bytes of node fields for one frame", need);
        return MK_EDECLINE;
    }
    plan->chunk_bytes = need;
    plan->ws_bytes = up256(sizeof(MkNodeRec) * (size_t)records(*plan)) +
                     up256(sizeof(float) * (size_t)wf) +
                     std::max(need, up256(8 * (size_t)MK_SUM_PARTS * n_frames));
    char *hb = static_cast<char *>(host_buf);
    size_t off = 0;
    auto put = [&](const void *p, size_t n) {
        const size_t at = off;
        if (n) memcpy(hb + at, p, n);
        off += up256(n);
        return (long long)at;
    };
    put(fr.data(), sizeof(MkNodeFrame) * fr.size());
    plan->off_src = put(src.data(), sizeof(MkNodeSrc) * src.size());
    plan->off_members = put(members.data(), sizeof(int) * members.size());
    plan->off_mid = put(mid.data(), sizeof(int) * mid.size());
    plan->off_wide = put(wide.data(), sizeof(int) * wide.size());
    plan->off_leaf = put(leaf.data(), sizeof(int) * leaf.size());
    plan->off_leaf_row = put(leaf_row.data(), sizeof(int) * leaf_row.size());
    plan->off_msrc = put(msrc.data(), sizeof(MkNodeSrc) * msrc.size());
    plan->off_morg = put(morg.data(), sizeof(double4) * morg.size());
    plan->off_msingle = put(msingle.data(), sizeof(int) * msingle.size());
    plan->off_mrow = put(mrow.data(), sizeof(int) * mrow.size());
    plan->buf_bytes = (long long)off;
    return MK_OK;
}

// --------------------------------------------------------------- kernels
struct MkNodeArgs {
    const MkNodeFrame *frames;
    int f_lo, f_hi;                  // frames of this pass
    int n1, n_groups, n_src, src_per_slice, tile_atoms;
    long long patches1, patch1_base; // fine patches of this pass, and before it
    long long pblk_base, part_base;
    const MkNodeSrc *src;
    float2 *V1;
    const double4 *origin;
    const float4 *tpos;
    const float2 *tamp;
    const double4 *q;
    const float4 *u;
    const float2 *ftab;
    long long ftab_n;
    const float *weights;
    double2 *partial;
    float kappa, fres_r;
    double kappa_d;
    int fresnel, decay;
};

// One merge: sources on n_in nodes per axis of level `in` to n_out of level
// `to`, patches and bases of this pass.
struct MkMergeArgs {
    const MkNodeFrame *frames;
    int f_lo, f_hi;
    int step, in, to, n_out;
    long long in_patches, in_base, to_patches, to_base, item_base, items;
    const MkNodeSrc *src;            // the runs or groups made
    const int *members;              // their tiles (null: sources in order)
    const double4 *origin;
    const MkNodeRec *rec;            // of level `to`, every frame
    const float *weights;
    const float2 *Vin;
    float2 *Vout;
    float kappa;
};

// First frame f in [lo, hi) whose key(f+1) exceeds i.
template <class Key>
__device__ __forceinline__ int mk_find_frame(int lo, int hi, long long i, Key key)
{
    --hi;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (key(mid) <= i) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ double mk_half_range(int len) { return 0.5 * (len - 1) + MK_NODE_PAD; }

// The Chebyshev nodes of one count and the inverse products of their Lagrange
// weights.
struct MkCheb {
    double x[MK_NODE_MAX], inv[MK_NODE_MAX];
    void fill(int n)
    {
        for (int i = 0; i < n; ++i) x[i] = std::cos((2 * i + 1) * MK_PI / (2.0 * n));
        for (int j = 0; j < n; ++j) {
            double den = 1.0;
            for (int i = 0; i < n; ++i)
                if (i != j) den *= x[j] - x[i];
            inv[j] = 1.0 / den;
        }
    }
};

// Lagrange weight j of n nodes at x (FP64 products), rounded to float32 so that
// the point's n weights still sum to 1: the rounding of each would be the same
// for every source and so a relative error of ~1e-7 of the whole sum. A group
// of `width` lanes (16 or 32) holds one point's weights (lane j weight j, j >= n
// 0); the largest takes what the sum is off by, the next largest what its own
// rounding leaves.
__device__ __forceinline__ float mk_lagrange(const MkCheb &C, double x, int n, int j, int width)
{
    double num = j < n ? C.inv[j] : 0.0;
    for (int i = 0; i < n; ++i)
        if (i != j) num *= x - C.x[i];
    float w = (float)num;
    double off = (double)w;
    for (int o = width >> 1; o > 0; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
    off = 1.0 - off;
    float key = fabsf(w);
    const unsigned lane = threadIdx.x & 31, group = width == 32 ? 0xffffffffu : 0xffffu << (lane & 16);
#pragma unroll
    for (int round = 0; round < 2; ++round) {
        float big = key;
        for (int o = width >> 1; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
        const int who = __ffs(__ballot_sync(0xffffffffu, key == big) & group) - 1;
        if ((int)lane == who) {
            const float to = (float)((double)w + off);
            off -= (double)to - (double)w;
            w = to;
            key = -1.f;
        }
        off = __shfl_sync(0xffffffffu, off, who);
    }
    return w;
}

// Node records and weight tables of every frame: one thread per node, 16 or 32
// lanes per point's weights (blocks before `node_blocks` the one, the rest the
// other). On one frame a chain of ~n FP64 products' latency, on many the FP64
// pipe: the nodes of every count come with the arguments (a block that made
// them itself spent ~100 operations of it a warp). With all n weights (and the
// nodes' cosines) in one thread it took 35 us on a 128 x 128 detector and 99 us
// for 16 frames; here 6 and 55 us.
struct MkPrepArgs {
    const MkNodeFrame *frames;
    int n[5];                            // nodes per axis of the levels, and of eighths of either class
    MkNodeRec *rec[5];
    int node_blocks;
    double kappa;
    const double *xyz;
    float *weights, *w_s[2];
    MkCheb cheb[5];
};
#define MK_PREP_NT 128
__global__ void __launch_bounds__(MK_PREP_NT) mk_node_prep_kernel(const MkPrepArgs A)
{
    __shared__ MkCheb s_c[5];              // of every level, and of eighths
    const int th = threadIdx.x;
    for (int i = th; i < 5 * 2 * MK_NODE_MAX; i += MK_PREP_NT)
        reinterpret_cast<double *>(s_c)[i] = reinterpret_cast<const double *>(A.cheb)[i];
    __syncthreads();
    const MkNodeFrame &F = A.frames[blockIdx.x];
    if ((int)blockIdx.y < A.node_blocks) {
        int first[6] = {0};
#pragma unroll
        for (int l = 0; l < 5; ++l) {
            const int g = l > 2 ? MK_COARSE : l;
            first[l + 1] = first[l] + F.py[g] * F.pz[g] * A.n[l] * A.n[l];
        }
        for (int t = blockIdx.y * MK_PREP_NT + th; t < first[5]; t += A.node_blocks * MK_PREP_NT) {
            int lv = 0, e = t;
#pragma unroll
            for (int l = 1; l < 5; ++l)
                if (t >= first[l]) { lv = l; e = t - first[l]; }
            const int g = lv > 2 ? MK_COARSE : lv;
            const int n = A.n[lv], py = F.py[g], ly = F.ly[g], lz = F.lz[g];
            const int p = e / (n * n), r = e - p * n * n, j = r / n, c = r - j * n;
            const int pz = p / py, pyi = p - pz * py;
            const double *X = s_c[lv].x;
            const double y = pyi * (double)ly + 0.5 * (ly - 1) + mk_half_range(ly) * X[c];
            const double z = pz * (double)lz + 0.5 * (lz - 1) + mk_half_range(lz) * X[j];
            double P[3], u[3], q[3], r2 = 0.0;
            for (int d = 0; d < 3; ++d) {
                P[d] = F.p0[d] + y * F.ey[d] + z * F.ez[d];
                r2 += P[d] * P[d];
            }
            const double inv = 1.0 / sqrt(r2);
            for (int d = 0; d < 3; ++d) {
                u[d] = P[d] * inv;
                q[d] = A.kappa * (F.b[d] - u[d]);
            }
            const float hx = (float)q[0], hy = (float)q[1], hz = (float)q[2];
            MkNodeRec R;
            R.w = make_float4((float)(F.b[0] - u[0]), (float)(F.b[1] - u[1]), (float)(F.b[2] - u[2]), (float)inv);
            R.u = make_float4((float)u[0], (float)u[1], (float)u[2], (float)F.b[0]);
            R.qh = make_float4(hx, hy, hz, (float)F.b[1]);
            R.ql = make_float4((float)(q[0] - hx), (float)(q[1] - hy), (float)(q[2] - hz), (float)F.b[2]);
            A.rec[lv][F.off[g] * n * n + e] = R;
        }
        return;
    }
    // points: pixel columns and rows in their fine patches, the nodes of a finer
    // level in a patch of the coarser one, and (frame 0) a tile's nodes among its
    // eighths'
    const MkNodeMerge &M1 = F.mg[1], &M0 = F.mg[0];
    const int above = A.n[MK_MIDDLE] ? MK_MIDDLE : MK_COARSE;
    const int e0 = F.ny + F.nz, e1 = e0 + (A.n[0] ? (M1.ratio_y + M1.ratio_z) * A.n[MK_FINE] : 0);
    const int e2 = e1 + (A.n[MK_MIDDLE] ? (M0.ratio_y + M0.ratio_z) * A.n[MK_MIDDLE] : 0);
    const int points = e2 + (blockIdx.x == 0 && A.n[3] ? 2 * A.n[0] : 0);
    const int width = max(A.n[0], max(A.n[1], A.n[2])) > 16 ? 32 : 16, lane = th & (width - 1);
    const int per = MK_PREP_NT / width, step = (gridDim.y - A.node_blocks) * per;
    // whole warps stay in the loop: the lanes of a warp's groups shuffle together
    for (int i0 = (blockIdx.y - A.node_blocks) * per + (th >> 5) * (32 / width); i0 < points; i0 += step) {
        const int at = i0 + (th & 31) / width, i = min(at, points - 1);
        double x;
        float *out;
        int lv = MK_FINE;
        if (i < e0) {
            const bool row = i >= F.ny;
            const int k = row ? i - F.ny : i, len = row ? F.lz[MK_FINE] : F.ly[MK_FINE];
            const double *P = A.xyz + 3 * (F.pix_off + (row ? (long long)k * F.ny : k));
            const double v = mk_axis_coord(P, F.p0, row ? F.ez : F.ey, mk_axis_inv(row ? F.ez : F.ey));
            x = (v - ((k / len) * (double)len + 0.5 * (len - 1))) / mk_half_range(len);
            out = A.weights + F.w_off + (long long)i * A.n[MK_FINE];
        } else if (i < e2) {
            const bool low = i < e1;             // into the fine patches
            const MkNodeMerge &M = low ? M1 : M0;
            const int m = i - (low ? e0 : e1), to = low ? MK_FINE : MK_MIDDLE, n_to = A.n[to];
            lv = low ? above : MK_COARSE;
            const bool row = m >= M.ratio_y * n_to;
            const int k = row ? m - M.ratio_y * n_to : m;
            const int l1 = row ? F.lz[to] : F.ly[to], l0 = row ? F.lz[lv] : F.ly[lv];
            const int sub = k / n_to, c = k - sub * n_to;
            const double v = sub * (double)l1 + 0.5 * (l1 - 1) + mk_half_range(l1) * s_c[to].x[c];
            x = (v - 0.5 * (l0 - 1)) / mk_half_range(l0);
            out = A.weights + M.w_off + (long long)m * A.n[lv];
        } else {
            const int c = i - e2 >= A.n[0], j = i - e2 - c * A.n[0];
            x = s_c[MK_COARSE].x[j];
            lv = 3 + c;
            out = A.w_s[c] + j * A.n[lv];
        }
        const int n = A.n[lv];
        const float w = mk_lagrange(s_c[lv], x, n, lane, width);
        if (lane < n && at < points) out[lane] = w;
    }
}

// A tile's field on the nodes: V[rows[list position]][node] (rows null: the list
// position). One node a thread,
// the tile's atoms (interleaved pairs) from shared memory, two atoms per
// packed instruction. Bound by the MUFU (two results a term, 16 per clock
// and SM); the phase is always reduced mod 1, so __sincosf stays at its
// 3.5e-7 absolute error.
__global__ void __launch_bounds__(256) mk_node_leaf_kernel(const MkNodeArgs A, const int *__restrict__ list,
                                                           const int *__restrict__ rows,
                                                           const MkNodeRec *__restrict__ rec,
                                                           long long n_nodes, float2 *__restrict__ V)
{
    extern __shared__ __align__(16) unsigned char leaf_smem[];
    const int T = A.tile_atoms;
    float4 *s_pos = reinterpret_cast<float4 *>(leaf_smem);
    float4 *s_amp = s_pos + T;
    const int t = list[blockIdx.x];
    const float4 *gp = A.tpos + (size_t)t * T;
    const float4 *ga = reinterpret_cast<const float4 *>(A.tamp + (size_t)t * T);
    for (int i = threadIdx.x; i < T; i += blockDim.x) s_pos[i] = gp[i];
    for (int i = threadIdx.x; i < T / 2; i += blockDim.x) s_amp[i] = ga[i];
    __syncthreads();
    const long long g = (long long)blockIdx.y * blockDim.x + threadIdx.x;
    if (g >= n_nodes) return;
    const double4 o = A.origin[t];
    const float ox = (float)o.x, oy = (float)o.y, oz = (float)o.z;
    const float4 w4 = rec[g].w, u4 = rec[g].u;
    const float uo = fmaf(u4.z, oz, fmaf(u4.y, oy, u4.x * ox));
    // w = b - u', u' the direction from the tile's origin
    const mk_f2 wx = f2_splat(fmaf(ox - uo * u4.x, w4.w, w4.x));
    const mk_f2 wy = f2_splat(fmaf(oy - uo * u4.y, w4.w, w4.y));
    const mk_f2 wz = f2_splat(fmaf(oz - uo * u4.z, w4.w, w4.z));
    const mk_f2 magic = f2_splat(MK_ROUND_MAGIC), two_pi = f2_splat(TWO_PI_F), m_one = f2_splat(-1.f);
    mk_f2 ar = 0ull, ai = 0ull;
    const ulonglong2 *P2 = reinterpret_cast<const ulonglong2 *>(s_pos);
    const ulonglong2 *E2 = reinterpret_cast<const ulonglong2 *>(s_amp);
    const bool fr = A.fresnel && (float)o.w > A.fres_r;
    mk_f2 bx = 0ull, by = 0ull, bz = 0ull, hq = 0ull;
    if (fr) {
        bx = f2_splat(u4.w);
        by = f2_splat(rec[g].qh.w);
        bz = f2_splat(rec[g].ql.w);
        hq = f2_splat(0.5f * w4.w / (A.kappa * fmaf(-uo, w4.w, 1.f)));
    }
#pragma unroll 4
    for (int p = 0; p < T / 2; ++p) {
        const ulonglong2 a = P2[2 * p], b = P2[2 * p + 1], e = E2[p];
        mk_f2 lin = f2_fma(b.x, wz, f2_fma(a.y, wy, f2_mul(a.x, wx)));
        if (fr) {
            const mk_f2 sp = f2_sub(f2_fma(b.x, bz, f2_fma(a.y, by, f2_mul(a.x, bx))), lin);
            lin = f2_fma(f2_fma(f2_mul(sp, m_one), sp, b.y), hq, lin);
        }
        const float2 r = f2_unpack(f2_mul(f2_sub(lin, f2_sub(f2_add(lin, magic), magic)), two_pi));
        float s0, c0, s1, c1;
        __sincosf(r.x, &s0, &c0);
        __sincosf(r.y, &s1, &c1);
        const mk_f2 c = f2_pack(c0, c1), s = f2_pack(s0, s1);
        ar = f2_fma(e.x, c, f2_fma(f2_mul(e.y, m_one), s, ar));
        ai = f2_fma(e.x, s, f2_fma(e.y, c, ai));
    }
    const float2 r2 = f2_unpack(ar), i2 = f2_unpack(ai);
    V[(long long)(rows ? rows[blockIdx.x] : (int)blockIdx.x) * n_nodes + g] = make_float2(mk_unshort(r2.x + r2.y), mk_unshort(i2.x + i2.y));
}

// A tile's field on its coarse nodes by way of its eighths (64 atoms, a
// stretch of the Hilbert curve): each on NS x NS nodes of the same patch
// relative to the centre of its own box, then interpolated to the tile's
// N0 x N0 nodes times exp(2 pi i w.centre) and added. A block is a (tile,
// coarse patch). An eighth wider than its nodes take (and every eighth of a
// tile that keeps the |d|^2 term) is added term by term at the tile's nodes.
// NS^2 terms an atom instead of N0^2: still bound by the MUFU. 10,321 tiles
// on four 20 x 20 node patches 3.88 ms directly, 2.07 so; 15,814 on one of 16 x 16
// 0.95 and 0.56 (all of them on 14 x 14 and 12 x 12 nodes: 2.78 and 0.74).
struct MkSubArgs {
    const int *list, *rows;              // tiles and the rows of their fields
    const MkNodeRec *rec;                // the eighths' nodes
    const float *w;                      // from those to the tile's, (N0, NS)
    float radius;                        // widest eighth [cycles]
    int patches;                         // of a block
};
// Threads: 96 for the 288 nodes of 6 x 6 (a thread one: 603 us for 64 frames; two
// 639), else 256, a thread two nodes (5.3M atoms on 12 x 12 and 14 x 14: 2.32 ->
// 2.07 ms). Blocks that the node count divides into (224, 288, 416) hold fewer
// warps an SM and were 1 to 25 % slower.
__host__ __device__ constexpr int mk_leaf8_threads(int ns) { return ns == 6 ? 96 : 256; }
// Sum of atom pairs' terms at direction w [cycles], phases relative to lin0, two
// atoms a packed instruction.
struct MkLeafSum {
    mk_f2 wx, wy, wz, l0, re, im;
    MkLeafSum() = default;
    __device__ __forceinline__ MkLeafSum(const float3 &w, float lin0)
        : wx(f2_splat(w.x)), wy(f2_splat(w.y)), wz(f2_splat(w.z)), l0(f2_splat(-lin0)), re(0ull), im(0ull) {}
    __device__ __forceinline__ void add(const ulonglong2 &a, const ulonglong2 &b, const ulonglong2 &e)
    {
        const mk_f2 magic = f2_splat(MK_ROUND_MAGIC), two_pi = f2_splat(TWO_PI_F), m_one = f2_splat(-1.f);
        const mk_f2 lin = f2_fma(b.x, wz, f2_fma(a.y, wy, f2_fma(a.x, wx, l0)));
        const float2 r = f2_unpack(f2_mul(f2_sub(lin, f2_sub(f2_add(lin, magic), magic)), two_pi));
        float s0, c0, s1, c1;
        __sincosf(r.x, &s0, &c0);
        __sincosf(r.y, &s1, &c1);
        const mk_f2 c = f2_pack(c0, c1), s = f2_pack(s0, s1);
        re = f2_fma(e.x, c, f2_fma(f2_mul(e.y, m_one), s, re));
        im = f2_fma(e.x, s, f2_fma(e.y, c, im));
    }
    __device__ __forceinline__ float2 sum() const
    {
        const float2 r = f2_unpack(re), i = f2_unpack(im);
        return make_float2(mk_unshort(r.x + r.y), mk_unshort(i.x + i.y));
    }
};

template <int N0, int NS>
__global__ void __launch_bounds__(mk_leaf8_threads(NS)) mk_node_leaf8_kernel(const MkNodeArgs A, const MkSubArgs B,
                                                                             const MkNodeRec *__restrict__ rec,
                                                                             long long n_nodes,
                                                                             float2 *__restrict__ V)
{
    constexpr int SQ = NS * NS, NT = mk_leaf8_threads(NS), RW = N0 % 4 == 0 ? 4 : 2, ND = NS == 6 ? 1 : 2;
    extern __shared__ __align__(16) unsigned char leaf_smem[];
    const int T = A.tile_atoms, pairs = T / 16;          // atom pairs of an eighth
    float4 *s_pos = reinterpret_cast<float4 *>(leaf_smem);
    float4 *s_amp = s_pos + T;
    float2 *s_v = reinterpret_cast<float2 *>(s_amp + T / 2);        // [8][SQ]
    float2 *s_t = s_v + 8 * SQ;                                     // [8][N0][NS]
    float *s_w = reinterpret_cast<float *>(s_t + 8 * N0 * NS);      // [NS][N0]
    __shared__ float4 s_c[8];                            // centre; 1 where the eighth has nodes
    const int t = B.list[blockIdx.x];
    const float4 *gp = A.tpos + (size_t)t * T;
    const float4 *ga = reinterpret_cast<const float4 *>(A.tamp + (size_t)t * T);
    for (int i = threadIdx.x; i < T; i += NT) s_pos[i] = gp[i];
    for (int i = threadIdx.x; i < T / 2; i += NT) s_amp[i] = ga[i];
    for (int i = threadIdx.x; i < N0 * NS; i += NT) s_w[i % NS * N0 + i / NS] = B.w[i];
    __syncthreads();
    const double4 o = A.origin[t];
    const float ox = (float)o.x, oy = (float)o.y, oz = (float)o.z;
    const bool fr = A.fresnel && (float)o.w > A.fres_r;
    for (int s = threadIdx.x >> 5; s < 8; s += NT / 32) {
        const int lane = threadIdx.x & 31;
        float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
        for (int p = s * pairs + lane; p < (s + 1) * pairs; p += 32) {
            const float4 a = s_pos[2 * p], b = s_pos[2 * p + 1];    // x0 x1 y0 y1, z0 z1
            lo[0] = fminf(lo[0], fminf(a.x, a.y)); hi[0] = fmaxf(hi[0], fmaxf(a.x, a.y));
            lo[1] = fminf(lo[1], fminf(a.z, a.w)); hi[1] = fmaxf(hi[1], fmaxf(a.z, a.w));
            lo[2] = fminf(lo[2], fminf(b.x, b.y)); hi[2] = fmaxf(hi[2], fmaxf(b.x, b.y));
        }
        float c[3], r2 = 0.f;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            for (int w = 16; w > 0; w >>= 1) {
                lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], w));
                hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], w));
            }
            c[d] = 0.5f * (lo[d] + hi[d]);
        }
        for (int p = s * pairs + lane; p < (s + 1) * pairs; p += 32) {
            const float4 a = s_pos[2 * p], b = s_pos[2 * p + 1];
            const float x0 = a.x - c[0], y0 = a.z - c[1], z0 = b.x - c[2];
            const float x1 = a.y - c[0], y1 = a.w - c[1], z1 = b.y - c[2];
            r2 = fmaxf(r2, fmaxf(fmaf(z0, z0, fmaf(y0, y0, x0 * x0)), fmaf(z1, z1, fmaf(y1, y1, x1 * x1))));
        }
        for (int w = 16; w > 0; w >>= 1) r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, w));
        if (lane == 0)
            s_c[s] = make_float4(c[0], c[1], c[2], !fr && r2 <= B.radius * B.radius ? 1.f : 0.f);
    }
    __syncthreads();
    const ulonglong2 *P2 = reinterpret_cast<const ulonglong2 *>(s_pos);
    const ulonglong2 *E2 = reinterpret_cast<const ulonglong2 *>(s_amp);
    // pairs [p0, p1) at direction w
    auto terms = [&](int p0, int p1, const float3 &w) {
        MkLeafSum a(w, 0.f);
#pragma unroll 4
        for (int p = p0; p < p1; ++p) a.add(P2[2 * p], P2[2 * p + 1], E2[p]);
        return a.sum();
    };
    // w = b - u', u' the direction from the tile's origin
    auto direction = [&](const float4 &w4, const float4 &u4) {
        const float uo = fmaf(u4.z, oz, fmaf(u4.y, oy, u4.x * ox));
        return make_float3(fmaf(ox - uo * u4.x, w4.w, w4.x), fmaf(oy - uo * u4.y, w4.w, w4.y),
                           fmaf(oz - uo * u4.z, w4.w, w4.z));
    };
    const int patches = (int)(n_nodes / (N0 * N0)), p_end = min((int)(blockIdx.y + 1) * B.patches, patches);
    for (int patch = blockIdx.y * B.patches; patch < p_end; ++patch) {
        const MkNodeRec *rs = B.rec + (long long)patch * SQ;
        // ND nodes a thread: an atom pair's 48 bytes from shared memory serve them all
        for (int i = threadIdx.x; i < 8 * (SQ / ND); i += NT) {
            const int s = i / (SQ / ND), q = i - s * (SQ / ND);
            const float4 c = s_c[s];
            float2 *v = s_v + s * SQ + q;
            if (c.w == 0.f) {
#pragma unroll
                for (int k = 0; k < ND; ++k) v[k * (SQ / ND)] = make_float2(0.f, 0.f);
                continue;
            }
            MkLeafSum a[ND];
#pragma unroll
            for (int k = 0; k < ND; ++k) {
                const MkNodeRec &R = rs[q + k * (SQ / ND)];
                const float3 w = direction(R.w, R.u);
                a[k] = MkLeafSum(w, fmaf(c.z, w.z, fmaf(c.y, w.y, c.x * w.x)));
            }
#pragma unroll 4 / ND
            for (int p = s * pairs; p < (s + 1) * pairs; ++p) {
                const ulonglong2 xy = P2[2 * p], z = P2[2 * p + 1], e = E2[p];
#pragma unroll
                for (int k = 0; k < ND; ++k) a[k].add(xy, z, e);
            }
#pragma unroll
            for (int k = 0; k < ND; ++k) v[k * (SQ / ND)] = a[k].sum();
        }
        __syncthreads();
        // along z: RW rows a thread share the eighth's column and read their weights at once
        for (int i = threadIdx.x; i < 8 * (N0 / RW) * NS; i += NT) {
            const int s = i / (N0 / RW * NS), r = i - s * (N0 / RW * NS), row = r / NS * RW, c = r % NS;
            mk_f2 a[RW];
#pragma unroll
            for (int k = 0; k < RW; ++k) a[k] = 0ull;
#pragma unroll
            for (int j = 0; j < NS; ++j) {
                alignas(16) float w[RW];
                if constexpr (RW == 4)
                    *reinterpret_cast<float4 *>(w) = *reinterpret_cast<const float4 *>(s_w + j * N0 + row);
                else
                    *reinterpret_cast<float2 *>(w) = *reinterpret_cast<const float2 *>(s_w + j * N0 + row);
                const mk_f2 v = *reinterpret_cast<const mk_f2 *>(&s_v[s * SQ + j * NS + c]);
#pragma unroll
                for (int k = 0; k < RW; ++k) a[k] = f2_fma(f2_splat(w[k]), v, a[k]);
            }
#pragma unroll
            for (int k = 0; k < RW; ++k) *reinterpret_cast<mk_f2 *>(&s_t[(s * N0 + row + k) * NS + c]) = a[k];
        }
        __syncthreads();
        const MkNodeRec *rn = rec + (long long)patch * N0 * N0;
        float2 *out = V + (long long)B.rows[blockIdx.x] * n_nodes + (long long)patch * N0 * N0;
        for (int g = threadIdx.x; g < N0 * N0; g += NT) {
            const int row = g / N0, col = g - row * N0;
            const float4 w4 = rn[g].w, u4 = rn[g].u;
            const float3 w = direction(w4, u4);
            float re = 0.f, im = 0.f, wy[NS];
#pragma unroll
            for (int i = 0; i < NS; ++i) wy[i] = s_w[i * N0 + col];
            for (int s = 0; s < 8; ++s) {
                const float4 c = s_c[s];
                if (c.w == 0.f) {               // uniform across the block
                    float2 v;
                    if (fr) {
                        // the |d|^2 term: 1 / (2 kappa |P - o|), db = D.b
                        const float uo = fmaf(u4.z, oz, fmaf(u4.y, oy, u4.x * ox));
                        const float hq = 0.5f * w4.w / (A.kappa * fmaf(-uo, w4.w, 1.f));
                        const float bx = u4.w, by = rn[g].qh.w, bz = rn[g].ql.w;
                        v = make_float2(0.f, 0.f);
                        for (int p = s * pairs; p < (s + 1) * pairs; ++p) {
                            MkAtom m[2];
                            mk_atom_pair(s_pos, s_amp, p, m[0], m[1]);
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const float4 a = m[h].a;
                                float lin = fmaf(a.z, w.z, fmaf(a.y, w.y, a.x * w.x));
                                const float sp = fmaf(a.z, bz, fmaf(a.y, by, a.x * bx)) - lin;
                                lin = fmaf(fmaf(-sp, sp, a.w), hq, lin);
                                float sn, cs;
                                __sincosf(mk_frac_nearest(lin) * TWO_PI_F, &sn, &cs);
                                v.x += m[h].e.x * cs - m[h].e.y * sn;
                                v.y += m[h].e.x * sn + m[h].e.y * cs;
                            }
                        }
                        v = make_float2(mk_unshort(v.x), mk_unshort(v.y));
                    } else {
                        v = terms(s * pairs, (s + 1) * pairs, w);
                    }
                    re += v.x;
                    im += v.y;
                    continue;
                }
                mk_f2 v = 0ull;
                const ulonglong2 *t2 = reinterpret_cast<const ulonglong2 *>(s_t + (s * N0 + row) * NS);
#pragma unroll
                for (int i = 0; i < NS / 2; ++i) {
                    const ulonglong2 tt = t2[i];
                    v = f2_fma(f2_splat(wy[2 * i]), tt.x, v);
                    v = f2_fma(f2_splat(wy[2 * i + 1]), tt.y, v);
                }
                float sn, cs;
                __sincosf(mk_frac_nearest(fmaf(c.z, w.z, fmaf(c.y, w.y, c.x * w.x))) * TWO_PI_F, &sn, &cs);
                const float2 vv = f2_unpack(v);
                re += mk_unshort(vv.x * cs - vv.y * sn);
                im += mk_unshort(vv.x * sn + vv.y * cs);
            }
            out[g] = make_float2(re, im);
        }
    }       // s_v is written again only after every thread has left the reads of s_t's making
}

__device__ __forceinline__ void mk_cp16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(mk_smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void mk_cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void mk_cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// q.d in cycles, mod 1 per component: two-float products.
__device__ __forceinline__ float mk_dot_frac(float3 qh, float3 ql, float3 dh, float3 dl)
{
    const float px = qh.x * dh.x, py = qh.y * dh.y, pz = qh.z * dh.z;
    float lo = fmaf(qh.x, dh.x, -px) + fmaf(qh.y, dh.y, -py) + fmaf(qh.z, dh.z, -pz);
    lo = fmaf(qh.x, dl.x, fmaf(ql.x, dh.x, lo));
    lo = fmaf(qh.y, dl.y, fmaf(ql.y, dh.y, lo));
    lo = fmaf(qh.z, dl.z, fmaf(ql.z, dh.z, lo));
    return (mk_frac_nearest(px) + mk_frac_nearest(py)) + (mk_frac_nearest(pz) + lo);
}

// acc += v (Kahan: c carries what the sum's last bit lost).
__device__ __forceinline__ void mk_kahan(float v, float &acc, float &c)
{
    const float y = __fsub_rn(v, c), z = __fadd_rn(acc, y);
    c = __fsub_rn(__fsub_rn(z, acc), y);
    acc = z;
}

// Sources s0 .. s0 + SB - 1's patch fields into shared memory (16-byte
// chunks: n^2 even).
template <int N>
__device__ __forceinline__ void mk_stage_fields(float2 (*s_v)[N * N], const float2 *V, long long ld,
                                                long long s0, int count)
{
    constexpr int CH = N * N / 2;
    for (int i = threadIdx.x; i < count * CH; i += blockDim.x) {
        const int s = i / CH, c = i - s * CH;
        mk_cp16(&s_v[s][2 * c], V + (s0 + s) * ld + 2 * c);
    }
}

// Merge: block = (group, strip of neighbouring fine patches, rows of their
// nodes); a thread one node column of the strip and ROWS rows. The group's
// tiles come SB at a time: first the interpolation along z to the block's
// rows, which all the strip's columns share, then along y per node. Bound by
// the FMA pipe: 2 N0 + ~47 FP32 operations a (tile, fine node), N0 from the
// interpolation along y. With one fine patch a block (the z interpolation,
// N0^2 / n1 packed FMAs a node, made again for every patch of a row) it took
// 6.72 ms for N0 = 20, n1 = 12 on the 1024 x 1024 detector and 1.46 ms for N0 =
// 16 on the 512 x 512 one; here 2.34 and 0.70 ms (4.5 and 5.2 ps a (tile, fine
// node)). Six or eight sources a step instead of four: 0.44 -> 0.42 ms for 15,814 tiles
// into runs on 16 x 16 middle nodes (at N0 = 20 slower).
template <int N0, int ROWS>
__global__ void __launch_bounds__(MK_MERGE_NT) mk_node_merge_kernel(const MkMergeArgs A)
{
    constexpr int SB = MK_NODE_SB(N0);
    constexpr int MAXR = 16;                 // rows of a block at most
    __shared__ __align__(16) float2 s_v[2][SB][N0 * N0];
    __shared__ __align__(16) float2 s_t[SB][MAXR][N0];
    __shared__ float s_wz[MAXR][N0];
    __shared__ __align__(16) float s_d[2][SB][8];
    const long long it = A.item_base + blockIdx.x % A.items;
    const int grp = (int)(blockIdx.x / A.items);
    const int n1 = A.n_out;
    const int f = mk_find_frame(A.f_lo, A.f_hi, it, [&](int i) { return A.frames[i].mg[A.step].item_off; });
    const MkNodeFrame &F = A.frames[f];
    const MkNodeMerge &M = F.mg[A.step];
    int e = (int)(it - M.item_off);
    const int chunk = e % M.chunks;
    e /= M.chunks;
    const int strip = e % M.strips;
    e /= M.strips;
    const int p0y = F.py[A.in], p1y = F.py[A.to];
    const int cy = e % p0y, pz = e / p0y;
    const int suby0 = strip * M.strip;
    const int patches = min(min(M.strip, M.ratio_y - suby0), p1y - (cy * M.ratio_y + suby0));
    if (patches <= 0) return;                // a last coarse patch with fewer fine ones
    const int width = M.strip * n1;          // node columns of a full strip
    const int cz = pz / M.ratio_z, subz = pz - cz * M.ratio_z;
    const int rows = M.rowg * ROWS, row0 = chunk * rows;      // rows of this block
    const float *W = A.weights + M.w_off;
    const float *Wy = W + (long long)suby0 * n1 * N0, *Wz = W + (M.ratio_y + subz) * n1 * N0;
    const int nrow = min(rows, n1 - row0);
    for (int i = threadIdx.x; i < nrow * N0; i += MK_MERGE_NT) s_wz[i / N0][i % N0] = Wz[row0 * N0 + i];
    const int rg = threadIdx.x / width, oc = threadIdx.x - rg * width;
    const bool live = oc < patches * n1 && rg * ROWS < nrow && rg < M.rowg;
    const int oc1 = live ? oc : 0, lr = live ? rg * ROWS : 0;
    mk_f2 wy[N0];
#pragma unroll
    for (int i = 0; i < N0; ++i) wy[i] = f2_splat(Wy[oc1 * N0 + i]);
    const MkNodeSrc &S = A.src[grp];
    if (S.count == 0) return;                // a single tile: its leaf wrote its row
    const double gx = S.o[0], gy = S.o[1], gz = S.o[2];
    // the thread's nodes: patch of its column, rows lr .. lr + ROWS - 1
    const int py = cy * M.ratio_y + suby0 + oc1 / n1;
    const long long node = (F.off[A.to] - A.to_base + (long long)pz * p1y + py) * n1 * n1 +
                           (row0 + lr) * n1 + oc1 % n1;
    const MkNodeRec *rec = A.rec + A.to_base * n1 * n1 + node;
    float3 qh[ROWS], ql[ROWS], u[ROWS];
    float half[ROWS], accr[ROWS], acci[ROWS], cr[ROWS], ci[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {         // directions from the group's origin
        const MkNodeRec R = rec[r * n1];
        const float ox = (float)gx, oy = (float)gy, oz = (float)gz;
        qh[r] = make_float3(R.qh.x, R.qh.y, R.qh.z);
        u[r] = make_float3(R.u.x, R.u.y, R.u.z);
        const float uo = fmaf(u[r].z, oz, fmaf(u[r].y, oy, u[r].x * ox));
        const float kr = A.kappa * R.w.w;
        ql[r] = make_float3(fmaf(ox - uo * u[r].x, kr, R.ql.x), fmaf(oy - uo * u[r].y, kr, R.ql.y),
                            fmaf(oz - uo * u[r].z, kr, R.ql.z));
        half[r] = 0.5f * kr / fmaf(-uo, R.w.w, 1.f);
        accr[r] = acci[r] = cr[r] = ci[r] = 0.f;
    }
    const float2 *V = A.Vin + (F.off[A.in] - A.in_base + cz * p0y + cy) * N0 * N0;
    const long long first = S.first;
    const int count = S.count;
    auto stage = [&](int s0, int buf) {
        const int m = min(SB, count - s0);
        mk_stage_fields<N0>(s_v[buf], V, A.in_patches * N0 * N0, first + s0, m);
        mk_cp_commit();
        if ((int)threadIdx.x < m) {
            const long long j = first + s0 + threadIdx.x;
            const double4 o = A.origin[A.members ? A.members[j] : j];
            const double d[3] = {o.x - gx, o.y - gy, o.z - gz};
            float *sd = s_d[buf][threadIdx.x], dd = 0.f;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float h = (float)d[c];
                sd[c] = h;
                sd[4 + c] = (float)(d[c] - (double)h);
                dd = fmaf(h, h, dd);
            }
            sd[3] = dd;
        }
    };
    stage(0, 0);
    for (int s0 = 0, buf = 0; s0 < count; s0 += SB, buf ^= 1) {
        const int m = min(SB, count - s0);
        if (s0 + SB < count) {
            stage(s0 + SB, buf ^ 1);
            mk_cp_wait<1>();
        } else {
            mk_cp_wait<0>();
        }
        __syncthreads();
        for (int i = threadIdx.x; i < m * nrow * N0; i += MK_MERGE_NT) {
            const int s = i / (nrow * N0), r = i - s * nrow * N0, row = r / N0, c = r - row * N0;
            mk_f2 a = 0ull;
#pragma unroll
            for (int j = 0; j < N0; ++j)
                a = f2_fma(f2_splat(s_wz[row][j]), *reinterpret_cast<const mk_f2 *>(&s_v[buf][s][j * N0 + c]), a);
            *reinterpret_cast<mk_f2 *>(&s_t[s][row][c]) = a;
        }
        __syncthreads();
        if (live) {
            for (int s = 0; s < m; ++s) {
                const float4 d4 = *reinterpret_cast<const float4 *>(s_d[buf][s]);
                const float4 l4 = *reinterpret_cast<const float4 *>(s_d[buf][s] + 4);
                const float3 dh = make_float3(d4.x, d4.y, d4.z), dl = make_float3(l4.x, l4.y, l4.z);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    mk_f2 v = 0ull;
                    const ulonglong2 *t2 = reinterpret_cast<const ulonglong2 *>(s_t[s][lr + r]);
#pragma unroll
                    for (int i = 0; i < N0 / 2; ++i) {
                        const ulonglong2 t = t2[i];
                        v = f2_fma(wy[2 * i], t.x, v);
                        v = f2_fma(wy[2 * i + 1], t.y, v);
                    }
                    const float ud = fmaf(u[r].z, dh.z, fmaf(u[r].y, dh.y, u[r].x * dh.x));
                    float ph = fmaf(fmaf(-ud, ud, d4.w), half[r], mk_dot_frac(qh[r], ql[r], dh, dl));
                    ph = mk_frac_nearest(ph);
                    float sn, cs;
                    __sincosf(ph * TWO_PI_F, &sn, &cs);
                    const float2 vv = f2_unpack(v);
                    mk_kahan(vv.x * cs - vv.y * sn, accr[r], cr[r]);
                    mk_kahan(vv.x * sn + vv.y * cs, acci[r], ci[r]);
                }
            }
        }
        __syncthreads();        // s_d and s_t are read; the next step may stage
    }
    if (live) {
        float2 *out = A.Vout + (long long)grp * (A.to_patches * n1 * n1) + node;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) out[r * n1] = make_float2(mk_unshort(accr[r] - cr[r]), mk_unshort(acci[r] - ci[r]));
    }
}

// Pixels: block = (32 x 16 pixels of one fine patch, slice of sources), a
// thread one column and four rows. Sources come SB at a time as in the
// merge; bound by the FMA pipe (about 2 N + 45 FP32 operations a source and
// pixel).
template <int N>
__global__ void __launch_bounds__(128) mk_node_pixels_kernel(const MkNodeArgs A)
{
    constexpr int SB = MK_NODE_SB(N);
    __shared__ __align__(16) float2 s_v[2][SB][N * N];
    __shared__ __align__(16) float2 s_t[SB][MK_PIX_ROWS][N];
    __shared__ float s_wz[MK_PIX_ROWS][N];
    const long long blk = A.pblk_base + blockIdx.x;
    const int f = mk_find_frame(A.f_lo, A.f_hi, blk, [&](int i) { return A.frames[i].pblk_off; });
    const MkNodeFrame &F = A.frames[f];
    const int per = F.bpy * F.bpz;
    const int lb = (int)(blk - F.pblk_off), lp = lb / per, sub = lb - lp * per;
    const int p1y = F.py[MK_FINE], l1y = F.ly[MK_FINE], l1z = F.lz[MK_FINE];
    const int pz = lp / p1y, py = lp - pz * p1y, bz = sub / F.bpy, by = sub - bz * F.bpy;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int col_end = min((py + 1) * l1y, F.ny), row_end = min((pz + 1) * l1z, F.nz);
    const int col = py * l1y + by * MK_PIX_COLS + lane;
    const int row0 = pz * l1z + bz * MK_PIX_ROWS;
    if (row0 >= row_end || py * l1y + by * MK_PIX_COLS >= col_end) return;   // whole block outside
    const float *Wy = A.weights + F.w_off, *Wz = Wy + (long long)N * F.ny;
    for (int i = threadIdx.x; i < MK_PIX_ROWS * N; i += blockDim.x)
        s_wz[i / N][i % N] = Wz[(long long)min(row0 + i / N, row_end - 1) * N + i % N];
    const int c0 = min(col, col_end - 1);
    mk_f2 wy[N];
#pragma unroll
    for (int i = 0; i < N; ++i) wy[i] = f2_splat(Wy[(long long)c0 * N + i]);
    float3 qh[4], ql[4], u[4];
    float inv[4];
    float accr[4], acci[4], cr[4], ci[4], tr[4], ti[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const long long g = F.pix_off + (long long)min(row0 + 4 * warp + r, row_end - 1) * F.ny + c0;
        const double4 q = A.q[g];
        const float4 uu = A.u[g];
        qh[r] = make_float3((float)q.x, (float)q.y, (float)q.z);
        ql[r] = make_float3((float)(q.x - (double)qh[r].x), (float)(q.y - (double)qh[r].y),
                            (float)(q.z - (double)qh[r].z));
        u[r] = make_float3(uu.x, uu.y, uu.z);
        inv[r] = uu.w;
        accr[r] = acci[r] = cr[r] = ci[r] = tr[r] = ti[r] = 0.f;
    }
    const int s_lo = blockIdx.y * A.src_per_slice, s_hi = min(A.n_src, s_lo + A.src_per_slice);
    const long long ld = A.patches1 * N * N;
    const float2 *V = A.V1 + (F.off[MK_FINE] - A.patch1_base + lp) * N * N;
    int species = A.src[s_lo].species;
    auto flush = [&](int s) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const long long g = F.pix_off + (long long)min(row0 + 4 * warp + r, row_end - 1) * F.ny + c0;
            const float2 fc = A.ftab[(long long)s * A.ftab_n + g];
            const float xr = mk_unshort(accr[r] - cr[r]), xi = mk_unshort(acci[r] - ci[r]);
            tr[r] += fc.x * xr - fc.y * xi;
            ti[r] += fc.x * xi + fc.y * xr;
            accr[r] = acci[r] = cr[r] = ci[r] = 0.f;
        }
    };
    mk_stage_fields<N>(s_v[0], V, ld, s_lo, min(SB, s_hi - s_lo));
    mk_cp_commit();
    for (int s0 = s_lo, buf = 0; s0 < s_hi; s0 += SB, buf ^= 1) {
        const int m = min(SB, s_hi - s0);
        if (s0 + SB < s_hi) {
            mk_stage_fields<N>(s_v[buf ^ 1], V, ld, s0 + SB, min(SB, s_hi - s0 - SB));
            mk_cp_commit();
            mk_cp_wait<1>();
        } else {
            mk_cp_wait<0>();
        }
        __syncthreads();
        for (int i = threadIdx.x; i < m * MK_PIX_ROWS * N; i += blockDim.x) {
            const int s = i / (MK_PIX_ROWS * N), e = i - s * MK_PIX_ROWS * N, row = e / N, c = e - row * N;
            mk_f2 a = 0ull;
#pragma unroll
            for (int j = 0; j < N; ++j)
                a = f2_fma(f2_splat(s_wz[row][j]), *reinterpret_cast<const mk_f2 *>(&s_v[buf][s][j * N + c]), a);
            *reinterpret_cast<mk_f2 *>(&s_t[s][row][c]) = a;
        }
        __syncthreads();
        for (int s = 0; s < m; ++s) {
            const float4 h4 = *reinterpret_cast<const float4 *>(A.src[s0 + s].dh);
            const float4 l4 = *reinterpret_cast<const float4 *>(A.src[s0 + s].dl);
            const int sp = __float_as_int(h4.w);
            if (sp != species) {            // uniform across the block
                flush(species);
                species = sp;
            }
            const float3 dh = make_float3(h4.x, h4.y, h4.z), dl = make_float3(l4.x, l4.y, l4.z);
            const float dd = fmaf(dh.z, dh.z, fmaf(dh.y, dh.y, dh.x * dh.x));
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                mk_f2 v = 0ull;
                const ulonglong2 *t2 = reinterpret_cast<const ulonglong2 *>(s_t[s][4 * warp + r]);
#pragma unroll
                for (int i = 0; i < N / 2; ++i) {
                    const ulonglong2 t = t2[i];
                    v = f2_fma(wy[2 * i], t.x, v);
                    v = f2_fma(wy[2 * i + 1], t.y, v);
                }
                const float ud = fmaf(u[r].z, dh.z, fmaf(u[r].y, dh.y, u[r].x * dh.x));
                float ph = fmaf(fmaf(-ud, ud, dd), 0.5f * A.kappa * inv[r], mk_dot_frac(qh[r], ql[r], dh, dl));
                ph = mk_frac_nearest(ph);
                float sn, cs;
                __sincosf(ph * TWO_PI_F, &sn, &cs);
                if (A.decay) {
                    const float dr = 1.f / fmaf(-ud, inv[r], 1.f);
                    sn *= dr;
                    cs *= dr;
                }
                const float2 vv = f2_unpack(v);
                mk_kahan(vv.x * cs - vv.y * sn, accr[r], cr[r]);
                mk_kahan(vv.x * sn + vv.y * cs, acci[r], ci[r]);
            }
        }
        __syncthreads();
    }
    flush(species);
    if (col >= col_end) return;
    const long long n_pix = (long long)F.ny * F.nz;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int row = row0 + 4 * warp + r;
        if (row < row_end)
            A.partial[F.part_off - A.part_base + blockIdx.y * n_pix + (long long)row * F.ny + col] =
                make_double2((double)tr[r], (double)ti[r]);
    }
}

// out[g] (+)= r_e phasor[g] sum over slices (FP64, fixed order).
__global__ void mk_node_reduce_kernel(const MkNodeFrame *__restrict__ frames, int f_lo, int f_hi,
                                      long long g0, long long n, int slices, long long part_base,
                                      const double2 *__restrict__ partial,
                                      const double2 *__restrict__ phasor, double2 *__restrict__ out,
                                      int accumulate)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long g = g0 + i;
    const int f = mk_find_frame(f_lo, f_hi, g, [&](int j) { return frames[j].pix_off; });
    const long long n_pix = (long long)frames[f].ny * frames[f].nz;
    const double2 *p = partial + (frames[f].part_off - part_base) + (g - frames[f].pix_off);
    double re = 0.0, im = 0.0;
    for (int s = 0; s < slices; ++s) {
        const double2 v = p[s * n_pix];
        re += v.x;
        im += v.y;
    }
    const double2 e = phasor[g];
    double2 o = make_double2(MK_R_E * (re * e.x - im * e.y), MK_R_E * (re * e.y + im * e.x));
    if (accumulate) {
        o.x += out[g].x;
        o.y += out[g].y;
    }
    out[g] = o;
}

// sums[f] = sum of |A|^2 over the frame's pixels: MK_SUM_PARTS fixed chunks a
// frame, each a fixed-order tree, then the chunks in order.
__global__ void __launch_bounds__(256) mk_node_sums_kernel(const MkNodeFrame *__restrict__ frames,
                                                           const double2 *__restrict__ field,
                                                           double *__restrict__ parts)
{
    __shared__ double red[256];
    const MkNodeFrame &F = frames[blockIdx.x];
    const long long n = (long long)F.ny * F.nz, step = (n + MK_SUM_PARTS - 1) / MK_SUM_PARTS;
    const long long lo = blockIdx.y * step, hi = min(n, lo + step);
    double acc = 0.0;
    for (long long p = lo + threadIdx.x; p < hi; p += 256) {
        const double2 v = field[F.pix_off + p];
        acc += v.x * v.x + v.y * v.y;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) parts[(long long)blockIdx.x * MK_SUM_PARTS + blockIdx.y] = red[0];
}

__global__ void mk_node_sums_final_kernel(int n_frames, const double *__restrict__ parts,
                                          double *__restrict__ sums)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_frames) return;
    double acc = 0.0;
    for (int i = 0; i < MK_SUM_PARTS; ++i) acc += parts[(long long)f * MK_SUM_PARTS + i];
    sums[f] = acc;
}

// ------------------------------------------------------- top-hat analyser
// Every atom's direction to a pixel is within `exc` of the pixel's own, so x =
// |u' - c|^2 is within 2 sqrt(x) exc + exc^2 of the pixel's: a pixel whose own
// x is farther than that from the acceptance edge takes one factor, 0 or 1,
// for every atom, which its factor-table entries carry; the others (the edge
// passes them within 1e-7 rad: a few of a detector) are zeroed and listed for
// the split kernel's per-atom test. FP64, one pass: 24 B read, 16 B a species.
__global__ void __launch_bounds__(256) mk_analyser_mask_kernel(long long n, const double *__restrict__ xyz,
                                                               double cx, double cy, double cz, double x_acc,
                                                               double exc, int n_species,
                                                               const float2 *__restrict__ in,
                                                               float2 *__restrict__ out,
                                                               int *__restrict__ edge, int cap)
{
    const long long p = (long long)blockIdx.x * 256 + threadIdx.x;
    if (p >= n) return;
    const double x0 = xyz[3 * p], y0 = xyz[3 * p + 1], z0 = xyz[3 * p + 2];
    const double inv = 1.0 / sqrt(x0 * x0 + y0 * y0 + z0 * z0);
    const double vx = x0 * inv - cx, vy = y0 * inv - cy, vz = z0 * inv - cz;
    const double x = vx * vx + vy * vy + vz * vz, m = 2.0 * sqrt(x) * exc + exc * exc + 1e-15;
    const bool inside = x + m <= x_acc, outside = x - m > x_acc;
    for (int s = 0; s < n_species; ++s)
        out[s * n + p] = inside ? in[s * n + p] : make_float2(0.f, 0.f);
    if (!inside && !outside) {          // NaN too
        const int i = atomicAdd(edge, 1);
        if (i < cap) edge[1 + i] = (int)p;
    }
}

extern "C" int mk_analyser_mask(const mk_pixels *px, const mk_physics *phys, double excursion, int n_species,
                                float *factor_out, int *edge, int edge_cap, void *stream)
{
    MK_REQUIRE(px && phys && px->xyz && px->factor && factor_out && edge && edge_cap >= 0 && n_species >= 1 &&
                   excursion >= 0.0,
               "mk_analyser_mask: bad arguments");
    MK_REQUIRE(phys->analyser == 1, "mk_analyser_mask: a top-hat analyser is needed");
    int kind;
    double ax, ay, az, xacc, hw;
    const int rc = mk_analyser_pack(phys, &kind, &ax, &ay, &az, &xacc, &hw);
    if (rc != MK_OK) return rc;
    const long long n = (long long)px->ny * px->nz;
    cudaStream_t st = mk_stream(stream);
    MK_CHECK_CUDA(cudaMemsetAsync(edge, 0, sizeof(int), st));
    mk_analyser_mask_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(
        n, px->xyz, ax, ay, az, xacc, excursion, n_species, reinterpret_cast<const float2 *>(px->factor),
        reinterpret_cast<float2 *>(factor_out), edge, edge_cap);
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

template <int N>
static void mk_launch_pixels(const MkNodeArgs &A, dim3 grid, cudaStream_t st)
{
    mk_node_pixels_kernel<N><<<grid, 128, 0, st>>>(A);
}
template <int N>
static void mk_launch_merge(const MkMergeArgs &A, unsigned grid, cudaStream_t st)
{
    switch (merge_rows(A.n_out)) {
    case 3: mk_node_merge_kernel<N, 3><<<grid, MK_MERGE_NT, 0, st>>>(A); break;
    case 4: mk_node_merge_kernel<N, 4><<<grid, MK_MERGE_NT, 0, st>>>(A); break;
    default: mk_node_merge_kernel<N, 5><<<grid, MK_MERGE_NT, 0, st>>>(A); break;
    }
}
static int mk_merge(const MkMergeArgs &A, int n_in, int n_runs, cudaStream_t st)
{
    const unsigned grid = (unsigned)(A.items * n_runs);
    switch (n_in) {
    case 8: mk_launch_merge<8>(A, grid, st); break;
    case 10: mk_launch_merge<10>(A, grid, st); break;
    case 12: mk_launch_merge<12>(A, grid, st); break;
    case 16: mk_launch_merge<16>(A, grid, st); break;
    case 20: mk_launch_merge<20>(A, grid, st); break;
    default: mk_set_error("mk_kin_nodes_f32: %d nodes to merge", n_in); return MK_EINVAL;
    }
    return MK_OK;
}

// A tile's atoms in shared memory. The kernels' limit is set to that of the
// largest tiles with every launch: threads with smaller ones must not lower it
// between another's setting it and its launch.
#define MK_TILE_ATOMS_MAX 4096
static size_t leaf_bytes(int tile_atoms) { return (size_t)tile_atoms * 24; }

template <int N0, int NS>
static int mk_launch_leaf8(const MkNodeArgs &A, MkSubArgs B, int n_list, const MkNodeRec *rec,
                           long long nodes, float2 *V, int sms, cudaStream_t st)
{
    const size_t fixed = 8 * 8 * (size_t)NS * (NS + N0) + 4 * (size_t)N0 * NS, smem = leaf_bytes(A.tile_atoms) + fixed;
    auto fn = mk_node_leaf8_kernel<N0, NS>;
    MK_CHECK_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(leaf_bytes(MK_TILE_ATOMS_MAX) + fixed)));
    // a block's patches share its tile's atoms and boxes; 16 blocks an SM first
    const int patches = (int)(nodes / (N0 * N0));
    B.patches = (int)std::max<long long>(1, std::min<long long>(8, (long long)n_list * patches / (16ll * sms)));
    fn<<<dim3(n_list, (patches + B.patches - 1) / B.patches), mk_leaf8_threads(NS), smem, st>>>(A, B, rec, nodes, V);
    return MK_OK;
}

extern "C" int mk_kin_nodes_f32(const mk_tiles *tiles, const mk_physics *phys, const mk_pixels *px,
                                const mk_node_plan *plan, const void *host_buf, const void *dev_buf,
                                int fresnel, double fresnel_radius_m, double *out, double *intensity_sums,
                                int accumulate, void *workspace, size_t ws_bytes, void *stream)
{
    MK_REQUIRE(tiles && phys && px && plan && host_buf && dev_buf && out, "mk_kin_nodes_f32: null argument");
    MK_REQUIRE(px->xyz && px->q && px->u && px->phasor && px->factor,
               "mk_kin_nodes_f32: pixels not prepared, or no factor table");
    MK_REQUIRE(tiles->origin && tiles->pos && tiles->amp && tiles->n_tiles == plan->n_tiles,
               "mk_kin_nodes_f32: the tiles are not the plan's");
    MK_REQUIRE(((uintptr_t)tiles->pos & 15) == 0 && ((uintptr_t)tiles->amp & 15) == 0 &&
                   ((uintptr_t)workspace & 255) == 0 && ((uintptr_t)dev_buf & 15) == 0,
               "mk_kin_nodes_f32: misaligned buffer");
    MK_REQUIRE(!phys->analyser && !phys->remove_forward && phys->k > 0.0,
               "mk_kin_nodes_f32: no analyser (a top-hat comes in the factor table, mk_analyser_mask) and "
               "no remove_forward here");
    MK_REQUIRE(tiles->tile_atoms >= 128 && tiles->tile_atoms <= MK_TILE_ATOMS_MAX,
               "mk_kin_nodes_f32: bad tile_atoms %d", tiles->tile_atoms);
    MK_REQUIRE(plan->n_src >= 1 && plan->n_frames >= 1 && plan->sms >= 1 && (long long)px->ny * px->nz >= plan->n_pix,
               "mk_kin_nodes_f32: empty plan or too few pixels");
    if (!workspace || ws_bytes < (size_t)plan->ws_bytes) {
        mk_set_error("mk_kin_nodes_f32: workspace %zu bytes, need %lld", ws_bytes, plan->ws_bytes);
        return MK_ENOMEM;
    }
    const int n0 = plan->n0, nm = plan->nm, n1 = plan->n1, T = tiles->tile_atoms;
    const MkNodeFrame *hf = static_cast<const MkNodeFrame *>(host_buf);
    const char *db = static_cast<const char *>(dev_buf);
    cudaStream_t st = mk_stream(stream);
    MkNodeArgs A;
    memset(&A, 0, sizeof(A));
    A.frames = reinterpret_cast<const MkNodeFrame *>(db);
    A.src = reinterpret_cast<const MkNodeSrc *>(db + plan->off_src);
    const int *members = reinterpret_cast<const int *>(db + plan->off_members);
    const int *mid = reinterpret_cast<const int *>(db + plan->off_mid);
    char *w = static_cast<char *>(workspace);
    MkPrepArgs prep;
    memset(&prep, 0, sizeof(prep));
    prep.frames = A.frames;
    prep.n[MK_COARSE] = n0;
    prep.n[MK_MIDDLE] = nm;
    prep.n[MK_FINE] = n1;
    MkNodeRec *rec[5];
    rec[0] = reinterpret_cast<MkNodeRec *>(w);
    rec[1] = rec[0] + plan->patches0 * n0 * n0;
    rec[2] = rec[1] + plan->patchesm * nm * nm;
    rec[3] = rec[2] + plan->patches1 * n1 * n1;
    rec[4] = rec[3] + plan->patches0 * plan->ns[0] * plan->ns[0];
    for (int l = 0; l < 5; ++l) prep.rec[l] = rec[l];
    w += up256(sizeof(MkNodeRec) * (size_t)records(*plan));
    float *weights = reinterpret_cast<float *>(w);
    w += up256(sizeof(float) * (size_t)plan->weights);
    A.weights = weights;
    MkSubArgs sub[2];
    for (int c = 0; c < 2; ++c) {
        const int from = c ? plan->n_narrow : 0;
        sub[c].list = reinterpret_cast<const int *>(db + plan->off_leaf) + from;
        sub[c].rows = reinterpret_cast<const int *>(db + plan->off_leaf_row) + from;
        sub[c].w = weights + plan->sub_w_off[c];
        sub[c].radius = (float)(plan->sub_radius_m[c] * phys->k / MK_TWO_PI);
        prep.n[3 + c] = plan->ns[c];
        prep.w_s[c] = weights + plan->sub_w_off[c];
    }
    A.n1 = n1;
    A.n_groups = plan->n_groups;
    A.n_src = plan->n_src;
    A.src_per_slice = plan->src_per_slice;
    A.tile_atoms = T;
    A.origin = reinterpret_cast<const double4 *>(tiles->origin);
    A.tpos = reinterpret_cast<const float4 *>(tiles->pos);
    A.tamp = reinterpret_cast<const float2 *>(tiles->amp);
    A.q = reinterpret_cast<const double4 *>(px->q);
    A.u = reinterpret_cast<const float4 *>(px->u);
    A.ftab = reinterpret_cast<const float2 *>(px->factor);
    A.ftab_n = (long long)px->ny * px->nz;
    A.kappa_d = phys->k / MK_TWO_PI;
    A.kappa = (float)A.kappa_d;
    A.fresnel = fresnel != 0;
    A.fres_r = fresnel_radius_m > 0.0 ? (float)fresnel_radius_m : 0.f;
    A.decay = phys->spherical_decay;

    int nodes = 0, points = 0;             // of the largest frame
    for (int f = 0; f < plan->n_frames; ++f) {
        const MkNodeFrame &F = hf[f];
        nodes = std::max(nodes, F.py[0] * F.pz[0] * (n0 * n0 + plan->ns[0] * plan->ns[0] + plan->ns[1] * plan->ns[1]) + F.py[1] * F.pz[1] * nm * nm +
                                    F.py[2] * F.pz[2] * n1 * n1);
        points = std::max(points, F.ny + F.nz + 2 * n0 + (F.mg[1].ratio_y + F.mg[1].ratio_z) * n1 +
                                      (F.mg[0].ratio_y + F.mg[0].ratio_z) * nm);
    }
    for (int l = 0; l < 5; ++l) prep.cheb[l].fill(prep.n[l]);
    const int most = std::max(1, 8 * plan->sms / plan->n_frames);
    prep.node_blocks = std::min((nodes + MK_PREP_NT - 1) / MK_PREP_NT, most);
    prep.kappa = A.kappa_d;
    prep.xyz = px->xyz;
    prep.weights = weights;
    mk_node_prep_kernel<<<dim3(plan->n_frames, prep.node_blocks + std::min((points + 3) / 4, most)), MK_PREP_NT, 0,
                          st>>>(prep);
    MK_CHECK_CUDA(cudaGetLastError());
    MK_CHECK_CUDA(cudaFuncSetAttribute((const void *)mk_node_leaf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)leaf_bytes(MK_TILE_ATOMS_MAX)));
    auto leaf = [&](const int *list, const int *rows, int n_list, const MkNodeRec *rec, long long nodes, float2 *V) {
        const int th = (int)std::min<long long>(256, (nodes + 31) / 32 * 32);
        mk_node_leaf_kernel<<<dim3(n_list, (unsigned)((nodes + th - 1) / th)), th, leaf_bytes(T), st>>>(
            A, list, rows, rec, nodes, V);
    };
    // passes of whole frames whose node fields and partials fit the chunk
    const size_t budget = std::max((size_t)plan->chunk_bytes, (size_t)1);
    for (int fa = 0; fa < plan->n_frames;) {
        Pass P;
        const int fb = next_pass(*plan, hf, fa, budget, &P);
        const MkNodeFrame &F = hf[fa];
        A.f_lo = fa;
        A.f_hi = fb;
        A.patches1 = P.patches[MK_FINE];
        A.patch1_base = F.off[MK_FINE];
        A.pblk_base = F.pblk_off;
        A.part_base = F.part_off;
        float2 *V[3];
        char *cw = w;
        for (int l = 0; l < 3; ++l) {
            V[l] = reinterpret_cast<float2 *>(cw);
            cw += P.field[l];
        }
        A.V1 = V[MK_FINE];
        A.partial = reinterpret_cast<double2 *>(cw);
        if (plan->n_members > 0) {
            const long long nodes0 = P.patches[MK_COARSE] * n0 * n0;
            const MkNodeRec *r0 = rec[MK_COARSE] + F.off[MK_COARSE] * n0 * n0;
            if (!plan->ns[0]) leaf(members, nullptr, plan->n_members, r0, nodes0, V[0]);
            for (int c = 0; c < 2 && plan->ns[0]; ++c) {
                const int n = c ? plan->n_members - plan->n_narrow : plan->n_narrow, ns = plan->ns[c];
                if (n == 0) continue;
                MkSubArgs B = sub[c];
                B.rec = rec[3 + c] + F.off[MK_COARSE] * ns * ns;
                int rc = MK_OK;
                switch (n0 * 100 + ns) {
                case 2014: rc = mk_launch_leaf8<20, 14>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                case 2012: rc = mk_launch_leaf8<20, 12>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                case 1612: rc = mk_launch_leaf8<16, 12>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                case 1610: rc = mk_launch_leaf8<16, 10>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                case 1210: rc = mk_launch_leaf8<12, 10>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                case 1208: rc = mk_launch_leaf8<12, 8>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                case 1008: rc = mk_launch_leaf8<10, 8>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                case 806: rc = mk_launch_leaf8<8, 6>(A, B, n, r0, nodes0, V[0], plan->sms, st); break;
                default: leaf(B.list, B.rows, n, r0, nodes0, V[0]);
                }
                if (rc != MK_OK) return rc;
            }
        }
        if (plan->n_msingle > 0)
            leaf(reinterpret_cast<const int *>(db + plan->off_msingle), reinterpret_cast<const int *>(db + plan->off_mrow),
                 plan->n_msingle, rec[MK_MIDDLE] + F.off[MK_MIDDLE] * nm * nm, P.patches[MK_MIDDLE] * nm * nm,
                 V[MK_MIDDLE]);
        MkMergeArgs G;
        memset(&G, 0, sizeof(G));
        G.frames = A.frames;
        G.f_lo = fa;
        G.f_hi = fb;
        G.weights = weights;
        G.kappa = A.kappa;
        auto merge = [&](int step, int in, int to, int n_runs) {
            G.step = step;
            G.in = in;
            G.to = to;
            G.n_out = prep.n[to];
            G.in_patches = P.patches[in];
            G.in_base = F.off[in];
            G.to_patches = P.patches[to];
            G.to_base = F.off[to];
            G.item_base = F.mg[step].item_off;
            G.items = P.items[step];
            G.rec = rec[to];
            G.Vin = V[in];
            G.Vout = V[to];
            return mk_merge(G, prep.n[in], n_runs, st);
        };
        if (nm) {
            // runs of no tiles (single ones) hold the leaf's field already
            G.src = reinterpret_cast<const MkNodeSrc *>(db + plan->off_msrc);
            G.members = members;
            G.origin = A.origin;
            int rc = merge(0, MK_COARSE, MK_MIDDLE, plan->n_msrc);
            if (rc != MK_OK) return rc;
            G.src = A.src;
            G.members = nullptr;
            G.origin = reinterpret_cast<const double4 *>(db + plan->off_morg);
            rc = merge(1, MK_MIDDLE, MK_FINE, plan->n_groups);
            if (rc != MK_OK) return rc;
        } else if (plan->n_groups > 0) {
            G.src = A.src;
            G.members = members;
            G.origin = A.origin;
            const int rc = merge(1, MK_COARSE, MK_FINE, plan->n_groups);
            if (rc != MK_OK) return rc;
        }
        if (plan->n_mid > 0)
            leaf(mid, nullptr, plan->n_mid, rec[MK_FINE] + A.patch1_base * n1 * n1, A.patches1 * n1 * n1,
                 A.V1 + (long long)plan->n_groups * A.patches1 * n1 * n1);
        const dim3 grid((unsigned)P.pblk, plan->slices);
        switch (n1) {
        case 6: mk_launch_pixels<6>(A, grid, st); break;
        case 8: mk_launch_pixels<8>(A, grid, st); break;
        case 10: mk_launch_pixels<10>(A, grid, st); break;
        case 12: mk_launch_pixels<12>(A, grid, st); break;
        case 16: mk_launch_pixels<16>(A, grid, st); break;
        default: mk_set_error("mk_kin_nodes_f32: %d nodes", n1); return MK_EINVAL;
        }
        mk_node_reduce_kernel<<<(unsigned)((P.pix + 255) / 256), 256, 0, st>>>(
            A.frames, fa, fb, hf[fa].pix_off, P.pix, plan->slices, A.part_base, A.partial,
            reinterpret_cast<const double2 *>(px->phasor), reinterpret_cast<double2 *>(out), accumulate);
        MK_CHECK_CUDA(cudaGetLastError());
        fa = fb;
    }
    if (intensity_sums) {       // the node fields are read: their space holds the chunks' sums
        double *parts = reinterpret_cast<double *>(w);
        mk_node_sums_kernel<<<dim3(plan->n_frames, MK_SUM_PARTS), 256, 0, st>>>(
            A.frames, reinterpret_cast<const double2 *>(out), parts);
        mk_node_sums_final_kernel<<<(plan->n_frames + 127) / 128, 128, 0, st>>>(plan->n_frames, parts,
                                                                                intensity_sums);
        MK_CHECK_CUDA(cudaGetLastError());
    }
    return MK_OK;
}
