// Staging kernels: per-pixel prologue, stage transform + incident amplitude,
// species-partitioned Morton order and atom tiles with FP64 origins.
#include <cub/device/device_radix_sort.cuh>

#include "mk_common.cuh"

// ------------------------------------------------------------------ pixels
// x / 1e10 correctly rounded: with y = RN(1e-10) = RN(1 / 1e10) the estimate
// q = RN(x y) is within an ulp, its remainder x - q 1e10 is exact in an FMA
// and RN(q + r y) is the rounded quotient (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34, 111 (1990)). Three FP64 operations instead of a division's ~20:
// the stage transform of 8.19M atoms was bound by the FP64 pipe.
__device__ __forceinline__ double mk_metres(double x)
{
    const double q = x * 1e-10;
    return fma(fma(-q, 1e10, x), 1e-10, q);
}

// x mod 2 pi for x >= 0 (2 pi the double), exactly as fmod: the remainder is
// representable, so an FMA with the right integer quotient returns it; the
// quotient from the product with 1 / 2 pi is at most one off.
__device__ __forceinline__ double mk_mod_2pi(double x)
{
    double r = fma(-trunc(x * (1.0 / MK_TWO_PI)), MK_TWO_PI, x);
    if (r < 0.0) r = fma(-(trunc(x * (1.0 / MK_TWO_PI)) - 1.0), MK_TWO_PI, x);
    else if (r >= MK_TWO_PI) r = fma(-(trunc(x * (1.0 / MK_TWO_PI)) + 1.0), MK_TWO_PI, x);
    return r;
}

// One pixel's prologue from its position and its two neighbours' (right and
// upper; edge pixels the inner one): see mk_pixels_kernel.
struct MkPixelOut {
    double r0;
    double4 q;
    float4 u;
    double2 phasor;
};

__device__ __forceinline__ MkPixelOut mk_pixel(const double (&t)[3], const double (&n0)[3], const double (&n1)[3],
                                               double kappa, double k, const double (&b)[3])
{
    MkPixelOut o;
    const double R = sqrt(t[0] * t[0] + t[1] * t[1] + t[2] * t[2]);
    double ux = 0.0, uy = 0.0, uz = 0.0;
    const double inv = R > 0.0 ? 1.0 / R : 0.0;
    if (R > 0.0) { ux = t[0] * inv; uy = t[1] * inv; uz = t[2] * inv; }
    o.r0 = R;
    o.u = make_float4((float)ux, (float)uy, (float)uz, (float)inv);
    double s, c;
    sincos(mk_mod_2pi(k * R), &s, &c);
    o.phasor = make_double2(c, s);
    double q2 = 0.0;
    for (int j = 0; j < 2; ++j) {
        const double (&m)[3] = j ? n1 : n0;
        const double Rr = sqrt(m[0] * m[0] + m[1] * m[1] + m[2] * m[2]);
        double cd = (Rr > 0.0) ? (ux * m[0] + uy * m[1] + uz * m[2]) / Rr : 1.0;
        cd = fmin(1.0, fmax(-1.0, cd));
        const double qn = k * sqrt(fmax(0.0, 2.0 * (1.0 - cd)));
        q2 += qn * qn;
    }
    o.q = make_double4(kappa * (b[0] - ux), kappa * (b[1] - uy), kappa * (b[2] - uz), 0.5 * sqrt(q2));
    return o;
}

// One thread per pixel. Everything of magnitude |P| is kept in double here so
// the sum kernels only ever see it as (i) an FP64 dot product with a tile
// origin and (ii) the per-pixel phasor exp(i k |P|).
__global__ void mk_pixels_kernel(int ny, int nz, const double *__restrict__ xyz, double kappa,
                                 double k, double bx, double by, double bz, double *__restrict__ r0,
                                 double4 *__restrict__ q, float4 *__restrict__ u,
                                 double2 *__restrict__ phasor)
{
    const int n = ny * nz;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    // Q_cut: half the pixel diagonal in Q from the right and upper neighbours,
    // edge pixels taking the inner one (compute_scattering_cffi, Beam.py:716-746).
    const int col = p % ny, row = p / ny;
    const int nb0 = (col + 1 < ny) ? p + 1 : ((col > 0) ? p - 1 : p);
    const int nb1 = (row + 1 < nz) ? p + ny : ((row > 0) ? p - ny : p);
    const double t[3] = {xyz[3 * p], xyz[3 * p + 1], xyz[3 * p + 2]};
    const double n0[3] = {xyz[3 * nb0], xyz[3 * nb0 + 1], xyz[3 * nb0 + 2]};
    const double n1[3] = {xyz[3 * nb1], xyz[3 * nb1 + 1], xyz[3 * nb1 + 2]};
    const double b[3] = {bx, by, bz};
    const MkPixelOut o = mk_pixel(t, n0, n1, kappa, k, b);
    r0[p] = o.r0;
    u[p] = o.u;
    phasor[p] = o.phasor;
    q[p] = o.q;
}

// A scan's frames: lab pixels (A) into the sample frame, P' = R^T (P - t) /
// 1e10, and their prologue, all frames in one launch. The product is rounded as
// NumPy's matrix product rounds it (first term, then one FMA each): k |P| is
// ~5e10 rad, where an ulp of a position turns a frame's phase by ~1e-5 rad. `frames`: 20 doubles
// each -- R (9), t (3), b (3), first pixel, ny, nz, lab offset, 1 unused -- and
// lab holds a frame's (3, ny nz) coordinates from that offset on (frames of one
// ROI may share them). FP64 pipe:
// ~250 operations a pixel. 64 frames of 128 x 128: the frames' transforms in
// NumPy and a launch each took 17 ms of host and 0.87 ms of GPU time; here
// 0.41 ms.
__global__ void __launch_bounds__(256) mk_scan_pixels_kernel(const double *__restrict__ frames,
                                                             const double *__restrict__ lab, double kappa,
                                                             double k, double *__restrict__ xyz,
                                                             double *__restrict__ r0, double4 *__restrict__ q,
                                                             float4 *__restrict__ u, double2 *__restrict__ phasor)
{
    const double *F = frames + 20ll * blockIdx.y;
    const long long off = (long long)F[15];
    const int ny = (int)F[16], nz = (int)F[17], n = ny * nz;
    const double b[3] = {F[12], F[13], F[14]};
    const double *L = lab + (long long)F[18];
    for (int p = blockIdx.x * 256 + threadIdx.x; p < n; p += gridDim.x * 256) {
        const int row = p / ny, col = p - row * ny;
        const int i0 = (col + 1 < ny) ? p + 1 : ((col > 0) ? p - 1 : p);
        const int i1 = (row + 1 < nz) ? p + ny : ((row > 0) ? p - ny : p);
        double P[3][3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int i = j == 0 ? p : (j == 1 ? i0 : i1);
            const double x = L[i] - F[9], y = L[n + i] - F[10], z = L[2ll * n + i] - F[11];
#pragma unroll
            for (int c = 0; c < 3; ++c) P[j][c] = mk_metres(fma(F[6 + c], z, fma(F[3 + c], y, __dmul_rn(F[c], x))));
        }
        const MkPixelOut o = mk_pixel(P[0], P[1], P[2], kappa, k, b);
        const long long g = off + p;
        xyz[3 * g] = P[0][0];
        xyz[3 * g + 1] = P[0][1];
        xyz[3 * g + 2] = P[0][2];
        r0[g] = o.r0;
        q[g] = o.q;
        u[g] = o.u;
        phasor[g] = o.phasor;
    }
}

extern "C" int mk_scan_pixels(int n_frames, const double *frames, int max_pix, const double *lab, double k,
                              double *xyz, const mk_pixels *px, void *stream)
{
    MK_REQUIRE(n_frames >= 1 && frames && max_pix >= 1 && lab && xyz && px && px->r0 && px->q && px->u &&
                   px->phasor && k > 0.0,
               "mk_scan_pixels: bad arguments");
    const int gx = std::min((max_pix + 255) / 256, 1024);
    for (int f = 0; f < n_frames; f += 65535) {
        const int m = std::min(n_frames - f, 65535);
        mk_scan_pixels_kernel<<<dim3(gx, m), 256, 0, mk_stream(stream)>>>(
            frames + 20ll * f, lab, k / MK_TWO_PI, k, xyz, px->r0, reinterpret_cast<double4 *>(px->q),
            reinterpret_cast<float4 *>(px->u), reinterpret_cast<double2 *>(px->phasor));
        MK_CHECK_CUDA(cudaGetLastError());
    }
    return MK_OK;
}

extern "C" int mk_pixels_prepare(const mk_pixels *px, const mk_physics *phys, void *stream)
{
    MK_REQUIRE(px && phys, "mk_pixels_prepare: null argument");
    MK_REQUIRE(px->ny > 0 && px->nz > 0, "mk_pixels_prepare: empty detector (%d x %d)", px->ny, px->nz);
    MK_REQUIRE(px->xyz && px->r0 && px->q && px->u && px->phasor,
               "mk_pixels_prepare: null pixel buffer");
    MK_REQUIRE(phys->k > 0.0, "mk_pixels_prepare: k must be positive");
    const int64_t n = (int64_t)px->ny * px->nz;
    MK_REQUIRE(n < (1ll << 31), "mk_pixels_prepare: too many pixels");
    const double kappa = phys->k / MK_TWO_PI;
    const int th = 256;
    mk_pixels_kernel<<<(unsigned)((n + th - 1) / th), th, 0, mk_stream(stream)>>>(
        px->ny, px->nz, px->xyz, kappa, phys->k, phys->beam_dir[0], phys->beam_dir[1],
        phys->beam_dir[2], px->r0, reinterpret_cast<double4 *>(px->q),
        reinterpret_cast<float4 *>(px->u), reinterpret_cast<double2 *>(px->phasor));
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

// ------------------------------------------------- stage transform + E_in
// float32 lab position r = R p + t with separately rounded products and sums
// (no contraction), then E0 sampled bilinearly at (u, v) = (y, z) with the
// reference's float32 arithmetic; 0 outside the grid (Beam.py:956-1045).
struct MkRot {
    float r[9];
    float t[3];
    double grid[4];
};

__global__ void mk_atoms_lab_kernel(int64_t n, const float *__restrict__ pin, MkRot R,
                                    const float2 *__restrict__ e0, int gny, int gnz,
                                    double *__restrict__ pos_lab, float2 *__restrict__ amp)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float x = pin[3 * i], y = pin[3 * i + 1], z = pin[3 * i + 2];
    float l[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        float acc = __fmul_rn(x, R.r[3 * r]);
        acc = __fadd_rn(acc, __fmul_rn(y, R.r[3 * r + 1]));
        acc = __fadd_rn(acc, __fmul_rn(z, R.r[3 * r + 2]));
        l[r] = __fadd_rn(acc, R.t[r]);
    }
    pos_lab[3 * i] = mk_metres(l[0]);       // float32 lab positions, widened
    pos_lab[3 * i + 1] = mk_metres(l[1]);
    pos_lab[3 * i + 2] = mk_metres(l[2]);
    float2 a = make_float2(1.f, 0.f);
    if (e0) {
        const float iu = __fadd_rn(__fdiv_rn(l[1], (float)R.grid[0]), (float)R.grid[2]);
        const float iv = __fadd_rn(__fdiv_rn(l[2], (float)R.grid[1]), (float)R.grid[3]);
        a = make_float2(0.f, 0.f);
        if (iu >= 0.f && iu <= (float)(gny - 1) && iv >= 0.f && iv <= (float)(gnz - 1)) {
            const int i0 = (int)floorf(iu), j0 = (int)floorf(iv);
            const int i1 = min(i0 + 1, gny - 1), j1 = min(j0 + 1, gnz - 1);
            const float fu = __fsub_rn(iu, (float)i0), fv = __fsub_rn(iv, (float)j0);
            const float gu = __fsub_rn(1.f, fu), gv = __fsub_rn(1.f, fv);
            const float w00 = __fmul_rn(gu, gv), w01 = __fmul_rn(gu, fv);
            const float w10 = __fmul_rn(fu, gv), w11 = __fmul_rn(fu, fv);
            const float2 e00 = e0[i0 * gnz + j0], e01 = e0[i0 * gnz + j1];
            const float2 e10 = e0[i1 * gnz + j0], e11 = e0[i1 * gnz + j1];
            float re = __fmul_rn(e00.x, w00), im = __fmul_rn(e00.y, w00);
            re = __fadd_rn(re, __fmul_rn(e01.x, w01));
            im = __fadd_rn(im, __fmul_rn(e01.y, w01));
            re = __fadd_rn(re, __fmul_rn(e10.x, w10));
            im = __fadd_rn(im, __fmul_rn(e10.y, w10));
            re = __fadd_rn(re, __fmul_rn(e11.x, w11));
            im = __fadd_rn(im, __fmul_rn(e11.y, w11));
            a = make_float2(re, im);
        }
    }
    amp[i] = a;
}

extern "C" int mk_atoms_lab(int64_t n, const float *pos_in, const float *rot, const float *trans,
                            const float *e0, int grid_ny, int grid_nz, const double *grid,
                            double *pos_lab, float *amp, void *stream)
{
    MK_REQUIRE(n >= 0, "mk_atoms_lab: negative atom count");
    if (n == 0) return MK_OK;
    MK_REQUIRE(pos_in && rot && trans && pos_lab && amp, "mk_atoms_lab: null argument");
    MK_REQUIRE(!e0 || (grid && grid_ny > 0 && grid_nz > 0 && grid[0] > 0.0 && grid[1] > 0.0),
               "mk_atoms_lab: beam grid needs positive sizes and spacings");
    MkRot R;
    for (int i = 0; i < 9; ++i) R.r[i] = rot[i];
    for (int i = 0; i < 3; ++i) R.t[i] = trans[i];
    for (int i = 0; i < 4; ++i) R.grid[i] = grid ? grid[i] : 1.0;
    const int th = 256;
    mk_atoms_lab_kernel<<<(unsigned)((n + th - 1) / th), th, 0, mk_stream(stream)>>>(
        n, pos_in, R, reinterpret_cast<const float2 *>(e0), grid_ny, grid_nz, pos_lab,
        reinterpret_cast<float2 *>(amp));
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

// ------------------------------------------------------------- species
// Byte species codes of a chunk -> the call's species indices, and how many
// atoms each has (added to counts), in one pass over the codes: 5 bytes an
// atom. An indexing pass and a histogram took 907 us for 8.19M atoms. Codes
// without an entry are written as 0 and not counted.
struct MkSpeciesLut {
    signed char to[256];
};

__global__ void __launch_bounds__(256) mk_species_kernel(int64_t n, const unsigned char *__restrict__ codes,
                                                         const __grid_constant__ MkSpeciesLut lut, int n_species,
                                                         int *__restrict__ out,
                                                         unsigned long long *__restrict__ counts)
{
    __shared__ signed char s_to[256];
    __shared__ int s_n[MK_MAX_SPECIES];
    s_to[threadIdx.x] = lut.to[threadIdx.x];
    if (threadIdx.x < MK_MAX_SPECIES) s_n[threadIdx.x] = 0;
    __syncthreads();
    const int64_t step = (int64_t)gridDim.x * 256;
    int mine = 0;       // lane s of a warp counts species s
    for (int64_t i0 = (int64_t)blockIdx.x * 256; i0 < n; i0 += step) {
        const int64_t i = i0 + threadIdx.x;
        int s = -1;
        if (i < n) {
            s = s_to[codes[i]];
            out[i] = max(s, 0);
        }
        for (int k = 0; k < n_species; ++k) {
            const int m = __popc(__ballot_sync(0xffffffffu, s == k));
            if ((int)(threadIdx.x & 31) == k) mine += m;
        }
    }
    if ((threadIdx.x & 31) < n_species && mine) atomicAdd(&s_n[threadIdx.x & 31], mine);
    __syncthreads();
    if (threadIdx.x < n_species && s_n[threadIdx.x])
        atomicAdd(&counts[threadIdx.x], (unsigned long long)s_n[threadIdx.x]);
}

extern "C" int mk_species_index(int64_t n, const unsigned char *codes, const int *lut, int n_lut,
                                int n_species, int *species, int64_t *counts, void *stream)
{
    MK_REQUIRE(n >= 0 && n_lut >= 1 && n_lut <= 256 && n_species >= 1 && n_species <= MK_MAX_SPECIES,
               "mk_species_index: bad sizes");
    if (n == 0) return MK_OK;
    MK_REQUIRE(codes && lut && species && counts, "mk_species_index: null argument");
    MkSpeciesLut L;
    for (int i = 0; i < 256; ++i) {
        const int v = i < n_lut ? lut[i] : -1;
        MK_REQUIRE(i >= n_lut || (v >= 0 && v < n_species), "mk_species_index: code %d maps to species %d of %d",
                   i, v, n_species);
        L.to[i] = (signed char)v;
    }
    const unsigned nb = (unsigned)std::min<int64_t>((n + 1023) / 1024, 152 * 8);
    mk_species_kernel<<<nb, 256, 0, mk_stream(stream)>>>(n, codes, L, n_species, species,
                                                        reinterpret_cast<unsigned long long *>(counts));
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

// ------------------------------------------------------------- tiles
// Bounding box of all atoms (for the Morton quantisation): one block-level
// min/max per block, combined with atomics on the ordered-integer image of
// the doubles.
__device__ __forceinline__ unsigned long long mk_ordered(double v)
{
    const unsigned long long b = __double_as_longlong(v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double mk_unordered(unsigned long long o)
{
    const unsigned long long b = (o & 0x8000000000000000ull) ? (o & ~0x8000000000000000ull) : ~o;
    return __longlong_as_double(b);
}

__global__ void mk_bbox_init(unsigned long long *bb, double *crowded)
{
    if (threadIdx.x == 0 && crowded) *crowded = 0.0;
    if (threadIdx.x < 3) bb[threadIdx.x] = ~0ull;       // min
    else if (threadIdx.x < 6) bb[threadIdx.x] = 0ull;   // max
}

// A thread always meets the same coordinate (the stride is a multiple of 3),
// so the loads are whole lines; six atomics a block.
#define MK_BBOX_NT 192
__global__ void __launch_bounds__(MK_BBOX_NT) mk_bbox_kernel(int64_t n, const double *__restrict__ pos,
                                                             unsigned long long *bb)
{
    __shared__ unsigned long long s_bb[6];
    if (threadIdx.x < 6) s_bb[threadIdx.x] = threadIdx.x < 3 ? ~0ull : 0ull;
    __syncthreads();
    unsigned long long lo = ~0ull, hi = 0ull;
    const int64_t step = (int64_t)gridDim.x * MK_BBOX_NT;
    for (int64_t i = (int64_t)blockIdx.x * MK_BBOX_NT + threadIdx.x; i < 3 * n; i += step) {
        const unsigned long long o = mk_ordered(pos[i]);
        lo = o < lo ? o : lo;
        hi = o > hi ? o : hi;
    }
    atomicMin(&s_bb[threadIdx.x % 3], lo);
    atomicMax(&s_bb[3 + threadIdx.x % 3], hi);
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(&bb[threadIdx.x], s_bb[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(&bb[threadIdx.x], s_bb[threadIdx.x]);
}

// Position along a 3-D Hilbert curve of 2^bits cells per axis (the
// axes-to-transpose construction of J. Skilling, "Programming the Hilbert
// curve", AIP Conf. Proc. 707, 381 (2004)): undo the rotations/reflections
// level by level, Gray-encode, then read the bits out MSB first, x first.
// Unlike a Z-order (Morton) curve, consecutive cells are always face
// neighbours, so a run of consecutive atoms never spans two distant corners
// of the sample and every tile stays compact.
#define MK_MAX_CUBES 128     // 7 bits of cube index at most

template <class Key>
__device__ __forceinline__ Key mk_hilbert3(uint32_t x, uint32_t y, uint32_t z, int bits)
{
    uint32_t X[3] = {x, y, z};
    for (uint32_t Q = 1u << (bits - 1); Q > 1; Q >>= 1) {
        const uint32_t P = Q - 1;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (X[i] & Q) {
                X[0] ^= P;
            } else {
                const uint32_t t = (X[0] ^ X[i]) & P;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    uint32_t t = 0;
    for (uint32_t Q = 1u << (bits - 1); Q > 1; Q >>= 1)
        if (X[2] & Q) t ^= Q - 1;
    X[0] ^= t;
    X[1] ^= t;
    X[2] ^= t;
    Key h = 0;
    for (int b = bits - 1; b >= 0; --b) {
        h = (h << 1) | ((X[0] >> b) & 1u);
        h = (h << 1) | ((X[1] >> b) & 1u);
        h = (h << 1) | ((X[2] >> b) & 1u);
    }
    return h;
}

// The cubes and the key's layout, from the bounding box, once per build.
struct MkKeyGrid {
    double lo[3];
    double inv[3];       // 1 / cube side, per axis
    int nc[3];           // cubes per axis
    int bits;            // Hilbert bits per axis
    int cube_bits;
};

__global__ void mk_key_grid_kernel(const unsigned long long *__restrict__ bb, int key_bits, int axis_bits,
                                   int species_bits, MkKeyGrid *__restrict__ out)
{
    MkKeyGrid G;
    double span[3], side = 0.0;
    for (int c = 0; c < 3; ++c) {
        G.lo[c] = mk_unordered(bb[c]);
        span[c] = mk_unordered(bb[3 + c]) - G.lo[c];
        if (!(span[c] < 1e30)) span[c] = 0.0;       // an atom at infinity or nowhere
        if (span[c] > 0.0 && (side == 0.0 || span[c] < side)) side = span[c];
    }
    if (!(side > 0.0)) side = 1.0;
    for (;;) {
        double all = 1.0;
        for (int c = 0; c < 3; ++c) {
            const double m = floor(span[c] / side + 0.5);
            G.nc[c] = (int)fmin(fmax(m, 1.0), 1e6);
            all *= G.nc[c];
        }
        if (!(all > MK_MAX_CUBES)) break;
        side *= 1.25;
    }
    for (int c = 0; c < 3; ++c) G.inv[c] = span[c] > 0.0 ? G.nc[c] / span[c] : 0.0;
    G.cube_bits = 0;
    while ((1 << G.cube_bits) < G.nc[0] * G.nc[1] * G.nc[2]) ++G.cube_bits;
    G.bits = min(axis_bits, (key_bits - species_bits - G.cube_bits) / 3);
    *out = G;
}

// Sort key: species on top, then a row of cubes, then the Hilbert index
// inside the atom's cube. The bounding box is cut into near-cubes, along each
// axis the whole number of the shortest extent (enlarged until at most
// MK_MAX_CUBES) that is nearest, taken x fastest. The curve runs from a
// cube's (0,0,0) corner to its (max,0,0) corner, so consecutive cubes along
// x join without a jump; only row ends do. Filling every cube keeps the curve
// out of empty space (where its excursions would put far-apart atoms next to
// each other in the order): cubes of one exact side left slivers of the
// longer extents as cubes of their own, a few atoms thick, and every tile
// that crossed one spanned the sample (5.4M atoms of a cubic polycrystal: 14
// tiles too wide for the node form, 2.1 ms in the split kernel at 1024^2).
// Short keys have 32 bits, or 24 below MK_SHORT_KEY_ATOMS atoms (four or three
// radix passes, at most 10 Hilbert bits an axis): in a filled box the cells then
// outnumber the atoms. Long ones have 62 (17 bits an axis, 8 passes) and resolve
// samples whose box is mostly empty -- particles far apart, an atom far off --
// where short cells hold many atoms each, in input order: the tile build reports
// more than a quarter of a tile in one cell. Fewer do not widen the tiles: two
// particles of 32,000 atoms 0.3 um apart, ~110 atoms a cell, have 2.04 nm tiles,
// 2.02 with long keys, whose build adds 230 us to a call of 1.44 ms; with 1,600 a
// cell they are 1.5 times as wide. Long keys, then cut in FP64
// by every thread, took 1355 us to make and 551 us to sort for 8.19M atoms, and
// 63 us to sort 32k.
#define MK_SHORT_KEY_ATOMS (1 << 17)
#define MK_LONG_KEY_BITS 62

// Real: what the cell coordinates are formed in; 17 bits of up to 128 cubes
// need FP64.
template <class Key, class Real>
__global__ void mk_keys_kernel(int64_t n, const double *__restrict__ pos,
                               const int *__restrict__ species, const MkKeyGrid *__restrict__ grid,
                               Key *__restrict__ keys, int *__restrict__ idx)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const MkKeyGrid &G = *grid;
    const int bits = G.bits;
    const Real top = (Real)((1u << bits) - 1);
    uint32_t q[3];
    int cube[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const Real t = (Real)(pos[3 * i + c] - G.lo[c]) * (Real)G.inv[c];
        cube[c] = min(G.nc[c] - 1, max(0, (int)floor(t)));
        const Real f = fmin(fmax(t - (Real)cube[c], (Real)0), (Real)1);
        q[c] = (uint32_t)(f * top);
    }
    const Key ci = (Key)((cube[2] * G.nc[1] + cube[1]) * G.nc[0] + cube[0]);
    keys[i] = ((((Key)species[i] << G.cube_bits) | ci) << (3 * bits)) | mk_hilbert3<Key>(q[0], q[1], q[2], bits);
    idx[i] = (int)i;
}

struct MkTileMap {
    int n_species;
    int tile_atoms;
    long long run_start[MK_MAX_SPECIES];  // first sorted index of each species
    long long run_count[MK_MAX_SPECIES];
    int tile_start[MK_MAX_SPECIES + 1];   // first tile of each species
};

// One block per tile: gather its atoms in sorted order; origin the centre of
// their bounding box, offsets k/2pi (a - o) formed in FP64 and rounded once to
// float32. The box is taken of the offsets from the tile's first atom, exact
// differences rounded to float32, so that its ~40 minima and maxima a thread
// stay off the FP64 pipe (2 lane operations per clock and SM), which bound
// the build at 39 operations an atom (645 us for 8.19M atoms; here 358). Tiles of
// up to 2 NT atoms hold their positions in registers, larger ones gather them
// again for the offsets. `keys` (short ones, or null): *crowded is set where
// atoms a quarter of a tile apart in the order have the same key.
template <int NT, bool HOLD>
__global__ void __launch_bounds__(NT) mk_tile_kernel(MkTileMap M, double kappa,
                                                      const double *__restrict__ pos,
                                                      const float2 *__restrict__ amp,
                                                      const int *__restrict__ order,
                                                      const uint32_t *__restrict__ keys, double *crowded,
                                                      double4 *__restrict__ origin,
                                                      int *__restrict__ tspecies,
                                                      float4 *__restrict__ tpos,
                                                      float2 *__restrict__ tamp)
{
    const int t = blockIdx.x;
    int s = 0;
    while (s + 1 < M.n_species && t >= M.tile_start[s + 1]) ++s;
    const long long first = M.run_start[s] + (long long)(t - M.tile_start[s]) * M.tile_atoms;
    const long long end = M.run_start[s] + M.run_count[s];
    __shared__ float red[6][NT / 32];
    __shared__ float rad2[NT / 32];
    if (keys && threadIdx.x < 8) {
        const long long i = first + (long long)threadIdx.x * (M.tile_atoms >> 3), j = i + (M.tile_atoms >> 2);
        if (j < end && keys[i] == keys[j]) *crowded = 1.0;
    }
    const long long a0 = order[first];
    const double fx = pos[3 * a0], fy = pos[3 * a0 + 1], fz = pos[3 * a0 + 2];

    double hx[2], hy[2], hz[2];             // HOLD: offsets from the first atom
    int ha[2];
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    auto meet = [&](double x, double y, double z) {
        const float v[3] = {(float)x, (float)y, (float)z};
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            lo[c] = fminf(lo[c], v[c]);
            hi[c] = fmaxf(hi[c], v[c]);
        }
    };
    if constexpr (HOLD) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = threadIdx.x + i * NT;
            const long long si = first + j;
            ha[i] = j < M.tile_atoms && si < end ? order[si] : -1;
            hx[i] = hy[i] = hz[i] = 0.0;
            if (ha[i] >= 0) {
                hx[i] = pos[3 * (long long)ha[i]] - fx;
                hy[i] = pos[3 * (long long)ha[i] + 1] - fy;
                hz[i] = pos[3 * (long long)ha[i] + 2] - fz;
                meet(hx[i], hy[i], hz[i]);
            }
        }
    } else {
        for (int j = threadIdx.x; j < M.tile_atoms && first + j < end; j += NT) {
            const long long a = order[first + j];
            meet(pos[3 * a] - fx, pos[3 * a + 1] - fy, pos[3 * a + 2] - fz);
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        for (int off = 16; off > 0; off >>= 1) {
            lo[c] = fminf(lo[c], __shfl_xor_sync(0xffffffffu, lo[c], off));
            hi[c] = fmaxf(hi[c], __shfl_xor_sync(0xffffffffu, hi[c], off));
        }
        if ((threadIdx.x & 31) == 0) {
            red[c][threadIdx.x >> 5] = lo[c];
            red[3 + c][threadIdx.x >> 5] = hi[c];
        }
    }
    __syncthreads();
    double org[3];                          // the box's centre, from the first atom
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float l = INFINITY, h = -INFINITY;
        for (int w = 0; w < NT / 32; ++w) {
            l = fminf(l, red[c][w]);
            h = fmaxf(h, red[3 + c][w]);
        }
        org[c] = (double)(0.5f * (l + h));
    }
    float r2max = 0.f;
    const long long base = (long long)t * M.tile_atoms;
    auto put = [&](int j, int a, double x, double y, double z) {
        float4 P = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 E = make_float2(0.f, 0.f);
        if (a >= 0) {
            const double dx = x - org[0], dy = y - org[1], dz = z - org[2];
            const double d2 = dx * dx + dy * dy + dz * dz;
            P = make_float4((float)(kappa * dx), (float)(kappa * dy), (float)(kappa * dz),
                            (float)(kappa * kappa * d2));
            r2max = fmaxf(r2max, P.w);
            E = amp[a];
        }
        // atom pairs interleaved: per pair (2q, 2q+1) the floats
        // x0 x1 y0 y1 z0 z1 w0 w1 and er0 er1 ei0 ei1, so that the sum
        // kernels load two atoms' coordinates as packed f32x2 operands
        float *pf = reinterpret_cast<float *>(tpos) + 4 * (base + (j & ~1));
        float *af = reinterpret_cast<float *>(tamp) + 2 * (base + (j & ~1));
        const int h = j & 1;
        pf[h] = P.x;
        pf[2 + h] = P.y;
        pf[4 + h] = P.z;
        pf[6 + h] = P.w;
        af[h] = E.x;
        af[2 + h] = E.y;
    };
    if constexpr (HOLD) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = threadIdx.x + i * NT;
            if (j < M.tile_atoms) put(j, ha[i], hx[i], hy[i], hz[i]);
        }
    } else {
        for (int j = threadIdx.x; j < M.tile_atoms; j += NT) {
            const int a = first + j < end ? order[first + j] : -1;
            if (a >= 0)
                put(j, a, pos[3 * (long long)a] - fx, pos[3 * (long long)a + 1] - fy,
                    pos[3 * (long long)a + 2] - fz);
            else
                put(j, a, 0.0, 0.0, 0.0);
        }
    }
    for (int off = 16; off > 0; off >>= 1) r2max = fmaxf(r2max, __shfl_xor_sync(0xffffffffu, r2max, off));
    if ((threadIdx.x & 31) == 0) rad2[threadIdx.x >> 5] = r2max;
    __syncthreads();
    if (threadIdx.x == 0) {
        float m = 0.f;
        for (int w = 0; w < NT / 32; ++w) m = fmaxf(m, rad2[w]);
        // |D|^2 was rounded to float32 (in cycles): a whole ulp up bounds it
        origin[t] = make_double4(fx + org[0], fy + org[1], fz + org[2],
                                 sqrt((double)m * (1.0 + 1.2e-7)) / kappa);
        tspecies[t] = s;
    }
}

static size_t mk_align256(size_t b) { return (b + 255) & ~(size_t)255; }

template <class Key>
static size_t mk_cub_temp_bytes(int64_t n)
{
    size_t tb = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tb, (Key *)nullptr, (Key *)nullptr, (int *)nullptr, (int *)nullptr,
                                    (int)n, 0, sizeof(Key) == 8 ? MK_LONG_KEY_BITS : 32);
    return tb;
}

extern "C" size_t mk_tiles_workspace_size_keys(int64_t n, int long_keys)
{
    if (n <= 0) return 256;
    const size_t key = long_keys ? 8 : 4;
    return mk_align256(64) + mk_align256(sizeof(MkKeyGrid)) + 2 * mk_align256(key * (size_t)n) +
           2 * mk_align256(4 * (size_t)n) +
           mk_align256(long_keys ? mk_cub_temp_bytes<unsigned long long>(n) : mk_cub_temp_bytes<uint32_t>(n));
}

extern "C" size_t mk_tiles_workspace_size(int64_t n) { return mk_tiles_workspace_size_keys(n, 1); }

// Sorted keys and order of the atoms, in the workspace `w`.
template <class Key, class Real>
static int mk_sort_atoms(int64_t n, const double *pos, const int *species, const MkKeyGrid *grid, char *w,
                         int key_bits, cudaStream_t st, const Key **keys, const int **order)
{
    Key *k_in = reinterpret_cast<Key *>(w);
    w += mk_align256(sizeof(Key) * (size_t)n);
    Key *k_out = reinterpret_cast<Key *>(w);
    w += mk_align256(sizeof(Key) * (size_t)n);
    int *i_in = reinterpret_cast<int *>(w);
    w += mk_align256(4 * (size_t)n);
    int *i_out = reinterpret_cast<int *>(w);
    w += mk_align256(4 * (size_t)n);
    size_t temp = mk_cub_temp_bytes<Key>(n);
    const int th = 256;
    mk_keys_kernel<Key, Real><<<(unsigned)((n + th - 1) / th), th, 0, st>>>(n, pos, species, grid, k_in, i_in);
    MK_CHECK_CUDA(cudaGetLastError());
    MK_CHECK_CUDA(cub::DeviceRadixSort::SortPairs(w, temp, k_in, k_out, i_in, i_out, (int)n, 0, key_bits, st));
    *keys = k_out;
    *order = i_out;
    return MK_OK;
}

extern "C" int mk_tiles_build(int64_t n, const double *pos, const int *species, const float *amp,
                              int n_species, const int64_t *counts, double k, mk_tiles *tiles,
                              void *workspace, size_t ws_bytes, void *stream)
{
    return mk_tiles_build_keys(n, pos, species, amp, n_species, counts, k, tiles, 1, nullptr, workspace,
                               ws_bytes, stream);
}

extern "C" int mk_tiles_build_keys(int64_t n, const double *pos, const int *species, const float *amp,
                                   int n_species, const int64_t *counts, double k, mk_tiles *tiles,
                                   int long_keys, double *crowded, void *workspace, size_t ws_bytes,
                                   void *stream)
{
    MK_REQUIRE(tiles && counts, "mk_tiles_build: null argument");
    MK_REQUIRE(n_species >= 1 && n_species <= MK_MAX_SPECIES, "mk_tiles_build: 1..%d species",
               MK_MAX_SPECIES);
    MK_REQUIRE(n > 0 && n < (1ll << 31), "mk_tiles_build: atom count %lld out of range",
               (long long)n);
    MK_REQUIRE(pos && species && amp && tiles->origin && tiles->species && tiles->pos && tiles->amp,
               "mk_tiles_build: null buffer");
    const int T = tiles->tile_atoms;
    MK_REQUIRE(T >= 128 && T <= 4096 && (T & (T - 1)) == 0,
               "mk_tiles_build: tile_atoms must be a power of two in [128, 4096]");
    MkTileMap M;
    memset(&M, 0, sizeof(M));
    M.n_species = n_species;
    M.tile_atoms = T;
    long long run = 0, total = 0;
    int tiles_needed = 0;
    for (int s = 0; s < n_species; ++s) {
        MK_REQUIRE(counts[s] >= 0, "mk_tiles_build: negative count");
        M.run_start[s] = run;
        M.run_count[s] = counts[s];
        M.tile_start[s] = tiles_needed;
        run += counts[s];
        tiles_needed += (int)((counts[s] + T - 1) / T);
        total += counts[s];
    }
    M.tile_start[n_species] = tiles_needed;
    MK_REQUIRE(total == n, "mk_tiles_build: species counts sum to %lld, expected %lld", total,
               (long long)n);
    MK_REQUIRE(tiles->n_tiles == tiles_needed, "mk_tiles_build: n_tiles %d, layout needs %d",
               tiles->n_tiles, tiles_needed);
    const size_t need = mk_tiles_workspace_size_keys(n, long_keys);
    if (!workspace || ws_bytes < need) {
        mk_set_error("mk_tiles_build: workspace %zu bytes, need %zu", ws_bytes, need);
        return MK_ENOMEM;
    }
    char *w = static_cast<char *>(workspace);
    unsigned long long *bb = reinterpret_cast<unsigned long long *>(w);
    w += mk_align256(64);
    MkKeyGrid *grid = reinterpret_cast<MkKeyGrid *>(w);
    w += mk_align256(sizeof(MkKeyGrid));
    cudaStream_t st = mk_stream(stream);
    const int key_bits = long_keys ? MK_LONG_KEY_BITS : n <= MK_SHORT_KEY_ATOMS ? 24 : 32;
    int species_bits = 0;
    while ((1 << species_bits) < n_species) ++species_bits;
    mk_bbox_init<<<1, 32, 0, st>>>(bb, crowded);
    const int nb = (int)std::min<int64_t>((3 * n + 4 * MK_BBOX_NT - 1) / (4 * MK_BBOX_NT), 152 * 10);
    mk_bbox_kernel<<<nb, MK_BBOX_NT, 0, st>>>(n, pos, bb);
    mk_key_grid_kernel<<<1, 1, 0, st>>>(bb, key_bits, long_keys ? 17 : 10, species_bits, grid);
    const uint32_t *keys = nullptr;
    const unsigned long long *keys64 = nullptr;
    const int *order = nullptr;
    const int rc = long_keys ? mk_sort_atoms<unsigned long long, double>(n, pos, species, grid, w, key_bits, st,
                                                                         &keys64, &order)
                             : mk_sort_atoms<uint32_t, float>(n, pos, species, grid, w, key_bits, st, &keys, &order);
    if (rc != MK_OK) return rc;
    if (tiles_needed > 0) {
        auto fn = T <= 512 ? mk_tile_kernel<256, true> : mk_tile_kernel<256, false>;
        fn<<<tiles_needed, 256, 0, st>>>(
            M, k / MK_TWO_PI, pos, reinterpret_cast<const float2 *>(amp), order, crowded ? keys : nullptr, crowded,
            reinterpret_cast<double4 *>(tiles->origin), tiles->species,
            reinterpret_cast<float4 *>(tiles->pos), reinterpret_cast<float2 *>(tiles->amp));
        MK_CHECK_CUDA(cudaGetLastError());
    }
    return MK_OK;
}
