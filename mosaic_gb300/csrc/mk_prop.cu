// Free-space angular-spectrum propagation of the detector field: padding,
// the transfer-function multiply on the spectrum, and the centre crop fused
// with |A|^2. The FFTs in between are cuFFT (through the caller).
//
// Transfer function (the reference's prop_mul_kernel, MOSAIC Beam.py:4747-4834):
//   kt = (ky + kgy, kz + kgz), kt^2 <= k^2:
//     H = exp(i [ -z kt^2 / (sqrt(k^2 - kt^2) + k) + z (k - kga) ])
//   otherwise (evanescent):
//     H = exp(-|z| sqrt(kt^2 - k^2)) exp(-i z kga)
// with ky, kz the FFT frequencies 2 pi fftfreq(N, d). The phase is formed
// and reduced in FP64 (the evanescent carrier z kga is ~1e10 rad), then
// sin/cos in FP64: the multiply is one pass over the spectrum, so its cost
// is memory traffic, not arithmetic.
#include <algorithm>

#include "mk_common.cuh"

__device__ __forceinline__ double mk_fftfreq(int i, int n, double d)
{
    const int half = (n - 1) / 2 + 1;      // numpy.fft.fftfreq ordering
    const int m = i < half ? i : i - n;
    return (double)m / ((double)n * d);
}

// Pad (nz, ny) into (nz2, ny2) centred at (z0, y0): edge replication
// (mode 0) or a constant (mode 1). PTS points a thread: two where rows have an
// even number of points and start on 16 bytes.
template <int PTS>
__global__ void mk_prop_pad_kernel(const float2 *__restrict__ in, int ny, int nz,
                                   float2 *__restrict__ out, int ny2, int nz2, int y0, int z0,
                                   int mode, float2 cval)
{
    const int x0 = PTS * (blockIdx.x * blockDim.x + threadIdx.x);
    const int y = blockIdx.y;
    if (x0 >= ny2 || y >= nz2) return;
    const int sz = y - z0;
    const bool off = mode == 1 && (sz < 0 || sz >= nz);
    const float2 *row = in + (size_t)min(max(sz, 0), nz - 1) * ny;
    float2 v[PTS];
#pragma unroll
    for (int i = 0; i < PTS; ++i) {
        const int sx = x0 + i - y0;
        v[i] = off || (mode == 1 && (sx < 0 || sx >= ny)) ? cval : row[min(max(sx, 0), ny - 1)];
    }
    float2 *o = out + (size_t)y * ny2 + x0;
    if (PTS == 2) *reinterpret_cast<float4 *>(o) = make_float4(v[0].x, v[0].y, v[PTS - 1].x, v[PTS - 1].y);
    else o[0] = v[0];
}

__global__ void mk_prop_mul_kernel(float2 *__restrict__ F, int ny2, int nz2, double dy, double dz,
                                   double k, double z, double kga, double kgy, double kgz)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= ny2 || y >= nz2) return;
    const double a = MK_TWO_PI * mk_fftfreq(x, ny2, dy) + kgy;
    const double b = MK_TWO_PI * mk_fftfreq(y, nz2, dz) + kgz;
    const double kt2 = a * a + b * b, kx2 = k * k - kt2;
    double ph, amp;
    if (kx2 >= 0.0) {
        ph = -z * kt2 / (sqrt(kx2) + k) + z * (k - kga);
        amp = 1.0;
    } else {
        amp = exp(-fabs(z) * sqrt(-kx2));
        ph = fmod(-z * kga, MK_TWO_PI);
    }
    double s, c;
    sincos(ph, &s, &c);
    const size_t i = (size_t)y * ny2 + x;
    const float2 g = F[i];
    const double hr = amp * c, hi = amp * s;
    F[i] = make_float2((float)(g.x * hr - g.y * hi), (float)(g.x * hi + g.y * hr));
}

// Centre crop of the inverse transform, fused with |A|^2; `scale` applies
// the inverse FFT's normalisation.
__global__ void mk_prop_crop_kernel(const float2 *__restrict__ G, int ny2, int nz2, int y0, int z0,
                                    int ny, int nz, float scale, float2 *__restrict__ field,
                                    float *__restrict__ intensity)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;
    if (x >= ny || y >= nz) return;
    const float2 g = G[(size_t)(y + z0) * ny2 + (x + y0)];
    const float2 v = make_float2(g.x * scale, g.y * scale);
    if (field) field[(size_t)y * ny + x] = v;
    if (intensity) intensity[(size_t)y * ny + x] = v.x * v.x + v.y * v.y;
}

// --------------------------------------------- fused spectral column pass
// The 2-D transform separates into a transform along y (rows) and one along
// z (columns), in either order. Taking the rows first and last,
//   G = R^-1 C^-1 [H o (C R P)] = R^-1 (C^-1 H C) R P,
// the column transform, the transfer-function multiply and the inverse
// column transform are adjacent: one kernel does all three for a group of
// W neighbouring columns in shared memory, so between the two row
// transforms (cuFFT, contiguous rows) the spectrum is read and written once
// instead of three times (column FFT, multiply, inverse column FFT).
//
// The padded rows need no memory: rows outside the field repeat its edge
// rows (their transforms too) or are constant (their transform is one bin),
// and only the field's rows are wanted back, so the kernel reads and writes
// the field's nz rows and forms the nz2 - nz others as it loads.
//
// N = 2^logn points are P passes of radix 8 and a last one of radix 2, 4 or
// 8, decimation in frequency forward and in time back, so that neither
// transform is permuted: the forward one ends with frequency k0 + 8 k1 + ..
// at position k0 N/8 + k1 N/64 + .., where H is applied. A thread holds 8
// points in registers per item; the first forward pass reads global memory,
// the last inverse pass writes it, and the radix-2/4/8 passes either side of
// H stay in registers: 2 P + 2 passes over shared memory of 8 bytes a point.
// A line's point i is at i + i/8 and lines are LD = 16/W (mod 16) points
// apart, which keeps the 8-byte accesses of a half warp (W lines x 16/W
// neighbouring points) on different banks at every stride; in place and
// unpadded, radix-2 stages fused by threes with a bit-reversal pass between
// the transforms ran 8-way conflicts and took 299 us for the 2048 x 4096
// spectrum of a 2048 x 1500 field; this 81 us (98 MB at copy bandwidth: 15).
// Twiddles exp(-2 pi i i k / M) of a pass over lines of M points come from a
// table made in FP64, its M / 8 values of one k side by side: a warp's i are
// neighbours. From one table of exp(-2 pi i t / N), read k 8^pass entries apart,
// the same passes took 91 us. The transfer
// function is formed in FP32 as the reference's prop_mul_kernel does
// (Beam.py:4763-4830), with the two large constant phases, z (k - k_axis) and
// -z k_axis, reduced mod 2 pi in FP64 on the host.
#define MK_FFT_NT 512
#define MK_FFT_MAX 8192
#define MK_FFT_SMEM (74 << 10)    // a block's lines where three blocks fit an SM
#define MK_FFT_SMEM_MAX (227u << 10)

__device__ __forceinline__ float2 mk_cmul(float2 a, float2 b)
{
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 mk_cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 mk_csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a times -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 mk_crot(float2 a)
{
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// DFT of R points in registers, natural order in and out.
template <int R, bool INV>
__device__ __forceinline__ void mk_dft(float2 *v)
{
    if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = mk_cadd(a, b);
        v[1] = mk_csub(a, b);
    } else if constexpr (R == 4) {
        const float2 a = mk_cadd(v[0], v[2]), b = mk_csub(v[0], v[2]);
        const float2 c = mk_cadd(v[1], v[3]), d = mk_crot<INV>(mk_csub(v[1], v[3]));
        v[0] = mk_cadd(a, c);
        v[1] = mk_cadd(b, d);
        v[2] = mk_csub(a, c);
        v[3] = mk_csub(b, d);
    } else {
        float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        mk_dft<4, INV>(e);
        mk_dft<4, INV>(o);
        const float h = 0.70710678118654752f;
        const float2 r1 = mk_crot<INV>(o[1]), r3 = mk_crot<INV>(o[3]);
        o[1] = make_float2(h * (o[1].x + r1.x), h * (o[1].y + r1.y));        // times w8
        o[2] = mk_crot<INV>(o[2]);
        o[3] = make_float2(h * (r3.x - o[3].x), h * (r3.y - o[3].y));        // times w8^3
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[j] = mk_cadd(e[j], o[j]);
            v[j + 4] = mk_csub(e[j], o[j]);
        }
    }
}

struct MkColsArgs {
    float2 *F;             // (nz, ny2) rows of the field's spectrum, in place
    int ny2, nz2, logn, W, ld;
    int z0, nz, mode;      // field rows at [z0, z0 + nz); 0 repeat the edges, 1 constant
    float2 cval;           // spectrum of a constant row at column 0
    const float2 *tw;
    const float *ky, *kz;
    float k, z, c_prop, c_evan;
};

__device__ __forceinline__ int mk_pad8(int i) { return i + (i >> 3); }

// Row r of column col of the padded, row-transformed field.
__device__ __forceinline__ float2 mk_cols_load(const MkColsArgs &A, int r, int col)
{
    const int s = r - A.z0;
    if (A.mode == 1 && (unsigned)s >= (unsigned)A.nz)
        return col == 0 ? A.cval : make_float2(0.f, 0.f);
    return A.F[(size_t)min(max(s, 0), A.nz - 1) * A.ny2 + col];
}

// H(ky, kz) times v.
__device__ __forceinline__ float2 mk_cols_mul(const MkColsArgs &A, float2 v, float a, float b)
{
    const float kt2 = fmaf(a, a, b * b);
    const float kt = sqrtf(kt2);
    float ph, amp;
    if (kt <= A.k) {
        // sqrt(k^2 - kt^2) - k = -kt^2 / (sqrt(k^2 - kt^2) + k)
        ph = -A.z * kt2 / (sqrtf((A.k - kt) * (A.k + kt)) + A.k) + A.c_prop;
        amp = 1.f;
    } else {
        amp = expf(-fabsf(A.z) * sqrtf((kt - A.k) * (kt + A.k)));
        ph = A.c_evan;
    }
    float sn, cs;
    sincosf(ph, &sn, &cs);
    return mk_cmul(v, make_float2(amp * cs, amp * sn));
}

// LAST: bits of the last radix (1, 2 or 3). Block = W neighbouring columns.
template <int LAST>
__global__ void __launch_bounds__(MK_FFT_NT, 2) mk_prop_cols_kernel(const __grid_constant__ MkColsArgs A)
{
    extern __shared__ __align__(16) float2 s_lines[];
    constexpr int RL = 1 << LAST;
    const int N = A.nz2, W = A.W, P = (A.logn - LAST) / 3;
    const int logw = 31 - __clz(W), items = W * (N >> 3);
    const int c0 = blockIdx.x * W;
    // forward passes
    const float2 *tw = A.tw;
    for (int p = 0; p < P; ++p) {
        const int logm = A.logn - 3 * (p + 1), m = 1 << logm;
        for (int t = threadIdx.x; t < items; t += MK_FFT_NT) {
            const int c = t & (W - 1), q = t >> logw;
            const int i = q & (m - 1), base = ((q >> logm) << (logm + 3)) + i;
            float2 *line = s_lines + c * A.ld;
            float2 v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
                v[r] = p == 0 ? mk_cols_load(A, base + (r << logm), c0 + c) : line[mk_pad8(base + (r << logm))];
            mk_dft<8, false>(v);
            line[mk_pad8(base)] = v[0];
#pragma unroll
            for (int k = 1; k < 8; ++k)
                line[mk_pad8(base + (k << logm))] = mk_cmul(v[k], __ldg(tw + (k - 1) * m + i));
        }
        tw += 7 * m;
        __syncthreads();
    }
    // last radix, H, and back: 8 consecutive positions a thread
    for (int t = threadIdx.x; t < items; t += MK_FFT_NT) {
        const int c = t & (W - 1), q = t >> logw;
        float2 *line = s_lines + c * A.ld + 9 * q;             // mk_pad8(8 q)
        const float a = A.ky[c0 + c];
        float2 v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = line[j];
#pragma unroll
        for (int g = 0; g < 8 / RL; ++g) {
            mk_dft<RL, false>(v + g * RL);
            // the frequency of position 8 q + g RL + k: its digits reversed
            const int pos = 8 * q + g * RL;
            int f = 0;
            for (int p = 0; p < P; ++p) f |= ((pos >> (A.logn - 3 * (p + 1))) & 7) << (3 * p);
#pragma unroll
            for (int k = 0; k < RL; ++k)
                v[g * RL + k] = mk_cols_mul(A, v[g * RL + k], a, A.kz[f + (k << (3 * P))]);
            mk_dft<RL, true>(v + g * RL);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) line[j] = v[j];
    }
    __syncthreads();
    // inverse passes
    for (int p = P - 1; p >= 0; --p) {
        const int logm = A.logn - 3 * (p + 1), m = 1 << logm;
        tw -= 7 * m;
        for (int t = threadIdx.x; t < items; t += MK_FFT_NT) {
            const int c = t & (W - 1), q = t >> logw;
            const int i = q & (m - 1), base = ((q >> logm) << (logm + 3)) + i;
            float2 *line = s_lines + c * A.ld;
            float2 v[8];
            v[0] = line[mk_pad8(base)];
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                float2 w = __ldg(tw + (k - 1) * m + i);
                w.y = -w.y;
                v[k] = mk_cmul(line[mk_pad8(base + (k << logm))], w);
            }
            mk_dft<8, true>(v);
            if (p > 0) {
#pragma unroll
                for (int r = 0; r < 8; ++r) line[mk_pad8(base + (r << logm))] = v[r];
            } else {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int s = base + (r << logm) - A.z0;
                    if ((unsigned)s < (unsigned)A.nz) A.F[(size_t)s * A.ny2 + c0 + c] = v[r];
                }
            }
        }
        if (p > 0) __syncthreads();
    }
}

// Column lengths 2, 4 and 8: a thread a column, in registers.
template <int N>
__global__ void mk_prop_cols_short_kernel(const __grid_constant__ MkColsArgs A)
{
    const int col = blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= A.ny2) return;
    float2 v[N];
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = mk_cols_load(A, r, col);
    mk_dft<N, false>(v);
#pragma unroll
    for (int r = 0; r < N; ++r) v[r] = mk_cols_mul(A, v[r], A.ky[col], A.kz[r]);
    mk_dft<N, true>(v);
#pragma unroll
    for (int r = 0; r < N; ++r) {
        const int s = r - A.z0;
        if ((unsigned)s < (unsigned)A.nz) A.F[(size_t)s * A.ny2 + col] = v[r];
    }
}

// The tables of a column pass: the passes' twiddles exp(-2 pi i i k / M), (7, M / 8)
// of every M = nz2, nz2 / 8, .. >= 8, from FP64 sincospi, and 2 pi fftfreq +
// offset of every column and row as float32 (numpy ordering, in FP64). A warp a
// block: the FP64 pipe of every SM.
__global__ void mk_prop_tables_kernel(float2 *__restrict__ tw, float *__restrict__ ky, float *__restrict__ kz,
                                      int ny2, int nz2, double dy, double dz, double offy, double offz)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nz2) {
        int M = nz2, e = i;
        while (M >= 8 && e >= 7 * (M / 8)) {
            e -= 7 * (M / 8);
            M /= 8;
        }
        if (M >= 8) {
            const int k = e / (M / 8) + 1, t = (e % (M / 8)) * k * (nz2 / M);
            double s, c;
            sincospi(-2.0 * (double)t / (double)nz2, &s, &c);
            tw[i] = make_float2((float)c, (float)s);
        }
        kz[i] = (float)(MK_TWO_PI * mk_fftfreq(i, nz2, dz) + offz);
    }
    if (i < ny2) ky[i] = (float)(MK_TWO_PI * mk_fftfreq(i, ny2, dy) + offy);
}

// Points between a line's start and the next: its padded length, rounded up to
// 16 / W (mod 16) points.
static int mk_prop_ld(int nz2, int W)
{
    int ld = nz2 + nz2 / 8;
    while (ld % 16 != (16 / W) % 16) ++ld;
    return ld;
}

// Columns a block: as many as three blocks an SM leave room for, at least 4
// (whole 32-byte sectors) where one block can hold them, at most 16 and the
// row length.
static int mk_prop_cols_width(int ny2, int nz2)
{
    int W = 16;
    while (W > 4 && sizeof(float2) * (size_t)W * mk_prop_ld(nz2, W) > MK_FFT_SMEM) W /= 2;
    while (W > 1 && sizeof(float2) * (size_t)W * mk_prop_ld(nz2, W) > MK_FFT_SMEM_MAX) W /= 2;
    return std::max(1, std::min(W, ny2));
}

extern "C" size_t mk_prop_cols_workspace_size(int ny2, int nz2)
{
    if (ny2 <= 0 || nz2 <= 0) return 0;
    return sizeof(float2) * (size_t)nz2 + sizeof(float) * ((size_t)ny2 + (size_t)nz2) + 256;
}

extern "C" int mk_prop_cols_rows(float *spectrum, int ny2, int nz2, int z0, int nz, int mode,
                                 float cval_re, float cval_im, double dy, double dz, double k,
                                 double z, double k_axis, double k_perp_y, double k_perp_z,
                                 void *workspace, size_t ws_bytes, void *stream)
{
    MK_REQUIRE(spectrum && ny2 > 0 && nz2 > 0 && dy > 0.0 && dz > 0.0 && k > 0.0,
               "mk_prop_cols: bad arguments");
    MK_REQUIRE((nz2 & (nz2 - 1)) == 0 && nz2 >= 2 && nz2 <= MK_FFT_MAX,
               "mk_prop_cols: the column length %d must be a power of two in [2, %d]", nz2,
               MK_FFT_MAX);
    MK_REQUIRE((ny2 & (ny2 - 1)) == 0, "mk_prop_cols: the row length %d must be a power of two",
               ny2);
    MK_REQUIRE(nz > 0 && z0 >= 0 && z0 + nz <= nz2 && (mode == 0 || mode == 1),
               "mk_prop_cols: %d rows at %d do not fit %d", nz, z0, nz2);
    const size_t need = mk_prop_cols_workspace_size(ny2, nz2);
    if (!workspace || ws_bytes < need) {
        mk_set_error("mk_prop_cols: workspace %zu bytes, need %zu", ws_bytes, need);
        return MK_ENOMEM;
    }
    MK_REQUIRE(((uintptr_t)workspace & 15) == 0, "mk_prop_cols: workspace must be 16-byte aligned");
    int logn = 0;
    while ((1 << logn) < nz2) ++logn;
    cudaStream_t st = mk_stream(stream);
    float2 *tw = reinterpret_cast<float2 *>(workspace);
    float *ky = reinterpret_cast<float *>(tw + nz2);
    float *kz = ky + ny2;
    mk_prop_tables_kernel<<<(std::max(ny2, nz2) + 31) / 32, 32, 0, st>>>(tw, ky, kz, ny2, nz2, dy, dz,
                                                                           k_perp_y, k_perp_z);
    MK_CHECK_CUDA(cudaGetLastError());
    MkColsArgs A;
    memset(&A, 0, sizeof(A));
    A.F = reinterpret_cast<float2 *>(spectrum);
    A.ny2 = ny2;
    A.nz2 = nz2;
    A.logn = logn;
    A.z0 = z0;
    A.nz = nz;
    A.mode = mode;
    A.cval = make_float2(cval_re * (float)ny2, cval_im * (float)ny2);
    A.tw = tw;
    A.ky = ky;
    A.kz = kz;
    A.k = (float)k;
    A.z = (float)z;
    A.c_prop = (float)fmod(z * (k - k_axis), MK_TWO_PI);
    A.c_evan = (float)fmod(-z * k_axis, MK_TWO_PI);
    if (logn <= 3) {
        auto fn = logn == 1 ? mk_prop_cols_short_kernel<2>
                            : (logn == 2 ? mk_prop_cols_short_kernel<4> : mk_prop_cols_short_kernel<8>);
        fn<<<(ny2 + 127) / 128, 128, 0, st>>>(A);
        MK_CHECK_CUDA(cudaGetLastError());
        return MK_OK;
    }
    A.W = mk_prop_cols_width(ny2, nz2);
    A.ld = mk_prop_ld(nz2, A.W);
    const size_t smem = sizeof(float2) * (size_t)A.W * (size_t)A.ld;
    const int last = logn % 3 == 0 ? 3 : logn % 3;
    auto fn = last == 1 ? mk_prop_cols_kernel<1> : (last == 2 ? mk_prop_cols_kernel<2> : mk_prop_cols_kernel<3>);
    // the same value with every launch: another thread's smaller transform must not
    // lower the limit before this one's launch
    if (smem > (48u << 10))
        MK_CHECK_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)MK_FFT_SMEM_MAX));
    fn<<<ny2 / A.W, MK_FFT_NT, smem, st>>>(A);
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

extern "C" int mk_prop_cols(float *spectrum, int ny2, int nz2, double dy, double dz, double k,
                            double z, double k_axis, double k_perp_y, double k_perp_z,
                            void *workspace, size_t ws_bytes, void *stream)
{
    return mk_prop_cols_rows(spectrum, ny2, nz2, 0, nz2, 0, 0.f, 0.f, dy, dz, k, z, k_axis, k_perp_y,
                             k_perp_z, workspace, ws_bytes, stream);
}

extern "C" int mk_prop_pad(const float *field, int ny, int nz, float *padded, int ny2, int nz2,
                           int y0, int z0, int mode, float cval_re, float cval_im, void *stream)
{
    MK_REQUIRE(field && padded && ny > 0 && nz > 0 && ny2 >= ny && nz2 >= nz,
               "mk_prop_pad: bad arguments");
    MK_REQUIRE(y0 >= 0 && z0 >= 0 && y0 + ny <= ny2 && z0 + nz <= nz2, "mk_prop_pad: bad offsets");
    MK_REQUIRE(mode == 0 || mode == 1, "mk_prop_pad: mode must be 0 (edge) or 1 (constant)");
    const bool two = ny2 % 2 == 0 && ((uintptr_t)padded & 15) == 0;
    dim3 g((ny2 / (two ? 2 : 1) + 255) / 256, nz2);
    auto fn = two ? mk_prop_pad_kernel<2> : mk_prop_pad_kernel<1>;
    fn<<<g, 256, 0, mk_stream(stream)>>>(reinterpret_cast<const float2 *>(field), ny, nz,
                                         reinterpret_cast<float2 *>(padded), ny2, nz2, y0, z0, mode,
                                         make_float2(cval_re, cval_im));
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

extern "C" int mk_prop_mul(float *spectrum, int ny2, int nz2, double dy, double dz, double k,
                           double z, double k_axis, double k_perp_y, double k_perp_z, void *stream)
{
    MK_REQUIRE(spectrum && ny2 > 0 && nz2 > 0 && dy > 0.0 && dz > 0.0 && k > 0.0,
               "mk_prop_mul: bad arguments");
    dim3 g((ny2 + 255) / 256, nz2);
    mk_prop_mul_kernel<<<g, 256, 0, mk_stream(stream)>>>(reinterpret_cast<float2 *>(spectrum), ny2,
                                                        nz2, dy, dz, k, z, k_axis, k_perp_y,
                                                        k_perp_z);
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}

extern "C" int mk_prop_crop_abs2(const float *grid, int ny2, int nz2, int y0, int z0, int ny,
                                 int nz, float scale, float *field, float *intensity, void *stream)
{
    MK_REQUIRE(grid && ny > 0 && nz > 0 && y0 >= 0 && z0 >= 0 && y0 + ny <= ny2 && z0 + nz <= nz2,
               "mk_prop_crop_abs2: bad arguments");
    MK_REQUIRE(field || intensity, "mk_prop_crop_abs2: nothing to write");
    dim3 g((ny + 255) / 256, nz);
    mk_prop_crop_kernel<<<g, 256, 0, mk_stream(stream)>>>(reinterpret_cast<const float2 *>(grid),
                                                         ny2, nz2, y0, z0, ny, nz, scale,
                                                         reinterpret_cast<float2 *>(field),
                                                         intensity);
    MK_CHECK_CUDA(cudaGetLastError());
    return MK_OK;
}
