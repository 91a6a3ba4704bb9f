// FP64 plain direct sum: the reference CPU kernel's arithmetic term for term
// (compute_scattering_cffi, MOSAIC Beam.py:748-808) on the GPU.
//
// This translation unit is compiled with --fmad=false so that, like the
// uncontracted C oracle, every product and sum rounds separately: the
// absolute phase k (x + r) is ~1e10 rad, where one double ulp is ~2e-6 rad,
// and a contracted build would differ from the CPU result at that level.
#include <type_traits>

#include "mk_common.cuh"

int mk_launch_reduce(const double2 *partial, int slices, int n_pix, const double2 *phasor,
                     double scale, double2 *out, int accumulate, cudaStream_t st);

#define F64_NT 128
#define F64_ATOMS 128   // atoms staged in shared memory per step

// x mod y with the sign of x, exactly as C fmod: the remainder of two doubles
// is representable, so fma(-q, y, x) with the right integer quotient q
// returns it without rounding; q from the product with 1/y (rounded, so at
// most one off for |x| < 2^52 y) is corrected when it lands on the wrong
// side. A division here cost ~20 operations of the FP64 pipe.
__device__ __forceinline__ double mk_fmod_exact(double x, double y, double inv_y)
{
    const double ax = fabs(x);
    if (ax < y) return x;
    double q = trunc(ax * inv_y);
    double r = fma(-q, y, ax);
    if (r < 0.0) { q -= 1.0; r = fma(-q, y, ax); }
    else if (r >= y) { q += 1.0; r = fma(-q, y, ax); }
    return x < 0.0 ? -r : r;
}

struct MkPlainArgs {
    MkSpecies sp;
    double k;
    int apply_pol, decay, remove_forward;
    double pdeg, ex, ey, ez;
    int analyser;                      // 0 off, 1 top-hat, 2 Darwin
    double ax, ay, az, x_accept, hw;   // axis, 4 sin^2(alpha/2), half-width
};

// Largest |a| / |P| at which the direction-dependent factors are taken from
// their expansion about the pixel's own direction. Per pixel and species the
// kernel holds the factor F there (f0 + f' + i f'', Debye-Waller, polarization)
// and the first two derivatives of f0 in cos(2 theta); per term only the
// CHANGE from the pixel's direction, 1 + eta, is formed in FP32 and multiplied
// into the phasor, and F into the sum of a species' terms. With e = |a| / |P|, d_i =
// b_i / (2 lambda^2) and f_i the Gaussians of f0, the change of f0 is at most sum
// |f_i| d_i (sin(2 theta) e + e^2); FP32 forms the change of cos(2 theta) to 3
// roundings of e and the product to 4 of itself. The expansion is taken where that
// stays below 1e-12 of |F|, the third order below 2e-13 and the Debye-Waller
// factor's roundings below 5e-13 of theirs (tested per pixel and species: it
// holds for tabulated atoms at 8 to 20 keV, and fails near forward at high
// energies, for very wide electron clouds and where F cancels). Polarization and
// decay change by e at most, their second order is below 1e-13 for P_pol > 1/4;
// with the sine and cosine below, a term is within 2e-12 of its size. Beyond
// the limit, with an analyser, at P_pol < 1/4 and at the Q_cut edge every factor
// is evaluated per term as the reference does.
//
// The phase k (a_x + r) keeps the reference's roundings bit for bit. r = the
// rounded root of v = |P - a|^2 comes from a start r0 = R0 - u.a + (|a|^2 -
// (u.a)^2) / 2 R0, its change from R0 in FP32: within |a| 2e-7 of r (240 ulps at
// the limit), so that r0 + (v - r0^2) / (2 r0), one Newton step with the residue
// from an FMA and 1 / r0 to 1e-14, is r to 1e-11 ulp before its rounding.
// The sine and cosine of fmod(x, 2 pi) (2 pi the double) come from a table: x =
// q h + d with h = 2 pi / 1024, q h exact to d's last bit in one FMA and q read
// off the low bits of x / h + 1.5 2^52 (|x| < 1e13); the rotation by d is
// 1 + i d in FP64, and its higher orders (d^2 / 2 <= 5e-6, d^3 / 6) in FP32,
// 3e-13 at most, next to the 2e-6 rad that one ulp of the phase is worth.
// FP32 values enter and leave FP64 by their bits: a conversion is an operation
// of the FP64 pipe too.
//
// The kernel is bound by that pipe (2 lane operations per clock and SM). A term
// was ~320 operations (5 exp, 2 divisions, 3 square roots, fmod, sincos):
// 32,000 atoms x 1,920 pixels 31.3 ms; ~60 with the factors expanded and a sine
// table of 256 angles and FP64 polynomials: 7.2 ms; 23 now (25 with complex
// amplitudes): 3.0 ms, in even slices 2.7.
#define F64_FAR 1.5e-7f
#define F64_PHASE_MAX 1e13   // largest phase the table's reduction takes [rad]
#define F64_CS 1024          // table angles

// A float's value by its bits; 0 below the smallest normal number.
__device__ __forceinline__ double mk_widen(float f)
{
    const unsigned b = __float_as_uint(f);
    const unsigned hi = (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20));
    return __hiloint2double((b & 0x7f800000u) ? (int)hi : 0, (b & 0x7f800000u) ? (int)(b << 29) : 0);
}

// A double in (1e-37, 1e38) or 0 rounded to float by its bits; smaller ones 0.
__device__ __forceinline__ float mk_narrow(double d)
{
    const long long b = __double_as_longlong(d) + (1ll << 28);
    const unsigned hi = (unsigned)(b >> 32), mag = hi & 0x7fffffffu;
    const unsigned m = __funnelshift_l((unsigned)b, mag - (896u << 20), 3);
    return __uint_as_float(mag > (897u << 20) ? (hi & 0x80000000u) | m : 0u);
}

template <bool FAR>
__global__ void __launch_bounds__(F64_NT) mk_plain_f64_kernel(
    int64_t n, int64_t atoms_per_slice, const double *__restrict__ pos,
    const int *__restrict__ species, const float2 *__restrict__ amp, int n_pix,
    const double *__restrict__ xyz, const double *__restrict__ r0v,
    const double4 *__restrict__ qv, const __grid_constant__ MkPlainArgs A,
    double2 *__restrict__ partial)
{
    __shared__ double s_pos[F64_ATOMS][3];
    __shared__ double2 s_amp[F64_ATOMS];
    __shared__ float4 s_posf[F64_ATOMS];          // position in FP32, species (bits)
    __shared__ float s_aa[F64_ATOMS];             // |a|^2
    __shared__ int s_complex;                     // an amplitude of the step has an imaginary part
    __shared__ double s_ani[MK_MAX_SPECIES];
    __shared__ float s_wk[MK_MAX_SPECIES][11];
    __shared__ double2 s_cs[FAR ? F64_CS : 1];    // cos, sin of j 2 pi / F64_CS
    __shared__ float2 s_csf[FAR ? F64_CS : 1];
    __shared__ unsigned s_far;                    // largest |a| of the step, float bits
    extern __shared__ __align__(16) double2 s_F[];           // FAR: [S][NT] F, then f0', f0''/2 and 1/F0
    float4 *s_df = reinterpret_cast<float4 *>(s_F + (FAR ? A.sp.n * F64_NT : 0));
    const int p = blockIdx.x * F64_NT + threadIdx.x;
    const bool live = p < n_pix;
    for (int i = threadIdx.x; i < MK_MAX_SPECIES * 11; i += F64_NT)
        s_wk[i / 11][i % 11] = A.sp.wk[i / 11][i % 11];
    if (threadIdx.x < MK_MAX_SPECIES) s_ani[threadIdx.x] = A.sp.ani[threadIdx.x];
    const double cx = live ? xyz[3 * p] : 0.0, cy = live ? xyz[3 * p + 1] : 0.0,
                 cz = live ? xyz[3 * p + 2] : 0.0;
    const double R0 = live ? r0v[p] : 0.0, qcut = live ? qv[p].w : 0.0;
    const double s_fac = 0.25e-10 / MK_PI;
    const double inv_2pi = 1.0 / MK_TWO_PI;
    double acc_r = 0.0, acc_i = 0.0;
    const int64_t a_lo = (int64_t)blockIdx.y * atoms_per_slice;
    const int64_t a_hi = min(n, a_lo + atoms_per_slice);

    // the pixel's own direction: ux = cos(2 theta), and what changes with it
    bool expand = false, forward = false;
    double scale0 = MK_R_E, half_inv = 0.0;
    float vx = 0.f, vy = 0.f, vz = 0.f, inv_R = 0.f, inv_P = 0.f, gx = 0.f, s2x = 0.f, ex = 0.f, ey = 0.f,
          ez = 0.f, eu = 0.f;
    if (FAR) {
        // every fourth angle by sincos, the three after it by rotation
        double c1[3], s1[3];
        for (int i = 0; i < 3; ++i) sincos((i + 1) * (MK_TWO_PI / F64_CS), &s1[i], &c1[i]);
        for (int i = threadIdx.x; i < F64_CS / 4; i += F64_NT) {
            double sn, c;
            sincos(i * (4.0 * MK_TWO_PI / F64_CS), &sn, &c);
            for (int j = 0; j < 4; ++j) {
                const double2 v = j == 0 ? make_double2(c, sn)
                                         : make_double2(fma(c, c1[j - 1], -(sn * s1[j - 1])),
                                                        fma(sn, c1[j - 1], c * s1[j - 1]));
                s_cs[4 * i + j] = v;
                s_csf[4 * i + j] = make_float2((float)v.x, (float)v.y);
            }
        }
        __syncthreads();
        if (live && R0 > 0.0) {
            expand = A.k * R0 < 0.25 * F64_PHASE_MAX;       // x = k (a_x + r) < 2.1 k R0
            const double ux = cx / R0;
            half_inv = 0.5 / R0;
            const double uy = cy / R0, uz = cz / R0;
            vx = (float)ux; vy = (float)uy; vz = (float)uz;
            inv_R = (float)(1.0 / R0);
            const float across0 = sqrtf(fmaf(vz, vz, vy * vy));          // sin(2 theta)
            const double g = fmax(2.0 * (1.0 - ux), 0.0), Q = A.k * sqrt(g);
            const double sk = s_fac * A.k, s2 = sk * sk * g, ds2 = -2.0 * sk * sk;   // d s2 / d ux
            s2x = (float)ds2;
            if (A.remove_forward) {
                forward = Q < qcut;
                if (!(fabs(Q - qcut) > 1e-6 * A.k)) expand = false;   // Q changes by k e at most
            }
            if (A.apply_pol) {
                const double e = A.ex * ux + A.ey * uy + A.ez * uz;
                const double P = 0.5 * (1.0 - A.pdeg) * (1.0 + ux * ux) + A.pdeg * (1.0 - e * e);
                if (!(P > 0.25)) expand = false;
                scale0 *= sqrt(fmin(P, 1.0));
                inv_P = (float)(1.0 / P);
                gx = (float)((1.0 - A.pdeg) * ux);
                eu = (float)e;
                ex = (float)A.ex; ey = (float)A.ey; ez = (float)A.ez;
            }
            for (int s = 0; s < A.sp.n; ++s) {
                const float *wk = s_wk[s];
                double f0 = wk[5], f1 = 0.0, f2 = 0.0, f1_abs = 0.0;
                float b_max = 0.f;
                for (int i = 0; i < 5; ++i) {
                    const double b = (double)wk[6 + i], t = (double)wk[i] * exp(-b * s2), d = -b * ds2, td = t * d;
                    f0 += t;
                    f1 += td;
                    f1_abs += fabs(td);
                    f2 += td * d;
                    b_max = fmaxf(b_max, fabsf(wk[6 + i]));
                }
                double fre = f0 + A.sp.anr[s], fim = A.sp.ani[s];
                if (forward) {
                    fre -= (double)A.sp.f0z[s] + A.sp.anr[s];
                    fim = 0.0;
                }
                // F0 + change as F0 (1 + change / F0), each remainder against F0
                const double m2 = fre * fre + fim * fim;
                const double round = f1_abs * (F64_FAR * 0x1p-24) * (double)(3.f + 4.f * across0);
                const double d_e = (double)(b_max * -s2x * F64_FAR), third = f1_abs * F64_FAR * d_e * d_e / 6.0;
                if (!(round * round <= 1e-24 * m2 && third * third <= 4e-26 * m2)) expand = false;
                double w = scale0;
                if (A.sp.has_dw) {
                    w *= exp(-(double)A.sp.dwb[s] * s2);
                    if (!(fabsf(A.sp.dwb[s] * s2x) * (F64_FAR * 0x1p-24f) * (3.f + 4.f * across0) <= 5e-13f))
                        expand = false;
                }
                s_F[s * F64_NT + threadIdx.x] = make_double2(fre * w, fim * w);
                s_df[s * F64_NT + threadIdx.x] =
                    make_float4((float)f1, (float)(0.5 * f2), (float)(fre / m2), (float)(-fim / m2));
            }
        }
    }
    for (int64_t a0 = a_lo; a0 < a_hi; a0 += F64_ATOMS) {
        const int m = (int)min((int64_t)F64_ATOMS, a_hi - a0);
        __syncthreads();
        if (threadIdx.x == 0) {
            s_far = 0u;
            s_complex = 0;
        }
        __syncthreads();
        for (int j = threadIdx.x; j < m; j += F64_NT) {
            const double x = pos[3 * (a0 + j)], y = pos[3 * (a0 + j) + 1], z = pos[3 * (a0 + j) + 2];
            s_pos[j][0] = x;
            s_pos[j][1] = y;
            s_pos[j][2] = z;
            const float2 e = amp[a0 + j];
            s_amp[j] = make_double2(e.x, e.y);
            s_posf[j] = make_float4((float)x, (float)y, (float)z, __int_as_float(species[a0 + j]));
            if (FAR) {
                const float aa = (float)x * (float)x + (float)y * (float)y + (float)z * (float)z, l = sqrtf(aa);
                s_aa[j] = aa;
                if (e.y != 0.f) s_complex = 1;
                atomicMax(&s_far, __float_as_uint(l <= 1e30f ? l : 1e30f));    // NaN: far out
            }
        }
        __syncthreads();
        if (!live) continue;
        if (FAR && expand && __uint_as_float(s_far) * inv_R < F64_FAR) {
            auto terms = [&](auto complex_amp) {
                double sr = 0.0, si = 0.0;
                int species = __float_as_int(s_posf[0].w);
                float4 df = s_df[species * F64_NT + threadIdx.x];
                auto flush = [&]() {
                    const double2 F = s_F[species * F64_NT + threadIdx.x];
                    acc_r = fma(F.x, sr, fma(-F.y, si, acc_r));
                    acc_i = fma(F.x, si, fma(F.y, sr, acc_i));
                };
                for (int j = 0; j < m; ++j) {
                    const double ax = s_pos[j][0], ay = s_pos[j][1], az = s_pos[j][2];
                    const float4 pf = s_posf[j];
                    const int s = __float_as_int(pf.w);
                    if (s != species) {            // uniform across the block
                        flush();
                        sr = si = 0.0;
                        species = s;
                        df = s_df[species * F64_NT + threadIdx.x];
                    }
                    const double dx = cx - ax, dy = cy - ay, dz = cz - az;
                    const double v = dx * dx + dy * dy + dz * dz;
                    const float ua = fmaf(vz, pf.z, fmaf(vy, pf.y, vx * pf.x)), across = fmaf(-ua, ua, s_aa[j]);
                    const float dr = fmaf(0.5f * inv_R, across, -ua);        // r - R0
                    const double r0 = R0 + mk_widen(dr);
                    const double r = fma(fma(-r0, r0, v), fma(half_inv, mk_widen(-dr * inv_R), half_inv), r0);
                    // cos and sin of the phase mod 2 pi
                    const double x = A.k * (ax + r), magic = 6755399441055744.0;
                    const double t52 = fma(x, F64_CS / MK_TWO_PI, magic);
                    const double d = fma(-(t52 - magic), MK_TWO_PI / F64_CS, x);
                    const int q = __double2loint(t52) & (F64_CS - 1);
                    const double2 cs = s_cs[q];
                    const float2 cf = s_csf[q];
                    const float d1 = mk_narrow(d), d2 = d1 * d1;
                    const float cd = d2 * fmaf(d2, 1.f / 24.f, -0.5f), sd = d1 * d2 * (-1.f / 6.f);   // cos d - 1, sin d - d
                    const float hc = fmaf(cf.x, cd, -cf.y * sd), hs = fmaf(cf.y, cd, cf.x * sd);
                    const float c1 = fmaf(-cf.y, d1, cf.x) + hc, s1 = fmaf(cf.x, d1, cf.y) + hs;
                    // change of cos(2 theta), to second order in e = a / R0
                    const float ue = ua * inv_R, exx = pf.x * inv_R;
                    const float t = fmaf(-exx, ue, fmaf(vx, ue, -exx)) +
                                    vx * fmaf(ue, ue, -0.5f * across * inv_R * inv_R);
                    float sig = A.decay ? ue : 0.f;      // R0 / r - 1
                    if (A.apply_pol) {
                        // P_pol's change over P_pol, and its root's; e.u' changes by te
                        const float te = -(fmaf(ez, pf.z, fmaf(ey, pf.y, ex * pf.x)) - ua * eu) * inv_R;
                        const float pd = (float)A.pdeg;
                        const float g = (t * fmaf(0.5f * (1.f - pd), t, gx) - pd * te * fmaf(2.f, eu, te)) * inv_P;
                        const float h = g * fmaf(-0.125f, g, 0.5f);
                        sig = fmaf(h, sig, h + sig);
                    }
                    if (A.sp.has_dw) {
                        const float b = -A.sp.dwb[s] * s2x * t, h = b * fmaf(0.5f, b, 1.f);
                        sig = fmaf(h, sig, h + sig);
                    }
                    // 1 + eta = (1 + change of f0 / F0) (1 + sig)
                    const float df0 = fmaf(df.y, t, df.x) * t, fr = df0 * df.z, fi = df0 * df.w;
                    const float er = fmaf(fr, sig, fr + sig), ei = fmaf(fi, sig, fi);
                    const double c = fma(-cs.y, d, cs.x) + mk_widen(fmaf(c1, er, fmaf(-s1, ei, hc)));
                    const double sn = fma(cs.x, d, cs.y) + mk_widen(fmaf(s1, er, fmaf(c1, ei, hs)));
                    const double2 E = s_amp[j];
                    sr = fma(E.x, c, sr);
                    si = fma(E.x, sn, si);
                    if constexpr (decltype(complex_amp)::value) {
                        sr = fma(-E.y, sn, sr);
                        si = fma(E.y, c, si);
                    }
                }
                flush();
            };
            if (s_complex) terms(std::true_type{});
            else terms(std::false_type{});
            continue;
        }
        for (int j = 0; j < m; ++j) {
            const double ax = s_pos[j][0], ay = s_pos[j][1], az = s_pos[j][2];
            const int s = __float_as_int(s_posf[j].w);
            const double dx = cx - ax, dy = cy - ay, dz = cz - az;
            const double r = sqrt(dx * dx + dy * dy + dz * dz);
            if (r == 0.0) continue;
            const double dotv = dx / r;
            const double g = 2.0 * (1.0 - dotv);
            const double Q = A.k * sqrt(g > 0.0 ? g : 0.0);
            const double sv = s_fac * Q, s2 = sv * sv;
            const float *wk = s_wk[s];
            double f0 = wk[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) f0 += (double)wk[i] * exp(-(double)wk[6 + i] * s2);
            const double fr = A.sp.anr[s], fi = A.sp.ani[s];
            double fre = f0 + fr, fim = fi;
            if (A.remove_forward && Q < qcut) {
                fre -= ((double)A.sp.f0z[s] + fr);
                fim -= fi;
            }
            if (A.sp.has_dw) {
                const double B = A.sp.dwb[s];
                if (B != 0.0) {
                    const double w = exp(-B * s2);
                    fre *= w;
                    fim *= w;
                }
            }
            const double er = s_amp[j].x, ei = s_amp[j].y;
            const double tr = er * fre - ei * fim, ti = er * fim + ei * fre;
            const double ph = mk_fmod_exact(A.k * (ax + r), MK_TWO_PI, inv_2pi);
            double sn, c;
            sincos(ph, &sn, &c);
            double scale = MK_R_E;
            if (A.decay && R0 > 0.0) scale *= R0 / r;
            if (A.apply_pol) {
                const double e = (A.ex * dx + A.ey * dy + A.ez * dz) / r;
                double P = 0.5 * (1.0 - A.pdeg) * (1.0 + dotv * dotv) + A.pdeg * (1.0 - e * e);
                P = P < 0.0 ? 0.0 : (P > 1.0 ? 1.0 : P);
                scale *= sqrt(P);
            }
            if (A.analyser) {
                const double vx = dx / r - A.ax, vy = dy / r - A.ay, vz = dz / r - A.az;
                scale *= mk_analyser_factor(A.analyser, vx * vx + vy * vy + vz * vz, A.x_accept,
                                            A.hw);
            }
            acc_r += (tr * c - ti * sn) * scale;
            acc_i += (tr * sn + ti * c) * scale;
        }
    }
    if (live) partial[(size_t)blockIdx.y * n_pix + p] = make_double2(acc_r, acc_i);
}

extern "C" size_t mk_sum_workspace_size(int n_pix, int slices)
{
    if (n_pix <= 0 || slices <= 0) return 256;
    return sizeof(double2) * (size_t)n_pix * (size_t)slices;
}

static int mk_plain_slices(int64_t n, int n_pix, int want)
{
    if (want > 0) return (int)std::min<int64_t>(want, std::max<int64_t>(1, (n + F64_ATOMS - 1) / F64_ATOMS));
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int64_t bx = (n_pix + F64_NT - 1) / F64_NT;
    int64_t s = (8LL * sms + bx - 1) / bx;
    s = std::min<int64_t>(s, std::max<int64_t>(1, (n + 4 * F64_ATOMS - 1) / (4 * F64_ATOMS)));
    return (int)std::max<int64_t>(1, std::min<int64_t>(s, 4096));
}

extern "C" int mk_kin_plain_f64(int64_t n, const double *pos, const int *species,
                                const float *amp, const mk_species *spc, const mk_physics *phys,
                                const mk_pixels *px, int slices, double *out, int accumulate,
                                void *workspace, size_t ws_bytes, void *stream)
{
    MK_REQUIRE(spc && phys && px && out, "mk_kin_plain_f64: null argument");
    MK_REQUIRE(n >= 0, "mk_kin_plain_f64: negative atom count");
    const int64_t np64 = (int64_t)px->ny * px->nz;
    MK_REQUIRE(px->ny > 0 && px->nz > 0 && np64 < (1ll << 31), "mk_kin_plain_f64: bad detector shape");
    MK_REQUIRE(n == 0 || (pos && species && amp), "mk_kin_plain_f64: null atom buffer");
    MK_REQUIRE(px->xyz && px->r0 && px->q, "mk_kin_plain_f64: pixels not prepared");
    MK_REQUIRE(phys->k > 0.0, "mk_kin_plain_f64: k must be positive");
    const int n_pix = (int)np64;
    MkPlainArgs A;
    int rc = mk_species_pack(spc, &A.sp);
    if (rc != MK_OK) return rc;
    A.k = phys->k;
    A.apply_pol = phys->apply_pol;
    A.decay = phys->spherical_decay;
    A.remove_forward = phys->remove_forward;
    A.pdeg = phys->pol_deg;
    A.ex = phys->pol_e[0];
    A.ey = phys->pol_e[1];
    A.ez = phys->pol_e[2];
    rc = mk_analyser_pack(phys, &A.analyser, &A.ax, &A.ay, &A.az, &A.x_accept, &A.hw);
    if (rc != MK_OK) return rc;
    cudaStream_t st = mk_stream(stream);
    if (n == 0) {
        if (!accumulate) MK_CHECK_CUDA(cudaMemsetAsync(out, 0, sizeof(double2) * (size_t)n_pix, st));
        return MK_OK;
    }
    const int ns = mk_plain_slices(n, n_pix, slices);
    const size_t need = sizeof(double2) * (size_t)ns * n_pix;
    if (!workspace || ws_bytes < need) {
        mk_set_error("mk_kin_plain_f64: workspace %zu bytes, need %zu (slices=%d)", ws_bytes, need, ns);
        return MK_ENOMEM;
    }
    int64_t per = (n + ns - 1) / ns;
    per = ((per + 31) / 32) * 32;
    const int ns_eff = (int)((n + per - 1) / per);
    dim3 grid((n_pix + F64_NT - 1) / F64_NT, ns_eff);
    double2 *part = static_cast<double2 *>(workspace);
    // expansions per (species, pixel): the factor and its derivatives
    const size_t smem = A.analyser ? 0 : (sizeof(double2) + sizeof(float4)) * (size_t)A.sp.n * F64_NT;
    auto fn = A.analyser ? mk_plain_f64_kernel<false> : mk_plain_f64_kernel<true>;
    // the same value with every launch: threads with fewer species must not lower
    // the limit between another's setting it and its launch
    MK_CHECK_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)((sizeof(double2) + sizeof(float4)) * MK_MAX_SPECIES * F64_NT)));
    fn<<<grid, F64_NT, smem, st>>>(n, per, pos, species, reinterpret_cast<const float2 *>(amp), n_pix, px->xyz,
                                   px->r0, reinterpret_cast<const double4 *>(px->q), A, part);
    MK_CHECK_CUDA(cudaGetLastError());
    return mk_launch_reduce(part, ns_eff, n_pix, nullptr, 1.0, reinterpret_cast<double2 *>(out),
                            accumulate, st);
}
