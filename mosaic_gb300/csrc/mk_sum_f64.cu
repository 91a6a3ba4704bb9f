// FP64 plain direct sum: the reference CPU kernel's arithmetic term for term
// (compute_scattering_cffi, MOSAIC Beam.py:748-808) on the GPU.
//
// This translation unit is compiled with --fmad=false so that, like the
// uncontracted C oracle, every product and sum rounds separately: the
// absolute phase k (x + r) is ~1e10 rad, where one double ulp is ~2e-6 rad,
// and a contracted build would differ from the CPU result at that level.
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
// kernel holds f0 and its first two derivatives in cos(2 theta); per term only
// the CHANGE from the pixel's direction is formed in FP32 and added to the
// FP64 value. At the limit, with c = b / (2 lambda^2) <= 240 (b <= 180 A^2, 20
// keV): the change is at most c e = 4e-5 of a term of f0, so FP32 leaves 2e-12
// of that term (1e-13 for the b ~ 1/s^2 that count at a reflection); f0's third
// order (c e)^3 / 6 is 8e-15, the direction's second order in polarization and
// decay below 1e-13 for P_pol > 1/4. Beyond the limit, with an analyser, at
// P_pol < 1/4 and at the Q_cut edge every factor is evaluated per term as the
// reference does.
// There the sine and cosine of fmod(x, 2 pi) (2 pi the double) come from a
// table: x = q h + d with h = 2 pi / 256, q h exact to d's last bit in one FMA
// and q read off the low bits of x / h + 1.5 2^52 (|x| < 1e13); cos and sin of
// d, |d| <= h / 2, are their Taylor polynomials to d^6 and d^5 (below 9e-18),
// and those of the table's angle rotate them. Absolute error ~2e-16, next to
// the 2e-6 rad that one ulp of the phase is worth.
// The kernel is bound by the FP64 pipe (2 lane operations per clock and SM):
// of ~320 operations a term most went to 5 exp, 2 divisions, 2 further square
// roots, fmod and sincos (32,000 atoms x 1,920 pixels: 31.3 ms); with the
// factors expanded 10.1 ms, with the table 7.2 ms.
#define F64_FAR 1.5e-7f
#define F64_PHASE_MAX 1e13   // largest phase the table's reduction takes [rad]
#define F64_CS 256           // table angles

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
    __shared__ double s_ani[MK_MAX_SPECIES];
    __shared__ float s_wk[MK_MAX_SPECIES][11];
    __shared__ double2 s_cs[FAR ? F64_CS : 1];    // cos, sin of j 2 pi / F64_CS
    __shared__ unsigned s_far;                    // largest |a| of the step, float bits
    extern __shared__ __align__(16) double s_f0[];           // FAR: [S][NT], then the derivatives
    float2 *s_df = reinterpret_cast<float2 *>(s_f0 + (FAR ? A.sp.n * F64_NT : 0));
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
    double ux = 0.0, scale0 = MK_R_E;
    float vx = 0.f, vy = 0.f, vz = 0.f, inv_R = 0.f, inv_P = 0.f, gx = 0.f, s2x = 0.f, ex = 0.f, ey = 0.f,
          ez = 0.f, eu = 0.f;
    if (FAR) {
        for (int i = threadIdx.x; i < F64_CS; i += F64_NT) {
            double sn, c;
            sincos(i * (MK_TWO_PI / F64_CS), &sn, &c);
            s_cs[i] = make_double2(c, sn);
        }
        __syncthreads();
        if (live && R0 > 0.0) {
            expand = A.k * R0 < 0.25 * F64_PHASE_MAX;       // x = k (a_x + r) < 2.1 k R0
            ux = cx / R0;
            const double uy = cy / R0, uz = cz / R0;
            vx = (float)ux; vy = (float)uy; vz = (float)uz;
            inv_R = (float)(1.0 / R0);
            const double g = fmax(2.0 * (1.0 - ux), 0.0), Q = A.k * sqrt(g);
            const double sk = s_fac * A.k, s2 = sk * sk * g, ds2 = -2.0 * sk * sk;   // d s2 / d ux
            s2x = (float)ds2;
            if (A.remove_forward) {
                forward = Q < qcut;
                if (!(fabs(Q - qcut) > 1e-6 * A.k)) expand = false;   // Q changes by k e at most
            }
            for (int s = 0; s < A.sp.n; ++s) {
                const float *wk = s_wk[s];
                double f0 = wk[5], f1 = 0.0, f2 = 0.0;
                for (int i = 0; i < 5; ++i) {
                    const double b = (double)wk[6 + i], t = (double)wk[i] * exp(-b * s2), d = -b * ds2;
                    f0 += t;
                    f1 += t * d;
                    f2 += t * d * d;
                }
                double fre = f0 + A.sp.anr[s];
                if (forward) fre -= (double)A.sp.f0z[s] + A.sp.anr[s];
                double w = 1.0;
                if (A.sp.has_dw) w = exp(-(double)A.sp.dwb[s] * s2);
                s_f0[s * F64_NT + threadIdx.x] = fre;
                s_df[s * F64_NT + threadIdx.x] = make_float2((float)f1, (float)(0.5 * f2));
                if (A.sp.has_dw) s_f0[(2 * A.sp.n + s) * F64_NT + threadIdx.x] = w;
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
        }
    }
    for (int64_t a0 = a_lo; a0 < a_hi; a0 += F64_ATOMS) {
        const int m = (int)min((int64_t)F64_ATOMS, a_hi - a0);
        __syncthreads();
        if (threadIdx.x == 0) s_far = 0u;
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
                const float l = sqrtf((float)x * (float)x + (float)y * (float)y + (float)z * (float)z);
                atomicMax(&s_far, __float_as_uint(l <= 1e30f ? l : 1e30f));    // NaN: far out
            }
        }
        __syncthreads();
        if (!live) continue;
        if (FAR && expand && __uint_as_float(s_far) * inv_R < F64_FAR) {
            for (int j = 0; j < m; ++j) {
                const double ax = s_pos[j][0], ay = s_pos[j][1], az = s_pos[j][2];
                const float4 pf = s_posf[j];
                const int s = __float_as_int(pf.w);
                const double dx = cx - ax, dy = cy - ay, dz = cz - az;
                const double r = sqrt(dx * dx + dy * dy + dz * dz);
                // cos and sin of the phase mod 2 pi
                const double x = A.k * (ax + r), magic = 6755399441055744.0;
                const double t52 = fma(x, F64_CS / MK_TWO_PI, magic);
                const double d = fma(-(t52 - magic), MK_TWO_PI / F64_CS, x);
                const double2 cs = s_cs[__double2loint(t52) & (F64_CS - 1)];
                const double d2 = d * d;
                const double sd = fma(d * d2, fma(d2, 1.0 / 120.0, -1.0 / 6.0), d);
                const double cd = d2 * fma(d2, fma(d2, -1.0 / 720.0, 1.0 / 24.0), -0.5);   // cos d - 1
                const double c = fma(cs.x, cd, fma(-cs.y, sd, cs.x));
                const double sn = fma(cs.y, cd, fma(cs.x, sd, cs.y));
                const float ua = fmaf(vz, pf.z, fmaf(vy, pf.y, vx * pf.x));
                // change of cos(2 theta): (dx - ux r) / r, the difference in FP64
                const float t = (float)(dx - ux * r) * inv_R;
                const float2 df = s_df[s * F64_NT + threadIdx.x];
                const double fre = s_f0[s * F64_NT + threadIdx.x] + (double)(fmaf(df.y, t, df.x) * t);
                const double fim = forward ? 0.0 : s_ani[s];
                float sig = A.decay ? ua * inv_R : 0.f;      // R0 / r - 1
                if (A.apply_pol) {
                    // P_pol's change over P_pol, and its root's; e.u' changes by te
                    const float te = -(fmaf(ez, pf.z, fmaf(ey, pf.y, ex * pf.x)) - ua * eu) * inv_R;
                    const float pd = (float)A.pdeg;
                    const float q = (t * fmaf(0.5f * (1.f - pd), t, gx) - pd * te * fmaf(2.f, eu, te)) * inv_P;
                    const float h = q * fmaf(-0.125f, q, 0.5f);
                    sig = fmaf(h, sig, h + sig);
                }
                double sc = scale0;
                if (A.sp.has_dw) {
                    const float d = -A.sp.dwb[s] * s2x * t, h = d * fmaf(0.5f, d, 1.f);
                    sig = fmaf(h, sig, h + sig);
                    sc *= s_f0[(2 * A.sp.n + s) * F64_NT + threadIdx.x];
                }
                const double scale = fma(sc, (double)sig, sc);
                const double er = s_amp[j].x, ei = s_amp[j].y;
                const double tr = er * fre - ei * fim, ti = er * fim + ei * fre;
                acc_r += (tr * c - ti * sn) * scale;
                acc_i += (tr * sn + ti * c) * scale;
            }
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
    per = ((per + F64_ATOMS - 1) / F64_ATOMS) * F64_ATOMS;
    const int ns_eff = (int)((n + per - 1) / per);
    dim3 grid((n_pix + F64_NT - 1) / F64_NT, ns_eff);
    double2 *part = static_cast<double2 *>(workspace);
    // expansions per (species, pixel): f0, its derivatives and the Debye-Waller factor
    const size_t smem = A.analyser ? 0 : (A.sp.has_dw ? 3 : 2) * sizeof(double) * (size_t)A.sp.n * F64_NT;
    auto fn = A.analyser ? mk_plain_f64_kernel<false> : mk_plain_f64_kernel<true>;
    MK_CHECK_CUDA(cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fn<<<grid, F64_NT, smem, st>>>(n, per, pos, species, reinterpret_cast<const float2 *>(amp), n_pix, px->xyz,
                                   px->r0, reinterpret_cast<const double4 *>(px->q), A, part);
    MK_CHECK_CUDA(cudaGetLastError());
    return mk_launch_reduce(part, ns_eff, n_pix, nullptr, 1.0, reinterpret_cast<double2 *>(out),
                            accumulate, st);
}
