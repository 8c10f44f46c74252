// Moment recombination, ES grid correction and reprojection with bilinear splat.
//
// One thread per rotated-frame pixel (SVDIntegratedImager.cu:1295-1463 fused_interpolation;
// archive/FIPkernels.cu:463-677 accumulation, scaling, coordschange, p2p, finalinterp):
//   t3 = -v33 + sgn(v33) sqrt(1 - (t1 + v13)^2 - (t2 + v23)^2)        (pixel skipped if < 0)
//   R  = | Re sum_slab sum_n J_n(alpha) c_n i^n e^{i beta_slab} M_{slab,n}(x, y) | * (-1)^(x+y)
//        / (Phi(|x|) Phi(|y|)) / N_s,  alpha = 2 pi t3 h, beta_slab = 2 pi t3 centre_slab
// then a SIN deprojection of the pixel to the output grid and a bilinear splat.
// Bessel coefficients and geometry in FP64 (the reference evaluates a FP32 power series,
// SVDIntegratedImager.cu:901-920, whose cancellation grows with alpha).
#include "svdi_internal.cuh"
#include "math.cuh"

namespace svdi {

namespace {

struct SplatTarget {
    double LL, MM;
    bool ok;
};

// Per-launch constants of the deprojection, computed once per block from Vin.
struct ReprojConst {
    double inv_v8;      // 1 / |V[8]|
    double dc_r0_sq;    // (cell in degrees / r0)^2, r0 = 180 / pi
    float xi_f, eta_f;  // V[6] / V[8], V[7] / V[8]
    float r0_dc;        // r0 / cell in degrees
};

__device__ inline ReprojConst reproj_const(const double* V, double dc_rad) {
    ReprojConst c;
    const double r0 = 180.0 / kPi, dc = dc_rad / kPi * 180.0;
    c.inv_v8 = 1.0 / fabs(V[8]);
    c.dc_r0_sq = (dc / r0) * (dc / r0);
    c.xi_f = (float)(V[6] / V[8]);
    c.eta_f = (float)(V[7] / V[8]);
    c.r0_dc = (float)(r0 / dc);
    return c;
}

// SVDIntegratedImager.cu:1325-1379 (simplified SIN deprojection; keeps p1, p2 when h > r0). With
// (x, y) the pixel's offset in degrees and h = |(x, y)|, the reference normalises (x, y) by h,
// scales it back by r = h and adds z r0 (xi, eta), z = 1 - sqrt(1 - (h / r0)^2): the target is
// (p1, p2) moved by z r0 (-xi, eta) / dc pixels. That is evaluated here directly: (p1, p2) in FP64,
// the displacement (at most some tens of pixels) in FP32 with z in the cancellation-free form
// s / (1 + sqrt(1 - s)), s = (h / r0)^2 -- no square root or division in FP64 per pixel.
__device__ inline SplatTarget reproject_sii(long long idx, long long idy, long long N, const ReprojConst& k,
                                            const double* V) {
    const double di2 = (double)N * 0.5;
    const long long half = N / 2;
    const double idxf = (double)idx - di2, idyf = (double)idy - di2;
    const double p1 = (-V[0] * idxf + V[3] * idyf) * k.inv_v8 + di2;
    const double p2 = (-V[1] * idxf + V[4] * idyf) * k.inv_v8 + di2;
    const double xo = p1 - (di2 + 1.0), yo = p2 - (di2 + 1.0);  // offset in pixels
    const double s = fma(xo, xo, yo * yo) * k.dc_r0_sq;          // (h / r0)^2
    double oi0 = p1, oi1 = p2;
    if (s <= 1.0) {  // h <= r0
        const float sf = (float)s;
        const float z = sf / (1.0f + sqrtf(1.0f - sf));
        const float m = z * k.r0_dc;
        oi0 = p1 - (double)(m * k.xi_f);
        oi1 = p2 + (double)(m * k.eta_f);
    }
    return {oi0 - (double)half, oi1 - (double)half, true};
}

// archive/FIPkernels.cu:552-624 (coordschange with the integer half size, then the
// trigonometric SIN p2p of Calabretta & Greisen that drops r^2 > 1)
__device__ inline SplatTarget reproject_fipk(long long idx, long long idy, long long N, double dc_rad,
                                             const double* V) {
    const long long half = N / 2;
    const double dc = dc_rad / kPi * 180.0;
    const double r0 = 180.0 / kPi;
    const double xi = V[6] / V[8], eta = V[7] / V[8];
    const double p1 = (-V[0] * (double)(idx - half) + V[3] * (double)(idy - half)) / fabs(V[8]) + (double)half;
    const double p2 = (-V[1] * (double)(idx - half) + V[4] * (double)(idy - half)) / fabs(V[8]) + (double)half;
    double x = -dc * (p1 - ((double)N / 2.0 + 1.0));
    double y = dc * (p2 - ((double)N / 2.0 + 1.0));
    const double x0 = x / r0, y0 = y / r0, r2 = x0 * x0 + y0 * y0;
    const double phi = (r2 != 0.0) ? atan2(x0, -y0) : 0.0;
    double theta;
    if (r2 < 0.5) theta = acos(sqrt(r2));
    else if (r2 <= 1.0) theta = asin(sqrt(1.0 - r2));
    else return {0.0, 0.0, false};
    double sx, cy;
    sincos(phi, &sx, &cy);
    const double t = kPi / 2.0 - fabs(theta);
    double z, costhe;
    if (t < 1.0e-5) {
        z = theta > 0.0 ? t * t / 2.0 : 2.0 - t * t / 2.0;
        costhe = t;
    } else {
        z = 1.0 - sin(theta);
        costhe = cos(theta);
    }
    const double r = r0 * costhe;
    const double w = xi * xi + eta * eta;
    if (w == 0.0) {
        x = r * sx;
        y = -r * cy;
    } else {
        z *= r0;
        x = r * sx + xi * z;
        y = -r * cy + eta * z;
    }
    const double oi0 = -1.0 / dc * x + (double)N / 2.0 + 1.0;
    const double oi1 = 1.0 / dc * y + (double)N / 2.0 + 1.0;
    return {oi0 - (double)half, oi1 - (double)half, true};
}

// A warp takes an 8 x 4 patch of pixels: the splat's targets are the patch turned by the snapshot's rotation,
// and its reductions cost the L2 one operation per 32-byte sector: about 14 sectors per warp instruction for
// a patch, up to 32 for a run of 32 pixels. (tx, ty): the thread's place in its block's 32 x 8 tile.
__device__ __forceinline__ void patch_pixel(int& tx, int& ty) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    tx = (warp & 3) * 8 + (lane & 7);
    ty = (warp >> 2) * 4 + (lane >> 3);
}

// floor of x, |x| < 2^31, as a double and an integer: one addition rounds x to the nearest integer, which
// the low word of the sum holds (the conversion unit, at a sixteenth of the FP64 rate, stays free).
__device__ __forceinline__ double floor_int(double x, int& i) {
    const double r = x + 6755399441055744.0;  // 1.5 * 2^52
    double f = r - 6755399441055744.0;
    i = __double2loint(r);
    if (f > x) {
        f -= 1.0;
        --i;
    }
    return f;
}

// Bilinear splat of one value at (LL, MM), pixels from the image centre (archive/FIPkernels.cu:627-677).
__device__ __forceinline__ void splat(float* __restrict__ out, int N, int half, double LL, double MM, double value) {
    if (!(fabs(LL) < (double)(half - 1) && fabs(MM) < (double)(half - 1))) return;
    int l, m;
    const double fl = LL - floor_int(LL, l), fm = MM - floor_int(MM, m);
    float* d = out + (long long)(m + half) * N + (l + half);
    // an exactly integer target adds its zero weights to its own cell
    const int dx = fl > 0.0 ? 1 : 0;
    const long long dy = fm > 0.0 ? N : 0;
    const double v0 = (1.0 - fl) * value, v1 = fl * value, gm = 1.0 - fm;
    atomicAdd(d, (float)(v0 * gm));
    atomicAdd(d + dy, (float)(v0 * fm));
    atomicAdd(d + dx, (float)(v1 * gm));
    atomicAdd(d + dy + dx, (float)(v1 * fm));
}

// From the sum over planes at pixel (x, y) to the image: checkerboard, grid correction, slab batches,
// |.| / N_s, reprojection and bilinear splat.
__device__ __forceinline__ void finish_pixel(long long x, long long y, double sum, long long N, double cell,
                                             const double* V, const float* __restrict__ corr, double inv_n,
                                             int reprojection, int presplat, float* __restrict__ out,
                                             double* __restrict__ acc, int final_batch, bool bad,
                                             const ReprojConst& kc) {
    const long long half = N / 2;
    const long long xr = x - half, yr = y - half;
    if ((xr + yr) & 1) sum = -sum;
    const long long ax = xr < 0 ? -xr : xr, ay = yr < 0 ? -yr : yr;
    double signed_sum = sum * (double)corr[ax] * (double)corr[ay];
    if (acc) {  // slab batches: the signed sums add up, |.| is taken once, in the last batch
        signed_sum += acc[y * N + x];
        if (!final_batch) {
            acc[y * N + x] = signed_sum;
            return;
        }
    }
    double value = fabs(signed_sum) * inv_n;
    // a NaN or Inf among the gridded values: every moment cell would be NaN after the FFT, so every
    // valid pixel is NaN (the reference's float atomics, SVDIntegratedImager.cu:1276-1290, carry it)
    if (bad) value = __longlong_as_double(0x7ff8000000000000LL);
    if (presplat) {
        out[y * N + x] = (float)value;
        return;
    }

    const SplatTarget tg = reprojection == SVDI_REPROJ_FIPK ? reproject_fipk(x, y, N, cell, V)
                                                            : reproject_sii(x, y, N, kc, V);
    if (!tg.ok) return;
    splat(out, (int)N, (int)half, tg.LL, tg.MM, value);
}

// One pixel (x, y) of the rotated frame: moments -> |Re sum| -> grid correction -> reprojection.
template <int KMAX>
__device__ __forceinline__ void recombine_pixel(long long x, long long y, const float2* __restrict__ moments,
                                                const GridGeom& g, long long N, double cell,
                                                const double* __restrict__ vin, const SlabParams& sp,
                                                const float* __restrict__ corr, double inv_n, int reprojection,
                                                int presplat, float* __restrict__ out, double* __restrict__ acc,
                                                int final_batch, bool bad, const ReprojConst& kc) {
    double V[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) V[k] = vin[k];
    const long long half = N / 2;
    const long long xr = x - half, yr = y - half;
    const double t1 = cell * (double)yr, t2 = cell * (double)xr;
    const double ra = 1.0 - (t1 + V[2]) * (t1 + V[2]) - (t2 + V[5]) * (t2 + V[5]);
    if (ra < 0.0) {
        if (presplat && final_batch) out[y * N + x] = __int_as_float(0x7fc00000);  // NaN
        return;
    }
    const double t3 = -V[8] + (V[8] >= 0.0 ? 1.0 : -1.0) * sqrt(ra);

    const int K = sp.K;
    double jv[KMAX];
    bessel_jn_fast(2.0 * kPi * t3 * sp.slab_half, K - 1, jv);
    const long long G = g.G, GG = G * G;
    const long long gidx = GG / 2 + G / 2 + yr * G + xr;  // SVDIntegratedImager.cu:1397
    double sum = 0.0;
    for (int j = 0; j < sp.nslab; ++j) {
        const double centre = sp.r3_min + ((double)j + 0.5) * sp.slab_width;
        const double ph = 2.0 * t3 * centre;     // e^{i pi ph}
        double sb, cb;
        if (fabs(ph) < 0x1p-8) {  // small phase: FP32 is exact to ~1e-7 of ph, far below 1e-9 rad
            float sf, cf;
            sincospif((float)ph, &sf, &cf);
            sb = (double)sf;
            cb = (double)cf;
        } else {
            sincospi(ph, &sb, &cb);
        }
        // the terms n = 4 i + q into four independent FP64 sums (the chain of dependent adds, not
        // the loads, set the pace: wide-field recombination 27.7 -> 22.7 ms)
        const float2* mp = moments + (long long)j * K * GG + gidx;
        double s4[4] = {0.0, 0.0, 0.0, 0.0};
        int n = 0;
        for (; n + 4 <= K; n += 4) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 m = mp[(long long)(n + q) * GG];
                const double amp = (n + q == 0) ? jv[0] : 2.0 * jv[n + q];
                double cr, ci;  // amp * i^(n + q) * e^{i beta}, n a multiple of 4
                switch (q) {
                    case 0: cr = amp * cb; ci = amp * sb; break;
                    case 1: cr = -amp * sb; ci = amp * cb; break;
                    case 2: cr = -amp * cb; ci = -amp * sb; break;
                    default: cr = amp * sb; ci = -amp * cb; break;
                }
                s4[q] += cr * (double)m.x - ci * (double)m.y;
            }
        }
        for (; n < K; ++n) {
            const float2 m = mp[(long long)n * GG];
            const double amp = (n == 0) ? jv[0] : 2.0 * jv[n];
            double cr, ci;  // amp * i^n * e^{i beta}
            switch (n & 3) {
                case 0: cr = amp * cb; ci = amp * sb; break;
                case 1: cr = -amp * sb; ci = amp * cb; break;
                case 2: cr = -amp * cb; ci = -amp * sb; break;
                default: cr = amp * sb; ci = -amp * cb; break;
            }
            s4[0] += cr * (double)m.x - ci * (double)m.y;
        }
        sum += (s4[0] + s4[1]) + (s4[2] + s4[3]);
    }
    finish_pixel(x, y, sum, N, cell, V, corr, inv_n, reprojection, presplat, out, acc, final_batch, bad, kc);
}

// Persistent over 32 x 8 pixel tiles: the per-launch constants (slab geometry, reprojection
// constants, the non-finite flag) are set up once per block.
template <int KMAX>
__global__ void __launch_bounds__(256, 4) k_recombine(const float2* __restrict__ moments, GridGeom g, long long N,
                                                  double cell, const double* __restrict__ vin,
                                                  SlabParams sp, const float* __restrict__ corr,
                                                  double inv_n, int reprojection, int presplat,
                                                  float* __restrict__ out, double* __restrict__ acc,
                                                  int final_batch, const DevPlan* __restrict__ plan,
                                                  const unsigned long long* __restrict__ nonfinite) {
    if (plan && first_thread()) plan_stamps(plan)[STAMP_IMAGE] = stamp_now();
    if (plan) {  // one batch of all slabs: the device plan's slab geometry
        sp.r3_min = plan->sp.r3_min;
        sp.slab_width = plan->sp.slab_width;
        sp.slab_half = plan->sp.slab_half;
        sp.inv_half = plan->sp.inv_half;
    }
    __shared__ ReprojConst kc;
    if (threadIdx.x == 0) kc = reproj_const(vin, cell);
    __syncthreads();
    const bool bad = nonfinite && *nonfinite;
    const long long ntx = (N + 31) / 32, nty = (N + 7) / 8;
    int px, py;
    patch_pixel(px, py);
    for (long long t = blockIdx.x; t < ntx * nty; t += gridDim.x) {
        const long long ty = t / ntx, tx = t - ty * ntx;
        const long long x = tx * 32 + px, y = ty * 8 + py;
        if (x < N && y < N)
            recombine_pixel<KMAX>(x, y, moments, g, N, cell, vin, sp, corr, inv_n, reprojection, presplat, out, acc,
                                  final_batch, bad, kc);
    }
    if (plan && threadIdx.x == 0) atomicMax(plan_stamps(plan) + STAMP_END, stamp_now());
}

// J_0 .. J_{KT-1}: bessel_jn_fast with the ascending series (|x| < 1e-3) unrolled in registers.
template <int KT>
__device__ __forceinline__ void bessel_few(double x, double (&j)[KT]) {
    if (fabs(x) < 1e-3) {
        const double h = 0.5 * x, q = -h * h;
        double lead = 1.0;  // (x/2)^n / n!
#pragma unroll
        for (int n = 0; n < KT; ++n) {
            if (n > 0) lead *= h * (1.0 / n);
            const double t1 = q * (1.0 / (n + 1));
            j[n] = fma(lead * t1, fma(q, 0.5 / (n + 2), 1.0), lead);
        }
        return;
    }
    double t[KT];
    bessel_jn_fast(x, KT - 1, t);
#pragma unroll
    for (int n = 0; n < KT; ++n) j[n] = t[n];
}

// Few Chebyshev terms, K = KT (the coplanar snapshots' orders 1 .. 4 and the bucket rule's 8): everything
// unrolled, what depends on the launch computed once: 330 warp instructions per 32 pixels at two terms, where
// the general kernel above takes 550 (term loops over a local array, 64-bit indices, conversions). With the
// patches, two terms: 1024^2 35 -> 24 us, 2048^2 115 -> 74 us (12 us of it the splat's reductions, 55 us before
// the patches). Four pixels of a row per thread, to share the row's part, was slower (80 us: fewer warps wait for
// more loads each).
template <int KT>
__global__ void __launch_bounds__(256, 3) k_recombine_few(const float2* __restrict__ moments, GridGeom g, int N,
                                                      double cell, const double* __restrict__ vin, SlabParams sp,
                                                      const float* __restrict__ corr, double inv_n, int reprojection,
                                                      int presplat, float* __restrict__ out, double* __restrict__ acc,
                                                      int final_batch, const DevPlan* __restrict__ plan,
                                                      const unsigned long long* __restrict__ nonfinite) {
    if (plan && first_thread()) plan_stamps(plan)[STAMP_IMAGE] = stamp_now();
    if (plan) {  // one batch of all slabs: the device plan's slab geometry
        sp.r3_min = plan->sp.r3_min;
        sp.slab_width = plan->sp.slab_width;
        sp.slab_half = plan->sp.slab_half;
    }
    __shared__ ReprojConst kc_s;
    if (threadIdx.x == 0) kc_s = reproj_const(vin, cell);
    __syncthreads();
    const ReprojConst kc = kc_s;
    const bool bad = nonfinite && *nonfinite;
    const int half = N / 2, G = (int)g.G;
    const long long GG = (long long)G * G;
    const double di2 = (double)N * 0.5;
    const double v13 = vin[2], v23 = vin[5], v33 = vin[8], sgn = v33 >= 0.0 ? 1.0 : -1.0;
    const double a0 = -vin[0] * kc.inv_v8, a3 = vin[3] * kc.inv_v8, b1 = -vin[1] * kc.inv_v8, b4 = vin[4] * kc.inv_v8;
    const double c_alpha = 2.0 * kPi * sp.slab_half;
    const int ntx = (N + 31) / 32, nty = (N + 7) / 8;
    int px, py;
    patch_pixel(px, py);
    for (int t = blockIdx.x; t < ntx * nty; t += gridDim.x) {
        const int ty = t / ntx, tx = t - ty * ntx;
        const int y = ty * 8 + py, yr = y - half;
        if (y >= N) continue;
        const double t1 = fma(cell, (double)yr, v13), r1 = 1.0 - t1 * t1;
        const double idyf = (double)y - di2;
        const double p1y = fma(a3, idyf, di2), p2y = fma(b4, idyf, di2);
        const double cy = (double)corr[yr < 0 ? -yr : yr];
        const float2* mrow = moments + (GG / 2 + G / 2 + (long long)yr * G) - half;
        const int x = tx * 32 + px, xr = x - half;
        if (x >= N) continue;
        const double xd = (double)xr;
        const double t2 = fma(cell, xd, v23), ra = r1 - t2 * t2;
        if (ra < 0.0) {
            if (presplat && final_batch) out[(long long)y * N + x] = __int_as_float(0x7fc00000);  // NaN
            continue;
        }
        const double t3 = fma(sgn, sqrt(ra), -v33);
        double jv[KT];
        bessel_few<KT>(t3 * c_alpha, jv);
        double sum = 0.0;
        for (int s = 0; s < sp.nslab; ++s) {
            const float2* mp = mrow + (long long)s * KT * GG + x;
            float2 m[KT];
#pragma unroll
            for (int n = 0; n < KT; ++n) m[n] = mp[n * GG];
            const double ph = 2.0 * t3 * (sp.r3_min + ((double)s + 0.5) * sp.slab_width);  // e^{i pi ph}
            double sb, cb;
            if (fabs(ph) < 0x1p-8) {  // the next terms of the series are below 1e-17
                const double z = kPi * ph, z2 = z * z;
                cb = fma(z2, fma(z2, fma(z2, -1.0 / 720.0, 1.0 / 24.0), -0.5), 1.0);
                sb = z * fma(z2, fma(z2, fma(z2, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), 1.0);
            } else {
                sincospi(ph, &sb, &cb);
            }
            double part = 0.0;
#pragma unroll
            for (int n = 0; n < KT; ++n) {
                const double amp = n == 0 ? jv[0] : 2.0 * jv[n];
                const double mx = (double)m[n].x, my = (double)m[n].y;
                double v;  // Re(i^n e^{i beta} M_n)
                switch (n & 3) {
                    case 0: v = cb * mx - sb * my; break;
                    case 1: v = -sb * mx - cb * my; break;
                    case 2: v = sb * my - cb * mx; break;
                    default: v = sb * mx + cb * my; break;
                }
                part = fma(amp, v, part);
            }
            sum += part;
        }
        if ((xr + yr) & 1) sum = -sum;
        double signed_sum = sum * (double)corr[xr < 0 ? -xr : xr] * cy;
        if (acc) {  // slab batches: the signed sums add up, |.| is taken once, in the last batch
            double* a = acc + (long long)y * N + x;
            signed_sum += *a;
            if (!final_batch) {
                *a = signed_sum;
                continue;
            }
        }
        double value = fabs(signed_sum) * inv_n;
        if (bad) value = __longlong_as_double(0x7ff8000000000000LL);  // as in finish_pixel
        if (presplat) {
            out[(long long)y * N + x] = (float)value;
            continue;
        }
        double LL, MM;
        if (reprojection == SVDI_REPROJ_FIPK) {
            const SplatTarget tg = reproject_fipk(x, y, N, cell, vin);
            if (!tg.ok) continue;
            LL = tg.LL;
            MM = tg.MM;
        } else {  // reproject_sii with the row's part of the rotation at hand
            const double idxf = (double)x - di2;
            const double p1 = fma(a0, idxf, p1y), p2 = fma(b1, idxf, p2y);
            const double xo = p1 - (di2 + 1.0), yo = p2 - (di2 + 1.0);
            const double s = fma(xo, xo, yo * yo) * kc.dc_r0_sq;
            LL = p1;
            MM = p2;
            if (s <= 1.0) {
                const float sf = (float)s;
                const float mv = sf / (1.0f + sqrtf(1.0f - sf)) * kc.r0_dc;
                LL -= (double)(mv * kc.xi_f);
                MM += (double)(mv * kc.eta_f);
            }
            LL -= (double)half;
            MM -= (double)half;
        }
        splat(out, N, half, LL, MM, value);
    }
    if (plan && threadIdx.x == 0) atomicMax(plan_stamps(plan) + STAMP_END, stamp_now());
}

template <int KT>
void launch_few(const float2* d_moments, const GridGeom& g, int N, double cell, const double* d_vin64,
                const SlabParams& sp, const float* d_corr, double inv_n, int reprojection, int presplat, float* d_out,
                cudaStream_t st, double* d_acc, int final_batch, const DevPlan* d_plan,
                const unsigned long long* d_nonfinite) {
    const long long tiles = ((N + 31LL) / 32) * ((N + 7) / 8);
    k_recombine_few<KT><<<(unsigned)std::min<long long>(tiles, 6LL * current_sm_count()), 256, 0, st>>>(
        d_moments, g, N, cell, d_vin64, sp, d_corr, inv_n, reprojection, presplat, d_out, d_acc, final_batch, d_plan,
        d_nonfinite);
}

// One pixel from w planes: Re sum_p e^{2 pi i w_p t3} M_p / psi^(dw t3). The phases advance by one
// rotation per plane in FP64 (two chains of every other plane).
__global__ void __launch_bounds__(256, 4) k_recombine_w(const float2* __restrict__ planes, GridGeom g, long long N,
                                                    double cell, const double* __restrict__ vin, WPlanes wp,
                                                    int plane_lo, int plane_hi, const float* __restrict__ corr,
                                                    double inv_n, int reprojection, int presplat,
                                                    float* __restrict__ out, double* __restrict__ acc,
                                                    int final_batch, const unsigned long long* __restrict__ nonfinite) {
    __shared__ ReprojConst kc;
    if (threadIdx.x == 0) kc = reproj_const(vin, cell);
    __syncthreads();
    const bool bad = nonfinite && *nonfinite;
    double V[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) V[k] = vin[k];
    const long long half = N / 2, G = g.G, GG = G * G;
    const long long ntx = (N + 31) / 32, nty = (N + 7) / 8;
    int px, py;
    patch_pixel(px, py);
    for (long long t = blockIdx.x; t < ntx * nty; t += gridDim.x) {
        const long long ty = t / ntx, tx = t - ty * ntx;
        const long long x = tx * 32 + px, y = ty * 8 + py;
        if (x >= N || y >= N) continue;
        const long long xr = x - half, yr = y - half;
        const double t1 = cell * (double)yr, t2 = cell * (double)xr;
        const double ra = 1.0 - (t1 + V[2]) * (t1 + V[2]) - (t2 + V[5]) * (t2 + V[5]);
        if (ra < 0.0) {
            if (presplat && final_batch) out[y * N + x] = __int_as_float(0x7fc00000);  // NaN
            continue;
        }
        const double t3 = -V[8] + (V[8] >= 0.0 ? 1.0 : -1.0) * sqrt(ra);
        const double w0 = wp.lo + (double)(plane_lo - (wp.W / 2 - 1)) * wp.dw;
        double si, co, dsi, dco;
        sincospi(2.0 * t3 * w0, &si, &co);
        sincospi(2.0 * t3 * wp.dw, &dsi, &dco);
        const float2* mp = planes + GG / 2 + G / 2 + yr * G + xr;
        double sum0 = 0.0, sum1 = 0.0;
        int n = plane_hi - plane_lo;
#pragma unroll 4
        for (; n >= 2; n -= 2) {
            const float2 m0 = mp[0], m1 = mp[GG];
            mp += 2 * GG;
            sum0 += co * (double)m0.x - si * (double)m0.y;
            double c1 = co * dco - si * dsi, s1 = si * dco + co * dsi;
            sum1 += c1 * (double)m1.x - s1 * (double)m1.y;
            co = c1 * dco - s1 * dsi;
            si = s1 * dco + c1 * dsi;
        }
        if (n) sum0 += co * (double)mp[0].x - si * (double)mp[0].y;
        // 1 / psi^ by Clenshaw's recurrence in 2 (t3 / max|t3|)^2 - 1
        const double kk = t3 * wp.dw / wp.kmax, z = 2.0 * kk * kk - 1.0;
        double b1 = 0.0, b2 = 0.0;
#pragma unroll
        for (int i = kWCorrTerms - 1; i > 0; --i) {
            const double b = fma(2.0 * z, b1, wp.corr[i] - b2);
            b2 = b1;
            b1 = b;
        }
        finish_pixel(x, y, (sum0 + sum1) * fma(z, b1, wp.corr[0] - b2), N, cell, V, corr, inv_n, reprojection,
                     presplat, out, acc, final_batch, bad, kc);
    }
}

}  // namespace

int launch_recombine(const float2* d_moments, const GridGeom& g, long long N, double cell,
                     const double* d_vin64, const SlabParams& sp, const float* d_corr,
                     double inv_n_total, int reprojection, int presplat, float* d_out,
                     cudaStream_t st, double* d_acc, bool final_batch, const DevPlan* d_plan,
                     const unsigned long long* d_nonfinite) {
    const dim3 block(256);
    const long long tiles = ((N + 31) / 32) * ((N + 7) / 8);
    const dim3 grid((unsigned)std::min<long long>(tiles, 8LL * current_sm_count()));
#define SVDI_FEW(KT)                                                                                          \
    launch_few<KT>(d_moments, g, (int)N, cell, d_vin64, sp, d_corr, inv_n_total, reprojection, presplat, d_out, st, \
                   d_acc, final_batch ? 1 : 0, d_plan, d_nonfinite)
    if (sp.K == 1) SVDI_FEW(1);
    else if (sp.K == 2) SVDI_FEW(2);
    else if (sp.K == 3) SVDI_FEW(3);
    else if (sp.K == 4) SVDI_FEW(4);
    else if (sp.K == 8) SVDI_FEW(8);
#undef SVDI_FEW
    else if (sp.K < 8) k_recombine<8><<<grid, block, 0, st>>>(d_moments, g, N, cell, d_vin64, sp, d_corr, inv_n_total, reprojection, presplat, d_out, d_acc, final_batch ? 1 : 0, d_plan, d_nonfinite);
    else if (sp.K <= 16) k_recombine<16><<<grid, block, 0, st>>>(d_moments, g, N, cell, d_vin64, sp, d_corr, inv_n_total, reprojection, presplat, d_out, d_acc, final_batch ? 1 : 0, d_plan, d_nonfinite);
    else if (sp.K <= 32) k_recombine<32><<<grid, block, 0, st>>>(d_moments, g, N, cell, d_vin64, sp, d_corr, inv_n_total, reprojection, presplat, d_out, d_acc, final_batch ? 1 : 0, d_plan, d_nonfinite);
    else if (sp.K <= kMaxTerms) k_recombine<kMaxTerms><<<grid, block, 0, st>>>(d_moments, g, N, cell, d_vin64, sp, d_corr, inv_n_total, reprojection, presplat, d_out, d_acc, final_batch ? 1 : 0, d_plan, d_nonfinite);
    else {
        set_error("recombine: too many Chebyshev terms");
        return SVDI_ERR_UNSUPPORTED;
    }
    SVDI_LAUNCHED();
    return SVDI_OK;
}

int launch_recombine_w(const float2* d_planes, const GridGeom& g, long long N, double cell, const double* d_vin64,
                       const WPlanes& wp, int plane_lo, int plane_hi, const float* d_corr, double inv_n_total,
                       int reprojection, int presplat, float* d_out, cudaStream_t st, double* d_acc, bool final_batch,
                       const unsigned long long* d_nonfinite) {
    const dim3 block(256);
    const long long tiles = ((N + 31) / 32) * ((N + 7) / 8);
    const dim3 grid((unsigned)std::min<long long>(tiles, 8LL * current_sm_count()));
    k_recombine_w<<<grid, block, 0, st>>>(d_planes, g, N, cell, d_vin64, wp, plane_lo, plane_hi, d_corr, inv_n_total,
                                          reprojection, presplat, d_out, d_acc, final_batch ? 1 : 0, d_nonfinite);
    SVDI_LAUNCHED();
    return SVDI_OK;
}

}  // namespace svdi
