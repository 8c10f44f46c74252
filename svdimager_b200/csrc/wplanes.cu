// Imaging through w planes: the error-target rule's path for large w ranges.
//
// The reference (and this library's other rules) expands e^{2 pi i r3 t3} in Chebyshev polynomials per
// w-slab: every sample enters all K terms of its slab, and nslab K planes are transformed. Where only an
// error target is asked for, the third axis can be interpolated like the other two: with planes w_p = lo +
// (p - (W/2 - 1)) dw and an ES kernel psi of W planes,
//   e^{2 pi i r3 t3} = (1 / psi^(dw t3)) sum_p psi(v - p) e^{2 pi i w_p t3},  v = (r3 - lo) / dw + W/2 - 1,
// so a sample enters W planes only, and dw = 1 / (2 sigma max|t3|) gives sigma alpha / pi + W planes. The
// image is a real part, and Re(V e^{i phi}) = Re(V* e^{-i phi}): samples with r3 < 0 enter as their mirror
// image (-r, V*), which halves the w range. Wide field (4 slabs x 59 terms = 236 planes): 86 planes.
//
// Gridding: planes hold 0.1 samples per 8 x 8 tile and plane there, so samples are not binned; a warp
// stages the taps of 32 samples (lane per sample), then takes them one by one: lane (row, column pair) holds
// two adjacent cells and adds them to each of the W planes with one 16-byte reduction (64-byte row pieces).
// What bounds it: the L2's reductions, 512-640 bytes per sample and plane.
#include "binning_rules.cuh"
#include "svdi_internal.cuh"

namespace svdi {

namespace {

using namespace binrules;

constexpr int kWarps = 8;
constexpr int kMaxW = 12;  // planes per sample

__device__ __forceinline__ void red_add_v4(float2* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d)
                 : "memory");
}

__device__ __forceinline__ void red_add_v2(float2* addr, float a, float b) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(addr), "f"(a), "f"(b) : "memory");
}

__device__ __forceinline__ float es_exact(float beta, float x) {
    if (fabsf(x) > 1.0f) return 0.0f;
    return expf(-beta * x * x / (1.0f + sqrtf((1.0f - x) * (1.0f + x))));
}

// Taps 0 .. W - 1 at fraction f (u = 2 f - 1): mirrored pieces share the even and odd parts.
template <int W>
__device__ __forceinline__ void taps(const EsPoly& p, float u, float* w) {
    const float v = u * u;
#pragma unroll
    for (int i = 0; i < W / 2; ++i) {
        const float* c = p.c[i];
        const float ev = fmaf(fmaf(fmaf(fmaf(c[8], v, c[6]), v, c[4]), v, c[2]), v, c[0]);
        const float od = fmaf(fmaf(fmaf(c[7], v, c[5]), v, c[3]), v, c[1]);
        w[i] = fmaf(u, od, ev);
        w[W - 1 - i] = fmaf(-u, od, ev);
    }
}
static_assert(kPolyDeg == 8, "taps() is written for degree 8");

// One staged sample. wy starts at slot (first column & 1): slot pairs are 16-byte aligned cells.
struct __align__(16) Staged {
    float wz[kMaxW];
    float wy[12];
    float wx[8];
    float2 v;
    long long off;   // cell of the first row's first slot
    int p0;          // first plane; -1: nothing to add
    int pad;
};

template <int W, int WZ>
__global__ void __launch_bounds__(32 * kWarps) k_grid_w(SampleSource src, GridGeom g, WPlanes wp, EsPoly pxy,
                                                        EsPoly pz, int plane_lo, int plane_hi,
                                                        float2* __restrict__ planes,
                                                        unsigned long long* __restrict__ dropped) {
    constexpr int HW = W / 2, HZ = WZ / 2;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Staged* st = reinterpret_cast<Staged*>(smem) + warp * 32;
    const int C = (int)(src.n / src.R);
    const int G = (int)g.G;
    const long long GG = (long long)G * G;
    // units of 32 consecutive samples along the channels of consecutive rows
    const long long units = (src.n + 31) / 32;
    unsigned int ndrop = 0, nbad = 0;
    const int rr = lane >> 2, cp = lane & 3;
    for (long long u = (long long)blockIdx.x * kWarps + warp; u < units; u += (long long)gridDim.x * kWarps) {
        const long long k = u * 32 + lane;
        Staged& me = st[lane];
        bool rare = false;
        int first = -1;
        if (k < src.n) {
            const unsigned int row = (unsigned int)k / (unsigned int)C;
            const int c = (int)((unsigned int)k - row * (unsigned int)C);
            const long long idx = row + (long long)c * src.R;
            const double* q = src.q + (long long)row * 3;
            const double sc = src.s[c];
            const double r1 = __dmul_rn(sc, q[0]), r2 = __dmul_rn(sc, q[1]), r3 = __dmul_rn(sc, q[2]);
            float vre = __fmul_rn(src.vr[idx], src.inv_det), vim = __fmul_rn(src.vi[idx], src.inv_det);
            double p1 = grid_pos(r1, g), p2 = grid_pos(r2, g);
            int tile, qrel;
            // the binned gridders' inclusion rule, on the sample as it is
            if (!quantise_axis(p1, g, g.T, tile, qrel) || !quantise_axis(p2, g, g.T2, tile, qrel)) {
                ++ndrop;
            } else {
                nbad += (((__float_as_uint(vre) & 0x7f800000u) == 0x7f800000u) |
                         ((__float_as_uint(vim) & 0x7f800000u) == 0x7f800000u));
                if (r3 < 0.0) {
                    p1 = -p1;
                    p2 = -p2;
                    vim = -vim;
                }
                const long long q1 = __double2ll_rd(p1 * 16777216.0), q2 = __double2ll_rd(p2 * 16777216.0);
                const int c1 = (int)(q1 >> 24), c2 = (int)(q2 >> 24);
                const int f1 = (int)(q1 & 0xFFFFFF), f2 = (int)(q2 & 0xFFFFFF);
                const double w = __dmul_rn(fabs(r3) - wp.lo, wp.inv_dw);  // >= 0 up to rounding
                const long long q3 = __double2ll_rd(w * 16777216.0);
                const int p0 = max(0, min((int)(q3 >> 24), wp.P - WZ));   // its first plane
                const float f3 = fminf(1.0f, fmaxf(0.0f, (float)(w - (double)p0)));
                taps<WZ>(pz, fmaf(2.0f, f3, -1.0f), me.wz);
                const int a1 = c1 - (HW - 1) - (int)g.gmin, a2 = c2 - (HW - 1) - (int)g.gmin;  // plane row, column
                const int low = r3 < 0.0 ? 1 : 0;  // -G / 2 mirrors G / 2, which is not on the grid
                rare = f1 == 0 || f2 == 0 || a1 < low || a2 < low || a1 + W > G || a2 + W > G;
                // planes [p0, p0 + WZ) against this launch's range
                if (p0 < plane_hi && p0 + WZ > plane_lo) {
                    me.v = make_float2(vre, vim);
                    if (!rare) {
                        float t[W];
                        taps<W>(pxy, fmaf((float)f1, 1.0f / 8388608.0f, -1.0f), t);
                        // the checkerboard sign of the first row and slot; the rest alternates
#pragma unroll
                        for (int i = 0; i < 8; ++i) me.wx[i] = i < W ? ((a1 + i) & 1 ? -t[i < W ? i : 0] : t[i < W ? i : 0]) : 0.0f;
                        taps<W>(pxy, fmaf((float)f2, 1.0f / 8388608.0f, -1.0f), t);
                        const int odd = a2 & 1;
#pragma unroll
                        for (int i = 0; i < 12; ++i) me.wy[i] = 0.0f;
#pragma unroll
                        for (int i = 0; i < W; ++i) me.wy[odd + i] = (odd + i) & 1 ? -t[i] : t[i];
                        me.off = (long long)a1 * G + (a2 - odd);
                    } else {  // cells one by one below: positions instead of taps
                        me.wx[0] = __int_as_float(c1);
                        me.wx[1] = __int_as_float(f1);
                        me.wx[2] = __int_as_float(c2);
                        me.wx[3] = __int_as_float(f2);
                        me.wx[4] = __int_as_float(r3 < 0.0 ? -1 : 1);
                    }
                    first = p0;
                } else {
                    rare = false;
                }
            }
        }
        me.p0 = first;
        const unsigned int rare_mask = __ballot_sync(0xffffffffu, rare);
        __syncwarp();
        for (int j = 0; j < 32; ++j) {
            const Staged& s = st[j];
            const int p0 = s.p0;
            if (p0 < 0) continue;
            if (rare_mask & (1u << j)) {
                // exactly integer positions (W + 1 cells) and footprints at the grid edge: the cells the
                // reference rule keeps of the sample as it is, mirrored with it (column G / 2 is column
                // -G / 2 of the periodic transform)
                const int m = __float_as_int(s.wx[4]);
                const int c1 = __float_as_int(s.wx[0]), f1 = __float_as_int(s.wx[1]);
                const int c2 = __float_as_int(s.wx[2]), f2 = __float_as_int(s.wx[3]);
                const int lo1 = f1 ? c1 - (HW - 1) : c1 - HW, n1 = f1 ? W : W + 1;
                const int lo2 = f2 ? c2 - (HW - 1) : c2 - HW, n2 = f2 ? W : W + 1;
                const float x0 = (float)f1 * (1.0f / 16777216.0f), y0 = (float)f2 * (1.0f / 16777216.0f);
                const int gmin = (int)g.gmin, gmax = (int)g.gmax;
                for (int e = lane; e < n1 * n2; e += 32) {
                    int y = lo1 + e / n2, x = lo2 + e % n2;
                    const float kv = es_exact(wp.beta_xy, ((float)(y - c1) - x0) / (float)HW) *
                                     es_exact(wp.beta_xy, ((float)(x - c2) - y0) / (float)HW);
                    if (m * y < gmin || m * y > gmax || m * x < gmin || m * x > gmax) continue;
                    if (y > gmax) y -= G;
                    if (x > gmax) x -= G;
                    const float sg = ((y - gmin + x - gmin) & 1) ? -kv : kv;
                    for (int n = 0; n < WZ; ++n) {
                        if (p0 + n < plane_lo || p0 + n >= plane_hi) continue;
                        const float z = sg * s.wz[n];
                        red_add_v2(planes + (long long)(p0 + n - plane_lo) * GG + (long long)(y - gmin) * G + (x - gmin),
                                   z * s.v.x, z * s.v.y);
                    }
                }
                continue;
            }
            const float2 v = s.v;
            const float wx = s.wx[rr];
            const float2 wy = *reinterpret_cast<const float2*>(&s.wy[2 * cp]);
            const float k0 = wx * wy.x, k1 = wx * wy.y;
            const float a0 = k0 * v.x, b0 = k0 * v.y, a1 = k1 * v.x, b1 = k1 * v.y;
            float2* d0 = planes + (long long)(p0 - plane_lo) * GG + s.off;
            float2* d = d0 + (long long)rr * G + 2 * cp;
            // the fifth pair of an odd first column (its first cell only), one lane per row
            const float w8 = s.wy[8];
            const float k8 = lane < 8 ? s.wx[lane & 7] * w8 : 0.0f;
            const float a8 = k8 * v.x, b8 = k8 * v.y;
            float2* d8 = d0 + (long long)(lane & 7) * G + 8;
            const bool whole = p0 >= plane_lo && p0 + WZ <= plane_hi;
            const bool tail = k8 != 0.0f && lane < W, on = rr < W;
#pragma unroll
            for (int n = 0; n < WZ; ++n) {
                if (whole || (p0 + n >= plane_lo && p0 + n < plane_hi)) {
                    const float z = s.wz[n];
                    if (on) red_add_v4(d, z * a0, z * b0, z * a1, z * b1);
                    if (tail) red_add_v2(d8, z * a8, z * b8);
                }
                d += GG;
                d8 += GG;
            }
        }
        __syncwarp();
    }
    for (int o = 16; o > 0; o >>= 1) {
        ndrop += __shfl_xor_sync(0xffffffffu, ndrop, o);
        nbad += __shfl_xor_sync(0xffffffffu, nbad, o);
    }
    if (lane == 0 && dropped) {
        if (ndrop) atomicAdd(dropped, (unsigned long long)ndrop);
        if (nbad && src.nonfinite) atomicAdd(src.nonfinite, (unsigned long long)nbad);
    }
}

template <int W, int WZ>
int launch_one(const SampleSource& src, const GridGeom& g, const WPlanes& wp, const EsPoly& pxy, const EsPoly& pz,
               int plane_lo, int plane_hi, float2* d_planes, unsigned long long* d_dropped, cudaStream_t st) {
    auto kern = k_grid_w<W, WZ>;
    const size_t smem = sizeof(Staged) * 32 * kWarps;
    SVDI_TRY(ensure_dynamic_smem((const void*)kern, smem, true));
    const long long units = (src.n + 31) / 32;
    const long long blocks = std::max<long long>(1, std::min<long long>((units + kWarps - 1) / kWarps, 4LL * current_sm_count()));
    kern<<<(int)blocks, 32 * kWarps, smem, st>>>(src, g, wp, pxy, pz, plane_lo, plane_hi, d_planes, d_dropped);
    SVDI_LAUNCHED();
    return SVDI_OK;
}

}  // namespace

int launch_grid_w(const SampleSource& src, const GridGeom& g, const WPlanes& wp, const EsPoly& pxy, const EsPoly& pz,
                  int plane_lo, int plane_hi, float2* d_planes, unsigned long long* d_dropped, cudaStream_t st) {
    if (g.W == 8 && wp.W == 10) return launch_one<8, 10>(src, g, wp, pxy, pz, plane_lo, plane_hi, d_planes, d_dropped, st);
    if (g.W == 8 && wp.W == 12) return launch_one<8, 12>(src, g, wp, pxy, pz, plane_lo, plane_hi, d_planes, d_dropped, st);
    if (g.W == 6 && wp.W == 10) return launch_one<6, 10>(src, g, wp, pxy, pz, plane_lo, plane_hi, d_planes, d_dropped, st);
    if (g.W == 6 && wp.W == 12) return launch_one<6, 12>(src, g, wp, pxy, pz, plane_lo, plane_hi, d_planes, d_dropped, st);
    set_error("w planes: unsupported kernel widths");
    return SVDI_ERR_INTERNAL;
}

}  // namespace svdi
