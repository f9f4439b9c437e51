// Energy-equation kernels of one SIMPLE outer iteration, plus the per-step
// laser and push-back kernels.  Each kernel names the reference routine it
// replaces; arithmetic follows the reference expression by expression so that
// the FP64 build matches the CPU solve to rounding.
#include "kernels.cuh"

namespace amcfd {

// ---------------------------------------------------------------------------
// updateLaser heat flux (BoundCondManager.cpp:128-159): Gaussian surface flux
// heatin[j][i] and the partial sums of areaij*heatin (heatinlaser).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void laser_kernel(Params p, Fields<T> g, double *red)
{
    pdl_enter();
    const Status *st = g.st;
    double acc = 0.0;
    const double rb2 = p.alasrb * p.alasrb;
    const double varlas = p.alaspow * p.alaseta;
    const double peakhin = p.alasfact * varlas / (M_PI * rb2);
    const double pw = (double)st->powerindicator;
    const int n = p.ni * p.nj;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        int j = q / p.ni, i = q - j * p.ni;
        double ydist = st->beamposy - g.y[j];
        double xdist = st->beamposx - g.x[i];
        double dist2 = (xdist * xdist) + (ydist * ydist);
        double hin = peakhin * exp(-p.alasfact * dist2 / rb2) * pw;
        if (p.alasfact < 1.0e-6 && dist2 < rb2) hin = varlas / (M_PI * rb2) * pw;
        g.heatin[(size_t)j * p.nip + i] = hin;
        acc += area_ij(p, g, i, j) * hin;
    }
    double v[1] = {acc};
    const int s[1] = {R_HEATIN};
    const bool m[1] = {false};
    block_reduce_store<1>(v, s, m, red, blockIdx.x);
}

// ---------------------------------------------------------------------------
// applyBCs(5) (BoundCondManager.cpp:565-654): top-surface flux balance and
// convective side planes.  Also advances the volumetric heat-source table the
// way calculateSource(5) does at the start of each outer iteration
// (CFDSolverManager.cpp:1707-1717).
// ---------------------------------------------------------------------------
template <typename T>
__global__ void energy_bc_kernel(Params p, Fields<T> g, double *red)
{
    pdl_enter();
    Status *st = g.st;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (p.nheattable > 0) {
            int it = st->heat_iter;
            if (st->timet > g.heattable[6 * it] && it < p.nheattable - 1) it += 1;
            st->heat_iter = it;
            const double *row = &g.heattable[6 * it];
            st->avolpow = row[1];
            st->apowseta = row[2];
            st->heatthick = row[3];
            st->heatrb = row[4];
            st->avolfact = row[5];
        }
    }
    const int ni = p.ni, nj = p.nj, nip = p.nip;
    const int nim1 = p.nim1, njm1 = p.njm1, nkm1 = p.nkm1, nim2 = p.nim2, njm2 = p.njm2,
              nkm2 = p.nkm2;
    const int ntop = (nim1 - 1) * (njm1 - 1);
    const int new_ = (nkm1 - 1) * (njm1 - 1);
    const int nns = (nkm1 - 1) * (nim1 - 1);
    double ahtop = 0.0;
    double a4 = p.tempamb;
    for (int q = 1; q < 4; q++) a4 *= p.tempamb;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < ntop + new_ + nns;
         q += gridDim.x * blockDim.x) {
        if (q < ntop) {
            int j = 1 + q / (nim1 - 1), i = 1 + q % (nim1 - 1);
            double t = (double)g.temp[cidx(i, j, nkm1, nj, nip)];
            double hlossevap = 0.0;
            if (p.isevap) {
                double psat = p.pressamb * exp(-p.evaplatent * p.molarmass / p.gasconst *
                                               (1.0 / t - 1.0 / p.evaptemp));
                double mdot = p.evapfact * psat * sqrt(p.molarmass / (2.0 * M_PI * p.gasconst * t));
                hlossevap = mdot * p.evaplatent;
            }
            double t4 = t;
            for (int r = 1; r < 4; r++) t4 *= t;
            double hlossradia = p.emiss * p.sigm * (t4 - a4);
            double ctmp1 = (double)g.diff_cur[cidx(i, j, nkm2, nj, nip)] * g.dzpbinv[nkm1];
            double hb = (double)g.h[cidx(i, j, nkm2, nj, nip)];
            g.h[cidx(i, j, nkm1, nj, nip)] =
                (T)(hb + (g.heatin[(size_t)j * nip + i] - hlossradia - hlossradia - hlossevap) / ctmp1);
            ahtop += (hlossradia + hlossradia + hlossevap) * area_ij(p, g, i, j);
        } else if (q < ntop + new_) {
            int r = q - ntop;
            int k = 1 + r / (njm1 - 1), j = 1 + r % (njm1 - 1);
            double hc = p.htci * ((double)g.temp[cidx(0, j, k, nj, nip)] - p.tempamb);
            double ctmp1 = (double)g.diff_cur[cidx(1, j, k, nj, nip)] * g.dxpwinv[1];
            g.h[cidx(0, j, k, nj, nip)] = (T)((double)g.h[cidx(1, j, k, nj, nip)] - hc / ctmp1);
            hc = p.htci * ((double)g.temp[cidx(nim1, j, k, nj, nip)] - p.tempamb);
            ctmp1 = (double)g.diff_cur[cidx(nim2, j, k, nj, nip)] * g.dxpwinv[nim2];
            g.h[cidx(nim1, j, k, nj, nip)] = (T)((double)g.h[cidx(nim2, j, k, nj, nip)] - hc / ctmp1);
        } else {
            int r = q - ntop - new_;
            int k = 1 + r / (nim1 - 1), i = 1 + r % (nim1 - 1);
            double hc = p.htcj * ((double)g.temp[cidx(i, 0, k, nj, nip)] - p.tempamb);
            double ctmp1 = (double)g.diff_cur[cidx(i, 1, k, nj, nip)] * g.dypsinv[1];
            g.h[cidx(i, 0, k, nj, nip)] = (T)((double)g.h[cidx(i, 1, k, nj, nip)] - hc / ctmp1);
            hc = p.htcj * ((double)g.temp[cidx(i, njm1, k, nj, nip)] - p.tempamb);
            ctmp1 = (double)g.diff_cur[cidx(i, njm2, k, nj, nip)] * g.dypsinv[njm2];
            g.h[cidx(i, njm1, k, nj, nip)] = (T)((double)g.h[cidx(i, njm2, k, nj, nip)] - hc / ctmp1);
        }
    }
    (void)ni;
    double v[1] = {ahtop};
    const int s[1] = {R_AHTOP};
    const bool m[1] = {false};
    block_reduce_store<1>(v, s, m, red, blockIdx.x);
}

// 1-D TDMA of the block correction (enhanceConvergenceSpeed(5),
// CFDSolverManager.cpp:2334-2349) for cells i0..i1 by one warp:
//   den_i = bl_i - blm_i pib_{i-1},  pib_i = blp_i / den_i,
//   qib_i = (blc_i + blm_i qib_{i-1}) / den_i,  delphi_i = pib_i delphi_{i+1} + qib_i,
// with pib_{i0-1} = qib_{i0-1} = 0 and delphi_{i1+1} = 0.  Each lane owns a
// contiguous chunk.  pib follows x -> blp / (bl - blm x), a Moebius map: the
// chunks' 2x2 matrices (rescaled as they are multiplied; the map ignores
// scale) are combined by a warp scan to give each chunk its entry value, and
// the chunk then runs the reference recurrence.  qib and delphi are affine in
// their predecessor and use warp scans of affine maps.  All in FP64.  On
// return bl holds den, blm holds pib and blp holds qib.
__device__ __forceinline__ double moebius_scale(double a, double b, double c, double d)
{
    const double mx = fmax(fmax(fabs(a), fabs(b)), fmax(fabs(c), fabs(d)));
    return mx > 0.0 ? 1.0 / mx : 1.0;
}

__device__ void block_tdma_warp(double *bl, double *blp, double *blm, const double *blc, int i0, int i1,
                                double *delphi)
{
    const int lane = threadIdx.x & 31;
    const int n = i1 - i0 + 1;
    if (n <= 0) return;
    const int L = (n + 31) >> 5;
    const int a = i0 + min(lane * L, n), e = i0 + min(lane * L + L, n);
    // chunk product of the Moebius matrices [[0, blp], [-blm, bl]] (later cells on the left)
    double m00 = 1.0, m01 = 0.0, m10 = 0.0, m11 = 1.0;
    for (int i = a; i < e; ++i) {
        const double n00 = blp[i] * m10, n01 = blp[i] * m11;
        const double n10 = -blm[i] * m00 + bl[i] * m10, n11 = -blm[i] * m01 + bl[i] * m11;
        const double sc = moebius_scale(n00, n01, n10, n11);
        m00 = n00 * sc; m01 = n01 * sc; m10 = n10 * sc; m11 = n11 * sc;
    }
    // inclusive scan: M_lane <- M_lane * M_{lane-o}
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double p00 = __shfl_up_sync(0xffffffffu, m00, o), p01 = __shfl_up_sync(0xffffffffu, m01, o);
        const double p10 = __shfl_up_sync(0xffffffffu, m10, o), p11 = __shfl_up_sync(0xffffffffu, m11, o);
        if (lane >= o) {
            const double n00 = m00 * p00 + m01 * p10, n01 = m00 * p01 + m01 * p11;
            const double n10 = m10 * p00 + m11 * p10, n11 = m10 * p01 + m11 * p11;
            const double sc = moebius_scale(n00, n01, n10, n11);
            m00 = n00 * sc; m01 = n01 * sc; m10 = n10 * sc; m11 = n11 * sc;
        }
    }
    // entry value pib_{a-1}: the exclusive prefix applied to x = 0
    double e01 = __shfl_up_sync(0xffffffffu, m01, 1), e11 = __shfl_up_sync(0xffffffffu, m11, 1);
    double pib = (lane == 0) ? 0.0 : e01 / e11;
    // the chunk runs the reference recurrence for den and pib; qib's affine maps
    double A = 1.0, B = 0.0;
    for (int i = a; i < e; ++i) {
        const double den = bl[i] - blm[i] * pib;
        const double pv = blp[i] / den;
        const double ca = blm[i] / den, cb = blc[i] / den;  // qib_i = ca qib_{i-1} + cb
        bl[i] = den;
        blm[i] = pv;
        blp[i] = cb;  // temporarily the affine offset
        pib = pv;
        B = ca * B + cb;
        A = ca * A;
        delphi[i] = ca;  // temporarily the affine slope
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double A2 = __shfl_up_sync(0xffffffffu, A, o), B2 = __shfl_up_sync(0xffffffffu, B, o);
        if (lane >= o) { B = A * B2 + B; A = A * A2; }
    }
    double Be = __shfl_up_sync(0xffffffffu, B, 1);
    double q = (lane == 0) ? 0.0 : Be;  // qib_{a-1} (qib_{i0-1} = 0)
    for (int i = a; i < e; ++i) {
        q = delphi[i] * q + blp[i];
        blp[i] = q;
    }
    // back substitution delphi_i = pib_i delphi_{i+1} + qib_i, delphi_{i1+1} = 0
    A = 1.0;
    B = 0.0;
    for (int i = e - 1; i >= a; --i) {
        B = blm[i] * B + blp[i];
        A = blm[i] * A;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double A2 = __shfl_down_sync(0xffffffffu, A, o), B2 = __shfl_down_sync(0xffffffffu, B, o);
        if (lane + o < 32) { B = A * B2 + B; A = A * A2; }
    }
    Be = __shfl_down_sync(0xffffffffu, B, 1);
    double d = (lane == 31) ? 0.0 : Be;
    for (int i = e - 1; i >= a; --i) {
        d = blm[i] * d + blp[i];
        delphi[i] = d;
    }
}

// ---------------------------------------------------------------------------
// Block correction solve (enhanceConvergenceSpeed(5), CFDSolverManager.cpp:2334-2349)
// and the energy residual resorh (:2099), in one launch.  Each CTA (32 i x 8
// strides of the partial rows, one of the four quantities) forms its per-i sums in
// a fixed order; the last CTA to finish solves the 1-D system with one warp while
// the others add up the residual's per-CTA partials (32 groups of 32, the strides
// of a 1024-thread block, then a tree over the groups).  Bound by latency: as two
// launches 9 us on 60x30x20 cells and 20 on 400x200x100, 5 and 13 as one.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) block_correct_kernel(Params p, Fields<T> g, const double *red_asm,
                                                            int nblk_asm, int check_finite, int ivar)
{
    pdl_enter();
    // 4 * nip; first the partial sums of the 8 rows of threads (rows of 1502 cells fit the
    // 48 KB that need no opt-in because they share the space)
    extern __shared__ double sm[];
    double (*sh)[33] = reinterpret_cast<double (*)[33]>(sm);
    __shared__ double grp[2][32];
    __shared__ int last;
    const int nip = p.nip, nim2 = p.nim2;
    {
        const int i = blockIdx.x * 32 + threadIdx.x, w = blockIdx.y;
        double s = 0.0;
        const double *src = g.bc + (size_t)w * nip + i;
#pragma unroll 8
        for (int part = threadIdx.y; part < g.npart; part += 8) s += src[(size_t)part * 4 * nip];
        sh[threadIdx.y][threadIdx.x] = s;
        __syncthreads();
        if (threadIdx.y == 0) {
            double t = 0.0;
            for (int y = 0; y < 8; ++y) t += sh[y][threadIdx.x];
            g.bcsum[(size_t)w * nip + i] = t;
            __threadfence();
            __syncwarp();
            if (threadIdx.x == 0) last = atomicAdd(&g.st->bc_done, 1) == (int)(gridDim.x * gridDim.y) - 1;
        }
        __syncthreads();
    }
    if (!last) return;
    __threadfence();
    const int tid = threadIdx.y * 32 + threadIdx.x, lane = threadIdx.x, warp = threadIdx.y;
    double *bl = sm, *blp = sm + nip, *blm = sm + 2 * nip, *blc = sm + 3 * nip;
    for (int q = tid; q < 4 * nip; q += 256) sm[q] = __ldcg(g.bcsum + q);
    __syncthreads();
    if (warp == 0) {
        block_tdma_warp(bl, blp, blm, blc, 1, nim2, g.delphi);
        if (lane == 0) g.st->bc_done = 0;
    } else {
        for (int v = warp - 1; v < 32; v += 7) {
            double sd = 0.0, sh2 = 0.0;
            for (int b = v * 32 + lane; b < nblk_asm; b += 1024) {
                sd += red_asm[(size_t)b * R_NSLOTS + R_SUMD];
                sh2 += red_asm[(size_t)b * R_NSLOTS + R_SUMH];
            }
            sd = warp_sum(sd);
            sh2 = warp_sum(sh2);
            if (lane == 0) {
                grp[0][v] = sd;
                grp[1][v] = sh2;
            }
        }
    }
    __syncthreads();
    if (warp == 1) {
        const double sd = warp_sum(grp[0][lane]), sh2 = warp_sum(grp[1][lane]);
        if (lane == 0) {
            Status *st = g.st;
            // resorh (calculateResiduals(5)) or resorc (calculateResiduals(6))
            const double res = sd / (sh2 + kSmall);
            if (ivar == 6) st->resorc = res; else st->resorh = res;
            if (check_finite && !isfinite(res)) st->nonfinite = 1;
        }
    }
}
// ---------------------------------------------------------------------------
// convertEnthalpyToTemp (CFDSolverManager.cpp:2531-2571), fused with the
// peak-temperature maximum (BoundCondManager.cpp:301) and the reductions of
// calculateFluxes (BoundCondManager.cpp:778-843): boundary conduction fluxes,
// heat accumulation and volumetric heat input.  H->T is evaluated in FP64.
// Bound by issue and by the FP64 conversions in FP32 (176 instructions a cell, XU 38 %,
// DRAM 32 %), by its divisions in FP64.  A warp that keeps to one chunk of the row, widths
// loaded once, the peak in the bulk precision and no conversion of a fraction that did not
// change: with the melt-pool step 88 -> 76 us on 400x200x100 cells, 178 -> 148 on
// 600x300x120, 26 -> 25 on 163x81x50; FP64 400x200x100 120 -> 115.  Three CTAs a SM: with
// four, some of the registers are spilled (80 us); five are as good on 400x200x100 but cost
// 120x60x40 3 us.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256, 3) h2t_kernel(Params p, Fields<T> g, double *red)
{
    pdl_wait();
    const Status *st = g.st;
    const int ni = p.ni, nj = p.nj, nk = p.nk, nip = p.nip;
    const int nim1 = p.nim1, njm1 = p.njm1, nkm1 = p.nkm1, nim2 = p.nim2, njm2 = p.njm2,
              nkm2 = p.nkm2;
    const double deltemp = p.tliquid - p.tsolid;
    const double delt = st->delt;
    // The FP64 build divides exactly as the reference; the FP32 build keeps the
    // inversion in FP64 but multiplies by reciprocals formed once per launch.
    constexpr bool kExact = sizeof(T) == sizeof(double);
    const double inv_acpl = 1.0 / p.acpl, inv_acpa = 1.0 / p.acpa,
                 inv_mush = 1.0 / (p.hlcal - p.hsmelt), inv_delt = 1.0 / delt;
    T tpeak = (T)-INFINITY;
    double accul = 0.0, heatvol = 0.0;
    const size_t sj = nip, sk = (size_t)nj * nip;
    const int js = st->jstart, is0 = st->istart;
    const double ts = p.tsolid;
    const bool steady = p.steady != 0;
    const bool volsrc = p.volsrc != 0;
    const int lane = threadIdx.x & 31;
    // Work unit: a chunk of 32 V cells of one x-line, V = 16 bytes per element;
    // lane l holds the 16-byte vector of cells base = chunk start + V l (the pitch
    // nip is a multiple of 32, so a vector lies wholly inside or wholly past the
    // padded row).  A warp keeps to one chunk of the row, so that what depends on x
    // alone is formed once, and steps over the rows (32-bit: their count is bounded
    // at context creation; a 64-bit division costs more than a chunk's enthalpy
    // inversions).
    constexpr int V = 16 / (int)sizeof(T);
    constexpr int RC = 32 * V;
    const unsigned cpr = ((unsigned)nip + RC - 1) / RC;  // chunks per row
    const unsigned unj = (unsigned)nj, nrows = (unsigned)nk * unj;
    const unsigned W = gridDim.x * (blockDim.x >> 5);
    const unsigned w0 = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const unsigned step = max(1u, W / cpr);  // warps a chunk of the row
    const double *dxw = g.dxpwinv, *dys = g.dypsinv, *dzb = g.dzpbinv;
    for (unsigned w = w0; w < cpr * step; w += W) {
        const int base = (int)(w % cpr) * RC + V * lane;
        const bool inrow = base < nip, whole = base + V <= ni;
        double xw[V + 1];  // the cells' faces (their difference is taken where it is used, so
                           // that a warp's first row is on its way before they are waited for)
#pragma unroll
        for (int v = 0; v <= V; ++v) xw[v] = g.xu[min(base + v, ni - 1)];
        for (unsigned r = w / cpr; r < nrows; r += step) {
            const int k = (int)(r / unj), j = (int)(r - (unsigned)k * unj);
            const size_t c0 = (size_t)r * nip + (inrow ? base : 0);
            T hv[V], hn[V], fln[V], rn[V], sv[V];
            ld16(g.h + c0, hv); ld16(g.hnot + c0, hn); ld16(g.fraclnot + c0, fln);
            ld16(g.rho_nxt + c0, rn);
            // the volumetric source input is zero everywhere without a volumetric source
            if (volsrc) ld16(g.sourceinput + c0, sv);
            const bool rowint = !steady && j >= 1 && j <= njm2 && k >= 1 && k <= nkm2;
            const double dy = rowint ? g.yv[j + 1] - g.yv[j] : 0.0, dz = rowint ? g.zw[k + 1] - g.zw[k] : 0.0;
            T tout[V], fout[V];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                tout[v] = fout[v] = T(0);
                if (!inrow || (!whole && base + v >= ni)) continue;
                const double h = (double)hv[v];
                double t;
                if (h >= p.hlcal) {
                    fout[v] = T(1);
                    t = (kExact ? (h - p.hlcal) / p.acpl : (h - p.hlcal) * inv_acpl) + p.tliquid;
                } else if (h <= p.hsmelt) {
                    const double root = sqrt(p.acpb * p.acpb + 2 * p.acpa * h) - p.acpb;
                    t = kExact ? root / p.acpa : root * inv_acpa;
                } else {
                    const double fl = kExact ? (h - p.hsmelt) / (p.hlcal - p.hsmelt) : (h - p.hsmelt) * inv_mush;
                    fout[v] = (T)fl;
                    t = deltemp * fl + p.tsolid;
                }
                tout[v] = (T)t;
                if (tout[v] > tpeak) tpeak = tout[v];
                if (!rowint || base + v < 1 || base + v > nim2) continue;
                double dh1 = h - (double)hn[v];
                if (fout[v] != fln[v]) dh1 += ((double)fout[v] - (double)fln[v]) * p.hlatnt;
                const double vol = (xw[v + 1] - xw[v]) * dy * dz;
                accul += kExact ? vol * (double)rn[v] * dh1 / delt : vol * (double)rn[v] * dh1 * inv_delt;
                if (volsrc) heatvol += (double)sv[v] * vol;
            }
            if (inrow) {
                if (whole) {
                    typename Vec16<T>::type w;
                    memcpy(&w, tout, 16);
                    *reinterpret_cast<typename Vec16<T>::type *>(g.temp + c0) = w;
                    memcpy(&w, fout, 16);
                    *reinterpret_cast<typename Vec16<T>::type *>(g.fracl + c0) = w;
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v)
                        if (base + v < ni) {
                            g.temp[c0 + v] = tout[v];
                            g.fracl[c0 + v] = fout[v];
                        }
                }
            }
            // melt-pool scan candidates (BoundCondManager.cpp:318-417), on the beam's
            // plane and on the top plane.  Most cells are solid, so each atomic is
            // issued only when it can still change the value (candidates only move one
            // way); the beam-row scalars are warp-reduced.
            if (k != nkm1 && (j != js || k < 1 || k > nkm2)) continue;
            int cmaxl = INT_MAX, cminl = INT_MIN;  // beam-row length candidates of this lane
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const int i = base + v;
                if (!inrow || i >= ni) continue;
                const double tt = (double)tout[v];
                if (j == js && k >= 1 && k <= nkm2 && tt < ts && k > *(volatile int *)&g.mp_kb[i])
                    atomicMax(&g.mp_kb[i], k);
                if (k == nkm1) {
                    if (j >= js && j <= njm2 && tt < ts && j < *(volatile int *)&g.mp_jup[i])
                        atomicMin(&g.mp_jup[i], j);
                    if (j >= 1 && j <= js && tt < ts && j > *(volatile int *)&g.mp_jdn[i])
                        atomicMax(&g.mp_jdn[i], j);
                    if (j == js) {
                        if (i >= is0 && i < nim1 && tt <= ts) cmaxl = min(cmaxl, i);
                        if (i >= 1 && i <= is0 && tt < ts) cminl = max(cminl, i);
                    }
                }
            }
            if (k == nkm1 && j == js) {  // row-uniform: every lane takes part
                const int wmin = __reduce_min_sync(0xffffffffu, cmaxl);
                const int wmax = __reduce_max_sync(0xffffffffu, cminl);
                if (lane == 0) {
                    if (wmin != INT_MAX) atomicMin(&g.st->mp_imax, wmin);
                    if (wmax != INT_MIN) atomicMax(&g.st->mp_imin, wmax);
                }
            }
        }
    }
    pdl_release();
    // Boundary conduction fluxes (BoundCondManager.cpp:778-843): a second pass
    // over the six interior boundary layers only, so that the bulk loop above
    // carries no flux accumulators.  Face f's layer is a 2-D index set.
    double fw = 0.0, fe = 0.0, fb = 0.0, ft = 0.0, fs = 0.0, fn = 0.0;
    {
        const int I = nim2, J = njm2, K = nkm2;  // interior extents
        // 32-bit: twice the faces of any domain whose arrays fit the memory
        const unsigned nx = (unsigned)J * K, ny = (unsigned)I * K, nz = (unsigned)I * J;
        const unsigned nall = 2 * (nx + ny + nz);
        const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
        const unsigned nthr = gridDim.x * blockDim.x;
        for (unsigned q = tid; q < nall; q += nthr) {
            unsigned r = q;
            int face, a, b;  // face 0..5 = W E B T S N
            if (r < 2 * nx) { face = (int)(r / nx); r %= nx; a = (int)(r % J); b = (int)(r / J); }
            else if ((r -= 2 * nx) < 2 * nz) { face = 2 + (int)(r / nz); r %= nz; a = (int)(r % I); b = (int)(r / I); }
            else { r -= 2 * nz; face = 4 + (int)(r / ny); r %= ny; a = (int)(r % I); b = (int)(r / I); }
            int i, j, k;
            if (face < 2) { i = face == 0 ? 1 : nim2; j = 1 + a; k = 1 + b; }
            else if (face < 4) { k = face == 2 ? 1 : nkm2; i = 1 + a; j = 1 + b; }
            else { j = face == 4 ? 1 : njm2; i = 1 + a; k = 1 + b; }
            const size_t c = cidx(i, j, k, nj, nip);
            const double h = (double)g.h[c];
            const double dn = (double)g.diff_nxt[c];
            switch (face) {
            case 0: fw += area_jk(p, g, j, k) * (dn * ((double)g.h[c - 1] - h) * dxw[1]); break;
            case 1: fe += area_jk(p, g, j, k) * (dn * ((double)g.h[c + 1] - h) * dxw[nim1]); break;
            case 2: fb += area_ij(p, g, i, j) * (dn * ((double)g.h[c - sk] - h) * dzb[1]); break;
            case 3: ft += area_ij(p, g, i, j) * (dn * ((double)g.h[c + sk] - h) * dzb[nkm1]); break;
            case 4: fs += area_ik(p, g, i, k) * (dn * ((double)g.h[c - sj] - h) * dys[1]); break;
            default: fn += area_ik(p, g, i, k) * (dn * ((double)g.h[c + sj] - h) * dys[njm1]); break;
            }
        }
    }
    double v[8] = {(double)tpeak, accul, heatvol, fw, fe, fb, ft, fs};
    const int s[8] = {R_TPEAK, R_ACCUL, R_HEATVOL, R_FW, R_FE, R_FB, R_FT, R_FS};
    const bool m[8] = {true, false, false, false, false, false, false, false};
    block_reduce_store<8>(v, s, m, red, blockIdx.x);
    __syncthreads();
    double v2[1] = {fn};
    const int s2[1] = {R_FN};
    const bool m2[1] = {false};
    block_reduce_store<1>(v2, s2, m2, red, blockIdx.x);
}

// Sentinels of the melt-pool scan candidates for the next outer iteration.
template <typename T>
__device__ void reset_scan_candidates(const Params &p, Fields<T> &g)
{
    for (int i = threadIdx.x; i < p.nip; i += blockDim.x) {
        g.mp_kb[i] = 0;
        g.mp_jup[i] = p.njm1;
        g.mp_jdn[i] = 0;
    }
    if (threadIdx.x == 0) {
        g.st->mp_imax = INT_MAX;
        g.st->mp_imin = INT_MIN;
    }
}

// ---------------------------------------------------------------------------
// getMeltPoolShape (BoundCondManager.cpp:280-447), one CTA.  The scans along
// i/j/k are evaluated per column in parallel, and so are the folds whose result
// depends on order (the NaN behaviour of std::max/min).  Also activates the momentum
// box (its exact-order ticket list is box_tickets_kernel's).
// ---------------------------------------------------------------------------
// The reference's folds acc = f(x_i, acc) in ascending i over the flagged columns,
// with f = std::max or std::min as the reference folds (maxd/mind): a NaN element
// makes acc NaN and the next element replaces it.  A fold therefore equals the
// extreme of the flagged elements after the last NaN, NaN when that NaN is the
// last flagged element, and includes init only when no NaN occurs -- which a
// block computes in two passes: the last flagged and the last NaN index, then
// the extreme after it.
__device__ __forceinline__ double fold_result(int last_flag, int last_nan, double ext, double init, bool is_max)
{
    if (last_flag < 0) return init;
    if (last_nan >= 0) return last_nan == last_flag ? (double)NAN : ext;
    return is_max ? ((ext < init) ? init : ext) : ((init < ext) ? init : ext);
}

// One CTA, bound by latency: a chain of block-wide reductions and gathered loads.
// The reductions go through one shared word per warp that every warp then reduces
// for itself (a block barrier each, four in all), and thread 0's loads for the pool
// length are issued with the columns'.  Measured on 120x60x40 cells 17.9 -> 9 us a
// launch (three folds of four barriers each, shared atomics from every thread).
template <typename T>
__global__ void __launch_bounds__(1024) meltpool_kernel(Params p, Fields<T> g, const double *red_h2t,
                                                        int nblk_h2t)
{
    pdl_enter();
    Status *st = g.st;
    extern __shared__ double colv[];  // 3 * nip doubles + nip ints
    __shared__ double wd[3][32];
    __shared__ int wi[6][32];
    const unsigned full = 0xffffffffu;
    const int nj = p.nj, nip = p.nip, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nim1 = p.nim1, nkm1 = p.nkm1, nim2 = p.nim2, njm2 = p.njm2, nkm2 = p.nkm2;
    const double ts = p.tsolid;
    const int js = st->jstart, is0 = st->istart, mp_imax = st->mp_imax, mp_imin = st->mp_imin;
    const double t0 = (double)g.temp[0];
    // peak temperature, and the column scans' candidates (gathered by h2t_kernel):
    // depth: per column i, mp_kb = the largest k in 1..nkm2 with T < Ts on the beam
    // plane (0 if none) -- the scan from nkm2 down visits nkm2..mp_kb+1.
    // width: mp_jup = first j >= jstart with T < Ts (njm1 if none), mp_jdn = first
    // j <= jstart going down with T < Ts (0 if none).
    double tp = -INFINITY;
    for (int b = threadIdx.x; b < nblk_h2t; b += blockDim.x)
        tp = fmax(tp, red_h2t[(size_t)b * R_NSLOTS + R_TPEAK]);
    int kmin_c = INT_MAX, jmax_c = INT_MIN, jmin_c = INT_MAX;
    for (int i = 1 + (int)threadIdx.x; i < nim1; i += blockDim.x) {
        const int kb = g.mp_kb[i], ju = g.mp_jup[i], jd = g.mp_jdn[i];
        if (kb < nkm2) kmin_c = min(kmin_c, kb + 1);
        if (ju > js) jmax_c = max(jmax_c, ju - 1);
        if (jd < js) jmin_c = min(jmin_c, jd + 1);
    }
    tp = warp_max(tp);
    kmin_c = __reduce_min_sync(full, kmin_c);
    jmax_c = __reduce_max_sync(full, jmax_c);
    jmin_c = __reduce_min_sync(full, jmin_c);
    if (lane == 0) {
        wd[0][warp] = tp;
        wi[0][warp] = kmin_c; wi[1][warp] = jmax_c; wi[2][warp] = jmin_c;
    }
    __syncthreads();
    tp = warp_max(wd[0][lane]);
    kmin_c = __reduce_min_sync(full, wi[0][lane]);
    jmax_c = __reduce_max_sync(full, wi[1][lane]);
    jmin_c = __reduce_min_sync(full, wi[2][lane]);
    if (isnan(t0)) tp = t0;  // std::max_element keeps a leading NaN
    if (threadIdx.x == 0) st->tpeak = tp;
    // every thread has read its candidates
    reset_scan_candidates(p, g);
    if (!(tp > ts)) {
        if (threadIdx.x == 0) {
            st->alen = 0.0;
            st->depth = 0.0;
            st->width = 0.0;
            st->momentum_active = 0;
        }
        return;
    }
    // Reads outside the node range (the reference reads past its arrays when the
    // pool touches the north/south boundary rows) return NaN instead.
    auto TT = [&](int i, int j, int k) {
        if (i < 0 || i >= p.ni || j < 0 || j >= nj || k < 0 || k >= p.nk) return (double)NAN;
        return (double)g.temp[cidx(i, j, k, nj, nip)];
    };
    auto YY = [&](int j) { return (j < 0 || j >= nj) ? (double)NAN : g.y[j]; };
    double *depv = colv, *wmax = colv + nip, *wmin = colv + 2 * nip;
    int *imaxc = (int *)(colv + 3 * nip);
    // length: first i >= istart on the top row with T <= Ts; last i <= istart with T < Ts
    const int imax = (is0 < nim1) ? (mp_imax == INT_MAX ? nim1 - 1 : mp_imax) : is0;
    const int imin = (is0 > 0) ? (mp_imin == INT_MIN ? 1 : mp_imin) : is0;
    const int kmin = min(nkm2, kmin_c) - 1;
    const int jmax = max(js, jmax_c) + 1;
    const int jmin = min(js, jmin_c) - 1;
    double xa[4], ta[4], za = 0.0, zb = 0.0;
    if (threadIdx.x == 0) {
        auto XX = [&](int i) { return (i < 0 || i >= p.ni) ? (double)NAN : g.x[i]; };
        const int at[4] = {imax, imax + 1, imin, imin - 1};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            xa[q] = XX(at[q]);
            ta[q] = TT(at[q], js, nkm1);
        }
        za = g.z[nkm1];
        zb = g.z[0];
    }
    // per-column interpolated values for the order-dependent folds
    // imaxc[i] bits: 1 = column enters the depth fold, 2 = the max-width fold,
    // 4 = the min-width fold (the reference's `continue` tests); per thread, and then
    // per block, the last flagged and the last NaN column of each fold
    int lf[3] = {-1, -1, -1}, ln[3] = {-1, -1, -1};
    for (int i = 1 + (int)threadIdx.x; i < nim1; i += blockDim.x) {
        int fl = 0;
        const bool d0 = kmin != 0 && !(TT(i, js, kmin + 1) < ts), d1 = jmax != js && !(TT(i, jmax - 1, nkm1) < ts),
                   d2 = jmin != js && !(TT(i, jmin + 1, nkm1) < ts);
        if (d0) {
            fl |= 1;
            double dtdzzinv = (g.z[kmin] - g.z[kmin - 1]) / (TT(i, js, kmin) - TT(i, js, kmin - 1));
            const double x = g.z[nkm1] - g.z[kmin] + (TT(i, js, kmin) - ts) * dtdzzinv;
            depv[i] = x;
            lf[0] = i;
            if (isnan(x)) ln[0] = i;
        }
        if (d1) {
            fl |= 2;
            double dtdyyinv = (YY(jmax) - YY(jmax + 1)) / (TT(i, jmax, nkm1) - TT(i, jmax + 1, nkm1));
            const double x = YY(jmax) + (ts - TT(i, jmax, nkm1)) * dtdyyinv;
            wmax[i] = x;
            lf[1] = i;
            if (isnan(x)) ln[1] = i;
        }
        if (d2) {
            fl |= 4;
            double dtdyyinv = (YY(jmin) - YY(jmin - 1)) / (TT(i, jmin, nkm1) - TT(i, jmin - 1, nkm1));
            const double x = YY(jmin) + (ts - TT(i, jmin, nkm1)) * dtdyyinv;
            wmin[i] = x;
            lf[2] = i;
            if (isnan(x)) ln[2] = i;
        }
        imaxc[i] = fl;
    }
    __syncthreads();  // the candidates' words are read
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        lf[q] = __reduce_max_sync(full, lf[q]);
        ln[q] = __reduce_max_sync(full, ln[q]);
        if (lane == 0) {
            wi[q][warp] = lf[q];
            wi[3 + q][warp] = ln[q];
        }
    }
    __syncthreads();
    double ex[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        lf[q] = __reduce_max_sync(full, wi[q][lane]);
        ln[q] = __reduce_max_sync(full, wi[3 + q][lane]);
        ex[q] = -INFINITY;  // of the elements, or of their negatives for the minimum
        const double *col = q == 0 ? depv : q == 1 ? wmax : wmin;
        for (int i = 1 + (int)threadIdx.x; i < nim1; i += blockDim.x)  // this thread's own columns
            if (i > ln[q] && (imaxc[i] >> q & 1)) ex[q] = fmax(ex[q], q == 2 ? -col[i] : col[i]);
        ex[q] = warp_max(ex[q]);
        if (lane == 0) wd[q][warp] = ex[q];
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) ex[q] = warp_max(wd[q][lane]);
    }
    if (threadIdx.x == 0) {
        const double depth_f = fold_result(lf[0], ln[0], ex[0], 0.0, true);
        const double ymax_f = fold_result(lf[1], ln[1], ex[1], g.y[0], true);
        const double ymin_f = fold_result(lf[2], ln[2], -ex[2], YY(js), false);
        double dtdxxinv = (xa[0] - xa[1]) / (ta[0] - ta[1]);
        double xxmax = xa[0] + (ts - ta[0]) * dtdxxinv;
        dtdxxinv = (xa[2] - xa[3]) / (ta[2] - ta[3]);
        double xxmin = xa[2] + (ts - ta[2]) * dtdxxinv;
        st->alen = xxmax - xxmin;
        st->depth = kmin == 0 ? za - zb : depth_f;
        const double yymax = jmax != js ? ymax_f : g.y[0];
        const double yymin = jmin != js ? ymin_f : YY(js);
        st->width = yymax - yymin;
        st->imax = imax; st->imin = imin; st->kmin = kmin; st->kmax = nkm2;
        st->jmax = jmax; st->jmin = jmin;
        st->istat = max(imin - 3, 1);
        st->iend = min(imax + 3, nim2);
        st->jstat = max(jmin - 3, 1);
        st->jend = min(jmax + 2, njm2);
        st->kstat = max(kmin - 2, 2);
        st->istatp1 = st->istat + 1;
        st->iendm1 = st->iend - 1;
        st->momentum_active = p.navierstokes ? 1 : 0;
        st->box_cells = st->momentum_active
            ? max(0, st->iendm1 - st->istatp1 + 1) * max(0, st->jend - st->jstat + 1) * max(0, nkm1 - st->kstat)
            : 0;
    }
}

// ---------------------------------------------------------------------------
// End of an outer iteration: calculateFluxes ratio (BoundCondManager.cpp:846-857),
// amaxres and the convergence test (CFDSolverManager.cpp:689-716).  One CTA.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void converge_kernel(Params p, Fields<T> gd, const double *red_h2t, int nb_h2t,
                                const double *red_bc, int nb_bc, const double *red_las, int nb_las,
                                const double *red_mom, int nb_mom, double tol, int check_finite,
                                LoopCtl lc)
{
    pdl_enter();
    // ten sums of per-CTA partials, each in the order of a one-slot block reduction
    // (strided per-thread sums, a warp tree, a tree over the warps); a warp takes
    // each sum's second tree, so the block meets twice instead of three times a sum
    // (9.8 -> 6 us a launch; latency)
    __shared__ double wsum[10][33];
    Status *st = gd.st;
    double list[5], tpeak = 0.0, resorh = 0.0;
    int power = 0;
    if (threadIdx.x == 0) {
        list[0] = st->resorm; list[1] = st->resoru; list[2] = st->resorv; list[3] = st->resorw; list[4] = st->resorc;
        tpeak = st->tpeak; resorh = st->resorh; power = st->powerindicator;
    }
    {
        const int slot[10] = {R_ACCUL, R_HEATVOL, R_FW, R_FE, R_FB, R_FT, R_FS, R_FN, R_AHTOP, R_HEATIN};
        double acc[10];
#pragma unroll
        for (int q = 0; q < 10; ++q) acc[q] = 0.0;
        for (int b = threadIdx.x; b < nb_h2t; b += blockDim.x) {
#pragma unroll
            for (int q = 0; q < 8; ++q) acc[q] += red_h2t[(size_t)b * R_NSLOTS + slot[q]];
        }
        for (int b = threadIdx.x; b < nb_bc; b += blockDim.x) acc[8] += red_bc[(size_t)b * R_NSLOTS + slot[8]];
        for (int b = threadIdx.x; b < nb_las; b += blockDim.x) acc[9] += red_las[(size_t)b * R_NSLOTS + slot[9]];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
#pragma unroll
        for (int q = 0; q < 10; ++q) acc[q] = warp_sum(acc[q]);
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 10; ++q) wsum[q][warp] = acc[q];
        }
        __syncthreads();
        if (warp < 10) {
            const double r = warp_sum(lane < nw ? wsum[warp][lane] : 0.0);
            if (lane == 0) wsum[warp][32] = r;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double accul = wsum[0][32], heatvol = wsum[1][32], fw = wsum[2][32], fe = wsum[3][32], fb = wsum[4][32],
                     ft = wsum[5][32], fs = wsum[6][32], fn = wsum[7][32], ahtop = wsum[8][32], heatin = wsum[9][32];
        st->accul = p.steady ? 0.0 : accul;
        st->heatvol = p.steady ? 0.0 : heatvol;
        st->fluxwest = fw; st->fluxeast = fe; st->fluxbottom = fb; st->fluxtop = ft;
        st->fluxsouth = fs; st->fluxnorth = fn;
        st->ahtoploss = ahtop;
        st->heatinlaser = heatin;
        const double heatout = (fn + fb + fw + fe + fs) - ahtop;
        st->heatout = heatout;
        double ratio = p.steady ? -heatout / heatin : (heatvol + heatin) / (accul - heatout);
        st->ratio = ratio;
        double amaxres = list[0];
        for (int q = 1; q < 5; q++)
            if (amaxres < list[q]) amaxres = list[q];
        int conv;
        if (p.steady)
            conv = (ratio <= 1.001 && ratio >= 0.999 && amaxres < tol);
        else if (power == 1)
            conv = (ratio <= 1.01 && ratio >= 0.99 && amaxres < tol);
        else
            conv = (resorh < 1e-6 && amaxres < tol);
        st->converged = conv;
        if (check_finite && (!isfinite(tpeak) || !isfinite(ratio) || !isfinite(resorh)))
            st->nonfinite = 1;
        if (lc.active) {
            // the host loop's bookkeeping: count the iteration, remember its box, and
            // continue unless converged, failed or out of iterations
            const int it = st->lp_niter + 1;
            st->lp_niter = it;
            st->lp_small += st->lp_mode;
            const int box = st->momentum_active ? st->box_cells : 0;
            st->lp_box = box;
            const int mode = lc.chain_nc > 0
                ? (!st->momentum_active || chain_box_fits(st->iendm1 - st->istatp1 + 1, st->jend - st->jstat + 1,
                                                          p.nkm2 - st->kstat + 1, lc.exact, lc.chain_nc))
                : lc.cap >= 0 && box <= lc.cap;
            st->lp_mode = mode;
            const int cont = !conv && !st->nonfinite && !*(volatile int *)&st->error && it < lc.maxit;
            if (lc.has_next) {
                cudaGraphSetConditional(lc.mode_next, (unsigned)mode);
                cudaGraphSetConditional(lc.cont, (unsigned)cont);
            }
        }
    }
    (void)red_mom; (void)nb_mom;
}

// Head of a step captured as one graph: the momentum path of its first outer
// iteration, which the host has chosen from the box of the last iteration before it.
__global__ void loop_init_kernel(Status *st, LoopCtl lc)
{
    cudaGraphSetConditional(lc.mode_next, (unsigned)st->lp_mode);
}
void launch_loop_init(Status *st, const LoopCtl &lc, cudaStream_t s)
{
    loop_init_kernel<<<1, 1, 0, s>>>(st, lc);
}

// ---------------------------------------------------------------------------
// updateSolutions (CFDSolverManager.cpp:2625-2687): solid velocities to zero and
// the previous-step copies.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void update_solutions_kernel(Params p, Fields<T> g, double trackindx, int trackid)
{
    pdl_enter();
    const size_t total = (size_t)p.nk * p.nj * p.nip;
    const T ts = (T)p.tsolid;
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < total;
         c += (size_t)gridDim.x * blockDim.x) {
        if (g.temp[c] <= ts) {
            g.uvel[c] = T(0);
            g.vvel[c] = T(0);
            g.wvel[c] = T(0);
        }
        g.unot[c] = g.uvel[c];
        g.vnot[c] = g.vvel[c];
        g.wnot[c] = g.wvel[c];
        g.hnot[c] = g.h[c];
        g.fraclnot[c] = g.fracl[c];
        if (p.powder) {  // CFDSolverManager.cpp:2666-2678
            const T fl = g.fracl[c];
            g.csfrac[c] = maxd(g.csfrac[c], fl);
            g.solfrac[c] = maxd(g.solfrac[c], (T)((double)fl * trackindx));
            if (g.temp[c] > ts) g.mpphase[c] = (T)trackid;
            if (g.temp[c] > (T)p.tliquid) g.mpliq[c] = (T)trackid;
        }
    }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename T> void launch_laser(Inst<T> &I)
{
    launch_k(I.pdl, laser_kernel<T>, I.nb_las, 256, 0, I.stream, I.p, I.g, I.red_las);
}
template <typename T> void launch_energy_bc(Inst<T> &I)
{
    launch_k(I.pdl, energy_bc_kernel<T>, I.nb_bc, 256, 0, I.stream, I.p, I.g, I.red_bc);
}
template <typename T> void launch_block_correct(Inst<T> &I, int ivar)
{
    launch_k(I.pdl, block_correct_kernel<T>, dim3(I.p.nip / 32, 4), dim3(32, 8),
             std::max(4 * I.p.nip, 8 * 33) * sizeof(double), I.stream,
             I.p, I.g, I.red_asm, I.nb_asm, I.check_finite, ivar);
}
// Field read-out: the padded [k][j][nip] array widened to FP64 and packed to
// the reference's unpadded [k][j][ni] layout (CFDSolverManager.cpp:249), so
// that a single contiguous copy moves it to the host.
template <typename T>
__global__ void pack_field_kernel(const T *src, double *dst, int ni, int nip, long long rows)
{
    const long long n = rows * ni;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const long long r = q / ni;
        const int i = (int)(q - r * ni);
        dst[q] = (double)src[r * nip + i];
    }
}
template <typename T> void launch_pack_field(const T *src, double *dst, int ni, int nip,
                                             long long rows, int sm_count, cudaStream_t s)
{
    pack_field_kernel<T><<<sm_count * 4, 256, 0, s>>>(src, dst, ni, nip, rows);
}

// Cell-centred velocity for output (vtsBinWriter::transferVelNodes,
// vtsBinWriter.cpp:497-522): the mean of the two faces of component `comp`
// (0 u, 1 v, 2 w) on interior nodes of the active domain, zero where T <= T_solidus,
// on the boundary nodes and on inactive powder layers, packed to FP64 [k][j][ni].
template <typename T>
__global__ void centre_velocity_kernel(Params p, Fields<T> g, int comp, double *dst)
{
    const long long n = (long long)p.ni * p.nj * p.nk_alloc;  // every allocated plane
    const T *f = comp == 0 ? g.uvel : comp == 1 ? g.vvel : g.wvel;
    const size_t step = comp == 0 ? 1 : comp == 1 ? (size_t)p.nip : (size_t)p.nj * p.nip;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n;
         q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q % p.ni);
        const long long r = q / p.ni;
        const int j = (int)(r % p.nj), k = (int)(r / p.nj);
        double v = 0.0;
        if (i >= 1 && i < p.nim1 && j >= 1 && j < p.njm1 && k >= 1 && k < p.nkm1) {
            const size_t c = cidx(i, j, k, p.nj, p.nip);
            v = ((double)f[c] + (double)f[c + step]) * 0.5;
            if ((double)g.temp[c] <= p.tsolid) v = 0.0;
        }
        dst[q] = v;
    }
}
template <typename T> void launch_centre_velocity(Inst<T> &I, int comp, double *dst)
{
    centre_velocity_kernel<T><<<I.grid_1d, 256, 0, I.stream>>>(I.p, I.g, comp, dst);
}

// Resident 256-thread CTAs of h2t_kernel per SM (its grid is one full wave).
template <typename T> int h2t_blocks_per_sm()
{
    int nb = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, h2t_kernel<T>, 256, 0);
    return nb > 0 ? nb : 1;
}
template <typename T> void launch_h2t(Inst<T> &I)
{
    launch_k(I.pdl, h2t_kernel<T>, I.nb_h2t, 256, 0, I.stream, I.p, I.g, I.red_h2t);
}
template <typename T> void launch_meltpool(Inst<T> &I)
{
    size_t smem = 3 * (size_t)I.p.nip * sizeof(double) + (size_t)I.p.nip * sizeof(int);
    launch_k(I.pdl, meltpool_kernel<T>, 1, 1024, smem, I.stream, I.p, I.g, I.red_h2t, I.nb_h2t);
}
template <typename T> void launch_converge(Inst<T> &I, double tol, const LoopCtl &lc)
{
    launch_k(I.pdl, converge_kernel<T>, 1, 1024, 0, I.stream, I.p, I.g, I.red_h2t, I.nb_h2t, I.red_bc, I.nb_bc,
                                                  I.red_las, I.nb_las, I.red_mom, I.nb_mom, tol,
                                                  I.check_finite, lc);
}
template <typename T> void launch_update_solutions(Inst<T> &I)
{
    launch_k(I.pdl, update_solutions_kernel<T>, I.grid_1d, 256, 0, I.stream, I.p, I.g, I.trackindx, I.trackid);
}

#define AMCFD_INST(T)                                        \
    template void launch_laser<T>(Inst<T> &);               \
    template void launch_energy_bc<T>(Inst<T> &);           \
    template void launch_block_correct<T>(Inst<T> &, int);  \
    template void launch_h2t<T>(Inst<T> &);                 \
    template int h2t_blocks_per_sm<T>();                    \
    template void launch_pack_field<T>(const T *, double *, int, int, long long, int, cudaStream_t); \
    template void launch_centre_velocity<T>(Inst<T> &, int, double *);                                \
    template void launch_meltpool<T>(Inst<T> &);            \
    template void launch_converge<T>(Inst<T> &, double, const LoopCtl &); \
    template void launch_update_solutions<T>(Inst<T> &);
AMCFD_INST(double)
AMCFD_INST(float)
#undef AMCFD_INST

}  // namespace amcfd
