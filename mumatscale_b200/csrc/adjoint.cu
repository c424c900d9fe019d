// adjoint.cu — frozen-CA replay and hand-written adjoint of the continuous
// part of one timestep: diffusion (growth.c:69-162) followed by the fraction-
// solid change (growth.c:220-273), with respect to the solute, liquid
// concentration and fraction-solid fields and to the parameters D_l, k and
// the Gibbs-Thomson coefficient.
//
// Frozen CA.  Everything discrete in a step is taken from a recorded forward
// run: which branch fs_change took in every cell (liquid reset, solid keep,
// growth, growth clamped at fs = 1, growth reset at fs < 0), nucleation and
// capture (which change no continuous value: a captured cell was reset to
// cl = ce, fs = 0 in the same step already), and the curvature used.  With
// those fixed, a step is a smooth map x_t -> x_{t+1} of (ce, cl, fs), and
// its transpose Jacobian is applied here cell by cell.
//
// The replay kernel evaluates the same expressions as the step's stencil
// (kernels.cu, cell_update), in the same order and precision, so with the
// recorded parameters it reproduces the recorded trajectory bit for bit.
#include <cuda.h>
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "mms_internal.h"

namespace mms {

constexpr int ADJ_NT = 256;

// The replay and the backward step: a CTA of 32 x 8 threads, one column of
// cells each, marches up `zc` planes.  The z neighbours stay in registers, the
// x and y neighbours come from the L1 cache.
constexpr int ADX = 32, ADY = 8;

struct Column {
    int i, j, k0, k1;
    bool on;
    long long c;  // cell (i, j, k0)
};

__device__ __forceinline__ Column column_of(const Geo &g, int zc)
{
    Column q;
    q.i = (int)blockIdx.x * ADX + (int)threadIdx.x + 1;
    q.j = (int)blockIdx.y * ADY + (int)threadIdx.y + 1;
    q.k0 = (int)blockIdx.z * zc + 1;
    q.k1 = min(q.k0 + zc - 1, g.gz);
    q.on = q.i <= g.gx && q.j <= g.gy;
    q.c = (long long)q.k0 * g.sz + (long long)q.j * g.sy + q.i;
    return q;
}

__device__ __forceinline__ bool interior_cell(const Geo &g, long long v, int &i, int &j, int &k, long long &c)
{
    long long n = (long long)g.gx * g.gy * g.gz;
    if (v >= n) return false;
    i = (int)(v % g.gx) + 1;
    long long r = v / g.gx;
    j = (int)(r % g.gy) + 1;
    k = (int)(r / g.gy) + 1;
    c = (long long)k * g.sz + (long long)j * g.sy + i;
    return true;
}

// ------------------------------------------------------------------ replay
// x_t (ce0, cl0, fs0) -> x_{t+1} (ce1, cl1, fs1) with the branches of step
// ts (flags) and the curvature it used, under the parameters in p.
// Bounded by the latency of a plane's loads, near the fields' bytes (57 a cell
// in FP64 with curvature: 18 us at 128^3, 24 measured; 33 when each thread
// divided its cell number in 64 bits and read all six neighbours).
template <typename Real>
__global__ void __launch_bounds__(ADJ_NT) k_replay(Geo g, Phys p, int zc, const Real *__restrict__ ce0,
                                                   const Real *__restrict__ cl0, const Real *__restrict__ fs0,
                                                   Real *__restrict__ ce1, Real *__restrict__ cl1,
                                                   Real *__restrict__ fs1, const unsigned char *__restrict__ flags,
                                                   const double *__restrict__ curv, unsigned long long ts)
{
    const Column col = column_of(g, zc);
    if (!col.on) return;
    const PhysR<Real> q = phys_r<Real>(p);
    const int i = col.i, j = col.j;
    const Real one_x = (Real)(1 - g.padx), one_y = (Real)(1 - g.pady), one_zp = (Real)(1 - g.padz_hi),
               one_zm = (Real)(1 - g.padz_lo);
    const Real ox_p = i == g.gx ? one_x : (Real)1, ox_m = i == 1 ? one_x : (Real)1;
    const Real oy_p = j == g.gy ? one_y : (Real)1, oy_m = j == 1 ? one_y : (Real)1;
    const bool in_xy = i > 1 && i < g.gx && j > 1 && j < g.gy;
    long long c = col.c;
    Real cl_m = cl0[c - g.sz], fs_m = fs0[c - g.sz], conc = cl0[c], lspfs = fs0[c];
    for (int k = col.k0; k <= col.k1; k++, c += g.sz) {
        const Real cl_p = cl0[c + g.sz], fs_p = fs0[c + g.sz], oce = ce0[c];
        const int br = flags[c];
        const Real nb_cl[6] = {cl0[c + 1], cl0[c - 1], cl0[c + g.sy], cl0[c - g.sy], cl_p, cl_m};
        const Real nb_fs[6] = {fs0[c + 1], fs0[c - 1], fs0[c + g.sy], fs0[c - g.sy], fs_p, fs_m};
        const Real one_m[6] = {ox_p, ox_m, oy_p, oy_m, k == g.gz ? one_zp : (Real)1, k == 1 ? one_zm : (Real)1};
        const bool interior = in_xy && k > 1 && k < g.gz;
        // diffusion sum: cell_update's expressions
        Real nbsum = 0;
        if (sizeof(Real) == 4) {
            const float B = 0.5f * ((float)q.rs - (float)q.rl);
            const float A = fmaf(B, (float)lspfs, (float)q.rl);
            float acc = 0.f;
#pragma unroll
            for (int n = 0; n < 6; n++) {
                float r = fmaf(B, (float)nb_fs[n], A);
                if (!interior) r *= (float)one_m[n];
                acc = fmaf(r, (float)nb_cl[n] - (float)conc, acc);
            }
            nbsum = (Real)acc;
        } else if (interior) {
#pragma unroll
            for (int n = 0; n < 6; n++) {
                Real fs_av = (Real)0.5 * (lspfs + nb_fs[n]);
                Real r = (q.rs * fs_av + q.rl * (1 - fs_av));
                nbsum += r * (nb_cl[n] - conc);
            }
        } else {
#pragma unroll
            for (int n = 0; n < 6; n++) {
                Real fs_av = (Real)0.5 * (lspfs + nb_fs[n]);
                Real r = (q.rs * fs_av + q.rl * (1 - fs_av)) * one_m[n];
                nbsum += r * (nb_cl[n] - conc);
            }
        }
        const Real cen = oce + nbsum;
        Real cl_new, fs_new;
        if (br == BR_RESET || br == BR_NEG) {
            cl_new = cen;
            fs_new = 0;
        } else if (br == BR_KEEP) {
            cl_new = (sizeof(Real) == 8) ? cen * q.k_inv : cen * q.k_inv + q.c0k;
            fs_new = lspfs;
        } else {
            const double Td = temp_cell(p, nullptr, nullptr, c, j, k, ts);
            if (sizeof(Real) == 8) {
                const Real Tcell = (Real)Td;
                Real c_int = q.cinit + q.m_inv * (Tcell - q.Tliq);
                if (p.tip_curv) c_int = q.cinit + q.m_inv * (Tcell - q.Tliq + q.gibbs * (Real)curv[c]);
                Real dce = cen - oce;
                Real dcl = (c_int - conc) * q.D_xt * 2 + dce / (1 - q.km * lspfs);
                Real dfs = (dcl * ((Real)1. - q.km * lspfs) - dce) * q.km_inv / conc;
                cl_new = conc + dcl;
                fs_new = lspfs + dfs;
            } else {
                const Real dT = (Real)(Td - p.Tliq);
                Real c_int = q.m_inv * dT;
                if (p.tip_curv) c_int = q.m_inv * (dT + q.gibbs * (Real)curv[c]);
                const float dce = (float)nbsum;
                const float u = 1.f - (float)q.km * (float)lspfs;
                const float t2 = ((float)c_int - (float)conc) * (2.f * (float)q.D_xt);
                const float dcl = t2 + __fdividef(dce, u);
                const float dfs = __fdividef(t2 * u * (float)q.km_inv, (float)conc + (float)q.cinit);
                cl_new = conc + dcl;
                fs_new = lspfs + dfs;
            }
            if (br == BR_CLAMP) fs_new = 1;
        }
        ce1[c] = cen;
        cl1[c] = cl_new;
        fs1[c] = fs_new;
        cl_m = conc;
        fs_m = lspfs;
        conc = cl_p;
        lspfs = fs_p;
    }
}

// ----------------------------------------------------------------- adjoint
// Adjoint of a cell's diffusion sum (nu) from the adjoints lce and lcl of ce
// and cl after the step; before: the adjoint of ce before the step.
template <typename Real>
__device__ __forceinline__ Real adj_nu(const Phys &p, int br, Real lce, Real lcl, Real fs, Real &before)
{
    Real n;
    if (br == BR_RESET || br == BR_NEG) {  // cl' = ce' = oce + nbsum
        n = lce + lcl;
        before = n;
    } else if (br == BR_KEEP) {            // cl' = ce' / k
        n = lce + lcl * (Real)p.k_inv;
        before = n;
    } else {                               // cl' = cl + t2 + nbsum / u
        const Real u = (Real)1 - (Real)p.km * fs;
        n = lce + lcl / u;
        before = lce;
    }
    return n;
}

// Parameter-gradient slots accumulated per block.
enum AdjSlot : int { AS_RL = 0, AS_DXT, AS_KM, AS_KMINV, AS_KINV, AS_GIBBS, AS_COUNT };

// One step backward.  In: the adjoints lce1, lcl1, lfs1 after the step; out:
// those before it, and the step's contribution to the parameter gradients,
// added to this block's own sums (partial: its blocks add up once, after the
// last step, in a fixed order).  A cell needs the diffusion-sum adjoints of its
// six neighbours: each plane's are formed once, with the tile's rim, in shared
// memory (two planes in turn, one barrier a plane).
// Bounded by the latency of a plane's loads, which are all issued before its
// barrier (64 us at 128^3 in FP64; 30 would be the fields' bytes, 12 words and
// the branch a cell).  As a pointwise pass that wrote them out (13 us), a gather
// pass (48) and a fold of all blocks' sums in one CTA after every step (24) it
// took 85.
template <typename Real>
__global__ void __launch_bounds__(ADJ_NT, 3) k_adj_step(Geo g, Phys p, int zc, const unsigned char *__restrict__ flags,
                                                     const double *__restrict__ curv, const Real *__restrict__ ce0,
                                                     const Real *__restrict__ cl0, const Real *__restrict__ fs0,
                                                     const Real *__restrict__ ce1, const Real *__restrict__ lce1,
                                                     const Real *__restrict__ lcl1, const Real *__restrict__ lfs1,
                                                     Real *__restrict__ lce0, Real *__restrict__ lcl0,
                                                     Real *__restrict__ lfs0, double *__restrict__ partial,
                                                     unsigned long long ts)
{
    constexpr int PW = ADX + 2, PN = PW * (ADY + 2);
    __shared__ Real s_nu[2][PN];
    const Column col = column_of(g, zc);
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * ADX + tx;
    const int i = col.i, j = col.j;
    // what nu of a cell is formed from; 0 outside the domain, where no
    // diffusion sum is formed
    struct Nu {
        int br;
        Real lce, lcl, fs;
    };
    auto fetch = [&](bool on, int I, int J, int K) -> Nu {
        if (!on || I < 1 || I > g.gx || J < 1 || J > g.gy || K < 1 || K > g.gz) return {BR_RESET, 0, 0, 0};
        const long long c = (long long)K * g.sz + (long long)J * g.sy + I;
        return {flags[c], lce1[c], lcl1[c], fs0[c]};
    };
    auto nu_of = [&](const Nu &v, Real &before) { return adj_nu<Real>(p, v.br, v.lce, v.lcl, v.fs, before); };
    // this thread's cell of the tile's rim (34 + 34 + 8 + 8 cells)
    const bool rim = tid < 2 * PW + 2 * ADY;
    const int ex = tid < 2 * PW ? tid % PW : (tid - 2 * PW < ADY ? 0 : PW - 1);
    const int ey = tid < 2 * PW ? (tid < PW ? 0 : ADY + 1) : 1 + (tid - 2 * PW) % ADY;
    const int ri = (int)blockIdx.x * ADX + ex, rj = (int)blockIdx.y * ADY + ey, rat = ey * PW + ex;
    double acc[AS_COUNT] = {0, 0, 0, 0, 0, 0};
    // absolute concentrations (the FP32 form stores ce, cl - Cinit)
    const Real off = (sizeof(Real) == 4) ? (Real)p.cinit : (Real)0;
    const Real rs = (Real)p.rs, rl = (Real)p.rl;
    const Real one_x = (Real)(1 - g.padx), one_y = (Real)(1 - g.pady), one_zp = (Real)(1 - g.padz_hi),
               one_zm = (Real)(1 - g.padz_lo);
    const Real ox_p = i == g.gx ? one_x : (Real)1, ox_m = i == 1 ? one_x : (Real)1;
    const Real oy_p = j == g.gy ? one_y : (Real)1, oy_m = j == 1 ? one_y : (Real)1;
    long long c = col.c;
    Real b_c = 0, b_p = 0, b_x;
    const Nu vm = fetch(true, i, j, col.k0 - 1), vc = fetch(true, i, j, col.k0), vr = fetch(rim, ri, rj, col.k0);
    Real cl_m = 0, fs_m = 0, cl_c = 0, fs_c = 0;
    if (col.on) {
        cl_m = cl0[c - g.sz];
        fs_m = fs0[c - g.sz];
        cl_c = cl0[c];
        fs_c = fs0[c];
    }
    const int at = (ty + 1) * PW + tx + 1;
    Real nu_m = nu_of(vm, b_x), nu_c = nu_of(vc, b_c);
    s_nu[col.k0 & 1][at] = nu_c;
    if (rim) s_nu[col.k0 & 1][rat] = nu_of(vr, b_x);
    for (int k = col.k0; k <= col.k1; k++, c += g.sz) {
        const Real *plane = s_nu[k & 1];
        // every load of the plane, and of the next one's nu, before the barrier
        Real ncl[6], nfs[6], a_cl = 0, a_fs = 0;
        int br = BR_RESET;
        if (col.on) {
            ncl[0] = cl0[c + 1], ncl[1] = cl0[c - 1], ncl[2] = cl0[c + g.sy], ncl[3] = cl0[c - g.sy];
            ncl[4] = cl0[c + g.sz], ncl[5] = cl_m;
            nfs[0] = fs0[c + 1], nfs[1] = fs0[c - 1], nfs[2] = fs0[c + g.sy], nfs[3] = fs0[c - g.sy];
            nfs[4] = fs0[c + g.sz], nfs[5] = fs_m;
            br = flags[c];
            a_cl = lcl1[c];
            a_fs = lfs1[c];
        }
        const Nu vp = fetch(true, i, j, k + 1), vq = fetch(rim && k < col.k1, ri, rj, k + 1);
        __syncthreads();
        const Real nu_p = nu_of(vp, b_p);
        // read after the next barrier
        s_nu[(k + 1) & 1][at] = nu_p;
        if (rim) s_nu[(k + 1) & 1][rat] = nu_of(vq, b_x);
        if (col.on) {
            const Real cl_p = ncl[4], fs_p = nfs[4];
            const Real conc = cl_c + off, lspfs = fs_c;
            const Real nnu[6] = {plane[at + 1], plane[at - 1], plane[at + PW], plane[at - PW], nu_p, nu_m};
            const Real one_m[6] = {ox_p, ox_m, oy_p, oy_m, k == g.gz ? one_zp : (Real)1, k == 1 ? one_zm : (Real)1};
            Real gcl = 0, gfs = 0, grl = 0;
#pragma unroll
            for (int n = 0; n < 6; n++) {
                const Real cl_n = ncl[n] + off, fs_n = nfs[n];
                const Real fs_av = (Real)0.5 * (lspfs + fs_n);
                const Real r = rs * fs_av + rl * ((Real)1 - fs_av);
                // a neighbour inside the domain sees this cell with factor 1
                const Real nu_n = nnu[n];
                gcl += nu_n * r - nu_c * r * one_m[n];
                gfs += (Real)0.5 * (rs - rl) * (nu_c * (cl_n - conc) * one_m[n] + nu_n * (conc - cl_n));
                grl += nu_c * ((Real)1 - fs_av) * (cl_n - conc) * one_m[n];
            }
            acc[AS_RL] += (double)grl;
            if (br == BR_KEEP) {
                gfs += a_fs;                                                    // fs' = fs
                acc[AS_KINV] += (double)a_cl * ((double)ce1[c] + (double)off);  // cl' = ce' k_inv
            } else if (br == BR_GROW || br == BR_CLAMP) {
                const Real D_xt = (Real)p.D_xt, km = (Real)p.km, km_inv = (Real)p.km_inv, m_inv = (Real)p.m_inv;
                const double Td = temp_cell(p, nullptr, nullptr, c, j, k, ts);
                const Real kap = p.tip_curv ? (Real)curv[c] : (Real)0;
                const Real c_int = (Real)p.cinit + m_inv * ((Real)(Td - p.Tliq) + (Real)p.gibbs * kap);
                const Real u = (Real)1 - km * lspfs;
                const Real dce = ce1[c] - ce0[c];          // the diffusion sum
                const Real t2 = (c_int - conc) * (Real)2 * D_xt;
                // cl' = cl + t2 + dce / u
                gcl += a_cl * ((Real)1 - (Real)2 * D_xt);
                gfs += a_cl * dce * km / (u * u);
                acc[AS_DXT] += (double)(a_cl * (Real)2 * (c_int - conc));
                acc[AS_KM] += (double)(a_cl * dce * lspfs / (u * u));
                acc[AS_GIBBS] += (double)(a_cl * (Real)2 * D_xt * m_inv * kap);
                if (br == BR_GROW) {
                    // fs' = fs + W km_inv / cl with W = dcl u - dce = t2 u
                    const Real W = t2 * u;
                    gcl += a_fs * km_inv * (-(Real)2 * D_xt * u / conc - W / (conc * conc));
                    gfs += a_fs * ((Real)1 - km * t2 * km_inv / conc);
                    acc[AS_DXT] += (double)(a_fs * (Real)2 * (c_int - conc) * u * km_inv / conc);
                    acc[AS_KM] += (double)(-a_fs * lspfs * t2 * km_inv / conc);
                    acc[AS_KMINV] += (double)(a_fs * W / conc);
                    acc[AS_GIBBS] += (double)(a_fs * (Real)2 * D_xt * m_inv * kap * u * km_inv / conc);
                }
            }
            lce0[c] = b_c;
            lcl0[c] = gcl;
            lfs0[c] = gfs;
            cl_m = cl_c;
            fs_m = fs_c;
            cl_c = cl_p;
            fs_c = fs_p;
        }
        nu_m = nu_c;
        nu_c = nu_p;
        b_c = b_p;
    }
    // block sums of the parameter terms, in a fixed order
    __shared__ double sh[AS_COUNT][ADJ_NT / 32];
#pragma unroll
    for (int s = 0; s < AS_COUNT; s++) {
        double v = acc[s];
        for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
        if (tx == 0) sh[s][ty] = v;
    }
    __syncthreads();
    if (tid < AS_COUNT) {
        double v = 0;
        for (int q = 0; q < ADJ_NT / 32; q++) v += sh[tid][q];
        const long long b = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
        partial[b * AS_COUNT + tid] += v;
    }
}

// The gradient from the blocks' sums (one block; fixed order, so the result
// is reproducible).
__global__ void k_adj_fold(const double *__restrict__ partial, int nblocks, double *__restrict__ grad)
{
    __shared__ double sh[AS_COUNT][32];
    const int s = threadIdx.y, lane = threadIdx.x;  // blockDim (32, AS_COUNT)
    double v = 0;
    for (int b = lane; b < nblocks; b += 32) v += partial[(long long)b * AS_COUNT + s];
    sh[s][lane] = v;
    __syncthreads();
    if (lane == 0) {
        double t = 0;
        for (int q = 0; q < 32; q++) t += sh[s][q];
        grad[s] = t;
    }
}

// Terminal adjoint of L = 1/2 sum (ce - target)^2 over interior cells:
// lce = ce - target, lcl = lfs = 0; per-block partial sums of the loss.
template <typename Real>
__global__ void __launch_bounds__(ADJ_NT) k_adj_terminal(Geo g, double cinit_off, const Real *__restrict__ ce,
                                                         const double *__restrict__ target, Real *lce, Real *lcl,
                                                         Real *lfs, double *__restrict__ partial)
{
    int i, j, k;
    long long c;
    double l = 0;
    if (interior_cell(g, blockIdx.x * (long long)ADJ_NT + threadIdx.x, i, j, k, c)) {
        const double d = ((double)ce[c] + cinit_off) - target[c];
        l = 0.5 * d * d;
        if (lce) {
            lce[c] = (Real)d;
            lcl[c] = 0;
            lfs[c] = 0;
        }
    }
    __shared__ double sh[ADJ_NT / 32];
    for (int d = 16; d > 0; d >>= 1) l += __shfl_down_sync(0xffffffffu, l, d);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int q = 0; q < ADJ_NT / 32; q++) t += sh[q];
        partial[blockIdx.x] = t;
    }
}

__global__ void k_sum_partials(const double *__restrict__ partial, int n, double *out)
{
    __shared__ double sh[256];
    double v = 0;
    for (int b = threadIdx.x; b < n; b += 256) v += partial[b];
    sh[threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int q = 0; q < 256; q++) t += sh[q];
        *out = t;
    }
}

// ------------------------------------------------------------------ launchers
static int adj_blocks(const Geo &g) { return (int)(((long long)g.gx * g.gy * g.gz + ADJ_NT - 1) / ADJ_NT); }

// Planes per CTA of the marching kernels: long columns save loads of the planes
// above and below, short ones give a small domain enough CTAs.  A gradient over
// 100 steps of 128^3 in FP64: 13.9, 11.6, 10.6, 10.8 and 10.7 ms with 1, 2, 4, 6
// and 11 planes (16: a fifth slower); over 40 steps of 57 x 63 x 49 in FP32:
// 0.79, 0.76, 0.89, 1.00 and 1.41 ms.  More where a grid would have over 65,535
// layers of them.
static int adj_zc(const Geo &g)
{
    const long long tiles = (long long)((g.gx + ADX - 1) / ADX) * ((g.gy + ADY - 1) / ADY);
    const long long zc = tiles * g.gz / (148 * 3);
    const int least = (g.gz + 65534) / 65535;
    return std::max(least, (int)(zc < 1 ? 1 : (zc > 6 ? 6 : zc)));
}

static dim3 adj_grid(const Geo &g, int zc)
{
    return dim3((g.gx + ADX - 1) / ADX, (g.gy + ADY - 1) / ADY, (g.gz + zc - 1) / zc);
}

int adj_nblocks(const Geo &g)
{
    const dim3 d = adj_grid(g, adj_zc(g));
    const int n = (int)(d.x * d.y * d.z);
    return n > adj_blocks(g) ? n : adj_blocks(g);
}

template <typename Real>
static void replay_t(const Geo &g, const Phys &p, const void *const x0[3], void *const x1[3],
                     const unsigned char *flags, const double *curv, unsigned long long ts, cudaStream_t st)
{
    const int zc = adj_zc(g);
    k_replay<Real><<<adj_grid(g, zc), dim3(ADX, ADY), 0, st>>>(
        g, p, zc, (const Real *)x0[0], (const Real *)x0[1], (const Real *)x0[2], (Real *)x1[0], (Real *)x1[1],
        (Real *)x1[2], flags, curv, ts);
}

int launch_replay(const Geo &g, const Phys &p, int precision, const void *const x0[3], void *const x1[3],
                  const unsigned char *flags, const double *curv, unsigned long long ts, void *stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (precision == MMS_PREC_F32) replay_t<float>(g, p, x0, x1, flags, curv, ts, st);
    else replay_t<double>(g, p, x0, x1, flags, curv, ts, st);
    return 1;
}

template <typename Real>
static void adj_step_t(const Geo &g, const Phys &p, const void *const x0[3], const void *ce1,
                       const unsigned char *flags, const double *curv, const void *const l1[3], void *const l0[3],
                       double *partial, unsigned long long ts, cudaStream_t st)
{
    const int zc = adj_zc(g);
    k_adj_step<Real><<<adj_grid(g, zc), dim3(ADX, ADY), 0, st>>>(
        g, p, zc, flags, curv, (const Real *)x0[0], (const Real *)x0[1], (const Real *)x0[2], (const Real *)ce1,
        (const Real *)l1[0], (const Real *)l1[1], (const Real *)l1[2], (Real *)l0[0], (Real *)l0[1], (Real *)l0[2],
        partial, ts);
}

int launch_adj_step(const Geo &g, const Phys &p, int precision, const void *const x0[3], const void *ce1,
                    const unsigned char *flags, const double *curv, const void *const l1[3], void *const l0[3],
                    double *partial, unsigned long long ts, void *stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    if (precision == MMS_PREC_F32) adj_step_t<float>(g, p, x0, ce1, flags, curv, l1, l0, partial, ts, st);
    else adj_step_t<double>(g, p, x0, ce1, flags, curv, l1, l0, partial, ts, st);
    return 1;
}

int launch_adj_fold(const Geo &g, const double *partial, double *grad, void *stream)
{
    const dim3 d = adj_grid(g, adj_zc(g));
    k_adj_fold<<<1, dim3(32, AS_COUNT), 0, (cudaStream_t)stream>>>(partial, (int)(d.x * d.y * d.z), grad);
    return 1;
}

int launch_adj_terminal(const Geo &g, int precision, double cinit_off, const void *ce, const double *target,
                        void *lce, void *lcl, void *lfs, double *partial, double *loss_out, void *stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    const int nb = adj_blocks(g);  // (no more than adj_nblocks)
    if (precision == MMS_PREC_F32)
        k_adj_terminal<float><<<nb, ADJ_NT, 0, st>>>(g, cinit_off, (const float *)ce, target, (float *)lce,
                                                      (float *)lcl, (float *)lfs, partial);
    else
        k_adj_terminal<double><<<nb, ADJ_NT, 0, st>>>(g, cinit_off, (const double *)ce, target, (double *)lce,
                                                       (double *)lcl, (double *)lfs, partial);
    k_sum_partials<<<1, 256, 0, st>>>(partial, nb, loss_out);
    return 2;
}

}  // namespace mms
