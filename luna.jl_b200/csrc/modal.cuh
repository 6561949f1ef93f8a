// Modal transform (TransModal with full=false, NonlinearRHS.jl:148-302) on the device.
//
// The reference evaluates, per transverse point r of a p-adaptive Clenshaw-Curtis rule on
// (0, a) (Cubature.pcubature_v, NonlinearRHS.jl:294-298):
//   Erω = Emω Ems(r) -> irfft -> responses -> towin -> rfft -> crop -> ωwin -> norm!
//   -> Prω Ems(r)^T, times 2πr,
// and sums the points with the rule's weights, doubling the rule until the L2 difference
// from the previous rule meets the tolerance. Everything between the two mode products is
// linear except the responses, and the mode products act on the mode index only, so the
// sum over points moves to the time samples:
//   E_m(t)  = irfft(pad Emω[:, m])                          time kernel, one CTA per mode
//   g_s,m(t) = sum_p Ems[s][m][p] towin P_p(sum_m' Ems[s][m'][p] E_m'(t))
//                                                           node kernel, per new node s
//   X_l,m   = rfft(sum_s W[l][s] g_s,m)                     level kernel, one CTA per mode
// with W[l][s] the level-l weight of node s (2πr and the half-width included). Each level
// costs one forward transform per mode instead of two transforms per point. The level
// kernel compares X_l (times the output factor crop ωwin norm!) with the previous level,
// and the last of its CTAs decides whether the cubature has converged; the kernels of the
// remaining levels then return at once. X of the last level taken is left in B for the
// store kernel of the column solver (radial.cuh), which applies the output factor.
//
// Time samples are kept in the buffer order of the block transforms (slot i of a buffer
// holds the sample pair n with Swz(split_pos(n)) == i), the same in every kernel, so node
// and level sums are plain element-wise loops over the buffers.
#pragma once
#include "dist.cuh"
#include "radial.cuh"

namespace luna {

#define MODAL_MAX_MODES 16
#define MODAL_MAX_LEVELS 9

struct ModalState {
    int done;         // the cubature of the current right-hand side has ended
    int nevals;       // integrand evaluations it took (2^(l+1) + 1 at level l)
    unsigned ticket;  // level-kernel CTAs that have finished the current level
    int pad;
    double err;       // L2 error estimate of the last level
    double part[2 * MODAL_MAX_MODES];  // per mode: sum |F_l - F_{l-1}|^2, sum |F_l|^2
    double part1[2 * MODAL_MAX_MODES]; // the same of the odd levels (modal_dist_kernel)
};

struct ModalArgs {
    int nmodes, npol, nslots, lmax, P;
    int Mt;                 // complex samples of a time buffer: No/2 pairs (real grid), No (envelope)
    const double* ems;      // [nslots][nmodes][npol] normalised mode fields at the nodes
    const double* wts;      // [lmax + 1][nslots] node weights of each level's rule
    double wlow;            // weight of node 0 in the midpoint rule (level 0's comparison)
    double rtol, atol;      // pcubature reltol / abstol on the L2 norm
    double kerr;            // sum of the Kerr coefficients (vector Kerr)
    const double2* outfac;  // [nmodes * Nw] crop * ωwin * norm!
    void* Et;               // [nmodes][M] field samples per mode (buffer order)
    void* G;                // [nslots][nmodes][M] projected polarisation per node
    ModalState* ms;
    const RadState* st;     // loop state of a solve (null for a plain evaluation)
    unsigned spin;          // rounds after which a cluster stops waiting for the others
};

__device__ __forceinline__ bool modal_skip(const ModalArgs& a) {
    return (a.st && a.st->finished) || a.ms->done;
}

// E_m(t) for every mode: to_time! of column m of the stage input A.
template <typename Rl>
__global__ void __launch_bounds__(LUNA_BLOCK, 1)
modal_time_kernel(const LunaInst* inst, const cpx<Rl>* A, ModalArgs a, TwTab<Rl> tw, int smem_bytes,
                  char* gscr, size_t gstride) {
    char* const smem = dsm;
    if (a.st && a.st->finished) return;
    __shared__ LunaInst sI;
    tws_fill(tw);
    const LunaInst& I = local_inst<Rl>(inst, &sI);
    const int c = blockIdx.x;
    if (c == 0 && threadIdx.x == 0) {
        a.ms->done = 0;
        a.ms->ticket = 0;
    }
    Ws<Rl> w;
    plan_ws<Rl>(I, smem, smem_bytes, w, tw, gscr ? gscr + (size_t)c * gstride : nullptr);
    const int M = I.No / 2, Mt = a.Mt;
    const cpx<Rl>* E = A + (size_t)c * I.Nw;
    int P;
    auto ld = [&](int k) { return cvt<double>(E[k]); };
    // envelope grids: to_time! with copy_scale_both! (NonlinearRHS.jl:16-32), No complex samples
    cpx<Rl>* x = (I.kind == 1) ? env_to_time<Rl>(I, w, ld, &P) : c2r_to_time<Rl>(w, M, I.Nw, ld, &P);
    cpx<Rl>* out = reinterpret_cast<cpx<Rl>*>(a.Et) + (size_t)c * Mt;
    for (int i = threadIdx.x; i < Mt; i += LUNA_BLOCK) out[i] = x[i];
}

// One polarisation component: one CTA per new node. The point's field is built in the
// CTA's transform buffer and the responses of the mode-averaged kernel (Kerr, plasma) and
// the time window are applied in place; the result times each mode's field at the node
// goes to G.
template <typename Rl>
__global__ void __launch_bounds__(LUNA_BLOCK, 1)
modal_node_kernel(const LunaInst* inst, ModalArgs a, int slot0, TwTab<Rl> tw, int smem_bytes, char* gscr,
                  size_t gstride, int* flags) {
    char* const smem = dsm;
    if (modal_skip(a)) return;
    __shared__ LunaInst sI;
    tws_fill(tw);
    const LunaInst& I = local_inst<Rl>(inst, &sI);
    const int slot = slot0 + blockIdx.x;
    Ws<Rl> w;
    plan_ws<Rl>(I, smem, smem_bytes, w, tw, gscr ? gscr + (size_t)blockIdx.x * gstride : nullptr);
    if (threadIdx.x == 0) *w.flag = 0;
    const int M = a.Mt, nm = a.nmodes;
    const int P = buf_split<Rl>(w.main_alt, M);
    const double* e = a.ems + (size_t)slot * nm;
    const cpx<Rl>* Et = reinterpret_cast<const cpx<Rl>*>(a.Et);
    cpx<Rl>* x = w.main;
    for (int i = threadIdx.x; i < M; i += LUNA_BLOCK) {
        double sx = 0, sy = 0;
        for (int m = 0; m < nm; ++m) {
            const cpx<Rl> v = Et[(size_t)m * M + i];
            sx += e[m] * (double)v.x;
            sy += e[m] * (double)v.y;
        }
        x[i] = mk<Rl>((Rl)sx, (Rl)sy);
    }
    __syncthreads();
    if (I.kind == 1) pointwise_env<Rl>(I, w, x, P, I.in_scale);  // Kerr_env(_thg), RamanPolarEnv
    else pointwise_real<Rl>(I, w, x, M, P, I.in_scale);
    cpx<Rl>* G = reinterpret_cast<cpx<Rl>*>(a.G) + (size_t)slot * nm * M;
    for (int m = 0; m < nm; ++m) {
        const double em = e[m];
        for (int i = threadIdx.x; i < M; i += LUNA_BLOCK) {
            const cpx<Rl> v = x[i];
            G[(size_t)m * M + i] = mk<Rl>((Rl)(em * (double)v.x), (Rl)(em * (double)v.y));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && *w.flag && flags) atomicOr(flags, *w.flag);
}

// Two polarisation components, Kerr only (KerrVector!, Nonlinear.jl:12-21): element-wise,
// so each new node is spread over gridDim.y CTAs.
template <typename Rl>
__global__ void __launch_bounds__(256) modal_kerr2_kernel(const LunaInst* inst, ModalArgs a, int slot0) {
    if (modal_skip(a)) return;
    const LunaInst& I = *inst;
    const int slot = slot0 + blockIdx.x;
    const int M = a.Mt, nm = a.nmodes, P = a.P, Lb = M / P;
    const double* e = a.ems + (size_t)slot * nm * 2;
    const cpx<Rl>* Et = reinterpret_cast<const cpx<Rl>*>(a.Et);
    cpx<Rl>* G = reinterpret_cast<cpx<Rl>*>(a.G) + (size_t)slot * nm * M;
    const double sc = I.in_scale, kc = a.kerr;
    if (I.kind == 1) {
        // KerrVectorEnv! (Nonlinear.jl:52-63): slot i holds the complex sample n
        for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < M; i += gridDim.y * blockDim.x) {
            const int sp = Swz<Rl>::f(i);
            const int n = (sp % Lb) * P + sp / Lb;
            cpx<double> ex = mk<double>(0, 0), ey = mk<double>(0, 0);
            for (int m = 0; m < nm; ++m) {
                const cpx<double> v = cvt<double>(Et[(size_t)m * M + i]);
                ex = ex + scale(e[2 * m], v);
                ey = ey + scale(e[2 * m + 1], v);
            }
            ex = scale(sc, ex);
            ey = scale(sc, ey);
            const double ax = abs2(ex), ay = abs2(ey), f = 0.75 * kc, tw = __ldg(I.towin + n);
            const cpx<double> px = scale(f, scale(ax + 2.0 / 3 * ay, ex) + scale(1.0 / 3, conj(ex) * (ey * ey)));
            const cpx<double> py = scale(f, scale(ay + 2.0 / 3 * ax, ey) + scale(1.0 / 3, conj(ey) * (ex * ex)));
            for (int m = 0; m < nm; ++m)
                G[(size_t)m * M + i] = cvt<Rl>(scale(tw, scale(e[2 * m], px) + scale(e[2 * m + 1], py)));
        }
        return;
    }
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < M; i += gridDim.y * blockDim.x) {
        const int sp = Swz<Rl>::f(i);            // the swizzle is its own inverse
        const int n = (sp % Lb) * P + sp / Lb;   // inverse of split_pos
        double ex0 = 0, ey0 = 0, ex1 = 0, ey1 = 0;
        for (int m = 0; m < nm; ++m) {
            const cpx<Rl> v = Et[(size_t)m * M + i];
            const double fx = e[2 * m], fy = e[2 * m + 1];
            ex0 += fx * (double)v.x;
            ey0 += fy * (double)v.x;
            ex1 += fx * (double)v.y;
            ey1 += fy * (double)v.y;
        }
        ex0 *= sc;
        ey0 *= sc;
        ex1 *= sc;
        ey1 *= sc;
        const double tw0 = __ldg(I.towin + 2 * n), tw1 = __ldg(I.towin + 2 * n + 1);
        const double f0 = kc * (ex0 * ex0 + ey0 * ey0), f1 = kc * (ex1 * ex1 + ey1 * ey1);
        const double px0 = f0 * ex0 * tw0, py0 = f0 * ey0 * tw0;
        const double px1 = f1 * ex1 * tw1, py1 = f1 * ey1 * tw1;
        for (int m = 0; m < nm; ++m) {
            const double fx = e[2 * m], fy = e[2 * m + 1];
            G[(size_t)m * M + i] = mk<Rl>((Rl)(fx * px0 + fy * py0), (Rl)(fx * px1 + fy * py1));
        }
    }
}

// Exclusive prefix of v over the CTA's threads (thread order) and the total; sh holds
// LUNA_WARPS doubles.
__device__ __forceinline__ double cta_exscan(double v, double* sh, double& total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    double x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        double t = (lane < LUNA_WARPS) ? sh[lane] : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < LUNA_WARPS) sh[lane] = t;
    }
    __syncthreads();
    const double base = wid ? sh[wid - 1] : 0.0;
    total = sh[LUNA_WARPS - 1];
    __syncthreads();
    return base + x - v;
}

// Maths.cumtrapz! (Maths.jl:323-328) of v[0..n) on one CTA, written as the prefix sum
// out[j] = dt (S_j - (v_0 + v_j)/2), S_j = v_0 + ... + v_j, each thread a contiguous run.
__device__ __forceinline__ void cta_cumtrapz(const double* v, double* out, int n, double dt, double* sh) {
    const int C = (n + LUNA_BLOCK - 1) / LUNA_BLOCK;
    const int b = threadIdx.x * C, e = min(n, b + C);
    const double v0 = v[0];  // read before the scan's barriers: out may alias v
    double s = 0;
    for (int j = b; j < e; ++j) s += v[j];
    double tot;
    double pre = cta_exscan(s, sh, tot);
    for (int j = b; j < e; ++j) {
        pre += v[j];
        out[j] = dt * (pre - 0.5 * (v0 + v[j]));
    }
    __syncthreads();
}

// Two polarisation components with the plasma response (PlasmaVector!, Nonlinear.jl:144-162)
// and vector Kerr (KerrVector!, Nonlinear.jl:12-21): one CTA per new node. The node's field
// (Ex, Ey) in natural time order, the rate of |E| = hypot(Ex, Ey) and the ionisation fraction,
// the phase integrands and currents of both components, their cumulative integrals, then
// the polarisation times the time window projected on each mode's field at the node.
// Scratch: 6 No doubles per CTA in global memory (vs).
template <typename Rl>
__global__ void __launch_bounds__(LUNA_BLOCK, 1)
modal_vec_kernel(const LunaInst* inst, ModalArgs a, int slot0, double* vscr, int* flags) {
    __shared__ double sh[LUNA_WARPS];
    __shared__ int flag;
    if (modal_skip(a)) return;
    const LunaInst& I = *inst;
    const int slot = slot0 + blockIdx.x;
    const int M = I.No / 2, No = I.No, nm = a.nmodes, P = a.P, Lb = M / P;
    const int tid = threadIdx.x;
    if (tid == 0) flag = 0;
    int ip = -1;
    for (int i = 0; i < I.nresp; ++i)
        if (I.resp[i].kind == LUNA_RESP_PLASMA_PPT || I.resp[i].kind == LUNA_RESP_PLASMA_ADK) ip = i;
    const LunaResp& r = I.resp[ip];
    const double* e = a.ems + (size_t)slot * nm * 2;
    const cpx<Rl>* Et = reinterpret_cast<const cpx<Rl>*>(a.Et);
    cpx<Rl>* G = reinterpret_cast<cpx<Rl>*>(a.G) + (size_t)slot * nm * M;
    double* ex = vscr + (size_t)blockIdx.x * 6 * No;
    double* ey = ex + No;
    double* rt = ey + No;   // rate, then Px
    double* fr = rt + No;   // cumulative rate, the fraction, then Py
    double* jx = fr + No;   // phase integrand and current, x
    double* jy = jx + No;   // phase integrand and current, y
    const double sc = I.in_scale, kc = a.kerr, dt = r.dt;
    __syncthreads();
    // the node's field in natural order (buffer slot i holds the sample pair n)
    for (int i = tid; i < M; i += LUNA_BLOCK) {
        const int sp = Swz<Rl>::f(i);
        const int n = (sp % Lb) * P + sp / Lb;
        double x0 = 0, y0 = 0, x1 = 0, y1 = 0;
        for (int m = 0; m < nm; ++m) {
            const cpx<Rl> v = Et[(size_t)m * M + i];
            const double fx = e[2 * m], fy = e[2 * m + 1];
            x0 += fx * (double)v.x;
            y0 += fy * (double)v.x;
            x1 += fx * (double)v.y;
            y1 += fy * (double)v.y;
        }
        ex[2 * n] = x0 * sc;
        ey[2 * n] = y0 * sc;
        ex[2 * n + 1] = x1 * sc;
        ey[2 * n + 1] = y1 * sc;
    }
    __syncthreads();
    for (int j = tid; j < No; j += LUNA_BLOCK) {
        const double Em = hypot(ex[j], ey[j]);
        rt[j] = (r.kind == LUNA_RESP_PLASMA_PPT) ? ppt_rate<double>(r, Em, &flag) : adk_rate<double>(r, Em);
    }
    __syncthreads();
    cta_cumtrapz(rt, fr, No, dt, sh);
    for (int j = tid; j < No; j += LUNA_BLOCK) {
        const double f = r.preion + 1.0 - exp(-fr[j]);
        fr[j] = f;
        jx[j] = f * r.eratio * ex[j];
        jy[j] = f * r.eratio * ey[j];
    }
    __syncthreads();
    // J = cumtrapz(phase) + ionpot rate (1 - fraction)/|E|^2 E per component, in place
    cta_cumtrapz(jx, jx, No, dt, sh);
    cta_cumtrapz(jy, jy, No, dt, sh);
    for (int j = tid; j < No; j += LUNA_BLOCK) {
        const double Em = hypot(ex[j], ey[j]);
        const double f = fr[j];
        if (fabs(Em) > 0) {
            const double pre = r.ionpot * rt[j] * (1.0 - f) / (Em * Em);
            jx[j] += pre * ex[j];
            jy[j] += pre * ey[j];
        }
    }
    __syncthreads();
    cta_cumtrapz(jx, rt, No, dt, sh);  // Px (the rates are no longer needed)
    cta_cumtrapz(jy, fr, No, dt, sh);  // Py
    const double coef = r.coef;
    for (int i = tid; i < M; i += LUNA_BLOCK) {
        const int sp = Swz<Rl>::f(i);
        const int n = (sp % Lb) * P + sp / Lb;
        double pxy[2][2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = 2 * n + h;
            const double Ex = ex[j], Ey = ey[j];
            const double fk = kc * (Ex * Ex + Ey * Ey);
            const double tw = __ldg(I.towin + j);
            pxy[h][0] = (fk * Ex + coef * rt[j]) * tw;
            pxy[h][1] = (fk * Ey + coef * fr[j]) * tw;
        }
        for (int m = 0; m < nm; ++m) {
            const double fx = e[2 * m], fy = e[2 * m + 1];
            G[(size_t)m * M + i] = mk<Rl>((Rl)(fx * pxy[0][0] + fy * pxy[0][1]), (Rl)(fx * pxy[1][0] + fy * pxy[1][1]));
        }
    }
    __syncthreads();
    if (tid == 0 && flag && flags) atomicOr(flags, flag);
}

// Level l of the rule for mode c: X_l = rfft(sum_s W[l][s] g_s,c) into B (level 0 first
// puts the midpoint rule there), the two L2 sums against the previous level, and the
// convergence decision by the last CTA to finish (Cubature's L2 error norm).
template <typename Rl>
__global__ void __launch_bounds__(LUNA_BLOCK, 1)
modal_level_kernel(const LunaInst* inst, ModalArgs a, int l, cpx<Rl>* B, TwTab<Rl> tw, int smem_bytes,
                   char* gscr, size_t gstride) {
    char* const smem = dsm;
    if (modal_skip(a)) return;
    __shared__ LunaInst sI;
    tws_fill(tw);
    const LunaInst& I = local_inst<Rl>(inst, &sI);
    const int c = blockIdx.x;
    Ws<Rl> w;
    plan_ws<Rl>(I, smem, smem_bytes, w, tw, gscr ? gscr + (size_t)c * gstride : nullptr);
    const int M = a.Mt, Nw = I.Nw, nm = a.nmodes;
    const int ns = (2 << l) - 1;  // interior nodes of level l
    const double* wl = a.wts + (size_t)l * a.nslots;
    const cpx<Rl>* G = reinterpret_cast<const cpx<Rl>*>(a.G);
    cpx<Rl>* Bc = B + (size_t)c * Nw;
    const cpx<double>* of = reinterpret_cast<const cpx<double>*>(a.outfac) + (size_t)c * Nw;
    double se = 0, sv = 0;
    for (int pass = (l == 0) ? 0 : 1; pass < 2; ++pass) {
        cpx<Rl>* x = w.main;
        for (int i = threadIdx.x; i < M; i += LUNA_BLOCK) {
            double sx = 0, sy = 0;
            if (pass == 0) {
                const cpx<Rl> v = G[(size_t)c * M + i];
                sx = a.wlow * (double)v.x;
                sy = a.wlow * (double)v.y;
            } else {
                for (int s = 0; s < ns; ++s) {
                    const double ws = wl[s];
                    const cpx<Rl> v = G[((size_t)s * nm + c) * M + i];
                    sx += ws * (double)v.x;
                    sy += ws * (double)v.y;
                }
            }
            x[i] = mk<Rl>((Rl)sx, (Rl)sy);
        }
        __syncthreads();
        const bool cmp = pass == 1;
        auto st = [&](int k, cpx<double> X) {
            if (cmp) {
                const cpx<double> o = ldg(of + k);
                se += abs2((X - cvt<double>(Bc[k])) * o);
                sv += abs2(X * o);
            }
            Bc[k] = cvt<Rl>(X);
        };
        if (I.kind == 1) env_to_freq<Rl>(I, w, x, st);
        else r2c_to_freq<Rl>(w, x, M, Nw, st);
    }
    double unused = 0;
    block_sum3(se, sv, unused, w.red);
    if (threadIdx.x == 0) {
        ModalState* ms = a.ms;
        ms->part[2 * c] = se;
        ms->part[2 * c + 1] = sv;
        __threadfence();
        const unsigned tk = atomicAdd(&ms->ticket, 1u);
        if (tk == (unsigned)nm - 1) {
            __threadfence();
            const volatile double* pp = ms->part;
            double e2 = 0, v2 = 0;
            for (int m = 0; m < nm; ++m) {
                e2 += pp[2 * m];
                v2 += pp[2 * m + 1];
            }
            const double err = sqrt(e2), val = sqrt(v2);
            ms->err = err;
            ms->nevals = (2 << l) + 1;
            if (err <= a.atol || err <= a.rtol * val || l >= a.lmax) ms->done = 1;
            ms->ticket = 0;
        }
    }
}

// ------------------------------------------------------------------ one launch on clusters (FP64)
// The whole transform in one launch, for time buffers from 2048 samples: clusters of R CTAs
// (the largest of 16, 8 and 4 that leaves 512 samples a CTA) take a mode's or a node's
// time samples together, as a distributed right-hand side does (dist.cuh). Time samples are in natural
// order, CTA q holding the block q. The kernels above run one CTA a mode, 17 to 19 launches of which
// those after convergence do nothing: at No = 16384 with one mode and 15 nodes 25 us for the field,
// 31 us for each level's nodes and 56 to 100 us for its integral, 332 us in all; 72 us here. Bound by the
// chain of one transform per level (16 k cycles each) and the exchange of its L2 sums.
//
// elem (Kerr responses alone): the integrand is local in time, so each level's sum over its nodes
// is evaluated in registers from the mode fields, without G; nothing but the convergence
// test crosses modes, and one mode needs a single cluster. Otherwise clusters take the new nodes of a
// level, leave the projections in G, and after a grid barrier sum them per mode. Several clusters are
// a cooperative launch: all are resident, and modal_gsync bounds its wait besides.
struct ModalBar {
    unsigned count, gen;
};

// Barrier of all clusters of the grid (C = 1: of the cluster). False when the wait of `spin` rounds ran
// out; every thread of a cluster returns the same.
template <int R>
__device__ __forceinline__ bool modal_gsync(DWs<double>& d, ModalBar* bar, int C, unsigned spin) {
    dsync();
    if (C == 1) return true;
    if (d.rank == 0 && threadIdx.x == 0) {
        volatile unsigned* vg = &bar->gen;
        const unsigned g = *vg;
        bool ok = true;
        __threadfence();
        if (atomicAdd(&bar->count, 1u) == (unsigned)C - 1) {
            bar->count = 0;
            __threadfence();
            *vg = g + 1;
        } else {
            unsigned n = 0;
            if (spin)
                while (*vg == g && ++n < spin) __nanosleep(20);
            ok = n < spin;
        }
        __threadfence();
        d.xs[15] = ok ? 1.0 : 0.0;
    }
    dsync();
    return *drem(&d.xs[15], 0) != 0.0;
}

// Polarisation of one slot of a node times e_c, Kerr responses only, without the time window: a
// sample pair of two components, or a complex envelope sample of one or two; the expressions of modal_node_kernel
// and modal_kerr2_kernel. f holds the components of the node's field.
__device__ __forceinline__ cpx<double> modal_kerr(const LunaInst& I, int npol, double kc, int n, cpx<double> fx,
                                                  cpx<double> fy, double ex, double ey) {
    if (I.kind == 0) {
        const double k0 = kc * (fx.x * fx.x + fy.x * fy.x), k1 = kc * (fx.y * fx.y + fy.y * fy.y);
        return mk<double>(ex * (k0 * fx.x) + ey * (k0 * fy.x), ex * (k1 * fx.y) + ey * (k1 * fy.y));
    }
    if (npol == 1) {
        cpx<double> P = mk<double>(0, 0);
        for (int i = 0; i < I.nresp; ++i) {
            const LunaResp& r = I.resp[i];
            if (r.cthg) {
                const cpx<double> C = ldg(reinterpret_cast<const cpx<double>*>(r.cthg) + n);
                P = P + scale(0.25 * r.coef, scale(3.0 * abs2(fx), fx) + C * (fx * fx) * fx);
            } else {
                P = P + scale(0.75 * r.coef * abs2(fx), fx);
            }
        }
        return scale(ex, P);
    }
    const double ax = abs2(fx), ay = abs2(fy), f = 0.75 * kc;
    const cpx<double> px = scale(f, scale(ax + 2.0 / 3 * ay, fx) + scale(1.0 / 3, conj(fx) * (fy * fy)));
    const cpx<double> py = scale(f, scale(ay + 2.0 / 3 * ax, fy) + scale(1.0 / 3, conj(fy) * (fx * fx)));
    return scale(ex, px) + scale(ey, py);
}

template <int R>
__global__ void __launch_bounds__(LUNA_BLOCK, 1)
modal_dist_kernel(const LunaInst* inst, const double2* A, ModalArgs a, double2* B, double2* dst, int elem,
                  TwTab<double> tw, int* flags, ModalBar* bar) {
    if (a.st && a.st->finished) return;
    __shared__ LunaInst sI;
    __shared__ int s_done;
    tws_fill(tw);
    const LunaInst& I = local_inst<double>(inst, &sI);
    DWs<double> d;
    plan_dws<double, R>(I, dsm, d, tw, (int)cooperative_groups::this_cluster().block_rank());
    const int tid = threadIdx.x, T = LUNA_BLOCK, p = d.rank;
    const int C = gridDim.x / R, cl = blockIdx.x / R;
    const int Mt = a.Mt, Mb = Mt / R, base = p * Mb, nm = a.nmodes, np = a.npol, Nw = I.Nw;
    const int No = I.No, N = I.N, h = I.N / 2;  // envelope grids: copy_scale_both! padding and cropping
    const double sc = I.in_scale;
    cpx<double>* Et = reinterpret_cast<cpx<double>*>(a.Et);
    cpx<double>* G = reinterpret_cast<cpx<double>*>(a.G);
    if (tid == 0) *d.flag = 0;
    dsync();  // every CTA of the cluster has started before its shared memory is addressed
    for (int m = cl; m < nm; m += C) {
        const cpx<double>* E = reinterpret_cast<const cpx<double>*>(A) + (size_t)m * Nw;
        if (I.kind == 1)
            dist_c2c_inv<R>(d, No, [&](int j) { return j < h ? E[j] : j >= No - h ? E[j - No + N] : mk<double>(0, 0); });
        else
            dist_c2r<double, R>(d, No / 2, Nw, [&](int k) { return E[k]; });
        for (int n = tid; n < Mb; n += T) Et[(size_t)m * Mt + base + n] = d.tb[Swz<double>::f(n)];
    }
    bool ok = modal_gsync<R>(d, bar, C, a.spin);
    for (int l = 0; ok; ++l) {
        const int ns = (2 << l) - 1;  // interior nodes of level l
        if (!elem) {
            const int s0 = (l == 0) ? 0 : (1 << l) - 1, nn = (l == 0) ? 1 : (1 << l);
            for (int s = s0 + cl; s < s0 + nn; s += C) {
                const double* e = a.ems + (size_t)s * nm;
                for (int n = tid; n < Mb; n += T) {
                    cpx<double> f = mk<double>(0, 0);
                    for (int m = 0; m < nm; ++m) f = f + scale(__ldg(e + m), Et[(size_t)m * Mt + base + n]);
                    d.tb[Swz<double>::f(n)] = f;
                }
                __syncthreads();
                if (I.kind == 1) dist_pointwise_env<R>(I, d, sc);
                else dist_pointwise<double, R>(I, d, Mt, sc);
                for (int n = tid; n < Mb; n += T) {
                    const cpx<double> v = d.tb[Swz<double>::f(n)];
                    for (int m = 0; m < nm; ++m) G[((size_t)s * nm + m) * Mt + base + n] = scale(__ldg(e + m), v);
                }
                dsync();  // the blocks may be written again
            }
            if (!(ok = modal_gsync<R>(d, bar, C, a.spin))) break;
        }
        const double* wl = a.wts + (size_t)l * a.nslots;
        // level 0 has one node: one transform gives its rule and the midpoint rule's value
        const double w0 = l == 0 ? 1.0 : 0.0, wa = l == 0 ? a.wlow : 0.0, wb = l == 0 ? __ldg(wl) : 1.0;
        ModalState* ms = a.ms;
        double* part = (l & 1) ? ms->part1 : ms->part;
        double e2 = 0, v2 = 0;
        for (int c = cl; c < nm; c += C) {
            for (int n = tid; n < Mb; n += T) {
                cpx<double> x = mk<double>(0, 0);
                if (elem) {
                    cpx<double> v[4];
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (m < nm) v[m] = Et[(size_t)m * Mt + base + n];
                    if (I.kind == 0 && np == 1) {  // the cubes of the field, the factors after the sum
#pragma unroll 4
                        for (int s = 0; s < ns; ++s) {
                            const double* e = a.ems + (size_t)s * nm;
                            cpx<double> f = mk<double>(0, 0);
#pragma unroll
                            for (int m = 0; m < 4; ++m)
                                if (m < nm) f = f + scale(__ldg(e + m), v[m]);
                            for (int m = 4; m < nm; ++m) f = f + scale(__ldg(e + m), Et[(size_t)m * Mt + base + n]);
                            const double we = (l == 0 ? w0 : __ldg(wl + s)) * __ldg(e + c);
                            x = x + scale(we, mk<double>(f.x * f.x * f.x, f.y * f.y * f.y));
                        }
                        x = scale(a.kerr * (sc * sc * sc), x);
                    } else {
                    for (int s = 0; s < ns; ++s) {
                        const double* e = a.ems + (size_t)s * nm * np;
                        cpx<double> fx = mk<double>(0, 0), fy = fx;
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            if (m >= nm) break;
                            fx = fx + scale(__ldg(e + m * np), v[m]);
                            if (np == 2) fy = fy + scale(__ldg(e + m * np + 1), v[m]);
                        }
                        for (int m = 4; m < nm; ++m) {
                            const cpx<double> u = Et[(size_t)m * Mt + base + n];
                            fx = fx + scale(__ldg(e + m * np), u);
                            if (np == 2) fy = fy + scale(__ldg(e + m * np + 1), u);
                        }
                        const double ey = np == 2 ? __ldg(e + c * np + 1) : 0.0;
                        const cpx<double> P = modal_kerr(I, np, a.kerr, base + n, scale(sc, fx), scale(sc, fy), __ldg(e + c * np), ey);
                        x = x + scale(l == 0 ? w0 : __ldg(wl + s), P);
                    }
                    }
                    if (I.kind == 1) {
                        x = scale(__ldg(I.towin + base + n), x);
                    } else {
                        const double2 t = __ldg(reinterpret_cast<const double2*>(I.towin) + base + n);
                        x = mk<double>(x.x * t.x, x.y * t.y);
                    }
                } else {
#pragma unroll 4
                    for (int s = 0; s < ns; ++s)
                        x = x + scale(l == 0 ? w0 : __ldg(wl + s), G[((size_t)s * nm + c) * Mt + base + n]);
                }
                d.tb[Swz<double>::f(n)] = x;
            }
            cpx<double>* Bc = reinterpret_cast<cpx<double>*>(B) + (size_t)c * Nw;
            const cpx<double>* of = reinterpret_cast<const cpx<double>*>(a.outfac) + (size_t)c * Nw;
            double se = 0, sv = 0;
            auto st = [&](int k, cpx<double> X) {
                const cpx<double> o = ldg(of + k), last = l == 0 ? scale(wa, X) : Bc[k];
                X = scale(wb, X);
                se += abs2((X - last) * o);
                sv += abs2(X * o);
                Bc[k] = X;
            };
            if (I.kind == 1)
                dist_c2c_fwd<R>(d, No, [&](int j, cpx<double> X) { if (j < h || j >= No - h) st(j < h ? j : j - No + N, X); });
            else
                dist_r2c<double, R>(d, Mt, Nw, st);
            double unused = 0;
            block_sum3(se, sv, unused, d.red);
            if (tid == 0) {
                d.xs[8] = se;
                d.xs[9] = sv;
            }
            dsync();
            if (tid < 32 && (C == 1 || p == 0)) {  // one cluster: every CTA adds the cluster's sums
                double x = tid < R ? drem(d.xs, tid)[8] : 0.0, y = tid < R ? drem(d.xs, tid)[9] : 0.0;
                x = warp_sum(x);
                y = warp_sum(y);
                e2 += x;
                v2 += y;
                if (C > 1 && tid == 0) {
                    part[2 * c] = x;
                    part[2 * c + 1] = y;
                }
            }
        }
        if (C > 1 && !(ok = modal_gsync<R>(d, bar, C, a.spin))) break;
        if (tid == 0) {  // every CTA adds the same sums in the same order: identical decisions
            if (C > 1) {
                e2 = v2 = 0;
                for (int m = 0; m < nm; ++m) {
                    e2 += __ldcg(part + 2 * m);
                    v2 += __ldcg(part + 2 * m + 1);
                }
            }
            const double err = sqrt(e2), val = sqrt(v2);
            s_done = err <= a.atol || err <= a.rtol * val || l >= a.lmax;
            if (blockIdx.x == 0) {
                ms->err = err;
                ms->nevals = (2 << l) + 1;
            }
        }
        __syncthreads();
        if (s_done) break;
    }
    if (!ok && tid == 0) atomicOr(flags, 1 << ST_WAIT_TIMEOUT);
    if (dst) {  // a cluster whose wait ran out leaves NaN in its modes (a call on a stream has no other answer)
        __syncthreads();
        for (int c = cl; c < nm; c += C)
            for (int k = p + R * tid; k < Nw; k += R * T) {
                const size_t e = (size_t)c * Nw + k;
                const cpx<double> X = reinterpret_cast<const cpx<double>*>(B)[e] * ldg(reinterpret_cast<const cpx<double>*>(a.outfac) + e);
                dst[e] = ok ? make_double2(X.x, X.y) : make_double2(nan(""), nan(""));
            }
    }
    if (tid == 0 && *d.flag) atomicOr(flags, *d.flag);
    dsync();  // no CTA leaves while another may read its shared memory
}

}  // namespace luna
