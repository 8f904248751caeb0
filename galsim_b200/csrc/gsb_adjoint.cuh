// Adjoint of the fused FFT draw (reverse mode), one CTA per stamp.
//
// The forward kernel computes, per stamp, image(x, y) = (1/N^2) sum_c w_c Re(sum_r X(c, r)
// e^{+2 pi i (c x + r y) / N}) over the Hermitian half plane c = 0..N/2 (w_c = 1 for c = 0 and
// N/2, else 2), where X is the wrapped k-image: the program summed over the aliases of (c, r)
// inside the Nk x Nk evaluation grid.  For a loss L with image cotangent G = dL/dimage,
//     dL = sum_{c,r} (w_c / N^2) Re(Ghat(c, r) dX(c, r)),
//     Ghat(c, r) = sum_pixels G(x, y) e^{+2 pi i (c x + r y) / N},
// i.e. Ghat is the forward-sign DFT of the zero-padded cotangent at the pixels' (x mod N,
// y mod N) positions.  The kernel computes Ghat with the same warp Stockham FFTs (rows in
// packed pairs, then columns), then visits every alias exactly as the forward gather does and
// runs the program in reverse at that k-point, accumulating
//   per leaf   d/dflux, d/dA, d/dB, d/dC, d/dD (its Jacobian), d/dn (Sersic index)
//   per phase  d/dcenx, d/dceny, d/dflux_scaling, d/dA..D (the phase's Jacobian)
//   per scale  d/dscale
// The k-grid is recomputed, never stored.
#pragma once

#include "gsb_draw.cuh"
#include "gsb_grad.cuh"

namespace gsb {

constexpr int kGradPerLeaf = 6;
constexpr int kGradPerPhase = 7;
constexpr int kMaxGrad = kGradPerLeaf * GSB_MAX_LEAVES + kGradPerPhase * GSB_MAX_PHASES + GSB_MAX_SCALES;

__host__ __device__ inline int grad_count(const gsb_template& tpl)
{
    return kGradPerLeaf * tpl.n_leaves + kGradPerPhase * tpl.n_phases + tpl.n_scales;
}

struct AdjArgs {
    gsb_template tpl;
    FactorPlan fac;
    int n_stamps;
    const gsb_leaf* leaves;
    const gsb_phase* phases;
    const double* scales;
    const gsb_stamp* stamps;
    const double* sersic_header;
    const double4* sersic_node;
    const double* sersic_dheader;
    const double4* sersic_dnode;
    int sersic_stride;
    const void* cot;      // cotangent images, same layout as the forward output
    int cot_dtype;
    double* grad;         // n_stamps * grad_count(tpl)
    unsigned want;        // records whose gradients are wanted (leaf l: bit l, phase p: 8 + p, scale q: 16 + q)
    void* work;           // per-CTA W slabs when W does not fit in shared memory
};

// Atoms of the factored adjoint held in registers.
constexpr int kAdjAtoms = 3;

struct AdjSmem {
    StampSmem S;
    SersicDnView dn[GSB_MAX_LEAVES];
    int child1[GSB_MAX_OPS];
    int child2[GSB_MAX_OPS];
    double gacc[kMaxGrad];
};

// Operand op indices of every op of the postfix program (thread 0).
__device__ inline void program_children(const gsb_template& tpl, int* c1, int* c2)
{
    int st[GSB_MAX_OPS];
    int sp = 0;
    for (int o = 0; o < tpl.n_ops; ++o) {
        const int code = tpl.op_code[o];
        c1[o] = c2[o] = -1;
        if (code == GSB_OP_LEAF) {
            st[sp++] = o;
        } else if (code == GSB_OP_MUL || code == GSB_OP_ADD) {
            c2[o] = st[--sp];
            c1[o] = st[sp - 1];
            st[sp - 1] = o;
        } else {
            c1[o] = st[sp - 1];
            st[sp - 1] = o;
        }
    }
}

// Reverse-mode pass of the ops [o0, o1) (a complete subtree, or the whole program) at k index
// (i, j) with output cotangent u (contribution Re(u * dF)); gradients are added into acc.
template <typename T, bool II = true>
__device__ __noinline__ void adjoint_range(const gsb_template& tpl, const AdjSmem& A, double dk, int i,
                                           int j, const GridRef& g, Cx<T> u, T* acc, int o0, int o1)
{
    const StampSmem& S = A.S;
    Cx<T> val[GSB_MAX_OPS];
    Cx<T> adj[GSB_MAX_OPS];
    LeafD<T> ld[GSB_MAX_LEAVES];
    Cx<T> pe[GSB_MAX_PHASES];
    const T kx = T(i) * T(dk), ky = T(j) * T(dk);
    const int n_ops = o1;
    for (int o = o0; o < n_ops; ++o) {
        const int code = tpl.op_code[o], arg = tpl.op_arg[o];
        const int a = A.child1[o], b = A.child2[o];
        if (code == GSB_OP_LEAF) {
            if (II && S.leaf[arg].type == GSB_INTERPOLATED) {
                // an image leaf enters with its complex value and no gradient entries of its own
                ld[arg] = LeafD<T>{T(0), T(0), T(0), T(0), T(0)};
                val[o] = ii_kvalue<T>(S.leaf[arg], dk, i, j);
            } else {
                ld[arg] = leaf_grad<T>(S.leaf[arg], S.sersic, A.dn, kx, ky, g, i - g.x0, j - g.y0);
                val[o] = cx<T>(ld[arg].v, T(0));
            }
        } else if (code == GSB_OP_MUL) {
            val[o] = cmul<T>(val[a], val[b]);
        } else if (code == GSB_OP_ADD) {
            val[o] = cadd<T>(val[a], val[b]);
        } else if (code == GSB_OP_PHASE) {
            double tt = i * S.phase_ax[arg] + j * S.phase_ay[arg];
            tt -= rint(tt);
            T sn, cs;
            sincospi(T(-2. * tt), &sn, &cs);
            pe[arg] = cx<T>(cs, sn);
            val[o] = cscale<T>(cmul<T>(val[a], pe[arg]), T(S.phase[arg].flux_scaling));
        } else {
            val[o] = cscale<T>(val[a], T(S.scale[arg]));
        }
        adj[o] = cx<T>(T(0), T(0));
    }
    adj[n_ops - 1] = u;
    const int pbase = kGradPerLeaf * tpl.n_leaves;
    const int sbase = pbase + kGradPerPhase * tpl.n_phases;
    for (int o = n_ops - 1; o >= o0; --o) {
        const int code = tpl.op_code[o], arg = tpl.op_arg[o];
        const int a = A.child1[o], b = A.child2[o];
        const Cx<T> w = adj[o];
        if (code == GSB_OP_LEAF) {
            const LeafD<T>& d = ld[arg];
            const T ar = w.x;
            T* gl = acc + kGradPerLeaf * arg;
            gl[0] += ar * d.unit;
            gl[1] += ar * d.gx * kx;
            gl[2] += ar * d.gy * kx;
            gl[3] += ar * d.gx * ky;
            gl[4] += ar * d.gy * ky;
            gl[5] += ar * d.gn;
        } else if (code == GSB_OP_MUL) {
            adj[a] = cadd<T>(adj[a], cmul<T>(w, val[b]));
            adj[b] = cadd<T>(adj[b], cmul<T>(w, val[a]));
        } else if (code == GSB_OP_ADD) {
            adj[a] = cadd<T>(adj[a], w);
            adj[b] = cadd<T>(adj[b], w);
        } else if (code == GSB_OP_PHASE) {
            const gsb_phase& P = S.phase[arg];
            const T fs = T(P.flux_scaling);
            const Cx<T> e = pe[arg];
            adj[a] = cadd<T>(adj[a], cscale<T>(cmul<T>(w, e), fs));
            const Cx<T> we = cmul<T>(cmul<T>(w, val[a]), e);
            const T z = fs * we.y;                   // dL/dtheta with f = fs exp(-i theta)
            const T cxp = T(P.cenx), cyp = T(P.ceny);
            T* gp = acc + pbase + kGradPerPhase * arg;
            gp[0] += z * (T(P.jac[0]) * kx + T(P.jac[2]) * ky);
            gp[1] += z * (T(P.jac[1]) * kx + T(P.jac[3]) * ky);
            gp[2] += we.x;
            gp[3] += z * kx * cxp;
            gp[4] += z * kx * cyp;
            gp[5] += z * ky * cxp;
            gp[6] += z * ky * cyp;
        } else {
            adj[a] = cadd<T>(adj[a], cscale<T>(w, T(S.scale[arg])));
            acc[sbase + arg] += cmul<T>(w, val[a]).x;
        }
    }
}

// The n-derivative nodes (value, second derivative) of the wanted Sersic leaves, in shared memory
// (whole block, with fill_caches).
__device__ inline void fill_dn_cache(const AdjSmem& A, const gsb_template& tpl, unsigned char* cache, bool have_dn)
{
    const StampSmem& S = A.S;
    for (int l = 0; l < tpl.n_leaves; ++l) {
        if (S.leaf[l].type != GSB_SERSIC || S.aux_cache[l] < 0 || !have_dn) continue;
        float2* dst = reinterpret_cast<float2*>(cache + S.aux_cache[l]);
        const double4* src = A.dn[l].node;
        for (int t = threadIdx.x; t < S.sersic[l].n; t += blockDim.x) dst[t] = make_float2(float(src[t].y), float(src[t].z));
    }
}

// leaf_grad with the shared-memory constants and nodes, for the kinds that have them (float): the
// same forms as leaf_points' values.
template <typename T>
__device__ __forceinline__ LeafD<T> leaf_grad_fast(const AdjSmem& A, const unsigned char* cache, int l, int i, int j,
                                                   int hk, const GridRef& g, T kx, T ky)
{
    const StampSmem& S = A.S;
    if constexpr (sizeof(T) == 4) {
        const LeafT<float>& L = leaf_const<float>(S, l);
        if (L.kind == kLeafSersic && S.aux_cache[l] >= 0) {
            const float u = L.a * float(i) + L.c * float(j), w = L.b * float(i) + L.d * float(j);
            const float k2 = u * u + w * w, flux = L.flux;
            const float inv0 = fast_rcp(k2), inv = fmaf(fmaf(-k2, inv0, 1.f), inv0, inv0);
            const float h = L.q[6], inv_h = L.q[7];
            float phi, dphi, dphin;
            if (k2 >= L.q[0] && k2 < L.q[1]) {
                const float4* node = reinterpret_cast<const float4*>(cache + L.cache);
                const float2* dnode = reinterpret_cast<const float2*>(cache + S.aux_cache[l]);
                const int q = max(1, min(__float_as_int(fmaf(fast_log2(k2), L.q[8], L.q[9]) + 12582912.f) - 0x4b400000, L.n - 1));
                const float4 n0 = node[q - 1], n1 = node[q];
                const float2 d0 = dnode[q - 1], d1 = dnode[q];
                const float e = (n1.w - k2) * inv0;
                float aa;
                if (h < 0.04f) {
                    float p = fmaf(e, -1.f / 16.f, 1.f / 14.f);      // ln(1 + e) / 2, as sersic_points
                    p = fmaf(e, p, -1.f / 12.f);
                    p = fmaf(e, p, 0.1f);
                    p = fmaf(e, p, -0.125f);
                    p = fmaf(e, p, 1.f / 6.f);
                    p = fmaf(e, p, -0.25f);
                    p = fmaf(e, p, 0.5f);
                    aa = e * p;
                } else {
                    aa = 0.5f * logf(n1.w * inv0);
                }
                const float bb = h - aa, P = aa * bb, s = aa * inv_h, c = s * bb * (-1.f / 6.f);
                const float Q = fmaf(aa + h, n0.z, (bb + h) * n1.z);
                const float f = fmaf(c, Q, fmaf(s, n0.y - n1.y, n1.y));
                const float fl = fmaf(fmaf(aa - bb, Q, P * (n1.z - n0.z)), -1.f / 6.f, n1.y - n0.y) * inv_h;
                const float Qn = fmaf(aa + h, d0.y, (bb + h) * d1.y);
                const float fn = fmaf(c, Qn, fmaf(s, d0.x - d1.x, d1.x));
                phi = quotient(f, k2, inv0);
                dphi = (0.5f * fl - f) * inv * inv;
                dphin = (fn - float(A.dn[l].dfront) * fl) * inv;     // the argument moves with the grid origin
            } else {
                sersic_phi_grad<float>(S.sersic[l], A.dn[l], k2, phi, dphi, dphin);
            }
            LeafD<float> r;
            r.unit = phi;
            r.v = flux * phi;
            r.gn = flux * dphin;
            const float d2 = 2.f * flux * dphi * L.size;              // dv/dk' = 2 k' dv/d|k'|^2
            r.gx = d2 * u;
            r.gy = d2 * w;
            return r;
        }
        if (L.kind == kLeafExpFast) {
            const ushort2 c = reinterpret_cast<const ushort2*>(cache + L.cache)[hk + j];
            LeafD<T> r{T(0), T(0), T(0), T(0), T(0)};
            if (i < int(c.x) || i >= int(c.y)) return r;
            const float u = L.a * float(i) + L.c * float(j), w = L.b * float(i) + L.d * float(j);
            const float s = refined_rsqrt(1.f + (u * u + w * w)), ss = s * s;
            r.unit = ss * s;
            r.v = L.flux * r.unit;
            const float d2 = -3.f * r.v * ss * L.size;
            r.gx = d2 * u;
            r.gy = d2 * w;
            return r;
        }
    }
    if (sizeof(T) == 8 && leaf_const<T>(S, l).kind == kLeafExp) {
        const LeafT<T>& L = leaf_const<T>(S, l);
        const ushort2 c = reinterpret_cast<const ushort2*>(cache + L.cache)[hk + j];
        LeafD<T> r{T(0), T(0), T(0), T(0), T(0)};
        if (i < int(c.x) || i >= int(c.y)) return r;
        const T u = L.a * kx + L.c * ky, w = L.b * kx + L.d * ky, r0 = L.q[0];
        const T p = T(1) + (u * u + w * w) * r0 * r0;
        const T phi = T(1) / (p * sqrt(p));
        r.unit = phi;
        r.v = L.flux * phi;
        const T d2 = T(-3) * r.v / p * r0 * r0;
        r.gx = d2 * u;
        r.gy = d2 * w;
        return r;
    }
    return leaf_grad<T>(S.leaf[l], S.sersic, A.dn, kx, ky, g, i - g.x0, j - g.y0);
}

// The unit phasor of phase p at (i, j): the product of its cached axis factors, or directly.
template <typename T>
__device__ __forceinline__ Cx<T> phase_unit(const StampSmem& S, const unsigned char* cache, int p, int i, int j, int hk)
{
    if (S.phase_cache[p] >= 0) {
        const Cx<T>* PX = reinterpret_cast<const Cx<T>*>(cache + S.phase_cache[p]);
        return cmul<T>(PX[i], PX[hk + 1 + j + hk]);
    }
    double tt = i * S.phase_ax[p] + j * S.phase_ay[p];
    tt -= rint(tt);
    T sn, cs;
    sincospi(T(-2. * tt), &sn, &cs);
    return cx<T>(cs, sn);
}

// Gradients of the leaves of a Sum atom (LEAF and ADD ops [o0, o1)) with cotangent w: each
// leaf receives w unchanged.
template <typename T>
__device__ __noinline__ void sum_atom_grads(const gsb_template& tpl, const AdjSmem& A, const unsigned char* cache,
                                            unsigned want, T kx, T ky, int i, int j, const GridRef& g, Cx<T> w, T* acc,
                                            int o0, int o1)
{
    const T ar = w.x;
    for (int o = o0; o < o1; ++o) {
        if (tpl.op_code[o] != GSB_OP_LEAF) continue;
        const int l = tpl.op_arg[o];
        if (!want_leaf(want, l)) continue;
        const LeafD<T> d = leaf_grad_fast<T>(A, cache, l, i, j, g.n / 2, g, kx, ky);
        T* gl = acc + kGradPerLeaf * l;
        gl[0] += ar * d.unit;
        gl[1] += ar * d.gx * kx;
        gl[2] += ar * d.gy * kx;
        gl[3] += ar * d.gx * ky;
        gl[4] += ar * d.gy * ky;
        gl[5] += ar * d.gn;
    }
}

// Values and derivatives of the two leaves of a Sum atom [o0, o0 + 3) (values only where not wanted).
template <typename T> struct LeafPair { LeafD<T> d[2]; };

template <typename T>
__device__ __noinline__ LeafPair<T> sum_pair_grads(const gsb_template& tpl, const AdjSmem& A, const unsigned char* cache,
                                                   unsigned want, T kx, T ky, int i, int j, const GridRef& g, int o0)
{
    LeafPair<T> r;
    r.d[0] = r.d[1] = LeafD<T>{T(0), T(0), T(0), T(0), T(0)};
#pragma unroll 1
    for (int q = 0; q < 2; ++q) {
        const int l = tpl.op_arg[o0 + q];
        LeafD<T> d{T(0), T(0), T(0), T(0), T(0)};
        if (want_leaf(want, l)) d = leaf_grad_fast<T>(A, cache, l, i, j, g.n / 2, g, kx, ky);
        else d.v = leaf_fast<T>(A.S, cache, l, i, j, g.n / 2, g.dk);
        r.d[1] = d;
        if (q == 0) r.d[0] = d;
    }
    return r;
}

// The first atom that is a Sum of two leaves with derivatives of their own (bulge + disk), or -1: its
// leaves are evaluated once, value and derivatives together, and their gradients stay in registers
// (any other Sum takes its value from eval_range and its derivatives from sum_atom_grads).
template <bool II>
__device__ __forceinline__ int sum_pair_atom(const gsb_template& tpl, const StampSmem& S)
{
    for (int t = 0; t < S.n_atoms; ++t) {
        const int o0 = S.atom_o0[t];
        if (S.atom_kind[t] != kAtomSum || S.atom_o1[t] - o0 != 3) continue;
        if (II && (S.leaf[tpl.op_arg[o0]].type == GSB_INTERPOLATED || S.leaf[tpl.op_arg[o0 + 1]].type == GSB_INTERPOLATED)) continue;
        return t;
    }
    return -1;
}

// Factored reverse pass at (i, j): F = prod_a atom_a * XS[i] YS[j]; the cotangent of atom a
// is u XS YS prod_{b != a} atom_b (prefix and suffix products, no division).  Leaf, phase and
// scale atoms accumulate into ga[a][*] (registers); subtree atoms run adjoint_range into acc.
template <typename T, bool II = true>
__device__ __forceinline__ void adjoint_point_factored(const gsb_template& tpl, const AdjSmem& A,
                                                       const unsigned char* cache, unsigned want, double dk,
                                                       int i, int j, const GridRef& g, Cx<T> u,
                                                       T (&ga)[kAdjAtoms][kGradPerPhase], T* acc, int pair,
                                                       T (&gs)[2][kGradPerLeaf])
{
    const StampSmem& S = A.S;
    const int hk = g.n / 2;
    const T kx = T(i) * T(dk), ky = T(j) * T(dk);
    const int na = S.n_atoms;
    // ld[a] holds a leaf atom's derivatives, or a phase atom's unit phasor in (gx, gy)
    Cx<T> val[kAdjAtoms], pre[kAdjAtoms];
    LeafD<T> ld[kAdjAtoms];
    LeafPair<T> ps;
    Cx<T> run = cx<T>(T(1), T(0));
#pragma unroll
    for (int a = 0; a < kAdjAtoms; ++a) {
        val[a] = cx<T>(T(1), T(0));
        ld[a] = LeafD<T>{T(0), T(0), T(0), T(0), T(0)};
        if (a < na) {
            const int kind = S.atom_kind[a];
            const int o0 = S.atom_o0[a], o1 = S.atom_o1[a];
            if (kind == kAtomPhase) {
                const int p = S.atom_arg[a];
                const Cx<T> e = phase_unit<T>(S, cache, p, i, j, hk);
                ld[a].gx = e.x;
                ld[a].gy = e.y;
                val[a] = cscale<T>(e, T(S.phase[p].flux_scaling));
            } else if (kind == kAtomScale) {
                val[a] = cx<T>(T(S.scale[S.atom_arg[a]]), T(0));
            } else if (o1 - o0 == 1) {
                const int l = tpl.op_arg[o0];
                if (want_leaf(want, l) && !(II && S.leaf[l].type == GSB_INTERPOLATED)) {
                    ld[a] = leaf_grad_fast<T>(A, cache, l, i, j, hk, g, kx, ky);
                    val[a] = cx<T>(ld[a].v, T(0));
                } else {
                    val[a] = leaf_cfast<T, II, !II && sizeof(T) == 4>(S, cache, l, i, j, g);
                }
            } else if (a == pair) {
                ps = sum_pair_grads<T>(tpl, A, cache, want, kx, ky, i, j, g, o0);
                val[a] = cx<T>(ps.d[0].v + ps.d[1].v, T(0));
            } else {
                val[a] = eval_range<T, II>(tpl, S, cache, dk, i, j, g, o0, o1);
            }
        }
        pre[a] = run;
        run = cmul<T>(run, val[a]);
    }
    const Cx<T>* XS = reinterpret_cast<const Cx<T>*>(cache + S.xy_cache);
    const Cx<T> us = cmul<T>(u, cmul<T>(XS[i], XS[hk + 1 + j + hk]));
    Cx<T> suf = cx<T>(T(1), T(0));
#pragma unroll
    for (int a = kAdjAtoms - 1; a >= 0; --a) {
        if (a < na) {
            const Cx<T> w = cmul<T>(cmul<T>(us, pre[a]), suf);
            const int kind = S.atom_kind[a];
            const int o0 = S.atom_o0[a], o1 = S.atom_o1[a];
            if (kind == kAtomPhase) {
                const gsb_phase& P = S.phase[S.atom_arg[a]];
                const Cx<T> we = cmul<T>(w, cx<T>(ld[a].gx, ld[a].gy));
                const T z = T(P.flux_scaling) * we.y;
                const T cxp = T(P.cenx), cyp = T(P.ceny);
                ga[a][0] += z * (T(P.jac[0]) * kx + T(P.jac[2]) * ky);
                ga[a][1] += z * (T(P.jac[1]) * kx + T(P.jac[3]) * ky);
                ga[a][2] += we.x;
                ga[a][3] += z * kx * cxp;
                ga[a][4] += z * kx * cyp;
                ga[a][5] += z * ky * cxp;
                ga[a][6] += z * ky * cyp;
            } else if (kind == kAtomScale) {
                ga[a][0] += w.x;
            } else if (o1 - o0 == 1) {
                const T ar = w.x;
                ga[a][0] += ar * ld[a].unit;
                ga[a][1] += ar * ld[a].gx * kx;
                ga[a][2] += ar * ld[a].gy * kx;
                ga[a][3] += ar * ld[a].gx * ky;
                ga[a][4] += ar * ld[a].gy * ky;
                ga[a][5] += ar * ld[a].gn;
            } else if (a == pair) {
                const T ar = w.x;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const T gx = ar * ps.d[q].gx, gy = ar * ps.d[q].gy;
                    gs[q][0] += ar * ps.d[q].unit;
                    gs[q][1] += gx * kx;
                    gs[q][2] += gy * kx;
                    gs[q][3] += gx * ky;
                    gs[q][4] += gy * ky;
                    gs[q][5] += ar * ps.d[q].gn;
                }
            } else if (kind == kAtomSum) {
                sum_atom_grads<T>(tpl, A, cache, want, kx, ky, i, j, g, w, acc, o0, o1);
            } else {
                adjoint_range<T, II>(tpl, A, dk, i, j, g, w, acc, o0, o1);
            }
            suf = cmul<T>(suf, val[a]);
        }
    }
}

// In-place transform of the warp's buffer (values at fft_slot).
template <typename T, int N>
__device__ __forceinline__ void adj_warp_fft(Cx<T>* buf, const Cx<T>* tw)
{
    warp_fft_io<T, N, +1, true, true>(buf, tw, [&](int i) { return buf[fft_slot(i)]; },
                                      [&](int i, Cx<T> z) { buf[fft_slot(i)] = z; });
}

template <typename T>
__device__ inline T load_cot(const void* p, int dtype, long long idx)
{
    return dtype == GSB_F32 ? T(reinterpret_cast<const float*>(p)[idx])
                            : T(reinterpret_cast<const double*>(p)[idx]);
}

// Warps per CTA: 16, or 8 where 16 FFT buffers of N complex T do not fit (double, N >= 768).
// In float at N <= 128, 8 warps of up to 128 registers, two CTAs an SM, as the forward.
template <typename T, int N>
__host__ __device__ constexpr int adj_warps()
{
    if (sizeof(T) == 4 && N <= 128) return kWarps / 2;
    return ((sizeof(AdjSmem) + 15) / 16 * 16 + sizeof(Cx<T>) * N * (1 + kWarps) + kCacheBytes + 4096 <=
            kSmemLimit) ? kWarps : kWarps / 2;
}

// PAIR: compiled for programs with a Sum of two leaves (sum_pair_atom), whose 22 registers the others
// should not pay for: bulge + disk gradients of 2048 stamps at N = 192 4.2 -> 2.3 ms (the leaf of an
// atom inlined included, 4.2 -> 3.1 by itself), a Sersic fit at N = 128 0.51 ms without against 0.69.
template <typename T, int N, bool WSMEM, bool II, bool PAIR>
__global__ void __launch_bounds__(adj_warps<T, N>() * 32, sizeof(T) == 4 && N <= 128 ? 2 : 1) adjoint_fused_kernel(const __grid_constant__ AdjArgs a)
{
    constexpr int NW = adj_warps<T, N>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int H = N / 2 + 1;
    constexpr int WS = N + 1;
    AdjSmem& A = *reinterpret_cast<AdjSmem*>(smem_raw);
    StampSmem& S = A.S;
    size_t off = (sizeof(AdjSmem) + 15) & ~size_t(15);
    Cx<T>* tw = reinterpret_cast<Cx<T>*>(smem_raw + off);
    off += sizeof(Cx<T>) * N;
    Cx<T>* scratch = reinterpret_cast<Cx<T>*>(smem_raw + off);
    off += sizeof(Cx<T>) * N * NW;
    Cx<T>* W = WSMEM ? reinterpret_cast<Cx<T>*>(smem_raw + off)
                     : reinterpret_cast<Cx<T>*>(a.work) + (size_t)blockIdx.x * H * WS;
    if (WSMEM) off += sizeof(Cx<T>) * H * WS;
    unsigned char* cache = smem_raw + ((off + 15) & ~size_t(15));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Cx<T>* buf = scratch + warp * N;
    fill_twiddles<T>(tw, N);
    const double dk = 2. * kPi / N;
    const T inv_n2 = T(1) / (T(N) * T(N));
    const int ng = grad_count(a.tpl);
    if (threadIdx.x == 0) program_children(a.tpl, A.child1, A.child2);

    for (int s = blockIdx.x; s < a.n_stamps; s += gridDim.x) {
        __syncthreads();
        load_stamp(S, a.tpl, s, a.leaves, a.phases, a.scales, a.stamps, a.sersic_header,
                   a.sersic_node, a.sersic_stride, 1. / N);
        if (threadIdx.x < a.tpl.n_leaves && S.leaf[threadIdx.x].type == GSB_SERSIC && a.sersic_dheader) {
            const int t = a.leaves[(size_t)s * a.tpl.n_leaves + threadIdx.x].table;
            const double* D = a.sersic_dheader + (size_t)t * kSersicDHeader;
            SersicDnView& v = A.dn[threadIdx.x];
            v.dkd2 = D[kSD_DKD2];
            v.dkd4 = D[kSD_DKD4];
            v.dhigha = D[kSD_DHIGHA];
            v.dhighb = D[kSD_DHIGHB];
            v.dlnre = D[kSD_DLNRE];
            v.dfront = D[kSD_DFRONT];
            v.node = a.sersic_dnode + (size_t)t * a.sersic_stride;
        }
        for (int k = threadIdx.x; k < ng; k += blockDim.x) A.gacc[k] = 0.;
        __syncthreads();
        const gsb_stamp& G = S.geom;
        const int Nk = G.Nk;
        const int hk = Nk / 2;
        const GridRef g{dk, 0, -hk, hk + 1, Nk + 1};
        if (threadIdx.x == 0) plan_caches<T, II>(S, a.tpl, a.fac, Nk, a.want);
        __syncthreads();
        fill_caches<T, II>(S, a.tpl, cache, dk, Nk);
        fill_dn_cache(A, a.tpl, cache, a.sersic_dheader != nullptr);
        __syncthreads();
        const bool factored = S.xy_cache >= 0 && S.n_atoms <= kAdjAtoms;
        const int pair = PAIR && factored ? sum_pair_atom<II>(a.tpl, S) : -1;
        bool subtree = !factored;
        if (factored)
            for (int t = 0; t < S.n_atoms; ++t)
                subtree |= t != pair && (S.atom_kind[t] == kAtomRange || S.atom_kind[t] == kAtomSum) &&
                           S.atom_o1[t] - S.atom_o0[t] > 1;

        // ---- row phase: forward-sign DFT of pairs of cotangent rows ----
        const int npairs = (G.ny + 1) / 2;
        for (int p = warp; p < npairs; p += NW) {
            const bool two = 2 * p + 1 < G.ny;
            for (int x = lane; x < N; x += 32) buf[x] = cx<T>(T(0), T(0));
            __syncwarp();
            const long long row1 = G.out_offset + (long long)(2 * p) * G.nx;
            for (int i = lane; i < G.nx; i += 32) {
                const T g1 = load_cot<T>(a.cot, a.cot_dtype, row1 + i);
                const T g2 = two ? load_cot<T>(a.cot, a.cot_dtype, row1 + G.nx + i) : T(0);
                buf[fft_slot(pmod(G.xmin + i, N))] = cx<T>(g1, g2);
            }
            __syncwarp();
            adj_warp_fft<T, N>(buf, tw);
            const int y1 = pmod(G.ymin + 2 * p, N), y2 = pmod(G.ymin + 2 * p + 1, N);
            for (int c = lane; c < H; c += 32) {
                const Cx<T> z = buf[fft_slot(c)];
                const Cx<T> zm = buf[fft_slot(c == 0 ? 0 : N - c)];
                W[(size_t)c * WS + y1] = cx<T>(T(0.5) * (z.x + zm.x), T(0.5) * (z.y - zm.y));
                if (two) W[(size_t)c * WS + y2] = cx<T>(T(0.5) * (z.y + zm.y), T(0.5) * (zm.x - z.x));
            }
            __syncwarp();
        }
        __syncthreads();

        // ---- column phase: forward-sign DFT along y, then the reverse pass per alias ----
        // Each lane accumulates its gradient terms over all of its warp's columns; the warp
        // reduces them once per stamp.
        T acc[kMaxGrad];
        T ga[kAdjAtoms][kGradPerPhase], gs[2][kGradPerLeaf];
        if (subtree)
            for (int k = 0; k < ng; ++k) acc[k] = T(0);
#pragma unroll
        for (int t = 0; t < kAdjAtoms; ++t)
#pragma unroll
            for (int e = 0; e < kGradPerPhase; ++e) ga[t][e] = T(0);
#pragma unroll
        for (int e = 0; e < kGradPerLeaf; ++e) gs[0][e] = gs[1][e] = T(0);
        for (int c = warp; c < H; c += NW) {
            const Cx<T>* Wc = W + (size_t)c * WS;
            warp_fft_io<T, N, +1, false, true>(
                buf, tw, [&](int y) { return pmod(y - G.ymin, N) < G.ny ? Wc[y] : cx<T>(T(0), T(0)); },
                [&](int i, Cx<T> z) { buf[fft_slot(i)] = z; });
            const T wc = (c == 0 || 2 * c == N) ? inv_n2 : T(2) * inv_n2;
            const int kx0 = c + ceil_div(-hk - c, N) * N;
            // the column's rows ky = -hk .. hk in order, every alias once, as the forward takes them
            for (int ky = -hk + lane; ky <= hk; ky += 32) {
                const Cx<T> gh = cscale<T>(buf[fft_slot(pmod(ky, N))], wc);
                for (int kx = kx0; kx <= hk; kx += N) {
                    const bool pos = kx >= 0;
                    // an alias taken as conj(F(-k)) contributes Re(Ghat conj(dF)) = Re(conj(Ghat) dF)
                    if (factored)
                        adjoint_point_factored<T, II>(a.tpl, A, cache, a.want, dk, pos ? kx : -kx,
                                                  pos ? ky : -ky, g, pos ? gh : cconj<T>(gh), ga, acc, pair, gs);
                    else
                        adjoint_range<T, II>(a.tpl, A, dk, pos ? kx : -kx, pos ? ky : -ky, g,
                                         pos ? gh : cconj<T>(gh), acc, 0, a.tpl.n_ops);
                }
            }
            __syncwarp();
        }
        if (subtree) {
            for (int k = 0; k < ng; ++k) {
                double v = double(acc[k]);
                for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                if (lane == 0) atomicAdd(&A.gacc[k], v);
            }
        }
        if (factored) {
            const int pbase = kGradPerLeaf * a.tpl.n_leaves;
            const int sbase = pbase + kGradPerPhase * a.tpl.n_phases;
#pragma unroll
            for (int t = 0; t < kAdjAtoms; ++t) {
                if (t >= S.n_atoms) break;
                const int kind = S.atom_kind[t];
                int base, cnt;
                if (kind == kAtomPhase) { base = pbase + kGradPerPhase * S.atom_arg[t]; cnt = kGradPerPhase; }
                else if (kind == kAtomScale) { base = sbase + S.atom_arg[t]; cnt = 1; }
                else if (S.atom_o1[t] - S.atom_o0[t] == 1 && want_leaf(a.want, S.atom_arg[t])) {
                    base = kGradPerLeaf * S.atom_arg[t]; cnt = kGradPerLeaf;
                } else continue;
#pragma unroll
                for (int e = 0; e < kGradPerPhase; ++e) {
                    if (e >= cnt) break;
                    double v = double(ga[t][e]);
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                    if (lane == 0) atomicAdd(&A.gacc[base + e], v);
                }
            }
            if (pair >= 0)
#pragma unroll
                for (int e = 0; e < 2 * kGradPerLeaf; ++e) {
                    double v = double(gs[e / kGradPerLeaf][e % kGradPerLeaf]);
                    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                    if (lane == 0)
                        atomicAdd(&A.gacc[kGradPerLeaf * a.tpl.op_arg[S.atom_o0[pair] + e / kGradPerLeaf] + e % kGradPerLeaf], v);
                }
        }
        __syncthreads();
        // Sersic leaves given by half-light radius: r0 = hlr / r_e(n), so at fixed hlr
        // d/dn picks up -d ln r_e/dn * d/d ln r0, and d/d ln r0 = sum_ij J_ij d/dJ_ij.
        if (threadIdx.x < a.tpl.n_leaves && want_leaf(a.want, threadIdx.x)) {
            const LeafParams& L = S.leaf[threadIdx.x];
            if (L.type == GSB_SERSIC && (L.flags & GSB_LEAF_SIZE_IS_HLR)) {
                double* gl = A.gacc + kGradPerLeaf * threadIdx.x;
                const double glnr0 = L.jac[0] * gl[1] + L.jac[1] * gl[2] + L.jac[2] * gl[3] + L.jac[3] * gl[4];
                gl[5] -= A.dn[threadIdx.x].dlnre * glnr0;
            }
        }
        __syncthreads();
        // entries of records outside the want mask are written as zero
        const int pbase = kGradPerLeaf * a.tpl.n_leaves;
        const int sbase = pbase + kGradPerPhase * a.tpl.n_phases;
        for (int k = threadIdx.x; k < ng; k += blockDim.x) {
            const bool w = k < pbase ? want_leaf(a.want, k / kGradPerLeaf)
                         : k < sbase ? want_phase(a.want, (k - pbase) / kGradPerPhase)
                                     : want_scale(a.want, k - sbase);
            a.grad[(size_t)s * ng + k] = w ? A.gacc[k] : 0.;
        }
    }
}

template <typename T, int N>
constexpr size_t adj_smem_bytes(bool wsmem)
{
    size_t off = (sizeof(AdjSmem) + 15) & ~size_t(15);
    off += sizeof(Cx<T>) * N * (1 + adj_warps<T, N>());
    if (wsmem) off += sizeof(Cx<T>) * (N / 2 + 1) * (N + 1);
    return ((off + 15) & ~size_t(15)) + kCacheBytes;
}

template <typename T, int N>
constexpr bool adj_w_fits_smem()
{
    return adj_smem_bytes<T, N>(true) <= kSmemLimit;
}

template <typename T, int N>
int adj_grid(int n_stamps)
{
    DeviceState* st = device_state();
    const size_t sm = adj_smem_bytes<T, N>(adj_w_fits_smem<T, N>());
    int per_sm = int(std::min<size_t>(kSmemLimit / sm, 4));
    if (per_sm < 1) per_sm = 1;
    return std::max(1, std::min(n_stamps, st->sm_count * per_sm));
}

template <typename T, int N>
size_t adj_workspace_bytes_for(int n_stamps)
{
    if (adj_w_fits_smem<T, N>()) return 0;
    return sizeof(Cx<T>) * (size_t)(N / 2 + 1) * (N + 1) * adj_grid<T, N>(n_stamps);
}

template <typename T, int N>
int launch_adjoint(const AdjArgs& args, size_t work_bytes, cudaStream_t stream)
{
    constexpr bool wsmem = adj_w_fits_smem<T, N>();
    constexpr size_t sm = adj_smem_bytes<T, N>(wsmem);
    const int grid = adj_grid<T, N>(args.n_stamps);
    if (!wsmem && (args.work == nullptr || work_bytes < adj_workspace_bytes_for<T, N>(args.n_stamps)))
        return set_error(GSB_ERR_INVALID, "adjoint workspace too small");
    auto run = [&](auto kernel) -> int {
        GSB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
        kernel<<<grid, adj_warps<T, N>() * 32, sm, stream>>>(args);
        return GSB_OK;
    };
    // programs without image leaves run the instance compiled without their code, and those with a Sum of
    // two leaves the one that keeps both in registers (float; in double the registers are not there)
    bool pair = false;
    for (int f = 0; f < args.fac.n; ++f)
        pair = pair || (args.fac.kind[f] == kFactorSum && args.fac.o1[f] - args.fac.o0[f] == 3);
    int rc;
    if (has_image_leaves(args.tpl)) rc = run(adjoint_fused_kernel<T, N, wsmem, true, false>);
    else if (pair && sizeof(T) == 4) rc = run(adjoint_fused_kernel<T, N, wsmem, false, sizeof(T) == 4>);
    else rc = run(adjoint_fused_kernel<T, N, wsmem, false, false>);
    if (rc) return rc;
    GSB_CUDA_CHECK(cudaGetLastError());
    return GSB_OK;
}

}  // namespace gsb
