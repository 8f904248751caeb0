// Fused FFT drawing kernels.
//
// draw_fused_kernel<T, N, W_IN_SMEM>: one CTA draws one stamp at a time (persistent loop over
// the stamps of an FFT-size bucket):
//   1. column phase: each warp takes columns kx = 0..N/2 of the wrapped k-image; every lane
//      builds the wrapped value of its rows by summing the program over all aliases
//      (kx + a N, ky + b N) inside the Nk x Nk evaluation grid -- the Hermitian wrap of
//      wrapImage(hermx=True) (src/Image.cpp:578-727) done as a gather -- then the warp
//      inverse-transforms the column (length N) and stores it into W (shared memory, or a
//      per-CTA global slab when it does not fit);
//   2. row phase: each warp packs two needed image rows as one complex row
//      (row1 + i row2, each Hermitian-extended in kx), inverse-transforms it and writes the
//      pixels that fall inside the stamp, scaled by 1/N^2, with the compensated flux sum.
// This is drawFFT (gsobject.py:2014-2045) = drawFFT_makeKImage + _drawKImage + wrap +
// irfft(shift_in, shift_out) (src/Image.cpp:815-912) + drawFFT_finish, with no k-image in
// HBM.  The output pixel (px, py) is the inverse DFT at (px mod N, py mod N), which is what
// irfft's half swap and (-1)^(i+j) pre-multiplication produce.
#pragma once
#include <algorithm>
#include <string>

#include "gsb_fft.cuh"
#include "gsb_internal.cuh"
#include "gsb_interp.cuh"
#include "gsb_profiles.cuh"

namespace gsb {


constexpr int kWarps = 16;          // most warps per CTA

// How a leaf's value is formed at a wave vector.  The named kinds read constants of type T formed
// once per stamp (LeafT); kLeafGeneric goes through leaf_kvalue.
enum LeafKind { kLeafGeneric = 0, kLeafSep, kLeafExp, kLeafExpFast, kLeafSersic, kLeafMoffat1, kLeafMoffat2, kLeafMoffat3,
                kLeafMoffatSum, kLeafKolm, kLeafAiry };

// A leaf's constants in the working precision: (u, v) = (a i + c j, b i + d j) is the wave vector of
// grid point (i, j) in the leaf's own units (Jacobian, dk and size in one factor each), so a point
// costs a multiply-add an axis and no conversion from the FP64 records.
template <typename T>
struct __align__(16) LeafT {
    T a, b, c, d;
    T flux;
    int kind, cache, n;
    T size;             // the leaf's size (in the units of its Jacobian's source), for derivatives
    T q[10];
};

struct StampSmem {
    LeafParams leaf[GSB_MAX_LEAVES];
    LeafT<double> leaf_t[GSB_MAX_LEAVES];   // holds LeafT<T> of the kernel's T (leaf_const)
    SersicTableView sersic[GSB_MAX_LEAVES];
    gsb_phase phase[GSB_MAX_PHASES];
    double phase_ax[GSB_MAX_PHASES];   // phase turns per k index, x and y
    double phase_ay[GSB_MAX_PHASES];
    double scale[GSB_MAX_SCALES];
    gsb_stamp geom;
    double flux_part[kWarps];
    // Per-stamp shared-memory caches (offsets in bytes into the cache area, -1 = not cached):
    // separable leaf factors X[i], Y[j + Nk/2]; phase factors PX[i], PY[j + Nk/2]; Sersic nodes.
    int leaf_cache[GSB_MAX_LEAVES];
    int phase_cache[GSB_MAX_PHASES];
    int sersic_cache[GSB_MAX_LEAVES];
    int ii_cache[GSB_MAX_LEAVES];      // InterpolatedImage taps per column / row (IITaps)
    // Exponential: kept columns per row; Moffat: quadrature nodes; Sersic: n-derivative nodes (adjoint)
    int aux_cache[GSB_MAX_LEAVES];
    int regstack;      // the program fits the 4-deep register stack
    // Factored form of the program (see plan_factored): the root is a product of atoms; the
    // separable atoms (diagonal Box / Gaussian leaves, phases, scales) are folded into
    // XS[i] YS[j + Nk/2] (complex, at offset xy_cache, -1 = not factored) and the others are
    // evaluated per k-point over their postfix op ranges [atom_o0, atom_o1).
    int xy_cache;
    int n_atoms;
    short atom_o0[GSB_MAX_OPS];
    short atom_o1[GSB_MAX_OPS];
    unsigned char atom_kind[GSB_MAX_OPS];      // kAtomRange, kAtomPhase (arg), kAtomScale (arg)
    unsigned char atom_arg[GSB_MAX_OPS];
    // evaluation list: the leaves of the atoms that are real leaves or sums of them, real_last marking
    // the last of an atom; the other atoms follow by index
    int n_real, n_other;
    unsigned char real_leaf[GSB_MAX_OPS], real_last[GSB_MAX_OPS], other[GSB_MAX_OPS];
    unsigned char leaf_sep[GSB_MAX_LEAVES];    // leaf folded into XS / YS
    unsigned char phase_sep[GSB_MAX_PHASES];   // phase folded into XS / YS
    unsigned char scale_sep[GSB_MAX_SCALES];   // scale folded into XS / YS
};

// Bytes of shared memory reserved for the per-stamp caches (kCacheBytes; the fused kernels in double at N = 768
// and 1024, one CTA an SM as it is, hold twice that, so that Nk = N stays factored).
constexpr int kCacheBytes = 24 * 1024;
template <typename T>
__host__ __device__ constexpr int form_budget(int N) { return sizeof(T) == 8 && N >= 768 ? 2 * kCacheBytes : kCacheBytes; }

constexpr size_t kSmemLimit = 227 * 1024;

// Warps per CTA of the fused kernels for (T, N): 16, or 8 where 16 per-warp FFT buffers of N
// complex T (plus twiddles, stamp state and caches) exceed the 227 KB of shared memory
// (double at N >= 768).
//
// In float, 8 warps of up to 128 registers where the shared memory leaves room for two CTAs on an
// SM (N <= 128, and N >= 256, whose W is in global memory): the evaluator takes four wave
// vectors a lane at a time, which needs the registers, and two CTAs cover one another's set-up.
// N = 192 fills an SM's shared memory with one CTA: 16 warps.
template <typename T, int N>
__host__ __device__ constexpr int fused_warps()
{
    if (sizeof(T) == 4 && N != 192) return kWarps / 2;
    return ((sizeof(StampSmem) + 15) / 16 * 16 + sizeof(Cx<T>) * N * (1 + kWarps) + kCacheBytes + 4096 <=
            kSmemLimit) ? kWarps : kWarps / 2;
}

// The factors of the program's root product, found once per launch on the host (plan_factors): MUL
// nodes are flattened, PHASE and SCALE nodes give a separable factor and pass their child on, and
// every other LEAF and every ADD subtree is a factor of its own.
enum { kFactorLeaf = 0, kFactorTree, kFactorSum, kFactorPhase, kFactorScale };
struct FactorPlan {
    int n;
    int depth;                                    // of the evaluation stack
    short o0[GSB_MAX_OPS], o1[GSB_MAX_OPS];       // ops of a leaf or subtree
    unsigned char kind[GSB_MAX_OPS], arg[GSB_MAX_OPS];
};

struct DrawArgs {
    gsb_template tpl;
    FactorPlan fac;
    int n_stamps;
    const gsb_leaf* leaves;
    const gsb_phase* phases;
    const double* scales;
    const gsb_stamp* stamps;
    const double* sersic_header;
    const double4* sersic_node;
    int sersic_stride;
    void* out;
    int out_dtype;
    int add;
    double* added_flux;
    void* work;          // per-CTA W slabs when W does not fit in shared memory
    int max_grid = 0;    // when > 0: CTAs for which `work` has a slab
};

__device__ inline int floor_div(int a, int n) { return a >= 0 ? a / n : -((-a + n - 1) / n); }
__device__ inline int ceil_div(int a, int n) { return -floor_div(-a, n); }
__device__ inline int pmod(int a, int n) { const int r = a % n; return r < 0 ? r + n : r; }

// Load stamp s's leaves / phases / scales into shared memory.
__device__ inline void load_stamp(StampSmem& S, const gsb_template& tpl, int s, const gsb_leaf* leaves,
                           const gsb_phase* phases, const double* scales, const gsb_stamp* stamps,
                           const double* sh, const double4* snode, int sstride, double dk_over_2pi)
{
    const int t = threadIdx.x;
    if (t < tpl.n_leaves) {
        const gsb_leaf& g = leaves[(size_t)s * tpl.n_leaves + t];
        LeafParams& L = S.leaf[t];
        for (int i = 0; i < 4; ++i) L.jac[i] = g.jac[i];
        L.flux = g.flux;
        for (int i = 0; i < 8; ++i) L.d[i] = g.d[i];
        L.flags = g.flags;
        L.type = tpl.leaf_type[t];
        L.table = t;
        if (L.type == GSB_SERSIC && sh) {
            const double* H = sh + (size_t)g.table * kSersicHeader;
            SersicTableView& v = S.sersic[t];
            v.n = int(H[kSH_NUSED]);
            v.front = H[kSH_FRONT];
            v.da = H[kSH_DA];
            v.ksq_min = H[kSH_KSQMIN];
            v.ksq_max = H[kSH_KSQMAX];
            v.kderiv2 = H[kSH_KD2];
            v.kderiv4 = H[kSH_KD4];
            v.highk_a = H[kSH_HIGHA];
            v.highk_b = H[kSH_HIGHB];
            v.node = snode + (size_t)g.table * sstride;
        }
    }
    if (t >= 32 && t < 32 + tpl.n_phases) {
        const int i = t - 32;
        const gsb_phase& P = phases[(size_t)s * tpl.n_phases + i];
        S.phase[i] = P;
        // exp(-i (kx' cx + ky' cy)) with k' = jac^T k and k = (i, j) dk:
        // argument = 2 pi (i ax + j ay), ax = (A cx + B cy) dk / 2 pi, ay = (C cx + D cy) dk / 2 pi
        S.phase_ax[i] = (P.jac[0] * P.cenx + P.jac[1] * P.ceny) * dk_over_2pi;
        S.phase_ay[i] = (P.jac[2] * P.cenx + P.jac[3] * P.ceny) * dk_over_2pi;
    }
    if (t >= 64 && t < 64 + tpl.n_scales) S.scale[t - 64] = scales[(size_t)s * tpl.n_scales + (t - 64)];
    if (t == 96 && stamps) S.geom = stamps[s];
}

// Evaluate the program at k index (i, j) (kx = i dk, ky = j dk) of grid g.
// II: the program may hold InterpolatedImage leaves (their code is compiled in only then).
template <typename T, bool II = true>
__device__ __noinline__ Cx<T> eval_program(const gsb_template& tpl, const StampSmem& S, double dk, int i, int j,
                              const GridRef& g)
{
    Cx<T> stack[GSB_MAX_OPS];
    int sp = 0;
    const T kx = T(i * dk), ky = T(j * dk);
    const int gi = i - g.x0, gj = j - g.y0;
    for (int o = 0; o < tpl.n_ops; ++o) {
        const int code = tpl.op_code[o], arg = tpl.op_arg[o];
        if (code == GSB_OP_LEAF) {
            if (II && S.leaf[arg].type == GSB_INTERPOLATED)
                stack[sp++] = ii_kvalue<T>(S.leaf[arg], dk, i, j);
            else
                stack[sp++] = cx<T>(leaf_kvalue<T>(S.leaf[arg], S.sersic, kx, ky, g, gi, gj), T(0));
        } else if (code == GSB_OP_MUL) {
            --sp;
            stack[sp - 1] = cmul<T>(stack[sp - 1], stack[sp]);
        } else if (code == GSB_OP_ADD) {
            --sp;
            stack[sp - 1] = cadd<T>(stack[sp - 1], stack[sp]);
        } else if (code == GSB_OP_PHASE) {
            double tt = i * S.phase_ax[arg] + j * S.phase_ay[arg];
            tt -= rint(tt);
            T sn, cs;
            sincospi(T(-2. * tt), &sn, &cs);
            const T fs = T(S.phase[arg].flux_scaling);
            stack[sp - 1] = cmul<T>(stack[sp - 1], cx<T>(fs * cs, fs * sn));
        } else if (code == GSB_OP_SCALE) {
            stack[sp - 1] = cscale<T>(stack[sp - 1], T(S.scale[arg]));
        }
    }
    return stack[0];
}

template <typename T> struct NodeT;
template <> struct NodeT<float> { using type = float4; };
template <> struct NodeT<double> { using type = double4; };

// kAtomSum: a subtree of LEAF and ADD ops only (e.g. bulge + disk), whose cotangent passes
// unchanged to each of its leaves.
enum { kAtomRange = 0, kAtomPhase = 1, kAtomScale = 2, kAtomSum = 3 };

// want bits: leaf l = bit l, phase p = bit 8 + p, scale q = bit 16 + q.
__device__ __forceinline__ bool want_leaf(unsigned want, int l) { return (want >> l) & 1u; }
__device__ __forceinline__ bool want_phase(unsigned want, int p) { return (want >> (8 + p)) & 1u; }
__device__ __forceinline__ bool want_scale(unsigned want, int q) { return (want >> (16 + q)) & 1u; }

// The factor list of a template (host).
inline void plan_factors(const gsb_template& tpl, FactorPlan& P)
{
    short c1[GSB_MAX_OPS], c2[GSB_MAX_OPS], start[GSB_MAX_OPS], st[GSB_MAX_OPS];
    int sp = 0;
    P.n = 0;
    P.depth = 0;
    for (int o = 0; o < tpl.n_ops; ++o) {
        const int code = tpl.op_code[o];
        c1[o] = c2[o] = -1;
        if (code == GSB_OP_LEAF) {
            start[o] = short(o);
            st[sp++] = short(o);
        } else if (code == GSB_OP_MUL || code == GSB_OP_ADD) {
            c2[o] = st[--sp];
            c1[o] = st[sp - 1];
            start[o] = start[c1[o]];
            st[sp - 1] = short(o);
        } else {
            c1[o] = st[sp - 1];
            start[o] = start[c1[o]];
            st[sp - 1] = short(o);
        }
        P.depth = std::max(P.depth, sp);
    }
    sp = 0;
    st[sp++] = short(tpl.n_ops - 1);
    while (sp > 0) {
        const int o = st[--sp];
        const int code = tpl.op_code[o];
        if (code == GSB_OP_MUL) {
            st[sp++] = c1[o];
            st[sp++] = c2[o];
            continue;
        }
        const int f = P.n++;
        P.o0[f] = short(o);
        P.o1[f] = short(o + 1);
        P.arg[f] = (unsigned char)tpl.op_arg[o];
        if (code == GSB_OP_PHASE || code == GSB_OP_SCALE) {
            P.kind[f] = code == GSB_OP_PHASE ? kFactorPhase : kFactorScale;
            st[sp++] = c1[o];
        } else if (code == GSB_OP_LEAF) {
            P.kind[f] = kFactorLeaf;
        } else {
            bool sum = true;
            for (int q = start[o]; q <= o && sum; ++q)
                sum = tpl.op_code[q] == GSB_OP_LEAF || tpl.op_code[q] == GSB_OP_ADD;
            P.o0[f] = start[o];
            P.kind[f] = sum ? kFactorSum : kFactorTree;
        }
    }
}

// Sort the factors into atoms and folded separable ones (thread 0).  A leaf is separable when its
// value is X(i) Y(j) (Box or Gaussian with a diagonal Jacobian: the reference's 1-d fill).  Factors
// named in `want` (the adjoint's differentiated records) are not folded: a wanted separable leaf
// stays a leaf atom, a wanted phase or scale becomes an atom of its own.
__device__ inline void plan_factored(StampSmem& S, const gsb_template& tpl, const FactorPlan& P, unsigned want = 0u)
{
    int n = 0, nl = 0, no = 0;
    for (int f = 0; f < P.n; ++f) {
        const int kind = P.kind[f], arg = P.arg[f];
        if (kind == kFactorPhase && !want_phase(want, arg)) { S.phase_sep[arg] = 1; continue; }
        if (kind == kFactorScale && !want_scale(want, arg)) { S.scale_sep[arg] = 1; continue; }
        if (kind == kFactorLeaf && !want_leaf(want, arg)) {
            const LeafParams& L = S.leaf[arg];
            if ((L.type == GSB_BOX || L.type == GSB_GAUSSIAN) && !(L.flags & GSB_LEAF_JAC_GENERAL)) {
                S.leaf_sep[arg] = 1;
                continue;
            }
        }
        S.atom_o0[n] = P.o0[f];
        S.atom_o1[n] = P.o1[f];
        S.atom_kind[n] = kind == kFactorPhase ? kAtomPhase : kind == kFactorScale ? kAtomScale
                         : kind == kFactorSum ? kAtomSum : kAtomRange;
        S.atom_arg[n] = (unsigned char)(kind == kFactorTree || kind == kFactorSum ? 0 : arg);
        bool real = kind == kFactorSum || kind == kFactorLeaf;
        for (int o = P.o0[f]; o < P.o1[f] && real; ++o)
            real = !(tpl.op_code[o] == GSB_OP_LEAF && tpl.leaf_type[tpl.op_arg[o]] == GSB_INTERPOLATED);
        if (real) {
            for (int o = P.o0[f]; o < P.o1[f]; ++o)
                if (tpl.op_code[o] == GSB_OP_LEAF) {
                    S.real_leaf[nl] = tpl.op_arg[o];
                    S.real_last[nl++] = 0;
                }
            S.real_last[nl - 1] = 1;
        } else {
            S.other[no++] = (unsigned char)n;
        }
        ++n;
    }
    S.n_atoms = n;
    S.n_real = nl;
    S.n_other = no;
}

// Trapezoid nodes of the Moffat sum (moffat_nodes).
constexpr int kMoffatNodes = 64;
constexpr double kMoffatTau = 0.25;

// Decide which factors of this stamp are cached in shared memory (thread 0), in order: the folded
// separable factors, Sersic spline nodes, phase factors, separable leaf factors, per-leaf tables, until
// the budget is used; image taps in what is left of the room.  What is not cached is evaluated in
// another form, so kernels that are to give the same bits plan with the same budget (form_budget).
template <typename T, bool II = true>
__device__ inline void plan_caches(StampSmem& S, const gsb_template& tpl, const FactorPlan& fac, int Nk,
                                   unsigned want = 0u, int budget = kCacheBytes, int room = 0)
{
    room = max(room, budget);
    const int hk = Nk / 2;
    int used = 0;
    S.regstack = fac.depth <= 4;
    S.xy_cache = -1;
    for (int l = 0; l < tpl.n_leaves; ++l) S.leaf_sep[l] = 0;
    for (int p = 0; p < tpl.n_phases; ++p) S.phase_sep[p] = 0;
    for (int q = 0; q < tpl.n_scales; ++q) S.scale_sep[q] = 0;
    {
        const int bytes = ((hk + 1 + Nk + 1) * (int)sizeof(Cx<T>) + 15) & ~15;
        if (S.regstack && bytes <= budget) {
            plan_factored(S, tpl, fac, want);
            S.xy_cache = used;
            used += bytes;
        }
    }
    for (int l = 0; l < tpl.n_leaves; ++l) {
        S.sersic_cache[l] = -1;
        S.leaf_cache[l] = -1;
        if (S.leaf[l].type == GSB_SERSIC) {
            const int bytes = (S.sersic[l].n * (int)sizeof(typename NodeT<T>::type) + 15) & ~15;
            if (used + bytes <= budget) { S.sersic_cache[l] = used; used += bytes; }
        }
    }
    for (int p = 0; p < tpl.n_phases; ++p) {
        S.phase_cache[p] = -1;
        if (S.phase_sep[p]) continue;
        const int bytes = ((hk + 1 + Nk + 1) * (int)sizeof(Cx<T>) + 15) & ~15;
        if (used + bytes <= budget) { S.phase_cache[p] = used; used += bytes; }
    }
    for (int l = 0; l < tpl.n_leaves; ++l) {
        const LeafParams& L = S.leaf[l];
        const bool sep = !(L.flags & GSB_LEAF_JAC_GENERAL) && (L.type == GSB_BOX || L.type == GSB_GAUSSIAN);
        if (!sep || S.leaf_sep[l]) continue;
        const int bytes = ((hk + 1 + Nk + 1) * (int)sizeof(T) + 15) & ~15;
        if (used + bytes <= budget) { S.leaf_cache[l] = used; used += bytes; }
    }
    for (int l = 0; l < tpl.n_leaves; ++l) {
        S.aux_cache[l] = -1;
        const LeafParams& L = S.leaf[l];
        int bytes = 0;
        if (L.type == GSB_EXPONENTIAL) bytes = ((Nk + 1) * (int)sizeof(ushort2) + 15) & ~15;
        else if (L.type == GSB_MOFFAT && sizeof(T) == 4 && int(L.d[2]) == 0) bytes = kMoffatNodes * (int)sizeof(float2);
        else if (L.type == GSB_SERSIC && sizeof(T) == 4 && want_leaf(want, l) && S.sersic_cache[l] >= 0)
            bytes = (S.sersic[l].n * (int)sizeof(float2) + 15) & ~15;
        else continue;
        if (hk < 65535 && used + bytes <= budget) { S.aux_cache[l] = used; used += bytes; }
    }
    // InterpolatedImage leaves with a diagonal Jacobian: the taps, weights and transform
    // factor of every column and row (the reference's separable fill caches the same per
    // column, SBInterpolatedImage.cpp:820-866).  Kept or not they are the same numbers, so they may
    // take what room there is.
    for (int l = 0; l < tpl.n_leaves; ++l) {
        S.ii_cache[l] = -1;
        const LeafParams& L = S.leaf[l];
        if (!II || L.type != GSB_INTERPOLATED || (L.flags & GSB_LEAF_JAC_GENERAL)) continue;
        const int bytes = ((hk + 1 + Nk + 1) * (int)sizeof(IITaps<T>) + 15) & ~15;
        if (used + bytes <= room) { S.ii_cache[l] = used; used += bytes; }
    }
}

template <typename T>
__device__ __forceinline__ LeafT<T>& leaf_const(StampSmem& S, int l)
{ return *reinterpret_cast<LeafT<T>*>(&S.leaf_t[l]); }
template <typename T>
__device__ __forceinline__ const LeafT<T>& leaf_const(const StampSmem& S, int l)
{ return *reinterpret_cast<const LeafT<T>*>(&S.leaf_t[l]); }

// The constants of leaf l in the working precision (one thread per leaf, after plan_caches).
//
// mixed: float arithmetic drawn into a double image (drawImage's default precision with an ImageD).  No
// rounding to a float pixel hides the arithmetic there, so every profile takes its general form, whose
// operations are correctly rounded and follow the reference's, and none the shared-constant forms with
// hardware approximations.
template <typename T>
__device__ __noinline__ void set_leaf_const(StampSmem& S, int l, double dk, bool mixed)
{
    const LeafParams& L = S.leaf[l];
    LeafT<T>& t = leaf_const<T>(S, l);
    t.kind = kLeafGeneric;
    t.cache = -1;
    t.n = 0;
    t.flux = T(L.flux);
    t.size = T(L.d[0]);
    double size = 1.;
    if (S.leaf_cache[l] >= 0) {
        t.kind = kLeafSep;
        t.cache = S.leaf_cache[l];
    } else if (L.type == GSB_EXPONENTIAL && S.aux_cache[l] >= 0 && sizeof(T) == 4 && !mixed) {
        t.kind = kLeafExpFast;
        t.cache = S.aux_cache[l];
        size = L.d[0];
    } else if (L.type == GSB_EXPONENTIAL && S.aux_cache[l] >= 0) {
        // (the general path's own order of operations: k = (i dk, j dk), then r0 squared)
        t.kind = kLeafExp;
        t.cache = S.aux_cache[l];
        t.q[0] = T(L.d[0]);
        t.q[1] = T(dk);
        t.a = T(L.jac[0]);
        t.b = T(L.jac[1]);
        t.c = T(L.jac[2]);
        t.d = T(L.jac[3]);
        return;
    } else if (L.type == GSB_SERSIC && S.sersic_cache[l] >= 0 && !(sizeof(T) == 4 && mixed)) {
        const SersicTableView& v = S.sersic[l];
        t.kind = kLeafSersic;
        t.cache = S.sersic_cache[l];
        t.n = v.n;
        size = L.d[0];
        t.q[0] = T(v.ksq_min);
        t.q[1] = T(v.ksq_max);
        t.q[2] = T(v.kderiv2);
        t.q[3] = T(v.kderiv4);
        t.q[4] = T(v.highk_a);
        t.q[5] = T(v.highk_b);
        t.q[6] = T(v.da);
        t.q[7] = T(1. / v.da);
        t.q[8] = T(0.34657359027997264 / v.da);          // node coordinate + 1/2: log2(k^2) q8 + q9
        t.q[9] = T(0.5 - v.front / v.da);
    } else if (L.type == GSB_MOFFAT) {
        const int mode = int(L.d[2]);
        size = L.d[0];
        t.flux = T(L.d[1]);
        if (mode >= 1 && mode <= 3 && sizeof(T) == 4 && !mixed) {
            t.kind = kLeafMoffat1 + mode - 1;
        } else if (mode == 0 && S.aux_cache[l] >= 0) {
            // terms a point at x needs: up to cosh t = 1 + B / x, B = 19 + nu ln 2B bounding the rest by 2e-9 of
            // the sum.  The smallest x of the grid sets the node count.
            const float nu = float(L.d[3]);
            float B = 20.f;
            for (int it = 0; it < 6; ++it) B = 19.f + nu * __logf(2.f * B);
            const float j0 = float(L.jac[0]), j1 = float(L.jac[1]), j2 = float(L.jac[2]), j3 = float(L.jac[3]);
            const float det = fabsf(j0 * j3 - j1 * j2);
            const float fro = sqrtf(j0 * j0 + j1 * j1 + j2 * j2 + j3 * j3);
            const float xmin = float(dk * size) * det / fro;      // <= dk rD times the smaller singular value
            const float tend = __logf(2.f + 2.f * B / xmin);
            const int need = int(tend * float(1. / kMoffatTau)) + 2;
            // the weights cosh(nu t) stay within FP32, and the nodes within the cache
            if (!mixed && xmin > 0.f && need <= kMoffatNodes && nu * tend < 80.f) {
                t.kind = kLeafMoffatSum;
                t.cache = S.aux_cache[l];
                t.n = need;
                t.q[0] = T(nu);
                t.q[1] = T(2.f * B);
            }
        }
    } else if (L.type == GSB_KOLMOGOROV && sizeof(T) == 4 && !mixed) {
        t.kind = kLeafKolm;
        size = L.d[0];
    } else if (L.type == GSB_AIRY && sizeof(T) == 4 && !mixed) {
        t.kind = kLeafAiry;
        size = L.d[0];
        t.flux = T(L.d[1]);
        t.q[0] = T(L.d[2]);
        t.q[1] = T(L.d[3]);
    }
    size *= dk;
    t.a = T(L.jac[0] * size);
    t.b = T(L.jac[1] * size);
    t.c = T(L.jac[2] * size);
    t.d = T(L.jac[3] * size);
}

// Columns [lo, hi) of row j that survive the Exponential's clip (exponential_keep, which keeps a
// range of columns in every row).
static __device__ __noinline__ ushort2 exponential_columns(const LeafParams& L, double dk, int hk, int j)
{
    const double r0 = L.d[0], ksqmax = L.d[1], kmax = L.d[2];
    int i1, i2;
    if (!(L.flags & GSB_LEAF_JAC_GENERAL)) {
        const double A = L.jac[0], D = L.jac[3];
        const int jq = j < 0 ? -j : j;
        kvalue_range_1d(hk + 1, kmax, ksqmax, 0., dk * A * r0, jq * (dk * D * r0), i1, i2);
    } else {
        const double A = L.jac[0], B = L.jac[1], C = L.jac[2], D = L.jac[3];
        const double y0 = -hk * dk;
        const double kx0 = (C * y0) * r0 + (j + hk) * (C * dk * r0);
        const double ky0 = (D * y0) * r0 + (j + hk) * (D * dk * r0);
        kvalue_range_2d(hk + 1, kmax, ksqmax, kx0, A * dk * r0, ky0, B * dk * r0, i1, i2);
    }
    if (i1 >= i2) return make_ushort2(0, 0);
    return make_ushort2((unsigned short)(i1 < 0 ? 0 : i1), (unsigned short)(i2 > hk + 1 ? hk + 1 : i2));
}

// Node j of the Moffat sum: (log2(e) cosh t_j, w_j).
static __device__ __noinline__ float2 moffat_node(double nu, double lognorm, int j)
{
    const double t = j * kMoffatTau;
    const double w = 0.5 * kMoffatTau * (exp(lognorm + nu * t) + exp(lognorm - nu * t));
    return make_float2(float(cosh(t) * 1.4426950408889634), float(j == 0 ? 0.5 * w : w));
}

// Fill the planned caches (whole block).
template <typename T, bool II = true>
__device__ inline void fill_caches(StampSmem& S, const gsb_template& tpl, unsigned char* cache,
                                   double dk, int Nk, bool mixed = false)
{
    const int hk = Nk / 2;
    // (the last warp forms the constants and the one before it the Moffat nodes, while the first
    // ones start on the tables)
    const int back = int(blockDim.x) - 1 - int(threadIdx.x);
    if (back < tpl.n_leaves) set_leaf_const<T>(S, back, dk, mixed);
    for (int l = 0; l < tpl.n_leaves; ++l) {
        if (S.aux_cache[l] < 0) continue;
        const LeafParams& L = S.leaf[l];
        if (L.type == GSB_SERSIC) {
            // (filled by the adjoint, which knows the derivative tables)
        } else if (L.type == GSB_EXPONENTIAL) {
            ushort2* R = reinterpret_cast<ushort2*>(cache + S.aux_cache[l]);
            for (int t = threadIdx.x; t < Nk + 1; t += blockDim.x) R[t] = exponential_columns(L, dk, hk, t - hk);
        } else {
            // c_nu x^nu K_nu(x) = x^nu sum_j w_j exp(-x cosh t_j)  (moffat_kv), w_j = e^lognorm tau cosh(nu t_j)
            float2* E = reinterpret_cast<float2*>(cache + S.aux_cache[l]);
            for (int t = back - 32; t < kMoffatNodes; t += blockDim.x)
                if (t >= 0) E[t] = moffat_node(L.d[3], L.d[4], t);
        }
    }
    for (int l = 0; l < tpl.n_leaves; ++l) {
        if (II && S.ii_cache[l] >= 0) {
            const LeafParams& L = S.leaf[l];
            IITaps<T>* E = reinterpret_cast<IITaps<T>*>(cache + S.ii_cache[l]);
            for (int t = threadIdx.x; t < hk + 1 + Nk + 1; t += blockDim.x) {
                const bool isx = t <= hk;
                const int idx = isx ? t : t - (hk + 1) - hk;
                // k' as ii_kvalue forms it for a diagonal Jacobian (the zero terms are exact)
                const double kp = isx ? L.jac[0] * (idx * dk) : L.jac[3] * (idx * dk);
                ii_axis_taps<T>(L, kp, true, isx, E[t]);
            }
        }
        if (S.sersic_cache[l] >= 0) {
            typename NodeT<T>::type* dst = reinterpret_cast<typename NodeT<T>::type*>(cache + S.sersic_cache[l]);
            const double4* src = S.sersic[l].node;
            for (int i = threadIdx.x; i < S.sersic[l].n; i += blockDim.x) {
                const double4 v = src[i];
                dst[i].x = T(v.x); dst[i].y = T(v.y); dst[i].z = T(v.z); dst[i].w = T(v.w);
            }
        }
        if (S.leaf_cache[l] >= 0) {
            const LeafParams& L = S.leaf[l];
            T* X = reinterpret_cast<T*>(cache + S.leaf_cache[l]);
            T* Y = X + hk + 1;
            const bool box = L.type == GSB_BOX;
            const double ax = L.jac[0] * dk * (box ? L.d[0] : L.d[0]);
            const double ay = L.jac[3] * dk * (box ? L.d[1] : L.d[0]);
            for (int i = threadIdx.x; i < hk + 1 + Nk + 1; i += blockDim.x) {
                const bool isx = i <= hk;
                const int idx = isx ? i : i - (hk + 1) - hk;
                const T u = T(idx * (isx ? ax : ay));
                const T v = box ? sinc_ref<T>(u) : exp(T(-0.5) * u * u);
                if (isx) X[i] = v; else Y[i - (hk + 1)] = v;
            }
        }
    }
    if (S.xy_cache >= 0) {
        // XS[i] = prod over folded atoms of their kx factor (flux, fs and scales in XS),
        // YS[j + hk] = prod of their ky factor.
        Cx<T>* XS = reinterpret_cast<Cx<T>*>(cache + S.xy_cache);
        Cx<T>* YS = XS + hk + 1;
        for (int t = threadIdx.x; t < hk + 1 + Nk + 1; t += blockDim.x) {
            const bool isx = t <= hk;
            const int idx = isx ? t : t - (hk + 1) - hk;
            Cx<T> v = cx<T>(T(1), T(0));
            for (int l = 0; l < tpl.n_leaves; ++l) {
                if (!S.leaf_sep[l]) continue;
                const LeafParams& L = S.leaf[l];
                const bool box = L.type == GSB_BOX;
                const double ax = L.jac[0] * dk * L.d[0];
                const double ay = L.jac[3] * dk * (box ? L.d[1] : L.d[0]);
                const T u = T(idx * (isx ? ax : ay));
                T f = box ? sinc_ref<T>(u) : exp(T(-0.5) * u * u);
                if (isx) f *= T(L.flux);
                v = cscale<T>(v, f);
            }
            for (int p = 0; p < tpl.n_phases; ++p) {
                if (!S.phase_sep[p]) continue;
                double tt = idx * (isx ? S.phase_ax[p] : S.phase_ay[p]);
                tt -= rint(tt);
                T sn, cs;
                sincospi(T(-2. * tt), &sn, &cs);
                v = cmul<T>(v, cx<T>(cs, sn));
                if (isx) v = cscale<T>(v, T(S.phase[p].flux_scaling));
            }
            if (isx)
                for (int q = 0; q < tpl.n_scales; ++q)
                    if (S.scale_sep[q]) v = cscale<T>(v, T(S.scale[q]));
            if (isx) XS[t] = v; else YS[t - (hk + 1)] = v;
        }
    }
    for (int p = 0; p < tpl.n_phases; ++p) {
        if (S.phase_cache[p] < 0) continue;
        Cx<T>* PX = reinterpret_cast<Cx<T>*>(cache + S.phase_cache[p]);
        Cx<T>* PY = PX + hk + 1;
        for (int i = threadIdx.x; i < hk + 1 + Nk + 1; i += blockDim.x) {
            const bool isx = i <= hk;
            const int idx = isx ? i : i - (hk + 1) - hk;
            double tt = idx * (isx ? S.phase_ax[p] : S.phase_ay[p]);
            tt -= rint(tt);
            T sn, cs;
            sincospi(T(-2. * tt), &sn, &cs);
            if (isx) PX[i] = cx<T>(cs, sn); else PY[i - (hk + 1)] = cx<T>(cs, sn);
        }
    }
}

// Sersic FT from shared-memory nodes (same arithmetic as sersic_kvalue).
template <typename T>
__device__ inline T sersic_kvalue_smem(const SersicTableView& tb, const typename NodeT<T>::type* node, T ksq)
{
    if (ksq >= T(tb.ksq_max)) return (T(tb.highk_a) + T(tb.highk_b) / sqrt(ksq)) / ksq;
    if (ksq < T(tb.ksq_min)) return T(1) + ksq * (T(tb.kderiv2) + ksq * T(tb.kderiv4));
    const T lk = T(0.5) * log(ksq) - T(tb.front);
    const T inv_da = T(1. / tb.da);
    int i = int(ceil(lk * inv_da));
    if (i >= tb.n) i = tb.n - 1;
    if (i <= 0) i = 1;
    const typename NodeT<T>::type n0 = node[i - 1], n1 = node[i];
    // The offset from the upper node is 0.5 ln(k_i^2 / k^2), the log of a ratio near 1, and
    // the spacing is the table's: both accurate in FP32 (a difference of two logs of size ~10,
    // or of rounded node positions, would cost up to ~1e-6 of the value).  bb = h - aa keeps
    // the weights aa / h + bb / h summing to 1.
    const T h = T(tb.da);
    const T aa = T(0.5) * log(n1.w / ksq);
    const T bb = h - aa;
    const T num = mul_add(-((T(1) / T(6)) * aa * bb), mul_add(aa + h, n0.z, mul_rn(bb + h, n1.z)),
                          mul_add(aa, n0.y, mul_rn(bb, n1.y)));
    return num / h / ksq;
}

// Flush-to-zero hardware approximations (one instruction each: the accurate forms' scaling for
// denormal arguments and results is not needed, a k-value below 1e-38 being 0 of the flux).
__device__ __forceinline__ float fast_exp2(float x) { float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float fast_log2(float x) { float y; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float fast_rcp(float x) { float y; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float fast_rsqrt(float x) { float y; asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }
__device__ __forceinline__ float fast_sqrt(float x) { float y; asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y; }

// f / x, inv the hardware's reciprocal of x: its quotient corrected once by the exact residual (rounded
// once, as a division; inv alone is wrong by up to one ulp, f inv by two).
__device__ __forceinline__ float quotient(float f, float x, float inv)
{
    const float q = mul_rn(f, inv);
    return fmaf(fmaf(-q, x, f), inv, q);
}

// 1 / sqrt(x): the hardware's, after one Newton step.
__device__ __forceinline__ float refined_rsqrt(float x)
{
    const float s = fast_rsqrt(x);
    return fmaf(0.5f * s, fmaf(-mul_rn(x, s), s, 1.f), s);
}

// Sersic FT at V points from the shared-memory nodes (FP32).  One reciprocal of k^2 serves the node
// offset and the final quotient; the offset's logarithm is a series in the ratio's excess over 1 (an
// exact difference) where the table is fine enough for its degree; the interval comes from the
// hardware logarithm (a point within rounding of a node may take the neighbouring cubic, which
// agrees there to third order).  The offset enters as a share s of the spacing, so that the two nodes'
// weights add up to 1 whatever the spacing's rounding.  Against the general form (divisions, logf) the rms
// error of a float image is 0.85 times as large; with f inv in place of the quotient and weights aa / h and
// bb / h by a rounded 1 / h it was 1.3 to 1.5 times.
template <int V>
__device__ __forceinline__ void sersic_points(const LeafT<float>& L, const unsigned char* cache,
                                              const float (&ksq)[V], float (&out)[V])
{
    const float4* node = reinterpret_cast<const float4*>(cache + L.cache);
    const float kmin = L.q[0], kmax = L.q[1], h = L.q[6], inv_h = L.q[7], is = L.q[8], io = L.q[9];
    const int last = L.n - 1;
    const bool fine = h < 0.04f;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const float k2 = ksq[v];
        const float inv = fast_rcp(k2);
        // i = ceil of the node coordinate: the coordinate + 1/2 rounded by adding 1.5 * 2^23
        const int i = max(1, min(__float_as_int(fmaf(fast_log2(k2), is, io) + 12582912.f) - 0x4b400000, last));
        const float4 n0 = node[i - 1], n1 = node[i];
        const float e = (n1.w - k2) * inv;       // k_i^2 / k^2 - 1
        float aa;
        if (fine) {
            // ln(1 + e) / 2, |e| < 0.084: the series to e^8 (next term 1.2e-11)
            float p = fmaf(e, -1.f / 16.f, 1.f / 14.f);
            p = fmaf(e, p, -1.f / 12.f);
            p = fmaf(e, p, 0.1f);
            p = fmaf(e, p, -0.125f);
            p = fmaf(e, p, 1.f / 6.f);
            p = fmaf(e, p, -0.25f);
            p = fmaf(e, p, 0.5f);
            aa = e * p;
        } else {
            aa = mul_rn(0.5f, logf(n1.w * inv));
        }
        const float bb = h - aa;
        const float s = mul_rn(aa, inv_h);
        const float lin = fmaf(s, n0.y - n1.y, n1.y);
        float r = quotient(fmaf(s * bb * (-1.f / 6.f), fmaf(aa + h, n0.z, mul_rn(bb + h, n1.z)), lin), k2, inv);
        if (!(k2 >= kmin && k2 < kmax)) {
            if (k2 >= kmax) r = k2 <= 3e38f ? quotient(fmaf(L.q[5], refined_rsqrt(k2), L.q[4]), k2, inv) : 0.f;
            else r = fmaf(k2, fmaf(k2, L.q[3], L.q[2]), 1.f);
        }
        out[v] = r;
    }
}

// x^nu sum_j w_j exp(-x cosh t_j) at V points, x^2 given (1 at x = 0).
template <int V>
__device__ __forceinline__ void moffat_sum_points(const LeafT<float>& L, const unsigned char* cache,
                                                  const float (&xsq)[V], float (&out)[V])
{
    const float2* E = reinterpret_cast<const float2*>(cache + L.cache);
    float sum[V], x[V], xs = 1e30f;
#pragma unroll
    for (int v = 0; v < V; ++v) {
        sum[v] = 0.f;
        x[v] = sqrtf(xsq[v]);
        if (x[v] > 0.f) xs = fminf(xs, x[v]);
    }
    // the smallest x of the V needs the most nodes: cosh t up to 1 + B / x
    const float need = fast_log2(fmaf(L.q[1], fast_rcp(xs), 2.f)) * float(0.6931471805599453 / kMoffatTau);
    const int nj = min(L.n, int(need) + 2);
    for (int j = 0; j < nj; ++j) {
        const float2 e = E[j];
#pragma unroll
        for (int v = 0; v < V; ++v) sum[v] = fmaf(e.y, fast_exp2(-x[v] * e.x), sum[v]);
    }
#pragma unroll
    for (int v = 0; v < V; ++v) out[v] = x[v] > 0.f ? sum[v] * exp2f(L.q[0] * log2f(x[v])) : 1.f;
}

// Real leaf l at the V points (i, j0 + v js) with the shared-memory caches: out[] times the returned factor.
template <typename T, int V>
__device__ __forceinline__ T leaf_points(const StampSmem& S, const unsigned char* cache, int l, int i, int j0,
                                            int js, int hk, double dk, T (&out)[V])
{
    const LeafT<T>& L = leaf_const<T>(S, l);
    const int kind = L.kind;
    if (kind == kLeafGeneric) {
        const GridRef g{dk, 0, -hk, hk + 1, 2 * hk + 1};
        const T kx = T(i) * T(dk);
#pragma unroll 1
        for (int v = 0; v < V; ++v) {
            const int j = j0 + v * js;
            const T val = leaf_kvalue<T>(S.leaf[l], S.sersic, kx, T(j) * T(dk), g, i, j + hk);
#pragma unroll
            for (int w = 0; w < V; ++w) if (w == v) out[w] = val;
        }
        return T(1);
    }
    const T flux = L.flux;
    if (kind == kLeafSep) {
        const T* X = reinterpret_cast<const T*>(cache + L.cache);
        const T x = flux * X[i];
#pragma unroll
        for (int v = 0; v < V; ++v) out[v] = x * X[hk + 1 + hk + j0 + v * js];
        return T(1);
    }
    const T jf = T(j0), jd = T(js);
    if constexpr (sizeof(T) == 8) {
        // (double: the remaining kinds gain nothing over the general path but its conversions)
        if (kind == kLeafSersic) {
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const T j = jf + T(v) * jd, u = mul_add(L.c, j, mul_rn(L.a, T(i))), w = mul_add(L.d, j, mul_rn(L.b, T(i)));
                out[v] = flux * sersic_kvalue_smem<T>(
                                    S.sersic[l], reinterpret_cast<const typename NodeT<T>::type*>(cache + L.cache),
                                    mul_add(u, u, mul_rn(w, w)));
            }
            return T(1);
        }
    }
    if (kind == kLeafExp) {
        // flux / (1 + k^2 r0^2)^(3/2) where the clip keeps it
        const ushort2* R = reinterpret_cast<const ushort2*>(cache + L.cache) + hk + j0;
        const T r0 = L.q[0], tdk = L.q[1], kx = T(i) * tdk;
        const T A = L.a, B = L.b, C = L.c, D = L.d;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const ushort2 r = R[v * js];
            const T ky = (jf + T(v) * jd) * tdk;
            const T u = mul_add(A, kx, mul_rn(C, ky)), w = mul_add(B, kx, mul_rn(D, ky));
            const T q = mul_add(mul_add(u, u, mul_rn(w, w)) * r0, r0, T(1));
            const T val = flux / (q * sqrt(q));
            out[v] = i >= int(r.x) && i < int(r.y) ? val : T(0);
        }
        return T(1);
    }
    if constexpr (sizeof(T) == 4) {
        float ksq[V];
        {
            const float ui = mul_rn(L.a, float(i)), wi = mul_rn(L.b, float(i)), c = L.c, d = L.d;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const float j = jf + float(v) * jd;
                const float u = mul_add(c, j, ui), w = mul_add(d, j, wi);
                ksq[v] = mul_add(u, u, mul_rn(w, w));
            }
        }
        if (kind == kLeafSersic) {
            sersic_points<V>(L, cache, ksq, out);
        } else if (kind == kLeafExpFast) {
            // (1 + k^2)^(-3/2) where the clip keeps it
            const ushort2* R = reinterpret_cast<const ushort2*>(cache + L.cache) + hk + j0;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const ushort2 r = R[v * js];
                const float s = fast_rsqrt(1.f + ksq[v]);
                out[v] = i >= int(r.x) && i < int(r.y) ? s * s * s : 0.f;
            }
        } else if (kind == kLeafKolm) {
            // exp(-(k^2)^(5/6)), the power as k^2 times its -1/6th power r, whose error is a sixth of the
            // logarithm's and is then taken out by a Newton step on r^6 k^2 = 1 (the general form's power
            // has 5/6 of the logarithm's: 1e-7 at k^2 = 4).  Below 1e-30 the value is 1, above 1e30 0; a NaN stays.
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const float k2 = ksq[v], x = k2 < 1e-30f ? 1e-30f : k2 > 1e30f ? 1e30f : k2;
                const float r = fast_exp2(fast_log2(x) * (-1.f / 6.f)), r3 = mul_rn(mul_rn(r, r), r);
                const float y = mul_rn(x, fmaf(mul_rn(r, 1.f / 6.f), fmaf(-mul_rn(x, r3), r3, 1.f), r));
                out[v] = expf(-y);
            }
        } else if (kind == kLeafMoffatSum) {
            moffat_sum_points<V>(L, cache, ksq, out);
        } else if (kind == kLeafAiry) {
#pragma unroll 1
            for (int v = 0; v < V; ++v) {
                float k2 = ksq[0];
#pragma unroll
                for (int w = 1; w < V; ++w) if (w == v) k2 = ksq[w];
                const float val = airy_kvalue<float>(k2, L.q[0], L.q[1]);
#pragma unroll
                for (int w = 0; w < V; ++w) if (w == v) out[w] = val;
            }
        } else {
            // Moffat beta = 1.5, 2.5, 3.5: exp(-k) times 1, 1 + k, 1 + k + k^2 / 3
            const float c1 = kind == kLeafMoffat1 ? 0.f : 1.f, c2 = kind == kLeafMoffat3 ? 1.f / 3.f : 0.f;
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const float k = sqrtf(ksq[v]);
                out[v] = expf(-k) * (1.f + k * (c1 + k * c2));
            }
        }
    }
    return flux;
}

// One leaf at k index (i, j) with the shared-memory caches.
template <typename T>
__device__ __noinline__ T leaf_fast(const StampSmem& S, const unsigned char* cache, int arg, int i, int j, int hk,
                                    double dk)
{
    T out[1];
    const T f = leaf_points<T, 1>(S, cache, arg, i, j, 0, hk, dk, out);
    return mul_rn(out[0], f);
}

// One leaf as a complex value: InterpolatedImage leaves are complex, the others real.  INL: compiled
// into the caller.
template <typename T, bool II = true, bool INL = false>
__device__ __forceinline__ Cx<T> leaf_cfast(const StampSmem& S, const unsigned char* cache, int arg, int i, int j,
                                            const GridRef& g)
{
    if (II && S.leaf[arg].type == GSB_INTERPOLATED) {
        if (S.ii_cache[arg] >= 0) {
            const IITaps<T>* E = reinterpret_cast<const IITaps<T>*>(cache + S.ii_cache[arg]);
            const int hk = g.n / 2;
            return ii_sum<T>(S.leaf[arg], E[i], E[hk + 1 + j + hk]);
        }
        return ii_kvalue<T>(S.leaf[arg], g.dk, i, j);
    }
    if constexpr (INL) {
        T out[1];
        const T f = leaf_points<T, 1>(S, cache, arg, i, j, 0, g.n / 2, g.dk, out);
        return cx<T>(mul_rn(out[0], f), T(0));
    }
    return cx<T>(leaf_fast<T>(S, cache, arg, i, j, g.n / 2, g.dk), T(0));
}

// Evaluation of the ops [o0, o1) (a complete subtree, or the whole program) with the caches and
// a 4-deep register stack (warp-uniform branches).
template <typename T, bool II = true>
__device__ __noinline__ Cx<T> eval_range(const gsb_template& tpl, const StampSmem& S,
                                            const unsigned char* cache, double dk, int i, int j,
                                            const GridRef& g, int o0, int o1)
{
    const int hk = g.n / 2;
    Cx<T> s0 = cx<T>(T(0), T(0)), s1 = s0, s2 = s0, s3 = s0;
    int sp = 0;
    for (int o = o0; o < o1; ++o) {
        const int code = tpl.op_code[o], arg = tpl.op_arg[o];
        if (code == GSB_OP_LEAF) {
            const Cx<T> c = leaf_cfast<T, II>(S, cache, arg, i, j, g);
            if (sp == 0) s0 = c; else if (sp == 1) s1 = c; else if (sp == 2) s2 = c; else s3 = c;
            ++sp;
        } else if (code == GSB_OP_MUL || code == GSB_OP_ADD) {
            --sp;
            const bool mul = code == GSB_OP_MUL;
            if (sp == 1) s0 = mul ? cmul_yx<T>(s0, s1) : cadd<T>(s0, s1);
            else if (sp == 2) s1 = mul ? cmul_yx<T>(s1, s2) : cadd<T>(s1, s2);
            else s2 = mul ? cmul_yx<T>(s2, s3) : cadd<T>(s2, s3);
        } else {
            Cx<T> f;
            if (code == GSB_OP_PHASE) {
                const T fs = T(S.phase[arg].flux_scaling);
                if (S.phase_cache[arg] >= 0) {
                    const Cx<T>* PX = reinterpret_cast<const Cx<T>*>(cache + S.phase_cache[arg]);
                    f = cscale<T>(cmul_yx<T>(PX[i], PX[hk + 1 + j + hk]), fs);
                } else {
                    double tt = i * S.phase_ax[arg] + j * S.phase_ay[arg];
                    tt -= rint(tt);
                    T sn, cs;
                    sincospi(T(-2. * tt), &sn, &cs);
                    f = cx<T>(fs * cs, fs * sn);
                }
            } else {
                f = cx<T>(T(S.scale[arg]), T(0));
            }
            if (sp == 1) s0 = cmul_yx<T>(s0, f);
            else if (sp == 2) s1 = cmul_yx<T>(s1, f);
            else if (sp == 3) s2 = cmul_yx<T>(s2, f);
            else s3 = cmul_yx<T>(s3, f);
        }
    }
    return s0;
}

// The factored program at the V points (i, j0 + v js): the folded separable factors XS[i] YS[j + hk]
// times the atoms.  Taking V points through each atom at a time shares the program's control flow
// and the atoms' constants, and gives the latencies V independent chains to overlap.  The value of point v is
// handed to fold(v, z, r) as a complex z and a real factor r, which the fold multiplies in (kahan_add).
template <typename T, int V> struct Values { Cx<T> v[V]; T r[V]; };

template <typename T, bool II, int V, class Fold>
__device__ __forceinline__ void eval_points_fold(const gsb_template& tpl, const StampSmem& S, const unsigned char* cache,
                                                 int i, int j0, int js, int hk, double dk, const Fold& fold)
{
    T r[V], sum[V];
#pragma unroll
    for (int v = 0; v < V; ++v) { r[v] = T(1); sum[v] = T(0); }
    const int nr = S.n_real;
#pragma unroll 1
    for (int q = 0; q < nr; ++q) {
        T t[V];
        const T f = leaf_points<T, V>(S, cache, S.real_leaf[q], i, j0, js, hk, dk, t);
        const bool last = S.real_last[q];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            sum[v] = mul_add(t[v], f, sum[v]);
            if (last) { r[v] *= sum[v]; sum[v] = T(0); }
        }
    }
    const Cx<T>* XS = reinterpret_cast<const Cx<T>*>(cache + S.xy_cache);
    const Cx<T>* YS = XS + hk + 1 + hk + j0;
    const Cx<T> x = XS[i];
    const int no = S.n_other;
    if (no == 0) {
#pragma unroll
        for (int v = 0; v < V; ++v) fold(v, cmul_yx<T>(x, YS[v * js]), r[v]);
        return;
    }
    const GridRef g{dk, 0, -hk, hk + 1, 2 * hk + 1};
#pragma unroll 1
    for (int v = 0; v < V; ++v) {
        const int j = j0 + v * js;
        Cx<T> c = cx<T>(T(1), T(0));
        for (int q = 0; q < no; ++q) {
            const int a = S.other[q], o0 = S.atom_o0[a], o1 = S.atom_o1[a];
            c = cmul<T>(c, o1 - o0 == 1 ? leaf_cfast<T, II>(S, cache, S.atom_arg[a], i, j, g)
                                        : eval_range<T, II>(tpl, S, cache, dk, i, j, g, o0, o1));
        }
        const Cx<T> z = cmul<T>(c, cmul_yx<T>(x, YS[v * js]));
#pragma unroll
        for (int w = 0; w < V; ++w) if (w == v) fold(w, z, r[w]);
    }
}

template <typename T, bool II, int V>
__device__ __noinline__ Values<T, V> eval_points(const gsb_template& tpl, const StampSmem& S,
                                                 const unsigned char* cache, int i, int j0, int js, int hk, double dk)
{
    Values<T, V> res;
    eval_points_fold<T, II, V>(tpl, S, cache, i, j0, js, hk, dk, [&](int v, Cx<T> z, T r) { res.v[v] = z; res.r[v] = r; });
    return res;
}

// V points of the program to fold(v, z, r), by the best of its three forms.  INL: compiled into the caller
// (else a function call per V points, so that the kernels of all sizes share one compiled body).
template <typename T, bool II, int V, bool INL, class Fold>
__device__ __forceinline__ void eval_any(const gsb_template& tpl, const StampSmem& S, const unsigned char* cache, int i,
                                         int j0, int js, int hk, double dk, const Fold& fold)
{
    if (S.xy_cache >= 0) {
        if constexpr (INL) {
            eval_points_fold<T, II, V>(tpl, S, cache, i, j0, js, hk, dk, fold);
        } else {
            const Values<T, V> z = eval_points<T, II, V>(tpl, S, cache, i, j0, js, hk, dk);
#pragma unroll
            for (int v = 0; v < V; ++v) fold(v, z.v[v], z.r[v]);
        }
        return;
    }
    const GridRef g{dk, 0, -hk, hk + 1, 2 * hk + 1};
#pragma unroll 1
    for (int v = 0; v < V; ++v) {
        const Cx<T> z = S.regstack ? eval_range<T, II>(tpl, S, cache, dk, i, j0 + v * js, g, 0, tpl.n_ops)
                                   : eval_program<T, II>(tpl, S, dk, i, j0 + v * js, g);
#pragma unroll
        for (int w = 0; w < V; ++w) if (w == v) fold(w, z, T(1));
    }
}

template <typename T, bool II, bool INL = false>
__device__ __forceinline__ Values<T, 1> eval_point(const gsb_template& tpl, const StampSmem& S, const unsigned char* cache,
                                            int i, int j, int hk, double dk)
{
    Values<T, 1> res;
    eval_any<T, II, 1, INL>(tpl, S, cache, i, j, 0, hk, dk, [&](int, Cx<T> z, T r) { res.v[0] = z; res.r[0] = r; });
    return res;
}

// acc += v r (conjugated where not pos) with Kahan's compensation term comp, componentwise.  The real
// part's product is not rounded before the compensation is taken off; the imaginary part's is.
template <typename T>
__device__ __forceinline__ void kahan_add(Cx<T>& acc, Cx<T>& comp, Cx<T> v, T r, bool pos)
{
    const T vy = mul_rn(v.y, r);
    const T yx = mul_add(v.x, r, -comp.x), yy = add_rn(pos ? vy : -vy, -comp.y);
    const T tx = acc.x + yx, ty = acc.y + yy;
    comp.x = (tx - acc.x) - yx;
    comp.y = (ty - acc.y) - yy;
    acc.x = tx;
    acc.y = ty;
}

template <typename T>
__device__ inline void store_pixel(void* out, int dtype, int add, long long idx, T v)
{
    if (dtype == GSB_F32) {
        float* o = reinterpret_cast<float*>(out) + idx;
        *o = add ? *o + float(v) : float(v);
    } else {
        double* o = reinterpret_cast<double*>(out) + idx;
        *o = add ? *o + double(v) : double(v);
    }
}

template <typename T, int N>
constexpr size_t smem_bytes(bool wsmem)
{
    size_t off = (sizeof(StampSmem) + 15) & ~size_t(15);
    off += sizeof(Cx<T>) * N * (1 + fused_warps<T, N>());
    if (wsmem) off += sizeof(Cx<T>) * (N / 2 + 1) * (N + 1);
    return ((off + 15) & ~size_t(15)) + form_budget<T>(N);
}

template <typename T, int N>
constexpr bool w_fits_smem()
{
    return smem_bytes<T, N>(true) <= kSmemLimit;
}

// Resident CTAs per SM that the shared memory allows (at most 2): the register budget is
// capped to match, so that code used only by some programs (the FP64 transform of image
// leaves, the general-Jacobian paths) cannot halve the occupancy of every other program.
constexpr size_t kSmemPerSM = 228 * 1024;

template <typename T, int N>
__host__ __device__ constexpr int fused_min_blocks()
{
    return kSmemPerSM / (smem_bytes<T, N>(w_fits_smem<T, N>()) + 1024) >= 2 ? 2 : 1;
}

// Bound by instruction issue and its latencies, with the 16 warps an SM that 128 registers leave: the
// k-space evaluation is half the instructions, the FFTs a sixth.  686 catalog stamps (Sersic x
// Kolmogorov) at N = 128: 222 us with the evaluator as a call and each FFT in its buffer, 182 with the
// evaluator of the float kernels compiled in place (its callers' registers need not be saved), the
// column FFT's last pass writing W and the rows' first reading it; N = 192 100 -> 89.  (Compiled in
// place for the double and image kernels, or a row FFT that writes pixels from its last pass, it
// spills: 239 us.)  Before both, one wave vector a lane with constants converted from the FP64
// records at each: bulge + disk x Moffat (general beta), 16384 stamps, N = 128 5.4 ms and N = 192 14.6
// against 2.9 and 6.0 with the calls.
template <typename T, int N, bool WSMEM, bool II = true>
__global__ void __launch_bounds__(fused_warps<T, N>() * 32, fused_min_blocks<T, N>()) draw_fused_kernel(const __grid_constant__ DrawArgs a)
{
    constexpr int NW = fused_warps<T, N>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int H = N / 2 + 1;
    constexpr int WS = N + 1;   // column stride of W (padding against bank conflicts)
    StampSmem& S = *reinterpret_cast<StampSmem*>(smem_raw);
    size_t off = (sizeof(StampSmem) + 15) & ~size_t(15);
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

    for (int s = blockIdx.x; s < a.n_stamps; s += gridDim.x) {
        __syncthreads();
        load_stamp(S, a.tpl, s, a.leaves, a.phases, a.scales, a.stamps, a.sersic_header,
                   a.sersic_node, a.sersic_stride, 1. / N);
        __syncthreads();
        const int Nk = S.geom.Nk;
        const int hk = Nk / 2;
        if (threadIdx.x == 0) plan_caches<T, II>(S, a.tpl, a.fac, Nk, 0u, form_budget<T>(N));
        __syncthreads();
        fill_caches<T, II>(S, a.tpl, cache, dk, Nk, sizeof(T) == 4 && a.out_dtype == GSB_F64);
        __syncthreads();

        // ---- column phase: wrapped k-values, inverse DFT along ky ----
        if constexpr (N % 32 == 0) {
            // A column's Nk + 1 rows ky = -hk .. hk go to the lanes in order, 32 a slot.  N is a multiple
            // of 32, so slots s, s + N/32, ... of a lane are the aliases of one wrapped row: the lane
            // folds them (with Kahan compensation) in registers, and a column costs
            // ceil((Nk + 1) / 32) slots.  When Nk is a multiple of 32 (Nk = N above all) the last slot
            // would hold the single point ky = hk: up to Nk = N, where a column has one alias in kx (but for
            // c = N / 2, which has a slot for them), those points of all the warp's columns are taken
            // together, one column a lane, before its columns, and folded in their turn.
            constexpr int NS = N / 32;
            constexpr int V = sizeof(T) == 8 ? (NS % 2 == 0 ? 2 : 1) : NS % 4 == 0 ? 4 : NS % 3 == 0 ? 3 : NS;
            constexpr int COLS = (H + NW - 1) / NW;
            const bool edge = COLS <= 32 && Nk % 32 == 0 && Nk <= N;
            Cx<T> edge_val = cx<T>(T(0), T(0));
            if (edge) {
                const int c = warp + lane * NW;
                if (c <= hk && c + c < N) {
                    const Values<T, 1> z = eval_point<T, II>(a.tpl, S, cache, c, hk, hk, dk);
                    edge_val = cscale<T>(z.v[0], z.r[0]);
                }
                __syncwarp();
            }
            int q = 0;
            for (int c = warp; c < H; c += NW, ++q) {
                const int kx0 = c + ceil_div(-hk - c, N) * N;
                const bool has_edge = edge && c <= hk && c + c < N;
                const int top = has_edge ? hk - 1 : hk;
                const int edge_slot = has_edge ? (Nk % N) / 32 : -1;
                for (int s0 = 0; s0 < NS; s0 += V) {
                    Cx<T> acc[V], comp[V];
#pragma unroll
                    for (int v = 0; v < V; ++v) acc[v] = comp[v] = cx<T>(T(0), T(0));
                    bool first = true;       // a lane's first value needs no compensation
                    for (int kx = kx0; kx <= hk; kx += N) {
                        const bool pos = kx >= 0;
                        const int ii = pos ? kx : -kx;
                        for (int e0 = -hk + 32 * s0; e0 <= top; e0 += N) {
                            if (e0 + 32 * V - 1 <= top) {
                                const int ky = e0 + lane;
                                eval_any<T, II, V, !II && sizeof(T) == 4>(
                                    a.tpl, S, cache, ii, pos ? ky : -ky, pos ? 32 : -32, hk, dk, [&](int v, Cx<T> z, T r) {
                                        if (first) {
                                            acc[v] = cscale<T>(z, r);
                                            if (!pos) acc[v].y = -acc[v].y;
                                        } else {
                                            kahan_add<T>(acc[v], comp[v], z, r, pos);
                                        }
                                    });
                                first = false;
                            } else {
                                // the last, partial slots of the column (lanes beyond it repeat its end)
#pragma unroll 1
                                for (int u = 0; u < V && e0 + 32 * u <= top; ++u) {
                                    const int ky = e0 + 32 * u + lane, kc = min(ky, top);
                                    const Values<T, 1> z = eval_point<T, II>(a.tpl, S, cache, ii, pos ? kc : -kc, hk, dk);
#pragma unroll
                                    for (int v = 0; v < V; ++v)
                                        if (v == u && ky <= top) kahan_add<T>(acc[v], comp[v], z.v[0], z.r[0], pos);
                                }
                                first = false;
                            }
                        }
                        if (edge_slot >= s0 && edge_slot < s0 + V) {
                            const Cx<T> e = cx<T>(__shfl_sync(0xffffffffu, edge_val.x, q), __shfl_sync(0xffffffffu, edge_val.y, q));
#pragma unroll
                            for (int v = 0; v < V; ++v)
                                if (lane == 0 && s0 + v == edge_slot) kahan_add<T>(acc[v], comp[v], e, T(1), true);
                        }
                    }
#pragma unroll
                    for (int v = 0; v < V; ++v) buf[fft_slot(pmod(-hk + 32 * (s0 + v) + lane, N))] = acc[v];
                }
                __syncwarp();
                Cx<T>* Wc = W + (size_t)c * WS;
                warp_fft_io<T, N, +1, true, false>(buf, tw, [&](int i) { return buf[fft_slot(i)]; },
                                                   [&](int i, Cx<T> z) { Wc[i] = z; });
            }
        } else {
            for (int c = warp; c < H; c += NW) {
                const int kx0 = c + ceil_div(-hk - c, N) * N;
                for (int r = lane; r < N; r += 32) {
                    const int kyc = r < N / 2 ? r : r - N;
                    // the fold (wrap) of the aliases, with Kahan compensation
                    Cx<T> acc = cx<T>(T(0), T(0)), comp = acc;
                    for (int kx = kx0; kx <= hk; kx += N) {
                        const bool pos = kx >= 0;
                        for (int ky = kyc + ceil_div(-hk - kyc, N) * N; ky <= hk; ky += N) {
                            const Values<T, 1> z = eval_point<T, II>(a.tpl, S, cache, pos ? kx : -kx, pos ? ky : -ky, hk, dk);
                            kahan_add<T>(acc, comp, z.v[0], z.r[0], pos);
                        }
                    }
                    buf[fft_slot(r)] = acc;
                }
                __syncwarp();
                Cx<T>* Wc = W + (size_t)c * WS;
                warp_fft_io<T, N, +1, true, false>(buf, tw, [&](int i) { return buf[fft_slot(i)]; },
                                                   [&](int i, Cx<T> z) { Wc[i] = z; });
            }
        }
        __syncthreads();

        // ---- row phase: two image rows per complex transform ----
        const gsb_stamp& G = S.geom;
        const int npairs = (G.ny + 1) / 2;
        const int xstart = pmod(G.xmin, N);
        double fsum = 0., fcomp = 0.;
        for (int p = warp; p < npairs; p += NW) {
            const int py1 = G.ymin + 2 * p;
            const bool two = 2 * p + 1 < G.ny;
            const int y1 = pmod(py1, N), y2 = pmod(py1 + 1, N);
            const long long row1 = G.out_offset + (long long)(2 * p) * G.nx;
            // the transform reads the two rows from W
            auto load = [&](int kx) {
                const bool up = kx < H;
                const Cx<T>* w = W + (size_t)(up ? kx : N - kx) * WS;
                Cx<T> a1 = w[y1], a2 = two ? w[y2] : cx<T>(T(0), T(0));
                if (!up) { a1 = cconj<T>(a1); a2 = cconj<T>(a2); }
                return cx<T>(a1.x - a2.y, a1.y + a2.x);
            };
            warp_fft_io<T, N, +1, false, true>(buf, tw, load, [&](int i, Cx<T> z) { buf[fft_slot(i)] = z; });
#pragma unroll 1
            for (int i = lane; i < G.nx; i += 32) {
                int x = xstart + i;
                while (x >= N) x -= N;
                const Cx<T> v = buf[fft_slot(x)];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    if (r == 1 && !two) break;
                    const T px = (r ? v.y : v.x) * inv_n2;
                    store_pixel<T>(a.out, a.out_dtype, a.add, row1 + (r ? G.nx : 0) + i, px);
                    const double d = double(px);
                    // (a lane's ~100 float pixels add up exactly in FP64 but for a range beyond 2^22: the float
                    // fluxes are within 4e-16 of the exact sum of the pixels, as with compensation)
                    if (sizeof(T) == 4) {
                        fsum += d;
                    } else {                       // Neumaier compensated sum in FP64
                        const double tsum = fsum + d;
                        fcomp += fabs(fsum) >= fabs(d) ? (fsum - tsum) + d : (d - tsum) + fsum;
                        fsum = tsum;
                    }
                }
            }
            __syncwarp();
        }
        if (a.added_flux) {
            double v = fsum + fcomp;
            for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
            if (lane == 0) S.flux_part[warp] = v;
            __syncthreads();
            if (threadIdx.x == 0) {
                double tot = 0.;
                for (int w = 0; w < NW; ++w) tot += S.flux_part[w];
                a.added_flux[s] = tot;
            }
        }
    }
}

template <typename T>
__global__ void draw_kimage_kernel(const __grid_constant__ gsb_template tpl, int n_stamps, const gsb_leaf* leaves,
                                   const gsb_phase* phases, const double* scales,
                                   const double* sh, const double4* snode, int sstride, double dk,
                                   int kxmin, int kymin, int nkx, int nky, void* out, int dtype)
{
    __shared__ StampSmem S;
    const long long per = (long long)nkx * nky;
    for (int s = blockIdx.y; s < n_stamps; s += gridDim.y) {
        __syncthreads();
        load_stamp(S, tpl, s, leaves, phases, scales, nullptr, sh, snode, sstride, dk / (2. * kPi));
        __syncthreads();
        const GridRef g{dk, kxmin, kymin, nkx, nky};
        for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < per;
             p += (long long)gridDim.x * blockDim.x) {
            const int i = int(p % nkx), j = int(p / nkx);
            const Cx<T> v = eval_program<T>(tpl, S, dk, kxmin + i, kymin + j, g);
            const long long o = (s * per + p) * 2;
            if (dtype == GSB_F32) {
                reinterpret_cast<float*>(out)[o] = float(v.x);
                reinterpret_cast<float*>(out)[o + 1] = float(v.y);
            } else {
                reinterpret_cast<double*>(out)[o] = double(v.x);
                reinterpret_cast<double*>(out)[o + 1] = double(v.y);
            }
        }
    }
}

inline bool has_image_leaves(const gsb_template& tpl)
{
    for (int l = 0; l < tpl.n_leaves; ++l)
        if (tpl.leaf_type[l] == GSB_INTERPOLATED) return true;
    return false;
}

template <typename T, int N>
int draw_grid(int n_stamps)
{
    DeviceState* st = device_state();
    const size_t sm = smem_bytes<T, N>(w_fits_smem<T, N>());
    int per_sm = int(std::min<size_t>(kSmemLimit / sm, 4));
    if (per_sm < 1) per_sm = 1;
    return std::max(1, std::min(n_stamps, st->sm_count * per_sm));
}

template <typename T, int N>
size_t workspace_bytes_for(int n_stamps)
{
    if (w_fits_smem<T, N>()) return 0;
    return sizeof(Cx<T>) * (size_t)(N / 2 + 1) * (N + 1) * draw_grid<T, N>(n_stamps);
}

template <typename T, int N>
int launch_fused(const DrawArgs& args, size_t work_bytes, cudaStream_t stream)
{
    constexpr bool wsmem = w_fits_smem<T, N>();
    constexpr size_t sm = smem_bytes<T, N>(wsmem);
    int grid = draw_grid<T, N>(args.n_stamps);
    if (!wsmem && args.max_grid > 0) grid = std::min(grid, args.max_grid);
    else if (!wsmem && (args.work == nullptr || work_bytes < workspace_bytes_for<T, N>(args.n_stamps)))
        return set_error(GSB_ERR_INVALID, "draw workspace too small");
    // programs without image leaves run the instance compiled without their code
    if (has_image_leaves(args.tpl)) {
        GSB_CUDA_CHECK(cudaFuncSetAttribute(draw_fused_kernel<T, N, wsmem, true>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
        draw_fused_kernel<T, N, wsmem, true><<<grid, fused_warps<T, N>() * 32, sm, stream>>>(args);
    } else {
        GSB_CUDA_CHECK(cudaFuncSetAttribute(draw_fused_kernel<T, N, wsmem, false>,
                                            cudaFuncAttributeMaxDynamicSharedMemorySize, int(sm)));
        draw_fused_kernel<T, N, wsmem, false><<<grid, fused_warps<T, N>() * 32, sm, stream>>>(args);
    }
    GSB_CUDA_CHECK(cudaGetLastError());
    return GSB_OK;
}

}  // namespace gsb
