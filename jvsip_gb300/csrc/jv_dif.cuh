// jv_dif.cuh -- the in-place mixed-radix kernel: whole transforms of any
// length N = R1*R2*...*Rp (codelets 2..16) in shared memory, decimated in
// frequency.
//
// Pass 1 reads the view: the butterfly of n' (< S1 = N/R1) takes elements
// n' + r*S1, multiplies output k1 by exp(-2 pi i k1 n'/N) and stores it at
// k1*P1 + n'.  Pass p transforms the R_p sub-blocks of S_p elements inside
// every block of M_p = R_p*S_p = S_(p-1) elements, twiddles output k_p by
// exp(-2 pi i k_p n/M_p) and puts it back where it came from.  The last pass
// (S = 1) writes the view: butterfly q = k1 + R1*(k2 + R2*(k3 ...)) holds
// outputs q + r*N/R_last.
//
// Every butterfly reads and writes the same R places, so a pass is a plain
// loop over butterflies with one barrier after it (the self-sorting passes of
// k_smem hold every butterfly of a thread in registers between two barriers),
// a butterfly's addresses are computed once, and any thread count serves any
// radix.  The pitch P1 of the k1 blocks is the one of 16 paddings whose
// accesses collide least in the shared-memory banks (dif_schedule).
#pragma once

#include "jv_kernels.cuh"

namespace jv {

constexpr int kDifMaxPass = 8;

// A pass's constants, read from the arguments ...
struct DifPass {
    int R, S;            // radix; distance of a butterfly's elements inside a k1 block
    int NR, mstep;       // butterflies per transform N/R; M - S
    int NB1, two;        // butterflies per k1 block; start of the pass's twiddle table
    unsigned mNR, mNB1;  // multiply-high magic of NR, NB1
    unsigned mS, mR;     // of S, R
    __device__ __forceinline__ int by_NR(int x) const { return mdiv(x, mNR); }
    __device__ __forceinline__ int by_NB1(int x) const { return mdiv(x, mNB1); }
    __device__ __forceinline__ int by_S(int x) const { return mdiv(x, mS); }
    __device__ __forceinline__ int by_R(int x) const { return mdiv(x, mR); }
};
// ... or of a schedule known at compile time (DifFix)
template <class F, int I> struct DifFixPass {
    static constexpr int R = F::radix(I), S = F::S(I), NR = F::N / R, mstep = F::M(I) - S, NB1 = F::N / F::radix(0) / R,
                         two = F::two(I);
    __device__ __forceinline__ int by_NR(int x) const { return x / NR; }
    __device__ __forceinline__ int by_NB1(int x) const { return x / (NB1 > 0 ? NB1 : 1); }
    __device__ __forceinline__ int by_S(int x) const { return x / S; }
    __device__ __forceinline__ int by_R(int x) const { return x / R; }
};

template <typename T> struct DifArgs {
    typedef typename cplx_t<T>::t C;
    // transform v starts at in + v*vs_in; element n follows at n*es_in (es 1 for rows)
    const C *in;
    C *out;
    const T *in_re, *in_im;  // split complex views
    T *out_re, *out_im;
    long es_in, vs_in, es_out, vs_out, nvec;
    int N, np, vpb, lgv;     // transforms per CTA (2^lgv for column tiles)
    int P1, LD;              // pitch of a k1 block; of a transform (rows)
    unsigned smask_in, smask_out;  // 0x80000000: conjugate on load / store
    int has_scale;
    T scale;
    const C *tw;             // per-pass tables: pass p at p.two, entry k*S + n = exp(-2 pi i k n/M)
    // the steps of a long transform (DIF_STEP): group y of the grid starts
    // y*bvs_in / y*bvs_out elements on, and output k of its transform t is
    // multiplied by W^(g*k), g = t*tw_ts + y*tw_ys (none when tw_lo is null),
    // W^m = tw_lo[m & tw_mask] * tw_hi[m >> tw_sh]
    long bvs_in, bvs_out;
    const C *tw_lo, *tw_hi;
    unsigned tw_mask, tw_sh, tw_ts, tw_ys;
    const C *tv;             // DIF_VEC1, DIF_VEC2: output k of transform t times tv[k*tv_st + t]
    int tv_st;
    // DIF_R2CT: real element n of row t times tp_n[n*tp_n_st], then times
    // tp_t[t*tp_t_st], written back through wb; DIF_POWER: output k of transform
    // t stores (p, Im X), p = g_scale |X|^2 added to gram[t*g_vs + k*g_es]
    const T *tp_n, *tp_t;
    long tp_n_st, tp_t_st;
    C *wb;
    T *gram;
    long g_es, g_vs;
    T g_scale;
    const C *thalf;          // real transforms: exp(-+ i pi k/N), k <= N
    unsigned mH;             // and the magic of the pair passes' work items per transform
    DifPass p[kDifMaxPass];
};

// DIF_VEC1, DIF_VEC2, DIF_VECR: the passes over a single long vector
// (launch_vec_f32).  DIF_R2CT, DIF_POWER: the k-omega pipeline's tapered R2C
// rows into a column-major spectrum, and its transforms over the sensors with
// the power accumulator (kw.c komega()).
enum DifKind {
    DIF_C2C = 0, DIF_SPLIT = 1, DIF_R2C = 2, DIF_C2R = 3, DIF_STEP = 4, DIF_VEC1 = 5, DIF_VEC2 = 6, DIF_VECR = 7,
    DIF_R2CT = 8, DIF_POWER = 9
};
template <int KIND> constexpr bool dif_groups() { return KIND >= DIF_STEP && KIND <= DIF_VECR; }
// rows whose last pass stores with consecutive threads on adjacent transforms
template <int KIND> constexpr bool dif_rows_tf() { return KIND == DIF_VECR || KIND == DIF_R2CT; }

template <int KIND, typename T>
__device__ __forceinline__ typename cplx_t<T>::t dif_in(const DifArgs<T> &a, long e) {
    typedef typename cplx_t<T>::t C;
    if constexpr (KIND == DIF_SPLIT) return mk<C>(a.in_re[e], a.in_im[e]);
    else return a.in[e];
}
template <int KIND, typename T>
__device__ __forceinline__ void dif_out(const DifArgs<T> &a, long e, typename cplx_t<T>::t c) {
    if constexpr (KIND == DIF_SPLIT) {
        a.out_re[e] = c.x;
        a.out_im[e] = c.y;
    } else {
        a.out[e] = c;
    }
}

// Schedules: the passes from the arguments (any length) ...
struct DifDyn {
    static constexpr int V = 0;  // transforms per column tile: from the arguments
    template <typename T> static __device__ __forceinline__ const DifPass &first(const DifArgs<T> &a) { return a.p[0]; }
    template <typename T> static __device__ __forceinline__ const DifPass &last(const DifArgs<T> &a) {
        return a.p[a.np - 1];
    }
    template <typename T> static __device__ __forceinline__ int P1(const DifArgs<T> &a) { return a.P1; }
    // position of butterfly q = k1 + R1*(k2 + R2*(...)) of the last pass
    template <typename T> static __device__ __forceinline__ int pos(const DifArgs<T> &a, int q) {
        int rem = mdiv(q, a.p[0].mR);
        int pos = (q - rem * a.p[0].R) * a.P1;
        for (int i = 1; i + 1 < a.np; i++) {
            const int n = mdiv(rem, a.p[i].mR);
            pos += (rem - n * a.p[i].R) * a.p[i].S;
            rem = n;
        }
        return pos;
    }
};
// ... or radices Rs and block pitch P known at compile time: strides and
// divisors are immediates and a kernel holds its own codelets only (2^24
// points in rows: 50-52 us for lengths of three passes against 56-62).  VT:
// transforms per column tile (1 for rows).
template <int VT, int P, int... Rs> struct DifFix {
    static constexpr int V = VT, np = sizeof...(Rs), N = (Rs * ...);
    static constexpr int radix(int i) {
        const int r[] = {Rs...};
        return r[i];
    }
    static constexpr int M(int i) {
        int m = N;
        for (int j = 0; j < i; j++) m /= radix(j);
        return m;
    }
    static constexpr int S(int i) { return M(i) / radix(i); }
    static constexpr int two(int i) {
        int t = 0;
        for (int j = 0; j < i; j++) t += M(j);
        return t;
    }
    template <typename T> static __device__ __forceinline__ DifFixPass<DifFix, 0> first(const DifArgs<T> &) { return {}; }
    template <typename T> static __device__ __forceinline__ DifFixPass<DifFix, np - 1> last(const DifArgs<T> &) {
        return {};
    }
    template <typename T> static __device__ __forceinline__ int P1(const DifArgs<T> &) { return P; }
    template <int I> static __device__ __forceinline__ int digits(int rem) {
        if constexpr (I + 1 < np) return rem % radix(I) * S(I) + digits<I + 1>(rem / radix(I));
        else return 0;
    }
    template <typename T> static __device__ __forceinline__ int pos(const DifArgs<T> &, int q) {
        return q % radix(0) * P + digits<1>(q / radix(0));
    }
};

// x / V, V a power of two
template <class SC, typename T> __device__ __forceinline__ int dif_by_v(const DifArgs<T> &a, int x) {
    return SC::V ? x / (SC::V ? SC::V : 1) : x >> a.lgv;
}

// First pass.  Rows: consecutive threads on consecutive n' of one transform;
// column tiles: on adjacent transforms (element i of transform t at i*vpb + t).
template <class SC, int KIND, bool COLS, int R, typename T>
__device__ __forceinline__ void dif_first(const DifArgs<T> &a, typename cplx_t<T>::t *s, int nt, long v0) {
    typedef typename cplx_t<T>::t C;
    const auto &p = SC::first(a);
    const int S = p.S, V = !COLS ? 1 : SC::V ? SC::V : a.vpb;
    const int nb = COLS ? S : nt * S;
    const int step = COLS ? dif_by_v<SC>(a, (int)blockDim.x) : (int)blockDim.x;
    const int ct = COLS ? ((int)threadIdx.x & (V - 1)) : 0;
    const int sp = SC::P1(a) * V;
    if (COLS && ct >= nt) return;
    for (int b = COLS ? dif_by_v<SC>(a, (int)threadIdx.x) : (int)threadIdx.x; b < nb; b += step) {
        int t = ct, j = b;
        if (!COLS && a.vpb > 1) {
            t = p.by_NR(b);
            j = b - t * S;
        }
        long e0 = (v0 + t) * a.vs_in + (COLS ? (long)j * a.es_in : (long)j);
        if constexpr (dif_groups<KIND>()) e0 += blockIdx.y * a.bvs_in;
        C v[R];
        if constexpr (COLS) {
            const long st = (long)S * a.es_in;
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = dif_in<KIND>(a, e0 + r * st);
        } else {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = dif_in<KIND>(a, e0 + r * S);
        }
        if constexpr (KIND == DIF_R2CT) {
            // kw.c: data = ts * data (VSIP_ROW), then data = arr * data (VSIP_COL)
            const T wt = a.tp_t[(v0 + t) * a.tp_t_st];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const long n = 2L * (j + r * S);
                v[r].x = mul_rn(mul_rn(a.tp_n[n * a.tp_n_st], v[r].x), wt);
                v[r].y = mul_rn(mul_rn(a.tp_n[(n + 1) * a.tp_n_st], v[r].y), wt);
                a.wb[e0 + r * S] = v[r];
            }
        }
#pragma unroll
        for (int r = 0; r < R; r++) v[r].y = flip_sign(v[r].y, a.smask_in);
        DftF<C, R>::run(v);
        const C *w = a.tw + j;
#pragma unroll
        for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(w + r * S));
        C *d = COLS ? s + (j * V + t) : s + (t * a.LD + j);
#pragma unroll
        for (int r = 0; r < R; r++) d[r * sp] = v[r];
    }
}

// Middle pass.
template <class SC, bool COLS, int R, typename T, class PD>
__device__ __forceinline__ void dif_mid(const DifArgs<T> &a, const PD &p, typename cplx_t<T>::t *s, int nt) {
    typedef typename cplx_t<T>::t C;
    const int S = p.S, V = !COLS ? 1 : SC::V ? SC::V : a.vpb;
    const int nb = COLS ? p.NR : nt * p.NR;
    const int step = COLS ? dif_by_v<SC>(a, (int)blockDim.x) : (int)blockDim.x;
    const int ct = COLS ? ((int)threadIdx.x & (V - 1)) : 0;
    const int sp = S * V;
    if (COLS && ct >= nt) return;
    for (int b = COLS ? dif_by_v<SC>(a, (int)threadIdx.x) : (int)threadIdx.x; b < nb; b += step) {
        int t = ct, j = b;
        if (!COLS && a.vpb > 1) {
            t = p.by_NR(b);
            j = b - t * p.NR;
        }
        const int k1 = p.by_NB1(j), u = j - k1 * p.NB1;
        const int c = p.by_S(u), n = u - c * S;
        const int pos = k1 * SC::P1(a) + u + c * p.mstep;
        C *d = COLS ? s + (pos * V + t) : s + (t * a.LD + pos);
        C v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = d[r * sp];
        DftF<C, R>::run(v);
        const C *w = a.tw + (p.two + n);
#pragma unroll
        for (int r = 1; r < R; r++) v[r] = cmul(v[r], __ldg(w + r * S));
#pragma unroll
        for (int r = 0; r < R; r++) d[r * sp] = v[r];
    }
}

// Last pass: to the view.
template <class SC, int KIND, bool COLS, int R, typename T>
__device__ __forceinline__ void dif_last(const DifArgs<T> &a, const typename cplx_t<T>::t *s, int nt, long v0) {
    typedef typename cplx_t<T>::t C;
    const auto &p = SC::last(a);
    // stores with consecutive threads on adjacent transforms: column tiles,
    // and the rows of a long vector's last pass
    constexpr bool TF = COLS || dif_rows_tf<KIND>();
    const int Q = p.NR, V = !TF ? 1 : SC::V ? SC::V : a.vpb;
    const int nb = TF ? Q : nt * Q;
    const int step = TF ? dif_by_v<SC>(a, (int)blockDim.x) : (int)blockDim.x;
    const int ct = TF ? ((int)threadIdx.x & (V - 1)) : 0;
    if (TF && ct >= nt) return;
    for (int b = TF ? dif_by_v<SC>(a, (int)threadIdx.x) : (int)threadIdx.x; b < nb; b += step) {
        int t = ct, q = b;
        if (!TF && a.vpb > 1) {
            t = p.by_NR(b);
            q = b - t * Q;
        }
        const int pos = SC::pos(a, q);
        const C *d = COLS ? s + (pos * V + t) : s + (t * a.LD + pos);
        C v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = COLS ? d[r * V] : d[r];
        DftF<C, R>::run(v);
        long e0 = (v0 + t) * a.vs_out + (TF ? (long)q * a.es_out : (long)q);
        const long st = TF ? (long)Q * a.es_out : (long)Q;
        if constexpr (dif_groups<KIND>()) e0 += blockIdx.y * a.bvs_out;
        if constexpr (KIND == DIF_STEP) {
            if (a.tw_lo) {
                const unsigned g = (unsigned)(v0 + t) * a.tw_ts + blockIdx.y * a.tw_ys;
#pragma unroll
                for (int r = 0; r < R; r++)
                    v[r] = cmul(v[r], tw_two_level(a.tw_lo, a.tw_hi, a.tw_mask, a.tw_sh, g * (unsigned)(q + r * Q)));
            }
        }
        if constexpr (KIND == DIF_VEC1) {
            // W_N^(k (v0 + t)) = base[k] * W_N^(k t)
            const C *base = s + a.LD * V + q, *w = a.tv + (q * V + t);
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = cmul(v[r], cmul(base[r * Q], __ldg(w + r * Q * V)));
        }
        if constexpr (KIND == DIF_VEC2) {
            const C *w = a.tv + ((long)q * a.tv_st + v0 + t);
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = cmul(v[r], __ldg(w + r * Q * a.tv_st));
        }
        if constexpr (KIND == DIF_POWER) {
            T *g = a.gram + (v0 + t) * a.g_vs + (long)q * a.g_es;
            T old[R];
#pragma unroll
            for (int r = 0; r < R; r++) old[r] = g[(long)(r * Q) * a.g_es];
#pragma unroll
            for (int r = 0; r < R; r++) {
                // p = |X|^2 (vsip_mcmagsq_f), p *= s (vsip_smmul_f),
                // gram = p + gram (vsip_madd_f), rounded in that order
                const C x = out_value(v[r], a.smask_out, a.has_scale != 0, a.scale);
                T p = add_rn(mul_rn(x.x, x.x), mul_rn(x.y, x.y));
                p = mul_rn(a.g_scale, p);
                g[(long)(r * Q) * a.g_es] = add_rn(p, old[r]);
                dif_out<KIND>(a, e0 + r * st, mk<C>(p, x.y));
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; r++)
                dif_out<KIND>(a, e0 + r * st, out_value(v[r], a.smask_out, a.has_scale != 0, a.scale));
        }
    }
}

// First pass of C2R rows: Y_n = X_n + conj X_{N-n} + i w_n (X_n - conj X_{N-n}),
// w_n = exp(+i pi n/N) (c_VSIP_src/VI_crfftmop_f_def.h:58-110), conjugated for
// the forward passes.  A thread takes the butterflies of n' and S - n' (one of
// them for n' = 0 and S/2), which hold each other's partners X_{N-n}, so every
// spectrum element is loaded once; w_{N-n} = -conj w_n.
template <class SC, int R, typename T>
__device__ __forceinline__ void dif_first_c2r(const DifArgs<T> &a, typename cplx_t<T>::t *s, int nt, long v0) {
    typedef typename cplx_t<T>::t C;
    const auto &p = SC::first(a);
    const int S = p.S, H = S / 2 + 1, P1 = SC::P1(a);
    for (int b = threadIdx.x; b < nt * H; b += blockDim.x) {
        const int t = mdiv(b, a.mH), j = b - t * H;
        const C *x = a.in + (v0 + t) * a.vs_in;
        const C *xu = x + j, *xw = x + (S - j), *h = a.thalf + j;
        C u[R], w[R];
#pragma unroll
        for (int r = 0; r < R; r++) u[r] = xu[r * S];
#pragma unroll
        for (int r = 0; r < R; r++) w[r] = xw[r * S];
#pragma unroll
        for (int r = 0; r < R; r++) {
            const C f = u[r], g = w[R - 1 - r], c = __ldg(h + r * S);
            const C d = mk<C>(g.x - f.x, f.y + g.y);
            u[r] = mk<C>(f.x + g.x + c.y * d.x - c.x * d.y, -(f.y - g.y - c.y * d.y - c.x * d.x));
            w[R - 1 - r] = mk<C>(f.x + g.x - c.y * d.x + c.x * d.y, -(g.y - f.y - c.y * d.y - c.x * d.x));
        }
        C *d = s + (t * a.LD + j);
        DftF<C, R>::run(u);
        const C *tu = a.tw + j;
#pragma unroll
        for (int r = 1; r < R; r++) u[r] = cmul(u[r], __ldg(tu + r * S));
#pragma unroll
        for (int r = 0; r < R; r++) d[r * P1] = u[r];
        if (j != 0 && 2 * j != S) {
            d += S - 2 * j;
            DftF<C, R>::run(w);
            const C *tw = a.tw + (S - j);
#pragma unroll
            for (int r = 1; r < R; r++) w[r] = cmul(w[r], __ldg(tw + r * S));
#pragma unroll
            for (int r = 0; r < R; r++) d[r * P1] = w[r];
        }
    }
}

// Last pass of R2C rows: Z from two butterflies q and Q - q (Q = N/R), which
// hold each other's partners Z_{N-k}, then X_k = ((Z_k + conj Z_{N-k}) - i w_k
// (Z_k - conj Z_{N-k}))/2, w_k = exp(-i pi k/N), Z_N = Z_0, the scale applied
// to Z first (c_VSIP_src/VI_rcfftmop_f_def.h:79-118): the spectrum leaves from
// registers, without another trip through shared memory.
template <class SC, int KIND, int R, typename T>
__device__ __forceinline__ void dif_last_r2c(const DifArgs<T> &a, const typename cplx_t<T>::t *s, int nt, long v0) {
    typedef typename cplx_t<T>::t C;
    const auto &p = SC::last(a);
    // a column-major spectrum (DIF_R2CT) is stored with consecutive threads on
    // adjacent rows: segments of 8 bytes times the tile's rows instead of single
    // elements a column apart
    constexpr bool TF = dif_rows_tf<KIND>();
    const int Q = p.NR, H = Q / 2 + 1, V = !TF ? 1 : SC::V ? SC::V : a.vpb;
    const int ct = TF ? ((int)threadIdx.x & (V - 1)) : 0;
    if (TF && ct >= nt) return;
    const int nb = TF ? H : nt * H, step = TF ? dif_by_v<SC>(a, (int)blockDim.x) : (int)blockDim.x;
    for (int b = TF ? dif_by_v<SC>(a, (int)threadIdx.x) : (int)threadIdx.x; b < nb; b += step) {
        const int t = TF ? ct : mdiv(b, a.mH), q = TF ? b : b - t * H;
        const C *su = s + (t * a.LD + SC::pos(a, q)), *sw = s + (t * a.LD + SC::pos(a, q ? Q - q : 0));
        C u[R], w[R];
#pragma unroll
        for (int r = 0; r < R; r++) u[r] = su[r];
#pragma unroll
        for (int r = 0; r < R; r++) w[r] = sw[r];
        DftF<C, R>::run(u);
        DftF<C, R>::run(w);
        if (a.has_scale) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                u[r] = cscale(u[r], a.scale);
                w[r] = cscale(w[r], a.scale);
            }
        }
        const C *h = a.thalf + q;
        C *o = a.out + (v0 + t) * a.vs_out;
        const bool both = q != 0 && 2 * q != Q;
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int k = q + r * Q;
            const C z = u[r], c = __ldg(h + r * Q);
            C n = w[R - 1 - r];
            if (q == 0) n = w[(R - r) % R];
            const C sm = mk<C>(z.x + n.x, z.y + n.y), df = mk<C>(z.x - n.x, z.y - n.y);
            o[(long)k * a.es_out] =
                mk<C>((T)0.5 * (sm.x + c.x * sm.y + c.y * df.x), (T)0.5 * (df.y - c.x * df.x + c.y * sm.y));
            if (both || (r == 0 && q == 0))
                o[(long)(a.N - k) * a.es_out] =
                    mk<C>((T)0.5 * (sm.x - c.x * sm.y - c.y * df.x), (T)0.5 * (-df.y - c.x * df.x + c.y * sm.y));
        }
    }
}

#define JV_DIF_SWITCH(RAD, CALL)     \
    switch (RAD) {                   \
        case 16: CALL(16); break;    \
        case 15: CALL(15); break;    \
        case 14: CALL(14); break;    \
        case 13: if constexpr (P13) CALL(13); break; \
        case 12: CALL(12); break;    \
        case 11: if constexpr (P13) CALL(11); break; \
        case 10: CALL(10); break;    \
        case 9: CALL(9); break;      \
        case 8: CALL(8); break;      \
        case 7: CALL(7); break;      \
        case 6: CALL(6); break;      \
        case 5: CALL(5); break;      \
        case 4: CALL(4); break;      \
        case 3: CALL(3); break;      \
        default: CALL(2); break;     \
    }

// the pair passes hold two butterflies, of at most this radix (at 10 the compiled-in
// R2C kernels that end on it, 19 of 147, spill 8 to 76 bytes; 9 and below none)
constexpr int kDifPairMax = 10;
#define JV_DIF_PAIR_SWITCH(RAD, CALL) \
    switch (RAD) {                    \
        case 10: CALL(10); break;     \
        case 9: CALL(9); break;       \
        case 8: CALL(8); break;       \
        case 7: CALL(7); break;       \
        case 6: CALL(6); break;       \
        case 5: CALL(5); break;       \
        case 4: CALL(4); break;       \
        case 3: CALL(3); break;       \
        default: CALL(2); break;      \
    }

// The passes of one CTA's transforms.  P13: with the codelets 11 and 13, which the
// lengths of batches and k-omega (2^a 3^b 5^c 7^d) do not reach.  Without them the
// batch kernels spill 156 and 296 bytes (208 and 384 with; a batch of 60 calls 143 us,
// 149, of 160 538 and 544).  k-omega's kernels keep them: without, the tapered rows
// spill less (4 bytes, 88) but 343 sensors x 2058 samples take 20.4 us (17.9), and the
// power columns spill more (556, 464; 448 x 2800 22.0 us, 21.1).
template <typename T, int KIND, bool COLS, bool P13>
__device__ __forceinline__ void dif_passes(const DifArgs<T> &a, typename cplx_t<T>::t *s, int nt, long v0) {
    typedef DifDyn SC;
    if constexpr (KIND == DIF_C2R) {
#define JV_DIF_FIRST(R) (dif_first_c2r<SC, R, T>(a, s, nt, v0))
        JV_DIF_PAIR_SWITCH(a.p[0].R, JV_DIF_FIRST)
#undef JV_DIF_FIRST
    } else {
#define JV_DIF_FIRST(R) (dif_first<SC, KIND, COLS, R, T>(a, s, nt, v0))
        JV_DIF_SWITCH(a.p[0].R, JV_DIF_FIRST)
#undef JV_DIF_FIRST
    }
    __syncthreads();
    for (int i = 1; i + 1 < a.np; i++) {
#define JV_DIF_MID(R) (dif_mid<SC, COLS, R, T>(a, a.p[i], s, nt))
        JV_DIF_SWITCH(a.p[i].R, JV_DIF_MID)
#undef JV_DIF_MID
        __syncthreads();
    }
    if constexpr (KIND == DIF_R2C || KIND == DIF_R2CT) {
#define JV_DIF_LAST(R) (dif_last_r2c<SC, KIND, R, T>(a, s, nt, v0))
        JV_DIF_PAIR_SWITCH(a.p[a.np - 1].R, JV_DIF_LAST)
#undef JV_DIF_LAST
    } else {
#define JV_DIF_LAST(R) (dif_last<SC, KIND, COLS, R, T>(a, s, nt, v0))
        JV_DIF_SWITCH(a.p[a.np - 1].R, JV_DIF_LAST)
#undef JV_DIF_LAST
    }
}
template <class F, int I, typename T, bool COLS>
__device__ __forceinline__ void dif_mids(const DifArgs<T> &a, typename cplx_t<T>::t *s, int nt) {
    if constexpr (I + 1 < F::np) {
        dif_mid<F, COLS, F::radix(I), T>(a, DifFixPass<F, I>(), s, nt);
        __syncthreads();
        dif_mids<F, I + 1, T, COLS>(a, s, nt);
    }
}
template <class F, typename T, int KIND, bool COLS>
__device__ __forceinline__ void dif_passes_fix(const DifArgs<T> &a, typename cplx_t<T>::t *s, int nt, long v0) {
    if constexpr (KIND == DIF_C2R) dif_first_c2r<F, F::radix(0), T>(a, s, nt, v0);
    else dif_first<F, KIND, COLS, F::radix(0), T>(a, s, nt, v0);
    __syncthreads();
    dif_mids<F, 1, T, COLS>(a, s, nt);
    if constexpr (KIND == DIF_R2C || KIND == DIF_R2CT) dif_last_r2c<F, KIND, F::radix(F::np - 1), T>(a, s, nt, v0);
    else dif_last<F, KIND, COLS, F::radix(F::np - 1), T>(a, s, nt, v0);
}

template <typename T, int KIND>
__device__ __forceinline__ void dif_prologue(const DifArgs<T> &a, typename cplx_t<T>::t *s, long v0) {
    if constexpr (KIND == DIF_VEC1) {
        // W_N^(k v0), k < the pass's length (k v0 < N), behind the tile
        for (int k = threadIdx.x; k < a.N; k += blockDim.x)
            s[a.LD * a.vpb + k] = tw_two_level(a.tw_lo, a.tw_hi, a.tw_mask, a.tw_sh, (unsigned)k * (unsigned)v0);
    }
}

template <typename T, int KIND, bool COLS>
__global__ void __launch_bounds__(sizeof(T) == 4 ? 1024 : 512) k_dif(const __grid_constant__ DifArgs<T> a) {
    typedef typename cplx_t<T>::t C;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    C *s = reinterpret_cast<C *>(smem_raw);
    const long v0 = (long)blockIdx.x * a.vpb;
    const int nt = (int)min((long)a.vpb, a.nvec - v0);
    dif_prologue<T, KIND>(a, s, v0);
    dif_passes<T, KIND, COLS, true>(a, s, nt, v0);
}

// The same with a schedule known at compile time, in CTAs of NT threads of
// which MB share an SM.
template <class F, typename T, int KIND, bool COLS, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_dif_fix(const __grid_constant__ DifArgs<T> a) {
    typedef typename cplx_t<T>::t C;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    C *s = reinterpret_cast<C *>(smem_raw);
    const long v0 = (long)blockIdx.x * a.vpb;
    const int nt = (int)min((long)a.vpb, a.nvec - v0);
    dif_prologue<T, KIND>(a, s, v0);
    dif_passes_fix<F, T, KIND, COLS>(a, s, nt, v0);
}

// One tile of a batch of calls: nt transforms from v0 of call `call`.
struct DifTile {
    int call, nt;
    long v0;
};

// The batching form's kernel: CTA b takes tile b of the queue, its call's
// arguments copied into shared memory.
template <bool COLS>
__global__ void __launch_bounds__(1024) k_dif_batch(const DifArgs<float> *__restrict__ calls,
                                                    const DifTile *__restrict__ q) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(16) DifArgs<float> a;
    float2 *s = reinterpret_cast<float2 *>(smem_raw);
    const DifTile d = q[blockIdx.x];
    static_assert(sizeof(DifArgs<float>) % 8 == 0, "copied by 8 bytes");
    for (int i = threadIdx.x; i < (int)(sizeof(a) / 8); i += blockDim.x)
        reinterpret_cast<unsigned long long *>(&a)[i] =
            __ldg(reinterpret_cast<const unsigned long long *>(&calls[d.call]) + i);
    __syncthreads();
    dif_passes<float, DIF_C2C, COLS, false>(a, s, d.nt, d.v0);
}

// static shared memory of k_dif_batch (the copied arguments), rounded up
constexpr size_t kStaticArgs = 1024;
static_assert(sizeof(DifArgs<float>) <= kStaticArgs, "arguments fit");

// A length whose schedule is compiled in (jv_dif_table.h) and its launchers
// (null: the kernel that reads the schedule from its arguments).
typedef bool (*DifFixGo)(const DifArgs<float> &a, size_t smem, cudaStream_t st, unsigned groups);
struct DifFixEntry {
    int N = 0, P1 = 0;
    int vpb = 1, nthr = 0;   // rows: transforms per CTA, threads
    int vcol = 0;            // transforms per column tile
    std::vector<int> radix;
    DifFixGo rows = nullptr, cols = nullptr, cols4 = nullptr;  // cols4: tiles of 4, for few columns
    DifFixGo step = nullptr, vec[3] = {nullptr, nullptr, nullptr};
    DifFixGo taper = nullptr, power = nullptr;  // k-omega: R2C tiles of vtaper rows; power rows
    int vtaper = 0;
};
const DifFixEntry *dif_fix(long N, int cls);  // cls 0: c2c, 1: R2C, 2: C2R; null: not in the table

// CTA shape of a call
struct DifCta {
    int nthr = 0;
    size_t smem = 0;
    bool rows = true, split = false;
};
// batch tiles that are to occupy `sms` SMs; false: not for k_dif
bool dif_tile_args(const Job &j, long tuned, long sms, DifArgs<float> &a, DifCta &c);
bool dif_batch_go(bool cols, const DifArgs<float> *calls, const DifTile *q, int ntiles, int nthr, size_t smem,
                  cudaStream_t st);

// Launches (nvec + vpb - 1)/vpb CTAs of nthr threads; instances in jv_dif*.cu.
template <typename T, int KIND, bool COLS>
bool dif_go(const DifArgs<T> &a, int nthr, size_t smem, cudaStream_t st);

template <typename T, int KIND, bool COLS>
inline bool dif_launch(const DifArgs<T> &a, int nthr, size_t smem, cudaStream_t st, unsigned gy = 1) {
    static std::atomic<bool> attr{false};  // set once; concurrent first calls both set it
    if (!attr) {
        if (!cuda_ok(cudaFuncSetAttribute(k_dif<T, KIND, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)device()->smem_optin),
                     "cudaFuncSetAttribute"))
            return false;
        attr = true;
    }
    const long grid = (a.nvec + a.vpb - 1) / a.vpb;
    if (grid > 0x7fffffffL) return false;
    k_dif<T, KIND, COLS><<<dim3((unsigned)grid, gy), (unsigned)nthr, smem, st>>>(a);
    count_launch();
    return cuda_ok(cudaGetLastError(), "k_dif launch");
}
#define JV_DIF_INSTANCE(T, KIND, COLS)                                                        \
    template <>                                                                               \
    bool dif_go<T, KIND, COLS>(const DifArgs<T> &a, int nthr, size_t smem, cudaStream_t st) { \
        return dif_launch<T, KIND, COLS>(a, nthr, smem, st);                                  \
    }
#define JV_DIF_DECLARE(T, KIND, COLS) \
    template <>                       \
    bool dif_go<T, KIND, COLS>(const DifArgs<T> &a, int nthr, size_t smem, cudaStream_t st);
JV_DIF_DECLARE(float, DIF_C2C, false)
JV_DIF_DECLARE(float, DIF_C2C, true)
JV_DIF_DECLARE(float, DIF_SPLIT, false)
JV_DIF_DECLARE(float, DIF_SPLIT, true)
JV_DIF_DECLARE(float, DIF_R2C, false)
JV_DIF_DECLARE(float, DIF_C2R, false)
JV_DIF_DECLARE(double, DIF_C2C, false)
JV_DIF_DECLARE(double, DIF_C2C, true)
bool dif_step_go(const DifArgs<float> &a, int nthr, size_t smem, cudaStream_t st, unsigned groups);
bool dif_komega_go(int kind, const DifArgs<float> &a, int nthr, size_t smem, cudaStream_t st);
bool dif_vec_go(int kind, const DifArgs<float> &a, int nthr, size_t smem, cudaStream_t st, unsigned groups);

}  // namespace jv
