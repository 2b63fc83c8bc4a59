// jv_batch.cu -- batching form: many independent c2c fftm calls (uneven
// lengths 2^a 3^b 5^c 7^d, uneven row counts, mixed directions and ROW/COL
// majors) in one launch per CTA-size class, fed by a device queue of tile
// descriptors.
//
// The host cuts every call on row-contiguous or adjacent transforms into tiles
// of the in-place mixed-radix kernel (jv_dif.cuh, k_dif_batch): one queue per
// block size, largest tiles first, one tile per CTA -- no CTA ever waits on
// another -- whose arguments (the call's) the CTA copies into shared memory.
// Columns from kColStepsMin points (adjacent; 32 or more below 8192 points) go
// through the plain calls' two steps on eight streams of their own.  Other layouts, and
// lengths without a schedule of two codelets, keep the general kernel's fused
// c2c passes in CTAs of 256, 512 or 1024 threads (k_batch; long adjacent
// columns in 4-CTA clusters, k_batch_cols), each CTA asking L2
// for the input of the descriptor one resident wave further down its queue.
// The launches run side by side on forked streams.  160 instances of 64-16384
// points (0.58 GB per buffer) on GB300: 0.56 ms against 0.80 with every tile
// on the general kernel's passes and only columns from 8192 points in steps.
// A captured batch (jvsip_fftm_batch_create_f) records the launches in a CUDA
// graph once; jvsip_fftm_batch_run_f replays it.
//
// No reference counterpart: VSIPL has no multi-plan call; the reference can
// only loop plan by plan (c_VSIP_src/VI_ccfftmop_f_def.h:20-29 per call).
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <new>
#include <vector>

#include <cooperative_groups.h>

#include "jv_dif.cuh"
#include "jv_dif_tile.h"
#include "jv_launch.cuh"

namespace jv {

// one tile: nt transforms [v0, v0+nt) of one call
struct TileDesc {
    const float *in;    // interleaved views, complex index off + v*vs + n*es
    float *out;
    long in_off, in_es, in_vs;
    long out_off, out_es, out_vs;
    const float2 *twg;  // per-pass [r][m] tables of the call's plan
    const uint4 *pc;    // per-pass constants of the plan's schedule
    unsigned long long passes;  // pass counts per codelet (pass_count)
    unsigned mnt;       // multiply-high magic of nt
    long v0;
    int N, nt, ld;
    unsigned char inv, vec_fast, cls;  // cls: CTA-size class (index into kClassBT)
    int has_scale;
    float scale;
};

constexpr int BT = 1024;      // threads of the largest batch CTA
constexpr int BEMAX = 16;     // complex values a thread keeps per pass: tiles of <= 16384 points
// CTA-size classes: a tile runs in the smallest CTA whose threads cover every
// pass of it, so small tiles share an SM (4 x 256 or 2 x 512 threads at 64
// registers) instead of idling most of a 1024-thread CTA
constexpr int kClasses = 4;
constexpr int kClassBT[kClasses] = {256, 512, 1024, 1024};  // the last: column clusters
constexpr int kColClass = 3;

__device__ __forceinline__ void batch_tile(const TileDesc &d, float2 *s) {
    TileIO<float> io;
    io.in = reinterpret_cast<const float2 *>(d.in) + (d.in_off + d.v0 * d.in_vs);
    io.out = reinterpret_cast<float2 *>(d.out) + (d.out_off + d.v0 * d.out_vs);
    io.in_es = d.in_es;
    io.in_vs = d.in_vs;
    io.out_es = d.out_es;
    io.out_vs = d.out_vs;
    io.smask_in = io.smask_out = d.inv ? 0x80000000u : 0u;
    io.has_scale = d.has_scale != 0;
    io.scale = d.has_scale ? d.scale : 1.f;
    io.vf = io.vf_out = d.vec_fast != 0;
    io.mnt = d.mnt;
    io.tw_lo = io.tw_hi = nullptr;
    c2c_tile<float, BEMAX>(s, d.ld, d.nt, d.passes, d.twg, d.pc, io);
}

__device__ __forceinline__ void prefetch_l2_line(const void *p) {
    asm volatile("{\n\t.reg .u64 a;\n\tcvta.to.global.u64 a, %0;\n\tprefetch.global.L2 [a];\n\t}" :: "l"(p));
}

// Ask L2 for the input of tile d: one 128-byte line per thread and step.
// Transforms contiguous in memory (|es| = 1) go by 16-element segments of each
// transform, adjacent transforms (|vs| = 1) by 16-element segments of each
// point's row of transforms; other layouts are not prefetched.
__device__ __forceinline__ void prefetch_tile(const TileDesc &d, int tid, int nthr) {
    const float2 *base = reinterpret_cast<const float2 *>(d.in) + (d.in_off + d.v0 * d.in_vs);
    // every address is an element of the tile (the last line of a segment
    // is taken at its last element)
    if (d.in_es == 1) {
        const int L = (d.N + 15) >> 4, tot = L * d.nt;
        for (int i = tid; i < tot; i += nthr) {
            const int v = i / L, l = i - v * L;
            prefetch_l2_line(base + (long)v * d.in_vs + min(16 * l, d.N - 1));
        }
    } else if (d.in_vs == 1) {
        const int L = (d.nt + 15) >> 4, tot = L * d.N;
        for (int i = tid; i < tot; i += nthr) {
            const int n = i / L, l = i - n * L;
            prefetch_l2_line(base + (long)n * d.in_es + min(16 * l, d.nt - 1));
        }
    }
}

// One launch over the whole queue: CTA b takes descriptor b.  The queue is
// sorted largest tile first, so the hardware's in-order CTA dispatch hands the
// long tiles out first and the short ones fill the tail.  (A persistent
// variant -- each CTA looping over an atomic queue head -- was built and
// measured against ptxas: keeping the pass state live across tile iterations
// spills the codelet registers at every block size, so the loop-free form is
// used.)
template <int CBT>
__global__ void __launch_bounds__(CBT, 1024 / CBT) k_batch(const TileDesc *__restrict__ q, int ntiles, int ahead) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *s = reinterpret_cast<float2 *>(smem_raw);
    __shared__ TileDesc sd, sn;  // descriptor fields are re-read from shared memory, not held in registers
    const int t = blockIdx.x;
    if (t >= ntiles) return;
    const int tn = t + ahead;  // the tile that takes this slot a wave later
    if (threadIdx.x == 0) {
        sd = q[t];
        if (ahead > 0 && tn < ntiles) sn = q[tn];
    }
    __syncthreads();
    if (ahead > 0 && tn < ntiles) prefetch_tile(sn, threadIdx.x, blockDim.x);
    batch_tile(sd, s);
}

// Columns of long transforms (one column fills a CTA): a 4-CTA cluster takes
// up to 4 adjacent columns, one column per CTA.  CTA c reads rows
// [c*Q, (c+1)*Q) of all the columns with the column index fastest -- every
// matrix row is one contiguous segment -- and stores each value into the
// owning CTA's shared memory (distributed shared memory, natural order); after
// a cluster barrier every CTA runs its column's passes locally (the first pass
// reads the natural order, the last writes the padded rows); after a second
// barrier CTA c writes rows [c*Q, (c+1)*Q) of all the columns, read from the
// owners' shared memory, and a third barrier keeps every CTA's shared memory
// alive until the others have read it.  Every thread of the cluster reaches
// every barrier: CTAs without a column skip only the passes.
constexpr int kColCluster = 4;

__device__ __forceinline__ void col_passes(float2 *s, int ld, unsigned long long packed, const float2 *twg,
                                           const uint4 *pc) {
    int fi = 0;
    while (fi < kRadices - 1 && pass_count(packed, fi) == 0) fi++;
    const uint4 pc0 = __ldg(&pc[0]);
    int Rf = 2;
#define JV_DENSE_FIRST(R) (smem_pass<float, R, BEMAX, 1>(s, ld, 1, 1, twg, pc0), Rf = R)
    JV_RADIX_SWITCH(fi, JV_DENSE_FIRST)
#undef JV_DENSE_FIRST
    int Ns = Rf, p = 1;
    const float2 *tp = twg + Rf;
    smem_passes_from<float, BEMAX>(s, ld, 1, packed - (1ull << (4 * fi)), tp, pc, Ns, p);
}

__global__ void __cluster_dims__(kColCluster, 1, 1) __launch_bounds__(BT, 1)
    k_batch_cols(const TileDesc *__restrict__ q, int ntiles) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2 *s = reinterpret_cast<float2 *>(smem_raw);
    __shared__ TileDesc sd;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int t = blockIdx.x / kColCluster;  // the same descriptor for the whole cluster
    if (t >= ntiles) return;                 // uniform over the cluster
    if (threadIdx.x == 0) sd = q[t];
    __syncthreads();
    // each phase reads its values from the shared descriptor, so none of them
    // stays live in registers across the passes (which use all 64)
    {
        // ---- load: (row, column) with the column fastest, four loads in flight
        const int tid = threadIdx.x, nthr = blockDim.x;
        const int N = sd.N, nt = sd.nt;
        const int Q = (N + kColCluster - 1) / kColCluster;
        const int n0 = rank * Q, nr = max(0, min(N, n0 + Q) - n0);
        const int tot = nr * nt;
        const unsigned mnt = sd.mnt;
        const float2 *in = reinterpret_cast<const float2 *>(sd.in) + (sd.in_off + sd.v0 * sd.in_vs);
        const long ies = sd.in_es, ivs = sd.in_vs;
        const float sgn = sd.inv ? -1.f : 1.f;
        for (int i0 = tid; i0 < tot; i0 += 4 * nthr) {
            float2 c[4];
            int kk[4], nn[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = i0 + u * nthr;
                kk[u] = 0;
                nn[u] = 0;
                if (i < tot) {
                    const int r = mdiv(i, mnt);
                    kk[u] = i - r * nt;
                    nn[u] = n0 + r;
                    c[u] = in[(long)kk[u] * ivs + (long)nn[u] * ies];
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                if (i0 + u * nthr < tot) {
                    float2 *dst = cl.map_shared_rank(s, kk[u]);
                    dst[nn[u]] = make_float2(c[u].x, c[u].y * sgn);
                }
            }
        }
    }
    cl.sync();
    if ((int)cl.block_rank() < sd.nt) col_passes(s, sd.ld, sd.passes, sd.twg, sd.pc);
    cl.sync();
    {
        // ---- store: rows [n0, n0 + nr) of the columns, from their owners
        const int tid = threadIdx.x, nthr = blockDim.x;
        const int N = sd.N, nt = sd.nt;
        const int Q = (N + kColCluster - 1) / kColCluster;
        const int n0 = (int)cl.block_rank() * Q, nr = max(0, min(N, n0 + Q) - n0);
        const int tot = nr * nt;
        const unsigned mnt = sd.mnt;
        float2 *out = reinterpret_cast<float2 *>(sd.out) + (sd.out_off + sd.v0 * sd.out_vs);
        const long oes = sd.out_es, ovs = sd.out_vs;
        const float scale = sd.has_scale ? sd.scale : 1.f, sy = (sd.inv ? -1.f : 1.f) * scale;
        for (int i = tid; i < tot; i += nthr) {
            const int r = mdiv(i, mnt), k = i - r * nt, n = n0 + r;
            const float2 *src = cl.map_shared_rank(s, k);
            const float2 v = src[spad(n)];
            out[(long)k * ovs + (long)n * oes] = make_float2(v.x * scale, v.y * sy);
        }
    }
    cl.sync();
}

// ---------------------------------------------------------------- host side
// A call the batch runs through the plain path instead of tiles: single-
// precision c2c columns (adjacent vectors on both sides) that the plain calls
// take as two steps, the groups along the grid's y.  Measured on the 160
// instances above: 0.60 ms with all of them in steps, 0.64 with columns of
// 3000-8191 points as tiles of 4 columns.
struct StepCall {
    Plan *p;
    const vsip_cmview_f *x, *y;
};

// Tiles of the in-place mixed-radix kernel of one block size, rows or columns.
struct DifGroup {
    bool cols = false;
    int nthr = 0;
    size_t smem = 0;
    long ntiles = 0;
    std::vector<int> calls;  // by their index, largest tiles first
};

struct BatchBuild {
    std::vector<DifArgs<float>> calls;   // of the groups' tiles
    std::vector<DifGroup> groups;
    std::vector<TileDesc> tiles[kClasses];
    size_t smem[kClasses] = {0, 0, 0, 0};
    std::vector<StepCall> steps;
    double bytes = 0;
};

static long tile_ld(long N, bool vf) {
    long ld = (N - 1) + (N - 1) / 16 + 1;
    if (vf && (ld % 2 == 0)) ld += 1;
    return ld;
}

// FFTs per tile for length N (transforms adjacent in memory or not).
long batch_fft_per_tile(long N, bool vf, long rows);
long batch_tuned_per_tile(long N, bool vf);  // the autotuner's entry, 0: none

// Cuts a call into tiles of the in-place mixed-radix kernel that are to occupy `sms`
// SMs; false when its views or length are not for it.
static bool dif_tiles(const Plan *p, const TileDesc &t, long nv, long sms, BatchBuild &bb) {
    Job j;
    j.kind = K_C2C;
    j.prec = P_F32;
    j.N = t.N;
    j.nvec = nv;
    j.inv = t.inv;
    j.has_scale = t.has_scale;
    j.scale = t.scale;
    j.dif = p->dif;
    j.no_fast = p->no_fast;
    j.no_dif = p->no_dif;
    j.cin.re = const_cast<float *>(t.in);
    j.cin.im = const_cast<float *>(t.in) + 1;
    j.cin.off = t.in_off;
    j.cin.es = t.in_es;
    j.cin.vs = t.in_vs;
    j.cout.re = t.out;
    j.cout.im = t.out + 1;
    j.cout.off = t.out_off;
    j.cout.es = t.out_es;
    j.cout.vs = t.out_vs;
    bb.calls.emplace_back();
    const DifArgs<float> &a = bb.calls.back();
    DifCta c;
    if (!dif_tile_args(j, batch_tuned_per_tile(t.N, t.vec_fast != 0), sms, bb.calls.back(), c) ||
        c.smem > device()->smem_optin - kStaticArgs) {
        bb.calls.pop_back();
        return false;
    }
    // block sizes in steps of 64, so that one launch takes tiles of many lengths
    c.nthr = dif_batch_threads(c.nthr);
    DifGroup *g = nullptr;
    for (DifGroup &h : bb.groups)
        if (h.cols == !c.rows && h.nthr == c.nthr) g = &h;
    if (!g) {
        bb.groups.emplace_back();
        g = &bb.groups.back();
        g->cols = !c.rows;
        g->nthr = c.nthr;
    }
    g->smem = std::max(g->smem, c.smem);
    g->ntiles += (nv + a.vpb - 1) / a.vpb;
    g->calls.push_back((int)bb.calls.size() - 1);
    return true;
}

static bool build_tiles(size_t n, const vsip_fftm_f *const plans[], const vsip_cmview_f *const in[],
                        const vsip_cmview_f *const out[], BatchBuild &bb) {
    Device *d = device();
    if (!d) return false;
    // a call's tiles are cut for the SMs that its share of the points fills: with the
    // whole GPU for every call each tile held one transform or four columns (64 calls
    // of 200 rows of 64 points 6.3 us, 18.4 so; of 128 points 10.4 and 24.7)
    double points = 0;
    bb.calls.reserve(n);
    for (size_t i = 0; i < n; i++)
        if (const Plan *p = plan_of(plans[i])) points += (double)p->MN * p->mN;
    for (size_t i = 0; i < n; i++) {
        Plan *p = plan_of(plans[i]);
        if (!p || p->prec != P_F32 || (p->type != JV_CCFFTOP && p->type != JV_CCFFTIP)) {
            set_error(E_ARG, "batch: every plan must be a single-precision c2c plan");
            return false;
        }
        if (!p->smooth || !p->d_twg || !p->d_pc || p->radix.empty() || p->MN > BEMAX * BT) {
            set_error(E_UNSUPPORTED, "batch: lengths must be 2^a 3^b 5^c 7^d and at most 16384");
            return false;
        }
        const vsip_cmview_f *x = in[i];
        const vsip_cmview_f *y = (p->type == JV_CCFFTIP || !out || !out[i]) ? x : out[i];
        if (!x || !y || !x->block || !y->block) {
            set_error(E_ARG, "batch: null view");
            return false;
        }
        Mirror *mx = mirror_find(x->block), *my = mirror_find(y->block);
        if (!mx || !my || x->block->cstride != 2 || y->block->cstride != 2) {
            set_error(E_ARG, "batch: views must be of admitted interleaved blocks");
            return false;
        }
        const long N = p->MN, nv = p->mN;
        long xl = (long)(p->major == 0 ? x->row_length : x->col_length);
        long xn = (long)(p->major == 0 ? x->col_length : x->row_length);
        long yl = (long)(p->major == 0 ? y->row_length : y->col_length);
        long yn = (long)(p->major == 0 ? y->col_length : y->row_length);
        if (xl < N || xn < nv || yl < N || yn < nv) {
            set_error(E_ARG, "batch: view smaller than its plan");
            return false;
        }
        TileDesc t;
        memset(&t, 0, sizeof(t));
        t.in = (const float *)mx->d;
        t.out = (float *)my->d;
        t.in_off = (long)x->offset;
        t.out_off = (long)y->offset;
        if (p->major == 0) {
            t.in_es = x->row_stride;
            t.in_vs = x->col_stride;
            t.out_es = y->row_stride;
            t.out_vs = y->col_stride;
        } else {
            t.in_es = x->col_stride;
            t.in_vs = x->row_stride;
            t.out_es = y->col_stride;
            t.out_vs = y->row_stride;
        }
        // bounds of both views inside their blocks
        auto span_ok = [&](long off, long es, long vs, long len, long cnt, long size) {
            long lo = off + std::min(0L, (cnt - 1) * vs) + std::min(0L, (len - 1) * es);
            long hi = off + std::max(0L, (cnt - 1) * vs) + std::max(0L, (len - 1) * es);
            return lo >= 0 && hi < size;
        };
        if (!span_ok(t.in_off, t.in_es, t.in_vs, N, nv, (long)x->block->size) ||
            !span_ok(t.out_off, t.out_es, t.out_vs, N, nv, (long)y->block->size)) {
            set_error(E_ARG, "batch: view outside its block");
            return false;
        }
        if (x->block == y->block && (t.in_off != t.out_off || t.in_es != t.out_es || t.in_vs != t.out_vs)) {
            set_error(E_UNSUPPORTED, "batch: x and y on one block must be the same view");
            return false;
        }
        t.twg = (const float2 *)p->d_twg;
        t.pc = (const uint4 *)p->d_pc;
        t.N = (int)N;
        if (!pack_passes(p->radix, &t.passes)) {
            set_error(E_UNSUPPORTED, "batch: pass schedule outside the codelets");
            return false;
        }
        t.inv = (p->dir == 1) ? 1 : 0;
        t.has_scale = (p->scale != 1.0) ? 1 : 0;
        t.scale = (float)p->scale;
        bool vf_in = labs(t.in_vs) == 1 && labs(t.in_es) != 1;
        bool vf_out = labs(t.out_vs) == 1 && labs(t.out_es) != 1;
        t.vec_fast = (vf_in || vf_out) ? 1 : 0;
        t.ld = (int)tile_ld(N, t.vec_fast);
        // columns below 8192 points in steps only where there are 32 of them, or a few
        // calls in all: a step is two launches (us, steps and tiles: 64 calls of 3000 x
        // 3 68 and 13, 3000 x 20 92 and 31, 3000 x 200 93 and 102, 6000 x 200 87 and 122;
        // one call 8 and 12)
        const bool long_call = N >= kColStepsMin && (N >= kLongFewMin || nv >= 32 || n <= 4);
        // the plan's scratch is had now (nothing may allocate while a batch is
        // recorded into its graph); without it the call goes in tiles
        if (long_call && resident_long_columns_f(p, x, y) && enqueue_resident_c2c_f(p, x, y, nullptr, true)) {
            bb.steps.push_back(StepCall{p, x, y});
            bb.bytes += 16.0 * N * nv;
            continue;
        }
        const long share = std::max(1L, (long)(d->sms * (double)N * nv / points));
        if (dif_tiles(p, t, nv, share, bb)) {
            bb.bytes += 16.0 * N * nv;
            continue;
        }
        if (t.vec_fast && 2 * N > BEMAX * BT) {
            // columns of long transforms: groups of up to kColCluster adjacent
            // columns, one cluster each (k_batch_cols)
            t.ld = (int)tile_ld(N, false);
            for (long v0 = 0; v0 < nv; v0 += kColCluster) {
                TileDesc u = t;
                u.v0 = v0;
                u.nt = (int)std::min((long)kColCluster, nv - v0);
                u.mnt = magic_host((unsigned long)u.nt);
                u.cls = (unsigned char)kColClass;
                bb.tiles[kColClass].push_back(u);
                bb.smem[kColClass] = std::max(bb.smem[kColClass], (size_t)u.ld * 8);
            }
            bb.bytes += 16.0 * N * nv;
            continue;
        }
        long per = batch_fft_per_tile(N, t.vec_fast, nv);
        // every pass of the tile must fit the CTA: a thread holds
        // pass_k(BEMAX, R) butterflies of radix R (the plan's schedule fits
        // one transform by construction)
        long min_pts = BEMAX;
        for (int r : p->radix) min_pts = std::min(min_pts, (long)r * pass_k(BEMAX, r));
        while (per > 1 && per * N > (long)BT * min_pts) per--;
        while (per > 1 && per * (long)t.ld * 8 > (long)d->smem_optin - 512) per--;
        for (long v0 = 0; v0 < nv; v0 += per) {
            TileDesc u = t;
            u.v0 = v0;
            u.nt = (int)std::min(per, nv - v0);
            u.mnt = magic_host((unsigned long)u.nt);
            // threads the tile's passes need: a thread holds pass_k(BEMAX, R) butterflies
            long need = 32;
            for (int r : p->radix) {
                const long K = pass_k(BEMAX, r);
                need = std::max(need, ((long)u.nt * N / r + K - 1) / K);
            }
            int c = 0;
            while (c < kClasses - 1 && need > kClassBT[c]) c++;
            u.cls = (unsigned char)c;
            bb.tiles[c].push_back(u);
            bb.smem[c] = std::max(bb.smem[c], (size_t)u.nt * u.ld * 8);
        }
        bb.bytes += 16.0 * N * nv;
    }
    // largest tiles first: each queue's tail is made of short work
    for (int c = 0; c < kClasses; c++)
        std::stable_sort(bb.tiles[c].begin(), bb.tiles[c].end(), [](const TileDesc &a, const TileDesc &b) {
            return (long)a.N * a.nt > (long)b.N * b.nt;
        });
    for (DifGroup &g : bb.groups)
        std::stable_sort(g.calls.begin(), g.calls.end(), [&](int x, int y) {
            const DifArgs<float> &a = bb.calls[x], &b = bb.calls[y];
            return (long)a.N * std::min((long)a.vpb, a.nvec) > (long)b.N * std::min((long)b.vpb, b.nvec);
        });
    // the groups of the largest CTAs are launched first
    std::stable_sort(bb.groups.begin(), bb.groups.end(), [](const DifGroup &a, const DifGroup &b) { return a.smem > b.smem; });
    return true;
}

struct DevBatch {
    TileDesc *q = nullptr;            // the classes' queues, one after the other
    int off[kClasses] = {0, 0, 0, 0};  // first descriptor of each class
    int n[kClasses] = {0, 0, 0, 0};    // descriptors of each class
    size_t smem[kClasses] = {0, 0, 0, 0};
    int total = 0;
    std::vector<StepCall> steps;      // calls run through the plain path
    struct Group {
        bool cols;
        int nthr, first, n;
        size_t smem;
    };
    DifArgs<float> *calls = nullptr;  // the in-place mixed-radix kernel's calls and tiles
    DifTile *tiles = nullptr;
    std::vector<Group> groups;
};

static bool upload(const BatchBuild &bb, DevBatch &db) {
    db.steps = bb.steps;
    // one buffer, one copy: [tiles of the classes | calls | tiles of the groups]
    size_t nq = 0, nt = 0;
    for (int c = 0; c < kClasses; c++) nq += bb.tiles[c].size();
    for (const DifGroup &g : bb.groups) nt += (size_t)g.ntiles;
    const size_t oc = (nq * sizeof(TileDesc) + 15) / 16 * 16, ot = oc + bb.calls.size() * sizeof(DifArgs<float>),
                 bytes = std::max<size_t>(1, ot + nt * sizeof(DifTile));
    std::vector<unsigned char> host(bytes);
    TileDesc *hq = (TileDesc *)host.data();
    for (int c = 0; c < kClasses; c++) {
        db.off[c] = db.total;
        db.n[c] = (int)bb.tiles[c].size();
        db.smem[c] = bb.smem[c];
        if (db.n[c]) memcpy(hq + db.total, bb.tiles[c].data(), bb.tiles[c].size() * sizeof(TileDesc));
        db.total += db.n[c];
    }
    if (!bb.calls.empty()) memcpy(host.data() + oc, bb.calls.data(), bb.calls.size() * sizeof(DifArgs<float>));
    DifTile *ht = (DifTile *)(host.data() + ot);
    for (const DifGroup &g : bb.groups) {
        int first = db.groups.empty() ? 0 : db.groups.back().first + db.groups.back().n;
        db.groups.push_back({g.cols, g.nthr, first, (int)g.ntiles, g.smem});
        for (int c : g.calls) {
            const DifArgs<float> &a = bb.calls[c];
            for (long v0 = 0; v0 < a.nvec; v0 += a.vpb)
                ht[first++] = DifTile{c, (int)std::min((long)a.vpb, a.nvec - v0), v0};
        }
    }
    if (nq + nt == 0) return true;
    db.q = (TileDesc *)dmalloc(bytes);
    if (!db.q) return false;
    db.calls = (DifArgs<float> *)((unsigned char *)db.q + oc);
    db.tiles = (DifTile *)((unsigned char *)db.q + ot);
    return cuda_ok(cudaMemcpyAsync(db.q, host.data(), bytes, cudaMemcpyHostToDevice, device()->stream),
                   "batch queue upload");
}

template <int CBT>
static bool launch_class(const DevBatch &db, int c, cudaStream_t st) {
    Device *d = device();
    static std::atomic<bool> attr{false};  // set once; concurrent first calls both set it
    if (!attr) {
        if (!cuda_ok(cudaFuncSetAttribute(k_batch<CBT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)d->smem_optin - 512),
                     "cudaFuncSetAttribute"))
            return false;
        attr = true;
    }
    // CTAs resident at once for this class: the descriptor that many places
    // further down the queue is the one a finishing CTA's slot takes next
    int per_sm = 0;
    if (!cuda_ok(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch<CBT>, CBT, db.smem[c]),
                 "batch occupancy"))
        return false;
    const int ahead = std::max(1, per_sm) * d->sms;
    k_batch<CBT><<<db.n[c], CBT, db.smem[c], st>>>(db.q + db.off[c], db.n[c], ahead);
    count_launch();
    return cuda_ok(cudaGetLastError(), "k_batch launch");
}

static bool launch_cols(const DevBatch &db, cudaStream_t st) {
    Device *d = device();
    static std::atomic<bool> attr{false};  // set once; concurrent first calls both set it
    if (!attr) {
        if (!cuda_ok(cudaFuncSetAttribute(k_batch_cols, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)d->smem_optin - 512),
                     "cudaFuncSetAttribute"))
            return false;
        attr = true;
    }
    const int c = kColClass;
    k_batch_cols<<<db.n[c] * kColCluster, BT, db.smem[c], st>>>(db.q + db.off[c], db.n[c]);
    count_launch();
    return cuda_ok(cudaGetLastError(), "k_batch_cols launch");
}

static bool launch_one(const DevBatch &db, int c, cudaStream_t st) {
    switch (c) {
        case 0: return launch_class<256>(db, c, st);
        case 1: return launch_class<512>(db, c, st);
        case 2: return launch_class<1024>(db, c, st);
        default: return launch_cols(db, st);
    }
}

// Streams and events the classes run on side by side (forked from and joined
// back to the caller's stream; the same pattern is recorded into the graph).
constexpr int kStepStreams = 8;  // streams of the calls run through the plain path
constexpr int kDifStreams = 8;   // streams of the in-place mixed-radix kernel's groups
constexpr int kBatchStreams = kClasses + kStepStreams + kDifStreams;
struct BatchStreams {
    cudaStream_t s[kBatchStreams] = {};  // the classes', the plain-path calls', the groups'
    cudaEvent_t fork = nullptr, join[kBatchStreams] = {};
    bool ready = false;
};
static BatchStreams g_bs;
static std::mutex g_bs_mu;

static bool batch_streams() {
    std::lock_guard<std::mutex> lk(g_bs_mu);
    if (g_bs.ready) return true;
    bool ok = cuda_ok(cudaEventCreateWithFlags(&g_bs.fork, cudaEventDisableTiming), "batch event");
    for (int c = 0; c < kBatchStreams && ok; c++)
        ok = cuda_ok(cudaStreamCreateWithFlags(&g_bs.s[c], cudaStreamNonBlocking), "batch stream") &&
             cuda_ok(cudaEventCreateWithFlags(&g_bs.join[c], cudaEventDisableTiming), "batch event");
    g_bs.ready = ok;
    return ok;
}

static bool launch_group(const DevBatch &db, const DevBatch::Group &g, cudaStream_t st) {
    return dif_batch_go(g.cols, db.calls, db.tiles + g.first, g.n, g.nthr, g.smem, st);
}

static bool launch(const DevBatch &db, cudaStream_t st) {
    if (db.total == 0 && db.steps.empty() && db.groups.empty()) return true;
    if (db.total == 0 && db.steps.empty() && db.groups.size() == 1) return launch_group(db, db.groups[0], st);
    int used = 0, only = 0;
    for (int c = 0; c < kClasses; c++)
        if (db.n[c]) {
            used++;
            only = c;
        }
    if (used == 1 && db.steps.empty() && db.groups.empty()) return launch_one(db, only, st);
    if (!batch_streams()) return false;
    bool ok = cuda_ok(cudaEventRecord(g_bs.fork, st), "batch fork");
    if (!db.steps.empty()) {
        // calls of one plan share its scratch, so they all go to one stream, in order
        bool on[kStepStreams] = {};
        std::map<const Plan *, int> stream_of;
        for (const StepCall &c : db.steps) {
            const int k = stream_of.emplace(c.p, (int)stream_of.size() % kStepStreams).first->second;
            cudaStream_t sl = g_bs.s[kClasses + k];
            if (!on[k]) ok = ok && cuda_ok(cudaStreamWaitEvent(sl, g_bs.fork, 0), "batch fork");
            on[k] = true;
            ok = ok && enqueue_resident_c2c_f(c.p, c.x, c.y, sl, false);
        }
        for (int k = 0; k < kStepStreams && ok; k++)
            if (on[k])
                ok = cuda_ok(cudaEventRecord(g_bs.join[kClasses + k], g_bs.s[kClasses + k]), "batch join") &&
                     cuda_ok(cudaStreamWaitEvent(st, g_bs.join[kClasses + k], 0), "batch join");
    }
    // largest CTAs first: they hold the longest tiles
    for (int c = kClasses - 1; c >= 0 && ok; c--) {
        if (!db.n[c]) continue;
        ok = cuda_ok(cudaStreamWaitEvent(g_bs.s[c], g_bs.fork, 0), "batch fork") && launch_one(db, c, g_bs.s[c]) &&
             cuda_ok(cudaEventRecord(g_bs.join[c], g_bs.s[c]), "batch join") &&
             cuda_ok(cudaStreamWaitEvent(st, g_bs.join[c], 0), "batch join");
    }
    const int base = kClasses + kStepStreams, ng = (int)db.groups.size();
    for (int i = 0; i < ng && ok; i++) {
        cudaStream_t sg = g_bs.s[base + i % kDifStreams];
        if (i < kDifStreams) ok = cuda_ok(cudaStreamWaitEvent(sg, g_bs.fork, 0), "batch fork");
        ok = ok && launch_group(db, db.groups[i], sg);
    }
    for (int i = 0; i < std::min(ng, kDifStreams) && ok; i++)
        ok = cuda_ok(cudaEventRecord(g_bs.join[base + i], g_bs.s[base + i]), "batch join") &&
             cuda_ok(cudaStreamWaitEvent(st, g_bs.join[base + i], 0), "batch join");
    return ok;
}

static void free_dev(DevBatch &db) {
    dfree(db.q);
    db.q = nullptr;
    db.calls = nullptr;
    db.tiles = nullptr;
}

}  // namespace jv

using namespace jv;

struct jvsip_fftm_batchplan_s {
    DevBatch db;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    std::vector<const void *> blocks;  // output blocks, marked device-newer after a run
};

static void mark_outputs(size_t n, const vsip_fftm_f *const plans[], const vsip_cmview_f *const in[],
                         const vsip_cmview_f *const out[]) {
    for (size_t i = 0; i < n; i++) {
        Plan *p = plan_of(plans[i]);
        const vsip_cmview_f *y = (p->type == JV_CCFFTIP || !out || !out[i]) ? in[i] : out[i];
        Mirror *m = mirror_find(y->block);
        if (m) m->device_newer = true;
    }
}

extern "C" {

int jvsip_fftm_batch_f(size_t n, const vsip_fftm_f *const plans[], const vsip_cmview_f *const in[],
                       const vsip_cmview_f *const out[]) {
    if (n == 0) return 0;
    if (!plans || !in) {
        set_error(E_ARG, "batch: null arrays");
        return E_ARG;
    }
    BatchBuild bb;
    if (!build_tiles(n, plans, in, out, bb)) return jvsip_gpu_last_error();
    DevBatch db;
    Device *d = device();
    bool ok = upload(bb, db) && launch(db, d->stream);
    free_dev(db);  // stream-ordered reuse of the pool
    if (!ok) return jvsip_gpu_last_error() ? jvsip_gpu_last_error() : E_CUDA;
    mark_outputs(n, plans, in, out);
    return 0;
}

jvsip_fftm_batchplan_f *jvsip_fftm_batch_create_f(size_t n, const vsip_fftm_f *const plans[],
                                                  const vsip_cmview_f *const in[], const vsip_cmview_f *const out[]) {
    if (!plans || !in) {
        set_error(E_ARG, "batch: null arrays");
        return nullptr;
    }
    BatchBuild bb;
    if (!build_tiles(n, plans, in, out, bb)) return nullptr;
    jvsip_fftm_batchplan_f *b = new (std::nothrow) jvsip_fftm_batchplan_f();
    if (!b) {
        set_error(E_ALLOC, "batch plan");
        return nullptr;
    }
    Device *d = device();
    if (!upload(bb, b->db) || !cuda_ok(cudaStreamSynchronize(d->stream), "batch upload")) {
        free_dev(b->db);
        delete b;
        return nullptr;
    }
    // record the launch once; runs replay the graph
    cudaStream_t cs = nullptr;
    bool ok = cuda_ok(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking), "capture stream");
    ok = ok && cuda_ok(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal), "begin capture");
    if (ok) {
        bool lk = launch(b->db, cs);
        ok = cuda_ok(cudaStreamEndCapture(cs, &b->graph), "end capture") && lk;
    }
    ok = ok && cuda_ok(cudaGraphInstantiate(&b->exec, b->graph, 0), "graph instantiate");
    if (cs) cudaStreamDestroy(cs);
    if (!ok) {
        if (b->exec) cudaGraphExecDestroy(b->exec);
        if (b->graph) cudaGraphDestroy(b->graph);
        free_dev(b->db);
        delete b;
        return nullptr;
    }
    for (size_t i = 0; i < n; i++) {
        Plan *p = plan_of(plans[i]);
        const vsip_cmview_f *y = (p->type == JV_CCFFTIP || !out || !out[i]) ? in[i] : out[i];
        b->blocks.push_back(y->block);
    }
    return b;
}

int jvsip_fftm_batch_run_f(jvsip_fftm_batchplan_f *b) {
    if (!b) return E_ARG;
    Device *d = device();
    if (!d) return E_NODEVICE;
    if (b->db.total == 0 && b->db.steps.empty() && b->db.groups.empty()) return 0;
    if (!cuda_ok(cudaGraphLaunch(b->exec, d->stream), "batch graph launch")) return E_CUDA;
    count_launch();
    for (const void *blk : b->blocks) {
        Mirror *m = mirror_find(blk);
        if (m) m->device_newer = true;
    }
    return 0;
}

int jvsip_fftm_loop_f(size_t n, const vsip_fftm_f *const plans[], const vsip_cmview_f *const in[],
                      const vsip_cmview_f *const out[]) {
    if (n && (!plans || !in)) {
        set_error(E_ARG, "loop: null arrays");
        return E_ARG;
    }
    for (size_t i = 0; i < n; i++) {
        Plan *p = plan_of(plans[i]);
        if (!p) {
            set_error(E_ARG, "loop: not a plan of this library");
            return E_ARG;
        }
        if (p->type == JV_CCFFTIP || !out || !out[i]) vsip_ccfftmip_f(plans[i], in[i]);
        else vsip_ccfftmop_f(plans[i], in[i], out[i]);
        const int e = jvsip_gpu_last_error();
        if (e) return e;
    }
    return 0;
}

int jvsip_fftm_batch_destroy_f(jvsip_fftm_batchplan_f *b) {
    if (!b) return 0;
    Device *d = device();
    if (d) cudaStreamSynchronize(d->stream);
    if (b->exec) cudaGraphExecDestroy(b->exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    free_dev(b->db);
    delete b;
    return 0;
}

}  // extern "C"
