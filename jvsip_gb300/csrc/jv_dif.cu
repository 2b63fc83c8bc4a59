// jv_dif.cu -- host side of the in-place mixed-radix kernel (jv_dif.cuh): the
// radix schedule and shared-memory pitch of a length (dif_schedule), its twiddle
// tables (shared by all plans of the length) and the launchers.
#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <new>
#include <tuple>

#include "jv_dif.cuh"
#include "jv_dif_tile.h"

namespace jv {

// arithmetic instructions per point of a codelet, R = 0..16
static const double kDifCost[17] = {0,   0,    2.0,  4.0,  4.0,  7.2,  7.3, 9.4, 7.0,
                                    9.8, 10.8, 13.6, 10.0, 15.7, 13.1, 13.3, 10.0};

// Cost of a radix-R pass in issue slots per point: the butterfly, and beside
// it the shared-memory accesses, addresses and twiddles (single precision) or
// the twiddles alone (double precision, bound by its FP64 pipe); per butterfly
// the index arithmetic.
static double pass_cost(int R, int prec) {
    return prec == P_F32 ? kDifCost[R] + 10.0 + 20.0 / R : kDifCost[R] + 4.5;
}

// multisets of codelet radices (descending) with product n
static void multisets(long n, int maxr, std::vector<int> &cur, std::vector<std::vector<int>> &out) {
    if (n == 1) {
        if (cur.size() >= 2 && (int)cur.size() <= kDifMaxPass) out.push_back(cur);
        return;
    }
    if ((int)cur.size() >= kDifMaxPass) return;
    for (int R = std::min<long>(maxr, n); R >= 2; R--) {
        if (n % R) continue;
        cur.push_back(R);
        multisets(n / R, R, cur, out);
        cur.pop_back();
    }
}

// shared-memory wavefronts of the middle (read and write) and last passes of
// schedule r with block pitch P1, sampled over groups of W lanes (W slots of
// one element each make a wavefront)
static long bank_waves(const std::vector<int> &r, long N, long P1, int W) {
    const int np = (int)r.size();
    long waves = 0;
    long M = N / r[0];
    for (int p = 1; p < np; p++) {
        const bool last = p == np - 1;
        const long S = last ? 1 : M / r[p], NR = N / r[p], NB1 = N / r[0] / r[p];
        const long ngr = (NR + W - 1) / W, take = std::min<long>(ngr, 6);
        for (long g = 0; g < take; g++) {
            const long b0 = g * ngr / take * W;
            int hit[16] = {0};
            int worst = 0;
            for (long b = b0; b < std::min(b0 + W, NR); b++) {
                long pos;
                if (last) {
                    long rem = b / r[0];
                    pos = (b % r[0]) * P1;
                    long Sq = N / r[0];
                    for (int i = 1; i + 1 < np; i++) {
                        Sq /= r[i];
                        pos += (rem % r[i]) * Sq;
                        rem /= r[i];
                    }
                } else {
                    const long k1 = b / NB1, u = b % NB1;
                    pos = k1 * P1 + u + (u / S) * (M - S);
                }
                worst = std::max(worst, ++hit[pos % W]);
            }
            waves += (last ? 1 : 2) * worst * ngr / take * r[p];
        }
        M = S;
    }
    return waves;
}

// The multiset of radices of least cost with product N (empty: N has a prime
// above 13 or fewer than two codelet factors).  Real transforms' pair pass (the
// last of R2C, the first of C2R) takes a radix of at most kDifPairMax.
static std::vector<int> least_cost(long N, int prec, int cls, double *cost) {
    std::vector<std::vector<int>> sets;
    std::vector<int> cur, pick;
    *cost = 1e30;
    if (N < 4 || N > 32768) return pick;
    multisets(N, 16, cur, sets);
    for (const std::vector<int> &m : sets) {
        if (cls && m.back() > kDifPairMax) continue;
        double c = 0;
        for (int R : m) c += pass_cost(R, prec);
        if (c < *cost) {
            *cost = c;
            pick = m;
        }
    }
    return pick;
}

// The schedule of length N: the radices of least cost, in the order and with
// the block pitch of the fewest shared-memory wavefronts (larger first radices
// on ties).
static bool dif_schedule(long N, int prec, int cls, std::vector<int> &rad, long *P1) {
    double cost;
    const std::vector<int> pick = least_cost(N, prec, cls, &cost);
    if (pick.empty()) return false;
    const int W = prec == P_F32 ? 16 : 8;
    long bw = -1;
    std::vector<int> q = pick;
    std::sort(q.begin(), q.end());
    int tried = 0;
    do {
        if (cls && (cls == 1 ? q.back() : q.front()) > kDifPairMax) continue;
        const long S1 = N / q[0];
        for (int pad = 0; pad < W; pad++) {
            const long w = bank_waves(q, N, S1 + pad, W);
            if (bw < 0 || w < bw || (w == bw && q[0] > rad[0])) {
                bw = w;
                rad = q;
                *P1 = S1 + pad;
            }
        }
    } while (++tried < 24 && std::next_permutation(q.begin(), q.end()));
    return true;
}

// ---------------------------------------------------------------- compiled-in schedules
void dif_fix_c2c_1(std::vector<DifFixEntry> &out);
void dif_fix_c2c_2(std::vector<DifFixEntry> &out);
void dif_fix_c2c_3(std::vector<DifFixEntry> &out);
void dif_fix_long_1(std::vector<DifFixEntry> &out);
void dif_fix_rows_1(std::vector<DifFixEntry> &out);
void dif_fix_rows_2(std::vector<DifFixEntry> &out);
void dif_fix_taper_1(std::vector<DifFixEntry> &out);
void dif_fix_taper_2(std::vector<DifFixEntry> &out);
void dif_fix_power_1(std::vector<DifFixEntry> &out);
void dif_fix_r2c_1(std::vector<DifFixEntry> &out);
void dif_fix_r2c_2(std::vector<DifFixEntry> &out);
void dif_fix_c2r_1(std::vector<DifFixEntry> &out);
void dif_fix_c2r_2(std::vector<DifFixEntry> &out);

const DifFixEntry *dif_fix(long N, int cls) {
    // built once, thread-safely, on the first call
    static const std::vector<std::map<long, DifFixEntry>> tab = []() {
        std::vector<std::map<long, DifFixEntry>> t(3);
        std::vector<DifFixEntry> v[6];
        dif_fix_c2c_1(v[0]);
        dif_fix_c2c_2(v[0]);
        dif_fix_c2c_3(v[0]);
        dif_fix_rows_1(v[0]);
        dif_fix_rows_2(v[0]);
        dif_fix_r2c_1(v[1]);
        dif_fix_r2c_2(v[1]);
        dif_fix_c2r_1(v[2]);
        dif_fix_c2r_2(v[2]);
        dif_fix_long_1(v[3]);
        dif_fix_taper_1(v[4]);
        dif_fix_taper_2(v[4]);
        dif_fix_power_1(v[5]);
        for (int c = 0; c < 3; c++)
            for (const DifFixEntry &e : v[c]) t[c][e.N] = e;
        for (const DifFixEntry &e : v[3]) {
            DifFixEntry &d = t[0][e.N];
            d.step = e.step;
            for (int i = 0; i < 3; i++) d.vec[i] = e.vec[i];
        }
        for (const DifFixEntry &e : v[4]) {
            t[1][e.N].taper = e.taper;
            t[1][e.N].vtaper = e.vtaper;
        }
        for (const DifFixEntry &e : v[5]) t[0][e.N].power = e.power;
        return t;
    }();
    auto it = tab[cls].find(N);
    return it == tab[cls].end() ? nullptr : &it->second;
}

// ---------------------------------------------------------------- tables
static std::mutex g_dif_mu;
static std::map<std::tuple<long, int, int>, DifTab> g_dif;
// schedules and CTA shapes found so far (host only; one small entry per length
// a program has planned, at most 16384 x 3): the search takes 0.1 to 0.3 ms
static std::map<std::tuple<long, int, int>, DifTab> g_found;

template <typename T>
static void *upload_tables(const std::vector<int> &rad, long N, const std::vector<double> &roots,
                           std::vector<int> &two) {
    std::vector<T> tw;
    long M = N;
    for (size_t p = 0; p + 1 < rad.size(); p++) {
        const long R = rad[p], S = M / R, step = N / M;
        two.push_back((int)(tw.size() / 2));
        for (long k = 0; k < R; k++)
            for (long n = 0; n < S; n++) {
                tw.push_back((T)roots[2 * (k * n * step)]);  // k*n < M
                tw.push_back((T)roots[2 * (k * n * step) + 1]);
            }
        M = S;
    }
    two.push_back(0);
    return table_upload(tw.data(), tw.size() * sizeof(T), "twiddle upload");
}

// Double precision: an FP64 instruction takes the pipe as long for one lane of a
// warp as for 32 and the pipe serves an SM's tiles one after another, so a call's
// time is the tiles of the fullest SM times the FP64 instructions of a tile's warps
// (of four warps at a time where an SM has one tile: its four quarters have a pipe
// each), at 0.30 ns per instruction and lane, and 1 us a pass.
static double f64_work(const int *rad, int np, long N, long v, bool smem, int lanes) {
    double c = 0;
    for (int i = 0; i < np; i++) {
        const int R = rad[i];
        // constants folded into 52 and 144 instructions here, products there
        double per = R == 16 && !smem ? 9.0 : R == 8 && !smem ? 6.5 : kDifCost[R];
        if (smem ? i > 0 : i + 1 < np) per += 4.0 * (R - 1) / R;  // the twiddles of a pass
        c += (double)((v * (N / R) + lanes - 1) / lanes * lanes) * per * R;
    }
    return c;
}
static double f64_time(const int *rad, int np, long N, long v, long nvec, bool smem, long sms) {
    const long tiles = (nvec + v - 1) / v, k = (tiles + sms - 1) / sms;
    double us = 0.0003 * k * f64_work(rad, np, N, v, smem, k > 1 ? 32 : 128) + 1.0 * np;
    const int most = *std::max_element(rad, rad + np);
    // passes of fewer than three warps leave quarters of the SM idle
    if (!smem && k > 1 && v * (N / most) < 96) us *= 1.2;
    if (smem && std::find(rad, rad + np, 7) != rad + np) us *= 1.4;  // 64 x 343 23.7 us, 11 here
    return us;
}

// Transforms per tile of a double-precision row call: of the least time, in up to
// 72 KB (three CTAs per SM).  Where several have it, the fewest if an SM has few
// tiles (a tile's chain of passes is shorter), else the fewest that give every pass
// four warps, one for each quarter of the SM (381300 x 22: 16 to a tile 646 us, 64 to
// a tile 355; 103563 x 81: 32 to a tile 423, 64 to a tile 454).
static long f64_rows_per_tile(const DifTab &t, long nvec, double *time) {
    static const long cand[] = {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 16, 20, 24, 28, 32, 40, 48, 56, 64};
    constexpr int kCand = sizeof cand / sizeof cand[0];
    const int np = (int)t.radix.size();
    const long ldb = t.radix[0] * t.P1 * 16, sms = device()->sms;
    double best = 1e300, e[kCand];
    int n = 0;
    for (; n < kCand && (n == 0 || cand[n] * ldb <= 72 * 1024); n++) {
        e[n] = f64_time(t.radix.data(), np, t.N, cand[n], nvec, false, sms);
        best = std::min(best, e[n]);
    }
    const long least = t.N / *std::max_element(t.radix.begin(), t.radix.end());
    int pick = 0, last = n - 1;
    while (e[pick] > 1.01 * best) pick++;
    while (e[last] > 1.01 * best) last--;
    if (nvec >= 4 * cand[last] * sms)
        while (pick < last && (cand[pick] * least < 128 || e[pick] > 1.01 * best)) pick++;
    *time = e[pick];
    return cand[pick];
}

// The tile of nvec rows, 0 where they run on the shared-memory kernel, whose schedule
// is rad and which takes 1024 points to a CTA: on this one where every tile has an SM,
// or by the times above.  Of 1756 calls (4-8192 points, 1 to 2^23 / N rows) 11 are 3 %
// or more slower than there and the average is 1.20x faster (us, there and here: 2^24
// points of 100 1114 and 867, 600 1470 and 1184; 16 x 343 23.7 and 11.0; 1000 x 972
// and 450 x 1620 stay there).  Schedules of radices 2^k do: their folded codelets take
// the same instructions.
static long f64_rows_or_smem(const DifTab &t, const int *rad, int np, long nvec, double hand = 1.0) {
    bool pow2 = true;
    for (int i = 0; i < np; i++) pow2 = pow2 && (rad[i] & (rad[i] - 1)) == 0;
    if (pow2 || np < 2) return 0;
    double time;
    const long v = f64_rows_per_tile(t, nvec, &time), sms = device()->sms;
    const bool pays = (nvec + v - 1) / v <= sms ||
                      hand * time < f64_time(rad, np, t.N, std::max(1L, std::min(nvec, 1024 / t.N)), nvec, true, sms);
    return pays ? v : 0;
}

// False where the radices alone, in whatever order, show that it would not pay: a
// plan that stays on the shared-memory kernel is made without the search for their
// order and pitch (0.1 to 0.3 ms).
static bool dif_f64_may_pay(long N, const std::vector<int> &smem, long nvec) {
    DifTab t;
    double cost;
    t.N = N;
    t.radix = least_cost(N, P_F64, 0, &cost);
    if (t.radix.empty()) return false;
    t.P1 = N / t.radix[0];
    return f64_rows_or_smem(t, smem.data(), (int)smem.size(), nvec, 0.95) > 0;
}

// Lengths without such a schedule (factors 11 and 13): whether `tiles` tiles of v
// transforms run here rather than as passes over global memory, which spread a call
// evenly over the SMs but cost 30 us and 17 us a pass at least, 21 for one of 13 (us,
// passes and here: 1 x 5632 55 and 78, 64 x 6500 97 and 115, 161 x 6500 196 and 223;
// 150 x 6500 173 and 116, 16 x 2816 51 and 39, 16 x 2197 76 and 45).
static bool dif_f64_beats_passes(const DifTab &t, long v, long nvec) {
    const int np = (int)t.radix.size();
    double per = 0, floor = 0;
    for (int i = 0; i < np; i++) {
        const int R = t.radix[i];
        floor += R == 13 ? 21.0 : 17.0;
        per += (kDifCost[R] + 4.0 * (R - 1) / R) * (R == 11 || R == 13 ? 1.13 : 1.45);
    }
    const long sms = device()->sms;
    const double passes = 0.0003 * per * t.N * nvec / sms;
    return f64_time(t.radix.data(), np, t.N, v, nvec, false, sms) < std::max(floor, 30.0 + passes);
}

long dif_f64_rows(const DifTab &t, const int *rad, int np, long nvec) {
    if (rad) return f64_rows_or_smem(t, rad, np, nvec);
    double time;
    const long v = f64_rows_per_tile(t, nvec, &time);
    return dif_f64_beats_passes(t, v, nvec) ? v : 0;
}

// CTA shape of row calls: vpb transforms in nthr threads, chosen by the idle
// thread slots of the passes' last rounds, the threads and points an SM then
// holds, and the CTA's size.  Small CTAs (1200 to 2400 points) are in
// different phases and end the last wave sooner; the weights are fitted to
// sweeps of 51 lengths on 2^24 points, of which the rule's choice is 2 % off
// the best on average (us, transforms x threads): 100 points 12 x 128 45.3, 24
// x 256 49.3, 32 x 192 49.3; 1200: 2 x 128 60.5, 4 x 256 62.6, 6 x 320 63.5;
// 2400: 1 x 160 62.1, 2 x 320 67.8, 3 x 512 70.1.
static void row_shape(DifTab &t, int cls) {
    if (t.prec == P_F64) return;  // by the call (f64_rows_per_tile)
    const long maxt = 1024, ldb = t.radix[0] * t.P1 * 8, unit = 1200;
    const size_t np = t.radix.size();
    double best = 1e30;
    t.vpb = 1;
    t.nthr = 96;
    for (long v = 1; v == 1 || v * t.N <= 2 * unit; v++) {
        for (long th = 96; th <= maxt; th += 32) {
            double slots = 0;
            for (size_t i = 0; i < np; i++) {
                const int R = t.radix[i];
                const bool pair = (cls == 1 && i + 1 == np) || (cls == 2 && i == 0);
                const long per = t.N / R, nb = v * (pair ? per / 2 + 1 : per);
                slots += (double)((nb + th - 1) / th) * pass_cost(R, t.prec) * R * (pair ? 2.0 : 1.0);
            }
            slots = slots * th / (double)(v * t.N);
            const long ctas = std::min({32L, maxt / th, 227L * 1024 / (v * ldb + 1024)});
            if (ctas < 1) continue;
            const double act = (double)ctas * th, want = 0.9 * maxt, pts = (double)ctas * v * t.N;
            if (act < want) slots *= sqrt(want / act);
            if (pts < 10.0 * unit) slots *= 10.0 * unit / pts;
            if (v > 1 && v * t.N > unit) slots *= pow((double)(v * t.N) / unit, 0.4);
            if (slots < best) {
                best = slots;
                t.vpb = v;
                t.nthr = (int)th;
            }
        }
    }
}

// the schedule's part of the kernel's arguments, made once for a table
template <typename T> static std::shared_ptr<const void> dif_fill(const DifTab &t) {
    auto made = std::make_shared<DifArgs<T>>();
    DifArgs<T> &a = *made;
    memset(&a, 0, sizeof a);
    a.N = (int)t.N;
    a.np = (int)t.radix.size();
    a.P1 = (int)t.P1;
    a.LD = (int)(t.radix[0] * t.P1);
    a.tw = (const typename cplx_t<T>::t *)t.d_tw;
    long M = t.N;
    for (int i = 0; i < a.np; i++) {
        DifPass &p = a.p[i];
        p.R = t.radix[i];
        p.S = (int)(M / p.R);
        p.NR = (int)(t.N / p.R);
        p.mstep = (int)M - p.S;
        p.NB1 = (int)(t.N / t.radix[0] / p.R);
        p.two = t.two[i];
        p.mNR = magic_host((unsigned long)p.NR);
        p.mNB1 = magic_host((unsigned long)p.NB1);
        p.mS = magic_host((unsigned long)p.S);
        p.mR = magic_host((unsigned long)p.R);
        M = p.S;
    }
    if (t.cls == 1) a.mH = magic_host((unsigned long)(a.p[a.np - 1].NR / 2 + 1));
    if (t.cls == 2) a.mH = magic_host((unsigned long)(a.p[0].S / 2 + 1));
    return made;
}
template <typename T> static const DifArgs<T> &dif_base(const DifTab &t) {
    return *static_cast<const DifArgs<T> *>(t.args.get());
}

const DifTab *dif_acquire(long N, int prec, int cls, const std::vector<double> *roots,
                          const std::vector<int> *other, long nvec) {
    if (N > (prec == P_F32 ? 16384 : 8192) || (prec == P_F64 && cls != 0)) return nullptr;
    std::lock_guard<std::mutex> lk(g_dif_mu);
    auto key = std::make_tuple(N, prec, cls);
    auto it = g_dif.find(key);
    if (it != g_dif.end()) {
        if (other && !f64_rows_or_smem(it->second, other->data(), (int)other->size(), nvec)) return nullptr;
        it->second.refs++;
        return &it->second;
    }
    DifTab t;
    const DifFixEntry *fix = prec == P_F32 ? dif_fix(N, cls) : nullptr;
    if (fix) {
        t.radix = fix->radix;
        t.P1 = fix->P1;
        t.fix = fix;
    }
    t.N = N;
    t.prec = prec;
    t.cls = cls;
    if (!fix) {
        auto seen = g_found.find(key);
        if (seen == g_found.end()) {
            if (other && !dif_f64_may_pay(N, *other, nvec)) return nullptr;
            if (dif_schedule(N, prec, cls, t.radix, &t.P1)) row_shape(t, cls);
            seen = g_found.emplace(key, t).first;
        }
        if (seen->second.radix.empty()) return nullptr;  // no schedule
        t = seen->second;
    }
    if (other && !f64_rows_or_smem(t, other->data(), (int)other->size(), nvec)) return nullptr;
    const int err0 = jvsip_gpu_last_error();
    std::vector<double> own;
    if (!roots) {
        own = unit_roots(N);
        roots = &own;
    }
    t.d_tw = prec == P_F32 ? upload_tables<float>(t.radix, N, *roots, t.two)
                           : upload_tables<double>(t.radix, N, *roots, t.two);
    if (!t.d_tw) {  // the general kernels take the plan's calls
        if (!err0 && jvsip_gpu_last_error()) jvsip_gpu_clear_error();
        return nullptr;
    }
    if (fix) {
        t.vpb = fix->vpb;
        t.nthr = fix->nthr;
    }
    t.args = prec == P_F32 ? dif_fill<float>(t) : dif_fill<double>(t);
    t.refs = 1;
    auto &slot = g_dif[key];
    slot = t;
    return &slot;
}

void dif_release(const DifTab *t) {
    if (!t) return;
    std::lock_guard<std::mutex> lk(g_dif_mu);
    auto it = g_dif.find(std::make_tuple(t->N, t->prec, t->cls));
    if (it == g_dif.end() || --it->second.refs > 0) return;
    dfree(it->second.d_tw);
    g_dif.erase(it);
}

// ---------------------------------------------------------------- launch
template <typename T> static bool interleaved_c(const CView &v) {
    return v.cst == 2 && (const T *)v.im == (const T *)v.re + 1 && (uintptr_t)v.re % (2 * sizeof(T)) == 0;
}
// rows of len elements that do not overlap
static bool apart(long vs, long len, long nvec) { return nvec <= 1 || labs(vs) >= len; }
// real rows of unit stride, even offset and pitch: x_2n, x_2n+1 one complex element
template <typename T> static bool real_pairs(const RView &r, long len, long nvec) {
    return r.rst == 1 && r.es == 1 && r.off % 2 == 0 && (nvec <= 1 || (r.vs % 2 == 0 && labs(r.vs) >= len)) &&
           (uintptr_t)r.a % (2 * sizeof(T)) == 0;
}

// Points of a column call from which tiles of 4 columns are too narrow.  Tiles of
// 4 against 8 (run-time schedule) at 2^26 points, us: 1125 points 475 and 321,
// 1350: 499 and 334, 1500: 499 and 436, 1792: 482 and 410, 1920: 441 and 336, 2048:
// 393 and 334 (1944: 422 and 485); at 2^25 points 1500: 214 and 222, 2000: 199 and
// 232, 2048: 150 and 168.
constexpr long kColWidePts = 5L << 23;

// The kernel's arguments for a call and its CTA: tuned > 0 asks for that many
// transforms (a power of two for column tiles); the call's tiles are to occupy
// `sms` SMs (a call of a batch has its share); column tiles become narrower than
// four for it where `narrow`.  False when the call does not qualify.
template <typename T>
static bool dif_args(const Job &j, long tuned, long sms, bool narrow, DifArgs<T> &a, DifCta &cta) {
    typedef typename cplx_t<T>::t C;
    const DifTab *t = j.dif;
    if (!t || j.no_fast || j.no_dif || j.nvec <= 0 || j.gram || j.taper_n) return false;
    const CView &ci = j.cin, &co = j.cout;
    a = dif_base<T>(*t);
    bool rows = true, split = false;
    if (j.kind == K_C2C) {
        split = ci.cst == 1 && co.cst == 1;
        if (!split && (!interleaved_c<T>(ci) || !interleaved_c<T>(co))) return false;
        rows = ci.es == 1 && co.es == 1;
        if (rows) {
            if (!apart(ci.vs, j.N, j.nvec) || !apart(co.vs, j.N, j.nvec)) return false;
        } else {
            // adjacent transforms, their elements at least the whole set apart
            if (labs(ci.vs) != 1 || labs(co.vs) != 1 || j.nvec < 2 || labs(ci.es) < j.nvec || labs(co.es) < j.nvec ||
                j.tma_columns == 1)
                return false;
        }
        if (split) {
            a.in_re = (const T *)ci.re + ci.off;
            a.in_im = (const T *)ci.im + ci.off;
            a.out_re = (T *)co.re + co.off;
            a.out_im = (T *)co.im + co.off;
        } else {
            a.in = (const C *)ci.re + ci.off;
            a.out = (C *)co.re + co.off;
        }
        a.es_in = ci.es;
        a.vs_in = ci.vs;
        a.es_out = co.es;
        a.vs_out = co.vs;
        a.smask_in = (j.conj_in < 0 ? j.inv : j.conj_in) ? 0x80000000u : 0u;
        a.smask_out = (j.conj_out < 0 ? j.inv : j.conj_out) ? 0x80000000u : 0u;
    } else if (sizeof(T) != 4 || !j.thalf) {
        return false;
    } else if (j.kind == K_R2C) {
        if (!real_pairs<T>(j.rin, 2 * j.N, j.nvec) || !interleaved_c<T>(co)) return false;
        // spectrum rows apart, or interleaved element by element (a column-major spectrum)
        if (co.es == 1 ? !apart(co.vs, j.N + 1, j.nvec)
                       : (co.es == 0 || co.vs == 0 || labs(co.vs) * j.nvec > labs(co.es)))
            return false;
        a.in = (const C *)j.rin.a + j.rin.off / 2;
        a.vs_in = j.rin.vs / 2;
        a.es_in = 1;
        a.out = (C *)co.re + co.off;
        a.es_out = co.es;
        a.vs_out = co.vs;
        a.thalf = (const C *)j.thalf;
    } else {
        if (!interleaved_c<T>(ci) || ci.es != 1 || !apart(ci.vs, j.N + 1, j.nvec) ||
            !real_pairs<T>(j.rout, 2 * j.N, j.nvec))
            return false;
        a.in = (const C *)ci.re + ci.off;
        a.vs_in = ci.vs;
        a.es_in = 1;
        a.out = (C *)j.rout.a + j.rout.off / 2;
        a.vs_out = j.rout.vs / 2;
        a.es_out = 1;
        a.smask_out = 0x80000000u;
        a.thalf = (const C *)j.thalf;
    }
    a.nvec = j.nvec;
    a.has_scale = j.has_scale;
    a.scale = j.has_scale ? (T)j.scale : (T)1;
    const size_t cap = device()->smem_optin;
    long vpb, nthr;
    if (rows && sizeof(T) == 8) {
        vpb = j.nvec == j.dif_rows_of ? j.dif_rows : dif_f64_rows(*t, j.twg ? j.radix : nullptr, j.npass, j.nvec);
        if (vpb < 1) return false;
        // rows on the host arrays: more, smaller CTAs keep the link busy (1000 x 1000 168
        // us, 196 with the tile of device rows)
        while (j.host && vpb > 1 && (j.nvec + vpb - 1) / vpb < 2L * sms) vpb = (vpb + 1) / 2;
        nthr = std::min(256L, (vpb * j.N / *std::min_element(t->radix.begin(), t->radix.end()) + 31) / 32 * 32);
    } else if (rows) {
        vpb = t->vpb;
        nthr = t->nthr;
        if (tuned > 0 && tuned != vpb) {
            vpb = std::max(1L, std::min(tuned, (long)(cap / (a.LD * sizeof(C)))));
            nthr = std::min(512L, std::max(64L, (vpb * j.N / 16 + 31) / 32 * 32));
        } else if (tuned <= 0) {
            // few transforms: smaller CTAs, so that more SMs work on them, with
            // every pass in one round
            while (vpb > 1 && (j.nvec + vpb - 1) / vpb < 2L * sms) vpb = (vpb + 1) / 2;
            if (vpb < t->vpb)
                nthr = std::min(256L, (vpb * j.N / *std::min_element(t->radix.begin(), t->radix.end()) + 31) / 32 * 32);
        }
    } else {
        // Column tiles, 64 KB or less: 16 adjacent transforms (128-byte rows of
        // the tile) up to 256 points, 8 up to 1200, 4 beyond, about 16 points
        // per thread.  Measured on 2^23 points (us; transforms x threads): 256
        // points 16 x 256 29.2, 32 x 512 31.5, 4 x 64 34.8; 640: 8 x 320 40.3,
        // 16 x 512 41.2, 4 x 160 45.4; 1200: 8 x 512 43.2, 4 x 320 45.0; 1500:
        // 4 x 320 43.2, 8 x 640 50.2; 3000: 4 x 512 53.6, 8 x 1024 59.9.
        const long pts = sizeof(T) == 4 ? 9600 : 4800;
        a.lgv = sizeof(T) == 4 ? 4 : 3;
        while (a.lgv > 2 && (j.N << a.lgv) > (a.lgv == 4 ? 4096 : pts)) a.lgv--;
        if (t->fix && t->fix->vcol)
            for (a.lgv = 0; (1 << a.lgv) < t->fix->vcol; a.lgv++) {
            }
        // calls far beyond L2: rows of 32 bytes, a megabyte and more apart, cost
        // memory twice their bytes, so tiles of 8 wherever they fit
        if (sizeof(T) == 4 && a.lgv == 2 && j.nbatch <= 1 && (j.N << 3) <= 16384 &&
            j.nvec * j.N >= kColWidePts)
            a.lgv = 3;
        // few columns: tiles of 4, so that more SMs work on them
        if (((j.nvec - 1) >> a.lgv) + 1 < sms && j.nbatch <= 1) a.lgv = std::min(a.lgv, 2);
        if (tuned > 0) a.lgv = dif_col_tuned(tuned, j.nvec);
        while (a.lgv > 0 && ((size_t)a.LD << a.lgv) * sizeof(C) > cap) a.lgv--;
        // down to one column where SMs would be idle and no compiled-in kernel
        // takes the tile: a tile's time is its chain of loads and passes then (us,
        // narrow against 4 to a tile: split columns 7000 x 16 16.7 and 26.4, 5000 x 2
        // 6.8 and 14.8, 3000 x 150 12.9 and 15.2, 7000 x 300 25.8 in twos, 34.8 in
        // fours and 46.7 in ones, two waves; 13312 x 100 24.8 and 35.3.  Compiled in,
        // fours stay: 1000 x 16 3.8 and 4.5 in ones)
        const bool fixed = sizeof(T) == 4 && !split && t->fix &&
                           ((t->fix->cols && (1 << a.lgv) == t->fix->vcol) || (t->fix->cols4 && a.lgv == 2));
        if (narrow && !fixed) a.lgv = dif_col_narrow(a.lgv, j.nvec, sms);
        vpb = 1L << a.lgv;
        // some columns of a long length that only this kernel takes in one launch: the
        // passes over global memory use more of the SMs (us, here and there: 14641 x 16
        // 30 and 22, split 13312 x 32 47 and 33, split 8788 x 32 32 and 25; 11264 x 16
        // 24 and 25, 13312 x 4 17 and 23, x 64 28 and 38)
        if (!j.twg && (sizeof(T) == 8 ? !dif_f64_beats_passes(*t, vpb, j.nvec)
                                      : (split ? 2 : 1) * j.N > 13000 && j.nvec >= 8 && j.nvec <= (split ? 64 : 32)))
            return false;
        nthr = dif_col_threads(j.N, a.lgv, sizeof(T) == 4, narrow && ((j.nvec - 1) >> a.lgv) < sms);
    }
    a.vpb = (int)vpb;
    cta.nthr = (int)nthr;
    cta.smem = (size_t)a.LD * vpb * sizeof(C);
    cta.rows = rows;
    cta.split = split;
    return cta.smem <= cap;
}

template <typename T>
static bool launch_dif_t(const Job &j, cudaStream_t st) {
    DifArgs<T> a;
    DifCta c;
    if (j.nbatch > 1 || j.tw_lo || !dif_args<T>(j, 0, device()->sms, true, a, c)) return false;
    if constexpr (sizeof(T) == 4) {
        const DifFixEntry *f = j.dif->fix;
        if (f && !c.split && c.rows && f->rows) return f->rows(a, c.smem, st, 1);
        if (f && !c.split && !c.rows && f->cols && a.vpb == f->vcol) return f->cols(a, c.smem, st, 1);
        if (f && !c.split && !c.rows && f->cols4 && a.vpb == 4) return f->cols4(a, c.smem, st, 1);
        if (j.kind == K_R2C) return dif_go<T, DIF_R2C, false>(a, c.nthr, c.smem, st);
        if (j.kind == K_C2R) return dif_go<T, DIF_C2R, false>(a, c.nthr, c.smem, st);
        if (c.split)
            return c.rows ? dif_go<T, DIF_SPLIT, false>(a, c.nthr, c.smem, st)
                          : dif_go<T, DIF_SPLIT, true>(a, c.nthr, c.smem, st);
    } else if (c.split || (!c.rows && j.twg)) {
        return false;  // columns: only lengths the shared-memory kernel has no codelets for
    }
    return c.rows ? dif_go<T, DIF_C2C, false>(a, c.nthr, c.smem, st) : dif_go<T, DIF_C2C, true>(a, c.nthr, c.smem, st);
}

// A step of a long transform of several adjacent vectors: column tiles, a
// group per grid row.
bool launch_dif_step_f32(const Job &j, cudaStream_t st) {
    DifArgs<float> a;
    DifCta c;
    if (j.kind != K_C2C || j.nbatch < 1 || j.nbatch > 65535 || !dif_args<float>(j, 0, device()->sms, false, a, c) || c.rows || c.split)
        return false;
    a.bvs_in = j.bvs_in;
    a.bvs_out = j.bvs_out;
    a.tw_lo = (const float2 *)j.tw_lo;
    a.tw_hi = (const float2 *)j.tw_hi;
    a.tw_mask = j.tw_mask;
    a.tw_sh = j.tw_sh;
    a.tw_ts = j.tw_ts;
    a.tw_ys = j.tw_ys;
    const DifFixEntry *f = j.dif->fix;
    if (f && f->step && a.vpb == 16) return f->step(a, c.smem, st, (unsigned)j.nbatch);
    return dif_step_go(a, c.nthr, c.smem, st, (unsigned)j.nbatch);
}

// ---------------------------------------------------------------- k-omega
// The tapered R2C rows into a column-major spectrum (kw.c creates it so):
// tiles of 4 to 16 rows in about 64 KB.  Row-major spectra are not taken.
bool launch_dif_komega_r2c_f32(const Job &j, cudaStream_t st) {
    const DifTab *t = j.dif;
    if (!t || j.no_fast || j.no_dif || j.kind != K_R2C || j.nvec <= 1 || !j.thalf || !j.taper_n || !j.taper_t ||
        !j.taper_back)
        return false;
    const CView &co = j.cout;
    if (!real_pairs<float>(j.rin, 2 * j.N, j.nvec) || !interleaved_c<float>(co) || co.vs != 1 || co.es < j.nvec)
        return false;
    DifArgs<float> a = dif_base<float>(*t);
    a.in = (const float2 *)j.rin.a + j.rin.off / 2;
    a.wb = const_cast<float2 *>(a.in);
    a.vs_in = j.rin.vs / 2;
    a.es_in = 1;
    a.out = (float2 *)co.re + co.off;
    a.es_out = co.es;
    a.vs_out = 1;
    a.thalf = (const float2 *)j.thalf;
    a.nvec = j.nvec;
    a.has_scale = j.has_scale;
    a.scale = j.has_scale ? (float)j.scale : 1.f;
    a.tp_n = (const float *)j.taper_n;
    a.tp_t = (const float *)j.taper_t;
    a.tp_n_st = j.taper_n_st;
    a.tp_t_st = j.taper_t_st;
    a.LD |= 1;
    const DifFixEntry *f = t->fix;
    a.lgv = 4;
    while (a.lgv > 2 && ((size_t)a.LD << a.lgv) * sizeof(float2) > 72 * 1024) a.lgv--;
    if (f && f->taper)
        for (a.lgv = 0; (1 << a.lgv) < f->vtaper; a.lgv++) {
        }
    // few sensors: fewer rows per tile, so that more SMs work on them
    while (a.lgv > 0 && 2 * (((j.nvec - 1) >> a.lgv) + 1) < device()->sms) a.lgv--;
    a.vpb = 1 << a.lgv;
    const size_t smem = (size_t)a.LD * a.vpb * sizeof(float2);
    if (smem > device()->smem_optin) return false;
    if (f && f->taper && a.vpb == f->vtaper) return f->taper(a, smem, st, 1);
    // 8 points a thread: without a compiled-in schedule, or with fewer rows to a tile,
    // few CTAs are there (16 x 3000 in all 15 us, 18 with 16 points; 128 x 8192 14.4
    // and 17.9)
    const long nthr = std::min(1024L, std::max(96L, (a.vpb * j.N / 8 + 31) / 32 * 32));
    return dif_komega_go(DIF_R2CT, a, (int)nthr, smem, st);
}

// Its transforms over the sensors, contiguous in that spectrum.
bool launch_dif_komega_power_f32(const Job &j, cudaStream_t st) {
    if (!j.gram) return false;
    Job q = j;
    q.gram = nullptr;
    DifArgs<float> a;
    DifCta c;
    if (j.kind != K_C2C || !dif_args<float>(q, 0, device()->sms, true, a, c) || !c.rows || c.split) return false;
    a.gram = (float *)j.gram;
    a.g_es = j.gram_es;
    a.g_vs = j.gram_vs;
    a.g_scale = (float)j.gram_scale;
    if (j.dif->fix && j.dif->fix->power) return j.dif->fix->power(a, c.smem, st, 1);
    return dif_komega_go(DIF_POWER, a, c.nthr, c.smem, st);
}

// ---------------------------------------------------------------- single long vectors
// N = A*B*C (or A*C, B = 1) points of one vector: with n = n1*BC + r and k =
// k1 + A*(k2 + B*k3), pass 1 transforms over n1 (A points BC apart, 16
// adjacent r per tile) and twiddles by W_N^(k1 r) into scratch[k1*BC + r];
// pass 2 does the same inside every block of BC over n2 (twiddle W_BC^(k2 n3),
// in place); the last pass transforms rows of C points and stores output k3 of
// 16 adjacent k1 side by side at y[k1 + A*(k2 + B*k3)].  Every pass reads and
// writes segments of 128 bytes or more, and every twiddle is a coalesced table
// load (pass 1: W_N^(k1 r0) of the tile's first r, computed once per tile, times
// W_N^(k1 t); pass 2: the whole table of BC entries), where the Stockham passes
// before took two gathers per point.
static double vec_cost(long n) {
    if (n < 16 || n > 1024) return 1e30;
    const DifFixEntry *fix = dif_fix(n, 0);
    double c;
    if (least_cost(n, P_F32, 0, &c).empty()) return 1e30;
    c += 25;  // global accesses and the pass's own twiddle
    if (fix && fix->vec[0]) return c;
    return n > 512 ? c * 1.3 : c * 1.15;  // tiles of 8 transforms; no compiled-in schedule
}

// Two factors up to kVecTwoMax points where there are two, by cost otherwise
// (2^20 points measured the same in two passes of 1024 and in three).
bool vec_factors(long N, long f[3]) {
    double best = 1e29;
    f[0] = f[1] = f[2] = 0;
    std::vector<long> d;
    std::map<long, double> cost;
    for (long a = 16; a <= 1024; a++)
        if (N % a == 0 && vec_cost(a) < 1e29) {
            d.push_back(a);
            cost[a] = vec_cost(a);
        }
    for (long a : d) {
        const long m = N / a;
        if (cost.count(m) && N <= kVecTwoMax && cost[a] + cost[m] < best) {
            best = cost[a] + cost[m];
            f[0] = a;
            f[1] = 1;
            f[2] = m;
        }
        if (N <= kVecTwoMax && f[1] == 1) continue;
        for (long b : d)
            if (m % b == 0 && cost.count(m / b) && cost[a] + cost[b] + cost[m / b] < best) {
                best = cost[a] + cost[b] + cost[m / b];
                f[0] = a;
                f[1] = b;
                f[2] = m / b;
            }
    }
    return f[0] != 0;
}

template <typename F> static void *upload_roots(long n, F exponent, long N) {
    std::vector<float> t(2 * n);
    for (long i = 0; i < n; i++) {
        double c, s;
        unit_root(exponent(i) % N, N, &c, &s);
        t[2 * i] = (float)c;
        t[2 * i + 1] = (float)s;
    }
    return table_upload(t.data(), t.size() * sizeof(float), "twiddle upload");
}

// adjacent transforms per tile: 128-byte segments, fewer while they leave SMs idle
static long vec_tile(long n, long N) {
    long v = n > 512 ? 8 : 16;
    while (v > 4 && N / n / v < 2L * device()->sms) v /= 2;
    return v;
}

void vec_release(VecPlan *v) {
    if (!v) return;
    for (const DifTab *t : v->tab) dif_release(t);
    dfree(v->d_t1);
    dfree(v->d_t2);
    delete v;
}

// nullptr when N does not factor so, or without memory (the other paths take
// the vector).
VecPlan *vec_acquire(long N) {
    long f[3];
    if (N >= (1L << 31) || !vec_factors(N, f)) return nullptr;
    const int err0 = jvsip_gpu_last_error();
    VecPlan *v = new (std::nothrow) VecPlan();
    if (!v) return nullptr;
    const long V = vec_tile(f[0], N), BC = f[1] * f[2];
    bool ok = true;
    for (int i = 0; i < 3; i++) {
        v->f[i] = f[i];
        if (f[i] > 1) ok = ok && (v->tab[i] = dif_acquire(f[i], P_F32, 0, nullptr, nullptr, 0)) != nullptr;
    }
    ok = ok && (v->d_t1 = upload_roots(f[0] * V, [&](long i) { return (i / V) * (i % V); }, N)) != nullptr;
    const long C = f[2];
    if (ok && f[1] > 1) ok = (v->d_t2 = upload_roots(BC, [&](long i) { return (i / C) * (i % C); }, BC)) != nullptr;
    if (ok) return v;
    vec_release(v);
    if (!err0 && jvsip_gpu_last_error()) jvsip_gpu_clear_error();
    return nullptr;
}

// One vector of unit stride from `in` to `out` through `scratch` (N points).
bool launch_vec_f32(const VecPlan &v, const float2 *in, float2 *out, float2 *scratch, const float2 *lo, const float2 *hi,
                    unsigned mask, unsigned sh, int conj_in, int conj_out, int has_scale, float scale, cudaStream_t st) {
    const long A = v.f[0], B = v.f[1], C = v.f[2];
    for (int i = 0; i < 3; i++) {
        if (!v.tab[i]) continue;
        DifArgs<float> a = dif_base<float>(*v.tab[i]);
        const long V = vec_tile(a.N, A * B * C);
        a.lgv = V == 16 ? 4 : V == 8 ? 3 : 2;
        a.vpb = (int)V;
        a.scale = 1.f;
        size_t smem;
        unsigned groups = 1;
        a.in = i == 0 ? in : scratch;
        a.out = i == 2 ? out : scratch;
        if (i < 2) {
            const long cols = i == 0 ? B * C : C;
            a.es_in = a.es_out = a.nvec = cols;
            a.vs_in = a.vs_out = 1;
            a.bvs_in = a.bvs_out = B * C;
            groups = i == 0 ? 1u : (unsigned)A;
            a.tv = (const float2 *)(i == 0 ? v.d_t1 : v.d_t2);
            a.tv_st = (int)C;
            a.tw_lo = lo;
            a.tw_hi = hi;
            a.tw_mask = mask;
            a.tw_sh = sh;
            a.smask_in = i == 0 && conj_in ? 0x80000000u : 0u;
            smem = ((size_t)a.LD * V + (i == 0 ? a.N : 0)) * sizeof(float2);
        } else {
            a.LD |= 1;
            a.es_in = 1;
            a.vs_in = B * C;
            a.bvs_in = C;
            a.nvec = A;
            a.es_out = A * B;
            a.vs_out = 1;
            a.bvs_out = A;
            groups = (unsigned)B;
            a.smask_out = conj_out ? 0x80000000u : 0u;
            a.has_scale = has_scale;
            if (has_scale) a.scale = scale;
            smem = (size_t)a.LD * V * sizeof(float2);
        }
        // up to 2^19 points the CTAs of a pass leave SMs half empty and its time is one
        // tile's chain: 4 points a thread instead of 16 (59049 points 8.6 us, 11.9 with
        // 16 and 10.1 in the two steps; 125000 8.8, 11.7, 11.3; 390625 12.6, 16.3, 16.9;
        // 786432 12.8 and 11.5 with 16)
        const long per = A * B * C <= (1L << 19) ? 4 : 16, most = per == 4 ? 1024 : 512;
        const int nthr = (int)std::min(most, std::max(64L, (V * a.N / per + 31) / 32 * 32));
        const DifFixEntry *f = v.tab[i]->fix;
        if (f && f->vec[i] && V == 16) {
            if (!f->vec[i](a, smem, st, groups)) return false;
            continue;
        }
        if (!dif_vec_go(i == 0 ? DIF_VEC1 : i == 1 ? DIF_VEC2 : DIF_VECR, a, nthr, smem, st, groups)) return false;
    }
    return true;
}

bool dif_tile_args(const Job &j, long tuned, long sms, DifArgs<float> &a, DifCta &c) {
    return j.kind == K_C2C && dif_args<float>(j, tuned, sms, true, a, c) && !c.split;
}

bool launch_dif_f32(const Job &j, cudaStream_t st) { return launch_dif_t<float>(j, st); }
bool launch_dif_f64(const Job &j, cudaStream_t st) { return launch_dif_t<double>(j, st); }

}  // namespace jv
