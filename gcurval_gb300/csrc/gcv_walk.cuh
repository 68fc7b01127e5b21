// The adaptive length walk with one list of pending panels per warp: the main
// pass of the mixed tables and of FP64 tables at tolerances from
// PLAIN_SPLIT_RTOL up.
//
// A warp holds up to WK_SLOTS knot intervals at a time and a stack of their
// panels still to be evaluated.  Each round its 32 lanes take 32 panels of any
// of those intervals, evaluate K15 and G7 in float-float (gcv_ff_eval.cuh), and
// either accept the panel (a leaf of the table) or replace it by its halves.
// Panels of an interval are nodes of a linked list in parameter order (a split
// puts the right half behind the left one), so leaves come out in order
// although they are evaluated in any order.  Finished intervals collect until
// there are WK_FLUSH of them; the warp then reserves their leaves' place in
// the pool with one atomic, sums them up in order, and writes the leaves
// together.  (Warps of 80 intervals, 32 written together: 10,000 cubics 0.76 ms,
// against 0.88 ms with 64 and 16.)
//
// What bounds it: issue (float-float panels on the FP32 pipes).  The
// lane-per-interval walk (gcv_length_impl.cuh) takes two global atomics in
// every round, lasts as long as its slowest lane's 31 panels one after another,
// and hands intervals of more than 16 leaves to two more passes that walk them
// again, one lane each; here an interval of L leaves takes as many rounds as
// its deepest leaf has levels.  Against it: FP64 tables, 10,000 cubics 3.28 ->
// 0.74 ms, 1,237 spatial curves (175k intervals) 3.16 -> 0.40 ms, 4,096 ellipses
// 0.35 -> 0.07 ms, 64 ellipses 0.24 -> 0.05 ms; mixed, 301 uneven curves 1.41 ->
// 0.24 ms, 50,000 spatial 2.68 -> 1.73 ms, 100,000 uneven with learned starts
// 14.2 -> 11.0 ms (of these two, 1.97 and 12.3 before the panels' inner steps were
// left unnormalised, gcv_ff.cuh).
#pragma once

#include "gcv_length_impl.cuh"
#include "gcv_leaf64.cuh"

namespace gcv {

constexpr int WK_THREADS = 64;
constexpr int WK_NODES = 192;   // panels of one warp's intervals, pending and accepted (ids in a byte)
constexpr int WK_SLOTS = 80;    // intervals of one warp, being walked or waiting to be written
constexpr int WK_RESERVE = 32;  // nodes kept free for splits when new intervals are taken
constexpr int WK_FLUSH = 32;    // finished intervals that are written together
constexpr int WK_LEAVES = 96;   // leaves of one interval; the deep passes take intervals with more
static_assert(2 * WK_LEAVES <= WK_NODES, "two intervals alone always finish");

// why a slot's interval is given up
enum WalkDead {
    WK_LIVE = 0,
    WK_DEEP = 1,   // too many leaves: to the deep list
    WK_LATER = 2,  // out of nodes: once more when the warp's other intervals are done
    WK_PLAIN = 3   // more than LCAP leaves from its learned start: once more from the whole interval
};

// node key: dyadic panel (k, depth), whether the learned start depths still have
// to be looked at, and whether a leaf was accepted short of the tolerance
constexpr unsigned long long WK_K_MASK = (1ull << 56) - 1;
constexpr unsigned long long WK_FLAG = 1ull << 63, WK_CAPPED = 1ull << 62;
__device__ __forceinline__ unsigned long long wk_key(unsigned long long k, int depth, bool flag)
{
    return k | ((unsigned long long)depth << 56) | (flag ? WK_FLAG : 0ull);
}
__device__ __forceinline__ int wk_depth(unsigned long long key) { return (int)(key >> 56) & 0x3F; }

// a slot's counts: panels to evaluate (low 16 bits), nodes of the list (8), evaluated
// panels that were split (8)
constexpr unsigned WK_ONE_NODE = 0x10001u, WK_ONE_SPLIT = 0x1000000u;
__device__ __forceinline__ int wk_nodes(unsigned count) { return (int)(count >> 16 & 0xFFu); }
__device__ __forceinline__ int wk_splits(unsigned count) { return (int)(count >> 24); }
static_assert(WK_LEAVES + 32 <= 256, "a limit and a round's splits beyond it fit eight bits");

struct WalkWarp {
    unsigned long long key[WK_NODES];
    double val[WK_NODES];   // the panel's K15 (float-float pair, then FP64), finally the running sum
    double whole[WK_SLOTS];  // float-float pair: K15 of the whole interval, or its chord (learned start)
    float tolf[WK_SLOTS];    // rtol times that
    int item[WK_SLOTS], sexp[WK_SLOTS];
    unsigned count[WK_SLOTS];  // see wk_nodes
    uint32_t dq[WK_SLOTS];  // learned quarter start depths (0: from the whole interval)
    unsigned char next[WK_NODES], slot[WK_NODES], stack[WK_NODES], freel[WK_NODES], order[WK_NODES];
    unsigned char head[WK_SLOTS], fslot[WK_SLOTS], done[WK_SLOTS], dead[WK_SLOTS], fits[WK_SLOTS], later[WK_SLOTS];
};

__device__ __forceinline__ double pack_ff(ff a)
{
    return __hiloint2double(__float_as_int(a.hi), __float_as_int(a.lo));
}
__device__ __forceinline__ ff unpack_ff(double x)
{
    return ff{__int_as_float(__double2hiint(x)), __int_as_float(__double2loint(x))};
}

// exponent of an interval's largest speed coefficient (FP64 table), the scale
// that brings its float-float panels near 1
template <int CODE>
__device__ __forceinline__ int interval_exponent(const double* __restrict__ seg)
{
    if constexpr (CODE == 0) {
        return exponent_of(fmax(fabs(seg[3]), fabs(seg[4])) * (PI * ELLIPSE_PIECE_SCALE));  // axes of either sign
    } else {
        constexpr int D = code_dim(CODE);
        int m = 0;
#pragma unroll
        for (int i = D; i < code_stride(CODE); ++i) m = max(m, __double2hiint(seg[i]) & 0x7FFFFFFF);
        const int raw = m >> 20;
        return raw == 0 || raw == 0x7FF ? 0 : raw - 1023;
    }
}

// K15 of a panel in FP64 whose float-float panel is infinite or NaN: with infinite
// control points FP64 has an infinite length where float-float has NaN, and
// samples are placed by it
template <int CODE>
__device__ __noinline__ double nonfinite_k15(const double* __restrict__ seg, unsigned long long k, int depth)
{
    double r[MAX_COEF];
    Eval<CODE>::load_speed(seg, r);
    const double hw = pow2_neg(depth);
    double K, G, fe, qe;
    panel_k15<CODE>(r, fma(__ull2double_rn(k), 2.0 * hw, -1.0), hw, K, G, fe, qe);
    return K;
}

// the FP64 error test of one panel of an FP64 table (panels whose float-float
// error estimate lands within 1 % or the float-float noise of the tolerance)
template <int CODE>
__device__ __noinline__ bool accept_fp64(const double* __restrict__ seg, unsigned long long k, int depth, double tol)
{
    double r[MAX_COEF];
    Eval<CODE>::load_speed(seg, r);
    const double hw = pow2_neg(depth);
    double K, G, fe, qe;
    panel_k15<CODE>(r, fma(__ull2double_rn(k), 2.0 * hw, -1.0), hw, K, G, fe, qe);
    if (depth == 0) tol *= fabs(K);
    return fabs(K - G) <= fmax(tol * hw, 50.0 * 2.220446049250313e-16 * fabs(K));
}

// Resident blocks per SM asked for, per curve code: 14 (at most 72 registers)
// for degree 3-5 in 3D, 16 (64) for the others.  The walk of the uneven batch of
// 100,000 curves took 11.5 ms at 10 / 12, 11.15 at 12 / 14, 11.0 at 14 / 16.
__host__ __device__ constexpr int walk_blocks(int code)
{
    return code > 0 && code_dim(code) == 3 && code_degree(code) >= 3 ? 14 : 16;
}

// PREC 1: float-float table, K15 in float-float; PREC 2: FP64 table, the
// partition from float-float panels with the FP64 test near the tolerance, and
// K15 of every leaf in FP64 (leaf_k15); PREC 3: the same without a table, for
// callers that only want the intervals' lengths: `src` gives an interval's
// FP64 coefficients when the walk takes it (kept in shared memory) and receives
// its length.
struct NoSource {};
template <int CODE, int PREC, typename SRC = NoSource>
__global__ void __launch_bounds__(WK_THREADS, PREC == 3 ? 6 : walk_blocks(CODE)) k_walk(LengthParams P, SRC src = SRC{})
{
    __shared__ WalkWarp s_walk[WK_THREADS / 32];
    // PREC 3: the slots' coefficients (an odd stride keeps the lanes' banks apart)
    constexpr int SLOT_COEF = code_stride(CODE) | 1;
    __shared__ double s_coef[WK_THREADS / 32][PREC == 3 ? WK_SLOTS * SLOT_COEF : 1];
    const Table& t = P.t;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt_mask = (1u << lane) - 1u;
    WalkWarp& W = s_walk[threadIdx.x >> 5];
    constexpr int STRIDE = code_stride(CODE);
    if constexpr (PREC == 3) {
        if (src.stop()) return;
    }
    const double eps50 = 50.0 * 1.4210854715202004e-14;  // 50 float-float units
    const float rtolf = (float)P.rtol;

    for (int i = lane; i < WK_NODES; i += 32) W.freel[i] = (unsigned char)i;
    for (int i = lane; i < WK_SLOTS; i += 32) W.fslot[i] = (unsigned char)i;
    __syncwarp(FULL);
    int nfree = WK_NODES, nslot = WK_SLOTS, nstack = 0, ndone = 0, nlater = 0;  // the same in all lanes
    bool exhausted = false;
    const int64_t n_items = P.n_items;
    // intervals per claim: 32, fewer when there are not 32 for every warp
    const int64_t share = (n_items + (int64_t)gridDim.x * (WK_THREADS / 32) - 1) / ((int64_t)gridDim.x * (WK_THREADS / 32));
    const int claim = share < 32 ? (int)share : 32;
    unsigned long long my_panels = 0;
    unsigned my_capped = 0, my_nonfinite = 0;

    double* slot_coef = s_coef[threadIdx.x >> 5];
    // FP64 coefficients of the interval in a slot
    auto coef64 = [&](int sl) -> const double* {
        if constexpr (PREC == 3)
            return slot_coef + sl * SLOT_COEF;
        else
            return t.coef + P.coef_base + (int64_t)W.item[sl] * STRIDE;
    };
    auto load = [&](int sl, ff* r) {
        if constexpr (PREC == 1)
            EvalFF<CODE>::load(P.coef_ff + P.coef_base + (int64_t)W.item[sl] * STRIDE, r);
        else
            EvalFF<CODE>::load(coef64(sl), r, W.sexp[sl]);
    };
    auto to_deep = [&](int s) {
        const unsigned long long o = atomicAdd(t.ctr + C_DEEP, 1ull);
        if ((int64_t)o < t.deep_cap)
            t.deep_list[o] = s;
        else
            raise_err(t, ERR_DEEP_LIST);
    };

    // slot sl (again) at its root, which goes to stack position `at`
    auto start = [&](int sl, int nd, uint32_t dq, int at) {
        W.head[sl] = (unsigned char)nd;
        W.count[sl] = WK_ONE_NODE;
        W.dead[sl] = WK_LIVE;
        W.dq[sl] = dq;
        W.key[nd] = wk_key(0ull, 0, dq != 0u);
        W.slot[nd] = (unsigned char)sl;
        W.stack[at] = (unsigned char)nd;
    };

    for (;;) {
        // ---- new intervals
        if (!exhausted && nstack < 32) {
            const int want = min(min(claim, nslot), nfree - WK_RESERVE);
            if (want > 0) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(P.work, (unsigned long long)want);
                base = __shfl_sync(FULL, base, 0);
                const int64_t left = n_items - (int64_t)base;
                const int n = left <= 0 ? 0 : (left < want ? (int)left : want);
                exhausted = left <= want;
                if (lane < n) {
                    const int item = (int)base + lane;
                    const int sl = W.fslot[nslot - 1 - lane], nd = W.freel[nfree - 1 - lane];
                    W.item[sl] = item;
                    if constexpr (PREC == 3) src.setup(item, slot_coef + sl * SLOT_COEF);
                    if constexpr (PREC >= 2) W.sexp[sl] = interval_exponent<CODE>(coef64(sl));
                    uint32_t dq = 0;
                    if constexpr (CODE > 0 && PREC != 3) {
                        // learned start: the predicted depths, tolerance from the chord
                        if (P.starts && (dq = P.starts[item]) != 0u) {
                            ff r[MAX_COEF];
                            load(sl, r);
                            const float ch = chord_of<CODE>(r);
                            W.tolf[sl] = rtolf * ch;
                            W.whole[sl] = pack_ff(ff{ch, 0.0f});
                            if (!(ch > 0.0f)) dq = 0;
                        }
                    }
                    start(sl, nd, dq, nstack + lane);
                }
                nslot -= n;
                nfree -= n;
                nstack += n;
                __syncwarp(FULL);
            }
        }
        if (nlater && nstack == 0 && ndone == 0) {  // every node is free: two of the postponed intervals
            const int n = nlater < 2 ? nlater : 2;
            if (lane < n) {
                const int sl = W.later[nlater - 1 - lane];
                start(sl, W.freel[nfree - 1 - lane], W.dq[sl], lane);
            }
            nlater -= n;
            nfree -= n;
            nstack = n;
            __syncwarp(FULL);
        }
        // ---- 32 panels
        const int n = nstack < 32 ? nstack : 32;
        nstack -= n;
        const bool active = lane < n;
        const int nd = active ? W.stack[nstack + lane] : 0;
        const int sl = active ? W.slot[nd] : 0;
        unsigned long long key = active ? W.key[nd] : 0ull;
        __syncwarp(FULL);  // the stack's entries are read before new ones overwrite them
        bool dead = active && W.dead[sl] != WK_LIVE;
        // replaces the lanes' panels (where `split`) by their halves: the lane
        // keeps the left one in place, the right one is a new node behind it
        auto split_nodes = [&](bool split, bool right_flag, bool left_to_stack) {
            const unsigned one = left_to_stack ? WK_ONE_NODE + WK_ONE_SPLIT : WK_ONE_NODE;
            if (split) {
                // the split's two nodes for the one are counted first: of the splits that
                // an interval wants at once, those beyond its limit see it, so it
                // is given up if and only if its tree has more leaves than
                // the limit, whichever rounds its splits fall in
                const bool learned = CODE > 0 && W.dq[sl] != 0u;
                if (wk_nodes(atomicAdd(&W.count[sl], one)) >= (learned ? LCAP : WK_LEAVES)) {
                    W.dead[sl] = learned ? WK_PLAIN : WK_DEEP;
                    dead = true;
                    split = false;
                    atomicSub(&W.count[sl], one);
                }
            }
            __syncwarp(FULL);
            const int rank = __popc(__ballot_sync(FULL, split) & lt_mask);
            const bool none_left = split && rank >= nfree;
            if (none_left) atomicSub(&W.count[sl], one);
            split = split && !none_left;
            const int cnt = __popc(__ballot_sync(FULL, split));
            if (split) {
                const unsigned long long k = (key & WK_K_MASK) << 1;
                const int depth = wk_depth(key) + 1, right = W.freel[nfree - 1 - rank];
                W.key[right] = wk_key(k + 1, depth, right_flag);
                W.slot[right] = (unsigned char)sl;
                W.next[right] = W.next[nd];
                W.next[nd] = (unsigned char)right;
                if (left_to_stack) {
                    W.key[nd] = wk_key(k, depth, false);
                    W.stack[nstack + 2 * rank] = (unsigned char)right;
                    W.stack[nstack + 2 * rank + 1] = (unsigned char)nd;
                } else {
                    key = wk_key(k, depth, true);
                    W.stack[nstack + rank] = (unsigned char)right;
                }
            }
            nfree -= cnt;
            nstack += left_to_stack ? 2 * cnt : cnt;
            __syncwarp(FULL);
            return none_left;
        };
        if constexpr (CODE > 0 && PREC != 3) {
            if (P.starts) {
                // down to the learned start depths without evaluating
                for (int guard = 0; guard < 16; ++guard) {
                    const bool down = active && !dead && (key & WK_FLAG) &&
                                      wk_depth(key) < learned_start(W.dq[sl], key & WK_K_MASK, wk_depth(key));
                    if (!__ballot_sync(FULL, down)) break;
                    if (split_nodes(down, true, false)) {
                        W.dead[sl] = WK_LATER;
                        dead = true;
                    }
                }
            }
        }
        const unsigned long long k = key & WK_K_MASK;
        const int depth = wk_depth(key);
        bool reject = false;
        if (active && !dead) {
            ff r[MAX_COEF], Kf, Gf;
            load(sl, r);
            panel_ff<CODE>(r, k, depth, Kf, Gf);
            const float hwf = __int_as_float((127 - depth) << 23);  // 2^-depth
            if (depth == 0) {
                W.tolf[sl] = rtolf * fabsf(Kf.hi);
                W.whole[sl] = pack_ff(Kf);
            }
            auto tolerance = [&] { return P.rtol * fabs(ff_to_double(unpack_ff(W.whole[sl]))); };
            const ff dkg = ff_add(Kf, ff_neg(Gf));
            const float errf = fabsf(dkg.hi);
            const bool finite = isfinite(Kf.hi) && isfinite(Gf.hi);
            bool ok;
            if constexpr (PREC == 1) {
                const float thr = fmaxf(W.tolf[sl] * hwf, (float)eps50 * fabsf(Kf.hi));
                if (errf < 0.99f * thr) {
                    ok = true;
                } else if (errf > 1.01f * thr && thr > 1e-30f) {
                    ok = false;
                } else {  // near the tolerance (or below FP32 range): the FP64 test
                    const double Kd = ff_to_double(Kf);
                    ok = fabs(ff_to_double(dkg)) <= fmax(tolerance() * pow2_neg(depth), eps50 * fabs(Kd));
                }
            } else {
                // FP64's own round-off floor, and what the float-float estimate
                // can be off by (16 units): between the two the FP64 test decides
                const float thr = fmaxf(W.tolf[sl] * hwf, 1.1102230246251565e-14f * fabsf(Kf.hi));
                const float noise = 2.3e-13f * fabsf(Kf.hi);
                if (errf + noise < 0.99f * thr)
                    ok = true;
                else if (errf - noise > 1.01f * thr)
                    ok = false;
                else
                    ok = !finite || accept_fp64<CODE>(coef64(sl), k, depth,
                                                      depth == 0 ? P.rtol : scalbn(tolerance(), W.sexp[sl]));
            }
            if (ok || depth >= P.max_depth || !finite) {
                my_nonfinite += !finite;
                W.val[nd] = pack_ff(Kf);
                W.key[nd] = !ok && finite ? key | WK_CAPPED : key;
            } else {
                reject = true;
            }
        }
        __syncwarp(FULL);
        if (__ballot_sync(FULL, reject)) {
            const int had = nfree;
            const bool retry = split_nodes(reject, true, true);
            unsigned rm = __ballot_sync(FULL, retry);
            if (rm) {
                // out of nodes: these panels go back on the stack until
                // finished intervals have returned theirs; when nothing else
                // moves, the first one's interval is postponed
                const bool stuck = had == 0 && ndone == 0 && !__ballot_sync(FULL, active && (!reject || dead));
                const int victim = stuck ? __ffs(rm) - 1 : -1;
                if (lane == victim) {
                    W.dead[sl] = WK_LATER;
                    dead = true;
                }
                rm = __ballot_sync(FULL, retry && !dead);
                if (retry && !dead) {
                    W.key[nd] = key;
                    W.stack[nstack + __popc(rm & lt_mask)] = (unsigned char)nd;
                }
                nstack += __popc(rm);
                __syncwarp(FULL);
            }
        }
        // ---- intervals whose last panel was accepted (or given up)
        const bool fin = active && (!reject || dead) && (atomicSub(&W.count[sl], 1u) & 0xFFFFu) == 1u;
        const unsigned fm = __ballot_sync(FULL, fin);
        if (fin) W.done[ndone + __popc(fm & lt_mask)] = (unsigned char)sl;
        ndone += __popc(fm);
        __syncwarp(FULL);
        // ---- write finished intervals out
        if (ndone && (ndone >= WK_FLUSH || nstack == 0 || nfree < WK_RESERVE + 32 || nslot < 32)) {
            const int m = ndone < 32 ? ndone : 32;
            ndone -= m;
            const bool mine = lane < m;
            const int fs = mine ? W.done[ndone + lane] : 0;
            const int why = mine ? W.dead[fs] : WK_LIVE;
            const bool gone = why != WK_LIVE;
            const unsigned counts = mine ? W.count[fs] : 0u;
            const int nodes = wk_nodes(counts);
            const int cnt = gone ? 0 : nodes;
            if (!gone) my_panels += cnt + wk_splits(counts);
            const int incl = warp_incl_scan(cnt, lane), total = __shfl_sync(FULL, incl, 31);
            unsigned long long base = 0;
            if constexpr (PREC != 3) {
                if (lane == 0) base = atomicAdd(t.ctr + C_LEAF_TOP, (unsigned long long)total);
                base = __shfl_sync(FULL, base, 0);
            }
            const int first = incl - cnt;
            const int64_t off = (int64_t)base + first;
            const bool fits = !gone && (PREC == 3 || off + cnt <= t.leaf_cap);
            if (mine) {
                W.fits[fs] = fits;
                int q = W.head[fs];
                for (int i = 0; i < cnt; ++i) {
                    W.order[first + i] = (unsigned char)q;
                    q = W.next[q];
                }
            }
            __syncwarp(FULL);
            if constexpr (PREC >= 2) {
                for (int g0 = 0; g0 < total; g0 += 32) {
                    const int g = g0 + lane, q = g < total ? W.order[g] : 0;
                    bool again = false;
                    if (g < total) {
                        const int qs = W.slot[q];
                        double K = 0.0;
                        if (W.fits[qs]) {
                            const unsigned long long k = W.key[q] & WK_K_MASK;
                            const int depth = wk_depth(W.key[q]);
                            K = isfinite(unpack_ff(W.val[q]).hi) ? leaf_k15<CODE>(coef64(qs), W.sexp[qs], k, depth, again)
                                                                 : nonfinite_k15<CODE>(coef64(qs), k, depth);
                        }
                        if (!again) W.val[q] = K;
                    }
                    if constexpr (CODE > 0) {
                        // two leaves at a time, 16 lanes each (the last one by both halves)
                        for (unsigned m = __ballot_sync(FULL, again); m;) {
                            const int a = __ffs(m) - 1;
                            m &= m - 1;
                            const int b = m ? __ffs(m) - 1 : a;
                            m &= m - 1;
                            const int qa = __shfl_sync(FULL, q, lane < 16 ? a : b), qs = W.slot[qa];
                            const double K =
                                leaf_k15_nodes<CODE>(coef64(qs), W.sexp[qs], W.key[qa] & WK_K_MASK, wk_depth(W.key[qa]));
                            if ((lane & 15) == 0) W.val[qa] = K;
                        }
                    }
                }
                __syncwarp(FULL);
            }
            if (mine) {
                double cum = 0.0;
                ff cumf{0.0f, 0.0f};
                for (int i = 0; i < cnt; ++i) {
                    const int q = W.order[first + i];
                    if constexpr (PREC == 1) {
                        cumf = ff_add(cumf, unpack_ff(W.val[q]));
                        cum = ff_to_double(cumf);
                    } else {
                        cum += W.val[q];
                    }
                    W.val[q] = cum;
                }
                const int s = PREC != 3 && P.list ? P.list[W.item[fs]] : W.item[fs];
                if constexpr (PREC == 3) {
                    if (why == WK_DEEP)
                        src.deep(s, coef64(fs));
                    else if (!gone)
                        src.finish(s, cum);
                } else if (why == WK_DEEP) {
                    to_deep(s);
                } else if (!gone) {
                    // a full pool: the pass is run again with a larger one
                    if (!fits) raise_err(t, ERR_POOL);
                    t.seg_len[s] = cnt == 1 && t.seg_t1[s] == t.seg_t0[s] ? 0.0 : cum;
                    t.leaf_off[s] = off;
                    t.leaf_cnt[s] = cnt;
                }
            }
            __syncwarp(FULL);
            for (int g = lane; g < total; g += 32) {
                const int q = W.order[g], qs = W.slot[q];
                const unsigned long long qk = W.key[q];
                my_capped += (qk & WK_CAPPED) != 0ull;
                if (PREC != 3 && W.fits[qs]) {
                    const int qd = wk_depth(qk);
                    // right end -1 + (k + 1) 2^(1 - depth): exact
                    const double vr = fma(__ull2double_rn((qk & WK_K_MASK) + 1), 2.0 * pow2_neg(qd), -1.0);
                    ff r[MAX_COEF];
                    load(qs, r);
                    float q32;
                    float f32 = EvalFF<CODE>::speed_slope32(r, f32_of_f64_trunc(vr), q32);
                    if constexpr (PREC == 2) {
                        f32 = scale_down(f32, -W.sexp[qs]);
                        q32 = scale_down(q32, -2 * W.sexp[qs]);
                    }
                    t.leaf_v[base + g] = vr;
                    t.leaf_cum[base + g] = W.val[q];
                    t.leaf_f[base + g] = f32;
                    t.leaf_q[base + g] = q32;
                }
                W.freel[nfree + g] = (unsigned char)q;
            }
            nfree += total;
            const unsigned back = __ballot_sync(FULL, mine && why != WK_LATER && why != WK_PLAIN);
            if (back >> lane & 1u) W.fslot[nslot + __popc(back & lt_mask)] = (unsigned char)fs;
            nslot += __popc(back);
            if (__ballot_sync(FULL, gone)) {  // the given-up intervals: their nodes, and those to walk again
                const int gincl = warp_incl_scan(gone ? nodes : 0, lane);
                if (gone) {
                    int q = W.head[fs];
                    for (int i = 0; i < nodes; ++i) {
                        W.freel[nfree + gincl - nodes + i] = (unsigned char)q;
                        q = W.next[q];
                    }
                }
                nfree += __shfl_sync(FULL, gincl, 31);
                __syncwarp(FULL);
                const unsigned later = __ballot_sync(FULL, why == WK_LATER), plain = __ballot_sync(FULL, why == WK_PLAIN);
                if (why == WK_LATER) W.later[nlater + __popc(later & lt_mask)] = (unsigned char)fs;
                if (why == WK_PLAIN) {
                    const int rank = __popc(plain & lt_mask);
                    start(fs, W.freel[nfree - 1 - rank], 0u, nstack + rank);
                }
                nlater += __popc(later);
                nfree -= __popc(plain);
                nstack += __popc(plain);
            }
            __syncwarp(FULL);
        }
        if (exhausted && nstack == 0 && ndone == 0 && nlater == 0) break;
    }
    // ---- statistics
    unsigned long long capped = my_capped, nonfinite = my_nonfinite;
    for (int o = 16; o > 0; o >>= 1) {
        my_panels += __shfl_xor_sync(FULL, my_panels, o);
        capped += __shfl_xor_sync(FULL, capped, o);
        nonfinite += __shfl_xor_sync(FULL, nonfinite, o);
    }
    if constexpr (PREC == 3) {
        if (lane == 0 && capped) src.count_capped(capped);
    } else if (lane == 0) {
        if (P.collect && my_panels) atomicAdd(t.ctr + C_PANELS, my_panels);
        if (capped) atomicAdd(t.ctr + C_CAPPED, capped);
        if (nonfinite) atomicAdd(t.ctr + C_NONFINITE, nonfinite);
    }
}

template <int CODE, int PREC, typename SRC>
cudaError_t walk_launch(const LengthParams& P, cudaStream_t stream, int sm_count, int blocks_per_sm_cap, SRC src)
{
    int occ = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_walk<CODE, PREC, SRC>, WK_THREADS, 0);
    if (e != cudaSuccess) return e;
    const int cap = blocks_per_sm_cap < 1 ? 1 : blocks_per_sm_cap;
    occ = occ < 1 ? 1 : (occ > cap ? cap : occ);
    // persistent: fill the GPU, with four intervals a warp or more
    const int64_t want = (P.n_items + 4 * (WK_THREADS / 32) - 1) / (4 * (WK_THREADS / 32));
    int64_t grid = (int64_t)sm_count * occ;
    if (want < grid) grid = want;
    if (grid < 1) grid = 1;
    k_walk<CODE, PREC, SRC><<<(unsigned)grid, WK_THREADS, 0, stream>>>(P, src);
    return cudaGetLastError();
}
template <int CODE, int PREC>
cudaError_t walk_launch(const LengthParams& P, cudaStream_t stream, int sm_count, int blocks_per_sm_cap)
{
    return walk_launch<CODE, PREC, NoSource>(P, stream, sm_count, blocks_per_sm_cap, NoSource{});
}

// the mixed and the FP64 walk of one curve code
#define GCV_WALK_INST(CODE)                                                                        \
    template cudaError_t walk_launch<CODE, 1>(const LengthParams&, cudaStream_t, int, int);        \
    template cudaError_t walk_launch<CODE, 2>(const LengthParams&, cudaStream_t, int, int);

}  // namespace gcv
