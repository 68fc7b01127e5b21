// The length pass with one half-warp per knot interval (float-float panels):
// the alternative mapping to k_walk's one lane per panel, chosen by the
// caller through gcv_options.mapping (GCV_MAP_HALF_WARP).
//
// The 16 lanes of a half-warp walk one interval's dyadic panels together: in
// each panel a lane evaluates one node (the seven Kronrod pairs and the centre,
// panel_ff_half), the nodes are gathered by shuffles and summed in k_walk's
// order, and the walk's state (panel (k, depth), running sums, tolerance) is
// the same in all lanes.  Lane 0 of the half stages accepted leaves in shared
// memory; the lanes write them out together when the interval is done.  The
// acceptance test, the learned start and the leaf table are those of
// k_walk<CODE, 1> (intervals of more than LCAP leaves go to the deep passes
// here), so both mappings build the same table up to float-float rounding (the
// square roots are scalar here and packed there): lengths differ by at most
// 6e-15 relative, curve parameters by 7e-13, over 1,500 uneven curves.
//
// Per panel this mapping spends 16 lanes on one node each, every one of which
// shifts the polynomials and adds up all pairs, where k_walk spends one lane on
// all of them; it finishes an interval's panel sooner.
#pragma once

#include "gcv_length_impl.cuh"  // chord_of and the shared parameter block

namespace gcv {

// K15 and G7 of a panel by the 16 lanes of a half-warp: lane hl evaluates one
// node of pair hl % 8 (the eighth pair is the centre), every lane then adds the
// pairs up in panel_ff's order, so the two agree to the rounding of
// the square root.  Every lane of the warp takes part.
template <int CODE>
__device__ __forceinline__ void panel_ff_half(ff* r, unsigned long long k, int depth, int hl, int half_base, ff& K, ff& G)
{
    const unsigned FULL = 0xffffffffu;
    const int i = hl & 7;
    const bool plus = hl >= 8;
    ff f;
    if constexpr (CODE == 0) {
        ff sm, cm;
        ff_sincospi(ff_add_f(ff_scale(panel_mid(k, depth), (float)ELLIPSE_PIECE_SCALE), r[2].hi), sm, cm);
        const float4 a = __ldg(reinterpret_cast<const float4*>(c_angle.ff[depth]) + i);
        const ff sd{a.x, a.y}, s = ff_fma(cm, plus ? sd : ff_neg(sd), ff_mul_open(sm, ff{a.z, a.w}));
        f = ff_sqrt(ff_fma(r[0], ff_mul_open(s, s), r[1]));
    } else {
        constexpr int P = code_degree(CODE), D = code_dim(CODE), N = P - 1;
        constexpr int JE = (N % 2 == 0) ? N : N - 1, JO = (N % 2 == 1) ? N : N - 1;
        panel_shift<P, D>(r, k, depth);
        const GkStep2 c = c_gk_step2[i >> 1];
        const ff x = i & 1 ? ff{c.xh.y, c.xl.y} : ff{c.xh.x, c.xl.x};
        const ff x2 = i & 1 ? ff{c.x2h.y, c.x2l.y} : ff{c.x2h.x, c.x2l.x};
        ff sum{0.0f, 0.0f};
#pragma unroll
        for (int d = 0; d < D; ++d) {
            ff e = r[JE * D + d];
#pragma unroll
            for (int j = JE - 2; j >= 0; j -= 2) e = ff_fma_open(e, x2, r[j * D + d]);
            if constexpr (JO >= 1) {
                ff o = r[JO * D + d];
#pragma unroll
                for (int j = JO - 2; j >= 1; j -= 2) o = ff_fma_open(o, x2, r[j * D + d]);
                o = ff_mul_open(o, x);
                e = ff_add(e, plus ? o : ff_neg(o));
            }
            sum = d == 0 ? ff_mul_open(e, e) : (d + 1 < D ? ff_fma_open(e, e, sum) : ff_fma(e, e, sum));
        }
        f = ff_sqrt(sum);
    }
    const ff pair = ff_add(f, ff{__shfl_xor_sync(FULL, f.hi, 8), __shfl_xor_sync(FULL, f.lo, 8)});
    ff kk[2] = {}, gg[2] = {};
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const ff s{__shfl_sync(FULL, pair.hi, half_base + p), __shfl_sync(FULL, pair.lo, half_base + p)};
        kk[p & 1] = ff_fma(to_ff(split_const(gk_pair_wk(p))), s, kk[p & 1]);
        if (p < 4) gg[p & 1] = ff_fma(to_ff(split_const(gk_pair_wg(p))), s, gg[p & 1]);
    }
    const float hw = __int_as_float((127 - depth) << 23);
    K = ff_scale(ff_add(kk[0], kk[1]), hw);
    G = ff_scale(ff_add(gg[0], gg[1]), hw);
}

template <int CODE>
__global__ void __launch_bounds__(LK_THREADS) k_length_hw(LengthParams P)
{
    static_assert(LK_THREADS % 32 == 0, "whole warps");
    constexpr int HALVES = LK_THREADS / 16;
    __shared__ double lf_v[LCAP][HALVES];
    __shared__ double lf_c[LCAP][HALVES];

    const Batch& b = P.b;
    const Table& t = P.t;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, hl = lane & 15, half_base = lane & 16, half = threadIdx.x >> 4;
    const unsigned half_mask = half_base ? 0xffff0000u : 0x0000ffffu;
    const double eps50 = 50.0 * 1.4210854715202004e-14;  // round-off floor: 50 float-float units

    const int64_t n_items = length_items(P);
    bool active = false, exhausted = false;
    int64_t s = 0;
    const float2* cff = nullptr;
    unsigned long long k = 0;
    int depth = 0, nleaf = 0;
    double cum = 0.0, tol_unit = 0.0;
    ff cumf{0.0f, 0.0f};
    float tol_f = 0.0f;
    uint32_t dq = 0;
    long long panels = 0;
    unsigned long long my_panels = 0, my_capped = 0, my_nonfinite = 0;

    for (;;) {
        bool fin = false, ovf = false;
        // ---- refill: lane 0 of each idle half takes the next interval
        const bool need = !active && !exhausted;  // the same in all lanes of a half
        unsigned long long item = 0;
        if (need && hl == 0) item = atomicAdd(P.work, 1ull);
        item = __shfl_sync(FULL, item, half_base);
        if (need) {
            if ((int64_t)item >= n_items) {
                exhausted = true;
            } else {
                s = P.list ? (int64_t)P.list[item] : (int64_t)item;
                if (P.by_item) {
                    cff = P.coef_ff + P.coef_base + (int64_t)item * code_stride(CODE);
                } else {
                    const int64_t c = b.seg_curve[s];
                    cff = P.coef_ff + b.coef_off[c] + (s - b.seg_off[c]) * code_stride(CODE);
                }
                k = 0;
                depth = 0;
                nleaf = 0;
                cum = 0.0;
                cumf = ff{0.0f, 0.0f};
                panels = 0;
                dq = 0;
                if constexpr (CODE > 0) {
                    if (P.starts) {
                        const uint32_t q = P.starts[P.by_item ? (int64_t)item : s];
                        ff rc[MAX_COEF];
                        EvalFF<CODE>::load(cff, rc);
                        const float ch = chord_of<CODE>(rc);
                        if (q != 0u && ch > 0.0f) {
                            dq = q;
                            tol_unit = P.rtol * (double)ch;
                            tol_f = (float)tol_unit;
                            learned_descend(dq, k, depth);
                        }
                    }
                }
                if (t.seg_t1[s] == t.seg_t0[s]) {  // zero-width knot interval: one empty leaf
                    if (hl == 0) {
                        lf_v[0][half] = 1.0;
                        lf_c[0][half] = 0.0;
                    }
                    nleaf = 1;
                    fin = true;
                } else {
                    active = true;
                }
            }
        }
        // ---- one panel per active half: each lane one node
        const float hwf = __int_as_float((127 - depth) << 23);  // 2^-depth
        ff Kf, Gf, rl[MAX_COEF];
        if (active) {
            EvalFF<CODE>::load(cff, rl);
        } else {
#pragma unroll
            for (ff& x : rl) x = ff{0.0f, 0.0f};
        }
        panel_ff_half<CODE>(rl, k, depth, hl, half_base, Kf, Gf);
        if (active) {
            if (depth == 0) {
                tol_unit = P.rtol * fabs(ff_to_double(Kf));
                tol_f = (float)tol_unit;
            }
            const ff dkg = ff_add(Kf, ff_neg(Gf));
            const float errf = fabsf(dkg.hi);
            const float thr = fmaxf(tol_f * hwf, (float)eps50 * fabsf(Kf.hi));
            const bool finite = isfinite(Kf.hi) && isfinite(Gf.hi);
            bool ok;
            if (errf < 0.99f * thr) {
                ok = true;
            } else if (errf > 1.01f * thr && thr > 1e-30f) {
                ok = false;
            } else {
                const double Kd = ff_to_double(Kf);
                ok = fabs(ff_to_double(dkg)) <= fmax(tol_unit * pow2_neg(depth), eps50 * fabs(Kd));
            }
            ++panels;
            const bool at_cap = depth >= P.max_depth || panels >= PANEL_BUDGET;
            if (ok || at_cap || !finite) {
                if (!ok && finite) ++my_capped;
                if (!finite) ++my_nonfinite;
                cumf = ff_add(cumf, Kf);
                cum = ff_to_double(cumf);
                const double vr = fma(__ull2double_rn(k + 1), 2.0 * pow2_neg(depth), -1.0);
                if (nleaf < LCAP) {
                    if (hl == 0) {
                        lf_v[nleaf][half] = vr;
                        lf_c[nleaf][half] = cum;
                    }
                } else {
                    ovf = true;
                }
                ++nleaf;
                ++k;
                const int tz = __ffsll((long long)k) - 1;
                k >>= tz;
                depth -= tz;
                if (dq && depth > 0) learned_descend(dq, k, depth);
                if (ovf) {
                    active = false;
                } else if (depth == 0) {
                    active = false;
                    fin = true;
                }
            } else {
                k <<= 1;
                ++depth;
            }
            if (!active && hl == 0) my_panels += (unsigned long long)panels;
        }
        // ---- finished intervals: the half writes its leaves together
        if (fin) {
            __syncwarp(half_mask);  // lane 0's staged leaves are visible to the half
            unsigned long long base = 0;
            if (hl == 0) base = atomicAdd(t.ctr + C_LEAF_TOP, (unsigned long long)nleaf);
            base = __shfl_sync(half_mask, base, half_base);
            const int64_t off = (int64_t)base;
            if (off + nleaf <= t.leaf_cap) {
                ff rl[MAX_COEF];
                EvalFF<CODE>::load(cff, rl);
                for (int i = hl; i < nleaf; i += 16) {
                    const double vi = lf_v[i][half];
                    float q32;
                    const float f32 = EvalFF<CODE>::speed_slope32(rl, (float)vi, q32);
                    t.leaf_v[off + i] = vi;
                    t.leaf_cum[off + i] = lf_c[i][half];
                    t.leaf_f[off + i] = f32;
                    t.leaf_q[off + i] = q32;
                }
            } else if (hl == 0) {
                // the pool is full: the deep passes redo this interval
                const unsigned long long o = atomicAdd(t.ctr + C_DEEP, 1ull);
                if ((int64_t)o < t.deep_cap)
                    t.deep_list[o] = int(s);
                else
                    raise_err(t, ERR_DEEP_LIST);
            }
            if (hl == 0) {
                t.seg_len[s] = nleaf == 1 && t.seg_t1[s] == t.seg_t0[s] ? 0.0 : cum;
                t.leaf_off[s] = off;
                t.leaf_cnt[s] = nleaf;
            }
            __syncwarp(half_mask);  // the staging slots are free for the next interval
        }
        if (ovf && hl == 0) {
            const unsigned long long o = atomicAdd(t.ctr + C_DEEP, 1ull);
            if ((int64_t)o < t.deep_cap)
                t.deep_list[o] = int(s);
            else
                raise_err(t, ERR_DEEP_LIST);
        }
        if (__all_sync(FULL, exhausted && !active)) break;
    }
    // ---- statistics (lane 0 of each half holds its counts)
    if (hl != 0) my_panels = my_capped = my_nonfinite = 0;
    for (int o = 16; o > 0; o >>= 1) {
        my_panels += __shfl_xor_sync(FULL, my_panels, o);
        my_capped += __shfl_xor_sync(FULL, my_capped, o);
        my_nonfinite += __shfl_xor_sync(FULL, my_nonfinite, o);
    }
    if (lane == 0) {
        if (P.collect && my_panels) atomicAdd(t.ctr + C_PANELS, my_panels);
        if (my_capped) atomicAdd(t.ctr + C_CAPPED, my_capped);
        if (my_nonfinite) atomicAdd(t.ctr + C_NONFINITE, my_nonfinite);
    }
}

template <int CODE>
cudaError_t length_launch_hw(const LengthParams& P, cudaStream_t stream, int sm_count, int blocks_per_sm_cap)
{
    int occ = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_length_hw<CODE>, LK_THREADS, 0);
    if (e != cudaSuccess) return e;
    const int cap = blocks_per_sm_cap < 1 ? 1 : blocks_per_sm_cap;
    occ = occ < 1 ? 1 : (occ > cap ? cap : occ);
    const int64_t want = (P.n_items + LK_THREADS / 16 - 1) / (LK_THREADS / 16);
    int64_t grid = (int64_t)sm_count * occ;
    if (want < grid) grid = want;
    if (grid < 1) grid = 1;
    k_length_hw<CODE><<<(unsigned)grid, LK_THREADS, 0, stream>>>(P);
    return cudaGetLastError();
}

#define GCV_LENGTH_HW_INST(CODE)                                                                  \
    template cudaError_t length_launch_hw<CODE>(const LengthParams&, cudaStream_t, int, int);

}  // namespace gcv
