// Importance sampling and replay, one warp per run, for networks whose
// locations are all exponential or zero-delay (no delay-bounding invariants,
// every rate a literal or a rate program): the runs, log-weights and training
// rows of is_warp_kernel (sim_is.cuh) bit for bit.
//
// In such a network nothing but the draws changes from step to step until a
// component moves, the rate table changes or the features reach another
// value, so everything else is computed then ("refresh") and kept: each
// component's tilted 1/rate (one shared-memory record), the warp's sum of
// rate changes and, in replay, the per-class sums of 1/rate, all in the same
// order of additions.  A step in between is one Philox block and four delays
// per lane, two integer minima, one FP64 product and sum for the log-weight,
// and the winner's edges.  The log of the winner's rate ratio is kept per
// location class.  Replay stores a step's four rows (160 bytes) with one word
// per lane.
//
// What bounds it: a launch of a few hundred runs (replay) the latency of a
// step, one of a few thousand (a training round) issue, about a third of it
// theta (1,500 instructions each time the features change).  Measured (B200)
// against is_warp_kernel, 100-agent epidemic to time 75: 4,000 runs 27.5 ->
// 9.6 ms, replay of 200 runs with the merge of its rows 21.0 -> 5.6 ms (of
// which two-warp CTAs, so that the runs do not share a scheduler).
#pragma once
#include "sim_is.cuh"

namespace csmc {
namespace detail {

// Run state of one warp: the layout run_receivers needs, one thread's view.
struct PlainView {
    VarView vars, rates, shadow;
    uint16_t *locv;   // global location index per component
    uint32_t *slotv;
    static constexpr uint32_t T = 1;
    __device__ __forceinline__ uint32_t loc(const Net &, uint32_t c) const { return locv[c]; }
    __device__ __forceinline__ void set_local(const Net &n, uint32_t c, uint32_t local) const {
        locv[c] = static_cast<uint16_t>(n.comp[c].loc_begin + local);
    }
};

// Log term of a location class's last tilted winner.
struct WinTerm {
    uint32_t inv, invp;
    double term;
};

template <bool TC, bool TRACE>
__global__ void __launch_bounds__(CSMC_IS_BLOCK, CSMC_IS_MIN_CTAS_PER_SM)
    is_plain_kernel(const __grid_constant__ IsParams ip) {
    const SimParams &p = ip.s;
    extern __shared__ __align__(16) uint8_t smem[];
    stage_network(smem, p.blob, p.blob_bytes);
    MlpSmem *mlp = reinterpret_cast<MlpSmem *>(smem + p.blob_bytes);
    stage_mlp(mlp, ip.mlp);
    __syncthreads();
    const Net n = net_view(smem, p.net);
    const uint32_t C = p.net.n_comps, V = p.net.n_vars, P = p.net.n_rate_prog;
    const bool rate_table = P > 0;
    const bool rates_read_clocks = !(p.net.flags & CSMC_NET_RATE_NO_CLOCK);
    const bool recv_any = (p.net.recv_lo | p.net.recv_hi) != 0;
    const uint32_t bits = ceil_log2(C), nb = (C + 3u) >> 2;
    const uint32_t lane = threadIdx.x & 31u;
    uint8_t *slab = smem + p.blob_bytes + sizeof(MlpSmem) + static_cast<size_t>(threadIdx.x >> 5) * ip.slab_bytes;
    float *h1s = reinterpret_cast<float *>(slab);
    if (!TC) slab += 4u * CSMC_MLP_HID * CSMC_MLP_CLASSES;
    WinTerm *terms = reinterpret_cast<WinTerm *>(slab);                       // [class]
    uint4 *rec = reinterpret_cast<uint4 *>(slab + 4u * sizeof(WinTerm));      // [half][block]: 1/rate' and form, twice
    float *invv = reinterpret_cast<float *>(rec + 2u * nb);                   // nominal 1/rate per component (0: none)
    PlainView rv;
    rv.slotv = reinterpret_cast<uint32_t *>(invv + 4u * nb);
    rv.vars = VarView{reinterpret_cast<float *>(rv.slotv + C), 1};
    rv.rates = VarView{rv.vars.base + V, 1};
    rv.shadow = VarView{rv.rates.base + P, 1};
    rv.locv = reinterpret_cast<uint16_t *>(rv.rates.base + P + (recv_any ? V : 0u));
    const MlpFeatures &F = ip.feat;

    unsigned long long acc_hits = 0, acc_steps = 0, acc_capped = 0;
    RunScalars sc{0.0, 0.0, 0, 0, -1, 0, 0};  // lane 0's copy is the run's
    // the last evaluated features (bits of x[4..9]; the rest are 0) and their class factors
    uint32_t x_last[6];
#pragma unroll
    for (int i = 0; i < 6; ++i) x_last[i] = 0xffffffffu;  // a NaN: never equal to a feature
    float mfac[CSMC_MLP_CLASSES] = {1.0f, 1.0f, 1.0f, 1.0f};
    if (lane < 4) terms[lane] = WinTerm{0xffffffffu, 0xffffffffu, 0.0};
    __syncwarp();
    // replay: this lane's words of a step's rows (word `lane`, and word 32 +
    // lane of lanes 0..7; ten words a row: features, a, b), and which row's a
    // or b it computes (lanes 8, 18, 28 and 6: a; 9, 19, 29 and 7: b)
    const uint32_t duty_row = lane < 8 ? 3u : lane / 10u;
    const bool duty_a = lane == 8 || lane == 18 || lane == 28 || lane == 6;
    const bool duty_b = lane == 9 || lane == 19 || lane == 29 || lane == 7;
    uint32_t xw0 = 0, xw1 = 0;

    for (;;) {
        unsigned long long ridx = 0;
        if (lane == 0) ridx = atomicAdd(p.scratch, 1ull);
        ridx = __shfl_sync(kFullWarp, ridx, 0);
        if (ridx >= p.n_runs) break;
        uint64_t run;
        float row_w = 0.0f;
        uint64_t row0 = 0;  // replay: the run's first row in the buffer
        if (TRACE) {
            run = p.first_run + ip.trace_runs[ridx];
            row_w = ip.trace_w[ridx];
            row0 = ip.row_offset[ridx];
        } else {
            run = p.first_run + ridx;
        }

        // run initialisation (run_init, across the lanes)
        for (uint32_t c = lane; c < C; c += 32u) {
            rv.set_local(n, c, n.comp[c].init_local);
            rv.slotv[c] = 0u;
        }
        for (uint32_t v = lane; v < V; v += 32u) rv.vars[v] = n.var[v].init;
        if (lane == 0) {
            double q0 = 0.0;
            if (p.var_id >= 0 && static_cast<uint32_t>(p.var_id) < V && n.var[p.var_id].kind == 0)
                q0 = static_cast<double>(n.var[p.var_id].init);
            sc = RunScalars{q0, q0, 0xcbf29ce484222325ull, 0, -1, 0, 0};
        }
        __syncwarp();

        float time = 0.0f, tf_last = -1.0f;
        uint32_t step = 0;
        int chan = 0, goal = 0;
        double logw = 0.0, lr = 0.0;  // lr: ln 2 * the warp's sum of rate changes
        double a_sum = 0.0;           // replay: the sum of 1/rate of this lane's duty row
        uint32_t present = 0;         // replay: classes with a tilted component
        bool new_rates = true, new_feat = true, refresh = true;
        for (;;) {
            const bool timeout = !(time < p.horizon);
            if (timeout || (p.loc_mode && goal) || step >= p.max_steps) {
                if (lane == 0) {
                    const RunEnd e =
                        run_end(sc, time, p.horizon, step, p.max_steps, p.loc_mode, p.is_max, p.threshold);
                    if (!TRACE) {
                        if (p.flags) p.flags[ridx] = static_cast<uint8_t>(e.flag);
                        if (p.values) p.values[ridx] = e.value;
                        if (p.steps) p.steps[ridx] = step;
                        if (ip.logw) ip.logw[ridx] = logw;
                        if (ip.wvals) ip.wvals[ridx] = e.flag ? exp2_d(d_mul(logw, 1.4426950408889634)) : 0.0;
                    }
                    acc_hits += e.flag;
                    acc_steps += step;
                    acc_capped += e.capped;
                }
                __syncwarp();
                break;
            }

            // pending broadcast receivers (serial, lane 0)
            if (chan > 0) {
                int moved = 0;
                if (lane == 0) moved = run_receivers<false, true>(n, C, V, rv, sc, p.seed, p.var_id, run, step);
                __syncwarp();
                if (__shfl_sync(kFullWarp, moved, 0)) {
                    new_rates = new_feat = refresh = true;
                    goal = __shfl_sync(kFullWarp, sc.goal, 0);
                }
                chan = 0;
            }
            if (rate_table && new_rates) {
                for (uint32_t j = lane; j < P; j += 32u) rv.rates[j] = inv_rate(eval(n, rv.vars, n.rate_prog[j]));
                __syncwarp();
                refresh = true;
            }
            new_rates = false;

            // the proposal's class factors
            const float tf = mlp_time_feature(time, p.horizon);
            if (new_feat || tf != tf_last) {
                float v4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (F.var[i] >= 0) v4[i] = rv.vars[F.var[i]];
                const float clk = F.clock_var >= 0 ? rv.vars[F.clock_var] : 0.0f;
                float x[CSMC_MLP_IN];
                mlp_features(0, F, v4, clk, time, p.horizon, x);
                tf_last = tf;
                new_feat = false;
                bool same = true;
#pragma unroll
                for (int i = 0; i < 6; ++i) same = same && __float_as_uint(x[4 + i]) == x_last[i];
                if (!same) {  // warp-uniform: every lane holds the same features
                    float theta[CSMC_MLP_CLASSES];
                    if (TC) theta_tc(mlp, x, theta);
                    else theta_exact(mlp, h1s, x, theta);
#pragma unroll
                    for (uint32_t l = 0; l < CSMC_MLP_CLASSES; ++l) mfac[l] = tilt_factor(theta[l]);
#pragma unroll
                    for (int i = 0; i < 6; ++i) x_last[i] = __float_as_uint(x[4 + i]);
                    refresh = true;
                    if (TRACE) {
#pragma unroll
                        for (uint32_t w = 0; w < 40u; ++w) {
                            const uint32_t l = w / 10u, f = 2u * (w % 10u);
                            if (f >= CSMC_MLP_IN) continue;
                            const uint32_t v =
                                f_to_bf16(feat_of(x, l, f)) | (static_cast<uint32_t>(f_to_bf16(feat_of(x, l, f + 1))) << 16);
                            if (w < 32u && lane == w) xw0 = v;
                            if (w >= 32u && lane == w - 32u) xw1 = v;
                        }
                    }
                }
            }

            // ---- refresh: the components' records and the warp's sums
            if (refresh) {
                double rate_sum = 0.0, inv_sum[CSMC_MLP_CLASSES];
#pragma unroll
                for (int l = 0; l < CSMC_MLP_CLASSES; ++l) inv_sum[l] = 0.0;
                uint32_t have = 0;
                // per class, the last tilted 1/rate of this lane and its quotients
                float k_inv[CSMC_MLP_CLASSES] = {-1.0f, -1.0f, -1.0f, -1.0f};
                double k_diff[CSMC_MLP_CLASSES] = {0.0, 0.0, 0.0, 0.0};
                double k_rec[CSMC_MLP_CLASSES] = {0.0, 0.0, 0.0, 0.0};
                for (uint32_t q = lane; q < nb; q += 32u) {
#pragma unroll 1
                    for (uint32_t k = 0; k < 4; ++k) {
                        const uint32_t c = 4u * q + k;
                        uint32_t form = 0u;
                        float inv = 0.0f, invp = __uint_as_float(0x7fffffffu);  // no component: a delay of NaN
                        if (c < C) {
                            const uint32_t li = rv.locv[c];
                            const uint32_t l = (li - n.comp[c].loc_begin) & 3u;
                            const uint64_t dsc = n.loc_desc[li];
                            const uint32_t lo = static_cast<uint32_t>(dsc), fl = static_cast<uint32_t>(dsc >> 32);
                            if (fl & CSMC_DESC_ZERO) {
                                form = 1u;
                            } else {
                                inv = (fl & CSMC_DESC_PROG) ? rv.rates[lo] : __uint_as_float(lo);
                                invp = inv;
                                if (tiltable(inv)) {
                                    invp = f_mul(inv, l == 0 ? mfac[0] : (l == 1 ? mfac[1] : (l == 2 ? mfac[2] : mfac[3])));
                                    const float kv = l == 0 ? k_inv[0] : (l == 1 ? k_inv[1] : (l == 2 ? k_inv[2] : k_inv[3]));
                                    if (kv != inv) {
                                        const double r = d_rcp(static_cast<double>(inv));
                                        const double diff = d_sub(d_rcp(static_cast<double>(invp)), r);  // rate_change
#pragma unroll
                                        for (int j = 0; j < CSMC_MLP_CLASSES; ++j)
                                            if (static_cast<uint32_t>(j) == l) {
                                                k_inv[j] = inv;
                                                k_diff[j] = diff;
                                                k_rec[j] = r;
                                            }
                                    }
                                    rate_sum = d_add(rate_sum, l == 0 ? k_diff[0] : (l == 1 ? k_diff[1] : (l == 2 ? k_diff[2] : k_diff[3])));
                                    if (TRACE) {
#pragma unroll
                                        for (int j = 0; j < CSMC_MLP_CLASSES; ++j)
                                            if (static_cast<uint32_t>(j) == l) inv_sum[j] = d_add(inv_sum[j], k_rec[j]);
                                        have |= 1u << l;
                                    }
                                }
                            }
                        }
                        invv[c] = inv;
                        reinterpret_cast<uint2 *>(rec + (k >> 1) * nb + q)[k & 1u] = make_uint2(__float_as_uint(invp), form);
                    }
                }
                const double ln2 = 0.6931471805599453;
                lr = d_mul(ln2, warp_sum_d(rate_sum));
                if (TRACE) {
#pragma unroll
                    for (int l = 0; l < CSMC_MLP_CLASSES; ++l) {
                        const double s = warp_sum_d(inv_sum[l]);
                        if (duty_row == static_cast<uint32_t>(l)) a_sum = s;
                    }
                    present = __reduce_or_sync(kFullWarp, have);
                }
                __syncwarp();
                refresh = false;
            }

            // ---- the race: per-lane minima, then the warp's
            uint32_t bkey = 0xffffffffu, bbr = 0xffffffffu;
            float bd = 0.0f;
            for (uint32_t q = lane; q < nb; q += 32u) {
                const uint4 r0 = rec[q], r1 = rec[nb + q];
                const u32x4 blk = philox_one(p.keys, step, run, q);
                float d0 = exp_delay(blk.x, __uint_as_float(r0.x)), d1 = exp_delay(blk.y, __uint_as_float(r0.z));
                float d2 = exp_delay(blk.z, __uint_as_float(r1.x)), d3 = exp_delay(blk.w, __uint_as_float(r1.z));
                if (r0.y | r0.w | r1.y | r1.w) {
                    if (r0.y) d0 = 0.0f;
                    if (r0.w) d1 = 0.0f;
                    if (r1.y) d2 = 0.0f;
                    if (r1.w) d3 = 0.0f;
                }
                // in order of bit-reversed index (0, 2, 1, 3): a later equal key loses
                uint32_t key = group_key(d0), kk = 0, o = group_key(d2);
                float d = d0;
                if (o < key) key = o, kk = 2, d = d2;
                o = group_key(d1);
                if (o < key) key = o, kk = 1, d = d1;
                o = group_key(d3);
                if (o < key) key = o, kk = 3, d = d3;
                const uint32_t br = bitrev_bits(4u * q + kk, bits);
                if (key < bkey || (key == bkey && key != 0xffffffffu && br < bbr)) {
                    bkey = key;
                    bbr = br;
                    bd = d;
                }
            }
            const uint32_t m = __reduce_min_sync(kFullWarp, bkey);
            if (m == 0xffffffffu) {  // every delay is NaN: the lowest index
                bbr = 0xffffffffu;
                for (uint32_t c = lane; c < C; c += 32u) bbr = min(bbr, bitrev_bits(c, bits));
            }
            const uint32_t win = bitrev_bits(__reduce_min_sync(kFullWarp, bkey == m ? bbr : 0xffffffffu), bits);
            const float dmin =
                m == 0xffffffffu ? __uint_as_float(0x7fffffffu) : __shfl_sync(kFullWarp, bd, (win >> 2) & 31u);
            const uint32_t li = rv.locv[win], base = n.comp[win].loc_begin;
            const uint32_t wl = (li - base) & 3u;
            const float inv_w = invv[win];
            const bool tilted_w = tiltable(inv_w);
            const bool finite = dmin < __uint_as_float(0x7f800000u);
            if (finite) {
                double r = d_mul(lr, static_cast<double>(dmin));
                if (tilted_w) {
                    const uint32_t invp_w = reinterpret_cast<const uint2 *>(rec + ((win >> 1) & 1u) * nb + (win >> 2))[win & 1u].x;
                    const WinTerm t = terms[wl];
                    double term = t.term;
                    if (t.inv != __float_as_uint(inv_w) || t.invp != invp_w) {
                        const double ln2 = 0.6931471805599453;
                        term = d_mul(ln2, log2_d(d_div(static_cast<double>(__uint_as_float(invp_w)),
                                                       static_cast<double>(inv_w))));
                        __syncwarp();
                        if (lane == 0) terms[wl] = WinTerm{__float_as_uint(inv_w), invp_w, term};
                        __syncwarp();
                    }
                    r = d_add(r, term);
                }
                logw = d_add(logw, r);
            }
            if (TRACE) {
                const bool has = finite && ((present >> duty_row) & 1u);
                uint32_t w0 = xw0, w1 = xw1;
                if (duty_a || duty_b) {
                    const float a = has ? row_a(a_sum, dmin, row_w) : 0.0f;
                    const float b = (has && tilted_w && wl == duty_row) ? row_w : 0.0f;
                    const uint32_t v = __float_as_uint(duty_a ? a : b);
                    if (lane < 8) w1 = v;
                    else w0 = v;
                }
                const uint64_t r = row0 + 4ull * step;
                uint32_t *out = reinterpret_cast<uint32_t *>(ip.rows + r);
                if (r + 3 < ip.rows_cap) {
                    out[lane] = w0;
                    if (lane < 8) out[32 + lane] = w1;
                } else {  // rows beyond the buffer are skipped and counted
                    if (r + lane / 10u < ip.rows_cap) out[lane] = w0;
                    if (lane < 4 && r + lane >= ip.rows_cap) atomicAdd(p.scratch + 4, 1ull);
                }
            }

            // ---- clocks, the winner's transition, time
            if (finite) {
                if (n.n_clocks) {
                    advance_clocks<false>(n, n.n_clocks, rv.vars, dmin, lane, 32u);
                    __syncwarp();
                    new_feat = true;
                    new_rates = rates_read_clocks;
                }
                const csmc_loc L = n.loc[li];
                uint32_t en = 0;
                if (L.n_edges) {
                    bool ok = false;
                    if (lane < L.n_edges) {
                        const csmc_edge e = n.edge[L.edge_begin + lane];
                        ok = e.channel >= 0 && guards_ok(n, rv.vars, e);
                    }
                    en = __ballot_sync(kFullWarp, ok);
                }
                if (en) {
                    int st = 0;
                    if (lane == 0) {
                        const uint32_t slots = write_slots(rv.slotv[win], en);
                        rv.slotv[win] = slots;
                        rv.set_local(n, win, take_edge<false>(n, rv.vars, sc, p.seed, p.var_id, run, step, win, li - base,
                                                              en, slots, 0));
                        st = sc.chan * 2 + sc.goal;
                    }
                    __syncwarp();
                    st = __shfl_sync(kFullWarp, st, 0);
                    chan = st >> 1;
                    goal = st & 1;
                    new_rates = new_feat = refresh = true;
                }
            }
            time = time_add(time, dmin);
            ++step;
        }
    }
    if (lane == 0) {
        if (acc_hits) atomicAdd(p.scratch + 1, acc_hits);
        if (acc_steps) atomicAdd(p.scratch + 2, acc_steps);
        if (acc_capped) atomicAdd(p.scratch + 3, acc_capped);
    }
}

}  // namespace detail
}  // namespace csmc
