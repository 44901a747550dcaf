// Lane-group simulation kernel (see sim.cuh for the mapping); instantiated
// per (lanes per run, components per lane) shape in sim_shapes_*.cu.
// Semantics follow the reference kernel; file:line references are to
// simulation/simulation.cu of the reference.
//
// What bounds it: a run's steps are a serial chain, so a launch that does not
// fill the GPU takes (steps of its longest run) x (latency of one step), and
// one that does is bound by instruction issue.  Both ask for few dependent
// instructions per step:
//   * what a component's delay needs is one 8-byte record (1/rate and the
//     delay's form) in shared memory, read as it is by the component's lane
//     and written again only when the component has moved or the rate table
//     has changed (kept in registers, the records of 4 to 16 components cost
//     more in spills than their 16-byte shared loads);
//   * the rate table is evaluated again only after a transition (unless a
//     rate reads a clock), the clocks advance by one float addition each;
//   * the race is two warp-wide integer minima (delay key, then bit-reversed
//     index) in a full warp, a butterfly of 32-bit words in a narrower group;
//   * a winner without edges is done there; else the lanes evaluate the
//     guards of its edges in parallel and one lane takes the chosen edge.
// All groups of a warp meet at the head of the step loop, so groups whose
// runs end at different steps keep advancing together.
// Measured (B200), against the form with a 64-bit butterfly, per-component
// location records read every step and every step's rate table evaluated:
// 100 agents, 32 lanes x 4, 64 runs 9.3 -> 2.7 ms, 65,536 runs 142 -> 45 ms;
// 256-process mutex, 32 x 8, 2,000 runs 237 -> 80 ms (1,370 -> 685 warp
// instructions a step).
#pragma once
#include "sim_common.cuh"

namespace csmc {
namespace detail {

struct RunState {  // per group, in shared memory (group_state_stride bytes)
    RunScalars sc;
    uint32_t pad2[2];
    float vars[1];  // n_vars entries, then n_rate_prog inverse rates, then
                    // (at group_vars_bytes) the delay records, the slot
                    // masks and the global location indices of the components
};

// Where a run's Philox round keys come from: the kernel's parameter bank
// (one network, one seed) or the seed itself (a batch job).
struct BankKeys {
    const PhiloxKeys &k;
    __device__ __forceinline__ u32x4 block(uint32_t step, uint64_t run, uint32_t q) const {
        return philox_one(k, step, run, q);
    }
};
struct SeedKeys {
    uint64_t seed;
    __device__ __forceinline__ u32x4 block(uint32_t step, uint64_t run, uint32_t q) const {
        return delay_block(seed, run, step, q);
    }
};

template <bool VERIFY>
static __device__ __noinline__ uint32_t group_take(const uint8_t *base, RunState *s, uint64_t seed, int32_t var_id,
                                                   uint64_t run, uint32_t step, uint32_t c, uint32_t cur_loc,
                                                   uint32_t en, uint32_t slot_mask, uint32_t which) {
    return take_edge<VERIFY>(net_view(base), VarView{s->vars, 1}, s->sc, seed, var_id, run, step, c, cur_loc, en,
                             slot_mask, which);
}

static __device__ __noinline__ uint32_t recv_mask(const uint8_t *base, RunState *s, uint32_t li, int chan) {
    return recv_edges(net_view(base), VarView{s->vars, 1}, li, chan);
}

// Delay of a component outside the cached forms (several invariants, a
// computed bound, a rate that is evaluated per component).
static __device__ __noinline__ float group_slow_delay(const uint8_t *base, const float *vars, const float *rates,
                                                      uint32_t li, uint32_t x) {
    return comp_delay(net_view(base), VarView{const_cast<float *>(vars), 1}, VarView{const_cast<float *>(rates), 1},
                      li, x);
}

// Form of a component's delay, the second word of its record: exponential,
// zero, through comp_delay, or the one-invariant word + kFormInv1.
constexpr uint32_t kFormExp = 0u, kFormZero = 1u, kFormSlow = 2u, kFormInv1 = 3u;

// Bit reversal of k over the K (a power of two) components of a lane.
static __host__ __device__ constexpr int lane_brev(int k, int K) {
    int r = 0;
    for (int b = 1; b < K; b <<= 1) {
        r = (r << 1) | (k & 1);
        k >>= 1;
    }
    return r;
}

// One run at a time simulated by the G lanes of a group of at most `cap`
// components, B NB of them per lane (B: of one Philox block; NB 0: given at
// run time by `cap`).  Few per lane (NB 1, 2) are consecutive: lane gl holds
// gl B NB ..; else lane gl holds the blocks gl, gl + G, gl + 2 G, .., so that a
// step draws ceil(blocks / G) blocks per lane whatever the shape's share
// (batches: one shape for networks of 4 to 512 components; 16 random
// networks, 16,000 runs 108 against 126 ms).  With two blocks per lane the
// consecutive form measured up to 11 % faster (random 64, 8 x 8, 131,072 runs:
// 89 against 99 ms).  The group's scalars, variables, rate table, slot masks
// and locations live in *s.
template <int G, int B, int NB, bool VERIFY>
struct GroupRun {
    static constexpr bool kStrided = NB == 0 || NB >= 4;
    RunState *s;
    uint32_t gl, gbase, gmask;
    uint2 *rec;        // delay records (rec_of)
    uint32_t *slotv;   // per component
    uint16_t *locv;    // per component: global location index
    float *rates;
    // this run
    float time;
    uint32_t step, chan, goal;
    bool dirty;        // variables changed since the rate table was evaluated
    uint32_t pm;       // bit k: this lane's component k has its rate from the table
    uint32_t cap;      // components the state is laid out for
    // one block per lane (NB 1): the next step's draws and their -log2, drawn
    // while the step before waits for its race and its tables
    uint32_t nx[NB == 1 ? B : 1];
    float nl[NB == 1 ? B : 1];

    __device__ __forceinline__ GroupRun(RunState *state, uint32_t lane, uint32_t capacity) {
        cap = NB ? G * B * NB : capacity;
        s = state;
        gl = lane % G;
        gbase = lane - gl;
        gmask = G == 32 ? 0xffffffffu : (((1u << (G & 31)) - 1u) << gbase);
    }

    // Record of this lane's component k (its b-th block's i-th: k = B b + i):
    // pairs of components side by side (one 16-byte load), lanes next to each
    // other.
    __device__ __forceinline__ uint2 *rec_of(int k) const {
        return B == 1 ? rec + gl : rec + 2 * ((k >> 1) * G + gl) + (k & 1);
    }
    // Component k of this lane, and the lane and k of a component.
    __device__ __forceinline__ uint32_t comp_of(uint32_t k) const {
        return kStrided ? 4u * (gl + G * (k >> 2)) + (k & 3u) : B * NB * gl + k;
    }
    static __device__ __forceinline__ uint32_t lane_of(uint32_t c) { return kStrided ? (c / B) % G : c / (B * NB); }
    static __device__ __forceinline__ int k_of(uint32_t c) {
        return static_cast<int>(kStrided ? 4u * ((c >> 2) / G) + (c & 3u) : c % (B * NB));
    }
    // This lane's components are 0 .. n_k - 1 (whole blocks).
    __device__ __forceinline__ uint32_t n_k(uint32_t C) const {
        if (!kStrided) return B * NB;
        const uint32_t nb = (C + 3u) >> 2;
        return gl < nb ? 4u * ((nb - gl + G - 1u) / G) : 0u;
    }
    // Writes the records of all of this lane's components.
    __device__ __forceinline__ void look_up_all(const Net &n) {
        const uint32_t kn = n_k(n.n_comps);
#pragma unroll 1
        for (uint32_t k = 0; k < kn; ++k) {
            const uint32_t c = comp_of(k);
            if (c < n.n_comps) look_up<true>(n, static_cast<int>(k), locv[c]);
            else *rec_of(static_cast<int>(k)) = make_uint2(0x7fffffffu, kFormExp);  // no component: a delay of NaN
        }
    }

    // Writes component k's record from its location li.  RATE false: a rate
    // from the table is left out (the next step evaluates the table and writes
    // it, and other lanes may be storing that table already).
    template <bool RATE>
    __device__ __forceinline__ void look_up(const Net &n, int k, uint32_t li) {
        const uint64_t dsc = n.loc_desc[li];
        const uint32_t lo = static_cast<uint32_t>(dsc), fl = static_cast<uint32_t>(dsc >> 32);
        uint32_t inv = lo, form = kFormExp;
        pm &= ~(1u << k);
        if (fl & CSMC_DESC_ZERO) {
            form = kFormZero;
        } else if ((fl & CSMC_DESC_EVAL) || (fl & (CSMC_DESC_INV | CSMC_DESC_INV1)) == CSMC_DESC_INV) {
            form = kFormSlow;
        } else {
            if (fl & CSMC_DESC_INV) {
                const uint32_t w = n.loc_inv1[li];
                form = w < 0xffffffffu - kFormInv1 ? w + kFormInv1 : kFormSlow;
            }
            if (fl & CSMC_DESC_PROG) {
                pm |= 1u << k;
                if (RATE) inv = __float_as_uint(rates[lo]);
            }
        }
        *rec_of(k) = make_uint2(inv, form);
    }

    template <class KEYS>
    __device__ __forceinline__ void draw(const KEYS &keys, uint64_t run, uint32_t at) {
        if constexpr (NB == 1) {
            const uint32_t c = gl * B;
            const u32x4 blk = keys.block(at, run, c >> 2);
#pragma unroll
            for (int i = 0; i < B; ++i) {
                nx[i] = B == 4 ? word_of(blk, i) : word_of(blk, (c + i) & 3u);
                nl[i] = neg_log2_draw(nx[i]);
            }
        }
    }

    // run initialisation (simulation.cu:766-831)
    template <class Q, class KEYS>
    __device__ __forceinline__ void init(const Net &n, const Q &q, const KEYS &keys, uint64_t run) {
        const uint32_t C = n.n_comps, V = n.n_vars;
        uint8_t *tail = reinterpret_cast<uint8_t *>(s) + group_vars_bytes(V, n.n_rate_prog);
        rec = reinterpret_cast<uint2 *>(tail);
        slotv = reinterpret_cast<uint32_t *>(tail + 8u * cap);
        locv = reinterpret_cast<uint16_t *>(tail + 12u * cap);
        rates = s->vars + V;
        __syncwarp(gmask);  // the lanes are done with the previous run's state
        for (uint32_t v = gl; v < V; v += G) s->vars[v] = n.var[v].init;
        if (gl == 0) {
            double q0 = 0.0;
            if (q.var_id >= 0 && static_cast<uint32_t>(q.var_id) < V && n.var[q.var_id].kind == 0)
                q0 = static_cast<double>(n.var[q.var_id].init);
            s->sc.qmin = q0;
            s->sc.qmax = q0;
            s->sc.chan = 0;
            s->sc.sender = -1;
            s->sc.goal = 0;
            s->sc.digest = 0xcbf29ce484222325ull;
        }
        for (uint32_t c = gl; c < C; c += G) {
            locv[c] = static_cast<uint16_t>(n.comp[c].loc_begin + n.comp[c].init_local);
            slotv[c] = 0u;
        }
        __syncwarp(gmask);
        time = 0.0f;
        step = 0;
        chan = 0;
        goal = 0;
        pm = 0;
        eval_rates(n);
        look_up_all(n);
        __syncwarp(gmask);  // before the first step may evaluate the rate table again
        dirty = false;
        draw(keys, run, 0u);
    }

    // distinct rate programs, spread over the lanes
    __device__ __forceinline__ void eval_rates(const Net &n) {
        if (!(n.flags & CSMC_NET_RATE_TABLE) || n.n_rate_prog == 0) return;
        for (uint32_t j = gl; j < n.n_rate_prog; j += G)
            rates[j] = inv_rate(eval(n, VarView{s->vars, 1}, n.rate_prog[j]));
        __syncwarp(gmask);
    }

    // Broadcast receivers of the previous step's sender (SyncInSerial,
    // simulation.cu:357-407): every enabled set is taken before any receiver
    // moves, then the receivers move in component order.
    template <class Q>
    __device__ __forceinline__ void receivers(const Net &n, const Q &q, uint64_t run) {
        const uint32_t C = n.n_comps;
        const int sender = s->sc.sender;
        uint32_t *const rmv = reinterpret_cast<uint32_t *>(rec);  // the records are written again below
        const uint32_t kn = n_k(C), kmax = !kStrided ? B * NB : 4u * ((((C + 3u) >> 2) + G - 1u) / G);
        // the masks overwrite the records: one lane's mask lies in another
        // lane's record, which that lane may have written at the end of the
        // step before
        __syncwarp(gmask);
#pragma unroll 1
        for (uint32_t k = 0; k < kn; ++k) {
            const uint32_t c = comp_of(k);
            uint32_t m = 0;
            if (c < C && static_cast<int>(c) != sender && n.loc[locv[c]].n_recv)
                m = recv_mask(n.base, s, locv[c], static_cast<int>(chan));
            rmv[k * G + gl] = m;
        }
        __syncwarp(gmask);
        // in component order: lane by lane, of the strided form block row by block row
        constexpr uint32_t kRow = kStrided ? B : B * NB;
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < kmax; k0 += kRow) {
            bool any = false;
            for (uint32_t k = k0; k < k0 + kRow && k < kn; ++k) any |= rmv[k * G + gl] != 0;
            uint32_t pending = (__ballot_sync(gmask, any) & gmask) >> gbase;
            if (pending) dirty = true;
            while (pending) {
                const uint32_t who = static_cast<uint32_t>(__ffs(pending) - 1);
                if (gl == who) {
#pragma unroll 1
                    for (uint32_t k = k0; k < k0 + kRow && k < kn; ++k) {
                        const uint32_t c = comp_of(k), rm = rmv[k * G + gl];
                        if (!rm) continue;
                        const uint32_t base = n.comp[c].loc_begin;
                        const uint32_t m = write_slots(slotv[c], rm);
                        slotv[c] = m;
                        if (VERIFY) mix(s->sc.digest, c | 0x80000000u);
                        locv[c] = static_cast<uint16_t>(base + group_take<VERIFY>(n.base, s, q.seed, q.var_id, run, step,
                                                                                  c, locv[c] - base, rm, m, 1));
                    }
                }
                __syncwarp(gmask);
                pending &= pending - 1;
            }
        }
        __syncwarp(gmask);
        look_up_all(n);
        goal = static_cast<uint32_t>(s->sc.goal);
    }

    // This lane's delays and their minimum (simulation.cu:409-541): key,
    // bit-reversed index and the delay itself.
    template <class KEYS>
    __device__ __forceinline__ void lane_min(const Net &n, const KEYS &keys, uint64_t run, uint32_t bits,
                                             uint32_t &bkey, uint32_t &bbr, float &bd) {
        const uint32_t C = n.n_comps;
        bkey = 0xffffffffu;
        bbr = 0xffffffffu;
        bd = 0.0f;
#pragma unroll 1
        for (int b = 0; NB == 0 || b < B * NB; b += B) {
            const uint32_t c = comp_of(b);
            if (NB != 1 && c >= C) break;  // no components from here on
            uint32_t iv[B], form[B];
            if (B == 1) {
                const uint2 r = rec[gl];
                iv[0] = r.x;
                form[0] = r.y;
            } else {
#pragma unroll
                for (int h = 0; h < B / 2; ++h) {
                    const uint4 r = *reinterpret_cast<const uint4 *>(rec_of(b + 2 * h));
                    iv[2 * h] = r.x;
                    form[2 * h] = r.y;
                    iv[2 * h + 1] = r.z;
                    form[2 * h + 1] = r.w;
                }
            }
            uint32_t xs[B];
            float d[B];
            uint32_t special = 0;
            if constexpr (NB == 1) {
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    xs[i] = nx[i];
                    d[i] = f_mul(nl[i], __uint_as_float(iv[i]));
                    special |= form[i];
                }
            } else {
                const u32x4 blk = keys.block(step, run, c >> 2);
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    xs[i] = B == 4 ? word_of(blk, i) : word_of(blk, (c + i) & 3u);
                    d[i] = exp_delay(xs[i], __uint_as_float(iv[i]));
                    special |= form[i];
                }
            }
            if (special) {
#pragma unroll
                for (int i = 0; i < B; ++i) {
                    const uint32_t x = xs[i];
                    if (form[i] >= kFormInv1) {
                        // uniform on (0, bound - clock] while the bound lies
                        // ahead (comp_delay's arithmetic, inv1_delay)
                        const uint32_t w = form[i] - kFormInv1;
                        double ttb = d_sub(n.konst[CSMC_INV1_CONST(w)], static_cast<double>(s->vars[CSMC_INV1_VAR(w)]));
                        if (CSMC_INV1_STRICT(w)) ttb = d_sub(ttb, 1e-6);
                        if (ttb >= 0) d[i] = uniform_delay(x, ttb);
                    } else if (form[i] == kFormZero) {
                        d[i] = 0.0f;
                    } else if (form[i] == kFormSlow) {
                        d[i] = group_slow_delay(n.base, s->vars, rates, locv[c + i], x);
                    }
                }
            }
            uint32_t key = 0xffffffffu;
            int kk = 0;
            float d0 = 0.0f;
#pragma unroll
            for (int j = 0; j < B; ++j) {
                // in order of bit-reversed index, so a later equal key loses
                const int i = lane_brev(j, B);
                const uint32_t kd = group_key(d[i]);
                if (kd < key) {
                    key = kd;
                    kk = i;
                    d0 = d[i];
                }
            }
            const uint32_t br = bitrev_bits(c + kk, bits);
            if (key < bkey || (key == bkey && key != 0xffffffffu && br < bbr)) {
                bkey = key;
                bbr = br;
                bd = d0;
            }
        }
    }

    // The lowest bit-reversed index among this lane's components (a race in
    // which every delay is NaN).
    __device__ __forceinline__ uint32_t lowest_brev(uint32_t C, uint32_t bits) const {
        uint32_t r = 0xffffffffu;
        for (uint32_t k = 0; k < n_k(C); ++k)
            if (comp_of(k) < C) r = min(r, bitrev_bits(comp_of(k), bits));
        return r;
    }

    static __device__ __forceinline__ uint32_t group_min(uint32_t v, uint32_t mask) {
        if (G == 32) return __reduce_min_sync(mask, v);
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) v = min(v, __shfl_xor_sync(mask, v, off, G));
        return v;
    }

    // One step of the run: receivers, rate table, delays, race, clock
    // advance, the winner's transition, time.
    template <class Q, class KEYS>
    __device__ __forceinline__ void advance(const Net &n, const Q &q, const KEYS &keys, uint64_t run, uint32_t bits) {
        const VarView vars{s->vars, 1};
        if (chan) {
            if (has_receivers(n, static_cast<int>(chan))) receivers(n, q, run);
            __syncwarp(gmask);
            if (gl == 0) {
                s->sc.chan = 0;
                s->sc.sender = -1;
            }
            chan = 0;
            __syncwarp(gmask);
        }
        if (dirty || !(n.flags & CSMC_NET_RATE_NO_CLOCK)) {
            eval_rates(n);
            for (uint32_t left = pm; left; left &= left - 1) {
                const int k = __ffs(left) - 1;
                rec_of(k)->x = __float_as_uint(rates[static_cast<uint32_t>(n.loc_desc[locv[comp_of(k)]])]);
            }
            dirty = false;
        }

        // ---- delays and the race (simulation.cu:409-628)
        uint32_t bkey, bbr;
        float bd;
        lane_min(n, keys, run, bits, bkey, bbr, bd);
        const uint32_t m = group_min(bkey, gmask);
        draw(keys, run, step + 1u);
        if (m == 0xffffffffu) {
            bbr = lowest_brev(n.n_comps, bits);
            bd = __uint_as_float(0x7fffffffu);
        }
        const uint32_t win = bitrev_bits(group_min(bkey == m ? bbr : 0xffffffffu, gmask), bits);
        const uint32_t owner = lane_of(win);
        const float dmin = G == 1 ? bd : __shfl_sync(gmask, bd, owner, G);
        if (VERIFY && gl == 0) {
            mix(s->sc.digest, step);
            mix(s->sc.digest, win);
            mix(s->sc.digest, f_bits(dmin));
        }
        if (dmin < __uint_as_float(0x7f800000u)) {
            // clocks advance (simulation.cu:632-651)
            if (n.n_clocks) {
                // (a full warp with many clocks per lane; narrower groups have no registers to spare)
                advance_clocks<(G == 32 && NB != 1)>(n, n.n_clocks, vars, dmin, gl, G);
                __syncwarp(gmask);
            }
            // the winner's enabled edges (simulation.cu:268-305), one lane per edge
            const uint32_t li = locv[win];
            const csmc_loc L = n.loc[li];
            uint32_t en = 0;
            for (uint32_t e0 = 0; e0 < L.n_edges; e0 += G) {
                bool ok = false;
                if (e0 + gl < L.n_edges) {
                    const csmc_edge e = n.edge[L.edge_begin + e0 + gl];
                    ok = e.channel >= 0 && guards_ok(n, vars, e);
                }
                const uint32_t b = G == 1 ? (ok ? 1u : 0u) : ((__ballot_sync(gmask, ok) & gmask) >> gbase);
                en |= b << e0;
            }
            if (en) {
                if (gl == 0) {
                    const uint32_t base = n.comp[win].loc_begin;
                    const uint32_t slots = write_slots(slotv[win], en);
                    slotv[win] = slots;
                    locv[win] = static_cast<uint16_t>(base + take_edge<VERIFY>(n, vars, s->sc, q.seed, q.var_id, run,
                                                                               step, win, li - base, en, slots, 0));
                }
                __syncwarp(gmask);
                dirty = true;
                chan = static_cast<uint32_t>(s->sc.chan);
                goal = static_cast<uint32_t>(s->sc.goal);
                if (gl == owner) look_up<false>(n, k_of(win), locv[win]);
            } else if (VERIFY && gl == 0) {
                mix(s->sc.digest, 0xffffffffu);
            }
        }
        time = time_add(time, dmin);  // simulation.cu:876-882
        ++step;
    }

    // Ended runs (simulation.cu:835-849, 887-893): true when the run is over;
    // the first lane writes its outputs and adds to its counters.
    template <class Q>
    __device__ __forceinline__ bool finish(const Net &n, const Q &q, uint64_t ridx, unsigned long long &acc_hits,
                                           unsigned long long &acc_steps, unsigned long long &acc_capped) {
        const bool timeout = !(time < q.horizon);
        const bool at_goal = q.loc_mode && goal;
        if (!timeout && !at_goal && step < q.max_steps) return false;
        if (gl == 0) {
            const double val = q.is_max ? s->sc.qmax : s->sc.qmin;
            uint32_t f = (!timeout && at_goal) ? 1u : 0u;
            if (!q.loc_mode) f = q.is_max ? (val > q.threshold) : (val < q.threshold);
            if (q.flags) q.flags[ridx] = static_cast<uint8_t>(f);
            if (q.values) q.values[ridx] = val;
            if (q.steps) q.steps[ridx] = step;
            if (VERIFY && q.digests) q.digests[ridx] = s->sc.digest;
            acc_hits += f;
            acc_steps += step;
            acc_capped += (!timeout && !at_goal) ? 1u : 0u;
        }
        if (VERIFY && q.final_state) {
            const uint32_t C = n.n_comps, V = n.n_vars;
            uint32_t *w = q.final_state + ridx * (C + V);
            for (uint32_t c = gl; c < C; c += G) w[c] = locv[c] - n.comp[c].loc_begin;
            for (uint32_t v = gl; v < V; v += G) w[C + v] = f_bits(s->vars[v]);
        }
        return true;
    }
};

// At most 512 threads per CTA, 128 registers a thread (16 warps per SM).
template <int G, int K, bool VERIFY>
__global__ void __launch_bounds__(512, 1) sim_kernel(const __grid_constant__ SimParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    stage_network(smem, p.blob, p.blob_bytes);
    __syncthreads();
    const Net n = net_view(smem, p.net);
    const uint32_t bits = ceil_log2(p.net.n_comps);
    const BankKeys keys{p.keys};
    GroupRun<G, (K < 4 ? K : 4), (K < 4 ? 1 : K / 4), VERIFY> r(
        reinterpret_cast<RunState *>(smem + p.blob_bytes + (threadIdx.x / G) * p.state_stride), threadIdx.x & 31u, G * K);

    unsigned long long acc_hits = 0, acc_steps = 0, acc_capped = 0;
    unsigned long long ridx = 0;
    if constexpr (G == 32) {  // one run per warp: no other group to meet
        for (;;) {
            if (r.gl == 0) ridx = atomicAdd(p.scratch, 1ull);
            ridx = __shfl_sync(0xffffffffu, ridx, 0);
            if (ridx >= p.n_runs) break;
            const uint64_t run = p.first_run + ridx;
            r.init(n, p, keys, run);
            while (!r.finish(n, p, ridx, acc_hits, acc_steps, acc_capped)) r.advance(n, p, keys, run, bits);
        }
    } else {
        bool have = false, drained = false;
        for (;;) {
            __syncwarp();
            if (!have && !drained) {
                if (r.gl == 0) ridx = atomicAdd(p.scratch, 1ull);
                ridx = __shfl_sync(r.gmask, ridx, 0, G);
                if (ridx >= p.n_runs) {
                    drained = true;
                } else {
                    have = true;
                    r.init(n, p, keys, p.first_run + ridx);
                }
            }
            if (__all_sync(0xffffffffu, drained)) break;
            if (have) {
                if (r.finish(n, p, ridx, acc_hits, acc_steps, acc_capped)) have = false;
                else r.advance(n, p, keys, p.first_run + ridx, bits);
            }
        }
    }
    if (r.gl == 0) {
        if (acc_hits) atomicAdd(p.scratch + 1, acc_hits);
        if (acc_steps) atomicAdd(p.scratch + 2, acc_steps);
        if (acc_capped) atomicAdd(p.scratch + 3, acc_capped);
    }
}

}  // namespace detail

template <int G, int K, bool VERIFY>
int launch_one(const SimParams &p, int grid, int block, size_t smem, void *stream) {
    auto fn = detail::sim_kernel<G, K, VERIFY>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    fn<<<grid, block, smem, static_cast<cudaStream_t>(stream)>>>(p);
    return static_cast<int>(cudaGetLastError());
}

template <int G, int K, bool VERIFY>
int occupancy_one(int block, size_t smem, int *ctas) {
    auto fn = detail::sim_kernel<G, K, VERIFY>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    return static_cast<int>(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, fn, block, smem));
}

// Explicit instantiation of the launch helpers for one shape.
#define CSMC_INSTANTIATE_SHAPE(GG, KK)                                                  \
    template int launch_one<GG, KK, false>(const SimParams &, int, int, size_t, void *); \
    template int launch_one<GG, KK, true>(const SimParams &, int, int, size_t, void *);  \
    template int occupancy_one<GG, KK, false>(int, size_t, int *);                        \
    template int occupancy_one<GG, KK, true>(int, size_t, int *);

}  // namespace csmc
