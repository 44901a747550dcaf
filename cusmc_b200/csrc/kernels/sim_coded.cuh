// Thread-per-run simulation kernel for networks with race classes: the
// race reads one packed word per four components.
//
// Every component's location is kept as one byte, local index (5 bits) |
// delay code (3 bits): 0..3 the location's race class, 7 a location whose
// delay goes through its descriptor (zero-delay types, invariant-bounded or
// unclassed exponential locations), 6 padding past the last component.  The
// bytes of components 4q..4q+3 form word q of the thread's state, so one
// shared load gives the codes of the four components that share Philox
// block q.  A class member contributes only its key, (24-bit draw) * 256 +
// (255 - bit-reversed q), to its class's largest key; each class keeps four
// independent maxima, one per word of the Philox block (chain k).  A block's
// four key words are loaded together, then stored together (the chains are
// disjoint; member by member, every load would wait behind the store before
// it), and the key's address is the thread's own key address plus the code
// field moved to the class stride: one mask, one shift-and-add.  After the
// components, the chains of a class are merged (a chain's keys stand for
// its part of the bit-reversed index) and the class takes part in the race
// with its largest key, as in race_classes (sim_run.cuh).  Where
// race_classes consults the second largest key (a lower draw that rounds to
// the same float delay could hide a member with a smaller index), this
// kernel falls back to race_exact whenever the largest draw of the winning
// class sits on such a flat spot of the delay function (about 2e-4 .. 4e-3
// per step for a class of 1-10 members, far less with many), and whenever
// two classes tie; delays do not increase with the draw, so no flat spot
// means no tie with a lower draw.
//
// The Philox blocks of a step are computed through philox_step /
// philox_block (csmc_numeric.h): the counter words the blocks share are
// folded once per step, and the round keys are kernel parameters.  The
// per-step rate table is evaluated again only after a step that moved a
// component, unless a rate program reads a clock.
//
// What bounds it: per block of four components and 32 runs, 16 wide multiplies
// of Philox at 4 cycles each on the FMA-heavy pipe and about 37 two-cycle
// integer operations on the ALU pipe; the race loop alone runs at 75 cycles a
// block with four warps per scheduler (both pipes full), the rest of a step
// (class delays, rate table, transition) is latency.  100-agent epidemic, 1e6
// runs (B200): 223 ms with one load-update-store per member in turn, 180 ms
// with a block's four loads first (and one flat-spot check per step).
//
// Members outside the classes race with a delay of their own, some 80
// instructions.  Evaluated where they come up in the race loop, a warp went
// through them for nearly every component, since some lane's run had that
// component in such a location; so the loop only notes their draws, and they
// are gone through afterwards, a run's first with another run's first: as many
// turns as the run with the most has.  Mutex of 8, 32, 64 and 128 processes,
// 400,000, 200,000, 100,000 and 65,536 runs: 50 -> 41, 214 -> 143, 131 -> 80
// and 213 -> 115 ms; with the one-invariant form inline instead of a call, the
// first three 35, 127 and 70.
//
// Results are those of serial_kernel: the same draws, the same race
// outcome, the same transitions.
//
// Reference: simulation/simulation.cu:674-901 (simulation_kernel).
#pragma once
#include "sim_run.cuh"

namespace csmc {
namespace detail {

constexpr uint32_t kCodeGeneral = 7u;  // delay through the location's descriptor
constexpr uint32_t kCodePad = 6u;      // no component
constexpr uint32_t kMaxCodedComps = 256u;
#ifndef CSMC_CODED_UNROLL
#define CSMC_CODED_UNROLL 2
#endif
constexpr int kCodedUnroll = CSMC_CODED_UNROLL;  // Philox blocks of the race loop in flight per iteration
// Bytes between the chains of a class and between classes (threads of a CTA
// next to each other, at most 128).
constexpr uint32_t kKeyChain = 4u * 128u, kKeyClass = 4u * kKeyChain;
static_assert(kKeyClass == CSMC_CODED_KEY_BYTES, "coded_slab_bytes");

static __device__ __forceinline__ uint32_t ld_key(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
static __device__ __forceinline__ void st_key(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v));
}

// Run state of one thread in the class-coded layout: vars[V] | rates[P] |
// shadow[V] (floats; only for networks with receiving edges, else the
// snapshot view aliases the variables and is never used) | class keys
// (kKeyClass bytes per class) | location words [ceil(C/4)] | slots[C]
// (all 4-byte words); element i of thread t at [i * T + t], the keys at
// class * kKeyClass + chain * kKeyChain + 4 t.
struct CodedView {
    VarView vars, rates, shadow;
    uint32_t keys;    // shared-memory address of this thread's chain 0 of class 0
    uint32_t *kp;     // the same as a pointer
    uint32_t *lw;     // this thread's location word 0; stride T
    uint32_t *slotv;  // this thread's element 0; stride T
    uint32_t T;

    __device__ __forceinline__ uint32_t byte_of(uint32_t c) const {
        return reinterpret_cast<const uint8_t *>(lw + (c >> 2) * T)[c & 3u];
    }
    // global location index of component c
    __device__ __forceinline__ uint32_t loc(const Net &n, uint32_t c) const {
        return n.comp[c].loc_begin + (byte_of(c) & 31u);
    }
    __device__ __forceinline__ void set_local(const Net &n, uint32_t c, uint32_t local) const {
        const uint32_t g = CSMC_DESC_CLASS(static_cast<uint32_t>(n.loc_desc[n.comp[c].loc_begin + local] >> 32));
        const uint32_t code = g < CSMC_RACE_CLASSES ? g : kCodeGeneral;
        reinterpret_cast<uint8_t *>(lw + (c >> 2) * T)[c & 3u] = static_cast<uint8_t>(local | (code << 5));
    }
};

// key_bytes: of the keys of all classes.
static __host__ __device__ __forceinline__ uint32_t coded_words(uint32_t C) { return (C + 3u) >> 2; }

static __device__ __forceinline__ CodedView carve_coded_view(uint8_t *st, uint32_t V, uint32_t P, uint32_t C,
                                                             uint32_t key_bytes, bool recv, uint32_t T, uint32_t t) {
    float *fb = reinterpret_cast<float *>(st);
    CodedView r;
    r.vars = VarView{fb + t, T};
    r.rates = VarView{fb + V * T + t, T};
    r.shadow = recv ? VarView{fb + (V + P) * T + t, T} : r.vars;
    const uint32_t kb = 4u * ((recv ? 2u : 1u) * V + P) * T;
    r.keys = static_cast<uint32_t>(__cvta_generic_to_shared(st + kb)) + 4u * t;
    r.kp = reinterpret_cast<uint32_t *>(st + kb) + t;
    const uint32_t lb = kb + key_bytes;
    r.lw = reinterpret_cast<uint32_t *>(st + lb) + t;
    r.slotv = reinterpret_cast<uint32_t *>(st + lb + 4u * coded_words(C) * T) + t;
    r.T = T;
    return r;
}

// Delay of a component through its location's descriptor (the general
// path of race_exact).
static __device__ __forceinline__ float desc_delay(const Net &n, const CodedView &rv, uint32_t li, uint32_t x) {
    const uint64_t dsc = n.loc_desc[li];
    const uint32_t lo = static_cast<uint32_t>(dsc), fl = static_cast<uint32_t>(dsc >> 32);
    if (fl & CSMC_DESC_ZERO) return 0.0f;
    float d;
    if ((fl & CSMC_DESC_INV1) && inv1_uniform(n, rv.vars, li, x, d)) return d;
    if ((fl & (CSMC_DESC_INV | CSMC_DESC_EVAL)) && !(fl & CSMC_DESC_INV1))
        return bounded_delay(n.base, rv.vars, rv.rates, li, x);
    const float inv = (fl & CSMC_DESC_PROG) ? rv.rates[lo] : __uint_as_float(lo);
    return exp_delay(x, inv);
}

// The address of member k's key: chain k of the class in byte k of wd.
template <uint32_t k>
static __device__ __forceinline__ uint32_t key_addr(const CodedView &rv, uint32_t wd) {
    static_assert(kKeyClass == 2048u, "the code field moves from bit 8k + 5 to bit 11");
    const uint32_t f = wd & (0xe0u << (8u * k));
    return rv.keys + (k == 0 ? f << 6 : f >> (8u * k - 6u));
}

// The members of a location word whose delay goes through its descriptor
// (code 7; padding has 6): bit 8k + 7 for member k.
static __device__ __forceinline__ uint32_t general_members(uint32_t wd) {
    static_assert(kCodeGeneral == 7u && kCodePad == 6u, "bits 7 and 5 of a byte");
    return wd & (wd << 2) & 0x80808080u;
}

// The four members of Philox block q.  cb: 255 minus the bit-reversed q, the
// low byte of their keys.  ALLCLS: all of them class members; else the bytes
// of the others are zero in wd and their bits set in out (bit 8k + 7 for
// member k): they leave class 0's key as it is.
template <bool ALLCLS>
static __device__ __forceinline__ void race_block(const CodedView &rv, uint32_t wd, uint32_t out, const u32x4 &x,
                                                  uint32_t cb) {
    const uint32_t a0 = key_addr<0>(rv, wd), a1 = key_addr<1>(rv, wd), a2 = key_addr<2>(rv, wd),
                   a3 = key_addr<3>(rv, wd);
    const uint32_t o0 = ld_key(a0), o1 = ld_key(a1 + kKeyChain), o2 = ld_key(a2 + 2u * kKeyChain),
                   o3 = ld_key(a3 + 3u * kKeyChain);
    const auto key = [&](uint32_t w, uint32_t k) {
        return ALLCLS || !(out & (0x80u << (8u * k))) ? (w & 0xffffff00u) | cb : 0u;
    };
    st_key(a0, max(o0, key(x.x, 0u)));
    st_key(a1 + kKeyChain, max(o1, key(x.y, 1u)));
    st_key(a2 + 2u * kKeyChain, max(o2, key(x.z, 2u)));
    st_key(a3 + 3u * kKeyChain, max(o3, key(x.w, 3u)));
}

// The last block of a network of 4 Q + m components, m = 1 .. 3 (all lanes
// alike), all of them class members: a0, a1, a2 are the members' key addresses.
static __device__ __forceinline__ void race_tail(uint32_t m, uint32_t a0, uint32_t a1, uint32_t a2, const u32x4 &x,
                                                 uint32_t cb) {
    st_key(a0, max(ld_key(a0), (x.x & 0xffffff00u) | cb));
    if (m > 1u) st_key(a1, max(ld_key(a1), (x.y & 0xffffff00u) | cb));
    if (m > 2u) st_key(a2, max(ld_key(a2), (x.z & 0xffffff00u) | cb));
}

// race_exact out of line: the view of the network is rebuilt, the run state's
// view passed by value.
struct RaceOutcome {
    unsigned long long best;
    float d;
};
static __device__ __noinline__ RaceOutcome coded_race_exact(const uint8_t *base, CodedView rv, uint64_t seed,
                                                            uint64_t run, uint32_t step) {
    const Net n = net_view(base);
    RaceOutcome r;
    race_exact(n, n.n_comps, ceil_log2(n.n_comps), rv, SeedBlocks{seed, run, step}, r.best, r.d);
    return r;
}

// The race decided from the class keys (race_classes' decision over the
// same keys); false: the caller runs race_exact.  src: each class's 1/rate
// source (CSMC_CLASS_SRC_PROG | slot, or float bits).  ALLCLS: every
// location is classed, so no block has a general member; the padding of a last
// block of one to three components is left out there.
template <bool ALLCLS>
static __device__ __forceinline__ bool race_coded(const Net &n, uint32_t C, uint32_t bits, uint32_t NG,
                                                  const CodedView &rv, const PhiloxKeys &K, const uint32_t *src,
                                                  uint64_t run, uint32_t step, unsigned long long &best,
                                                  float &bestd) {
    const uint32_t T = rv.T;
    for (uint32_t g = 0; g < NG; ++g)
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) st_key(rv.keys + g * kKeyClass + k * kKeyChain, 0u);
    best = ~0ull;
    bestd = 0.0f;
    const PhiloxStep ps = philox_step(K, step, run);
    // bit reversal of component 4q + k over `bits` (>= 2) bits: the two low
    // bits (k) become the top two, q the low bits - 2 reversed
    const uint32_t hi_shift = bits - 2u;  // bits >= 2: the plan needs at least four components
    const uint32_t Q = ALLCLS ? C >> 2 : (C + 3u) >> 2;
    // members outside the classes: the blocks that have some, their draws
    uint64_t general_blocks = 0;
    uint32_t n_general = 0, draws[ALLCLS ? 1 : kMaxCodedComps];
#pragma unroll kCodedUnroll
    for (uint32_t q = 0; q < Q; ++q) {
        const uint32_t wd = rv.lw[q * T];
        const u32x4 blk = philox_block(K, ps, q);
        const uint32_t cb = 255u - (hi_shift ? (__brev(q) >> (32u - hi_shift)) : 0u);
        const uint32_t out = ALLCLS ? 0u : wd & 0x80808080u;
        race_block<ALLCLS>(rv, ALLCLS ? wd : wd & ~((out >> 7) * 0xffu), out, blk, cb);
        if (!ALLCLS) {
            const uint32_t general = general_members(wd);
            if (general) {
                general_blocks |= 1ull << q;
                if (general & 0x80u) draws[n_general++] = blk.x;
                if (general & 0x8000u) draws[n_general++] = blk.y;
                if (general & 0x800000u) draws[n_general++] = blk.z;
                if (general & 0x80000000u) draws[n_general++] = blk.w;
            }
        }
    }
    if (ALLCLS && (C & 3u)) {
        const uint32_t wd = rv.lw[Q * T];
        const u32x4 blk = philox_block(K, ps, Q);
        race_tail(C & 3u, key_addr<0>(rv, wd), key_addr<1>(rv, wd) + kKeyChain, key_addr<2>(rv, wd) + 2u * kKeyChain, blk,
                  255u - (__brev(Q) >> (32u - hi_shift)));
    }
    // their delays, one member of each run at a time: a warp goes through as
    // many as its run with the most has, not through every component that is
    // outside the classes in one of its runs
    if (!ALLCLS && n_general) {
        uint32_t q = 0, wd = 0, general = 0;
        for (uint32_t i = 0; i < n_general; ++i) {
            if (!general) {
                q = static_cast<uint32_t>(__ffsll(static_cast<long long>(general_blocks))) - 1u;
                general_blocks &= general_blocks - 1u;
                wd = rv.lw[q * T];
                general = general_members(wd);
            }
            const uint32_t m = (static_cast<uint32_t>(__ffs(static_cast<int>(general))) >> 3) - 1u, c = 4u * q + m;
            general &= general - 1u;
            const float d = desc_delay(n, rv, n.comp[c].loc_begin + ((wd >> (8u * m)) & 31u), draws[i]);
            const unsigned long long key =
                (static_cast<unsigned long long>(delay_key(d)) << 32) | bitrev_bits(c, bits);
            if (key < best) {
                best = key;
                bestd = d;
            }
        }
    }
    // each class races with its largest key
    uint32_t inf_classes = 0, wtop = 0;
    float winv = 0.0f;
    bool tie = false, from_class = false;
#pragma unroll
    for (uint32_t g = 0; g < CSMC_RACE_CLASSES; ++g) {
        if (g >= NG) continue;
        const uint32_t kg = rv.keys + g * kKeyClass;
        const uint32_t o0 = ld_key(kg), o1 = ld_key(kg + kKeyChain), o2 = ld_key(kg + 2u * kKeyChain),
                       o3 = ld_key(kg + 3u * kKeyChain);
        // no chain key is 0 (its low byte is 255 minus at most 63)
        if ((o0 | o1 | o2 | o3) == 0u) continue;
        const uint32_t a = max(max(o0, o1 ? o1 - (2u << hi_shift) : 0u),
                               max(o2 ? o2 - (1u << hi_shift) : 0u, o3 ? o3 - (3u << hi_shift) : 0u));
        const uint32_t sg = src[g];
        const float inv = (sg & CSMC_CLASS_SRC_PROG) ? rv.rates[sg & 0xffffu] : __uint_as_float(sg);
        if (!(inv > 0.0f)) return false;  // delays 0, negative or NaN for the whole class
        if (!(inv <= 3.40282347e38f)) {   // +inf: the class's delays are +inf (NaN at u = 1)
            inf_classes |= 1u << g;
            continue;
        }
        const float d1 = exp_delay(a & 0xffffff00u, inv);
        const unsigned long long key =
            (static_cast<unsigned long long>(f_bits(d1) | 0x80000000u) << 32) | (255u - (a & 255u));  // d1 >= 0
        tie |= static_cast<uint32_t>(key >> 32) == static_cast<uint32_t>(best >> 32);
        if (key < best) {
            tie = static_cast<uint32_t>(key >> 32) == static_cast<uint32_t>(best >> 32);
            best = key;
            bestd = d1;
            wtop = a >> 8;
            winv = inv;
            from_class = true;
        }
    }
    // a class can hide a tie (a lower draw of a member with a smaller index
    // that rounds to the same delay) only when its delay is the race's
    // minimum and its largest draw sits on a flat spot of the delay; the
    // exact race decides those steps, and those in which two delays tie
    if (tie) return false;
    if (from_class && wtop > 0u && exp_delay((wtop - 1u) << 8, winv) == bestd) return false;
    if (inf_classes && static_cast<uint32_t>(best >> 32) >= delay_key(__uint_as_float(0x7f800000u))) return false;
    return true;
}

#ifndef CSMC_CODED_MIN_CTAS_PER_SM
#define CSMC_CODED_MIN_CTAS_PER_SM 4
#endif

template <bool VERIFY, bool SLOTS, bool ALLCLS>
__global__ void __launch_bounds__(128, CSMC_CODED_MIN_CTAS_PER_SM) coded_kernel(const __grid_constant__ SimParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    stage_network(smem, p.blob, p.blob_bytes);
    const uint32_t C = p.net.n_comps, V = p.net.n_vars, P = p.net.n_rate_prog;
    const uint32_t T = blockDim.x, t = threadIdx.x;
    const bool recv = (p.net.recv_lo | p.net.recv_hi) != 0;
    const CodedView rv = carve_coded_view(smem + p.blob_bytes, V, P, C, p.net.n_classes * kKeyClass, recv, T, t);
    // padding bytes of the last location word never change
    if (C & 3u) rv.lw[(C >> 2) * T] = kCodePad * 0x20202020u;  // 0xc0 in every byte
    __syncthreads();
    const Net n = net_view(smem, p.net);
    const bool rate_table = (p.net.flags & CSMC_NET_RATE_TABLE) && P > 0;
    const bool rate_every_step = !(p.net.flags & CSMC_NET_RATE_NO_CLOCK);
    const uint32_t bits = ceil_log2(C);
    const uint32_t NG = p.net.n_classes;  // classes in use: only these keys are kept

    const uint32_t lane = threadIdx.x & 31u;
    unsigned long long acc_hits = 0, acc_steps = 0, acc_capped = 0;

    bool have = false, drained = false;
    unsigned long long ridx = 0;
    uint64_t run = 0;
    float time = 0.0f;
    uint32_t step = 0;
    bool dirty = true;  // variables changed since the rate table was evaluated
    RunScalars sc{0.0, 0.0, 0, 0, -1, 0, 0};

    for (;;) {
        // all lanes meet here, so that a warp's runs advance in one stream
        // however their branches differed in the last step; the warp goes on
        // until its last run has ended
        __syncwarp();
        // ---- refill finished lanes from the work counter
        const bool need = !have && !drained;
        const unsigned want = __ballot_sync(0xffffffffu, need);
        if (want) {
            const int leader = __ffs(want) - 1;
            unsigned long long base = 0;
            if (static_cast<int>(lane) == leader)
                base = atomicAdd(p.scratch, static_cast<unsigned long long>(__popc(want)));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (need) {
                ridx = base + __popc(want & ((1u << lane) - 1u));
                if (ridx >= p.n_runs) {
                    drained = true;
                } else {
                    have = true;
                    run = p.first_run + ridx;
                    run_init<SLOTS>(n, C, V, rv, sc, p.var_id);
                    time = 0.0f;
                    step = 0;
                    dirty = true;
                }
            }
            if (__all_sync(0xffffffffu, drained)) break;
        }
        if (!have) continue;

        // ---- end of run (simulation.cu:835-849, 887-893)
        const RunEnd e = run_end(sc, time, p.horizon, step, p.max_steps, p.loc_mode, p.is_max, p.threshold);
        if (e.done) {
            if (p.flags) p.flags[ridx] = static_cast<uint8_t>(e.flag);
            if (p.values) p.values[ridx] = e.value;
            if (p.steps) p.steps[ridx] = step;
            if (VERIFY) {
                if (p.digests) p.digests[ridx] = sc.digest;
                if (p.final_state) run_final_state(n, C, V, rv, p.final_state + ridx * (C + V));
            }
            acc_hits += e.flag;
            acc_steps += step;
            acc_capped += e.capped;
            have = false;
            continue;
        }

        // ---- one step: receivers, rate table, race, commit
        if (run_receivers<VERIFY, SLOTS>(n, C, V, rv, sc, p.seed, p.var_id, run, step)) dirty = true;
        if (rate_table && (dirty || rate_every_step)) {
            for (uint32_t j = 0; j < P; ++j) rv.rates[j] = inv_rate(eval(n, rv.vars, n.rate_prog[j]));
            dirty = false;
        }
        unsigned long long best;
        float bestd;
        if (!race_coded<ALLCLS>(n, C, bits, NG, rv, p.keys, p.class_src, run, step, best, bestd)) {
            const RaceOutcome r = coded_race_exact(n.base, rv, p.seed, run, step);
            best = r.best;
            bestd = r.d;
        }
        const uint32_t win = bitrev_bits(static_cast<uint32_t>(best & 0xffffffffull), bits);
        if (run_commit<VERIFY, SLOTS>(n, p.net.n_clocks, rv, sc, p.seed, p.var_id, run, step, time, win, bestd))
            dirty = true;
    }
    if (acc_hits) atomicAdd(p.scratch + 1, acc_hits);
    if (acc_steps) atomicAdd(p.scratch + 2, acc_steps);
    if (acc_capped) atomicAdd(p.scratch + 3, acc_capped);
}

}  // namespace detail

template <bool VERIFY, bool SLOTS, bool ALLCLS>
int coded_launch_one(const SimParams &p, int grid, int block, size_t smem, void *stream) {
    auto fn = detail::coded_kernel<VERIFY, SLOTS, ALLCLS>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    fn<<<grid, block, smem, static_cast<cudaStream_t>(stream)>>>(p);
    return static_cast<int>(cudaGetLastError());
}

template <bool VERIFY, bool SLOTS, bool ALLCLS>
int coded_occupancy_one(int block, size_t smem, int *ctas) {
    auto fn = detail::coded_kernel<VERIFY, SLOTS, ALLCLS>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return static_cast<int>(e);
    return static_cast<int>(cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, fn, block, smem));
}

}  // namespace csmc
