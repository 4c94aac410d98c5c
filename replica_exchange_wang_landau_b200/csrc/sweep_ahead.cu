// sweep_ahead.cu — the dense REWL sweep: WangLandauWalker::run_attempts / attempt_flip
// (src/wang_landau.cpp:244-315) for one batch of exchange_interval attempts, then the
// walker-local flatness / 1/t check of run_rewl (src/parallel.cpp:395-407).
//
// What bounds it: a walker is one dependent chain (field of the drawn site -> proposed energy ->
// bin -> log g -> decision -> field of the next site), about 110 cycles of latencies per attempt
// that nothing inside the walker can overlap.  So one warp does the chain and nothing else, and
// everything that does not decide an attempt is done beside it by other warps of the CTA:
//
// * Draws do not depend on the walk.  They are taken in blocks of kStep = 30: lane j of the
//   walker warp holds the local field of the site that draw 30 b + j would select (the lanes 30
//   and 31 are the next block's first two draws, so that the two candidates of an attempt's
//   successor -- the next draw, or the one after it when the attempt consumes its acceptance
//   uniform -- are always in a lane).  An accepted flip is then ONE fma per lane with J between
//   the flipped site and the lane's site, instead of an update of all N fields; the other
//   fields are not needed until a later block draws their sites.
// * warp 1 (draws): generates the draws, their sites and log u, up to `slots` block records ahead.
// * warps 3 and 4 (pairs): gather, ahead of the walker, the couplings between the block's own sites
//   (what an accepted flip adds to the lanes) and between its sites and the next block's.
// * warp 2 (look-ahead): while the walker is in block b it builds the lanes of block b + 1: their
//   fields as of the end of block b - 1, then, following the walker's published decisions, the
//   flips of block b in order, one fma each.  At the walker's last decision of the block it hands
//   the lanes over.
// * the remaining warps (fields): after a block, apply its accepted flips to all N fields in
//   shared memory, each field its flips in order, the J rows read coalesced from L2 with eight
//   rows in flight; they have the whole next block's time for it.
//
// Bit-exactness: every field receives the reference's updates in the reference's order, each
// rounded once (fma(m, J, h) with m = +-2 rounds the real number h + m J, as the reference's
// multiply and add do, because m J is exact); a rejected flip's update is skipped or made with
// m = 0, which changes no field (a field is never -0.0: sums start at +0.0 and a sum that
// reaches zero is +0.0).  E + (-2s)h is evaluated as fma(m, h, E), equal for the same reason;
// with a power-of-two bin width (E' - min) / width as fma(E', 1/width, -min/width), equal because
// scaling by a power of two is exact and commutes with rounding.  log(max(u, 2^-53)) < log_ratio
// uses the CUDA log.  BF16 couplings carry a row scale s: m s b is exact in FP64, so tables of s b
// give the same sums.
//
// All waits are bounded: on timeout the walker records WLG_ERR_TIMEOUT, every role leaves and no
// state is written back.
#include "engine.hpp"
#include "walker_dev.cuh"

namespace wlg {

namespace {

constexpr int kStep = 30;             // draws per block
constexpr int kMinSlots = 4;          // block records: the walker's, the next one, two ahead of it
constexpr int kMaxSlots = 6;
constexpr int kOwnTables = 3;         // tables of a block's own pairs: the walker's, the next one, one being made
constexpr int kNextTables = 3;        // tables of the pairs with the next block
constexpr uint32_t kPolls = 1u << 22; // bound of every wait (a poll takes about 40 cycles)
constexpr int kRoleWarps = 5;         // walker, draws, look-ahead, two pairs warps
constexpr int kMaxFieldWarps = 8;
constexpr int kMaxRoles = kRoleWarps + kMaxFieldWarps;

// The role of a CTA's warp.  With the SM to itself (kAlone) the walker also gets a scheduler to
// itself: warps 4, 8 and 12, which the SM would run on the walker's scheduler, stay idle (the
// gathers' scattered loads in the walker's load queue cost it 256 -> 316 cycles per attempt).
template <bool kAlone>
__device__ __forceinline__ int role_of(int warp) {
    if constexpr (!kAlone) return warp;
    return warp == 0 ? 0 : (warp & 3) == 0 ? kMaxRoles : warp - (warp >> 2);
}
__host__ __device__ constexpr int warps_for(int roles, bool alone) { return alone ? roles + (roles - 2) / 3 : roles; }

// named barriers between the look-ahead warp and the field warps (0 is __syncthreads)
constexpr int kBarList = 1, kBarFields = 2;

// ent[] entry of one attempt: the high word of m for an accepted flip (0x40000000 / 0xC0000000)
// or 0, plus
constexpr uint32_t kEntValid = 1u;    // written
constexpr uint32_t kEntUniform = 2u;  // the attempt consumed its acceptance uniform
constexpr uint32_t kEntStop = 4u;     // no attempt: the batch has ended (or failed)

struct alignas(16) BinRecord {  // one bin of the walker's window
    double log_g;
    uint32_t visits;  // of this batch
    uint32_t active;
};
struct alignas(16) FlipRecord {  // one accepted flip of a block, for the field warps
    double m;         // -2 * old spin (times the BF16 row scale)
    uint64_t row;     // byte offset of the site's J row
};

struct SlotLayout {  // one block record
    size_t lnu, scale, site, same, misc, total;
};
__host__ __device__ inline SlotLayout slot_layout(bool scaled) {
    SlotLayout L;
    size_t at = 0;
    L.lnu = at; at += 32 * 8;             // log(max(u, 2^-53)) of each draw
    L.scale = at; at += scaled ? 32 * 8 : 0;
    L.site = at; at += 32 * 4;            // -1: bounded() rejects the draw
    L.same = at; at += 32 * 4;            // lanes that drew the same site
    L.misc = at; at += 48;                // rng[4] at the block's first draw, rejected-draw mask
    L.total = at;
    return L;
}
constexpr size_t kTable = kStep * 32 * 8;
struct AheadLayout {
    size_t slots, own_pairs, next_pairs, cross, flips, hand, factors, ent, ctl, fields, bins, spins, total;
};
__host__ __device__ inline AheadLayout ahead_layout(int ld, int mwb, bool scaled, int slots) {
    AheadLayout L;
    size_t at = 0;
    L.slots = at; at += static_cast<size_t>(slots) * slot_layout(scaled).total;
    L.own_pairs = at; at += kOwnTables * kTable;    // J[site of draw k][site of lane j]
    L.next_pairs = at; at += kNextTables * kTable;  // J[site of draw k][site of the next block's lane j]
    L.cross = at; at += kNextTables * 32 * 4;       // lanes of the next block that drew the site of draw k
    L.flips = at; at += 2 * 32 * sizeof(FlipRecord);
    L.hand = at; at += 2 * 32 * 8 + 16;             // handed lanes: fields, then their spin masks
    L.factors = at; at += 32 * 8;                   // 1/t stage: what the next 32 attempts add to log g
    L.ent = at; at += 2 * 32 * 4;
    L.ctl = at; at += 64;
    L.fields = at; at += static_cast<size_t>(ld) * 8;
    L.bins = at; at += (static_cast<size_t>(mwb) + 1) * sizeof(BinRecord);
    L.spins = at; at += round16(static_cast<size_t>(ld));
    L.total = at;
    return L;
}
// words of ctl
constexpr int kProduced = 0;  // block records published by the draws warp
constexpr int kHanded = 1;    // blocks whose lanes the walker may take over
constexpr int kAheadIn = 2;   // block the look-ahead warp follows
constexpr int kWalkerIn = 3;  // block the walker is in
constexpr int kStop = 4;      // the walker has ended its batch
constexpr int kFail = 5;      // a bounded wait gave up
constexpr int kFinal = 6;     // the flips handed to the field warps are the batch's last
constexpr int kCount = 8;     // [8], [9]: flips of the two flip lists
constexpr int kOwnMade = 10;  // blocks whose own pairs are gathered
constexpr int kNextMade = 11; // blocks whose pairs with the next block are gathered

__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) { *reinterpret_cast<volatile uint32_t*>(p) = v; }
__device__ __forceinline__ void st_release(uint32_t* p, uint32_t v) {
    __threadfence_block();
    st_relaxed(p, v);
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
// Warp-uniform bounded wait until *p >= want (wrap-safe).  0: reached, 1: *stop became nonzero
// first, 2: gave up.
__device__ __forceinline__ int wait_at_least(const uint32_t* p, uint32_t want, const uint32_t* stop) {
    for (uint32_t k = 0; k < kPolls; ++k) {
        const bool there = static_cast<int32_t>(ld_relaxed(p) - want) >= 0;
        if (__all_sync(kFull, there)) {
            __threadfence_block();
            return 0;
        }
        if (stop && __all_sync(kFull, ld_relaxed(stop) != 0)) {
            __threadfence_block();
            return 1;
        }
    }
    return 2;
}

template <int kPrec> struct Stored;
template <> struct Stored<WLG_PRECISION_FP64> { using T = double; };
template <> struct Stored<WLG_PRECISION_FP32> { using T = float; };
template <> struct Stored<WLG_PRECISION_BF16> { using T = __nv_bfloat16; };

template <int kPrec>
__device__ __forceinline__ const typename Stored<kPrec>::T* coupling_rows(const EngineView& v) {
    if constexpr (kPrec == WLG_PRECISION_FP64) return v.J64;
    else if constexpr (kPrec == WLG_PRECISION_FP32) return v.J32;
    else return v.J16;
}
// One coupling and the pair (2c, 2c + 1) of a row in global memory, widened exactly.
template <int kPrec>
__device__ __forceinline__ double coupling_one(const typename Stored<kPrec>::T* p) {
    if constexpr (kPrec == WLG_PRECISION_FP64) return __ldg(p);
    else if constexpr (kPrec == WLG_PRECISION_FP32) return static_cast<double>(__ldg(p));
    else return static_cast<double>(__bfloat162float(*p));
}
template <int kPrec> struct Pair;
template <> struct Pair<WLG_PRECISION_FP64> { using T = double2; };
template <> struct Pair<WLG_PRECISION_FP32> { using T = float2; };
template <> struct Pair<WLG_PRECISION_BF16> { using T = uint32_t; };
template <int kPrec>
__device__ __forceinline__ double2 widen(typename Pair<kPrec>::T p) {
    if constexpr (kPrec == WLG_PRECISION_FP64) return p;
    else if constexpr (kPrec == WLG_PRECISION_FP32) return make_double2(p.x, p.y);
    else  // BF16: element 2c in the low half of the word, 2c + 1 in the high half
        return make_double2(static_cast<double>(__uint_as_float(p << 16)),
                            static_cast<double>(__uint_as_float(p & 0xffff0000u)));
}

// The flips list[0..kRows) on one pair of fields, in order, all rows loaded before the first is used.
template <int kPrec, int kRows>
__device__ __forceinline__ void apply_rows(const char* column, const FlipRecord* list, double2& h) {
    using PairT = typename Pair<kPrec>::T;
    PairT x[kRows];
#pragma unroll
    for (int u = 0; u < kRows; ++u) x[u] = __ldg(reinterpret_cast<const PairT*>(column + list[u].row));
#pragma unroll
    for (int u = 0; u < kRows; ++u) {
        const double m = list[u].m;
        const double2 y = widen<kPrec>(x[u]);
        h.x = fma(m, y.x, h.x);
        h.y = fma(m, y.y, h.y);
    }
}

// Starts the copy of J between the sites of the block's draws 0..29 and this lane's column to `out`
// (row k at 32 k); with `upper` only what lies above the diagonal.  FP64 couplings go from L2 to
// shared memory without passing registers (cp.async, one group per call), so that the next block's
// gather runs while this one's is in flight: a gather's 30 scattered loads take 840 cycles that way,
// 1940 as two batches of loads waited for.  The narrow forms are widened on the way (exactly; BF16
// times its row scale) and are complete when the call returns.
template <int kPrec>
__device__ __forceinline__ void gather_pairs(const typename Stored<kPrec>::T* J, int ld, int my_row, double my_scale,
                                             int column, bool upper, double* out, int lane) {
    if constexpr (kPrec == WLG_PRECISION_FP64) {
        const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(out + lane));
#pragma unroll 6
        for (int k = 0; k < kStep; ++k) {
            const int row = __shfl_sync(kFull, my_row, k);
            const double* from = J + static_cast<size_t>(row) * ld + column;
            if (!upper || lane > k)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + 256u * k), "l"(from) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    } else {
#pragma unroll 1
        for (int k0 = 0; k0 < kStep; k0 += 15) {
            double x[15];
#pragma unroll
            for (int u = 0; u < 15; ++u) {
                const int row = __shfl_sync(kFull, my_row, k0 + u);
                x[u] = 0.0;
                if (!upper || lane > k0 + u) x[u] = coupling_one<kPrec>(J + static_cast<size_t>(row) * ld + column);
            }
#pragma unroll
            for (int u = 0; u < 15; ++u) {
                double y = x[u];
                if constexpr (kPrec == WLG_PRECISION_BF16) y *= __shfl_sync(kFull, my_scale, k0 + u);
                out[(k0 + u) * 32 + lane] = y;
            }
        }
    }
}

template <int kPrec, bool kPow2, bool kAlone>
__global__ void __launch_bounds__(32 * warps_for(kAlone ? kMaxRoles : kMaxRoles - 1, kAlone), kAlone ? 1 : 2) sweep_ahead_kernel(EngineView v, WalkArgs a,
                                                                                                        int slots, int field_warps) {
    using JT = typename Stored<kPrec>::T;
    constexpr bool kScaled = kPrec == WLG_PRECISION_BF16;
    extern __shared__ __align__(128) unsigned char smem[];
    // The role's warp index through a shuffle, so that the compiler knows the roles' branches to be
    // warp-uniform: the attempt loop then runs on the uniform datapath without reconvergence
    // instructions (292 -> 195 cycles per attempt for the loop alone, 185 with two attempts per trip).
    const int role = role_of<kAlone>(__shfl_sync(kFull, static_cast<int>(threadIdx.x >> 5), 0)), lane = threadIdx.x & 31;
    if (static_cast<int>(blockIdx.x) >= a.count) return;
    const int w = a.first + static_cast<int>(blockIdx.x);
    Control* ctl = v.ctl;
    // one answer for the whole CTA: another walker's error may set the flag meanwhile
    if (__syncthreads_or(a.epoch_mode && *reinterpret_cast<volatile int32_t*>(&ctl->done))) return;

    const int ld = v.ld;
    const SlotLayout SL = slot_layout(kScaled);
    const AheadLayout L = ahead_layout(ld, v.max_window_bins, kScaled, slots);
    FlipRecord* flips = reinterpret_cast<FlipRecord*>(smem + L.flips);
    double* hand_fields = reinterpret_cast<double*>(smem + L.hand);
    uint32_t* hand_masks = reinterpret_cast<uint32_t*>(smem + L.hand + 2 * 32 * 8);
    double* factors = reinterpret_cast<double*>(smem + L.factors);
    uint32_t* ent = reinterpret_cast<uint32_t*>(smem + L.ent);
    uint32_t* word = reinterpret_cast<uint32_t*>(smem + L.ctl);
    double* f_s = reinterpret_cast<double*>(smem + L.fields);
    BinRecord* bins = reinterpret_cast<BinRecord*>(smem + L.bins);
    int8_t* sp_s = reinterpret_cast<int8_t*>(smem + L.spins);

    // the walker's scalars are read where they are used (by one role each), so that no role holds them all
    const WalkerState* ws = v.ws + w;
    const int wb = v.win_begin[ws->window], nbins = v.win_end[ws->window] - wb;
    if (ws->cur_bin < wb || ws->cur_bin >= wb + nbins) {  // "Walker escaped its energy window"
        if (threadIdx.x == 0) record_error(ctl, WLG_ERR_ESCAPED, w);
        return;
    }
    const DeviceParams& P = v.p;
    uint32_t batch;
    {
        uint64_t b = a.fixed_batch ? a.fixed_batch : P.exchange_interval;
        if (!a.fixed_batch && P.max_attempts) {
            const uint64_t remaining = ws->attempted < P.max_attempts ? P.max_attempts - ws->attempted : 0;
            b = remaining < b ? remaining : b;
        }
        batch = static_cast<uint32_t>(b < 0xffffffffULL ? b : 0xffffffffULL);
    }
    const size_t boff = static_cast<size_t>(w) * static_cast<size_t>(v.grid.count) + static_cast<size_t>(wb);
    double* fg = v.fields + static_cast<size_t>(ws->slot) * ld;
    int8_t* sg = v.spins + static_cast<size_t>(ws->slot) * ld;
    const JT* J = coupling_rows<kPrec>(v);

    // ---- stage the walker ------------------------------------------------------------------
    for (int k = threadIdx.x; k < (ld >> 1); k += blockDim.x)
        reinterpret_cast<double2*>(f_s)[k] = reinterpret_cast<const double2*>(fg)[k];
    for (int k = threadIdx.x; k < (ld >> 4); k += blockDim.x)
        reinterpret_cast<int4*>(sp_s)[k] = reinterpret_cast<const int4*>(sg)[k];
    for (int b = threadIdx.x; b <= nbins; b += blockDim.x) {
        BinRecord r{0.0, 0u, 1u};  // [nbins]: read for a proposal outside the window, never used
        if (b < nbins) {
            r.log_g = v.log_g[boff + b];
            r.active = v.active[boff + b] != 0 ? 1u : 0u;
        }
        bins[b] = r;
    }
    if (threadIdx.x < 64) ent[threadIdx.x] = 0;
    if (threadIdx.x < 16) word[threadIdx.x] = 0;
    __syncthreads();

    auto slot_of = [&](int s) { return smem + L.slots + static_cast<size_t>(s) * SL.total; };

    if (role == 0) {
        // ---- the walker ----------------------------------------------------------------------
        double E = ws->energy, factor = ws->factor;
        int32_t stage = ws->stage;
        uint64_t since = ws->attempted - ws->last_accepted;
        uint32_t n_acc = 0, n_forced = 0;
        uint32_t active32 = static_cast<uint32_t>(ws->active_count);  // at most the window's bins
        int cur = ws->cur_bin - wb;
        int s = 0;
        uint32_t k = 0;  // draw (lane) of the current attempt's site
        bool failed = wait_at_least(word + kOwnMade, 1, nullptr) != 0;
        const Grid g = v.grid;
        const double neg_min_scaled = -g.minimum * g.inv_width;
        // q + this, rounded toward -infinity, is 1.5 * 2^52 + (floor(q) - wb) exactly for |q| < 2^51 (unit
        // in the last place 1): the low word is the window's bin, and the high word is kBinHigh exactly
        // when 0 <= floor(q) - wb < 2^32
        const double bin_magic = 0x1.8p52 - static_cast<double>(wb);
        constexpr int kBinHigh = 0x43380000;
        const uint32_t last_bin = static_cast<uint32_t>(static_cast<int>(g.count) - 1 - wb);  // E == maximum
        uint32_t b = 0;
        uint32_t own = 0;  // the block's table of its own pairs
        // (set from the shared-memory base here, never null: the compiler then knows the address space)
        const double* pair_rows = reinterpret_cast<const double*>(smem + L.own_pairs);
        const double* lnus = reinterpret_cast<const double*>(smem + L.slots + SL.lnu);
        const uint32_t* sames = reinterpret_cast<const uint32_t*>(smem + L.slots + SL.same);
        uint32_t* e_s = ent;
        uint32_t rejected = 0;
        auto enter = [&]() {  // the record of block b
            const unsigned char* rec = slot_of(s);
            pair_rows = reinterpret_cast<const double*>(smem + L.own_pairs + own * kTable);
            lnus = reinterpret_cast<const double*>(rec + SL.lnu);
            sames = reinterpret_cast<const uint32_t*>(rec + SL.same);
            rejected = reinterpret_cast<const uint32_t*>(rec + SL.misc)[8];
            e_s = ent + 32 * (b & 1u);
        };
        // the first draw at or after `from` that leaves the fast path: rejected by bounded(), or the
        // next block's
        auto limit = [&](uint32_t from) {
            const uint32_t r = from < 32 ? (rejected >> from) << from : 0u;
            const uint32_t at = r ? static_cast<uint32_t>(__ffs(static_cast<int>(r))) - 1u : 32u;
            return at < static_cast<uint32_t>(kStep) ? at : static_cast<uint32_t>(kStep);
        };
        double fc = 0.0, h = 0.0;  // the lane's field; the current site's
        uint32_t up = 0;           // bit j: the spin of lane j's site is up
        uint32_t klim = 0;
        int m_hi = 0;              // high word of -2 * spin of the current site
        auto sign_of = [&](uint32_t at) {
            return static_cast<int>(((up << (31u - at)) & 0x80000000u) | 0x40000000u);
        };
        if (!failed) {
            enter();
            const int site = reinterpret_cast<const int32_t*>(slot_of(0) + SL.site)[lane];
            fc = f_s[site < 0 ? 0 : site];
            up = __ballot_sync(kFull, sp_s[site < 0 ? 0 : site] > 0);
            h = __shfl_sync(kFull, fc, 0);
            m_hi = sign_of(0);
            klim = limit(0);
        }
        uint32_t t = 0;  // attempts made
        uint32_t* e_p = e_s;
        double lg_cur = bins[cur].log_g;
        uint32_t visits = 0;
        uint32_t active = bins[cur].active;  // 0 at first when an exchange brought a bin not visited before
        const uint64_t att0 = ws->attempted + ws->time_offset;
        const uint64_t force_limit = P.force_after != 0 ? P.force_after : ~0ULL;
        uint32_t acc_t = 0;  // without forced acceptance: the attempts made at the last acceptance

        // Attempts until the batch ends or, in the 1/t stage, the walker freezes.  kIT: the 1/t
        // stage; kForce: forced acceptance (force_accept_after_attempts != 0).
        auto run = [&](auto it_tag, auto force_tag) {
            constexpr bool kIT = decltype(it_tag)::value;
            constexpr bool kForce = decltype(force_tag)::value;
            // what an attempt adds to log g of its bin: ln f, or -0.0 (which changes nothing) once frozen
            const double constant = stage == kFrozen ? -0.0 : factor;
            uint32_t t0 = t;         // 1/t stage: the attempt factors[0] belongs to
            uint32_t frozen_at = 0;  // 1/t stage: the attempts made once the walker freezes, 0 = not in the table
            double quotient = factor;
            uint32_t tlim = kIT ? t : batch;
#pragma unroll 2
            while (true) {
                if (k >= klim || t >= tlim) {
                    if (t >= tlim) {
                        if (kIT && t != t0) factor = __shfl_sync(kFull, quotient, static_cast<int>(t - 1 - t0));
                        if (kIT && frozen_at != 0 && t == frozen_at) {
                            stage = kFrozen;
                            return;
                        }
                        if (t >= batch) return;
                        if constexpr (kIT) {
                            // update_inverse_time_factor (src/wang_landau.cpp:300-315) of the next 32
                            // attempts, lane j dividing for attempt j; made again when a new bin has
                            // become active
                            t0 = t;
                            quotient = active32 == 0 ? factor
                                                     : static_cast<double>(active32) /
                                                           static_cast<double>(att0 + t + static_cast<uint64_t>(lane) + 1);
                            const bool frz = quotient <= P.final_factor;
                            const uint32_t fm = __ballot_sync(kFull, frz);
                            __syncwarp();
                            factors[lane] = frz ? -0.0 : quotient;
                            __syncwarp();
                            const uint32_t steps = fm ? static_cast<uint32_t>(__ffs(static_cast<int>(fm))) : 32u;
                            frozen_at = fm ? t + steps : 0;
                            tlim = batch - t < steps ? batch : t + steps;
                            if (frozen_at > tlim) frozen_at = 0;
                        }
                    }
                    if (k >= klim) {
                        if (k >= static_cast<uint32_t>(kStep)) {  // the next block
                            ++b;
                            if (wait_at_least(word + kHanded, b, nullptr) != 0) {
                                failed = true;
                                return;
                            }
                            k -= kStep;
                            s = s + 1 == slots ? 0 : s + 1;
                            own = own + 1 == kOwnTables ? 0 : own + 1;
                            fc = hand_fields[32 * (b & 1u) + lane];
                            up = hand_masks[b & 1u];
                            enter();
                            e_p = e_s;
                            // (by every lane: a branch on the lane number anywhere in this loop costs the
                            // whole loop its uniform form, 250 -> 350 cycles per attempt)
                            st_release(word + kWalkerIn, b);
                        } else if ((rejected >> k) & 1u) {  // bounded() rejects the draw: the next one is the site
                            st_relaxed(e_p, kEntValid);
                            ++e_p;
                            ++k;
                            h = __shfl_sync(kFull, fc, static_cast<int>(k));
                            m_hi = sign_of(k);
                        }
                        klim = limit(k);
                        continue;  // the next draw may be another block's, or rejected as well
                    }
                }
                const uint32_t k1 = k + 1, k2 = k + 2;  // the candidates for the next site
                const double* row = pair_rows + 32 * k;
                const double lnu = lnus[k1];
                const double r1 = row[k1], r2 = row[k2], rl = row[lane];
                const uint32_t same = sames[k];
                const double add = kIT ? factors[t - t0] : constant;
                const double fc1 = __shfl_sync(kFull, fc, static_cast<int>(k1));
                const double fc2 = __shfl_sync(kFull, fc, static_cast<int>(k2));

                // attempt_flip (src/wang_landau.cpp:244-262)
                const double m = __hiloint2double(m_hi, 0);
                const double Ep = fma(m, h, E);
                const double q = kPow2 ? fma(Ep, g.inv_width, neg_min_scaled) : (Ep - g.minimum) / g.width;
                const double fl = __dadd_rd(q, bin_magic);
                const bool top = Ep == g.maximum;  // the grid's upper edge belongs to its last bin
                const uint32_t nb = top ? last_bin : static_cast<uint32_t>(__double2loint(fl));
                const bool in_window = nb < static_cast<uint32_t>(nbins) &&
                                       (top || (__double2hiint(fl) == kBinHigh && Ep < g.maximum));
                const uint32_t nb_read = nb < static_cast<uint32_t>(nbins) ? nb : static_cast<uint32_t>(nbins);
                const BinRecord rec = bins[nb_read];
                const double log_ratio = lg_cur - rec.log_g;
                const bool det = log_ratio >= 0.0;
                bool accepted, need_u;
                if constexpr (kForce) {
                    const bool forced = in_window && !det && since >= force_limit;
                    need_u = in_window && !det && !forced;
                    accepted = in_window && (det || forced || lnu < log_ratio);
                    n_forced += forced ? 1u : 0u;
                    since = accepted ? 0 : since + 1;
                } else {
                    need_u = in_window && !det;
                    accepted = in_window && lnu < log_ratio;  // lnu < 0, so det accepts as well
                }
                const int me_hi = accepted ? m_hi : 0;
                const double m_eff = __hiloint2double(me_hi, 0);
                h = fma(m_eff, need_u ? r2 : r1, need_u ? fc2 : fc1);
                up ^= accepted ? same : 0u;
                const uint32_t x = static_cast<uint32_t>(me_hi) | (need_u ? kEntValid | kEntUniform : kEntValid);
                k = need_u ? k2 : k1;
                m_hi = sign_of(k);
                st_relaxed(e_p, x);
                ++e_p;
                fc = fma(m_eff, rl, fc);
                E = accepted ? Ep : E;
                n_acc += accepted ? 1u : 0u;
                ++t;
                if constexpr (!kForce) acc_t = accepted ? t : acc_t;
                // update_current_bin (src/wang_landau.cpp:277-278)
                cur = accepted ? static_cast<int>(nb) : cur;
                lg_cur = (accepted ? rec.log_g : lg_cur) + add;
                visits = (accepted ? rec.visits : visits) + 1u;
                const bool opened = (accepted ? rec.active : active) == 0;
                active = 1;
                active32 += opened ? 1u : 0u;
                if (kIT) tlim = opened ? t : tlim;
                BinRecord now;
                now.log_g = lg_cur;
                now.visits = visits;
                now.active = 1u;
                bins[cur] = now;
            }
        };
        while (!failed && t < batch) {
            if (P.force_after != 0) {
                if (stage == kInverseTime) run(std::true_type{}, std::true_type{});
                else run(std::false_type{}, std::true_type{});
            } else {
                if (stage == kInverseTime) run(std::true_type{}, std::false_type{});
                else run(std::false_type{}, std::false_type{});
            }
        }
        if (P.force_after == 0) since = n_acc ? static_cast<uint64_t>(batch - acc_t) : since + batch;
        __syncwarp();
        if (failed && lane == 0) st_relaxed(word + kFail, 1u);
        // the stop entry; a batch that ended with its block's last draw puts it into the next block's
        uint32_t* stop_at = k >= static_cast<uint32_t>(kStep) && !failed ? ent + 32 * ((b + 1) & 1u) : e_p;
        if (lane == 0) {
            st_release(word + kStop, 1u);
            st_release(stop_at, kEntValid | kEntStop);
        }
        bar_sync(0, static_cast<int>(blockDim.x));  // every role has left
        if (ld_relaxed(word + kFail) != 0) {
            if (lane == 0) record_error(ctl, WLG_ERR_TIMEOUT, w);
            return;
        }
        WalkerState st = *ws;
        // the generator after the draws consumed: the block's first state, k draws on
        {
            const uint64_t* m = reinterpret_cast<const uint64_t*>(slot_of(s) + SL.misc);
            Rng rng{m[0], m[1], m[2], m[3]};
            for (uint32_t d = 0; d < k; ++d) rng.next();
            st.rng[0] = rng.s0;
            st.rng[1] = rng.s1;
            st.rng[2] = rng.s2;
            st.rng[3] = rng.s3;
        }
        st.energy = E;
        st.factor = factor;
        st.stage = stage;
        st.attempted += batch;
        st.accepted += n_acc;
        st.forced += n_forced;
        st.last_accepted = st.attempted - since;
        st.active_count = active32;
        st.cur_bin = cur + wb;

        // write the window back: the visits of the batch are folded into H, and the check reads its sums
        uint64_t covered = 0, least = ~0ULL, total = 0;
        for (int b = lane; b < nbins; b += 32) {
            const BinRecord r = bins[b];
            const uint64_t hist = v.hist[boff + b] + r.visits;
            v.log_g[boff + b] = r.log_g;
            v.hist[boff + b] = hist;
            v.active[boff + b] = static_cast<uint8_t>(r.active);
            if (r.active) {
                covered += hist != 0 ? 1 : 0;
                least = hist < least ? hist : least;
                total += hist;
            }
        }
        if (a.epoch_mode && st.stage == kWangLandau) {
            const bool at_limit = P.max_attempts != 0 && st.attempted >= P.max_attempts;
            if (st.attempted - st.last_check >= P.check_interval || at_limit) {
                st.last_check = st.attempted;
                const HistStats hs = histogram_statistics_of(covered, least, total, st.active_count);
                st.last_flatness = P.inverse_time ? hs.coverage : hs.min_over_mean;
                if (stats_ready(hs, st.stage, P)) warp_begin_next_iteration(st, v.hist + boff, nullptr, nbins, P, lane);
            }
        }
        if (lane == 0) {
            v.ws[w] = st;
            if (a.epoch_mode) {
                if (st.stage == kFrozen) atomicAdd(&ctl->frozen, 1u);
                if (P.max_attempts != 0 && st.attempted >= P.max_attempts) atomicAdd(&ctl->at_limit, 1u);
            }
        }
        return;
    }
    if (role == 1) {
        // ---- draws ---------------------------------------------------------------------------
        const FastMod fm = v.site_mod;
        Rng first{ws->rng[0], ws->rng[1], ws->rng[2], ws->rng[3]};  // before the block's first draw
        int s = 0;
        bool open = P.withhold_draws == 0;  // withheld (failure injection): the walker's wait runs out
        for (uint32_t b = 0; open; ++b) {
            if (b >= static_cast<uint32_t>(slots)) {  // the record's last readers: the walker and the look-ahead
                const uint32_t need = b - static_cast<uint32_t>(slots) + 1;
                int r = wait_at_least(word + kAheadIn, need, word + kStop);
                if (r == 0) r = wait_at_least(word + kWalkerIn, need, word + kStop);
                if (r == 2 && lane == 0) st_relaxed(word + kFail, 1u);
                if (r != 0) break;
            } else if (__all_sync(kFull, ld_relaxed(word + kStop) != 0)) {
                break;
            }
            unsigned char* rec = slot_of(s);
            Rng rng = first;
            // every lane steps through the block and keeps s1 at its own draw: a draw's value is a
            // function of s1 alone, evaluated once per lane after the loop
            Rng own = rng, next = rng;
#pragma unroll 4
            for (int j = 0; j < 32; ++j) {
                if (j == kStep) next = rng;
                own.s1 = lane == j ? rng.s1 : own.s1;
                rng.next();
            }
            const uint64_t mine = own.next();
            const int site = mine < fm.threshold ? -1 : static_cast<int>(fast_mod(fm, mine));
            if constexpr (kScaled)
                reinterpret_cast<double*>(rec + SL.scale)[lane] = static_cast<double>(v.Jscale[site < 0 ? 0 : site]);
            const uint32_t rejected = __ballot_sync(kFull, site < 0);
            reinterpret_cast<int32_t*>(rec + SL.site)[lane] = site;
            reinterpret_cast<uint32_t*>(rec + SL.same)[lane] = __match_any_sync(kFull, site);
            if (lane == 0) {
                uint64_t* m = reinterpret_cast<uint64_t*>(rec + SL.misc);
                m[0] = first.s0;
                m[1] = first.s1;
                m[2] = first.s2;
                m[3] = first.s3;
                reinterpret_cast<uint32_t*>(m + 4)[0] = rejected;
            }
            reinterpret_cast<double*>(rec + SL.lnu)[lane] = log(fmax(to_uniform(mine), 0x1.0p-53));
            first = next;
            __syncwarp();
            if (lane == 0) st_release(word + kProduced, b + 1);
            s = s + 1 == slots ? 0 : s + 1;
        }
    } else if (role == 2) {
        // ---- look-ahead ----------------------------------------------------------------------
        const int barrier_threads = 32 + 32 * field_warps;
        int s = 0, k = 0;
        uint32_t table = 0;
        for (uint32_t b = 0;; ++b) {
            if (lane == 0) st_release(word + kAheadIn, b);
            const int s_next = s + 1 == slots ? 0 : s + 1;
            const unsigned char* rec = slot_of(s);
            const double* pairs = reinterpret_cast<const double*>(smem + L.next_pairs + table * kTable);
            const uint32_t* cross = reinterpret_cast<const uint32_t*>(smem + L.cross) + 32 * table;
            int r = wait_at_least(word + kNextMade, b + 1, word + kStop);
            if (r == 0) r = wait_at_least(word + kOwnMade, b + 2, word + kStop);
            bool gave_up = r == 2;
            int mine = 0;  // the next block's site of this lane
            if (r == 0) {
                mine = reinterpret_cast<const int32_t*>(slot_of(s_next) + SL.site)[lane];
                mine = mine < 0 ? 0 : mine;
            }
            if (b > 0) bar_sync(kBarFields, barrier_threads);  // the fields are up to block b - 1
            double f = f_s[mine];
            uint32_t up = __ballot_sync(kFull, sp_s[mine] > 0);
            uint32_t* e_s = ent + 32 * (b & 1u);
            // Follow the walker: the block's entries are read together (lane e reads entry e) and taken
            // as bit masks, and the flips found are applied four at a time, so that the four table
            // loads overlap (one flip at a time, catching up took 150 cycles a flip).
            const int k0 = k;
            int done = 0;  // entries followed
            bool stop = false;
            uint32_t acc = 0, neg = 0, uni = 0;
            uint32_t polls = 0;
            while (!gave_up && !stop && k < kStep) {
                const uint32_t x = ld_relaxed(e_s + lane);
                const uint32_t missing = __ballot_sync(kFull, x == 0);
                const int there = missing ? __ffs(static_cast<int>(missing)) - 1 : 32;
                if (there == done) {
                    gave_up = ++polls >= kPolls;
                    continue;
                }
                acc = __ballot_sync(kFull, x & 0x40000000u);
                neg = __ballot_sync(kFull, x & 0x80000000u);
                uni = __ballot_sync(kFull, x & kEntUniform);
                stop = __any_sync(kFull, x & kEntStop);  // the last entry there, never accepted
                uint32_t flipped = there < 32 ? acc & ((1u << there) - 1u) : acc;
                flipped = (flipped >> done) << done;
                while (flipped) {
                    double m[4], pair[4];
                    uint32_t same[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int e = flipped ? __ffs(static_cast<int>(flipped)) - 1 : 0;
                        const int at = k0 + e + __popc(uni & ((1u << e) - 1u));  // the entry's draw
                        const int hi = (neg >> e) & 1u ? static_cast<int>(0xC0000000u) : 0x40000000;
                        m[u] = __hiloint2double(flipped ? hi : 0, 0);
                        pair[u] = pairs[at * 32 + lane];
                        same[u] = flipped ? cross[at] : 0u;
                        flipped &= flipped - 1u;
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        f = fma(m[u], pair[u], f);
                        up ^= same[u];
                    }
                }
                done = there - (stop ? 1 : 0);
                k = k0 + done + __popc(uni & (done < 32 ? (1u << done) - 1u : kFull));
            }
            const bool last = stop || gave_up;
            const uint32_t followed = done < 32 ? (1u << done) - 1u : kFull;
            if (!last) {
                hand_fields[32 * ((b + 1) & 1u) + lane] = f;
                if (lane == 0) hand_masks[(b + 1) & 1u] = up;
                e_s[lane] = 0;  // for block b + 2
                __syncwarp();
                if (lane == 0) st_release(word + kHanded, b + 1);
            }
            // the block's flips: the field warps' list and the spins (a site's last flip sets its spin)
            acc &= followed;
            const uint32_t below = (1u << lane) - 1u;
            const bool mine_flipped = (acc >> lane) & 1u;
            const int at = k0 + lane + __popc(uni & below);
            const int site = mine_flipped ? reinterpret_cast<const int32_t*>(rec + SL.site)[at] : -1 - lane;
            const uint32_t group = __match_any_sync(kFull, site);
            if (mine_flipped) {
                const bool down = (neg >> lane) & 1u;  // m = -2 * old spin
                FlipRecord fr;
                fr.m = down ? -2.0 : 2.0;
                if constexpr (kScaled) fr.m *= reinterpret_cast<const double*>(rec + SL.scale)[at];
                fr.row = static_cast<uint64_t>(site) * static_cast<uint64_t>(ld) * sizeof(JT);
                flips[32 * (b & 1u) + __popc(acc & below)] = fr;
                if ((group >> lane) == 1u) sp_s[site] = down ? -1 : 1;
            }
            // pad with flips that change nothing (the first flip's row, m = 0) to a multiple of four
            const int flips_made = __popc(acc);
            const int first_site = __shfl_sync(kFull, site, flips_made ? __ffs(static_cast<int>(acc)) - 1 : 0);
            if (lane >= flips_made && lane < ((flips_made + 3) & ~3))
                flips[32 * (b & 1u) + lane] =
                    FlipRecord{0.0, static_cast<uint64_t>(first_site) * static_cast<uint64_t>(ld) * sizeof(JT)};
            if (lane == 0) {
                word[kCount + (b & 1u)] = static_cast<uint32_t>(flips_made);
                if (last) word[kFinal] = 1u;
                if (gave_up) st_relaxed(word + kFail, 1u);
            }
            __syncwarp();
            bar_arrive(kBarList, barrier_threads);
            if (last) break;
            k -= kStep;
            s = s_next;
            table = table + 1 == kNextTables ? 0 : table + 1;
        }
    } else if (role < kRoleWarps) {
        // ---- pairs ---------------------------------------------------------------------------
        const bool with_next = role == 4;
        uint32_t* made = word + (with_next ? kNextMade : kOwnMade);
        const uint32_t* reader = word + (with_next ? kAheadIn : kWalkerIn);  // the tables' reader
        const uint32_t tables = with_next ? kNextTables : kOwnTables, draws = with_next ? 2 : 1;
        int s = 0;
        uint32_t table = 0, published = 0;
        for (uint32_t b = 0;; ++b) {
            // the block's draws are made, and the reader has left the table's last block
            const bool now = static_cast<int32_t>(ld_relaxed(word + kProduced) - (b + draws)) >= 0 &&
                             (b < tables || static_cast<int32_t>(ld_relaxed(reader) - (b - tables + 1)) >= 0);
            if (__all_sync(kFull, now)) {
                __threadfence_block();
            } else {
                if (published < b) {  // complete what is in flight first
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) st_release(made, b);
                    published = b;
                }
                int r = wait_at_least(word + kProduced, b + draws, word + kStop);
                if (r == 0 && b >= tables) r = wait_at_least(reader, b - tables + 1, word + kStop);
                if (r == 2 && lane == 0) st_relaxed(word + kFail, 1u);
                if (r != 0) break;
            }
            const int s_next = s + 1 == slots ? 0 : s + 1;
            const int site = reinterpret_cast<const int32_t*>(slot_of(s) + SL.site)[lane];
            const double scale = kScaled ? reinterpret_cast<const double*>(slot_of(s) + SL.scale)[lane] : 1.0;
            int column = with_next ? reinterpret_cast<const int32_t*>(slot_of(s_next) + SL.site)[lane] : site;
            column = column < 0 ? 0 : column;
            double* out = reinterpret_cast<double*>(smem + (with_next ? L.next_pairs : L.own_pairs) + table * kTable);
            gather_pairs<kPrec>(J, ld, site < 0 ? 0 : site, scale, column, !with_next, out, lane);
            if (with_next) {
                uint32_t mask = 0;
#pragma unroll 6
                for (int k = 0; k < kStep; ++k) {
                    const uint32_t lanes = __ballot_sync(kFull, __shfl_sync(kFull, site, k) == column);
                    mask = lane == k ? lanes : mask;
                }
                reinterpret_cast<uint32_t*>(smem + L.cross)[32 * table + lane] = mask;
            }
            asm volatile("cp.async.wait_group 1;" ::: "memory");  // the block before
            __syncwarp();
            if (lane == 0 && published < b) st_release(made, b);
            published = b;
            s = s_next;
            table = table + 1 == tables ? 0 : table + 1;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (role < kRoleWarps + field_warps) {
        // ---- fields --------------------------------------------------------------------------
        using PairT = typename Pair<kPrec>::T;
        const int threads = 32 * field_warps;
        const int me = 32 * (role - kRoleWarps) + lane;
        const int barrier_threads = 32 + threads;
        const int pairs = ld >> 1;
        double2* f2 = reinterpret_cast<double2*>(f_s);
        for (uint32_t b = 0;; ++b) {
            bar_sync(kBarList, barrier_threads);
            const FlipRecord* list = flips + 32 * (b & 1u);
            const int n = static_cast<int>(word[kCount + (b & 1u)]);
            const bool last = word[kFinal] != 0;
            const bool write = last && ld_relaxed(word + kFail) == 0;
            double2* out = write ? reinterpret_cast<double2*>(fg) : f2;
            // eight rows in flight, then the last flips by fours (the list is padded with m = 0)
            const int groups = (n + 3) >> 2;
#pragma unroll 1
            for (int p = me; p < pairs; p += threads) {
                const char* column = reinterpret_cast<const char*>(J) + static_cast<size_t>(p) * sizeof(PairT);
                double2 h = f2[p];
                int q = 0;
#pragma unroll 1
                for (; q + 2 <= groups; q += 2) apply_rows<kPrec, 8>(column, list + 4 * q, h);
                if (q < groups) apply_rows<kPrec, 4>(column, list + 4 * q, h);
                out[p] = h;
            }
            if (last) break;
            bar_arrive(kBarFields, barrier_threads);
        }
    }

    bar_sync(0, static_cast<int>(blockDim.x));  // the walker has ended its batch and every role has left
    if (ld_relaxed(word + kFail) != 0) return;
    for (int i = static_cast<int>(threadIdx.x) - 32; i < (ld >> 4); i += static_cast<int>(blockDim.x) - 32)
        reinterpret_cast<int4*>(sg)[i] = reinterpret_cast<const int4*>(sp_s)[i];
}

using AheadFn = void (*)(EngineView, WalkArgs, int, int);

template <int kPrec, bool kPow2, bool kAlone>
AheadFn ahead_fn() {
    static bool configured = false;
    if (!configured) {
        check_cuda(cudaFuncSetAttribute(reinterpret_cast<const void*>(&sweep_ahead_kernel<kPrec, kPow2, kAlone>),
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024),
                   "cudaFuncSetAttribute");
        configured = true;
    }
    return &sweep_ahead_kernel<kPrec, kPow2, kAlone>;
}

template <int kPrec>
AheadFn pick_ahead(bool pow2, bool alone) {
    if (alone) return pow2 ? ahead_fn<kPrec, true, true>() : ahead_fn<kPrec, false, true>();
    return pow2 ? ahead_fn<kPrec, true, false>() : ahead_fn<kPrec, false, false>();
}

int sm_count() {
    static int count = 0;
    if (count == 0) {
        int device = 0;
        check_cuda(cudaGetDevice(&device), "cudaGetDevice");
        check_cuda(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    }
    return count;
}

}  // namespace

bool launch_sweep_ahead(const EngineView& v, const WalkArgs& a, cudaStream_t stream) {
    if (v.csr || v.p.collect || v.p.nalivaiko) return false;
    const bool scaled = v.precision == WLG_PRECISION_BF16;
    int slots = v.split_ring_log == 5 ? kMaxSlots : kMinSlots;
    if (ahead_layout(v.ld, v.max_window_bins, scaled, slots).total > 227 * 1024) slots = kMinSlots;
    const size_t bytes = ahead_layout(v.ld, v.max_window_bins, scaled, slots).total;
    if (bytes > 227 * 1024) return false;
    const bool pow2 = v.grid.pow2_width != 0, alone = v.walkers <= sm_count();
    AheadFn fn = v.precision == WLG_PRECISION_FP32   ? pick_ahead<WLG_PRECISION_FP32>(pow2, alone)
                 : v.precision == WLG_PRECISION_BF16 ? pick_ahead<WLG_PRECISION_BF16>(pow2, alone)
                                                     : pick_ahead<WLG_PRECISION_FP64>(pow2, alone);
    // one thread per pair of fields, up to eight warps
    const int field_warps = std::max(1, std::min(alone ? kMaxFieldWarps : kMaxFieldWarps - 1, (v.ld / 2 + 31) / 32));
    fn<<<static_cast<unsigned>(a.count), 32 * warps_for(kRoleWarps + field_warps, alone), bytes, stream>>>(
        v, a, slots, field_warps);
    check_cuda(cudaGetLastError(), "sweep_ahead_kernel");
    return true;
}

}  // namespace wlg
