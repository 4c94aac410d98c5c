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
// * the books (one warp, only with pilot statistics): follows the entries as well and keeps the squared
//   displacements, round trips and representatives on an energy and spins of its own (N = 343,
//   8 x 4 walkers: 1.69 -> 0.33 us per attempt against the ring sweep that kept them in the walker's
//   warp).
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
// Measured (8x8x8 sites, 16 x 8 walkers, FP64, an epoch of 512 attempts with its exchange): 175 us with the
// sweep that kept all fields in the walker's warp, 88 with this one and an exchange kernel, 72 with
// many epochs to a launch; 2458 sites, 32 x 8 walkers: 3.28 -> 0.97 ms per epoch of 2458 attempts.  The
// rows an accepted flip reads, 224 MB an epoch at 8x8x8, come from L2 at 2.8 TB/s.
//
// All waits are bounded: on timeout the walker records WLG_ERR_TIMEOUT and every role leaves.  A launch of
// one epoch then writes no state back.  In a launch of several, which has written fields and spins at each
// epoch's end, the run ends with that epoch: every walker that made it writes the state it has, and one that
// failed the state it had before the epoch (from what it left in its mailbox), so that a walker's
// configuration, estimates and generator always belong together, as they do after epochs launched one by one.
#include <type_traits>

#include "engine.hpp"
#include "walker_dev.cuh"

namespace wlg {

namespace {

constexpr int kStep = 30;             // draws per block
constexpr int kMinSlots = 4;          // block records: the walker's, the next one, two ahead of it
constexpr int kMaxSlots = 6;
constexpr int kOwnTables = 3;         // tables of a block's own pairs: the walker's, the next one, one being made
constexpr int kNextTables = 3;        // tables of the pairs with the next block
constexpr uint32_t kPolls = 1u << 24; // bound of every wait (a poll takes about 40 cycles)
constexpr uint32_t kSyncPolls = 1u << 24;  // of the waits across CTAs (a poll and a sleep, about 0.3 us)
constexpr int kRoleWarps = 5;         // walker, draws, look-ahead, two pairs warps
constexpr int kMaxFieldWarps = 8;
constexpr int kMaxRoles = kRoleWarps + kMaxFieldWarps;  // one more with pilot statistics

// The role of a CTA's warp.  With the SM to itself (kAlone) the walker also gets a scheduler to
// itself: warps 4, 8 and 12, which the SM would run on the walker's scheduler, stay idle (the
// gathers' scattered loads in the walker's load queue cost it 256 -> 316 cycles per attempt).
template <bool kAlone>
__device__ __forceinline__ int role_of(int warp) {
    if constexpr (!kAlone) return warp;
    return warp == 0 ? 0 : (warp & 3) == 0 ? 2 * kMaxRoles : warp - (warp >> 2);
}
__host__ __device__ constexpr int warps_for(int roles, bool alone) { return alone ? roles + (roles - 2) / 3 : roles; }

// named barriers between the look-ahead warp and the field warps (0 is __syncthreads)
constexpr int kBarList = 1, kBarFields = 2;

// The entry of one attempt: the high word of m for an accepted flip (0x40000000 / 0xC0000000) or
// 0, plus
constexpr uint32_t kEntValid = 1u;    // written
constexpr uint32_t kEntUniform = 2u;  // the attempt consumed its acceptance uniform
constexpr uint32_t kEntStop = 4u;     // no attempt: the batch has ended (or failed)
constexpr uint32_t kEntSkip = 8u;     // no attempt: the draw was rejected by bounded()

using BinRecord = FusedBin;  // one bin of the walker's window; visits: not in the histogram yet
// A block's attempts: what the walker publishes of each, and (1/t stage) what each adds to log g;
// both at eight bytes per attempt, so that one running address serves them.
struct alignas(16) Attempts {
    uint2 entry[32];  // .x; .y the bin the attempt started from (pilot statistics)
    double add[32];
    double field[32]; // local field of the attempt's site (pilot statistics)
};
constexpr int kAddWords = 64, kFieldWords = 128;  // from entry[i].x to add[i] and to field[i], in words

// What an attempt whose site is draw k needs of the draws, ahead of the couplings of its site with the
// lanes' sites: one record, two 16-byte loads.
struct alignas(16) DrawRecord {
    double lnu;       // log(max(u, 2^-53)) of draw k + 1
    double pair1;     // J[site of draw k][site of draw k + 1]
    double pair2;     // ... of draw k + 2
    uint32_t same;    // lanes that drew the site of draw k
    uint32_t pad;
    double pair[32];  // J[site of draw k][site of lane j]
};

// The same towards the next block's lanes.
struct alignas(16) NextRecord {
    uint32_t cross;   // lanes that drew the site of draw k
    uint32_t pad[3];
    double pair[32];  // J[site of draw k][site of lane j]
};

struct alignas(16) FlipRecord {  // one accepted flip of a block, for the field warps
    double m;         // -2 * old spin (times the BF16 row scale)
    uint64_t row;     // byte offset of the site's J row
};

// A lane's field handed from the look-ahead warp to the walker: each 64-bit word, which is stored
// and loaded whole, carries half of the field and the block it belongs to, so the walker needs no
// flag and no fence to know that what it reads is complete (a flag behind a fence cost the walker
// 600 cycles per block).  The 33rd record holds the spin mask.
struct alignas(16) HandWords {
    uint64_t low, high;  // (block << 32) | half
};

// words of ctl
constexpr int kProduced = 0;  // block records published by the draws warp
constexpr int kAheadIn = 2;   // block the look-ahead warp follows
constexpr int kWalkerIn = 3;  // block the walker is in
constexpr int kStop = 4;      // the walker has ended its last batch
constexpr int kFail = 5;      // a bounded wait gave up
constexpr int kFinal = 6;     // the flips handed to the field warps are the batch's last (kFinalGood, kFinalFailed)
constexpr uint32_t kFinalGood = 1u, kFinalFailed = 2u;
constexpr int kGo = 1;        // epochs closed: (count << 2) | flags
constexpr uint32_t kGoLeave = 1u, kGoReload = 2u, kGoGaveUp = 3u;  // (kGoGaveUp: leave, a role did not get the word)
constexpr int kCount = 8;     // [8], [9]: flips of the two flip lists
constexpr int kOwnMade = 10;  // blocks whose own pairs are gathered
constexpr int kNextMade = 11; // blocks whose pairs with the next block are gathered
constexpr int kAccepted = 12; // accepted flips of the batch
constexpr int kLastAcc = 13;  // attempts made at the last of them
constexpr int kSettled = 14;  // field warps that have settled an epoch's end, counted on
constexpr int kSlot = 15;     // configuration slot of the walker
constexpr int kReloaded = 16; // warps that have reloaded an exchanged configuration, counted on
constexpr int kBooked = 17;   // blocks entered in the books (pilot statistics)
constexpr int kBoundary = 18; // block before whose first attempt the batch has ended, 0: none
constexpr int kEnded = 19;    // epochs the walker has ended (what it leaves in EpochIo is complete)
constexpr int kWords = 32;

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
constexpr size_t kIoBytes = 112;  // EpochIo
constexpr size_t kOwnTable = kStep * sizeof(DrawRecord);
constexpr size_t kNextTable = kStep * sizeof(NextRecord);
struct AheadLayout {
    size_t slots, own_pairs, next_pairs, flips, hand, attempts, ctl, state, io, fields, bins, spins;
    size_t sq, ds, book_spins, total;  // pilot statistics
};
__host__ __device__ inline AheadLayout ahead_layout(int ld, int mwb, bool scaled, int slots, bool collect) {
    AheadLayout L;
    size_t at = 0;
    L.slots = at; at += static_cast<size_t>(slots) * slot_layout(scaled).total;
    L.own_pairs = at; at += kOwnTables * kOwnTable;     // DrawRecord of each draw
    L.next_pairs = at; at += kNextTables * kNextTable;  // NextRecord of each draw
    L.flips = at; at += 2 * 32 * sizeof(FlipRecord);
    L.hand = at; at += 2 * 33 * 16;                 // handed lanes (HandWords), then their spin mask
    L.attempts = at; at += 2 * sizeof(Attempts);
    L.ctl = at; at += 4 * kWords;
    L.state = at; at += round16(sizeof(WalkerState));
    L.io = at; at += round16(kIoBytes);
    L.fields = at; at += static_cast<size_t>(ld) * 8;
    L.bins = at; at += (static_cast<size_t>(mwb) + 1) * sizeof(BinRecord);
    L.spins = at; at += round16(static_cast<size_t>(ld));
    L.sq = at; at += collect ? round16(static_cast<size_t>(mwb) * 8) : 0;
    L.ds = at; at += collect ? round16(static_cast<size_t>(mwb) * 8) : 0;
    L.book_spins = at; at += collect ? round16(static_cast<size_t>(ld)) : 0;
    L.total = at;
    return L;
}
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) { return *reinterpret_cast<const volatile uint32_t*>(p); }
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) { *reinterpret_cast<volatile uint32_t*>(p) = v; }
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];"
                 : "=r"(v)
                 : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p)))
                 : "memory");
    return v;
}
__device__ __forceinline__ void st_release(uint32_t* p, uint32_t v) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))),
                 "r"(v)
                 : "memory");
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
    if constexpr (kPrec == WLG_PRECISION_FP64) return v.rows64;
    else if constexpr (kPrec == WLG_PRECISION_FP32) return v.rows32;
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
// (row k at `stride` k doubles); with `upper` only what lies above the diagonal.  FP64 couplings go from L2 to
// shared memory without passing registers (cp.async, one group per call), so that the next block's
// gather runs while this one's is in flight: a gather's 30 scattered loads take 840 cycles that way,
// 1940 as two batches of loads waited for.  The narrow forms are widened on the way (exactly; BF16
// times its row scale) and are complete when the call returns.
template <int kPrec>
__device__ __forceinline__ void gather_pairs(const typename Stored<kPrec>::T* J, int ld, int my_row, double my_scale,
                                             int column, bool upper, double* out, int stride, int lane) {
    if constexpr (kPrec == WLG_PRECISION_FP64) {
        const uint32_t to = static_cast<uint32_t>(__cvta_generic_to_shared(out + lane));
#pragma unroll 6
        for (int k = 0; k < kStep; ++k) {
            const int row = __shfl_sync(kFull, my_row, k);
            const double* from = J + static_cast<size_t>(row) * ld + column;
            if (!upper || lane > k)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(to + static_cast<uint32_t>(8 * stride * k)), "l"(from) : "memory");
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
                out[(k0 + u) * stride + lane] = y;
            }
        }
    }
}

// ---- the close of an epoch in a launch of several (all CTAs of the cooperative launch resident) ----

struct EpochClose {
    int status;   // 0; 1: another walker failed; else this walker's status
    bool done;    // the run has terminated
    bool swapped; // this walker has taken its partner's configuration:
    double energy;
    int bin, slot;
    bool left;    // this walker is the pair's left one
    int pairs;    // pairs offered an exchange in this epoch
};

// One walker's end of an epoch, by its warp: what the exchange kernel does for all pairs
// (src/parallel.cpp:157-166, 410-421, src/wang_landau.cpp:483-508, and the termination test of
// src/parallel.cpp:527-533).  Each walker leaves its energy, bin, slot and bins in a mailbox of the
// epoch's parity (the bins also for itself, should it fail in the next epoch) and arrives at a grid-wide count; when all have arrived, the two walkers of a pair
// evaluate the same expression from the same numbers, so that no second barrier is needed.  A mailbox
// is written again two epochs later, after every walker has arrived once more; the termination counts
// rotate over three sets, the first walker clearing the set that is two epochs ahead.
__device__ __forceinline__ EpochClose close_epoch(const EngineView& v, const FusedEpochs& fe, uint32_t epochs, int w,
                                                  int wb, int nbins, const BinRecord* bins, const WalkerState& st,
                                                  uint64_t epoch, bool frozen, bool at_limit, int status, int lane) {
    EpochClose c{status, false, false, 0.0, 0, 0, false, 0};
    const uint32_t parity_box = epochs & 1u, set = epochs % 3u;
    const int walkers = v.walkers, wpw = v.walkers_per_window;
    FusedSync* sync = fe.sync;
    FusedMail* box = fe.mail + static_cast<size_t>(parity_box) * walkers;
    FusedBin* box_bins = fe.mail_bins + static_cast<size_t>(parity_box) * walkers * v.max_window_bins;
    if (status == 0 && (v.windows > 1 || epochs < fe.epochs))
        for (int i = lane; i < nbins; i += 32) box_bins[static_cast<size_t>(w) * v.max_window_bins + i] = bins[i];
    if (lane == 0) {
        if (status != 0 && atomicCAS(&v.ctl->error, 0, status) == 0) v.ctl->error_walker = w;
        box[w] = FusedMail{st.energy, st.cur_bin, st.slot};
        if (frozen) atomicAdd(&sync->frozen[set], 1u);
        if (at_limit) atomicAdd(&sync->at_limit[set], 1u);
        if (status != 0) atomicAdd(&sync->failed[set], 1u);
    }
    __syncwarp();
    uint32_t there = 0;
    if (lane == 0) {
        __threadfence();
        atomicAdd(&sync->arrived, 1u);
        const uint32_t all = static_cast<uint32_t>(walkers) * epochs;
        for (uint32_t polls = 0; polls < kSyncPolls; ++polls) {
            if (static_cast<int32_t>(*reinterpret_cast<volatile uint32_t*>(&sync->arrived) - all) >= 0) {
                there = 1;
                break;
            }
            __nanosleep(40);
        }
        __threadfence();
    }
    there = __shfl_sync(kFull, there, 0);
    if (!there) {
        if (lane == 0 && atomicCAS(&v.ctl->error, 0, WLG_ERR_TIMEOUT) == 0) v.ctl->error_walker = w;
        c.status = WLG_ERR_TIMEOUT;
        return c;
    }
    const uint32_t all_frozen = __ldcg(&sync->frozen[set]), limit = __ldcg(&sync->at_limit[set]);
    const uint32_t any_failed = __ldcg(&sync->failed[set]);
    if (w == 0 && lane == 0) {
        const uint32_t clear = (epochs + 2u) % 3u;
        sync->frozen[clear] = 0;
        sync->at_limit[clear] = 0;
        sync->failed[clear] = 0;
    }
    if (any_failed != 0) {
        if (c.status == 0) c.status = 1;
        c.done = true;
        return c;
    }
    c.done = all_frozen == static_cast<uint32_t>(walkers) ||
             (v.p.max_attempts != 0 && limit == static_cast<uint32_t>(walkers));
    // the even/odd pairing left[p] <-> right[(p + epoch) % wpw] (src/parallel.cpp:410-421)
    const int parity = static_cast<int>(epoch & 1ULL);
    const int bounds = v.windows - 2 < parity ? 0 : (v.windows - 2 - parity) / 2 + 1;
    c.pairs = bounds * wpw;
    const int window = st.window, p = w - window * wpw;
    const int shift = static_cast<int>(epoch % static_cast<uint64_t>(wpw));
    int boundary = -1, partner = 0;
    if (window >= parity && ((window - parity) & 1) == 0 && window + 1 < v.windows) {
        boundary = window;
        c.left = true;
        partner = (window + 1) * wpw + (p + shift) % wpw;
    } else if (window - 1 >= parity && ((window - 1 - parity) & 1) == 0) {
        boundary = window - 1;
        partner = boundary * wpw + (p - shift + wpw) % wpw;
    }
    if (boundary < 0) return c;
    const int4 raw = __ldcg(reinterpret_cast<const int4*>(box + partner));
    const FusedMail other{__hiloint2double(raw.y, raw.x), raw.z, raw.w};
    const int ow = c.left ? window + 1 : window - 1;
    const int ob = v.win_begin[ow], oe = v.win_end[ow], we = wb + nbins;
    const int mine = st.cur_bin, theirs = other.bin;
    if (mine < wb || mine >= we || theirs < wb || theirs >= we || mine < ob || mine >= oe || theirs < ob || theirs >= oe)
        return c;  // exchange_log_probability is -infinity
    const FusedBin* other_bins = box_bins + static_cast<size_t>(partner) * v.max_window_bins;
    const double own_mine = bins[mine - wb].log_g, own_theirs = bins[theirs - wb].log_g;
    const double other_mine = __ldcg(&other_bins[mine - ob].log_g);
    const double other_theirs = __ldcg(&other_bins[theirs - ob].log_g);
    // ga[x] - ga[y] + gb[y] - gb[x] with a the left walker, x its bin, y the right walker's
    const double logp = c.left ? own_mine - own_theirs + other_theirs - other_mine
                               : other_theirs - other_mine + own_mine - own_theirs;
    bool accept = false;
    if (isfinite(logp)) {
        if (logp >= 0.0) {
            accept = true;
        } else {
            Rng rng;
            rng.seed(v.p.seed ^ (epoch * 0x9e3779b97f4a7c15ULL), static_cast<uint64_t>(boundary));
            accept = log(fmax(to_uniform(rng.next()), 0x1.0p-53)) < logp;
        }
    }
    c.swapped = accept;
    c.energy = other.energy;
    c.bin = other.bin;
    c.slot = other.slot;
    return c;
}

// What the walker leaves for the look-ahead warp's end_epoch, and finds there afterwards: in an epoch, bin
// and active are those of its start.
struct EpochIo {
    double energy, factor;
    int32_t stage, bin, status;
    uint32_t active, forced, batch;
    uint32_t exchanged;
    int32_t rt_state;     // pilot statistics: of the books
    uint64_t trips;
    uint64_t epoch0, offered;
    uint64_t rng[4];      // the generator at the last epoch's end, `draws` draws on
    uint32_t draws;
    int32_t good;         // the launch's last epoch was made: its state is to be written
};

// The end of an epoch, by the look-ahead warp: the walker's state, its check, the epoch's close with
// the other walkers, and the word to the other roles; the flags of that word.  It is not the walker's
// warp that does this, because a branch on the lane number (or a call) inside the loop that holds the
// attempt loop costs every attempt: 85 -> 107 us per epoch of the 8x8x8 workload.
__device__ __noinline__ uint32_t end_epoch(const EngineView& v, const WalkArgs& a, const FusedEpochs& fe, EpochIo* io,
                                           WalkerState* st_s, BinRecord* bins, uint32_t* word, const uint64_t* generator,
                                           uint32_t draws, int w, int wb, int nbins, uint32_t epochs, uint32_t settlers,
                                           int lane) {
    const DeviceParams& P = v.p;
    const bool fused = fe.epochs != 0;
    // A look-ahead warp that has given up comes here ahead of the walker, whose own waits then run out, each
    // within kPolls of its faster polls.
    int walker_ended = 2;
    for (int tries = 0; tries < 4 && walker_ended != 0; ++tries)
        walker_ended = wait_at_least(word + kEnded, epochs, nullptr);
    const uint32_t batch = io->batch;
    const uint64_t epoch0 = io->epoch0;
    int status = io->status;
    bool failed = status != 0;
    uint32_t exchanged = io->exchanged;
    uint64_t offered = io->offered;
    const size_t boff = static_cast<size_t>(w) * static_cast<size_t>(v.grid.count) + static_cast<size_t>(wb);
    // the field warps have brought the fields up to date, in shared memory and in HBM
    if (walker_ended != 0 || wait_at_least(word + kSettled, epochs * settlers, nullptr) != 0 ||
        ld_relaxed(word + kFinal) != kFinalGood) {
        failed = true;
        if (status == 0) status = WLG_ERR_TIMEOUT;
    }
    WalkerState st = *st_s;
    const bool at_limit = P.max_attempts != 0 && st.attempted + batch >= P.max_attempts;
    if (!failed) {
        const uint32_t n_acc = word[kAccepted];
        st.energy = io->energy;
        st.factor = io->factor;
        st.stage = io->stage;
        const uint64_t since = n_acc ? static_cast<uint64_t>(batch - word[kLastAcc])
                                     : st.attempted - st.last_accepted + batch;
        st.attempted += batch;
        st.accepted += n_acc;
        st.forced += io->forced;
        st.last_accepted = st.attempted - since;
        st.active_count = io->active;
        st.cur_bin = io->bin;
        if (P.collect) {
            st.rt_state = io->rt_state;
            st.round_trips = io->trips;
            st.rep_pending = 0;
        }
        if (a.epoch_mode && st.stage == kWangLandau && (st.attempted - st.last_check >= P.check_interval || at_limit)) {
            // the check reads H: fold the visits into it
            uint64_t covered = 0, least = ~0ULL, total = 0;
            for (int i = lane; i < nbins; i += 32) {
                const BinRecord r = bins[i];
                const uint64_t hist = v.hist[boff + i] + r.visits;
                v.hist[boff + i] = hist;
                bins[i].visits = 0;
                if (r.active) {
                    covered += hist != 0 ? 1 : 0;
                    least = hist < least ? hist : least;
                    total += hist;
                }
            }
            st.last_check = st.attempted;
            const HistStats hs = histogram_statistics_of(covered, least, total, st.active_count);
            st.last_flatness = P.inverse_time ? hs.coverage : hs.min_over_mean;
            if (stats_ready(hs, st.stage, P)) warp_begin_next_iteration(st, v.hist + boff, nullptr, nbins, P, lane);
        }
        if (lane < 4) io->rng[lane] = generator[lane];
        io->draws = draws;
    } else if (fused) {
        // back to the epoch's start: the bins as this walker left them in its mailbox, or as the launch found
        // them; the state, the generator and, in HBM, the fields and spins are those of that time still
        const FusedBin* box = fe.mail_bins + (static_cast<size_t>((epochs - 1) & 1u) * v.walkers + w) * v.max_window_bins;
        for (int i = lane; i < nbins; i += 32)
            bins[i] = epochs > 1 ? box[i] : BinRecord{v.log_g[boff + i], 0u, v.active[boff + i] != 0 ? 1u : 0u};
    }
    bool leave = true, reload = false, done = false;
    bool ended = failed;  // the run ends with a failure, this walker's or another's
    if (fused) {
        // every walker arrives with its configuration's energy and bin, and each pair's two walkers
        // then decide their exchange alike
        const EpochClose c = close_epoch(v, fe, epochs, w, wb, nbins, bins, st, epoch0 + epochs - 1,
                                         st.stage == kFrozen, at_limit, failed ? status : 0, lane);
        ended = ended || c.status != 0;
        if (c.status > 1) status = c.status;
        leave = ended || c.done || epochs == fe.epochs;
        if (c.swapped) {
            st.energy = c.energy;
            st.cur_bin = c.bin;
            st.slot = c.slot;
            reload = !leave;
            exchanged += c.left ? 1u : 0u;
            if (P.collect) {
                round_trip_update(st.energy, window_lower(v, wb), window_lower(v, wb + nbins), P.round_trip_margin,
                                  st.rt_state, st.round_trips);
                st.rep_pending = leave ? 1 : 0;  // the books refresh the representatives after the reload
            }
        }
        offered += static_cast<uint64_t>(c.pairs);
        done = c.done;
    }
    __syncwarp();
    uint32_t flags = (leave ? kGoLeave : 0u) | (reload ? kGoReload : 0u);
    if (lane == 0) {
        if (ended) st_relaxed(word + kFail, 1u);
        *st_s = st;  // (a failed epoch's is as it was)
        word[kSlot] = static_cast<uint32_t>(st.slot);
        io->good = failed ? 0 : 1;
        io->energy = st.energy;
        io->factor = st.factor;
        io->stage = st.stage;
        io->bin = st.cur_bin;
        io->status = status;
        io->exchanged = exchanged;
        io->offered = offered;
        // The word is replaced, not stored: a role that has given up waiting for it has put its own there,
        // and then this warp leaves as well (it would otherwise wait at a barrier for warps that have left).
        __threadfence_block();
        const uint32_t before = ld_relaxed(word + kGo);
        if ((before >> 2) == (epochs & 0x3fffffffu) || atomicCAS(word + kGo, before, (epochs << 2) | flags) != before)
            flags = kGoGaveUp;
        if (flags & kGoLeave) st_release(word + kStop, 1u);
        if (fused && w == 0 && (flags & kGoLeave)) {
            v.ctl->exchange_attempted += offered;
            v.ctl->epoch = epoch0 + epochs - (ended ? 1u : 0u);  // (an epoch that failed somewhere is not counted)
            v.ctl->done = done || ended || flags == kGoGaveUp ? 1 : 0;
        }
    }
    return __shfl_sync(kFull, flags, 0);
}

template <int kPrec, bool kPow2, bool kAlone, bool kCollect>
__global__ void __launch_bounds__(32 * warps_for((kAlone ? kMaxRoles : kMaxRoles - 1) + (kCollect ? 1 : 0), kAlone), kAlone ? 1 : 2) sweep_ahead_kernel(const __grid_constant__ EngineView v,
                                                                                                        const __grid_constant__ WalkArgs a,
                                                                                                        int slots, int field_warps,
                                                                                                        const __grid_constant__ FusedEpochs fe) {
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
    const AheadLayout L = ahead_layout(ld, v.max_window_bins, kScaled, slots, kCollect);
    FlipRecord* flips = reinterpret_cast<FlipRecord*>(smem + L.flips);
    HandWords* hand = reinterpret_cast<HandWords*>(smem + L.hand);
    Attempts* attempts = reinterpret_cast<Attempts*>(smem + L.attempts);
    uint32_t* word = reinterpret_cast<uint32_t*>(smem + L.ctl);
    double* f_s = reinterpret_cast<double*>(smem + L.fields);
    BinRecord* bins = reinterpret_cast<BinRecord*>(smem + L.bins);
    int8_t* sp_s = reinterpret_cast<int8_t*>(smem + L.spins);

    const bool fused = fe.epochs != 0;  // several epochs with their exchanges in this launch
    // the walker's scalars are read where they are used (by one role each), so that no role holds them all
    const WalkerState* ws = v.ws + w;
    const int wb = v.win_begin[ws->window], nbins = v.win_end[ws->window] - wb;
    const bool escaped = ws->cur_bin < wb || ws->cur_bin >= wb + nbins;  // "Walker escaped its energy window"
    const DeviceParams& P = v.p;
    const size_t boff = static_cast<size_t>(w) * static_cast<size_t>(v.grid.count) + static_cast<size_t>(wb);
    const JT* J = coupling_rows<kPrec>(v);

    // ---- stage the walker ------------------------------------------------------------------
    // fields and spins of a configuration slot, by `threads` threads (past L1, which may hold what
    // another CTA has replaced since)
    auto load_fields = [&](int slot, int me, int threads) {
        const double2* from = reinterpret_cast<const double2*>(v.fields + static_cast<size_t>(slot) * ld);
        for (int k = me; k < (ld >> 1); k += threads) reinterpret_cast<double2*>(f_s)[k] = __ldcg(from + k);
    };
    auto load_spins = [&](int slot, int me, int threads) {
        const int4* from = reinterpret_cast<const int4*>(v.spins + static_cast<size_t>(slot) * ld);
        for (int k = me; k < (ld >> 4); k += threads) reinterpret_cast<int4*>(sp_s)[k] = __ldcg(from + k);
    };
    load_fields(ws->slot, static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x));
    load_spins(ws->slot, static_cast<int>(threadIdx.x), static_cast<int>(blockDim.x));
    WalkerState* st_s = reinterpret_cast<WalkerState*>(smem + L.state);
    for (int b = threadIdx.x; b <= nbins; b += blockDim.x) {
        BinRecord r{0.0, 0u, 1u};  // [nbins]: read for a proposal outside the window, never used
        if (b < nbins) {
            r.log_g = v.log_g[boff + b];
            r.active = v.active[boff + b] != 0 ? 1u : 0u;
        }
        bins[b] = r;
    }
    if (threadIdx.x < 64) attempts[threadIdx.x >> 5].entry[threadIdx.x & 31] = make_uint2(0, 0);
    if (threadIdx.x < 66) hand[threadIdx.x] = HandWords{0, 0};
    if (threadIdx.x < kWords) word[threadIdx.x] = 0;
    if (threadIdx.x == 32) *st_s = *ws;
    static_assert(sizeof(EpochIo) <= kIoBytes, "EpochIo");
    if (threadIdx.x == 64) {
        EpochIo first{};
        first.bin = escaped ? wb : ws->cur_bin;
        first.active = static_cast<uint32_t>(ws->active_count);
        first.epoch0 = ctl->epoch;
        for (int k = 0; k < 4; ++k) first.rng[k] = ws->rng[k];
        *reinterpret_cast<EpochIo*>(smem + L.io) = first;
    }
    __syncthreads();
    if (threadIdx.x == 0) word[kSlot] = static_cast<uint32_t>(st_s->slot);
    __syncthreads();
    // the warp's writes are visible to who has seen the count
    auto settle = [&](int counter) {
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            atomicAdd(word + counter, 1u);
        }
    };
    // Waits for the word on the end of epoch `count`; its flags.  A role that gives up puts a word of its own in
    // place of the one it saw last, for all: either the look-ahead warp's word came first and holds, or every
    // role, the look-ahead warp among them, leaves (by all lanes: no branch on the lane number here).
    auto wait_go = [&](uint32_t count) -> uint32_t {
        uint32_t x = 0;
        for (uint32_t polls = 0; polls < kSyncPolls; ++polls) {
            x = ld_relaxed(word + kGo);
            if (__all_sync(kFull, (x >> 2) == (count & 0x3fffffffu))) {
                __threadfence_block();
                return __shfl_sync(kFull, x, 0) & 3u;
            }
            __nanosleep(100);
        }
        atomicCAS(word + kGo, x, (count << 2) | kGoGaveUp);
        __syncwarp();
        __threadfence_block();
        x = __shfl_sync(kFull, ld_relaxed(word + kGo), 0) & 3u;
        if (x == kGoGaveUp) st_relaxed(word + kFail, 1u);
        return x;
    };

    auto slot_of = [&](int s) { return smem + L.slots + static_cast<size_t>(s) * SL.total; };

    if (role == 0) {
        // ---- the walker ----------------------------------------------------------------------
        double E = ws->energy, factor = ws->factor;
        int32_t stage = ws->stage;
        uint64_t since = 0;
        uint32_t n_forced = 0;
        uint32_t active32 = static_cast<uint32_t>(ws->active_count);  // at most the window's bins
        int cur = escaped ? 0 : ws->cur_bin - wb;
        EpochIo* io = reinterpret_cast<EpochIo*>(smem + L.io);
        int s = 0;
        uint32_t k = 0;  // draw (lane) of the current attempt's site
        int status = escaped ? WLG_ERR_ESCAPED : 0;
        bool failed = escaped;
        if (!failed && wait_at_least(word + kOwnMade, 1, nullptr) != 0) {
            failed = true;
            status = WLG_ERR_TIMEOUT;
        }
        const Grid g = v.grid;
        const double neg_min_scaled = -g.minimum * g.inv_width;
        // q + this, rounded toward -infinity, is 1.5 * 2^52 + (floor(q) - wb) exactly for |q| < 2^51 (unit
        // in the last place 1): the low word is the window's bin, and the high word is kBinHigh exactly
        // when 0 <= floor(q) - wb < 2^32
        const double bin_magic = 0x1.8p52 - static_cast<double>(wb);
        constexpr int kBinHigh = 0x43380000;
        const double half_clear = 0.5 - (static_cast<double>(g.count) + 2.0) * 0x1p-49;
        const uint32_t last_bin = static_cast<uint32_t>(static_cast<int>(g.count) - 1 - wb);  // E == maximum
        uint32_t b = 0;
        uint32_t own = 0;  // the block's table of draw records
        // (set from the shared-memory base here, never null: the compiler then knows the address space)
        const DrawRecord* draws = reinterpret_cast<const DrawRecord*>(smem + L.own_pairs);
        uint32_t rejected = 0;
        auto enter = [&]() {  // the records of block b
            draws = reinterpret_cast<const DrawRecord*>(smem + L.own_pairs + own * kOwnTable);
            rejected = reinterpret_cast<const uint32_t*>(slot_of(s) + SL.misc)[8];
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
        // the lanes from the fields in shared memory, which are complete
        auto load_lanes = [&]() {
            const int site = reinterpret_cast<const int32_t*>(slot_of(s) + SL.site)[lane];
            fc = f_s[site < 0 ? 0 : site];
            up = __ballot_sync(kFull, sp_s[site < 0 ? 0 : site] > 0);
            h = __shfl_sync(kFull, fc, static_cast<int>(k));
            m_hi = sign_of(k);
        };
        if (!failed) {
            enter();
            load_lanes();
        }
        uint32_t t = 0;  // attempts made at the entry e_mark of the block
        uint32_t* e_p = &attempts[0].entry[0].x;
        const uint32_t* e_mark = e_p;
        double lg_cur = bins[cur].log_g;
        uint32_t visits = 0, batch = 0;
        bool opens = bins[cur].active == 0;  // an exchange brought a bin not visited before
        uint64_t att0 = 0;
        const uint64_t force_limit = P.force_after != 0 ? P.force_after : ~0ULL;

        // Attempts until the batch ends or, in the 1/t stage, the walker freezes.  kIT: the 1/t stage;
        // kForce: forced acceptance (force_accept_after_attempts != 0); kTop: the window holds the grid's
        // last bin, to which the energy E == maximum belongs.  Everything an attempt does not need is
        // left to the look-ahead warp (the counts of attempts and acceptances come from the entries) or
        // to the rare path at the top, which one comparison guards: `klim` is the first draw at which
        // the block, the batch, the 1/t table or the active-bin count may change.
        auto run = [&](auto it_tag, auto force_tag, auto top_tag) {
            constexpr bool kIT = decltype(it_tag)::value;
            constexpr bool kForce = decltype(force_tag)::value;
            constexpr bool kTop = decltype(top_tag)::value;
            // what an attempt adds to log g of its bin: ln f, or -0.0 (which changes nothing) once frozen
            const double constant = stage == kFrozen ? -0.0 : factor;
            uint32_t frozen_at = 0;  // 1/t stage: the attempts made once the walker freezes, 0 = not in the table
            double quotient = factor;
            const uint32_t* quotient_mark = e_mark;  // 1/t stage: the entry the table starts at
            uint32_t polls = 0, klim_next = 0;
            bool waiting = false;  // for the lanes of the block just entered
            [[maybe_unused]] bool exact = false;  // the next attempt's bin (fl_exact) has been worked out exactly
            [[maybe_unused]] const uint32_t* exact_at = nullptr;
            [[maybe_unused]] double fl_exact = 0.0;
            klim = 0;
            while (true) {
                if (k >= klim) {
                    // (the attempt loop is the polling loop too: a loop of its own inside it costs every
                    // attempt about ten cycles; and no branch here may be on the lane number, which would
                    // cost the whole loop its uniform form, 250 -> 350 cycles per attempt)
                    if (!waiting) {
                        const uint32_t made = static_cast<uint32_t>(e_p - e_mark) >> 1;
                        if (made != 0) {
                            // an initial bin not visited before is opened by the first attempt if that stayed there
                            // (the epoch's bin and count are where its start left them: the look-ahead warp may
                            // have cleared the attempt's entry by now, when it was the block's last)
                            if (t == 0 && opens && opened_by_staying(cur + wb, io->bin, active32, io->active)) ++active32;
                            if (kIT)
                                factor = __shfl_sync(kFull, quotient, static_cast<int>((e_p - quotient_mark) >> 1) - 1);
                            t += made;
                            e_mark = e_p;
                        }
                        if (kIT && frozen_at != 0 && t == frozen_at) {
                            stage = kFrozen;
                            return;
                        }
                        if (t >= batch) return;
                        if (k >= static_cast<uint32_t>(kStep)) {  // the next block
                            if (!__all_sync(kFull, static_cast<int32_t>(ld_acquire(word + kOwnMade) - (b + 2)) >= 0)) {
                                if (++polls < kPolls) continue;
                                failed = true;
                                return;
                            }
                            ++b;
                            polls = 0;
                            k -= kStep;
                            s = s + 1 == slots ? 0 : s + 1;
                            own = own + 1 == kOwnTables ? 0 : own + 1;
                            enter();
                            e_p = &attempts[b & 1u].entry[0].x;
                            e_mark = e_p;
                            st_release(word + kWalkerIn, b);
                            waiting = true;
                        }
                        // Every attempt consumes a draw, so that at draw k + left at most `left` were made
                        // (the first attempt by itself when it may open the initial bin).
                        const uint32_t left = opens && t == 0 ? 1u : batch - t;
                        klim_next = limit(k);
                        klim_next = left < klim_next - k ? k + left : klim_next;
                        if constexpr (!kPow2) {  // the attempt whose bin is worked out exactly, by itself
                            exact = exact_at == e_p;
                            klim_next = exact ? k + 1 : klim_next;
                            if (exact) {
                                const double offset = fma(__hiloint2double(m_hi, 0), h, E) - g.minimum;
                                fl_exact = floor_near_integer(offset, g.width, rint(offset * g.inv_width)) + bin_magic;
                            }
                        }
                        if constexpr (kIT) {
                            // update_inverse_time_factor (src/wang_landau.cpp:300-315) of the block's
                            // coming attempts, lane j dividing for attempt j from here; at a new block while
                            // its lanes are on their way
                            const double made_d = static_cast<double>(att0 + t + static_cast<uint64_t>(lane) + 1);
                            quotient = quotient_rn(static_cast<double>(active32 == 0 ? 1u : active32), made_d,
                                                   static_cast<double>(__fdividef(1.0f, static_cast<float>(made_d))));
                            quotient = active32 == 0 ? factor : quotient;
                            const bool frz = quotient <= P.final_factor;
                            const uint32_t fm = __ballot_sync(kFull, frz);
                            const uint32_t e0 = static_cast<uint32_t>(e_p - &attempts[b & 1u].entry[0].x) >> 1;
                            attempts[b & 1u].add[(e0 + lane) & 31u] = frz ? -0.0 : quotient;
                            __syncwarp();
                            quotient_mark = e_p;
                            frozen_at = 0;
                            if (fm) {
                                const uint32_t steps = static_cast<uint32_t>(__ffs(static_cast<int>(fm)));
                                frozen_at = t + steps;
                                klim_next = steps < klim_next - k ? k + steps : klim_next;
                            }
                        }
                    }
                    if (waiting) {
                        const volatile HandWords* mine = hand + 33 * (b & 1u) + lane;
                        const volatile HandWords* mask = hand + 33 * (b & 1u) + 32;
                        const uint64_t w0 = mine->low, w1 = mine->high, w2 = mask->low;
                        const bool there = static_cast<uint32_t>(w0 >> 32) == b && static_cast<uint32_t>(w1 >> 32) == b &&
                                           static_cast<uint32_t>(w2 >> 32) == b;
                        if (!__all_sync(kFull, there)) {
                            klim = 0;
                            if (++polls < kPolls) continue;
                            failed = true;
                            return;
                        }
                        polls = 0;
                        waiting = false;
                        fc = __hiloint2double(static_cast<int>(static_cast<uint32_t>(w1)),
                                              static_cast<int>(static_cast<uint32_t>(w0)));
                        up = __shfl_sync(kFull, static_cast<uint32_t>(w2), 0);
                    }
                    klim = klim_next;
                    if ((rejected >> k) & 1u) {  // bounded() rejects the draw: the next one is the site
                        st_relaxed(e_p, kEntValid | kEntSkip);
                        e_p += 2;
                        e_mark = e_p;
                        ++k;
                        h = __shfl_sync(kFull, fc, static_cast<int>(k));
                        m_hi = sign_of(k);
                        klim = 0;  // the next draw may be another block's, or rejected as well
                        continue;
                    }
                }
                const uint32_t k1 = k + 1, k2 = k + 2;  // the candidates for the next site
                const DrawRecord* d = draws + k;
                const double2 d0 = *reinterpret_cast<const double2*>(&d->lnu);    // lnu, pair1
                const double2 d1 = *reinterpret_cast<const double2*>(&d->pair2);  // pair2, same
                const double rl = d->pair[lane];
                const double add = kIT ? *reinterpret_cast<const double*>(e_p + kAddWords) : constant;
                const double fc1 = __shfl_sync(kFull, fc, static_cast<int>(k1));
                const double fc2 = __shfl_sync(kFull, fc, static_cast<int>(k2));

                // attempt_flip (src/wang_landau.cpp:244-262)
                const double m = __hiloint2double(m_hi, 0);
                const double Ep = fma(m, h, E);
                double fl;
                [[maybe_unused]] bool unclear = false;
                if constexpr (kPow2) {
                    fl = __dadd_rd(fma(Ep, g.inv_width, neg_min_scaled), bin_magic);
                } else {
                    // q differs from the reference's rounded quotient by less than |q| 2^-51, so both
                    // have the same floor unless q lies that near to an integer; then the attempt is
                    // made again with the floor worked out exactly
                    const double q = (Ep - g.minimum) * g.inv_width;
                    fl = __dadd_rd(q, bin_magic);
                    unclear = !exact && !(fabs(q - (fl - bin_magic) - 0.5) < half_clear);
                    fl = exact ? fl_exact : fl;
                }
                uint32_t nb = static_cast<uint32_t>(__double2loint(fl));
                bool in_window;
                if constexpr (kTop) {
                    const bool top = Ep == g.maximum;
                    nb = top ? last_bin : nb;
                    in_window = nb < static_cast<uint32_t>(nbins) &&
                                (top || (__double2hiint(fl) == kBinHigh && Ep < g.maximum));
                } else {  // a bin below the grid's last one: its energies are below the maximum
                    in_window = nb < static_cast<uint32_t>(nbins) && __double2hiint(fl) == kBinHigh;
                }
                const BinRecord rec = bins[nb < static_cast<uint32_t>(nbins) ? nb : static_cast<uint32_t>(nbins)];
                const double log_ratio = lg_cur - rec.log_g;
                const bool det = log_ratio >= 0.0;
                if constexpr (!kPow2) {
                    if (unclear) {
                        exact_at = e_p;
                        klim = 0;
                        continue;
                    }
                }
                bool accepted, need_u;
                if constexpr (kForce) {
                    const bool forced = in_window && !det && since >= force_limit;
                    need_u = in_window && !det && !forced;
                    accepted = in_window && (det || forced || d0.x < log_ratio);
                    n_forced += forced ? 1u : 0u;
                    since = accepted ? 0 : since + 1;
                } else {
                    need_u = in_window && !det;
                    accepted = in_window && d0.x < log_ratio;  // lnu < 0, so det accepts as well
                }
                const int me_hi = accepted ? m_hi : 0;
                const double m_eff = __hiloint2double(me_hi, 0);
                [[maybe_unused]] const double h_site = h;
                h = fma(m_eff, need_u ? d1.x : d0.y, need_u ? fc2 : fc1);
                up ^= accepted ? static_cast<uint32_t>(__double2loint(d1.y)) : 0u;
                const uint32_t x = static_cast<uint32_t>(me_hi) | (need_u ? kEntValid | kEntUniform : kEntValid);
                k = need_u ? k2 : k1;
                m_hi = sign_of(k);
                if constexpr (kCollect) {  // the books read the field and the bin left once the entry is there
                    *reinterpret_cast<volatile double*>(e_p + kFieldWords) = h_site;
                    st_relaxed(e_p + 1, static_cast<uint32_t>(cur));
                    st_release(e_p, x);
                } else {
                    st_relaxed(e_p, x);
                }
                e_p += 2;
                fc = fma(m_eff, rl, fc);
                E = accepted ? Ep : E;
                // update_current_bin (src/wang_landau.cpp:277-278)
                cur = accepted ? static_cast<int>(nb) : cur;
                lg_cur = (accepted ? rec.log_g : lg_cur) + add;
                visits = (accepted ? rec.visits : visits) + 1u;
                const bool opened = accepted && rec.active == 0;
                active32 += opened ? 1u : 0u;
                if (kIT) klim = opened ? 0u : klim;
                BinRecord now;
                now.log_g = lg_cur;
                now.visits = visits;
                now.active = 1u;
                bins[cur] = now;
            }
        };
        auto run_stage = [&](auto force_tag, auto top_tag) {
            if (stage == kInverseTime) run(std::true_type{}, force_tag, top_tag);
            else run(std::false_type{}, force_tag, top_tag);
        };
        const bool top_window = wb + nbins == static_cast<int>(g.count);
        // (no branch on the lane number and no call in this loop: see end_epoch)
        uint32_t reloads = 0;  // warps that have to have reloaded
        for (uint32_t epochs = 1;; ++epochs) {
            const uint64_t made = st_s->attempted;
            uint64_t left = a.fixed_batch ? a.fixed_batch : P.exchange_interval;
            if (!a.fixed_batch && P.max_attempts) {
                const uint64_t remaining = made < P.max_attempts ? P.max_attempts - made : 0;
                left = remaining < left ? remaining : left;
            }
            batch = static_cast<uint32_t>(left < 0xffffffffULL ? left : 0xffffffffULL);
            att0 = made + st_s->time_offset;
            since = made - st_s->last_accepted;
            n_forced = 0;
            while (!failed && t < batch) {
                if (P.force_after != 0) run_stage(std::true_type{}, std::true_type{});
                else if (top_window) run_stage(std::false_type{}, std::true_type{});
                else run_stage(std::false_type{}, std::false_type{});
            }
            if (failed && status == 0) status = WLG_ERR_TIMEOUT;
            const bool block_done = k >= static_cast<uint32_t>(kStep) && !failed;
            io->energy = E;
            io->factor = factor;
            io->stage = stage;
            io->bin = cur + wb;
            io->status = status;
            io->active = active32;
            io->forced = n_forced;
            io->batch = batch;
            st_release(word + kEnded, epochs);
            if (failed) st_relaxed(word + kFail, 1u);
            if (failed || !fused) st_release(word + kStop, 1u);
            // the stop entry; a batch that ended with its block's last draw has no entry left for it (the
            // next block's may still be cleared by who follows)
            st_release(block_done ? word + kBoundary : e_p, block_done ? b + 1 : kEntValid | kEntStop);
            const uint32_t go = wait_go(epochs);
            if (go & kGoLeave) break;
            if (go & kGoReload) {
                reloads += 1u + static_cast<uint32_t>(field_warps) + (kCollect ? 1u : 0u);
                failed = wait_at_least(word + kReloaded, reloads, nullptr) != 0;
            }
            if (block_done) failed = failed || wait_at_least(word + kOwnMade, b + 2, nullptr) != 0;
            E = io->energy;
            factor = io->factor;
            stage = io->stage;
            cur = io->bin - wb;
            if (block_done) {
                ++b;
                k -= kStep;
                s = s + 1 == slots ? 0 : s + 1;
                own = own + 1 == kOwnTables ? 0 : own + 1;
                enter();
                st_release(word + kWalkerIn, b);
            }
            load_lanes();
            e_p = &attempts[b & 1u].entry[0].x;
            e_mark = e_p;
            t = 0;
            lg_cur = bins[cur].log_g;
            visits = bins[cur].visits;
            opens = bins[cur].active == 0;
        }
        bar_sync(0, static_cast<int>(blockDim.x));  // every role has left
        if (failed || ld_relaxed(word + kFail) != 0) {
            // (in a launch of several epochs the first error is there already, unless a role gave up since)
            if (lane == 0) record_error(ctl, io->status > 0 ? io->status : WLG_ERR_TIMEOUT, w);
            if (!fused && !io->good) return;
        }
        const uint32_t exchanged = io->exchanged;
        WalkerState st = *st_s;
        // the generator after the draws consumed: the block's first state, some draws on
        {
            Rng rng{io->rng[0], io->rng[1], io->rng[2], io->rng[3]};
            for (uint32_t d = 0; d < io->draws; ++d) rng.next();
            st.rng[0] = rng.s0;
            st.rng[1] = rng.s1;
            st.rng[2] = rng.s2;
            st.rng[3] = rng.s3;
        }
        for (int i = lane; i < nbins; i += 32) {
            const BinRecord r = bins[i];
            v.log_g[boff + i] = r.log_g;
            v.hist[boff + i] += r.visits;
            v.active[boff + i] = static_cast<uint8_t>(r.active);
        }
        if (lane == 0) {
            v.ws[w] = st;
            if (fused) {
                if (exchanged) atomicAdd(reinterpret_cast<unsigned long long*>(&ctl->exchange_accepted),
                                         static_cast<unsigned long long>(exchanged));
            } else if (a.epoch_mode) {
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
        const uint32_t most = blocks_published(P, w);  // failure injection: the walker's wait runs out
        for (uint32_t b = 0; b < most; ++b) {
            if (b >= static_cast<uint32_t>(slots)) {  // the record's last readers: the walker and the look-ahead
                const uint32_t need = b - static_cast<uint32_t>(slots) + 1;
                int r = wait_at_least(word + kAheadIn, need, word + kStop);
                if (r == 0) r = wait_at_least(word + kWalkerIn, need, word + kStop);
                if (kCollect && r == 0) r = wait_at_least(word + kBooked, need, word + kStop);
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
        EpochIo* io = reinterpret_cast<EpochIo*>(smem + L.io);
        int s = 0, k = 0;
        uint32_t table = 0;
        uint32_t made = 0, n_acc = 0, last_acc = 0;  // attempts followed; accepted; attempts made at the last acceptance
        uint32_t lists = 0, epochs = 0, reloads = 0;
        bool fresh = true;  // the fields in shared memory are complete (no list is being applied)
        for (uint32_t b = 0;;) {
            if (lane == 0) st_release(word + kAheadIn, b);
            const int s_next = s + 1 == slots ? 0 : s + 1;
            const unsigned char* rec = slot_of(s);
            const NextRecord* next = reinterpret_cast<const NextRecord*>(smem + L.next_pairs + table * kNextTable);
            int r = wait_at_least(word + kNextMade, b + 1, word + kStop);
            if (r == 0) r = wait_at_least(word + kOwnMade, b + 2, word + kStop);
            bool gave_up = r == 2;
            int mine = 0;  // the next block's site of this lane
            if (r == 0) {
                mine = reinterpret_cast<const int32_t*>(slot_of(s_next) + SL.site)[lane];
                mine = mine < 0 ? 0 : mine;
            }
            if (!fresh) bar_sync(kBarFields, barrier_threads);  // the fields are up to block b - 1
            fresh = false;
            double f = f_s[mine];
            uint32_t up = __ballot_sync(kFull, sp_s[mine] > 0);
            uint2* e_s = attempts[b & 1u].entry;
            // Follow the walker.  First what it has published already: lane e reads entry e and works
            // out its draw, and the flips found are applied in order, eight at a time with their table
            // loads overlapped.
            const int k0 = k;
            const uint32_t below = (1u << lane) - 1u;
            int done = 0;  // entries followed
            bool stop = false;
            if (!gave_up) {
                const uint32_t x = ld_relaxed(&e_s[lane].x);
                const uint32_t missing = __ballot_sync(kFull, x == 0);
                const int there = missing ? __ffs(static_cast<int>(missing)) - 1 : 32;
                const uint32_t uni = __ballot_sync(kFull, x & kEntUniform);
                stop = __any_sync(kFull, x & kEntStop);  // the last entry there, never accepted
                // the draw, and the high word of m above it (0 unless accepted)
                const uint32_t mine_x = lane < there && (x & 0x40000000u)
                                            ? (x & 0xC0000000u) | static_cast<uint32_t>(k0 + lane + __popc(uni & below))
                                            : 0u;
#pragma unroll 1
                for (; done < there; done += 8) {  // (without a branch inside: each would wait for its operands)
                    uint32_t of[8], same[8];
                    double pair[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        of[u] = __shfl_sync(kFull, mine_x, (done + u) & 31);
                        of[u] = done + u < there ? of[u] : 0u;
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const NextRecord* row = next + (of[u] & 31u);
                        pair[u] = row->pair[lane];
                        same[u] = row->cross;
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        f = fma(__hiloint2double(static_cast<int>(of[u] & 0xC0000000u), 0), pair[u], f);
                        up ^= of[u] ? same[u] : 0u;
                    }
                }
                done = there - (stop ? 1 : 0);
                k = k0 + done + __popc(uni & (done < 32 ? (1u << done) - 1u : kFull));
            }
            // Then one entry at a time, its table row loaded before it is there: quicker than the walker,
            // so that the lanes are complete right after its last attempt of the block.
            while (!gave_up && !stop && k < kStep) {
                const double pair = next[k].pair[lane];
                const uint32_t same = next[k].cross;
                uint32_t x = ld_relaxed(&e_s[done].x);  // one word: the same for every lane
                for (uint32_t polls = 0; x == 0 && polls < kPolls; ++polls) {
                    x = ld_relaxed(&e_s[done].x);
                    if (done == 0 && x == 0 && b != 0 && ld_relaxed(word + kBoundary) == b) x = kEntValid | kEntStop;
                }
                f = fma(__hiloint2double(static_cast<int>(x & 0xC0000000u), 0), pair, f);  // m = 0 unless accepted
                up ^= (x & 0x40000000u) ? same : 0u;
                stop = (x & kEntStop) != 0;
                gave_up = x == 0;
                if (stop || gave_up) break;
                k += (x & kEntUniform) ? 2 : 1;
                ++done;
            }
            __syncwarp();
            const bool last = stop || gave_up;
            if constexpr (kCollect) {
                // the books, too, read the entries: the buffer of the block before, which the walker gets back
                // with the lanes, is cleared when they are through with it
                if (!last && b > 0) {
                    if (wait_at_least(word + kBooked, b, nullptr) != 0) st_relaxed(word + kFail, 1u);
                    attempts[(b + 1) & 1u].entry[lane] = make_uint2(0, 0);
                    __syncwarp();
                    __threadfence_block();
                }
            }
            if (!last) {  // hand the lanes over
                volatile HandWords* out = hand + 33 * ((b + 1) & 1u) + lane;
                const uint64_t tag = static_cast<uint64_t>(b + 1) << 32;
                out->low = tag | static_cast<uint32_t>(__double2loint(f));
                out->high = tag | static_cast<uint32_t>(__double2hiint(f));
                (out + 32 - lane)->low = tag | up;
            }
            const uint32_t x = lane < done ? ld_relaxed(&e_s[lane].x) : 0u;
            const uint32_t neg = __ballot_sync(kFull, x & 0x80000000u), uni = __ballot_sync(kFull, x & kEntUniform);
            const uint32_t skip = __ballot_sync(kFull, x & kEntSkip), acc = __ballot_sync(kFull, x & 0x40000000u);
            if constexpr (!kCollect) e_s[lane] = make_uint2(0, 0);  // the walker writes there only in block b + 2, or in the next epoch
            // the block's flips for the field warps
            const bool mine_flipped = (acc >> lane) & 1u;
            const int at = mine_flipped ? k0 + lane + __popc(uni & below) : 0;
            const int site = reinterpret_cast<const int32_t*>(rec + SL.site)[at];
            const int flips_made = __popc(acc);
            const int first_site = __shfl_sync(kFull, site, flips_made ? __ffs(static_cast<int>(acc)) - 1 : 0);
            // padded with flips that change nothing (the first flip's row, m = 0) to a multiple of four
            const bool pad = lane >= flips_made && lane < ((flips_made + 3) & ~3);
            FlipRecord fr;
            fr.m = (neg >> lane) & 1u ? -2.0 : 2.0;
            if constexpr (kScaled) fr.m *= reinterpret_cast<const double*>(rec + SL.scale)[at];
            fr.row = static_cast<uint64_t>(site) * static_cast<uint64_t>(ld) * sizeof(JT);
            if (mine_flipped) flips[32 * (lists & 1u) + __popc(acc & below)] = fr;
            fr.m = 0.0;
            fr.row = static_cast<uint64_t>(first_site) * static_cast<uint64_t>(ld) * sizeof(JT);
            if (pad) flips[32 * (lists & 1u) + lane] = fr;
            // the epoch was made if the walker says so and its entries have been followed to the end; what this
            // decides, the writes of fields, spins and state, all go by this one word
            const bool good = last && !gave_up && *reinterpret_cast<volatile int32_t*>(&io->status) == 0;
            if (lane == 0) {
                word[kCount + (lists & 1u)] = static_cast<uint32_t>(flips_made);
                word[kFinal] = !last ? 0u : good ? kFinalGood : kFinalFailed;
                if (gave_up) st_relaxed(word + kFail, 1u);
            }
            __syncwarp();
            bar_arrive(kBarList, barrier_threads);
            ++lists;
            // the spins: each flip turns 0x01 into 0xff or back, in whatever order a site's flips are counted
            if (mine_flipped) atomicXor(reinterpret_cast<uint32_t*>(sp_s) + (site >> 2), 0xfeu << (8 * (site & 3)));
            if (flips_made) {
                const int e = 31 - __clz(static_cast<int>(acc));  // the last accepted attempt of the block
                n_acc += static_cast<uint32_t>(flips_made);
                last_acc = made + static_cast<uint32_t>(e + 1 - __popc(skip & ((2u << e) - 1u)));
            }
            made += static_cast<uint32_t>(done - __popc(skip));
            if (lane == 0) {
                word[kAccepted] = n_acc;
                word[kLastAcc] = last_acc;
            }
            __syncwarp();
            if (last) {  // the epoch's end
                ++epochs;
                if (good) {
                    int4* to = reinterpret_cast<int4*>(v.spins + static_cast<size_t>(word[kSlot]) * ld);
                    for (int i = lane; i < (ld >> 4); i += 32) to[i] = reinterpret_cast<const int4*>(sp_s)[i];
                }
                const uint32_t settlers = static_cast<uint32_t>(field_warps) + (kCollect ? 1u : 0u);
                if constexpr (kCollect) {
                    if (wait_at_least(word + kSettled, epochs * settlers, nullptr) != 0) st_relaxed(word + kFail, 1u);
                    attempts[0].entry[lane] = make_uint2(0, 0);
                    attempts[1].entry[lane] = make_uint2(0, 0);
                }
                st_relaxed(word + kBoundary, 0u);
                __syncwarp();
                const uint32_t go = end_epoch(v, a, fe, io, st_s, bins, word,
                                              reinterpret_cast<const uint64_t*>(rec + SL.misc), static_cast<uint32_t>(k), w,
                                              wb, nbins, epochs, settlers, lane);
                if (go & kGoLeave) break;
                if (go & kGoReload) {
                    load_spins(static_cast<int>(word[kSlot]), lane, 32);
                    settle(kReloaded);
                    reloads += 1u + settlers;
                    // every field warp's part, too, before the first field is read
                    if (wait_at_least(word + kReloaded, reloads, word + kStop) == 2) st_relaxed(word + kFail, 1u);
                }
                made = n_acc = last_acc = 0;
                fresh = true;
                continue;  // the rest of the block
            }
            ++b;
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
        int s = 0, s_made = 0;
        uint32_t table = 0, table_made = 0, published = 0;
        // the last block gathered is complete: its draws' records, then its number
        auto publish = [&](uint32_t blocks) {
            __syncwarp();
            if (!with_next) {
                DrawRecord* out = reinterpret_cast<DrawRecord*>(smem + L.own_pairs + table_made * kOwnTable) + lane;
                if (lane < kStep) {
                    out->lnu = reinterpret_cast<const double*>(slot_of(s_made) + SL.lnu)[lane + 1];
                    out->pair1 = out->pair[lane + 1];
                    out->pair2 = out->pair[lane + 2];
                    out->same = reinterpret_cast<const uint32_t*>(slot_of(s_made) + SL.same)[lane];
                }
                __syncwarp();
            }
            if (lane == 0) st_release(made, blocks);
            published = blocks;
        };
        for (uint32_t b = 0;; ++b) {
            // the block's draws are made, and the reader has left the table's last block
            const bool now = static_cast<int32_t>(ld_relaxed(word + kProduced) - (b + draws)) >= 0 &&
                             (b < tables || static_cast<int32_t>(ld_relaxed(reader) - (b - tables + 1)) >= 0);
            if (__all_sync(kFull, now)) {
                __threadfence_block();
            } else {
                if (published < b) {  // complete what is in flight first
                    asm volatile("cp.async.wait_group 0;" ::: "memory");
                    publish(b);
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
            NextRecord* next = reinterpret_cast<NextRecord*>(smem + L.next_pairs + table * kNextTable);
            double* out = with_next ? next->pair
                                    : reinterpret_cast<DrawRecord*>(smem + L.own_pairs + table * kOwnTable)->pair;
            gather_pairs<kPrec>(J, ld, site < 0 ? 0 : site, scale, column, !with_next, out,
                                static_cast<int>((with_next ? sizeof(NextRecord) : sizeof(DrawRecord)) / 8), lane);
            if (with_next) {
                uint32_t mask = 0;
#pragma unroll 6
                for (int k = 0; k < kStep; ++k) {
                    const uint32_t lanes = __ballot_sync(kFull, __shfl_sync(kFull, site, k) == column);
                    mask = lane == k ? lanes : mask;
                }
                if (lane < kStep) next[lane].cross = mask;
            }
            asm volatile("cp.async.wait_group 1;" ::: "memory");  // the block before
            if (published < b) publish(b);
            s_made = s;
            table_made = table;
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
        uint32_t epochs = 0;
        for (uint32_t lists = 0;; ++lists) {
            bar_sync(kBarList, barrier_threads);
            const FlipRecord* list = flips + 32 * (lists & 1u);
            const int n = static_cast<int>(word[kCount + (lists & 1u)]);
            const uint32_t final = word[kFinal];
            const bool last = final != 0;
            // an epoch's end: the fields go to HBM as well
            double2* out = final == kFinalGood
                               ? reinterpret_cast<double2*>(v.fields + static_cast<size_t>(word[kSlot]) * ld)
                               : nullptr;
            // eight rows in flight, then the last flips by fours (the list is padded with m = 0); sixteen
            // in flight measured slower (85.0 against 82.9 us per epoch of the 8x8x8 workload)
            const int groups = (n + 3) >> 2;
#pragma unroll 1
            for (int p = me; p < pairs; p += threads) {
                const char* column = reinterpret_cast<const char*>(J) + static_cast<size_t>(p) * sizeof(PairT);
                double2 h = f2[p];
                int q = 0;
#pragma unroll 1
                for (; q + 2 <= groups; q += 2) apply_rows<kPrec, 8>(column, list + 4 * q, h);
                if (q < groups) apply_rows<kPrec, 4>(column, list + 4 * q, h);
                f2[p] = h;
                if (out) out[p] = h;
            }
            if (!last) {
                bar_arrive(kBarFields, barrier_threads);
                continue;
            }
            settle(kSettled);
            const uint32_t go = wait_go(++epochs);
            if (go & kGoLeave) break;
            if (go & kGoReload) {
                load_fields(static_cast<int>(word[kSlot]), me, threads);
                settle(kReloaded);
            }
        }
    } else if (kCollect && role == kRoleWarps + field_warps) {
        // ---- the books: pilot statistics (src/wang_landau.cpp:272-276, 317-342) ----------------
        // Follows the walker's entries and keeps, in the reference's order, the squared displacements
        // and sample counts of the bins, the round trips and the representatives, on an energy and
        // spins of its own, so that none of it is on the walker's chain.
        double* sq_s = reinterpret_cast<double*>(smem + L.sq);
        uint64_t* ds_s = reinterpret_cast<uint64_t*>(smem + L.ds);
        int8_t* spins = reinterpret_cast<int8_t*>(smem + L.book_spins);
        EpochIo* io = reinterpret_cast<EpochIo*>(smem + L.io);
        const double lower = window_lower(v, wb), upper = window_lower(v, wb + nbins);
        double E = st_s->energy;
        int32_t rt_state = st_s->rt_state;
        uint64_t trips = st_s->round_trips;
        const size_t rep0 = static_cast<size_t>(w) * kRepresentatives + (lane < kRepresentatives ? lane : 0);
        const double target = v.rep_target[rep0];
        double nearest = lane < kRepresentatives ? v.rep_dist[rep0] : -1.0;
        auto represent = [&]() {
            if (!__any_sync(kFull, fabs(E - target) < nearest)) return;
            warp_update_representatives(v, w, E, spins, lane);
            nearest = lane < kRepresentatives ? __ldcg(v.rep_dist + rep0) : -1.0;
        };
        auto load_book_spins = [&](int slot) {
            const int4* from = reinterpret_cast<const int4*>(v.spins + static_cast<size_t>(slot) * ld);
            for (int i = lane; i < (ld >> 4); i += 32) reinterpret_cast<int4*>(spins)[i] = __ldcg(from + i);
            __syncwarp();
        };
        load_book_spins(st_s->slot);
        for (int i = lane; i < nbins; i += 32) {
            sq_s[i] = v.sqdisp[boff + i];
            ds_s[i] = v.dsamples[boff + i];
        }
        __syncwarp();
        if (st_s->rep_pending) represent();  // a replica exchange changed the configuration
        bool complete = true;
        auto save = [&]() {  // after an epoch that was made: should the next one fail, these are what it started from
            if (!complete || !io->good) return;
            for (int i = lane; i < nbins; i += 32) {
                v.sqdisp[boff + i] = sq_s[i];
                v.dsamples[boff + i] = ds_s[i];
            }
        };
        int s = 0, k = 0;
        uint32_t epochs = 0;
        for (uint32_t b = 0;;) {
            const int32_t* sites = reinterpret_cast<const int32_t*>(slot_of(s) + SL.site);
            const Attempts* block = attempts + (b & 1u);
            int e = 0;
            // The look-ahead warp clears this buffer of the entries of two blocks before when it is through with
            // the last block, which is later than here where its fields come late (two walkers to an SM,
            // or thousands of sites).  It enters every block that the walker has ended, also after the walker
            // has stopped.
            bool stop = wait_at_least(word + kAheadIn, b, nullptr) != 0, gave_up = stop;
            while (!stop && k < kStep) {
                uint32_t x = ld_relaxed(&block->entry[e].x);
                for (uint32_t polls = 0; x == 0 && polls < kPolls; ++polls) {
                    x = ld_relaxed(&block->entry[e].x);
                    if (e == 0 && x == 0 && b != 0 && ld_relaxed(word + kBoundary) == b) x = kEntValid | kEntStop;
                }
                __syncwarp();
                __threadfence_block();
                gave_up = x == 0;
                stop = gave_up || (x & kEntStop) != 0;
                if (stop) break;
                if (!(x & kEntSkip)) {
                    const bool accepted = (x & 0x40000000u) != 0;
                    const int bin = static_cast<int>(ld_relaxed(&block->entry[e].y));
                    const double field = *reinterpret_cast<const volatile double*>(&block->field[e]);
                    const double m = __hiloint2double(static_cast<int>(x & 0xC0000000u), 0);
                    const double displacement = accepted ? m * field : 0.0;
                    if (lane == 0) {
                        sq_s[bin] += displacement * displacement;
                        ++ds_s[bin];
                        if (accepted) spins[sites[k]] = (x & 0x80000000u) ? -1 : 1;  // m = -2 * old spin
                    }
                    __syncwarp();
                    if (accepted) {
                        E = fma(m, field, E);
                        round_trip_update(E, lower, upper, P.round_trip_margin, rt_state, trips);
                        represent();
                    }
                }
                k += (x & kEntUniform) ? 2 : 1;
                ++e;
            }
            if (!stop) {
                __syncwarp();
                if (lane == 0) st_release(word + kBooked, b + 1);
                ++b;
                k -= kStep;
                s = s + 1 == slots ? 0 : s + 1;
                continue;
            }
            if (lane == 0) {
                if (gave_up) st_relaxed(word + kFail, 1u);
                io->rt_state = rt_state;
                io->trips = trips;
            }
            settle(kSettled);
            complete = complete && !gave_up;
            const uint32_t go = wait_go(++epochs);
            if (go & kGoLeave) break;
            save();
            if (go & kGoReload) {
                load_book_spins(static_cast<int>(word[kSlot]));
                E = st_s->energy;
                represent();
                settle(kReloaded);
            }
            rt_state = st_s->rt_state;
            trips = st_s->round_trips;
        }
        bar_sync(0, static_cast<int>(blockDim.x));  // every role has left
        save();
        return;
    }

    bar_sync(0, static_cast<int>(blockDim.x));  // every role has left
}

using AheadFn = void (*)(EngineView, WalkArgs, int, int, FusedEpochs);

template <int kPrec, bool kPow2, bool kAlone, bool kCollect>
AheadFn ahead_fn() {
    static SharedMemoryOptIn opt_in;
    check_cuda(opt_in(reinterpret_cast<const void*>(&sweep_ahead_kernel<kPrec, kPow2, kAlone, kCollect>)), "cudaFuncSetAttribute");
    return &sweep_ahead_kernel<kPrec, kPow2, kAlone, kCollect>;
}

template <int kPrec, bool kCollect>
AheadFn pick_ahead(bool pow2, bool alone) {
    if (alone) return pow2 ? ahead_fn<kPrec, true, true, kCollect>() : ahead_fn<kPrec, false, true, kCollect>();
    return pow2 ? ahead_fn<kPrec, true, false, kCollect>() : ahead_fn<kPrec, false, false, kCollect>();
}
template <int kPrec>
AheadFn pick_ahead(bool pow2, bool alone, bool collect) {
    return collect ? pick_ahead<kPrec, true>(pow2, alone) : pick_ahead<kPrec, false>(pow2, alone);
}

// Block records made ahead of the walker for a staging depth of 2^log draws.
int slots_of(int log) { return log == 5 ? kMaxSlots : kMinSlots; }

// How the kernel is launched for an engine; fn is null when the sweep does not serve it.
struct AheadLaunch {
    AheadFn fn = nullptr;
    unsigned threads = 0;
    size_t bytes = 0;
    int slots = 0, field_warps = 0, sms = 0;
};
AheadLaunch ahead_launch(const EngineView& v) {
    AheadLaunch l;
    if (v.p.nalivaiko || v.split_sweep) return l;
    const bool collect = v.p.collect != 0;
    if (v.csr && !v.rows64 && !v.rows32) return l;
    const bool scaled = v.precision == WLG_PRECISION_BF16;
    l.slots = slots_of(v.staging_log);
    l.bytes = ahead_layout(v.ld, v.max_window_bins, scaled, l.slots, collect).total;
    if (l.bytes > 227 * 1024) return l;
    int device = 0;
    check_cuda(cudaGetDevice(&device), "cudaGetDevice");
    check_cuda(cudaDeviceGetAttribute(&l.sms, cudaDevAttrMultiProcessorCount, device), "cudaDeviceGetAttribute");
    // With more walkers than SMs two CTAs share an SM and its registers: walkers that meet at every
    // exchange would otherwise take two rounds.  (A batch's engines do not meet and are each launched as if
    // alone: 96 x 2 walkers, four epochs of 8192 attempts, 8.5 ms as branches of a graph.)
    const bool pow2 = v.grid.pow2_width != 0, alone = v.walkers <= l.sms;
    l.fn = v.precision == WLG_PRECISION_FP32   ? pick_ahead<WLG_PRECISION_FP32>(pow2, alone, collect)
           : v.precision == WLG_PRECISION_BF16 ? pick_ahead<WLG_PRECISION_BF16>(pow2, alone, collect)
                                               : pick_ahead<WLG_PRECISION_FP64>(pow2, alone, collect);
    // one thread per pair of fields, up to eight warps
    l.field_warps = std::max(1, std::min(alone ? kMaxFieldWarps : kMaxFieldWarps - 1, (v.ld / 2 + 31) / 32));
    l.threads = static_cast<unsigned>(32 * warps_for(kRoleWarps + l.field_warps + (collect ? 1 : 0), alone));
    return l;
}

}  // namespace

// The staging depths wlg_engine_set_staging_ring accepts (log2 of the draws): those whose block records fit
// beside the walker, for dense systems of at most 1024 sites without pilot statistics or the Nalivaiko mask.
std::vector<int> staging_logs(const EngineView& v) {
    std::vector<int> out;
    if (v.csr || v.p.collect || v.p.nalivaiko || v.ld > 1024) return out;
    if (v.split_sweep) return {4, 5};
    for (int log = 4; log <= 5; ++log)
        if (ahead_layout(v.ld, v.max_window_bins, v.precision == WLG_PRECISION_BF16, slots_of(log), false).total <= 227 * 1024)
            out.push_back(log);
    return out;
}

bool sweep_ahead_serves(const EngineView& v) { return ahead_launch(v).fn != nullptr; }

bool launch_sweep_ahead(const EngineView& v, const WalkArgs& a, cudaStream_t stream) {
    const AheadLaunch l = ahead_launch(v);
    if (!l.fn) return false;
    l.fn<<<static_cast<unsigned>(a.count), l.threads, l.bytes, stream>>>(v, a, l.slots, l.field_warps, FusedEpochs{});
    check_cuda(cudaGetLastError(), "sweep_ahead_kernel");
    return true;
}

bool ahead_epochs_fit(const EngineView& v) { return v.walkers <= ahead_resident(v); }

int ahead_resident(const EngineView& v) {
    const AheadLaunch l = ahead_launch(v);
    if (!l.fn) return 0;
    int per_sm = 0;
    check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, reinterpret_cast<const void*>(l.fn),
                                                             static_cast<int>(l.threads), l.bytes),
               "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    return per_sm * l.sms;
}

void launch_ahead_epochs(const EngineView& v, const FusedEpochs& epochs, cudaStream_t stream) {
    AheadLaunch l = ahead_launch(v);
    WalkArgs a{};
    a.count = v.walkers;
    a.epoch_mode = 1;
    FusedEpochs fe = epochs;
    EngineView view = v;
    check_cuda(cudaMemsetAsync(fe.sync, 0, sizeof(FusedSync), stream), "memset");
    void* args[] = {&view, &a, &l.slots, &l.field_warps, &fe};
    check_cuda(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(l.fn), dim3(static_cast<unsigned>(v.walkers)),
                                           dim3(l.threads), args, l.bytes, stream),
               "sweep_ahead_kernel");
}

}  // namespace wlg
