// wf_wave.cuh -- slim persistent wavefront walker (diagonal sub-steps, sentinel hand-off).
//
// Only the discharge propagates downstream in a kinematic-wave sweep, so the walker carries
// nothing but the solve: per-node terms that do not depend on the upstream discharge are
// prepared by the per-cell kernels before the sweep, and every output that nothing downstream
// reads (water depths, storages, averages, soil-column updates) is finished by per-cell
// kernels after it. What remains on the critical path of a chain position is the gather of
// the upstream discharges and the solve.
//
// A warp takes items (a chunk's chain-member pairs, or a part of them) from a global ticket counter: a
// bounded number of the longest chains first, one to a warp, then the others in the plan's
// dependency order (chain length for plans without heavy-child hints), and walks each chain leaf ->
// chain end. Chain ends publish the discharge of each sub-step into end_q, which is filled with a
// sentinel bit pattern before the launch; a consumer reads the slot with a relaxed 64-bit load until
// the sentinel is gone (one round trip instead of flag-then-value). No value other than the published
// discharge itself crosses warps, so no acquire/release pairing is needed: 64-bit aligned stores and
// loads are single-copy atomic.
//
// Every wait is bounded by a wall-clock budget (globaltimer); a wait that runs out sets
// WF_DEV_SPIN_TIMEOUT in the device status word and all lanes abort.
#pragma once

#include <cstdint>
#include <cstring>

#include "wf_ff.cuh"
#include "wf_fields.cuh"

namespace wfv {

// The fill of end_q: a NaN, read as a double (the FP64 form, snow transport) or as a pair of floats (the
// split form). A NaN of that pattern from the inputs keeps it through FP64 arithmetic, so another
// pattern that is NaN in both readings is published in its place.
constexpr unsigned long long SENTINEL = 0xFFFFFFFFFFFFFFFFULL;
constexpr unsigned long long QUIET_NAN = 0x7FFFFFFF7FFFFFFFULL;
constexpr int MAX_GROUP = 16;  // sub-steps per launch of the slim walker

// The relaxed loads and stores of published discharges carry no ordering duty (a consumer uses
// only the value it reads), so they have no compiler memory clobber: a clobber would make the
// compiler reload every shared-memory value it holds in registers after each of them.
__device__ __forceinline__ unsigned long long ld_relaxed(const void* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void st_relaxed(void* p, unsigned long long v) {
    if (v == SENTINEL) v = QUIET_NAN;
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v));
}
__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ int32_t status_ld(const int32_t* s) {
    return *reinterpret_cast<const volatile int32_t*>(s);
}

// end_q index of chain `chain`, member m, sub-step s of the launch (members innermost, so a
// warp of 32 members reads 256 contiguous bytes). Each slot holds one packed double-FP32
// discharge (wf_ff.cuh).
__device__ __forceinline__ int64_t end_index(const WfDevGraph& g, int64_t chain, int m, int s) {
    return (chain * g.s_cap + s) * g.M + m;
}

// Whether a wait since t0 goes on. Called after a poll that failed: the order matters, a poll takes a round
// trip to L2 and so does the status word.
__device__ __forceinline__ bool wait_goes_on(const WfSweep& sw, uint64_t t0, int32_t* status) {
    if (status_ld(status) & WF_DEV_SPIN_TIMEOUT) return false;
    if (now_ns() - t0 <= sw.wait_ns) return true;
    atomicOr(status, WF_DEV_SPIN_TIMEOUT);
    return false;
}

// The word of chain lt (negative: none) at sub-step s; w holds the value loaded earlier (or the sentinel).
// False when the budget ran out or another lane aborted. A non-zero sw.wait_offset (test hook, 0 in
// production) makes every wait run out.
__device__ __forceinline__ bool await_one(const WfDevGraph& g, const WfSweep& sw, int32_t lt, int m, int s,
                                          unsigned long long& w, int32_t* status) {
    if (lt < 0) return true;
    const unsigned long long* p = reinterpret_cast<const unsigned long long*>(&g.end_q[end_index(g, lt, m, s)]);
    if (w == SENTINEL) w = ld_relaxed(p);
    if (w != SENTINEL && sw.wait_offset == 0) return true;
    const uint64_t t0 = now_ns();
    while (true) {
        __nanosleep(32);
        w = ld_relaxed(p);
        if (w != SENTINEL && sw.wait_offset == 0) return true;
        if (!wait_goes_on(sw, t0, status)) return false;
    }
}

// The words of the chains lt0 and lt1 (negative: none) at sub-step s, waited for together: for the FP64 form
// (daily overland flow of 160 x 160 cells 2.46 ms in turn, 2.27 together). The split form waits in turn
// (hourly steps of 1024 x 1024 cells: overland 2.57 ms together, 2.43 in turn; river 2.73 and 2.59).
__device__ __forceinline__ bool await_two(const WfDevGraph& g, const WfSweep& sw, int32_t lt0, int32_t lt1, int m, int s,
                                          unsigned long long& w0, unsigned long long& w1, int32_t* status) {
    auto missing = [&]() {
        if (lt0 >= 0 && w0 == SENTINEL) w0 = ld_relaxed(&g.end_q[end_index(g, lt0, m, s)]);
        if (lt1 >= 0 && w1 == SENTINEL) w1 = ld_relaxed(&g.end_q[end_index(g, lt1, m, s)]);
        return (lt0 >= 0 && (w0 == SENTINEL || sw.wait_offset != 0)) ||
               (lt1 >= 0 && (w1 == SENTINEL || sw.wait_offset != 0));
    };
    if (!missing()) return true;
    const uint64_t t0 = now_ns();
    while (true) {
        __nanosleep(32);
        if (!missing()) return true;
        if (!wait_goes_on(sw, t0, status)) return false;
    }
}

__device__ __forceinline__ void publish(const WfDevGraph& g, int64_t chain, int m, int s, wff::ff q) {
    st_relaxed(&g.end_q[end_index(g, chain, m, s)], wff::pack(q));
}

// Up to GROUP entries of a node's upstream list, for the nodes with more than two light children. Their
// chains are loaded together, then their words, then waited for together: one at a time, each entry took
// three dependent loads, and with 24 sub-steps in a warp some lane is at such a node in most steps of a
// long chain (daily overland flow: 64 x 64 cells in FP64 3.15 -> 2.70 ms, 40 uneven catchments in the
// split form 15.2 -> 12.4).
constexpr int GROUP = 4;
struct UpGroup {
    int32_t chain[GROUP];  // -1: the heavy child, -2: no entry
    unsigned long long word[GROUP];
};
// Entries from o on (o1: end of the list) of `chains` at sub-step s; the first `skip` light children are left out.
__device__ __forceinline__ bool gather_group(const WfDevGraph& g, const WfSweep& sw, const int32_t* chains, int32_t o,
                                             int32_t o1, int& skip, int m, int s, int32_t* status, UpGroup& u) {
#pragma unroll
    for (int i = 0; i < GROUP; ++i) u.chain[i] = o + i < o1 ? __ldg(chains + o + i) : -2;
#pragma unroll
    for (int i = 0; i < GROUP; ++i) {
        if (u.chain[i] >= 0 && --skip >= 0) u.chain[i] = -2;
        u.word[i] = u.chain[i] >= 0 ? ld_relaxed(&g.end_q[end_index(g, u.chain[i], m, s)]) : 0ull;
    }
    auto missing = [&]() {
        bool any = sw.wait_offset != 0;
#pragma unroll
        for (int i = 0; i < GROUP; ++i) any |= u.word[i] == SENTINEL;
        return any;
    };
    if (!missing()) return true;
    const uint64_t t0 = now_ns();
    while (true) {
        __nanosleep(32);
#pragma unroll
        for (int i = 0; i < GROUP; ++i)
            if (u.word[i] == SENTINEL) u.word[i] = ld_relaxed(&g.end_q[end_index(g, u.chain[i], m, s)]);
        if (!missing()) return true;
        if (!wait_goes_on(sw, t0, status)) return false;
    }
}

// Upstream inflow record of one node. A node at chain position k > 0 has its heavy child at
// position k - 1 (its discharge stays with the lane); its light children are chain ends of shorter
// chains. The first two light children come from the per-slot record (one 16-byte load, no dependent
// index loads), the rare further ones from the CSR list; the end_q words of the first two for the
// sub-step are prefetched (load_words), so a producer that finished earlier costs no round trip.
struct UpRec {
    int32_t lt0, lt1;     // chains of light children 0 and 1 (-1: none)
    float w_lt0, w_lt1;   // their weights
    float w_hv;           // weight of the heavy child
    int32_t n_lt;         // light children in all
};
// Weighted upstream sum at sub-step s: qin = sum w*q (w = 1 - fraction to river on land, 1 on
// rivers) in double-FP32, heavy child first, then the light children. `qh` is the heavy child's
// word of this sub-step, `heavy` whether the node has one (chain position > 0); w0 / w1 are the
// end_q words of light children 0 / 1 at sub-step s loaded earlier (SENTINEL when not loaded or
// not yet published).
template <bool WEIGHTED>
__device__ __forceinline__ bool gather_w(const WfDevGraph& g, const WfSweep& sw, const UpRec& r, unsigned long long w0,
                                         unsigned long long w1, int64_t slot, int m, int s, bool heavy,
                                         unsigned long long qh, int32_t* status, wff::ff& qin) {
    wff::ff acc = {0.0f, 0.0f};
    if (heavy) {
        const wff::ff q = wff::unpack(qh);
        acc = WEIGHTED ? wff::mul(q, r.w_hv) : q;
    }
    if (!await_one(g, sw, r.lt0, m, s, w0, status)) return false;
    if (r.lt0 >= 0) {
        const wff::ff q = wff::unpack(w0);
        acc = WEIGHTED ? wff::add(acc, wff::mul(q, r.w_lt0)) : wff::add(acc, q);
    }
    if (!await_one(g, sw, r.lt1, m, s, w1, status)) return false;
    if (r.lt1 >= 0) {
        const wff::ff q = wff::unpack(w1);
        acc = WEIGHTED ? wff::add(acc, wff::mul(q, r.w_lt1)) : wff::add(acc, q);
    }
    if (r.n_lt > 2) {  // further light children, in up-list order after the first two
        int skip = 2;
        const int32_t o1 = __ldg(g.up_ptr + slot + 1);
        for (int32_t o = __ldg(g.up_ptr + slot); o < o1; o += GROUP) {
            UpGroup u;
            if (!gather_group(g, sw, g.up_chain, o, o1, skip, m, s, status, u)) return false;
#pragma unroll
            for (int i = 0; i < GROUP; ++i) {
                if (u.chain[i] < 0) continue;
                const wff::ff q = wff::unpack(u.word[i]);
                acc = WEIGHTED ? wff::add(acc, wff::mul(q, __ldg(g.up_wf + o + i))) : wff::add(acc, q);
            }
        }
    }
    qin = acc;
    return true;
}

// The end_q words of light children 0 and 1 (chains lt0, lt1) at sub-step s (SENTINEL for a missing
// child); a load that finds the producer not yet done also returns the sentinel.
__device__ __forceinline__ void load_words(const WfDevGraph& g, int m, int32_t lt0, int32_t lt1, int s,
                                           unsigned long long& w0, unsigned long long& w1) {
    w0 = lt0 >= 0 ? ld_relaxed(&g.end_q[end_index(g, lt0, m, s)]) : SENTINEL;
    w1 = lt1 >= 0 ? ld_relaxed(&g.end_q[end_index(g, lt1, m, s)]) : SENTINEL;
}

// ---- items, positions --------------------------------------------------------------------------
//
// Work items are parts of a chunk's chain-member pairs in dependency (chain length) order. One ticket
// takes a batch of consecutive short items (chunk length <= SHORT_LEN: the bulk of a drainage forest is
// short tributary chains, and a ticket per chain would pay the ticket, the descriptor loads and the
// prefetch start-up per chain), or a single longer item. The items of a batch are walked as one
// sequence of positions, so the prefetch runs on across item boundaries. Order and progress are
// unchanged: a batch holds consecutive items and a chain waits only for chains that come earlier in
// the order, or for chains of its own chunk that end before it needs them (wf_plan.cpp: the lanes
// of a warp advance together).
//
// SL lanes (a power of two) serve a chain-member pair, of which the first SU = min(SL, S) work. Sub-step
// s of the node at chain position k depends only on (k - 1, s), its heavy child, and (k, s - 1), its own
// previous state: in round r lane l takes sub-step r SU + l and at time step t works on position
// t - l. A chain of L positions takes ceil(S / SU) rounds of L + SU - 1 time steps instead of L S.
constexpr int BATCH = 2;
constexpr int SHORT_LEN = 8;

struct Batch {  // per-warp shared descriptors of the items of the current ticket
    struct Item {
        int64_t slot0;           // slot of position 0 of the item's first pair
        int32_t chain, m, Gc, L;  // chain and member of that pair, chains per position, positions
    } item[BATCH];
    int32_t len[BATCH][32];  // length of each lane's chain (0: the lane idles in that item)
};

// A lane's pair within an item: what its slot, chain and member add to the item's first pair
struct LanePair {
    int32_t gi, m;  // chains and members
};

// A position of a lane's sequence, resolved from the item descriptors
struct Pos {
    int64_t slot;
    int32_t m, chain, flags;  // flags 0: no node here
};
constexpr int32_t P_VALID = 1, P_END = 2, P_HEAVY = 4;

// Walks over the positions (item it, chain position k) of a ticket
struct Cursor {
    int it, k, L;
    __device__ __forceinline__ void reset(const Batch* b, int count) {
        it = k = 0;
        L = b->item[0].L;
    }
    __device__ __forceinline__ void advance(const Batch* b, int count) {
        if (++k < L || it >= count) return;
        k = 0;
        if (++it < count) L = b->item[it].L;
    }
    __device__ __forceinline__ void resolve(const Batch* b, int count, const LanePair& lp, Pos& p) const {
        p.flags = 0;
        if (it >= count) return;
        const int len = b->len[it][threadIdx.x & 31u];
        if (k >= len) return;
        const Batch::Item& d = b->item[it];
        p.slot = d.slot0 + (int64_t)(k * d.Gc + lp.gi);
        p.m = d.m + lp.m;
        p.chain = d.chain + lp.gi;
        p.flags = P_VALID | (k == len - 1 ? P_END : 0) | (k > 0 ? P_HEAVY : 0);
    }
};

// Descriptors of the `count` items from `first` (ipc items per chunk, SL lanes per pair) for a warp;
// lanes with `use` false idle. npos: positions of the sequence. False when no lane has work.
__device__ __forceinline__ bool fill_batch(const WfDevGraph& g, int64_t first, int count, int SL, int64_t ipc, bool use,
                                           Batch* wb, LanePair& lp, int& npos) {
    const unsigned lane = threadIdx.x & 31u;
    const int M = g.M, J = 32 / SL, j = (int)lane / SL;
    const int gi = M <= J ? j / M : 0;  // M is a power of two or a multiple of 32
    lp.gi = gi;
    lp.m = M <= J ? j - gi * M : j;
    if ((int)lane < count) {
        const int64_t item = first + lane, chunk = item / ipc;
        const int p0 = (int)(item - chunk * ipc) * J;
        const int gi0 = M <= 32 ? p0 / M : 0;
        Batch::Item& d = wb->item[lane];
        d.slot0 = g.chunk_base[chunk] + gi0;
        d.chain = (int32_t)g.chunk_chain0[chunk] + gi0;
        d.m = M <= 32 ? p0 - gi0 * M : p0;
        d.Gc = g.chunk_g[chunk];
        d.L = g.chunk_len[chunk];
        wb->len[lane][0] = d.Gc - gi0;  // chains left in the chunk from the item's first (read below)
    }
    __syncwarp();
    int left[BATCH];
#pragma unroll
    for (int it = 0; it < BATCH; ++it) left[it] = it < count ? wb->len[it][0] : 0;
    __syncwarp();
    npos = 0;
    int work = 0;
#pragma unroll
    for (int it = 0; it < BATCH; ++it) {
        if (it >= count) break;
        const Batch::Item& d = wb->item[it];
        int len = 0;
        if (use && gi < left[it] && d.m + lp.m < M) len = g.chain_len[d.chain + gi];
        wb->len[it][lane] = len;
        work |= len;
        npos += d.L;
    }
    __syncwarp();
    return __any_sync(0xffffffffu, work > 0);
}

template <class T>
__device__ __forceinline__ void shfl_up_pod(T& v, int width) {
    static_assert(sizeof(T) % 4 == 0, "shuffled structs are whole 32-bit words");
    uint32_t w[sizeof(T) / 4];
    memcpy(w, &v, sizeof(T));
#pragma unroll
    for (int i = 0; i < (int)(sizeof(T) / 4); ++i) w[i] = __shfl_up_sync(0xffffffffu, w[i], 1, width);
    memcpy(&v, w, sizeof(T));
}

// ---- staged walk ---------------------------------------------------------------------------------
//
// The lead lane of a pair (lane 0 of its SL) copies the inputs of the position RING_D ahead into a
// per-warp ring in shared memory with asynchronous copies (cp.async, one commit group per position,
// issued whether or not the lane has work there). The light children's words are loaded two positions
// ahead from the staged records, so the copies issued in a step are waited for at the start of the
// next: they have one position to arrive, the words two. Each
// lane reads back only what it copied itself, so the waits are per thread (cp.async.wait_group) and
// no barrier is involved. At the end of a time step every lane hands what the node's next sub-step needs
// (Pass, its state, the words of its light children, loaded during the step) to the next lane with warp
// shuffles; launches of one sub-step skip the hand-over.
//
// A position's bookkeeping is on the critical path of a chain as much as its solve. Its inputs are
// 16-byte vectors (4 or 5 copies instead of 12 to 15 words), and its index arithmetic is resolved once, when
// it is staged, from per-ticket descriptors, and kept in the ring beside them. Measured on the hourly step
// of a 1024 x 1024 domain, longest chain 1867 positions: subsurface 2.05 -> 1.60 ms, overland 2.9 -> 2.5,
// river (4 sub-steps) 3.2 -> 2.8, against words staged singly and resolved twice; of the 1600 cycles that
// a subsurface position takes, the solve and the wait for the tributaries are two thirds.
//
// Phys interface:
//   struct In;                                            inputs of a node, including an UpRec `up`
//   struct St;                                            state carried from sub-step to sub-step
//   struct Pass;                                          what later sub-steps need of the inputs (pack, unpack)
//   static constexpr int kVecs;                           16-byte input vectors per position
//   static constexpr bool kWeighted;                      the land graph's weights (else all 1)
//   void copy(int64_t slot, int64_t e, float4* v)         starts their copies to v[32 i] (cpa)
//   void from_vecs(const float4* v, In&)                  the inputs from the staged vectors (v[32 i])
//   void start(const In&, St&)                            state at the start of a round
//   bool active(m, first)                                 whether member m takes the launch's sub-step;
//                                                         adaptive sub-steps: first of the model step
//   bool gather(const In&, const St&, w0, w1, slot, m, s, heavy, qh_in, qin, tr)
//     the inflow of sub-step s: w0 / w1 the light children's end_q words (or SENTINEL), qh_in the
//     heavy child's packed discharge. False to abort.
//   void sub(const In&, St&, qin, tr, slot, e, m, s, chain, is_end, qh_out)
//     the sub-step after its gather; qh_out the node's packed discharge
//   void finish(const St&, e, add_stored)                 stores after the last sub-step of a round
//                                                         (add_stored: add the stored cumulative sums)
// The copies and their commit carry no compiler memory clobber (it would force every shared
// value held in registers to be reloaded after each copy); cp.async.wait_group has one, so the
// reads of a slot stay after the wait that covers it, and a slot's earlier reads stay before the
// next wait, which precedes its refill.
// positions staged ahead: one for the copies to arrive (1000 cycles and more, a memory round trip) and the
// two for the words
constexpr int RING_D = 3;
constexpr int RING_R = RING_D + 1;  // ring slots (the slot refilled is the one read a position ago)

__device__ __forceinline__ void cpa16(void* smem, const void* gmem) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(gmem));
}
// a short vector goes to the start of a 16-byte slot
__device__ __forceinline__ void cpa(float4* smem, const float4* gmem) { cpa16(smem, gmem); }
__device__ __forceinline__ void cpa(float4* smem, const float2* gmem) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(gmem));
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void cpa_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cpa_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Bytes of one warp: its descriptors, and per ring slot kVecs input vectors, the record and the resolved
// position of 32 lanes.
__host__ __device__ constexpr size_t lean_warp_bytes(int vecs) {
    return (sizeof(Batch) + 15) / 16 * 16 + (size_t)RING_R * (vecs + 2) * 512;
}
__host__ __device__ constexpr size_t lean_smem(int threads, int vecs) {
    return (size_t)(threads / 32) * lean_warp_bytes(vecs);
}

template <class Phys, bool MULTI>
__device__ __forceinline__ bool ticket(const WfDevGraph& g, const WfSweep& sw, Phys& phys, int32_t* status, int count,
                                       int SL, const LanePair& lp, int npos, Batch* wb, float4* ring) {
    using In = typename Phys::In;
    using St = typename Phys::St;
    constexpr int KV = Phys::kVecs;
    const unsigned lane = threadIdx.x & 31u;
    const int M = g.M;
    const int sl = (int)lane & (SL - 1);
    const int SU = MULTI ? min(SL, sw.S) : 1;
    const int rounds = MULTI ? (sw.S + SU - 1) / SU : 1;
    const bool lead = sl == 0;
    if (status_ld(status) & WF_DEV_SPIN_TIMEOUT) return false;
    ring += lane;
    auto vecs_of = [&](int r) { return ring + r * (KV + 2) * 32; };
    auto rec_of = [&](int r) { return reinterpret_cast<int4*>(ring + (r * (KV + 2) + KV) * 32); };
    auto pos_of = [&](int r) { return reinterpret_cast<int4*>(ring + (r * (KV + 2) + KV + 1) * 32); };
    for (int r = 0; r < rounds; ++r) {
        const int s = r * SU + sl, s0 = r * SU;
        const bool works = sl < SU && s < sw.S;
        const bool last_lane = (s == sw.S - 1) || (sl == SU - 1);
        Cursor sc;  // staging cursor, RING_D positions ahead
        sc.reset(wb, count);
        int slot_s = 0;  // ring slot of the position staged next
        auto stage = [&]() {
            if (lead) {
                Pos p;
                sc.resolve(wb, count, lp, p);
                int4 v = make_int4(0, 0, 0, 0);
                if (p.flags) {
                    phys.copy(p.slot, p.slot * M + p.m, vecs_of(slot_s));
                    cpa16(rec_of(slot_s), &g.up_rec[p.slot]);
                    v = make_int4((int)(p.slot & 0xffffffff), (int)(p.slot >> 32) | p.flags << 28, p.m, p.chain);
                }
                *pos_of(slot_s) = v;
                sc.advance(wb, count);
            }
            slot_s = (slot_s + 1) & (RING_R - 1);
            cpa_commit();
        };
        static_assert((RING_R & (RING_R - 1)) == 0, "the ring slots wrap by a mask");
        // the light children's words of the position in ring slot k (issued, not awaited)
        auto look = [&](int k, unsigned long long& a, unsigned long long& b) {
            if (!lead) return;
            const int4 v = *pos_of(k);
            if (!v.y) return;
            const int4 q = *rec_of(k);
            load_words(g, v.z, q.x, q.y, s0, a, b);
        };
#pragma unroll
        for (int d = 0; d < RING_D; ++d) stage();
        cpa_wait<RING_D - 2>();
        unsigned long long a0 = SENTINEL, b0 = SENTINEL, a1 = SENTINEL, b1 = SENTINEL, a2 = SENTINEL, b2 = SENTINEL;
        look(0, a0, b0);
        look(1, a1, b1);
        In x;
        St st;
        int4 ps = make_int4(0, 0, 0, 0);  // the node in hand, packed as in the ring
        unsigned long long w0 = SENTINEL, w1 = SENTINEL, hq = 0ull;
        bool ok = true;
        int tt = 0;
        const int steps = npos + SU - 1;
        // One time step: ac / bc hold position t's words (looked up two steps ago), af / bf receive those
        // of position t + 2. The three register sets rotate by unrolling (below) rather than by copies: a
        // copy of a register whose load is in flight would wait for it.
        auto step = [&](unsigned long long& ac, unsigned long long& bc, unsigned long long& af,
                        unsigned long long& bf) -> bool {
            if (tt >= steps) return false;
            cpa_wait<RING_D - 3>();  // every group, up to position t + 2, complete
            look((tt + 2) & (RING_R - 1), af, bf);
            if (lead) {
                const int k = tt & (RING_R - 1);
                ps = *pos_of(k);
                if (ps.y) {
                    phys.from_vecs(vecs_of(k), x);
                    const int4 q = *rec_of(k);
                    x.up.lt0 = q.x;
                    x.up.lt1 = q.y;
                    x.up.w_lt0 = Phys::kWeighted ? __int_as_float(q.z) : 1.0f;
                    x.up.w_lt1 = Phys::kWeighted ? __int_as_float(q.w) : 1.0f;
                    if (!Phys::kWeighted) x.up.w_hv = 1.0f;
                    w0 = ac;
                    w1 = bc;
                    phys.start(x, st);
                }
            }
            stage();
            unsigned long long v0 = SENTINEL, v1 = SENTINEL;  // words of sub-step s + 1 for the next lane
            const bool here = ps.y && works;
            const int flags = (unsigned)ps.y >> 28, m = ps.z, chain = ps.w;
            const int64_t slot = ((int64_t)(ps.y & 0x0fffffff) << 32) | (uint32_t)ps.x;
            bool first_of_step = sw.first == 0;
            const bool acts = here && phys.active(m, first_of_step);
            if (here && MULTI && sl + 1 < SU && s + 1 < sw.S) load_words(g, m, x.up.lt0, x.up.lt1, s + 1, v0, v1);
            wff::ff qin = {0.0f, 0.0f}, tr = {0.0f, 0.0f};
            if (acts) ok = phys.gather(x, st, w0, w1, slot, m, s, (flags & P_HEAVY) != 0, hq, qin, tr);
            // The lanes meet after their waits: lanes that wait differently would otherwise run the rest of
            // the step group by group (daily steps of 40 uneven catchments: overland 12.4 -> 9.1 ms, river
            // 12.4 -> 9.5).
            if (__any_sync(0xffffffffu, !ok)) {
                ok = false;
                return false;
            }
            if (acts) {
                const int64_t e = slot * M + m;
                phys.sub(x, st, qin, tr, slot, e, m, s, chain, (flags & P_END) != 0, hq);
                if (last_lane) phys.finish(st, e, r > 0 || !first_of_step);
            }
            __syncwarp();
            if constexpr (MULTI) {
                if (SL > 1) {  // hand the node to the next lane
                    typename Phys::Pass pass;
                    phys.pack(x, pass);
                    shfl_up_pod(pass, SL);
                    phys.unpack(pass, x);
                    int4 up = make_int4(x.up.lt0, x.up.lt1, __float_as_int(x.up.w_lt0), __float_as_int(x.up.w_lt1));
                    if constexpr (Phys::kWeighted) {
                        shfl_up_pod(up, SL);
                        x.up.w_lt0 = __int_as_float(up.z);
                        x.up.w_lt1 = __int_as_float(up.w);
                    } else {
                        up.x = __shfl_up_sync(0xffffffffu, up.x, 1, SL);
                        up.y = __shfl_up_sync(0xffffffffu, up.y, 1, SL);
                    }
                    x.up.lt0 = up.x;
                    x.up.lt1 = up.y;
                    shfl_up_pod(st, SL);
                    shfl_up_pod(ps, SL);
                    w0 = __shfl_up_sync(0xffffffffu, v0, 1, SL);
                    w1 = __shfl_up_sync(0xffffffffu, v1, 1, SL);
                }
            }
            ++tt;
            return true;
        };
        while (step(a0, b0, a2, b2) && step(a1, b1, a0, b0) && step(a2, b2, a1, b1)) {
        }
        cpa_wait_all();  // the ring is refilled by the next round or ticket
        __syncwarp();    // and the round's stores are read by the next round's copies
        if (!ok) return false;
    }
    return true;
}

// Tickets: the last p_chunks chunks (one long chain each) longest first, with SLp lanes per pair, then
// the other chunks in dependency order, the short ones with SLs lanes in batches of `batch`, the rest
// with SLr lanes.
template <class Phys, bool MULTI>
__device__ __forceinline__ void walk(Phys& phys, int64_t p_chunks, int SLp, int SLs, int SLr, int batch, int32_t* status) {
    extern __shared__ __align__(16) unsigned char lean_ring[];
    const WfDevGraph& g = phys.g;
    const WfSweep& sw = phys.sw;
    const unsigned lane = threadIdx.x & 31u;
    unsigned char* mine = lean_ring + (size_t)(threadIdx.x >> 5) * lean_warp_bytes(Phys::kVecs);
    Batch* wb = reinterpret_cast<Batch*>(mine);
    float4* ring = reinterpret_cast<float4*>(mine + (sizeof(Batch) + 15) / 16 * 16);
    const int64_t ipp = wf_items_per_chunk(1, g.M, SLp), ips = wf_items_per_chunk(g.G, g.M, SLs),
                  ipr = wf_items_per_chunk(g.G, g.M, SLr);
    const int64_t nd = p_chunks * ipp, rest = g.n_chunks - p_chunks;
    const int64_t short_chunks = min(g.n_short_chunks, rest), n_short = short_chunks * ips;
    const int64_t n_sb = (n_short + batch - 1) / batch;
    const int64_t total = nd + n_sb + (rest - short_chunks) * ipr;
    while (true) {
        unsigned long long t0 = 0;
        if (lane == 0) t0 = atomicAdd(g.ticket, 1ULL);
        const int64_t t = (int64_t)__shfl_sync(0xffffffffu, t0, 0);
        if (t >= total) return;
        int64_t first = g.n_chunks * ipp - 1 - t, ipc = ipp;
        int count = 1, SL = SLp, npos;
        if (t >= nd) {
            const int64_t v = t - nd;
            const bool is_short = v < n_sb;
            first = is_short ? v * batch : short_chunks * ipr + (v - n_sb);
            if (is_short) count = (int)min((int64_t)batch, n_short - first);
            SL = is_short ? SLs : SLr;
            ipc = is_short ? ips : ipr;
        }
        LanePair lp;
        if (!fill_batch(g, first, count, SL, ipc, MULTI || (lane & (SL - 1)) == 0, wb, lp, npos)) continue;
        if (!ticket<Phys, MULTI>(g, sw, phys, status, count, SL, lp, npos, wb, ring)) return;
    }
}

}  // namespace wfv
