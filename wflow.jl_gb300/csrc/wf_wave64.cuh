// wf_wave64.cuh -- slim persistent wavefront walker of the FP64 plain form.
//
// Only the discharge propagates downstream in a kinematic-wave sweep. A chain position costs a warp
// 64 cycles per FP64 instruction (wf_math.cuh), and chains are as long as the catchment is deep, so
// the walker executes nothing but what depends on the upstream discharge: the gather, the solve and,
// when the launch holds several sub-steps, the terms of the node's next one. The terms that the
// previous state gives (u = Q^0.2 and the first Newton iterate's residual, derivative and
// reciprocal) are prepared by a per-cell kernel before the sweep; depths, storages, averages and the
// soil column are finished by another after it. Every operation is the reference's, in its order,
// wherever it runs, so the results are those of a plain sweep bit for bit.
//
// Schedule: the diagonal one of wf_wave.cuh. SL lanes serve a chain-member pair, lane l
// takes sub-step r SL + l of round r and at time t works on position t - l; the node's state goes from
// lane to lane by warp shuffles, the heavy child's discharge stays in the lane. Launches of one
// sub-step (SL = 1) skip the hand-over. Chain ends publish their discharge's bits into end_q, filled
// with a sentinel before the launch (wf_wave.cuh await_two).
//
// The loads of a position (inputs, light children's words) are issued one position ahead, its
// upstream record two ahead: a position takes 3000 cycles and more, several times a memory round
// trip.
#pragma once

#include "wf_math.cuh"
#include "wf_wave.cuh"

namespace wfz {

using wfv::SENTINEL;

// Upstream record of a node (up_rec64): the chains of the first two light children (-1 none), flags
// with the number of light children, and where its upstream list starts. The reference adds the inflows
// in ascending cell order: with up to two light children that order only matters when the heavy child is
// the last of three.
constexpr int32_t REC_HEAVY_LAST = 1;
constexpr int32_t REC_WEIGHTED = 2;     // land: some child sends a fraction of its discharge to the river
constexpr int32_t REC_NO_INFLOW = 4;    // land: no surface flow width, the overland inflow does not count
constexpr int32_t REC_ABSTRACTION = 8;  // river: a negative external inflow, limited by the storage
constexpr int REC_LIGHTS = 8;           // flags: number of light children from this bit on
struct Rec {
    int32_t lt0, lt1, flags, list;
    __device__ __forceinline__ int n_lt() const { return flags >> REC_LIGHTS; }
};

__device__ __forceinline__ Rec load_rec(const WfDevGraph& g, int64_t slot) {
    const int4 v = g.up_rec64[slot];
    return {v.x, v.y, v.z, v.w};
}

// What the gather of the position after the next reads besides the words, into L1
template <bool LAND>
__device__ __forceinline__ void prefetch_lists(const WfDevGraph& g, int64_t slot, const Rec& r) {
    auto l1 = [](const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); };
    if (r.n_lt() > 2) {
        l1(g.up_chain + r.list);
        if (LAND) {
            l1(g.up_w + r.list);
            l1(g.up_fr + r.list);
        }
    } else if (LAND && (r.flags & REC_WEIGHTED)) {
        l1(g.up_w64 + slot * 6);
        l1(g.up_w64 + slot * 6 + 5);
    }
}

__device__ __forceinline__ void load_words(const WfDevGraph& g, int m, const Rec& r, int s, unsigned long long& w0,
                                           unsigned long long& w1) {
    w0 = r.lt0 >= 0 ? wfv::ld_relaxed(&g.end_q[wfv::end_index(g, r.lt0, m, s)]) : SENTINEL;
    w1 = r.lt1 >= 0 ? wfv::ld_relaxed(&g.end_q[wfv::end_index(g, r.lt1, m, s)]) : SENTINEL;
}

__device__ __forceinline__ void publish(const WfDevGraph& g, int64_t chain, int m, int s, double q) {
    wfv::st_relaxed(&g.end_q[wfv::end_index(g, chain, m, s)], wfm::to_bits(q));
}

// Sum of the heavy child's term (heavy) and the light ones in the reference's order (n light terms)
__device__ __forceinline__ double sum_up(const Rec& r, bool heavy, double h, double a, double b) {
    if (r.lt0 < 0) return heavy ? h : 0.0;
    if (!heavy) return r.lt1 < 0 ? a : a + b;
    if (r.lt1 < 0) return h + a;
    return (r.flags & REC_HEAVY_LAST) ? (a + b) + h : (h + a) + b;
}

// Inflow of a node at sub-step s: qin = sum of the upstream discharges (LAND: of the part that does
// not go to the river), and with TR tr = sum of the parts that go to the river. hq is the heavy
// child's discharge (heavy: it has one), w0 / w1 the light children's words loaded earlier.
template <bool LAND, bool TR>
__device__ __forceinline__ bool gather(const WfDevGraph& g, const WfSweep& sw, const Rec& r, unsigned long long w0,
                                       unsigned long long w1, int64_t slot, int m, int s, bool heavy, double hq,
                                       int32_t* status, double& qin, double& tr) {
    tr = 0.0;
    if (r.n_lt() > 2) {
        double acc = 0.0;
        int skip = 0;
        const int32_t o1 = r.list + r.n_lt() + (heavy ? 1 : 0);
        for (int32_t o = r.list; o < o1; o += wfv::GROUP) {
            double wt[wfv::GROUP] = {}, fr[wfv::GROUP] = {};
            if (LAND)
#pragma unroll
                for (int i = 0; i < wfv::GROUP; ++i)
                    if (o + i < o1) {
                        wt[i] = __ldg(g.up_w + o + i);
                        if (TR) fr[i] = __ldg(g.up_fr + o + i);
                    }
            wfv::UpGroup u;
            if (!wfv::gather_group(g, sw, g.up_chain, o, o1, skip, m, s, status, u)) return false;
#pragma unroll
            for (int i = 0; i < wfv::GROUP; ++i) {
                if (u.chain[i] < -1) continue;
                const double q = u.chain[i] < 0 ? hq : wfm::from_bits(u.word[i]);
                if (LAND) {
                    acc = acc + q * wt[i];
                    if (TR) tr = tr + q * fr[i];
                } else {
                    acc = acc + q;
                }
            }
        }
        qin = acc;
        return true;
    }
    if (!wfv::await_two(g, sw, r.lt0, r.lt1, m, s, w0, w1, status)) return false;
    double a = wfm::from_bits(w0), b = wfm::from_bits(w1);  // read only where there is a child
    if (LAND && (r.flags & REC_WEIGHTED)) {
        // {1 - fr, fr} of the heavy child and light children 0 and 1
        const double2* w = reinterpret_cast<const double2*>(g.up_w64 + slot * 6);
        const double2 wh = __ldg(w), wa = __ldg(w + 1), wb = __ldg(w + 2);
        if (TR) tr = sum_up(r, heavy, hq * wh.y, a * wa.y, b * wb.y);
        hq = hq * wh.x;
        if (r.lt0 >= 0) a = a * wa.x;
        if (r.lt1 >= 0) b = b * wb.x;
    }
    qin = sum_up(r, heavy, hq, a, b);
    return true;
}

// ---- kinematic wave for surface flow (routing/surface/surface_process.jl:24-70) ------------------

constexpr double MIN_FLOW_QROOT = 0x1.0c6f7a0b5ed8ap-20;  // 1e-30^0.2 (routing/utils.jl:2)

// What the solve needs of the node's previous discharge: u = q^0.2, A = alpha u^3, and of the first
// Newton iterate u (u > 0) P = u^3 (dt_dx u^2 + alpha), the derivative df and 1 / df (rcp_kept).
struct KwState {
    double u, A, P, df, rdf;
};

__device__ __forceinline__ void kw_state(double q_prev, double dt_dx, double alpha, double c1, double c2, KwState& k) {
    k.u = wfm::lt_(q_prev, 0.0) || wfm::isnan_(q_prev) ? 0.0 : wfm::pow(q_prev, 0.2);
    k.A = alpha * k.u * k.u * k.u;
    k.P = k.df = 0.0;
    k.rdf = 0.0;
    if (wfm::gt0_(k.u)) {
        const double u2 = k.u * k.u;
        const double u3 = u2 * k.u;
        k.P = u3 * (dt_dx * u2 + alpha);
        k.df = u2 * (c1 * u2 + c2);
        k.rdf = wfm::rcp_kept(k.df);
    }
}

// |f| <= 1e-12, the solve's stop (false for NaN)
__device__ __forceinline__ bool converged(double f) {
    return (wfm::to_bits(f) & 0x7fffffffffffffffULL) <= 0x3d719799812dea11ULL;
}

// cterm < -1e-12: then f(u) = u^3 (dt_dx u^2 + alpha) - cterm is above 1e-12 for every u > 0, so no
// iterate passes the stop; each Newton step from u > 0 goes down, in the end to u <= 0, which the solve
// replaces by MIN_FLOW_QROOT, and the step from there (f / f' >= 1e-12 / (3e-12 alpha + ...) > 1e-6 as
// long as alpha and dt_dx are below 1e4) repeats it: the end of the iteration. A step from a negative
// first iterate stays on the side of the negative root and ends there as well.
__device__ __forceinline__ bool no_root(double cterm, double dt_dx, double alpha) {
    return wfm::to_bits(cterm) > 0xbd719799812dea11ULL && wfm::to_bits(cterm) < 0xfff0000000000000ULL &&
           wfm::f32_of(alpha) < 1e4f && wfm::f32_of(dt_dx) < 1e4f;
}

// Discharge for cterm = dt/dx q_in + alpha u^3 + dt q_lat; u is the final iterate (at least
// MIN_FLOW_QROOT). The first iteration is the prepared one: 5 FP64 instructions, the later ones 16,
// the last residual 6.
__device__ __forceinline__ double kw_solve(const KwState& k, double cterm, double dt_dx, double alpha, double c1,
                                           double c2, double& u_out) {
    double u, u2 = 0.0, u3 = 0.0;
    int it = 0;
    bool done = false;
    if (no_root(cterm, dt_dx, alpha)) {  // a cell that its evaporation drains: up to 30 iterations otherwise
        u = MIN_FLOW_QROOT;
        u2 = u * u;
        u3 = u2 * u;
        done = true;
    } else if (wfm::gt0_(k.u)) {
        u = k.u;
        const double fu = k.P - cterm;
        if (converged(fu)) {
            done = true;
            u2 = u * u;
            u3 = u2 * u;
        } else {
            u = u - (wfm::is_zero_(k.rdf) ? fu / k.df : wfm::div_by_(fu, k.df, k.rdf));
            if (wfm::isnan_(u) || wfm::le0_(u)) u = MIN_FLOW_QROOT;
            if (wfm::to_bits(u) == wfm::to_bits(k.u)) {  // an iterate that repeats itself
                done = true;
                u2 = u * u;
                u3 = u2 * u;
            }
            it = 1;
        }
    } else {
        u = wfm::cbrt(wfm::div_(cterm, alpha));
    }
    while (!done) {
        u2 = u * u;
        u3 = u2 * u;
        const double fu = u3 * (dt_dx * u2 + alpha) - cterm;
        if (it >= 3000 || converged(fu)) break;
        const double df = u2 * (c1 * u2 + c2);
        const double u_old = u;
        u = u - wfm::div_(fu, df);
        if (wfm::isnan_(u) || wfm::le0_(u)) u = MIN_FLOW_QROOT;
        if (wfm::to_bits(u) == wfm::to_bits(u_old)) break;
        ++it;
    }
    if (!wfm::le_(MIN_FLOW_QROOT, u)) {  // max(u, MIN_FLOW_QROOT)
        u = wfm::jmax(u, MIN_FLOW_QROOT);
        u3 = u * u * u;
    }
    u_out = u;
    return u3 * u * u;
}

// ---- walker --------------------------------------------------------------------------------------
//
// Phys interface:
//   struct In; struct St;                        inputs of a node; state handed from sub-step to sub-step
//   void load(slot, e, m, fresh, resumed, In&)   issues the loads (fresh: before the model step's first
//                                                sub-step; resumed: after another round of the launch)
//   void start(const In&, St&)
//   static constexpr bool kLand, kTr             arguments of gather
//   bool active(m, St&)                          whether member m takes the sub-step
//   void sub(const In&, St&, rec, qin, tr, slot, e, m, s, chain, is_end, hq, more)
//     one sub-step after its gather; on return hq is what the node hands downstream; more: the launch
//     holds another sub-step after s.
//   void finish(const St&, e, bool last_round)   stores after the last sub-step of a round

using wfv::Batch;
using wfv::Cursor;
using wfv::P_END;
using wfv::P_HEAVY;
using wfv::Pos;

__host__ __device__ constexpr size_t walk_smem(int threads) { return (size_t)(threads / 32) * sizeof(Batch); }

// SL lanes per chain-member pair, of which the first SU = min(SL, S) work (more lanes than sub-steps
// only keep other chains out of the warp).
template <class Phys, bool MULTI>
__device__ __forceinline__ bool ticket(const WfDevGraph& g, const WfSweep& sw, Phys& phys, int32_t* status, int count,
                                       int SL, const wfv::LanePair& lp, int npos, Batch* wb) {
    using In = typename Phys::In;
    using St = typename Phys::St;
    const unsigned lane = threadIdx.x & 31u;
    const int M = g.M;
    const int sl = (int)lane & (SL - 1);
    const int SU = MULTI ? min(SL, sw.S) : 1;
    const int rounds = MULTI ? (sw.S + SU - 1) / SU : 1;
    if (wfv::status_ld(status) & WF_DEV_SPIN_TIMEOUT) return false;
    const bool lead = sl == 0;
    for (int r = 0; r < rounds; ++r) {
        const int s = r * SU + sl;
        const int s0 = r * SU;
        const bool works = sl < SU && s < sw.S;
        const bool last_lane = (s == sw.S - 1) || (sl == SU - 1);
        const bool fresh = r == 0 && sw.first == 0;
        // the lead lane's pipeline: position t (pc), t + 1 (pn) and t + 2
        In cur, nxt;
        Rec ucur{-1, -1, 0, 0}, unxt{-1, -1, 0, 0};
        unsigned long long c0 = SENTINEL, c1 = SENTINEL;
        Pos pc{0, 0, 0, 0}, pn{0, 0, 0, 0};
        Cursor cur2;
        cur2.reset(wb, count);
        if (lead) {
            cur2.resolve(wb, count, lp, pc);
            if (pc.flags) {
                ucur = load_rec(g, pc.slot);
                phys.load(pc.slot, pc.slot * M + pc.m, pc.m, fresh, r > 0, cur);
                load_words(g, pc.m, ucur, s0, c0, c1);
            }
            cur2.advance(wb, count);
            cur2.resolve(wb, count, lp, pn);
            if (pn.flags) unxt = load_rec(g, pn.slot);
        }
        In x;
        St st;
        Rec u{-1, -1, 0, 0};
        unsigned long long w0 = SENTINEL, w1 = SENTINEL;
        Pos ps{0, 0, 0, 0};
        double hq = 0.0;
        for (int tt = 0; tt < npos + SU - 1; ++tt) {
            unsigned long long n0 = SENTINEL, n1 = SENTINEL;
            Rec unn{-1, -1, 0, 0};
            Pos pnn{0, 0, 0, 0};
            if (lead) {
                x = cur;
                u = ucur;
                w0 = c0;
                w1 = c1;
                ps = pc;
                phys.start(x, st);
                if (pn.flags) {
                    phys.load(pn.slot, pn.slot * M + pn.m, pn.m, fresh, r > 0, nxt);
                    load_words(g, pn.m, unxt, s0, n0, n1);
                    prefetch_lists<Phys::kLand>(g, pn.slot, unxt);
                }
                cur2.advance(wb, count);
                cur2.resolve(wb, count, lp, pnn);
                if (pnn.flags) unn = load_rec(g, pnn.slot);
            }
            bool ok = true;
            unsigned long long v0 = SENTINEL, v1 = SENTINEL;  // words of sub-step s + 1 for the next lane
            const bool here = ps.flags && works;
            const bool acts = here && phys.active(ps.m, st);
            double qin = 0.0, tr = 0.0;
            if (here && MULTI && sl + 1 < SU && s + 1 < sw.S) load_words(g, ps.m, u, s + 1, v0, v1);
            if (acts)
                ok = gather<Phys::kLand, Phys::kTr>(g, sw, u, w0, w1, ps.slot, ps.m, s, (ps.flags & P_HEAVY) != 0, hq,
                                                    status, qin, tr);
            // The lanes meet after their waits: lanes that wait differently would otherwise run the rest of
            // the step group by group, each at the full price of its FP64 instructions (a daily step of
            // 64 x 64 cells: overland 2.70 -> 1.25 ms, river 6.2 -> 3.5).
            if (__any_sync(0xffffffffu, !ok)) return false;
            if (here) {
                const int64_t e = ps.slot * M + ps.m;
                if (acts)
                    phys.sub(x, st, u, qin, tr, ps.slot, e, ps.m, s, ps.chain, (ps.flags & P_END) != 0, hq,
                             MULTI && s + 1 < sw.S);
                if (last_lane) phys.finish(st, e, s == sw.S - 1);
            }
            __syncwarp();
            if (MULTI) {  // hand the node to the next lane
                wfv::shfl_up_pod(x, SL);
                wfv::shfl_up_pod(st, SL);
                wfv::shfl_up_pod(u, SL);
                Pos up = ps;
                wfv::shfl_up_pod(up, SL);
                const unsigned long long v0_up = __shfl_up_sync(0xffffffffu, v0, 1, SL);
                const unsigned long long v1_up = __shfl_up_sync(0xffffffffu, v1, 1, SL);
                if (!lead) {
                    ps = up;
                    w0 = v0_up;
                    w1 = v1_up;
                }
            }
            if (lead) {
                cur = nxt;
                ucur = unxt;
                unxt = unn;
                c0 = n0;
                c1 = n1;
                pc = pn;
                pn = pnn;
            }
        }
        __syncwarp();  // the round's stores before the next round's loads
    }
    return true;
}

// Tickets: the last p_chunks chunks (one long chain each) longest first, with SLp lanes per pair, then
// the other chunks in dependency order, the short ones with SLs lanes in batches of `batch`, the rest
// with SLr lanes.
template <class Phys, bool MULTI>
__device__ __forceinline__ void walk(Phys& phys, int64_t p_chunks, int SLp, int SLs, int SLr, int batch, int32_t* status) {
    extern __shared__ unsigned long long wave_smem[];
    const WfDevGraph& g = phys.g;
    const WfSweep& sw = phys.sw;
    const unsigned lane = threadIdx.x & 31u;
    Batch* wb = reinterpret_cast<Batch*>(wave_smem) + (threadIdx.x >> 5);
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
        wfv::LanePair lp;
        __syncwarp();
        if (!wfv::fill_batch(g, first, count, SL, ipc, MULTI || (lane & (SL - 1)) == 0, wb, lp, npos)) continue;
        if (!ticket<Phys, MULTI>(g, sw, phys, status, count, SL, lp, npos, wb)) return;
    }
}

}  // namespace wfz
