// twins-b200: the persistent slot kernel.
//
// One cooperative launch runs up to `max_slots_per_launch` slots of every world in the batch.
// Warps own entities for the whole launch (host units of `host_lanes` hosts, one thread each;
// one switch per warp), so that an entity's records are its SM's alone; link messages cross SMs
// through L2 (ld/st.cg). A warp stages the link messages its unit reads in
// shared memory first. Slots are separated by a grid barrier (tb_sync.cuh) whose last arriving block does the
// slot bookkeeping of the reference's ticket block (src/kernel.cuh:79-112): finish when every
// message is done, else the exact idle skip to the earliest host wake-up when nothing was sent in
// this or the previous slot. Every wait is bounded; a barrier that times out sets an error flag
// and ends the launch.
#include "tb_switch.cuh"
#include "tb_sync.cuh"
#include "tb_kernel.h"

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

namespace tb
{

constexpr int WARPS_PER_BLOCK = TB_WARPS_PER_BLOCK;
// resident blocks per SM that each instantiation's register budget allows. Several hosts per warp: 3
// (168 registers: with 4 blocks, 128 registers, the connection core spills and 96 k=8 worlds take
// 186 ms, with 3 163 ms). One host per warp: 2, and up to 255 registers (with 3 blocks the event loop
// spills: 12 leaf-spine worlds 297 / 233 ms, 96 k=8 worlds 281 / 252 ms).
constexpr int MIN_BLOCKS_MANY = 3, MIN_BLOCKS_ONE = 2;
constexpr long long BARRIER_SPIN_LIMIT = 1ll << 22; // polls of >= 64 ns: several seconds

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// An L1 line brought in ahead by a load whose value nobody waits for (prefetch.global.L1 left the
// loads that follow it as slow as without it here: with the loads, and every sector and ring head an
// event reads among them, k=16 takes 89.9 ms against 94.1 ms, three k=8 worlds 237 against 244 ms).
__device__ __forceinline__ void prefetch_l1(const void *p)
{
    unsigned v;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(p));
    (void)v;
}
// (the L1 fills by 32-byte sectors: a prefetch per sector, not per line)
__device__ __forceinline__ void prefetch_l1(const void *p, int bytes)
{
    for (int b = 0; b < bytes; b += 32)
        prefetch_l1((const char *)p + b);
}

// the stream's look-ahead rows (tb_common.cuh), in global memory, read through the read-only path
__device__ const RngAhead g_rng_ahead = make_rng_ahead();

// The world's rule for this slot (reference src/kernel.cuh:79-112, per world): the next launch
// slot its entities run, and its time origin; both read through L2 (the controller of another SM
// writes them)
__device__ __forceinline__ int64_t world_next(const Sim &s, int w) { return __ldcg(&s.wctl[w].next); }
__device__ __forceinline__ int64_t world_t0(const Sim &s, int w) { return __ldcg(&s.wctl[w].t0); }

// a host's slot results into its world's record (wake: a world-local slot)
__device__ __forceinline__ void host_report(const Sim &s, int w, int64_t t0, bool act, int64_t wake, unsigned done)
{
    WorldCtl *wc = &s.wctl[w];
    if (act)
        atomicOr(&wc->act, 1u);
    if (wake != INT64_MAX)
        atomicMin(&wc->wake, (unsigned long long)(wake + t0));
    if (done)
        atomicAdd(&wc->fdone, done);
}

// host_step's timer scan on the whole warp: the timers of the host's active connections due before
// E0, in host_step's order (senders' retransmission then SYN timers, then receivers' delayed-ACK,
// SYN, last-ACK and FIN timers, each list in its order), the first DUE_CAP of them into `due`; the
// count kept is returned (every lane), the count left out goes to *ovf.
__device__ int collect_due_warp(const Sim &s, const HostRec &hr, int h, int64_t E0, int lane, Due *due, int *ovf)
{
    const unsigned FULL = 0xffffffffu;
    const int *as = s.act_snd + (size_t)h * s.act_cap, *ar = s.act_rcv + (size_t)h * s.act_cap;
    const int ns = hr.n_snd, nr = hr.n_rcv;
    int n = 0;
    auto place = [&](int cnt) {
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1)
        {
            const int v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o)
                incl += v;
        }
        const int at = n + incl - cnt;
        n += __shfl_sync(FULL, incl, 31);
        return at;
    };
    for (int i0 = 0; i0 < ns; i0 += 32)
    {
        const int i = i0 + lane;
        int f = 0;
        int64_t v[2] = {-1, -1};
        if (i < ns)
        {
            f = as[i];
            v[0] = s.snd[f].rto_at;
            v[1] = s.snd[f].syn_at;
        }
        const int kinds[2] = {0, 2};
        int at = place((v[0] >= 0 && v[0] < E0) + (v[1] >= 0 && v[1] < E0));
        for (int j = 0; j < 2; j++)
            if (v[j] >= 0 && v[j] < E0)
            {
                if (at < DUE_CAP)
                    due[at] = {v[j], f, kinds[j]};
                at++;
            }
    }
    for (int i0 = 0; i0 < nr; i0 += 32)
    {
        const int i = i0 + lane;
        int f = 0;
        int64_t v[4] = {-1, -1, -1, -1};
        if (i < nr)
        {
            f = ar[i];
            const RcvRec &R = s.rcv[f];
            v[0] = R.delack_at;
            v[1] = R.syn_at;
            v[2] = R.last_at;
            v[3] = R.frx_at;
        }
        const int kinds[4] = {1, 3, 4, 5};
        int cnt = 0;
        for (int j = 0; j < 4; j++)
            cnt += v[j] >= 0 && v[j] < E0;
        int at = place(cnt);
        for (int j = 0; j < 4; j++)
            if (v[j] >= 0 && v[j] < E0)
            {
                if (at < DUE_CAP)
                    due[at] = {v[j], f, kinds[j]};
                at++;
            }
    }
    *ovf = n > DUE_CAP ? n - DUE_CAP : 0;
    return n < DUE_CAP ? n : DUE_CAP;
}

// host_step's last phase on the whole warp: the host's finished connections leave its active
// lists (the others keep their order; lanes read a chunk of 32 entries, then write the kept ones
// back at or below it) and the earliest timer of the connections that stay is returned (every
// lane). The host's lists and counts are those its lane 0 has just written.
__device__ int64_t prune_lists_warp(const Sim &s, int h, int lane)
{
    const unsigned FULL = 0xffffffffu, below = (1u << lane) - 1;
    HostRec &hr = s.hosts[h];
    int *as = s.act_snd + (size_t)h * s.act_cap, *ar = s.act_rcv + (size_t)h * s.act_cap;
    int64_t next = INT64_MAX;
    const int ns = hr.n_snd, nr = hr.n_rcv;
    int k = 0;
    for (int i0 = 0; i0 < ns; i0 += 32)
    {
        const int i = i0 + lane;
        int f = 0;
        bool keep = false;
        if (i < ns)
        {
            f = as[i];
            const SndRec &S = s.snd[f];
            keep = S.st != S_DONE;
            if (keep && S.rto_at >= 0 && S.rto_at < next)
                next = S.rto_at;
            if (keep && S.syn_at >= 0 && S.syn_at < next)
                next = S.syn_at;
        }
        const unsigned m = __ballot_sync(FULL, keep);
        __syncwarp(); // (every lane has read its entry)
        if (keep)
            as[k + __popc(m & below)] = f;
        k += __popc(m);
    }
    const int ks = k;
    k = 0;
    for (int i0 = 0; i0 < nr; i0 += 32)
    {
        const int i = i0 + lane;
        int f = 0;
        bool keep = false;
        if (i < nr)
        {
            f = ar[i];
            const RcvRec &R = s.rcv[f];
            keep = !rcv_idle_for_good(R);
            if (keep)
            {
                const int64_t v[4] = {R.delack_at, R.syn_at, R.last_at, R.frx_at};
                for (int j = 0; j < 4; j++)
                    if (v[j] >= 0 && v[j] < next)
                        next = v[j];
            }
        }
        const unsigned m = __ballot_sync(FULL, keep);
        __syncwarp();
        if (keep)
            ar[k + __popc(m & below)] = f;
        k += __popc(m);
    }
    for (int o = 16; o > 0; o >>= 1)
    {
        const int64_t v = __shfl_xor_sync(FULL, next, o);
        next = v < next ? v : next;
    }
    __syncwarp(); // (every lane has read the counts)
    if (lane == 0)
    {
        hr.n_snd = ks;
        hr.n_rcv = k;
    }
    return next;
}

// A host unit at launch slot t: one host per warp (host_lanes 1) or one per lane. With one host
// per warp, the warp reads the host's link-message tags (by launch slot) together with its world's
// rule; a host whose world does not run this slot, or that has no frame arriving, no timer due and
// an empty queue, only reports its wake-up. Otherwise the warp copies the host's incoming link
// messages to shared memory (one cooperative pass) and prefetches into L1 what the host's events
// will read: the records of the frames' connections with the heads of their sent lists and RTT
// histories, the head frames of the host's egress queue, and the timers of its active
// connections; then lane 0 runs the host's slot (host_step) on the staged frames, or in place
// when they do not fit. With several hosts per warp each lane runs its own host in place: the
// unit's hosts are h0 .. h0 + nh - 1. Flows completed are added to *done_sink.
template <bool MANY>
__device__ __forceinline__ void host_unit(const Sim &s, int h0, int nh, int64_t t, int lane, SwShared &sh, unsigned &ties,
                                          unsigned *done_sink)
{
    int h, w = 0, first2 = 0, n2 = 0, n1 = 0, due_n = 0, due_ovf = 0;
    int64_t t0 = 0;
    bool run = false;
    const Frame *stage = nullptr;
    Due *due = nullptr;
    if constexpr (!MANY)
    {
        h = h0;
        const HostRec &hr = s.hosts[h];
        w = hr.world;
        const int link = hr.in_link;
        const MsgTag a2 = msg_tag(s, t - 2, link), a1 = msg_tag(s, t - 1, link);
        first2 = a2.early;
        n2 = a2.n - a2.early;
        n1 = a1.early;
        const int n = n2 + n1;
        const int64_t next = world_next(s, w);
        t0 = world_t0(s, w);
        if (t < next)
            return;
        if (n == 0 && t - t0 < hr.wake && hr.q_size == 0)
        {
            if (lane == 0 && hr.wake != INT64_MAX)
                atomicMin(&s.wctl[w].wake, (unsigned long long)(hr.wake + t0));
            return;
        }
        const bool staged = n <= sh.cap;
        if (staged)
            for (int i = lane; i < n; i += 32)
                frame_load_link(sh.fr()[i], i < n2 ? msg_frames(s, t - 2, link) + first2 + i : msg_frames(s, t - 1, link) + (i - n2));
        __syncwarp();
        const bool cubic = s.worlds[w].cc == CC_CUBIC;
        if (staged)
            for (int i = lane; i < n; i += 32)
            {
                const Frame &f = sh.fr()[i];
                if (f.to_sender)
                {
                    const SndRec *S = &s.snd[f.flow];
                    prefetch_l1(S, sizeof(SndCore));
                    prefetch_l1(&S->rchain, sizeof(Chain));
                    if (cubic)
                        prefetch_l1((const char *)S + sizeof(SndCore), 80);
                    // the heads of its sent list and RTT history, where the list grows, its message
                    const uint64_t off = S->it_off;
                    const uint32_t cap = S->it_cap, hd = S->it_head, hh = S->h_head, n = S->it_n;
                    const uint32_t tl = hd + n < cap ? hd + n : hd + n - cap;
                    prefetch_l1(&s.it_start[off + hd], min(64, (int)(4 * (cap - hd))));
                    prefetch_l1(&s.it_fl[off + 4 * (hd >> 3)]); // (the flag word of the head's eight)
                    prefetch_l1(&s.it_fl[off + 4 * (tl >> 3)]);
                    prefetch_l1(&s.h_end[off + hh], min(64, (int)(4 * (cap - hh))));
                    prefetch_l1(&s.h_t[off + hh], min(96, (int)(8 * (cap - hh))));
                    if (S->m_dn < S->m_cnt)
                        prefetch_l1(&s.msgs[S->m_first + S->m_dn].end);
                }
                else
                {
                    prefetch_l1(&s.rcv[f.flow], sizeof(RcvRec));
                }
            }
        if (lane < 8 && lane < hr.q_size)
        {
            int at = hr.q_head + lane;
            if (at >= s.ring)
                at -= s.ring;
            prefetch_l1(&s.host_ring[(size_t)h * s.ring + at], sizeof(Frame));
        }
        if (sh.due_fit(DUE_CAP * sizeof(Due)))
        {
            due = reinterpret_cast<Due *>(sh.due_area()); // (the word arrays, unused by a host)
            due_n = collect_due_warp(s, hr, h, (t - t0 + 1) * SLOT_PS, lane, due, &due_ovf);
        }
        else
        {
            const int *as = s.act_snd + (size_t)h * s.act_cap, *ar = s.act_rcv + (size_t)h * s.act_cap;
            for (int i = lane; i < hr.n_snd; i += 32)
                prefetch_l1(&s.snd[as[i]].rto_at);
            for (int i = lane; i < hr.n_rcv; i += 32)
                prefetch_l1(&s.rcv[ar[i]].delack_at);
        }
        __syncwarp();
        stage = staged ? sh.fr() : nullptr;
        run = lane == 0;
    }
    else
    {
        h = h0 + lane;
        if (lane < nh)
        {
            const HostRec &hr = s.hosts[h];
            w = hr.world;
            t0 = world_t0(s, w);
            run = t >= world_next(s, w);
            if (run)
            {
                // all lanes at once: the tags of the host's link messages, then the records of
                // the connections of its first arrivals into L1 (the lanes' event loops diverge
                // next, and would each wait for these one after the other)
                const int link = hr.in_link;
                const MsgTag a2 = msg_tag(s, t - 2, link), a1 = msg_tag(s, t - 1, link);
                first2 = a2.early;
                n2 = a2.n - a2.early;
                n1 = a1.early;
                const Frame *m2 = msg_frames(s, t - 2, link) + first2, *m1 = msg_frames(s, t - 1, link);
                for (int j = 0; j < 4 && j < n2 + n1; j++)
                {
                    const Frame *f = j < n2 ? &m2[j] : &m1[j - n2];
                    const uint32_t flow = __ldcg(&f->flow);
                    const uint8_t to_snd = __ldcg(&f->to_sender);
                    prefetch_l1(to_snd ? (const void *)&s.snd[flow] : (const void *)&s.rcv[flow]);
                }
                if (hr.q_size > 0)
                    prefetch_l1(&s.host_ring[(size_t)h * s.ring + hr.q_head]);
            }
        }
    }
    int64_t wake = INT64_MAX;
    unsigned done = 0;
    bool act = false;
    if (run)
    {
        act = host_step<!MANY>(s, h, t - t0, t, &wake, &ties, &done, sh.offered(), stage, first2, n2, n1, due, due_n, due_ovf);
        if constexpr (MANY)
            host_report(s, w, t0, act, wake, done);
    }
    if constexpr (!MANY)
    {
        // the whole warp prunes the host's active lists; the earliest timer left bounds the wake-up
        __syncwarp();
        const int64_t nt = prune_lists_warp(s, h, lane);
        if (lane == 0)
        {
            HostRec &hr = s.hosts[h];
            if (hr.q_size == 0 && nt != INT64_MAX && nt / SLOT_PS < hr.wake)
                hr.wake = nt / SLOT_PS;
            host_report(s, w, t0, act, hr.wake, done);
        }
    }
    if (run && done)
        atomicAdd(done_sink, done);
    __syncwarp(); // (the staging area is reused by the warp's next unit)
}

// a slot's messages beyond the staging area: the phases through L2, a port per lane
__device__ __noinline__ bool switch_unstaged(const SwCtx &x, SwShared &sh, int lane, SwCounts &c)
{
    const bool on = lane < x.sr->k;
    if (on)
    {
        sw_phase_clear(x, sh, lane);
        c.pk = (unsigned)input_of(x, sh, lane).count();
    }
    __syncwarp();
    if (x.spray)
    {
        if (lane == 0)
            sw_phase_spray(x, sh, c.ties);
        __syncwarp();
    }
    if (on)
        c.drops += sw_phase_count(x, sh, lane);
    __syncwarp();
    if (on)
        sw_phase_offsets(x, sh, lane);
    __syncwarp();
    if (on)
        sw_phase_base(x, sh, lane);
    __syncwarp();
    if (on)
        sw_phase_scatter(x, sh, lane);
    __syncwarp();
    return on && sw_phase_egress(x, sh, lane, c);
}

// one switch, one slot (launch slot gt), by its warp; nothing when its world does not run this slot
__device__ __forceinline__ bool switch_step(const Sim &s, int sw, int64_t gt, int lane, SwShared &sh, unsigned &ties)
{
    const unsigned FULL = 0xffffffffu;
    const SwRec &sr = s.sws[sw];
    const int64_t next = world_next(s, sr.world), t0 = world_t0(s, sr.world);
    const int k = sr.k;
    const bool on = lane < k;
    int link = -1, first2 = 0, n2 = 0, n1 = 0, qn = 0, qh = 0;
    if (on)
    {
        const PortRec &pr = s.ports[sr.port0 + lane];
        link = pr.in_link;
        qn = pr.q_size;
        qh = pr.q_head;
        if (link >= 0)
        {
            const MsgTag a2 = msg_tag(s, gt - 2, link), a1 = msg_tag(s, gt - 1, link);
            first2 = a2.early;
            n2 = a2.n - a2.early;
            n1 = a1.early;
        }
    }
    // its world does not run this slot; or no frame arriving and every queue empty: nothing to do
    // (its link messages of this slot stay unwritten, and a stale tag reads as an empty message)
    if (gt < next || !__any_sync(FULL, (n2 | n1 | qn) != 0))
        return false;
#ifdef TB_PROFILE
    unsigned long long sp0 = globaltimer();
#endif
    SwCtx x;
    x.s = &s;
    x.wd = &s.worlds[sr.world];
    x.sr = &sr;
    x.sw = sw;
    x.ports = s.ports + sr.port0;
    x.scratch = (size_t)sw * s.kmax * 2 * MAX_TX;
    x.t = gt - t0;
    x.gt = gt;
    x.spray = x.wd->spray != 0;
    SwCounts c{};
    int incl = n2 + n1;
    for (int o = 1; o < 32; o <<= 1)
    {
        const int v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o)
            incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31), first = incl - n2 - n1;
    sh.win[lane][0] = first2;
    sh.win[lane][1] = first2 + n2;
    sh.win[lane][2] = n1;
    sh.link[lane] = link;
    sh.cnt[lane] = 0;
    bool act;
    if (total <= sh.cap)
    {
        uint32_t *key = sh.key(), *mem = sh.mem();
        uint16_t *src = sh.src();
        uint8_t *out = sh.out();
        const int64_t S0 = x.t * SLOT_PS;
        // each staged frame's port (5 bits) and place in its message (9 bits, 1: of msg[t-1])
        for (int j = 0; j < n2 + n1; j++)
            src[first + j] = (uint16_t)(j < n2 ? lane << 10 | (first2 + j) : lane << 10 | 0x200 | (j - n2));
        if (lane == 0)
            sh.tied = 0;
        // the queue's next frames, which the slot starts (a slot sends 8 full frames), into L1
        if (on && qn)
        {
            const Frame *ring = s.port_ring + (size_t)(sr.port0 + lane) * s.ring;
            for (int j = 0; j < 9 && j < qn; j++)
                prefetch_l1(&ring[qh + j < s.ring ? qh + j : qh + j - s.ring], sizeof(Frame));
        }
        __syncwarp();
        c.pk = n2 + n1;
        // the frames: copied, their keys
        for (int i = lane; i < total; i += 32)
        {
            const int v = src[i], q = v >> 10, l = sh.link[q];
            const bool m1 = v & 0x200;
            Frame f;
            frame_load_link(f, msg_frames(s, m1 ? gt - 1 : gt - 2, l) + (v & 0x1FF));
            frame_copy(&sh.fr()[i], &f);
            uint32_t ky = (uint32_t)(f.ts - S0);
            if (x.spray)
            {
                const int ep = x.wd->n_fail ? epoch_of(*x.wd, f.ts) : 0;
                const bool draws = !port_down(*x.wd, sr.local, q, ep) && routes_to(*x.wd, sr.local, f.dst, ep) > 0;
                ky = ky << 12 | (uint32_t)(2047 - f.len) << 1 | (draws ? 0u : 1u);
            }
            key[i] = ky;
        }
        if (lane < 4 && total + lane < SwShared::pad4(total))
            key[total + lane] = ~0u; // (the draws' scan reads whole fours)
        __syncwarp();
#ifdef TB_PROFILE
        unsigned long long sp2 = globaltimer();
        if (lane == 0)
            atomicAdd(&s.ctl->prof_phase[11], sp2 - sp0);
#endif
        if (x.spray)
        {
            sw_spray_staged(x, sh, lane, total, first, first + n2 + n1, g_rng_ahead, c.ties);
            __syncwarp();
        }
#ifdef TB_PROFILE
        unsigned long long sp3 = globaltimer();
        if (lane == 0)
            atomicAdd(&s.ctl->prof_phase[12], sp3 - sp2);
#endif
        // each frame's egress port
        for (int i = lane; i < total; i += 32)
        {
            const int e = sw_egress_for(x, sh.fr()[i], src[i] >> 10, x.spray ? out[i] : 0);
            if (e < 0)
                c.drops++;
            else
                atomicAdd(&sh.cnt[e], 1);
            out[i] = (uint8_t)e;
        }
        __syncwarp();
        const int n = sh.cnt[lane];
        int ei = n;
        for (int o = 1; o < 32; o <<= 1)
        {
            const int v = __shfl_up_sync(FULL, ei, o);
            if (lane >= o)
                ei += v;
        }
        const int base = ei - n, kept = __shfl_sync(FULL, ei, 31);
        sh.base[lane] = base;
        __syncwarp();
        // by egress port (in any order), then each to its place among its port's
        for (int i = lane; i < total; i += 32)
        {
            const int e = (int8_t)out[i];
            if (e >= 0)
                mem[sh.base[e] + atomicSub(&sh.cnt[e], 1) - 1] = (x.spray ? key[i] >> 12 : key[i]) << 9 | (uint32_t)i;
        }
        sh.num[lane] = n;
        __syncwarp();
        for (int j = lane; j < kept; j += 32)
        {
            const uint32_t v = mem[j];
            const int e = out[v & 511], b = sh.base[e], m = sh.num[e];
            int rank = 0, same = 0;
            for (int i = b; i < b + m; i++)
            {
                const uint32_t u = mem[i];
                rank += u < v;
                same += u >> 9 == v >> 9;
            }
            key[b + rank] = v;
            if (same > 1)
                atomicOr(&sh.tied, 1u << e);
        }
        __syncwarp();
        if (sh.tied >> lane & 1)
            sw_order_ties(sh, key + base, n, c.ties);
#ifdef TB_PROFILE
        unsigned long long sp1 = globaltimer();
        if (lane == 0)
            atomicAdd(&s.ctl->prof_phase[6], sp1 - sp0);
#endif
        __syncwarp();
        act = on && sw_egress_staged(x, sh, lane, key + base, n, c);
#ifdef TB_PROFILE
        __syncwarp();
        if (lane == 0)
            atomicAdd(&s.ctl->prof_phase[7], globaltimer() - sp1);
#endif
    }
    else
    {
        __syncwarp();
#ifdef TB_QTRACE
        if (lane == 0)
            ev_add(s, sr.world, EV_UNSTAGED, 1);
#endif
        // (copies: what a call is given the address of lives in memory, and the staged slot's is to stay
        // in registers)
        const SwCtx y = x;
        SwCounts d = c;
        act = switch_unstaged(y, sh, lane, d);
        c = d;
    }
    __syncwarp();
    // warp totals, one atomic each
    c.pk = __reduce_add_sync(FULL, c.pk);
    c.drops = __reduce_add_sync(FULL, c.drops);
    c.marks = __reduce_add_sync(FULL, c.marks);
    c.ovf = __reduce_add_sync(FULL, c.ovf);
    c.ties = __reduce_add_sync(FULL, c.ties);
    if (lane == 0)
    {
        ev_add(s, sr.world, EV_SW_PKT, c.pk);
        ev_add(s, sr.world, EV_DROPS, c.drops);
        ev_add(s, sr.world, EV_MARKS, c.marks);
        ev_add(s, sr.world, EV_OVF_TX, c.ovf);
        ev_add(s, sr.world, EV_TIES, c.ties);
        ties += c.ties;
    }
    return __any_sync(FULL, act);
}

// MIN_BLOCKS: the register budget. Separate instantiations, chosen per launch. The parameters stay in
// the constant bank (__grid_constant__): the code takes their address, which otherwise copies them to
// local memory, where every use of an array's base is a load (96 k=8 worlds 138 ms, now 125 ms).
template <int MIN_BLOCKS>
__global__ void __launch_bounds__(WARPS_PER_BLOCK * 32, MIN_BLOCKS) slot_kernel(const __grid_constant__ Sim s, int max_slots_per_launch, int host_lanes, int stage_cap)
{
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    __shared__ unsigned blk_done;
    __shared__ int blk_last;
    __shared__ unsigned long long blk_next;
    __shared__ unsigned blk_alive;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gwarp = blockIdx.x * WARPS_PER_BLOCK + warp, nwarps = gridDim.x * WARPS_PER_BLOCK;
    const int host_units = (s.H + host_lanes - 1) / host_lanes;
    const int units = host_units + s.S;
    SwShared &sh = *sw_shared_at(dyn_smem + (size_t)warp * sw_shared_bytes(stage_cap), stage_cap); // the warp's scratch
    __syncwarp();
    SlotCtl *ctl = s.ctl;
    volatile SlotCtl *vc = ctl;
    for (int it = 0; it < max_slots_per_launch; it++)
    {
        if (threadIdx.x == 0)
            blk_done = 0;
        __syncthreads();
        // (written by the last block of the previous barrier, before it released the others)
        if (vc->finished)
            return;
        const int64_t t = vc->slot;
        unsigned ties = 0;
        const int n_iter = s.unit_list ? s.n_list : units;
        for (int i = gwarp; i < n_iter; i += nwarps)
        {
            const int u = s.unit_list ? __ldg(&s.unit_list[i]) : i;
#ifdef TB_PROFILE
            unsigned long long p0 = globaltimer();
#endif
            if (u < host_units)
            {
                const int h0 = u * host_lanes;
                host_unit<MIN_BLOCKS == MIN_BLOCKS_MANY>(s, h0, min(host_lanes, s.H - h0), t, lane, sh, ties, &blk_done);
            }
            else
            {
                const int sw = u - host_units;
                if (switch_step(s, sw, t, lane, sh, ties) && lane == 0)
                    atomicOr(&s.wctl[s.sws[sw].world].act, 1u);
            }
#ifdef TB_PROFILE
            if (lane == 0)
                atomicMax(u < host_units ? &ctl->prof_host_max : &ctl->prof_sw_max, globaltimer() - p0);
#endif
        }
        __syncthreads();
        unsigned g = 0; // (thread 0: the barrier generation before it arrives)
        if (threadIdx.x == 0)
        {
            if (blk_done)
                atomicAdd(&ctl->flows_done, blk_done);
            blk_next = ~0ull;
            blk_alive = 0;
            // grid barrier: the last block to arrive ends the slot and releases the others
            g = ld_relaxed(&ctl->gen);
            blk_last = add_release(&ctl->arrive, 1u) + 1 == gridDim.x;
            if (blk_last)
                acquire(&ctl->arrive);
        }
        __syncthreads();
        if (blk_last)
        {
            // every world's next slot: finished worlds stop; a world where nothing was sent in
            // this or the previous slot skips to its earliest wake-up
            for (int w = threadIdx.x; w < s.W; w += blockDim.x)
            {
                WorldCtl *wc = &s.wctl[w];
                volatile WorldCtl *vw = wc;
                int64_t nx = vw->next;
                if (nx == INT64_MAX)
                    continue;
                const unsigned cur = atomicExch(&wc->act, 0u), prev = vw->prev;
                const unsigned long long wake = atomicExch(&wc->wake, (unsigned long long)INT64_MAX);
                vw->prev = cur;
                if (t >= nx)
                {
                    if (atomicAdd(&wc->fdone, 0u) >= (unsigned)s.worlds[w].n_msgs)
                    {
                        vw->next = INT64_MAX;
                        continue;
                    }
                    nx = (cur == 0 && prev == 0 && (int64_t)wake > t + 1) ? (int64_t)wake : t + 1;
                    vw->next = nx;
                }
                atomicMin(&blk_next, (unsigned long long)nx);
                atomicAdd(&blk_alive, 1u);
            }
            __syncthreads();
            if (threadIdx.x == 0)
            {
                vc->arrive = 0;
                int64_t next = (int64_t)blk_next;
                if (next > s.max_slots)
                    next = s.max_slots;
                if (blk_alive == 0)
                    next = t + 1; // (finished: nothing left to skip to)
                if (blk_alive == 0 || t + 1 >= s.max_slots)
                    vc->finished = 1;
                vc->slot = next > t + 1 ? next : t + 1;
                vc->slots_run = vc->slots_run + 1;
#ifdef TB_PROFILE
                unsigned long long now = globaltimer();
                if (vc->prof_release)
                    vc->prof_slot_sum = vc->prof_slot_sum + (now - vc->prof_release);
                vc->prof_release = now;
                vc->prof_host_sum = vc->prof_host_sum + atomicAdd(&ctl->prof_host_max, 0ull);
                vc->prof_sw_sum = vc->prof_sw_sum + atomicAdd(&ctl->prof_sw_max, 0ull);
                vc->prof_host_max = 0;
                vc->prof_sw_max = 0;
#endif
                add_release(&ctl->gen, 1u);
            }
        }
        else if (threadIdx.x == 0)
        {
            long long spins = 0;
            while (ld_relaxed(&ctl->gen) == g)
            {
                if (++spins > BARRIER_SPIN_LIMIT)
                {
                    atomicExch(&ctl->error, 1);
                    atomicExch(&ctl->finished, 1);
                    atomicAdd(&s.ev[EV_BARRIER_TIMEOUT], 1ull);
                    break;
                }
                __nanosleep(64);
            }
            acquire(&ctl->gen);
        }
        __syncthreads();
    }
}


// ------------------------------------------------------------------ batches without a grid barrier
// A batch's worlds are independent: each runs its own slots on a barrier of its own, so that a
// slot of one world waits only for that world's units, not for the slowest unit of the batch.
// The launch's unit list holds host units (first host h < H; up to host_lanes hosts of one world)
// and switches (H + switch). A warp cycles over its units and runs every one whose world runs a
// slot the unit has not done; the unit's lane 0, after the warp, counts it in its world's
// `arrive`, and the world's last unit closes the slot: the world's slot rule (finish, the exact
// idle skip), then the next slot is published (or the world parks: its slot budget for this
// launch is spent, or it is done). A warp whose units are all parked leaves; one that finds
// nothing to run waits (bounded) for its worlds to move.

// the world's slot t is done by all its units: its next slot, or parked (by the unit's lane 0)
__device__ void world_close(const Sim &s, int w, int64_t t)
{
    WorldCtl *wc = &s.wctl[w];
    volatile WorldCtl *vw = wc;
    const unsigned cur = atomicExch(&wc->act, 0u), prev = vw->prev;
    const unsigned long long wake = atomicExch(&wc->wake, (unsigned long long)INT64_MAX);
    vw->prev = cur;
    vw->last = t;
    int64_t nx;
    if (atomicAdd(&wc->fdone, 0u) >= (unsigned)s.worlds[w].n_msgs)
        nx = INT64_MAX;
    else
    {
        nx = (cur == 0 && prev == 0 && (int64_t)wake > t + 1) ? (int64_t)wake : t + 1;
        if (nx >= s.max_slots)
        {
            nx = INT64_MAX; // (the run ends at max_slots with flows unfinished, as the batch's does)
            vw->last = s.max_slots - 1;
        }
    }
    atomicAdd((unsigned long long *)&s.ctl->slots_run, 1ull);
    const unsigned budget = vw->budget - 1;
    vw->budget = budget;
    vw->next = nx;
    vw->arrive = 0;
    st_release(&wc->run, (nx == INT64_MAX || budget == 0) ? RUN_PARKED : nx);
}

// before a launch: every world runs from its next slot with a budget; every unit has done nothing
__global__ void free_open(Sim s, unsigned budget)
{
    const int stride = gridDim.x * blockDim.x;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < s.n_list; i += stride)
        s.unit_done[i] = RUN_PARKED;
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < s.W; w += stride)
    {
        WorldCtl &c = s.wctl[w];
        c.arrive = 0;
        c.units = s.w_units[w];
        c.budget = budget;
        c.run = c.next == INT64_MAX || c.units == 0 ? RUN_PARKED : c.next;
    }
}

template <int MIN_BLOCKS>
__global__ void __launch_bounds__(WARPS_PER_BLOCK * 32, MIN_BLOCKS) free_kernel(const __grid_constant__ Sim s, int host_lanes, int stage_cap)
{
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gwarp = blockIdx.x * WARPS_PER_BLOCK + warp, nwarps = gridDim.x * WARPS_PER_BLOCK;
    SwShared &sh = *sw_shared_at(dyn_smem + (size_t)warp * sw_shared_bytes(stage_cap), stage_cap); // the warp's scratch
    __syncwarp();
    const unsigned FULL = 0xffffffffu;
    long long idle = 0;
    for (;;)
    {
        bool live = false, ran = false;
        for (int i = gwarp; i < s.n_list; i += nwarps)
        {
            const int v = __ldg(&s.unit_list[i]);
            const bool host = v < s.H;
            const int w = host ? s.hosts[v].world : s.sws[v - s.H].world;
            int64_t t = 0, done = 0;
            if (lane == 0)
            {
                t = ld_relaxed(&s.wctl[w].run);
                done = s.unit_done[i];
            }
            t = __shfl_sync(FULL, t, 0);
            done = __shfl_sync(FULL, done, 0);
            if (t == RUN_PARKED)
                continue;
            live = true;
            if (done == t)
                continue; // (done; its world's other units are not)
            ran = true;
            if (lane == 0)
                acquire(&s.wctl[w].run);
            __syncwarp();
            unsigned ties = 0;
            if (host)
            {
                const WorldDesc &wd = s.worlds[w];
                host_unit<MIN_BLOCKS == MIN_BLOCKS_MANY>(s, v, min(host_lanes, wd.host0 + wd.H1 - v), t, lane, sh, ties,
                                                         &s.ctl->flows_done);
            }
            else if (switch_step(s, v - s.H, t, lane, sh, ties) && lane == 0)
                atomicOr(&s.wctl[w].act, 1u);
            __syncwarp();
            if (lane == 0)
            {
                s.unit_done[i] = t;
                if (add_release(&s.wctl[w].arrive, 1u) + 1 == __ldcg(&s.wctl[w].units))
                {
                    acquire(&s.wctl[w].arrive);
                    world_close(s, w, t);
                }
            }
            __syncwarp();
        }
        if (!live)
            return;
        if (ran)
        {
            idle = 0;
            continue;
        }
        if (++idle > BARRIER_SPIN_LIMIT || ld_relaxed((const unsigned *)&s.ctl->error))
        {
            if (lane == 0 && idle > BARRIER_SPIN_LIMIT)
            {
                atomicExch(&s.ctl->error, 1);
                atomicAdd(&s.ev[EV_BARRIER_TIMEOUT], 1ull);
            }
            return;
        }
        __nanosleep(64);
    }
}

// dynamic shared memory of a block: one switch scratch (with its staging area) per warp
static size_t smem_bytes(int stage_cap) { return sw_shared_bytes(stage_cap) * WARPS_PER_BLOCK; }

// the instantiation of a launch shape: several hosts per warp or one host per warp; each with the
// grid barrier or without (F_*: batches)
enum
{
    K_MANY,
    K_ONE,
    F_MANY,
    F_ONE,
    K_N
};
static int kind_of(int host_lanes, bool free = false) { return (host_lanes > 1 ? K_MANY : K_ONE) + (free ? F_MANY : 0); }
static const void *kernel_of(int k)
{
    switch (k)
    {
    case K_MANY:
        return (const void *)slot_kernel<MIN_BLOCKS_MANY>;
    case K_ONE:
        return (const void *)slot_kernel<MIN_BLOCKS_ONE>;
    case F_MANY:
        return (const void *)free_kernel<MIN_BLOCKS_MANY>;
    default:
        return (const void *)free_kernel<MIN_BLOCKS_ONE>;
    }
}

static bool smem_attr(int k)
{
    static bool ok[K_N], tried[K_N];
    if (!tried[k])
    {
        tried[k] = true;
        ok[k] = cudaFuncSetAttribute(kernel_of(k), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(SW_STAGE_MAX)) == cudaSuccess;
    }
    return ok[k];
}

// The preferred shared-memory carveout, in percent of the SM's maximum: the shared memory of the
// blocks a launch puts on one SM and no more, so that the rest of the SM's unified L1 / shared
// memory is L1, which holds the units' records, ring heads and prefetched lines through a slot.
static int carveout[K_N] = {-1, -1, -1, -1}; // the last ones set (-1: none)
static void set_carveout(int k, int pct)
{
    if (pct != carveout[k] && cudaFuncSetAttribute(kernel_of(k), cudaFuncAttributePreferredSharedMemoryCarveout, pct) == cudaSuccess)
        carveout[k] = pct;
}

int slot_kernel_blocks_per_sm(int stage_cap, int host_lanes, bool free)
{
    int n = 0;
    const int k = kind_of(host_lanes, free);
    if (stage_cap < 1 || stage_cap > SW_STAGE_MAX || !smem_attr(k))
        return 0;
    set_carveout(k, 100); // (occupancy with all of the shared memory)
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel_of(k), WARPS_PER_BLOCK * 32, smem_bytes(stage_cap)) != cudaSuccess)
        return 0;
    return n;
}

// a cooperative launch of kernel kind k (all its blocks resident: the waits need it)
static int launch_kind(int k, void **args, int grid, int stage_cap, cudaStream_t stream)
{
    int dev = 0, sms = 1, max_smem = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    const long long per_sm = (grid + sms - 1) / sms;
    const size_t bytes = smem_bytes(stage_cap);
    const long long need = per_sm * (long long)(bytes + 2048); // (+ the block's reserved and static shared memory)
    set_carveout(k, (int)std::min<long long>(100, (need * 100 + max_smem - 1) / max_smem));
    cudaError_t e = cudaLaunchCooperativeKernel(kernel_of(k), dim3(grid), dim3(WARPS_PER_BLOCK * 32), args, bytes, stream);
    if (e == cudaErrorCooperativeLaunchTooLarge)
    {
        // (the carveout left too little shared memory for the blocks to be resident at once)
        cudaGetLastError();
        set_carveout(k, 100);
        e = cudaLaunchCooperativeKernel(kernel_of(k), dim3(grid), dim3(WARPS_PER_BLOCK * 32), args, bytes, stream);
    }
    return e == cudaSuccess ? 0 : (int)e;
}

int launch_slots(const Sim &s, int grid, int max_slots_per_launch, int host_lanes, int stage_cap, cudaStream_t stream)
{
    const int k = kind_of(host_lanes);
    if (!smem_attr(k) || stage_cap < 1 || stage_cap > SW_STAGE_MAX)
        return (int)cudaErrorInvalidValue;
    void *args[] = {(void *)&s, (void *)&max_slots_per_launch, (void *)&host_lanes, (void *)&stage_cap};
    return launch_kind(k, args, grid, stage_cap, stream);
}

int launch_free(const Sim &s, int grid, int slots_per_world, int host_lanes, int stage_cap, cudaStream_t stream)
{
    const int k = kind_of(host_lanes, true);
    if (!smem_attr(k) || stage_cap < 1 || stage_cap > SW_STAGE_MAX || !s.unit_list || !s.unit_done || !s.w_units || slots_per_world < 1)
        return (int)cudaErrorInvalidValue;
    const int n = std::max(s.n_list, s.W);
    free_open<<<(n + 255) / 256, 256, 0, stream>>>(s, (unsigned)slots_per_world);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return (int)e;
    void *args[] = {(void *)&s, (void *)&host_lanes, (void *)&stage_cap};
    return launch_kind(k, args, grid, stage_cap, stream);
}

// A launch as a CUDA graph: the launch is captured once per shape, slot count and unit list and
// replayed as a graph; where capturing or instantiating fails, plain launches follow for good.
// free: the batch kernel without a grid barrier (launch_free), with its opening kernel.
int launch_slots_graph(SlotGraph &g, const Sim &s, int grid, int max_slots_per_launch, int host_lanes, int stage_cap,
                       cudaStream_t stream, bool free)
{
    const unsigned long long key[8] = {(unsigned long long)grid, (unsigned long long)max_slots_per_launch, (unsigned long long)host_lanes,
                                       (unsigned long long)stage_cap, (unsigned long long)(uintptr_t)s.unit_list,
                                       (unsigned long long)s.n_list, (unsigned long long)s.max_slots, (unsigned long long)free};
    auto go = [&]() {
        return free ? launch_free(s, grid, max_slots_per_launch, host_lanes, stage_cap, stream)
                    : launch_slots(s, grid, max_slots_per_launch, host_lanes, stage_cap, stream);
    };
    if (g.broken)
        return go();
    if (!g.exec || memcmp(key, g.key, sizeof key) != 0)
    {
        if (g.exec)
            cudaGraphExecDestroy((cudaGraphExec_t)g.exec);
        g.exec = nullptr;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        int e = 1;
        if (cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess)
        {
            e = go();
            if (cudaStreamEndCapture(stream, &graph) != cudaSuccess)
                e = 1;
        }
        if (e == 0 && graph && cudaGraphInstantiate(&exec, graph, 0) == cudaSuccess)
        {
            g.exec = exec;
            memcpy(g.key, key, sizeof key);
        }
        if (graph)
            cudaGraphDestroy(graph);
        if (!g.exec)
        {
            cudaGetLastError(); // (the failed capture's error)
            g.broken = true;
            return go();
        }
    }
    g.replays++;
    return cudaGraphLaunch((cudaGraphExec_t)g.exec, stream) == cudaSuccess ? 0 : (int)cudaGetLastError();
}

void release_graph(SlotGraph &g)
{
    if (g.exec)
        cudaGraphExecDestroy((cudaGraphExec_t)g.exec);
    g.exec = nullptr;
}

} // namespace tb
