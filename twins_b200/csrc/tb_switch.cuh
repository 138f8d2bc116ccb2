// twins-b200: one slot of one switch by its warp (k <= 32 ports).
// Reference: src/step.cuh:2748-2886 (switch_step), :2709-2745 (spray_draws).
//
// A staged slot (its ingress link messages fit the warp's staging area) spreads every step over the
// lanes: a frame per lane for the copy, the arrival window, the route, the spraying draw and the
// arrival's place among its egress port's arrivals; then a port per lane for the egress, where each
// iteration of one loop moves one frame on every port at once, whether it starts on the wire or
// joins the queue. (A serial loop per port of its own, each with its own start and enqueue loops,
// ran the ports of a warp one after the other: with it a FatTree k=16 DCTCP world of 2,253 flows
// took 207 ms, with this split 128 ms; 96 k=8 worlds 274 ms, with it 177 ms.) A slot whose messages exceed the staging area runs a port per lane in phases
// through L2 (sw_phase_*).
#pragma once
#include "tb_slot.cuh"

namespace tb
{

// per-warp shared scratch of a switch (also a host unit's staging area). The staging arrays
// follow the header in the warp's part of the block's dynamic shared memory; their capacity
// (`cap` frames) is chosen per launch.
struct SwShared
{
    int base[32], cnt[32];
    int num[32];            // arrivals per egress port
    int win[32][3];         // each ingress port's frames of the slot: msg[t-2] from the first to the second, msg[t-1] to the third
    int link[32];           // the port's ingress link
    unsigned tied;          // egress ports with arrivals at one instant
    int cap;
    // the arrays after this header, addressed from the scratch itself (so that the compiler keeps
    // them in the shared address space): a host's offered frames [OUT_FRAMES], the staged frames
    // [cap], two words, a half-word and a byte per frame (padded to four entries)
    TB_D unsigned char *bytes() { return reinterpret_cast<unsigned char *>(this); }
    TB_D const unsigned char *bytes() const { return reinterpret_cast<const unsigned char *>(this); }
    TB_D Frame *offered() { return reinterpret_cast<Frame *>(bytes() + header()); }
    TB_D Frame *fr() { return offered() + OUT_FRAMES; }
    TB_D const Frame *fr() const { return const_cast<SwShared *>(this)->fr(); }
    TB_D uint32_t *key() { return reinterpret_cast<uint32_t *>(fr() + cap); }
    TB_D uint32_t *mem() { return key() + pad4(cap); }
    TB_D uint16_t *src() { return reinterpret_cast<uint16_t *>(mem() + pad4(cap)); }
    TB_D uint8_t *out() { return reinterpret_cast<uint8_t *>(src() + pad4(cap)); }
    // a host's due timers, in the word arrays (when they are large enough: due_fit)
    TB_D unsigned char *due_area() { return reinterpret_cast<unsigned char *>(key()); }
    TB_D bool due_fit(size_t bytes) const { return (size_t)pad4(cap) * 8 >= bytes; }
    // (unstaged) [ingress][egress] counts, then offsets, in place of the staged frames
    typedef int Row[33];
    TB_D Row *rows() { return reinterpret_cast<Row *>(fr()); }
    static TB_HDI size_t header();
    static TB_HDI int pad4(int n);
};

TB_HDI size_t SwShared::header() { return (sizeof(SwShared) + 15) & ~(size_t)15; }
TB_HDI int SwShared::pad4(int n) { return (n + 3) & ~3; }
// bytes of one warp's scratch with `cap` staged frames (16-byte multiple)
TB_HDI size_t sw_shared_bytes(int cap)
{
    const size_t staged = (size_t)cap * sizeof(Frame) + (size_t)SwShared::pad4(cap) * 11, rows = 32 * sizeof(SwShared::Row);
    return SwShared::header() + OUT_FRAMES * sizeof(Frame) + (((staged > rows ? staged : rows) + 15) & ~(size_t)15);
}
// a warp's scratch at `p` (every lane may call it: the same value is written)
TB_D SwShared *sw_shared_at(unsigned char *p, int cap)
{
    SwShared *sh = reinterpret_cast<SwShared *>(p);
    sh->cap = cap;
    return sh;
}

// (unstaged) a port's frames of the slot: the late ones of msg[t-2], the early ones of msg[t-1]
struct Input
{
    const Frame *m2, *m1;
    int i2, n2, n1;
    TB_D int count() const { return (n2 - i2) + n1; }
    TB_D const Frame *at(int j) const { return j < n2 - i2 ? &m2[i2 + j] : &m1[j - (n2 - i2)]; }
    TB_D void load(Frame &f, int j) const { frame_load_link(f, at(j)); }
    TB_D int64_t ts(int j) const { return ts_load_link(at(j)); }
};

struct SwCtx
{
    const Sim *s;
    const WorldDesc *wd;
    const SwRec *sr;
    int sw;          // global switch id
    PortRec *ports;  // the switch's ports
    size_t scratch;  // its region in sw_ts / sw_ref / sw_up
    int64_t t;       // the world's own slot (time)
    int64_t gt;      // the launch's slot (indexes the link messages)
    bool spray;
};

// the egress port of an arrival at port q (-1: dropped on arrival at a down interface); `up`: its
// spraying choice
TB_D int sw_egress_for(const SwCtx &x, const Frame &f, int q, int up)
{
    const WorldDesc &wd = *x.wd;
    int ep = wd.n_fail ? epoch_of(wd, f.ts) : 0;
    if (port_down(wd, x.sr->local, q, ep))
        return -1;
    if (x.spray)
        return route_up(wd, x.sr->local, f.dst, up, ep);
    return route(*x.s, wd, x.sr->local, f, ep);
}

// ------------------------------------------------------------------ staged slots
// The spraying draws of a staged slot: one per forwarded packet, in the order the packets arrive at
// the node (all ports merged). key[i] of a frame is its offset in the slot (20 bits), 2047 - its length
// (11 bits; the longer of two simultaneous frames first) and whether it draws nothing (1 bit); ~0
// fills the last four. pos .. end - 1: the frames of the lane's port. A frame's place among the draws is the number of
// drawing frames with smaller keys: a frame per lane counts them, and every draw is computed at
// once from the stream's state and its look-ahead rows. Where two frames' keys tie, the places come
// from a merge of the ports' frames instead, a port per lane, in which the ties are decided by the
// chains in port order. A merge of every slot took one warp-wide step per frame. Each frame's
// choice goes to out[i]; the stream's state moves on by the slot's draws.
__device__ void sw_spray_staged(const SwCtx &x, SwShared &sh, int lane, int total, int pos, int end, const RngAhead &ahead, unsigned &ties)
{
    const unsigned FULL = 0xffffffffu;
    uint32_t *key = sh.key(), *place = sh.mem();
    uint8_t *up = sh.out();
    const WorldDesc &wd = *x.wd;
    bool tie = false;
    int draws = 0;
    for (int i0 = 0; i0 < total; i0 += 32)
    {
        const int i = i0 + lane;
        const uint32_t mine = i < total ? key[i] : ~0u, m = mine >> 1;
        int rank = 0, same = 0;
        const uint4 *k4 = reinterpret_cast<const uint4 *>(key);
        for (int j = 0; j < total; j += 4)
        {
            const uint4 v = k4[j >> 2];
            rank += (v.x >> 1 < m && !(v.x & 1)) + (v.y >> 1 < m && !(v.y & 1)) + (v.z >> 1 < m && !(v.z & 1)) + (v.w >> 1 < m && !(v.w & 1));
            same += (v.x >> 1 == m) + (v.y >> 1 == m) + (v.z >> 1 == m) + (v.w >> 1 == m);
        }
        if (i < total)
            place[i] = (uint32_t)rank;
        tie |= mine != ~0u && same > 1;
        draws += __popc(__ballot_sync(FULL, mine != ~0u && !(mine & 1)));
    }
    if (__any_sync(FULL, tie))
    {
        __syncwarp();
        uint32_t head = pos < end ? key[pos] >> 1 : ~0u;
        int run = 0;
        for (;;)
        {
            const uint32_t m = __reduce_min_sync(FULL, head);
            if (m == ~0u)
                break;
            const unsigned cand = __ballot_sync(FULL, head == m);
            int best = __ffs(cand) - 1;
            if (cand & (cand - 1))
            {
                // equal times and lengths: the upstream chains, then the connection id
                const Frame *bf = nullptr;
                for (unsigned cc = cand; cc; cc &= cc - 1)
                {
                    const int q = __ffs(cc) - 1;
                    const int pq = __shfl_sync(FULL, pos, q);
                    if (lane == 0)
                    {
                        const Frame *f = &sh.fr()[pq];
                        if (!bf || frame_before(*f, *bf, ties))
                        {
                            best = q;
                            bf = f;
                        }
                    }
                }
                best = __shfl_sync(FULL, best, 0);
            }
            bool drew = false;
            if (lane == best)
            {
                place[pos] = (uint32_t)run;
                drew = !(key[pos] & 1);
                pos++;
                head = pos < end ? key[pos] >> 1 : ~0u;
            }
            run += __any_sync(FULL, drew);
        }
    }
    __syncwarp();
    const Rng st = x.s->sw_rng[x.sw];
    for (int i = lane; i < total; i += 32)
    {
        uint32_t u = 0;
        if (!(key[i] & 1))
        {
            const Frame &f = sh.fr()[i];
            const uint32_t nr = (uint32_t)routes_to(wd, x.sr->local, f.dst, wd.n_fail ? epoch_of(wd, f.ts) : 0);
            const uint32_t *row = ahead.r[place[i] + 1];
            u = int_of_u01(u01_of(rng_ahead_value<RNG_M1>(row, st.s), rng_ahead_value<RNG_M2>(row + 3, st.s + 3)), nr);
        }
        up[i] = (uint8_t)u;
    }
    // the stream after the slot's draws: each component's last three values
    __syncwarp(); // (every lane has read the stream)
    if (lane < 6)
    {
        const int cmp = lane / 3, m = draws - 2 + lane % 3;
        const uint32_t *row = ahead.r[m > 0 ? m : 1] + 3 * cmp;
        x.s->sw_rng[x.sw].s[lane] = m <= 0 ? st.s[3 * cmp + m + 2]
                                           : (cmp ? rng_ahead_value<RNG_M2>(row, st.s + 3) : rng_ahead_value<RNG_M1>(row, st.s));
    }
}

// Egress e's arrivals list[0..n) (offset << 9 | staged frame, ascending) where some fall at one instant:
// each run of one offset in ns-3's order (insertion in ingress order)
TB_D void sw_order_ties(SwShared &sh, uint32_t *list, int n, unsigned &ties)
{
    for (int i = 1; i < n; i++)
    {
        const uint32_t v = list[i];
        int j = i - 1;
        for (; j >= 0 && list[j] >> 9 == v >> 9 && frame_before(sh.fr()[v & 511], sh.fr()[list[j] & 511], ties); j--)
            list[j + 1] = list[j];
        list[j + 1] = v;
    }
}

// the counters of a switch's slot
struct SwCounts
{
    unsigned pk, drops, marks, ovf, ties;
};

// Egress port e of a staged slot (its lane): list[0..n), its arrivals in order (offset in the slot <<
// 9 | staged frame). The sending end of a link as Egress describes it, for a whole slot at once:
// every iteration moves one frame, which starts on the wire (the queue's first when the wire is
// free by the next arrival, or an arrival that finds the queue empty and the wire idle) or joins the
// queue (RED's mark or drop first), so that the warp's ports run side by side whatever each has to
// do. Times are offsets in the slot. A queued frame always begins when the wire gets free: it was
// queued because the wire was busy beyond its arrival (an arrival at an idle wire starts at once,
// which is when Egress's next step would start it), so its chain is the child of the wire's
// frame's. A frame that joins the queue stays where it is staged, and goes to the queue's ring in
// memory if it still waits when the slot ends: read back from the ring it would wait for its own store
// (600 cycles). Bound by the latency of a frame's load and chain, well under 1 us per iteration; the
// ring's first frames are in L1. Returns true if the port sent or holds frames.
TB_D bool sw_egress_staged(const SwCtx &x, SwShared &sh, int e, uint32_t *list, int n, SwCounts &c)
{
    const Sim &s = *x.s;
    constexpr int SLOT = (int)SLOT_PS;
    PortRec &pr = x.ports[e];
    const int port = x.sr->port0 + e, cap = s.ring, out_link = s.H + port;
    if (n == 0 && pr.q_size == 0)
    {
        msg_seal(s, x.gt, out_link, 0, 0);
        return false;
    }
    const int red_k = pr.red_k, qcap = pr.qcap;
    const int64_t S0 = x.t * SLOT_PS;
    Frame *ring = s.port_ring + (size_t)port * cap;
    Frame *msg = s.msg + msg_index(s, x.gt, out_link) * MAX_TX;
    int head = pr.q_head, size = pr.q_size, n_out = 0, early = 0;
    // the wire: busy until `busy` with a frame of tx_len bytes that began at `began` (a wire free
    // since before the slot: only that it is matters)
    int busy = -1, began = -SLOT, tx_len = 0;
    if (pr.link_free >= S0)
    {
        busy = (int)(pr.link_free - S0);
        tx_len = (int)((uint32_t)(pr.link_free - pr.last_start) / (uint32_t)PS_PER_BYTE);
        began = busy - tx_len * (int)PS_PER_BYTE;
    }
    Chain wire = pr.last;
    // queued: `held` frames of the ring, then lq from list[jq] on (~0: dropped)
    int i = 0, held = size, jq = 0, lq = 0;
    uint32_t next = n > 0 ? list[0] : 0;
    for (;;)
    {
        const int ta = i < n ? (int)(next >> 9) : SLOT;
        size = held + lq;
        const bool start = size > 0 && busy < SLOT && busy <= ta;
        if (!start && i >= n)
            break;
        Frame f;
        Frame *const here = &sh.fr()[(start ? list[jq] : next) & 511];
        frame_copy(&f, start && held ? &ring[head] : here);
        const bool idle = size == 0 && busy <= ta; // (an arrival at an idle wire)
        bool sends = start || idle, gone = false;
        if (sends && n_out == MAX_TX)
        {
            c.ovf++;
            break; // (more frames than a slot holds: counted, never seen)
        }
        const bool behind = start || (busy == ta && tx_len > 0);
        // an arrival: its event's chain; a start behind a frame: the child of its TransmitComplete
        const bool tc = sends && behind;
        Chain par;
#pragma unroll
        for (int r = 0; r < RUNS; r++)
            par.run[r] = tc ? wire.run[r] : f.ch.run[r];
        par.root = tc ? wire.root : f.ch.root;
        chain_child(f.ch, par, tc ? code_tc(tx_len) : code_arrival(f.len));
        if (!start)
        {
            const int backlog = !size || busy <= ta ? size : size - (began < ta ? 1 : 0);
            f.ts = S0 + ta;
            if (backlog >= red_k && backlog > 1)
            {
                if (f.flags & F_ECT)
                {
                    f.flags |= F_CE;
                    c.marks++;
                }
                else
                    gone = true;
            }
            gone |= backlog >= qcap;
            c.drops += gone;
#ifdef TB_QTRACE
            if (!gone)
                qtrace_enqueue(s, x.wd->H1 + x.sr->local, e + 1, f, backlog, f.ts);
#endif
            if (!gone && !sends && size == cap)
            {
                c.ovf++;
                gone = true;
            }
            if (gone)
                list[i] = ~0u;
            if (lq == 0)
                jq = gone || sends ? i + 1 : i;
            lq += !gone && !sends;
            i++;
            next = i < n ? list[i] : 0;
        }
        if (gone)
            continue;
        if (sends)
        {
            wire = f.ch;
            began = start ? busy : ta;
            tx_len = f.len;
            busy = began + tx_len * (int)PS_PER_BYTE;
            early += busy < SLOT;
            f.ts = S0 + busy + PROP_PS;
            frame_store_link(&msg[n_out++], f);
            if (start && held)
            {
                head = head + 1 == cap ? 0 : head + 1;
                held--;
            }
            else if (start)
            {
                lq--;
                jq++;
                while (jq < i && list[jq] == ~0u)
                    jq++;
            }
        }
        else
            frame_copy(here, &f);
    }
    for (; lq; jq++)
    {
        if (list[jq] == ~0u)
            continue;
        const int at = head + held;
        frame_copy(&ring[at < cap ? at : at - cap], &sh.fr()[list[jq] & 511]);
        held++;
        lq--;
    }
    size = held;
    msg_seal(s, x.gt, out_link, n_out, early);
    pr.q_head = head;
    pr.q_size = size;
    if (n_out)
    {
        pr.link_free = S0 + busy;
        pr.last_start = S0 + began;
        pr.last = wire;
    }
    return n_out > 0 || size > 0;
}

// ------------------------------------------------------------------ slots beyond the staging area
TB_D Input input_of(const SwCtx &x, const SwShared &sh, int q)
{
    Input in;
    in.i2 = sh.win[q][0];
    in.n2 = sh.win[q][1];
    in.n1 = sh.win[q][2];
    int link = x.ports[q].in_link;
    if (link < 0)
        link = 0; // (an unused port's window is empty; any link gives valid pointers)
    in.m2 = x.gt >= 2 ? msg_frames(*x.s, x.gt - 2, link) : nullptr;
    in.m1 = x.gt >= 1 ? msg_frames(*x.s, x.gt - 1, link) : nullptr;
    return in;
}

// phase 1 (lane q < k): clear its row
TB_D void sw_phase_clear(const SwCtx &x, SwShared &sh, int q)
{
    for (int i = 0; i <= x.sr->k; i++)
        sh.rows()[q][i] = 0;
}

TB_D int sw_egress_of(const SwCtx &x, const Input &in, int q, int j)
{
    Frame f;
    frame_load_link(f, in.at(j));
    return sw_egress_for(x, f, q, x.spray ? x.s->sw_up[x.scratch + (size_t)q * 2 * MAX_TX + j] : 0);
}

// phase 2 (one lane): per-packet ECMP draws, one per forwarded packet in the order the packets
// arrive at the node (all ports merged), from the switch's MRG32k3a stream
TB_D void sw_phase_spray(const SwCtx &x, const SwShared &sh, unsigned &ties)
{
    const int k = x.sr->k;
    int pos[32];
    for (int q = 0; q < k; q++)
        pos[q] = 0;
    Rng st = x.s->sw_rng[x.sw];
    const WorldDesc &wd = *x.wd;
    for (;;)
    {
        int best = -1;
        Frame bf, f;
        for (int q = 0; q < k; q++)
        {
            Input in = input_of(x, sh, q);
            if (pos[q] >= in.count())
                continue;
            in.load(f, pos[q]);
            if (best < 0 || f.ts < bf.ts || (f.ts == bf.ts && frame_before(f, bf, ties)))
            {
                best = q;
                bf = f;
            }
        }
        if (best < 0)
            break;
        int ep = wd.n_fail ? epoch_of(wd, bf.ts) : 0;
        if (!port_down(wd, x.sr->local, best, ep))
        {
            int nr = routes_to(wd, x.sr->local, bf.dst, ep);
            x.s->sw_up[x.scratch + (size_t)best * 2 * MAX_TX + pos[best]] = (uint8_t)(nr ? rand_int(st, (uint32_t)nr) : 0);
        }
        pos[best]++;
    }
    x.s->sw_rng[x.sw] = st;
}

// phase 3 (lane q): count arrivals per egress port; returns the drops at a down interface
TB_D unsigned sw_phase_count(const SwCtx &x, SwShared &sh, int q)
{
    Input in = input_of(x, sh, q);
    unsigned dropped = 0;
    int n = in.count();
    for (int j = 0; j < n; j++)
    {
        int e = sw_egress_of(x, in, q, j);
        if (e >= 0)
            sh.rows()[q][e]++;
        else
            dropped++;
    }
    return dropped;
}

// phase 4 (lane e): offsets of each ingress port's arrivals within egress e
TB_D void sw_phase_offsets(const SwCtx &x, SwShared &sh, int e)
{
    int off = 0;
    for (int j = 0; j < x.sr->k; j++)
    {
        int c = sh.rows()[j][e];
        sh.rows()[j][e] = off;
        off += c;
    }
    sh.cnt[e] = off;
}

// phase 5 (lane e): egress e's region
TB_D void sw_phase_base(const SwCtx &x, SwShared &sh, int e)
{
    int b = 0;
    for (int j = 0; j < e; j++)
        b += sh.cnt[j];
    sh.base[e] = b;
}

// phase 6 (lane q): scatter (time, source) of each arrival to its egress region
TB_D void sw_phase_scatter(const SwCtx &x, SwShared &sh, int q)
{
    Input in = input_of(x, sh, q);
    int64_t *ts = x.s->sw_ts + x.scratch;
    uint32_t *ref = x.s->sw_ref + x.scratch;
    int n = in.count();
    for (int j = 0; j < n; j++)
    {
        int e = sw_egress_of(x, in, q, j);
        if (e < 0)
            continue;
        int at = sh.base[e] + sh.rows()[q][e]++;
        ts[at] = in.ts(j);
        ref[at] = (uint32_t)(q << 16 | j);
    }
}

// phase 7 (lane e): egress e's arrivals in time order (ties: ns-3's order, insertion sort in
// ingress order), each enqueued (RED) with its arrival event's chain; then the starts of the
// slot. Returns true if the port sent or holds frames.
TB_D bool sw_phase_egress(const SwCtx &x, SwShared &sh, int e, SwCounts &cn)
{
    const Sim &s = *x.s;
    const int n = sh.cnt[e];
    int64_t *ts = s.sw_ts + x.scratch + sh.base[e];
    uint32_t *ref = s.sw_ref + x.scratch + sh.base[e];
    auto load_ref = [&](Frame &f, uint32_t r) { input_of(x, sh, (int)(r >> 16)).load(f, (int)(r & 0xFFFF)); };
    for (int i = 1; i < n; i++)
    {
        int64_t tx = ts[i];
        uint32_t r = ref[i];
        int j = i - 1;
        while (j >= 0)
        {
            if (ts[j] < tx)
                break;
            if (ts[j] == tx)
            {
                Frame a, b;
                load_ref(a, r);
                load_ref(b, ref[j]);
                if (!frame_before(a, b, cn.ties))
                    break;
            }
            ts[j + 1] = ts[j];
            ref[j + 1] = ref[j];
            j--;
        }
        ts[j + 1] = tx;
        ref[j + 1] = r;
    }
    PortRec &pr = x.ports[e];
    const int port = x.sr->port0 + e;
    Egress eg;
    const int out_link = s.H + port;
    eg.open(s.port_ring + (size_t)port * s.ring, s.ring, pr.q_head, pr.q_size, pr.link_free, pr.last_start, &pr.last, pr.red_k, pr.qcap,
            (x.t + 1) * SLOT_PS, s.msg + msg_index(s, x.gt, out_link) * MAX_TX);
#ifdef TB_QTRACE
    eg.qs = &s;
    eg.qnode = x.wd->H1 + x.sr->local;
    eg.qdev = e + 1;
#endif
    for (int i = 0; i < n; i++)
    {
        Frame p;
        load_ref(p, ref[i]);
        chain_child(p.ch, p.ch, code_arrival(p.len)); // queued: the arrival event's chain
        eg.enqueue(p, p.ts);
    }
    eg.advance(eg.horizon - 1);
    msg_seal(s, x.gt, out_link, eg.n_out, eg.early);
    pr.q_head = eg.head;
    pr.q_size = eg.size;
    pr.link_free = eg.busy_until;
    pr.last_start = eg.began;
    cn.drops += eg.drops;
    cn.marks += eg.marks;
    cn.ovf += eg.ovf;
    return eg.n_out > 0 || eg.size > 0;
}

} // namespace tb
