// twins-b200: one slot of a host, and a switch's routes.
//   host_step   (reference: src/step.cuh:2250-2528) one thread per host: every event of the host
//               in [t us, t+1 us) in ns-3's order: arrivals, timers, application starts
//   route, ...  (reference: src/step.cuh:2530-2705) a frame's egress port (per-flow ECMP or a spraying
//               choice, link failures) and ns-3's order of simultaneous arrivals; the switch's slot itself
//               is tb_switch.cuh's and tb_kernel.cu's switch_step
#pragma once
#include "tb_tcp.cuh"

namespace tb
{

// the chain of a timer (due_chain, step.cuh:2241-2247)
TB_D const Chain &due_chain(const Sim &s, const Due &d)
{
    switch (d.kind)
    {
    case 1:
    case 3:
    case 4:
        return s.rcv[d.flow].dchain;
    case 5:
        return s.rcv[d.flow].fchain;
    case 2:
        return s.snd[d.flow].st == S_EST ? s.snd[d.flow].schain : s.snd[d.flow].rchain;
    default:
        return s.snd[d.flow].rchain;
    }
}

// a receiver that can arm no timer any more: all its timers idle and everything received (or,
// with FIN, the connection closed)
TB_D bool rcv_idle_for_good(const RcvRec &R)
{
    if (R.delack_at >= 0 || R.syn_at >= 0 || R.last_at >= 0 || R.frx_at >= 0)
        return false;
    if (R.fin_on)
        return R.st == R_CLOSED;
    return R.est && R.rcv_nxt >= R.bytes;
}

// One slot of host h. Returns true if it sent or holds frames; *wake: the next slot it must run.
// t: the world's own slot (time); gt: the launch's slot, which indexes the link messages (equal
// in a batch; a world that joins a running launch starts its own time at a later launch slot).
// Its arrivals: n2 frames of msg[gt-2] from frame first2 on, then the first n1 of msg[gt-1]; `stage`: copied
// to shared memory by its warp, or null to read them in place.
// KEEP (one host per warp): the records last used stay in registers between events (Recs); the active
// lists are left unpruned and *wake counts only the host's queue and its next application start; the
// caller prunes them (prune_lists_warp) and lowers the wake-up to the earliest timer of the
// connections that stay. `due`: the timers due in the slot, already collected
// in this function's scan order (the first DUE_CAP of them; due_ovf more were left out), with room
// for DUE_CAP, or null to scan the active lists here.
// `out` (KEEP): the list of the frames its events offer, room for OUT_FRAMES.
template <bool KEEP>
TB_D bool host_step(const Sim &s, int h, int64_t t, int64_t gt, int64_t *wake, unsigned *ties_out, unsigned *done_out, Frame *out,
                    const Frame *stage, int first2, int n2, int n1, Due *due = nullptr,
                    int due_n = 0, int due_ovf = 0)
{
    const int64_t S0 = t * SLOT_PS, E0 = S0 + SLOT_PS;
    TB_PHASE_START
    HostRec &hr = s.hosts[h];
    const Frame *m2 = stage ? stage : msg_frames(s, gt - 2, hr.in_link) + first2, *m1 = stage ? stage + n2 : msg_frames(s, gt - 1, hr.in_link);
    int i2 = 0, i1 = 0;
    auto frame_at = [&](Frame &d, const Frame *m, int j) {
        if (stage)
            d = m[j];
        else
            frame_load_link(d, &m[j]);
    };
    if (n2 == 0 && n1 == 0 && t < hr.wake && hr.q_size == 0)
    {
        *wake = hr.wake;
        return false;
    }
    const WorldDesc &wd = s.worlds[hr.world];
    HostCtx c;
    c.s = &s;
    c.wd = &wd;
    c.h = h;
    c.dctcp = wd.cc == CC_DCTCP;
    c.cubic = wd.cc == CC_CUBIC;
    c.slot_end = E0;
    c.retx = c.rtos = c.ovf = c.done = 0;
    c.pkts = c.snd_pkts = 0;
    HostNic nic;
    c.list = KEEP;
    c.nic = &nic;
    c.out = out;
    c.out_n = 0;
    c.kicked = -1;
    if (KEEP)
        nic.open(s, hr, s.host_ring + (size_t)h * s.ring, wd, S0, s.msg + msg_index(s, gt, h) * MAX_TX);
    else
    {
        c.eg.open(s.host_ring + (size_t)h * s.ring, s.ring, hr.q_head, hr.q_size, hr.link_free, hr.last_start, &hr.last, wd.red_k, wd.qcap,
                  E0, s.msg + msg_index(s, gt, h) * MAX_TX);
#ifdef TB_QTRACE
        c.eg.qs = &s;
        c.eg.qnode = hr.local;
        c.eg.qdev = 1;
#endif
    }
    unsigned ties = 0;
    Recs<KEEP> recs;

    TB_PHASE(0)
    // timers due in this slot (new timers lie >= 10 us ahead, except the 1 ps Send deferral,
    // which timer_in_slot adds), by time
    int *act_snd = s.act_snd + (size_t)h * s.act_cap, *act_rcv = s.act_rcv + (size_t)h * s.act_cap;
    const int ns = hr.n_snd, nr = hr.n_rcv;
    c.nd = 0;
    c.di = 0;
    Due own[DUE_CAP];
    c.due = due ? due : own;
    if (due)
    {
        c.nd = due_n;
        c.ovf += due_ovf;
    }
    for (int i = 0; i < (due ? 0 : ns); i++)
    {
        int f = act_snd[i];
        const SndRec &S = s.snd[f];
        int64_t a = S.rto_at, b = S.syn_at;
        if (a >= 0 && a < E0)
        {
            if (c.nd < DUE_CAP)
                c.due[c.nd++] = {a, f, 0};
            else
                c.ovf++;
        }
        if (b >= 0 && b < E0)
        {
            if (c.nd < DUE_CAP)
                c.due[c.nd++] = {b, f, 2};
            else
                c.ovf++;
        }
    }
    for (int i = 0; i < (due ? 0 : nr); i++)
    {
        int f = act_rcv[i];
        const RcvRec &R = s.rcv[f];
        int64_t v[4] = {R.delack_at, R.syn_at, R.last_at, R.frx_at};
        const int kinds[4] = {1, 3, 4, 5};
        for (int j = 0; j < 4; j++)
            if (v[j] >= 0 && v[j] < E0)
            {
                if (c.nd < DUE_CAP)
                    c.due[c.nd++] = {v[j], f, kinds[j]};
                else
                    c.ovf++;
            }
    }
    for (int i = 1; i < c.nd; i++)
    {
        Due x = c.due[i];
        int j = i - 1;
        while (j >= 0 && c.due[j].at > x.at)
        {
            c.due[j + 1] = c.due[j];
            j--;
        }
        c.due[j + 1] = x;
    }
    TB_PHASE(1)
    int pn = hr.pend_next;
    const int pe = hr.pend_end;
    Frame p;
    bool have_p = false; // p holds the next arrival
    // the next application event and its start (at or after E0: none this slot)
    int pm = -1;
    int64_t pst = INT64_MAX;
    auto next_pend = [&]() {
        pm = pn < pe ? s.pend_msg[pn] : -1;
        pst = pm >= 0 ? s.msgs[pm].start : INT64_MAX;
    };
    next_pend();
    for (;;)
    {
        int64_t tr = INT64_MAX, td = INT64_MAX, tp = INT64_MAX;
        if (!have_p)
        {
            if (i2 < n2)
            {
                frame_at(p, m2, i2);
                have_p = true;
            }
            else if (i1 < n1)
            {
                frame_at(p, m1, i1);
                have_p = true;
            }
        }
        if (have_p)
            tr = p.ts;
        if (c.di < c.nd)
            td = c.due[c.di].at;
        if (pst < E0)
            tp = pst;
        int64_t now = tr < td ? tr : td;
        now = now < tp ? now : tp;
        if (now == INT64_MAX)
            break;
        if (now < S0)
            now = S0;
        TB_PHASE(2)
        if (!KEEP)
            c.eg.advance(now);
        if (now == tp)
        {
            app_event(c, recs, hr, act_snd, pm, now);
            pn++;
            next_pend();
            TB_PHASE(10)
            continue;
        }
        bool timer = now == td;
        if (KEEP && timer && recs.S.f == c.due[c.di].flow)
            recs.flush(); // (its chain is read from the record)
        if (timer && now == tr)
        {
            // a timer and an arrival at the same instant: the one scheduled first
            Chain arr;
            chain_child(arr, p.ch, code_arrival(p.len));
            int r = chain_cmp(due_chain(s, c.due[c.di]), arr);
            if (r == 0)
                ties++;
            timer = r <= 0; // (undecided: the timer)
        }
        if (timer)
        {
            const Due d = c.due[c.di++];
            c.ech = due_chain(s, d);
            timer_event(c, recs, d, now);
            TB_PHASE(10)
            continue;
        }
        // the arrival
        if (i2 < n2)
            i2++;
        else
            i1++;
        have_p = false;
        c.pkts++;
        c.snd_pkts += p.to_sender;
        chain_child(c.ech, p.ch, code_arrival(p.len));
        on_frame(c, recs, hr, p, now);
        TB_PHASE(9)
    }
    if (KEEP)
        recs.flush();
    TB_PHASE(2)
    int sent, early, held;
    unsigned drops, marks, ovf, offered;
    if (KEEP)
    {
        nic_run(&nic, c.out, c.out_n, (int)SLOT_PS - 1);
        nic.close(hr);
        sent = nic.n_out, early = nic.early, held = nic.size;
        drops = nic.drops, marks = nic.marks, ovf = nic.ovf, offered = nic.offered;
    }
    else
    {
        c.eg.advance(E0 - 1);
        hr.q_head = c.eg.head;
        hr.q_size = c.eg.size;
        hr.link_free = c.eg.busy_until;
        hr.last_start = c.eg.began;
        sent = c.eg.n_out, early = c.eg.early, held = c.eg.size;
        drops = c.eg.drops, marks = c.eg.marks, ovf = c.eg.ovf, offered = c.eg.offered;
    }
    TB_PHASE(8)
    msg_seal(s, gt, h, sent, early);
    hr.pend_next = pn;

    TB_PHASE(3)
    // drop finished connections from the active lists; the next wake-up
    int64_t next = INT64_MAX;
    if (!KEEP)
    {
        int k = 0, n = hr.n_snd;
        for (int i = 0; i < n; i++)
        {
            int f = act_snd[i];
            const SndRec &S = s.snd[f];
            if (S.st == S_DONE)
                continue;
            act_snd[k++] = f;
            if (S.rto_at >= 0 && S.rto_at < next)
                next = S.rto_at;
            if (S.syn_at >= 0 && S.syn_at < next)
                next = S.syn_at;
        }
        hr.n_snd = k;
    }
    if (!KEEP)
    {
        int k = 0, n = hr.n_rcv;
        for (int i = 0; i < n; i++)
        {
            int f = act_rcv[i];
            const RcvRec &R = s.rcv[f];
            if (rcv_idle_for_good(R))
                continue;
            act_rcv[k++] = f;
            int64_t v[4] = {R.delack_at, R.syn_at, R.last_at, R.frx_at};
            for (int j = 0; j < 4; j++)
                if (v[j] >= 0 && v[j] < next)
                    next = v[j];
        }
        hr.n_rcv = k;
    }
    if (pst < next)
        next = pst;
    hr.wake = held > 0 ? t + 1 : (next == INT64_MAX ? INT64_MAX : next / SLOT_PS);
    *wake = hr.wake;
    TB_PHASE(4)
    // counters
    ev_add(s, hr.world, EV_DROPS, drops);
    ev_add(s, hr.world, EV_MARKS, marks);
    ev_add(s, hr.world, EV_RETX, c.retx);
    ev_add(s, hr.world, EV_RTO, c.rtos);
    ev_add(s, hr.world, EV_HOST_PKT, c.pkts);
    ev_add(s, hr.world, EV_HOST_SND, c.snd_pkts);
    ev_add(s, hr.world, EV_HOST_FRAMES, offered);
    ev_add(s, hr.world, EV_OVF_RING, c.ovf);
    ev_add(s, hr.world, EV_OVF_TX, ovf);
    ev_add(s, hr.world, EV_TIES, ties);
    *ties_out += ties;
    *done_out += c.done;
    TB_PHASE(5)
    return sent > 0 || held > 0;
}

// ------------------------------------------------------------------ switches
TB_D int epoch_of(const WorldDesc &wd, int64_t ts)
{
    int e = 0;
    while (e < wd.n_fail && ts >= wd.fail_t[e])
        e++;
    return e;
}
// the egress port at switch sw (world-local) towards host dst (world-local); `up` indexes the
// equal-cost routes (reference: src/step.cuh:2554-2591)
TB_D int route_up(const WorldDesc &wd, int sw, int dst, int up, int ep)
{
    if (wd.kind == TOPO_GRAPH)
    {
        int e = wd.host_sw[dst];
        if (e == sw)
            return wd.host_port[dst];
        size_t r = ((size_t)ep * wd.S1 + sw) * wd.S1 + e;
        return wd.rt_ports[wd.rt_off[r] + up];
    }
    if (wd.kind == TOPO_LEAFSPINE)
    {
        if (sw < wd.leaves)
            return dst / wd.hpl == sw ? dst % wd.hpl : wd.hpl + up;
        return dst / wd.hpl;
    }
    const int k = wd.k, hk = wd.hk, E = k * hk;
    int dst_pod = dst / (hk * hk), dst_edge = (dst / hk) % hk;
    if (sw < E)
        return (dst_pod == sw / hk && dst_edge == sw % hk) ? dst % hk : hk + up;
    if (sw < 2 * E)
        return dst_pod == (sw - E) / hk ? dst_edge : hk + up;
    return dst_pod;
}
TB_D int route(const Sim &s, const WorldDesc &wd, int sw, const Frame &p, int ep)
{
    if (wd.kind == TOPO_GRAPH)
    {
        int e = wd.host_sw[p.dst];
        if (e == sw)
            return wd.host_port[p.dst];
        // the flow hash modulo the routes at this switch
        const SndRec &S = s.snd[p.flow];
        uint32_t hsh = p.to_sender ? S.hash_ack : S.hash_data;
        return route_up(wd, sw, p.dst, (int)(hsh % wd.rt_n[((size_t)ep * wd.S1 + sw) * wd.S1 + e]), ep);
    }
    return route_up(wd, sw, p.dst, p.up, ep);
}
TB_D bool port_down(const WorldDesc &wd, int sw, int q, int ep)
{
    return wd.n_fail && wd.port_dn[((size_t)ep * wd.S1 + sw) * wd.k + q];
}
// equal-cost routes Ipv4GlobalRouting finds from sw towards dst (0: the host is attached)
TB_D int routes_to(const WorldDesc &wd, int sw, int dst, int ep)
{
    if (wd.kind == TOPO_GRAPH)
        return wd.host_sw[dst] == sw ? 0 : wd.rt_n[((size_t)ep * wd.S1 + sw) * wd.S1 + wd.host_sw[dst]];
    if (wd.kind == TOPO_LEAFSPINE)
        return sw < wd.leaves ? (dst / wd.hpl == sw ? 0 : wd.ecmp_n) : 1;
    const int hk = wd.hk, E = wd.k * hk;
    int dst_pod = dst / (hk * hk), dst_edge = (dst / hk) % hk;
    if (sw < E)
        return dst_pod == sw / hk && dst_edge == sw % hk ? 0 : wd.ecmp_n;
    if (sw < 2 * E)
        return dst_pod == (sw - E) / hk ? 1 : wd.ecmp_n;
    return 1;
}

// simultaneous arrivals at a switch, as ns-3 orders their Receive events: the longer frame
// started earlier upstream; else the chains of the upstream starts; else the lower connection id
// (a guess, counted) (frame_before, step.cuh:2693-2705)
TB_D bool frame_before(const Frame &a, const Frame &b, unsigned &ties)
{
    if (a.len != b.len)
        return a.len > b.len;
    int c = chain_cmp(a.ch, b.ch);
    if (c == 0)
        ties++;
    return c != 0 ? c < 0 : a.flow < b.flow;
}

} // namespace tb
