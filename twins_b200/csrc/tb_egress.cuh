// twins-b200: frame moves and the egress port (a point-to-point device: one-packet device queue
// under a RED queue disc), used by hosts and switch ports.
#pragma once
#include "tb_state.cuh"

namespace tb
{

// Frames that cross entities (link messages) move through L2 only: readers in later slots run
// on other SMs, whose L1 would otherwise hold stale lines (the persistent kernel is never
// relaunched between slots).
TB_D void frame_copy(Frame *d, const Frame *s)
{
    const uint4 *a = reinterpret_cast<const uint4 *>(s);
    uint4 *b = reinterpret_cast<uint4 *>(d);
    uint4 v[FRAME_WORDS];
#pragma unroll
    for (int i = 0; i < FRAME_WORDS; i++)
        v[i] = a[i];
#pragma unroll
    for (int i = 0; i < FRAME_WORDS; i++)
        b[i] = v[i];
}
TB_D void frame_load_link(Frame &d, const Frame *s)
{
#if defined(__CUDA_ARCH__)
    const uint4 *a = reinterpret_cast<const uint4 *>(s);
    uint4 *b = reinterpret_cast<uint4 *>(&d);
#pragma unroll
    for (int i = 0; i < FRAME_WORDS; i++)
        b[i] = __ldcg(a + i);
#else
    d = *s;
#endif
}
TB_D void frame_store_link(Frame *d, const Frame &s)
{
#if defined(__CUDA_ARCH__)
    const uint4 *a = reinterpret_cast<const uint4 *>(&s);
    uint4 *b = reinterpret_cast<uint4 *>(d);
#pragma unroll
    for (int i = 0; i < FRAME_WORDS; i++)
        __stcg(b + i, a[i]);
#else
    *d = s;
#endif
}
TB_D int64_t ts_load_link(const Frame *s)
{
#if defined(__CUDA_ARCH__)
    return __ldcg(&s->ts);
#else
    return s->ts;
#endif
}
TB_D int64_t tag_load(const int64_t *p)
{
#if defined(__CUDA_ARCH__)
    return __ldcg(p);
#else
    return *p;
#endif
}
TB_D void tag_store(int64_t *p, int64_t v)
{
#if defined(__CUDA_ARCH__)
    __stcg(p, v);
#else
    *p = v;
#endif
}

TB_D void ev_add(const Sim &s, int world, int i, unsigned long long n)
{
    if (!n)
        return;
#if defined(__CUDA_ARCH__)
    atomicAdd(&s.ev[i], n);
    atomicAdd(&s.ev_w[(size_t)world * EV_N + i], n);
#else
    s.ev[i] += n;
    s.ev_w[(size_t)world * EV_N + i] += n;
#endif
}

// link messages: slot `slot` of link `link`
TB_D size_t msg_index(const Sim &s, int64_t slot, int link) { return (size_t)(slot & (NB - 1)) * s.L + link; }
// Its frames and how many of them arrive in the slot after it, the first ones; the others arrive in the
// next. The sender, which knows the arrival times, says so in the tag, so that a reader takes the
// frames of its slot and no others: the late ones of the message before last, the early ones of the last.
struct MsgTag
{
    int n, early;
};
TB_D MsgTag msg_tag(const Sim &s, int64_t slot, int link)
{
    const int64_t v = slot >= 0 ? tag_load(&s.msg_tag[msg_index(s, slot, link)]) : -1;
    MsgTag m = {0, 0};
    if (slot >= 0 && (v >> 20) == slot)
        m = {(int)(v & 1023), (int)(v >> 10 & 1023)};
    return m;
}
static_assert(MAX_TX < 1024, "a tag's counts");
TB_D void msg_seal(const Sim &s, int64_t slot, int link, int n, int early)
{
    tag_store(&s.msg_tag[msg_index(s, slot, link)], slot << 20 | (int64_t)early << 10 | n);
}
TB_D const Frame *msg_frames(const Sim &s, int64_t slot, int link) { return s.msg + msg_index(s, slot, link) * MAX_TX; }

#ifdef TB_QTRACE
// the enqueue trace: frame g joined the queue disc of (node, dev) at `now` behind `backlog` frames
TB_D void qtrace_enqueue(const Sim &s, int node, int dev, const Frame &g, int backlog, int64_t now)
{
    if (!s.qtrace || now >= s.qtrace_until || now < s.qtrace_from)
        return;
#if defined(__CUDA_ARCH__)
    const unsigned long long i = atomicAdd(s.qtrace_cnt, 1ull);
#else
    const unsigned long long i = (*s.qtrace_cnt)++;
#endif
    if (i >= s.qtrace_n)
        return;
    QRec &r = s.qtrace[i];
    const SndRec &S = s.snd[g.flow];
    r.ts = now;
    r.node = node;
    r.dev = dev;
    r.src = g.to_sender ? S.dst_local : S.src_local;
    r.dst = g.to_sender ? S.src_local : S.dst_local;
    r.sa = g.sa;
    r.len = g.len;
    r.qlen = (uint16_t)(backlog + 1);
    r.flags = g.flags;
}
#endif

// The sending end of a point-to-point link for one slot: ns-3's RED queue disc over a one-packet
// device queue over the wire (reference: src/step.cuh:163-317). `ring` holds the frames that have
// not started, each stamped with its enqueue time; the wire is busy until `busy_until` with the
// frame that began at `began`, whose chain is *tx_chain. A frame begins at max(its enqueue time,
// busy_until); its transmission's copy, stamped with its arrival at the far end, goes to this
// slot's link message `msg` (at most MAX_TX; more is counted as an overflow). (Hosts that share a warp,
// and a switch port in a slot beyond the staging area; HostNic and sw_egress_staged are the same device a
// slot at a time.)
struct Egress
{
    Frame *ring;
    int cap, head, size;
    int64_t busy_until, began;
    Chain *tx_chain;
    int red_k, qcap;
    int64_t horizon;    // the slot's end: nothing begins at or after it
    int64_t kicked;     // the instant of a ScheduleNow'd event being handled (-1: none)
    int64_t idle_began; // the last start this slot on an idle wire (-1: none)
    Frame *msg;
    int n_out, early; // frames started, of which the first `early` arrive in the next slot
    unsigned drops, marks, ovf, offered;
#ifdef TB_QTRACE
    const Sim *qs; // the trace's sink; the queue's ns-3 node and device
    int qnode, qdev;
#endif

    TB_D void open(Frame *ring_, int cap_, int head_, int size_, int64_t busy_until_, int64_t began_, Chain *tx_chain_, int red_k_,
                   int qcap_, int64_t horizon_, Frame *msg_)
    {
        ring = ring_;
        cap = cap_;
        head = head_;
        size = size_;
        busy_until = busy_until_;
        began = began_;
        tx_chain = tx_chain_;
        red_k = red_k_;
        qcap = qcap_;
        horizon = horizon_;
        kicked = idle_began = -1;
        msg = msg_;
        n_out = early = 0;
        drops = marks = ovf = offered = 0;
    }

    // every waiting frame that begins by `until` (and before the horizon) goes on the wire; a frame
    // that found the wire busy begins at the previous one's TransmitComplete, whose chain is its
    // parent's; one that found it idle begins at its own enqueue, its chain unchanged
    TB_D void advance(int64_t until)
    {
        for (; size; size--)
        {
            const Frame &f = ring[head];
            const int64_t t0 = f.ts > busy_until ? f.ts : busy_until;
            if (t0 > until || t0 >= horizon)
                return;
            if (n_out == MAX_TX)
            {
                ovf++;
                return;
            }
            const int64_t t1 = t0 + (int64_t)f.len * PS_PER_BYTE; // (its end, read before the stores below)
            const bool behind = busy_until >= f.ts && busy_until > began;
            Frame o;
            frame_copy(&o, &f);
            if (behind)
                chain_child(o.ch, *tx_chain, code_tc((int)((busy_until - began) / PS_PER_BYTE)));
            else
                idle_began = t0;
            *tx_chain = o.ch;
            began = t0;
            busy_until = t1;
            o.ts = t1 + PROP_PS;
            frame_store_link(&msg[n_out++], o);
            early += t1 < horizon; // (PROP_PS is a slot)
            head = head + 1 == cap ? 0 : head + 1;
        }
    }

    // the frames RED counts at `now`: the waiting ones, less the one the device queue holds while
    // the wire is busy, once the Wake that refills it has run. The Wake is ScheduleNow'd when a
    // transmission begins, so it has run for one that began earlier; for one that began at this
    // instant only a ScheduleNow'd event sees it, after a start on an idle wire (a start at a
    // TransmitComplete comes after the arrivals that scheduled such events).
    TB_D int disc_backlog(int64_t now) const
    {
        if (!size || busy_until <= now)
            return size;
        const bool woken = began < now || (kicked == now && idle_began == now);
        return size - (woken ? 1 : 0);
    }

    // a frame offered at `now` (its ts becomes now): the wire first takes what begins by now; RED
    // with MinTh = MaxTh = K and weight 1 (no averaging) marks an ECT frame or drops another when
    // the backlog is at least K (and above 1); then the disc's limit drops. False: dropped.
    TB_D bool enqueue(Frame &g, int64_t now)
    {
        offered++;
        advance(now);
        const int backlog = disc_backlog(now);
        g.ts = now;
        if (backlog >= red_k && backlog > 1)
        {
            if (!(g.flags & F_ECT))
            {
                drops++;
                return false;
            }
            g.flags |= F_CE;
            marks++;
        }
        if (backlog >= qcap)
        {
            drops++;
            return false;
        }
#ifdef TB_QTRACE
        qtrace_enqueue(*qs, qnode, qdev, g, backlog, now);
#endif
        if (size == cap)
        {
            ovf++;
            return false;
        }
        const int at = head + size < cap ? head + size : head + size - cap;
        frame_copy(&ring[at], &g);
        size++;
        return true;
    }
};
// The sending end of a host that has a warp of its own (the same device). The sockets never look at it, so the slot's events only
// append the frames they offer, each stamped with its time, to a list on chip, and `run` plays the
// list through the device, a frame per iteration that starts on the wire or joins the queue, in
// offsets in the slot; what is still queued then joins the ring. (With the device's code at every
// place that sends a frame, and each frame written to the ring in memory and read back to start,
// the event loop took more instructions and waited on every frame: a load from a line that was just
// stored takes 600 cycles longer than another.) OFFER_KICK in a
// frame's to_sender: offered by a ScheduleNow'd event of its instant.
constexpr uint8_t OFFER_KICK = 2;
constexpr int OUT_FRAMES = 16; // the list's capacity (a slot takes 8 full frames; more frames in a slot are played in parts)
struct HostNic
{
    const Sim *s;
    Frame *ring;
    int cap, head, size; // the ring
    int busy, began, tx_len; // the wire: busy until `busy` with a frame of tx_len bytes that began at `began` (offsets)
    int idle_at;         // the last start this slot on an idle wire (-1: none)
    int red_k, qcap;
    int64_t S0;
    Frame *msg;
    Chain *wire;         // the chain of the frame on the wire
    int n_out, early;
    unsigned drops, marks, ovf, offered;
    int node;

    TB_D void open(const Sim &s_, HostRec &hr, Frame *ring_, const WorldDesc &wd, int64_t S0_, Frame *msg_)
    {
        s = &s_;
        ring = ring_;
        cap = s_.ring;
        head = hr.q_head;
        size = hr.q_size;
        S0 = S0_;
        busy = -1;
        began = -(int)SLOT_PS;
        tx_len = 0;
        if (hr.link_free >= S0)
        {
            busy = (int)(hr.link_free - S0);
            tx_len = (int)((uint32_t)(hr.link_free - hr.last_start) / (uint32_t)PS_PER_BYTE);
            began = busy - tx_len * (int)PS_PER_BYTE;
        }
        idle_at = -1;
        red_k = wd.red_k;
        qcap = wd.qcap;
        msg = msg_;
        wire = &hr.last;
        n_out = early = 0;
        drops = marks = ovf = offered = 0;
        node = hr.local;
    }
    TB_D void close(HostRec &hr) const
    {
        hr.q_head = head;
        hr.q_size = size;
        if (n_out)
        {
            hr.link_free = S0 + busy;
            hr.last_start = S0 + began;
        }
    }

    // the frames list[0..n), offered in this order, and every start by `until` (an offset). A queued
    // frame begins when the wire gets free (it was queued because the wire was busy beyond its
    // offer), behind the frame on the wire, whose chain is its parent's; one offered at an idle wire
    // begins at once, its chain unchanged. RED as in Egress; a ScheduleNow'd event also sees the
    // Wake of a start on an idle wire at its own instant.
    TB_D void run_list(Frame *list, int n, int until)
    {
        constexpr int SLOT = (int)SLOT_PS;
        Chain on = *wire;
        int i = 0, jq = 0, lq = 0; // the next offer; list[jq]: the first queued from the list; their number
        const int n_out0 = n_out;
        for (;;)
        {
            const int waiting = size + lq;
            const int ta = i < n ? (int)(list[i].ts - S0) : until;
            const bool room = n_out < MAX_TX, start = waiting > 0 && busy < SLOT && busy <= ta && room;
            if (!start && i >= n)
                break;
            Frame f;
            frame_copy(&f, start ? (size ? &ring[head] : &list[jq]) : &list[i]);
            const bool kick = f.to_sender & OFFER_KICK;
            f.to_sender &= 1; // (the list's mark is no part of the frame: not on the wire, not in the trace)
            if (!start)
                offered++;
            const bool idle = waiting == 0 && busy <= ta && room;
            if (start || idle)
            {
                const bool behind = start || (busy == ta && tx_len > 0);
                if (behind)
                    chain_child(f.ch, on, code_tc(tx_len));
                else
                    idle_at = ta;
#ifdef TB_QTRACE
                if (!start)
                    qtrace_enqueue(*s, node, 1, f, 0, f.ts);
#endif
                on = f.ch;
                began = start ? busy : ta;
                tx_len = f.len;
                busy = began + tx_len * (int)PS_PER_BYTE;
                f.ts = S0 + busy + PROP_PS;
                frame_store_link(&msg[n_out++], f);
                early += busy < SLOT;
                if (!start)
                {
                    i++;
                    jq = i;
                }
                else if (size)
                {
                    head = head + 1 == cap ? 0 : head + 1;
                    size--;
                }
                else
                {
                    lq--;
                    jq++;
                    while (jq < i && list[jq].len == 0)
                        jq++; // (dropped)
                }
                continue;
            }
            // an offer that finds the wire busy, or frames waiting
            const bool woken = began < ta || (kick && idle_at == ta);
            const int backlog = !waiting || busy <= ta ? waiting : waiting - (woken ? 1 : 0);
            bool gone = false;
            ovf += !room;
            if (backlog >= red_k && backlog > 1)
            {
                if (f.flags & F_ECT)
                {
                    f.flags |= F_CE;
                    list[i].flags = f.flags;
                    marks++;
                }
                else
                    gone = true;
            }
            gone |= backlog >= qcap;
            drops += gone;
#ifdef TB_QTRACE
            if (!gone)
                qtrace_enqueue(*s, node, 1, f, backlog, f.ts);
#endif
            if (!gone && waiting == cap)
            {
                ovf++;
                gone = true;
            }
            if (gone)
                list[i].len = 0;
            if (lq == 0)
                jq = gone ? i + 1 : i;
            lq += !gone;
            i++;
        }
        for (; lq; jq++)
        {
            if (list[jq].len == 0)
                continue;
            const int at = head + size;
            list[jq].to_sender &= 1;
            frame_copy(&ring[at < cap ? at : at - cap], &list[jq]);
            size++;
            lq--;
        }
        if (n_out != n_out0)
            *wire = on;
    }
};

} // namespace tb
