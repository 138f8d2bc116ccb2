// A randomized check of the two forms of a switch port's slot (twins_b200/csrc/tb_switch.cuh), built with g++
// for the host, in the enqueue trace's build, by tests/test_host_nic.py: the same arrivals, slot after slot,
// go to sw_egress_staged (a slot staged in shared memory, a frame per iteration) and to an Egress as
// sw_phase_egress drives it (a slot run from L2). Queues small and deep, arrivals at one instant and at the
// instant the wire gets free: the link messages and their tags (chains among them), the held frames, the
// port's record, the counts and the traced enqueues must be the same. Exit status 0: all agree.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

struct uint4
{
    unsigned x, y, z, w;
};
// (the header's warp-wide code is compiled, not run, here)
#define __device__
static inline void __syncwarp() {}
static inline unsigned __ballot_sync(unsigned, bool b) { return b; }
static inline bool __any_sync(unsigned, bool b) { return b; }
static inline unsigned __reduce_min_sync(unsigned, unsigned v) { return v; }
static inline int __shfl_sync(unsigned, int v, int) { return v; }
static inline int __popc(unsigned v) { return __builtin_popcount(v); }
static inline int __ffs(int v) { return __builtin_ffs(v); }
#define TB_QTRACE
#include "tb_switch.cuh"

using namespace tb;

namespace
{
constexpr int FLOWS = 4, QREC = 4096, CAP = 384;

struct Side
{
    Sim s{};
    WorldDesc wd{};
    SwRec sr{};
    PortRec pr{};
    std::vector<Frame> ring, msg;
    std::vector<int64_t> tag;
    std::vector<SndRec> snd;
    std::vector<QRec> q;
    std::vector<uint4> shared;
    unsigned long long nq = 0;
    SwCounts c{};
    bool act = false;

    Side(int red_k, int qcap)
        : ring(qcap + 2), msg((size_t)NB * MAX_TX), tag(NB, -1), snd(FLOWS), q(QREC), shared(sw_shared_bytes(CAP) / 16)
    {
        for (int f = 0; f < FLOWS; f++)
        {
            snd[f].src_local = 7 + f;
            snd[f].dst_local = 90 + f;
        }
        s.ring = qcap + 2;
        s.L = 1;
        s.port_ring = ring.data();
        s.msg = msg.data();
        s.msg_tag = tag.data();
        s.snd = snd.data();
        s.qtrace = q.data();
        s.qtrace_cnt = &nq;
        s.qtrace_n = QREC;
        s.qtrace_until = INT64_MAX;
        wd.H1 = 128;
        sr.local = 3;
        sr.k = 1;
        pr.red_k = red_k;
        pr.qcap = qcap;
    }
    void staged(int64_t t, const std::vector<Frame> &in)
    {
        SwShared &sh = *sw_shared_at(reinterpret_cast<unsigned char *>(shared.data()), CAP);
        SwCtx x{};
        x.s = &s;
        x.wd = &wd;
        x.sr = &sr;
        x.ports = &pr;
        x.t = x.gt = t;
        // (staged in another order than that of their arrivals)
        const int n = (int)in.size();
        uint32_t *list = sh.key();
        for (int i = 0; i < n; i++)
        {
            const int at = (i * 7 + 3) % (n % 7 ? n : n + 1);
            sh.fr()[at] = in[i];
            list[i] = (uint32_t)(in[i].ts - t * SLOT_PS) << 9 | (uint32_t)at;
        }
        nq = 0;
        act = sw_egress_staged(x, sh, 0, list, n, c);
    }
    void unstaged(int64_t t, const std::vector<Frame> &in)
    {
        Egress eg;
        eg.open(ring.data(), s.ring, pr.q_head, pr.q_size, pr.link_free, pr.last_start, &pr.last, pr.red_k, pr.qcap, (t + 1) * SLOT_PS,
                s.msg + msg_index(s, t, 0) * MAX_TX);
        eg.qs = &s;
        eg.qnode = wd.H1 + sr.local;
        eg.qdev = 1;
        nq = 0;
        for (Frame p : in)
        {
            chain_child(p.ch, p.ch, code_arrival(p.len));
            eg.enqueue(p, p.ts);
        }
        eg.advance(eg.horizon - 1);
        msg_seal(s, t, 0, eg.n_out, eg.early);
        pr.q_head = eg.head;
        pr.q_size = eg.size;
        pr.link_free = eg.busy_until;
        pr.last_start = eg.began;
        c.drops += eg.drops;
        c.marks += eg.marks;
        c.ovf += eg.ovf;
        act = eg.n_out > 0 || eg.size > 0;
    }
};

bool check(const Side &a, const Side &b, int trial, int64_t t)
{
    auto differ = [&](const char *what, long long x, long long y) {
        if (x != y)
            printf("trial %d slot %lld: %s %lld, staged %lld\n", trial, (long long)t, what, x, y);
        return x != y;
    };
    const int at = (int)(t & (NB - 1)), n = (int)(a.tag[at] & 1023);
    if (differ("tag", a.tag[at], b.tag[at]) || differ("active", a.act, b.act) || differ("held", a.pr.q_size, b.pr.q_size) ||
        differ("drops", a.c.drops, b.c.drops) || differ("marks", a.c.marks, b.c.marks) || differ("overflows", a.c.ovf, b.c.ovf) ||
        differ("wire free", a.pr.link_free, b.pr.link_free) || differ("last start", a.pr.last_start, b.pr.last_start) ||
        differ("traced", (long long)a.nq, (long long)b.nq))
        return false;
    if (memcmp(&a.pr.last, &b.pr.last, sizeof(Chain)) != 0)
        return printf("trial %d slot %lld: the wire's chain\n", trial, (long long)t), false;
    for (int i = 0; i < n; i++)
        if (memcmp(&a.msg[(size_t)at * MAX_TX + i], &b.msg[(size_t)at * MAX_TX + i], sizeof(Frame)) != 0)
            return printf("trial %d slot %lld: frame %d sent\n", trial, (long long)t, i), false;
    for (int i = 0; i < a.pr.q_size; i++)
        if (memcmp(&a.ring[(a.pr.q_head + i) % a.s.ring], &b.ring[(b.pr.q_head + i) % b.s.ring], sizeof(Frame)) != 0)
            return printf("trial %d slot %lld: frame %d held\n", trial, (long long)t, i), false;
    for (unsigned long long i = 0; i < a.nq; i++)
    {
        const QRec &x = a.q[i], &y = b.q[i];
        if (x.ts != y.ts || x.node != y.node || x.dev != y.dev || x.src != y.src || x.dst != y.dst || x.sa != y.sa || x.len != y.len ||
            x.qlen != y.qlen || x.flags != y.flags)
            return printf("trial %d slot %lld: enqueue %llu\n", trial, (long long)t, i), false;
    }
    return true;
}
} // namespace

int main()
{
    std::mt19937 rng(11);
    auto below = [&](int n) { return (int)(rng() % (unsigned)n); };
    long long sent = 0, held = 0, traced = 0, dropped = 0, marked = 0, ties = 0, meets = 0;
    for (int trial = 0; trial < 500; trial++)
    {
        const int red_k = 1 + below(trial % 3 ? 6 : 40), qcap = red_k + below(trial % 2 ? 3 : 60);
        const int lens[4] = {CTRL_LEN, SYN_LEN, 42 + 700, 42 + (int)MSS}, most = trial % 5 == 0 ? 120 : 14;
        Side a(red_k, qcap), b(red_k, qcap);
        for (int64_t t = 0; t < 60; t++)
        {
            const int64_t S0 = t * SLOT_PS;
            std::vector<Frame> in;
            int64_t now = S0 + (below(4) ? below((int)SLOT_PS) : 0), free = a.pr.link_free;
            for (int left = below(3) ? below(most) : 0; left > 0 && now < S0 + SLOT_PS; left--)
            {
                const int f = below(FLOWS), data = below(2);
                Frame p;
                memset(&p, 0, sizeof p);
                p.ts = now;
                p.flow = (uint32_t)f;
                p.sa = rng();
                p.len = (uint16_t)lens[data ? 2 + below(2) : below(2)];
                p.dst = (uint16_t)(90 + f);
                p.flags = (uint8_t)((data ? F_DATA : F_ACK) | (below(3) ? F_ECT : 0));
                p.to_sender = (uint8_t)(!data);
                p.up = (uint16_t)below(16);
                chain_app_root(p.ch, below(50), f);
                for (int r = below(12); r > 0; r--)
                    chain_child(p.ch, p.ch, (uint16_t)(1 + below(5000)));
                in.push_back(p);
                // (the wire's next free instant if nothing is dropped: an arrival may fall on it)
                free = (free > now ? free : now) + p.len * PS_PER_BYTE;
                const int how = below(5);
                ties += how == 0;
                if (how == 1 && free < S0 + SLOT_PS)
                    now = free, meets++;
                else if (how)
                    now += 1 + below(most > 14 ? 30'000 : 150'000);
            }
            a.unstaged(t, in);
            b.staged(t, in);
            if (!check(a, b, trial, t))
                return 1;
            sent += a.tag[t & (NB - 1)] & 1023;
            held += a.pr.q_size > 0;
            traced += (long long)a.nq;
        }
        dropped += a.c.drops;
        marked += a.c.marks;
    }
    printf("%lld frames sent, %lld slots ended with frames held, %lld enqueues, %lld drops, %lld marks, %lld ties, %lld on the wire's end\n", sent,
           held, traced, dropped, marked, ties, meets);
    return sent && held && traced && dropped && marked && ties && meets ? 0 : 2;
}
