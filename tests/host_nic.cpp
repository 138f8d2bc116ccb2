// A randomized check of the two forms of a host's sending end (twins_b200/csrc/tb_egress.cuh), built with
// g++ for the host, in the enqueue trace's build, by tests/test_host_nic.py: the same offers through
// to_device go to an Egress frame by frame and to the list that HostNic plays at the slot's end (and in
// parts when more are offered than it holds). Slot after slot, with small queues and deep ones, offers at
// one instant, at the instant the wire gets free and from a ScheduleNow'd event of their instant, both
// must send the same frames (their chains among them), hold the same ones, count the same and trace the
// same enqueues. Exit status 0: all agree.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

struct uint4 // (the frame copies of the included headers name CUDA's vector type)
{
    unsigned x, y, z, w;
};
#define TB_QTRACE
#include "tb_tcp.cuh"

using namespace tb;

namespace
{
constexpr int FLOWS = 4, QREC = 4096;

// one host and one form of its sending end
struct Side
{
    Sim s{};
    WorldDesc wd{};
    HostRec hr{};
    HostNic nic{};
    HostCtx c{};
    std::vector<Frame> ring, msg;
    std::vector<SndRec> snd;
    std::vector<QRec> q;
    unsigned long long nq = 0;
    Frame out[OUT_FRAMES];
    int sent = 0, early = 0;
    unsigned drops = 0, marks = 0, ovf = 0, offered = 0;

    Side(bool list, int red_k, int qcap) : ring(qcap + 2), msg(MAX_TX), snd(FLOWS), q(QREC)
    {
        for (int f = 0; f < FLOWS; f++)
        {
            snd[f].src_local = 7 + f;
            snd[f].dst_local = 90 + f;
        }
        s.ring = qcap + 2;
        s.snd = snd.data();
        s.qtrace = q.data();
        s.qtrace_cnt = &nq;
        s.qtrace_n = QREC;
        s.qtrace_until = INT64_MAX;
        wd.red_k = red_k;
        wd.qcap = qcap;
        hr.local = 7;
        hr.link_free = hr.last_start = 0;
        c.s = &s;
        c.wd = &wd;
        c.dctcp = true;
        c.list = list;
        c.nic = &nic;
        c.out = out;
    }
    void open(int64_t t)
    {
        nq = 0;
        c.out_n = 0;
        c.kicked = -1;
        if (c.list)
            nic.open(s, hr, ring.data(), wd, t * SLOT_PS, msg.data());
        else
        {
            c.eg.open(ring.data(), s.ring, hr.q_head, hr.q_size, hr.link_free, hr.last_start, &hr.last, wd.red_k, wd.qcap, (t + 1) * SLOT_PS,
                      msg.data());
            c.eg.qs = &s;
            c.eg.qnode = hr.local;
            c.eg.qdev = 1;
        }
    }
    void close(int64_t t)
    {
        if (c.list)
        {
            nic_run(&nic, c.out, c.out_n, (int)SLOT_PS - 1);
            nic.close(hr);
            sent = nic.n_out, early = nic.early;
            drops += nic.drops, marks += nic.marks, ovf += nic.ovf, offered += nic.offered;
            return;
        }
        c.eg.advance((t + 1) * SLOT_PS - 1);
        hr.q_head = c.eg.head;
        hr.q_size = c.eg.size;
        hr.link_free = c.eg.busy_until;
        hr.last_start = c.eg.began;
        sent = c.eg.n_out, early = c.eg.early;
        drops += c.eg.drops, marks += c.eg.marks, ovf += c.eg.ovf, offered += c.eg.offered;
    }
};

bool same_rec(const QRec &a, const QRec &b)
{
    return a.ts == b.ts && a.node == b.node && a.dev == b.dev && a.src == b.src && a.dst == b.dst && a.sa == b.sa && a.len == b.len &&
           a.qlen == b.qlen && a.flags == b.flags;
}

bool check(const Side &a, const Side &b, int trial, int64_t t)
{
    auto differ = [&](const char *what, long long x, long long y) {
        if (x != y)
            printf("trial %d slot %lld: %s %lld, the list's %lld\n", trial, (long long)t, what, x, y);
        return x != y;
    };
    if (differ("frames sent", a.sent, b.sent) || differ("early", a.early, b.early) || differ("held", a.hr.q_size, b.hr.q_size) ||
        differ("drops", a.drops, b.drops) || differ("marks", a.marks, b.marks) || differ("overflows", a.ovf, b.ovf) ||
        differ("offered", a.offered, b.offered) || differ("wire free", a.hr.link_free, b.hr.link_free) ||
        differ("last start", a.hr.last_start, b.hr.last_start) || differ("traced", (long long)a.nq, (long long)b.nq))
        return false;
    if (memcmp(&a.hr.last, &b.hr.last, sizeof(Chain)) != 0)
        return printf("trial %d slot %lld: the wire's chain\n", trial, (long long)t), false;
    for (int i = 0; i < a.sent; i++)
        if (memcmp(&a.msg[i], &b.msg[i], sizeof(Frame)) != 0)
            return printf("trial %d slot %lld: frame %d sent\n", trial, (long long)t, i), false;
    for (int i = 0; i < a.hr.q_size; i++)
        if (memcmp(&a.ring[(a.hr.q_head + i) % a.s.ring], &b.ring[(b.hr.q_head + i) % b.s.ring], sizeof(Frame)) != 0)
            return printf("trial %d slot %lld: frame %d held\n", trial, (long long)t, i), false;
    for (unsigned long long i = 0; i < a.nq; i++)
        if (!same_rec(a.q[i], b.q[i]))
            return printf("trial %d slot %lld: enqueue %llu: %d -> %d qlen %d flags %d, the list's %d -> %d qlen %d flags %d\n", trial,
                          (long long)t, i, a.q[i].src, a.q[i].dst, a.q[i].qlen, a.q[i].flags, b.q[i].src, b.q[i].dst, b.q[i].qlen,
                          b.q[i].flags),
                   false;
    return true;
}
} // namespace

int main()
{
    std::mt19937 rng(7);
    auto below = [&](int n) { return (int)(rng() % (unsigned)n); };
    long long parts = 0, kicks = 0, traced = 0, dropped = 0, marked = 0;
    for (int trial = 0; trial < 400; trial++)
    {
        const int red_k = 1 + below(trial % 3 ? 6 : 40), qcap = red_k + below(trial % 2 ? 3 : 60);
        const int lens[4] = {CTRL_LEN, SYN_LEN, 42 + 700, 42 + (int)MSS}, most = trial % 4 == 0 ? 60 : 12;
        Side a(false, red_k, qcap), b(true, red_k, qcap);
        for (int64_t t = 0; t < 60; t++)
        {
            const int64_t S0 = t * SLOT_PS;
            a.open(t);
            b.open(t);
            int64_t now = S0 + (below(4) ? below((int)SLOT_PS) : 0);
            for (int left = below(3) ? below(most) : 0; left > 0 && now < S0 + SLOT_PS;)
            {
                a.c.eg.advance(now);
                if (below(4) == 0) // a SYN's arrival: what it schedules now runs at this instant
                {
                    a.c.kicked = b.c.kicked = now;
                    kicks++;
                }
                for (int k = 1 + below(3); k > 0 && left > 0; k--, left--)
                {
                    const int f = below(FLOWS), data = below(2), len = lens[data ? 2 + below(2) : below(2)], up = below(16);
                    chain_app_root(a.c.ech, below(50), f);
                    for (int r = below(12); r > 0; r--)
                        chain_child(a.c.ech, a.c.ech, (uint16_t)(1 + below(5000)));
                    b.c.ech = a.c.ech;
                    const uint32_t num = rng();
                    const bool back = !data && below(2);
                    if (b.c.out_n == OUT_FRAMES)
                        parts++;
                    for (Side *x : {&a, &b})
                    {
                        x->c.dctcp = data; // (a frame without ECT is dropped where another is marked)
                        to_device(x->c, f, (uint8_t)(data ? F_DATA : F_ACK), num, (uint16_t)len, back, (uint32_t)up, 90 + f, now);
                    }
                }
                // the next event: at this instant, when the wire gets free, or later
                const int how = below(4);
                now = how == 0 ? now : how == 1 && a.c.eg.busy_until > now ? a.c.eg.busy_until : now + 1 + below(150'000);
            }
            a.close(t);
            b.close(t);
            if (!check(a, b, trial, t))
                return 1;
            traced += (long long)a.nq;
        }
        dropped += a.drops;
        marked += a.marks;
    }
    printf("%lld lists played in parts, %lld kicks, %lld enqueues, %lld drops, %lld marks\n", parts, kicks, traced, dropped, marked);
    return parts && kicks && traced && dropped && marked ? 0 : 2;
}
