// A check of the device arrays that an RDMA batch keeps between its runs (twins_b200/csrc/tr_arrays.h) over a
// model of the memory, built with g++ by tests/test_rdma_arrays.py. Every run must find its zeroed arrays
// zero and its images whole, whatever the run before left in them: a run like the one before (the same
// memory, none allocated), one whose tail ring grew (that piece alone is allocated anew), one of fewer
// arrays, one that finds no memory (it fails, and what it holds is given back). Exit status 0: all hold.
#include "tr_arrays.h"

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>

namespace
{
struct Model
{
    using Stream = int;
    static std::map<void *, size_t> held;
    static int allocs;
    static size_t limit, in_use;
    static bool alloc(void **p, size_t n)
    {
        if (in_use + n > limit)
            return false;
        *p = malloc(n);
        memset(*p, 0xA5, n); // (as found: not zero)
        held[*p] = n;
        in_use += n;
        allocs++;
        return true;
    }
    static void release(void *p)
    {
        if (!p)
            return;
        auto it = held.find(p);
        if (it == held.end())
        {
            printf("released what is not held\n");
            exit(1);
        }
        in_use -= it->second;
        held.erase(it);
        free(p);
    }
    static bool inside(void *p, size_t n)
    {
        auto it = held.find(p);
        return it != held.end() && n <= it->second;
    }
    static bool zero(void *p, size_t n, Stream)
    {
        if (!inside(p, n))
            return false;
        memset(p, 0, n);
        return true;
    }
    static bool copy(void *p, const void *from, size_t n, Stream)
    {
        if (!inside(p, n))
            return false;
        memcpy(p, from, n);
        return true;
    }
};
std::map<void *, size_t> Model::held;
int Model::allocs = 0;
size_t Model::limit = SIZE_MAX, Model::in_use = 0;

// one run's arrays: an image, an empty image, a zeroed array, the tail ring, an image behind it, and
// (a traced run) one more
struct Run
{
    uint32_t *image;
    char *none;
    uint64_t *zero, *tail;
    int16_t *after, *trace = nullptr;
};

bool upload(tr::RunArrays<Model> &d, Run &r, int tail_log2, bool trace, uint32_t seed)
{
    d.begin(1);
    std::vector<uint32_t> image(1000);
    for (size_t i = 0; i < image.size(); i++)
        image[i] = seed + (uint32_t)i;
    std::vector<int16_t> after(77, (int16_t)seed);
    if (!(d.copy(&r.image, image) && d.copy(&r.none, std::vector<char>()) && d.zeroed(&r.zero, 500) && d.zeroed(&r.tail, (size_t)1 << tail_log2) &&
          d.copy(&r.after, after) && (!trace || d.zeroed(&r.trace, 300))))
        return false;
    bool ok = !memcmp(r.image, image.data(), 4000) && !memcmp(r.after, after.data(), 154) && *r.none == 0;
    for (int i = 0; i < 500; i++)
        ok &= r.zero[i] == 0;
    for (size_t i = 0; i < (size_t)1 << tail_log2; i++)
        ok &= r.tail[i] == 0;
    for (int i = 0; trace && i < 300; i++)
        ok &= r.trace[i] == 0;
    if (!ok || d.bytes != 4000 + 1 + 4000 + (8ull << tail_log2) + 154 + (trace ? 600 : 0))
    {
        printf("seed %u: contents, or %zu bytes taken\n", seed, d.bytes);
        exit(1);
    }
    // the run leaves its own values everywhere
    for (auto &m : d.mem)
        memset(m.p, 0x5A, m.bytes);
    return true;
}

void expect(bool ok, const char *what)
{
    if (!ok)
    {
        printf("%s (%d allocations, %zu pieces, %zu bytes)\n", what, Model::allocs, Model::held.size(), Model::in_use);
        exit(1);
    }
}
} // namespace

int main()
{
    {
        tr::RunArrays<Model> d;
        Run a, b;
        expect(upload(d, a, 10, false, 1) && Model::allocs == 5, "the first run");
        expect(upload(d, b, 10, false, 2) && Model::allocs == 5 && a.image == b.image && a.tail == b.tail, "a run like the one before");
        expect(upload(d, b, 11, false, 3) && Model::allocs == 6 && Model::held.size() == 5 && b.image == a.image && b.after == a.after,
               "a tail ring that grew");
        expect(upload(d, b, 11, true, 4) && Model::allocs == 7, "an array more");
        expect(upload(d, b, 11, false, 5) && Model::allocs == 7, "an array fewer");
        Model::limit = Model::in_use + 100;
        Run c;
        expect(!upload(d, c, 12, false, 6), "no memory");
        d.release();
        expect(Model::held.empty() && Model::in_use == 0 && d.bytes == 0, "a failed run gives back what it holds");
        Model::limit = SIZE_MAX;
        expect(upload(d, c, 10, false, 7) && Model::held.size() == 5, "the run after a failed one");
    }
    expect(Model::held.empty(), "the end of the batch");
    return 0;
}
