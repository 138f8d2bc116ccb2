// twins-b200: the device arrays of an RDMA run, kept from one run of a batch to the next (plain C++17; the
// memory's operations are a parameter, so that the tests check the bookkeeping on the CPU).
#pragma once
#include <cstddef>
#include <vector>

namespace tr
{

// The run's arrays that start as set-up images, the ones that start zeroed, and the tail ring. A run
// takes them in one order and of one size (but for a tail ring that grew), so the next run of the
// batch fills the same memory again: allocating and freeing some forty arrays, gigabytes in all, took
// 10 ms of a small run and up to 100 ms when the driver was slow about it.
// Mem: static alloc(void **, bytes), release(void *), zero(void *, bytes, Stream), copy(void *, const void *,
// bytes, Stream), the last two in the stream's order; false on an error.
template <class Mem>
struct RunArrays
{
    using Stream = typename Mem::Stream;
    struct Piece
    {
        void *p;
        size_t bytes;
    };
    std::vector<Piece> mem;
    size_t at = 0, bytes = 0; // the next piece; the bytes taken by this run
    Stream stream{};
    ~RunArrays() { release(); }
    void release()
    {
        for (Piece &m : mem)
            Mem::release(m.p);
        mem.clear();
        at = bytes = 0;
    }
    void begin(Stream s)
    {
        stream = s;
        at = bytes = 0;
    }
    template <class T>
    bool take(T **p, size_t n)
    {
        const size_t b = sizeof(T) * (n ? n : 1);
        if (at == mem.size())
            mem.push_back({nullptr, 0});
        Piece &m = mem[at++];
        if (m.bytes != b)
        {
            Mem::release(m.p);
            m = {nullptr, 0};
            if (!Mem::alloc(&m.p, b))
                return false;
            m.bytes = b;
        }
        *p = (T *)m.p;
        bytes += b;
        return true;
    }
    template <class T>
    bool zeroed(T **p, size_t n)
    {
        return take(p, n) && Mem::zero(*p, sizeof(T) * (n ? n : 1), stream);
    }
    template <class T>
    bool copy(T **p, const std::vector<T> &v)
    {
        if (v.empty())
            return zeroed(p, 0);
        return take(p, v.size()) && Mem::copy(*p, v.data(), sizeof(T) * v.size(), stream);
    }
};

} // namespace tr
