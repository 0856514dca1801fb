// fe_sort_scratch.h — the device buffers that fe_sort_pairs keeps per device.
// Host code without CUDA types, so that a host program can run it with an
// allocator of its own.
#pragma once

#include <cstddef>
#include <cstdint>

namespace fe {

struct SortBuffers {
    uint32_t* tk = nullptr;      // cap words each: the other half of the ping-pong
    uint32_t* tv = nullptr;
    uint32_t cap = 0;
    uint32_t* words = nullptr;   // nwords: histograms and status words
    size_t nwords = 0;
    uint32_t* flags = nullptr;   // kSortFlagWords: the error word, an allocation of its
                                 // own, which sorts without other scratch use too
};
constexpr size_t kSortFlagWords = 8;

inline bool sort_buffers_hold(const SortBuffers& S, uint32_t n, size_t words) {
    return S.cap >= n && S.nwords >= words;
}

// Frees the ping-pong and scratch buffers and allocates larger ones.  The
// capacities are 0 until all of them are there: after an allocation that failed,
// the next sort that needs them grows them again, whatever its size.
// alloc(void**, bytes) returns 0 or an error, which is returned; release(void*)
// takes NULL too.
template <class Alloc, class Release>
auto sort_buffers_grow(SortBuffers& S, uint32_t n, size_t words, Alloc&& alloc,
                       Release&& release) -> decltype(alloc((void**)nullptr, (size_t)0)) {
    const uint32_t cap = n > S.cap ? n : S.cap;
    const size_t nwords = words > S.nwords ? words : S.nwords;
    release(S.tk);
    release(S.tv);
    release(S.words);
    S.tk = S.tv = S.words = nullptr;
    S.cap = 0;
    S.nwords = 0;
    auto e = alloc((void**)&S.tk, (size_t)cap * 4);
    if (!e) e = alloc((void**)&S.tv, (size_t)cap * 4);
    if (!e) e = alloc((void**)&S.words, nwords * 4);
    if (e) return e;
    S.cap = cap;
    S.nwords = nwords;
    return e;
}

}  // namespace fe
