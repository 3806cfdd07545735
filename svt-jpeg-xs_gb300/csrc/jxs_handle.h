/*
 * What a handle's frames share on the host (plain C++, any thread).
 */
#ifndef JXS_HANDLE_H
#define JXS_HANDLE_H

#include <atomic>

/* A handle's frames in flight (submitted and not yet waited for).  For one
 * frame at a time, a result for pageable memory is best written there by the
 * kernel that makes it, when the device reaches that memory directly: no
 * staging, no copy after the host has seen the frame done (1920x1080 4:2:2
 * 8 bit decodes in 99 us instead of 157, the first frame of a new handle in
 * 127 instead of 180).  With more in flight the copy engines carry it beside
 * the next frames' kernels, which otherwise wait on the link.  A pipeline is
 * at times down to no frame; that one frame then goes the first way makes no
 * difference to it (4K frames encoded and decoded from and to pageable memory:
 * 24.4 to 24.6 Gpix/s in six runs, and 11.7 to 24.4 where only the fifth such
 * frame in a row did; one handle with two or three frames in flight the same
 * within 1 %, with pauses between them up to 4 % faster). */
struct HandleLoad {
    std::atomic<int> in_flight{0};
    int submit() { return in_flight.fetch_add(1) == 0; } /* 1: write results in place */
    void done() { in_flight.fetch_sub(1); }
};

/* What a decoder's frames told about its stream, for the frames after them:
 * set by the completion thread, read by the submitting ones. */
struct DecHints {
    /* the stream uses vertical prediction (decoded slice by slice) */
    std::atomic<int> vpred{0};
    /* Device codestreams whose slices are not at the constant-bit-rate split:
     * the precincts of this many frames to come are located first, which
     * costs a 4K frame 11 us, where finding that out costs a decode.  Each
     * time the split fails again after that, twice as many. */
    static constexpr int kFirst = 16, kMost = 4096;
    std::atomic<int> left{0}, next{kFirst};
    int locate() { /* 1: locate this frame's precincts first */
        int n = left.load();
        while (n > 0 && !left.compare_exchange_weak(n, n - 1)) {}
        return n > 0;
    }
    void elsewhere() { /* a frame not at the split was decoded after all */
        int none = 0;
        const int n = next.load();
        if (left.compare_exchange_strong(none, n)) next.store(n < kMost ? 2 * n : kMost);
    }
};

#endif
