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

#endif
