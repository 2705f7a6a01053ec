// serve_claim.hpp -- how a serving decoder takes the next published work item.
// Written over the words it reads and changes (Words), so that the same code
// runs in the decoders (decoder.cu: words in device memory) and in a test's
// model of many decoders under a chosen order of their accesses.
#pragma once

#ifdef __CUDACC__
#define PLP_HD __host__ __device__ __forceinline__
#else
#define PLP_HD inline
#endif

namespace plpb {

// Notices whether any decoder of the launch has taken an item: a launch in use
// keeps the decoders that find none, so that a burst after hours of small
// requests, or a request that outgrows its tile, meets all of them.
struct ClaimWatch {
    int seen = -1;   // the first look only notes the counts
    template <class Words>
    PLP_HD bool moved(Words& w) {
        const int now = w.head() + w.deep_head(), was = seen;
        seen = now;
        return now != was;
    }
};
constexpr int WATCH_POLLS = 256;   // empty polls between looks (about 1 ms)

// The next item's number, or -1 once the host has asked the launch to stop and
// every published item is taken, or after `polls` empty polls (rounded up to
// looks) in which no decoder took an item, overflow decoders included.
//
// Two counters, so that a claim is two additions, which the L2 serves one after
// the other (a compare-and-swap of one counter, which one decoder wins per round
// trip, held a launch to 3 restarts per us whatever their size). A decoder first
// counts itself among the claims; if the count before it is below the tail, an
// item is left for it and the head's next value is that item, else it takes its
// count back. The count is the claims that succeeded and those about to be taken
// back, so no more succeed than are published.
//
// A claim is tried only where the count was read below the tail. Claims about
// to be taken back can then keep nobody from a free item: after the count was
// read below the tail, the next addition is one that succeeds, so there is no
// round of failures without a claim between. (Tried whenever the head is below
// the tail, failures alone hold the count up, and idle decoders, of which there
// are some 2000, keep all of each other from a request of a few restarts.)
//
// The stop word is read before the head and the tail that it is obeyed by, so a
// decoder leaves no item that was published before the stop.
template <class Words>
PLP_HD int serve_claim(Words& w, int polls) {
    unsigned ns = 32;
    ClaimWatch watch;
    for (int k = 0; k < polls; k++) {
        const int t = w.tail();
        if (w.claims() < t) {
            if (w.claim() < t) {
                const int i = w.take();
                if (i >= t) (void)w.tail();   // published since: its words were written before
                return i;
            }
            w.unclaim();
        }
        if (w.stopped() && w.head() >= w.tail()) return -1;
        w.pause(ns);
        if (ns < 4096) ns <<= 1;
        if (k % WATCH_POLLS == WATCH_POLLS - 1 && watch.moved(w)) k = -1;
    }
    return -1;
}

// An overflow decoder's next item (a ticket of the overflow ring), or -1 once
// every main decoder has left and no item is left, or after `polls` empty polls
// in which no decoder took an item.
//
// It waits for the main decoders only, not for the stop word: those leave by
// themselves after their idle bound, and a launch that overflow decoders alone
// keep running takes no new request. (A request whose restarts overflowed for
// longer than that bound left the next ones waiting for the overflow decoders'
// bound, a minute.) Main decoders push before they leave, so once none is left
// the count of items seen after that is final.
template <class Words>
PLP_HD int serve_claim_deep(Words& w, int polls) {
    unsigned ns = 64;
    ClaimWatch watch;
    for (int k = 0; k < polls; k++) {
        const int t = w.deep_tail();
        int h = w.deep_head();
        while (h < t) {
            const int prev = w.deep_take(h);
            if (prev == h) return h;
            h = prev;
        }
        if (w.alive() == 0 && w.deep_tail() <= h) return -1;
        w.pause(ns);
        if (ns < 8192) ns <<= 1;
        if (k % WATCH_POLLS == WATCH_POLLS - 1 && watch.moved(w)) k = -1;
    }
    return -1;
}

}  // namespace plpb
