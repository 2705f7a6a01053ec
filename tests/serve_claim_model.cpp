// Many serving decoders on one set of claim words, one access at a time in the
// order a scheduler picks: it likes to leave decoders between a failed claim and
// taking it back, but lets every decoder go on after a bounded wait.
//   serve_claim_model progress   16 items while failed claims are pending
//   serve_claim_model stop       the same, with the stop word set
// Prints "<items taken> <items published> <accesses granted>". Modes with a dash
// in their name run one decoder on a script (see scripted()).
#include <condition_variable>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "serve_claim.hpp"

namespace {

constexpr int DECODERS = 64, PENDING = 20, WAIT = 8 * DECODERS, LIMIT = 8000;

struct Model {
    std::mutex mu;
    std::condition_variable cv;        // the scheduler's
    int head = 0, tail = 0, claims = 0;
    bool stop = false, over = false;
    int turn = -1;                     // the decoder that may make one access
    struct Decoder {
        std::condition_variable cv;
        bool waiting = false, unclaims = false, done = false;
        int since = 0, got = -1;
    };
    std::vector<Decoder> d = std::vector<Decoder>(DECODERS);

    // blocks until the scheduler grants this decoder one access
    template <class F>
    auto access(int i, bool unclaims, const F& f) {
        std::unique_lock<std::mutex> lk(mu);
        d[i].waiting = true;
        d[i].unclaims = unclaims;
        cv.notify_one();
        d[i].cv.wait(lk, [&] { return turn == i || over; });
        d[i].waiting = false;
        if (turn == i) turn = -1;
        return f();
    }
};

struct Words {
    Model& m;
    int i;
    int tail() { return m.access(i, false, [&] { return m.tail; }); }
    int claims() { return m.access(i, false, [&] { return m.claims; }); }
    int head() { return m.access(i, false, [&] { return m.head; }); }
    int claim() { return m.access(i, false, [&] { return m.claims++; }); }
    void unclaim() { m.access(i, true, [&] { m.claims--; }); }
    int take() { return m.access(i, false, [&] { return m.head++; }); }
    bool stopped() { return m.access(i, false, [&] { return m.stop || m.over; }); }
    int deep_head() { return m.access(i, false, [] { return 0; }); }
    void pause(unsigned) {}
};

// One decoder whose surroundings follow a script over its empty polls.
struct Script {
    int polls = 0, n_tail = 0, n_head = 0, n_deep_tail = 0, n_deep_head = 0, n_alive = 1;
    int others_until = 0, item_at = -1;   // the others take an item every 100 polls until here
    bool deep = false;                    // this is an overflow decoder (the others are main ones)
    int tail() { return n_tail; }
    int claims() { return n_head; }
    int head() { return n_head; }
    int claim() { return n_head; }
    void unclaim() {}
    int take() { return n_head++; }
    bool stopped() { return false; }
    int deep_tail() { return n_deep_tail; }
    int deep_head() { return n_deep_head; }
    int deep_take(int) { return n_deep_head++; }
    int alive() { return n_alive; }
    void pause(unsigned) {
        polls++;
        if (polls <= others_until && polls % 100 == 0) {
            if (deep) n_tail = ++n_head;
            else n_deep_tail = ++n_deep_head;
        }
        if (polls == item_at) (deep ? n_deep_tail : n_tail)++;
    }
};

// "<took an item> <empty polls>"
int scripted(const char* mode) {
    Script w;
    int got = -1;
    if (!std::strcmp(mode, "main-waits")) {          // overflow decoders at work, an item after a long while
        w.others_until = w.item_at = 20000;
        got = plpb::serve_claim(w, 2000);
    } else if (!std::strcmp(mode, "main-idle")) {    // nobody takes anything any more
        w.others_until = 5000;
        got = plpb::serve_claim(w, 2000);
    } else if (!std::strcmp(mode, "deep-waits")) {   // main decoders at work, the first overflow after a long while
        w.deep = true;
        w.others_until = w.item_at = 20000;
        got = plpb::serve_claim_deep(w, 2000);
    } else if (!std::strcmp(mode, "deep-left")) {    // the main decoders have left, no stop
        w.deep = true;
        w.n_alive = 0;
        got = plpb::serve_claim_deep(w, 2000);
    } else {
        return 2;
    }
    std::printf("%d %d\n", got >= 0, w.polls);
    return 0;
}

}  // namespace

int main(int argc, char** argv) {
    if (argc > 1 && std::strchr(argv[1], '-')) return scripted(argv[1]);
    const bool stop = argc > 1 && !std::strcmp(argv[1], "stop");
    Model m;
    // a decoder that ends (with an item, or without) takes part no further, as
    // one that decodes for long does
    std::vector<std::thread> ts;
    for (int i = 0; i < DECODERS; i++)
        ts.emplace_back([&m, i] {
            Words w{m, i};
            const int got = plpb::serve_claim(w, LIMIT);
            std::lock_guard<std::mutex> lk(m.mu);
            m.d[i].got = got;
            m.d[i].done = true;
            m.cv.notify_one();
        });
    // four items, whose claims race with the other decoders' until some of those are pending
    m.tail = 4;
    int published = 4, granted = 0, next = 0, taken = 0;
    for (;;) {
        std::unique_lock<std::mutex> lk(m.mu);
        m.cv.wait(lk, [&] {
            if (m.turn >= 0) return false;
            for (const auto& x : m.d)
                if (!x.waiting && !x.done) return false;
            return true;
        });
        int pending = 0, live = 0, oldest = -1;
        taken = 0;
        for (int i = 0; i < DECODERS; i++) {
            auto& x = m.d[i];
            taken += x.done && x.got >= 0;
            if (x.done) continue;
            live++;
            if (x.unclaims) {
                pending++;
                if (oldest < 0 || x.since < m.d[oldest].since) oldest = i;
            }
        }
        if (!live || granted == LIMIT || (taken == 20 && !stop)) {
            m.over = true;
            for (auto& x : m.d) x.cv.notify_one();
            break;
        }
        // later items, once failed claims are pending (or nobody is in between)
        if (published == 4 && (pending >= PENDING || granted > 4 * WAIT)) {
            published = m.tail = 20;
            m.stop = stop;
        }
        int pick = -1;
        if (pending > PENDING || (oldest >= 0 && granted - m.d[oldest].since > WAIT)) pick = oldest;
        for (int k = 0; pick < 0 && k < DECODERS; k++, next = (next + 1) % DECODERS)
            if (!m.d[next].done && !m.d[next].unclaims) pick = next;
        if (pick < 0) pick = oldest;
        m.d[pick].unclaims = false;
        m.d[pick].since = granted++;
        m.turn = pick;
        m.d[pick].cv.notify_one();
    }
    for (auto& t : ts) t.join();
    std::printf("%d %d %d\n", taken, published, granted);
    return 0;
}
