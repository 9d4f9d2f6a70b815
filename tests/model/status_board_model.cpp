// Drives csrc/status_board.h with a model of streams and events: a stream is a queue of copies that land only when it is
// run, an event the place in a stream's queue behind which it was recorded last.  Exits non-zero at the first failure.
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <stdexcept>
#include <string>
#include <thread>

#include "status_board.h"

#define REQUIRE(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); exit(1); } } while (0)

struct Stream {
    std::deque<std::function<void()>> queue;
    size_t enqueued = 0, ran = 0;
    void run(size_t upto) {
        while (ran < upto) { queue.front()(); queue.pop_front(); ++ran; }
    }
};
struct EventState { Stream* stream = nullptr; size_t at = 0; };
static std::deque<EventState> g_events;
static int g_waits = 0, g_asked = 0;
struct Gpu {
    typedef EventState* Event;
    typedef ::Stream* Stream;
    static int32_t* alloc_words(int slots) { return static_cast<int32_t*>(calloc(slots, 16)); }
    static Event make_event(int) { g_events.emplace_back(); return &g_events.back(); }
    static void copy(int32_t* dst, const void* src, Stream st) {
        st->queue.push_back([=] { memcpy(dst, src, 16); });
        ++st->enqueued;
    }
    static void record(Event e, Stream st) { e->stream = st; e->at = st->enqueued; }
    static bool done(Event e) { ++g_asked; return !e->stream || e->stream->ran >= e->at; }
    static void wait(Event e) { ++g_waits; if (e->stream) e->stream->run(e->at); }
};
typedef hdla_host::StatusBoard<Gpu> Board;

struct Reported { int32_t w[4]; };
static void fail(const int32_t* w) { Reported r; memcpy(r.w, w, 16); throw r; }
static int32_t reported(Board& b, bool wait, int word) {          // 0: nothing
    try { b.check(wait); } catch (const Reported& r) { return r.w[word]; }
    return 0;
}
struct Words { int32_t w[4]; };
static Words words(int code, int overflow, float decay) {
    Words x{{code, overflow, 0, 0}};
    memcpy(&x.w[2], &decay, 4);
    return x;
}

// one stream lags while another makes more calls than there are published words: nobody's words land in another's slot
static void lagging_stream(int other_calls, bool take_words) {
    Board board(0, fail);
    Stream a, b;
    const Words bad = words(7, 0, 100.f);
    board.publish(board.post(&bad, &a));
    for (int i = 0; i < other_calls; ++i) {
        const Words mine = words(0, i % 2, 80.f + i);
        if (take_words) {
            int32_t got[4];
            board.take(board.post(&mine, &b), got);
            REQUIRE(memcmp(got, mine.w, 16) == 0);
            REQUIRE(reported(board, false, 0) == 0);              // (a has not run: its report is still to come)
        } else {
            const Words clean = words(0, 0, 1.f);
            board.publish(board.post(&clean, &b));
            b.run(b.enqueued);
            REQUIRE(reported(board, false, 0) == 0);
        }
    }
    REQUIRE(a.ran == 0);
    REQUIRE(reported(board, true, 0) == 7);
    REQUIRE(reported(board, true, 0) == 0);
}

// words that a forward waits for are not consumed by whoever looks at the device meanwhile
static void words_have_one_owner() {
    Board board(0, fail);
    Stream a;
    const Words over = words(0, 1, 200.f);
    Board::Slot* s = board.post(&over, &a);
    a.run(a.enqueued);
    REQUIRE(reported(board, false, 1) == 0 && reported(board, true, 1) == 0);
    const Words clean = words(0, 0, 1.f);
    for (int i = 0; i < 200; ++i) { board.publish(board.post(&clean, &a)); a.run(a.enqueued); board.check(false); }
    int32_t got[4];
    board.take(s, got);
    REQUIRE(got[1] == 1);
    REQUIRE(board.decay() == 200.0);
}

// published words are bounded: a call beyond them waits for the oldest, and what that reports is not lost
static void published_words_are_bounded() {
    Board board(0, fail);
    Stream a;
    const Words clean = words(0, 0, 1.f), bad = words(5, 0, 1.f);
    board.publish(board.post(&bad, &a));
    for (int i = 1; i < 64; ++i) board.publish(board.post(&clean, &a));
    REQUIRE(g_waits == 0 && a.ran == 0);
    const int asked = g_asked;
    board.check(false);
    REQUIRE(g_asked == asked + 1);               // one question per stream that lags, not one per call
    int32_t code = 0;
    try { board.publish(board.post(&clean, &a)); } catch (const Reported& r) { code = r.w[0]; }
    REQUIRE(code == 5 && g_waits == 1 && a.ran == 1);
    for (int i = 0; i < 1000; ++i) board.publish(board.post(&clean, &a));
    REQUIRE(reported(board, true, 0) == 0);
    REQUIRE(g_events.size() == 64);
}

// every report of several is seen, one per look; NaN in the decay word says nothing
static void reports_come_one_by_one() {
    Board board(0, fail);
    Stream a;
    const Words x[4] = {words(0, 0, NAN), words(3, 0, NAN), words(0, 1, 160.f), words(4, 0, 2.f)};
    for (const Words& w : x) board.publish(board.post(&w, &a));
    REQUIRE(reported(board, false, 0) == 0 && board.decay() != board.decay());
    REQUIRE(reported(board, true, 0) == 3);
    REQUIRE(reported(board, true, 1) == 1);
    REQUIRE(reported(board, true, 0) == 4);
    REQUIRE(reported(board, true, 0) == 0 && board.decay() == 160.0);
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "lagging") for (int n : {1, 62, 63, 64, 65, 200}) { lagging_stream(n, true); lagging_stream(n, false); }
    else if (what == "owner") words_have_one_owner();
    else if (what == "bounded") published_words_are_bounded();
    else if (what == "reports") reports_come_one_by_one();
    else return 2;
    return 0;
}
