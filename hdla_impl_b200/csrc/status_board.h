// Status words of the calls in flight on one device (host side; see include/hdla.h for the words).
//
// After a call its words are copied to pinned host memory on the call's stream, without waiting.  A slot -- the pinned
// words and the event behind the copy -- belongs to one call from the moment the copy is enqueued until its event has
// been seen complete; only then is it used again, so that no two copies in flight share one, however far streams drift
// apart.  The call then either takes its words itself (take: a forward that must know whether to run again; nobody else
// can consume them) or publishes the slot, and check() of whoever uses the device next looks at it.
//
// `Gpu` supplies events and copies (a model of them stands in for CUDA in the tests on the CPU):
//   Event, Stream;  int32_t* alloc_words(int slots);  Event make_event(int dev);
//   void copy(int32_t* dst, const void* src, Stream);  void record(Event, Stream);  bool done(Event);  void wait(Event)
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>
#include <deque>
#include <mutex>
#include <vector>

namespace hdla_host {

template <class Gpu>
class StatusBoard {
public:
    struct Slot { int32_t* words; typename Gpu::Event event; typename Gpu::Stream stream; };
    typedef void (*Fail)(const int32_t* words);              // throws

    StatusBoard(int dev, Fail fail) : dev_(dev), fail_(fail) {}

    // Enqueue the copy of the words at `ws` (device memory) in a slot of the call's own.
    Slot* post(const void* ws, typename Gpu::Stream stream) {
        Slot* s = acquire();
        try {
            Gpu::copy(s->words, ws, stream);
            Gpu::record(s->event, stream);
            s->stream = stream;
        } catch (...) {
            release(s);
            throw;
        }
        return s;
    }
    void publish(Slot* s) {
        std::lock_guard<std::mutex> lk(mu_);
        posted_.push_back(s);
    }
    // Wait for the words of a slot that was not published.
    void take(Slot* s, int32_t* w) {
        try {
            Gpu::wait(s->event);
        } catch (...) {
            release(s);
            throw;
        }
        memcpy(w, s->words, 16);
        std::lock_guard<std::mutex> lk(mu_);
        note(w);
        free_.push_back(s);
    }
    // Look at the published words that have landed (with `wait`, at all of them); fails at the first that report a problem.
    void check(bool wait) {
        std::unique_lock<std::mutex> lk(mu_);
        if (wait) {
            const std::deque<Slot*> todo = posted_;
            lk.unlock();
            for (Slot* s : todo) Gpu::wait(s->event);        // (one that is consumed and reused meanwhile: a longer wait)
            lk.lock();
        }
        std::vector<typename Gpu::Stream> busy;              // what follows an unfinished copy on its stream is not asked about
        for (size_t i = 0; i < posted_.size();) {
            Slot* s = posted_[i];
            bool skip = false;
            for (const auto& b : busy) skip = skip || b == s->stream;
            if (!skip && !Gpu::done(s->event)) { busy.push_back(s->stream); skip = true; }
            if (skip) { ++i; continue; }
            int32_t w[4];
            memcpy(w, s->words, 16);
            posted_.erase(posted_.begin() + static_cast<std::ptrdiff_t>(i));
            free_.push_back(s);
            note(w);
            if (w[0] || w[1]) {
                lk.unlock();
                fail_(w);
                lk.lock();
            }
        }
    }
    // Largest chunk decay seen (NAN: nothing seen yet).
    double decay() { std::lock_guard<std::mutex> lk(mu_); return decay_; }
    void set_decay(double x) { std::lock_guard<std::mutex> lk(mu_); decay_ = x; }

private:
    static constexpr size_t kPosted = 64;        // published words kept at most; a further call waits for the oldest
    static constexpr int kBlock = 64;            // slots allocated at a time (beyond the first: callers that wait at once)

    Slot* acquire() {
        std::unique_lock<std::mutex> lk(mu_);
        while (posted_.size() >= kPosted) {
            typename Gpu::Event oldest = posted_.front()->event;
            lk.unlock();
            Gpu::wait(oldest);
            check(false);
            lk.lock();
        }
        if (free_.empty()) {
            int32_t* words = Gpu::alloc_words(kBlock);
            for (int i = 0; i < kBlock; ++i) {
                all_.push_back(Slot{words + 4 * i, Gpu::make_event(dev_), {}});
                free_.push_back(&all_.back());
            }
        }
        Slot* s = free_.back();
        free_.pop_back();
        return s;
    }
    void release(Slot* s) {
        std::lock_guard<std::mutex> lk(mu_);
        free_.push_back(s);
    }
    void note(const int32_t* w) {                // (with mu_ held)
        float seen;
        memcpy(&seen, &w[2], 4);
        if (seen == seen && !(decay_ > seen)) decay_ = seen;
    }

    const int dev_;
    const Fail fail_;
    std::mutex mu_;
    std::deque<Slot> all_;                       // (a deque: slots keep their addresses)
    std::vector<Slot*> free_;
    std::deque<Slot*> posted_;
    double decay_ = NAN;
};

}  // namespace hdla_host
