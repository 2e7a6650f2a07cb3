// Staging ring of a context: task arrays go to pinned host memory and from there to the
// same offset in device memory, and launches read them there.
//
// Outside a Batch an array is uploaded when it is staged, on the stream of its launch.
// Inside one, launches are held; flush() uploads all of their arrays in one copy and
// makes them.  When an array does not fit behind the others, the ring wraps: what is
// held is launched, the host waits for everything, and the ring starts again at its
// beginning.  So every array has to be launched, or held, before the ring wraps: a
// later array of the same Batch could take its place, and reach the device before the
// launch that reads it.  A launch with several arrays therefore makes room for all of
// them (stage_room) before it stages the first; one that does not is refused at the wrap.
//
// C is the context: it has a Ring `ring`, a current stream `cur`, and
//   int ring_upload(size_t off, size_t n)   host to device on the current stream
//   int ring_wait_current()                 the host waits for the current stream
//   int ring_wait_all()                     the host waits for all streams
#pragma once
#include <cstddef>
#include <cstring>
#include <functional>
#include <vector>

namespace tlr {

struct Ring {
    char *h = nullptr, *d = nullptr;
    size_t bytes = 0, off = 0;
    bool batching = false;                    // launches wait for one upload of their arrays
    bool split = false;                       // the ring wrapped inside the Batch: part of it is launched
    bool unlaunched = false;                  // an array is staged whose launch is not held yet
    size_t held_from = 0;                     // staged bytes from here on are not uploaded yet
    std::vector<std::function<int()>> held;   // the launches, in order
};

// Ring bytes of an array of `raw` bytes.
inline size_t ring_bytes(size_t raw) { return (raw + 1 + 255) / 256 * 256; }

// Uploads what is staged on the current stream and makes the held launches.  Other
// streams join the current one by an event held among them, so after the upload; once
// a part of the Batch with such an event is launched, the host waits for the upload.
template <class C>
int issue_held(C *c) {
    Ring &r = c->ring;
    int rc = r.off > r.held_from ? c->ring_upload(r.held_from, r.off - r.held_from) : 0;
    if (!rc && r.split) rc = c->ring_wait_current();
    if (rc) return rc;
    r.held_from = r.off;
    std::vector<std::function<int()>> q;
    q.swap(r.held);
    const auto st = c->cur;
    for (size_t i = 0; i < q.size() && !rc; ++i) rc = q[i]();
    c->cur = st;
    return rc;
}

// A launch (or an event call) on the current stream: made now, or held inside a Batch.
template <class C, class F>
int issue(C *c, F f) {
    Ring &r = c->ring;
    r.unlaunched = false;
    if (!r.batching) return f();
    const auto st = c->cur;
    r.held.push_back([c, st, f]() {
        c->cur = st;
        return f();
    });
    return 0;
}

// While a Batch lives, the helpers stage their task arrays and hold their launches;
// flush() uploads all arrays in one copy on the current stream, then launches.  A copy
// per launch sits in the stream before it: 3 us of copy and 6 us of gaps to a launch of
// 20 to 200 us in the chains of a late panel.  One copy a batch: 2D requests of 27,000
// and 97,200 unknowns 77.3, 314 ms -> 73.3, 299; 60 x 60 tiles 390 -> 377.
template <class C>
struct BatchOf {
    C *c;
    bool mine;
    explicit BatchOf(C *ctx) : c(ctx), mine(!ctx->ring.batching) {
        if (!mine) return;
        c->ring.batching = true;
        c->ring.split = c->ring.unlaunched = false;
        c->ring.held_from = c->ring.off;
    }
    int flush() { return mine ? issue_held(c) : 0; }
    ~BatchOf() {
        if (!mine) return;
        c->ring.held.clear();       // left only by an error
        c->ring.batching = false;
    }
    BatchOf(const BatchOf &) = delete;
    BatchOf &operator=(const BatchOf &) = delete;
};

// Room for `n` ring bytes behind what is staged: wraps if there is none.
template <class C>
int stage_room(C *c, size_t n) {
    Ring &r = c->ring;
    if (n > r.bytes) return -1;
    if (r.off + n <= r.bytes) return 0;
    if (r.batching) {
        if (r.unlaunched) return -1;
        r.split = true;
        if (int rc = issue_held(c)) return rc;
    }
    if (int rc = c->ring_wait_all()) return rc;
    r.off = r.held_from = 0;
    return 0;
}

// Device address of an array for a launch on the current stream; null on failure.
template <class C, class T>
T *stage(C *c, const T *src, size_t n) {
    Ring &r = c->ring;
    const size_t raw = n * sizeof(T), at_end = ring_bytes(raw);
    if (stage_room(c, at_end)) return nullptr;
    std::memcpy(r.h + r.off, src, raw);
    if (!r.batching && c->ring_upload(r.off, raw)) return nullptr;
    T *d = (T *)(r.d + r.off);
    r.off += at_end;
    r.unlaunched = true;
    return d;
}

// The two arrays of one launch.
template <class C, class T, class U>
bool stage_both(C *c, const std::vector<T> &a, const std::vector<U> &b, T **da, U **db) {
    if (stage_room(c, ring_bytes(a.size() * sizeof(T)) + ring_bytes(b.size() * sizeof(U)))) return false;
    *da = stage(c, a.data(), a.size());
    *db = stage(c, b.data(), b.size());
    return *da && *db;
}

}  // namespace tlr
