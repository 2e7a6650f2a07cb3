// Device memory of the descriptors, kept for the next ones.
//
// A program that evaluates likelihoods makes and destroys a descriptor for each.  Mapping
// and unmapping its memory every time costs 0.6 ms for the smallest and about 0.4 and 0.8
// ms a GB, more on a busy host.  A region that is given back is therefore kept, up
// to `limit` bytes and MAX_REGIONS regions of a device, the oldest going first, and
// handed out again for a size that wastes at most a fifth of it.  Whatever is kept goes
// back to the driver when an allocation fails and with the device's last context.
//
// Regions come from cudaMalloc.  A stream-ordered pool took 56 ms and more to grow by 15 GB
// where cudaMalloc takes 3 to 4, and 21 to 363 ms when its free pieces had to be mapped
// side by side for another size: preparing a factorization of 162,000 unknowns 437 ms,
// 261 to 335 with regions; four serving threads 1.5 to 2.1 requests a second, 3.3 with
// regions (2.9 one after the other).
//
// Api: static int alloc(void **, size_t) (0, or the error), static bool is_oom(int),
// static void release(void *), for the current device.  Thread-safe.
#pragma once
#include <cstddef>
#include <list>
#include <map>
#include <mutex>

namespace tlr {

template <class Api>
class Regions {
public:
    static constexpr size_t MAX_REGIONS = 256;

    // A context uses the device from enter() to leave(); the last leave() frees what is kept.
    void enter(size_t limit) {
        std::lock_guard<std::mutex> lk(mu);
        limit_ = limit;
        ++users_;
    }
    void leave() {
        {
            std::lock_guard<std::mutex> lk(mu);
            if (--users_ > 0) return;
        }
        trim();
    }

    // A region of at least `bytes` bytes, of any content; 0, or the error of the allocation.
    int take(void **p, size_t bytes) {
        const size_t n = bytes <= SMALL ? (bytes + 511) / 512 * 512 : (bytes + GRAIN - 1) / GRAIN * GRAIN;
        {
            std::lock_guard<std::mutex> lk(mu);
            auto best = kept_.end();
            for (auto it = kept_.begin(); it != kept_.end(); ++it)
                if (it->bytes >= n && it->bytes <= n + n / 4 && (best == kept_.end() || it->bytes < best->bytes)) best = it;
            if (best != kept_.end()) {
                *p = best->p;
                held_ -= best->bytes;
                kept_.erase(best);
                return 0;
            }
        }
        int e = alloc(p, n);
        if (e) {
            *p = nullptr;
            return e;
        }
        std::lock_guard<std::mutex> lk(mu);
        size_[*p] = n;
        return 0;
    }

    // Nothing on the device uses the region any more.  keep: it may be handed out again.
    void give(void *p, bool keep) {
        std::list<Region> out;
        {
            std::lock_guard<std::mutex> lk(mu);
            auto f = size_.find(p);
            if (f == size_.end()) return;
            const size_t n = f->second;
            if (!keep || users_ <= 0 || n > limit_) {
                out.push_back({p, n});
            } else {
                kept_.push_back({p, n});
                held_ += n;
                while (held_ > limit_ || kept_.size() > MAX_REGIONS) {
                    held_ -= kept_.front().bytes;
                    out.splice(out.end(), kept_, kept_.begin());
                }
            }
            for (auto &r : out) size_.erase(r.p);
        }
        for (auto &r : out) Api::release(r.p);
    }

    // Everything that is kept goes back to the driver; true if there was something.
    bool trim() {
        std::list<Region> out;
        {
            std::lock_guard<std::mutex> lk(mu);
            out.swap(kept_);
            held_ = 0;
            for (auto &r : out) size_.erase(r.p);
        }
        for (auto &r : out) Api::release(r.p);
        return !out.empty();
    }

    // An allocation of another kind on this device, tried again after trim().
    int alloc(void **p, size_t bytes) {
        int e = Api::alloc(p, bytes);
        if (e && Api::is_oom(e) && trim()) e = Api::alloc(p, bytes);
        return e;
    }

    size_t held() {
        std::lock_guard<std::mutex> lk(mu);
        return held_;
    }

private:
    static constexpr size_t SMALL = (size_t)1 << 20, GRAIN = (size_t)2 << 20;
    struct Region {
        void *p;
        size_t bytes;
    };
    std::mutex mu;
    std::list<Region> kept_;                  // oldest first
    std::map<void *, size_t> size_;           // of every region, handed out or kept
    size_t held_ = 0, limit_ = 0;
    int users_ = 0;
};

}  // namespace tlr
