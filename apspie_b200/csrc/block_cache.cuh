// Device memory of library-owned matrices: freed blocks are kept and handed out again.
//
// A call that returns a matrix used to spend more time in cudaMalloc and cudaFree than on the
// device (building R-MAT scale 20, 256 MB of output: 1.7 ms + 1.2 ms beside 1.65 ms of
// kernels): the driver maps and unmaps the memory each time. Blocks that are freed are kept
// instead, up to a bound in each CUDA context, and handed out again for requests of about their
// size.
//
// A block is reused and given back in the CUDA context it was made in and nowhere else: when
// something larger needs the room among the kept blocks, when an allocation of the library fails
// (all of them are made by alloc or take), when the caller asks for it (apspie_ctx_trim), and with
// the last apspie_ctx of that CUDA context. The blocks of a CUDA context that was reset went with it,
// and their addresses may be someone else's by now: they are forgotten, not freed.
//
// Freeing a matrix waits for nothing (cudaFree does, and so may not be called in a stream capture
// of the default mode); the device is waited for when a block is handed out again, if it has not
// been since the block was freed. The calls that ask for one wait for their own stream anyway.
//
// Gpu is CUDA (ctx.cu), or what a test puts in its place: Error with Gpu::kOk and
// Gpu::kOutOfMemory, the id of the current CUDA context (0: none or unknown), alloc, free, wait.
#pragma once

#include <cstddef>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace apspie {

template <class Gpu>
class BlockCache {
  public:
    using Error = typename Gpu::Error;
    explicit BlockCache(std::size_t most) : most_(most) {}

    // An apspie_ctx made in CUDA context `id` comes, or goes (here: `id` is the current one).
    void enter(unsigned long long id) {
        std::lock_guard<std::mutex> lock(mu_);
        ++of_[id].contexts;
    }
    void leave(unsigned long long id, bool here) {
        std::lock_guard<std::mutex> lock(mu_);
        auto it = of_.find(id);
        if (it == of_.end() || --it->second.contexts > 0) return;
        if (here) trim(it->second, 0);
        of_.erase(it);
    }

    // Memory of any use, without the kept blocks when there is not enough beside them.
    Error alloc(void **p, std::size_t bytes) {
        Error e = Gpu::alloc(p, bytes);
        if (e != Gpu::kOutOfMemory) return e;
        {
            std::lock_guard<std::mutex> lock(mu_);
            auto it = of_.find(Gpu::context());
            if (it == of_.end() || it->second.kept.empty()) return e;
            trim(it->second, 0);
        }
        return Gpu::alloc(p, bytes);
    }

    // Memory of a matrix, and its end.
    Error take(void **p, std::size_t bytes) {
        // whole granules, so that matrices of nearly the same size share blocks
        const std::size_t granule = bytes >= (std::size_t(1) << 20) ? std::size_t(1) << 20 : 4096;
        bytes = (bytes + granule - 1) / granule * granule;
        const unsigned long long id = Gpu::context();
        Block got{nullptr, 0, 0};
        bool idle = false;
        unsigned long long until = 0;
        {
            std::lock_guard<std::mutex> lock(mu_);
            auto it = of_.find(id);
            if (it != of_.end()) {
                List &l = it->second;
                std::size_t best = l.kept.size();
                for (std::size_t i = 0; i < l.kept.size(); ++i)
                    if (l.kept[i].bytes >= bytes && l.kept[i].bytes <= bytes + bytes / 4 &&
                        (best == l.kept.size() || l.kept[i].bytes < l.kept[best].bytes))
                        best = i;
                if (best < l.kept.size()) {
                    got = l.kept[best];
                    l.kept.erase(l.kept.begin() + static_cast<std::ptrdiff_t>(best));
                    l.bytes -= got.bytes;
                    idle = got.freed <= l.idle;
                    until = frees_;
                }
            }
        }
        if (got.p) {
            // what was in flight when the block was freed may still use it, on any stream
            const Error e = idle ? Gpu::kOk : Gpu::wait();
            if (e != Gpu::kOk) {
                Gpu::free(got.p);
                return e;
            }
            std::lock_guard<std::mutex> lock(mu_);
            auto it = of_.find(id);
            if (it != of_.end() && it->second.idle < until) it->second.idle = until;
            live_[got.p] = Live{got.bytes, id};
            *p = got.p;
            return Gpu::kOk;
        }
        const Error e = alloc(p, bytes);
        if (e == Gpu::kOk && id != 0) {
            std::lock_guard<std::mutex> lock(mu_);
            live_[*p] = Live{bytes, id};
        }
        return e;
    }
    void give(void *p) {
        if (!p) return;
        const unsigned long long id = Gpu::context();
        Live b{0, 0};
        {
            std::lock_guard<std::mutex> lock(mu_);
            auto it = live_.find(p);
            if (it != live_.end()) {
                b = it->second;
                live_.erase(it);
            } else {
                // a matrix freed twice (through a copy of its struct): the block is not the
                // caller's any more, and freeing it would leave it among the kept ones
                for (const auto &l : of_)
                    for (const Block &k : l.second.kept)
                        if (k.p == p) return;
            }
        }
        // another context's block, or one too large to keep
        if (b.id == 0 || b.id != id || b.bytes > most_ / 2) {
            Gpu::free(p);
            return;
        }
        std::lock_guard<std::mutex> lock(mu_);
        auto it = of_.find(id);
        if (it == of_.end() || it->second.contexts <= 0) {
            Gpu::free(p);
            return;
        }
        trim(it->second, most_ - b.bytes);
        it->second.kept.push_back(Block{p, b.bytes, ++frees_});
        it->second.bytes += b.bytes;
    }

    // Gives every kept block of the current CUDA context back.
    void trim() {
        std::lock_guard<std::mutex> lock(mu_);
        auto it = of_.find(Gpu::context());
        if (it != of_.end()) trim(it->second, 0);
    }

  private:
    struct Block {
        void *p;
        std::size_t bytes;
        unsigned long long freed;  // number of the free that kept it
    };
    struct Live {
        std::size_t bytes;
        unsigned long long id;  // the CUDA context it was made in
    };
    struct List {  // of one CUDA context
        std::vector<Block> kept;  // oldest first
        std::size_t bytes = 0;
        int contexts = 0;  // apspie_ctx alive
        unsigned long long idle = 0;  // the device has been waited for since this free
    };

    // Gives the oldest blocks of the current CUDA context's list back until at most `most` bytes
    // are kept (mu_ held).
    static void trim(List &l, std::size_t most) {
        std::size_t n = 0;
        for (; n < l.kept.size() && l.bytes > most; ++n) {
            Gpu::free(l.kept[n].p);
            l.bytes -= l.kept[n].bytes;
        }
        l.kept.erase(l.kept.begin(), l.kept.begin() + static_cast<std::ptrdiff_t>(n));
    }

    const std::size_t most_;
    std::mutex mu_;
    std::unordered_map<void *, Live> live_;  // handed out
    std::unordered_map<unsigned long long, List> of_;
    unsigned long long frees_ = 0;
};

}  // namespace apspie
