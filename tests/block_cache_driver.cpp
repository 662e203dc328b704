// The cache of matrix memory on a stand-in for CUDA (no GPU): a table of who holds which address
// in which CUDA context. Freeing or handing out what is not the cache's is an error.
#include <cstdio>
#include <cstring>
#include <map>

#include "../apspie_b200/csrc/block_cache.cuh"

namespace {
constexpr std::size_t MB = std::size_t(1) << 20;
int g_bad = 0;
void check(bool ok, const char *what) {
    if (ok) return;
    ++g_bad;
    std::printf("%s\n", what);
}

// Context k is on device k / 10. Every device has addresses of its own; the lowest free one is
// handed out first, whichever of the device's contexts asks.
struct Fake {
    using Error = int;
    static constexpr Error kOk = 0, kOutOfMemory = 2;
    static unsigned long long now;                       // the current CUDA context
    static std::map<unsigned long long, std::map<std::size_t, std::size_t>> held;  // context -> address -> bytes
    static std::size_t room;                             // bytes a context can hold
    static int waits, wait_error;

    static unsigned long long context() { return now; }
    static Error alloc(void **p, std::size_t bytes) {
        std::size_t at = (now / 10 + 1) << 44, used = 0;
        for (auto &b : held[now]) {
            used += b.second;
            if (at + bytes <= b.first) break;
            at = b.first + b.second;
        }
        used = 0;
        for (auto &b : held[now]) used += b.second;
        if (used + bytes > room) return kOutOfMemory;
        held[now][at] = bytes;
        *p = reinterpret_cast<void *>(at);
        return kOk;
    }
    static void free(void *p) {
        std::size_t n = 0;
        for (auto &c : held) n += c.second.erase(reinterpret_cast<std::size_t>(p));
        check(n == 1, "freed what nobody holds");
    }
    static Error wait() { return ++waits, wait_error; }
};
unsigned long long Fake::now = 1;
std::map<unsigned long long, std::map<std::size_t, std::size_t>> Fake::held;
std::size_t Fake::room = std::size_t(64) << 30;
int Fake::waits = 0, Fake::wait_error = 0;

std::size_t held_by(unsigned long long id) {
    std::size_t n = 0;
    for (auto &b : Fake::held[id]) n += b.second;
    return n;
}
using Cache = apspie::BlockCache<Fake>;

// A block comes back for a request of about its size, and the kept blocks are bounded.
void reuse() {
    Cache c(64 * MB);
    c.enter(1);
    void *a, *b;
    c.take(&a, 10 * MB);
    c.give(a);
    c.take(&b, 9 * MB);
    check(a == b, "a block of about the size is reused");
    c.give(b);
    c.take(&a, 5 * MB);
    check(a != b, "a block of twice the size is not");
    void *p[20];
    for (auto &x : p) c.take(&x, 16 * MB);
    for (auto &x : p) c.give(x);
    check(held_by(1) <= 64 * MB + 5 * MB, "the kept blocks are bounded");
    c.give(a);
    c.leave(1, true);
    check(held_by(1) == 0, "the last context gives everything back");
}

// The blocks of a context that was reset are forgotten: their addresses belong to others.
void reset() {
    Cache c(64 * MB);
    c.enter(1);
    void *a, *other = nullptr, *b;
    c.take(&a, 20 * MB);
    c.give(a);
    Fake::held[1].clear();  // the device is reset: context 1 and its memory are gone
    Fake::now = 2;
    Fake::alloc(&other, 20 * MB);  // another user of the device
    check(other == a, "the stand-in hands the address out again");
    c.enter(2);
    for (int k = 0; k < 6; ++k) {  // more than fits among the kept blocks
        void *p[4];
        for (auto &x : p) c.take(&x, (16 + k) * MB), check(x != other, "a foreign block is handed out");
        for (auto &x : p) c.give(x);
    }
    check(c.alloc(&b, Fake::room - 30 * MB) == Fake::kOk, "kept blocks make room");
    Fake::free(b);
    c.leave(1, false);
    c.leave(2, true);
    check(held_by(2) == 20 * MB, "the other user's memory is left alone");
}

// Each device's blocks go with its own last context, whatever the other devices do.
void devices() {
    Cache c(64 * MB);
    void *a, *b;
    c.enter(1);
    c.enter(11);
    Fake::now = 11;
    c.take(&b, 20 * MB);
    c.give(b);
    Fake::now = 1;
    c.take(&a, 20 * MB);
    c.give(a);
    Fake::now = 11;
    c.leave(11, true);
    check(held_by(11) == 0 && held_by(1) == 20 * MB, "a device's blocks go with its last context");
    Fake::now = 1;
    c.take(&b, 20 * MB);
    check(b == a, "the other device still has its block");
    Fake::now = 11;
    c.enter(11);
    c.give(b);  // freed with another device current: not kept
    check(held_by(1) == 0, "another device's block is freed");
    c.leave(11, true);
    Fake::now = 1;
    c.leave(1, true);
}

// A second free of a matrix does nothing, as long as its memory has not been handed out again.
void twice() {
    Cache c(64 * MB);
    c.enter(1);
    void *a, *b, *d;
    c.take(&a, 20 * MB);
    c.give(a);
    c.give(a);
    check(held_by(1) == 20 * MB, "the kept block stays kept");
    c.take(&b, 20 * MB);
    c.take(&d, 20 * MB);
    check(b == a && d != b && held_by(1) == 40 * MB, "the block is handed out once");
    c.give(b);
    Fake::now = 11;
    c.give(b);  // with another device current
    Fake::now = 1;
    c.give(d);
    c.leave(1, true);
    check(held_by(1) == 0, "everything is given back");
}

// Freeing waits for nothing; a block is handed out when the device has been waited for since.
void waits() {
    Cache c(64 * MB);
    c.enter(1);
    void *a, *b, *d;
    c.take(&a, 10 * MB);
    c.take(&b, 20 * MB);
    Fake::waits = 0;
    c.give(a);
    c.give(b);
    check(Fake::waits == 0, "a free does not wait");
    c.take(&d, 20 * MB);
    check(d == b && Fake::waits == 1, "a reuse waits");
    c.take(&b, 10 * MB);
    check(b == a && Fake::waits == 1, "once for all blocks freed before");
    c.give(d);
    c.take(&a, 20 * MB);
    check(a == d && Fake::waits == 2, "and again for one freed since");
    c.give(a);
    Fake::wait_error = 1;
    c.take(&d, 20 * MB);
    check(held_by(1) == 10 * MB, "a block is not reused when the device reports an error");
    Fake::wait_error = 0;
    c.give(b);
    c.leave(1, true);
}

// The kept blocks make room for any allocation, and go when they are asked to, in their context.
void room() {
    Cache c(64 * MB);
    c.enter(1);
    c.enter(11);
    void *a, *b;
    Fake::room = 100 * MB;
    c.take(&a, 30 * MB);
    c.give(a);
    Fake::now = 11;
    check(c.alloc(&b, 101 * MB) == Fake::kOutOfMemory && held_by(1) == 30 * MB, "another device's blocks are no room");
    c.trim();
    check(held_by(1) == 30 * MB, "nor are they given back from there");
    Fake::now = 1;
    check(c.alloc(&b, 90 * MB) == Fake::kOk && held_by(1) == 90 * MB, "the kept block makes room");
    Fake::free(b);
    c.take(&a, 30 * MB);
    c.give(a);
    c.trim();
    check(held_by(1) == 0, "the kept blocks are given back");
    c.leave(1, true);
    Fake::now = 11;
    c.leave(11, true);
}
}  // namespace

int main(int argc, char **argv) {
    const struct {
        const char *name;
        void (*f)();
    } all[] = {{"reuse", reuse}, {"reset", reset}, {"devices", devices}, {"twice", twice}, {"waits", waits}, {"room", room}};
    for (auto &s : all)
        if (argc > 1 && !std::strcmp(argv[1], s.name)) {
            s.f();
            return g_bad ? 1 : 0;
        }
    return 2;
}
