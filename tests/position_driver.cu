// Host-side check of the arithmetic on entry positions (no GPU): the library's own helpers,
// walked as the kernels walk them, around the largest nnz (2^31 - 1).
#include <cstdio>

#include "../apspie_b200/csrc/common.cuh"

using namespace apspie;

namespace {
int g_bad = 0;
void check(bool ok, const char *what, long long a, long long b) {
    if (ok) return;
    ++g_bad;
    std::printf("%s: %lld %lld\n", what, a, b);
}

// Tiles of `tile` edges through unit u of a queue of E edges: every edge of the unit once.
void walk_unit(int u, int shift, int E, int tile) {
    const long long first = static_cast<long long>(u) << shift;
    const long long last = first + (1ll << shift) < E ? first + (1ll << shift) : E;
    const int end = static_cast<int>(last);
    long long want = first;
    int steps = 0;
    for (int t0 = u << shift, t1; t0 < end && steps <= (1 << shift) / tile; t0 = t1, ++steps) {
        t1 = step_end(t0, tile, end);
        check(t1 > t0 && t1 <= end, "tile", t0, t1);
        for (int x = 0; x < tile; ++x)
            if (x < t1 - t0) check(t0 + x == want++, "edge", t0 + x, want);
    }
    check(want == last, "edges of a unit", want, last);
}

// Steps of `step` entries through a row [r0, r1), in parts of `part`.
void walk_row(long long r0, long long r1, int step, int part) {
    long long want = r0;
    int parts = 0;
    for (int from = static_cast<int>(r0); from < r1 && parts < 64; ++parts) {
        const int lim = step_end(from, part, static_cast<int>(r1));
        check(lim > from && lim <= r1, "part", from, lim);
        int steps = 0;
        for (Pos e = from; e < static_cast<Pos>(lim) && steps <= part / step; e += step, ++steps)
            for (int k = 0; k < step; ++k)
                if (e + k < static_cast<Pos>(lim)) check(static_cast<long long>(e + k) == want++, "entry", e + k, want);
        from = lim;
        if (lim == r1) break;
    }
    check(want == r1, "entries of a row", want, r1);
}
}  // namespace

int main() {
    const long long most = 0x7fffffffll;
    for (long long E : {1ll, 127ll, 128ll, 129ll, 5000ll, most - 129, most - 128, most - 127, most - 1, most})
        for (int shift : {7, 11, 16}) {
            const int units = static_cast<int>((E - 1) >> shift) + 1;
            for (int u = units > 2 ? units - 2 : 0; u < units; ++u) walk_unit(u, shift, static_cast<int>(E), 128);
        }
    for (long long len : {0ll, 1ll, 3ll, 8ll, 9ll, 130ll, 2048ll, 2049ll, 20000ll})
        for (long long r1 : {len, most - 5, most - 1, most})
            for (int step : {4, 64, 128, 1024})
                for (int part : {1024, 2048, 16384}) walk_row(r1 - len, r1, step, part);
    return g_bad ? 1 : 0;
}
