// Walks of csrc/index.h over ranges that end at the largest index of their type.
// Compiled with traps on signed overflow; prints "ok" when every walk has taken
// each entry of its range once.
#include <climits>
#include <cstdio>
#include <vector>

#include "index.h"

static int failures = 0;

static void expect(bool ok, const char *what, long long a, long long b)
{
    if (ok) return;
    ++failures;
    std::printf("%s: %lld %lld\n", what, a, b);
}

template <int BLOCK, int ILP>
static void check_walk_range(int len, int e)
{
    const int s = e - len;
    std::vector<int> seen(len, 0);
    long long calls = -1;
    for (int t = 0; t < BLOCK; t++) {
        long long mine = 0, taken = 0;
        gbfs::walk_range<BLOCK, ILP>(
            s, e, t,
            [&](int i) {
                expect(i >= s && i < e, "walk_range reads outside", i, e);
                if (i >= s && i < e) seen[i - s]++;
                return (unsigned)i;
            },
            [&](unsigned v, bool in) {
                mine++;
                taken += in;
                expect(!in || (int)v >= s, "walk_range value", v, s);
            });
        if (calls < 0) calls = mine;
        expect(mine == calls, "threads differ in their calls", mine, calls);
    }
    for (int k = 0; k < len; k++) expect(seen[k] == 1, "walk_range entry", k, seen[k]);
}

// A range in steps of W x ILP entries, lane by lane: the form of the warps' walks
// over a row (W = 32) and of one thread's (W = 1).
template <typename T>
static void check_steps(T b, T e, int w, int ilp)
{
    std::vector<int> seen((size_t)(e - b), 0);
    long long steps = 0;
    for (T i0 = b; gbfs::idx_before(i0, e) && steps < 1 << 20; i0 = gbfs::idx_add(i0, w * ilp), steps++)
        for (int t = 0; t < ilp; t++)
            for (int lane = 0; lane < w; lane++) {
                const T i = gbfs::idx_add(i0, t * w + lane);
                if (!gbfs::idx_before(i, e)) continue;
                expect(i >= b && i < e, "a step outside", (long long)i, (long long)e);
                if (i >= b && i < e) seen[(size_t)(i - b)]++;
            }
    expect(steps == (long long)((e - b) + (w * ilp - 1)) / (w * ilp), "steps", steps, (long long)(e - b));
    for (size_t k = 0; k < seen.size(); k++) expect(seen[k] == 1, "an entry", (long long)k, seen[k]);
}

// A row in pieces: piece j is [b + j * piece, ...) up to the row's end.
template <typename T>
static void check_pieces(T b, T e, int piece, int count)
{
    long long total = 0;
    for (int j = 0; j < count; j++) {
        const T s = gbfs::idx_add(b, j * piece), x = gbfs::idx_end(s, piece, e);
        if (!gbfs::idx_before(s, e)) continue;  // past the row's end: no entries
        expect(s >= b && x > s && x <= e, "a piece outside", (long long)s, (long long)x);
        total += x - s;
    }
    expect(total == (long long)(e - b), "entries in pieces", total, (long long)(e - b));
}

template <typename T>
static void check_rows(T last)
{
    for (int back : {0, 1, 3, 31, 127, 255, 4095})
        for (int len : {0, 1, 2, 4, 5, 31, 33, 129, 2049, 5000, 9000}) {
            const T e = last - back, b = e - len;
            for (int ilp : {1, 2, 4, 8}) {
                check_steps<T>(b, e, 32, ilp);
                check_steps<T>(b, e, 1, ilp);
            }
            check_pieces<T>(b, e, 2048, (len + 2047) / 2048);
            check_pieces<T>(b, e, 512, 4 * ((len + 2047) / 2048));
        }
    expect(gbfs::idx_mid<T>(last - 1, last) == last - 1, "idx_mid", (long long)gbfs::idx_mid<T>(last - 1, last), (long long)last);
    expect(gbfs::idx_mid<T>(last / 2 + 1, last) > last / 2, "idx_mid", 0, (long long)last);
    expect(gbfs::idx_mid<T>(3, 3) == 3 && gbfs::idx_mid<T>(3, 4) == 3 && gbfs::idx_mid<T>(3, 5) == 4, "idx_mid", 3, 5);
}

int main()
{
    check_rows<int>(INT_MAX);
    check_rows<long long>((1ll << 33) + 5);
    for (int len : {0, 1, 1023, 1024, 8191, 8192, 8193, 16385, 1 << 20})
        for (int e : {len, INT_MAX - 8192, INT_MAX - 1, INT_MAX}) check_walk_range<1024, 8>(len, e);
    if (failures) return 1;
    std::printf("ok\n");
    return 0;
}
