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

int main()
{
    for (int len : {0, 1, 1023, 1024, 8191, 8192, 8193, 16385, 1 << 20})
        for (int e : {len, INT_MAX - 8192, INT_MAX - 1, INT_MAX}) check_walk_range<1024, 8>(len, e);
    if (failures) return 1;
    std::printf("ok\n");
    return 0;
}
