// csrc/retry.h: prints how many of `calls` calls tried an allocation that is
// refused for the first `refused` calls, and the call that succeeded (-1: none).
#include <cstdio>
#include <cstdlib>

#include "retry.h"

int main(int argc, char **argv)
{
    const long calls = argc > 1 ? std::atol(argv[1]) : 0, refused = argc > 2 ? std::atol(argv[2]) : 0;
    gbfs::Retry r;
    long tries = 0, at = -1;
    for (long i = 0; i < calls && at < 0; i++) {
        if (!r.due()) continue;
        tries++;
        if (i < refused) {
            r.failed();
        } else {
            r.succeeded();
            at = i;
        }
    }
    std::printf("%ld %ld\n", tries, at);
    return 0;
}
