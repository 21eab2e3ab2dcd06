// Host check of alloc_or_release (kbw_gb300/csrc/retry.h) with a fake allocator.
#include <stdio.h>

#include "../../kbw_gb300/csrc/retry.h"

enum Code { OK, OUT, OTHER };

int main() {
    int bad = 0;
    auto run = [&](Code first, bool idle, Code second, Code want, int want_allocs, int want_releases) {
        int allocs = 0, releases = 0;
        const Code got = kbwg::alloc_or_release(
            OUT, [&] { return ++allocs == 1 ? first : second; },
            [&] {
                releases++;
                return idle;
            });
        if (got != want || allocs != want_allocs || releases != want_releases) {
            printf("first %d idle %d: got %d after %d allocations, %d releases\n", first, idle, got, allocs, releases);
            bad++;
        }
    };
    run(OK, true, OTHER, OK, 1, 0);     // enough memory: nothing is given up
    run(OTHER, true, OK, OTHER, 1, 0);  // another error: likewise
    run(OUT, false, OK, OUT, 1, 1);     // nothing idle: no second try
    run(OUT, true, OK, OK, 2, 1);
    run(OUT, true, OUT, OUT, 2, 1);     // still short: the error stands
    return bad;
}
