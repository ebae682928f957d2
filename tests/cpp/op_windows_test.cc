// The windows of the resolver's bitmap sort (xkaapi_b200/csrc/op_windows.h): they follow one another
// without a gap, end exactly at the last op and number no op past an int, up to the most ops a batch may have.
#include "../../xkaapi_b200/csrc/op_windows.h"

#include <cstdio>
#include <initializer_list>

using namespace xkb;

static int check(int nops, int words)
{
    long windows = 0;
    int at = 0;
    while (at < nops)
    {
        const OpWindow w = OpWindow::from(at, words, nops);
        if (w.first != at || w.last <= at || w.last > nops) return 1;
        if ((long) w.last - w.first > 32L * words) return 2;
        if (w.last < nops && w.last - w.first != 32 * words) return 3;
        if (!w.holds(at) || !w.holds(w.last - 1) || w.holds(w.last) || (at > 0 && w.holds(at - 1))) return 4;
        at = w.last;
        ++windows;
    }
    return windows == ((long) nops + 32L * words - 1) / (32L * words) ? 0 : 5;
}

int main()
{
    const int most = (int) RESOLVE_MAX_OPS;
    for (int words : {1, 7, 1024, 40960})
        for (int nops : {1, 31, 32, 33, 32 * words - 1, 32 * words, 32 * words + 1, 1000003, most - 1, most, INT_MAX - 1, INT_MAX})
        {
            if (words < 1024 && nops > 2000000) continue;
            if (const int e = check(nops, words)) { fprintf(stderr, "nops %d, words %d: %d\n", nops, words, e); return 1; }
        }
    // a thread of a grid of up to 2^20 threads steps past the last op without leaving an int
    if (RESOLVE_MAX_OPS + (1u << 20) > (uint64_t) INT_MAX) { fprintf(stderr, "no room for a grid's step\n"); return 1; }
    puts("ok");
    return 0;
}
