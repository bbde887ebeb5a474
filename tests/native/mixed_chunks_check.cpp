// CPU check of the mixed tile kernel's source chunks (plan_tools.h): mixed_chunk_time against the CTAs
// dealt out one by one, and mixed_chunk_count never more than 15 % above the best chunk
// count by it.
#include <cmath>
#include <cstdio>
#include <functional>
#include <queue>
#include <vector>

#include "../../red.cuda.closeencounter_gb300/csrc/plan_tools.h"

static double dealt(int sinks, int src, int tiles, int slots)
{
    std::priority_queue<double, std::vector<double>, std::greater<double>> free;
    for (int k = 0; k < slots; k++) free.push(0.0);
    double end = 0.0;
    for (int at = 0; at < src; at += tiles) {
        const int n = src - at < tiles ? src - at : tiles;
        for (int s = 0; s < sinks; s++) {
            const double t = free.top() + n + redgb::MIXED_START_COST;
            free.pop();
            free.push(t);
            if (t > end) end = t;
        }
    }
    return end;
}

int main()
{
    int cases = 0, bad = 0;
    for (int sinks = 1; sinks < 260; sinks += 1 + sinks / 9)
        for (int src = 1; src < 140; src += 1 + src / 7)
            for (int sm : {8, 152}) {
                const int slots = 2 * sm;
                double best = 1e300;
                for (int tiles = 1; tiles <= src; tiles += 1 + tiles / 5) {
                    const double a = redgb::mixed_chunk_time(sinks, src, tiles, slots), b = dealt(sinks, src, tiles, slots);
                    cases++;
                    if (std::fabs(a - b) > 1e-6 * b) {
                        bad++;
                        printf("%d x %d by %d on %d: %g, not %g\n", sinks, src, tiles, slots, a, b);
                    }
                }
                for (int n = 1; n <= src; n++) best = std::fmin(best, dealt(sinks, src, (src + n - 1) / n, slots));
                const int n = redgb::mixed_chunk_count(sinks, src, sm);
                const double took = n >= 1 && n <= src ? dealt(sinks, src, (src + n - 1) / n, slots) : 1e300;
                cases++;
                if (took > 1.1501 * best) {
                    bad++;
                    printf("%d x %d on %d: %d chunks take %g, %g is possible\n", sinks, src, slots, n, took, best);
                }
            }
    // sizes that lost by chunks of six tiles at least: (bodies + 127) / 128 sinks, (bodies + 258) / 256 sources
    const int sizes[] = {6600, 6800, 8200, 8500, 8800, 9200, 9600}, tiles[] = {5, 5, 4, 4, 9, 9, 10};
    for (int k = 0; k < 7; k++) {
        const int src = (sizes[k] + 258) / 256, n = redgb::mixed_chunk_count((sizes[k] + 127) / 128, src, 152);
        cases++;
        if ((src + n - 1) / n != tiles[k]) {
            bad++;
            printf("%d bodies: chunks of %d\n", sizes[k], (src + n - 1) / n);
        }
    }
    printf("cases %d bad %d\n", cases, bad);
    return bad ? 1 : 0;
}
