// CPU check of fp64_block_form and PairparSinks (plan_tools.h): the form of the blocks on both sides of
// each line, no line crossed twice along a block's sinks or sources, and the sinks of a CTA against a
// count of waves and steps made here.
#include <cmath>
#include <cstdio>
#include <initializer_list>

#include "../../red.cuda.closeencounter_gb300/csrc/plan_tools.h"

using namespace redgb;

int main()
{
    int bad = 0, cases = 0;
    auto expect = [&](long rows, long sources, Fp64Form want) {
        cases++;
        const Fp64Form got = fp64_block_form(rows, rows * sources);
        if (got != want) {
            bad++;
            printf("%ld rows of %ld: form %d, not %d\n", rows, sources, (int)got, (int)want);
        }
    };
    // sinks x sources: rows up to 300 + 3 sources + sources^2 / 250 ...
    for (long src : {65, 103, 203, 303, 403}) {
        const long line = (300000 + 3000 * src + 4 * src * src) / 1000;
        expect(1, src, FP64_FORM_ROWS);
        expect(line, src, FP64_FORM_ROWS);
        expect(line + 1, src, FP64_FORM_PAIRPAR);
        const long last = 1200000 / (src - 60);  // ... pair by pair up to rows (sources - 60) = 1 200 000
        expect(last, src, FP64_FORM_PAIRPAR);
        expect(last + 1, src, FP64_FORM_CERT);
        expect(1000000, src, FP64_FORM_CERT);
    }
    expect(3016, 603, FP64_FORM_ROWS);
    expect(5000, 603, FP64_FORM_CERT);
    expect(1500, 1500, FP64_FORM_ROWS);  // square blocks by their pairs
    expect(1501, 1501, FP64_FORM_CERT);
    expect(131074, 131074, FP64_FORM_CERT);
    expect(268435456, 65, FP64_FORM_CERT);
    expect(3, 268435456, FP64_FORM_CERT);
    expect(0, 0, FP64_FORM_ROWS);
    for (long src = 65; src < 3000; src += 7) {  // along the sinks: rows, pair by pair, certified, each once
        int before = 0;
        for (long rows = 1; rows < 400000; rows += 1 + rows / 50) {
            const Fp64Form f = fp64_block_form(rows, rows * src);
            const int now = f == FP64_FORM_ROWS ? 0 : (f == FP64_FORM_PAIRPAR ? 1 : 2);
            cases++;
            bad += now < before;
            before = now;
        }
    }
    for (int n : {1, 3, 28, 65, 103, 1000, 5000, 20000, 50000})
        for (int src : {33, 65, 73, 103, 128, 129, 203, 403})
            for (int blocks : {1, 8, 64, 1000}) {
                PairparSinks p;
                for (int k = 0; k < blocks; k++) p.add(n, src);
                const int S = p.best(3, 152);
                double least = 1e300;
                int want = 0;
                for (int q : {4, 8, 16, 32}) {
                    const long ctas = (long)blocks * ((n + q - 1) / q);
                    long steps = 2;
                    for (int j = 0; j < src; j += 1024 / q) {  // a tile of sources: a step per 256 pairs
                        const int m = src - j < 1024 / q ? src - j : 1024 / q;
                        steps += (m * q + 255) / 256;
                    }
                    const double waves = (double)ctas / 456.0;
                    const double cost = (2.0 * std::ceil(waves) + (waves > 1.0 ? waves : 1.0)) * (double)steps;
                    if (cost < least) {
                        least = cost;
                        want = q;
                    }
                }
                cases++;
                if (S != want) {
                    bad++;
                    printf("%d blocks of %d sinks, %d sources: %d, not %d\n", blocks, n, src, S, want);
                }
            }
    PairparSinks none;
    bad += none.best(3, 152) != 8;
    printf("cases %d bad %d\n", cases, bad);
    return bad ? 1 : 0;
}
