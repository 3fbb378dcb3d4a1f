// The launch plans of the decode attention over batches, heads, capacities and devices: splits of an int8 cache are never longer than
// those of an fp16 one, whatever room the sequences have.  Built with the undefined-behaviour checks of the host compiler; no CUDA
// call is made.
#include "handle.cu"
#include "mmha.cu"

#include <cstdio>

int main()
{
    int failures = 0;
    const int heads[][2] = {{32, 32}, {64, 8}, {8, 1}, {40, 40}, {4, 4}};
    for (auto& hh : heads) {
        for (int B : {1, 2, 4, 13, 21, 64, 300}) {
            for (int capacity : {0, 1, 64, 200, 1024, 2047, 2049, 4096, 8192, 16384, 131072}) {
                for (int sms : {148, 66, 1}) {
                    const tmb::MmhaPlan i8 = tmb::mmha_plan(B, hh[0], hh[1], capacity, sms, 0, 0, true), f16 = tmb::mmha_plan(B, hh[0], hh[1], capacity, sms, 0, 0, false);
                    for (const tmb::MmhaPlan& pl : {i8, f16}) {
                        if (pl.chunk >= 64 && pl.chunk % 64 == 0 && (long long)pl.chunk * pl.max_splits >= capacity) continue;
                        ++failures;
                        std::fprintf(stderr, "%d x %d heads, capacity %d, %d SMs: splits of %d do not cover it\n", B, hh[0], capacity, sms, pl.chunk);
                    }
                    if (i8.chunk > f16.chunk && i8.chunk > 192) {
                        ++failures;
                        std::fprintf(stderr, "%d x %d / %d heads, capacity %d, %d SMs: splits of %d, fp16 %d\n", B, hh[0], hh[1], capacity, sms, i8.chunk, f16.chunk);
                    }
                }
            }
        }
    }
    if (!failures) std::puts("plans ok");
    return failures ? 1 : 0;
}
