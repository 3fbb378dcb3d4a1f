// The plans of the W4A16 column-owner kernel over products and devices: strips that clusters share are resident at once, by what a
// CTA's shared memory leaves of an SM and (on 148 SMs) by the clusters that a B200 holds.  Built with the undefined-behaviour checks of
// the host compiler; no CUDA call is made.
#include "handle.cu"
#include "gemm_s4_f16_small.cu"

#include <cstdio>

int main()
{
    // clusters of 1 to 8 CTAs that a B200 holds with three and with two CTAs on an SM (cudaOccupancyMaxActiveClusters)
    const int most[2][9] = {{0, 444, 222, 142, 104, 82, 71, 56, 48}, {0, 296, 148, 93, 71, 56, 45, 37, 33}};
    const int max_smem = 227 * 1024;
    int       failures = 0;
    for (int N = 32; N <= 16384; N += 32) {
        for (int K : {128, 1024, 4096, 8192, 11008, 24704, 28672, 32768}) {
            for (int T : {1, 8, 12, 16}) {
                for (int variant : {1, 2}) {
                    for (int sms : {148, 132, 20}) {
                        const tmb::GemmSmallPlan pl = tmb::gemm_small_plan(N, T, K, sms, max_smem, variant);
                        if (!pl.cols_tiles) continue;
                        const int strips = (N / 32 + pl.cols_tiles - 1) / pl.cols_tiles, per_sm = (int)((max_smem + 1024) / (pl.smem_bytes + 1024));
                        const int wanted = pl.cols_tiles == 1 && T <= 8 ? 3 : 2, slots = sms * (per_sm < wanted ? per_sm : wanted);
                        bool      ok = pl.ctas == strips * pl.cols_cluster && pl.cols_cluster >= 1 && pl.cols_cluster <= 8 && pl.smem_bytes <= (size_t)max_smem;
                        if (pl.cols_cluster > 1) ok = ok && pl.ctas <= slots && (sms != 148 || strips <= most[slots == 444 ? 0 : 1][pl.cols_cluster]);
                        if (ok) continue;
                        ++failures;
                        std::fprintf(stderr, "%d x %d, %d tokens, variant %d, %d SMs: clusters of %d on %d strips, %d CTAs an SM\n", N, K, T, variant, sms,
                                     pl.cols_cluster, strips, per_sm);
                    }
                }
            }
        }
    }
    if (!failures) std::puts("plans ok");
    return failures ? 1 : 0;
}
