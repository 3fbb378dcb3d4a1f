// The launch plans of the W4A16 tensor-core GEMM over a range of products and devices: every plan covers the product, and CTAs
// that wait for one another are resident together.  Built with the undefined-behaviour checks of the host compiler; no CUDA call is made.
#include "handle.cu"
#include "gemm_s4_f16_tc.cu"

#include <cstdio>

static int failures = 0;

static void check(bool ok, const char* what, int N, int T, int K, int sms, int balance)
{
    if (ok) return;
    ++failures;
    std::fprintf(stderr, "%s: %d x %d, %d tokens, %d SMs, balance %d\n", what, N, K, T, sms, balance);
}

static void check_tc(int N, int T, int K, int sms, bool balance)
{
    const tmb::GemmTcPlan pl = tmb::gemm_tc_plan(N, T, K, sms, balance);
    const int             G  = K / 128;
    const long long       tiles = (long long)pl.t_chunks * pl.n_col_tiles;
    check(pl.units_per_cta >= 1 && pl.ctas >= 1, "an empty plan", N, T, K, sms, balance);
    if (pl.parts_per_tile) {
        check(pl.ctas == pl.n_col_tiles * pl.parts_per_tile, "parts", N, T, K, sms, balance);
        check((long long)pl.parts_per_tile * pl.units_per_cta >= G && (pl.parts_per_tile - 1) * pl.units_per_cta < G, "parts of a tile", N, T, K, sms, balance);
    }
    else {
        check((long long)pl.ctas * pl.units_per_cta >= pl.total_units && (long long)(pl.ctas - 1) * pl.units_per_cta < pl.total_units, "units", N, T, K, sms, balance);
    }
    if (pl.units_per_cta % G) {
        check((long long)pl.ctas * pl.t_chunks <= sms, "CTAs that wait for one another do not fit", N, T, K, sms, balance);
        check(pl.workspace_floats > 0, "no workspace", N, T, K, sms, balance);
    }
    check(pl.last_sums == (tiles >= sms && pl.units_per_cta != G), "who sums", N, T, K, sms, balance);
    if (!balance && tiles >= sms) check(pl.units_per_cta == G && pl.workspace_floats == 0, "cut without balance", N, T, K, sms, balance);
}

int main()
{
    const int shapes[][2] = {{12288, 4096}, {4096, 4096}, {22016, 4096}, {4096, 11008}, {57344, 8192}, {8192, 28672}, {10240, 8192}, {1280, 8192},
                             {57344, 1024}, {32, 128}, {288, 384}, {128000, 128}};
    for (auto& s : shapes) {
        for (int T : {1, 9, 16, 17, 21, 32, 33, 128, 129, 200, 1000, 1600, 4096, 20000}) {
            for (int sms : {148, 132, 66, 2, 1}) {
                check_tc(s[0], T, s[1], sms, false);
                check_tc(s[0], T, s[1], sms, true);
            }
        }
    }
    // the sizes that tests/test_gpu_many_tokens.py runs as products cut evenly although there is a tile for every SM
    const int even[][3] = {{57344, 1024, 17}, {40960, 2048, 100}, {22016, 4096, 200}};
    for (auto& s : even) {
        const tmb::GemmTcPlan pl = tmb::gemm_tc_plan(s[0], s[2], s[1], 148, true);
        check(pl.last_sums && pl.units_per_cta % (s[1] / 128) && pl.t_chunks * pl.n_col_tiles >= 148, "not cut evenly", s[0], s[2], s[1], 148, true);
    }
    if (!failures) std::puts("plans ok");
    return failures ? 1 : 0;
}
