// Walks the delay kernel's lists (delay_plan.h) as its gather does and compares every sum
// with the direct one: prints one line per plan, "plan accepted passes tile_src tiles
// threads smem near_k rest" and "sum <hash of all sums>", and returns 1 on any difference.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "../cubnm_b200/csrc/delay_plan.h"

using namespace cbnm;

template <class R>
static int check(int n, int n_sims, int sms, double density, int dmin, int dmax, int tables, int n_noise) {
    std::mt19937 g(n * 1000 + dmax);
    std::uniform_real_distribution<double> u(0, 1);
    const size_t nn = (size_t)n * n;
    std::vector<double> sc(nn);
    for (double &v : sc) v = u(g) < density ? u(g) : 0.0;
    std::vector<int> delay(nn * tables), sc_of(n_sims, 0), table_of(n_sims);
    for (int t = 0; t < tables; ++t)   // table t: the first one's delays at (t + 1) times the speed
        for (size_t i = 0; i < nn; ++i) {
            delay[t * nn + i] = t ? std::max(1, delay[i] / (t + 1)) : dmin + (int)(u(g) * (dmax - dmin + 1));
        }
    for (int s = 0; s < n_sims; ++s) table_of[s] = s % tables;
    DelayPlan p;
    const bool ok = build_delay_plan<R>(p, n, n_sims, n_noise, sms, sc.data(), sc_of.data(), delay, table_of, (size_t)1 << 30);
    std::printf("plan %d passes %d tile_src %d tiles %d threads %d smem %d near_k %d rest %d", ok, p.passes, p.tile_src, p.tiles, p.threads,
                p.smem, p.near_k, (int)p.rest.size());
    if (!ok) {
        std::printf(" sum 0\n");
        return 0;
    }
    std::vector<int> table(p.n_pairs, -1);   // delay table of each pair that is taken
    int most = 0;
    for (int s : p.sims) table[p.pair[s]] = table_of[s];
    for (int t : table)
        for (size_t i = 0; i < nn; ++i)
            if (sc[i] != 0.0) most = std::max(most, delay[t * nn + i]);
    if ((int)(p.sims.size() + p.rest.size()) != n_sims) return 1;
    const int W = p.window, WS = delay_stride(W), nh = (n + p.passes - 1) / p.passes;
    if (p.smem > DELAY_SMEM_SM - 1024 || p.tile_src * WS > 65536 || W < most) return 1;
    std::vector<R> x((size_t)n * (W + DELAY_BLOCK));   // x_k(t0 - W + i); i >= W: this block's values
    for (R &v : x) v = (R)u(g);
    uint64_t hash = 1469598103934665603ull;
    for (int q = 0; q < p.n_pairs; ++q) {
        const int *d = delay.data() + (size_t)table[q] * nn;
        for (int pass = 0; pass < p.passes; ++pass) {
            const int h0 = pass * nh, h1 = std::min(n, h0 + nh);
            std::vector<R> row((size_t)(h1 - h0) * 32, R(0));
            for (int t = 0; t < p.tiles; ++t) {
                const int *at = p.blob_at.data() + ((size_t)q * p.passes + pass) * (p.tiles + 1) + t;
                const unsigned char *b = p.blob.data() + 16 * (size_t)at[0];
                if ((at[1] - at[0]) * 16 > p.blob_max) return 1;
                const TileHead *h = (const TileHead *)b;
                const unsigned *end = (const unsigned *)(b + sizeof(TileHead));
                const int s0 = t * p.tile_src, cnt = std::min(p.tile_src, n - s0);
                std::vector<R> win((size_t)p.tile_src * WS, R(0));   // windows, then zeros
                for (int k = 0; k < cnt; ++k)
                    for (int i = 0; i < W; ++i) win[(size_t)k * WS + i] = x[(size_t)(s0 + k) * (W + DELAY_BLOCK) + i];
                unsigned e = 0;
                for (int j = 0; j < h1 - h0; ++j)
                    for (; e < end[j]; ++e)
                        for (int two = 0; two < 2; ++two) {
                            const int o = ((const uint16_t *)(b + h->off_at))[2 * e + two];
                            const R w = ((const R *)(b + h->w_at))[2 * e + two];
                            for (int lane = 0; lane < 32; ++lane) {
                                if (o + lane >= cnt * WS) return 1;
                                R &acc = row[(size_t)j * 32 + lane];
                                acc = std::fma(w, win[o + lane], acc);
                            }
                        }
            }
            for (int j = h0; j < h1; ++j)
                for (int lane = 0; lane < 32; ++lane) {
                    R gather = R(0), steps = R(0), got = row[(size_t)(j - h0) * 32 + lane], late = R(0);
                    for (int k = 0; k < n; ++k) {
                        const double v = sc[(size_t)k * n + j];
                        if (v == 0.0) continue;
                        const int dk = d[(size_t)k * n + j], i = W + lane - dk;
                        const R xk = x[(size_t)k * (W + DELAY_BLOCK) + i];
                        if (i < W) gather = std::fma((R)v, xk, gather);
                        else steps = std::fma((R)v, xk, steps);
                    }
                    for (int r = 0; r < p.near_cnt[q]; ++r) {   // the step loop's share
                        const size_t at = ((size_t)q * p.near_k + r) * n + j;
                        const int o = p.near[at], dk = o % DELAY_BLOCK;
                        if (dk && lane >= dk)
                            late = std::fma((R)p.near_w[at], x[(size_t)(o / DELAY_BLOCK) * (W + DELAY_BLOCK) + W + lane - dk], late);
                    }
                    if (got != gather || late != steps) return 1;
                    unsigned char bytes[sizeof(R)];
                    std::memcpy(bytes, &got, sizeof(R));
                    for (unsigned char c : bytes) hash = (hash ^ c) * 1099511628211ull;
                }
        }
    }
    std::printf(" sum %llx\n", (unsigned long long)hash);
    return 0;
}

int main(int argc, char **argv) {
    if (argc != 10) return 2;
    const int n = std::atoi(argv[2]), sims = std::atoi(argv[3]), sms = std::atoi(argv[4]);
    const double density = std::atof(argv[5]);
    const int dmin = std::atoi(argv[6]), dmax = std::atoi(argv[7]), tables = std::atoi(argv[8]), noise = std::atoi(argv[9]);
    return argv[1][0] == 'd' ? check<double>(n, sims, sms, density, dmin, dmax, tables, noise)
                             : check<float>(n, sims, sms, density, dmin, dmax, tables, noise);
}
