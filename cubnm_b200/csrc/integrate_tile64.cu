// FP64 integrators for networks of up to 128 nodes without delays: the reference's time
// loop (src/ext/bnm.cu:117-505) with the SC in registers.
//
// The per-simulation kernel (integrate_sim.cuh) runs one thread per node; at every step a
// thread walks its SC column in one chain of dependent additions, loading each weight
// again, then the update (two exponentials and two divisions for rWW) runs on as many
// threads as nodes.  At 100 nodes a step took about 4,200 cycles alone on an SM and
// 1,264 cycles per simulation with the SM full, of which the FP64 pipe (64 lanes an SM)
// needs about 370.  Two forms replace it:
//
//  * k_one64, small batches: one CTA per simulation.  The n x n product with x is spread
//    over the lanes: a group of eight holds four rows of SC^T, each lane one chain of the
//    sources, in registers; partial sums meet in a transposing butterfly (4 shuffles) and
//    the update runs on one thread per node.  Bound by latency: product, two barriers,
//    update chain.
//  * k_tile64, larger batches: eight simulations sharing an SC per CTA, the product as
//    mma.sync m8n8k4 (FP64), SC^T fragments in registers, so that a weight read serves
//    eight simulations and the sums need no shuffles.  DMMA runs at the FP64 pipe's rate
//    on sm_100a (measured 63.7 multiply-adds a cycle and SM for both), so this saves
//    loads and latency, not FP64 work: bound by the FP64 pipe (product 169 cycles per
//    simulation and step at 100 nodes, update about 180).  The Balloon-Windkessel model
//    of a tile runs in up to four more warps, a millisecond behind.
//
// Both form a sum in one order, so that a simulation has the same bits in any batch: chain
// (h, e), h < 4, e < 2, runs over sources 8 c + 2 t + e, c = h, h + 4, .., t = 0 .. 3, by
// fused multiply-adds from zero (m8n8k4 adds its four products one after the other, rounding
// each: equal to the chain of fma in all of 65,536 random sums); then e = 0 and e = 1 each
// ((h0 + h2) + (h1 + h3)), then both.  Measured against two chains of free order: tiles
// 1-5 % slower (rWW 100 nodes, 1,184 simulations, 21.9 -> 22.6 ms per simulated second), one
// simulation at 100 nodes 8.2 -> 7.5 ms (four rows a group of eight lanes instead of two a
// group of sixteen halve the loads of x; rWW 68 nodes 6.4 -> 6.5).
//
// Noise rows are copied to shared memory a chunk of steps ahead.  The sums are formed in
// another order than the reference's, and multiply-adds are fused, in the update too.
#include <algorithm>
#include <cstdint>
#include "engine.h"
#include "models.cuh"
#include "tc_common.cuh"

namespace cbnm {
namespace {

constexpr int TS = 8;            // simulations per tile (MMA N)
constexpr int NOISE_CHUNK = 10;  // steps of noise per shared-memory buffer (two buffers)

__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}
template <int B>
__device__ __forceinline__ void cp_small(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_u32(dst)), "l"(src), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Noise of `cnt` steps from inner step i0 of Balloon-Windkessel step b to dst [step][n][NN]
// (sh_ts is [repeats][noise_bw_it], one run of Balloon-Windkessel steps).
template <int NN>
__device__ __forceinline__ void stage_noise(const IntegrateArgs &a, int b, int i0, int cnt, double *dst, int nwarps) {
    const int n = a.nodes, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int *shn = a.sh_nodes + (size_t)(b / a.noise_bw_it) * n;
    const double *src = a.noise + ((long long)__ldg(a.sh_ts + b) * a.inner_it + i0) * n * NN;
    for (int q = warp; q < cnt; q += nwarps)
        for (int k = lane; k < n; k += 32)
            cp_small<NN * 8>(dst + ((size_t)q * n + k) * NN, src + ((size_t)q * n + __ldg(shn + k)) * NN);
}

// States of a sample: the time series, or the sum of the kept samples in the output itself.
template <class M>
__device__ __forceinline__ void states_out(const IntegrateArgs &a, const double (&s)[M::NS], int sim, int j, int states_i) {
    const int n = a.nodes;
    const size_t ext = a.states_ts ? (size_t)n * a.states_len : (size_t)n;
#pragma unroll
    for (int v = 0; v < M::NS; ++v) {
        double *out = a.states + ((size_t)v * a.n_sims + sim) * ext + j;
        if (a.states_ts) {
            if (states_i < a.states_len) out[(size_t)states_i * n] = s[v];
        } else if (states_i == a.n_states_samples_remove) {
            *out = 0.0 + s[v];
        } else if (states_i > a.n_states_samples_remove) {
            *out += s[v];
        }
    }
}
template <class M>
__device__ __forceinline__ void states_mean(const IntegrateArgs &a, int sim, int j, int states_i) {
    const int pts = states_i - a.n_states_samples_remove;
#pragma unroll
    for (int v = 0; v < M::NS; ++v) {
        double &out = a.states[((size_t)v * a.n_sims + sim) * (size_t)a.nodes + j];
        out = (pts > 0 ? out : 0.0) / pts;   // no kept sample: 0 / pts
    }
}

// Place of source k in k_one64's x: a lane reads two of its chain's sources in 16 bytes, the
// eight lanes of a group 128 in a row.
__device__ __forceinline__ int one_pos(int k) {
    const int t = (k >> 1) & 3, l = ((k >> 3) & 3) * 2 + (k & 1);
    return ((k >> 5) * 4 + (t & 2)) * 8 + 2 * l + (t & 1);
}

__device__ __forceinline__ double bold_of(const IntegrateArgs &a, double q, double nu) {  // bnm.cpp:316-335
    return a.bw.V_0 * (a.bw.k1 * (1 - q) + a.bw.k2 * (1 - q / nu) + a.bw.k3 * (1 - nu));
}

// ---------------------------------------------------------------- one simulation per CTA
__host__ __device__ constexpr bool one_par_smem(int nc) { return nc == 3; }   // parameters too
// NC: compiled count of 32-source blocks (32 NC >= n).  The Balloon-Windkessel state,
// touched once a millisecond, is in shared memory: the weights take 32 NC registers.
template <class M, int NC>
__global__ void __launch_bounds__(NC * 64) k_one64(const __grid_constant__ IntegrateArgs a) {
    constexpr int NN = M::NN;
    constexpr bool PAR_SMEM = one_par_smem(NC);
    extern __shared__ __align__(16) double sh[];
    const int n = a.nodes, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, l = lane & 7, nwarps = blockDim.x >> 5;
    const int chunk = min(a.inner_it, NOISE_CHUNK);
    double *x = sh, *in_s = x + 32 * NC, *bws = in_s + 32 * NC, *par = bws + 128 * NC;   // [32 NC], [32 NC], [4][32 NC]
    double *noise_s = par + (PAR_SMEM ? (M::NR + M::NG) * 32 * NC : 0);   // parameters [NR + NG][32 NC]; noise [2][chunk][n][NN]
    const int row0 = warp * 16 + (lane >> 3) * 4;                     // the four rows of this group of eight lanes
    const int my_row = row0 + (l >> 1);                               // the row whose sum this lane ends with
    const int j = tid;
    const bool act = j < n;
    for (int sim = blockIdx.x; sim < a.n_sims; sim += gridDim.x) {
        const double *SC = a.sc + (size_t)a.sc_idx[sim] * n * n;
        double w[4][4 * NC];   // chain l: sources 32 b + 8 (l / 2) + 2 t + l % 2
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int i = 0; i < 4 * NC; ++i) {
                const int k = (i >> 2) * 32 + (l >> 1) * 8 + 2 * (i & 3) + (l & 1);
                w[r][i] = row0 + r < n && k < n ? SC[(size_t)k * n + row0 + r] : 0.0;
            }
        double g[M::NG], iv[M::NI], r[M::NR], s[M::NS];
        const size_t rstride = (size_t)a.n_sims * n;
#pragma unroll
        for (int i = 0; i < M::NG; ++i) g[i] = a.gparams[(size_t)i * a.n_sims + sim];
#pragma unroll
        for (int i = 0; i < M::NR; ++i) r[i] = act ? a.rparams[i * rstride + (size_t)sim * n + j] : 0.0;
#pragma unroll
        for (int i = 0; i < M::NI; ++i) iv[i] = 0.0;
#pragma unroll
        for (int i = 0; i < M::NS; ++i) s[i] = 0.0;
        M::init(s, iv, g, r);
        if (PAR_SMEM && act) {
#pragma unroll
            for (int i = 0; i < M::NR; ++i) par[i * 32 * NC + j] = r[i];
#pragma unroll
            for (int i = 0; i < M::NG; ++i) par[(M::NR + i) * 32 * NC + j] = g[i];
        }
        double *const b = bws + j;   // x, f, nu, q at stride 32 NC
        if (act) {
            b[0] = 0.0;
            b[32 * NC] = b[64 * NC] = b[96 * NC] = 1.0;
        }
        for (int k = tid; k < 32 * NC; k += blockDim.x) x[k] = 0.0;   // padding
        __syncthreads();
        if (act) x[one_pos(j)] = s[M::CONN];
        stage_noise<NN>(a, 0, 0, chunk, noise_s, nwarps);
        cp_commit();
        cp_wait_all();
        __syncthreads();
        int nbuf = 0, bold_i = 0, states_i = 0, to_tr = a.bold_tr_iters, to_sample = a.states_sampling_iters;
        for (int bw_i = 0; bw_i < a.bw_it; ++bw_i) {
            for (int i0 = 0; i0 < a.inner_it; i0 += chunk) {
                const bool next_bw = i0 + chunk >= a.inner_it;
                double *nxt = noise_s + (size_t)(nbuf ^ 1) * chunk * n * NN;
                if (!next_bw) stage_noise<NN>(a, bw_i, i0 + chunk, min(chunk, a.inner_it - i0 - chunk), nxt, nwarps);
                else if (bw_i + 1 < a.bw_it) stage_noise<NN>(a, bw_i + 1, 0, chunk, nxt, nwarps);
                cp_commit();
                const int i1 = min(i0 + chunk, a.inner_it);
                for (int inner = i0; inner < i1; ++inner) {
                    double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
                    for (int i = 0; i < 4 * NC; i += 2) {
                        const double2 xk = *reinterpret_cast<const double2 *>(x + i * 8 + 2 * l);
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = fma(w[q][i + 1], xk.y, fma(w[q][i], xk.x, v[q]));
                    }
                    // transposing butterfly: lanes keep rows {0,1} / {2,3}, then one row, then its sum
                    const bool up = l & 4, odd = l & 2;
                    double m0 = up ? v[2] : v[0], m1 = up ? v[3] : v[1];
                    m0 += __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 4);
                    m1 += __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 4);
                    double m = odd ? m1 : m0;
                    m += __shfl_xor_sync(0xffffffffu, odd ? m0 : m1, 2);
                    m += __shfl_xor_sync(0xffffffffu, m, 1);
                    if ((l & 1) == 0) in_s[my_row] = m;
                    __syncthreads();
                    if (act) {
                        const double *z = noise_s + ((size_t)(nbuf * chunk + inner - i0) * n + j) * NN;
                        if constexpr (PAR_SMEM) {
#pragma unroll
                            for (int i = 0; i < M::NR; ++i) r[i] = par[i * 32 * NC + j];
#pragma unroll
                            for (int i = 0; i < M::NG; ++i) g[i] = par[(M::NR + i) * 32 * NC + j];
                        }
                        M::step(s, iv, g, r, in_s[j], z[0], NN > 1 ? z[NN - 1] : 0.0, a.K);
                        x[one_pos(j)] = s[M::CONN];
                    } else {   // assigned on every path, outputs of a step hold no register during the product
#pragma unroll
                        for (int i = 0; i < M::NS; ++i) s[i] = 0.0;
#pragma unroll
                        for (int i = 0; i < M::NI; ++i) iv[i] = 0.0;
                        if constexpr (PAR_SMEM) {
#pragma unroll
                            for (int i = 0; i < M::NR; ++i) r[i] = 0.0;
#pragma unroll
                            for (int i = 0; i < M::NG; ++i) g[i] = 0.0;
                        }
                    }
                    if (inner == i1 - 1) cp_wait_all();   // the next chunk's noise, before the barrier
                    __syncthreads();
                }
                nbuf ^= 1;
            }
            const bool tr = --to_tr == 0;
            if (act) {
                double bx = b[0], bf = b[32 * NC], bnu = b[64 * NC], bq = b[96 * NC];
                bw_step64(bx, bf, bnu, bq, s[M::BOLDV], a.bwf);
                b[0] = bx; b[32 * NC] = bf; b[64 * NC] = bnu; b[96 * NC] = bq;
                if (tr && bold_i < a.bold_len) a.bold[((size_t)sim * a.bold_len + bold_i) * n + j] = bold_of(a, bq, bnu);
            }
            if (tr) {
                to_tr = a.bold_tr_iters;
                ++bold_i;   // a sample past bold_len has no slot
            }
            if (--to_sample == 0) {
                to_sample = a.states_sampling_iters;
                if (a.ext_out) {
                    if (act) states_out<M>(a, s, sim, j, states_i);
                    ++states_i;
                }
            }
        }
        if (act && a.ext_out && !a.states_ts) states_mean<M>(a, sim, j, states_i);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- eight simulations per CTA
struct Layout {
    int mt, rs;                 // 8-node tiles (= node warps); doubles per simulation row of x (8 mod 16: no bank conflicts)
    int x, noise, bw, z, bytes; // byte offsets: x [2][8][rs], noise [2][chunk][n][NN], Balloon-Windkessel
                                // state [4][8 n] and inputs [2][8 n]
};
__host__ __device__ inline Layout layout(int n, int nn, int chunk) {
    Layout l;
    l.mt = (n + 7) / 8;
    l.rs = l.mt * 8 + (l.mt % 2 ? 0 : 8);
    l.x = 0;
    l.noise = 2 * TS * l.rs * 8;
    l.bw = l.noise + 2 * chunk * n * nn * 8;
    l.z = l.bw + 4 * TS * n * 8;
    l.bytes = l.z + 2 * TS * n * 8;
    return l;
}
// Balloon-Windkessel warps beside `mt` node warps: up to a multiple of four (a warp's
// registers come from its quarter of the SM).
__host__ __device__ constexpr int bw_warps(int mt) { return mt % 4 ? 4 - mt % 4 : mt < 16 ? 4 : 0; }
__host__ __device__ constexpr int min_ctas(int ks) { return ks <= 4 ? 2 : 1; }

// The Balloon-Windkessel warps: for every tile and millisecond, wait for the inputs of the
// 8 n items (item s n + j), step them two at a time, write BOLD at TR.
template <bool CALL>
__device__ __forceinline__ void bw_items(const IntegrateArgs &a, const int *td, double *b, const double *z, int tid, int nthr,
                                         bool tr, int bold_i) {
    const int n = a.nodes, items = TS * n;
    for (int i0 = tid; i0 < items; i0 += 2 * nthr) {
        const int at[2] = {i0, i0 + nthr < items ? i0 + nthr : i0};   // the last one may be alone: computed twice
        double x[2], f[2], nu[2], q[2], zz[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            x[u] = b[at[u]]; f[u] = b[items + at[u]]; nu[u] = b[2 * items + at[u]]; q[u] = b[3 * items + at[u]];
            zz[u] = z[at[u]];
        }
        bw_step64_n<2, CALL>(x, f, nu, q, zz, a.bwf);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            b[at[u]] = x[u]; b[items + at[u]] = f[u]; b[2 * items + at[u]] = nu[u]; b[3 * items + at[u]] = q[u];
            if (tr && bold_i < a.bold_len) {   // a sample past bold_len has no slot
                const int s = at[u] / n, j = at[u] - s * n, sim = td[1 + s];
                if (sim >= 0) a.bold[(size_t)sim * a.bold_len * n + (size_t)bold_i * n + j] = bold_of(a, q[u], nu[u]);
            }
        }
    }
}
template <bool CALL>
__device__ __forceinline__ void bw_role(const IntegrateArgs &a, double *b, const double *zs, int tid, int nthr) {
    const int items = TS * a.nodes;
    for (int tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
        const int *td = a.tiles + (size_t)tile * (TS + 1);
        for (int i = tid; i < items; i += nthr) {   // x = 0, f = nu = q = 1
            b[i] = 0.0;
            b[items + i] = b[2 * items + i] = b[3 * items + i] = 1.0;
        }
        int to_tr = a.bold_tr_iters, bold_i = 0;
        for (int bw_i = 0; bw_i < a.bw_it; ++bw_i) {
            const bool tr = --to_tr == 0;
            bar_sync(2, blockDim.x);
            bw_items<CALL>(a, td, b, zs + (bw_i & 1) * items, tid, nthr, tr, bold_i);
            if (tr) {
                to_tr = a.bold_tr_iters;
                ++bold_i;
            }
        }
        bar_sync(2, blockDim.x);
    }
}

// KS: compiled count of 8-node tiles (two K steps of 4 each), at least the run's.
template <class M, int KS>
__global__ void __launch_bounds__((KS + bw_warps(KS)) * 32, min_ctas(KS)) k_tile64(const __grid_constant__ IntegrateArgs a) {
    constexpr int NN = M::NN;
    constexpr bool BW_CALL = KS >= 13;   // see bw_step64_n
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = a.nodes, tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int chunk = min(a.inner_it, NOISE_CHUNK);
    const Layout L = layout(n, NN, chunk);
    double *xb = reinterpret_cast<double *>(smem + L.x);
    double *noise_s = reinterpret_cast<double *>(smem + L.noise);
    double *bws = reinterpret_cast<double *>(smem + L.bw), *zs = reinterpret_cast<double *>(smem + L.z);
    const int items = TS * n, node_threads = L.mt * 32;
    const bool bw_here = bw_warps(L.mt) == 0;   // 16 node warps: they do the Balloon-Windkessel work themselves
    if (warp >= L.mt) {
        bw_role<BW_CALL>(a, bws, zs, tid - node_threads, nthr - node_threads);
        return;
    }
    const int j = warp * 8 + g;                 // this lane's node; simulations 2t, 2t + 1 of the tile
    const bool act = j < n;
    const int jn = act ? j : 0;
    const size_t rstride = (size_t)a.n_sims * n;
    double w[KS][2];
    int sc_loaded = -1;
    for (int tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
        const int *td = a.tiles + (size_t)tile * (TS + 1);
        const int sc_idx = td[0];
        const int sims[2] = {td[1 + 2 * t], td[2 + 2 * t]};
        if (sc_idx != sc_loaded) {              // K step (c, e): lane t holds source 8 c + 2 t + e
            const double *SC = a.sc + (size_t)sc_idx * n * n;
#pragma unroll
            for (int c = 0; c < KS; ++c)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int k = 8 * c + 2 * t + e;
                    w[c][e] = act && k < n ? SC[(size_t)k * n + j] : 0.0;
                }
            sc_loaded = sc_idx;
        }
        double gl[2][M::NG], iv[2][M::NI], r[2][M::NR], s[2][M::NS];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const bool live = sims[u] >= 0;
#pragma unroll
            for (int i = 0; i < M::NG; ++i) gl[u][i] = live ? a.gparams[(size_t)i * a.n_sims + sims[u]] : 0.0;
#pragma unroll
            for (int i = 0; i < M::NR; ++i)
                r[u][i] = live && act ? a.rparams[i * rstride + (size_t)sims[u] * n + j] : 0.0;
#pragma unroll
            for (int i = 0; i < M::NI; ++i) iv[u][i] = 0.0;
#pragma unroll
            for (int i = 0; i < M::NS; ++i) s[u][i] = 0.0;
            M::init(s[u], iv[u], gl[u], r[u]);
        }
        if (bw_here)
            for (int i = tid; i < items; i += nthr) {
                bws[i] = 0.0;
                bws[items + i] = bws[2 * items + i] = bws[3 * items + i] = 1.0;
            }
        double *xc = xb, *xn = xb + TS * L.rs;
        auto write_x = [&](double *x) {
            x[(2 * t) * L.rs + j] = act ? s[0][M::CONN] : 0.0;
            x[(2 * t + 1) * L.rs + j] = act ? s[1][M::CONN] : 0.0;
        };
        write_x(xc);
        stage_noise<NN>(a, 0, 0, chunk, noise_s, L.mt);
        cp_commit();
        cp_wait_all();
        bar_sync(1, node_threads);
        int nbuf = 0, bold_i = 0, states_i = 0, to_tr = a.bold_tr_iters, to_sample = a.states_sampling_iters;
        for (int bw_i = 0; bw_i < a.bw_it; ++bw_i) {
            for (int i0 = 0; i0 < a.inner_it; i0 += chunk) {
                const bool next_bw = i0 + chunk >= a.inner_it;
                double *nxt = noise_s + (size_t)(nbuf ^ 1) * chunk * n * NN;
                if (!next_bw) stage_noise<NN>(a, bw_i, i0 + chunk, min(chunk, a.inner_it - i0 - chunk), nxt, L.mt);
                else if (bw_i + 1 < a.bw_it) stage_noise<NN>(a, bw_i + 1, 0, chunk, nxt, L.mt);
                cp_commit();
                const int i1 = min(i0 + chunk, a.inner_it);
                for (int inner = i0; inner < i1; ++inner) {
                    const double *xr = xc + g * L.rs + 2 * t;
                    auto chain = [&](int h, double (&d)[2][2]) {   // 8-source tiles h, h + 4, ..
                        d[0][0] = d[0][1] = d[1][0] = d[1][1] = 0.0;
#pragma unroll
                        for (int c = h; c < KS; c += 4)
                            if (c < L.mt) {
                                const double2 b = *reinterpret_cast<const double2 *>(xr + 8 * c);
                                mma_f64(d[0], w[c][0], b.x);
                                mma_f64(d[1], w[c][1], b.y);
                            }
                    };
                    double in2[2], d0[2][2], d1[2][2];
                    {
                        double d2[2][2];
                        chain(0, d0);
                        chain(2, d2);
#pragma unroll
                        for (int e = 0; e < 2; ++e)
#pragma unroll
                            for (int u = 0; u < 2; ++u) d0[e][u] += d2[e][u];
                        chain(1, d1);
                        chain(3, d2);
#pragma unroll
                        for (int e = 0; e < 2; ++e)
#pragma unroll
                            for (int u = 0; u < 2; ++u) d0[e][u] += d1[e][u] + d2[e][u];
#pragma unroll
                        for (int u = 0; u < 2; ++u) in2[u] = d0[0][u] + d0[1][u];
                    }
                    const double *z = noise_s + ((size_t)(nbuf * chunk + inner - i0) * n + jn) * NN;
                    const double n0 = z[0], n1 = NN > 1 ? z[NN - 1] : 0.0;
#pragma unroll
                    for (int u = 0; u < 2; ++u) M::step(s[u], iv[u], gl[u], r[u], in2[u], n0, n1, a.K);
                    write_x(xn);
                    if (inner == i1 - 1) cp_wait_all();   // the next chunk's noise, before the barrier
                    bar_sync(1, node_threads);
                    double *sw = xc;
                    xc = xn;
                    xn = sw;
                }
                nbuf ^= 1;
            }
            // this millisecond's Balloon-Windkessel inputs; the barrier also waits for the last one's
            double *z = zs + (bw_i & 1) * items;
            if (act) {
                z[(2 * t) * n + j] = s[0][M::BOLDV];
                z[(2 * t + 1) * n + j] = s[1][M::BOLDV];
            }
            bar_sync(2, nthr);
            const bool tr = --to_tr == 0;
            if (bw_here) bw_items<BW_CALL>(a, td, bws, z, tid, nthr, tr, bold_i);
            if (tr) {
                to_tr = a.bold_tr_iters;
                ++bold_i;
            }
            if (--to_sample == 0) {
                to_sample = a.states_sampling_iters;
                if (a.ext_out) {
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                        if (act && sims[u] >= 0) states_out<M>(a, s[u], sims[u], j, states_i);
                    ++states_i;
                }
            }
        }
        if (a.ext_out && !a.states_ts)
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (act && sims[u] >= 0) states_mean<M>(a, sims[u], j, states_i);
        bar_sync(2, nthr);   // the tile's Balloon-Windkessel work is done with its inputs
    }
}

// CTAs an SM holds.
template <class K>
cudaError_t occupancy(K kernel, int threads, size_t smem, int *occ) {
    const cudaError_t e = allow_dynamic_smem(kernel);
    return e != cudaSuccess ? e : cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, kernel, threads, smem);
}
int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

// A kernel's instance for a run: launched over `items`, or with occ set, only asked for its occupancy.
template <class K>
cudaError_t use(K kernel, const IntegrateArgs &a, int items, int threads, size_t smem, cudaStream_t st, int *occ) {
    int fits = 0;
    const cudaError_t e = occupancy(kernel, threads, smem, &fits);
    if (e != cudaSuccess) return e;
    if (fits < 1) return cudaErrorInvalidConfiguration;
    if (occ) {
        *occ = fits;
        return cudaSuccess;
    }
    kernel<<<std::min(items, fits * sm_count()), threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <class M, int NC>
cudaError_t use_one(const IntegrateArgs &a, cudaStream_t st, int *occ) {
    const int chunk = std::min(a.inner_it, NOISE_CHUNK);
    const size_t smem = 8 * ((size_t)(192 + (one_par_smem(NC) ? 32 * (M::NR + M::NG) : 0)) * NC + (size_t)2 * chunk * a.nodes * M::NN);
    return use(k_one64<M, NC>, a, a.n_sims, ((a.nodes + 15) / 16) * 32, smem, st, occ);
}
template <class M, int KS>
cudaError_t use_tile(const IntegrateArgs &a, cudaStream_t st, int *occ) {
    const Layout L = layout(a.nodes, M::NN, std::min(a.inner_it, NOISE_CHUNK));
    return use(k_tile64<M, KS>, a, a.n_tiles, (L.mt + bw_warps(L.mt)) * 32, L.bytes, st, occ);
}

// Compiled extents; a run takes the least that holds its nodes.
template <class M>
cudaError_t use_model(const IntegrateArgs &a, bool tiles, cudaStream_t st, int *occ) {
    if (!tiles) {
        const int nc = (a.nodes + 31) / 32;
        if (nc <= 1) return use_one<M, 1>(a, st, occ);
        if (nc <= 2) return use_one<M, 2>(a, st, occ);
        if (nc <= 3) return use_one<M, 3>(a, st, occ);
        return use_one<M, 4>(a, st, occ);
    }
    const int mt = (a.nodes + 7) / 8;
    if (mt <= 4) return use_tile<M, 4>(a, st, occ);
    if (mt <= 8) return use_tile<M, 8>(a, st, occ);
    if (mt <= 11) return use_tile<M, 11>(a, st, occ);
    if (mt <= 13) return use_tile<M, 13>(a, st, occ);
    return use_tile<M, 16>(a, st, occ);
}

cudaError_t use_any(int model, const IntegrateArgs &a, bool tiles, cudaStream_t st, int *occ) {
    switch (model) {
        case MODEL_RWW: return use_model<RWWm<double>>(a, tiles, st, occ);
        case MODEL_WC: return use_model<WCm<double>>(a, tiles, st, occ);
        case MODEL_JR: return use_model<JRm<double>>(a, tiles, st, occ);
        case MODEL_RWWEX: return use_model<RWWExm<double>>(a, tiles, st, occ);
        default: break;
    }
    return cudaErrorNotSupported;
}

// Time of `items` CTAs of which an SM holds occ at once, in units of one alone on its SM;
// each further one on an SM adds `share` of that.
double waves(int items, int occ, double share) {
    const int sms = sm_count(), load = (items + sms - 1) / sms;   // CTAs of the fullest SM
    const int full = load / occ, rest = load % occ;
    return full * (1.0 + share * (occ - 1)) + (rest ? 1.0 + share * (rest - 1) : 0.0);
}

}  // namespace

// Whether n_tiles tiles of eight are faster than n_sims CTAs of one simulation: by the
// waves that either form takes on this GPU.  A tile's step takes n / 34 of a single
// simulation's, at least 1.25 (ms per simulated second alone on an SM, one / tile: rWW 32
// nodes 5.2 / 6.3, 64 nodes 5.5 / 9.8, 68 nodes 6.5 / 14.4, 100 nodes 7.5 / 22.6, 128 nodes
// 7.5 / 27.6; WC 100 nodes 7.0 / 22.6, JR 9.7 / 30.7, rWWEx 6.3 / 18.3), a second CTA on an
// SM costs a fifth more (rWW 68 nodes 6.5 -> 7.8).  So 444 simulations of 100 nodes on 148
// SMs take 22.6 ms in either form, 450 take 22.6 in tiles and 30.1 one by one, and 600 with
// an SC each (600 tiles of one live column) 113 in tiles and 37.7 one by one.
cudaError_t tile64_choose(int model, const IntegrateArgs &a, int n_tiles, bool *tiles) {
    int occ1 = 0, occ8 = 0;
    cudaError_t e = use_any(model, a, false, nullptr, &occ1);
    if (e == cudaSuccess) e = use_any(model, a, true, nullptr, &occ8);
    if (e != cudaSuccess) return e;
    *tiles = std::max(1.25, a.nodes / 34.0) * waves(n_tiles, occ8, 0.3) < waves(a.n_sims, occ1, 0.2);
    return cudaSuccess;
}

// Without delays and numerical FIC (whose restarts are per simulation), up to 128 nodes.
bool tile64_supported(int model, int nodes) {
    return nodes >= 1 && nodes <= 128 &&
           (model == MODEL_RWW || model == MODEL_WC || model == MODEL_JR || model == MODEL_RWWEX);
}

cudaError_t launch_integrate_tile64(int model, const IntegrateArgs &a, cudaStream_t st) {
    return use_any(model, a, a.tiles != nullptr, st, nullptr);
}

}  // namespace cbnm
