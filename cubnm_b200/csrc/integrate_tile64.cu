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
//  * k_one64, batches of up to four simulations per SM: one CTA per simulation.  The n x n
//    product with x is spread over 4 lanes per node: a group of 16 lanes holds four rows
//    of SC^T, each lane the sources k = lane mod 16, in registers; partial sums meet in a
//    transposing butterfly (5 shuffles) and the update runs on one thread per node.  Bound
//    by latency: product, two barriers, update chain.
//  * k_tile64, larger batches: eight simulations sharing an SC per CTA, the product as
//    mma.sync m8n8k4 (FP64), SC^T fragments in registers, so that a weight read serves
//    eight simulations and the sums need no shuffles.  DMMA runs at the FP64 pipe's rate
//    on sm_100a (measured 63.7 multiply-adds a cycle and SM for both), so this saves
//    loads and latency, not FP64 work: bound by the FP64 pipe (product 169 cycles per
//    simulation and step at 100 nodes, update about 180).  The Balloon-Windkessel model
//    of a tile runs in up to four more warps, a millisecond behind.
//
// Noise rows are copied to shared memory a chunk of steps ahead.  The sums are formed in
// another order than the reference's, with fused multiply-adds.
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

__device__ __forceinline__ double bold_of(const IntegrateArgs &a, double q, double nu) {  // bnm.cpp:316-335
    return a.bw.V_0 * (a.bw.k1 * (1 - q) + a.bw.k2 * (1 - q / nu) + a.bw.k3 * (1 - nu));
}

// ---------------------------------------------------------------- one simulation per CTA
// KPL: compiled sources per lane (16 KPL >= n).
template <class M, int KPL>
__global__ void __launch_bounds__(KPL * 64) k_one64(const __grid_constant__ IntegrateArgs a) {
    constexpr int NN = M::NN;
    extern __shared__ __align__(16) double sh[];
    const int n = a.nodes, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, l = lane & 15, nwarps = blockDim.x >> 5;
    const int chunk = min(a.inner_it, NOISE_CHUNK);
    double *x = sh, *in_s = x + 16 * KPL, *noise_s = in_s + 16 * KPL;   // [16 KPL], [16 KPL], [2][chunk][n][NN]
    const int row0 = warp * 8 + (lane >> 4) * 4;                        // the four rows of this half-warp
    const int my_row = row0 + (l >> 3) * 2 + ((l >> 2) & 1);            // the row whose sum this lane ends with
    const int j = tid;
    const bool act = j < n;
    for (int sim = blockIdx.x; sim < a.n_sims; sim += gridDim.x) {
        const double *SC = a.sc + (size_t)a.sc_idx[sim] * n * n;
        double w[4][KPL];
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int i = 0; i < KPL; ++i) {
                const int k = l + 16 * i;
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
        double bx = 0.0, bf = 1.0, bnu = 1.0, bq = 1.0;
        double *bold = a.bold + (size_t)sim * a.bold_len * n;
        if (tid < 16 * KPL) x[tid] = act ? s[M::CONN] : 0.0;
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
                    for (int i = 0; i < KPL; ++i) {
                        const double xk = x[l + 16 * i];
#pragma unroll
                        for (int q = 0; q < 4; ++q) v[q] = fma(w[q][i], xk, v[q]);
                    }
                    // transposing butterfly: lanes keep rows {0,1} / {2,3}, then one row, then its sum
                    const bool up = l & 8, odd = l & 4;
                    double s0 = up ? v[0] : v[2], s1 = up ? v[1] : v[3];
                    double m0 = up ? v[2] : v[0], m1 = up ? v[3] : v[1];
                    m0 += __shfl_xor_sync(0xffffffffu, s0, 8);
                    m1 += __shfl_xor_sync(0xffffffffu, s1, 8);
                    s0 = odd ? m0 : m1;
                    m0 = odd ? m1 : m0;
                    m0 += __shfl_xor_sync(0xffffffffu, s0, 4);
                    m0 += __shfl_xor_sync(0xffffffffu, m0, 2);
                    m0 += __shfl_xor_sync(0xffffffffu, m0, 1);
                    if ((l & 3) == 0) in_s[my_row] = m0;
                    __syncthreads();
                    if (act) {
                        const double *z = noise_s + ((size_t)(nbuf * chunk + inner - i0) * n + j) * NN;
                        M::step(s, iv, g, r, in_s[j], z[0], NN > 1 ? z[NN - 1] : 0.0, a.K);
                        x[j] = s[M::CONN];
                    }
                    if (inner == i1 - 1) cp_wait_all();   // the next chunk's noise, before the barrier
                    __syncthreads();
                }
                nbuf ^= 1;
            }
            if (act) bw_step64(bx, bf, bnu, bq, s[M::BOLDV], a.bwf);
            if (--to_tr == 0) {
                to_tr = a.bold_tr_iters;
                if (act && bold_i < a.bold_len) bold[(size_t)bold_i * n + j] = bold_of(a, bq, bnu);
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
        bw_step64_n<2>(x, f, nu, q, zz, a.bwf);
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
            bw_items(a, td, b, zs + (bw_i & 1) * items, tid, nthr, tr, bold_i);
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
        bw_role(a, bws, zs, tid - node_threads, nthr - node_threads);
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
                    double d[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
                    const double *xr = xc + g * L.rs + 2 * t;
#pragma unroll
                    for (int c = 0; c < KS; ++c) {
                        if (c < L.mt) {
                            const double2 b = *reinterpret_cast<const double2 *>(xr + 8 * c);
                            mma_f64(d[0], w[c][0], b.x);
                            mma_f64(d[1], w[c][1], b.y);
                        }
                    }
                    const double *z = noise_s + ((size_t)(nbuf * chunk + inner - i0) * n + jn) * NN;
                    const double n0 = z[0], n1 = NN > 1 ? z[NN - 1] : 0.0;
#pragma unroll
                    for (int u = 0; u < 2; ++u) M::step(s[u], iv[u], gl[u], r[u], d[0][u] + d[1][u], n0, n1, a.K);
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
            if (bw_here) bw_items(a, td, bws, z, tid, nthr, tr, bold_i);
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

template <class K>
cudaError_t launch(K kernel, const IntegrateArgs &a, int items, int threads, size_t smem, cudaStream_t st) {
    cudaError_t e = allow_dynamic_smem(kernel);
    int dev = 0, sms = 0, occ = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, threads, smem);
    if (e != cudaSuccess) return e;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    kernel<<<std::min(items, occ * sms), threads, smem, st>>>(a);
    return cudaGetLastError();
}

template <class M, int KPL>
cudaError_t launch_one(const IntegrateArgs &a, cudaStream_t st) {
    const int chunk = std::min(a.inner_it, NOISE_CHUNK);
    const size_t smem = 8 * ((size_t)32 * KPL + (size_t)2 * chunk * a.nodes * M::NN);
    return launch(k_one64<M, KPL>, a, a.n_sims, ((a.nodes + 7) / 8) * 32, smem, st);
}
template <class M, int KS>
cudaError_t launch_tile(const IntegrateArgs &a, cudaStream_t st) {
    const Layout L = layout(a.nodes, M::NN, std::min(a.inner_it, NOISE_CHUNK));
    return launch(k_tile64<M, KS>, a, a.n_tiles, (L.mt + bw_warps(L.mt)) * 32, L.bytes, st);
}

// Compiled extents; a run takes the least that holds its nodes.
template <class M>
cudaError_t launch_model(const IntegrateArgs &a, cudaStream_t st) {
    if (!a.tiles) {
        const int kpl = (a.nodes + 15) / 16;
        if (kpl <= 2) return launch_one<M, 2>(a, st);
        if (kpl <= 4) return launch_one<M, 4>(a, st);
        if (kpl <= 5) return launch_one<M, 5>(a, st);
        if (kpl <= 7) return launch_one<M, 7>(a, st);
        return launch_one<M, 8>(a, st);
    }
    const int mt = (a.nodes + 7) / 8;
    if (mt <= 4) return launch_tile<M, 4>(a, st);
    if (mt <= 8) return launch_tile<M, 8>(a, st);
    if (mt <= 11) return launch_tile<M, 11>(a, st);
    if (mt <= 13) return launch_tile<M, 13>(a, st);
    return launch_tile<M, 16>(a, st);
}

}  // namespace

// Without delays and numerical FIC (whose restarts are per simulation), up to 128 nodes.
bool tile64_supported(int model, int nodes) {
    return nodes >= 1 && nodes <= 128 &&
           (model == MODEL_RWW || model == MODEL_WC || model == MODEL_JR || model == MODEL_RWWEX);
}

cudaError_t launch_integrate_tile64(int model, const IntegrateArgs &a, cudaStream_t st) {
    switch (model) {
        case MODEL_RWW: return launch_model<RWWm<double>>(a, st);
        case MODEL_WC: return launch_model<WCm<double>>(a, st);
        case MODEL_JR: return launch_model<JRm<double>>(a, st);
        case MODEL_RWWEX: return launch_model<RWWExm<double>>(a, st);
        default: break;
    }
    return cudaErrorNotSupported;
}

}  // namespace cbnm
