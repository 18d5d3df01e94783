// Integrator for conduction delays: one CTA per simulation, the time loop in
// blocks of 32 steps.
//
// The per-step form (integrate_sim.cuh; src/ext/bnm.cu:28-77) gathers, at every
// step and for every nonzero, one value x_k(t - d_kj) from a ring buffer ordered
// [slot][node]: each 4- or 8-byte value costs a 32-byte sector, and the 32 lanes of
// a warp touch 32 lines, so the load unit serves one value a cycle.  Here the ring
// buffer is [node][slot] and 32 steps are gathered at once, step t0 + b on lane b:
//
//  1. gather: the ring buffers of a tile of source nodes are copied to shared memory,
//     unrolled to the window [t0 - W, t0) (W = ring length), with the tile's entry
//     lists; a warp takes target node j and runs over the nonzeros of its SC column
//     within the tile; its 32 lanes read x_k(t0 + b - d), b = 0..31, 32 consecutive
//     words, and accumulate w x.  Pairs with d >= 32 ("far") need only values from
//     before t0; of the others ("near") the lanes b >= d read zeros behind the window.
//  2. steps: thread j integrates node j through the 32 steps with the sums of 1
//     in shared memory, adding the near pairs' terms with b >= d from the values
//     this block has already produced.  Those are read by other threads, so a
//     barrier (of the warps that hold nodes) is due every min(near d) steps; with no
//     near pair there is none.  The noise of the steps is copied to shared memory
//     beforehand, into the tile buffers, which are free now.
//     (Networks whose 32 sums per node leave little shared memory for tiles gather them in
//     two passes over the targets, the sums parked in global memory and brought back in
//     chunks with the noise: at 1,000 nodes tiles of 73 sources instead of 25.)
//  3. the block's 32 values per node go to the ring buffer, one line per node.
//
// What bounds it: step 1 is shared-memory bandwidth (one wavefront per entry and 32
// steps, half a wavefront for the entry itself), step 2 the latency of the update's
// dependency chain.  Gathering straight from global memory through L1 took 5.3 cycles
// an entry (the 128-byte window is unaligned: two lines, five sectors) against about
// 1.5 from shared memory.  A target's sum runs over its sources in ascending order, then
// over the near pairs whose value the block has produced, so that it depends neither on the
// tiles nor on what else is in the batch.
#pragma once
#include <algorithm>
#include "delay_plan.h"
#include "engine.h"
#include "integrate_sim.cuh"
#include "tc_common.cuh"

namespace cbnm {
namespace delayblk {

constexpr int DB = 32;            // steps per block = lanes
constexpr int NEAR_REGS = 4;      // near pairs of a node held in registers
constexpr int DROW = DB + 1;      // shared-memory row of a node: 32 sums, then its 32 new values in their place

template <class R>
struct Arr;
template <>
struct Arr<float> {
    __device__ static float *hist(const IntegrateArgs &a) { return a.hist_f32; }
    __device__ static float *sums(const IntegrateArgs &a) { return static_cast<float *>(a.db_sums); }
    __device__ static const float *near_w(const IntegrateArgs &a) { return a.db_near_w32; }
    __device__ static const ModelKf &consts(const IntegrateArgs &a) { return a.Kf; }
    __device__ static void pair(const float *w, unsigned p, float &w0, float &w1) {
        const float2 q = reinterpret_cast<const float2 *>(w)[p];
        w0 = q.x; w1 = q.y;
    }
    __device__ static float mad(float x, float y, float c) { return fmaf(x, y, c); }
};
template <>
struct Arr<double> {
    __device__ static double *hist(const IntegrateArgs &a) { return a.hist; }
    __device__ static double *sums(const IntegrateArgs &a) { return static_cast<double *>(a.db_sums); }
    __device__ static const double *near_w(const IntegrateArgs &a) { return a.db_near_w64; }
    __device__ static const ModelK &consts(const IntegrateArgs &a) { return a.K; }
    __device__ static void pair(const double *w, unsigned p, double &w0, double &w1) {
        const double2 q = reinterpret_cast<const double2 *>(w)[p];
        w0 = q.x; w1 = q.y;
    }
    __device__ static double mad(double x, double y, double c) { return fma(x, y, c); }
};

__device__ __forceinline__ void cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// B = 4, 8 or 16 bytes
template <int B>
__device__ __forceinline__ void cp_small(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_u32(dst)), "l"(src), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Copies tile `t` to buf: the entry lists (one 16-byte-aligned blob), then the window
// of each source, the ring rotated so that it ends at t0.
template <class R>
__device__ __forceinline__ void stage_tile(const IntegrateArgs &a, int pair, int pass, int t, const R *hist,
                                           unsigned char *buf, int t0m) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int *at = a.db_blob_at + ((size_t)pair * a.db_passes + pass) * (a.db_tiles + 1) + t;
    const int b0 = __ldg(at), b1 = __ldg(at + 1);   // in units of 16 bytes
    const int4 *src = reinterpret_cast<const int4 *>(a.db_blob) + b0;
    for (int i = threadIdx.x; i < b1 - b0; i += blockDim.x) cp16(buf + 16 * (size_t)i, src + i);
    R *win = reinterpret_cast<R *>(buf + a.db_blob_max);
    const int W = a.db_window, WS = W + DB, s0 = t * a.db_tile_src, cnt = min(a.db_tile_src, a.nodes - s0);
    constexpr int V = 16 / sizeof(R);
    for (int k = warp; k < cnt; k += nwarps) {
        const R *h = hist + (size_t)(s0 + k) * W;
        win[(size_t)k * WS + W + lane] = R(0);   // where the steps of a near pair read that the block has not done
        for (int c = lane * V; c < W; c += 32 * V) {
            int p = t0m + c;
            if (p >= W) p -= W;
            cp16(win + (size_t)k * WS + c, h + p);
        }
    }
}

// Copies the noise of `steps` steps from step t on to shared memory, [step][node][NN]:
// row (time shuffle, inner step), column = the repeat's node shuffle.  sh_ts is
// [repeats][noise_bw_it], one run of Balloon-Windkessel steps.
template <int NN, class R>
__device__ __noinline__ void stage_noise(const IntegrateArgs &a, const R *noise, int t, int steps, R *buf) {
    const int n = a.nodes, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int chunks = (n + 31) >> 5;   // (step, 32 nodes) pairs over the warps
    int q = warp / chunks, c = warp - q * chunks;
    const int dq = nwarps / chunks, dc = nwarps - dq * chunks;
#pragma unroll 2
    for (; q < steps;) {
        const int k = c * 32 + lane;
        if (k < n) {
            const int bw = (t + q) / a.inner_it, inner = (t + q) - bw * a.inner_it;
            const int shk = __ldg(a.sh_nodes + (size_t)(bw / a.noise_bw_it) * n + k);
            const R *src = noise + ((long long)__ldg(a.sh_ts + bw) * a.inner_it + inner) * n * NN;
            cp_small<NN * (int)sizeof(R)>(buf + ((size_t)q * n + k) * NN, src + (size_t)shk * NN);
        }
        q += dq;
        c += dc;
        if (c >= chunks) { c -= chunks; ++q; }
    }
}

// Step 1 of a block: the sums of targets [h0, h1) into row[target - h0][lane].  Out of line,
// so that the node state's registers are saved once per block instead of limiting this loop.
template <class R>
__device__ __noinline__ void gather_block(const IntegrateArgs &a, int pair, int pass, int h0, int h1, const R *hist,
                                          R *row, unsigned char *bufs, int t0m) {
    using A = Arr<R>;
    const int nh = h1 - h0, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int k0 = (int)((long long)nh * warp / nwarps), k1 = (int)((long long)nh * (warp + 1) / nwarps);
    const int tiles = a.db_tiles;
    const bool two = a.db_bufs == 2;
    stage_tile<R>(a, pair, pass, 0, hist, bufs, t0m);
    cp_commit();
    for (int t = 0; t < tiles; ++t) {
        unsigned char *buf = bufs + (two ? (t & 1) * (size_t)a.db_buf_bytes : 0);
        if (two && t + 1 < tiles) {
            stage_tile<R>(a, pair, pass, t + 1, hist, bufs + ((t + 1) & 1) * (size_t)a.db_buf_bytes, t0m);
            cp_commit();
            cp_wait<1>();
        } else {
            cp_wait<0>();
        }
        __syncthreads();
        const TileHead *head = reinterpret_cast<const TileHead *>(buf);
        const unsigned *rend = reinterpret_cast<const unsigned *>(buf + sizeof(TileHead));
        const unsigned *off = reinterpret_cast<const unsigned *>(buf + head->off_at);   // two 16-bit offsets a word
        const R *wgt = reinterpret_cast<const R *>(buf + head->w_at);
        const R *win = reinterpret_cast<const R *>(buf + a.db_blob_max) + lane;
        unsigned p = k0 > 0 ? rend[k0 - 1] : 0;   // in pairs of entries
        for (int k = k0; k < k1; ++k) {
            const unsigned pe = rend[k];
            if (t > 0 && p == pe) continue;
            R acc = t == 0 ? R(0) : row[k * DROW + lane];
#pragma unroll 4
            for (; p < pe; ++p) {
                const unsigned o = off[p];
                R w0, w1;
                A::pair(wgt, p, w0, w1);
                acc = A::mad(w0, win[o & 0xffff], acc);
                acc = A::mad(w1, win[o >> 16], acc);
            }
            row[k * DROW + lane] = acc;
        }
        __syncthreads();   // the buffer is free; after the last tile the sums are complete
        if (!two && t + 1 < tiles) {
            stage_tile<R>(a, pair, pass, t + 1, hist, bufs, t0m);
            cp_commit();
        }
    }
}

// States of node j at a sample: the time series, or the sum of the kept samples in the
// output itself (once per sample, so not held in registers).
template <int NS, class R>
__device__ __noinline__ void states_out(const IntegrateArgs &a, const R *s, int sim, int j, int states_i) {
    const int n = a.nodes;
    const size_t ext = a.states_ts ? (size_t)n * a.states_len : (size_t)n;
    for (int v = 0; v < NS; ++v) {
        double *out = a.states + ((size_t)v * a.n_sims + sim) * ext + j;
        if (a.states_ts) {
            if (states_i < a.states_len) out[(size_t)states_i * n] = (double)s[v];
        } else if (states_i == a.n_states_samples_remove) {
            *out = 0.0 + (double)s[v];
        } else if (states_i > a.n_states_samples_remove) {
            *out += (double)s[v];
        }
    }
}

// Registers: FP32 at 64 a thread (1,024 threads an SM); FP64 at 128 (512 threads an SM:
// at 80 the update spilled and two CTAs on an SM took as long as one after the other),
// but 64 for networks of more than 512 nodes.
template <class R, int MAXT>
constexpr int min_ctas() { return MAXT > 512 ? 1 : (sizeof(R) == 4 ? 1024 : 512) / MAXT; }

template <class M, class R, int MAXT>
__global__ void __launch_bounds__(MAXT, min_ctas<R, MAXT>()) k_integrate_delay(const __grid_constant__ IntegrateArgs a) {
    static_assert(!M::OSC, "the phase model's coupling depends on the target's current phase");
    using A = Arr<R>;
    using P = typename M::P;
    constexpr bool TWO = sizeof(R) == 4 && MAXT == 1024;   // two passes over the targets are possible
    const bool two = TWO && a.db_passes == 2;
    const int n = a.nodes;
    const int j = threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const bool act = j < n;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R *row = reinterpret_cast<R *>(smem_raw);   // [n][DROW]
    unsigned char *bufs = smem_raw + a.db_buf_at;
    // during the steps: noise of a chunk of them [step][n][NN], with two passes then their sums [step][n]
    R *const nzb = reinterpret_cast<R *>(smem_raw + a.db_noise_at);
    const R *nz = nzb + (size_t)j * M::NN;
    const int ns = (n + 3) & ~3;   // row of sums
    R *const sum_s = nzb + (((size_t)a.db_noise_steps * n * M::NN + 3) & ~(size_t)3);
    R *const sums = two ? A::sums(a) + (size_t)blockIdx.x * DB * ns : nullptr;
    const int node_threads = (n + 31) & ~31;
    __shared__ int s_trial, s_adjust, s_failed;
    const int W = a.db_window;
    R *const hist = A::hist(a) + (size_t)blockIdx.x * ((size_t)n * W);
    const R *const noise = SimArrays<R>::noise(a);
    const size_t rstride = (size_t)a.n_sims * n;
    const size_t ext = a.states_ts ? (size_t)n * a.states_len : (size_t)n;
    const int total = a.bw_it * a.inner_it;

    for (int i = blockIdx.x; i < a.sim_list_n; i += gridDim.x) {
        const int sim = a.sim_list[i];
        const int pair = a.db_pair[sim];                       // (SC, delay table) of this simulation
        const int *const near_off = a.db_near + (size_t)pair * a.db_near_k * n;   // k * 32 + d, padding 0 (d = 0)
        const R *const near_w = A::near_w(a) + (size_t)pair * a.db_near_k * n;
        const int near_n = a.db_near_cnt[pair];               // longest near list
        const int sync_every = near_n ? a.db_near_min[pair] : DB;
        int no[NEAR_REGS];   // this node's first near pairs
        R nw[NEAR_REGS];
#pragma unroll
        for (int q = 0; q < NEAR_REGS; ++q) {
            const bool has = act && q < near_n;
            no[q] = has ? __ldg(near_off + (size_t)q * n + j) : 0;
            nw[q] = has ? __ldg(near_w + (size_t)q * n + j) : R(0);
        }
        R g[M::NG], iv[M::NI];
        P r[M::NR];
        R s[M::NS];
#pragma unroll
        for (int i = 0; i < M::NG; ++i) g[i] = (R)a.gparams[(size_t)i * a.n_sims + sim];
#pragma unroll
        for (int i = 0; i < M::NR; ++i) r[i] = act ? (P)a.rparams[i * rstride + (size_t)sim * n + j] : P(0);
#pragma unroll
        for (int i = 0; i < M::NI; ++i) iv[i] = R(0);
#pragma unroll
        for (int i = 0; i < M::NS; ++i) s[i] = R(0);
        M::init(s, iv, g, r);
        double fic_sum = 0.0, fic_delta = a.init_delta;   // numerical FIC (rww.cpp:233-298)
        if (j == 0) { s_trial = 0; s_adjust = (a.do_fic && a.max_fic_trials > 0) ? 1 : 0; s_failed = 0; }
        double bx = 0.0, bf = 1.0, bnu = 1.0, bq = 1.0;
        double *const bold = a.bold + (size_t)sim * a.bold_len * n;
        int bw_i = 0, inner = 0, bold_i = 0, states_i = 0;   // inner: steps done of Balloon-Windkessel step bw_i
        int t0 = 0, t0m = 0;   // first step of the block, and its slot
        bool fill = true;   // the ring buffer holds the initial state (start and FIC restarts)
        while (t0 < total) {
            if (fill) {
                __syncthreads();  // the previous simulation's or trial's reads are done
                if (act) row[j * DROW] = s[M::CONN];
                __syncthreads();
                for (int k = warp; k < n; k += nwarps) {
                    const R v = row[k * DROW];
                    for (int p = lane; p < W; p += 32) hist[(size_t)k * W + p] = v;
                }
                fill = false;
                __syncthreads();
            }
            // ---- 1. gather, lane = step of the block
            if (!two) {
                gather_block<R>(a, pair, 0, 0, n, hist, row, bufs, t0m);
            } else {   // half of the targets at a time; their sums wait in global memory, [step][node]
                const int nh = (n + 1) / 2;
                for (int h = 0; h < 2; ++h) {
                    const int h0 = h * nh, h1 = min(n, h0 + nh);
                    gather_block<R>(a, pair, h, h0, h1, hist, row, bufs, t0m);
                    for (int b = warp; b < DB; b += nwarps)
                        for (int k = h0 + lane; k < h1; k += 32) sums[(size_t)b * ns + k] = row[(k - h0) * DROW + b];
                    __syncthreads();
                }
            }
            // ---- 2. the block's steps, thread = node, in chunks of the noise that the buffers hold
            const int nb = min(DB, total - t0);
            bool restart = false;
            int next_sync = sync_every;
            for (int b = 0; b < nb;) {
                if (b % a.db_noise_steps == 0) {
                    if (b) __syncthreads();   // the previous chunk is used
                    const int cnt = min(a.db_noise_steps, nb - b);
                    stage_noise<M::NN, R>(a, noise, t0 + b, cnt, nzb);
                    if (two)
                        for (int i = threadIdx.x * 4; i < cnt * ns; i += blockDim.x * 4)
                            cp16(sum_s + i, sums + (size_t)b * ns + i);
                    cp_commit();
                    cp_wait<0>();
                    __syncthreads();
                }
                const int chunk = b - b % a.db_noise_steps;
                const int e = min(min(nb, chunk + a.db_noise_steps), b + a.inner_it - inner);
                inner += e - b;
                if (j < node_threads) {
                    for (; b < e; ++b) {
                        if (b == next_sync) {   // near pairs read values of up to sync_every steps ago
                            asm volatile("bar.sync 1, %0;" ::"r"(node_threads) : "memory");
                            next_sync += sync_every;
                        }
                        if (!act) continue;
                        R in = two ? sum_s[(b - chunk) * ns + j] : row[j * DROW + b];
                        const R *z = nz + (size_t)(b - chunk) * n * M::NN;
                        const R n0 = z[0], n1 = M::NN > 1 ? z[1] : R(0);
                        if (near_n) {  // d = 0: the padding of shorter lists
                            R xq[NEAR_REGS];
#pragma unroll
                            for (int q = 0; q < NEAR_REGS; ++q) {
                                const int d = no[q] & (DB - 1);
                                xq[q] = R(0);
                                if (d != 0 && b >= d) xq[q] = row[(no[q] >> 5) * DROW + b - d];
                            }
#pragma unroll
                            for (int q = 0; q < NEAR_REGS; ++q) in = A::mad(nw[q], xq[q], in);
                            for (int q = NEAR_REGS; q < near_n; ++q) {
                                const int o = __ldg(near_off + (size_t)q * n + j);
                                const int d = o & (DB - 1);
                                if (d != 0 && b >= d)
                                    in = A::mad(__ldg(near_w + (size_t)q * n + j), row[(o >> 5) * DROW + b - d], in);
                            }
                        }
                        M::step(s, iv, g, r, in, n0, n1, A::consts(a));
                        row[j * DROW + b] = s[M::CONN];
                    }
                }
                b = e;
                if (inner < a.inner_it) continue;
                // ---- end of a Balloon-Windkessel step
                inner = 0;
                const int now = bw_i;
                if (act) bw_step64(bx, bf, bnu, bq, (double)s[M::BOLDV], a.bwf);
                if ((now + 1) % a.bold_tr_iters == 0) {  // bnm.cpp:316-335; no slot for a sample past bold_len
                    if (act && bold_i < a.bold_len)
                        bold[(size_t)bold_i * n + j] =
                            a.bw.V_0 * (a.bw.k1 * (1 - bq) + a.bw.k2 * (1 - bq / bnu) + a.bw.k3 * (1 - bnu));
                    bold_i++;
                }
                if (a.ext_out && (now + 1) % a.states_sampling_iters == 0) {  // bnm.cpp:337-355
                    if (act) {
                        R out[M::NS];   // a copy: s itself must not have its address taken
#pragma unroll
                        for (int v = 0; v < M::NS; ++v) out[v] = s[v];
                        states_out<M::NS, R>(a, out, sim, j, states_i);
                    }
                    states_i++;
                }
                if constexpr (M::POSTBW) {  // numerical FIC, rww.cpp:233-298
                    const int t = now + 1;
                    if (a.do_fic && a.max_fic_trials > 0 && t <= a.I_end && s_adjust) {  // block-uniform
                        if (act && t >= a.I_start) fic_sum += (double)s[0];
                        if (t == a.I_end) {
                            const int trial = s_trial;
                            int need = 0;
                            if (act) {
                                fic_sum /= a.I_dur;
                                const double diff = fic_sum - a.K.rww.b_a_ratio_E;
                                if (fabs(diff + 0.026) > 0.005) {
                                    need = 1;
                                    if (trial < a.max_fic_trials) {
                                        if (diff < -0.026) {
                                            r[2] = (P)((double)r[2] - fic_delta);
                                            fic_delta -= 0.001;
                                            fic_delta = fmax(fic_delta, 0.001);
                                        } else {
                                            r[2] = (P)((double)r[2] + fic_delta);
                                        }
                                    }
                                }
                            }
                            const int any = __syncthreads_or(need);
                            if (any) {
                                if (trial < a.max_fic_trials) {
                                    restart = true;
                                    if (j == 0) s_trial = trial + 1;
                                } else if (j == 0) {
                                    s_adjust = 0;
                                    s_failed = 1;
                                }
                            } else if (j == 0) {
                                s_adjust = 0;
                            }
                            __syncthreads();
                        }
                    }
                }
                bw_i++;
                if (restart) break;
            }
            if (restart) {  // bnm.cpp:386-434
                if (act) M::restart(s, iv, r);
                fic_sum = 0.0;
                bx = 0.0; bf = 1.0; bnu = 1.0; bq = 1.0;
                bold_i = 0; states_i = 0; bw_i = 0; inner = 0;
                t0 = 0;
                t0m = 0;
                fill = true;
                continue;
            }
            t0 += DB;
            if (t0 >= total) break;
            __syncthreads();
            // ---- 3. the block's values into the ring buffer
            for (int k = warp; k < n; k += nwarps)
                hist[(size_t)k * W + t0m + lane] = row[k * DROW + lane];
            t0m = t0m + DB == W ? 0 : t0m + DB;
            __syncthreads();
        }
        if constexpr (M::POSTBW) {
            if (a.do_fic) {  // rww.cpp:300-314 post_integration
                if (act) a.rparams_out[2 * rstride + (size_t)sim * n + j] = (double)r[2];
                if (j == 0) {
                    a.gints[sim] = s_trial;
                    a.gbools[(size_t)a.n_sims + sim] = (unsigned char)s_failed;
                }
            }
        }
        if (act && a.ext_out && !a.states_ts) {
            const int pts = states_i - a.n_states_samples_remove;
#pragma unroll
            for (int v = 0; v < M::NS; ++v) {   // no kept sample: 0 / pts
                double &out = a.states[((size_t)v * a.n_sims + sim) * ext + j];
                out = (pts > 0 ? out : 0.0) / pts;
            }
        }
        __syncthreads();  // the next simulation resets the shared words
    }
}

// CTAs an SM holds of a launch shape (threads and shared memory chosen by the host).
template <class M, class R, int MAXT>
cudaError_t occupancy(const DelayLaunch &c, int *occ) {
    cudaError_t e = allow_dynamic_smem(k_integrate_delay<M, R, MAXT>);
    return e != cudaSuccess
               ? e
               : cudaOccupancyMaxActiveBlocksPerMultiprocessor(occ, k_integrate_delay<M, R, MAXT>, c.threads, c.smem);
}

template <class M, class R>
cudaError_t config_model(const IntegrateArgs &a, int sms, DelayLaunch *c) {
    // the two-pass form is compiled for the FP32 kernel of more than 512 threads only
    if (a.db_passes != 1 && (sizeof(R) != 4 || c->threads <= 512)) return cudaErrorInvalidValue;
    int occ = 0;
    const cudaError_t e = c->threads <= 256   ? occupancy<M, R, 256>(*c, &occ)
                          : c->threads <= 512 ? occupancy<M, R, 512>(*c, &occ)
                                              : occupancy<M, R, 1024>(*c, &occ);
    if (e != cudaSuccess) return e;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    c->grid = std::min(a.sim_list_n, occ * sms);
    return cudaSuccess;
}

template <class M, class R>
cudaError_t launch_model(const IntegrateArgs &a, const DelayLaunch &c, cudaStream_t st) {
    if (c.threads <= 256) k_integrate_delay<M, R, 256><<<c.grid, c.threads, c.smem, st>>>(a);
    else if (c.threads <= 512) k_integrate_delay<M, R, 512><<<c.grid, c.threads, c.smem, st>>>(a);
    else k_integrate_delay<M, R, 1024><<<c.grid, c.threads, c.smem, st>>>(a);
    return cudaGetLastError();
}

template <class R>
cudaError_t config(int model, const IntegrateArgs &a, int sms, DelayLaunch *c) {
    switch (model) {
        case MODEL_RWW: return config_model<RWWm<R>, R>(a, sms, c);
        case MODEL_WC: return config_model<WCm<R>, R>(a, sms, c);
        case MODEL_JR: return config_model<JRm<R>, R>(a, sms, c);
        case MODEL_RWWEX: return config_model<RWWExm<R>, R>(a, sms, c);
    }
    return cudaErrorInvalidValue;
}

template <class R>
cudaError_t launch(int model, const IntegrateArgs &a, const DelayLaunch &c, cudaStream_t st) {
    switch (model) {
        case MODEL_RWW: return launch_model<RWWm<R>, R>(a, c, st);
        case MODEL_WC: return launch_model<WCm<R>, R>(a, c, st);
        case MODEL_JR: return launch_model<JRm<R>, R>(a, c, st);
        case MODEL_RWWEX: return launch_model<RWWExm<R>, R>(a, c, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace delayblk
}  // namespace cbnm
