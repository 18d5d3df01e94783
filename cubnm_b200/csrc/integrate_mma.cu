// FP32 integrator for shared-SC batches without delays: eight simulations per CTA,
// the coupling as warp-level matrix products with the SC held in registers.
//
// The time loop is the reference's (src/ext/bnm.cu:117-505).  Per 0.1-ms step the
// coupling of a tile (bnm.cu:48-77) is the small product D[j][s] = sum_k SC[k][j] x_k^s,
// n x n by n x 8, whose input is the step before: its latency, not its throughput, is
// on the critical path.  The tcgen05 form of it (32 simulations per CTA, operands
// through shared memory and tensor memory, one barrier pair and one MMA commit a step)
// took 5,237 cycles a step of 32 simulations at 100 nodes: about 1,460 for the 21 MMAs,
// the update after them, 52 % issue, and a batch below 32 x 148 simulations left SMs
// idle.  Here:
//
//  * warp m owns target nodes 16 m .. 16 m + 15 and keeps its rows of SC^T as mma.sync
//    m16n8k16 A fragments in registers for the whole run (FP16 hi and lo; for more than
//    96 nodes lo in shared memory); a step loads the eight simulations' x as B
//    fragments (one 16-byte load per 16 sources brings hi and lo) and issues the
//    products hi hi, hi lo, lo hi.  FP16, with each row of SC^T scaled by a power of two
//    and lo by 2^11, holds 22 bits (x is at most 1 in all four models).  The tensor pipe
//    truncates where it accumulates: hi hi products chained over the K steps gave three
//    times the error in BOLD, so the FP32 pipe adds them, and above 128 nodes the mean of
//    what is lost within one product is added back (HH_BIAS).  Errors against FP64 beside
//    launch_integrate_mma; 100-node rWW 3.3e-8 relative in BOLD, 1.1e-7 in BF16 halves (the
//    tcgen05 form);
//  * the accumulator layout is the update's layout: lane (g, t) holds nodes g, g + 8 of
//    the warp and simulations 2t, 2t + 1, state and parameters in registers, stepped as
//    pairs in packed FP32x2.  K is ordered so that the two nodes of a lane are adjacent
//    in the next product's B operand: a lane writes hi and lo of both in 8 bytes;
//  * x is double-buffered, so a step has one barrier; several CTAs share an SM and run
//    out of step, one's product under another's update;
//  * noise rows (shared by all simulations) are copied to shared memory a chunk of steps
//    ahead;
//  * one to four more warps integrate the FP64 Balloon-Windkessel model of the tile, a
//    millisecond behind, from the inputs left in shared memory (state there too).  Inside
//    the node warps its chain of some 300 cycles and its registers cost 545 of 2,240
//    cycles a step.
//
// mma.sync reaches a quarter of tcgen05's rate on sm_100a (measured 950 FP16 multiply-
// adds a cycle and SM), but a tile's 147 products at 100 nodes are 316 cycles of it, in
// the shadow of the other CTA's update.  Measured at 100 nodes: 1,500 cycles a step with
// one CTA an SM (8 simulations), 2,290 with two (200 nodes, one: 3,930).  What bounds a step then: the phases of a
// CTA's warps (product, MUFU, update) follow one another between its barriers, with two
// CTAs to overlap; more do not fit the registers.
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <cstring>
#include <cuda_fp16.h>
#include <type_traits>
#include "engine.h"
#include "tc_common.cuh"

namespace cbnm {
namespace {

constexpr int TS = 8;            // simulations per tile (MMA N)
constexpr int NOISE_CHUNK = 10;  // steps of noise per shared-memory buffer (two buffers)

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint4 &a, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// v = hi + lo / LO_SCALE to 22 bits for 2^-14 <= |v| < 2^15, to 2^-36 below.
constexpr float LO_SCALE = 2048.0f;
// Share of the hi hi sums added back above 128 nodes and for rWWEx above 80, 2^-25: the tensor pipe drops what is
// below the last place of the largest of its 16 products, on average half a unit of that
// place a product, always towards zero (mean of the relative error of sums of 16 positive
// products, x in [0.05, 0.95]: -4.0e-8 with all weights nonzero, -1.5e-8 with a quarter of
// them; 2^-25 is 2.98e-8).
constexpr float HH_BIAS = 2.98023224e-8f;
__device__ __forceinline__ void split_f16x2(float2 v, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __float22half2_rn(v);
    const float2 hf = __half22float2(h);
    const __half2 l = __float22half2_rn(__ffma2_rn(hf, make_float2(-LO_SCALE, -LO_SCALE),
                                                   make_float2(v.x * LO_SCALE, v.y * LO_SCALE)));
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}
// The same from zero: the tensor pipe truncates as it accumulates, so that sums of many
// K steps drift; the hi hi products, which carry it, are added by the FP32 pipe instead.
__device__ __forceinline__ void mma_f16_add(float2 (&d)[2], const uint4 &a, uint32_t b0, uint32_t b1) {
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    mma_f16(c, a, b0, b1);
    d[0] = __fadd2_rn(d[0], make_float2(c[0], c[1]));
    d[1] = __fadd2_rn(d[1], make_float2(c[2], c[3]));
}
template <int B>
__device__ __forceinline__ void cp_small(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_u32(dst)), "l"(src), "n"(B) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// rWWEx with the FP32 update of the per-simulation kernels (models.cuh, rwwex.cpp:48-73),
// a pair of simulations at a time.
struct RWWExs32 {
    using K = ModelKf;
    static constexpr bool PAIR = true, ACC = true;
    static constexpr int NP = 4, NS = 1, NN = 1, NOUT = 3, CV = 0, BV = 0;
    __device__ static void params(float *p, double G, const double *r, const K &k) {   // w J_N, G J_N, I_0, sigma
        p[0] = (float)r[0] * k.rwwex.J_N; p[1] = (float)G * k.rwwex.J_N; p[2] = (float)r[1]; p[3] = (float)r[2];
    }
    __device__ static void pair_params(float2 *) {}
    __device__ static void init(float *s) { s[0] = 0.001f; }
    __device__ static void step2(float2 *s, const float2 *p, float2 in, float n0, float, const K &k, float2 *o) {
        const RWWExKt<float> &m = k.rwwex;
        const float2 x = __fadd2_rn(__ffma2_rn(p[1], in, __fmul2_rn(p[0], s[0])), p[2]);
        const float2 r = rate2_acc(__ffma2_rn(f2(m.a), x, f2(-m.b)), m.d, 1.0f / m.d);
        float2 ds = __fmul2_rn(f2(m.dt_gamma), __fmul2_rn(__ffma2_rn(s[0], f2(-1.0f), f2(1.0f)), r));
        ds = __ffma2_rn(f2(-m.dt_itau), s[0], ds);
        ds = __ffma2_rn(f2(n0 * m.sqrt_dt), p[3], ds);
        const float2 n = __fadd2_rn(s[0], ds);
        s[0] = make_float2(__saturatef(n.x), __saturatef(n.y));
        o[0] = x; o[1] = r; o[2] = s[0];
    }
};
template <class M>
__device__ __forceinline__ const typename M::K &model_consts(const IntegrateArgs &a) {
    if constexpr (std::is_same<typename M::K, ModelKf>::value) return a.Kf;
    else return *reinterpret_cast<const typename M::K *>(a.k32);
}

// Shared-memory layout, from the node count and the model's noise terms.
struct Layout {
    int mt, ps;                   // 16-node tiles (= node warps); words per simulation pair of x
    int x, noise, bw, z, alo, bytes;   // byte offsets: x [2][4][ps], noise [2][chunk][n][NN],
                                       // Balloon-Windkessel [4][8 n] and inputs [2][8 n], A lo
};
__host__ __device__ inline Layout layout(int n, int nn, int chunk, int ks, bool lo_smem) {
    Layout l;
    l.mt = (n + 15) / 16;
    l.ps = ks * 32 + 16;          // 16 mod 32: the four pairs of a store hit two bank halves
    l.x = 0;
    l.noise = l.x + 2 * 4 * l.ps * 4;
    l.bw = (l.noise + 2 * chunk * n * nn * 4 + 15) & ~15;
    l.z = l.bw + 4 * TS * n * 8;
    l.alo = (l.z + 2 * TS * n * 4 + 15) & ~15;
    l.bytes = l.alo + (lo_smem ? l.mt * ks * 32 * 16 : 0);
    return l;
}

__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__host__ __device__ constexpr bool lo_in_smem(int ks) { return ks > 6; }   // A lo

// Balloon-Windkessel warps beside `mt` node warps: up to a multiple of four (a warp's
// registers come from its quarter of the SM), at least one.
__host__ __device__ constexpr int bw_warps(int mt) { return mt % 4 ? 4 - mt % 4 : mt <= 4 ? 4 : 2; }
// CTAs an SM should hold: about 128 registers a thread, fewer for 8 node warps.
__host__ __device__ constexpr int min_ctas(int ks) { return ks <= 8 ? 2 : 1; }

// The Balloon-Windkessel warps: for every tile and millisecond, wait for the inputs of the
// 8 n items (item s n + j), step them two at a time, write BOLD at TR.
__device__ __forceinline__ void bw_role(const IntegrateArgs &a, double *b, const float *zs, int tid, int nthr) {
    const int n = a.nodes, items = TS * n;
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
            const float *zb = zs + (bw_i & 1) * items;
            for (int i0 = tid; i0 < items; i0 += 2 * nthr) {
                int at[2] = {i0, i0 + nthr < items ? i0 + nthr : i0};   // the last one may be alone: computed twice
                double x[2], f[2], nu[2], q[2], z[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    x[u] = b[at[u]]; f[u] = b[items + at[u]]; nu[u] = b[2 * items + at[u]]; q[u] = b[3 * items + at[u]];
                    z[u] = (double)zb[at[u]];
                }
                bw_step64_n<2>(x, f, nu, q, z, a.bwf);
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    b[at[u]] = x[u]; b[items + at[u]] = f[u]; b[2 * items + at[u]] = nu[u]; b[3 * items + at[u]] = q[u];
                    if (tr && bold_i < a.bold_len) {   // a sample past bold_len has no slot
                        const int s = at[u] / n, j = at[u] - s * n, sim = td[1 + s];
                        if (sim >= 0)
                            a.bold[(size_t)sim * a.bold_len * n + (size_t)bold_i * n + j] = bold64(q[u], nu[u], a.bwf);
                    }
                }
            }
            if (tr) {
                to_tr = a.bold_tr_iters;
                ++bold_i;
            }
        }
        bar_sync(2, blockDim.x);
    }
}

// KS: compiled count of 16-node tiles (K steps), at least the run's.
template <class M, int KS>
__global__ void __launch_bounds__((KS + bw_warps(KS)) * 32, min_ctas(KS)) k_integrate_mma(const __grid_constant__ IntegrateArgs a) {
    constexpr bool LO_SMEM = lo_in_smem(KS);
    constexpr int NN = M::NN;
    using Step = PairStep<M>;
    extern __shared__ __align__(16) unsigned char smem[];
    const int n = a.nodes, tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int chunk = min(a.inner_it, NOISE_CHUNK);
    const Layout L = layout(n, NN, chunk, KS, LO_SMEM);
    const int ps = L.ps;
    uint32_t *xb = reinterpret_cast<uint32_t *>(smem + L.x);
    float *noise_s = reinterpret_cast<float *>(smem + L.noise);
    double *bws = reinterpret_cast<double *>(smem + L.bw);
    float *zs = reinterpret_cast<float *>(smem + L.z);
    const int items = TS * n, node_threads = L.mt * 32;
    uint4 *alo_s = reinterpret_cast<uint4 *>(smem + L.alo) + (size_t)warp * KS * 32 + lane;
    const typename M::K &K = model_consts<M>(a);
    const size_t rstride = (size_t)a.n_sims * n;
    const size_t ext = a.states_ts ? (size_t)n * a.states_len : (size_t)n;
    const int node[2] = {warp * 16 + g, warp * 16 + g + 8};
    const bool act[2] = {node[0] < n, node[1] < n};
    const int nzoff[2] = {act[0] ? node[0] * NN : 0, act[1] ? node[1] * NN : 0};
    // this lane's words of x: writes (hi, lo) of its two nodes for simulation 2t (+16 words: 2t + 1),
    // reads 16 bytes per K step for simulation g
    const int xw = t * ps + warp * 32 + (g & 3) * 4 + (g >> 2) * 2;
    const int xr = (g >> 1) * ps + (g & 1) * 16 + t * 4;

    for (int i = tid; i < 2 * 4 * ps; i += nthr) xb[i] = 0;   // K steps past the last tile stay zero
    __syncthreads();
    if (warp >= L.mt) {
        bw_role(a, bws, zs, tid - node_threads, nthr - node_threads);
        return;
    }
    uint4 ahi[KS], alo[LO_SMEM ? 1 : KS];
    int sc_loaded = -1;
    float unscale[2] = {1.0f, 1.0f};   // of the rows of its two nodes

    for (int tile = blockIdx.x; tile < a.n_tiles; tile += gridDim.x) {
        const int *td = a.tiles + (size_t)tile * (TS + 1);
        const int sc_idx = td[0];
        const int sims[2] = {td[1 + 2 * t], td[2 + 2 * t]};
        if (sc_idx != sc_loaded) {
            // K step c, position 2p (+1) of K = source node 16 c + p (+ 8)
            const float *SC = a.sc_f32 + (size_t)sc_idx * n * n;
            // a row's weights times the power of two that puts its largest into [2^14, 2^15)
            float scale[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                float most = 0.0f;
                if (act[u])
                    for (int k = t; k < n; k += 4) most = fmaxf(most, fabsf(SC[(size_t)k * n + node[u]]));
                most = fmaxf(most, __shfl_xor_sync(~0u, most, 1));
                most = fmaxf(most, __shfl_xor_sync(~0u, most, 2));
                const int e = most > 0.0f && most <= FLT_MAX ? min(14 - ilogbf(most), 126) : 0;
                scale[u] = scalbnf(1.0f, e);
                unscale[u] = scalbnf(1.0f, -e);
            }
            auto w2 = [&](int c, int p, int u, uint32_t &hi, uint32_t &lo) {
                const int k0 = 16 * c + p, k1 = k0 + 8;
                split_f16x2(make_float2(act[u] && k0 < n ? SC[(size_t)k0 * n + node[u]] * scale[u] : 0.0f,
                                        act[u] && k1 < n ? SC[(size_t)k1 * n + node[u]] * scale[u] : 0.0f), hi, lo);
            };
#pragma unroll
            for (int c = 0; c < KS; ++c) {
                uint4 h, l;
                w2(c, t, 0, h.x, l.x);
                w2(c, t, 1, h.y, l.y);
                w2(c, t + 4, 0, h.z, l.z);
                w2(c, t + 4, 1, h.w, l.w);
                ahi[c] = h;
                if constexpr (LO_SMEM) {
                    alo_s[c * 32] = l;
                } else {
                    alo[c] = l;
                }
            }
            sc_loaded = sc_idx;
        }
        float2 p2[2][M::NP], s2[2][M::NS];   // per node, the simulation pair
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            float pa[2][M::NP], sa[2][M::NS];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                M::init(sa[w]);
#pragma unroll
                for (int q = 0; q < M::NP; ++q) pa[w][q] = 0.0f;
                if (act[u] && sims[w] >= 0) {
                    double rr[8];
                    for (int q = 0; q < 8; ++q)
                        rr[q] = q < a.n_regional ? a.rparams[(size_t)q * rstride + (size_t)sims[w] * n + node[u]] : 0.0;
                    M::params(pa[w], a.gparams[sims[w]], rr, K);
                }
            }
#pragma unroll
            for (int q = 0; q < M::NP; ++q) p2[u][q] = make_float2(pa[0][q], pa[1][q]);
#pragma unroll
            for (int q = 0; q < M::NS; ++q) s2[u][q] = make_float2(sa[0][q], sa[1][q]);
            Step::params(p2[u]);
        }
        // the two nodes' x of simulation 2t and 2t + 1 (padded nodes write 0)
        auto write_x = [&](uint32_t *x) {
            uint32_t h, l;
            split_f16x2(make_float2(act[0] ? s2[0][M::CV].x : 0.0f, act[1] ? s2[1][M::CV].x : 0.0f), h, l);
            *reinterpret_cast<uint2 *>(x + xw) = make_uint2(h, l);
            split_f16x2(make_float2(act[0] ? s2[0][M::CV].y : 0.0f, act[1] ? s2[1][M::CV].y : 0.0f), h, l);
            *reinterpret_cast<uint2 *>(x + xw + 16) = make_uint2(h, l);
        };
        // noise of `cnt` steps from inner step i0 of Balloon-Windkessel step b
        auto stage = [&](int b, int i0, int buf) {
            const int cnt = min(chunk, a.inner_it - i0);
            const int *shn = a.sh_nodes + (size_t)(b / a.noise_bw_it) * n;   // sh_ts: [repeats][noise_bw_it], one run
            const float *src = a.noise_f32 + ((long long)__ldg(a.sh_ts + b) * a.inner_it + i0) * n * NN;
            for (int q = warp; q < cnt; q += L.mt)
                for (int k = lane; k < n; k += 32)
                    cp_small<NN * 4>(noise_s + ((size_t)(buf * chunk + q) * n + k) * NN,
                                     src + ((size_t)q * n + __ldg(shn + k)) * NN);
        };
        uint32_t *xc = xb, *xn = xb + 4 * ps;
        write_x(xc);
        stage(0, 0, 0);
        cp_commit();
        cp_wait_all();
        bar_sync(1, node_threads);
        int nbuf = 0, states_i = 0, to_sample = a.states_sampling_iters;
        for (int bw_i = 0; bw_i < a.bw_it; ++bw_i) {
            const bool sample = --to_sample == 0 && a.ext_out;
            if (to_sample == 0) to_sample = a.states_sampling_iters;
            for (int i0 = 0; i0 < a.inner_it; i0 += chunk) {
                const bool next_bw = i0 + chunk >= a.inner_it;
                if (!next_bw) stage(bw_i, i0 + chunk, nbuf ^ 1);
                else if (bw_i + 1 < a.bw_it) stage(bw_i + 1, 0, nbuf ^ 1);
                cp_commit();
                const int i1 = min(i0 + chunk, a.inner_it);
                for (int inner = i0; inner < i1; ++inner) {
                    float2 hh[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
                    float hl[4] = {0.0f, 0.0f, 0.0f, 0.0f}, lh[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int k = 0; k < KS; ++k) {   // K steps past the nodes hold zeros
                        const uint4 w = *reinterpret_cast<const uint4 *>(xc + xr + k * 32);
                        mma_f16_add(hh, ahi[k], w.x, w.z);
                        mma_f16(hl, ahi[k], w.y, w.w);
                        if constexpr (LO_SMEM) mma_f16(lh, alo_s[k * 32], w.x, w.z);
                        else mma_f16(lh, alo[k], w.x, w.z);
                    }
                    const float *nz = noise_s + (size_t)(nbuf * chunk + inner - i0) * n * NN;
                    const bool last = inner == a.inner_it - 1;
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        float n0, n1 = 0.0f;
                        if constexpr (NN == 2) {
                            const float2 v = *reinterpret_cast<const float2 *>(nz + nzoff[u]);
                            n0 = v.x; n1 = v.y;
                        } else {
                            n0 = nz[nzoff[u]];
                        }
                        float2 o[M::NOUT];
                        const float lo_unscale = unscale[u] * (1.0f / LO_SCALE);
                        float2 lo = make_float2(hl[2 * u] + lh[2 * u], hl[2 * u + 1] + lh[2 * u + 1]);
                        if constexpr (KS > 8 || M::ACC) lo = __ffma2_rn(hh[u], make_float2(HH_BIAS * LO_SCALE, HH_BIAS * LO_SCALE), lo);
                        const float2 in = __ffma2_rn(lo,
                                                     make_float2(lo_unscale, lo_unscale),
                                                     make_float2(hh[u].x * unscale[u], hh[u].y * unscale[u]));
                        Step::step(s2[u], p2[u], in, n0, n1, K, o);
                        if (last && sample && act[u]) {
#pragma unroll
                            for (int w = 0; w < 2; ++w) {
                                if (sims[w] < 0) continue;
#pragma unroll
                                for (int v = 0; v < M::NOUT; ++v) {
                                    const double ov = (double)(w ? o[v].y : o[v].x);
                                    double *out = a.states + ((size_t)v * a.n_sims + sims[w]) * ext + node[u];
                                    if (a.states_ts) {
                                        if (states_i < a.states_len) out[(size_t)states_i * n] = ov;
                                    } else if (states_i == a.n_states_samples_remove) {
                                        *out = ov;   // the sum of the kept samples, in the output itself
                                    } else if (states_i > a.n_states_samples_remove) {
                                        *out += ov;
                                    }
                                }
                            }
                        }
                    }
                    write_x(xn);
                    if (inner == i1 - 1) cp_wait_all();   // the next chunk's noise, before the barrier
                    bar_sync(1, node_threads);
                    uint32_t *sw = xc;
                    xc = xn;
                    xn = sw;
                }
                nbuf ^= 1;
            }
            // this millisecond's Balloon-Windkessel inputs; the barrier also waits for the last one's
            float *z = zs + (bw_i & 1) * items;
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (act[u]) {
                    z[(2 * t) * n + node[u]] = s2[u][M::BV].x;
                    z[(2 * t + 1) * n + node[u]] = s2[u][M::BV].y;
                }
            bar_sync(2, nthr);
            if (sample) ++states_i;
        }
        if (a.ext_out && !a.states_ts) {
            const int pts = states_i - a.n_states_samples_remove;
#pragma unroll
            for (int u = 0; u < 2; ++u)
#pragma unroll
                for (int w = 0; w < 2; ++w)
                    if (act[u] && sims[w] >= 0)
                        for (int v = 0; v < M::NOUT; ++v) {
                            double &out = a.states[((size_t)v * a.n_sims + sims[w]) * ext + node[u]];
                            out = (pts > 0 ? out : 0.0) / pts;   // no kept sample: 0 / pts
                        }
        }
        bar_sync(2, nthr);   // the tile's Balloon-Windkessel warps are done with its inputs
    }
}

template <class M, int KS>
cudaError_t launch_ks(const IntegrateArgs &a, cudaStream_t st) {
    const Layout L = layout(a.nodes, M::NN, std::min(a.inner_it, NOISE_CHUNK), KS, lo_in_smem(KS));
    cudaError_t e = allow_dynamic_smem(k_integrate_mma<M, KS>);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, occ = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int threads = (L.mt + bw_warps(L.mt)) * 32;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_integrate_mma<M, KS>, threads, L.bytes);
    if (e != cudaSuccess) return e;
    if (occ < 1) return cudaErrorInvalidConfiguration;
    k_integrate_mma<M, KS><<<std::min(a.n_tiles, occ * sms), threads, L.bytes, st>>>(a);
    return cudaGetLastError();
}

// Compiled K extents; a run takes the least that holds its nodes.  X is the model above 80
// nodes, Z above 128.
template <class M, class X, class Z>
cudaError_t launch_model(const IntegrateArgs &a, cudaStream_t st) {
    const int mt = (a.nodes + 15) / 16;
    if (mt <= 2) return launch_ks<M, 2>(a, st);
    if (mt <= 4) return launch_ks<M, 4>(a, st);
    if (mt <= 5) return launch_ks<M, 5>(a, st);
    if (mt <= 6) return launch_ks<X, 6>(a, st);
    if (mt <= 7) return launch_ks<X, 7>(a, st);
    if (mt <= 8) return launch_ks<X, 8>(a, st);
    if (mt <= 10) return launch_ks<Z, 10>(a, st);
    if (mt <= 13) return launch_ks<Z, 13>(a, st);
    if (mt <= 14) return launch_ks<Z, 14>(a, st);
    return cudaErrorInvalidValue;
}

}  // namespace

// No delays, up to 224 nodes: A lo and the Balloon-Windkessel state of more do not fit
// shared memory together.
bool fp32_supported(int model, int nodes, bool has_delay) {
    if (has_delay || nodes > 224 || nodes < 1) return false;
    return model == MODEL_RWW || model == MODEL_WC || model == MODEL_JR || model == MODEL_RWWEX;
}

void fill_k32(int model, const ModelK &K, float *k32) {
    auto put = [&](const auto &k) {
        static_assert(sizeof(k) <= 24 * sizeof(float), "FP32 constants");
        std::memcpy(k32, &k, sizeof(k));
    };
    switch (model) {
        case MODEL_RWW: put(RWW32::make(K)); break;
        case MODEL_WC: put(WC32::make(K)); break;
        case MODEL_JR: put(JR32::make(K)); break;
        case MODEL_RWWEX: put(RWWEx32::make(K)); break;
        default: break;
    }
}

// The rates by rate2_acc where FP32 sums or better ones were there before, so that no run is
// farther from FP64 than it was: BOLD, relative, geometric mean of 4-6 batches of 40 at
// densities 0.25 / 0.8, per-simulation kernel (FP32 sums, expm1), fast rates, as here: rWW
// 200 nodes 2.46e-8 / 2.30e-8, 3.03e-8 / 2.88e-8, 2.41e-8 / 2.28e-8; rWWEx 200 nodes 1.34e-7 /
// 1.87e-7, 1.61e-7 / 2.05e-7, 1.18e-7 / 1.48e-7; WC 200 nodes 3.15e-8 / 3.12e-8, as here 2.02e-8 /
// 2.03e-8; rWWEx 128 nodes 2.87e-7 / 1.69e-7 (tcgen05, BF16 halves), 1.70e-7 / 2.10e-7 with the
// fast rate.  They cost 10-17 % (rWW 200 nodes 18.4 -> 20.0 ms per simulated second).
cudaError_t launch_integrate_mma(int model, const IntegrateArgs &a, cudaStream_t st) {
    switch (model) {
        case MODEL_RWW: return launch_model<RWW32, RWW32, RWW32T<true>>(a, st);
        case MODEL_WC: return launch_model<WC32, WC32, WC32>(a, st);
        case MODEL_JR: return launch_model<JR32, JR32, JR32>(a, st);
        case MODEL_RWWEX: return launch_model<RWWEx32, RWWExs32, RWWExs32>(a, st);
        default: break;
    }
    return cudaErrorNotSupported;
}

}  // namespace cbnm
