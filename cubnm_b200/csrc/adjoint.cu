// Adjoint (reverse-mode) gradient of an FP32 rWW batch with the noise held fixed.
//
// Forward (k_adj_forward): the FP32 per-simulation rWW time loop of
// integrate_sim.cuh (same expressions, same coupling order, so the same BOLD),
// plus a checkpoint of (S_E, S_I) and the FP64 Balloon-Windkessel state
// (x, f, nu, q) at the start of every segment of seg_bw Balloon-Windkessel
// steps (seg_bw * inner_it integration steps).
//
// Backward (k_adj_backward): segments in reverse.  Each segment is recomputed
// from its checkpoint, storing the pre-step S_E, S_I and coupling input of every
// step and the pre-step Balloon-Windkessel state of every millisecond in a
// scratch; then the steps are run backwards.  With lambda the adjoint of each
// state, per integration step of node j (reference step: rww.cpp:194-232):
//   u_E = S_E + sigma sqrt(dt) n0 + dt g_E (1 - S_E) r_E - dt/t_E S_E  (clamped: lambda passes only inside [0, 1])
//   u_I = S_I + sigma sqrt(dt) n1 + dt g_I r_I - dt/t_I S_I
//   r(x) = x / (1 - e^{-d x}),  r'(x) = ((1 - e) - d x e) / (1 - e)^2,  e = e^{-d x}
//   I_E = wEI0 + w_p J_N S_E + G J_N in_j - wIE S_I,   I_I = wII0 + J_N S_E - wII S_I
//   in_j = sum_k SC[k][j] S_E,k  =>  lambda_S_E,k += sum_j SC[k][j] lambda_in,j  (a transposed product:
//   both products as the FP32 sum of integrate_sim.cuh)
// and per millisecond the reverse of the Balloon-Windkessel Euler step
// (bw.cu:4-15; the f update uses the new x, the q update the new nu) with the
// BOLD sample (bnm.cpp:316-320) adding dL/dBOLD * dBOLD/d(q, nu).
// Up to 208 nodes the SC (and, in the reverse sweep, its transpose) is in registers:
// k_adj_*_reg, a group of 16 lanes per four rows, lane l the sources k = l mod 16, the
// lanes' partial sums met in a transposing butterfly; the node's own work follows on one
// thread per node.  One thread per node over SC in L1 / L2 (k_adj_forward / _backward,
// kept for larger networks) made a step of a fit of 64 simulations x 200 nodes a chain of
// 200 dependent loads per product: 22,000 cycles per forward and backward step together.
// The node's adjoints, gradient sums and parameters rest in shared memory between steps,
// so that the weights keep their registers.
// Parameter gradients (G per simulation; w_p, J_N, wIE, sigma per node) are
// accumulated in FP64 by the thread of each node; G is summed over nodes at
// the end.  Adjoint states are FP32 like the forward state, Balloon-Windkessel
// adjoints FP64 like its state.
#include "integrate_sim.cuh"

namespace cbnm {
namespace {

using M = RWWm<float>;

__device__ __forceinline__ int noise_ts(const IntegrateArgs &a, int bw_i, int &repeat) {
    repeat = bw_i / a.noise_bw_it;
    return a.sh_ts[(bw_i % a.noise_bw_it) + repeat * a.noise_bw_it];
}

// d r / d x for r(x) = x / (1 - e^{-d x}); series near 0 where the closed form cancels.
// u is capped at -43, where r' is below 1e-16 and the square of the divisor still finite.
__device__ __forceinline__ float rate_deriv(float x, float d) {
    const float u = fmaxf(d * x, -43.0f);
    const bool small = fabsf(u) < 1e-2f;
    const float e = expf(-u), den = small ? 1.0f : -expm1f(-u);
    return small ? 0.5f + u * (1.0f / 6.0f) : div_nr(den - u * e, den * den);
}

__device__ double block_sum_d(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0) {
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        red[32] = t;
    }
    __syncthreads();
    return red[32];
}

struct Params {
    float g[M::NG];
    float r[M::NR];
};

__device__ __forceinline__ Params load_params(const IntegrateArgs &a, int sim, int j, bool act) {
    Params P;
    P.g[0] = (float)a.gparams[sim];
    const size_t rstride = (size_t)a.n_sims * a.nodes;
#pragma unroll
    for (int i = 0; i < M::NR; ++i) P.r[i] = act ? (float)a.rparams[i * rstride + (size_t)sim * a.nodes + j] : 0.0f;
    return P;
}

// Reverse of one integration step of a node: its adjoints lE, lI become those before the
// step (without the transposed coupling), and the step's share of the gradients.
struct StepGrad { float in, w_p, J_N, G, wIE, sigma; };
__device__ __forceinline__ StepGrad step_reverse(float &lE, float &lI, float SE, float SI, float in, float n0, float n1,
                                                 const Params &P, const RWWKt<float> &m) {
    const float w_p = P.r[0], J_N = P.r[1], wIE = P.r[2], sig = P.r[3], G = P.g[0], sqdt = m.sqrt_dt;
    // forward pieces, as RWWm<float>::step
    const float IE = m.w_E__I_0 + w_p * J_N * SE + in * G * J_N - wIE * SI;
    const float II = m.w_I__I_0 + J_N * SE - m.w_II * SI;
    const float xE = m.a_E * IE - m.b_E;
    const float xI = m.a_I * II - m.b_I;
    const float rE = rate_of(xE, m.d_E);
    const float rI = rate_of(xI, m.d_I);
    const float uE = SE + (n0 * sig * sqdt + m.dt_gamma_E * ((1.0f - SE) * rE) - m.dt_itau_E * SE);
    const float uI = SI + (n1 * sig * sqdt + m.dt_gamma_I * rI - m.dt_itau_I * SI);
    const float luE = (uE >= 0.0f && uE <= 1.0f) ? lE : 0.0f;
    const float luI = (uI >= 0.0f && uI <= 1.0f) ? lI : 0.0f;
    const float lrE = luE * m.dt_gamma_E * (1.0f - SE);
    const float lrI = luI * m.dt_gamma_I;
    float lSE = luE * (1.0f - m.dt_gamma_E * rE - m.dt_itau_E);
    float lSI = luI * (1.0f - m.dt_itau_I);
    const float lIE = lrE * rate_deriv(xE, m.d_E) * m.a_E;
    const float lII = lrI * rate_deriv(xI, m.d_I) * m.a_I;
    lSE += lIE * w_p * J_N + lII * J_N;
    lSI += -lIE * wIE - lII * m.w_II;
    StepGrad d;
    d.in = lIE * G * J_N;
    d.w_p = lIE * J_N * SE;
    d.J_N = lIE * (w_p * SE + G * in) + lII * SE;
    d.G = lIE * J_N * in;
    d.wIE = -lIE * SI;
    d.sigma = (luE * n0 + luI * n1) * sqdt;
    lE = lSE;
    lI = lSI;
    return d;
}

// Reverse of one Balloon-Windkessel step from the state f0, nu0, q0 before it, with the
// BOLD sample's dL/dBOLD where it is one; returns the adjoint of its input.
__device__ __forceinline__ double bw_reverse(double &lx, double &lf, double &lnu, double &lq, double f0, double nu0,
                                             double q0, double gb, bool sample, const IntegrateArgs &a) {
    const BWConst &c = a.bw;
    const double ct = c.dt_itau, ia = c.ialpha;
    const double inv_f = 1.0 / f0, p0 = pow_nu(nu0, a.bwf), E = pow_omr(f0, inv_f, a.bwf);
    const double nu1 = nu0 + ct * (f0 - p0), inv_nu1 = 1.0 / nu1;
    const double A1 = pow_nu(nu1, a.bwf) * inv_nu1;                  // nu1^(a-1)
    if (sample) {  // BOLD = V0 (k1 (1-q) + k2 (1-q/nu) + k3 (1-nu))
        const double q1 = q0 + ct * (f0 * (1.0 - E) / c.rho - A1 * q0);
        lq += gb * c.V_0 * (-c.k1 - c.k2 * inv_nu1);
        lnu += gb * c.V_0 * (c.k2 * q1 * inv_nu1 * inv_nu1 - c.k3);
    }
    const double dq_dq0 = 1.0 - ct * A1;
    const double dq_dnu1 = -ct * q0 * (ia - 1.0) * A1 * inv_nu1;
    const double dq_df0 = ct / c.rho * ((1.0 - E) + E * a.bwf.ln_omr * inv_f);
    const double lq0 = lq * dq_dq0;
    const double lnu1 = lnu + lq * dq_dnu1;
    double lf0 = lq * dq_df0;
    const double lnu0 = lnu1 * (1.0 - ct * ia * (p0 / nu0));
    lf0 += lnu1 * ct;
    lf0 += lf;
    const double lx1 = lx + lf * c.dt;
    lf0 += lx1 * (-c.dt * c.y);
    lx = lx1 * (1.0 - c.dt * c.kappa);
    lf = lf0; lnu = lnu0; lq = lq0;
    return lx1 * c.dt;
}

// One integration step of node j (the coupling input already formed), exactly as
// k_integrate_sim<RWWm<float>, false, float, ...>.
__device__ __forceinline__ void fwd_step(float *s, const Params &P, float in, const IntegrateArgs &a, int sh_ts,
                                         int inner, int sh_j) {
    const long long ni = ((long long)sh_ts * a.inner_it + inner) * a.nodes * M::NN + (long long)sh_j * M::NN;
    const float n0 = a.noise_f32[ni], n1 = a.noise_f32[ni + 1];
    float iv[M::NI];
    M::step(s, iv, P.g, P.r, in, n0, n1, a.Kf);
}

__global__ void __launch_bounds__(1024) k_adj_forward(const AdjArgs A) {
    const IntegrateArgs &a = A.ia;
    const int sim = A.sim_begin + blockIdx.x;
    const int j = threadIdx.x, n = a.nodes;
    const bool act = j < n;
    extern __shared__ __align__(16) float x1[];
    const float *SC = a.sc_f32 + (size_t)a.sc_idx[sim] * n * n;
    const Params P = load_params(a, sim, j, act);
    float s[M::NS];
#pragma unroll
    for (int i = 0; i < M::NS; ++i) s[i] = 0.0f;
    float iv0[M::NI];
    M::init(s, iv0, P.g, P.r);
    double bx = 0.0, bf = 1.0, bnu = 1.0, bq = 1.0;
    if (act) x1[j] = s[M::CONN];
    double *bold = a.bold + (size_t)sim * a.bold_len * n;
    int bold_i = 0;
    for (int bw_i = 0; bw_i < a.bw_it; ++bw_i) {
        if (bw_i % A.seg_bw == 0 && act) {
            const size_t c = (size_t)sim * A.n_seg + bw_i / A.seg_bw;
            A.ck_s[(c * 2 + 0) * n + j] = s[4];
            A.ck_s[(c * 2 + 1) * n + j] = s[5];
            A.ck_bw[(c * 4 + 0) * n + j] = bx;
            A.ck_bw[(c * 4 + 1) * n + j] = bf;
            A.ck_bw[(c * 4 + 2) * n + j] = bnu;
            A.ck_bw[(c * 4 + 3) * n + j] = bq;
        }
        int repeat;
        const int sh_ts = noise_ts(a, bw_i, repeat);
        const int sh_j = act ? a.sh_nodes[(size_t)repeat * n + j] : 0;
        for (int inner = 0; inner < a.inner_it; ++inner) {
            __syncthreads();
            float in = 0.0f;
            if (act) {
                in = coupling_f32(SC, x1, n, j);
                fwd_step(s, P, in, a, sh_ts, inner, sh_j);
            }
            __syncthreads();
            if (act) x1[j] = s[M::CONN];
        }
        if (act) bw_step(bx, bf, bnu, bq, (double)s[M::BOLDV], a.bw);
        if ((bw_i + 1) % a.bold_tr_iters == 0) {
            if (act && bold_i < a.bold_len)  // no slot for a sample past bold_len
                bold[(size_t)bold_i * n + j] =
                    a.bw.V_0 * (a.bw.k1 * (1 - bq) + a.bw.k2 * (1 - bq / bnu) + a.bw.k3 * (1 - bnu));
            bold_i++;
        }
    }
}

__global__ void __launch_bounds__(1024) k_adj_backward(const AdjArgs A) {
    const IntegrateArgs &a = A.ia;
    const int sim = A.sim_begin + blockIdx.x;
    const int j = threadIdx.x, n = a.nodes;
    const bool act = j < n;
    extern __shared__ __align__(16) float sh[];
    float *x1 = sh;                          // S_E of every node (forward recompute)
    float *lin = sh + ((n + 3) & ~3);        // adjoint of every node's coupling input (16-byte aligned)
    __shared__ double red[33];
    const float *SC = a.sc_f32 + (size_t)a.sc_idx[sim] * n * n;
    const float *SCT = A.sct_f32 + (size_t)a.sc_idx[sim] * n * n;
    const Params P = load_params(a, sim, j, act);
    const int steps_seg = A.seg_bw * a.inner_it;
    float *scr_s = A.scr_s + (size_t)blockIdx.x * steps_seg * 3 * n;
    float *scr_z = A.scr_z + (size_t)blockIdx.x * A.seg_bw * n;
    double *scr_bw = A.scr_bw + (size_t)blockIdx.x * A.seg_bw * 4 * n;
    const double *dbold = A.dbold + (size_t)sim * a.bold_len * n;

    float lE = 0.0f, lI = 0.0f;                        // adjoints of S_E, S_I
    double lx = 0.0, lf = 0.0, lnu = 0.0, lq = 0.0;    // adjoints of the Balloon-Windkessel state
    double gG = 0.0, gWp = 0.0, gJ = 0.0, gWIE = 0.0, gSig = 0.0;

    for (int seg = A.n_seg - 1; seg >= 0; --seg) {
        const int bw0 = seg * A.seg_bw;
        const int nb = min(A.seg_bw, a.bw_it - bw0);
        // ---- recompute the segment from its checkpoint
        float s[M::NS];
#pragma unroll
        for (int i = 0; i < M::NS; ++i) s[i] = 0.0f;
        double bx = 0.0, bf = 1.0, bnu = 1.0, bq = 1.0;
        if (act) {
            const size_t ck = (size_t)sim * A.n_seg + seg;
            s[4] = A.ck_s[(ck * 2 + 0) * n + j];
            s[5] = A.ck_s[(ck * 2 + 1) * n + j];
            bx = A.ck_bw[(ck * 4 + 0) * n + j];
            bf = A.ck_bw[(ck * 4 + 1) * n + j];
            bnu = A.ck_bw[(ck * 4 + 2) * n + j];
            bq = A.ck_bw[(ck * 4 + 3) * n + j];
        }
        __syncthreads();
        if (act) x1[j] = s[M::CONN];
        for (int b = 0; b < nb; ++b) {
            const int bw_i = bw0 + b;
            int repeat;
            const int sh_ts = noise_ts(a, bw_i, repeat);
            const int sh_j = act ? a.sh_nodes[(size_t)repeat * n + j] : 0;
            if (act) {
                scr_bw[((size_t)b * 4 + 0) * n + j] = bx;
                scr_bw[((size_t)b * 4 + 1) * n + j] = bf;
                scr_bw[((size_t)b * 4 + 2) * n + j] = bnu;
                scr_bw[((size_t)b * 4 + 3) * n + j] = bq;
            }
            for (int inner = 0; inner < a.inner_it; ++inner) {
                __syncthreads();
                float in = 0.0f;
                if (act) {
                    in = coupling_f32(SC, x1, n, j);
                    const size_t t = (size_t)b * a.inner_it + inner;
                    scr_s[(t * 3 + 0) * n + j] = s[4];
                    scr_s[(t * 3 + 1) * n + j] = s[5];
                    scr_s[(t * 3 + 2) * n + j] = in;
                    fwd_step(s, P, in, a, sh_ts, inner, sh_j);
                }
                __syncthreads();
                if (act) x1[j] = s[M::CONN];
            }
            if (act) {
                scr_z[(size_t)b * n + j] = s[M::BOLDV];
                bw_step(bx, bf, bnu, bq, (double)s[M::BOLDV], a.bw);
            }
        }
        // ---- reverse through the segment
        for (int b = nb - 1; b >= 0; --b) {
            const int bw_i = bw0 + b;
            int repeat;
            const int sh_ts = noise_ts(a, bw_i, repeat);
            const int sh_j = act ? a.sh_nodes[(size_t)repeat * n + j] : 0;
            if (act) {
                const double f0 = scr_bw[((size_t)b * 4 + 1) * n + j];
                const double nu0 = scr_bw[((size_t)b * 4 + 2) * n + j], q0 = scr_bw[((size_t)b * 4 + 3) * n + j];
                const int vol = (bw_i + 1) / a.bold_tr_iters - 1;
                const bool sample = (bw_i + 1) % a.bold_tr_iters == 0 && vol < a.bold_len;
                lE += (float)bw_reverse(lx, lf, lnu, lq, f0, nu0, q0, sample ? dbold[(size_t)vol * n + j] : 0.0, sample, a);
            }
            for (int inner = a.inner_it - 1; inner >= 0; --inner) {
                float lin_j = 0.0f, SE = 0.0f, SI = 0.0f, in = 0.0f;
                if (act) {
                    const size_t t = (size_t)b * a.inner_it + inner;
                    SE = scr_s[(t * 3 + 0) * n + j];
                    SI = scr_s[(t * 3 + 1) * n + j];
                    in = scr_s[(t * 3 + 2) * n + j];
                    const long long ni = ((long long)sh_ts * a.inner_it + inner) * n * M::NN + (long long)sh_j * M::NN;
                    const StepGrad d = step_reverse(lE, lI, SE, SI, in, a.noise_f32[ni], a.noise_f32[ni + 1], P, a.Kf.rww);
                    gWp += (double)d.w_p;
                    gJ += (double)d.J_N;
                    gG += (double)d.G;
                    gWIE += (double)d.wIE;
                    gSig += (double)d.sigma;
                    lin_j = d.in;
                    lin[j] = lin_j;
                }
                __syncthreads();
                if (act) {  // lambda_S_E,j += sum_k SC[j][k] lambda_in,k
                    lE += coupling_f32(SCT, lin, n, j);
                }
                __syncthreads();
            }
        }
    }
    const double gG_all = block_sum_d(act ? gG : 0.0, red);
    if (j == 0) A.grad_g[sim] = gG_all;
    if (act) {
        const size_t rs = (size_t)a.n_sims * n, o = (size_t)sim * n + j;
        A.grad_r[0 * rs + o] = gWp;
        A.grad_r[1 * rs + o] = gJ;
        A.grad_r[2 * rs + o] = gWIE;
        A.grad_r[3 * rs + o] = gSig;
    }
}

// ---------------------------------------------------------------- SC in registers (<= 16 KPL nodes)
// The rows row0 .. row0 + 3 of this half-warp, sources l + 16 i on lane l.
template <int KPL>
struct Rows {
    float2 w[2][KPL];
    int row0, l;
    // m[k][j]: row = source
    __device__ __forceinline__ void load(const float *m, int n) {
        const int lane = threadIdx.x & 31;
        l = lane & 15;
        row0 = (threadIdx.x >> 5) * 8 + (lane >> 4) * 4;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < KPL; ++i) {
                const int k = l + 16 * i, j0 = row0 + 2 * r;
                w[r][i] = make_float2(k < n && j0 < n ? m[(size_t)k * n + j0] : 0.0f,
                                      k < n && j0 + 1 < n ? m[(size_t)k * n + j0 + 1] : 0.0f);
            }
    }
    // sums[j] = sum_k m[k][j] x[k] for the half-warp's rows
    __device__ __forceinline__ void product(const float *x, float *sums) const {
        float2 v[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
#pragma unroll
        for (int i = 0; i < KPL; ++i) {
            const float xk = x[l + 16 * i];
#pragma unroll
            for (int r = 0; r < 2; ++r) v[r] = __ffma2_rn(w[r][i], make_float2(xk, xk), v[r]);
        }
        const bool up = l & 8, odd = l & 4;   // lanes keep rows {0,1} / {2,3}, then one row, then its sum
        float2 keep = up ? v[1] : v[0], send = up ? v[0] : v[1];
        keep.x += __shfl_xor_sync(0xffffffffu, send.x, 8);
        keep.y += __shfl_xor_sync(0xffffffffu, send.y, 8);
        float s = odd ? keep.y : keep.x;
        s += __shfl_xor_sync(0xffffffffu, odd ? keep.x : keep.y, 4);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if ((l & 3) == 0) sums[row0 + (up ? 2 : 0) + (odd ? 1 : 0)] = s;
    }
};

// Shared memory of the register kernels; n16 = 16 KPL.
template <int KPL>
struct AdjSmem {
    static constexpr int N = 16 * KPL;
    double bw[4][N];     // Balloon-Windkessel state (recompute), or its adjoints (reverse)
    double bwl[4][N];    // adjoints x, f, nu, q
    double acc[5][N];    // gradient sums G, w_p, J_N, wIE, sigma
    float x[N], sums[N]; // product input and result
    float sI[N], lE[N], lI[N];
    float par[5][N];     // w_p, J_N, wIE, sigma, G
};

template <int KPL>
__device__ __forceinline__ Params smem_params(const AdjSmem<KPL> &sm, int j) {
    Params P;
#pragma unroll
    for (int q = 0; q < 4; ++q) P.r[q] = sm.par[q][j];
    P.g[0] = sm.par[4][j];
    return P;
}

// Noise of node j at inner step `inner` of Balloon-Windkessel step bw_i.
__device__ __forceinline__ float2 noise_at(const IntegrateArgs &a, int bw_i, int inner, int j) {
    const int repeat = bw_i / a.noise_bw_it, sh_ts = __ldg(a.sh_ts + bw_i);   // [repeats][noise_bw_it], one run
    const int sh_j = __ldg(a.sh_nodes + (size_t)repeat * a.nodes + j);
    return *reinterpret_cast<const float2 *>(a.noise_f32 + (((size_t)sh_ts * a.inner_it + inner) * a.nodes + sh_j) * 2);
}

// One step of the time loop: the product with all warps, the update on thread j < n
// (S_E in sm.x, S_I in sm.sI).  RECORD: the state before it and the coupling input go to scr.
template <int KPL, bool RECORD>
__device__ __forceinline__ void reg_step(const IntegrateArgs &a, AdjSmem<KPL> &sm, const Rows<KPL> &W, int j, bool act,
                                         float2 nz, float *scr) {
    W.product(sm.x, sm.sums);
    __syncthreads();
    if (act) {
        const Params P = smem_params(sm, j);
        float s[M::NS], iv[M::NI];
        s[4] = sm.x[j];
        s[5] = sm.sI[j];
        const float in = sm.sums[j];
        if (RECORD) {
            scr[j] = s[4];
            scr[a.nodes + j] = s[5];
            scr[2 * a.nodes + j] = in;
        }
        M::step(s, iv, P.g, P.r, in, nz.x, nz.y, a.Kf);
        sm.x[j] = s[4];
        sm.sI[j] = s[5];
    }
    __syncthreads();
}

template <int KPL>
__device__ __forceinline__ void reg_bw_step(const IntegrateArgs &a, AdjSmem<KPL> &sm, int j) {
    double x = sm.bw[0][j], f = sm.bw[1][j], nu = sm.bw[2][j], q = sm.bw[3][j];
    bw_step64(x, f, nu, q, (double)sm.x[j], a.bwf);
    sm.bw[0][j] = x; sm.bw[1][j] = f; sm.bw[2][j] = nu; sm.bw[3][j] = q;
}

template <int KPL>
__global__ void __launch_bounds__(KPL * 64) k_adj_forward_reg(const __grid_constant__ AdjArgs A) {
    extern __shared__ __align__(16) unsigned char raw[];
    AdjSmem<KPL> &sm = *reinterpret_cast<AdjSmem<KPL> *>(raw);
    const IntegrateArgs &a = A.ia;
    const int sim = A.sim_begin + blockIdx.x, j = threadIdx.x, n = a.nodes;
    const bool act = j < n;
    Rows<KPL> W;
    W.load(a.sc_f32 + (size_t)a.sc_idx[sim] * n * n, n);
    for (int k = j; k < 16 * KPL; k += blockDim.x) sm.x[k] = 0.0f;   // padding
    __syncthreads();
    if (act) {
        const Params P = load_params(a, sim, j, true);
#pragma unroll
        for (int q = 0; q < 4; ++q) sm.par[q][j] = P.r[q];
        sm.par[4][j] = P.g[0];
        float s[M::NS], iv[M::NI];
        M::init(s, iv, P.g, P.r);
        sm.x[j] = s[4];
        sm.sI[j] = s[5];
        sm.bw[0][j] = 0.0;
        sm.bw[1][j] = sm.bw[2][j] = sm.bw[3][j] = 1.0;
    }
    __syncthreads();
    double *bold = a.bold + (size_t)sim * a.bold_len * n;
    int bold_i = 0;
    float2 nz = act ? noise_at(a, 0, 0, j) : make_float2(0.0f, 0.0f);
    for (int bw_i = 0; bw_i < a.bw_it; ++bw_i) {
        if (bw_i % A.seg_bw == 0 && act) {
            const size_t c = (size_t)sim * A.n_seg + bw_i / A.seg_bw;
            A.ck_s[(c * 2 + 0) * n + j] = sm.x[j];
            A.ck_s[(c * 2 + 1) * n + j] = sm.sI[j];
#pragma unroll
            for (int q = 0; q < 4; ++q) A.ck_bw[(c * 4 + q) * n + j] = sm.bw[q][j];
        }
        for (int inner = 0; inner < a.inner_it; ++inner) {
            const float2 z = nz;   // the next step's is on its way during this one
            const bool last = inner == a.inner_it - 1;
            if (act && !(last && bw_i + 1 == a.bw_it)) nz = last ? noise_at(a, bw_i + 1, 0, j) : noise_at(a, bw_i, inner + 1, j);
            reg_step<KPL, false>(a, sm, W, j, act, z, nullptr);
        }
        if (act) reg_bw_step(a, sm, j);
        if ((bw_i + 1) % a.bold_tr_iters == 0) {
            if (act && bold_i < a.bold_len)  // no slot for a sample past bold_len
                bold[(size_t)bold_i * n + j] = a.bw.V_0 * (a.bw.k1 * (1 - sm.bw[3][j]) + a.bw.k2 * (1 - sm.bw[3][j] / sm.bw[2][j]) +
                                                           a.bw.k3 * (1 - sm.bw[2][j]));
            bold_i++;
        }
    }
}

template <int KPL>
__global__ void __launch_bounds__(KPL * 64) k_adj_backward_reg(const __grid_constant__ AdjArgs A) {
    extern __shared__ __align__(16) unsigned char raw[];
    AdjSmem<KPL> &sm = *reinterpret_cast<AdjSmem<KPL> *>(raw);
    __shared__ double red[33];
    const IntegrateArgs &a = A.ia;
    const int sim = A.sim_begin + blockIdx.x, j = threadIdx.x, n = a.nodes;
    const bool act = j < n;
    const int steps_seg = A.seg_bw * a.inner_it;
    float *scr_s = A.scr_s + (size_t)blockIdx.x * steps_seg * 3 * n;
    double *scr_bw = A.scr_bw + (size_t)blockIdx.x * A.seg_bw * 4 * n;
    const double *dbold = A.dbold + (size_t)sim * a.bold_len * n;
    for (int k = j; k < 16 * KPL; k += blockDim.x) sm.x[k] = 0.0f;   // padding
    __syncthreads();
    if (act) {
        const Params P = load_params(a, sim, j, true);
#pragma unroll
        for (int q = 0; q < 4; ++q) sm.par[q][j] = P.r[q];
        sm.par[4][j] = P.g[0];
        sm.lE[j] = sm.lI[j] = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) sm.bwl[q][j] = 0.0;
#pragma unroll
        for (int q = 0; q < 5; ++q) sm.acc[q][j] = 0.0;
    }
    Rows<KPL> W;
    for (int seg = A.n_seg - 1; seg >= 0; --seg) {
        const int bw0 = seg * A.seg_bw, nb = min(A.seg_bw, a.bw_it - bw0);
        // ---- recompute the segment from its checkpoint
        W.load(a.sc_f32 + (size_t)a.sc_idx[sim] * n * n, n);
        __syncthreads();
        float2 nz = make_float2(0.0f, 0.0f);
        if (act) {
            const size_t ck = (size_t)sim * A.n_seg + seg;
            sm.x[j] = A.ck_s[(ck * 2 + 0) * n + j];
            sm.sI[j] = A.ck_s[(ck * 2 + 1) * n + j];
#pragma unroll
            for (int q = 0; q < 4; ++q) sm.bw[q][j] = A.ck_bw[(ck * 4 + q) * n + j];
            nz = noise_at(a, bw0, 0, j);
        }
        __syncthreads();
        for (int b = 0; b < nb; ++b) {
            if (act) {
#pragma unroll
                for (int q = 0; q < 4; ++q) scr_bw[((size_t)b * 4 + q) * n + j] = sm.bw[q][j];
            }
            for (int inner = 0; inner < a.inner_it; ++inner) {
                const float2 z = nz;
                const bool last = inner == a.inner_it - 1;
                if (act && !(last && b + 1 == nb)) nz = last ? noise_at(a, bw0 + b + 1, 0, j) : noise_at(a, bw0 + b, inner + 1, j);
                reg_step<KPL, true>(a, sm, W, j, act, z, scr_s + ((size_t)b * a.inner_it + inner) * 3 * n);
            }
            if (act) reg_bw_step(a, sm, j);
        }
        // ---- reverse through the segment: lambda_S_E,j += sum_k SC[j][k] lambda_in,k
        W.load(A.sct_f32 + (size_t)a.sc_idx[sim] * n * n, n);
        // the state before the step and its noise, one step ahead of the sweep
        float SE = 0.0f, SI = 0.0f, in = 0.0f;
        auto fetch = [&](int b, int inner) {
            const float *p = scr_s + ((size_t)b * a.inner_it + inner) * 3 * n + j;
            SE = p[0];
            SI = p[n];
            in = p[2 * n];
            nz = noise_at(a, bw0 + b, inner, j);
        };
        if (act) fetch(nb - 1, a.inner_it - 1);
        for (int b = nb - 1; b >= 0; --b) {
            const int bw_i = bw0 + b;
            if (act) {
                double lx = sm.bwl[0][j], lf = sm.bwl[1][j], lnu = sm.bwl[2][j], lq = sm.bwl[3][j];
                const int vol = (bw_i + 1) / a.bold_tr_iters - 1;
                const bool sample = (bw_i + 1) % a.bold_tr_iters == 0 && vol < a.bold_len;
                sm.lE[j] += (float)bw_reverse(lx, lf, lnu, lq, scr_bw[((size_t)b * 4 + 1) * n + j],
                                              scr_bw[((size_t)b * 4 + 2) * n + j], scr_bw[((size_t)b * 4 + 3) * n + j],
                                              sample ? dbold[(size_t)vol * n + j] : 0.0, sample, a);
                sm.bwl[0][j] = lx; sm.bwl[1][j] = lf; sm.bwl[2][j] = lnu; sm.bwl[3][j] = lq;
            }
            for (int inner = a.inner_it - 1; inner >= 0; --inner) {
                if (act) {
                    const float sE = SE, sI = SI, c = in;
                    const float2 z = nz;
                    if (inner > 0) fetch(b, inner - 1);
                    else if (b > 0) fetch(b - 1, a.inner_it - 1);
                    float lE = sm.lE[j], lI = sm.lI[j];
                    const StepGrad d = step_reverse(lE, lI, sE, sI, c, z.x, z.y, smem_params(sm, j), a.Kf.rww);
                    sm.x[j] = d.in;
                    sm.lE[j] = lE;
                    sm.lI[j] = lI;
                    sm.acc[0][j] += (double)d.G;
                    sm.acc[1][j] += (double)d.w_p;
                    sm.acc[2][j] += (double)d.J_N;
                    sm.acc[3][j] += (double)d.wIE;
                    sm.acc[4][j] += (double)d.sigma;
                }
                __syncthreads();
                W.product(sm.x, sm.sums);
                __syncthreads();
                if (act) sm.lE[j] += sm.sums[j];
            }
        }
        __syncthreads();   // sm.x and sm.sums are reused by the next segment
    }
    const double gG = block_sum_d(act ? sm.acc[0][j] : 0.0, red);
    if (j == 0) A.grad_g[sim] = gG;
    if (act) {
        const size_t rs = (size_t)a.n_sims * n, o = (size_t)sim * n + j;
#pragma unroll
        for (int q = 0; q < 4; ++q) A.grad_r[q * rs + o] = sm.acc[q + 1][j];
    }
}

template <int KPL>
cudaError_t launch_reg(const AdjArgs &a, bool forward, cudaStream_t st) {
    const int threads = ((a.ia.nodes + 7) / 8) * 32;
    const size_t smem = sizeof(AdjSmem<KPL>);
    cudaError_t e = forward ? allow_dynamic_smem(k_adj_forward_reg<KPL>) : allow_dynamic_smem(k_adj_backward_reg<KPL>);
    if (e != cudaSuccess) return e;
    if (forward) k_adj_forward_reg<KPL><<<a.sim_count, threads, smem, st>>>(a);
    else k_adj_backward_reg<KPL><<<a.sim_count, threads, smem, st>>>(a);
    return cudaGetLastError();
}
// Compiled extents; false above 208 nodes.
bool launch_reg_any(const AdjArgs &a, bool forward, cudaStream_t st, cudaError_t *e) {
    const int kpl = (a.ia.nodes + 15) / 16;
    if (kpl <= 3) *e = launch_reg<3>(a, forward, st);
    else if (kpl <= 7) *e = launch_reg<7>(a, forward, st);
    else if (kpl <= 10) *e = launch_reg<10>(a, forward, st);
    else if (kpl <= 13) *e = launch_reg<13>(a, forward, st);
    else return false;
    return true;
}

__global__ void k_transpose_sc(const double *sc, float *scf, float *sct, int n_scs, int n) {
    const size_t nn = (size_t)n * n, total = nn * n_scs;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t s = e / nn, r = e % nn;
        const int row = (int)(r / n), col = (int)(r % n);
        const float v = (float)sc[e];
        scf[e] = v;
        sct[s * nn + (size_t)col * n + row] = v;
    }
}

}  // namespace

cudaError_t launch_adjoint_forward(const AdjArgs &a, cudaStream_t st) {
    cudaError_t e;
    if (launch_reg_any(a, true, st, &e)) return e;
    const int threads = ((a.ia.nodes + 31) / 32) * 32;
    k_adj_forward<<<a.sim_count, threads, sizeof(float) * a.ia.nodes, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_backward(const AdjArgs &a, cudaStream_t st) {
    cudaError_t e;
    if (launch_reg_any(a, false, st, &e)) return e;
    const int threads = ((a.ia.nodes + 31) / 32) * 32;
    k_adj_backward<<<a.sim_count, threads, sizeof(float) * 2 * ((a.ia.nodes + 3) & ~3), st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_transpose_sc(const double *sc, float *sc_f32, float *sct_f32, int n_scs, int nodes, cudaStream_t st) {
    k_transpose_sc<<<592, 256, 0, st>>>(sc, sc_f32, sct_f32, n_scs, nodes);
    return cudaGetLastError();
}

}  // namespace cbnm
