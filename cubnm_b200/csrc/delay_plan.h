// Host side of the delay kernel (integrate_delay.cuh): its tiles and entry lists.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <map>
#include <utility>
#include <vector>

namespace cbnm {

constexpr int DELAY_BLOCK = 32;          // integration steps per block of the kernel
constexpr int DELAY_SMEM_SM = 227 * 1024;   // shared memory of an SM that CTAs can use, and 1 KB of it per CTA is the system's

struct DelayPlan {
    int window = 0, tiles = 0, tile_src = 0, bufs = 1, threads = 0, blob_max = 0, buf_bytes = 0, passes = 1, buf_at = 0, noise_at = 0, noise_steps = 0;
    int smem = 0, n_pairs = 0, near_k = 1;
    std::vector<int> sims, pair;   // the simulations that run on the kernel, and each one's pair (as all of [n_sims])
    std::vector<int> rest;         // the others: their pair is not for it
    std::vector<int> blob_at, near, near_cnt, near_min;
    std::vector<unsigned char> blob;
    std::vector<double> near_w;
};

// The pairs (SC, delay table) that the simulations use.
inline std::vector<std::pair<int, int>> delay_pairs(DelayPlan &p, int n_sims, const int *sc_of,
                                                    const std::vector<int> &table_of) {
    std::map<std::pair<int, int>, int> id;
    std::vector<std::pair<int, int>> pairs;
    p.pair.resize(n_sims);
    for (int s = 0; s < n_sims; ++s) {
        const auto key = std::make_pair(sc_of[s], table_of[s]);
        const auto it = id.emplace(key, (int)pairs.size());
        if (it.second) pairs.push_back(key);
        p.pair[s] = it.first->second;
    }
    p.n_pairs = (int)pairs.size();
    return pairs;
}

// Words between the windows of two sources in shared memory: a window of p.window steps
// before the block, then DELAY_BLOCK zeros, where the lanes b >= d of a pair with
// d < DELAY_BLOCK read (their values are not there yet; the step loop adds them).
inline int delay_stride(int window) { return window + DELAY_BLOCK; }

// A tile's entry lists (per pass over the targets), 16-byte aligned: this header, unsigned
// end[targets] (pairs of entries up to and with the target's), then at the byte offsets
// given the offsets of x(t0 - d) in the tile's windows (16 bits each, a target's padded to a
// pair by repeating one with weight 0) and the weights.  A target's sources are in ascending
// order, so that its sum over all tiles is one chain in that order whatever the tiles are.
struct TileHead { int off_at, w_at, unused[2]; };

// The nonzeros of one SC by target, sources ascending; loaded again only when the SC changes,
// so that many delay tables of one SC are walked by their entries, not by all n x n.
struct DelayColumns {
    int loaded = -1;
    int full = 0;               // most sources of a target
    std::vector<int> at, src;   // target j: entries at[j] .. at[j + 1]
    std::vector<double> w;
    void load(const double *sc, int id, int n) {
        if (id == loaded) return;
        loaded = id;
        const double *S = sc + (size_t)id * n * n;
        at.assign(n + 1, 0);
        for (int k = 0; k < n; ++k)
            for (int j = 0; j < n; ++j) at[j + 1] += S[(size_t)k * n + j] != 0.0;
        full = *std::max_element(at.begin(), at.end());
        for (int j = 0; j < n; ++j) at[j + 1] += at[j];
        src.resize(at[n]);
        w.resize(at[n]);
        std::vector<int> next(at.begin(), at.end() - 1);
        for (int k = 0; k < n; ++k)
            for (int j = 0; j < n; ++j) {
                const double v = S[(size_t)k * n + j];
                if (v == 0.0) continue;
                src[next[j]] = k;
                w[next[j]++] = v;
            }
    }
};

// Lists of all pairs for tiles of p.tile_src sources; R = float or double.  False where all
// lists exceed max_bytes.
template <class R>
inline bool delay_blobs(DelayPlan &p, int n, const double *sc, const std::vector<int> &delay,
                        const std::vector<std::pair<int, int>> &pairs, DelayColumns &cols, size_t max_bytes) {
    const size_t nn = (size_t)n * n;
    const int W = p.window, WS = delay_stride(W);
    p.tiles = (n + p.tile_src - 1) / p.tile_src;
    p.blob.clear();
    p.blob_at.clear();
    p.blob_max = 0;
    const int nh = (n + p.passes - 1) / p.passes;
    std::vector<unsigned> end(nh);
    std::vector<int> at(nh);   // a target's next entry: tiles take them in order
    std::vector<uint16_t> off;
    std::vector<R> w;
    auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    for (const auto &pr : pairs) {
        cols.load(sc, pr.first, n);
        const int *d = delay.data() + (size_t)pr.second * nn;
        for (int pt = 0; pt < p.passes * p.tiles; ++pt) {
            const int pass = pt / p.tiles, t = pt % p.tiles;
            const int s0 = t * p.tile_src, s1 = std::min(n, s0 + p.tile_src), h0 = pass * nh, h1 = std::min(n, h0 + nh);
            if (t == 0) std::copy(cols.at.begin() + h0, cols.at.begin() + h1, at.begin());
            off.clear();
            w.clear();
            for (int j = h0; j < h1; ++j) {
                int &e = at[j - h0];
                for (; e < cols.at[j + 1] && cols.src[e] < s1; ++e) {
                    const int k = cols.src[e];
                    off.push_back((uint16_t)((k - s0) * WS + (W - d[(size_t)k * n + j])));
                    w.push_back((R)cols.w[e]);
                }
                if (off.size() % 2) {
                    off.push_back(off.back());
                    w.push_back(R(0));
                }
                end[j - h0] = (unsigned)(off.size() / 2);
            }
            TileHead h{};
            h.off_at = (int)up16(sizeof(h) + sizeof(unsigned) * nh);
            h.w_at = (int)up16(h.off_at + sizeof(uint16_t) * off.size());
            const size_t bytes = up16(h.w_at + sizeof(R) * w.size()), to = p.blob.size();
            p.blob_at.push_back((int)(to / 16));
            p.blob.resize(to + bytes);
            unsigned char *b = p.blob.data() + to;
            std::memcpy(b, &h, sizeof(h));
            std::memcpy(b + sizeof(h), end.data(), sizeof(unsigned) * (h1 - h0));
            if (!off.empty()) {
                std::memcpy(b + h.off_at, off.data(), sizeof(uint16_t) * off.size());
                std::memcpy(b + h.w_at, w.data(), sizeof(R) * w.size());
            }
            p.blob_max = std::max(p.blob_max, (int)bytes);
            if (p.blob.size() > max_bytes) return false;
            if (t == p.tiles - 1) p.blob_at.push_back((int)(p.blob.size() / 16));
        }
    }
    return true;
}

// Whether a pair's simulations are for the kernel, by its longest near list and most sources
// of a target: in FP32 up to a quarter near (and 8 in any case), in FP64 up to 0.56.  The
// step loop takes an entry of the near list at a time from L1 or L2, 400 and more cycles
// where a barrier is due every step, and the per-step kernel all sources at once.  ms per
// simulated second, 148 simulations, delay / per-step kernel (velocity in m/s: near of all):
// FP32 200 nodes, 30 %: 12 (10 of 89) 23.5 / 55, 15 (14 of 93) 29 / 51, 20 (31 of 102) 71 / 46,
// 40 (69 of 102) 141 / 39; FP32 1,000 nodes, 10 %: 15 (33 of 156) 151 / 247; FP64 200 nodes: 20
// 47 / 95, 30 (58 of 113) 75 / 92, 40 86 / 90; FP64 400 nodes, 20 %: 40 (99 of 137) 139 / 128.
template <class R>
inline bool delay_pair_fits(int near, int all) {
    return near <= std::max(8.0, (sizeof(R) == 4 ? 0.25 : 0.56) * all);
}

// Chooses the simulations that run on the kernel, the tile and launch shape, and builds the
// lists.  sc [n_scs][n*n] (row = source), delay [n_tables][n*n] steps (>= 1).  A pair (SC,
// delay table) is taken if delay_pair_fits and its windows leave tiles of at least 4 sources,
// whatever else is in the batch.  As many CTAs per SM as the batch can
// fill while a tile still holds about three entries per target (each target and tile costs
// a read and a write of its sums and half an entry of padding); alone on its SM a CTA
// keeps two tile buffers.  Returns false where no simulation is taken, the lists exceed
// max_bytes (counted before they are built), or of a batch larger than the GPU's SMs most
// are not taken: the two kernels then run one after the other, and what is left of the
// per-step kernel's batch takes about as long as all of it (FP32, 500 simulations of 68 nodes
// at 10-60 m/s: 45 ms per simulated second in two, 33 on the per-step kernel).
template <class R>
inline bool build_delay_plan(DelayPlan &p, int n, int n_sims, int n_noise, int sms, const double *sc, const int *sc_of,
                             const std::vector<int> &delay, const std::vector<int> &table_of, size_t max_bytes) {
    std::vector<std::pair<int, int>> pairs = delay_pairs(p, n_sims, sc_of, table_of);
    const size_t nn = (size_t)n * n;
    const int rows = (int)(sizeof(R) * n * (DELAY_BLOCK + 1) + 15) & ~15;
    // sums of half the targets where two passes over them are possible
    const double least_rows = sizeof(R) == 4 && n > 512 ? rows / 2 : rows;
    // near lists (d < DELAY_BLOCK) for the steps within a block, by rank q: counted first
    std::vector<int> new_id(pairs.size(), -1);
    std::vector<std::pair<int, int>> taken;
    DelayColumns cols;
    size_t nnz = 0, entries = 0;   // of the fullest pair, of all
    int max_delay = 1;
    for (size_t q = 0; q < pairs.size(); ++q) {
        cols.load(sc, pairs[q].first, n);
        const int *d = delay.data() + (size_t)pairs[q].second * nn;
        int least = DELAY_BLOCK, most = 1, cnt = 0;
        for (int j = 0; j < n && delay_pair_fits<R>(cnt, cols.full); ++j) {
            int near = 0;
            for (int e = cols.at[j]; e < cols.at[j + 1]; ++e) {
                const int dk = d[(size_t)cols.src[e] * n + j];
                most = std::max(most, dk);
                near += dk < DELAY_BLOCK;
                least = std::min(least, dk);
            }
            cnt = std::max(cnt, near);
        }
        const int stride = delay_stride((most + DELAY_BLOCK - 1) / DELAY_BLOCK * DELAY_BLOCK), few = std::min(n, 4);
        const double bytes = least_rows + n * (4 + 0.6 * (2 + sizeof(R))) + 2048 +
                             few * (stride * (double)sizeof(R) + 1.2 * cols.full * (2 + sizeof(R)));
        if (!delay_pair_fits<R>(cnt, cols.full) || bytes > DELAY_SMEM_SM || few * (long long)stride > 65535) continue;
        new_id[q] = (int)taken.size();
        taken.push_back(pairs[q]);
        p.near_cnt.push_back(cnt);
        p.near_min.push_back(least);
        p.near_k = std::max(p.near_k, cnt);
        max_delay = std::max(max_delay, most);
        nnz = std::max(nnz, cols.src.size());
        entries += cols.src.size();
    }
    for (int s = 0; s < n_sims; ++s) {
        p.pair[s] = new_id[p.pair[s]];
        (p.pair[s] >= 0 ? p.sims : p.rest).push_back(s);
    }
    p.n_pairs = (int)taken.size();
    pairs = taken;
    if (p.sims.empty() || entries * (2 + sizeof(R)) > max_bytes || (size_t)p.n_pairs * p.near_k * n * 16 > max_bytes) return false;
    if (n_sims > sms && 2 * p.rest.size() > (size_t)n_sims) return false;
    n_sims = (int)p.sims.size();
    p.window = (max_delay + DELAY_BLOCK - 1) / DELAY_BLOCK * DELAY_BLOCK;
    p.near.assign((size_t)p.n_pairs * p.near_k * n, 0);
    p.near_w.assign(p.near.size(), 0.0);
    for (int q = 0; q < p.n_pairs; ++q) {
        if (p.near_cnt[q] == 0) continue;
        cols.load(sc, pairs[q].first, n);
        const int *d = delay.data() + (size_t)pairs[q].second * nn;
        for (int j = 0; j < n; ++j) {
            int rank = 0;
            for (int e = cols.at[j]; e < cols.at[j + 1]; ++e) {
                const int k = cols.src[e], dk = d[(size_t)k * n + j];
                if (dk >= DELAY_BLOCK) continue;
                const size_t to = ((size_t)q * p.near_k + rank++) * n + j;
                p.near[to] = k * DELAY_BLOCK + dk;
                p.near_w[to] = cols.w[e];
            }
        }
    }
    // tile and launch shape
    const int least = (n + 31) / 32 * 32, stride = delay_stride(p.window);
    const bool f64 = sizeof(R) == 8;
    const double nnz_node = (double)nnz / n;
    const int thr_sm = f64 ? 512 : 1024;   // by registers, see min_ctas
    const int step_bytes = (int)sizeof(R) * n * n_noise;   // noise of a step
    for (int c = std::min({8, (n_sims + sms - 1) / sms, std::max(1, thr_sm / least)}); c >= 1; --c) {
        const int most_smem = DELAY_SMEM_SM / c - 1024;
        auto fit = [&](int bufs) {   // sources whose windows and entries, with row ends and padding, fill a buffer
            const double fixed = (double)n / p.passes * (4 + 0.6 * (2 + sizeof(R))) + 512;
            const double src = (double)stride * sizeof(R) + nnz_node / p.passes * 1.1 * (2 + sizeof(R));
            return std::min<int>({n, 65535 / stride, (int)(((most_smem - p.buf_at) / bufs - fixed) / src)});
        };
        p.bufs = p.passes = 1;
        p.buf_at = p.noise_at = rows;
        p.tile_src = fit(1);
        if (p.tile_src < n && c == 1 && nnz_node * fit(2) / n >= 12.0) {   // alone on its SM: load during the gather
            p.bufs = 2;
            p.tile_src = fit(2);
        }
        if (c > 1 && p.tile_src < n && nnz_node * p.tile_src / n < 3.0) continue;
        if (!f64 && n > 512 && c == 1 && p.tile_src < n && nnz_node * p.tile_src / n < 6.0 &&
             most_smem - rows >= 4 * (step_bytes + (int)sizeof(R) * n)) {
            p.passes = 2;                          // half the sums, larger tiles; then at least 4 steps of noise and sums
            p.buf_at = ((int)sizeof(R) * ((n + 1) / 2) * (DELAY_BLOCK + 1) + 15) & ~15;
            p.tile_src = fit(1);
        }
        if (p.tile_src < std::min(n, 4)) continue;
        const int most = c == 1 ? (f64 ? 512 : n <= 256 ? 512 : 1024) : std::min(f64 ? 256 : 512, thr_sm / c / 32 * 32);
        p.threads = std::max(least, most);
        for (int shrink = 0; shrink < 8 && p.tile_src >= 1; ++shrink) {
            if (!delay_blobs<R>(p, n, sc, delay, pairs, cols, max_bytes)) return false;
            p.buf_bytes = ((p.blob_max + p.tile_src * stride * (int)sizeof(R)) + 15) & ~15;
            p.smem = p.buf_at + p.bufs * p.buf_bytes;
            if (p.smem <= most_smem) {
                if (p.passes == 2) p.smem = most_smem & ~15;
                p.noise_steps = std::min(DELAY_BLOCK, (p.smem - p.noise_at - 16) / (step_bytes + (p.passes == 2 ? (int)sizeof(R) * ((n + 3) & ~3) : 0)));
                return p.noise_steps > 0;
            }
            p.tile_src = (int)(p.tile_src * 0.93);
        }
    }
    return false;
}

}  // namespace cbnm
