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
    int smem = 0, n_pairs = 0, near_k = 1, far_max = 0;
    std::vector<int> pair, blob_at, near, near_cnt, near_min;
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

// Lists of all pairs for tiles of p.tile_src sources; R = float or double.  False where all
// lists exceed max_bytes.
template <class R>
inline bool delay_blobs(DelayPlan &p, int n, const double *sc, const std::vector<int> &delay,
                        const std::vector<std::pair<int, int>> &pairs, size_t max_bytes) {
    const size_t nn = (size_t)n * n;
    const int W = p.window, WS = delay_stride(W);
    p.tiles = (n + p.tile_src - 1) / p.tile_src;
    p.blob.clear();
    p.blob_at.clear();
    p.blob_max = 0;
    const int nh = (n + p.passes - 1) / p.passes;
    std::vector<unsigned> end(nh);
    std::vector<uint16_t> off;
    std::vector<R> w;
    auto up16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    for (const auto &pr : pairs) {
        const double *S = sc + (size_t)pr.first * nn;
        const int *d = delay.data() + (size_t)pr.second * nn;
        for (int pt = 0; pt < p.passes * p.tiles; ++pt) {
            const int pass = pt / p.tiles, t = pt % p.tiles;
            const int s0 = t * p.tile_src, s1 = std::min(n, s0 + p.tile_src), h0 = pass * nh, h1 = std::min(n, h0 + nh);
            off.clear();
            w.clear();
            for (int j = h0; j < h1; ++j) {
                for (int k = s0; k < s1; ++k) {
                    const double v = S[(size_t)k * n + j];
                    if (v == 0.0) continue;
                    off.push_back((uint16_t)((k - s0) * WS + (W - d[(size_t)k * n + j])));
                    w.push_back((R)v);
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
            const size_t bytes = up16(h.w_at + sizeof(R) * w.size()), at = p.blob.size();
            p.blob_at.push_back((int)(at / 16));
            p.blob.resize(at + bytes);
            unsigned char *b = p.blob.data() + at;
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

// Chooses the tile and launch shape and builds the lists.  sc [n_scs][n*n] (row =
// source), delay [n_tables][n*n] steps (>= 1).  As many CTAs per SM as the batch can
// fill while a tile still holds about three entries per target (each target and tile costs
// a read and a write of its sums and half an entry of padding); alone on its SM a CTA
// keeps two tile buffers.  Returns false where the kernel does
// not apply: tiles of under 4 sources, most pairs near, or lists beyond max_bytes.
template <class R>
inline bool build_delay_plan(DelayPlan &p, int n, int n_sims, int n_noise, int sms, const double *sc, const int *sc_of,
                             const std::vector<int> &delay, const std::vector<int> &table_of, int max_delay,
                             size_t max_bytes) {
    p.window = (std::max(max_delay, DELAY_BLOCK) + DELAY_BLOCK - 1) / DELAY_BLOCK * DELAY_BLOCK;
    const auto pairs = delay_pairs(p, n_sims, sc_of, table_of);
    const size_t nn = (size_t)n * n;
    // near lists (d < DELAY_BLOCK) for the steps within a block, by rank q: counted first
    p.near_cnt.assign(p.n_pairs, 0);
    p.near_min.assign(p.n_pairs, DELAY_BLOCK);
    size_t nnz = 0;   // of the fullest pair
    if ((size_t)p.n_pairs * nn > max_bytes) return false;
    std::vector<int> near(n), all(n);
    for (int q = 0; q < p.n_pairs; ++q) {
        const double *S = sc + (size_t)pairs[q].first * nn;
        const int *d = delay.data() + (size_t)pairs[q].second * nn;
        std::fill(near.begin(), near.end(), 0);
        std::fill(all.begin(), all.end(), 0);
        for (int k = 0; k < n; ++k)
            for (int j = 0; j < n; ++j) {
                if (S[(size_t)k * n + j] == 0.0) continue;
                const int dk = d[(size_t)k * n + j];
                ++all[j];
                if (dk >= DELAY_BLOCK) continue;
                ++near[j];
                p.near_min[q] = std::min(p.near_min[q], dk);
            }
        p.near_cnt[q] = *std::max_element(near.begin(), near.end());
        p.far_max = std::max(p.far_max, *std::max_element(all.begin(), all.end()) - p.near_cnt[q]);
        size_t sum = 0;
        for (int c : all) sum += c;
        nnz = std::max(nnz, sum);
    }
    for (int c : p.near_cnt) p.near_k = std::max(p.near_k, c);
    if (p.near_k > std::max(8, p.far_max / 4) || (size_t)p.n_pairs * p.near_k * n * 16 > max_bytes) return false;
    p.near.assign((size_t)p.n_pairs * p.near_k * n, 0);
    p.near_w.assign(p.near.size(), 0.0);
    for (int q = 0; q < p.n_pairs; ++q) {
        const double *S = sc + (size_t)pairs[q].first * nn;
        const int *d = delay.data() + (size_t)pairs[q].second * nn;
        if (p.near_cnt[q] == 0) continue;
        std::fill(near.begin(), near.end(), 0);
        for (int k = 0; k < n; ++k)
            for (int j = 0; j < n; ++j) {
                const double v = S[(size_t)k * n + j];
                const int dk = d[(size_t)k * n + j];
                if (v == 0.0 || dk >= DELAY_BLOCK) continue;
                const size_t at = ((size_t)q * p.near_k + near[j]++) * n + j;
                p.near[at] = k * DELAY_BLOCK + dk;
                p.near_w[at] = v;
            }
    }
    // tile and launch shape
    const int least = (n + 31) / 32 * 32, stride = delay_stride(p.window);
    const bool f64 = sizeof(R) == 8;
    const int rows = (int)(sizeof(R) * n * (DELAY_BLOCK + 1) + 15) & ~15;
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
            if (!delay_blobs<R>(p, n, sc, delay, pairs, max_bytes)) return false;
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
