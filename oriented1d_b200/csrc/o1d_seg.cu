// Segment kernels: configuration and launches (see o1d_seg.cuh).
#include <string.h>

#include <memory>
#include <vector>

#include "o1d_seg.cuh"

namespace o1d {

namespace {

int round_up(int v, int m) { return (v + m - 1) / m * m; }

// Lines of one chunk: pairs of channels per canonical line, and the reach that a tile needs.
struct Chunk {
    int pairs[8];
    int reach_h, reach_w;
};
Chunk chunk_of(const int8_t *chan, int c0, int c1, int K) {
    Chunk k{};
    for (int c = c0; c < c1; c += 2) {
        k.pairs[chan[c]]++;
        if (c + 1 < c1 && chan[c + 1] != chan[c]) k.pairs[chan[c + 1]]++;
    }
    for (int o = 0; o < 8; o++)
        if (k.pairs[o]) {
            // the bodies run all taps of their reach, missing ones with weight zero
            const int rh = kCanonDh[o][kHalf - (K <= 15 ? 7 : 15)], rw = kCanonDw[o][kHalf - (K <= 15 ? 7 : 15)];
            if (abs(rh) > k.reach_h) k.reach_h = abs(rh);
            if (abs(rw) > k.reach_w) k.reach_w = abs(rw);
        }
    return k;
}

constexpr double kPieceCycles = 2.4;         // TMA, per pixel of a tile

double compute_cycles(const Chunk &k, int imgs, int lenh, int lenw, int LT) {
    double sum = 0;
    for (int o = 0; o < 8; o++) {
        const int n = k.pairs[o], per = n ? seg::class_pairs(n) : 1, split = ceil_div(n, per);
        if (!n) continue;
        const int lpg = 32 / per, fr = seg::frame_of(o), kind = seg::kind_of(o);
        const int plen = fr == seg::FR_H ? lenw : lenh, llen = fr == seg::FR_H ? lenh : lenw;
        const int lines = kind == KIND_AXIS ? llen : kind == KIND_DIAG ? lenw + seg::kTD - 1 : ceil_div(llen, seg::kSR);
        const int bl = kind == KIND_SLANT ? seg::kST : kind == KIND_AXIS ? LT : seg::kTD;
        sum += split * (double)ceil_div(imgs * lines, lpg) * ceil_div(plen, bl) * seg::task_cycles(kind, LT);
    }
    return sum / 4;                          // schedulers
}

// Best way to cut the maps for these lines.  Whole maps need no halo (a border of one pixel of zeros is
// enough); maps that do not fit twice are cut along the axis the lines reach least.
bool choose_geo(const Chunk &k, const SegParams &p, int room, int LT, SegGeo *out, double *cycles) {
    double best = 0;
    for (int nth = 1; nth <= 64; nth++) {
        const int TH = ceil_div(p.H, nth);
        if (nth > 1 && TH < 6) break;
        if (ceil_div(p.H, TH) != nth) continue;
        for (int ntw = 1; ntw <= 64; ntw++) {
            const int TW = ceil_div(p.W, ntw);
            if (ntw > 1 && TW < 6) break;
            if (ceil_div(p.W, TW) != ntw) continue;
            SegGeo g{};
            g.nth = nth; g.ntw = ntw; g.TH = TH; g.TW = TW;
            g.halo_h = nth > 1; g.halo_w = ntw > 1;
            g.oh = g.halo_h ? k.reach_h : 1;
            g.ow = g.halo_w ? k.reach_w : 0;
            g.RT = g.halo_h ? TH + 2 * k.reach_h : TH + 2;
            g.P = (g.halo_w ? TW + 2 * k.reach_w : TW + 1) | 1;
            if (g.P > 256 || g.RT > 256) continue;
            g.plo_h = g.halo_h ? -g.oh : -1;
            g.phi_h = g.halo_h ? g.RT - g.oh - 1 : TH;
            g.plo_w = g.halo_w ? -g.ow : -1;
            g.phi_w = g.halo_w ? g.P - g.ow - 1 : TW;
            g.img_bytes = g.RT * g.P * p.px;
            if (round_up(g.img_bytes + p.px, 128) > room) continue;
            g.G = 1;
            if (nth * ntw == 1)              // small maps: enough lines to fill the lanes of twelve warps
                while (g.G < 64 && g.G < p.N && g.G * p.H * p.W < 1024 && 2 * round_up((g.G + 1) * g.img_bytes + p.px, 128) <= room) g.G++;
            g.tile_bytes = g.G * g.img_bytes;
            g.buf_bytes = round_up(g.tile_bytes + p.px, 128);     // ends in a pixel of zeros
            g.nbuf = room / g.buf_bytes;
            if (g.nbuf > seg::kMaxBuf) g.nbuf = seg::kMaxBuf;
            g.items = ceil_div(p.N, g.G) * nth * ntw;
            const double load = kPieceCycles * g.G * g.RT * g.P * (p.px == 64 ? 1.5 : p.px == 48 ? 1.25 : 1.0);
            const double comp = compute_cycles(k, g.G, TH, TW, LT);
            // one buffer: every load is exposed
            const double cyc = (g.nbuf == 1 ? comp + load : comp > load ? comp : load) + 300;
            if (best == 0 || cyc * g.items < best) { best = cyc * g.items; *out = g; *cycles = cyc; }
        }
        if (best != 0 && nth > 4 && TH < 16) break;
    }
    return best != 0;
}

bool same_geo(const SegGeo &a, const SegGeo &b) { return memcmp(&a, &b, sizeof(SegGeo)) == 0; }

// Plan for chunks of `px` bytes and line blocks of LT outputs; the estimated time in *cycles.
bool plan_chunks(const int8_t *chan, SegParams &p, int px, int esize, int LT, int room, int *ngeos, double *cycles) {
    p.px = px;
    p.CC = px / esize;
    p.nruns = 0;
    const int nch = ceil_div(p.C, p.CC);
    int geos = 0;
    double total = 0;
    Chunk prev{};
    std::vector<double> cyc;
    for (int i = 0; i < nch; i++) {
        const int c0 = i * p.CC, c1 = c0 + p.CC < p.C ? c0 + p.CC : p.C;
        const Chunk k = chunk_of(chan, c0, c1, p.K);
        if (p.nruns && memcmp(&k, &prev, sizeof(k)) == 0) {
            p.run[p.nruns - 1].nchunks++;
        } else {
            if (p.nruns == kSegRuns) return false;
            SegGeo g;
            double c;
            if (!choose_geo(k, p, room, LT, &g, &c)) return false;
            int at = 0;
            while (at < geos && !same_geo(p.geo[at], g)) at++;
            if (at == geos) {
                if (geos == kSegGeos) return false;
                p.geo[geos++] = g;
            }
            p.run[p.nruns++] = SegRun{i, 1, at, 0, 0};
            cyc.push_back(c);
            prev = k;
        }
        total += cyc.back() * p.geo[p.run[p.nruns - 1].geo].items;
    }
    p.total_cost = 0;
    for (int r = 0; r < p.nruns; r++) {
        p.run[r].cost = (int)(cyc[r] / 16) + 1;
        p.total_cost += (long long)p.run[r].cost * p.geo[p.run[r].geo].items * seg::kParts * p.run[r].nchunks;
    }
    *ngeos = geos;
    *cycles = total;
    return true;
}

bool make_config(const int8_t *chan, int N, int H, int W, int C, int K, int esize, int smem_optin, int sms, bool wgrad, SegConfig *cfg) {
    if (C % 8 != 0 || K > kMaxTaps) return false;
    // Pairs of channels on different lines are computed twice and stored by halves: at most one pair in four.
    // Patchy layers (one pair in eight, or less than six channels in a row on a line) are taken, but behind the
    // tiled kernels where those are at their best: each line of a chunk is a body of its own.
    int mixed = 0, lines = 1;
    for (int c = 0; c + 1 < C; c++) {
        if (chan[c] == chan[c + 1]) continue;
        lines++;
        if (c % 2 == 0) mixed++;
    }
    if (mixed * 8 > C) return false;
    const int tail = round_up((int)sizeof(seg::Tables), 16) + 12 * seg::kMaxBuf + 128;
    const int room = smem_optin - round_up(seg::kPadBytes, 128) - tail;
    double best = 0;
    for (int px = 32; px <= 64; px += 16)
        for (int LT = 14; LT <= 28; LT += 14) {
            SegConfig t{};
            t.p.N = N; t.p.H = H; t.p.W = W; t.p.C = C; t.p.K = K;
            double cyc;
            if (!plan_chunks(chan, t.p, px, esize, LT, room, &t.ngeos, &cyc)) continue;
            if (best == 0 || cyc < best) { best = cyc; t.line_block = LT; *cfg = t; }
        }
    if (best == 0) return false;
    SegParams &p = cfg->p;
    int bytes = 0;
    long long items = 0;
    for (int i = 0; i < cfg->ngeos; i++)
        if (p.geo[i].nbuf * p.geo[i].buf_bytes > bytes) bytes = p.geo[i].nbuf * p.geo[i].buf_bytes;
    for (int r = 0; r < p.nruns; r++) items += (long long)p.run[r].nchunks * p.geo[p.run[r].geo].items;
    if (wgrad && bytes < seg::kWarps * 32 * seg::kMaxPairs * 8) bytes = seg::kWarps * 32 * seg::kMaxPairs * 8;   // sums over warps
    p.off_tile = round_up(seg::kPadBytes, 128);
    p.off_tab = p.off_tile + bytes;
    p.off_bar = p.off_tab + round_up((int)sizeof(seg::Tables), 16);
    cfg->patchy = lines * 6 > C || mixed * 16 > C;
    cfg->esize = esize;
    cfg->short_reach = K <= 15;
    cfg->smem_bytes = p.off_bar + 12 * seg::kMaxBuf;
    cfg->grid = items * 4 < sms ? (int)items * 4 : sms;          // no CTA with less than a quarter item
    // CTAs per chunk in proportion to cost, where that comes out even enough
    const int nch = ceil_div(C, p.CC);
    p.per_chunk = nch * 3 <= cfg->grid;
    if (p.per_chunk) {
        int left = cfg->grid;
        double worst = 0;
        auto load = [&](int r) { return (double)p.run[r].cost * p.geo[p.run[r].geo].items; };
        for (int r = 0; r < p.nruns; r++) {
            p.run[r].ctas = (int)(load(r) * seg::kParts * cfg->grid / p.total_cost);
            if (p.run[r].ctas < 1) p.run[r].ctas = 1;
            left -= p.run[r].ctas * p.run[r].nchunks;
        }
        while (left > 0) {               // the rest to the slowest runs
            int at = -1;
            for (int r = 0; r < p.nruns; r++)
                if (p.run[r].nchunks <= left && (at < 0 || load(r) / p.run[r].ctas > load(at) / p.run[at].ctas)) at = r;
            if (at < 0) break;
            p.run[at].ctas++;
            left -= p.run[at].nchunks;
        }
        for (int r = 0; r < p.nruns; r++)
            if (load(r) / p.run[r].ctas > worst) worst = load(r) / p.run[r].ctas;
        const double even = (double)p.total_cost / seg::kParts / cfg->grid;
        if (left < 0 || worst > 1.3 * even) p.per_chunk = 0;
        else cfg->grid -= left;
    }
    return cfg->smem_bytes <= smem_optin;
}

// Configurations of the last requests of this thread (they depend on the shape and the lines only).  A
// classifier has about 20 per image size, so that a loader of two dozen sizes finds its own again; an entry
// takes 1 KB and a byte per channel.
struct Key {
    int N, H, W, C, K, esize, smem, sms, wgrad;
    bool operator==(const Key &o) const { return memcmp(this, &o, sizeof(Key)) == 0; }
};
struct Entry {
    Key key;
    bool taken;
    std::vector<int8_t> chan;
    SegConfig cfg;
};
constexpr size_t kKept = 512;
uint64_t hash_of(const Key &k) {                 // FNV-1a
    const int v[] = {k.N, k.H, k.W, k.C, k.K, k.esize, k.smem, k.sms, k.wgrad};
    uint64_t h = 1469598103934665603ull;
    for (int x : v) h = (h ^ (uint32_t)x) * 1099511628211ull;
    return h;
}

}  // namespace

bool seg_configure(const int8_t *chan, int N, int H, int W, int C, int K, int esize, int smem_optin, int sms, bool wgrad,
                   SegConfig **cfg) {
    thread_local std::vector<std::unique_ptr<Entry>> kept;
    thread_local std::vector<uint64_t> hashes;   // of the entries, side by side
    thread_local size_t oldest = 0;
    const Key key{N, H, W, C, K, esize, smem_optin, sms, wgrad};
    const uint64_t hash = hash_of(key);
    for (size_t i = 0; i < hashes.size(); i++)
        if (hashes[i] == hash && kept[i]->key == key && memcmp(kept[i]->chan.data(), chan, C) == 0) {
            *cfg = &kept[i]->cfg;
            return kept[i]->taken;
        }
    auto e = std::make_unique<Entry>();
    e->key = key;
    e->chan.assign(chan, chan + C);
    e->taken = make_config(chan, N, H, W, C, K, esize, smem_optin, sms, wgrad, &e->cfg);
    *cfg = &e->cfg;
    const bool taken = e->taken;
    if (kept.size() < kKept) {
        kept.push_back(std::move(e));
        hashes.push_back(hash);
    } else {                                     // a full cache gives up its entries in turn
        kept[oldest] = std::move(e);
        hashes[oldest] = hash;
        oldest = (oldest + 1) % kKept;
    }
    return taken;
}

namespace {
struct Args {
    const SegMaps *maps, *dy_maps;
    const void *w, *bias;
    int wbf16;
    const int8_t *chan;
    void *y;
    float *partial;
    int *err_flag;
    SegParams p;
    cudaStream_t st;
};
template <typename T, int R, int LT, bool WG, bool MERGED> cudaError_t launch(const SegConfig &cfg, const Args &a) {
    auto kern = seg::seg_kernel<T, R, LT, WG, MERGED>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cfg.smem_bytes);
    if (e != cudaSuccess) return e;
    kern<<<cfg.grid, seg::kThreads, cfg.smem_bytes, a.st>>>(*a.maps, *a.dy_maps, a.w, a.bias, a.wbf16, a.chan, (T *)a.y, a.partial,
                                                            a.err_flag, a.p);
    return cudaGetLastError();
}
template <typename T, bool WG, bool MERGED> cudaError_t launch_any(const SegConfig &cfg, const Args &a) {
    if (cfg.short_reach) return cfg.line_block == 28 ? launch<T, 7, 28, WG, MERGED>(cfg, a) : launch<T, 7, 14, WG, MERGED>(cfg, a);
    return cfg.line_block == 28 ? launch<T, 15, 28, WG, MERGED>(cfg, a) : launch<T, 15, 14, WG, MERGED>(cfg, a);
}
}  // namespace

cudaError_t seg_launch_conv(const SegConfig &cfg, const SegMaps &maps, const void *w, const void *bias, int wbf16,
                            const int8_t *chan, void *y, int flip, int identity, int order, int *err_flag, cudaStream_t st) {
    Args a{&maps, &maps, w, bias, wbf16, chan, y, nullptr, err_flag, cfg.p, st};
    a.p.flip = flip;
    a.p.identity = identity;
    if (cfg.esize == 4) return launch_any<float, false, true>(cfg, a);
    return order == SEG_ASCENDING ? launch_any<__nv_bfloat16, false, false>(cfg, a) : launch_any<__nv_bfloat16, false, true>(cfg, a);
}

size_t seg_wgrad_bytes(const SegConfig &cfg) {
    const int slots = cfg.grid + (cfg.p.per_chunk ? 0 : ceil_div(cfg.p.C, cfg.p.CC));
    return (size_t)slots * cfg.p.CC * 32 * sizeof(float);
}

cudaError_t seg_launch_wgrad(const SegConfig &cfg, const SegMaps &maps, const SegMaps &dy_maps, const int8_t *chan, const void *dy,
                             void *dw, void *db, int out_bf16, float *partial, int *err_flag, cudaStream_t st) {
    Args a{&maps, &dy_maps, nullptr, nullptr, 0, chan, const_cast<void *>(dy), partial, err_flag, cfg.p, st};
    const cudaError_t e = cfg.esize == 4 ? launch_any<float, true, true>(cfg, a) : launch_any<__nv_bfloat16, true, true>(cfg, a);
    if (e != cudaSuccess) return e;
    seg::seg_wgrad_final_kernel<<<dim3(ceil_div(cfg.p.C, cfg.p.CC), ceil_div(cfg.p.CC * 32, 256)), 256, 0, st>>>(partial, chan, dw, db, out_bf16, cfg.grid, cfg.p);
    return cudaGetLastError();
}

}  // namespace o1d
