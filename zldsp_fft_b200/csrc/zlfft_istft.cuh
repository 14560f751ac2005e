// G9: inverse STFT with overlap-add, the backward-side counterpart of the STFT
// front end. Per frame f (bins X_f, N_c + 1 of them, N_c = 2^P):
//
//     x_f = RFFT::backward(H * X_f)                      (2 N_c reals)
//     y[f hop + n] += w[n] x_f[n],   f = 0, 1, ... in order
//
// with an optional spectral filter H (N_c + 1 bins, each complex product
// rounded operation by operation) and an optional synthesis window w. The
// inverse transform is the tile kernel's backward RFFT
// (src/common/zldsp_fft_common_execute.hpp:399-451 pre-step, then the
// swap-based backward CFFT), so x_f carries the reference's bits. With H
// the identity, the spectrum of a fast convolution, or an STFT's bins, the
// launch is inverse-STFT synthesis or overlap-add convolution.
//
// Determinism: the output is cut into blocks of `hop` reals; block m takes
// frames m - K + 1 .. m (K = 2 N_c / hop). Each CTA owns a run of consecutive
// blocks and transforms its frames in ascending order into a ring of K blocks
// in shared memory, beginning K - 1 frames before its first block (those
// frames' contributions to earlier blocks are dropped). After frame f, block
// f holds its final sum, is written once, and its ring slots are cleared for
// block f + K. Every output real is thus the sum of its frames' terms in
// ascending frame order, from zero, one rounding per term, whatever the grid:
// the same value as a sequential loop over frames, with no atomics.
#pragma once

#include "zlfft_launch.cuh"

namespace zlfft {

struct IstftArgs {
    const void* filt;    // H: N_c + 1 complex bins (null: none)
    const void* win;     // w: 2 N_c reals (null: none)
    void* sig;           // y: (n_frames - 1) * hop + 2 N_c reals
    long long n_frames;
    long long hop;       // reals: even, divides 2 N_c
    long long blocks;    // output blocks of hop reals: n_frames + K - 1
    long long run;       // blocks per CTA (set by the launch)
    int k;               // K: frames that overlap one block
};

// Last-group sink of the backward RFFT (TileWorker::run): adds the windowed
// sample pair (2 pos, 2 pos + 1) of frame f to the ring, whose slot for real
// sample j of the output is (j / 2) mod N_c.
template <typename F>
struct OlaSink {
    using C = Cx<F>;
    static constexpr bool kActive = true;
    const C* h;      // spectral filter (read by the pre-step)
    const C* w;      // synthesis window pairs
    bool has_h, has_w;
    C* ring;         // shared memory, N_c pairs
    uint32_t base;   // (f * hop / 2) mod N_c
    uint32_t mask;   // N_c - 1
    __device__ __forceinline__ bool filtered() const { return has_h; }
    __device__ __forceinline__ C filter(int k) const { return h[k]; }
    __device__ __forceinline__ void add(int pos, C x) const {
        if (has_w) {
            const C ww = w[pos];
            x = cx<C>(mul_rn(x.x, ww.x), mul_rn(x.y, ww.y));
        }
        C& r = ring[(base + (uint32_t)pos) & mask];
        r = cx<C>(add_rn(r.x, x.x), add_rn(r.y, x.y));
    }
};

// One CTA per SM of GROUPS groups of T threads, each a worker of its own: an
// exchange buffer, a ring and a run of blocks. What the groups share is the
// tables in shared memory, one copy per SM: the transform's middle twiddles
// and split twiddles, the filter and the window, as many as fit without
// costing a group. (A CTA per group, reading all four from global memory:
// 1420 us for 131069 frames of order 12 at hop N / 4 against 1365, 319 against
// 289 for 4096 frames of order 14. A copy per CTA would not fit.) The bins are
// read directly: staging them costs a group.
//
// Where every group transforms one frame and few of them share an SM, copying
// the tables costs more than it saves, and a CTA is one group that reads them
// from global memory (SHARED false; istft_single).
template <typename F, int P, bool SHARED>
struct IstftCfg {
    using C = Cx<F>;
    static constexpr int N = 1 << P;                  // complex points (frame length / 2)
    static constexpr int T = N / tile_elems(P);       // threads per transform
    using Tile = TileCfg<F, P, kC2RBwd, (T > 0 ? T : 1)>;
    static constexpr size_t RING = Tile::XBYTES;                    // a group's ring, behind its exchange
    static constexpr size_t GBYTES = RING + (size_t)N * sizeof(C);  // bytes of a group
    // whole warps, and the exchange and ring in shared memory
    static constexpr bool kOK = T >= 32 && Tile::TPC == 1 && GBYTES <= 200 * 1024;
    static_assert(!kOK || Tile::THREADS == T, "one transform per group of T threads");
    static constexpr size_t kSm = 226 * 1024;
    static constexpr int REGS = sizeof(F) == 4 && P <= 11 ? 96 : 128;
    static constexpr int by_regs = 65536 / (REGS * (T > 0 ? T : 1)), by_smem = (int)(kSm / GBYTES);
    static constexpr int G0 = by_regs < by_smem ? by_regs : by_smem;
    static constexpr int G1 = G0 > 1024 / (T > 0 ? T : 1) ? 1024 / (T > 0 ? T : 1) : G0;
    static constexpr int GROUPS = !SHARED ? 1 : T > 32 && G1 > 15 ? 15 : (G1 > 0 ? G1 : 1);
    static constexpr int THREADS = T * GROUPS;
    static constexpr size_t BASE = GBYTES * GROUPS;
    static constexpr size_t cxs = sizeof(C);
    static constexpr size_t mid_b = Tile::TW_MID * cxs, rw_b = ((N / 2 + 1) * cxs + 15) / 16 * 16,
                            h_b = ((N + 1) * cxs + 15) / 16 * 16, w_b = N * cxs;
    static constexpr bool kMid = SHARED && BASE + mid_b <= kSm;
    static constexpr size_t O_MID = BASE, O_RW = O_MID + (kMid ? mid_b : 0);
    static constexpr bool kRw = SHARED && O_RW + rw_b <= kSm;
    static constexpr size_t O_H = O_RW + (kRw ? rw_b : 0);
    static constexpr bool kH = SHARED && O_H + h_b <= kSm;
    static constexpr size_t O_W = O_H + (kH ? h_b : 0);
    static constexpr bool kW = SHARED && O_W + w_b <= kSm;
    static constexpr size_t SMEM = O_W + (kW ? w_b : 0);
    static constexpr int TABS = (kMid ? kTabMid : 0) | (kRw ? kTabRw : 0);
    static constexpr int MINB = SHARED ? 1 : Tile::MINB;
};

template <typename F, int P, int IL, bool SHARED>
__global__ void __launch_bounds__(IstftCfg<F, P, SHARED>::THREADS, IstftCfg<F, P, SHARED>::MINB)
    istft_kernel(const TileArgs a, const IstftArgs o) {
    using Cfg = IstftCfg<F, P, SHARED>;
    using C = Cx<F>;
    using W = TileWorker<F, P, kC2RBwd, IL, kAoS, Cfg::T, false, false, false, false, 0, 1, Cfg::TABS, SHARED>;
    constexpr int N = Cfg::N, T = Cfg::T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int grp = (int)threadIdx.x / T, lt = (int)threadIdx.x % T;
    C* t_mid = reinterpret_cast<C*>(smem_raw + Cfg::O_MID);
    C* t_rw = reinterpret_cast<C*>(smem_raw + Cfg::O_RW);
    C* t_h = reinterpret_cast<C*>(smem_raw + Cfg::O_H);
    C* t_w = reinterpret_cast<C*>(smem_raw + Cfg::O_W);
    if constexpr (Cfg::kMid) copy_table(t_mid, static_cast<const C*>(a.tws), Cfg::Tile::TW_MID);
    if constexpr (Cfg::kRw) copy_table(t_rw, static_cast<const C*>(a.rw), N / 2 + 1);
    W wk(a, smem_raw + (size_t)grp * Cfg::GBYTES, t_mid, t_rw);
    C* ring = reinterpret_cast<C*>(smem_raw + (size_t)grp * Cfg::GBYTES + Cfg::RING);
    C* sig = static_cast<C*>(o.sig);
    const long long hp = o.hop / 2;  // hop in sample pairs
    const C zero = cx<C>((F)0, (F)0);
    for (int i = lt; i < N; i += T) ring[i] = zero;
    pdl_wait();
    pdl_trigger();
    const long long m0 = ((long long)grp * gridDim.x + blockIdx.x) * o.run;
    const long long m1 = (m0 + o.run < o.blocks) ? m0 + o.run : o.blocks;
    const long long f0 = (m0 - o.k + 1 > 0) ? m0 - o.k + 1 : 0;
    const long long f1 = (m1 - 1 < o.n_frames - 1) ? m1 - 1 : o.n_frames - 1;
    // The bins come from HBM with nothing else to do meanwhile: one thread asks
    // L2 for the next frame's before this one is transformed (1639 -> 1365 us for
    // 131069 frames of order 12 at hop N / 4; with it the shared tables are worth
    // 4% there, without it nothing). A CTA of one group and one frame only asks
    // where it is a single warp (order 10, 74 frames 6.3 us against 7.9; order 13
    // 7.4 against 6.1).
    auto prefetch = [&](long long f) {
        if ((!SHARED && T > 32) || lt != 0 || f > f1 || m0 >= m1) return;
        if constexpr (IL == kSoA) {
            prefetch_l2(static_cast<const F*>(a.in0) + f * a.in_stride, (N + 1) * sizeof(F));
            prefetch_l2(static_cast<const F*>(a.in1) + f * a.in_stride, (N + 1) * sizeof(F));
        } else {
            prefetch_l2(static_cast<const C*>(a.in0) + f * a.in_stride, (N + 1) * sizeof(C));
        }
    };
    prefetch(f0);
    if (Cfg::kH && o.filt) copy_table(t_h, static_cast<const C*>(o.filt), N + 1);
    if (Cfg::kW && o.win) copy_table(t_w, static_cast<const C*>(o.win), N);
    __syncthreads();
    if (m0 >= m1) return;  // (the groups meet at no barrier from here on)
    OlaSink<F> sink{Cfg::kH ? t_h : static_cast<const C*>(o.filt), Cfg::kW ? t_w : static_cast<const C*>(o.win),
                    o.filt != nullptr, o.win != nullptr, ring, 0u, (uint32_t)(N - 1)};
    for (long long f = f0; f <= f1; ++f) {
        prefetch(f + 1);
        sink.base = (uint32_t)((f * hp) & (N - 1));
        wk.run(a, f, false, [] {}, sink);  // ends with a barrier: the frame is in the ring
        // block f is final: write it when this group owns it, clear its slots
        for (long long i = lt; i < hp; i += T) {
            const uint32_t r = (uint32_t)((f * hp + i) & (N - 1));
            if (f >= m0) sig[f * hp + i] = ring[r];
            ring[r] = zero;
        }
        wk.sync();
    }
    // blocks after the last frame are final once every frame is in
    for (long long m = (f1 + 1 > m0 ? f1 + 1 : m0); m < m1; ++m)
        for (long long i = lt; i < hp; i += T) sig[m * hp + i] = ring[(uint32_t)((m * hp + i) & (N - 1))];
}

// Blocks per run for `blocks` blocks of K overlapping frames over num_sms SMs
// that hold `groups` groups each. A full load takes one wave of the resident
// groups, at least 4 (K - 1) blocks each, so that the K - 1 frames a group
// transforms ahead of its run add at most a quarter to the work. A smaller
// one weighs those frames against idle SMs: a run of r blocks costs r + K - 1
// frames, and a frame takes about 3 units of time on an SM whose other groups
// idle, 2 g with g groups at work (frames of order 12: 3.5 us alone, 9.8 with five
// groups at work, 9.8 / 3.5 = 2.8 against 10 / 3). For each g only the shortest run that needs
// no more than g groups per SM can be the cheapest, so `groups` runs are
// weighed, whatever K.
inline long long istft_run(long long blocks, int k, long long num_sms, int groups) {
    const long long longest = 4LL * (k - 1);
    long long run = (blocks + num_sms * groups - 1) / (num_sms * groups), best = -1;
    for (int g = groups; g >= 1; --g) {
        const long long r = (blocks + num_sms * g - 1) / (num_sms * g);
        if (r > longest) break;
        const long long used = ((blocks + r - 1) / r + num_sms - 1) / num_sms;
        const long long cost = (r + k - 1) * (2 * used > 3 ? 2 * used : 3);
        if (best < 0 || cost < best) {
            best = cost;
            run = r;
        }
    }
    return run;
}

// Sizes that have a kernel of one group per CTA (of `groups` that share tables on an SM
// otherwise), and whether `runs` runs of `frames` frames each go to it, `slots` of its
// CTAs filling the GPU: one frame each, one wave. Measured at hop N, orders 10 / 11 / 12, groups that share
// tables against one group a CTA, us: one frame by itself 9.2 / 8.3 / 10.1 against 7.1 / 6.0 /
// 8.4, in a chain of calls 5.5 / 5.1 / 6.7 against 5.1 / 4.1 / 6.4; 148 frames in a chain 7.6 /
// 6.7 / 8.2 against 6.3 / 4.6 / 6.9, 740 frames 8.2 / 8.6 / 12.2 against 6.8 / 7.0 / 11.4. Order
// 13 (two groups) gains up to 4 frames and loses 7-14% at 8-100. Of several frames a
// group, the tables and the prefetch pay: order 12, hop N / 4, 16 frames 17.8
// against 20.8.
constexpr bool istft_has_single(int groups) { return groups > 3; }
inline bool istft_single(long long runs, long long frames, long long slots) { return frames == 1 && runs <= slots; }

using IstftLaunchFn = cudaError_t (*)(const TileArgs&, const IstftArgs&, cudaStream_t, const LaunchCtx&);

// The kernel's launch, and the CTAs of it that fit on an SM.
template <typename F, int P, int IL, bool SHARED>
struct IstftLaunch {
    using Cfg = IstftCfg<F, P, SHARED>;
    static int per_sm() {
        auto kern = istft_kernel<F, P, IL, SHARED>;
        static ResidentSlots slots;
        return resident_ctas(slots, [kern] { return occupancy_setup(kern, Cfg::THREADS, Cfg::SMEM, kSmemPerCta); });
    }
    static cudaError_t run(const TileArgs& a, const IstftArgs& o, long long grid, cudaStream_t stream, const LaunchCtx& ctx) {
        const size_t smem = balanced_smem(ctx, grid, per_sm(), Cfg::SMEM);
        if (ctx.launches) ++*ctx.launches;
        return launch_dependent(istft_kernel<F, P, IL, SHARED>, (unsigned)grid, Cfg::THREADS, smem, stream, a, o);
    }
};

// One group per run of blocks. Run r is group r / grid of CTA r % grid, so that
// few runs still spread over all SMs.
template <typename F, int P, int IL>
cudaError_t launch_istft(const TileArgs& a, const IstftArgs& o, cudaStream_t stream, const LaunchCtx& ctx) {
    if (o.n_frames <= 0 || o.blocks <= 0) return cudaSuccess;
    constexpr int GROUPS = IstftCfg<F, P, true>::GROUPS;
    IstftArgs oo = o;
    oo.run = istft_run(o.blocks, o.k, ctx.num_sms, GROUPS);
    const long long runs = (o.blocks + oo.run - 1) / oo.run;
    const long long ahead = oo.run + o.k - 1;  // frames that a whole run takes
    if constexpr (istft_has_single(GROUPS)) {
        using Single = IstftLaunch<F, P, IL, false>;
        if (istft_single(runs, ahead < o.n_frames ? ahead : o.n_frames, (long long)ctx.num_sms * Single::per_sm()))
            return Single::run(a, oo, runs, stream, ctx);
    }
    return IstftLaunch<F, P, IL, true>::run(a, oo, runs < ctx.num_sms ? runs : ctx.num_sms, stream, ctx);
}

// [complex order][input layout]; null where the order has no ISTFT kernel
struct IstftTable {
    IstftLaunchFn fn[kTileMaxP + 1][2];
};

template <typename F, int... Ps>
void fill_istft_orders(IstftTable& t, std::integer_sequence<int, Ps...>) {
    (
        [&] {
            if constexpr (IstftCfg<F, Ps, true>::kOK) {
                t.fn[Ps][kAoS] = launch_istft<F, Ps, kAoS>;
                t.fn[Ps][kSoA] = launch_istft<F, Ps, kSoA>;
            }
        }(),
        ...);
}
void fill_istft_f32(IstftTable& t);
void fill_istft_f64(IstftTable& t);

}  // namespace zlfft
