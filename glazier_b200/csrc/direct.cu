// The direct sweep: a colour pass with no staging at all, the labels and
// tallies read where they lie. It takes every lean model (contact, volume and
// surface terms) but the planes small enough for the cluster, and every model
// with more terms.
//
// What bounds it is latency. A pass is a chain of dependent reads (labels,
// then the two cells' tallies and types, then for some copies moments,
// fields or activity) and a copy's arithmetic, on too few targets to fill the
// GPU, so the work is laid out to shorten that chain and to keep a warp's
// lanes on the same part of it:
//   - Everything a pass can do before the previous pass has finished comes
//     before its programmatic wait: the tables into shared memory, each
//     thread's target and its pick's draw (the clock of a replayed step is
//     written a whole graph earlier).
//   - A small pass prices each target in its own thread; in a plane the
//     neighbour labels come with the target's own, so the chain is labels,
//     tallies, commit. A larger one gathers the unlike targets, about a
//     fifth, into a queue that whole warps price from its front; the largest
//     give each warp a run of targets and a queue of its own.
//   - Pricing has no branch on the common path, so its reads and sums overlap.
//   - The tally rotation is shared out over the grid and taken by each
//     block's last threads.
// Measured per MCS, queued back to back, against the pass that read its launch
// from shared memory and its tables where they lie, and launched plainly: lean
// planes of two types 25.3 -> 14.7 us at 512^2; the two-field tissue (length,
// chemotaxis) 55.5 -> 26.1 us at 256^2, 61.3 -> 27.3 at 512^2 and 223 -> 110
// at 2048^2. A pass of a 256^2 lean plane is 2.5 us, of which 0.8 is the
// kernel boundary and the rest the chain.

#include <atomic>
#include <cstdlib>
#include <type_traits>

#include "direct.cuh"

namespace glz {

// The view of a pass: from the launch, or for a step replayed from a graph
// from the engine's clock (the pass's number gives the tally slots, the step
// its draws), as pass_launch (engine.cu) sets them on the host.
struct DirectView {
    PassView v;
    TermView t;
    int2 *vs_next_base;
    long long *vs_clear;
    long long *mom_next_base;
    long long *mom_clear;
};

__device__ __forceinline__ DirectView direct_view(const SweepLaunch &a) {
    DirectView d;
    if (!a.clock) {
        d.v = PassView{a.colour, a.key_pick, a.key_accept, a.vs_base, a.vs_prev, a.vs_cur};
        d.t = TermView{a.mom_base, a.mom_prev, a.mom_cur, a.field_cur, nullptr};
        d.vs_next_base = a.vs_next_base;
        d.vs_clear = a.vs_clear;
        d.mom_next_base = a.mom_next_base;
        d.mom_clear = a.mom_clear;
        return d;
    }
    const EngineClock c = *a.clock;
    const unsigned long long p = (unsigned long long)(c.pass + a.colour);
    const int32_t step = (int32_t)c.step;
    const int b = (int)(p % 2), n = 1 - b, cur = (int)(p % 3), next = cur == 2 ? 0 : cur + 1,
              prev = cur == 0 ? 2 : cur - 1;
    d.v = PassView{a.colour,
                   stream_key(a.seed, step, a.colour, 0),
                   stream_key(a.seed, step, a.colour, 1),
                   a.tal.vs_base[b],
                   a.tal.vs_delta[prev],
                   reinterpret_cast<unsigned long long *>(a.tal.vs_delta[cur])};
    d.t = TermView{a.tal.mom_base[b], a.tal.mom_delta[prev],
                   reinterpret_cast<unsigned long long *>(a.tal.mom_delta[cur]), c.field_cur, nullptr};
    d.vs_next_base = a.tal.vs_base[n];
    d.vs_clear = a.tal.vs_delta[next];
    d.mom_next_base = a.tal.mom_base[n];
    d.mom_clear = a.tal.mom_delta[next];
    return d;
}

// This block's share of the tally rotation (engine.h): an equal run of the
// labels, and of the moment words, from the block's last thread back.
template <bool EXTRAS>
__device__ __forceinline__ void rotate_share(const SweepLaunch &a, const DirectView &d) {
    int n = a.n_labels, share = a.rotate_share;
    if (a.n_live) {
        n = *a.n_live;
        share = (n + (int)gridDim.x - 1) / (int)gridDim.x;
    }
    const int from = (int)(blockDim.x - 1u - threadIdx.x);
    const int first = (int)blockIdx.x * share, last = min(n, first + share);
    for (int l = first + from; l < last; l += (int)blockDim.x) {
        int dv, ds;
        unpack_delta(d.v.vs_prev[l], dv, ds);
        const int2 b = d.v.vs_base[l];
        d.vs_next_base[l] = make_int2(b.x + dv, b.y + ds);
        d.vs_clear[l] = 0;
    }
    if (EXTRAS && a.tracks) {
        const long long words = (long long)last * a.g.nm;
        for (long long k = (long long)first * a.g.nm + from; k < words; k += blockDim.x) {
            d.mom_next_base[k] = d.t.base[k] + d.t.prev[k];
            d.mom_clear[k] = 0;
        }
    }
}

// How a pass's targets are shared out (the launch's FORM).
constexpr int kPlain = 0;  // one target per thread, priced where it lies
constexpr int kWarp = 1;   // each warp queues the unlike of a run of targets, and prices it a whole round at a time
constexpr int kBlock = 2;  // each block gathers the unlike of its targets into one queue

// Past what one wave of gathering blocks holds, each warp takes a run of
// consecutive targets by itself, 32 kWarpK a step, with no block barrier: what
// a step leaves in its queue short of a whole round of 32 waits for the next
// step, so but for the run's last every round is full. Per MCS, priced a step
// at a time from labels read twice, and so: 41.3 and 37.5 us at 2048^2, 75.6
// and 64.5 at 3000^2, 139.8 and 107.6 at 4096^2, 0.37 and 0.23 ms at 256^3;
// the two-field tissue at 2048^2 122 and 107 (a step of 64 targets 121 at
// 4096^2, of 192 112, of 256 115; the next step's labels read ahead of the
// pricing 114, and 124 for the tissue, which spills). The large planes'
// tiled kernel, windows by tensor copies through a ring in shared memory, took
// 51.3, 103.7 and 131.3 us at these sizes (8192^2: 490 against 399; four
// neighbours at 4096^2: 326 against 151; two types: 189 against 146). A pass
// of 4096^2 is bound by issue, 61 % of cycles: 18.8 M warp instructions, and
// its reads are 1.5 lattices through L2 (2.3 TB/s).
constexpr int kWarpK = 4;
// A run's targets at most: longer ones leave the warps further apart in the
// lattice, shorter ones end in short rounds more often (per MCS with 512, 1024
// and 2048: 121, 108 and 108 us at 4096^2, 402, 399 and 419 at 8192^2; of the
// volume with 256 and 1024: 0.234 and 0.248 ms at 256^3).
constexpr int kRunMost = 1024;
constexpr int kRunMostVolume = 256;
// A block's targets per thread at most (per MCS at 1024^2: 37.3 us with two,
// 52.0 with one).
constexpr int kBlockK = 2;
constexpr int kBlockThreads = 256;

// Every-term passes of more targets than the device's blocks hold at once
// gather in blocks of kBlockThreads at 64 registers, some spilled: what the
// spills cost is less than what the warps give (per MCS of the two-field
// tissue, 128 registers and 64: 53.7 and 46.7 us at 1024^2, 162.6 and 130.2
// at 2048^2; 31.9 and 37.0 at 640^2, where a pass is a single wave).
constexpr int kBlockWide = 3;

// Blocks of kBlockThreads an SM holds, which caps a thread's registers. The
// lean models' 64 registers make a 2^18-target pass of two targets a thread
// one wave (at 128^3: 0.060 ms per MCS against 0.073 uncapped, 0.065 at 48);
// small every-term passes keep 128 (uncapped they take up to 200, one block:
// 48 against 70 us per MCS for the 512^2 tissue), large ones 64.
// In place, a volume of several types also takes 128, so that its neighbours'
// labels and types are in flight together (64 and 128 registers: 35.1 and
// 28.9 us per MCS at 64^3 with 26 neighbours, 39.0 and 35.7 at 80^3; 31.1 and
// 44.2 with 80).
constexpr int direct_blocks(int form, bool extras, bool mixed_volume = false) {
    return (extras && (form == kPlain || form == kBlock)) || (mixed_volume && form == kPlain) ? 2 : 4;
}

template <int DIM, int NOFF, bool UNIFORM, int FORM, int TERMS>
__global__ void __launch_bounds__(kBlockThreads, direct_blocks(FORM, TERMS > 0, DIM == 3 && !UNIFORM))
    direct_sweep_kernel(const __grid_constant__ SweepLaunch a) {
    constexpr bool EXTRAS = TERMS > 0;
    const int targets = (a.g.w / 2) * (a.g.h / 2) * (DIM == 3 ? a.g.d / 2 : 1);
    __shared__ TypeSmem<EXTRAS> types;
    const TypeTables T = UNIFORM && !EXTRAS ? a.t : load_types<EXTRAS>(a, types);
    DirectView d = direct_view(a);
    __shared__ float logs[TERMS == 2 ? kLogs : 1];
    if (TERMS == 2) {
        for (int k = (int)threadIdx.x; k < kLogs; k += (int)blockDim.x) logs[k] = k ? motility_log((float)k) : 0.0f;
        d.t.logs = logs;
    }
    const PassView &v = d.v;
    const GlobalPass acc{a, v};
    const int tid = (int)threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned below = (1u << lane) - 1u;
    if constexpr (FORM == kPlain) {
        const int j = (int)(blockIdx.x * blockDim.x) + tid;
        int x = 0, y = 0, z = 0, pick = 0;
        if (j < targets) {
            direct_site<DIM>(a, a.colour, j, x, y, z);
            pick = pick_of<NOFF>(draw(v.key_pick, (uint32_t)((z * a.g.h + y) * a.g.w + x)));
        }
        grid_wait();
        if (!(UNIFORM && !EXTRAS)) __syncthreads();  // the tables are in place
        if (j < targets) {
            if constexpr (DIM == 2) {
                // a plane's neighbour labels come with the target's own: one
                // round trip, not two
                NeighbourLabels<DIM, NOFF, GlobalPass> ln(a, acc, x, y, z);
                ln.load();
                const uint32_t old = acc.label(x, y, z), nw = ln.picked(pick);
                if (old != nw)
                    direct_copy<DIM, NOFF, UNIFORM, GlobalPass, NeighbourLabels<DIM, NOFF, GlobalPass>, TERMS>(
                        a, T, acc, ln, v.key_accept, x, y, z, pick, old, nw, &d.t);
            } else {
                const uint32_t old = acc.label(x, y, z), nw = picked_label<DIM, NOFF>(a, acc, x, y, z, pick);
                const NeighbourReads<DIM, NOFF, GlobalPass> ln(a, acc, x, y, z);
                if (old != nw)
                    direct_copy<DIM, NOFF, UNIFORM, GlobalPass, NeighbourReads<DIM, NOFF, GlobalPass>, TERMS>(
                        a, T, acc, ln, v.key_accept, x, y, z, pick, old, nw, &d.t);
            }
        }
        rotate_share<EXTRAS>(a, d);
    } else if constexpr (FORM == kBlock || FORM == kBlockWide) {
        __shared__ int queue[kBlockThreads * kBlockK];
        __shared__ uint8_t picks[kBlockThreads * kBlockK];
        __shared__ uint2 pair[kBlockThreads * kBlockK];  // (old, new) labels of each queued copy
        __shared__ int total;
        const int nt = (int)blockDim.x;
        // the block's targets: direct_span of them, at most nt kBlockK
        const int first = (int)blockIdx.x * a.direct_span;
        const int last = min(first + a.direct_span, targets);
        if (tid == 0) total = 0;
        int site[kBlockK], picked[kBlockK];
        int tx[kBlockK], ty[kBlockK], tz[kBlockK];
#pragma unroll
        for (int k = 0; k < kBlockK; ++k) {
            const int j = first + k * nt + tid;
            site[k] = j < last ? j : -1;
            picked[k] = 0;
            tx[k] = ty[k] = tz[k] = 0;
            if (j < last) {
                direct_site<DIM>(a, a.colour, j, tx[k], ty[k], tz[k]);
                picked[k] = pick_of<NOFF>(draw(v.key_pick, (uint32_t)((tz[k] * a.g.h + ty[k]) * a.g.w + tx[k])));
            }
        }
        __syncthreads();  // the count (and the tables) in place
        grid_wait();
        unsigned masks[kBlockK];
        uint2 labels[kBlockK];
        int mine = 0;
#pragma unroll
        for (int k = 0; k < kBlockK; ++k) {
            labels[k] = make_uint2(0u, 0u);
            if (site[k] >= 0)
                labels[k] = make_uint2(acc.label(tx[k], ty[k], tz[k]),
                                       picked_label<DIM, NOFF>(a, acc, tx[k], ty[k], tz[k], picked[k]));
        }
#pragma unroll
        for (int k = 0; k < kBlockK; ++k) {
            masks[k] = __ballot_sync(0xffffffffu, labels[k].x != labels[k].y);
            mine += __popc(masks[k]);
        }
        // A warp's slots at once; the queue's order changes nothing, since a
        // pass's copies read only its snapshot and other colours' labels and
        // commit by atomics. What bounds a gathering pass is issue: of the
        // volume's instructions about half are this light part's, so it has no
        // division (the rotation's share comes with the launch), no chain of
        // selects (pick_offset) and no loop over the warps' counts (per MCS,
        // with those and without: 46.3 and 45.0 us at 128^3, 17.3 and 16.2 at
        // 1024^2, 28.6 and 28.1 for the 512^2 tissue).
        int at = 0;
        if (lane == 0 && mine) at = atomicAdd(&total, mine);
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int k = 0; k < kBlockK; ++k) {
            if (masks[k] & (1u << lane)) {
                const int e = at + __popc(masks[k] & below);
                queue[e] = site[k];
                picks[e] = (uint8_t)picked[k];
                pair[e] = labels[k];
            }
            at += __popc(masks[k]);
        }
        __syncthreads();
        const int queued = total;
        for (int e = tid; e < queued; e += nt) {
            int x, y, z;
            direct_site<DIM>(a, a.colour, queue[e], x, y, z);
            const NeighbourReads<DIM, NOFF, GlobalPass> ln(a, acc, x, y, z);
            direct_copy<DIM, NOFF, UNIFORM, GlobalPass, NeighbourReads<DIM, NOFF, GlobalPass>, TERMS>(
                a, T, acc, ln, v.key_accept, x, y, z, picks[e], pair[e].x, pair[e].y, &d.t);
        }
        rotate_share<EXTRAS>(a, d);
    } else {
        constexpr int kQueue = 32 * (kWarpK + 1);  // a step's targets after fewer than 32 left of the last
        __shared__ int queue[kBlockThreads / 32][kQueue];
        __shared__ uint8_t picks[kBlockThreads / 32][kQueue];
        __shared__ uint2 pair[kBlockThreads / 32][kQueue];  // (old, new) labels of each queued copy
        // the warp's run of consecutive targets: direct_span of them
        const int first = ((int)blockIdx.x * (kBlockThreads / 32) + warp) * a.direct_span;
        const int last = min(first + a.direct_span, targets);
        int total = 0;
        if (!(UNIFORM && !EXTRAS)) __syncthreads();  // the tables are in place
        for (int t = first; t < last; t += 32 * kWarpK) {
            int tx[kWarpK], ty[kWarpK], tz[kWarpK], pick[kWarpK];
#pragma unroll
            for (int k = 0; k < kWarpK; ++k) {
                // past the run's end a lane reads its first target again: no
                // branch, so the step's reads leave together
                const int j = t + k * 32 + lane;
                direct_site<DIM>(a, a.colour, j < last ? j : first, tx[k], ty[k], tz[k]);
                pick[k] = pick_of<NOFF>(draw(v.key_pick, (uint32_t)((tz[k] * a.g.h + ty[k]) * a.g.w + tx[k])));
            }
            if (t == first) grid_wait();  // the first step's draws come before it
            uint2 labels[kWarpK];
#pragma unroll
            for (int k = 0; k < kWarpK; ++k)
                labels[k] = make_uint2(acc.label(tx[k], ty[k], tz[k]),
                                       picked_label<DIM, NOFF>(a, acc, tx[k], ty[k], tz[k], pick[k]));
#pragma unroll
            for (int k = 0; k < kWarpK; ++k) {
                const int j = t + k * 32 + lane;
                const bool unlike = j < last && labels[k].x != labels[k].y;
                const unsigned m = __ballot_sync(0xffffffffu, unlike);
                if (unlike) {
                    const int e = total + __popc(m & below);
                    queue[warp][e] = j;
                    picks[warp][e] = (uint8_t)pick[k];
                    pair[warp][e] = labels[k];
                }
                total += __popc(m);
            }
            __syncwarp();
            // whole rounds of 32 off the queue's end; fewer stay for the next
            // step, and the last step's are priced as they are
            const bool more = t + 32 * kWarpK < last;
            while (total >= 32 || (!more && total > 0)) {
                const int e = total - 32 + lane;
                if (e >= 0) {
                    int x, y, z;
                    direct_site<DIM>(a, a.colour, queue[warp][e], x, y, z);
                    const NeighbourReads<DIM, NOFF, GlobalPass> ln(a, acc, x, y, z);
                    direct_copy<DIM, NOFF, UNIFORM, GlobalPass, NeighbourReads<DIM, NOFF, GlobalPass>, TERMS>(
                        a, T, acc, ln, v.key_accept, x, y, z, picks[warp][e], pair[warp][e].x, pair[warp][e].y, &d.t);
                }
                total = total > 32 ? total - 32 : 0;
                __syncwarp();
            }
        }
        if (first >= last) grid_wait();
        rotate_share<EXTRAS>(a, d);
    }
}

int programmatic_launch() {
    static const int on = [] {
        const char *env = std::getenv("GLAZIER_SWEEP_PDL");
        return env && env[0] == '0' ? 0 : 1;
    }();
    return on;
}

// The device's SM count, or 0 if it cannot be read: a device attribute only,
// so a launch being captured into a graph may ask.
static int sm_count() {
    static std::atomic<int> sms_once{0};  // handles on other host threads may launch too
    int sms = sms_once.load(std::memory_order_acquire);
    if (!sms) {
        int dev = 0;
        if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) {
            cudaGetLastError();
            return 0;
        }
        sms_once.store(sms, std::memory_order_release);
    }
    return sms;
}

template <int DIM, int NOFF, bool UNIFORM>
cudaError_t launch_direct(const SweepLaunch &a, cudaStream_t stream) {
    const int targets = (a.g.w / 2) * (a.g.h / 2) * (DIM == 3 ? a.g.d / 2 : 1);
    const bool warp = a.compact == 1, block = a.compact == 2;
    const bool wide = block && !a.lean && targets >= kDirectGatherFrom;
    SweepLaunch b = a;
    // Every-term blocks of 128 registers a thread are half as wide: four of
    // 128 threads fill an SM as two of 256 do but wait for one another less
    // (62.7 against 64.9 us per MCS at 1024^2).
    const int threads = block && !a.lean && !wide ? kBlockThreads / 2 : kBlockThreads;
    int per_block = threads * (warp ? kWarpK : (block ? kBlockK : 1));
    int grid = (targets + per_block - 1) / per_block;
    if (block) {
        const int slots = sm_count() * direct_blocks(kBlock, false);
        if (a.lean && slots > 0) {
            // Spread the pass evenly over whole waves of resident blocks, so
            // that no SM holds more of its targets than another (at 128^3 and
            // 1024^2: 592 blocks of 443 targets instead of 512 of 512 on 148
            // SMs).
            const int spread = (grid + slots - 1) / slots * slots;
            per_block = (targets + spread - 1) / spread;
            grid = (targets + per_block - 1) / per_block;
        }
        b.direct_span = per_block;
    }
    if (warp) {
        // Equal runs of whole lanes over whole waves of resident warps (or of
        // the capped grid's), none longer than kRunMost targets unless capped.
        const int most = DIM == 3 ? kRunMostVolume : kRunMost;
        long long slots = (long long)sm_count() * direct_blocks(kWarp, false) * (kBlockThreads / 32);
        if (slots > 0 && a.max_ctas <= 0) slots *= (targets + slots * most - 1) / (slots * most);
        if (a.max_ctas > 0) slots = (long long)a.max_ctas * (kBlockThreads / 32);
        const long long even = slots > 0 ? (targets + slots - 1) / slots : 32 * kWarpK;
        b.direct_span = (int)((even + 31) / 32 * 32);
        per_block = b.direct_span * (kBlockThreads / 32);
        grid = (targets + per_block - 1) / per_block;
    }
    b.rotate_share = (a.n_labels + grid - 1) / grid;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = programmatic_launch();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const auto launch = [&](auto terms) {  // the form's kernel with these terms
        constexpr int TERMS = decltype(terms)::value;
        if (warp) return cudaLaunchKernelEx(&cfg, direct_sweep_kernel<DIM, NOFF, UNIFORM, kWarp, TERMS>, b);
        if constexpr (TERMS > 0)
            if (wide) return cudaLaunchKernelEx(&cfg, direct_sweep_kernel<DIM, NOFF, UNIFORM, kBlockWide, TERMS>, b);
        if (block) return cudaLaunchKernelEx(&cfg, direct_sweep_kernel<DIM, NOFF, UNIFORM, kBlock, TERMS>, b);
        return cudaLaunchKernelEx(&cfg, direct_sweep_kernel<DIM, NOFF, UNIFORM, kPlain, TERMS>, b);
    };
    if (a.lean) return launch(std::integral_constant<int, 0>{});
    return a.has_motility ? launch(std::integral_constant<int, 2>{}) : launch(std::integral_constant<int, 1>{});
}

template cudaError_t launch_direct<2, 4, true>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<2, 4, false>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<2, 8, true>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<2, 8, false>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<3, 6, true>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<3, 6, false>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<3, 18, true>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<3, 18, false>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<3, 26, true>(const SweepLaunch &, cudaStream_t);
template cudaError_t launch_direct<3, 26, false>(const SweepLaunch &, cudaStream_t);

}  // namespace glz
