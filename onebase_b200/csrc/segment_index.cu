// Token sort + segment index on the device: the five tensors vLLM's LoRAKernelMeta.prepare_tensors builds with torch
// sort / unique / cumsum (vllm/lora/ops/triton_ops/lora_kernel_metadata.py:110-168), bit for bit, including its
// statefulness: the three segment arrays are always reset; a batch whose every token is -1 stops there and leaves the
// token map and the sorted indices as they were.
//
// One CTA, a stable counting sort.  A warp owns a contiguous chunk of the tokens and its own histogram of slot ids (bin 0 =
// "-1") in shared memory, filled 32 tokens at a time: lanes with the same id find one another with match, the lowest of
// them adds their number.  Per bin the chunks' counts become exclusive offsets, the bins are compacted (sorted unique ids)
// and scanned, and every warp places its own chunk with the ranks it has already worked out.  What bounds it is latency --
// dependent shared-memory steps of one SM -- so the tokens are split over the warps and not the bins, and a batch takes no more
// warps than it has groups of tokens.  On the device, 32 slots: 8192 tokens 12.8 us (33.3 with a warp per bin walking all the
// tokens), 512 3.2 (4.5), 32 2.5 (2.65; 4.3 with 32 warps whatever the batch), one 2.4 (2.6).  A call from Python takes 12 us.
#include "ob_common.cuh"

namespace ob {

constexpr int kSegThreads = 1024;
constexpr int kSegMinThreads = 128;
constexpr int kSegKeep = 8;              // tokens per lane whose ids and ranks stay in registers (8192 tokens over 32 warps)
constexpr int kSegSmemInts = 10240;      // room for the warps' histograms: 32 of them up to 309 slots, fewer beyond

__global__ void __launch_bounds__(kSegThreads, 1) segment_index_kernel(const int32_t* token_lora, int M, int L, int n_warps,
                                                                    int32_t* tok, int32_t* srt, int32_t* seg_n,
                                                                    int32_t* seg_start, int32_t* seg_ids) {
    extern __shared__ int32_t sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_threads = blockDim.x;
    const int bins = L + 1;
    int32_t* hist = sm;                   // [n_warps][bins] counts of a warp's chunk, then where in the bin its next token goes
    int32_t* start = sm + n_warps * bins; // [bins] tokens of each bin, then its first sorted position
    const int chunk = ((M + n_warps - 1) / n_warps + 31) / 32 * 32;
    const int lo = warp * chunk, hi = warp < n_warps ? min(M, lo + chunk) : 0;
    const uint32_t below = (1u << lane) - 1u;

    int id[kSegKeep];                     // the chunk's first tokens, all requested at once
#pragma unroll
    for (int q = 0; q < kSegKeep; ++q) {
        const int i = lo + q * 32 + lane;
        id[q] = i < hi ? token_lora[i] : 0;
    }
    for (int i = tid; i < n_warps * bins; i += n_threads) hist[i] = 0;
    for (int i = tid; i < bins; i += n_threads) {
        seg_n[i] = 0;
        seg_ids[i] = -1;
    }
    for (int i = tid; i < L + 2; i += n_threads) seg_start[i] = 0;
    __syncthreads();
    int32_t* own = hist + warp * bins;
    uint32_t same[kSegKeep];              // lanes of the group of 32 with this lane's id
    bool mine = false;
    auto count = [&](int i, int v) {
        const bool in = i < hi;
        const int bin = (v >= 0 && v < L) ? v + 1 : 0;
        mine |= in && bin > 0;
        const uint32_t m = __match_any_sync(0xffffffffu, in ? bin : -1);
        if (in && (m & below) == 0) own[bin] += __popc(m);
        __syncwarp();
        return m;
    };
#pragma unroll
    for (int q = 0; q < kSegKeep; ++q) {
        if (lo + q * 32 >= hi) break;
        same[q] = count(lo + q * 32 + lane, id[q]);
    }
    for (int base = lo + kSegKeep * 32; base < hi; base += 32) count(base + lane, base + lane < hi ? token_lora[base + lane] : 0);
    if (!__syncthreads_or(mine)) return;  // no adapter: the reset is all that happens; tok / srt stay stale
    // a bin's counts -> the chunks' offsets within it, and their total (one chunk: the scan below does it)
    for (int b = n_warps > 1 ? tid : bins; b < bins; b += n_threads) {
        int at = 0;
        for (int w0 = 0; w0 < n_warps; w0 += 8) {
            int c[8];                     // (eight loads on their way together)
#pragma unroll
            for (int u = 0; u < 8; ++u) c[u] = w0 + u < n_warps ? hist[(w0 + u) * bins + b] : 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (w0 + u < n_warps) hist[(w0 + u) * bins + b] = at;
                at += c[u];
            }
        }
        start[b] = at;
    }
    if (n_warps > 1) __syncthreads();
    if (warp == 0) {                      // compaction + scan over the bins, 32 at a time, in order
        int n_seg = 0, run = 0;
        for (int base = 0; base < bins; base += 32) {
            const int b = base + lane;
            const int c = b >= bins ? 0 : n_warps > 1 ? start[b] : hist[b];
            if (n_warps == 1 && b < bins) hist[b] = 0;
            const uint32_t m = __ballot_sync(0xffffffffu, c > 0);
            int incl = c;                 // inclusive scan of the counts within the warp
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += t;
            }
            if (b < bins) start[b] = run + incl - c;
            if (c > 0) {
                const int slot = n_seg + __popc(m & below);
                seg_ids[slot] = b - 1;
                seg_n[slot] = c;
                seg_start[slot + 1] = run + incl;
            }
            n_seg += __popc(m);
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
    auto place = [&](int i, int v, uint32_t m) {
        const bool in = i < hi;
        const int bin = (v >= 0 && v < L) ? v + 1 : 0;
        const int at = in ? own[bin] : 0;
        __syncwarp();
        if (in) {
            srt[start[bin] + at + __popc(m & below)] = i;
            tok[i] = v;
            if ((m & below) == 0) own[bin] = at + __popc(m);
        }
        __syncwarp();
    };
#pragma unroll
    for (int q = 0; q < kSegKeep; ++q) {
        if (lo + q * 32 >= hi) break;
        place(lo + q * 32 + lane, id[q], same[q]);
    }
    for (int base = lo + kSegKeep * 32; base < hi; base += 32) {
        const int i = base + lane, v = i < hi ? token_lora[i] : 0;
        place(i, v, __match_any_sync(0xffffffffu, i < hi ? ((v >= 0 && v < L) ? v + 1 : 0) : -1));
    }
}

cudaError_t launch_segment_index(const int32_t* token_lora, int M, int L, int32_t* tok, int32_t* srt, int32_t* seg_n,
                                 int32_t* seg_start, int32_t* seg_ids, cudaStream_t stream) {
    const int bins = L + 1;
    int n_warps = kSegThreads / 32;
    // no more warps than the tokens have groups of 32 -- every warp's histogram is cleared and added up -- and two groups to a warp
    // between 257 and 1024 tokens, where that measured better (32 slots, 1024 tokens: 4.1 against 4.75 us; 128: 3.15 against 2.9)
    const int groups = (M + 31) / 32, want = M > 256 && M <= 1024 ? (groups + 1) / 2 : groups;
    while (n_warps > 1 && n_warps / 2 >= want) n_warps /= 2;
    while (n_warps > 1 && (n_warps + 1) * bins > kSegSmemInts) n_warps /= 2;
    const int threads = n_warps * 32 > kSegMinThreads ? n_warps * 32 : kSegMinThreads;   // (the others clear and add up bins)
    segment_index_kernel<<<1, threads, sizeof(int32_t) * (n_warps + 1) * bins, stream>>>(token_lora, M, L, n_warps, tok, srt,
                                                                                            seg_n, seg_start, seg_ids);
    return cudaGetLastError();
}

}  // namespace ob
