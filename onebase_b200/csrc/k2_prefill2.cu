// K2 for prefill batches on CTA PAIRS: two CTAs of a cluster compute one tile of 256 tokens x 256 (NVFP4
// base, or an FP8 launch of few tiles) or 512 (FP8 base) output features with tcgen05.mma.cta_group::2
// (kind::mxf4nvf4.block_scale or kind::f8f6f4, M = 256 tokens, N = 256 features, the 512-feature tile as two such MMAs filling
// all 512 accumulator columns: unlike the decode kernels the tokens are the MMA's rows here, so an accumulator lane is a token
// and its columns are consecutive features -- a thread of the epilogue stores 64 contiguous bytes of a row of y per
// tensor-memory load).
//
// Why pairs: a ring slot costs its single-thread roles a fixed time (every wait, copy issue, tcgen05.cp / mma / commit costs
// its issuing thread 50-250 cycles), whatever the slot holds.  In a pair each CTA supplies its own 128 rows of W per 256
// features and only HALF of the token tile (the MMA reads the other half out of the partner's shared memory), so a CTA takes
// in 32 KB (FP8) or 38 KB (NVFP4) per 256-feature slot -- 54 KB if it worked alone -- and with the tokens on the accumulator's
// lanes the epilogue needs no staging: W [128 x 128 B], x_q [128 tokens x 128 B], for NVFP4 its tokens' block scales (2 KB)
// and the W block scales of all 256 features (4 KB; every CTA needs the scales of all of B's rows in its own tensor memory).
// No load is multicast.  With one wave of pairs the main loop runs at the tensor rate (FP8: 0.33 us per 128-element k-block of
// 256 features, 0.57 us of 512, against 0.28 and 0.55 at the nominal peak); the rest of a launch is its 10 us of start-up,
// first loads and last read-out, the expand steps (as long as a k-block each) and idle pairs.
//
// Slices may end anywhere in a tile (widths in steps of 8 features): the tile's W, B and scale boxes run on into whatever
// follows or past the tensor's end (zeros), those columns are computed and not stored.  An expand step multiplies min(R, 64)
// ranks, its boxes 32, 64 or 128 bytes wide.
//
// Stored adapters (FP8 / NVFP4 codes): the epilogue's eight warps, which have nothing to do while a tile's main loop runs, turn
// the codes of the tile's expand steps into the slots' bf16 B tiles (scales folded in, one rounding, as k2_gemm.cu does),
// all eight on one step (two groups on steps in turn measured 180 against 160 us: 2048 tokens of gate_up, NVFP4 base), each
// step's codes requested two steps ahead; the producer hands them a slot through a count once it is free, they arrive
// on their CTA's `conv` barrier of the slot, and rank 1's warp 1 passes its CTA's completion on to rank 0's.
//
// Per CTA (512 threads): warp 0 = TMA producer of the CTA's own operands -- every load a tensor load of the
// cta_group::2 form, whose bytes are counted on the slot barrier of the pair's rank-0 CTA, so one wait there covers
// both CTAs' operands (the block scales are fetched as 8 x 256-byte boxes of a [rows, 256] byte tensor for that
// reason); warp 1 = in the pair's rank-0 CTA the MMA issuer for both; warp 2 = tile
// scout (row map, output scale, expand steps; both CTAs compute the same list); warps 4..11 = epilogue of the CTA's own
// 128 tokens (straight from tensor memory to y; two warps per lane quarter, half of the features each);
// warps 3, 12, 13 = in rank 0 the scale copiers (tcgen05.cp of a slot's scale factors into both CTAs' tensor memory).  The
// epilogue's two warpgroups take registers from the other two, so that a warp can hold 128 features of its tokens as bf16 and
// the accumulator is free after eight loads; 512-feature tiles are read out, and started, one 256-feature half after the other.
// (8192 tokens of gate_up: from the accumulator's last MMA to the next tile's first 3.5 -> 0.8 us, the call 822 -> 790.)  The
// issuer's commits arrive on the slot-free and accumulator-full barriers of BOTH CTAs (tcgen05.commit ... multicast::cluster, an arrival, not a load).  The kernel is persistent: a pair walks the launch's
// tiles, and the ring runs ahead into the next tile while the epilogue drains; the accumulators are single-buffered except
// for 256-feature FP8 tiles (NVFP4: 256 columns + 5 x 48 scale columns).  The LoRA expand is folded into the accumulator,
// y = s (W_q x_q + B_l h / s): per (tenant of the tile, rank chunk) one M = 256, N = 256 MMA of kind::f16 of the tenant's h
// blocks -- each CTA fetches its own 128 tokens' block, zeros (a TMA box outside the tensor) if the tenant has none of them --
// with B_l's rows.  Every wait is bounded; a CTA whose wait runs out records where,
// stops, and still joins the cluster barrier of the teardown, so its partner's own waits run out and both leave.
// Computes what lowbit_lora/kernels/nvfp4_lora_vllm.py:219-357 computes for a prefill batch.
#include <atomic>

#include "ob_common.cuh"
#include "ob_ptx.cuh"
#include "stored_adapters.cuh"

namespace ob {

constexpr int kP2Threads = 512;
constexpr int kP2RegsRoles = 88, kP2RegsEpilogue = 168;      // per thread; 2 x 88 + 2 x 168 = the 4 x 128 a launch has per lane
static_assert(2 * kP2RegsRoles + 2 * kP2RegsEpilogue <= 4 * 128, "register split");
constexpr int kP2Tokens = 256;               // tokens per tile: 128 per CTA (the MMA's M)
constexpr int kP2WBytes = 128 * 128;         // 128 rows of W (or B_l) of a slot
constexpr int kP2XBytes = 128 * 128;         // this CTA's half of the token tile
constexpr int kP2SfCols = 48;                // NVFP4: tensor-memory columns of one slot's scale factors (16 tokens' + 32 W)
constexpr int kP2MaxSteps = 512;
// Ring depth and slot size of a tile of `halves` 256-feature halves (NVFP4: one N = 256 MMA; FP8: one or two -- two take all
// 512 accumulator columns, with one the accumulators are double-buffered)
constexpr int kP2MaxStages = 6;
__host__ __device__ constexpr int p2_stages(bool fp4, int halves) { return fp4 ? 5 : halves == 2 ? 4 : 6; }
__host__ __device__ constexpr int p2_slot_bytes(bool fp4, int halves) {
    return halves * kP2WBytes + kP2XBytes + (fp4 ? 3 * kSfSlotBytes : 0);   // 38 KB / 48 KB or 32 KB
}

constexpr uint16_t kP2NoEntry = 0xFFFFu;
struct P2Step {
    uint16_t lora, chunk;                    // tenant, rank chunk
    uint16_t entry[2];                       // the tenant's entry in the list of each 128-token block (kP2NoEntry: not in it)
};

struct P2Meta {
    int n_steps;
    int rowmap[kP2Tokens];
    float scale[kP2Tokens];
    P2Step steps[kP2MaxSteps];
};

struct P2Ctrl {
    uint64_t full[kP2MaxStages];     // rank 0's: both CTAs' operands of the slot have landed (rank 1's is unused)
    uint64_t sf_ready[kP2MaxStages]; // rank 0 only (NVFP4): the slot's scale factors are in both CTAs' tensor memory
    uint64_t conv[kP2MaxStages];     // stored adapters: this CTA's B tiles of the expand step are in the slot (its 8 epilogue warps) ...
                                     // ... and, rank 0's, the partner's are (its relay's arrival)
    uint64_t empty[kP2MaxStages];    // the pair's MMAs on the slot are done (arrives in both CTAs)
    uint64_t meta_full[2];
    uint64_t meta_empty[2];
    uint64_t acc_full[2];            // per accumulator buffer; arrives in both CTAs
    uint64_t acc_empty[2];           // rank 0 only: both CTAs' epilogue warps (16 arrivals)
    uint32_t tmem_base;
    volatile int abort_flag;
    volatile int b_grant;            // stored adapters: expand steps whose slot the producer has acquired for the epilogue warps to fill
    int go_flag;
    P2Meta meta[2];
};

__device__ __forceinline__ void p2_timeout(const K2pParams& p, P2Ctrl* c, int where, int it) {
    c->abort_flag = 1;
    if (atomicCAS(p.status, OB_DEV_OK, OB_DEV_WAIT_TIMEOUT) == OB_DEV_OK) {
        p.status[1] = 300 + where;
        p.status[2] = blockIdx.x;
        p.status[3] = 0;
        p.status[4] = 0;
        p.status[5] = it;
    }
}

// Bounded wait of a role's thread: the abort flag and the clock are looked at only once the first poll has failed -- a wait that
// finds its phase complete is on the critical path of the single-thread roles.
template <bool CLUSTER>
__device__ __forceinline__ bool p2_wait(const K2pParams& p, P2Ctrl* c, uint64_t* bar, uint32_t parity, uint64_t limit_ns, int where, int it) {
    if (CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    for (uint32_t n = 1;; ++n) {
        if (CLUSTER ? mbar_try_wait_cluster(bar, parity) : mbar_try_wait(bar, parity)) return true;
        if ((n & 15u) == 0) {
            if (c->abort_flag) return false;
            if (global_timer_ns() - t0 > limit_ns) {
                p2_timeout(p, c, where, it);
                return false;
            }
        }
    }
}

// Two bf16 sums, each the fp32 sum rounded once (as k2_gemm.cu's residual add).
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(bf16_lo(a) + bf16_lo(b), bf16_hi(a) + bf16_hi(b));
    return *reinterpret_cast<const uint32_t*>(&r);
}

// A tile: `rows` features of one slice (the slice's last tile may be ragged: what lies beyond the slice is computed and not
// stored) x 256 tokens.
struct P2Tile {
    int t0, s, n_s, slice_off, n0_local, m_idx;
    int sf_tile;                             // NVFP4: the tile's first 128-row tile in the packed W scales (per slice, rounded up)
};
__host__ __device__ inline int p2_n_tiles(const int32_t* widths, int S, int rows) {
    int n = 0;
    for (int s = 0; s < S; ++s) n += (widths[s] + rows - 1) / rows;
    return n;
}
__device__ __forceinline__ P2Tile p2_tile(const K2pParams& p, int t, int m_tiles, int rows) {
    P2Tile r;
    r.m_idx = t % m_tiles;
    r.t0 = r.m_idx * kP2Tokens;
    int s = 0, n_tile = t / m_tiles, off = 0, sf = 0;
    while (s < p.S - 1 && n_tile >= (p.widths[s] + rows - 1) / rows) {
        n_tile -= (p.widths[s] + rows - 1) / rows;
        off += p.widths[s];
        sf += (p.widths[s] + kTileN - 1) / kTileN;
        ++s;
    }
    r.s = s;
    r.n_s = p.widths[s];
    r.slice_off = off;
    r.n0_local = n_tile * rows;
    r.sf_tile = sf + r.n0_local / kTileN;
    return r;
}

// A tile's ring slots, the same in every role: `lead` k-blocks, then the remaining k-blocks and the expand steps.  bf16
// adapters: all k-blocks lead, so that a tile's first loads need no list.  Stored adapters: the steps are spread evenly among
// the k-blocks behind the first ring's worth, so that converting one tile hides behind the k-blocks in between (a step's
// conversion takes a microsecond or two from its slot's release to its arrival; at the tile's end, one after the other, that was
// a third of the kernel).
struct P2Walk {
    int lead, rem, n_steps, acc = 0;
    __device__ P2Walk(int lead_blocks, int kblocks, int steps) : lead(lead_blocks), rem(kblocks - lead_blocks + steps), n_steps(steps) {}
    __device__ bool next_is_step() {                          // of the next slot behind the lead
        acc += n_steps;
        if (acc < rem) return false;
        acc -= rem;
        return true;
    }
    __device__ int slot_of_step(int li) const { return lead + ((li + 1) * rem + n_steps - 1) / n_steps - 1; }   // within the tile
};

// EXTRA: the launch adds a residual stream in its stores; every other launch runs an instantiation without that code.  The
// residual's pieces are asked into L2 under the main loop and loaded just before the step's transposes.  down at 2048 tokens with SiLU * mul
// and residual, whole projection: 458 us (128-token tiles of k2_gemm.cu, the transform evaluated three times) -> 197 us.
template <bool FP4, int HALVES, bool EXTRA, bool STORED>
__global__ void __launch_bounds__(kP2Threads, 1)
k2_prefill_pair_kernel(const K2pParams p, const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                       const __grid_constant__ CUtensorMap tm_h, const __grid_constant__ CUtensorMap tm_b0,
                       const __grid_constant__ CUtensorMap tm_b1, const __grid_constant__ CUtensorMap tm_b2,
                       const __grid_constant__ CUtensorMap tm_b3, const __grid_constant__ CUtensorMap tm_wsf,
                       const __grid_constant__ CUtensorMap tm_xsf) {
    extern __shared__ uint8_t smem_raw[];
    // (the dynamic shared memory starts at the same offset in both CTAs of a pair: the MMA applies one descriptor to both)
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int kHalves = HALVES, kRows = 256 * HALVES, kStages = p2_stages(FP4, HALVES), kSlot = p2_slot_bytes(FP4, HALVES);
    constexpr int kAccBufs = !FP4 && HALVES == 1 ? 2 : 1;     // (NVFP4: the scale factors take the rest of tensor memory)
    constexpr int kXOff = kHalves * kP2WBytes;                // the token tile (or h block) follows the W (or B_l) rows in a slot
    uint8_t* ring = smem;
    P2Ctrl* ctrl = reinterpret_cast<P2Ctrl*>(smem + (size_t)kStages * kSlot);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_cta_rank();                 // 0: issues the pair's MMAs
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    griddep_launch_dependents();
    const uint64_t limit_ns = (uint64_t)p.wait_ms * 1000000ull;
    const int m_tiles = (p.M + kP2Tokens - 1) / kP2Tokens;
    const int n_tiles = m_tiles * p2_n_tiles(p.widths, p.S, kRows);
    const int rc = min(p.R, 64), n_chunks = p.R / rc;         // an expand step multiplies rc ranks

    if (tid == 0) {
        for (int i = 0; i < kStages; ++i) {
            // rank 0's: one arrival whose transaction count covers both CTAs' bytes (every load is a tensor load, and the
            // partner's complete on this barrier directly); rank 1's is never used
            mbar_init(&ctrl->full[i], 1);
            mbar_init(&ctrl->sf_ready[i], 3);   // one commit per copier thread
            mbar_init(&ctrl->conv[i], rank == 0 ? 9 : 8);
            mbar_init(&ctrl->empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ctrl->meta_full[i], 1);
            mbar_init(&ctrl->meta_empty[i], STORED && rank == 1 ? 9 : 8);   // the epilogue warps, and the relay
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&ctrl->acc_full[i], 1);
            mbar_init(&ctrl->acc_empty[i], 16);
        }
        ctrl->abort_flag = 0;
        ctrl->b_grant = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc_pair(&ctrl->tmem_base, 512);
        tmem_relinquish_pair();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_w);
        tma_prefetch_desc(&tm_x);
        tma_prefetch_desc(&tm_h);
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();                                         // both CTAs' barriers exist before either is signalled from outside
    cluster_wait();
    tc_fence_after();
    const uint32_t tmem_base = ctrl->tmem_base;

    if (warp < 4 || warp >= 12) {
        regs_dec<kP2RegsRoles>();
    if (warp == 0) {
        // =========================================================== TMA producer of this CTA's operands
        if (lane == 0) {
            griddep_wait();                                   // x_q and the h blocks come from the preceding kernels
            int it = 0, st = 0, granted = 0;
            uint32_t ph = 1;                                  // parity of the phase that frees the slot (the first round passes)
            bool ok = true;
            for (int t = pair, i = 0; t < n_tiles && ok; t += n_pairs, ++i) {
                const P2Tile tl = p2_tile(p, t, m_tiles, kRows);
                const CUtensorMap* tmb = (tl.s == 0) ? &tm_b0 : (tl.s == 1) ? &tm_b1 : (tl.s == 2) ? &tm_b2 : &tm_b3;
                const int row0 = tl.n0_local + (int)rank * 128;           // this CTA's rows of each 256-feature half
                const int lead = STORED ? min(kStages, p.kblocks) : p.kblocks;
                P2Walk walk(lead, p.kblocks, 0);
                int total = p.kblocks;                        // (grows by the steps once the list is there)
                for (int q = 0, kb = 0, li = 0;; ++q, ++it) {
                    bool step = false;
                    if (q >= lead) {
                        if (q == lead) {
                            if (!p2_wait<false>(p, ctrl, &ctrl->meta_full[i & 1], (uint32_t)((i >> 1) & 1), limit_ns, 2, it)) {
                                ok = false;
                                break;
                            }
                            walk = P2Walk(lead, p.kblocks, ctrl->meta[i & 1].n_steps);
                            total += walk.n_steps;
                        }
                        if (q >= total) break;
                        step = walk.next_is_step();
                    }
                    if (!p2_wait<true>(p, ctrl, &ctrl->empty[st], ph, limit_ns, 1, it)) {
                        ok = false;
                        break;
                    }
                    uint8_t* slot = ring + (size_t)st * kSlot;
                    // every load is a tensor load, so both CTAs' bytes are counted on rank 0's barrier and no relay stands
                    // between the partner's data and the MMAs
                    const uint32_t bar0 = cluster_peer_addr(smem_u32(&ctrl->full[st]), 0);
                    if (!step) {
                        if (rank == 0) mbar_arrive_expect_tx(&ctrl->full[st], (uint32_t)(2 * kSlot));
#pragma unroll
                        for (int h = 0; h < kHalves; ++h)
                            tma_load_2d_pair(slot + h * kP2WBytes, &tm_w, bar0, kb * 128, tl.slice_off + row0 + h * 256);
                        tma_load_2d_pair(slot + kXOff, &tm_x, bar0, kb * 128, tl.t0 + (int)rank * 128);
                        if (FP4) {
                            // scales, as 8 x 256-byte rows of a [rows, 256] byte tensor per 2 KB atom: this CTA's 128 tokens (the
                            // MMA's A rows), then both 128-feature tiles of W (every CTA needs the scales of all of B's 256 rows in
                            // its own tensor memory)
                            uint8_t* sf = slot + kXOff + kP2XBytes;
                            tma_load_2d_pair(sf, &tm_xsf, bar0, 0, ((tl.m_idx * p.kblocks + kb) * 2 + (int)rank) * 8);
                            tma_load_2d_pair(sf + kSfSlotBytes, &tm_wsf, bar0, 0, (tl.sf_tile * p.kblocks + kb) * 8);
                            tma_load_2d_pair(sf + 2 * kSfSlotBytes, &tm_wsf, bar0, 0, ((tl.sf_tile + 1) * p.kblocks + kb) * 8);
                        }
                        ++kb;
                    } else {
                        const P2Step e = ctrl->meta[i & 1].steps[li];
                        // B_l: this CTA's 128 features of each half.  h: this CTA's 128 tokens' block of the tenant.  A tenant with no
                        // token among them must add nothing to those rows of the M = 256 MMA, so the CTA fetches a box that lies
                        // wholly outside the tensor, which TMA fills with zeros.
                        const int entry = rank == 0 ? e.entry[0] : e.entry[1];
                        const bool in = entry != kP2NoEntry;
                        const int h_row = in ? tl.s * p.max_m + tl.t0 + (int)rank * 128 : p.S * p.max_m + 128;
                        const int h_col = in ? entry * p.R + (int)e.chunk * rc : 0;
                        if (STORED) {                         // the slot is free: the epilogue warps fill its B tiles
                            __threadfence_block();
                            ctrl->b_grant = ++granted;
                        }
                        if (rank == 0) mbar_arrive_expect_tx(&ctrl->full[st], (uint32_t)(2 * ((STORED ? 0 : kHalves) + 1) * 128 * rc * 2));
#pragma unroll
                        for (int h = 0; !STORED && h < kHalves; ++h)
                            tma_load_2d_pair(slot + h * kP2WBytes, tmb, bar0, (int)e.chunk * rc, (int)e.lora * tl.n_s + row0 + h * 256);
                        tma_load_2d_pair(slot + kXOff, &tm_h, bar0, h_col, h_row);
                        ++li;
                    }
                    if (++st == kStages) { st = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // =========================================================== MMA issuer of the pair
            // A = tokens (each CTA's 128 are its accumulator's lanes), B = features (128 from each CTA per 256-wide half)
            const uint32_t idesc4 = umma_idesc_nvfp4(256, 256);
            const uint32_t idesc8 = umma_idesc(0, 0, 256, 256);
            const uint32_t idesc16 = umma_idesc(1, 1, 256, 256);
            const uint32_t row_bytes = (uint32_t)rc * 2;      // an expand tile's row: 32, 64 or 128 bytes, swizzled accordingly
            const uint32_t lt = row_bytes == 128 ? 2u : row_bytes == 64 ? 4u : 6u;
            int it = 0, st = 0;
            uint32_t ph = 0, sf_par = 0, conv_par = 0;        // phase of the slot; per slot: of its scale barrier, of its `conv` barrier
            const uint32_t ring_addr = smem_u32(ring);
            const uint64_t d_w0 = umma_smem_desc(ring_addr, 1024, 2), d_x0 = umma_smem_desc(ring_addr + kXOff, 1024, 2);
            const uint64_t d_b0 = umma_smem_desc(ring_addr, row_bytes * 8, lt), d_h0 = umma_smem_desc(ring_addr + kXOff, row_bytes * 8, lt);
            uint32_t acc = tmem_base;
            auto half_fp8 = [&](int slot, int h, uint32_t first) {        // one half of a k-block
                const uint64_t off = (uint64_t)(uint32_t)(slot * (kSlot >> 4));
                const uint64_t dx = d_x0 + off, dw = d_w0 + off + (uint64_t)(h * (kP2WBytes >> 4));
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    umma_f8f6f4_pair(acc + (uint32_t)(h * 256), dx + (uint64_t)(k * 2), dw + (uint64_t)(k * 2), idesc8, k > 0 ? 1u : first);
            };
            auto advance = [&]() {
                umma_commit_pair(&ctrl->empty[st], 3);
                ++it;
                if (++st == kStages) { st = 0; ph ^= 1u; }
            };
            auto k_block = [&](uint32_t first) -> bool {      // `first`: 0 for the tile's first (the accumulator starts there)
                if (FP4) {
                    // the scale copier saw both CTAs' operands land before it copied: one wait covers data and scales; the
                    // barrier completes once per K-BLOCK use of the slot -- expand steps pass it by -- so it has its own parity
                    if (!p2_wait<false>(p, ctrl, &ctrl->sf_ready[st], (sf_par >> st) & 1u, limit_ns, 4, it)) return false;
                    sf_par ^= 1u << st;
                    tc_fence_after();
                    const uint64_t off = (uint64_t)(uint32_t)(st * (kSlot >> 4));
                    const uint64_t dx = d_x0 + off, dw = d_w0 + off;
                    const uint32_t sft = tmem_base + 256u + (uint32_t)(st * kP2SfCols);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t ta = sft + (uint32_t)k * 4u, tb = sft + 16u + (uint32_t)k * 8u;
                        umma_nvfp4_pair(acc, dx + (uint64_t)(k * 2), dw + (uint64_t)(k * 2), idesc4, ta, tb, k > 0 ? 1u : first);
                    }
                } else {
                    if (!p2_wait<true>(p, ctrl, &ctrl->full[st], ph, limit_ns, 4, it)) return false;
#pragma unroll
                    for (int h = 0; h < kHalves; ++h) half_fp8(st, h, first);
                }
                advance();
                return true;
            };
            auto expand_step = [&]() -> bool {
                if (!p2_wait<true>(p, ctrl, &ctrl->full[st], ph, limit_ns, 6, it)) return false;
                if (STORED) {                                 // (completes once per EXPAND use of the slot: a parity of its own)
                    if (!p2_wait<true>(p, ctrl, &ctrl->conv[st], (conv_par >> st) & 1u, limit_ns, 16, it)) return false;
                    conv_par ^= 1u << st;
                }
                const uint64_t off = (uint64_t)(uint32_t)(st * (kSlot >> 4));
                const uint64_t dh = d_h0 + off;
#pragma unroll
                for (int h = 0; h < kHalves; ++h) {
                    const uint64_t db = d_b0 + off + (uint64_t)(h * (kP2WBytes >> 4));
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (k * 16 < rc)
                            umma_f16_pair(acc + (uint32_t)(h * 256), dh + (uint64_t)(k * 2), db + (uint64_t)(k * 2), idesc16, 1u);
                }
                advance();
                return true;
            };
            bool ok = true;
            for (int t = pair, i = 0; t < n_tiles && ok; t += n_pairs, ++i) {
                acc = tmem_base + (uint32_t)(i % kAccBufs) * 256u;
                const int use = kHalves == 2 ? i : i / kAccBufs;          // the epilogues have read the accumulator's previous tile
                if (use > 0) {
                    if (!p2_wait<true>(p, ctrl, &ctrl->acc_empty[kHalves == 2 ? 0 : i % kAccBufs], (uint32_t)((use - 1) & 1), limit_ns, 8, i)) break;
                    tc_fence_after();
                }
                int kb = 0;
                if (kHalves == 2) {
                    // The halves of the accumulator come free one after the other: the first ring's worth of k-blocks goes into the
                    // first half while the epilogues still read the second, then into the second.
                    const int n = min(kStages, p.kblocks);
                    int s2 = st;
                    uint32_t ph2 = ph;
                    for (int j = 0; j < n && ok; ++j) {
                        ok = p2_wait<true>(p, ctrl, &ctrl->full[s2], ph2, limit_ns, 4, it + j);
                        if (ok) half_fp8(s2, 0, j > 0 ? 1u : 0u);
                        if (++s2 == kStages) { s2 = 0; ph2 ^= 1u; }
                    }
                    if (ok && use > 0) {
                        ok = p2_wait<true>(p, ctrl, &ctrl->acc_empty[1], (uint32_t)((use - 1) & 1), limit_ns, 8, i);
                        tc_fence_after();
                    }
                    if (!ok) break;
                    for (; kb < n; ++kb) {
                        half_fp8(st, 1, kb > 0 ? 1u : 0u);
                        advance();
                    }
                }
                const int lead = STORED ? min(kStages, p.kblocks) : p.kblocks;
                for (; kb < lead && ok; ++kb) ok = k_block(kb > 0 ? 1u : 0u);
                if (!ok || !p2_wait<false>(p, ctrl, &ctrl->meta_full[i & 1], (uint32_t)((i >> 1) & 1), limit_ns, 5, it)) { ok = false; break; }
                const int n_steps = ctrl->meta[i & 1].n_steps;
                if (STORED) {
                    P2Walk walk(lead, p.kblocks, n_steps);
                    for (int q = 0; q < walk.rem && ok; ++q) ok = walk.next_is_step() ? expand_step() : k_block(1u);
                } else {
                    for (int li = 0; li < n_steps && ok; ++li) ok = expand_step();
                }
                if (ok) umma_commit_pair(&ctrl->acc_full[i % kAccBufs], 3);
            }
        }
        if (STORED && lane == 0 && rank == 1) {
            // =========================================================== stored adapters: relay of rank 1's `conv` arrivals.
            // Rank 0's thread issues the MMA that reads rank 1's converted tiles, which takes a release at cluster scope.  From
            // the converting warps themselves that release waits for everything they have in flight -- the codes
            // requested two steps ahead, the stores to y.  So they arrive here at CTA scope, and this thread, which has nothing in
            // flight, passes the arrival on: the release is cumulative over what its own wait has acquired.  (gate_up at 2048
            // tokens, FP8-stored on an NVFP4 base, whole call: 229 us so, 240 with the converting warps' release; o at 1111,
            // NVFP4-stored: 82 and 92.)
            int it = 0, st = 0;
            uint32_t conv_par = 0;
            bool ok = true;
            for (int t = pair, i = 0; t < n_tiles && ok; t += n_pairs, ++i) {
                if (!p2_wait<false>(p, ctrl, &ctrl->meta_full[i & 1], (uint32_t)((i >> 1) & 1), limit_ns, 18, it)) break;
                const int lead = min(kStages, p.kblocks);
                P2Walk walk(lead, p.kblocks, ctrl->meta[i & 1].n_steps);
                mbar_arrive(&ctrl->meta_empty[i & 1]);        // (nothing else of the list is read here)
                const int total = p.kblocks + walk.n_steps;
                for (int q = 0; q < total; ++q, ++it) {
                    if (q >= lead && walk.next_is_step()) {
                        if (!p2_wait<false>(p, ctrl, &ctrl->conv[st], (conv_par >> st) & 1u, limit_ns, 19, it)) {
                            ok = false;
                            break;
                        }
                        conv_par ^= 1u << st;
                        mbar_arrive_remote_release(cluster_peer_addr(smem_u32(&ctrl->conv[st]), 0));
                    }
                    if (++st == kStages) st = 0;
                }
            }
        }
    } else if (warp == 3 || warp >= 12) {
        // =========================================================== scale copiers (NVFP4, rank 0; warps 3, 12, 13): a k-block
        // slot's scale factors -> both CTAs' tensor memory, ahead of the MMAs.  Threads of their own because every tcgen05
        // instruction costs its issuer some 50 cycles: twelve copies per slot from one thread (with its wait and commit, 920
        // cycles) bounded the main loop, whose four MMAs take the tensor pipe some 540.  Copier 0 moves the tokens' scales,
        // copiers 1 and 2 those of the two 128-feature halves of W: four copies each per slot.
        const int cpi = warp == 3 ? 0 : warp - 11;
        if (FP4 && lane == 0 && rank == 0 && cpi < 3) {
            int it = 0, st = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int t = pair, i = 0; t < n_tiles && ok; t += n_pairs, ++i) {
                // the tile's expand steps use ring slots too: read their number now (the scout is a tile ahead), while this
                // thread's own copies still stand between the read and the buffer's next writer
                if (!mbar_wait(&ctrl->meta_full[i & 1], (uint32_t)((i >> 1) & 1), limit_ns)) {
                    p2_timeout(p, ctrl, 14, it);
                    break;
                }
                const int lead = STORED ? min(kStages, p.kblocks) : p.kblocks;
                P2Walk walk(lead, p.kblocks, ctrl->meta[i & 1].n_steps);
                const int total = p.kblocks + walk.n_steps;
                for (int q = 0; q < total; ++q, ++it) {
                    const bool step = q >= lead && walk.next_is_step();
                    if (!p2_wait<true>(p, ctrl, &ctrl->full[st], ph, limit_ns, 13, it)) {
                        ok = false;
                        break;
                    }
                    // (the expand steps' slots carry no scales, but this thread still follows their barriers phase by phase: a
                    // parity wait entered a whole phase early would pass at once)
                    if (!step) {
                        tc_fence_after();
                        const uint32_t sfs = smem_u32(ring + (size_t)st * kSlot) + (uint32_t)(kXOff + kP2XBytes);
                        const uint32_t sft = tmem_base + 256u + (uint32_t)(st * kP2SfCols);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const uint32_t dst = cpi == 0 ? sft + (uint32_t)k * 4u : sft + 16u + (uint32_t)k * 8u + (uint32_t)(cpi - 1) * 4u;
                            tmem_cp_sf_pair(dst, sf_smem_desc(sfs + (uint32_t)cpi * kSfSlotBytes + (uint32_t)k * 512u));
                        }
                        umma_commit_pair(&ctrl->sf_ready[st], 1);      // (arrives in rank 0 only)
                    }
                    if (++st == kStages) { st = 0; ph ^= 1u; }
                }
            }
        }
    } else if (warp == 2) {
        // =========================================================== tile scout (the same list in both CTAs)
        int n_all, n_ad;
        segment_totals(p.meta, p.L, lane, n_all, n_ad);
        n_all = min(n_all, p.M);
        griddep_wait();                                       // K1's s_x from here on
        const float s_w = __ldg(p.s_w);
        for (int t = pair, i = 0; t < n_tiles; t += n_pairs, ++i) {
            P2Meta& mt = ctrl->meta[i & 1];
            int go = 1;
            if (lane == 0 && i >= 2) {
                go = ctrl->abort_flag ? 0 : 1;
                if (go && !mbar_wait(&ctrl->meta_empty[i & 1], (uint32_t)(((i >> 1) - 1) & 1), limit_ns)) {
                    p2_timeout(p, ctrl, 9, i);
                    go = 0;
                }
            }
            go = __shfl_sync(0xffffffffu, go, 0);
            if (!go) break;
            const P2Tile tl = p2_tile(p, t, m_tiles, kRows);
            for (int c = lane; c < kP2Tokens; c += 32) {
                const int pos = tl.t0 + c;
                mt.rowmap[c] = pos < p.M ? position_row(p.meta, pos, p.M, n_all, n_ad) : -1;
                // FP8: the token's activation scale times the weight scale; NVFP4: alpha = 1 / (x_global * w_global) for all
                mt.scale[c] = pos < p.M ? expand_scale((p.sx ? __ldcg(p.sx + pos) : 1.0f) * s_w) : 0.0f;
            }
            // Expand steps: the tenants of the first 128-token block in segment order, then those of the second.  A tenant that
            // crosses the blocks' edge is the last of the one and the first of the other: ONE step serves both.
            int total = 0, last = -1;                         // last: the first block's last tenant
            if (n_ad > 0) {
                for (int blk = 0; blk < 2; ++blk) {
                    const int b0 = tl.t0 + blk * 128;
                    int entries = 0;
                    for (int base = 0; base <= p.L; base += 32) {
                        const int j = base + lane;
                        int lora = -1, lo = 0, hi = 0;
                        if (j <= p.L) {
                            lora = p.meta.seg_ids[j];
                            const int cnt = p.meta.seg_n[j], sst = p.meta.seg_start[j];
                            lo = max(sst, b0);
                            hi = min(min(sst + cnt, b0 + 128), n_all);
                            if (cnt <= 0 || sst < 0) lora = -1;
                        }
                        const bool hit = lora >= 0 && lora < p.L && lo < hi;
                        const uint32_t mask = __ballot_sync(0xffffffffu, hit);
                        if (mask == 0) continue;
                        const int first_lane = __ffs(mask) - 1, first_lora = __shfl_sync(0xffffffffu, lora, first_lane);
                        const bool merge = blk == 1 && entries == 0 && first_lora == last;
                        const int rk = __popc(mask & ((1u << lane) - 1u));
                        const int entry = entries + rk;
                        if (hit && entry < kMaxTileTenants) {
                            const bool joined = merge && rk == 0;
                            const int at = joined ? total - n_chunks : total + (rk - (merge ? 1 : 0)) * n_chunks;
                            for (int c = 0; c < n_chunks; ++c)
                                if (at + c < kP2MaxSteps) {
                                    if (joined) mt.steps[at + c].entry[1] = (uint16_t)entry;
                                    else
                                        mt.steps[at + c] = P2Step{(uint16_t)lora, (uint16_t)c,
                                                                  {blk == 0 ? (uint16_t)entry : kP2NoEntry, blk == 1 ? (uint16_t)entry : kP2NoEntry}};
                                }
                        }
                        const int n_hit = min(__popc(mask), kMaxTileTenants - entries);
                        entries += n_hit;
                        total += (n_hit - (merge ? 1 : 0)) * n_chunks;
                        if (blk == 0) last = __shfl_sync(0xffffffffu, lora, 31 - __clz(mask));
                    }
                    if (blk == 0 && entries >= kMaxTileTenants) last = -1;   // (its last tenants may have been left out)
                    __syncwarp();
                }
            }
            if (lane == 0) mt.n_steps = min(total, kP2MaxSteps);
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctrl->meta_full[i & 1]);
        }
    }
    } else {
        regs_inc<kP2RegsEpilogue>();
        // =========================================================== epilogue (warps 4..11): this CTA's 128 tokens -> y
        // Two warps per 32-lane quarter of tensor memory, one per half of the tile's features.
        const int te = tid - 128;                             // 0..255 over the eight warps
        const int q = warp & 3;                               // the 32 tensor-memory lanes this warp may read
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        int it = 0, taken = 0;                                // stored adapters: ring slots and expand steps so far
        for (int t = pair, i = 0; t < n_tiles; t += n_pairs, ++i) {
            const P2Meta& mt = ctrl->meta[i & 1];
            const P2Tile tl = p2_tile(p, t, m_tiles, kRows);
            if (te == 0) {
                int go = ctrl->abort_flag ? 0 : 1;
                if (go && !mbar_wait(&ctrl->meta_full[i & 1], (uint32_t)((i >> 1) & 1), limit_ns)) {
                    p2_timeout(p, ctrl, 10, i);
                    go = 0;
                }
                ctrl->go_flag = go;
            }
            if constexpr (STORED) {
                asm volatile("bar.sync 1, 256;" ::: "memory");
                const bool meta_ok = ctrl->go_flag != 0;
                const int n_steps = meta_ok ? mt.n_steps : 0;
                const P2Walk walk(min(kStages, p.kblocks), p.kblocks, n_steps);
                // Row r of the CTA's kHalves * 128 rows of B, in items of 16 codes: thread -> item te % ipr of rows te / ipr,
                // + 256 / ipr, ... (ipr = items per row = rc / 16; a row's items lie in neighbouring lanes)
                const int ipr = rc / 16, ipr_log = rc == 64 ? 2 : rc == 32 ? 1 : 0;
                constexpr int kItems = kHalves * 128 * 4 / 256;                   // per thread, for rc = 64
                const int n_items = kHalves * 128 * ipr;
                constexpr int kAhead = 2;                         // steps whose codes are on their way in registers
                uint4 cur[kAhead][kItems];
                float csc[kAhead][kItems];
                auto request = [&](uint4 (&c)[kItems], float (&sc)[kItems], int li) {
                    const P2Step e = mt.steps[li < n_steps ? li : 0];
#pragma unroll
                    for (int v = 0; v < kItems; ++v) {
                        const int u = te + v * 256, r = u >> ipr_log, c16 = u & (ipr - 1);
                        const int n = tl.n0_local + (r >> 7) * 256 + (int)rank * 128 + (r & 127);   // feature within the slice
                        c[v] = make_uint4(0u, 0u, 0u, 0u);
                        sc[v] = 0.0f;
                        if (li < n_steps && u < n_items && n < tl.n_s) {
                            const size_t row = (size_t)e.lora * tl.n_s + (size_t)n;
                            const size_t el = row * p.R + (size_t)e.chunk * rc + (size_t)c16 * 16;
                            if (p.lora_fmt == kLoraFp8) {
                                c[v] = ldg_ahead16(static_cast<const uint8_t*>(p.b[tl.s]) + el);
                                sc[v] = ldg_ahead_f32(static_cast<const float*>(p.sb[tl.s]) + row);
                            } else {
                                const uint2 w = ldg_ahead8(static_cast<const uint8_t*>(p.b[tl.s]) + el / 2);
                                c[v] = make_uint4(w.x, w.y, ldg_ahead_u8(static_cast<const uint8_t*>(p.sb[tl.s]) + el / 16), 0u);
                                sc[v] = ldg_ahead_f32(p.bg + (size_t)tl.s * p.L + e.lora);
                            }
                        }
                    }
                };
#pragma unroll
                for (int a = 0; a < kAhead; ++a) request(cur[a], csc[a], a);
                bool conv_ok = true;
                auto convert = [&](uint4 (&c)[kItems], float (&sc)[kItems], int li) {
                    const int st = (it + walk.slot_of_step(li)) % kStages;
                    int go = 1;
                    if (lane == 0) {                          // the producer has acquired the step's slot
                        const uint64_t t_start = ctrl->b_grant <= taken + li ? global_timer_ns() : 0;
                        for (uint32_t spin = 1; ctrl->b_grant <= taken + li; ++spin) {
                            if (ctrl->abort_flag) { go = 0; break; }
                            if ((spin & 63u) == 0 && global_timer_ns() - t_start > limit_ns) {
                                p2_timeout(p, ctrl, 17, it + li);
                                go = 0;
                                break;
                            }
                        }
                        __threadfence_block();
                    }
                    conv_ok = __shfl_sync(0xffffffffu, go, 0) != 0;
                    if (!conv_ok) return;
                    uint8_t* slot = ring + (size_t)st * kSlot;
#pragma unroll
                    for (int v = 0; v < kItems; ++v) {
                        const int u = te + v * 256, r = u >> ipr_log, c16 = u & (ipr - 1);
                        if (u < n_items) {
                            uint32_t o[8];
                            if (p.lora_fmt == kLoraFp8) e4m3x16_to_bf16(c[v], sc[v], o);
                            else e2m1x16_to_bf16(c[v].x, c[v].y, c[v].z, sc[v], o);
                            uint8_t* half = slot + (r >> 7) * kP2WBytes;
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                uint32_t off = (uint32_t)(r & 127) * (uint32_t)(rc * 2) + (uint32_t)(2 * c16 + h) * 16u;
                                off ^= ((off >> 7) & (uint32_t)(2 * ipr - 1)) << 4;
                                *reinterpret_cast<uint4*>(half + off) = make_uint4(o[4 * h], o[4 * h + 1], o[4 * h + 2], o[4 * h + 3]);
                            }
                        }
                    }
                    fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctrl->conv[st]);
                    request(c, sc, li + kAhead);
                };
                for (int li = 0; li < n_steps && conv_ok; li += kAhead) {
#pragma unroll
                    for (int a = 0; a < kAhead; ++a)
                        if (li + a < n_steps && conv_ok) convert(cur[a], csc[a], li + a);
                }
                it += p.kblocks + n_steps;
                taken += n_steps;
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            if constexpr (EXTRA) {
                // The tile's piece of the residual stream on its way to L2 while the main loop runs: one request per 128 bytes
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (ctrl->go_flag) {
                    for (int u = te; u < 128 * (kRows / 64); u += 256) {
                        const int rr = mt.rowmap[(int)rank * 128 + u / (kRows / 64)];
                        if (rr >= 0 && (u % (kRows / 64)) * 64 < tl.n_s - tl.n0_local)
                            prefetch_l2(p.residual + (int64_t)rr * p.ldr + tl.slice_off + tl.n0_local + (u % (kRows / 64)) * 64);
                    }
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            if (te == 0) {
                int go = ctrl->go_flag != 0 && ctrl->abort_flag == 0;
                if (go && !mbar_wait_cluster(&ctrl->acc_full[i % kAccBufs], (uint32_t)((i / kAccBufs) & 1), limit_ns)) {
                    p2_timeout(p, ctrl, 7, i);
                    go = 0;
                }
                ctrl->go_flag = go;
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const int go = ctrl->go_flag;
            asm volatile("bar.sync 1, 256;" ::: "memory");    // everyone has read the flag before its next writer runs
            if (!go) break;
            tc_fence_after();
            // Thread = one token (tensor-memory lane); a load brings 32 consecutive features of it, 64 contiguous bytes of
            // the token's row in y.  Stored as they come, a warp's store instruction would touch 32 rows with 16 bytes each and
            // the tile's read-out is bound by the store unit (measured: 18 k cycles per 512-feature tile, a third of the
            // kernel, spent with the tensor pipe idle).  So every four lanes transpose their 4 x 4 sixteen-byte pieces first
            // (two shuffle stages): lane j of a group then holds piece j of each of the group's four tokens, and a store
            // instruction writes 64 contiguous bytes of 8 rows.  No staging in shared memory, no barrier between the warps.
            const int c_tok = (int)rank * 128 + q * 32 + lane;
            const int row = mt.rowmap[c_tok];
            const float sc = mt.scale[c_tok];
            const int lj = lane & 3;
            const int n_left = tl.n_s - tl.n0_local - lj * 8;  // features of this lane's pieces that lie in the slice: whole pieces (widths % 8 == 0)
            int rr4[4];                                       // the rows of y this lane stores pieces of (-1: none)
#pragma unroll
            for (int r = 0; r < 4; ++r) rr4[r] = __shfl_sync(0xffffffffu, row, (lane & ~3) + r);
            const int64_t col = tl.slice_off + tl.n0_local + lj * 8;
            const uint32_t acc = tmem_base + (uint32_t)(i % kAccBufs) * 256u + lane_addr;
#pragma unroll 1
            for (int h = 0; h < kHalves; ++h) {
                // This warp's 128 features of the half, scaled and rounded to bf16 into registers first: the accumulator is free
                // for the next tile's MMAs after eight tensor-memory loads instead of at the pace of the stores.
                const int cb = h * 256 + (warp >= 8 ? 128 : 0);
                uint32_t pk[64];
#pragma unroll
                for (int c = 0; c < 8; ++c) {                 // (16 columns a load: 32 spilled)
                    uint32_t r[16];
                    tmem_ld16(acc + (uint32_t)(cb + c * 16), r);
                    tmem_ld_wait();
#pragma unroll
                    for (int u = 0; u < 8; ++u) pk[c * 8 + u] = pack_bf16x2(__uint_as_float(r[2 * u]) * sc, __uint_as_float(r[2 * u + 1]) * sc);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(cluster_peer_addr(smem_u32(&ctrl->acc_empty[kHalves == 2 ? h : i % kAccBufs]), 0));
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int c0 = cb + c * 32;
                    uint32_t* o = pk + c * 16;                // o[4 v + u]: piece v (8 features), register u
                    uint4 res[4];                             // EXTRA: the residual's pieces (the same thread reads and writes an
                    if constexpr (EXTRA) {                    // element: y may be the residual)
#pragma unroll
                        for (int r4 = 0; r4 < 4; ++r4)
                            res[r4] = rr4[r4] >= 0 && c0 < n_left ? *reinterpret_cast<const uint4*>(p.residual + (int64_t)rr4[r4] * p.ldr + col + c0)
                                                                  : make_uint4(0u, 0u, 0u, 0u);
                    }
#pragma unroll
                    for (int v = 0; v < 2; ++v)               // 2 x 2 blocks of pieces change places between lanes j and j ^ 2
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint32_t send = (lj & 2) ? o[v * 4 + u] : o[(v + 2) * 4 + u];
                            const uint32_t recv = __shfl_xor_sync(0xffffffffu, send, 2);
                            if (lj & 2) o[v * 4 + u] = recv; else o[(v + 2) * 4 + u] = recv;
                        }
#pragma unroll
                    for (int v = 0; v < 4; v += 2)            // then the pieces inside each block between lanes j and j ^ 1
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const uint32_t send = (lj & 1) ? o[v * 4 + u] : o[(v + 1) * 4 + u];
                            const uint32_t recv = __shfl_xor_sync(0xffffffffu, send, 1);
                            if (lj & 1) o[v * 4 + u] = recv; else o[(v + 1) * 4 + u] = recv;
                        }
                    if constexpr (EXTRA) {
#pragma unroll
                        for (int r4 = 0; r4 < 4; ++r4) {
                            o[r4 * 4] = add_bf16x2(o[r4 * 4], res[r4].x);
                            o[r4 * 4 + 1] = add_bf16x2(o[r4 * 4 + 1], res[r4].y);
                            o[r4 * 4 + 2] = add_bf16x2(o[r4 * 4 + 2], res[r4].z);
                            o[r4 * 4 + 3] = add_bf16x2(o[r4 * 4 + 3], res[r4].w);
                        }
                    }
#pragma unroll
                    for (int r4 = 0; r4 < 4; ++r4)            // o[4 r4 ..]: piece lj of the group's token r4
                        if (rr4[r4] >= 0 && c0 < n_left)
                            *reinterpret_cast<uint4*>(p.y + (int64_t)rr4[r4] * p.ldy + col + c0) =
                                make_uint4(o[r4 * 4], o[r4 * 4 + 1], o[r4 * 4 + 2], o[r4 * 4 + 3]);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&ctrl->meta_empty[i & 1]);
        }
    }
    // ---- teardown: neither CTA leaves (or frees tensor memory) while its partner may still read its shared memory, write
    // its tensor memory or arrive on its barriers
    if (ctrl->abort_flag) __nanosleep(200000);
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base, 512);
    }
}

template <bool FP4, int HALVES>
static void pair_launch_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int pairs, int pdl, cudaStream_t stream) {
    *cfg = cudaLaunchConfig_t{};
    cfg->gridDim = dim3((unsigned)(2 * pairs));
    cfg->blockDim = dim3(kP2Threads);
    cfg->dynamicSmemBytes = 1024 + (size_t)p2_stages(FP4, HALVES) * (size_t)p2_slot_bytes(FP4, HALVES) + sizeof(P2Ctrl) + 64;
    cfg->stream = stream;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg->attrs = attr;
    cfg->numAttrs = pdl ? 2 : 1;
}

int k2_prefill_pair_max_steps() { return kP2MaxSteps; }
int k2_prefill_pair_tiles(const int32_t* widths, int S, int halves) { return p2_n_tiles(widths, S, 256 * halves); }

// Resident pairs of the kernel on the current device (a pair sits inside one GPC, so fewer may fit than SMs / 2); 0 if the
// device takes none.
int k2_prefill_pair_capacity() {
    static std::atomic<int> cached[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return 0; }
    int n = cached[dev].load();
    if (n > 0) return n;
    if (cudaFuncSetAttribute(k2_prefill_pair_kernel<false, 2, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    pair_launch_config<false, 2>(&cfg, attr, 148, 0, nullptr);
    n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k2_prefill_pair_kernel<false, 2, false, false>, &cfg) != cudaSuccess) { (void)cudaGetLastError(); return 0; }
    cached[dev].store(n);
    return n;
}

template <bool FP4, int HALVES, bool EXTRA, bool STORED>
static cudaError_t launch_pair_impl(const K2pParams& p, const CUtensorMap& tm_w, const CUtensorMap& tm_x, const CUtensorMap& tm_h,
                                    const CUtensorMap* tm_b, const CUtensorMap* tm_sf, int pairs, int pdl, cudaStream_t stream) {
    static std::atomic<unsigned long long> configured{0};     // devices whose limit on dynamic shared memory was raised
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && !(configured.load() & (1ull << dev))) {
        // the epilogue's warps wait for the registers the others give back: a build that launched with fewer than the split adds
        // up to would wait for good, so it is refused here
        cudaFuncAttributes fa;
        e = cudaFuncGetAttributes(&fa, k2_prefill_pair_kernel<FP4, HALVES, EXTRA, STORED>);
        if (e != cudaSuccess) return e;
        if (fa.numRegs * 4 < 2 * kP2RegsRoles + 2 * kP2RegsEpilogue) return cudaErrorLaunchOutOfResources;
        e = cudaFuncSetAttribute(k2_prefill_pair_kernel<FP4, HALVES, EXTRA, STORED>, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024);
        if (e != cudaSuccess) return e;
        configured.fetch_or(1ull << dev);
    }
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[2];
    pair_launch_config<FP4, HALVES>(&cfg, attr, pairs, pdl, stream);
    return cudaLaunchKernelEx(&cfg, k2_prefill_pair_kernel<FP4, HALVES, EXTRA, STORED>, p, tm_w, tm_x, tm_h, tm_b[0], tm_b[1], tm_b[2],
                              tm_b[3], FP4 ? tm_sf[0] : tm_w, FP4 ? tm_sf[1] : tm_w);
}

template <bool EXTRA, bool STORED>
static cudaError_t launch_pair_form(const K2pParams& p, const CUtensorMap& tm_w, const CUtensorMap& tm_x, const CUtensorMap& tm_h,
                                    const CUtensorMap* tm_b, const CUtensorMap* tm_sf, int pairs, int fp4, int halves, int pdl,
                                    cudaStream_t stream) {
    return fp4           ? launch_pair_impl<true, 1, EXTRA, STORED>(p, tm_w, tm_x, tm_h, tm_b, tm_sf, pairs, pdl, stream)
           : halves == 1 ? launch_pair_impl<false, 1, EXTRA, STORED>(p, tm_w, tm_x, tm_h, tm_b, tm_sf, pairs, pdl, stream)
                         : launch_pair_impl<false, 2, EXTRA, STORED>(p, tm_w, tm_x, tm_h, tm_b, tm_sf, pairs, pdl, stream);
}

// tm_sf: NVFP4 base only, the packed W block scales and the workspace's token block scales as [rows, 256] byte tensors
cudaError_t launch_k2_prefill_pair(const K2pParams& p, const CUtensorMap& tm_w, const CUtensorMap& tm_x, const CUtensorMap& tm_h,
                                   const CUtensorMap* tm_b, const CUtensorMap* tm_sf, int pairs, int fp4, int halves, int pdl,
                                   cudaStream_t stream) {
    const bool extra = p.residual != nullptr, stored = p.lora_fmt != kLoraBf16;
    if (extra)
        return stored ? launch_pair_form<true, true>(p, tm_w, tm_x, tm_h, tm_b, tm_sf, pairs, fp4, halves, pdl, stream)
                      : launch_pair_form<true, false>(p, tm_w, tm_x, tm_h, tm_b, tm_sf, pairs, fp4, halves, pdl, stream);
    return stored ? launch_pair_form<false, true>(p, tm_w, tm_x, tm_h, tm_b, tm_sf, pairs, fp4, halves, pdl, stream)
                  : launch_pair_form<false, false>(p, tm_w, tm_x, tm_h, tm_b, tm_sf, pairs, fp4, halves, pdl, stream);
}

}  // namespace ob
