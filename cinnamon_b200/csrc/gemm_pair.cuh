// Two-SM variant of the dense block-scaled FP8 GEMM (included by gemm.cu).
//
// A cluster of two CTAs on neighbouring SMs computes a 256 x 256 output tile with
// tcgen05.mma.cta_group::2: CTA r holds rows [128 r, 128 r + 128) of A and columns
// [128 r, 128 r + 128) of B in its own shared memory and the 128 x 256 accumulator rows
// in its own tensor memory.  Each SM therefore stages 32 KiB per K block instead of 48 KiB
// and the tensor pipe reads a third less shared memory per MMA.  One thread of the even
// (leader) CTA issues the MMAs for the pair; completion is signalled to a barrier in each
// CTA.  TMA loads are plain per-CTA loads: each CTA fetches only its own halves and reports
// the bytes to the leader's "operands landed" barrier.
//
// Roles per CTA (12 warps): 0-7 promotion, 8 TMA producer, 9 TMEM allocation and, in the leader, the MMAs; 10 hands finished
// tiles to the TMA unit; 11 brings the scales and the tiles' coordinates.  All waits are bounded exactly as in the one-SM kernel.
//
// The promotion warps are the bound (a K block took them 840 cycles where its MMAs take 512, a tile 3500 around its K blocks), so
// they do nothing else: a tile's coordinates cost them 850 cycles of divisions, its stores up to 1000 of waiting for the TMA unit, and
// the scales registers and a round trip per tile.  The scales now arrive through shared memory, on the barrier that reports
// the MMAs.  16384 x 7168 -> 18432 1915 -> 1708 us, 16384 x 576 -> 7168 102 -> 81, 32768 x 512 -> 1024 32.7 -> 28.3, 32768 rows of 7168 -> 4096 by
// 32 experts and the way back with it 4.38 -> 4.29 ms, all cool.  (Sixteen warps of 64 columns, to hide more latency: 1957, 89 and 30.)
#pragma once

namespace pair {

constexpr int PM = 256;                 // rows of the pair's tile
constexpr int PN = 256;                 // columns of the pair's tile
constexpr int PSTAGES = 4;               // even (see the one-SM kernel); leaves room for a whole output tile
constexpr int PA_BYTES = 128 * BK;      // A rows of this CTA: 16 KiB
constexpr int PB_BYTES = 128 * BK;      // B columns of this CTA: 16 KiB
constexpr int PEPI = 8;                 // promotion warps: four TMEM lane quarters x two groups of PCOLS columns
constexpr int PCOLS = PN / (PEPI / 4);
constexpr int PTMA = PEPI, PMMA = PEPI + 1, PSTORE = PEPI + 2, PSCALE = PEPI + 3;
constexpr int PTHREADS = (PEPI + 4) * 32;
constexpr int PFETCH = 8;               // K blocks whose scales are on their way
constexpr int PSCALE_SLOTS = 16;        // K blocks whose scales have a place: one per row, two columns'
constexpr int PSCALES = 128 + 4;
constexpr int PSCALE_BYTES = PSCALE_SLOTS * PSCALES * 4;
constexpr int PTILE_SLOTS = 16;         // coordinates of the next tiles: {m0, n0, one past the last row, expert}
// dynamic shared memory: operand stages | two 4 KiB output boxes per promotion warp = the CTA's whole 128 x 256 tile of a
// 2-byte type (TMA-store boxes; also the 2 KiB-per-warp staging of the non-TMA path) | scales | tiles | 256 B of barriers and
// flags, plus 1 KiB of slack to align the stages to 1024 bytes
constexpr int PSTAGE_OFF = PSTAGES * (PA_BYTES + PB_BYTES);
constexpr int PBOX_BYTES = STORE_ROWS * 128;  // one TMA-store box
constexpr int PBOXES = 16 / PEPI;       // boxes per promotion warp: a round of them all is 64 KiB, a CTA's tile of a 2-byte type
constexpr int PC_BYTES = PEPI * PBOXES * PBOX_BYTES;
constexpr size_t PSMEM_BYTES = (size_t)PSTAGE_OFF + PC_BYTES + PSCALE_BYTES + PTILE_SLOTS * 16 + 256 + 1024;

__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// shared::cluster address of the same shared-memory offset in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on a barrier of the other CTA.  Relaxed: the barrier hands over a tensor-memory buffer whose reads
// are already complete (tcgen05.wait::ld + tcgen05.fence), no generic-memory data is published by it, and a
// cluster-scope release here costs over a thousand cycles per K block.
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// TMA load into this CTA's shared memory whose byte count is reported to a barrier that may live in
// the other CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(const CUtensorMap* map, uint32_t bar_cluster, uint32_t dst, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar_cluster), "r"(x), "r"(y) : "memory");
}
// Both are called by a whole warp and issued by the lane that elect.sync chooses.
// Completion of the pair's MMAs issued so far is reported to the barrier at the same offset in BOTH CTAs:
// one commit per CTA, each naming that CTA's barrier by its cluster address.
__device__ __forceinline__ void tc_commit_pair(uint32_t own, uint32_t peer) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t"
        "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%1];\n\t}"
        ::"r"(own), "r"(peer) : "memory");
}
// The four MMAs of a K block, by one election; only the low words of the descriptors vary.  STEP_B: 16-byte units from one step's B to the next
template <int STEP_B>
__device__ __forceinline__ void tc_mma_f8_pair(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
    constexpr uint32_t hi = (uint32_t)((((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61)) >> 32);
    asm volatile(
        "{\n\t.reg .pred e;\n\t.reg .b64 a, b;\n\t.reg .b32 x, y;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "mov.b64 a, {%1, %4};\n\tmov.b64 b, {%2, %4};\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], a, b, %3, 0;\n\t"
        "add.u32 x, %1, 2;\n\tadd.u32 y, %2, %5;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], a, b, %3, 1;\n\t"
        "add.u32 x, %1, 4;\n\tadd.u32 y, %2, %6;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], a, b, %3, 1;\n\t"
        "add.u32 x, %1, 6;\n\tadd.u32 y, %2, %7;\n\tmov.b64 a, {x, %4};\n\tmov.b64 b, {y, %4};\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], a, b, %3, 1;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(hi), "n"(STEP_B), "n"(2 * STEP_B), "n"(3 * STEP_B) : "memory");
}
__host__ __device__ constexpr uint32_t make_idesc_pair(bool b_mn_major) {
    return (1u << 4) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(PN >> 3) << 17) | ((uint32_t)(PM >> 4) << 24);
}

struct PairTile { int m0, n0; };

__device__ __forceinline__ int pair_total(const GemmParams& p) {
    return ((p.M + PM - 1) / PM) * ((p.N + PN - 1) / PN);
}
__device__ __forceinline__ PairTile pair_tile(const GemmParams& p, int t) {
    const int m_tiles = (p.M + PM - 1) / PM, n_tiles = (p.N + PN - 1) / PN;
    constexpr int GROUP = 16;                      // 16 x 256 rows per L2 group
    const int per_group = GROUP * n_tiles;
    const int g = t / per_group;
    const int first_m = g * GROUP;
    const int gsize = min(GROUP, m_tiles - first_m);
    const int r = t - g * per_group;
    PairTile ti;
    ti.m0 = (first_m + r % gsize) * PM;
    ti.n0 = (r / gsize) * PN;
    return ti;
}

// GK ("grouped K"): E independent problems of the same M x N whose reduction ranges differ - the weight gradients
// of the experts, dW[e] = dY[rows of e]^T @ x[rows of e].  Both operands are K-major over one padded token axis on
// which expert e owns the K blocks [kb_start[e], kb_start[e + 1]) (p.starts holds that int array, p.E = E); tile t
// belongs to expert t / (tiles per expert) and is stored at rows e * M + ... of the (E * M, N) output.  An expert
// without rows gets zeros.  Without kb_start (null) the E "experts" are equal pieces of one problem's reduction, whose partial sums
// split_sum_kernel adds.  The kernel keeps the array in shared memory: while the stores saturate memory, each role's two loads per
// tile cost it thousands of cycles (32 experts of 512 rows, 2048 x 2048 in bf16: 182 -> 172 us).
// OWN: the promotion warps load their scales themselves, for experts of few K blocks: see fp8_gemm_grouped_k.
//
// GR ("grouped rows"): E independent problems of the same N x K over the ragged row ranges [starts[e], ends[e]) of A and C
// (device arrays), B stacked (E * b_rows_per_expert rows).  The tiles of all experts are one list, found through a prefix sum
// of their tile counts in shared memory behind the barriers; a CTA whose 128 rows are not all its expert's stores them with
// row predicates.  Worth it from a few tiles of rows per expert on: see fp8_grouped_gemm.
template <bool B_MN, int OUT, bool GK = false, bool GR = false, bool OWN = false>
__global__ void __launch_bounds__(PTHREADS, 1)
fp8_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem + PSTAGES * PA_BYTES;
    uint8_t* c_stage = smem + PSTAGE_OFF;
    float* scales = reinterpret_cast<float*>(c_stage + PC_BYTES);
    int4* tiles = reinterpret_cast<int4*>(c_stage + PC_BYTES + PSCALE_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + PTILE_SLOTS);
    // [0, S) full (used in the leader), [S, 2S) empty, [2S, 2S+2) tmem full, [2S+2, 2S+4) tmem empty (leader), then: all boxes of a
    // round are staged, they have been read
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * PSTAGES + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* cum = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + 256);  // E + 1 prefix counts, GR: of row tiles, GK: of K blocks

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();           // 0 = leader
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + PSTAGES);
    const uint32_t tfull0 = smem_u32(bars + 2 * PSTAGES), tempty0 = smem_u32(bars + 2 * PSTAGES + 2);
    const uint32_t staged = smem_u32(bars + 2 * PSTAGES + 4), taken = smem_u32(bars + 2 * PSTAGES + 5);

    if (threadIdx.x == 0) *abort_flag = 0;
    if (warp == PTMA && lane == 0) {
        for (int s = 0; s < PSTAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tfull0 + 8 * b, OWN ? 1 : 2); mbar_init(tempty0 + 8 * b, 2 * PEPI); }
        mbar_init(staged, PEPI);
        mbar_init(taken, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == PMMA) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();                                        // (all of the above is this block's own; from here on, memory is read)
    if (warp == PMMA) pdl_trigger();
    if constexpr (GR) {
        if (warp == 0) tile_prefix_sum(p, cum, PM, lane);
    }
    if constexpr (GK) {
        const int* start = reinterpret_cast<const int*>(p.starts);
        for (int e = threadIdx.x; e <= p.E; e += PTHREADS)
            cum[e] = start ? start[e] : (int)((int64_t)((p.K + BK - 1) / BK) * e / p.E);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                    // both CTAs' barriers exist before anyone signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // A 4-byte tile leaves in two rounds, and the experts' gradients of either size are bound by their stores: there the promotion warps
    // hand over their own boxes, so that each waits for its own to be read and not for everybody's (weight gradients of 32 experts
    // of 64 rows, 2048 x 2048 in bf16, with their quantisers 98 -> 91 us).
    constexpr bool TWO_BYTE = sizeof(typename OutT<OUT>::type) == 2, STORE_WARP = TWO_BYTE && !GK;
    const int KB_dense = (p.K + BK - 1) / BK;
    const int per_expert = pair_total(p);
    const int n_tiles = (p.N + PN - 1) / PN;
    const int n_total = GR ? cum[p.E] * n_tiles : (GK ? per_expert * p.E : per_expert);
    const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    // tile t -> its coordinates inside one problem (GR: among all rows), the expert it belongs to, its K blocks, and one past
    // the last row it may write
    auto locate = [&](int t, PairTile& ti, int& e, int& kb0, int& KB, int& m_end) {
        m_end = p.M;
        if constexpr (GR) {
            const int mt = t / n_tiles;
            int lo = 0, hi = p.E;                      // largest e with cum[e] <= mt
            while (hi - lo > 1) {
                const int mid = (lo + hi) >> 1;
                if (cum[mid] <= mt) lo = mid; else hi = mid;
            }
            e = lo; kb0 = 0; KB = KB_dense;
            const long long first = p.starts[lo], last = p.ends[lo];
            ti.m0 = (int)first + (mt - cum[lo]) * PM;
            ti.n0 = (t - mt * n_tiles) * PN;
            m_end = (int)(last < (long long)p.M ? last : (long long)p.M);
        } else if constexpr (GK) {
            e = t / per_expert;
            ti = pair_tile(p, t - e * per_expert);
            kb0 = cum[e];
            KB = cum[e + 1] - kb0;
        } else {
            e = 0; kb0 = 0; KB = KB_dense;
            ti = pair_tile(p, t);
        }
    };

    if (warp == PTMA) {
        // ------------------------------ TMA producer (both CTAs) ------------------------------
        if (lane == 0) {
            const uint32_t full_leader = mapa(full0, 0);
            uint32_t it = 0;
            bool alive = true;
            for (int t = cluster_id; t < n_total && alive; t += n_clusters) {
                PairTile ti; int e, kb0, KB, m_end;
                locate(t, ti, e, kb0, KB, m_end);
                const int b_row0 = GR ? e * p.b_rows_per_expert : 0;
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const int s = it % PSTAGES;
                    const uint32_t ph = (it / PSTAGES) & 1;
                    if (!mbar_wait(empty0 + 8 * s, ph ^ 1, abort_flag, (1 << 8) | 1)) { alive = false; break; }
                    if (rank == 0) mbar_expect_tx(full0 + 8 * s, 2 * (PA_BYTES + PB_BYTES));
                    const uint32_t fb = full_leader + 8 * s;
                    tma_load_2d_pair(&tmA, fb, smem_u32(smem_a + s * PA_BYTES), (kb0 + kb) * BK, ti.m0 + 128 * (int)rank);
                    if constexpr (!B_MN) tma_load_2d_pair(&tmB, fb, smem_u32(smem_b + s * PB_BYTES), (kb0 + kb) * BK, b_row0 + ti.n0 + 128 * (int)rank);
                    else tma_load_2d_pair(&tmB, fb, smem_u32(smem_b + s * PB_BYTES), ti.n0 + 128 * (int)rank, b_row0 + (kb0 + kb) * BK);
                }
            }
            if (!alive) {
                // abandoned: the barrier that counts this CTA's copies may live in the other CTA, so just give
                // the copies already issued ample time to land before shared memory is given up
                const long long t0 = clock64();
                while (clock64() - t0 < 2000000LL) { }
            }
        }
    } else if (!OWN && warp == PSCALE) {
        // ------------------ scales (both CTAs): this CTA's rows' and both column blocks', K block by K block ------------------
        // Copied to where they are read, PFETCH blocks ahead.  Through registers, a block's values waited for the loads issued last, four
        // blocks on: a miss for every row each eighth block (8837 x 17024 -> 320, one wave of tiles: 101 us so, 69 like this).  Multiplied here
        // and not by their readers: 1 to 2 % slower on long reductions (the warp takes issue slots of two promotion warps).
        const float* a_ptr[4];
        const float* b_ptr[2];
        int t = cluster_id - n_clusters, left = 0;     // K blocks of the tile that are still to be fetched
        uint32_t entered = 0;
        uint32_t fetched = 0;
        auto copy4 = [](uint32_t dst, const float* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); };
        auto fetch = [&](uint32_t block) {
            while (left == 0) {
                t += n_clusters;
                if (t >= n_total) { t = n_total; return; }           // (and stays there)
                PairTile ti; int e, kb0, m_end;
                locate(t, ti, e, kb0, left, m_end);
                // (sixteen slots: the slot's last tile has left the promotion warps even when tiles have one K block)
                if (lane == 0) tiles[entered % PTILE_SLOTS] = make_int4(ti.m0, ti.n0, m_end, e);
                ++entered;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int row = ti.m0 + 128 * (int)rank + i * 32 + lane;
                    a_ptr[i] = p.sA + (int64_t)(row < m_end ? row : (GR ? ti.m0 : 0)) * p.sa_stride_m + (int64_t)kb0 * p.sa_stride_k;
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int col = ti.n0 + c * 128;
                    b_ptr[c] = p.sB + (int64_t)(col < p.N ? col / 128 : 0) * p.sb_stride_n + (int64_t)kb0 * p.sb_stride_k
                               + (GR ? (int64_t)e * p.sb_stride_e : 0);
                }
            }
            const uint32_t to = smem_u32(scales + block % PSCALE_SLOTS * PSCALES);
#pragma unroll
            for (int i = 0; i < 4; ++i) { copy4(to + (i * 32 + lane) * 4, a_ptr[i]); a_ptr[i] += p.sa_stride_k; }
            if (lane < 2) copy4(to + (128 + lane) * 4, lane == 0 ? b_ptr[0] : b_ptr[1]);
#pragma unroll
            for (int c = 0; c < 2; ++c) b_ptr[c] += p.sb_stride_k;
            --left;
            ++fetched;
        };
#pragma unroll 1
        for (int u = 0; u < PFETCH; ++u) {
            fetch(u);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        for (uint32_t it = 0; it < fetched; ++it) {
            asm volatile("cp.async.wait_group %0;" ::"n"(PFETCH - 1) : "memory");
            __syncwarp();
            // (that barrier cannot complete again without the arrival below; and once the MMAs of block it - 2 are done, every reader of
            // block it - 4 has released its buffer, so that the slot of block it - 8 may be filled again)
            if (it >= 2 && !mbar_wait_warp(tfull0 + 8 * (it & 1), ((it - 2) >> 1) & 1, abort_flag, (4 << 8) | 1)) break;
            if (lane == 0) mbar_arrive(tfull0 + 8 * (it & 1));
            fetch(it + PFETCH);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == PSTORE || warp == PSCALE) {
        // ------------------------------ finished tiles to the TMA unit (both CTAs) ------------------------------
        // A lane sends a box.  A tile's 64 KiB leave the SM in a thousand cycles and an issue blocks until the unit
        // takes it: promotion warps that issued their own stores stood still for most of that.
        if (STORE_WARP && warp == PSTORE && p.tma_out) {
            constexpr int EPR = 128 / (int)sizeof(typename OutT<OUT>::type);
            const int w = lane / PBOXES, q = w & 3, h = w >> 2;
            uint32_t round = 0;
            bool alive = true;
            for (int t = cluster_id; t < n_total && alive; t += n_clusters) {
                PairTile ti; int e, kb0, KB, m_end;
                locate(t, ti, e, kb0, KB, m_end);
                const int row = ti.m0 + 128 * (int)rank + q * 32;
                const int out_row0 = GR ? 0 : e * p.M;
                for (int r = 0; r < PCOLS / (PBOXES * EPR); ++r, ++round) {
                    const int col = ti.n0 + h * PCOLS + (r * PBOXES + lane % PBOXES) * EPR;
                    if (!mbar_wait_warp(staged, round & 1, abort_flag, (5 << 8) | 1)) { alive = false; break; }
                    if (lane < PEPI * PBOXES) {
                        if (col < p.N && (!(GR || GK) || row + 32 <= m_end)) tma_store_2d(&tmC, smem_u32(c_stage) + lane * PBOX_BYTES, col, out_row0 + row);
                        tma_store_commit();
                        tma_store_wait_read();
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(taken);
                }
            }
            if (lane < PEPI * PBOXES) tma_store_wait_all();     // the boxes have reached global memory
        }
    } else if (warp == PMMA) {
        // ------------------ MMA issuer (leader only; a whole warp, as in the one-SM kernel) ------------------
        if (rank == 0) {
            constexpr uint32_t idesc = make_idesc_pair(B_MN);
            const uint32_t tfull_own = mapa(tfull0, 0), tfull_peer = mapa(tfull0, 1);
            const uint32_t empty_own = mapa(empty0, 0), empty_peer = mapa(empty0, 1);
            const uint32_t a0 = ((smem_u32(smem_a) >> 4) & 0x3FFF) | (1u << 16), b0 = ((smem_u32(smem_b) >> 4) & 0x3FFF) | (1u << 16);
            uint32_t it = 0;
            bool alive = true;
            for (int t = cluster_id; t < n_total && alive; t += n_clusters) {
                int KB = KB_dense;
                if constexpr (GK) {
                    PairTile ti_; int e_, kb0_, end_;
                    locate(t, ti_, e_, kb0_, KB, end_);
                }
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    const uint32_t s = it % PSTAGES, ph = (it / PSTAGES) & 1;
                    const uint32_t b = it & 1, bph = (it >> 1) & 1;
                    if (!mbar_wait_warp(full0 + 8 * s, ph, abort_flag, (2 << 8) | 1)) { alive = false; break; }
                    if (!mbar_wait_warp(tempty0 + 8 * b, bph ^ 1, abort_flag, (2 << 8) | 2)) { alive = false; break; }
                    tc_fence_after();
                    tc_mma_f8_pair<B_MN ? 256 : 2>(tmem_base + b * PN, a0 + s * (PA_BYTES >> 4), b0 + s * (PB_BYTES >> 4), idesc);
                    tc_commit_pair(tfull_own + 8 * b, tfull_peer + 8 * b);
                    tc_commit_pair(empty_own + 8 * s, empty_peer + 8 * s);
                }
            }
            if (alive && it) mbar_wait(tfull0 + 8 * ((it - 1) & 1), ((it - 1) >> 1) & 1, abort_flag, (2 << 8) | 3);
        }
    } else {
        // ------------------------------ promotion / epilogue (both CTAs) ------------------------------
        const int q = warp & 3, h = warp >> 2;
        const uint32_t tempty_leader = mapa(tempty0, 0);
        uint32_t it = 0;
        bool alive = true;
        const float* my_scales = scales + q * 32 + lane;
        const float* column_scale = scales + 128 + h * PCOLS / 128;
        const bool vec_ok = (OUT == CINN_F32 || OUT == CINN_F32_BF16) ? (p.ldc % 4 == 0) : (p.ldc % 8 == 0);
        uint32_t seen = 0, round = 0;
        for (int t = cluster_id; t < n_total && alive; t += n_clusters) {
            PairTile ti; int e, kb0, KB = KB_dense, m_end;
            if constexpr (GK) locate(t, ti, e, kb0, KB, m_end);       // (a tile without K blocks does not pass through the scale warp)
            float acc[PCOLS];
#pragma unroll
            for (int i = 0; i < PCOLS; ++i) acc[i] = 0.0f;
            // OWN: the warp's own scales, three blocks ahead
            const float *sa_ptr = nullptr, *sb_ptr = nullptr;
            float sa[3], sb[3];
            if constexpr (OWN) {
                sa_ptr = p.sA + (int64_t)(ti.m0 + 128 * (int)rank + q * 32 + lane) * p.sa_stride_m + (int64_t)kb0 * p.sa_stride_k;
                sb_ptr = p.sB + (int64_t)(ti.n0 / 128 + h) * p.sb_stride_n + (int64_t)kb0 * p.sb_stride_k;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    if (i < KB) { sa[i] = ld_scale(sa_ptr + i * p.sa_stride_k); sb[i] = ld_scale(sb_ptr + i * p.sb_stride_k); }
            }
            for (int kb = 0; kb < KB; ++kb, ++it) {
                const uint32_t b = it & 1, bph = (it >> 1) & 1;
                float s;
                if constexpr (OWN) {
                    s = sa[0] * sb[0];
                    sa[0] = sa[1]; sb[0] = sb[1]; sa[1] = sa[2]; sb[1] = sb[2];
                    if (kb + 3 < KB) { sa[2] = ld_scale(sa_ptr + (kb + 3) * p.sa_stride_k); sb[2] = ld_scale(sb_ptr + (kb + 3) * p.sb_stride_k); }
                }
                if (!mbar_wait_warp(tfull0 + 8 * b, bph, abort_flag, (3 << 8) | 1)) { alive = false; break; }
                tc_fence_after();
                if constexpr (!OWN) s = my_scales[(it % PSCALE_SLOTS) * PSCALES] * column_scale[(it % PSCALE_SLOTS) * PSCALES];
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + b * PN + h * PCOLS;
                // packed fp32x2 FMAs: half the issue slots of scalar ones, the same IEEE result in every lane
                uint64_t s2;
                asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
                for (int c = 0; c < PCOLS / 16; ++c) {
                    float v[16];
                    tc_ld16(taddr + c * 16, v);
#pragma unroll
                    for (int j = 0; j < 16; j += 2)
                        asm("{\n\t.reg .b64 a, x;\n\t"
                            "mov.b64 a, {%0, %1};\n\t"
                            "mov.b64 x, {%2, %3};\n\t"
                            "fma.rn.f32x2 a, x, %4, a;\n\t"
                            "mov.b64 {%0, %1}, a;\n\t}"
                            : "+f"(acc[c * 16 + j]), "+f"(acc[c * 16 + j + 1]) : "f"(v[j]), "f"(v[j + 1]), "l"(s2));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_remote(tempty_leader + 8 * b);
            }
            if (!alive) break;
            if constexpr (!GK) {                       // in shared memory since the tile's first scales (the divisions took 850 cycles here)
                const int4 x = tiles[seen++ % PTILE_SLOTS];
                ti.m0 = x.x; ti.n0 = x.y; m_end = x.z; e = x.w;
            }
            const int row = ti.m0 + 128 * (int)rank + q * 32 + lane;
            const bool rvalid = row < m_end;
            const int col0 = ti.n0 + h * PCOLS;
            const bool cvalid = col0 < p.N;
            const int out_row0 = GR ? 0 : e * p.M;                      // GK: the expert's slice of the (E * M, N) output
            if (GK || p.tma_out) {                                      // (what GK writes always goes through TMA)
                // The tile leaves through TMA stores.  Every promotion warp owns two boxes of 32 rows x 128 bytes (128-byte swizzle) of the
                // staging area, where its lanes drop their rows in 16-byte chunks.  A 2-byte output fits the warp's 128 columns in one
                // round, and the store warp issues it; a 4-byte output takes two rounds of 64.  Rows of two owners leave as
                // staged 16-byte stores.
                using T = typename OutT<OUT>::type;
                constexpr int EPR = 128 / (int)sizeof(T);          // elements per 128-byte box row
                constexpr int PER16 = 16 / (int)sizeof(T);
                const uint32_t slot = smem_u32(c_stage) + warp * PBOXES * PBOX_BYTES;
                const bool whole = !(GR || (GK && !TWO_BYTE)) || row - lane + 32 <= m_end;
#pragma unroll
                for (int r = 0; r < PCOLS / (PBOXES * EPR); ++r, ++round) {
                    if constexpr (STORE_WARP) {                   // the previous boxes have been read
                        if (!mbar_wait_warp(taken, (round & 1) ^ 1, abort_flag, (3 << 8) | 2)) { alive = false; break; }
                    } else {
                        if (lane == 0) tma_store_wait_read();
                        __syncwarp();
                    }
                    if (whole) {
#pragma unroll
                        for (int j = 0; j < PBOXES * 8; ++j) {
                            const uint4 v = pack16<OUT>(&acc[(r * PBOXES + (j >> 3)) * EPR + (j & 7) * PER16]);
                            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                                         ::"r"(slot + (j >> 3) * PBOX_BYTES + lane * 128 + (((j & 7) ^ (lane & 7)) << 4)), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
                        }
                        fence_async_smem();
                    } else if (r == 0 && cvalid) {
                        store_rows_staged<OUT, PCOLS>(acc, c_stage + warp * PBOXES * PBOX_BYTES, p.C, p.ldc, out_row0 + ti.m0 + 128 * (int)rank + q * 32,
                                                      out_row0 + m_end, col0, p.N, lane);
                    }
                    __syncwarp();
                    if constexpr (STORE_WARP) {
                        if (lane == 0) mbar_arrive(staged);
                    } else {
                        if (whole && lane == 0) {
#pragma unroll
                            for (int b = 0; b < PBOXES; ++b) {
                                const int col = col0 + (r * PBOXES + b) * EPR;
                                if (col < p.N) tma_store_2d(&tmC, slot + b * PBOX_BYTES, col, out_row0 + row);
                            }
                            tma_store_commit();
                        }
                        __syncwarp();   // the lane rejoins its warp before the next warp-collective instruction
                    }
                }
            } else if (vec_ok) {
                // an output that TMA cannot write: staged 16-byte stores
                if (cvalid) store_rows_staged<OUT, PCOLS>(acc, c_stage + warp * PBOXES * PBOX_BYTES, p.C, p.ldc,
                                                          out_row0 + ti.m0 + 128 * (int)rank + q * 32, out_row0 + m_end, col0, p.N, lane);
            } else if (rvalid && cvalid) {
                const int64_t base = (int64_t)(out_row0 + row) * p.ldc + col0;
#pragma unroll
                for (int j = 0; j < PCOLS / 8; ++j) {
                    const int ncols = p.N - (col0 + j * 8);
                    if (ncols > 0) store8<OUT>(p.C, base + j * 8, &acc[j * 8], false, ncols);
                }
            }
        }
        if (!STORE_WARP && lane == 0) tma_store_wait_all();            // this warp's boxes have reached global memory
    }

    // nobody leaves while the other CTA may still read this CTA's shared memory or signal its barriers
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == PMMA) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace pair
