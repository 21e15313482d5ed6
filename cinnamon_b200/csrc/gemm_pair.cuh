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
// Roles per CTA (11 warps): 0-7 promotion/epilogue, 8 TMA producer, 9 TMEM allocation;
// warps 9 and 10 of the leader issue the MMAs of alternate K blocks.  All waits are bounded exactly as in the one-SM kernel.
#pragma once

namespace pair {

constexpr int PM = 256;                 // rows of the pair's tile
constexpr int PN = 256;                 // columns of the pair's tile
constexpr int PSTAGES = 4;               // even (see the one-SM kernel); leaves room for a whole output tile
constexpr int PA_BYTES = 128 * BK;      // A rows of this CTA: 16 KiB
constexpr int PB_BYTES = 128 * BK;      // B columns of this CTA: 16 KiB
constexpr int PTHREADS = 11 * 32;
// dynamic shared memory: operand stages | two 4 KiB output boxes per promotion warp = the CTA's whole 128 x 256 tile of a
// 2-byte type (TMA-store boxes; also the 2 KiB-per-warp staging of the non-TMA path) | 256 B of barriers and flags, plus 1 KiB of
// slack to align the stages to 1024 bytes
constexpr int PSTAGE_OFF = PSTAGES * (PA_BYTES + PB_BYTES);
constexpr int PBOX_BYTES = STORE_ROWS * 128;  // one TMA-store box
constexpr int PC_BYTES = 8 * 2 * PBOX_BYTES;
constexpr size_t PSMEM_BYTES = (size_t)PSTAGE_OFF + PC_BYTES + 256 + 1024;

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
__device__ __forceinline__ void tc_mma_f8_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
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
// without rows gets zeros.  M and N are multiples of 256 here, so every tile is whole.
//
// GR ("grouped rows"): E independent problems of the same N x K over the ragged row ranges [starts[e], ends[e]) of A and C
// (device arrays), B stacked (E * b_rows_per_expert rows).  The tiles of all experts are one list, found through a prefix sum
// of their tile counts in shared memory behind the barriers; a CTA whose 128 rows are not all its expert's stores them with
// row predicates.  Worth it from a few tiles of rows per expert on: see fp8_grouped_gemm.
template <bool B_MN, int OUT, bool GK = false, bool GR = false>
__global__ void __launch_bounds__(PTHREADS, 1)
fp8_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const GemmParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* smem_a = smem;
    uint8_t* smem_b = smem + PSTAGES * PA_BYTES;
    uint8_t* c_stage = smem + PSTAGE_OFF;
    uint64_t* bars = reinterpret_cast<uint64_t*>(c_stage + PC_BYTES);
    // [0, S) full (used in the leader), [S, 2S) empty, [2S, 2S+2) tmem full, [2S+2, 2S+4) tmem empty (leader)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * PSTAGES + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* cum = reinterpret_cast<int*>(reinterpret_cast<uint8_t*>(bars) + 256);  // GR: E + 1 prefix counts of row tiles

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();           // 0 = leader
    const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + PSTAGES);
    const uint32_t tfull0 = smem_u32(bars + 2 * PSTAGES), tempty0 = smem_u32(bars + 2 * PSTAGES + 2);

    if (threadIdx.x == 0) *abort_flag = 0;
    if (warp == 8 && lane == 0) {
        for (int s = 0; s < PSTAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(tfull0 + 8 * b, 1); mbar_init(tempty0 + 8 * b, 16); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    pdl_wait();                                        // (all of the above is this block's own; from here on, memory is read)
    pdl_trigger();
    if constexpr (GR) {
        if (warp == 0) tile_prefix_sum(p, cum, PM, lane);
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();                                    // both CTAs' barriers exist before anyone signals them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    const int KB_dense = (p.K + BK - 1) / BK;
    const int per_expert = pair_total(p);
    const int n_tiles = (p.N + PN - 1) / PN;
    const int n_total = GR ? cum[p.E] * n_tiles : (GK ? per_expert * p.E : per_expert);
    const int cluster_id = blockIdx.x >> 1, n_clusters = gridDim.x >> 1;
    const int* kb_start = reinterpret_cast<const int*>(p.starts);
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
            kb0 = kb_start[e];
            KB = kb_start[e + 1] - kb0;
        } else {
            e = 0; kb0 = 0; KB = KB_dense;
            ti = pair_tile(p, t);
        }
    };

    if (warp == 8) {
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
    } else if (warp >= 9) {
        // ------------------ MMA issuers (leader only; whole warps, as in the one-SM kernel) ------------------
        if (rank == 0) {
            constexpr uint32_t idesc = make_idesc_pair(B_MN);
            const uint32_t tfull_own = mapa(tfull0, 0), tfull_peer = mapa(tfull0, 1);
            const uint32_t empty_own = mapa(empty0, 0), empty_peer = mapa(empty0, 1);
            const uint32_t mine = (uint32_t)(warp - 9);
            uint32_t it = 0, last = 0xffffffffu;
            bool alive = true;
            for (int t = cluster_id; t < n_total && alive; t += n_clusters) {
                int KB = KB_dense;
                if constexpr (GK) {
                    PairTile ti_; int e_, kb0_, end_;
                    locate(t, ti_, e_, kb0_, KB, end_);
                }
                for (int kb = 0; kb < KB; ++kb, ++it) {
                    if ((it & 1u) != mine) continue;
                    last = it;
                    const int s = it % PSTAGES;
                    const uint32_t ph = (it / PSTAGES) & 1;
                    const uint32_t b = it & 1, bph = (it >> 1) & 1;
                    if (!mbar_wait_warp(full0 + 8 * s, ph, abort_flag, (2 << 8) | 1)) { alive = false; break; }
                    if (!mbar_wait_warp(tempty0 + 8 * b, bph ^ 1, abort_flag, (2 << 8) | 2)) { alive = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem_a + s * PA_BYTES);
                    const uint32_t b_addr = smem_u32(smem_b + s * PB_BYTES);
                    const uint32_t d = tmem_base + b * PN;
#pragma unroll
                    for (int k = 0; k < BK / 32; ++k) {
                        const uint64_t ad = make_smem_desc(a_addr + k * 32, 16, 1024);
                        const uint64_t bd = B_MN ? make_smem_desc(b_addr + k * 32 * 128, 16, 1024)
                                                 : make_smem_desc(b_addr + k * 32, 16, 1024);
                        tc_mma_f8_pair(d, ad, bd, idesc, k > 0 ? 1u : 0u);
                    }
                    tc_commit_pair(tfull_own + 8 * b, tfull_peer + 8 * b);
                    tc_commit_pair(empty_own + 8 * s, empty_peer + 8 * s);
                }
            }
            if (alive && last != 0xffffffffu) mbar_wait(tfull0 + 8 * (last & 1), (last >> 1) & 1, abort_flag, (2 << 8) | 3);
        }
    } else {
        // ------------------------------ promotion / epilogue (both CTAs) ------------------------------
        const int q = warp & 3, h = warp >> 2;
        const uint32_t tempty_leader = mapa(tempty0, 0);
        uint32_t it = 0;
        bool alive = true;
        const bool vec_ok = (OUT == CINN_F32 || OUT == CINN_F32_BF16) ? (p.ldc % 4 == 0) : (p.ldc % 8 == 0);
        for (int t = cluster_id; t < n_total && alive; t += n_clusters) {
            PairTile ti; int e, kb0, KB, m_end;
            locate(t, ti, e, kb0, KB, m_end);
            const int row = ti.m0 + 128 * (int)rank + q * 32 + lane;
            const bool rvalid = row < m_end;
            const int col0 = ti.n0 + h * 128;
            const bool cvalid = col0 < p.N;
            const float* sa_ptr = p.sA + (int64_t)(rvalid ? row : (GR ? ti.m0 : 0)) * p.sa_stride_m + (int64_t)kb0 * p.sa_stride_k;
            const float* sb_ptr = p.sB + (int64_t)(cvalid ? col0 / 128 : 0) * p.sb_stride_n + (int64_t)kb0 * p.sb_stride_k
                                  + (GR ? (int64_t)e * p.sb_stride_e : 0);
            const int out_row0 = GR ? 0 : e * p.M;                      // GK: the expert's slice of the (E * M, N) output
            float acc[128];
#pragma unroll
            for (int i = 0; i < 128; ++i) acc[i] = 0.0f;
            float sa0 = ld_scale(sa_ptr), sb0 = ld_scale(sb_ptr);
            float sa1 = 0.f, sb1 = 0.f, sa2 = 0.f, sb2 = 0.f;
            if (KB > 1) { sa1 = ld_scale(sa_ptr + p.sa_stride_k); sb1 = ld_scale(sb_ptr + p.sb_stride_k); }
            if (KB > 2) { sa2 = ld_scale(sa_ptr + 2 * p.sa_stride_k); sb2 = ld_scale(sb_ptr + 2 * p.sb_stride_k); }
            for (int kb = 0; kb < KB; ++kb, ++it) {
                const float s = sa0 * sb0;
                sa0 = sa1; sb0 = sb1; sa1 = sa2; sb1 = sb2;
                if (kb + 3 < KB) {
                    sa2 = ld_scale(sa_ptr + (int64_t)(kb + 3) * p.sa_stride_k);
                    sb2 = ld_scale(sb_ptr + (int64_t)(kb + 3) * p.sb_stride_k);
                }
                const uint32_t b = it & 1, bph = (it >> 1) & 1;
                if (!mbar_wait_warp(tfull0 + 8 * b, bph, abort_flag, (3 << 8) | 1)) { alive = false; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + b * PN + h * 128;
                // packed fp32x2 FMAs: half the issue slots of 128 scalar ones, the same IEEE result in every lane
                uint64_t s2;
                asm("mov.b64 %0, {%1, %1};" : "=l"(s2) : "f"(s));
#pragma unroll
                for (int c = 0; c < 8; ++c) {
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
            if (alive && p.tma_out && (!GR || row - lane + 32 <= m_end)) {
                // The tile leaves through TMA stores.  Every promotion warp owns 8 KiB of the staging area, two boxes of 32 rows
                // x 128 bytes (128-byte swizzle): its lanes drop their rows in 16-byte chunks and one lane hands the boxes to
                // the TMA unit.  A 2-byte output fits the warp's 128 columns in one round; a 4-byte output takes two rounds of
                // 64 columns.  Nobody waits for the unit until the boxes are needed again, and no warp for another: with boxes
                // of 128 rows, four warps met at two barriers for each (16384 x 7168 -> 2048: 211 us, where this takes 195;
                // 32768 x 512 -> 1024: 29.8 and 27.4).
                using T = typename OutT<OUT>::type;
                constexpr int EPR = 128 / (int)sizeof(T);          // elements per 128-byte box row
                constexpr int PER16 = 16 / (int)sizeof(T);
                constexpr int ROUNDS = 128 / (2 * EPR);
                const uint32_t slot = smem_u32(c_stage) + warp * 2 * PBOX_BYTES;
#pragma unroll
                for (int r = 0; r < ROUNDS; ++r) {
                    if (lane == 0) tma_store_wait_read();             // the previous boxes have left the slots
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const uint4 v = pack16<OUT>(&acc[r * 2 * EPR + (j >> 3) * EPR + (j & 7) * PER16]);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                                     ::"r"(slot + (j >> 3) * PBOX_BYTES + lane * 128 + (((j & 7) ^ (lane & 7)) << 4)),
                                       "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
                    }
                    fence_async_smem();
                    __syncwarp();
                    if (lane == 0) {
#pragma unroll
                        for (int sl = 0; sl < 2; ++sl) {
                            const int col = col0 + r * 2 * EPR + sl * EPR;
                            if (col < p.N) tma_store_2d(&tmC, slot + sl * PBOX_BYTES, col, out_row0 + row);
                        }
                        tma_store_commit();
                    }
                    __syncwarp();       // the lane rejoins its warp before the next warp-collective instruction
                }
            } else if (alive && vec_ok) {
                // rows of two owners, or an output that TMA cannot write: staged 16-byte stores
                if (p.tma_out) {
                    if (lane == 0) tma_store_wait_read();
                    __syncwarp();
                }
                if (cvalid) store_rows_staged<OUT, 128>(acc, c_stage + warp * 2 * PBOX_BYTES, p.C, p.ldc,
                                                        out_row0 + ti.m0 + 128 * (int)rank + q * 32, out_row0 + m_end, col0, p.N, lane);
            } else if (alive && rvalid && cvalid) {
                const int64_t base = (int64_t)(out_row0 + row) * p.ldc + col0;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int ncols = p.N - (col0 + j * 8);
                    if (ncols > 0) store8<OUT>(p.C, base + j * 8, &acc[j * 8], false, ncols);
                }
            }
        }
        if (lane == 0) tma_store_wait_all();                // this warp's boxes have reached global memory
    }

    // nobody leaves while the other CTA may still read this CTA's shared memory or signal its barriers
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace pair
