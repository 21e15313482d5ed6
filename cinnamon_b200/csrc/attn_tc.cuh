// Shared pieces of the tensor-core sparse attention (attn_tc.cu): operand panels, splits, tensor-memory moves.
//
// Queries pick K of the keys behind them, but K is a sizeable share of a sequence of a few thousand, and the gather
// kernels (sparse_attn.cu) move every picked row through the L1 once per query: 26 GB of it at 32 x 8 x 1024 queries x
// 128 keys against 0.7 GB of tensors.  Here a tile of 128 queries meets tiles of 128 keys on the tensor cores and a
// map says which of the products are picked.  At C5's density of 1/4 (causal) that is four times the arithmetic on
// hardware that has thirty times the rate.
//
// fp32 and fp16 inputs are split into three bf16 parts each (8 + 8 + 8 bits: the fp32 mantissa, exactly) and a product
// is the six partial products down to 2^-16 x 2^-8 of the largest, accumulated in fp32: the arithmetic has fp32's
// precision.  bf16 inputs are one part; probabilities and score gradients, which are fp32, always are three.
#pragma once
#include "tcgen05.cuh"

namespace cinn {
namespace atc {

constexpr int T = 128;                     // queries per tile, keys per tile
constexpr int PANEL = T * 128;             // bytes of 128 rows x 64 bf16 columns, 128-byte swizzle
constexpr int PARTS = 3;                   // bf16 parts of an fp32 value
constexpr int MAX_SLOTS = 512;             // K: a warp permutes a row of probabilities in registers
constexpr int MAX_COUNT = 255;             // times one query may pick one key

// What the queries picked, per (batch, query): one bit per key; the rank of every slot's key among the query's picked
// keys in ascending order (0xffff for an index that takes no part); and how often each picked key was picked, by rank.
struct Picks {
    const uint32_t* bits;                  // (B, L, Lp / 32)
    const uint16_t* rank;                  // (B, L, K)
    const uint8_t* count;                  // (B, L, K)
    const uint16_t* before;                // (B, L, Lp / 32): picked keys before each word
    const int* repeats;                    // (B, tiles): whether a query of the tile picked a key more than once
};

// D[tmem] (+)= A[tmem] * B[smem desc]
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// 32 lanes x 32 columns, without waiting
__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, "
        "%19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
          "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr) : "memory");
}
__device__ __forceinline__ void st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint32_t bar, uint32_t dst, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}

// a box of shared memory to global memory, written or added (fp32, rounded to nearest, in L2)
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_add_3d(const CUtensorMap* map, uint32_t src, int x, int y, int z) {
    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(y), "r"(z) : "memory");
}
// two fp32 values as three packed bf16 pairs whose sum they are
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    auto pack = [](float x, float y) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(x, y);
        return *reinterpret_cast<const uint32_t*>(&t);
    };
    hi = pack(a, b);
    a -= __uint_as_float(hi << 16); b -= __uint_as_float(hi & 0xffff0000u);
    mid = pack(a, b);
    a -= __uint_as_float(mid << 16); b -= __uint_as_float(mid & 0xffff0000u);
    lo = pack(a, b);
}

// e^x; a result below 2^-126 is 0
__device__ __forceinline__ float exp_fast(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950408889634f));
    return r;
}

// if (take) *p = x, as a predicated instruction: as a branch it costs a warp some sixty cycles
__device__ __forceinline__ void store_if(float* p, float x, uint32_t take) {
    asm volatile(
        "{\n\t.reg .pred t;\n\t"
        "setp.ne.u32 t, %2, 0;\n\t"
        "@t st.global.f32 [%0], %1;\n\t}"
        ::"l"(p), "f"(x), "r"(take) : "memory");
}

// *p = (x, y) if take is not zero, as one predicated instruction
__device__ __forceinline__ void store2_if(float2* p, float x, float y, uint32_t take) {
    asm volatile(
        "{\n\t.reg .pred t;\n\t"
        "setp.ne.u32 t, %3, 0;\n\t"
        "@t st.global.v2.f32 [%0], {%1, %2};\n\t}"
        ::"l"(p), "f"(x), "f"(y), "r"(take) : "memory");
}
__device__ __forceinline__ void st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr) : "memory");
}
// Writes 32 consecutive reduction positions (keys or queries) of this lane's row as an A operand in tensor memory: the
// leading parts in 16 columns at `lead`, the second and third in 32 columns at `rest`.
__device__ __forceinline__ void store_parts32(uint32_t rest, uint32_t lead, const float (&v)[32]) {
    uint32_t hi[16], mid[16], lo[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) split2(v[2 * i], v[2 * i + 1], hi[i], mid[i], lo[i]);
    st16(lead, hi);
    st16(rest, mid);
    st16(rest + 16, lo);
}
// A panel used K-major (its 64 columns are the reduction axis; a step of four takes 16 of them) and MN-major (its 128 rows
// are; a step of eight takes 16 of them): the descriptor of the first step, to which the steps are added.  One thread
// issues all MMAs, so what it computes between two of them is time the tensor core waits.
constexpr uint64_t K_STEP = 32 >> 4, MN_STEP = 2048 >> 4;
__device__ __forceinline__ uint64_t panel_desc(uint32_t panel) { return make_smem_desc(panel, 16, 1024); }

// D (+)= A B over the 64 columns of two K-major panels; the first step overwrites D when `fresh`
__device__ __forceinline__ void mma_panels(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool fresh) {
    tc_mma_f16(d, a, b, idesc, fresh ? 0u : 1u);
#pragma unroll
    for (int s = 1; s < 4; ++s) tc_mma_f16(d, a + s * K_STEP, b + s * K_STEP, idesc, 1u);
}

// the same for one half (0 or 1) of the 32 positions
__device__ __forceinline__ void store_parts16(uint32_t rest, uint32_t lead, int half, const float (&v)[16]) {
    uint32_t hi[8], mid[8], lo[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) split2(v[2 * i], v[2 * i + 1], hi[i], mid[i], lo[i]);
    st8(lead + half * 8, hi);
    st8(rest + half * 8, mid);
    st8(rest + 16 + half * 8, lo);
}

// D (+)= part X of a tensor-memory operand of 16 STEPS positions (store_parts32) times an MN-major panel
template <int X, int STEPS = 8>
__device__ __forceinline__ void mma_part_at(uint32_t d, uint32_t rest, uint32_t lead, uint64_t b, uint32_t idesc, bool fresh) {
    auto column = [&](int s) { return X == 0 ? lead + s * 8 : rest + (s >> 1) * 32 + (X - 1) * 16 + (s & 1) * 8; };
    mma_ts(d, column(0), b, idesc, fresh ? 0u : 1u);
#pragma unroll
    for (int s = 1; s < STEPS; ++s) mma_ts(d, column(s), b + s * MN_STEP, idesc, 1u);
}

}  // namespace atc
}  // namespace cinn
