// qm_gemm_pair.cu — matmul over Q4_K weights by CTA pairs: C[m][n] = sum_k A[m][k] * W[n][k], A bf16
// activations, W dequantized on the fly straight into tensor memory, fp32 out.
//
// Two CTAs of a cluster (one SM each) compute a 256 (weight rows) x N (tokens, <= 256) tile of C^T with
// tcgen05.mma.cta_group::2: CTA r holds the 128 weight rows 128r.. as the A operand in its tensor memory and
// HALF of the tokens as the B operand in its shared memory. What this split is for: shared memory moves 128
// bytes per cycle for copies and MMA operands together, and with A in shared memory and all of B per SM a
// 128 x 512 tile needs 1408 cycles of it per 64 columns against 1024 cycles of MMA. Here A never touches shared
// memory (tcgen05.st writes the bf16 row of a thread into the thread's own lane) and B costs half.
//
//   * warp 0 copies the CTA's half of the tokens' 64-column chunk with 2-D TMA tile loads (128-byte swizzle, no
//     multicast) into a ring of `stages` stages; both halves complete on the leader's barrier;
//   * warp 2 copies the CTA's weight items (8 items of 16 rows x 256 columns, 2304 contiguous bytes each) into a
//     ring of `raw_ring` units with bulk copies, so that HBM latency is hidden by the ring and not by registers;
//   * warps 8..23 dequantize: group g (four warps, one thread per weight row) takes quant group g (64 columns)
//     of every unit, forms the bf16 columns (byte 0x43 beside a code = bf16 128+q, minus 128, d*sc*q - dmin*m as
//     one bf16x2 FMA per pair) and stores them into tensor memory;
//   * one thread of the leader's warp 1 issues four MMAs (K = 16 each) per chunk for both CTAs; its commit frees
//     the stage in both;
//   * warps 4..7 read finished accumulators and store C. With two accumulators (bn <= 128) that overlaps the
//     next tile: the launch is persistent, pair p takes the tiles p, p + pairs, ...
// Few tokens: `splitk` pairs (or single CTAs) of a cluster of at most four CTAs share a tile's K range; the partial
// tiles meet in shared memory and every CTA adds one band of tokens from the others' in order of the shares: no
// scratch, no atomics, the same bits every run.
// Measured against the kernel before it (A and B in shared memory, one CTA per tile), us: 4096 x 4096 at 64 / 512 /
// 2048 tokens 16.4 -> 13.3, 35 -> 24, 79 -> 69; 6144 x 4096 at 391 47 -> 25; 14336 x 4096 at 1024 144 -> 109. At up to
// 128 tokens per tile the dequantizing warps' instruction issue bounds it (with one of eight MMAs issued the time is
// the same), at 256 the MMAs.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include "qm_kernel_args.h"
#include "qm_pipe.cuh"

using namespace qm;

namespace {

constexpr int kMaxStages = 8, kMaxRaw = 8;
constexpr int kRawBytes = 8 * QM_Q4K_ITEM_BYTES;   // one unit (256 columns) of a CTA's 128 rows

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}
__device__ __forceinline__ uint32_t bsub2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t bfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t bf2(float v) {   // (v, v) as bf16x2
    __nv_bfloat162 h = __float2bfloat162_rn(v);
    return *reinterpret_cast<uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_cta(uint32_t addr, uint32_t rank) {   // the same offset in CTA `rank` of the cluster
    uint32_t d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(rank));
    return d;
}
__device__ __forceinline__ void arrive_cluster(uint32_t mapped) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(mapped) : "memory");
}
__device__ __forceinline__ void arrive_local(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait of a whole warp. The lanes leave the polling loop one by one as far as the language goes, and the
// .sync.aligned instructions that follow need all of them.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
    const bool ok = mbar_wait_bounded(bar, parity);
    return __all_sync(0xFFFFFFFFu, ok);
}
// Tile load into this CTA's shared memory that completes on a barrier of the pair's leader.
template <int CG>
__device__ __forceinline__ void tma_load(uint32_t dst, const void *tmap, int x, int y, uint32_t leader_bar) {
    if (CG == 2)
        asm volatile(
            "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
            "l"(tmap), "r"(x), "r"(y), "r"(leader_bar)
            : "memory");
    else
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
            "l"(tmap), "r"(x), "r"(y), "r"(leader_bar)
            : "memory");
}
// K-major, 128-byte swizzle, 8-row groups 1024 bytes apart (sm_100 descriptor version 1)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// One lane of a converged warp. (The MMA loop is run by the whole warp and only the issue is elected: with the loop
// inside `if (lane == 0)` the operands do not stay in uniform registers, and a chunk's four MMAs took 350 cycles to
// issue whatever their N.)
__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xFFFFFFFF;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(pred));
    return pred != 0;
}
template <int CG>
__device__ __forceinline__ void umma(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    if (CG == 2)
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
            "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(acc)
            : "memory");
    else
        asm volatile(
            "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
            "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(acc)
            : "memory");
}
// Arrival at the barrier of both CTAs of the pair (of this CTA) when the MMAs issued so far are complete.
template <int CG>
__device__ __forceinline__ void commit(uint32_t bar, uint16_t cta_mask) {
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                     "h"(cta_mask)
                     : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(addr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t mapped) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(mapped));
    return v;
}

// The tiles of one pair (or, with split K, one cluster), in the order every role walks them.
struct Tiles {
    int it, e, base;        // next item; grouped: expert and its first item
    int rt, m0, mv, row_off;   // row tile, first token, tokens, first activation row of the expert
    __device__ __forceinline__ Tiles(int first) : it(first), e(0), base(0) {}
    __device__ __forceinline__ bool next(const QmPairArgs &a, const int *offsets, int stride) {
        if (!a.grouped) {
            if (it >= a.items) return false;
            rt = it % a.row_tiles;
            m0 = it / a.row_tiles * a.bn;
            mv = min(a.bn, a.m - m0);
            row_off = 0;
        } else {
            int nt;
            while (true) {
                if (e >= a.experts) return false;
                row_off = offsets[e];
                mv = offsets[e + 1] - row_off;
                nt = (mv + a.bn - 1) / a.bn;
                if (it < base + nt * a.row_tiles) break;
                base += nt * a.row_tiles;
                e++;
            }
            rt = (it - base) / nt;   // an expert's token tiles of one row tile follow one another
            m0 = (it - base) % nt * a.bn;
            mv = min(a.bn, mv - m0);
        }
        it += stride;
        return true;
    }
};

}  // namespace

namespace {

template <int CG>
__device__ __forceinline__ void pair_body(const QmPairArgs &a) {
    extern __shared__ uint8_t smem_raw[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t crank = cluster_rank(), leader = crank & ~(uint32_t)(CG - 1);
    const int rank = crank & (CG - 1), share = crank / CG;   // CTA of the pair; the pair's share of K
    const int S = a.stages, R = a.raw_ring;
    const uint32_t box_bytes = (uint32_t)a.bn * (128 / CG), stage_bytes = 2 * box_bytes;   // the CTA's tokens x 64 columns of bf16, twice
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *raw = smem + S * stage_bytes;
    uint64_t *bars = reinterpret_cast<uint64_t *>(raw + R * kRawBytes);
    const uint32_t full = smem_u32(bars), empty = full + 8 * kMaxStages, raw_full = empty + 8 * kMaxStages,
                   raw_empty = raw_full + 8 * kMaxRaw, acc_full = raw_empty + 8 * kMaxRaw, acc_empty = acc_full + 16;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * kMaxStages + 2 * kMaxRaw + 4);
    volatile uint32_t *failed = tmem_slot + 1;
    int *offsets = reinterpret_cast<int *>(tmem_slot + 2);
    const uint32_t smem_base = smem_u32(smem), raw_base = smem_u32(raw);

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(full + 8 * s, 8 * CG + 1);   // eight dequantizing warps in each CTA, the leader's byte count
            mbar_init(empty + 8 * s, 1);
        }
        for (int s = 0; s < R; s++) {
            mbar_init(raw_full + 8 * s, 1);
            mbar_init(raw_empty + 8 * s, 16);
        }
        for (int s = 0; s < 2; s++) {
            mbar_init(acc_full + 8 * s, 1);
            mbar_init(acc_empty + 8 * s, 4 * CG);
        }
        *failed = 0;
        fence_barrier_init();
    }
    if (a.grouped)
        for (int i = tid; i <= a.experts; i += blockDim.x) offsets[i] = a.offsets[i];
    __syncwarp();
    if (warp == 3) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync();   // the other CTA's barriers exist before anything arrives there
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t a_base = tmem_base + (uint32_t)(a.nacc * a.bn);   // A stages behind the accumulators, 64 columns each

    const int first = blockIdx.x / (CG * a.splitk), stride = gridDim.x / (CG * a.splitk);
    const int u_lo = a.units * share / a.splitk, nu = a.units * (share + 1) / a.splitk - u_lo;   // this pair's units of K
    Tiles t(first);
    auto fail = [&]() {
        atomicOr(a.status, QM_STATUS_TIMEOUT);
        *failed = 1;
    };

    if (warp == 0) {
        // ---- activation chunks: this CTA's half of the tokens -------------------------------------------
        if (lane == 0) {
            int s = 0;
            uint32_t ph = 1;   // parity of the release before the stage's first use: passes at once
            bool ok = true;
            while (ok && t.next(a, offsets, stride)) {
                const int half = qm_pair_mma_n(t.mv, CG) / CG, box = a.box_rows, nrows = (half + box - 1) / box * box;
                const int y = t.row_off + t.m0 + rank * half;
                for (int kc = 0; kc < nu * 2; kc++) {
                    if (!mbar_wait_bounded(empty + 8 * s, ph)) { fail(); ok = false; break; }
                    if (rank == 0) mbar_expect_tx(full + 8 * s, (uint32_t)nrows * 256 * CG);   // both CTAs' halves
                    const uint32_t bar = map_cta(full + 8 * s, leader);
#pragma unroll
                    for (int j = 0; j < 2; j++)
                        for (int nb = 0; nb < nrows; nb += box)
                            tma_load<CG>(smem_base + s * stage_bytes + j * box_bytes + nb * 128, &a.tmap_act,
                                         ((u_lo * 2 + kc) * 2 + j) * 64, y + nb, bar);
                    if (++s == S) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 2) {
        // ---- weight items ----------------------------------------------------------------------------------
        int s = 0;
        uint32_t ph = 1;
        bool ok = true;
        while (ok && t.next(a, offsets, stride)) {
            // the CTA's eight 16-row tiles; with SwiGLU gate and up tiles take turns, so that a warp's 32 lanes
            // hold 16 gate rows and the 16 up rows that belong to them
            const int i = lane & 7;
            const int tile16 = a.swiglu ? (t.rt * CG + rank) * 4 + (i >> 1) + (i & 1) * (a.up_offset >> 4) : (t.rt * CG + rank) * 8 + i;
            const uint8_t *src = (a.grouped ? a.wq_list[t.e] : a.wq) + ((int64_t)min(tile16, a.tiles16 - 1) * a.units + u_lo) * QM_Q4K_ITEM_BYTES;
            for (int u = 0; u < nu; u++) {
                if (!warp_wait(raw_empty + 8 * s, ph)) { if (lane == 0) fail(); ok = false; break; }
                if (lane == 0) mbar_expect_tx(raw_full + 8 * s, kRawBytes);
                __syncwarp();
                if (lane < 8)
                    bulk_g2s(raw_base + s * kRawBytes + lane * QM_Q4K_ITEM_BYTES, src + (int64_t)u * QM_Q4K_ITEM_BYTES,
                             QM_Q4K_ITEM_BYTES, raw_full + 8 * s);
                if (++s == R) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issue, for both CTAs ----------------------------------------------------------------------
        if (rank == 0) {
            // kind::f16, fp32 accumulate, A and B bf16, both K-major, M = 128 per CTA
            const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(8 * CG) << 24);
            const uint16_t mask = (uint16_t)(3u << leader);
            const uint64_t bdesc0 = smem_desc(smem_base);
            const uint32_t a_tmem0 = __shfl_sync(0xFFFFFFFFu, a_base, 0), d_tmem0 = __shfl_sync(0xFFFFFFFFu, tmem_base, 0);
            int s = 0, acc = 0;
            uint32_t ph = 0, acc_ph = 1;
            bool ok = true;
            while (ok && t.next(a, offsets, stride)) {
                // N: bits 17..22 hold N / 8
                const uint32_t idesc = __shfl_sync(0xFFFFFFFFu, idesc0 | ((uint32_t)qm_pair_mma_n(t.mv, CG) << 14), 0);
                const uint32_t d_tmem = d_tmem0 + (uint32_t)(acc * a.bn);
                if (!warp_wait(acc_empty + 8 * acc, acc_ph)) { if (lane == 0) fail(); break; }
                for (int kc = 0; kc < nu * 2; kc++) {
                    if (!warp_wait(full + 8 * s, ph)) { if (lane == 0) fail(); ok = false; break; }
                    __syncwarp();
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bdesc = bdesc0 + (uint32_t)s * (stage_bytes >> 4);
                    const uint32_t a_tmem = a_tmem0 + (uint32_t)(s * 64);
                    if (elect_one()) {
#pragma unroll
                        for (int k16 = 0; k16 < 8; k16++)   // 16 bf16: 8 tensor memory columns of A, 2 descriptor units of B
                            umma<CG>(d_tmem, a_tmem + 8 * k16, bdesc + (k16 >> 2) * (box_bytes >> 4) + 2 * (k16 & 3), idesc, (kc | k16) != 0);
                        commit<CG>(empty + 8 * s, mask);   // frees the stage in both CTAs when these MMAs have read it
                    }
                    __syncwarp();
                    if (++s == S) { s = 0; ph ^= 1; }
                }
                if (elect_one()) commit<CG>(acc_full + 8 * acc, mask);
                __syncwarp();
                if (++acc == a.nacc) { acc = 0; acc_ph ^= 1; }
            }
        }
    } else if (warp >= 8) {
        // ---- dequantize into tensor memory -----------------------------------------------------------------
        // Groups 0, 1 fill the unit's first stage, 2, 3 its second; a stage's release can be told from the one before
        // it only while a group is at most one release behind, which holds for S >= 2.
        const int g = (warp - 8) >> 2, q = warp & 3;
        const uint32_t item = (uint32_t)((2 * q + (lane >> 4)) * QM_Q4K_ITEM_BYTES), rr = lane & 15;
        const uint32_t lane_base = a_base + ((uint32_t)(q * 32) << 16);
        int s = g >> 1, rs = 0;
        uint32_t ph = 1, rph = 0;
        bool ok = true;
        while (ok && t.next(a, offsets, stride)) {
            for (int u = 0; u < nu; u++) {
                if (!warp_wait(raw_full + 8 * rs, rph)) { if (lane == 0) fail(); ok = false; break; }
                const uint8_t *src = raw + rs * kRawBytes + item;
                const uint4 h4 = *reinterpret_cast<const uint4 *>(src + 16 * rr);
                const uint4 qa = *reinterpret_cast<const uint4 *>(src + 256 + 512 * g + 32 * rr);
                const uint4 qb = *reinterpret_cast<const uint4 *>(src + 256 + 512 * g + 32 * rr + 16);
                __syncwarp();
                if (lane == 0) arrive_local(raw_empty + 8 * rs);   // the copies above are in registers
                if (++rs == R) { rs = 0; rph ^= 1; }
                // scales and minima of the unit half's four sub-blocks, one per byte; this group's are 2 * (g & 1) and the next
                const uint32_t sc = (g & 2) ? (h4.w & 0x0F0F0F0Fu) | ((h4.y >> 2) & 0x30303030u) : h4.y & 0x3F3F3F3Fu;
                const uint32_t mn = (g & 2) ? ((h4.w >> 4) & 0x0F0F0F0Fu) | ((h4.z >> 2) & 0x30303030u) : h4.z & 0x3F3F3F3Fu;
                const float2 dd = __half22float2(*reinterpret_cast<const __half2 *>(&h4.x));   // d, dmin
                const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
                if (!warp_wait(empty + 8 * s, ph)) { if (lane == 0) fail(); ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int hs = 0; hs < 2; hs++) {
                    // (a byte as a float: 2^23 + byte, minus 2^23)
                    const uint32_t sel = 0x7440u | (uint32_t)(2 * (g & 1) + hs);
                    const float scf = __uint_as_float(prmt(sc, 0x4B000000u, sel)) - 8388608.f;
                    const float mnf = __uint_as_float(prmt(mn, 0x4B000000u, sel)) - 8388608.f;
                    const uint32_t av = bf2(dd.x * scf), bv = bf2(-dd.y * mnf);
                    uint32_t o[16];
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        // four codes of this nibble half, then each next to the byte 0x43: bf16 128+q
                        const uint32_t nib = hs ? (w[i] >> 4) & 0x0F0F0F0Fu : w[i] & 0x0F0F0F0Fu;
                        o[2 * i] = bfma2(bsub2(prmt(nib, 0x43434343u, 0x4140u), 0x43004300u), av, bv);
                        o[2 * i + 1] = bfma2(bsub2(prmt(nib, 0x43434343u, 0x4342u), 0x43004300u), av, bv);
                    }
                    tmem_st16(lane_base + (uint32_t)(s * 64 + (g & 1) * 32 + hs * 16), o);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) arrive_cluster(map_cta(full + 8 * s, leader));
                s += 2;
                if (s >= S) { s -= S; ph ^= 1; }
            }
        }
    } else if (warp >= 4) {
        // ---- epilogue: accumulator lane r holds C[m0..m0+mv)[row r] ----------------------------------------
        const int q = warp & 3;
        const uint32_t quarter = tmem_base + ((uint32_t)(q * 32) << 16);
        float *part = reinterpret_cast<float *>(smem);   // split K: [token][128 rows] over the drained rings
        int acc = 0;
        uint32_t ph = 0;
        while (t.next(a, offsets, stride)) {
            if (!warp_wait(acc_full + 8 * acc, ph)) { if (lane == 0) fail(); break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t src = quarter + (uint32_t)(acc * a.bn);
            if (a.swiglu) {
                // lanes 0..15 hold gate rows, lanes 16..31 their up rows: of two neighbouring tokens the lower half
                // takes the first, the upper half the second
                const int n = ((t.rt * CG + rank) * 4 + q) * 16 + (lane & 15), odd = lane >> 4;
                uint16_t *hp = a.h + (int64_t)(t.row_off + t.m0 + odd) * a.ldh + n;
                for (int c0 = 0; c0 < t.mv; c0 += 16) {
                    uint32_t v[16];
                    tmem_ld16(src + (uint32_t)c0, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 16; j += 2) {
                        const uint32_t got = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[j] : v[j + 1], 16);
                        const float gv = __uint_as_float(odd ? got : v[j]), uv = __uint_as_float(odd ? v[j + 1] : got);
                        // (fast division: the quotient is rounded to bf16 next)
                        const __nv_bfloat16 hv = __float2bfloat16_rn(__fdividef(gv, 1.f + __expf(-gv)) * uv);
                        if (n < a.n && c0 + j + odd < t.mv) hp[(int64_t)(c0 + j) * a.ldh] = *reinterpret_cast<const uint16_t *>(&hv);
                    }
                }
            } else {
                const int n = (t.rt * CG + rank) * 128 + q * 32 + lane;
                float *cp = a.c + (int64_t)(t.row_off + t.m0) * a.ldc + n;
                for (int c0 = 0; c0 < t.mv; c0 += 32) {   // two blocks per wait where there are two
                    uint32_t v[16], w[16];
                    const bool two = c0 + 16 < t.mv;
                    tmem_ld16(src + (uint32_t)c0, v);
                    if (two) tmem_ld16(src + (uint32_t)(c0 + 16), w);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (a.splitk > 1) {
#pragma unroll
                        for (int j = 0; j < 16; j++) {
                            part[(c0 + j) * 128 + q * 32 + lane] = __uint_as_float(v[j]);
                            if (two) part[(c0 + 16 + j) * 128 + q * 32 + lane] = __uint_as_float(w[j]);
                        }
                    } else if (n < a.n) {
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (c0 + j < t.mv) cp[(int64_t)(c0 + j) * a.ldc] = __uint_as_float(v[j]);
                        if (two) {
#pragma unroll
                            for (int j = 0; j < 16; j++)
                                if (c0 + 16 + j < t.mv) cp[(int64_t)(c0 + 16 + j) * a.ldc] = __uint_as_float(w[j]);
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_cluster(map_cta(acc_empty + 8 * acc, leader));
            if (++acc == a.nacc) { acc = 0; ph ^= 1; }
        }
    }
    __syncwarp();
    __syncthreads();
    if (*failed) {   // let copies that are still in flight land before the memory they write is given up
        const long long t0 = clock64();
        while (clock64() - t0 < 4000000ll) {}
    }
    cluster_sync();   // every CTA is done with the others' barriers and operands (and the partial tiles are written)
    __syncwarp();
    if (warp == 3) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
    if (a.splitk > 1) {
        // one tile per cluster: this CTA adds a band of its row half's tokens, shares in order
        Tiles t1(first);
        if (t1.next(a, offsets, stride)) {
            const int n0 = (t1.rt * CG + rank) * 128;
            const int lo = t1.mv * share / a.splitk, hi = t1.mv * (share + 1) / a.splitk;
            const bool vec = (a.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(a.c) & 15) == 0;
            for (int i = lo * 32 + tid; i < hi * 32; i += blockDim.x) {   // four rows of one token
                const int n = n0 + 4 * (i & 31);
                float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int z = 0; z < a.splitk; z++) {
                    const float4 v = ld_cluster4(map_cta(smem_base + 16u * i, CG * z + rank));
                    sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
                }
                float *cp = a.c + (int64_t)(t1.row_off + t1.m0 + (i >> 5)) * a.ldc + n;
                if (vec && n + 3 < a.n) *reinterpret_cast<float4 *>(cp) = sum;
                else {
                    if (n < a.n) cp[0] = sum.x;
                    if (n + 1 < a.n) cp[1] = sum.y;
                    if (n + 2 < a.n) cp[2] = sum.z;
                    if (n + 3 < a.n) cp[3] = sum.w;
                }
            }
        }
        cluster_sync();   // no CTA leaves while another still reads its partial tile
    }
}

}  // namespace

extern "C" __global__ void __launch_bounds__(768, 1) qm_gemm_q4k_pair(const __grid_constant__ QmPairArgs a) { pair_body<2>(a); }
// One CTA per tile of 128 weight rows: few tokens, where more tiles and K shares matter more than the operand traffic.
extern "C" __global__ void __launch_bounds__(768, 1) qm_gemm_q4k_solo(const __grid_constant__ QmPairArgs a) { pair_body<1>(a); }
