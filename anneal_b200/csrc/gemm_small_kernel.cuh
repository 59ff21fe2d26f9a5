// One-CTA tcgen05 contraction kernel for outputs that leave most CTA pairs of the two-CTA kernel idle:
// a few rows against a large weight matrix (serving), a thousand-cubed training step, a head layer.  Compiled
// at run time (NVRTC, sm_100a) once per configuration, like gemm_pair_kernel.cuh, with which it shares the
// arithmetic: f16 operands, f32 accumulation in tensor memory, ONE rounding to f16, then optionally the
// elementwise kernel that the schedule runs next and the per-32-row partial column sums of what was stored.
//
// What bounds such a shape is not the tensor pipe but how few SMs share the loads, and the fixed cost of a
// launch.  So a cluster of CFG_SPLITS CTAs shares one 128 x CFG_NT tile: each CTA multiplies its own slice of K
// (TMA ring -> tcgen05.mma -> 128 x CFG_NT accumulator in tensor memory), leaves the f32 partial tile in its
// shared memory, and the CTAs then add the partials in rank order through distributed shared memory, each
// finishing its share of the tile: the same bits on every run, no scratch memory, no second launch.  The kernel is
// not persistent: about 100 KB of shared memory a CTA lets two sit on an SM, and one's loads run under the
// other's epilogue.
//
// Measured alone (B200, warm L2, the 6 to 7 us of the timing events included), against the route before: 32 x 4096 x 4096
// 16.4 us against 155 (generated, one block per output); 999 x 250 x 1000 12.3 against 31.8 and 1024-cubed 12.3 to 13.2
// against 17.3 (pair kernel).  A training step at 999 x 1000 with 250 classes, whose head gradients (rows off 16-byte
// boundaries) were generated kernels of 125 and 92 us, went from 326 to 122 us.
//
// f32 operands (CFG_TF32 = 1) take the same kernel in the 3 x TF32 form of the pair kernel: every operand arrives as two
// k-contiguous f32 arrays, hi and lo, a k-block is 32 deep and is staged as four parts, and three products are
// accumulated on them, without copies of the output in memory or a launch to add them up.
//
// Tensor memory cuts each partial sum instead of rounding it, an error that grows with the number of additions.  A
// slice of more than CFG_CHUNK k-blocks is therefore accumulated in chunks of that many, in two accumulators by turns: eight
// more warps than the two that load and multiply take each finished chunk to registers and add it to the ones before, in f32
// round-to-nearest, while the next one is multiplied.  Error against float64 (rms with normal values | mean with positive
// ones), slices of 1024 f32 terms in one go, in chunks of 256, on the pair kernel: 256 x 1024 x 4096 7.1e-6 | 1.1e-5, 1.7e-6 |
// 2.3e-6, 1.7e-6 | 2.3e-6 (37.9, 39.9, 37.9 us alone, with the operand splits and the events); 2048 x 1024 x 1024 7.1e-6 | 1.1e-5,
// 1.7e-6 | 2.3e-6, 3.5e-6 | 5.1e-6 (35.8, 37.9, 46.1 us).  Eight f16 slices of 8192 terms lost 4.7e-5 of a positive sum, in chunks
// of 1024 they lose 5.6e-6, beside the 1.4e-4 rms of the rounding to f16 (40 x 4096 x 16384 34.8 and 38.9 us).
//
// With fewer than 128 rows only CFG_PROWS of them are loaded and staged; the MMA still reads 128 rows of
// shared memory and the accumulator rows past the matrix are never stored (rows do not mix).
//
// Every wait on an mbarrier is bounded; a wait that runs out records a code in a host-visible status word and
// the CTA drains and frees its tensor memory.
//
// The host prepends the configuration:
//   CFG_A_MN, CFG_B_MN   1 when the operand's m / n index is the contiguous one (else k is)
//   CFG_NT               tile width in columns: 32, 64 or 128 (64 or 128 when CFG_B_MN)
//   CFG_PROWS            rows of A staged per k-block: 16, 32, 64 or 128 (128 when CFG_A_MN)
//   CFG_STAGES           depth of the shared-memory ring of k-blocks
//   CFG_SPLITS           CTAs per tile: 1, 2, 4 or 8
//   CFG_CHUNK            k-blocks accumulated in tensor memory at a time; 0 when no slice is longer than a chunk
//   CFG_TF32             1: f32 operands as hi and lo parts, f32 output (k-contiguous only, no fused consumer, no column sums)
//   CFG_EPI              1 when a fused elementwise consumer has been prepended (gemm_pair_kernel.cuh says how)
//   CFG_NAME             namespace of this configuration
//   CFG_ALONE            1: the text ends in a kernel of its own; 0: it is there twice, and the host appends the kernel of both
//
// Two contractions that do not depend on each other, a layer's weight gradient and its input gradient, run as ONE launch of
// both configurations: one CTA of each sits on an SM, so that one's loads (94 bytes a ns for a ring of 100 KB, of the 145 an
// SM can take from L2) and finish run beside the other's, and one launch's fixed cost is saved.  Training step of 1024 rows,
// 4 x 1024 wide, 144.1 -> 130.4 us, of 999 rows, 2 x 1000 wide, 111.0 -> 97.2.
#ifndef ANL_SMALL_GEMM_COMMON
#define ANL_SMALL_GEMM_COMMON

struct SmallGemmArgs {
    void* d_raw;            // [M, N] f16 (f32): the contraction itself; null when nothing else reads it
    void* d_out;            // [M, N] f16: output of the fused consumer; null without one
    float* colsum;          // [ceil(M/32), N] f32 partial column sums of the last value stored; null when not wanted
    const void* ep[6];      // operands of the fused consumer, in its parameter order
    int M, N, K;
    int tiles_m;
    int b_settled;          // 1: B is not written by any launch that may still run when this one starts
    int* status;
};

#ifdef ANL_SMALL_GEMM_DEVICE_CODE

#include <cuda_fp16.h>

struct alignas(64) TensorMap { unsigned long long opaque[16]; };

constexpr unsigned WAIT_LIMIT = 1u << 20;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// Bounded wait: false when the phase did not complete within WAIT_LIMIT polls, or when another role of this
// CTA has already given up.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, const volatile int* failed) {
    for (unsigned i = 0; i < WAIT_LIMIT; i++) {
        if (failed && (i & 255u) == 255u && *failed) return false;
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}\n"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ unsigned cluster_ctarank() { unsigned r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ unsigned map_to_cta(unsigned saddr, unsigned rank) {
    unsigned r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank)); return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(unsigned addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same without an order on memory, where nothing that was written before is read after it and what was read has been
// used: it does not wait for the stores of the outputs (32 rows through 4 x 4096, five launches, 60.4 -> 59.3 us).
__device__ __forceinline__ void cluster_meet_all() {
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void tma_load_2d(unsigned dst, const TensorMap* map, int c0, int c1, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar) : "memory");
}
// Shared-memory matrix descriptor, 128-byte swizzle: bits [0,14) start address >> 4, [16,30) leading byte
// offset >> 4, [32,46) stride byte offset >> 4, [46,48) version 1, [61,64) layout type 2.
__device__ __forceinline__ unsigned long long make_desc(unsigned saddr, unsigned lbo_bytes, unsigned sbo_bytes) {
    return (unsigned long long)((saddr >> 4) & 0x3FFF) | ((unsigned long long)((lbo_bytes >> 4) & 0x3FFF) << 16) |
           ((unsigned long long)((sbo_bytes >> 4) & 0x3FFF) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr) : "memory");
}

#endif  // ANL_SMALL_GEMM_DEVICE_CODE
#endif  // ANL_SMALL_GEMM_COMMON

#ifdef ANL_SMALL_GEMM_DEVICE_CODE
namespace CFG_NAME {

// a k-block is one 128-byte swizzle row of k: 64 f16 or 32 f32 elements; in the f32 form each operand is staged as hi, then lo
constexpr int BM = 128, BK = CFG_TF32 ? 32 : 64, PARTS = CFG_TF32 ? 2 : 1, NT = CFG_NT, NSTAGE = CFG_STAGES, SPLITS = CFG_SPLITS, CHUNK = CFG_CHUNK, THREADS = CHUNK ? 320 : 256;
constexpr int P_PART = CFG_PROWS * 128, Q_PART = NT * 128, P_BYTES = PARTS * P_PART, STAGE_BYTES = P_BYTES + PARTS * Q_PART;
static_assert(!(CFG_TF32 && (CFG_A_MN || CFG_B_MN || CFG_EPI)), "the f32 form takes k-contiguous operands and no consumer");
constexpr int LDT = NT + 4;              // floats per row of the staged f32 tile: rows 16 bytes apart in the banks
constexpr int TMEM_COLS = CHUNK ? 2 * NT : NT;
// Pieces of the finish (8 rows x 32 columns) that a warp takes together.  A piece alone is a chain of latencies (its operands
// from L2, the arithmetic of an activation), and a warp has few of them to hide it behind: four at a time where registers hold
// them and the partials are at hand, their operands asked for while the products are still running.  Training step of 1024 rows,
// 4 x 1024 wide, 146.6 -> 143.3 us, of 999 rows 111.5 -> 109.9.  Where the partials come from other CTAs or chunks have taken
// the registers, pieces by twos and fours were slower than one at a time (500 rows, 3 x 2048 wide, 67.8 us against 63.9).
#if CFG_EPI
constexpr int BATCH = SPLITS > 1 || CHUNK ? 1 : EPI_NRAW > 3 ? 2 : 4;
#else
constexpr int BATCH = SPLITS > 1 || CHUNK ? 1 : 4;
#endif
static_assert(!CFG_A_MN || CFG_PROWS == 128, "an m-contiguous operand is staged whole");
static_assert(!CFG_B_MN || NT % 64 == 0, "an n-contiguous operand is staged in boxes of 64");

__device__ __forceinline__ void umma_f16(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
#if CFG_TF32
        " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n"
#else
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
#endif
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}

// `block`: number of this CTA among the contraction's own
__device__ __forceinline__ void run(const TensorMap& map_a, const TensorMap& map_b,
#if CFG_TF32
                                    const TensorMap& map_a_lo, const TensorMap& map_b_lo,
#endif
                                    const SmallGemmArgs& g, const unsigned block) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long full_bar[NSTAGE], empty_bar[NSTAGE];
#if CFG_CHUNK
    __shared__ __align__(8) unsigned long long acc_full[2], acc_empty[2];
#else
    __shared__ __align__(8) unsigned long long acc_full;
#endif
    __shared__ unsigned tmem_base_slot;
    __shared__ volatile int failed;

    const unsigned smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;   // swizzle atoms need 1 KiB alignment
    float* const tile = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));   // the ring's memory, once the ring is done
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = SPLITS > 1 ? cluster_ctarank() : 0u;
    const int t = (int)(block / SPLITS);
    const int m0 = (t % g.tiles_m) * BM, n0 = (t / g.tiles_m) * NT;
    const int kblocks = (g.K + BK - 1) / BK;
    // this CTA's slice: at least one k-block, as the host gives no tile more CTAs than it has k-blocks
    const int kb0 = (int)((long long)kblocks * rank / SPLITS), nkb = (int)((long long)kblocks * (rank + 1) / SPLITS) - kb0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NSTAGE; s++) { mbar_init(smem_u32(&full_bar[s]), 1); mbar_init(smem_u32(&empty_bar[s]), 1); }
#if CFG_CHUNK
        for (int a = 0; a < 2; a++) { mbar_init(smem_u32(&acc_full[a]), 1); mbar_init(smem_u32(&acc_empty[a]), 8); }
#else
        mbar_init(smem_u32(&acc_full), 1);
#endif
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const unsigned tmem_base = tmem_base_slot;
    // Set up while the launch in front still runs; its results are not touched before it has finished.  A weight matrix
    // that nothing writes meanwhile is asked for at once: the ring is full when the activations arrive.
    if (warp != 0) asm volatile("griddepcontrol.wait;" ::: "memory");

    if (warp == 0) {
        // ── producer ──
        if (lane == 0) {
            unsigned stage = 0, phase = 0;
            bool ok = true;
            int issued = 0;
            auto load_b = [&](unsigned sq, int k0, unsigned fb) {
                if (CFG_B_MN) { for (int j = 0; j < NT / 64; j++) tma_load_2d(sq + j * (BK * 128), &map_b, n0 + 64 * j, k0, fb); }
                else tma_load_2d(sq, &map_b, k0, n0, fb);
#if CFG_TF32
                tma_load_2d(sq + Q_PART, &map_b_lo, k0, n0, fb);
#endif
            };
            const int early = !g.b_settled ? 0 : nkb < NSTAGE ? nkb : NSTAGE;
            for (int it = 0; it < early; it++) {
                mbar_expect_tx(smem_u32(&full_bar[it]), STAGE_BYTES);
                load_b(smem_base + it * STAGE_BYTES + P_BYTES, (kb0 + it) * BK, smem_u32(&full_bar[it]));
            }
            asm volatile("griddepcontrol.wait;" ::: "memory");
            for (int it = 0; it < nkb; it++) {
                if (!mbar_wait(smem_u32(&empty_bar[stage]), phase ^ 1, &failed)) { ok = false; *(volatile int*)g.status = 21; break; }
                const unsigned fb = smem_u32(&full_bar[stage]);
                const unsigned sp = smem_base + stage * STAGE_BYTES, sq = sp + P_BYTES;
                const int k0 = (kb0 + it) * BK;
                if (it >= early) mbar_expect_tx(fb, STAGE_BYTES);
                if (CFG_A_MN) { for (int j = 0; j < BM / 64; j++) tma_load_2d(sp + j * (BK * 128), &map_a, m0 + 64 * j, k0, fb); }
                else tma_load_2d(sp, &map_a, k0, m0, fb);
#if CFG_TF32
                tma_load_2d(sp + P_PART, &map_a_lo, k0, m0, fb);
#endif
                if (it >= early) load_b(sq, k0, fb);
                issued++;
                if (++stage == NSTAGE) { stage = 0; phase ^= 1; }
            }
            if (!ok) {
                failed = 1;
                // let copies already in flight land before the CTA goes away
                const int pending = issued < NSTAGE ? issued : NSTAGE;
                for (int i = 0; i < pending; i++) { stage = stage == 0 ? NSTAGE - 1 : stage - 1; mbar_wait(smem_u32(&full_bar[stage]), 0, nullptr); mbar_wait(smem_u32(&full_bar[stage]), 1, nullptr); }
            }
        }
    } else if (warp == 1) {
        // ── MMA issuer ──
        if (lane == 0) {
            // instruction descriptor: f32 accumulate, operand formats (0 f16, 2 tf32) at bits 7 and 10, majors, N >> 3 at bit 17, M >> 4 at bit 24
            const unsigned idesc = (1u << 4) | ((CFG_TF32 ? 2u : 0u) << 7) | ((CFG_TF32 ? 2u : 0u) << 10) | ((CFG_A_MN ? 1u : 0u) << 15) | ((CFG_B_MN ? 1u : 0u) << 16) | ((unsigned)(NT >> 3) << 17) | ((unsigned)(BM >> 4) << 24);
            unsigned stage = 0, phase = 0;
            bool ok = true;
#if CFG_CHUNK
            // chunk ch has accumulator ch & 1, which the chunk two before it has to have left
            for (int ch = 0, first = 0; first < nkb && ok; ch++, first += CHUNK) {
            if (!mbar_wait(smem_u32(&acc_empty[ch & 1]), ((unsigned)(ch >> 1) & 1u) ^ 1u, &failed)) { ok = false; *(volatile int*)g.status = 24; break; }
            const int end = first + CHUNK < nkb ? first + CHUNK : nkb;
            const unsigned acc = tmem_base + (ch & 1) * NT;
            for (int it = first; it < end; it++) {
#else
            constexpr int first = 0;
            const unsigned acc = tmem_base;
            for (int it = 0; it < nkb; it++) {
#endif
                if (!mbar_wait(smem_u32(&full_bar[stage]), phase, &failed)) { ok = false; *(volatile int*)g.status = 22; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const unsigned sp = smem_base + stage * STAGE_BYTES, sq = sp + P_BYTES;
#if CFG_TF32
                // A_lo · B_hi, A_hi · B_lo, A_hi · B_hi
#pragma unroll
                for (int pass = 0; pass < 3; pass++) {
                    const unsigned pp = pass == 0 ? sp + P_PART : sp, pq = pass == 1 ? sq + Q_PART : sq;
#pragma unroll
                    for (int k = 0; k < 4; k++) umma_f16(acc, make_desc(pp + k * 32, 16, 1024), make_desc(pq + k * 32, 16, 1024), idesc, ((it - first) | pass | k) != 0);
                }
#else
#pragma unroll
                for (int k = 0; k < BK / 16; k++) {
                    // K-major: 32 bytes inside the 128-byte row, 8-row groups 1 KiB apart.  MN-major: 16 k-rows of
                    // 128 bytes, 64-wide m/n groups one box apart.
                    const unsigned long long ad = CFG_A_MN ? make_desc(sp + k * 2048, BK * 128, 1024) : make_desc(sp + k * 32, 16, 1024);
                    const unsigned long long bd = CFG_B_MN ? make_desc(sq + k * 2048, BK * 128, 1024) : make_desc(sq + k * 32, 16, 1024);
                    umma_f16(acc, ad, bd, idesc, ((it - first) | k) != 0);
                }
#endif
                umma_commit(smem_u32(&empty_bar[stage]));
                if (++stage == NSTAGE) { stage = 0; phase ^= 1; }
            }
#if CFG_CHUNK
            if (ok) umma_commit(smem_u32(&acc_full[ch & 1]));
            }
            if (!ok) failed = 1;
#else
            if (ok) umma_commit(smem_u32(&acc_full));
            else failed = 1;
#endif
        }
    }
    __syncwarp();

    // pieces of the finish that this warp takes: piece j, its first row and column in the tile for this lane, and whether it has any
    constexpr int WARPS = THREADS / 32;
    const int per = g.colsum ? 4 : 1, units = (BM / 8 / per) * (NT / 32);
    const int pieces = (units + SPLITS * WARPS - 1) / (SPLITS * WARPS) * per;
    auto piece = [&](int j, int& trow, int& tcol) -> bool {
        const int u = (int)rank * WARPS + warp + (per == 4 ? j >> 2 : j) * (SPLITS * WARPS);
        const int rg = u / (NT / 32), cg = u - rg * (NT / 32);
        trow = (rg * per + (per == 4 ? j & 3 : 0)) * 8 + (lane >> 2);
        tcol = cg * 32 + 8 * (lane & 3);
        return j < pieces && u < units && m0 + trow < g.M && n0 + tcol < g.N;
    };
#if CFG_EPI
    // operands of BATCH pieces in registers: 16 of them for each operand
    constexpr int EPI_NR = EPI_NRAW > 0 ? EPI_NRAW : 1;
    __half2 raw[BATCH][EPI_NR][4];
    auto load_operands = [&](int j0) {
#pragma unroll
        for (int q = 0; q < BATCH; q++) {
            int trow, tcol;
            if (piece(j0 + q, trow, tcol)) epi8_load_(m0 + trow, n0 + tcol, g.ep, raw[q]);
        }
    };
#if !CFG_CHUNK
    load_operands(0);
#endif
#endif

#if CFG_CHUNK
    // ── the eight other warps: a quadrant of the accumulators each, half of the columns, from chunk to chunk in registers and
    // then to shared memory.  When the last chunk is complete, every TMA write has been consumed and every MMA has read
    // its operands: the ring's memory is free. ──
    if (warp >= 2) {
        const int quad = warp & 3, half = (warp - 2) >> 2;
        const bool used = m0 + quad * 32 < g.M;
        const int chunks = (nkb + CHUNK - 1) / CHUNK;
        float sum[NT / 2];
        bool ok = true;
        for (int ch = 0; ch < chunks && ok; ch++) {
            ok = mbar_wait(smem_u32(&acc_full[ch & 1]), (unsigned)(ch >> 1) & 1u, &failed);
            if (!ok && lane == 0) { *(volatile int*)g.status = 23; failed = 1; }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (used) {
#pragma unroll
                for (int c = 0; c < NT / 32; c++) {
                    unsigned v[16];
                    tmem_ld16(tmem_base + ((unsigned)(quad * 32) << 16) + (ch & 1) * NT + half * (NT / 2) + c * 16, v);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 16; j++) sum[c * 16 + j] = ch ? sum[c * 16 + j] + __uint_as_float(v[j]) : __uint_as_float(v[j]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[ch & 1]));
        }
        if (ok && used) {
            float4* const dst = reinterpret_cast<float4*>(tile + (quad * 32 + lane) * LDT + half * (NT / 2));
#pragma unroll
            for (int q = 0; q < NT / 8; q++) dst[q] = make_float4(sum[4 * q], sum[4 * q + 1], sum[4 * q + 2], sum[4 * q + 3]);
        }
    }
#else
    // ── every warp: its quadrant of the accumulator, half of the columns, to shared memory ──
    // The accumulator is complete, so every TMA write has been consumed and every MMA has read its operands: the
    // ring's memory is free.
    bool ok = mbar_wait(smem_u32(&acc_full), 0, &failed);
    if (!ok && lane == 0) { *(volatile int*)g.status = 23; failed = 1; }
    ok = __all_sync(0xffffffffu, ok);
    const int quad = warp & 3, half = warp >> 2;
    if (ok && m0 + quad * 32 < g.M) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < NT / 32; c++) {
            const int col = half * (NT / 2) + c * 16;
            unsigned v[16];
            tmem_ld16(tmem_base + ((unsigned)(quad * 32) << 16) + col, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            float4* const dst = reinterpret_cast<float4*>(tile + (quad * 32 + lane) * LDT + col);
#pragma unroll
            for (int q = 0; q < 4; q++) dst[q] = make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]), __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3]));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
#endif
    // The next launch may start now, beside the finish.  Let in when this CTA had been set up, it and the ones behind it, which let
    // in the next in turn, took places, L2 and issue slots from the loads and products: 21 layers of 64 x 512 fused with GELU 169 us,
    // now 132, of 512 x 1024 273 and 203; a step of 1024 rows, 4 x 1024 wide, 129.7 and 118.6, of 999 rows, 2 x 1000 wide, 97.5 and 91.0;
    // four layers of 32 x 4096 59.7 and 54.8.  Let in by a CTA's end only: 146, 216, 121, 94 and 62.
    asm volatile("griddepcontrol.launch_dependents;");
    __syncthreads();
    if (SPLITS > 1) cluster_sync_all();                  // all partial tiles are in place

    // ── sum of the partials, narrowing, fused consumer, stores: pieces of 8 rows x 32 columns, dealt out over all
    // warps of the cluster (four pieces below one another when column sums over 32 rows are wanted).  Four lanes hold 64
    // contiguous bytes of a row. ──
    const bool vec_ok = (g.N & 7) == 0;
#if !CFG_TF32
    __half* const d_raw = (__half*)g.d_raw;
#endif
    (void)vec_ok;
#if CFG_EPI
    __half* const d_out = (__half*)g.d_out;
#endif
    if (!failed) {
        float x[8];
        for (int j0 = 0; j0 < pieces; j0 += BATCH) {
#if CFG_EPI
            if (j0 > 0 || CHUNK) load_operands(j0);
#endif
            float4 a[BATCH][SPLITS], b[BATCH][SPLITS];
            int trow[BATCH], tcol[BATCH];
            bool on[BATCH];
#pragma unroll
            for (int q = 0; q < BATCH; q++) {
                on[q] = piece(j0 + q, trow[q], tcol[q]);
                if (!on[q]) continue;
                const float* const at = tile + trow[q] * LDT + tcol[q];
                if (SPLITS == 1) { a[q][0] = *reinterpret_cast<const float4*>(at); b[q][0] = *reinterpret_cast<const float4*>(at + 4); }
                else {
#pragma unroll
                    for (int r = 0; r < SPLITS; r++) { const unsigned p = map_to_cta(smem_u32(at), r); a[q][r] = ld_cluster_f4(p); b[q][r] = ld_cluster_f4(p + 16); }
                }
            }
#pragma unroll
            for (int q = 0; q < BATCH; q++) {
                const int j = j0 + q, row = m0 + trow[q], col = n0 + tcol[q];
#if !CFG_TF32
                if ((j & 3) == 0) {
#pragma unroll
                    for (int e = 0; e < 8; e++) x[e] = 0.0f;
                }
#endif
                if (on[q]) {
                    float s[8] = {a[q][0].x, a[q][0].y, a[q][0].z, a[q][0].w, b[q][0].x, b[q][0].y, b[q][0].z, b[q][0].w};
#pragma unroll
                    for (int r = 1; r < SPLITS; r++) { s[0] += a[q][r].x; s[1] += a[q][r].y; s[2] += a[q][r].z; s[3] += a[q][r].w; s[4] += b[q][r].x; s[5] += b[q][r].y; s[6] += b[q][r].z; s[7] += b[q][r].w; }
                    const size_t off = (size_t)row * g.N + col;
#if CFG_TF32
                    float* const d = (float*)g.d_raw + off;
                    if ((g.N & 3) == 0) {
                        *reinterpret_cast<float4*>(d) = make_float4(s[0], s[1], s[2], s[3]);
                        if (col + 4 < g.N) *reinterpret_cast<float4*>(d + 4) = make_float4(s[4], s[5], s[6], s[7]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 8; e++) if (col + e < g.N) d[e] = s[e];
                    }
#else
                    uint4 T;
                    __half2* const t2 = reinterpret_cast<__half2*>(&T);
#pragma unroll
                    for (int e = 0; e < 4; e++) t2[e] = __floats2half2_rn(s[2 * e], s[2 * e + 1]);     // the single narrowing
                    if (vec_ok) {
                        if (d_raw) *reinterpret_cast<uint4*>(d_raw + off) = T;
#if CFG_EPI
                        uint4 O;
                        epi8_(row, col, t2, reinterpret_cast<__half2*>(&O), g.ep, raw[q]);
                        *reinterpret_cast<uint4*>(d_out + off) = O;
                        T = O;
#endif
                        if (g.colsum) {
#pragma unroll
                            for (int e = 0; e < 4; e++) { const float2 f = __half22float2(t2[e]); x[2 * e] += f.x; x[2 * e + 1] += f.y; }
                        }
                    } else {
                        // row stride not a multiple of 16 bytes (no fused consumer on this route)
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            if (col + 2 * e < g.N) d_raw[off + 2 * e] = __low2half(t2[e]);
                            if (col + 2 * e + 1 < g.N) d_raw[off + 2 * e + 1] = __high2half(t2[e]);
                        }
                    }
#endif
                }
#if !CFG_TF32
                if (g.colsum && (j & 3) == 3) {
                    // the eight lanes of a column piece hold rows i * 8 + lane / 4: their sums, across the lanes
#pragma unroll
                    for (int o = 4; o <= 16; o <<= 1)
#pragma unroll
                        for (int e = 0; e < 8; e++) x[e] += __shfl_xor_sync(0xffffffffu, x[e], o);
                    const int row0 = m0 + (trow[q] & ~31);
                    if (lane < 4 && trow[q] < BM && row0 < g.M && col < g.N) {        // warps past the last unit have rows past the tile
                        float* const cs = g.colsum + (size_t)(row0 >> 5) * g.N + col;
#pragma unroll
                        for (int e = 0; e < 8; e++) cs[e] = x[e];
                    }
                }
#endif
            }
        }
    }
    __syncthreads();
    if (SPLITS > 1) cluster_meet_all();                  // the others' tiles stay until they have been read
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
    }
}

}  // namespace CFG_NAME

#if CFG_ALONE
#if CFG_TF32
extern "C" __global__ void __launch_bounds__(CFG_NAME::THREADS, 2)
gemm_f16_tcgen05_small(const __grid_constant__ TensorMap map_a, const __grid_constant__ TensorMap map_b,
                       const __grid_constant__ TensorMap map_a_lo, const __grid_constant__ TensorMap map_b_lo, const __grid_constant__ SmallGemmArgs g) {
    CFG_NAME::run(map_a, map_b, map_a_lo, map_b_lo, g, blockIdx.x);
}
#else
extern "C" __global__ void __launch_bounds__(CFG_NAME::THREADS, 2)
gemm_f16_tcgen05_small(const __grid_constant__ TensorMap map_a, const __grid_constant__ TensorMap map_b, const __grid_constant__ SmallGemmArgs g) {
    CFG_NAME::run(map_a, map_b, g, blockIdx.x);
}
#endif
#endif
#endif  // ANL_SMALL_GEMM_DEVICE_CODE
