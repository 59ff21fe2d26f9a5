// Dense contractions on the 5th-generation tensor cores: D[M,N] = sum_k A[m,k] * B[n,k], f16
// operands, f32 accumulation in tensor memory, one rounding to f16 at the store — the arithmetic
// the reference specifies for an f16 REDUCE (f32 accumulator, operands widened, narrowed once:
// codegen/lower.go:654-719), reached through tcgen05.mma instead of its one-thread-per-output loop.
//
// This file is the host side of two kernels, both compiled at run time, once per configuration (operand
// major-ness, tile, ring depth, fused elementwise consumer), so that the consumer's generated code can sit in
// their epilogue and the tunables are compile-time constants a search can vary:
//   gemm_pair_kernel.cuh   persistent CTA pairs with 256-row tiles, for outputs with enough tiles to occupy them;
//                          the same text serves f32 contractions in 3 x TF32 form (operand split pre-pass, K
//                          slices and their sum are further down);
//   gemm_small_kernel.cuh  128-row tiles shared by a cluster of CTAs that split K, for the others.
// Either operand may be K-major (k contiguous) or MN-major (m / n contiguous): the forward pass
// x·Wᵀ is K/K, the input gradient dY·W is K/MN, the weight gradient dYᵀ·X is MN/MN.  No operand
// is transposed in memory; the layout goes into the shared-memory and instruction descriptors.  An operand whose
// rows do not start on 16-byte boundaries (TMA's rule) is copied to scratch with padded rows first.
// No multicast is used anywhere: every CTA issues its own loads.
//
// Every wait on an mbarrier is bounded; a wait that runs out records a code in a host-visible
// status word and the CTA drains and frees its tensor memory instead of spinning.
#include <cuda_fp16.h>

#include <cstdlib>
#include <cstring>

#include "gemm_pair_kernel.cuh"      // argument blocks only: the device code is compiled at run time
#include "gemm_small_kernel.cuh"
#include "runtime.hpp"

namespace anl {

// texts of the two kernels, written beside the objects by the build step
static const char* const kPairKernelSource =
#include "gemm_pair_src.inc"
    ;
static const char* const kSmallKernelSource =
#include "gemm_small_src.inc"
    ;

constexpr int BM = 128, BK = 64;
constexpr int A_TILE_BYTES = BM * BK * 2;          // 16 KiB
constexpr int PAIR_THREADS = 320;        // two-CTA kernel: producer, MMA issuer and eight epilogue warps

struct GemmPlan {
    Contraction c;
    bool a_mn = false, b_mn = false;     // MN-major operands
    int64_t lda = 0, ldb = 0;            // elements between consecutive rows of the 2-D global views
    bool pad_a = false, pad_b = false;   // rows not on 16-byte boundaries: copied to scratch with padded rows at launch
    bool f32 = false;                    // f32 operands: the FP32-pipe kernel instead of tcgen05
    GemmTuning tune;                     // zero fields: heuristics
};

static int encode_map(anl_device* dev, CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint64_t row_stride_elems,
                      uint32_t box_inner, uint32_t box_outer, bool f32 = false) {
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {row_stride_elems * (f32 ? 4 : 2)};
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = dev->drv.TensorMapEncodeTiled(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) { const char* s = nullptr; dev->drv.GetErrorString(r, &s); return dev->fail(ANL_ERR_CUDA, std::string("gemm: cuTensorMapEncodeTiled: ") + (s ? s : "?")); }
    return ANL_OK;
}

// Host-visible status word and tile counters of this device.  A launch draws tile numbers from the
// counter that belongs to its stream, so contractions queued on different streams cannot disturb
// each other's draw; launches on one stream run one after the other and share one.
static int ensure_gemm_state(anl_device* dev) {
    if (!dev->gemm_status_host) {
        if (cudaHostAlloc((void**)&dev->gemm_status_host, 64, cudaHostAllocMapped) != cudaSuccess) return dev->fail(ANL_ERR_CUDA, "gemm: cannot allocate the status word");
        *dev->gemm_status_host = 0;
        if (cudaHostGetDevicePointer((void**)&dev->gemm_status_dev, dev->gemm_status_host, 0) != cudaSuccess) return dev->fail(ANL_ERR_CUDA, "gemm: cannot map the status word");
    }
    if (!dev->gemm_tile_counter) {
        const size_t bytes = (size_t)anl_device::kGemmCounterSlots * 256;
        if (cudaMalloc((void**)&dev->gemm_tile_counter, bytes) != cudaSuccess) return dev->fail(ANL_ERR_CUDA, "gemm: cannot allocate the tile counters");
        if (cudaMemset(dev->gemm_tile_counter, 0, bytes) != cudaSuccess) return dev->fail(ANL_ERR_CUDA, "gemm: cannot clear the tile counters");   // launches leave them zeroed again
    }
    return ANL_OK;
}

int counter_slot(anl_device* dev, cudaStream_t stream) {
    for (size_t k = 0; k < dev->gemm_counter_streams.size(); k++) if (dev->gemm_counter_streams[k] == stream) return (int)k;
    if ((int)dev->gemm_counter_streams.size() >= anl_device::kGemmCounterSlots) return 0;      // more streams than slots: those share the first one (never the case for this runtime's three)
    dev->gemm_counter_streams.push_back(stream);
    return (int)dev->gemm_counter_streams.size() - 1;
}
static int* tile_counter_for(anl_device* dev, cudaStream_t stream) { return dev->gemm_tile_counter + counter_slot(dev, stream) * 64; }

// A barrier wait that ran out leaves its code in the status word and the tile counters undefined (a
// CTA that gives up does not sign off).  Called where the host has just waited for the device: report
// once, clear the word and zero the counters so that later launches, replays included, start clean.
int gemm_check_status(anl_device* dev) {
    if (!dev->gemm_status_host || *dev->gemm_status_host == 0) return ANL_OK;
    const int code = *dev->gemm_status_host;
    cudaDeviceSynchronize();
    if (dev->gemm_tile_counter) cudaMemset(dev->gemm_tile_counter, 0, (size_t)anl_device::kGemmCounterSlots * 256);
    *dev->gemm_status_host = 0;
    return dev->fail(ANL_ERR_CUDA, "gemm: a launch timed out on a barrier (code " + std::to_string(code) + "); its output is incomplete");
}

// Test hook: puts the device in the state a timed-out barrier wait leaves behind (a code in the
// status word, a tile counter that was not signed off), without making any wait run out.
int gemm_inject_status(anl_device* dev, int code, int counter_value) {
    if (int rc = ensure_gemm_state(dev)) return rc;
    cudaStreamSynchronize(dev->stream);
    int words[2] = {counter_value, 0};
    for (int k = 0; k < anl_device::kGemmCounterSlots; k++)
        if (cudaMemcpy(dev->gemm_tile_counter + k * 64, words, sizeof words, cudaMemcpyHostToDevice) != cudaSuccess) return dev->fail(ANL_ERR_CUDA, "gemm: cannot write the tile counter");
    *dev->gemm_status_host = code;
    return ANL_OK;
}

// Is this f16 contraction worth a tensor-core launch instead of the generated kernel of lanes that share an output?
static bool gemm_f16_worth(const GemmPlan& gp) {
    const Contraction& c = gp.c;
    const bool padded = gp.pad_a || gp.pad_b;
    if (!padded && c.M >= 64 && c.N >= 64 && c.K >= 32) return true;
    // A handful of outputs: a tile has eight CTAs at most, the generated reduction is split over the whole machine, and adds in
    // f32 with rounding.  Tensor cores against generated kernel in us (K at 16384 / 262144): 64 outputs 17 / 145 against 8 / 12,
    // 256 outputs 16 / 145 against 10 / 25, 1024 outputs 18 / 148 against 10 / 76 with both operands k-contiguous; with neither,
    // 1024 outputs are 27 / 148 against 20 / 180, and from 4096 on the tensor cores are ahead (20 / 148 against 20 / 221 and
    // 27 / 150 against 41 / 804).
    if (c.M * c.N <= 1024) return false;
    // Few rows or few columns: most of a 128-row tile is empty, so it takes enough work to pay for the launch;
    // with an operand that has to be copied first, more.  The generated kernel adds these sums in f32 with rounding, tensor
    // memory cuts them, in chunks of at most 1024 terms: 5.6e-6 of a sum of positive terms, a twenty-fifth of what the one
    // rounding to f16 leaves (1.4e-4 rms).
    const double work = (double)c.M * (double)c.N * (double)c.K;
    return c.K >= 64 && work >= (padded ? 1 << 23 : 1 << 20);
}

int plan_gemm(const Item& item, const GemmTuning& tune, Plan& plan) {
    Contraction c;
    if (!match_contraction(item, c)) return ANL_ERR_UNSUPPORTED;
    const bool dynamic = c.m_sym || c.k_sym;
    if (c.in_dtype == DT_F32 && c.out_dtype == DT_F32) {
        if (c.a_sk != 1 && c.a_sm != 1) return ANL_ERR_UNSUPPORTED;
        if (c.b_sk != 1 && c.b_sn != 1) return ANL_ERR_UNSUPPORTED;
        if (!dynamic && !gemm_f32_worth(c.M, c.N, c.K, c.a_sm, c.a_sk, c.b_sn, c.b_sk)) return ANL_ERR_UNSUPPORTED;
        if (c.N < 64) return ANL_ERR_UNSUPPORTED;
        auto gp = std::make_shared<GemmPlan>();
        gp->c = c; gp->f32 = true;
        plan.gemm = gp;
        plan.gemm_dynamic = dynamic;
        if (!dynamic) {
            plan.r.klass = KC_GEMM;
            plan.r.note = "gemm f32 M=" + std::to_string(c.M) + " N=" + std::to_string(c.N) + " K=" + std::to_string(c.K);
        }
        return ANL_OK;
    }
    if (c.in_dtype != DT_F16 || c.out_dtype != DT_F16) return ANL_ERR_UNSUPPORTED;
    if (dynamic) return ANL_ERR_UNSUPPORTED;                                   // tcgen05 path: static extents only
    if (c.M >= (1ll << 31) || c.N >= (1ll << 31) || c.K >= (1ll << 31)) return ANL_ERR_UNSUPPORTED;
    auto gp = std::make_shared<GemmPlan>();
    gp->c = c;
    gp->tune = tune;
    // A: either k contiguous (K-major, row stride a_sm) or m contiguous (MN-major, row stride a_sk)
    if (c.a_sk == 1 && (c.M == 1 || c.a_sm >= c.K)) { gp->a_mn = false; gp->lda = c.M == 1 ? (c.K + 7) & ~7ll : c.a_sm; }
    else if (c.a_sm == 1 && c.a_sk >= c.M) { gp->a_mn = true; gp->lda = c.a_sk; }
    else return ANL_ERR_UNSUPPORTED;
    if (c.b_sk == 1 && c.b_sn >= c.K) { gp->b_mn = false; gp->ldb = c.b_sn; }
    else if (c.b_sn == 1 && c.b_sk >= c.N) { gp->b_mn = true; gp->ldb = c.b_sk; }
    else return ANL_ERR_UNSUPPORTED;
    // TMA: 16-byte aligned bases and row strides
    gp->pad_a = gp->lda % 8 != 0 || c.a_off % 8 != 0;
    gp->pad_b = gp->ldb % 8 != 0 || c.b_off % 8 != 0;
    if (!gemm_f16_worth(*gp)) return ANL_ERR_UNSUPPORTED;
    plan.gemm = gp;
    plan.r.klass = KC_GEMM;
    plan.r.note = std::string("gemm tcgen05 ") + (gp->a_mn ? "A:MN" : "A:K") + (gp->b_mn ? " B:MN" : " B:K") + " M=" + std::to_string(c.M) + " N=" + std::to_string(c.N) + " K=" + std::to_string(c.K);
    return ANL_OK;
}

// SMs the persistent GEMM may occupy.  When gradients are reduced while the backward pass is still
// running, a few SMs can be left free so that the collective's blocks (and the update kernels behind
// them) find a place at once instead of waiting for a persistent grid to drain.
static int gemm_sm_budget(anl_device* dev) {
    if (!dev) return 148;                                  // rendering without a device: a B200's count
    int sms = dev->prop.multiProcessorCount;
    int want = dev->nranks > 1 ? sms - dev->comm_reserved_sms : sms;
    want = std::max(2, std::min(want, sms));
    return want & ~1;
}

double gemm_flops(const Plan& plan, int64_t sym_value) {
    const Contraction& c = plan.gemm->c;
    return 2.0 * (double)(c.m_sym ? sym_value : c.M) * (double)c.N * (double)(c.k_sym ? sym_value : c.K);
}

int64_t gemm_window_rows(const Plan& plan, int64_t* row_elems) {
    if (!gemm_fusable(plan) || plan.gemm->pad_a || plan.gemm->pad_b) return 0;
    if (row_elems) *row_elems = plan.gemm->c.N;
    return plan.gemm->c.M;
}

bool gemm_taken(const Plan& plan, int64_t sym_value) {
    if (!plan.gemm) return false;
    if (!plan.gemm_dynamic) return plan.r.klass == KC_GEMM;
    const Contraction& c = plan.gemm->c;
    return gemm_f32_worth(c.m_sym ? sym_value : c.M, c.N, c.k_sym ? sym_value : c.K, c.a_sm, c.a_sk, c.b_sn, c.b_sk);
}

// a shape that fills a 256-row tile: the sources anl_lower_gemm shows
bool gemm_pair_shape(const Plan& plan) {
    return gemm_fusable(plan) && plan.gemm->tune.single_cta == 0 && plan.gemm->c.M >= 2 * BM && plan.gemm->c.N >= BM;
}
bool gemm_fusable(const Plan& plan) { return plan.gemm && !plan.gemm_dynamic && plan.r.klass == KC_GEMM && !plan.gemm->f32; }

int gemm_b_param(const Plan& plan) { return plan.gemm->c.b_param; }
void gemm_shape(const Plan& plan, int64_t* M, int64_t* N, int64_t* K) { *M = plan.gemm->c.M; *N = plan.gemm->c.N; *K = plan.gemm->c.K; }

// ── the run-time compiled two-CTA kernel ──────────────────────────────────────────────────────
namespace {

struct PairVariant { int bnt, stages, group_m, stream_stores; bool a_mn, b_mn; bool split_tail; bool tf32 = false; };
constexpr int kDefaultStages = 7;      // the deepest ring that fits beside a 256-wide tile; 1% faster than 6 on every large shape measured

int pair_smem_bytes(int bnt, int stages, bool tf32 = false) { return stages * (tf32 ? 2 : 1) * (A_TILE_BYTES + (bnt / 2) * BK * 2) + 1024; }

// ring depth that fits beside the static barriers: 227 KiB per CTA
int max_stages(int bnt) { int s = 8; while (s > 2 && pair_smem_bytes(bnt, s) > 227 * 1024 - 512) s--; return s; }

std::string pair_source(const PairVariant& v, const std::string& epilogue) {
    std::string s;
    s += "#define ANL_PAIR_GEMM_DEVICE_CODE 1\n";
    s += "#define CFG_A_MN " + std::to_string(v.a_mn ? 1 : 0) + "\n#define CFG_B_MN " + std::to_string(v.b_mn ? 1 : 0) + "\n";
    s += "#define CFG_BNT " + std::to_string(v.bnt) + "\n#define CFG_STAGES " + std::to_string(v.stages) + "\n";
    s += "#define CFG_GROUP_M " + std::to_string(v.group_m) + "\n#define CFG_STREAM_STORES " + std::to_string(v.stream_stores) + "\n";
    s += "#define CFG_EPI " + std::string(epilogue.empty() ? "0" : "1") + "\n";
    s += "#define CFG_TF32 " + std::string(v.tf32 ? "1" : "0") + "\n";
    s += epilogue;
    s += kPairKernelSource;
    return s;
}

int load_gemm_kernel(anl_device* dev, const std::string& source, const char* entry, int smem_bytes, const std::string& key, CUfunction* fn) {
    std::shared_ptr<Module> m;
    if (int rc = compile_source(dev, source, m)) return rc;
    auto f = m->fn.find(entry);
    if (f != m->fn.end()) { *fn = f->second; dev->pair_kernels[key] = (void*)*fn; return ANL_OK; }
    CUresult cr = dev->drv.ModuleGetFunction(fn, m->mod, entry);
    if (cr != CUDA_SUCCESS) return dev->fail(ANL_ERR_CUDA, std::string("gemm: ") + entry + ": entry point missing");
    cr = dev->drv.FuncSetAttribute(*fn, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, smem_bytes);
    if (cr != CUDA_SUCCESS) { const char* e = nullptr; dev->drv.GetErrorString(cr, &e); return dev->fail(ANL_ERR_CUDA, std::string("gemm: cuFuncSetAttribute: ") + (e ? e : "?")); }
    m->fn[entry] = *fn;
    dev->pair_kernels[key] = (void*)*fn;
    return ANL_OK;
}

int get_pair_kernel(anl_device* dev, const PairVariant& v, const std::string& epilogue, CUfunction* fn) {
    // looked up by the configuration, so that a launch does not assemble and hash 40 KB of source
    char head[96];
    std::snprintf(head, sizeof head, "%d,%d,%d,%d,%d,%d,%d|", v.bnt, v.stages, v.group_m, v.stream_stores, (int)v.a_mn, (int)v.b_mn, (int)v.tf32);
    const std::string key = head + epilogue;
    auto hit = dev->pair_kernels.find(key);
    if (hit != dev->pair_kernels.end()) { *fn = (CUfunction)hit->second; return ANL_OK; }
    return load_gemm_kernel(dev, pair_source(v, epilogue), "gemm_f16_tcgen05_pair", pair_smem_bytes(v.bnt, v.stages, v.tf32), key, fn);
}

PairVariant choose_variant(anl_device* dev, const GemmPlan& gp_in, int64_t M) {
    // the plan's own tunables (a search result) first, then the device's defaults, then the heuristics
    GemmPlan gp = gp_in;
    if (dev) {
        const GemmTuning& d = dev->gemm_defaults;
        if (!gp.tune.tile_n) gp.tune.tile_n = d.tile_n;
        if (!gp.tune.stages) gp.tune.stages = d.stages;
        if (!gp.tune.group_m) gp.tune.group_m = d.group_m;
        if (!gp.tune.stream_stores) gp.tune.stream_stores = d.stream_stores;
        if (!gp.tune.no_split_tail) gp.tune.no_split_tail = d.no_split_tail;
    }
    const Contraction& c = gp.c;
    PairVariant v{};
    v.a_mn = gp.a_mn; v.b_mn = gp.b_mn;
    const int npairs = gemm_sm_budget(dev) / 2;
    const int tm2 = (int)((M + 2 * BM - 1) / (2 * BM));
    if (gp.tune.tile_n == 128 || gp.tune.tile_n == 256) v.bnt = gp.tune.tile_n;
    else {
        // The narrow tile fills the last wave of tiles better but stages 1.5x the bytes per flop and
        // measured 25% slower on 4096x4096x8192 (it becomes L2-bound), so it is only taken when the
        // wide tile would leave most pairs idle.
        auto fill = [&](int bnt) { long long t = (long long)tm2 * ((c.N + bnt - 1) / bnt); long long w = (t + npairs - 1) / npairs; return (double)t / (double)(w * npairs); };
        v.bnt = (fill(128) * 0.7 > fill(256)) ? 128 : 256;
    }
    v.stages = gp.tune.stages > 0 ? std::max(2, std::min(gp.tune.stages, max_stages(v.bnt))) : std::min(kDefaultStages, max_stages(v.bnt));
    v.group_m = gp.tune.group_m > 0 ? gp.tune.group_m : (gp.tune.group_m < 0 ? 0 : kDefaultGroupM);
    v.stream_stores = gp.tune.stream_stores > 0 ? 1 : 0;
    v.split_tail = gp.tune.no_split_tail == 0;
    return v;
}

}  // namespace

// ── the run-time compiled one-CTA kernel ──────────────────────────────────────────────────────
namespace {

struct SmallVariant { bool a_mn, b_mn; int nt, prows, stages, splits, chunk; bool tf32; int threads() const { return chunk ? 320 : 256; } };
// k extent the 3 x TF32 form accumulates in tensor memory before adding to the output in f32.  Measured on
// 4096 x 2048 x 8192 (error against float64, of the largest output): 1024 -> 7.6e-6 at 226 TFLOP/s,
// 512 -> 3.5e-6 at 207, 256 -> 1.7e-6 at 146; the reference's serial f32 loop: 3.6e-6 (9.4e-6 at K = 65536).
constexpr int kTf32ChunkK = 1024;

// shared memory of one CTA: the ring (the MMA reads 128 rows from the start of a stage's A part, whatever was
// staged there), later the f32 tile of the rows that exist
int small_smem_bytes(const SmallVariant& v) {
    const int parts = v.tf32 ? 2 : 1, stage = parts * (v.prows + v.nt) * 128;
    const int ring = std::max(v.stages * stage, (v.stages - 1) * stage + (parts - 1) * v.prows * 128 + A_TILE_BYTES);
    return std::max(ring, v.prows * (v.nt + 4) * 4) + 1024;
}

SmallVariant choose_small(int64_t M, int64_t N, int64_t K, bool a_mn, bool b_mn, bool tf32) {
    SmallVariant v{};
    v.a_mn = a_mn; v.b_mn = b_mn; v.tf32 = tf32;
    v.prows = 128;
    // rows of the f32 tile are written by whole 32-lane quadrants
    if (!a_mn && M <= 64) v.prows = M <= 32 ? 32 : 64;
    const int parts = tf32 ? 2 : 1, bk = tf32 ? 32 : BK;
    const int64_t kblocks = (K + bk - 1) / bk, tm = (M + BM - 1) / BM;
    const int most = tf32 ? 8 : 16;           // k-blocks of a chunk: 256 f32 or 1024 f16 terms
    double best = 1e30, best_ctas = 0;
    for (int nt : {128, 64, 32}) {
        if (b_mn && nt < 64) continue;
        for (int splits : {1, 2, 4, 8}) {
            if (splits > 1 && kblocks / splits < 2) break;
            const int64_t per = (kblocks + splits - 1) / splits;
            const double ctas = (double)(tm * ((N + nt - 1) / nt) * splits);
            // Time of the busiest SM in us, fitted to a sweep over 24 shapes from 1 x 4096 x 4096 to 2048-cubed: 3 for
            // the launch, prologue and epilogue; its k-blocks' loads at 100 bytes a ns for one CTA, 135 for two
            // or more that take turns, a quarter of a microsecond a k-block at least (32 x 4096 x 4096 in 128 narrow
            // tiles without a split: 20 us against 10); the cluster's barriers and the sum of its partials.  Clusters of eight
            // land two CTAs to an SM even where there are SMs to spare, and clusters that do not all fit
            // at once start late (512 x 4096 x 4096 split four ways: 39 us against 22.6 split two ways).
            const bool alone = tf32 && nt == 128 && v.prows == 128;         // 64 KB a stage: one CTA an SM
            const double n = std::max(std::ceil(ctas / 148.0), splits == 8 ? 2.0 : 1.0);
            const double load = std::max(n * per * (double)(parts * (v.prows + nt) * 128) / (n > 1 && !alone ? 135e3 : 100e3), std::ceil(alone ? n : n / 2) * per * 0.25);
            double t = 3.0 + load + (splits == 1 ? 0.0 : splits == 2 ? 2.0 : splits == 4 ? 2.5 : 7.0);
            if (splits > 1 && ctas > 2 * 148) t *= 2;
            if (t < best) { best = t; best_ctas = ctas; v.nt = nt; v.splits = splits; v.chunk = per > most ? most : 0; }
        }
    }
    // two CTAs an SM, at most 110 KB each, unless each has an SM for itself or two stages do not fit that way
    v.stages = 8;
    SmallVariant two = v; two.stages = 2;
    const int room = tf32 && (best_ctas <= 148 || small_smem_bytes(two) > 110 * 1024) ? 220 * 1024 : 110 * 1024;
    while (v.stages > 2 && small_smem_bytes(v) > room) v.stages--;
    return v;
}
SmallVariant choose_small(const GemmPlan& gp, int64_t M) {
    SmallVariant v = choose_small(M, gp.c.N, gp.c.K, gp.a_mn, gp.b_mn, false);
    // a search may set the tile's width and the depth of the ring; the slices of K, and with them the order of the additions, stay
    if (!gp.tune.single_cta) return v;
    const int nt = gp.tune.tile_n;
    if (nt == 128 || nt == 64 || (nt == 32 && !gp.b_mn)) {
        v.nt = nt;
        for (v.stages = 8; v.stages > 2 && small_smem_bytes(v) > 110 * 1024;) v.stages--;
    }
    if (gp.tune.stages >= 2) for (v.stages = std::min(gp.tune.stages, 8); v.stages > 2 && small_smem_bytes(v) > 220 * 1024;) v.stages--;
    return v;
}

// `name`: empty for a kernel of its own, else the namespace of one of two configurations in a text
std::string small_source(const SmallVariant& v, const std::string& epilogue, const std::string& name = std::string()) {
    std::string s;
    s += "#define ANL_SMALL_GEMM_DEVICE_CODE 1\n";
    s += "#define CFG_NAME " + (name.empty() ? std::string("alone") : name) + "\n#define CFG_ALONE " + (name.empty() ? "1" : "0") + "\n";
    s += "#define CFG_A_MN " + std::to_string(v.a_mn ? 1 : 0) + "\n#define CFG_B_MN " + std::to_string(v.b_mn ? 1 : 0) + "\n";
    s += "#define CFG_NT " + std::to_string(v.nt) + "\n#define CFG_PROWS " + std::to_string(v.prows) + "\n";
    s += "#define CFG_STAGES " + std::to_string(v.stages) + "\n#define CFG_SPLITS " + std::to_string(v.splits) + "\n";
    s += "#define CFG_EPI " + std::string(epilogue.empty() ? "0" : "1") + "\n";
    s += "#define CFG_TF32 " + std::string(v.tf32 ? "1" : "0") + "\n#define CFG_CHUNK " + std::to_string(v.chunk) + "\n";
    if (name.empty()) s += epilogue;
    else if (!epilogue.empty()) s += "#include <cuda_fp16.h>\nnamespace " + name + " {\n" + epilogue + "}\n";
    s += kSmallKernelSource;
    return s;
}

// Both configurations in one kernel: the first `ctas` CTAs are the first one's.
std::string small_pair_source(const SmallVariant& v0, const std::string& epi0, const SmallVariant& v1, const std::string& epi1) {
    std::string s = small_source(v0, epi0, "first");
    for (const char* m : {"ANL_SMALL_GEMM_DEVICE_CODE", "CFG_NAME", "CFG_ALONE", "CFG_A_MN", "CFG_B_MN", "CFG_NT", "CFG_PROWS", "CFG_STAGES", "CFG_SPLITS", "CFG_EPI", "CFG_TF32", "CFG_CHUNK", "EPI_NRAW"}) s += std::string("#undef ") + m + "\n";
    s += small_source(v1, epi1, "second");
    s += "extern \"C\" __global__ void __launch_bounds__(first::THREADS, 2)\n"
         "gemm_f16_tcgen05_small_two(const __grid_constant__ TensorMap map_a0, const __grid_constant__ TensorMap map_b0, const __grid_constant__ TensorMap map_a1,\n"
         "                           const __grid_constant__ TensorMap map_b1, const __grid_constant__ SmallGemmArgs g0, const __grid_constant__ SmallGemmArgs g1, const unsigned ctas) {\n"
         "    static_assert(first::THREADS == second::THREADS && first::SPLITS == second::SPLITS, \"one launch, one block and cluster shape\");\n"
         "    if (blockIdx.x < ctas) first::run(map_a0, map_b0, g0, blockIdx.x);\n"
         "    else second::run(map_a1, map_b1, g1, blockIdx.x - ctas);\n}\n";
    return s;
}

std::string small_key(const SmallVariant& v, const std::string& epilogue) {
    char head[96];
    std::snprintf(head, sizeof head, "s%d,%d,%d,%d,%d,%d,%d,%d|", v.nt, v.prows, v.stages, v.splits, v.chunk, (int)v.a_mn, (int)v.b_mn, (int)v.tf32);
    return head + epilogue;
}
int get_small_kernel(anl_device* dev, const SmallVariant& v, const std::string& epilogue, CUfunction* fn) {
    const std::string key = small_key(v, epilogue);
    auto hit = dev->pair_kernels.find(key);
    if (hit != dev->pair_kernels.end()) { *fn = (CUfunction)hit->second; return ANL_OK; }
    return load_gemm_kernel(dev, small_source(v, epilogue), "gemm_f16_tcgen05_small", small_smem_bytes(v), key, fn);
}

// Which of the two kernels?  The pair kernel's 256 x 256 tiles move the fewest bytes per product, but half of the
// 74 pairs have to get one, or (K up to 2048, where the pair kernel's longer prologue still shows) all of them.
// Measured, one-CTA against pair in us, events included: 1024-cubed 12.3 / 16.4, 512 x 4096 x 4096 28.7 / 32.8,
// 1024 x 1024 x 8192 32.7 / 54.2 (16 tiles); 2048-cubed 23.5 / 25.5, 4096 x 1024 x 1024 16.4 / 19.4 (64 tiles); the
// other way 2048 x 2048 x 8192 63.5 / 59.4 and 1000 x 4096 x 8192 94.2 / 61.4 (64 tiles); from 81 tiles on the two are
// equal at K = 1024 and the pair kernel is ahead above.
bool small_takes(const GemmPlan& gp, int64_t M) {
    const Contraction& c = gp.c;
    if (gp.tune.single_cta || M < 2 * BM || c.N < 128) return true;
    if (gp.tune.tile_n) return false;
    const int64_t tiles = ((M + 255) / 256) * ((c.N + 255) / 256);
    return tiles <= 36 || (tiles <= 74 && c.K <= 2048);
}

}  // namespace

// A one-CTA launch that is ready but waits for the next contraction.
struct HeldGemm { SmallVariant v; std::string epilogue; CUtensorMap ma, mb; SmallGemmArgs g; int64_t ctas; };
void drop_held(HeldGemm* h) { delete h; }
bool gemm_holdable(const Plan& plan) { return gemm_fusable(plan) && !plan.gemm->pad_a && !plan.gemm->pad_b && small_takes(*plan.gemm, plan.gemm->c.M); }
// One CTA of each on an SM, and one launch's shape for both.  (The larger ones fill the machine by themselves.)
bool gemm_pairs(const HeldGemm& a, const HeldGemm& b) {
    return a.v.splits == b.v.splits && a.v.threads() == b.v.threads() && a.ctas <= 148 && b.ctas <= 148 &&
           small_smem_bytes(a.v) <= 110 * 1024 && small_smem_bytes(b.v) <= 110 * 1024;
}
int launch_held(anl_device* dev, HeldGemm& a, HeldGemm* b, cudaStream_t stream) {
    CUfunction fn;
    if (!b) {
        if (int rc = get_small_kernel(dev, a.v, a.epilogue, &fn)) return rc;
        void* params[3] = {&a.ma, &a.mb, &a.g};
        if (int rc = launch_kernel(dev, fn, KernelShape{(unsigned)a.ctas, 1, 1, (unsigned)a.v.threads(), 1, 1, (unsigned)small_smem_bytes(a.v), (unsigned)a.v.splits}, stream, params, true, "gemm_f16_tcgen05_small")) return rc;
        dev->stats.gemm_launched++;
        return ANL_OK;
    }
    const int smem = std::max(small_smem_bytes(a.v), small_smem_bytes(b->v));
    const std::string key = small_key(a.v, a.epilogue) + "&" + small_key(b->v, b->epilogue);
    auto hit = dev->pair_kernels.find(key);
    if (hit != dev->pair_kernels.end()) fn = (CUfunction)hit->second;
    else if (int rc = load_gemm_kernel(dev, small_pair_source(a.v, a.epilogue, b->v, b->epilogue), "gemm_f16_tcgen05_small_two", smem, key, &fn)) return rc;
    unsigned ctas = (unsigned)a.ctas;
    void* params[7] = {&a.ma, &a.mb, &b->ma, &b->mb, &a.g, &b->g, &ctas};
    if (int rc = launch_kernel(dev, fn, KernelShape{(unsigned)(a.ctas + b->ctas), 1, 1, (unsigned)a.v.threads(), 1, 1, (unsigned)smem, (unsigned)a.v.splits}, stream, params, true, "gemm_f16_tcgen05_small_two")) return rc;
    dev->stats.gemm_launched += 2;
    return ANL_OK;
}

int gemm_small_parts(const Plan& plan) {
    if (!gemm_fusable(plan) || !small_takes(*plan.gemm, plan.gemm->c.M)) return 0;
    const SmallVariant v = choose_small(*plan.gemm, plan.gemm->c.M);
    return v.splits * (v.chunk ? 2 : 1);
}

// Is a consumer worth joining where its output has to move for it (run_items)?  Not where one wave of large tiles leaves the whole
// finish exposed: us a layer with GELU, joined against apart, two-CTA kernel 706 x 3840 (45 tiles for 74 pairs) +1.0, 1024 x 3840
// (60) +0.6, 1500 x 3840 (90) -2.8; one-CTA kernel, 128 x 128 tiles of whole K on an SM each, 2048 x 1024 +0.3, 1500 x 1024 0.0;
// narrower ones 1024 x 1024 -0.8, 512 x 512 -0.9, split ones 384 x 1024 -1.9.
bool gemm_joins_moved(anl_device* dev, const Plan& plan) {
    const Contraction& c = plan.gemm->c;
    if (small_takes(*plan.gemm, c.M)) {
        const SmallVariant v = choose_small(*plan.gemm, c.M);
        const int64_t tiles = ((c.M + BM - 1) / BM) * ((c.N + v.nt - 1) / v.nt);
        return v.splits > 1 || v.nt < 128 || v.prows < 128 || tiles > gemm_sm_budget(dev);
    }
    const PairVariant v = choose_variant(dev, *plan.gemm, c.M);
    return ((c.M + 2 * BM - 1) / (2 * BM)) * ((c.N + v.bnt - 1) / v.bnt) > gemm_sm_budget(dev) / 2;
}

// the source that a launch of this plan will use, and the kernel itself
int gemm_source(anl_device* dev, const Plan& plan, const std::string& epilogue, std::string& out) {
    if (!gemm_fusable(plan)) return ANL_ERR_UNSUPPORTED;
    const int64_t M = plan.gemm->c.M;
    out = small_takes(*plan.gemm, M) ? small_source(choose_small(*plan.gemm, M), epilogue) : pair_source(choose_variant(dev, *plan.gemm, M), epilogue);
    return ANL_OK;
}

// Copies of f16 matrices with rows padded to a multiple of 8 elements (the padding zero), 8 elements a thread;
// blockIdx.y picks one of the two operands of a contraction.
struct PadArgs { const __half* src[2]; __half* dst[2]; long long rows[2], cols[2], ld[2], ldp[2]; };
__global__ void __launch_bounds__(256) pad_rows_f16(const PadArgs a) {
    enter_kernel();
    const int w = blockIdx.y;
    const long long per_row = a.ldp[w] >> 3, total = a.rows[w] * per_row;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const long long r = t / per_row, c = (t - r * per_row) << 3;
        const __half* p = a.src[w] + r * a.ld[w] + c;
        __align__(16) __half v[8];
#pragma unroll
        for (int j = 0; j < 8; j++) v[j] = c + j < a.cols[w] ? p[j] : __float2half_rn(0.0f);
        *reinterpret_cast<uint4*>(a.dst[w] + r * a.ldp[w] + c) = *reinterpret_cast<const uint4*>(v);
    }
}

// ── f32 contractions on the tensor cores: 3 x TF32 ────────────────────────────────────────────
// hi = the operand rounded to TF32 (11 significant bits, round to nearest, ties away), lo = operand - hi
// (exact in f32), itself rounded to TF32.
__global__ void __launch_bounds__(256) split_tf32(const float* __restrict__ src, long long ld, long long rows, long long cols, long long ldo,
                                                  float* __restrict__ hi, float* __restrict__ lo) {
    enter_kernel();
    const long long per_row = ldo >> 2;
    const long long total = rows * per_row;
    for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
        const long long r = t / per_row, c = (t - r * per_row) << 2;
        float v[4], h[4], l[4];
        const float* p = src + r * ld + c;
        if (c + 3 < cols && (reinterpret_cast<uintptr_t>(p) & 15) == 0) {
            const float4 q = *reinterpret_cast<const float4*>(p);
            v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = (c + j < cols) ? p[j] : 0.0f;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            unsigned u, w;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(v[j]));
            h[j] = __uint_as_float(u);
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(w) : "f"(v[j] - h[j]));     // the tensor core would cut it; rounding halves that error
            l[j] = __uint_as_float(w);
        }
        *reinterpret_cast<float4*>(hi + r * ldo + c) = make_float4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<float4*>(lo + r * ldo + c) = make_float4(l[0], l[1], l[2], l[3]);
    }
}

// The same split for an operand stored with its row index contiguous (element (r, k) at src[k * ld + r]):
// written out k-contiguous through a 32 x 32 shared-memory tile, so the tensor-core kernel sees one
// operand layout.  Block (32, 8); grid (ceil(k / 32), ceil(rows / 32)), rows folded into y then z.
__global__ void __launch_bounds__(256) split_tf32_transposed(const float* __restrict__ src, long long ld, long long rows, long long cols, long long ldo,
                                                             float* __restrict__ hi, float* __restrict__ lo) {
    enter_kernel();
    __shared__ float tile[32][33];
    const long long k0 = (long long)blockIdx.x * 32;
    const long long r0 = ((long long)blockIdx.z * gridDim.y + blockIdx.y) * 32;
    if (r0 >= rows) return;
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        const long long k = k0 + threadIdx.y + j, r = r0 + threadIdx.x;
        tile[threadIdx.y + j][threadIdx.x] = (k < cols && r < rows) ? src[k * ld + r] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 32; j += 8) {
        const long long r = r0 + threadIdx.y + j, k = k0 + threadIdx.x;
        if (r < rows && k < ldo) {
            const float v = tile[threadIdx.x][threadIdx.y + j];
            unsigned u, w;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(v));
            const float h = __uint_as_float(u);
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(w) : "f"(v - h));
            hi[r * ldo + k] = h;
            lo[r * ldo + k] = __uint_as_float(w);
        }
    }
}

// out[i] = copies[0][i] + copies[1][i] + ... in that order: finishes a contraction whose K was split
// between draws of the same tile.
__global__ void __launch_bounds__(256) sum_split_copies(const float* __restrict__ copies, long long stride, int n_copies, long long n, float* __restrict__ out) {
    enter_kernel();
    const long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (i >= n) return;
    if (i + 3 < n && (stride & 3) == 0) {
        float4 v = *reinterpret_cast<const float4*>(copies + i);
        for (int c = 1; c < n_copies; c++) {
            const float4 w = *reinterpret_cast<const float4*>(copies + c * stride + i);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
        *reinterpret_cast<float4*>(out + i) = v;
    } else {
        for (long long j = i; j < n && j < i + 4; j++) {
            float v = copies[j];
            for (int c = 1; c < n_copies; c++) v += copies[c * stride + j];
            out[j] = v;
        }
    }
}

// f32 contractions of more than a few rows take the two-CTA tensor-core kernel in 3 x TF32 form unless
// the device was opened with ANL_OPEN_NO_TF32X3: operands contiguous along k or along their row index.
static bool tf32x3_shape_ok(const Contraction& c, int64_t M, int64_t K) { return gemm_tf32_shape_ok(M, c.N, K, c.a_sm, c.a_sk, c.b_sn, c.b_sk); }
static bool tf32x3_applies(anl_device* dev, const Contraction& c, int64_t M, int64_t K) {
    return !(dev->flags & ANL_OPEN_NO_TF32X3) && tf32x3_shape_ok(c, M, K);
}
static PairVariant tf32_variant() {
    PairVariant v{};
    v.a_mn = v.b_mn = false;        // the split pre-pass hands both operands over k-contiguous
    v.bnt = 256; v.tf32 = true; v.split_tail = false;
    v.stages = 3;                   // 64 KB each: hi and lo parts of both operands
    v.group_m = kDefaultGroupM;
    return v;
}
bool gemm_tf32_eligible(const Plan& plan) {
    if (!plan.gemm || plan.gemm_dynamic || plan.r.klass != KC_GEMM || !plan.gemm->f32) return false;
    return tf32x3_shape_ok(plan.gemm->c, plan.gemm->c.M, plan.gemm->c.K);
}
int gemm_tf32_source(const Plan& plan, std::string& out, std::string& note) {
    if (!gemm_tf32_eligible(plan)) return ANL_ERR_UNSUPPORTED;
    const PairVariant v = tf32_variant();
    out = pair_source(v, std::string());
    const Contraction& c = plan.gemm->c;
    note = std::string("gemm tcgen05 3xTF32 A:") + (c.a_sk == 1 ? "K" : "MN") + " B:" + (c.b_sk == 1 ? "K" : "MN") + " (both rewritten k-contiguous by the split pre-pass) M=" + std::to_string(c.M) + " N=" + std::to_string(c.N) + " K=" + std::to_string(c.K);
    return ANL_OK;
}

// The one-CTA kernel for f32 contractions with few tiles.  Measured against the pair kernel (and the launch that adds its
// copies up), us with the operand splits and the events: 256 x 4096 x 1024 29.7 / 35.8, 64 x 4096 x 1024 25.6 / 31.7,
// 100 x 1000 x 700 17.4 / 29.7, 600-cubed 19.5 / 29.7, 1024-cubed 27.6 / 34.8, 512 x 4096 x 1024 39.9 / 46.1, 2048 x 1024 x 1024
// 37.9 / 46.1 (32 tiles), 1024 x 1024 x 2048 42.0 / 46.0, 300 x 1024 x 4096 44.0 / 44.0; the other way 256 x 1024 x 4096 39.9 / 37.9
// and 40 x 1024 x 4096 35.8 / 31.7 (the pair kernel has 16 slices where a cluster has 4), 1024 x 4096 x 1024 (64 tiles) and
// 1024 x 1024 x 8192 198 / 126.  Its error is no larger there: chunks of 256 terms, where the pair kernel takes 256 to 1024.
static bool tf32_small_takes(int64_t M, int64_t N, int64_t K) {
    const int64_t tiles = ((M + 255) / 256) * ((N + 255) / 256);
    return tiles <= 36 && K <= 4096;
}

static int launch_gemm_tf32x3(anl_device* dev, const GemmPlan& gp, const float* a, const float* b, float* d, int64_t M, int64_t K,
                              cudaStream_t stream, std::vector<void*>* keep_scratch) {
    const Contraction& c = gp.c;
    const int64_t N = c.N;
    if (int rc = ensure_gemm_state(dev)) return rc;
    if (*dev->gemm_status_host != 0) return dev->fail(ANL_ERR_CUDA, "gemm: an earlier launch timed out on a barrier (code " + std::to_string(*dev->gemm_status_host) + ")");
    // both operands are rewritten as [rows, K] with k contiguous (rows = m or n), K padded to 4 floats
    const bool a_mn = !(c.a_sk == 1), b_mn = !(c.b_sk == 1);
    const int64_t ldo = (K + 3) & ~3ll;
    void* scratch[4] = {nullptr, nullptr, nullptr, nullptr};
    const size_t a_bytes = (size_t)M * ldo * 4, b_bytes = (size_t)N * ldo * 4;
    int rc = ANL_OK;
    for (int k = 0; k < 4 && rc == ANL_OK; k++) rc = dev->alloc(k < 2 ? a_bytes : b_bytes, &scratch[k]);
    auto done = [&](int code) {
        for (void* p : scratch) if (p) { if (keep_scratch) keep_scratch->push_back(p); else dev->release(p); }
        return code;
    };
    if (rc) return done(rc);
    float *a_hi = (float*)scratch[0], *a_lo = (float*)scratch[1], *b_hi = (float*)scratch[2], *b_lo = (float*)scratch[3];
    const int sms = dev->prop.multiProcessorCount;
    auto split = [&](const float* src, bool mn, int64_t rows, int64_t ld, float* hi, float* lo) {
        if (!mn) {
            const unsigned grid = (unsigned)std::max<int64_t>(1, std::min<int64_t>((rows * (ldo / 4) + 255) / 256, (int64_t)sms * 16));
            return launch_static(dev, split_tf32, dim3(grid), dim3(256), stream, 1, src, ld, rows, K, ldo, hi, lo);
        } else {
            const int64_t rt = (rows + 31) / 32;
            const unsigned gy = (unsigned)std::min<int64_t>(rt, 32768), gz = (unsigned)((rt + gy - 1) / gy);
            return launch_static(dev, split_tf32_transposed, dim3((unsigned)((ldo + 31) / 32), gy, gz), dim3(32, 8), stream, 1, src, ld, rows, K, ldo, hi, lo);
        }
    };
    if (split(a, a_mn, M, a_mn ? c.a_sk : c.a_sm, a_hi, a_lo) != cudaSuccess || split(b, b_mn, N, b_mn ? c.b_sk : c.b_sn, b_hi, b_lo) != cudaSuccess) return done(dev->fail(ANL_ERR_CUDA, "gemm: operand split launch failed"));
    dev->stats.kernels_launched += 2;

    constexpr int BK32 = 32;
    CUtensorMap ma_hi, ma_lo, mb_hi, mb_lo;
    CUfunction fn;
    if (tf32_small_takes(M, N, K)) {
        const SmallVariant v = choose_small(M, N, K, false, false, true);
        if ((rc = encode_map(dev, &ma_hi, a_hi, (uint64_t)K, (uint64_t)M, (uint64_t)ldo, BK32, v.prows, true)) || (rc = encode_map(dev, &ma_lo, a_lo, (uint64_t)K, (uint64_t)M, (uint64_t)ldo, BK32, v.prows, true)) ||
            (rc = encode_map(dev, &mb_hi, b_hi, (uint64_t)K, (uint64_t)N, (uint64_t)ldo, BK32, v.nt, true)) || (rc = encode_map(dev, &mb_lo, b_lo, (uint64_t)K, (uint64_t)N, (uint64_t)ldo, BK32, v.nt, true))) return done(rc);
        if ((rc = get_small_kernel(dev, v, std::string(), &fn))) return done(rc);
        SmallGemmArgs g{};
        g.d_raw = d;
        g.M = (int)M; g.N = (int)N; g.K = (int)K;
        g.tiles_m = (int)((M + BM - 1) / BM);
        g.status = dev->gemm_status_dev;
        const int64_t ctas = (int64_t)g.tiles_m * ((N + v.nt - 1) / v.nt) * v.splits;
        void* params[5] = {&ma_hi, &mb_hi, &ma_lo, &mb_lo, &g};
        if ((rc = launch_kernel(dev, fn, KernelShape{(unsigned)ctas, 1, 1, (unsigned)v.threads(), 1, 1, (unsigned)small_smem_bytes(v), (unsigned)v.splits}, stream, params, true, "gemm_f16_tcgen05_small (f32)"))) return done(rc);
        dev->stats.gemm_launched++;
        return done(ANL_OK);
    }
    const PairVariant v = tf32_variant();
    if ((rc = get_pair_kernel(dev, v, std::string(), &fn))) return done(rc);
    auto enc_a = [&](CUtensorMap* m, const float* base) { return encode_map(dev, m, base, (uint64_t)K, (uint64_t)M, (uint64_t)ldo, BK32, BM, true); };
    auto enc_b = [&](CUtensorMap* m, const float* base) { return encode_map(dev, m, base, (uint64_t)K, (uint64_t)N, (uint64_t)ldo, BK32, v.bnt / 2, true); };
    if ((rc = enc_a(&ma_hi, a_hi)) || (rc = enc_a(&ma_lo, a_lo)) || (rc = enc_b(&mb_hi, b_hi)) || (rc = enc_b(&mb_lo, b_lo))) return done(rc);
    PairGemmArgsF32 g{};
    g.d_raw = d;
    g.M = (int)M; g.N = (int)N; g.ldd = (int)N;
    g.tiles_m = (int)((M + 2 * BM - 1) / (2 * BM)); g.tiles_n = (int)((N + v.bnt - 1) / v.bnt);
    g.full_tiles = g.tiles_m * g.tiles_n;
    g.status = dev->gemm_status_dev;
    g.tile_counter = tile_counter_for(dev, stream);
    const int npairs = gemm_sm_budget(dev) / 2;
    const int pairs = std::min(g.full_tiles, npairs);
    KernelShape shape{2u * pairs, 1, 1, PAIR_THREADS, 1, 1, (unsigned)pair_smem_bytes(v.bnt, v.stages, v.tf32), 2};
    g.K = (int)K;
    g.chunk_kb = kTf32ChunkK / BK32;
    // few tiles and a long K: draw every tile several times, each draw a slice of K into its own copy
    // of the output (at least 8 k-blocks a slice), and add the copies afterwards in order
    const int kblocks = (int)((K + BK32 - 1) / BK32);
    int splits = std::min(npairs / std::max(1, g.full_tiles), kblocks / 8);
    void* copies = nullptr;
    if (splits > 1) {
        g.kb_per_split = (kblocks + splits - 1) / splits;
        splits = (kblocks + g.kb_per_split - 1) / g.kb_per_split;
    }
    if (splits > 1) {
        g.k_splits = splits;
        g.split_stride = (long long)(((M * N) + 3) & ~3ll);
        if ((rc = dev->alloc((size_t)splits * (size_t)g.split_stride * 4, &copies))) return done(rc);
        g.d_raw = copies;
        shape.gx = 2 * std::min(g.full_tiles * splits, npairs);
    }
    auto done2 = [&](int code) {
        if (copies) { if (keep_scratch) keep_scratch->push_back(copies); else dev->release(copies); }
        return done(code);
    };
    g.draw_late = g.full_tiles * std::max(1, g.k_splits) <= 2 * npairs;
    void* params[5] = {&ma_hi, &mb_hi, &ma_lo, &mb_lo, &g};
    if ((rc = launch_kernel(dev, fn, shape, stream, params, true, "gemm_f16_tcgen05_pair (f32)"))) return done2(rc);
    if (splits > 1) {
        const long long n = (long long)M * N;
        if (launch_static(dev, sum_split_copies, dim3((unsigned)((n + 1023) / 1024)), dim3(256), stream, 1, (const float*)copies, g.split_stride, splits, n, d) != cudaSuccess) return done2(dev->fail(ANL_ERR_CUDA, "gemm: split sum launch failed"));
        dev->stats.kernels_launched++;
    }
    dev->stats.gemm_launched++;
    return done2(ANL_OK);
}

int launch_gemm(anl_device* dev, const Plan& plan, void* const* bufs, int64_t sym_value, cudaStream_t stream, int64_t m_begin, int64_t m_end,
                const GemmFusion* fusion, std::vector<void*>* keep_scratch, bool b_settled, HeldGemm** hold) {
    const GemmPlan& gp = *plan.gemm;
    const Contraction& c = gp.c;
    // an optional row window [m_begin, m_end) of the output: the caller splits a contraction so that
    // a collective on the first rows can start while the remaining rows are still being computed
    const bool window = m_end >= 0;
    if (window && (gp.f32 || c.m_sym || m_begin < 0 || m_end > c.M || m_begin >= m_end || (m_begin % 8)))
        return dev->fail(ANL_ERR_INVALID, "gemm: bad row window");
    if (fusion && (window || gp.f32)) return dev->fail(ANL_ERR_INVALID, "gemm: a fused consumer needs the whole f16 contraction");
    const int64_t M = window ? m_end - m_begin : c.M;
    if (gp.f32) {
        const int64_t Mv = c.m_sym ? sym_value : c.M, Kv = c.k_sym ? sym_value : c.K;
        if (tf32x3_applies(dev, c, Mv, Kv))
            return launch_gemm_tf32x3(dev, gp, (const float*)bufs[c.a_param] + c.a_off, (const float*)bufs[c.b_param] + c.b_off, (float*)bufs[0], Mv, Kv, stream, keep_scratch);
        return launch_gemm_f32(dev, (const float*)bufs[c.a_param] + c.a_off, (const float*)bufs[c.b_param] + c.b_off, (float*)bufs[0],
                               Mv, c.N, Kv, c.a_sm, c.a_sk, c.b_sn, c.b_sk, stream);
    }
    if (int rc = ensure_gemm_state(dev)) return rc;
    if (*dev->gemm_status_host != 0) return dev->fail(ANL_ERR_CUDA, "gemm: an earlier launch timed out on a barrier (code " + std::to_string(*dev->gemm_status_host) + ")");
    const __half* a = (const __half*)bufs[c.a_param] + c.a_off + (window ? m_begin * c.a_sm : 0);
    const __half* b = (const __half*)bufs[c.b_param] + c.b_off;
    int64_t lda = gp.lda, ldb = gp.ldb;
    int rc = ANL_OK;
    void* padded[2] = {nullptr, nullptr};
    auto done = [&](int code) {
        for (void* p : padded) if (p) { if (keep_scratch) keep_scratch->push_back(p); else dev->release(p); }
        return code;
    };
    if (gp.pad_a || gp.pad_b) {
        PadArgs pa{};
        int n = 0;
        auto add = [&](const __half*& src, int64_t& ld, int64_t rows, int64_t cols) -> int {
            const int64_t ldp = (cols + 7) & ~7ll;
            if (int r = dev->alloc((size_t)rows * ldp * 2, &padded[n])) return r;
            pa.src[n] = src; pa.dst[n] = (__half*)padded[n]; pa.rows[n] = rows; pa.cols[n] = cols; pa.ld[n] = ld; pa.ldp[n] = ldp;
            src = (const __half*)padded[n]; ld = ldp;
            n++;
            return ANL_OK;
        };
        if (gp.pad_a && (rc = gp.a_mn ? add(a, lda, c.K, M) : add(a, lda, M, c.K))) return done(rc);
        if (gp.pad_b && (rc = gp.b_mn ? add(b, ldb, c.K, c.N) : add(b, ldb, c.N, c.K))) return done(rc);
        long long most = 0;
        for (int k = 0; k < n; k++) most = std::max(most, pa.rows[k] * (pa.ldp[k] >> 3));
        if (launch_static(dev, pad_rows_f16, dim3((unsigned)std::min<long long>((most + 255) / 256, dev->prop.multiProcessorCount * 16), (unsigned)n), dim3(256), stream, 1, pa) != cudaSuccess) return done(dev->fail(ANL_ERR_CUDA, "gemm: operand copy launch failed"));
        dev->stats.kernels_launched++;
    }
    CUtensorMap ma, mb;
    if (small_takes(gp, M)) {
        const SmallVariant v = choose_small(gp, M);
        if (gp.a_mn) rc = encode_map(dev, &ma, a, (uint64_t)M, (uint64_t)c.K, (uint64_t)lda, 64, BK);
        else rc = encode_map(dev, &ma, a, (uint64_t)c.K, (uint64_t)M, (uint64_t)lda, BK, v.prows);
        if (rc) return done(rc);
        if (gp.b_mn) rc = encode_map(dev, &mb, b, (uint64_t)c.N, (uint64_t)c.K, (uint64_t)ldb, 64, BK);
        else rc = encode_map(dev, &mb, b, (uint64_t)c.K, (uint64_t)c.N, (uint64_t)ldb, BK, v.nt);
        if (rc) return done(rc);
        SmallGemmArgs g{};
        __half* out0 = (__half*)bufs[0] + (window ? m_begin * c.N : 0);
        g.d_raw = (!fusion || fusion->store_raw) ? out0 : nullptr;
        g.d_out = fusion ? fusion->d_out : nullptr;
        g.colsum = fusion ? fusion->colsum : nullptr;
        if (fusion) for (int k = 0; k < 6; k++) g.ep[k] = fusion->ep[k];
        g.M = (int)M; g.N = (int)c.N; g.K = (int)c.K;
        g.tiles_m = (int)((M + BM - 1) / BM);
        g.status = dev->gemm_status_dev;
        const int64_t ctas = (int64_t)g.tiles_m * ((c.N + v.nt - 1) / v.nt) * v.splits;
        if (ctas > 0x7fffffffLL) return done(dev->fail(ANL_ERR_LIMIT, "gemm: grid too large"));
        g.b_settled = b_settled && !gp.pad_b;
        HeldGemm h{v, fusion && fusion->epilogue ? *fusion->epilogue : std::string(), ma, mb, g, ctas};
        if (hold && !window && !gp.pad_a && !gp.pad_b) { *hold = new HeldGemm(std::move(h)); return ANL_OK; }
        if ((rc = launch_held(dev, h, nullptr, stream))) return done(rc);
        return done(ANL_OK);
    }
    if (gp.a_mn) rc = encode_map(dev, &ma, a, (uint64_t)M, (uint64_t)c.K, (uint64_t)lda, 64, BK);
    else rc = encode_map(dev, &ma, a, (uint64_t)c.K, (uint64_t)M, (uint64_t)lda, BK, BM);
    if (rc) return done(rc);
    int* const counter = tile_counter_for(dev, stream);
    const PairVariant v = choose_variant(dev, gp, M);
    // B is loaded in halves of bnt/2 columns, so its tensor map gets a box of that many rows; a
    // second map with half that box serves the half-width tiles of the last wave
    CUtensorMap mbh;
    if (gp.b_mn) rc = encode_map(dev, &mb, b, (uint64_t)c.N, (uint64_t)c.K, (uint64_t)ldb, 64, BK);
    else rc = encode_map(dev, &mb, b, (uint64_t)c.K, (uint64_t)c.N, (uint64_t)ldb, BK, v.bnt / 2);
    if (rc) return done(rc);
    if (gp.b_mn) mbh = mb;
    else if ((rc = encode_map(dev, &mbh, b, (uint64_t)c.K, (uint64_t)c.N, (uint64_t)ldb, BK, v.bnt / 4))) return done(rc);
    CUfunction fn;
    if ((rc = get_pair_kernel(dev, v, fusion && fusion->epilogue ? *fusion->epilogue : std::string(), &fn))) return done(rc);
    PairGemmArgs g{};
    __half* out0 = (__half*)bufs[0] + (window ? m_begin * c.N : 0);
    g.d_raw = (!fusion || fusion->store_raw) ? out0 : nullptr;
    g.d_out = fusion ? fusion->d_out : nullptr;
    g.colsum = fusion ? fusion->colsum : nullptr;
    if (fusion) for (int k = 0; k < 6; k++) g.ep[k] = fusion->ep[k];
    g.M = (int)M; g.N = (int)c.N; g.K = (int)c.K; g.ldd = (int)c.N;
    g.tiles_m = (int)((M + 2 * BM - 1) / (2 * BM)); g.tiles_n = (int)((c.N + v.bnt - 1) / v.bnt);
    g.status = dev->gemm_status_dev;
    g.tile_counter = counter;
    const int npairs = gemm_sm_budget(dev) / 2;
    // Last wave: when the tiles left over after the full waves would occupy at most half of the
    // pairs, they are drawn as half-width tiles and the wave costs half a tile instead of a whole one.
    const int whole = g.tiles_m * g.tiles_n;
    const int rest = whole % npairs;
    g.full_tiles = (v.split_tail && v.bnt == 256 && whole > npairs && rest > 0 && 2 * rest <= npairs) ? whole - rest : whole;
    const int pairs = std::min(whole + (whole - g.full_tiles), npairs);
    g.draw_late = (whole + (whole - g.full_tiles)) <= 2 * pairs;
    void* params[4] = {&ma, &mb, &mbh, &g};
    if ((rc = launch_kernel(dev, fn, KernelShape{2u * pairs, 1, 1, PAIR_THREADS, 1, 1, (unsigned)pair_smem_bytes(v.bnt, v.stages, v.tf32), 2}, stream, params, true, "gemm_f16_tcgen05_pair"))) return done(rc);
    dev->stats.gemm_launched++;
    return done(ANL_OK);
}

// Finishes a bias gradient whose per-32-row partial column sums a contraction's epilogue left in
// `partials` [parts, N]: summed in f32 in a fixed order, one narrowing to f16 — the arithmetic of the REDUCE
// the schedule holds for it (f32 accumulator, narrowed once), with the rows grouped.
__global__ void __launch_bounds__(256) colsum_finish(const float* __restrict__ partials, int parts, int n, __half* __restrict__ out) {
    // A warp owns 8 columns (a sector), its four groups of lanes a contiguous quarter of the parts each (ascending, eight loads in
    // flight), and the four sums are added in order.  No shared memory: beside a two-CTA contraction, which leaves
    // 1.5 KB of an SM's, these blocks find a place at once; with 1 KB of their own they ran before the next
    // contraction instead of beside it (step of 8192 rows, 4 x 4096 wide, at burst clocks 2746 -> 2726 us; at those of a long run
    // no more than two runs differ by).
    enter_kernel();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = lane >> 3;
    const int col = (blockIdx.x * 8 + warp) * 8 + (lane & 7);
    const int per = (parts + 3) / 4, p0 = group * per, p1 = (p0 + per) < parts ? (p0 + per) : parts;
    float acc = 0.0f;
    if (col < n) {
        int p = p0;
        for (; p + 8 <= p1; p += 8) {
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = partials[(size_t)(p + u) * n + col];
#pragma unroll
            for (int u = 0; u < 8; u++) acc = acc + v[u];
        }
        for (; p < p1; p++) acc = acc + partials[(size_t)p * n + col];
    }
    float v = __shfl_sync(0xffffffffu, acc, lane & 7);
#pragma unroll
    for (int q = 1; q < 4; q++) v = v + __shfl_sync(0xffffffffu, acc, q * 8 + (lane & 7));
    if (group == 0 && col < n) out[col] = __float2half_rn(v);
}

int launch_colsum_finish(anl_device* dev, const float* partials, int64_t parts, int64_t n, void* out, cudaStream_t stream) {
    cudaError_t e = launch_static(dev, colsum_finish, dim3((unsigned)((n + 63) / 64)), dim3(256), stream, 1, partials, (int)parts, (int)n, (__half*)out);
    if (e != cudaSuccess) return dev->fail(ANL_ERR_CUDA, std::string("gemm: column-sum finish: ") + cudaGetErrorString(e));
    dev->stats.kernels_launched++;
    return ANL_OK;
}

}  // namespace anl
