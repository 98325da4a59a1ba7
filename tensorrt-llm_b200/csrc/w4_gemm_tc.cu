// Prefill-regime kernel: weight-only GEMM on the 5th-generation tensor cores (tcgen05 + TMEM).
//
// Replaces CutlassFpAIntBGemmRunner::gemm of the reference project
// (cpp/tensorrt_llm/kernels/cutlass_kernels/fpA_intB_gemm/fpA_intB_gemm_template.h:394-465), which
// on compute capability 10.x runs an Ampere mma.sync kernel. Same math as that kernel: every
// weight is dequantised to T as round_T(fma(q, scale, zero))
// (cpp/tensorrt_llm/cutlass_extensions/include/cutlass_extensions/gemm/warp/mma_tensorop_dequantizer.h:247-262),
// products are accumulated in fp32, alpha and bias are applied in the epilogue.
//
// Orientation. The output tile is computed transposed: D[n, m] = sum_k W[n, k] * A[m, k]. The
// dequantised weights are the MMA's "A" operand and live in tensor memory (one TMEM lane per
// output column n), written there straight from registers by the conversion warps, so they never
// travel through shared memory; the activations are the "B" operand, brought by TMA into
// 128-byte-swizzled shared memory and consumed by the MMA unmodified.
//
// A CTA pair (cluster of two, cta_group::2) owns a tile of 256 weight columns x BM activation rows,
// BM a multiple of 32 up to 256 chosen per problem: each CTA converts its own 128 columns and holds
// half of the activation rows, which the pair's MMAs read from both shared memories. That halves the
// activation bytes a CTA has to pull out of L2 (at 256 rows 20 KB of operands per 64 k and 512
// tensor cycles instead of 36 KB, which alone would exceed what L2 delivers to all SMs) and leaves
// room for deep rings.
//
// Warp roles (one CTA pair per two SMs, persistent over tiles, n-fastest tile order):
//   warps 0..3            epilogue: tcgen05.ld, alpha/bias, convert, store; the accumulator is double
//                         buffered up to 128 rows
//   warps 4..4+4G-1       conversion, G groups of four warps (one per TMEM lane quadrant) that take
//                         alternate steps: shared memory -> registers -> exact int->T
//                         conversion, scale/zero -> tcgen05.st into the TMEM ring
//   next                  weight producer: packed weights and their scale/zero rows, one TMA box each
//                         per step, a ring of its own that runs far ahead (its latency is
//                         HBM's) and, with static weights, ahead of the preceding kernel
//   next                  activation producer: two boxes of 64 k x BM/2 rows per step
//   last                  MMA issuer (first CTA of the pair) and TMEM alloc/free (both)
// A step is 128 k (eight tcgen05.mma of K = 16). Hand-offs, all mbarriers: `w_full` / `w_empty` (weight
// ring, local), `full` (first CTA: both CTAs' halves of the step's activations landed and the eight
// conversion warps of both CTAs stored their part of the step's weights), `empty` (tcgen05.commit,
// multicast to both CTAs: the step's activation stage and TMEM stage are free), `d_full` /
// `d_empty` (accumulator).
// All waits are bounded; a timeout sets the device status word and the CTAs drain and exit.
#include <atomic>
#include <mutex>
#include <type_traits>

#include "w4_common.cuh"
#include "w4_internal.h"
#include "w4_tma.h"

namespace w4
{
namespace tc
{

constexpr int BN = 128;            // weight columns per CTA (TMEM lanes)
constexpr int kPairN = 2 * BN;     // weight columns per CTA pair
constexpr int kMaxBM = 256;        // activation rows per tile at most
constexpr int kTmemCols = 512;
constexpr int kStageCols = 64;     // TMEM columns of one converted 128-k stage
constexpr int kConvGroups = 3;
constexpr int kEpiWarps = 4;
constexpr int kConvWarp0 = kEpiWarps;
constexpr int kWProdWarp = kConvWarp0 + 4 * kConvGroups;
constexpr int kActWarp = kWProdWarp + 1;
constexpr int kMmaWarp = kWProdWarp + 2;
constexpr int kThreads = 32 * (kWProdWarp + 4);
constexpr int kMaxStages = 8;      // activation / TMEM ring
constexpr int kMaxWStages = 12;    // weight ring
constexpr int kMaxExperts = 32;    // experts of one launch

struct Args
{
    void const* bias;
    void* out;
    float alpha;
    int m, n, k;
    int group_shift; // log2(group size), 31 = per-channel
    int bm;          // activation rows per tile
    int tiles_n;
    // Experts (an ordinary GEMM is one): expert e has rows first_row[e] .. first_row[e + 1] - 1 of the
    // activations and of the output, tiles first_tile[e] .. first_tile[e + 1] - 1, the weights, scales and zeros
    // of slice slice[e] of their tensors, and bias + slice[e] * n.
    int num_experts;
    int groups; // scale rows per expert
    int first_row[kMaxExperts + 1], first_tile[kMaxExperts + 1], slice[kMaxExperts];
    int num_stages, num_wstages;
    int d_bufs;      // accumulators in TMEM: 2 up to 128 rows, else 1
    int weights_static;
    // Split-k: an output tile's k range is cut into `splits` work items that run on different CTA pairs.
    int splits;       // 1 = off
    int steps_split;  // 128-wide k steps per work item
    float* partial;   // [splits, m, n] fp32 (SPLIT_WORKSPACE)
};

// Where the fp32 partial tiles of a split tile meet. CLUSTER: the splits' CTA pairs form one cluster of
// 2 * splits CTAs, every CTA leaves its partial tile in its own shared memory and adds a share of the rows
// over all of them through distributed shared memory. WORKSPACE: partial tiles in the caller's workspace,
// added by a second kernel; for more splits than a cluster can hold, and where the device cannot
// co-schedule such clusters. Both add in split order (deterministic).
enum SplitMode
{
    SPLIT_NONE,
    SPLIT_CLUSTER,
    SPLIT_WORKSPACE
};
constexpr int kMaxClusterSplits = 8; // clusters of 16 CTAs

struct __align__(16) Barriers
{
    uint64_t full[kMaxStages];    // first CTA: activations of both CTAs landed, 8 conversion warps stored
    uint64_t empty[kMaxStages];   // the MMAs of the step completed: activation stage and TMEM stage are free
    // Weights of a step landed, one barrier per (conversion group, stage): copies land out of order, and a
    // group that met only some of a stage's phases could take the parity of an older phase for its own.
    // (The `empty` phases come from commits, which complete in order.)
    uint64_t w_full[kConvGroups][kMaxWStages];
    uint64_t w_empty[kMaxWStages];
    uint64_t d_full[2];           // accumulator complete
    uint64_t d_empty[2];          // first CTA: the epilogue warps of both CTAs drained the accumulator
    uint32_t tmem_base;
    int abort_flag;
};

// Bounded wait on an mbarrier phase, executed by a converged warp (every lane polls the same word).
// CLUSTER: the phase was completed by the other CTA's arrivals as well.
template <bool CLUSTER>
__device__ __forceinline__ bool mbar_poll(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    if (CLUSTER)
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    return __all_sync(0xffffffffu, ok) != 0; // warp-uniform: the code behind a wait is executed converged
}

template <bool CLUSTER>
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile int* abort_flag)
{
    for (uint32_t polls = 1; !mbar_poll<CLUSTER>(bar, parity); ++polls)
    {
        if ((polls & 1023u) == 0 && (*abort_flag || polls >= kMaxWaitPolls))
        {
            *abort_flag = 1;
            atomicExch(&g_device_status, kDeviceTimeout);
            return false;
        }
    }
    return true;
}

// Address of this CTA's shared variable in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, uint32_t rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// The following are executed by a whole (converged) warp; one elected lane performs the operation.
// Keeping the surrounding control flow warp-uniform lets the compiler hold addresses and
// descriptors in uniform registers, which is what the tensor-core and TMA instructions consume;
// issued from inside a divergent `if (lane == 0)` every operand has to be moved across first.
__device__ __forceinline__ void tc_mma4_ts_elect(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc)
{
    // the four K = 16 instructions of 64 k: one election for all
    asm volatile(
        "{\n"
        ".reg .pred p, pt, pe;\n"
        "elect.sync _|pe, 0xffffffff;\n"
        "setp.ne.b32 p, %10, 0;\n"
        "setp.eq.b32 pt, 0, 0;\n"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %5, %9, p;\n"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [%2], %6, %9, pt;\n"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [%3], %7, %9, pt;\n"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [%4], %8, %9, pt;\n"
        "}\n" ::"r"(d_tmem),
        "r"(a_tmem), "r"(a_tmem + 8), "r"(a_tmem + 16), "r"(a_tmem + 24), "l"(b_desc), "l"(b_desc + 2), "l"(b_desc + 4),
        "l"(b_desc + 6), "r"(idesc), "r"(acc)
        : "memory");
}

// Arrives on the barrier at this offset in both CTAs of the pair (`mask`: their ranks in the cluster) once
// all MMAs issued so far have completed.
__device__ __forceinline__ void tc_commit_pair_elect(uint32_t bar_addr, uint16_t mask)
{
    asm volatile(
        "{\n"
        ".reg .pred pe;\n"
        "elect.sync _|pe, 0xffffffff;\n"
        "@pe tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
        "}\n" ::"r"(bar_addr),
        "h"(mask)
        : "memory");
}

// 2-D tile load of this CTA's half of an activation step; completion is counted on `bar_addr`, which
// is the first CTA's barrier for both.
__device__ __forceinline__ void elect_tma_load_2d_pair(uint32_t dst, void const* tensor_map, int c0, int c1, uint32_t bar_addr)
{
    asm volatile(
        "{\n"
        ".reg .pred pe;\n"
        "elect.sync _|pe, 0xffffffff;\n"
        "@pe cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
        "}\n" ::"r"(dst),
        "l"(tensor_map), "r"(c0), "r"(c1), "r"(bar_addr)
        : "memory");
}

__device__ __forceinline__ void elect_tma_load_3d(uint32_t dst, void const* tensor_map, int c0, int c1, int c2, uint32_t bar_addr)
{
    asm volatile(
        "{\n"
        ".reg .pred pe;\n"
        "elect.sync _|pe, 0xffffffff;\n"
        "@pe cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
        "}\n" ::"r"(dst),
        "l"(tensor_map), "r"(c0), "r"(c1), "r"(c2), "r"(bar_addr)
        : "memory");
}

__device__ __forceinline__ void arrive_local(uint32_t bar_addr)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_addr) : "memory");
}

// Publishes tensor-memory accesses (ordered by tcgen05.wait and tcgen05.fence::before_thread_sync in
// front of it) to the first CTA's MMA warp. Relaxed: with release semantics every arrival waits for a
// cluster-scope fence, about half a microsecond that the conversion warp spends idle (the kernel took
// 0.33 us per 64 k instead of 0.17).
__device__ __forceinline__ void arrive_cluster_relaxed(uint32_t addr)
{
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

__device__ __forceinline__ void tc_st32(uint32_t taddr, uint32_t const (&v)[32])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&v)[32])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,"
        "%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
        "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
        "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor of a K-major, 128-byte-swizzled tile of T whose rows are 128
// bytes (64 elements) wide: 8-row groups are 1024 bytes apart, descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr)
{
    uint64_t d = uint64_t((smem_addr & 0x3ffffu) >> 4);
    d |= uint64_t(1024 >> 4) << 32; // stride between 8-row groups
    d |= uint64_t(1) << 46;         // version
    d |= uint64_t(2) << 61;         // SWIZZLE_128B
    return d;
}


template <typename T, int BITS, bool HAS_ZERO, int SPLIT>
__global__ void __launch_bounds__(kThreads, 1)
    gemm_kernel(Args const a, __grid_constant__ CUtensorMap const tm_act, __grid_constant__ CUtensorMap const tm_w,
        __grid_constant__ CUtensorMap const tm_s, __grid_constant__ CUtensorMap const tm_z)
{
    using P = Pair<T>;
    constexpr int IL = BITS == 4 ? 4 : 2;
    constexpr int SEG_CHUNKS = 8 / IL;               // 16-byte chunks of one column inside a 128-byte line (64 k)
    constexpr int LINE_TILE = (BN / IL) * 128;       // this CTA's interleaved rows x one line
    constexpr int W_BYTES = 2 * LINE_TILE;           // a step: two lines per row
    constexpr int W_STAGE = W_BYTES + 1024;          // + up to two rows of 128 scales, and of zeros
    constexpr uint32_t kFmt = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u; // 0 = fp16, 1 = bf16

    // The 128-byte swizzle of the TMA copies and of the MMA descriptors is a function of the
    // shared-memory address: the rings start on a 1024-byte boundary (declared, and checked below).
    extern __shared__ __align__(1024) uint8_t smem[];
    uint32_t const smem_base = smem_u32(smem);
    int const act_half = a.bm * 64;       // bm / 2 rows of 128 bytes: 64 k
    int const act_stage = 2 * act_half;
    uint32_t const w_ring = smem_base + uint32_t(a.num_stages) * act_stage;
    Barriers* bars = reinterpret_cast<Barriers*>(smem + size_t(a.num_stages) * act_stage + size_t(a.num_wstages) * W_STAGE);
    volatile int* abort_flag = &bars->abort_flag;

    int const warp = __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    uint32_t cta_rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(cta_rank));
    uint32_t const rank = cta_rank & 1u, lead_rank = cta_rank & ~1u; // in the pair; the pair's first CTA
    // Work items: (tile, split), splits adjacent. With SPLIT_CLUSTER a pair has exactly one: the grid is one
    // cluster per tile and a pair's rank in it is its split.
    int const pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
    int const num_items = a.first_tile[a.num_experts] * (SPLIT != SPLIT_NONE ? a.splits : 1);
    int const steps_all = (a.k + 127) >> 7; // the second half of the last step may lie past k: zeros, not multiplied

    bool const aligned = (smem_base & 1023u) == 0; // never false; the check keeps a wrong layout from being read
    if (threadIdx.x == 0)
    {
        for (int s = 0; s < a.num_stages; ++s)
        {
            mbar_init(&bars->full[s], 1 + 8); // expect_tx of the first CTA + four conversion warps of each CTA
            mbar_init(&bars->empty[s], 1);
        }
        for (int s = 0; s < a.num_wstages; ++s)
        {
            for (int g = 0; g < kConvGroups; ++g)
                mbar_init(&bars->w_full[g][s], 1);
            mbar_init(&bars->w_empty[s], 4);
        }
        for (int b = 0; b < 2; ++b)
        {
            mbar_init(&bars->d_full[b], 1);
            mbar_init(&bars->d_empty[b], 2 * kEpiWarps);
        }
        bars->abort_flag = aligned ? 0 : 1;
        if (!aligned)
            atomicExch(&g_device_status, kDeviceTimeout);
        mbar_fence_init();
    }
    if (warp == kMmaWarp)
    {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&bars->tmem_base)),
                     "r"(uint32_t(kTmemCols))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all(); // the barriers of both CTAs are initialised before either arrives on the other's
    tc_fence_after();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    uint32_t const tmem = bars->tmem_base;
    uint32_t const a_ring = tmem + uint32_t(a.d_bufs * a.bm); // TMEM ring of converted weights, behind the accumulators

    uint32_t const full0 = smem_u32(&bars->full[0]), empty0 = smem_u32(&bars->empty[0]);
    uint32_t const w_full0 = smem_u32(&bars->w_full[0][0]), w_empty0 = smem_u32(&bars->w_empty[0]);

    struct Item
    {
        int n0;             // first column of the pair's tile
        int row0, row_end;  // rows of the tile, and the end of the expert's
        int slice, split;
        int st0, st1;       // k steps
    };
    auto item_of = [&](int item)
    {
        Item it;
        int const tile = SPLIT != SPLIT_NONE ? item / a.splits : item;
        it.split = SPLIT != SPLIT_NONE ? item - tile * a.splits : 0;
        it.st0 = it.split * a.steps_split;
        it.st1 = SPLIT != SPLIT_NONE ? min(steps_all, it.st0 + a.steps_split) : steps_all;
        int e = 0;
        while (e + 1 < a.num_experts && tile >= a.first_tile[e + 1])
            ++e;
        int const t = tile - a.first_tile[e], tm = t / a.tiles_n;
        it.n0 = (t - tm * a.tiles_n) * kPairN;
        it.row0 = a.first_row[e] + tm * a.bm;
        it.row_end = a.first_row[e + 1];
        it.slice = a.slice[e];
        return it;
    };

    if (!aligned)
    {
        // nothing: fall through to the teardown
    }
    else if (warp == kWProdWarp)
    {
        // ------------------------------------------------------------------ weight producer
        if (lane == 0)
        {
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_w) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_s) : "memory");
            if (HAS_ZERO)
                asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_z) : "memory");
        }
        __syncwarp();
        // Weights that the preceding kernel may still be writing must not be fetched early.
        if (!a.weights_static)
            asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t const scale_bytes = a.group_shift == 6 ? 512u : 256u;
        uint32_t const tx = W_BYTES + scale_bytes * (HAS_ZERO ? 2 : 1);
        int s = 0, turn = 0; // turn: the group that converts the step
        uint32_t ph = 0;
        bool ok = true;
        for (int item = pair; item < num_items && ok; item += num_pairs)
        {
            Item const it = item_of(item);
            int const n0 = it.n0 + int(rank) * BN, w_row = it.slice * (a.n / IL) + n0 / IL, s_row = it.slice * a.groups;
            for (int st = it.st0; st < it.st1; ++st)
            {
                ok = wait_bar<false>(w_empty0 + 8 * s, ph ^ 1, abort_flag);
                if (!ok)
                    break;
                uint32_t const dst = w_ring + uint32_t(s) * W_STAGE, bar = w_full0 + 8 * (turn * kMaxWStages + s);
                int const g = s_row + (a.group_shift >= 31 ? 0 : (st << 7) >> a.group_shift);
                elect_expect_tx(bar, tx);
                elect_tma_load_3d(dst, &tm_w, 0, w_row, 2 * st, bar);
                elect_tma_load_2d(dst + W_BYTES, &tm_s, n0, g, bar);
                if (HAS_ZERO)
                    elect_tma_load_2d(dst + W_BYTES + 512, &tm_z, n0, g, bar);
                turn = turn + 1 == kConvGroups ? 0 : turn + 1;
                if (++s == a.num_wstages)
                {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    }
    else if (warp == kActWarp)
    {
        // ------------------------------------------------------------------ activation producer
        if (lane == 0)
            asm volatile("prefetch.tensormap [%0];" ::"l"(&tm_act) : "memory");
        __syncwarp();
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t const lead_full0 = cluster_addr(full0, lead_rank);
        int s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (int item = pair; item < num_items && ok; item += num_pairs)
        {
            Item const it = item_of(item);
            int const row0 = it.row0 + int(rank) * (a.bm >> 1);
            for (int st = it.st0; st < it.st1; ++st)
            {
                ok = wait_bar<false>(empty0 + 8 * s, ph ^ 1, abort_flag);
                if (!ok)
                    break;
                uint32_t const dst = smem_base + uint32_t(s) * act_stage, bar = lead_full0 + 8 * s;
                if (rank == 0)
                    elect_expect_tx(full0 + 8 * s, uint32_t(a.bm) * 256u); // both CTAs' rows
                elect_tma_load_2d_pair(dst, &tm_act, st * 128, row0, bar);
                elect_tma_load_2d_pair(dst + act_half, &tm_act, st * 128 + 64, row0, bar);
                if (++s == a.num_stages)
                {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
        // the last commits arrive on this CTA's barriers from the first CTA: stay until they have
        for (int i = 0; i < a.num_stages && ok; ++i)
        {
            ok = wait_bar<false>(empty0 + 8 * s, ph ^ 1, abort_flag);
            if (++s == a.num_stages)
            {
                s = 0;
                ph ^= 1;
            }
        }
    }
    else if (warp == kMmaWarp)
    {
        // ------------------------------------------------------------------ MMA issuer
        if (rank == 0)
        {
            uint32_t const idesc = (1u << 4)             // fp32 accumulator
                | (kFmt << 7) | (kFmt << 10)             // A and B types (both K-major)
                | (uint32_t(a.bm >> 3) << 17)            // MMA N = activation rows
                | (uint32_t(kPairN >> 4) << 24);         // MMA M = weight columns of the pair
            uint64_t const desc0 = smem_desc_sw128(smem_base);
            uint64_t const desc_stage = uint64_t(act_stage >> 4), desc_half = uint64_t(act_half >> 4); // 16-byte units
            uint32_t const d_empty0 = smem_u32(&bars->d_empty[0]), d_full0 = smem_u32(&bars->d_full[0]);
            uint16_t const both = uint16_t(3u << lead_rank);
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            uint32_t dph = 0; // bit b: parity of accumulator b's next drain
            int db = 0, done = 0;
            for (int item = pair; item < num_items && ok; item += num_pairs, ++done)
            {
                Item const it = item_of(item);
                if (done >= a.d_bufs)
                {
                    ok = wait_bar<true>(d_empty0 + 8 * db, (dph >> db) & 1u, abort_flag);
                    if (!ok)
                        break;
                    dph ^= 1u << db;
                    tc_fence_after();
                }
                uint32_t const d_tmem = tmem + uint32_t(db * a.bm);
                uint32_t accumulate = 0;
                for (int st = it.st0; st < it.st1; ++st)
                {
                    ok = wait_bar<true>(full0 + 8 * s, ph, abort_flag);
                    if (!ok)
                        break;
                    tc_fence_after();
                    uint64_t const desc = desc0 + uint64_t(s) * desc_stage;
                    uint32_t const a_col = a_ring + uint32_t(s) * kStageCols;
                    tc_mma4_ts_elect(d_tmem, a_col, desc, idesc, accumulate);
                    if (st * 128 + 64 < a.k)
                        tc_mma4_ts_elect(d_tmem, a_col + 32, desc + desc_half, idesc, 1u);
                    accumulate = 1u;
                    tc_commit_pair_elect(empty0 + 8 * s, both); // frees the activation stage and the TMEM stage
                    if (++s == a.num_stages)
                    {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok)
                    tc_commit_pair_elect(d_full0 + 8 * db, both);
                db = db + 1 == a.d_bufs ? 0 : db + 1;
            }
            // stay until the other CTA's last arrivals have landed
            for (int i = 0; i < a.d_bufs && i < done && ok; ++i)
            {
                db = db == 0 ? a.d_bufs - 1 : db - 1;
                ok = wait_bar<true>(d_empty0 + 8 * db, (dph >> db) & 1u, abort_flag);
            }
        }
    }
    else if (warp >= kConvWarp0 && warp < kWProdWarp)
    {
        // ------------------------------------------------------------------ conversion
        int const quad = warp & 3;                     // TMEM lane quadrant this warp may touch
        int const cgroup = (warp - kConvWarp0) >> 2;   // which k blocks this warp converts
        int const n_local = quad * 32 + lane;          // weight column inside the CTA's tile = TMEM lane
        uint32_t const lane_ring = a_ring + (uint32_t(quad * 32) << 16);
        uint32_t const lead_full0 = cluster_addr(full0, lead_rank);
        // This thread's 16-byte chunk c of a line sits at w_off ^ (c << 4): the TMA's 128-byte swizzle
        // exchanges chunk index and row modulo 8, which makes the reads conflict-free.
        int const w_row = n_local / IL;
        uint32_t const w_off = uint32_t(w_row * 128 + ((((n_local % IL) * SEG_CHUNKS) ^ (w_row & 7)) << 4));

        // Own steps are every kConvGroups-th, counted over all items; the rings run on from item to item.
        int s = cgroup, ws = cgroup;
        uint32_t ph = 0;
        uint32_t w_seen = 0; // bit ws: parity of this group's next phase on w_full[cgroup][ws]
        int skip = cgroup;   // steps from the start of the item to the next own step
        bool ok = true;
        for (int item = pair; item < num_items && ok; item += num_pairs)
        {
            Item const it = item_of(item);
            int st = it.st0 + skip;
            for (; st < it.st1; st += kConvGroups)
            {
                ok = wait_bar<false>(w_full0 + 8 * (cgroup * kMaxWStages + ws), (w_seen >> ws) & 1u, abort_flag);
                if (!ok)
                    break;
                w_seen ^= 1u << ws;
                uint8_t const* wst = smem + (w_ring - smem_base) + size_t(ws) * W_STAGE;
                uint16_t const* sc = reinterpret_cast<uint16_t const*>(wst + W_BYTES) + n_local;
                uint4 raw[2][SEG_CHUNKS];
                uint32_t s2[2], z2[2];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    int const grow = h && a.group_shift == 6 ? 128 : 0;
                    s2[h] = sc[grow];
                    s2[h] = prmt(s2[h], s2[h], 0x1010u);
                    if (HAS_ZERO)
                    {
                        z2[h] = sc[grow + 256];
                        z2[h] = prmt(z2[h], z2[h], 0x1010u);
                    }
#pragma unroll
                    for (int c = 0; c < SEG_CHUNKS; ++c)
                        raw[h][c] = *reinterpret_cast<uint4 const*>(wst + h * LINE_TILE + (w_off ^ uint32_t(c << 4)));
                }
                __syncwarp();
                if (lane == 0)
                    arrive_local(w_empty0 + 8 * ws);
                uint32_t const a_col = lane_ring + uint32_t(s) * kStageCols;
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    uint32_t v[32]; // TMEM columns of the half step: k = 2 * column (+1)
#pragma unroll
                    for (int c = 0; c < SEG_CHUNKS; ++c)
                    {
                        uint32_t const r[4] = {raw[h][c].x, raw[h][c].y, raw[h][c].z, raw[h][c].w};
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                        {
                            // pair p of register j holds k = 32c + 2j + 8p (+1) (int4), 16c + 2j + 8p (+1) (int8)
                            constexpr int PAIRS = BITS == 4 ? 4 : 2;
                            uint32_t q[PAIRS];
                            if constexpr (BITS == 4)
                                cvt_int4x8<T>(r[j], q);
                            else
                                cvt_int8x4<T>(r[j], q);
#pragma unroll
                            for (int p = 0; p < PAIRS; ++p)
                                v[4 * PAIRS * c + j + 4 * p] = HAS_ZERO ? P::fma(q[p], s2[h], z2[h]) : P::mul(q[p], s2[h]);
                        }
                    }
                    if (h == 0)
                    {
                        ok = wait_bar<false>(empty0 + 8 * s, ph ^ 1, abort_flag);
                        if (!ok)
                            break;
                        tc_fence_after();
                    }
                    tc_st32(a_col + 32 * h, v);
                }
                if (!ok)
                    break;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    arrive_cluster_relaxed(lead_full0 + 8 * s);
                ws += kConvGroups;
                ws -= ws >= a.num_wstages ? a.num_wstages : 0;
                s += kConvGroups;
                if (s >= a.num_stages)
                {
                    s -= a.num_stages;
                    ph ^= 1;
                }
            }
            skip = st - it.st1;
        }
    }
    else if (warp < kEpiWarps)
    {
        // ------------------------------------------------------------------ epilogue
        asm volatile("griddepcontrol.wait;" ::: "memory");
        uint32_t const lane_addr = tmem + (uint32_t(warp * 32) << 16);
        uint16_t const* bias = static_cast<uint16_t const*>(a.bias);
        uint32_t const d_full0 = smem_u32(&bars->d_full[0]), lead_d_empty0 = cluster_addr(smem_u32(&bars->d_empty[0]), lead_rank);
        uint32_t dph = 0;
        int db = 0;
        bool ok = true;
        for (int item = pair; item < num_items && ok; item += num_pairs)
        {
            Item const it = item_of(item);
            int const n = it.n0 + int(rank) * BN + warp * 32 + lane;
            bool const n_ok = n < a.n; // n is a multiple of 32: uniform over the warp
            int const m0 = it.row0;
            float const bias_f = (SPLIT == SPLIT_NONE && bias && n_ok) ? P::to_float(bias[size_t(it.slice) * a.n + n]) : 0.f;
            ok = wait_bar<false>(d_full0 + 8 * db, (dph >> db) & 1u, abort_flag);
            if (!ok)
                break;
            dph ^= 1u << db;
            tc_fence_after();
            float* part = SPLIT == SPLIT_WORKSPACE ? a.partial + size_t(it.split) * a.m * a.n + n : nullptr;
            // two rows at a time: neighbouring lanes exchange halves, so that the even lane stores columns
            // n, n + 1 of the first row and the odd lane columns n - 1, n of the second
            uint16_t* out = static_cast<uint16_t*>(a.out) + (n & ~1);
            uint32_t const sel = lane & 1 ? 0x3276u : 0x5410u;
            int const c_end = min(a.bm, it.row_end - m0);
#pragma unroll 1
            for (int c0 = 0; c0 < c_end; c0 += 32)
            {
                uint32_t v[32];
                tc_ld32(lane_addr + uint32_t(db * a.bm + c0), v);
                if (c0 + 32 >= c_end)
                {
                    // everything is in registers: the accumulator may be overwritten
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0)
                        arrive_cluster_relaxed(lead_d_empty0 + 8 * db);
                }
                if (SPLIT == SPLIT_CLUSTER)
                {
                    // [row][128 columns] in the activation ring, which no copy or MMA uses any more
                    float* dst = reinterpret_cast<float*>(smem) + c0 * BN + warp * 32 + lane;
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        dst[j * BN] = __uint_as_float(v[j]);
                    continue;
                }
                if (!n_ok)
                    continue;
                if (SPLIT == SPLIT_WORKSPACE)
                {
                    // fp32 partial tile; splitk_reduce_kernel, next on the stream, adds the partial tiles in
                    // split order (deterministic) and writes the output
                    float* dst = part + size_t(m0 + c0) * a.n;
                    int const rows = it.row_end - m0 - c0;
#pragma unroll
                    for (int j = 0; j < 32; ++j, dst += a.n)
                        if (j < rows)
                            __stcg(dst, __uint_as_float(v[j]));
                }
                else
                {
                    // (row pointers are advanced, not computed from the row: with an address product per
                    // row and a bounds test in front of every store a chunk took twice as long)
                    uint32_t o[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        o[j] = P::pack2(fmaf(a.alpha, __uint_as_float(v[2 * j]), bias_f),
                            fmaf(a.alpha, __uint_as_float(v[2 * j + 1]), bias_f));
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        o[j] = prmt(o[j], __shfl_xor_sync(0xffffffffu, o[j], 1), sel);
                    int const mrow = m0 + c0 + (lane & 1), rows = it.row_end - mrow; // this lane's rows: mrow, mrow + 2, ..
                    uint16_t* dst = out + size_t(mrow) * a.n;
                    size_t const two_rows = size_t(a.n) * 2;
                    if (m0 + c0 + 32 <= it.row_end)
                    {
#pragma unroll
                        for (int j = 0; j < 16; ++j, dst += two_rows)
                            *reinterpret_cast<uint32_t*>(dst) = o[j];
                    }
                    else
                    {
#pragma unroll
                        for (int j = 0; j < 16; ++j, dst += two_rows)
                            if (2 * j < rows)
                                *reinterpret_cast<uint32_t*>(dst) = o[j];
                    }
                }
            }
            db = db + 1 == a.d_bufs ? 0 : db + 1;
        }
    }

    // Teardown: both CTAs meet here (also after a timeout), then the allocating warps free TMEM.
    tc_fence_before();
    __syncthreads();
    if (*abort_flag)
        for (int i = 0; i < 64; ++i)
            __nanosleep(10000); // copies and MMAs that are still in flight end before the memory is given back
    cluster_sync_all();
    if (SPLIT == SPLIT_CLUSTER)
    {
        // Every CTA adds the rows row % splits == its split of its 128 columns: a warp per row, four columns
        // per lane, the other splits' values from their shared memory.
        Item const it = item_of(pair);
        int const split = it.split, m0 = it.row0, rows = min(a.bm, it.row_end - m0);
        int const n = it.n0 + int(rank) * BN + 4 * lane;
        if (n < a.n) // n is a multiple of 32
        {
            float b[4] = {0.f, 0.f, 0.f, 0.f};
            if (a.bias)
            {
                uint2 const bw = *reinterpret_cast<uint2 const*>(static_cast<uint16_t const*>(a.bias) + size_t(it.slice) * a.n + n);
                P::unpack2(bw.x, b[0], b[1]);
                P::unpack2(bw.y, b[2], b[3]);
            }
            for (int row = split + a.splits * warp; row < rows; row += a.splits * (kThreads / 32))
            {
                uint32_t const local = smem_base + uint32_t(row * BN + 4 * lane) * 4u;
                float4 x[kMaxClusterSplits];
#pragma unroll
                for (int q = 0; q < kMaxClusterSplits; ++q)
                    if (q < a.splits)
                        x[q] = ld_cluster_f4(cluster_addr(local, 2 * q + rank));
                float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int q = 0; q < kMaxClusterSplits; ++q)
                    if (q < a.splits)
                    {
                        sum.x += x[q].x;
                        sum.y += x[q].y;
                        sum.z += x[q].z;
                        sum.w += x[q].w;
                    }
                uint2 o;
                o.x = P::pack2(fmaf(a.alpha, sum.x, b[0]), fmaf(a.alpha, sum.y, b[1]));
                o.y = P::pack2(fmaf(a.alpha, sum.z, b[2]), fmaf(a.alpha, sum.w, b[3]));
                *reinterpret_cast<uint2*>(static_cast<uint16_t*>(a.out) + size_t(m0 + row) * a.n + n) = o;
            }
        }
        cluster_sync_all(); // nobody leaves while its shared memory is being read
    }
    if (warp == kMmaWarp)
    {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(uint32_t(kTmemCols))
                     : "memory");
    }
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------
static size_t split_align(size_t bytes)
{
    return (bytes + 255) & ~size_t(255);
}

// Workspace for split-k: `splits` fp32 copies of the output.
static size_t split_bytes(int m, int n, int splits)
{
    return size_t(splits) * m * n * sizeof(float);
}

// out[m, n] = alpha * sum over splits (in order) of partial[s, m, n] + bias[n]; four columns per thread.
template <typename T>
__global__ void __launch_bounds__(256)
    splitk_reduce_kernel(T* out, float const* partial, T const* bias, float alpha, size_t mn_vec, int n_vec, int splits)
{
    using P = Pair<T>;
    // programmatic dependent of the GEMM: its launch overlaps the GEMM's tail
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    size_t const i = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= mn_vec)
        return;
    float4 const* src = reinterpret_cast<float4 const*>(partial) + i;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    int sp = 0;
    for (; sp + 4 <= splits; sp += 4)
    {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            v[u] = __ldcg(src + size_t(sp + u) * mn_vec);
#pragma unroll
        for (int u = 0; u < 4; ++u)
        {
            acc.x += v[u].x;
            acc.y += v[u].y;
            acc.z += v[u].z;
            acc.w += v[u].w;
        }
    }
    for (; sp < splits; ++sp)
    {
        float4 const v = __ldcg(src + size_t(sp) * mn_vec);
        acc.x += v.x;
        acc.y += v.y;
        acc.z += v.z;
        acc.w += v.w;
    }
    float b[4] = {0.f, 0.f, 0.f, 0.f};
    if (bias)
    {
        uint2 const bw = *reinterpret_cast<uint2 const*>(bias + size_t(i % n_vec) * 4);
        P::unpack2(bw.x, b[0], b[1]);
        P::unpack2(bw.y, b[2], b[3]);
    }
    uint2 o;
    o.x = uint32_t(P::from_float(fmaf(alpha, acc.x, b[0]))) | (uint32_t(P::from_float(fmaf(alpha, acc.y, b[1]))) << 16);
    o.y = uint32_t(P::from_float(fmaf(alpha, acc.z, b[2]))) | (uint32_t(P::from_float(fmaf(alpha, acc.w, b[3]))) << 16);
    *reinterpret_cast<uint2*>(out + i * 4) = o;
}

// Launches a kernel as a programmatic dependent of whatever precedes it in the stream (every kernel
// here orders itself with griddepcontrol.wait before it touches what its predecessors may write).
template <typename... KArgs, typename... Args_>
static int launch_pdl(void (*kernel)(KArgs...), int grid, int threads, size_t smem, int cluster, cudaStream_t stream,
    Args_ const&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(unsigned(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = unsigned(cluster);
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess ? W4_OK : W4_ERR_CUDA;
}

// The experts of a launch: neighbours, out of the `slices` of the weight tensor, that have rows. Those that are
// computed elsewhere get no tiles.
struct Experts
{
    int num, slices;
    int slice[kMaxExperts], first_row[kMaxExperts + 1];
    bool elsewhere[kMaxExperts];

    int rows(int e) const
    {
        return elsewhere[e] ? 0 : first_row[e + 1] - first_row[e];
    }
};

template <typename T, int BITS, bool HAS_ZERO, int SPLIT>
static int launch_one(W4GemmParams const& p, void const* act, Experts const& ex, DeviceInfo const& dev, cudaStream_t stream,
    TcPlan const& plan)
{
    constexpr int IL = BITS == 4 ? 4 : 2;
    constexpr int W_STAGE = 2 * (BN / IL) * 128 + 1024;
    auto kernel = gemm_kernel<T, BITS, HAS_ZERO, SPLIT>;

    Args a{};
    a.bias = p.bias;
    a.out = p.out;
    a.alpha = p.alpha;
    a.m = p.m;
    a.n = p.n;
    a.k = p.k;
    a.group_shift = p.group_size == 64 ? 6 : (p.group_size == 128 ? 7 : 31);
    a.bm = plan.bm;
    a.tiles_n = (p.n + kPairN - 1) / kPairN;
    a.groups = p.group_size ? p.k / p.group_size : 1;
    a.num_experts = ex.num;
    for (int e = 0; e < ex.num; ++e)
    {
        a.slice[e] = ex.slice[e];
        a.first_row[e] = ex.first_row[e];
        a.first_tile[e + 1] = a.first_tile[e] + (ex.rows(e) + plan.bm - 1) / plan.bm * a.tiles_n;
    }
    a.first_row[ex.num] = ex.first_row[ex.num];
    a.weights_static = (p.flags & W4_GEMM_WEIGHTS_STATIC) ? 1 : 0;
    a.splits = plan.splits;
    a.steps_split = plan.steps_split;
    if (SPLIT == SPLIT_WORKSPACE)
    {
        // partial tiles go to the workspace, behind the scaled copy of the activations if there is one
        size_t const act_copy = (act != p.act) ? split_align(size_t(p.m) * p.k * 2) : 0;
        a.partial = reinterpret_cast<float*>(static_cast<char*>(p.workspace) + act_copy);
    }
    // Rings: as many 128-k steps as fit TMEM next to the accumulators (4 at 256 and at 128 rows, more in
    // between and below), the rest of shared memory for weight blocks.
    a.d_bufs = plan.bm <= 128 ? 2 : 1;
    int const stages = (kTmemCols - a.d_bufs * plan.bm) / kStageCols;
    a.num_stages = stages < kMaxStages ? stages : kMaxStages;
    size_t const fixed = sizeof(Barriers) + 16;
    size_t const act_bytes = size_t(a.num_stages) * plan.bm * 128;
    if (size_t(dev.max_smem_optin) < fixed + act_bytes + 3 * W_STAGE)
        return W4_ERR_CUDA;
    size_t const wstages = (size_t(dev.max_smem_optin) - fixed - act_bytes) / W_STAGE;
    a.num_wstages = wstages < size_t(kMaxWStages) ? int(wstages) : kMaxWStages;
    size_t const smem = act_bytes + size_t(a.num_wstages) * W_STAGE + fixed;

    // Activations [m, k] of T, boxes of 64 k x bm / 2 rows, 128-byte swizzle (rows past m read as 0).
    // Weights as bytes [k / 64 lines, n / IL interleaved rows, 128], boxes of two lines x 128 / IL rows.
    // Scales / zeros [groups, n], boxes of the rows of a 128-wide k step x 128 columns.
    CUtensorMap tm_act, tm_w, tm_s, tm_z;
    CUtensorMapDataType const dt
        = std::is_same<T, __nv_bfloat16>::value ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    if (!make_tensor_map_2d(&tm_act, dt, act, uint64_t(p.k), uint64_t(p.m), uint64_t(p.k) * 2, 64, uint32_t(plan.bm / 2),
            CU_TENSOR_MAP_SWIZZLE_128B))
        return W4_ERR_CUDA;
    if (!make_tensor_map_3d(&tm_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.weight, 128, uint64_t(p.n / IL) * ex.slices, uint64_t(p.k / 64),
            uint64_t(p.k) * 2, 128, 128, BN / IL, 2, CU_TENSOR_MAP_SWIZZLE_128B))
        return W4_ERR_CUDA;
    uint64_t const groups = uint64_t(a.groups) * ex.slices;
    uint32_t const box_rows = p.group_size == 64 ? 2 : 1;
    if (!make_tensor_map_2d(&tm_s, CU_TENSOR_MAP_DATA_TYPE_UINT16, p.scales, uint64_t(p.n), groups, uint64_t(p.n) * 2, BN,
            box_rows, CU_TENSOR_MAP_SWIZZLE_NONE))
        return W4_ERR_CUDA;
    tm_z = tm_s;
    if (HAS_ZERO
        && !make_tensor_map_2d(&tm_z, CU_TENSOR_MAP_DATA_TYPE_UINT16, p.zeros, uint64_t(p.n), groups, uint64_t(p.n) * 2, BN,
            box_rows, CU_TENSOR_MAP_SWIZZLE_NONE))
        return W4_ERR_CUDA;

    {
        // per-function, per-device attribute: set once (this block is instantiated once per kernel)
        static std::mutex mu;
        static bool configured[64] = {};
        std::lock_guard<std::mutex> lock(mu);
        if (dev.device < 0 || dev.device >= 64 || !configured[dev.device])
        {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.max_smem_optin)
                    != cudaSuccess
                || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
                return W4_ERR_CUDA;
            if (dev.device >= 0 && dev.device < 64)
                configured[dev.device] = true;
        }
    }
    int const items = a.first_tile[ex.num] * a.splits;
    int const pairs = SPLIT == SPLIT_CLUSTER || items < dev.num_sms / 2 ? items : dev.num_sms / 2;
    int rc = launch_pdl(kernel, 2 * pairs, kThreads, smem, SPLIT == SPLIT_CLUSTER ? 2 * a.splits : 2, stream, a, tm_act, tm_w,
        tm_s, tm_z);
    if (rc == W4_OK && SPLIT == SPLIT_WORKSPACE)
    {
        size_t const mn_vec = size_t(p.m) * p.n / 4; // n is a multiple of 32
        rc = launch_pdl(splitk_reduce_kernel<T>, int((mn_vec + 255) / 256), 256, 0, 1, stream, static_cast<T*>(p.out),
            static_cast<float const*>(a.partial), static_cast<T const*>(p.bias), p.alpha, mn_vec, p.n / 4, a.splits);
    }
    return rc;
}

template <typename T, int BITS, bool HAS_ZERO>
static int dispatch_split(W4GemmParams const& p, void const* act, Experts const& ex, DeviceInfo const& dev, cudaStream_t stream)
{
    int rows[kMaxExperts];
    for (int e = 0; e < ex.num; ++e)
        rows[e] = ex.rows(e);
    // The form of split-k that uses the caller's workspace needs room for the partial tiles there, and its second
    // kernel adds up and stores all p.m rows with one bias: not for the experts of a 3-D weight, also where a
    // launch has one expert only.
    size_t const act_copy = (act != p.act) ? split_align(size_t(p.m) * p.k * 2) : 0;
    TcPlan plan = gemm_tc_plan(rows, ex.num, p.n, p.k, dev.num_sms, p.weight_bits, p.act_dtype, ex.slices == 1);
    if (plan.splits > 1 && !plan.cluster && (!p.workspace || p.workspace_bytes < act_copy + split_bytes(p.m, p.n, plan.splits)))
        plan = gemm_tc_plan(rows, ex.num, p.n, p.k, dev.num_sms, p.weight_bits, p.act_dtype, false);
    if (plan.splits == 1)
        return launch_one<T, BITS, HAS_ZERO, SPLIT_NONE>(p, act, ex, dev, stream, plan);
    return plan.cluster ? launch_one<T, BITS, HAS_ZERO, SPLIT_CLUSTER>(p, act, ex, dev, stream, plan)
                        : launch_one<T, BITS, HAS_ZERO, SPLIT_WORKSPACE>(p, act, ex, dev, stream, plan);
}

template <typename T>
static int dispatch(W4GemmParams const& p, void const* act, Experts const& ex, DeviceInfo const& dev, cudaStream_t stream)
{
    bool const z = p.zeros != nullptr;
    if (p.weight_bits == 4)
        return z ? dispatch_split<T, 4, true>(p, act, ex, dev, stream) : dispatch_split<T, 4, false>(p, act, ex, dev, stream);
    return z ? dispatch_split<T, 8, true>(p, act, ex, dev, stream) : dispatch_split<T, 8, false>(p, act, ex, dev, stream);
}

// Clusters of 2 * splits CTAs the current device runs side by side, by splits: fixed by how its SMs are grouped.
// Without a device, the numbers of a B200 with all 148 SMs.
static int const* max_clusters()
{
    struct Limits
    {
        std::atomic<bool> known{false};
        int clusters[kMaxClusterSplits + 1] = {0, 74, 33, 22, 15, 11, 7, 7, 7};
    };
    static std::mutex mu;
    static Limits devices[64], none;
    DeviceInfo const& dev = current_device_info();
    Limits& l = dev.num_sms > 0 ? devices[dev.device] : none;
    if (dev.num_sms <= 0 || l.known.load(std::memory_order_acquire))
        return l.clusters;
    std::lock_guard<std::mutex> lock(mu);
    if (!l.known.load(std::memory_order_relaxed))
    {
        auto kernel = gemm_kernel<__nv_bfloat16, 4, true, SPLIT_CLUSTER>;
        bool const ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.max_smem_optin) == cudaSuccess
            && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
        for (int s = 1; s <= kMaxClusterSplits; ++s)
        {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(unsigned(2 * s));
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = size_t(dev.max_smem_optin);
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = unsigned(2 * s);
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int n = 0;
            l.clusters[s] = ok && cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess ? n : 0;
        }
        (void) cudaGetLastError(); // a cluster size the device refuses is no error of the caller's
        l.known.store(true, std::memory_order_release);
    }
    return l.clusters;
}

} // namespace tc

// Microseconds per 128-wide k step of a CTA pair (measured on B200): up to 96 rows the conversion's, which
// takes most of the issue slots and, for int8 to bf16, more instructions per weight; above, the MMAs'
// (1024 tensor cycles at 256 rows).
static double step_us(int bm, int bits, int act_dtype)
{
    double const conv = bits == 8 && act_dtype == W4_DTYPE_BF16 ? 0.33 : 0.25, mma = bm * (0.57 / 256);
    return conv > mma ? conv : mma;
}

// The plan with the shortest estimated time: row tiles in steps of 32 and, where the tiles leave pairs idle
// (and only up to 256 rows, where the fp32 partial tiles stay small), split factors. A launch costs 2.5 us plus
// the waves of its work items; an item's epilogue 0.3 us per 32 rows, of which the double-buffered
// accumulators hide all but the last. Splits that share a cluster add the exchange of the partial tiles
// (clusters of 4 and 8 CTAs about 1 us; 6 and more than 8 wait longer for enough free SMs side by side), splits
// through the workspace a second kernel and their traffic. Fitted to 4096 and 8192 x 1024..14336 at 16 to
// 777 rows, each launch by itself: within 1 us of the best plan found by trying all at 14 of 16 points. Beyond
// that, and in long runs at the power limit, it is too low (14336 x 4096 at 4096 rows 228 us, measured 302 cool
// and 356 sustained) and says only which row tile has the fewest waves.
TcPlan gemm_tc_plan(int const* rows, int experts, int n, int k, int num_sms, int bits, int act_dtype, bool may_use_workspace)
{
    int const pairs = num_sms > 1 ? num_sms / 2 : 1;
    int const steps = (k + 127) / 128;
    long const tiles_n = (n + tc::kPairN - 1) / tc::kPairN;
    int const* const clusters = tc::max_clusters();
    TcPlan best{};
    int m = 0; // most rows of an expert
    for (int e = 0; e < experts; ++e)
        m = m > rows[e] ? m : rows[e];
    int const most = m >= tc::kMaxBM ? tc::kMaxBM : (m + 31) & ~31;
    for (int bm = 32; bm <= most; bm += 32)
    {
        long tiles = 0;
        for (int e = 0; e < experts; ++e)
            tiles += tiles_n * ((rows[e] + bm - 1) / bm);
        double const step = step_us(bm, bits, act_dtype), drain = 0.01 * bm;
        int splits_max = m <= 256 && tiles < pairs ? int(pairs / tiles) : 1;
        splits_max = splits_max > 16 ? 16 : splits_max;
        for (int s = 1; s <= splits_max; ++s)
        {
            int const per = (steps + s - 1) / s;
            if ((steps + per - 1) / per != s || (s > 1 && per < 2))
                continue; // an empty work item, or too little in each
            bool const cluster = s > 1 && s <= tc::kMaxClusterSplits && tiles <= clusters[s];
            if (s > 1 && !cluster && !may_use_workspace)
                continue;
            double const waves = double((tiles * s + pairs - 1) / pairs);
            double us = 2.5 + drain + waves * per * step + (waves - 1) * (bm <= 128 ? 0.1 : drain + 0.3);
            if (cluster)
                us += (s == 2 || s == 4 ? 1.0 : 3.0) + 0.008 * bm;
            else if (s > 1)
                us += 2.5 + double(s) * m * n * 8.0 / 6.0e6;
            if (!best.bm || us < best.us)
            {
                best.bm = bm;
                best.splits = s;
                best.steps_split = per;
                best.cluster = cluster;
                best.us = us;
            }
        }
    }
    return best;
}

size_t gemm_tc_workspace_min(int m, int k, int has_act_scale)
{
    // the pre-quant scale is applied to a copy of the activations, as the reference plugin does
    // (weightOnlyGroupwiseQuantMatmulPlugin.cpp:444-458 of the reference project)
    return has_act_scale ? size_t(m) * k * 2 : 0;
}

size_t gemm_tc_workspace_bytes(int m, int n, int k, int has_act_scale, int bits, int act_dtype)
{
    // what lets the kernel use every form of split-k; with less (but at least the minimum) it runs with the
    // forms that need none
    DeviceInfo const& dev = current_device_info();
    int const sms = dev.num_sms > 0 ? dev.num_sms : 148;
    int const splits = gemm_tc_plan(&m, 1, n, k, sms, bits, act_dtype, true).splits;
    size_t bytes = gemm_tc_workspace_min(m, k, has_act_scale);
    if (splits > 1)
        bytes = tc::split_align(bytes) + tc::split_bytes(m, n, splits);
    return bytes;
}

int launch_gemm_tc(W4GemmParams const& p, cudaStream_t stream)
{
    DeviceInfo const& dev = current_device_info();
    if (dev.num_sms <= 0)
        return W4_ERR_CUDA;
    void const* act = p.act;
    if (p.act_scale)
    {
        int const rc = launch_pre_quant_scale(p.workspace, p.act, p.act_scale, p.m, p.k, p.act_dtype, stream);
        if (rc != W4_OK)
            return rc;
        act = p.workspace;
    }
    tc::Experts const one{1, 1, {0}, {0, p.m}, {false}};
    return p.act_dtype == W4_DTYPE_FP16 ? tc::dispatch<__half>(p, act, one, dev, stream)
                                        : tc::dispatch<__nv_bfloat16>(p, act, one, dev, stream);
}

int launch_gemm_tc_experts(W4GemmParams const& p, int num_experts, int const* first_row, bool (*joins)(W4GemmParams const&, int),
    cudaStream_t stream)
{
    DeviceInfo const& dev = current_device_info();
    if (dev.num_sms <= 0)
        return W4_ERR_CUDA;
    tc::Experts ex{};
    ex.slices = num_experts;
    bool any = false;
    for (int e = 0; e < num_experts; ++e)
    {
        int const rows = first_row[e + 1] - first_row[e];
        if (rows > 0)
        {
            ex.slice[ex.num] = e;
            ex.first_row[ex.num] = first_row[e];
            ex.elsewhere[ex.num] = !joins(p, rows);
            any |= !ex.elsewhere[ex.num];
            ex.first_row[++ex.num] = first_row[e + 1];
        }
        if (ex.num < tc::kMaxExperts && e + 1 < num_experts)
            continue;
        if (any)
        {
            int const rc = p.act_dtype == W4_DTYPE_FP16 ? tc::dispatch<__half>(p, p.act, ex, dev, stream)
                                                        : tc::dispatch<__nv_bfloat16>(p, p.act, ex, dev, stream);
            if (rc != W4_OK)
                return rc;
        }
        ex.num = 0;
        any = false;
    }
    return W4_OK;
}

} // namespace w4
