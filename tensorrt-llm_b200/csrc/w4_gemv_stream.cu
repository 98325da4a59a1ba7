// Decode kernel for int4 weights with 128-wide groups or one scale per column, a few rows and large matrices:
// weights go from HBM straight into registers. The kernel of w4_gemv.cu stages them in shared memory, which
// takes a copy, a wait and a release per tile and two shared-memory reads per 32 bytes; here every warp
// streams its own share, equal to within two units whatever the shape, and no barrier is met between the
// activations and the final sum.
//
// One CTA per SM owns a contiguous range of interleaved rows (layout and columns of a group of 16 as in
// w4_gemv.cu). Its work is a list of units of 16 columns x 128 k (1 KB of weights), column group by column
// group, which the 16 warps share out evenly. A warp keeps four units in flight in registers (64 KB per SM;
// a plain read with that pattern reaches 6.4 TB/s on 235 MB and 4.3 TB/s on 29 MB, launch included) and feeds
// them to mma.sync, weights as the 16-row A operand. The activations of all of K (or of as few equal panels as
// fit) are laid out once in shared memory as the B operands of every unit.
//
// Arithmetic: for fp16 and bf16 activations alike the multiplication is fp16 x integer with fp32 sums. Nibbles
// become fp16 numbers where they lie: alone in the low mantissa bits they are the subnormals u * 2^-24 (bits 0..3)
// and u * 2^-20 (bits 4..7), which the tensor cores multiply exactly (one shift for eight weights; bf16 with its
// 7-bit mantissa takes three and 40 % more integer instructions, whose pipe is the second bound). Under an
// exponent, as 1024 + u, they take as long, but then 1032 sum(a) has to cancel in every unit: positive
// activations on integers of -1, 0 and 1 at 28672 k gave outputs 2.3e-3 (bf16) and 1.2e-2 (fp16) of their size
// from the exact ones, now 1.6e-3 and 2.2e-4, the output's rounding. The two kinds have accumulators of their
// own; scale, zero, the powers of two and the bias of 8 are applied to the unit's sums. bf16 activations become
// fp16 exactly: each row of a unit is scaled by the power of two that brings its largest value to 2^14, the
// factor is taken back with the sums.
//
// Measured against the kernel of w4_gemv.cu (zeros, group 128): 4096 x 14336 at one row 10.5 -> 9.1 us, 14336 x 4096
// 12.2 -> 9.7, 2048 x 8192 6.7 -> 4.5, 8192 x 57344 at one row 54 -> 47 and at four 58 -> 50 (4.9 TB/s).
#include <mutex>
#include <type_traits>

#include "w4_common.cuh"
#include "w4_internal.h"

namespace w4
{
namespace stream
{

constexpr int kDepth = 4; // units in flight per warp (12 or 8 warps with more each were slower)
constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;
constexpr int kUnitK = 128;
constexpr int kPieces = 4; // 16-byte pieces of a lane's activation fragment of a unit: one per weight register

constexpr float kBias = 8.f;           // weights are stored as u = q + 8
constexpr float kEven = 16777216.f;    // 2^24: what a sum over even nibbles has to be multiplied by
constexpr float kOddByEven = 0.0625f;  // the odd ones lie four bits higher

struct Args
{
    uint8_t const* weight;
    void const* act;
    void const* act_scale;
    void const* scales;
    void const* zeros;
    void const* bias;
    void* out;
    float alpha;
    int m, n, k;
    int num_rows;    // interleaved rows: n / 4
    int64_t s_unit;  // bytes from a unit's scales to the next unit's (0 per channel)
    int slots;       // column groups that one warp can meet in a panel
    int num_panels, panel_duos; // pairs of units whose activations are in shared memory at a time
    int weights_static;
};

// The loads are ordinary ones, not non-coherent: this kernel is resident while the kernels in front write its
// activations (and, where they are not static, its weights); volatile, so that they stay behind
// griddepcontrol.wait. Weights are read once and pass L1 by; activations and scales stay in it.
__device__ __forceinline__ uint4 ld_stream16(uint8_t const* p)
{
    uint4 v;
    asm volatile("ld.global.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}

__device__ __forceinline__ uint4 ld_act16(void const* p)
{
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ uint32_t ld_scale4(uint8_t const* p)
{
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// Share of warp `w` of `items` items: its first item; the last is in front of the next warp's first.
__device__ __forceinline__ int share_begin(int items, int w)
{
    return int((int64_t(items) * w) / kWarps);
}

template <typename T, bool HAS_ZERO>
__global__ void __launch_bounds__(kThreads, 1) stream_kernel(Args const a)
{
    using P = Pair<T>;
    using H = Pair<__half>;
    // shared memory: activation fragments and row factors of a k panel, the warps' sums
    extern __shared__ __align__(16) uint8_t smem[];

    int const tid = threadIdx.x;
    int const warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31; // (uniform for the compiler as well)
    int const g = lane >> 2, t = lane & 3;

    // Row range of this CTA (balanced to within one interleaved row).
    int const r0 = int((int64_t(a.num_rows) * blockIdx.x) / gridDim.x);
    int const r1 = int((int64_t(a.num_rows) * (blockIdx.x + 1)) / gridDim.x);
    int const num_cg = (r1 - r0 + 3) >> 2;
    int const num_units = a.k / kUnitK, num_duos = (num_units + 1) >> 1;
    int64_t const row_bytes = int64_t(2) * a.k;

    int const MT = (a.m + 1) >> 1, MR = 2 * MT;            // lanes t below MT have rows of their own
    uint4* const act_s = reinterpret_cast<uint4*>(smem);   // [unit][piece][row][t]
    float4* const row_s = reinterpret_cast<float4*>(act_s + size_t(2 * a.panel_duos) * kPieces * a.m * 4); // [unit][MR]
    float* const red = reinterpret_cast<float*>(row_s + size_t(2 * a.panel_duos) * MR); // [warp][slot][g * MT + t] x 4
    int const cg_floats = 8 * MT * 4;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // ---- weight stream. Lane (g, t) holds logical mma rows g and g + 8 = columns 2g and 2g + 1 of a group,
    // whose segments are adjacent in one interleaved row. Units come in duos, neighbours in k; the last duo may
    // lack its second: its activations are zeros and the first unit is loaded in its place.
    struct Unit
    {
        uint32_t wa[4], wb[4]; // columns 2g, 2g + 1
        uint32_t s, z;
    };
    Unit ring[kDepth];
    int const in_row = (t >> 1) * 128 + (g & 1) * 64 + (t & 1) * 16;
    int const tail_duo = num_units & 1 ? num_duos - 1 : -1;

    // Share of this warp in a k panel: duos in the order column group, k.
    int ld_left, ld_duo, ld_end, ld_begin, ld_cg;
    uint8_t const *ld_w, *ld_s, *ld_z;
    auto seek_group = [&]()
    {
        // A lane whose row lies past the CTA's range reads the range's last row (and its columns' scales)
        // instead: its results are not written.
        int const row = min(r0 + ld_cg * 4 + (g >> 1), r1 - 1);
        ld_w = a.weight + row * row_bytes + in_row + int64_t(ld_duo) * (4 * kUnitK);
        int64_t const o = int64_t(row * 4 + 2 * (g & 1)) * 2 + ld_duo * (2 * a.s_unit);
        ld_s = static_cast<uint8_t const*>(a.scales) + o;
        ld_z = static_cast<uint8_t const*>(a.zeros) + o;
    };
    auto begin_panel = [&](int panel)
    {
        ld_begin = panel * a.panel_duos;
        ld_end = min(ld_begin + a.panel_duos, num_duos);
        int const n = ld_end - ld_begin, items = num_cg * n, u0 = share_begin(items, warp);
        ld_left = share_begin(items, warp + 1) - u0;
        ld_cg = u0 / n;
        ld_duo = ld_begin + u0 - ld_cg * n;
        seek_group();
    };
    auto load_unit = [&](Unit& u, uint8_t const* w, int64_t so)
    {
        uint4 const va = ld_stream16(w), vb = ld_stream16(w + 32);
        u.wa[0] = va.x, u.wa[1] = va.y, u.wa[2] = va.z, u.wa[3] = va.w;
        u.wb[0] = vb.x, u.wb[1] = vb.y, u.wb[2] = vb.z, u.wb[3] = vb.w;
        u.s = ld_scale4(ld_s + so);
        if (HAS_ZERO)
            u.z = ld_scale4(ld_z + so);
    };
    auto load_next = [&](Unit& u0, Unit& u1)
    {
        if (ld_left > 0)
        {
            bool const both = ld_duo != tail_duo;
            load_unit(u0, ld_w, 0);
            load_unit(u1, ld_w + (both ? 2 * kUnitK : 0), both ? a.s_unit : 0);
            --ld_left;
            ld_w += 4 * kUnitK;
            ld_s += 2 * a.s_unit;
            ld_z += 2 * a.s_unit;
            if (++ld_duo == ld_end)
            {
                ld_duo = ld_begin;
                ++ld_cg;
                seek_group();
            }
        }
    };

    // Weights that the preceding kernel may still be writing must not be fetched early.
    if (!a.weights_static)
        asm volatile("griddepcontrol.wait;" ::: "memory");
    if (num_cg > 0)
    {
        begin_panel(0);
#pragma unroll
        for (int i = 0; i < kDepth; i += 2)
            load_next(ring[i], ring[i + 1]);
    }
    // Slots of this warp: its share of a panel begins in column group num_cg * warp / kWarps whatever the
    // panel's length. Each lane owns its entries.
    float* const slot0 = red + warp * a.slots * cg_floats + (g * MT + t) * 4;
    if (t < MT)
        for (int i = 0; i < a.slots; ++i)
            *reinterpret_cast<float4*>(slot0 + i * cg_floats) = make_float4(0.f, 0.f, 0.f, 0.f);

    // ---- activations of a k panel as mma B fragments in the order of the weights, with the pre-quant scale
    // applied. A thread takes one lane's fragment of one row of a unit.
    T const* act = static_cast<T const*>(a.act);
    T const* act_scale = static_cast<T const*>(a.act_scale);
    auto stage_act = [&](int unit0, int units)
    {
        for (int i = tid; i < ((units * a.m * 4 + 31) & ~31); i += kThreads)
        {
            int const ft = i & 3, ur = i >> 2, u = ur / a.m, row = ur - u * a.m;
            bool const inside = u < units;
            int const k0 = (unit0 + u) * kUnitK + ft * 32;
            bool const valid = inside && k0 < a.k;
            uint4 v[4];
#pragma unroll
            for (int p = 0; p < 4; ++p)
                v[p] = valid ? ld_act16(act + int64_t(row) * a.k + k0 + 8 * p) : make_uint4(0, 0, 0, 0);
            if (act_scale && valid)
#pragma unroll
                for (int p = 0; p < 4; ++p)
                {
                    uint4 const ps = ld_act16(act_scale + k0 + 8 * p);
                    v[p].x = P::mul(v[p].x, ps.x);
                    v[p].y = P::mul(v[p].y, ps.y);
                    v[p].z = P::mul(v[p].z, ps.z);
                    v[p].w = P::mul(v[p].w, ps.w);
                }
            // v[p] holds pair p of weight registers 0..3; per register: pairs 0, 2 (even nibbles), 1, 3 (odd)
            uint32_t x[16] = {v[0].x, v[2].x, v[1].x, v[3].x, v[0].y, v[2].y, v[1].y, v[3].y, v[0].z, v[2].z, v[1].z, v[3].z,
                v[0].w, v[2].w, v[1].w, v[3].w};
            float unscale = 1.f;
            if constexpr (std::is_same<T, __nv_bfloat16>::value)
            {
                uint32_t top2 = 0; // exponent and mantissa bits order like the magnitudes
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    top2 = __vmaxu2(top2, x[j] & 0x7fff7fffu);
                top2 = __vmaxu2(top2, __shfl_xor_sync(0xffffffffu, top2, 1));
                top2 = __vmaxu2(top2, __shfl_xor_sync(0xffffffffu, top2, 2));
                // the factor 2^(141 - e) and its inverse are normal numbers from exponent 15 on
                int const e = max(int(max(top2 & 0xffffu, top2 >> 16) >> 7), 15);
                float const scale = __uint_as_float(uint32_t(127 + 14 + 127 - e) << 23);
                unscale = __uint_as_float(uint32_t(e - 14) << 23);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                {
                    float lo, hi;
                    P::unpack2(x[j], lo, hi);
                    x[j] = H::pack2(lo * scale, hi * scale);
                }
            }
            // Sums over k by the tensor cores: the four lanes of a (unit, row) are one column of the B operand, an
            // all-ones A operand adds up what they hold. Lane (g, t) gets the sums of columns 2t and 2t + 1.
            constexpr uint32_t one = 0x3c003c00u;
            uint32_t const ones[4] = {one, one, one, one};
            float even[4], odd[4];
            H::mma0(even, ones, x[0], x[1]);
            H::mma0(odd, ones, x[2], x[3]);
#pragma unroll
            for (int r = 1; r < 4; ++r)
            {
                H::mma(even, ones, x[4 * r], x[4 * r + 1]);
                H::mma(odd, ones, x[4 * r + 2], x[4 * r + 3]);
            }
            // column lane / 4 is entry (lane / 4) % 2 of lane (lane / 4) / 2
            int const from = lane >> 3;
            float const e0 = __shfl_sync(0xffffffffu, even[0], from), e1 = __shfl_sync(0xffffffffu, even[1], from);
            float const o0 = __shfl_sync(0xffffffffu, odd[0], from), o1 = __shfl_sync(0xffffffffu, odd[1], from);
            float const se = (lane >> 2) & 1 ? e1 : e0, so = (lane >> 2) & 1 ? o1 : o0;
            if (inside)
            {
#pragma unroll
                for (int p = 0; p < kPieces; ++p)
                    act_s[((u * kPieces + p) * a.m + row) * 4 + ft] = make_uint4(x[4 * p], x[4 * p + 1], x[4 * p + 2], x[4 * p + 3]);
                if (ft == 0)
                    row_s[u * MR + row] = make_float4(unscale, -kBias * (se + so), unscale * (se + so), 0.f);
            }
        }
    };

    float acc[4] = {0.f, 0.f, 0.f, 0.f}; // running sums of the column group
    // This lane's activations: row g (rows past m repeat the last: an mma keeps the rows apart), factors of
    // rows 2t and 2t + 1.
    int const act_lane = min(g, a.m - 1) * 4 + t, row_lane = 2 * min(t, MT - 1), piece = a.m * 4;

    // One unit: 16 columns x 128 k, added to the running sums. `act`, `rows`: the unit's activations and factors.
    auto process = [&](Unit const& u, uint4 const* act, float4 const* rows)
    {
        float even[4], odd[4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
        {
            uint32_t const ra = u.wa[jj], rb = u.wb[jj], sa = ra >> 8, sb = rb >> 8;
            uint32_t const ev[4] = {ra & 0x000f000fu, rb & 0x000f000fu, sa & 0x000f000fu, sb & 0x000f000fu};
            uint32_t const od[4] = {ra & 0x00f000f0u, rb & 0x00f000f0u, sa & 0x00f000f0u, sb & 0x00f000f0u};
            uint4 const b = act[jj * piece + act_lane];
            if (jj == 0)
            {
                H::mma0(even, ev, b.x, b.y);
                H::mma0(odd, od, b.z, b.w);
            }
            else
            {
                H::mma(even, ev, b.x, b.y);
                H::mma(odd, od, b.z, b.w);
            }
        }
        // s f (S - 8 sum(a)) + z f sum(a) with the row's factor f
        float s[2], z[2] = {0.f, 0.f};
        P::unpack2(u.s, s[0], s[1]);
        if (HAS_ZERO)
            P::unpack2(u.z, z[0], z[1]);
        float4 const f0 = rows[row_lane], f1 = rows[row_lane + 1];
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
            float4 const& f = c & 1 ? f1 : f0;
            acc[c] = fmaf(s[c >> 1] * f.x, fmaf(fmaf(odd[c], kOddByEven, even[c]), kEven, f.y), acc[c]);
            if (HAS_ZERO)
                acc[c] = fmaf(z[c >> 1], f.z, acc[c]);
        }
    };

    // Activations (and, later, the output) belong to the preceding kernels: wait for them here.
    asm volatile("griddepcontrol.wait;" ::: "memory");

    int const act_unit = kPieces * piece;
    for (int panel = 0; panel < a.num_panels; ++panel)
    {
        int const d0 = panel * a.panel_duos, n = min(a.panel_duos, num_duos - d0), items = num_cg * n;
        if (panel > 0)
            __syncthreads(); // the previous panel's activations have been read
        stage_act(2 * d0, 2 * n);
        int const u0 = share_begin(items, warp);
        int left = share_begin(items, warp + 1) - u0;
        int to_end = n - u0 % n; // duos to the end of the column group
        uint4 const* act_p = act_s + (n - to_end) * 2 * act_unit;
        float4 const* row_p = row_s + (n - to_end) * 2 * MR;
        float* dst = slot0;
        __syncthreads();
        while (left > 0)
        {
#pragma unroll
            for (int i = 0; i < kDepth; i += 2)
                if (left > 0)
                {
                    process(ring[i], act_p, row_p);
                    process(ring[i + 1], act_p + act_unit, row_p + MR);
                    load_next(ring[i], ring[i + 1]);
                    act_p += 2 * act_unit;
                    row_p += 2 * MR;
                    --left;
                    if (--to_end == 0 || left == 0)
                    {
                        // the group ends, or the share: add its sums to the slot
                        to_end = n;
                        act_p = act_s;
                        row_p = row_s;
                        if (t < MT)
                        {
                            float4* const d = reinterpret_cast<float4*>(dst);
                            float4 const v = *d;
                            *d = make_float4(v.x + acc[0], v.y + acc[1], v.z + acc[2], v.w + acc[3]);
                        }
                        dst += cg_floats;
                        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                    }
                }
        }
        if (panel + 1 < a.num_panels && num_cg > 0)
        {
            begin_panel(panel + 1);
#pragma unroll
            for (int i = 0; i < kDepth; i += 2)
                load_next(ring[i], ring[i + 1]);
        }
    }

    // Combine the warps' sums in a fixed order (deterministic) and write the columns.
    __syncthreads();
    for (int o = tid; o < num_cg * 16 * a.m; o += kThreads)
    {
        int const col_in = o & 15, rc = o >> 4, cb = rc / a.m, row = rc - cb * a.m;
        if (r0 + cb * 4 + col_in / 4 >= r1)
            continue;
        int const col = (r0 + cb * 4) * 4 + col_in;
        float const* src = red + ((col_in >> 1) * MT + (row >> 1)) * 4 + (col_in & 1) * 2 + (row & 1);
        float sum = 0.f;
        int const w1 = ((cb + 1) * kWarps - 1) / num_cg; // the last warp whose share can begin in or before cb
        for (int w = cb * kWarps / num_cg; w <= w1; ++w)
            sum += src[(w * a.slots + cb - num_cg * w / kWarps) * cg_floats];
        float v = a.alpha * sum;
        if (a.bias)
            v += P::to_float(static_cast<uint16_t const*>(a.bias)[col]);
        static_cast<uint16_t*>(a.out)[size_t(row) * a.n + col] = P::from_float(v);
    }
}

template <typename T, bool HAS_ZERO>
static int launch_one(Args a, DeviceInfo const& dev, cudaStream_t stream)
{
    auto kernel = stream_kernel<T, HAS_ZERO>;
    int const grid = a.num_rows < dev.num_sms ? a.num_rows : dev.num_sms;
    int const groups = ((a.num_rows + grid - 1) / grid + 3) / 4;
    // a share of groups * duos / warps, rounded up, wherever it starts
    a.slots = groups < 2 ? 1 : (groups + kWarps - 1) / kWarps + 1;
    int const mt = (a.m + 1) / 2;
    size_t const duo_bytes = 2 * (size_t(kUnitK) * a.m * 2 + size_t(2 * mt) * 16);
    size_t const fixed = size_t(kWarps) * a.slots * 8 * mt * 16;
    constexpr size_t kSmemMost = 195 * 1024; // leaves L1 60 KB (see the launch attribute below)
    if (fixed + duo_bytes > kSmemMost)
        return W4_ERR_UNSUPPORTED;
    int const duos = (a.k / kUnitK + 1) / 2, most = int((kSmemMost - fixed) / duo_bytes);
    a.num_panels = (duos + most - 1) / most;
    a.panel_duos = (duos + a.num_panels - 1) / a.num_panels;
    a.num_panels = (duos + a.panel_duos - 1) / a.panel_duos;
    {
        // per-function, per-device attribute: set once
        static std::mutex mu;
        static bool configured[64] = {};
        std::lock_guard<std::mutex> lock(mu);
        if (dev.device < 0 || dev.device >= 64 || !configured[dev.device])
        {
            if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dev.max_smem_optin) != cudaSuccess)
                return W4_ERR_CUDA;
            if (dev.device >= 0 && dev.device < 64)
                configured[dev.device] = true;
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(grid));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = fixed + duo_bytes * a.panel_duos;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    // The loads in flight need their place in L1. Left alone the runtime keeps the split that the kernel in front
    // had, and behind one that takes all shared memory 28 KB of L1 hold the loads back: 80 us instead of 47 at
    // 8192 x 57344, one row. Half of the memory (more where the activations need it) is far from that: at 85 %
    // some sizes of shared memory, 16 or 24 KB among them, still met the largest split, at 0 to 70 % none did.
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = 50;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, a) == cudaSuccess ? W4_OK : W4_ERR_CUDA;
}

} // namespace stream

int launch_gemv_stream(W4GemmParams const& p, cudaStream_t stream)
{
    DeviceInfo const& dev = current_device_info();
    if (dev.num_sms <= 0)
        return W4_ERR_CUDA;
    stream::Args a{};
    a.weight = static_cast<uint8_t const*>(p.weight);
    a.act = p.act;
    a.act_scale = p.act_scale;
    a.scales = p.scales;
    a.zeros = p.zeros;
    a.bias = p.bias;
    a.out = p.out;
    a.alpha = p.alpha;
    a.m = p.m;
    a.n = p.n;
    a.k = p.k;
    a.num_rows = p.n / 4;
    a.s_unit = p.group_size ? int64_t(p.n) * 2 : 0;
    a.weights_static = (p.flags & W4_GEMM_WEIGHTS_STATIC) ? 1 : 0;
    bool const z = p.zeros != nullptr;
    if (p.act_dtype == W4_DTYPE_FP16)
        return z ? stream::launch_one<__half, true>(a, dev, stream) : stream::launch_one<__half, false>(a, dev, stream);
    return z ? stream::launch_one<__nv_bfloat16, true>(a, dev, stream) : stream::launch_one<__nv_bfloat16, false>(a, dev, stream);
}

} // namespace w4
