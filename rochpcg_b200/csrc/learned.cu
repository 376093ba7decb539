// Learned smoother kernels on the 5th-generation tensor cores (tcgen05).  No
// reference counterpart: the conv-net smoother is new in this library.
//
// Convolution (k_conv16).  16 -> 16 channels, 3x3x3: layer 2, and the gradient of
// its input (the transposed convolution is a convolution with mirrored taps and
// swapped channels).  Bricks of 14 x 8 x 4 points, the dx and dz taps stacked in
// the MMA's N.  Layer 3 (k_layer3_tc, one output channel) is the same brick plan,
// layer 1 (k_layer1_tc, one input channel, also the gradient of layer 3's input)
// has the 27 taps as K.
//
// Weight gradient (k_conv16_wgrad).  dW[tap][ci][co] = sum_p x[p+tap][ci] *
// g[p][co] is a GEMM over points with both operands MN-major (8 channels = one
// 16-byte core-matrix row): M = (input line, input channel), N = (gradient
// plane, line, output channel), K = 16 points along x, one accumulator per dx and
// plane.  Per-CTA partial sums are reduced in a fixed order, so the gradient is
// deterministic.
//
// Operand layouts without a swizzle are the canonical "interleaved" forms, in
// 16-byte units: K-major ((8,m),2):((1,SBO),LBO); MN-major
// ((1,m),(8,k)):((.,SBO),(1,LBO)).
//
// Waits.  All waits are on mbarriers (TMA, tcgen05.commit, the roles' arrivals);
// each is bounded.  On timeout the CTA records an error in *status, waits once more
// (bounded) for its MMAs, leaves its loop as a whole block and still frees its
// TMEM, so the context stays usable.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <cmath>

#include "learned.cuh"

namespace hb {

namespace tc {

constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle (layout type 0), sm_100 version.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// Descriptor of a K-major operand with 32-byte rows (K = 16 BF16) in the
// 32-byte swizzle (layout type 6): 8-row groups 256 B apart (SBO), the two
// 16-byte halves of a row 16 B apart (LBO).  Start addresses must keep the
// 256-byte atom phase (base offset 0).
__device__ __forceinline__ uint64_t umma_desc_sw32(uint32_t saddr)
{
    return umma_desc(saddr, 16, 256) | ((uint64_t)6 << 61);
}

// Instruction descriptor of kind::f16: BF16 x BF16 -> FP32, M x N.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N, bool a_mn_major, bool b_mn_major)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// One lane of the (converged) warp.
__device__ __forceinline__ bool elect_one()
{
    uint32_t p;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        ".reg .b32 r;\n\t"
        "elect.sync r|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_commit(uint64_t* mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(mbar))
                 : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mbar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Bounded wait for the completion of phase `parity`; false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* mbar, uint32_t parity)
{
    const uint32_t a = smem_u32(mbar);
    for(uint32_t i = 0; i < kSpinLimit; ++i)
    {
        uint32_t done;
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if(done) return true;
    }
    return false;
}

__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_alloc(uint32_t* holder, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// 16 consecutive FP32 columns of this thread's TMEM lane (32x32b shape: warp
// w of a warpgroup reads lanes 32(w%4) .. 32(w%4)+31).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for(int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 48 consecutive columns: issued here, there after tmem_wait48.
__device__ __forceinline__ void tmem_ld48(uint32_t taddr, uint32_t (&r)[48])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
          "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47])
        : "r"(taddr + 32));
}

// the values as operands: nothing that uses them moves above the wait
__device__ __forceinline__ void tmem_wait48(uint32_t (&r)[48])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                   "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                   "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                   "+r"(r[29]), "+r"(r[30]), "+r"(r[31]), "+r"(r[32]), "+r"(r[33]), "+r"(r[34]), "+r"(r[35]),
                   "+r"(r[36]), "+r"(r[37]), "+r"(r[38]), "+r"(r[39]), "+r"(r[40]), "+r"(r[41]), "+r"(r[42]),
                   "+r"(r[43]), "+r"(r[44]), "+r"(r[45]), "+r"(r[46]), "+r"(r[47])::"memory");
}

// Four groups of four columns, `stride` columns apart.
__device__ __forceinline__ void tmem_ld4x4(uint32_t taddr, uint32_t stride, float (&v)[4][4])
{
    uint32_t r[4][4];
#pragma unroll
    for(int k = 0; k < 4; ++k)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[k][0]), "=r"(r[k][1]), "=r"(r[k][2]), "=r"(r[k][3])
                     : "r"(taddr + k * stride));
    // the values as operands: nothing that uses them moves above the wait
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0][0]), "+r"(r[0][1]), "+r"(r[0][2]), "+r"(r[0][3]), "+r"(r[1][0]), "+r"(r[1][1]),
                   "+r"(r[1][2]), "+r"(r[1][3]), "+r"(r[2][0]), "+r"(r[2][1]), "+r"(r[2][2]), "+r"(r[2][3]),
                   "+r"(r[3][0]), "+r"(r[3][1]), "+r"(r[3][2]), "+r"(r[3][3])::"memory");
#pragma unroll
    for(int k = 0; k < 4; ++k)
#pragma unroll
        for(int i = 0; i < 4; ++i) v[k][i] = __uint_as_float(r[k][i]);
}

}  // namespace tc

using namespace tc;

PermMap make_perm_map(const StencilLevel& L)
{
    PermMap pm{};
    for(int v = 0; v <= 8; ++v) pm.offsets[v] = L.offsets[v];
    for(int v = 0; v < 8; ++v)
    {
        pm.bx[v] = L.bx[v];
        pm.by[v] = L.by[v];
        pm.color_of_par[v] = L.color_of_par[v];
    }
    return pm;
}

__device__ __forceinline__ int perm_row(const PermMap& pm, int z, int y, int x)
{
    const int v = pm.color_of_par[((x & 1) << 2) | ((y & 1) << 1) | (z & 1)];
    return pm.offsets[v] + ((z >> 1) * pm.by[v] + (y >> 1)) * pm.bx[v] + (x >> 1);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ uint4 pack_bf16x8(const float* v)
{
    __align__(16) __nv_bfloat162 h[4];
#pragma unroll
    for(int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    return *reinterpret_cast<uint4*>(h);
}

// The 32 bytes of one point's 16 BF16 channels in one access (256-bit, sm_100):
// two 16-byte ones each touch half of every sector of the warp's points.  p is
// 32-byte aligned.
__device__ __forceinline__ void store_point(void* p, uint4 a, uint4 b)
{
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                 "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}

// K-major no-swizzle offset (bytes) of row r, 8-element K chunk c, for
// 16-column (K = 16) operands with SBO = 256 B, LBO = 128 B.
__host__ __device__ constexpr uint32_t kmajor_off(int r, int c) { return (uint32_t)((r >> 3) * 256 + c * 128 + (r & 7) * 16); }

// Weight tile slot (16 output-channel rows x 16 input channels, 512 B) of tap
// t = (dz+1)*9 + (dy+1)*3 + (dx+1): ordered [dy][dz = +1, 0, -1][dx], so the
// 9 taps of one dy form one 144-row K-major B operand (SBO 256 B) whose rows
// are (dz, dx, output channel) -- any run of its dz blocks is contiguous.
__host__ __device__ constexpr int weight_slot(int t) { return ((t / 3) % 3) * 9 + (2 - t / 9) * 3 + t % 3; }

// ------------------------------------------------------------ forward conv
//
// Warp-specialised persistent kernel, one CTA per SM.  A brick is 14 x 8 x kTZ
// output points; its input box is 16 x 10 x (kTZ + 2) points (one point of
// halo on every side), one TMA load of 32-byte swizzled rows.  The dx and dz
// taps are stacked in N: for each staged plane q and row shift dy, ONE MMA
// (M = 128 staged points of the plane, K = 16 input channels) multiplies the
// shifted plane by the weights of all (dz, dx) taps it feeds, N = 48 per
// output plane (3 dx x 16 channels) for the 1-3 output planes q - 1 - dz;
// the epilogue adds the dx = -1 / +1 blocks of the x-neighbouring rows (lane
// shuffles), so the two halo columns of the box produce no output.
//   warp 0      TMA producer into kStages shared-memory stages (zero fill
//               outside the grid);
//   warp 1      TMEM owner and MMA issuer: 3 (kTZ + 2) + kTZ - 1 MMAs per
//               brick (21 for kTZ = 4) into one of two accumulators of
//               kTZ x 48 columns;
//   warps 2-9   epilogue: tcgen05.ld of the finished accumulator, the dx
//               combination, ReLU / mask, global stores
//               (eight warps instead of four: a training batch, whose masked
//               passes read the activations too, 371 -> 361 us).
// Two samples of 128^3 took 96 us; with a sixth of the box rows loaded 94, a
// third of the MMAs 76, no stores 92: latencies on the roles' paths, not a unit,
// were the bound.  Carried brick coordinates, an elected issuer lane and one
// tcgen05.ld wait a plane with the next plane's columns in flight: 81 us.
// Stage and accumulator hand-offs are mbarriers (TMA complete_tx, MMA commit,
// epilogue arrivals), so loads, MMAs and stores of consecutive bricks overlap.

#ifndef HB_CONV_TZ
#define HB_CONV_TZ 4
#endif
#ifndef HB_CONV_STAGES
#define HB_CONV_STAGES 4
#endif
#ifndef HB_CONV_CTAS
#define HB_CONV_CTAS 1
#endif
constexpr int kTX = 16, kTY = 8, kTZ = HB_CONV_TZ;  // staged x width (with halo), output y, output z
constexpr int kOX = kTX - 2;                          // output x per brick
constexpr int kHY = kTY + 2, kHZ = kTZ + 2;
constexpr int kCopyRows = kTX * kHY * kHZ;            // 960 staged points
constexpr int kRowBytes = kNetCh * 2;                 // the 16 BF16 channels of a point: one 32-byte swizzle row
constexpr int kCopyBytes = kCopyRows * kRowBytes;     // 30720 B = one TMA box
constexpr int kStageBytes = kCopyBytes;
constexpr int kStages = HB_CONV_STAGES;
constexpr int kPlaneCols = 3 * kNetCh;                // one output plane: 3 dx blocks of 16 channels
constexpr int kAccCols = kTZ * kPlaneCols;            // FP32 columns of one brick's accumulator (192)
constexpr int kTmemCols = 512;                        // two accumulators, rounded to a power of two
constexpr int kEpiWarps = 8;                          // two per TMEM lane quadrant, half of the planes each
constexpr int kEpiThreads = 32 * kEpiWarps;
constexpr int kConvThreads = 64 + kEpiThreads;
static_assert(kTZ % 2 == 0, "planes per epilogue warp");
constexpr int kConvSmem = kStages * kStageBytes + kNetWeightTileBytes + 256 + 1024;

static_assert(kRowBytes == 32, "one point per 32-byte swizzle row (K = 16 per MMA)");
static_assert(kTX * kTY == 128, "one z plane of the brick is one 128-row M tile");
static_assert(kStageBytes % 1024 == 0, "stages start on swizzle-atom boundaries");
static_assert(2 * kAccCols <= kTmemCols && kTmemCols <= 512, "TMEM accumulators");
static_assert(3 * kPlaneCols <= 256, "MMA N");
static_assert(kConvSmem <= 227 * 1024, "shared memory per CTA");

struct Brick
{
    int b, x0, y0, z0;
};

// The bricks of a CTA: tile, tile + step, ... with x fastest.  Their coordinates
// are carried along (the divisions of a 64-bit tile number, done by every role for
// every brick, were on each role's path).
struct BrickWalk
{
    int tx, ty, tz;          // bricks per axis
    int b, bz, by, bx;       // the current one
    int sb, sz, sy, sx;      // the step

    __device__ BrickWalk(const ConvGrid& g, int ox, int oy, int oz, long tile, long step)
        : tx((g.nx + ox - 1) / ox), ty((g.ny + oy - 1) / oy), tz((g.nz + oz - 1) / oz)
    {
        split(tile, b, bz, by, bx);
        split(step, sb, sz, sy, sx);
    }

    __device__ void split(long t, int& tb, int& tbz, int& tby, int& tbx) const
    {
        const long q1 = t / tx, q2 = q1 / ty;
        tbx = (int)(t - q1 * tx);
        tby = (int)(q1 - q2 * ty);
        tb = (int)(q2 / tz);
        tbz = (int)(q2 - (long)tb * tz);
    }

    __device__ long count(int nb) const { return (long)tx * ty * tz * nb; }

    __device__ __forceinline__ void next()
    {
        bx += sx;
        int carry = bx >= tx;
        bx -= carry ? tx : 0;
        by += sy + carry;
        carry = by >= ty;
        by -= carry ? ty : 0;
        bz += sz + carry;
        carry = bz >= tz;
        bz -= carry ? tz : 0;
        b += sb + carry;
    }

    // first output point
    __device__ __forceinline__ Brick at(int ox, int oy, int oz) const { return Brick{b, bx * ox, by * oy, bz * oz}; }
};

__device__ __forceinline__ void mbar_expect_tx(uint64_t* mbar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(mbar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* mbar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(mbar)) : "memory");
}

// Tiled 5-D TMA load (no multicast) completing on mbar.
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t* mbar)
{
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(mbar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

// Bounded wait that also gives up when another role aborted.
__device__ __forceinline__ bool role_wait(uint64_t* mbar, uint32_t parity, volatile int* abort_flag, int* status,
                                          int code)
{
    const uint32_t a = smem_u32(mbar);
    for(uint32_t i = 0; i < kSpinLimit; ++i)
    {
        uint32_t done;
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if(done) return true;
        if((i & 255) == 255 && *abort_flag) return false;
    }
    *abort_flag = 1;
    atomicExch(status, code);
    return false;
}

template <int kOut>
__global__ void __launch_bounds__(kConvThreads, HB_CONV_CTAS)
    k_conv16(const __grid_constant__ CUtensorMap in_map, ConvGrid g, const __nv_bfloat16* __restrict__ wB, void* out,
             const __nv_bfloat16* __restrict__ act, int* status)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = smem;                                   // kStages x kStageBytes
    unsigned char* sW = smem + kStages * kStageBytes;           // weights
    uint64_t* full = (uint64_t*)(sW + kNetWeightTileBytes);     // [kStages] TMA -> MMA
    uint64_t* empty = full + kStages;                           // [kStages] MMA -> TMA
    uint64_t* tfull = empty + kStages;                          // [2] MMA -> epilogue
    uint64_t* tempty = tfull + 2;                               // [2] epilogue -> MMA
    uint32_t* tholder = (uint32_t*)(tempty + 2);
    volatile int* abort_flag = (volatile int*)(tholder + 1);

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    BrickWalk walk(g, kOX, kTY, kTZ, blockIdx.x, gridDim.x);
    const long ntiles = walk.count(g.nb);

    for(int i = tid; i < kNetWeightTileBytes / 16; i += kConvThreads)
        reinterpret_cast<uint4*>(sW)[i] = reinterpret_cast<const uint4*>(wB)[i];
    if(tid == 0)
    {
        for(int s = 0; s < kStages; ++s)
        {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for(int a = 0; a < 2; ++a)
        {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], kEpiThreads);
        }
        *abort_flag = 0;
    }
    if(warp == 1) tmem_alloc(tholder, kTmemCols);
    fence_async_smem();  // the weights are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tholder;
    pdl_launch_dependents();  // not before this CTA has its tensor memory
    pdl_wait();  // from here on the previous kernel's output is read

    if(warp == 0 && lane == 0)
    {
        // ---- TMA producer
        long issued = 0;
        for(long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, walk.next(), ++issued)
        {
            const int st = (int)(issued % kStages);
            const uint32_t ph = (uint32_t)((issued / kStages) & 1);
            if(!role_wait(&empty[st], ph ^ 1u, abort_flag, status, 3)) break;
            const Brick bk = walk.at(kOX, kTY, kTZ);
            mbar_expect_tx(&full[st], (uint32_t)kCopyBytes);
            tma_load_5d(sA + st * kStageBytes, &in_map, 0, bk.x0 - 1, bk.y0 - 1, bk.z0 - 1, bk.b, &full[st]);
        }
        if(*abort_flag)
        {
            // let the loads already issued land before the CTA's shared memory goes away
            for(long k = issued - kStages < 0 ? 0 : issued - kStages; k < issued; ++k)
                mbar_wait(&full[k % kStages], (uint32_t)((k / kStages) & 1));
        }
    }
    else if(warp == 1)
    {
        // ---- MMA issuer: the whole warp walks the loop, one elected lane issues
        const uint64_t bd0 = umma_desc(smem_u32(sW), 128, 256);
        long i = 0;
        for(long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++i)
        {
            const int st = (int)(i % kStages);
            const uint32_t ph = (uint32_t)((i / kStages) & 1);
            const int acc = (int)(i & 1);
            const uint32_t aph = (uint32_t)((i >> 1) & 1);
            const bool ready = role_wait(&tempty[acc], aph ^ 1u, abort_flag, status, 4) &&
                               role_wait(&full[st], ph, abort_flag, status, 5);
            if(!__all_sync(0xffffffffu, ready)) break;
            tc_fence_after();
            // descriptors = base + compile-time offset (the 14-bit start field
            // holds address / 16 and stays below 2^14 for any smem address)
            const uint64_t ad0 = umma_desc_sw32(smem_u32(sA + st * kStageBytes));
            const uint32_t d0 = tmem + (uint32_t)(acc * kAccCols);
            // staged plane q (z = z0 - 1 + q) feeds output planes mt = q - 1 - dz
            // in [lo, hi]; output plane mt takes dz block j = mt - q + 2 of the
            // row shift's 144-row operand.  Output plane q is first written at
            // (q, dy = -1), with the accumulate flag off, by an MMA of its own.
            if(elect_one())
            {
#pragma unroll
                for(int q = 0; q < kTZ + 2; ++q)
                {
                    const int lo = q - 2 < 0 ? 0 : q - 2;
                    const int hi = q < kTZ - 1 ? q : kTZ - 1;
#pragma unroll
                    for(int dyi = 0; dyi < 3; ++dyi)
                    {
                        const int row0 = (q * kHY + dyi) * kTX;
                        const uint64_t ad = ad0 + (uint64_t)((row0 * kRowBytes) >> 4);
                        const uint64_t bs = bd0 + (uint64_t)((dyi * 9 * 512) >> 4);
                        auto mma = [&](int m0, int m1, uint32_t accumulate) {
                            const uint32_t idesc = umma_idesc_bf16(128, (m1 - m0 + 1) * kPlaneCols, false, false);
                            mma_bf16(d0 + m0 * kPlaneCols, ad, bs + (uint64_t)(((m0 - q + 2) * 3 * 512) >> 4), idesc,
                                     accumulate);
                        };
                        if(q <= kTZ - 1 && dyi == 0)
                        {
                            if(hi > lo) mma(lo, hi - 1, 1u);
                            mma(hi, hi, 0u);
                        }
                        else
                        {
                            mma(lo, hi, 1u);
                        }
                    }
                }
                mma_commit(&empty[st]);   // stage free once these MMAs have read it
                mma_commit(&tfull[acc]);  // accumulator ready for the epilogue
            }
            __syncwarp();
        }
        if(*abort_flag && i > 0)
        {
            // MMAs in flight must finish before TMEM is released
            const long k = i - 1;
            mbar_wait(&tfull[k & 1], (uint32_t)((k >> 1) & 1));
        }
    }
    else if(warp >= 2)
    {
        // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31
        const int qd = warp & 3;
        const int m = qd * 32 + lane;
        constexpr int kPlanes = kTZ / 2;
        static_assert(kPlanes == 2 && kPlaneCols == 48, "two planes a warp");
        const int mt0 = (warp - 2) / 4 * kPlanes;  // this warp's output planes of a brick
        const bool wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0;
        long i = 0;
        for(long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, walk.next(), ++i)
        {
            const int acc = (int)(i & 1);
            const uint32_t aph = (uint32_t)((i >> 1) & 1);
            const Brick bk = walk.at(kOX, kTY, kTZ);
            // row m is staged point (xi, yi) of the plane; xi = 0 and kTX - 1
            // are the halo columns
            const int xi = m % kTX;
            const int x = bk.x0 - 1 + xi, y = bk.y0 + m / kTX;
            const bool halo = xi == 0 || xi == kTX - 1;
            // masked output: the row's activations of the whole brick, loaded while
            // its MMAs run (loaded where they are used they cost a memory round
            // trip a plane: 55 us against 27 unmasked on 2 x 64 samples of 16^3)
            uint4 mask[kOut == kOutMaskBf16 ? 2 * kPlanes : 1];
            if constexpr(kOut == kOutMaskBf16)
            {
#pragma unroll
                for(int mt = 0; mt < kPlanes; ++mt)
                {
                    const int z = bk.z0 + mt0 + mt;
                    mask[2 * mt] = mask[2 * mt + 1] = make_uint4(0, 0, 0, 0);
                    if(halo || x >= g.nx || y >= g.ny || z >= g.nz) continue;
                    const uint4* ap = reinterpret_cast<const uint4*>(
                        act + ((((long)bk.b * g.nz + z) * g.ny + y) * g.nx + x) * kNetCh);
                    mask[2 * mt] = __ldg(ap);
                    mask[2 * mt + 1] = __ldg(ap + 1);
                }
            }
            const bool ok = role_wait(&tfull[acc], aph, abort_flag, status, 6);
            if(!__all_sync(0xffffffffu, ok)) break;  // tcgen05.ld is warp-collective
            tc_fence_after();
            // out(x) = D_{dx=-1}[x - 1] + D_{dx=0}[x] + D_{dx=+1}[x + 1]: rows
            // x +- 1 are the neighbouring lanes of the same 16-lane line
            auto finish = [&](int mt, const uint32_t (&d)[48]) {
                float v[16];
#pragma unroll
                for(int c = 0; c < 16; ++c)
                {
                    const float left = __shfl_up_sync(0xffffffffu, __uint_as_float(d[c]), 1);
                    const float right = __shfl_down_sync(0xffffffffu, __uint_as_float(d[32 + c]), 1);
                    v[c] = (left + __uint_as_float(d[16 + c])) + right;
                }
                const int z = bk.z0 + mt0 + mt;
                if(halo || x >= g.nx || y >= g.ny || z >= g.nz) return;
                const long p = (((long)bk.b * g.nz + z) * g.ny + y) * g.nx + x;
                if constexpr(kOut == kOutReluBf16 || kOut == kOutMaskBf16)
                {
                    if constexpr(kOut == kOutReluBf16)
                    {
#pragma unroll
                        for(int c = 0; c < 16; ++c) v[c] = v[c] > 0.f ? v[c] : 0.f;
                    }
                    else
                    {
                        __align__(16) __nv_bfloat16 h[16];
                        *reinterpret_cast<uint4*>(h) = mask[2 * mt];
                        *reinterpret_cast<uint4*>(h + 8) = mask[2 * mt + 1];
#pragma unroll
                        for(int c = 0; c < 16; ++c) v[c] = __bfloat162float(h[c]) > 0.f ? v[c] : 0.f;
                    }
                    uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(out) + p * kNetCh);
                    if(wide) store_point(dst, pack_bf16x8(v), pack_bf16x8(v + 8));
                    else
                    {
                        dst[0] = pack_bf16x8(v);
                        dst[1] = pack_bf16x8(v + 8);
                    }
                }
                else if constexpr(kOut == kOutF32)
                {
                    float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(out) + p * kNetCh);
#pragma unroll
                    for(int c = 0; c < 4; ++c)
                        dst[c] = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
                }
                else
                {
                    reinterpret_cast<float*>(out)[p] = v[0];
                }
            };
            // the second plane's columns on their way while the first is finished
            const uint32_t ta = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(acc * kAccCols + mt0 * kPlaneCols);
            uint32_t d0[48], d1[48];
            tmem_ld48(ta, d0);
            tmem_wait48(d0);
            tmem_ld48(ta + kPlaneCols, d1);
            finish(0, d0);
            __syncwarp();
            tmem_wait48(d1);
            tc_fence_before();
            mbar_arrive(&tempty[acc]);  // the accumulator may take the next brick
            finish(1, d1);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if(warp == 1) tmem_free(tmem, kTmemCols);
}

// ------------------------------------------------------------ layer 3 (16 -> 1)
//
// What bounds it: reading the two branches' activations (64 B a point of the
// odd pair).  The 14 x 8 x 4 bricks, boxes, MMA plan and lane shuffles are the
// 16 -> 16 convolution's with one output channel: a plane's accumulator is a
// group of 16 columns of which dx = -1, 0, +1 take three, and every staged plane q
// and row shift dy is ONE MMA for the 1-3 output planes it feeds (N = 16, 32 or
// 48; 21 a brick, 42 with the pair).  In the odd evaluation the branch of -r
// multiplies the negated weights, both halved, so the accumulator already holds
// (y(r) - y(-r)) / 2.  The epilogue is one small tcgen05.ld and two lane shuffles
// per output plane.  (All 27 taps in N with the sums gathered from shared
// memory, 27 floats a staged point, was bound by that gather: 120 us on an odd
// 128^3 sample; this form takes 52, of it 42 MMAs a brick about 30.  The whole
// network there: 301 -> 216 us; 256^3 learned V-cycle 661 -> 651 us.)
//   warp 0      TMA producer: per brick one (two with the pair) box;
//   warp 1      TMEM owner and MMA issuer, two accumulators of 4 x 16 columns;
//   warps 2-5   epilogue.
constexpr int k3EpiThreads = 128;
constexpr int k3Threads = 64 + k3EpiThreads;
constexpr int k3Stages = 3;
constexpr int k3BoxBytes = kStageBytes;
constexpr int k3StageBytes = 2 * k3BoxBytes;                    // the two branches of the pair
constexpr int k3PlaneCols = 16;                                 // 3 dx and 13 zero columns (MMA N is a multiple of 16)
constexpr int k3AccCols = kTZ * k3PlaneCols;
constexpr int k3TmemCols = 2 * k3AccCols;
constexpr int k3Tile = k3PlaneCols * kRowBytes;                 // 16 columns x 16 channels, K-major
constexpr int k3Tiles = 9;                                      // [dy][dz = +1, 0, -1]
constexpr int k3Smem = k3Stages * k3StageBytes + 2 * k3Tiles * k3Tile + 256 + 1024;
static_assert(kTZ == 4, "tmem_ld4x4 reads the four planes");

static_assert(k3TmemCols == 128, "TMEM allocations are powers of two");
static_assert(k3Smem <= 227 * 1024, "shared memory per CTA");

template <int kOut, bool kPair>
__global__ void __launch_bounds__(k3Threads, 1)
    k_layer3_tc(const __grid_constant__ CUtensorMap in_map, ConvGrid g, const float* __restrict__ w3, float* out,
                PermMap pm, int* status)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* sA = smem;                                       // k3Stages x k3StageBytes
    unsigned char* sW = smem + k3Stages * k3StageBytes;             // + and - weight tiles
    uint64_t* full = (uint64_t*)(sW + 2 * k3Tiles * k3Tile);
    uint64_t* empty = full + k3Stages;
    uint64_t* tfull = empty + k3Stages;
    uint64_t* tempty = tfull + 2;
    uint32_t* tholder = (uint32_t*)(tempty + 2);
    volatile int* abort_flag = (volatile int*)(tholder + 1);

    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    BrickWalk walk(g, kOX, kTY, kTZ, blockIdx.x, gridDim.x);
    const long ntiles = walk.count(g.nb);

    // weight tile (dy, dz): column dx + 1 takes that tap, the others are zero
    for(int i = tid; i < k3Tiles * k3PlaneCols * kNetCh; i += k3Threads)
    {
        const int c = i % kNetCh, col = i / kNetCh % k3PlaneCols, tile = i / (kNetCh * k3PlaneCols);
        float w = 0.f;
        if(col < 3)
        {
            const int t = (2 - tile % 3) * 9 + tile / 3 * 3 + col;
            w = __bfloat162float(__float2bfloat16_rn(w3[(t * kNetCh + c) * kNetCh]));
            if(kPair) w *= 0.5f;  // exact in bf16
        }
        const uint32_t off = (uint32_t)(tile * k3Tile) + kmajor_off(col, c >> 3) + (uint32_t)(c & 7) * 2;
        *reinterpret_cast<__nv_bfloat16*>(sW + off) = __float2bfloat16_rn(w);
        *reinterpret_cast<__nv_bfloat16*>(sW + k3Tiles * k3Tile + off) = __float2bfloat16_rn(-w);
    }
    if(tid == 0)
    {
        for(int s = 0; s < k3Stages; ++s)
        {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for(int a = 0; a < 2; ++a)
        {
            mbar_init(&tfull[a], 1);
            mbar_init(&tempty[a], k3EpiThreads);
        }
        *abort_flag = 0;
    }
    if(warp == 1) tmem_alloc(tholder, k3TmemCols);
    fence_async_smem();  // the weights are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tholder;
    pdl_launch_dependents();  // not before this CTA has its tensor memory
    pdl_wait();  // from here on the previous kernel's output is read
    constexpr uint32_t kBoxTx = (uint32_t)kCopyBytes * (kPair ? 2u : 1u);

    if(warp == 0 && lane == 0)
    {
        // ---- TMA producer
        long issued = 0;
        for(long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, walk.next(), ++issued)
        {
            const int st = (int)(issued % k3Stages);
            const uint32_t ph = (uint32_t)((issued / k3Stages) & 1);
            if(!role_wait(&empty[st], ph ^ 1u, abort_flag, status, 3)) break;
            const Brick bk = walk.at(kOX, kTY, kTZ);
            mbar_expect_tx(&full[st], kBoxTx);
            unsigned char* dst = sA + st * k3StageBytes;
            tma_load_5d(dst, &in_map, 0, bk.x0 - 1, bk.y0 - 1, bk.z0 - 1, bk.b, &full[st]);
            if(kPair)
                tma_load_5d(dst + k3BoxBytes, &in_map, 0, bk.x0 - 1, bk.y0 - 1, bk.z0 - 1, bk.b + g.nb, &full[st]);
        }
        if(*abort_flag)
        {
            // let the loads already issued land before the CTA's shared memory goes away
            for(long k = issued - k3Stages < 0 ? 0 : issued - k3Stages; k < issued; ++k)
                mbar_wait(&full[k % k3Stages], (uint32_t)((k / k3Stages) & 1));
        }
    }
    else if(warp == 1)
    {
        // ---- MMA issuer: the whole warp walks the loop, one elected lane issues
        const uint64_t bd = umma_desc(smem_u32(sW), 128, 256);
        long i = 0;
        for(long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++i)
        {
            const int st = (int)(i % k3Stages);
            const uint32_t ph = (uint32_t)((i / k3Stages) & 1);
            const int acc = (int)(i & 1);
            const uint32_t aph = (uint32_t)((i >> 1) & 1);
            const bool ready = role_wait(&tempty[acc], aph ^ 1u, abort_flag, status, 4) &&
                               role_wait(&full[st], ph, abort_flag, status, 5);
            if(!__all_sync(0xffffffffu, ready)) break;
            tc_fence_after();
            const uint64_t a0 = umma_desc_sw32(smem_u32(sA + st * k3StageBytes));
            const uint32_t d0 = tmem + (uint32_t)(acc * k3AccCols);
            // as in k_conv16: plane q feeds output planes mt in [lo, hi] with dz
            // tile mt - q + 2, and first writes plane q by an MMA of its own
            if(elect_one())
            {
#pragma unroll
                for(int q = 0; q < kTZ + 2; ++q)
                {
                    const int lo = q - 2 < 0 ? 0 : q - 2;
                    const int hi = q < kTZ - 1 ? q : kTZ - 1;
#pragma unroll
                    for(int dyi = 0; dyi < 3; ++dyi)
                    {
                        const uint64_t ad = a0 + (uint64_t)(((q * kHY + dyi) * kTX * kRowBytes) >> 4);
                        auto mma = [&](int m0, int m1, uint32_t accumulate) {
                            const uint32_t idesc = umma_idesc_bf16(128, (m1 - m0 + 1) * k3PlaneCols, false, false);
                            const uint64_t bs = bd + (uint64_t)(((dyi * 3 + m0 - q + 2) * k3Tile) >> 4);
                            const uint32_t d = d0 + (uint32_t)(m0 * k3PlaneCols);
                            mma_bf16(d, ad, bs, idesc, accumulate);
                            if(kPair)
                                mma_bf16(d, ad + (uint64_t)(k3BoxBytes >> 4), bs + (uint64_t)((k3Tiles * k3Tile) >> 4),
                                         idesc, 1u);
                        };
                        if(q <= kTZ - 1 && dyi == 0)
                        {
                            if(hi > lo) mma(lo, hi - 1, 1u);
                            mma(hi, hi, 0u);
                        }
                        else
                        {
                            mma(lo, hi, 1u);
                        }
                    }
                }
                mma_commit(&empty[st]);   // stage free once these MMAs have read it
                mma_commit(&tfull[acc]);  // accumulator ready for the epilogue
            }
            __syncwarp();
        }
        if(*abort_flag && i > 0)
        {
            // MMAs in flight must finish before TMEM is released
            const long k = i - 1;
            mbar_wait(&tfull[k & 1], (uint32_t)((k >> 1) & 1));
        }
    }
    else if(warp >= 2)
    {
        // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31
        const int qd = warp & 3;
        const int m = qd * 32 + lane;
        long i = 0;
        for(long tile = blockIdx.x; tile < ntiles; tile += gridDim.x, walk.next(), ++i)
        {
            const int acc = (int)(i & 1);
            const uint32_t aph = (uint32_t)((i >> 1) & 1);
            const bool ok = role_wait(&tfull[acc], aph, abort_flag, status, 6);
            if(!__all_sync(0xffffffffu, ok)) break;  // tcgen05.ld is warp-collective
            tc_fence_after();
            float v[kTZ][4];
            tmem_ld4x4(tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(acc * k3AccCols), k3PlaneCols, v);
            tc_fence_before();
            mbar_arrive(&tempty[acc]);  // the accumulator may take the next brick
            const Brick bk = walk.at(kOX, kTY, kTZ);
            // row m is staged point (xi, yi) of a plane; xi = 0 and kTX - 1 are the halo columns
            const int xi = m % kTX;
            const int x = bk.x0 - 1 + xi, y = bk.y0 + m / kTX;
            const bool halo = xi == 0 || xi == kTX - 1;
#pragma unroll
            for(int mt = 0; mt < kTZ; ++mt)
            {
                // out(x) = D_{dx=-1}[x - 1] + D_{dx=0}[x] + D_{dx=+1}[x + 1]
                const float left = __shfl_up_sync(0xffffffffu, v[mt][0], 1);
                const float right = __shfl_down_sync(0xffffffffu, v[mt][2], 1);
                const float sum = (left + v[mt][1]) + right;
                const int z = bk.z0 + mt;
                if(halo || x >= g.nx || y >= g.ny || z >= g.nz) continue;
                if constexpr(kOut == 2)
                {
                    out[(((long)bk.b * g.nz + z) * g.ny + y) * g.nx + x] = sum;
                }
                else
                {
                    float* xo = out + perm_row(pm, z, y, x);
                    if constexpr(kOut == 1) *xo += sum;
                    else *xo = sum;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if(warp == 1) tmem_free(tmem, k3TmemCols);
}

// ------------------------------------------------------------ weight gradient

// What bounds it: an im2col operand would write every point's 16 channels to
// shared memory 27 times (64 points by 27 taps per MMA block, gathered with
// their index arithmetic: 452 us on 2 x 64 samples of 16^3).  Here both
// operands are plain bricks of points, MN-major, and a tap is a start address.
// With x contiguous in shared memory ([plane][line][8-channel half][x], 16 B a
// point) a descriptor's K direction runs along x, and its M (N) direction steps
// uniformly over (line, half): one MMA multiplies five lines of the input (M =
// (line, channel), 80 of 128 rows used, the rest reads the bytes behind and is
// ignored) with the three lines of each gradient plane it meets (N = (plane,
// line, channel) = 144) over 16 x, for one dx: the start x of A.  The three column
// blocks of a dx are the dz taps, the (line, line) pairs one apart the dy taps,
// summed at the end; the nine blocks take 432 TMEM columns.  (One MMA per (dz, dx)
// with N = 48 takes 53 cycles, N = 144 takes 75: 3800 -> 2000 cycles a unit.)  A
// CTA walks units of 3 lines x 16 x x 8 planes: eight warps fetch units into a
// ring of three stages, two units on their way in registers (one: 2600 cycles a
// unit, the bound with this plan; cp.async straight into the ring was slower
// still, 5000), a ninth issues the MMAs from one elected lane.  2 x 64 samples of
// 16^3, with the reduction: 41.6 -> 33.4 us, four times as many 104 -> 77.  A
// gradient step of 64 samples: im2col 1572 us, bricks 361, with the warps' split
// 299, 266 with the one-channel forms of layers 1 and 3, with this plan 244.
constexpr int kWgX = 16, kWgLines = 3, kWgZ = 8;                  // gradient points of a unit
constexpr int kWgXA = kWgX + 2, kWgLinesA = kWgLines + 2, kWgZA = kWgZ + 2;  // input points, with the halo
constexpr int kWgRowA = kWgXA * 16, kWgRowB = kWgX * 16;          // bytes of one line of one half
constexpr int kWgPlaneA = kWgLinesA * 2 * kWgRowA, kWgPlaneB = kWgLines * 2 * kWgRowB;
constexpr int kWgN = kWgLines * kNetCh;                           // 48 columns per (dz, dx)
constexpr int kWgOffB = kWgZA * kWgPlaneA;
constexpr int kWgStage = kWgOffB + kWgZ * kWgPlaneB;
constexpr int kWgThreads = 256;                                   // loaders (and one warp that issues the MMAs)
constexpr int kWgItemsA = kWgZA * kWgLinesA * kWgXA * 2, kWgItemsB = kWgZ * kWgLines * kWgX * 2;  // 16 B each
constexpr int kWgLoadsA = (kWgItemsA + kWgThreads - 1) / kWgThreads;
constexpr int kWgLoadsB = (kWgItemsB + kWgThreads - 1) / kWgThreads;
constexpr int kWgLoads = kWgLoadsA + kWgLoadsB;
constexpr int kWgStages = 3;
constexpr int kWgSmem = kWgStages * kWgStage + 128;
static_assert(9 * kWgN <= 512 && kWgStage % 128 == 0, "accumulators and stages");
// the last plane's A operand reads 16 halves and two 8-point groups from its start
static_assert((kWgZA - 1) * kWgPlaneA + 15 * kWgRowA + 256 + 32 <= kWgStage, "A reads stay in the stage");
static_assert(kNetLayerWeights * 4 <= kWgStage, "the sums fit a stage");

struct WgUnits
{
    int tx, ty, tz;
    long count;
};

__host__ __device__ inline WgUnits wg_units(const ConvGrid& g)
{
    const int tx = (g.nx + kWgX - 1) / kWgX, ty = (g.ny + kWgLines - 1) / kWgLines, tz = (g.nz + kWgZ - 1) / kWgZ;
    return WgUnits{tx, ty, tz, (long)g.nb * tz * ty * tx};
}

__global__ void __launch_bounds__(kWgThreads + 32, 1)
    k_conv16_wgrad(ConvGrid g, const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ gr,
                   float* __restrict__ partial, int* status)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
    __shared__ uint64_t full[kWgStages], empty[kWgStages], finished;
    __shared__ uint32_t tholder;
    __shared__ int gave_up;
    volatile int* abort_flag = &gave_up;

    const int tid = threadIdx.x;
    const int warp = tid >> 5;
    const WgUnits U = wg_units(g);

    if(tid == 0)
    {
        for(int k = 0; k < kWgStages; ++k)
        {
            mbar_init(&full[k], kWgThreads);
            mbar_init(&empty[k], 1);
        }
        mbar_init(&finished, 1);
        gave_up = 0;
    }
    if(warp == 0) tmem_alloc(&tholder, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tholder;

    if(tid < kWgThreads)
    {
        // ---- loaders: a thread's 16-byte items (plane, line, x, half) are the same in every
        // unit; zero outside the sample.  Two units are on their way in registers.
        long at[kWgLoads];  // element, from the halo's corner
        int to[kWgLoads], where[kWgLoads];  // byte of the stage; x | y << 8 | z << 16
#pragma unroll
        for(int j = 0; j < kWgLoads; ++j)
        {
            const bool in_a = j < kWgLoadsA;
            const int i = tid + (in_a ? j : j - kWgLoadsA) * kWgThreads, q = i >> 1, half = i & 1;
            const int wide = in_a ? kWgXA : kWgX, lines = in_a ? kWgLinesA : kWgLines, halo = in_a ? 0 : 1;
            const int line = q / wide, px = q % wide + halo, py = line % lines + halo, pz = line / lines + halo;
            to[j] = i >= (in_a ? kWgItemsA : kWgItemsB)
                        ? -1
                        : (in_a ? 0 : kWgOffB) + (line * 2 + half) * (in_a ? kWgRowA : kWgRowB) + q % wide * 16;
            where[j] = px | py << 8 | pz << 16;
            at[j] = (((long)pz * g.ny + py) * g.nx + px) * kNetCh + half * 8;
        }
        BrickWalk walk(g, kWgX, kWgLines, kWgZ, blockIdx.x, gridDim.x);
        long next = blockIdx.x;  // unit the walk is at
        auto load = [&](uint4 (&v)[kWgLoads]) {
            if(next >= U.count) return;
            const Brick bk = walk.at(kWgX, kWgLines, kWgZ);
            const long corner =
                ((((long)bk.b * g.nz + bk.z0 - 1) * g.ny + bk.y0 - 1) * g.nx + bk.x0 - 1) * kNetCh;
#pragma unroll
            for(int j = 0; j < kWgLoads; ++j)
            {
                const int xx = bk.x0 - 1 + (where[j] & 255), y = bk.y0 - 1 + (where[j] >> 8 & 255),
                          z = bk.z0 - 1 + (where[j] >> 16);
                const bool in = to[j] >= 0 && (unsigned)xx < (unsigned)g.nx && (unsigned)y < (unsigned)g.ny &&
                                (unsigned)z < (unsigned)g.nz;
                v[j] = make_uint4(0, 0, 0, 0);
                if(in) v[j] = __ldg(reinterpret_cast<const uint4*>((j < kWgLoadsA ? x : gr) + corner + at[j]));
            }
            walk.next();
            next += gridDim.x;
        };
        int k = 0;
        // unit k from v into its stage, then unit k + 2 on its way into v
        auto step = [&](uint4 (&v)[kWgLoads]) {
            const int st = k % kWgStages;
            // the MMAs that read this stage kWgStages units ago
            if(!role_wait(&empty[st], (uint32_t)((k / kWgStages) & 1) ^ 1u, abort_flag, status, 2)) return false;
            unsigned char* sA = smem + st * kWgStage;
#pragma unroll
            for(int j = 0; j < kWgLoads; ++j)
                if(to[j] >= 0) *reinterpret_cast<uint4*>(sA + to[j]) = v[j];
            fence_async_smem();
            mbar_arrive(&full[st]);
            load(v);
            ++k;
            return true;
        };
        uint4 even[kWgLoads], odd[kWgLoads];
        load(even);
        load(odd);
        for(long u = blockIdx.x; u < U.count; u += 2 * (long)gridDim.x)
        {
            if(!step(even)) break;
            if(u + gridDim.x < U.count && !step(odd)) break;
        }
    }
    else
    {
        // ---- MMA issuer: the whole warp walks the loop, one elected lane issues
        int k = 0;
        for(long u = blockIdx.x; u < U.count; u += gridDim.x, ++k)
        {
            const int st = k % kWgStages;
            const bool there = role_wait(&full[st], (uint32_t)((k / kWgStages) & 1), abort_flag, status, 2);
            if(!__all_sync(0xffffffffu, there)) break;
            tc_fence_after();
            const uint64_t ad = umma_desc(smem_u32(smem + st * kWgStage), 128, kWgRowA);
            const uint64_t bd = umma_desc(smem_u32(smem + st * kWgStage + kWgOffB), 128, kWgRowB);
            if(elect_one())
            {
                // input plane q meets gradient planes q - 2 .. q, column block j the
                // plane q - 2 + j (dz = 1 - j); a plane with all three goes first, it
                // starts the accumulators
#pragma unroll
                for(int i = 0; i < kWgZA; ++i)
                {
                    const int q = (i + 2) % kWgZA;
                    const int lo = q < 2 ? 2 - q : 0, hi = q > kWgZ - 1 ? kWgZ + 1 - q : 2;
                    const uint32_t idesc = umma_idesc_bf16(128, (hi - lo + 1) * kWgN, true, true);
#pragma unroll
                    for(int t = 0; t < 3; ++t)
                        mma_bf16(tmem + (uint32_t)((3 * t + lo) * kWgN), ad + (uint64_t)((q * kWgPlaneA + t * 16) >> 4),
                                 bd + (uint64_t)(((q - 2 + lo) * kWgPlaneB) >> 4), idesc, (k == 0 && i == 0) ? 0u : 1u);
                }
                mma_commit(&empty[st]);
            }
            __syncwarp();
        }
        // every MMA issued (also after a time-out: they finish before the CTA leaves)
        if(elect_one()) mma_commit(&finished);
        __syncwarp();
    }
    if(!mbar_wait(&finished, 0)) *abort_flag = 1;
    __syncthreads();
    const bool ok = *abort_flag == 0;
    if(!ok && tid == 0) atomicExch(status, 2);
    tc_fence_after();

    // accumulator row = (input line yy, channel), column group r = gradient line: dy = yy - 1 - r
    float* sums = reinterpret_cast<float*>(smem);
    for(int i = tid; i < kNetLayerWeights; i += blockDim.x) sums[i] = 0.f;
    __syncthreads();
    for(int r = 0; r < kWgLines; ++r)
    {
        if(warp < 3)  // lanes 0..79 hold the five input lines
        {
            const int yy = tid >> 4, ci = tid & 15, dy = yy - 1 - r;
            for(int t = 0; t < 9; ++t)
            {
                float v[16];
                // t = 3 (dz + 1) + (dx + 1)
                const int block = 3 * (t % 3) + 2 - t / 3;
                tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(block * kWgN + r * kNetCh), v);
                if(yy < kWgLinesA && dy >= -1 && dy <= 1)
                {
                    // [tap][co][ci]: the lanes of a line on consecutive words
                    float* d = sums + (t / 3 * 9 + (dy + 1) * 3 + t % 3) * kNetCh * kNetCh + ci;
#pragma unroll
                    for(int c = 0; c < 16; ++c) d[c * kNetCh] += v[c];
                }
            }
        }
        __syncthreads();
    }
    float* dst = partial + (size_t)blockIdx.x * kNetLayerWeights;
    for(int i = tid; i < kNetLayerWeights; i += blockDim.x)
        dst[i] = ok ? sums[(i & ~255) | ((i & 15) << 4) | ((i >> 4) & 15)] : 0.f;
    tc_fence_before();
    __syncthreads();
    if(warp == 0) tmem_free(tmem, 512);
}

// dw = the CTAs' partial sums: eight groups of them per output, then the
// groups in order (a thread per output over all partials: 22 us).
constexpr int kWgReduceGroups = 8;

__global__ void __launch_bounds__(256) k_wgrad_reduce(int nparts, const float* __restrict__ partial,
                                                      float* __restrict__ dw)
{
    __shared__ float red[kWgReduceGroups][32];
    const int o = threadIdx.x & 31, grp = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + o;
    float s = 0.f;
#pragma unroll 4
    for(int c = grp; c < nparts; c += kWgReduceGroups) s += partial[(size_t)c * kNetLayerWeights + i];
    red[grp][o] = s;
    __syncthreads();
    if(grp) return;
#pragma unroll
    for(int k = 1; k < kWgReduceGroups; ++k) s += red[k][o];
    dw[i] = s;
}
static_assert(kNetLayerWeights % 32 == 0, "reduction blocks");

// ------------------------------------------------------------ small kernels

// w[tap][ci][co] (FP32) -> per-tap K-major B operand (N = co rows, K = ci).
// flip != 0: W'[t][ci'][co'] = W[26-t][co'][ci'] (transposed convolution).
__global__ void k_prepare_weights(const float* __restrict__ w, __nv_bfloat16* __restrict__ wB, int flip)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= kNetLayerWeights) return;
    const int t = i / 256, nn = (i / 16) % 16, kk = i % 16;
    const float v = flip ? w[((26 - t) * 16 + nn) * 16 + kk] : w[(t * 16 + kk) * 16 + nn];
    unsigned char* base = reinterpret_cast<unsigned char*>(wB) + weight_slot(t) * 512;
    *reinterpret_cast<__nv_bfloat16*>(base + kmajor_off(nn, kk >> 3) + (kk & 7) * 2) = __float2bfloat16_rn(v);
}

__device__ __forceinline__ void store_embed(__nv_bfloat16* a, long p, float r0)
{
    const float v[8] = {r0, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    store_point(a + p * kNetCh, pack_bf16x8(v), make_uint4(0, 0, 0, 0));
}

// Natural <-> colour-permuted copies of a level vector (training-pair set-up).
template <typename Tin, typename Tout, bool kToNatural>
__global__ void k_perm_copy(PermMap pm, int nz, int ny, int nx, const Tin* __restrict__ in, Tout* __restrict__ out)
{
    const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= (long)nz * ny * nx) return;
    const int z = (int)(p / ((long)ny * nx));
    const long rem = p - (long)z * ny * nx;
    const int y = (int)(rem / nx), x = (int)(rem - (long)y * nx);
    const int row = perm_row(pm, z, y, x);
    if(kToNatural) out[p] = (Tout)in[row];
    else out[row] = (Tout)in[p];
}

// 1 / sum e^2 (one block, FP64 accumulation).
__global__ void k_inv_sumsq(long n, const float* __restrict__ e, float* __restrict__ out)
{
    __shared__ double red[32];
    double s = 0.0;
    for(long i = threadIdx.x; i < n; i += blockDim.x) s += (double)e[i] * e[i];
    s = block_sum(s, red);
    if(threadIdx.x == 0) *out = (float)(1.0 / s);
}

// Sum of a step's loss partials into acc (one block, fixed order).
__global__ void k_loss_accumulate(int parts, const float* __restrict__ partial, double* __restrict__ acc)
{
    __shared__ double red[32];
    double s = 0.0;
    for(int i = threadIdx.x; i < parts; i += blockDim.x) s += partial[i];
    s = block_sum(s, red);
    if(threadIdx.x == 0) *acc += s;
}

// b ~ N(0,1) by natural row id: SplitMix64 finalizer over (key + 2i, key + 2i + 1)
// with key = mix(seed), 53-bit uniforms u1 in (0,1], u2 in [0,1), Box-Muller
// sqrt(-2 ln u1) cos(2 pi u2).  Stored at out[perm[i]] (perm may be null).
__device__ __forceinline__ unsigned long long splitmix(unsigned long long z)
{
    z += 0x9E3779B97F4A7C15ULL;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

__global__ void k_normal_rhs(long long m, unsigned long long seed, const int* __restrict__ perm, double* out64,
                             float* out32)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= m) return;
    const unsigned long long key = splitmix(seed);
    const unsigned long long a = splitmix(key + 2ULL * (unsigned long long)i);
    const unsigned long long b = splitmix(key + 2ULL * (unsigned long long)i + 1ULL);
    const double u1 = ((double)(a >> 11) + 1.0) * (1.0 / 9007199254740992.0);
    const double u2 = (double)(b >> 11) * (1.0 / 9007199254740992.0);
    const double v = sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
    const long long o = perm ? perm[i] : i;
    if(out64) out64[o] = v;
    if(out32) out32[o] = (float)v;
}

__global__ void k_embed_f32(long n, const float* __restrict__ r, __nv_bfloat16* __restrict__ a, int pair)
{
    const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= n) return;
    store_embed(a, p, r[p]);
    if(pair) store_embed(a, p + n, -r[p]);
}

// 27-point stencil (diagonal 26, off-diagonals -1, zero outside the sample's grid).
__device__ __forceinline__ float stencil_at(const ConvGrid& g, const float* __restrict__ v, long p)
{
    const long per = (long)g.nz * g.ny * g.nx;
    const long b = p / per;
    const long q = p - b * per;
    const int z = (int)(q / ((long)g.ny * g.nx));
    const long rem = q - (long)z * g.ny * g.nx;
    const int y = (int)(rem / g.nx), x = (int)(rem - (long)y * g.nx);
    const float* vb = v + b * per;
    float off = 0.f;
#pragma unroll
    for(int t = 0; t < 27; ++t)
    {
        const int z2 = z + t / 9 - 1, y2 = y + (t / 3) % 3 - 1, x2 = x + t % 3 - 1;
        if(t != 13 && z2 >= 0 && z2 < g.nz && y2 >= 0 && y2 < g.ny && x2 >= 0 && x2 < g.nx)
            off += vb[((long)z2 * g.ny + y2) * g.nx + x2];
    }
    return 26.f * v[p] - off;
}

// Bf16 scalar field of a level: r (x == nullptr), or the residual r - A x of the
// 27-point stencil (diagonal diag32, off-diagonals -1), read from colour-permuted
// level vectors at natural point p.
__global__ void k_embed_scalar_level(PermMap pm, int nz, int ny, int nx, const float* __restrict__ r,
                                     const float* __restrict__ x, const float* __restrict__ diag32,
                                     __nv_bfloat16* __restrict__ s1)
{
    pdl_begin();
    const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if(p >= (long)nz * ny * nx) return;
    const int z = (int)(p / ((long)ny * nx));
    const long rem = p - (long)z * ny * nx;
    const int y = (int)(rem / nx), xx = (int)(rem - (long)y * nx);
    const int row = perm_row(pm, z, y, xx);
    float v = r[row];
    if(x)
    {
        float off = 0.f;
#pragma unroll
        for(int t = 0; t < 27; ++t)
        {
            const int z2 = z + t / 9 - 1, y2 = y + (t / 3) % 3 - 1, x2 = xx + t % 3 - 1;
            if(t != 13 && z2 >= 0 && z2 < nz && y2 >= 0 && y2 < ny && x2 >= 0 && x2 < nx)
                off += x[perm_row(pm, z2, y2, x2)];
        }
        v = v - (diag32[row] * x[row] - off);
    }
    s1[p] = __float2bfloat16_rn(v);
}

__device__ __forceinline__ float in_value(const __nv_bfloat16* v, long q) { return __bfloat162float(v[q]); }
__device__ __forceinline__ float in_value(const float* v, long q) { return __bfloat162float(__float2bfloat16_rn(v[q])); }


// ------------------------------------------------------------ layer 1 (1 -> 16)
//
// One input channel: the 27 taps are the K dimension, of two MMAs per plane of a
// 16 x 8 x 4 brick (M = 128 points, N = 16 channels, K = 16 each, 5 zero taps).
// What bounds it: it has 64 B a point of the odd pair to write; gathering every
// point's 27 neighbours from a staged field and rounding each again cost 57 us on
// a 128^3 sample.  Here A is MN-major: eight points along x are the 16 bytes of
// one tap.  A thread reads ten points of one line of the halo'd brick, rounds
// them once, and the three shifted runs of eight (dx = -1, 0, +1) are stored for
// each of the up to nine (dz, dy) the line serves: 27 16-byte stores, 216 values
// of the operand from ten points read.  Tap runs of an 8-point group are contiguous (K core matrices 128 B
// apart), groups 528 B apart, which spreads a store over all banks.  The
// epilogue writes relu(z) and, for the odd pair, relu(-z) as BF16, a point's 32
// bytes at a time (in two halves the stores were the bound: the new gather alone
// gained 1 us, with whole points 45).  The next brick's points are on their way
// meanwhile, and several CTAs per SM overlap.
constexpr int k1X = 16, k1Y = 8, k1Z = 4;
constexpr int k1Threads = 128;               // one thread per point of a plane
constexpr int k1Lines = 2 * (k1Y + 2) * (k1Z + 2);  // (plane, line, 8-point half) of the halo'd brick: a thread each
constexpr int k1K = 32;                      // 27 taps + 5 zeros
constexpr int k1Group = k1K * 16 + 16;       // bytes of an 8-point group
constexpr int k1PlaneBytes = 16 * k1Group;
constexpr int k1Cols = k1Z * kNetCh;         // TMEM columns per brick
constexpr int k1WBytes = kNetCh * k1K * 2;   // B: 16 channel rows x 32 taps
constexpr int k1Smem = k1Z * k1PlaneBytes + k1WBytes + 128;
constexpr int k1CtasPerSm = 6;

static_assert(k1X * k1Y == k1Threads && k1X == 16, "one plane of the brick is one 128-row M tile");
static_assert(k1Lines <= k1Threads, "a thread per staged line");
static_assert(k1Cols * k1CtasPerSm <= 512, "TMEM columns of the co-resident CTAs");
static_assert(k1CtasPerSm * (k1Smem + 1024) <= 227 * 1024, "shared memory of the co-resident CTAs");

// K-major no-swizzle offset of row r, 8-element K chunk c8 of the weights' 32-wide
// K: chunks 128 B apart (LBO), 8-row groups 512 B apart (SBO).
__host__ __device__ constexpr uint32_t k1_off(int r, int c8)
{
    return (uint32_t)((r >> 3) * 512 + c8 * 128 + (r & 7) * 16);
}

// kMask: the gradient of layer 3 instead.  in is dL/dy (one value a point, the
// second branch's being its negative), w1 are layer 3's weights, used transposed,
// and the result is kept where act > 0.  (As a 16 -> 16 convolution of dL/dy with
// 15 zero channels: 30 us on 2 x 64 samples of 16^3, here 18.)
template <typename Tin, bool kPair, bool kMask>
__global__ void __launch_bounds__(k1Threads, k1CtasPerSm)
    k_layer1_tc(ConvGrid g, const Tin* __restrict__ in, const float* __restrict__ w1, __nv_bfloat16* __restrict__ a1,
                const __nv_bfloat16* __restrict__ act, int* status)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
    unsigned char* sA = smem;                     // k1Z planes of tap runs
    unsigned char* sW = sA + k1Z * k1PlaneBytes;  // weights
    __shared__ uint64_t mbar;
    __shared__ uint32_t tholder;

    const int tid = threadIdx.x, warp = tid >> 5;
    for(int i = tid; i < kNetCh * k1K; i += k1Threads)
    {
        const int co = i / k1K, t = i % k1K;
        // w1[t][0][co], or w3[26 - t][co][0]
        const int at = kMask ? (26 - t) * kNetCh * kNetCh + co * kNetCh : t * kNetCh * kNetCh + co;
        const float w = t < 27 ? w1[at] : 0.f;
        *reinterpret_cast<__nv_bfloat16*>(sW + k1_off(co, t >> 3) + (t & 7) * 2) = __float2bfloat16_rn(w);
    }
    // the zero taps stay
    for(int i = tid; i < k1Z * 16 * (k1K - 27); i += k1Threads)
        *reinterpret_cast<uint4*>(sA + i / (k1K - 27) * k1Group + (27 + i % (k1K - 27)) * 16) = make_uint4(0, 0, 0, 0);
    if(tid == 0) mbar_init(&mbar, 1);
    if(warp == 0) tmem_alloc(&tholder, k1Cols);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tholder;
    pdl_launch_dependents();  // not before this CTA has its tensor memory
    pdl_wait();  // from here on the previous kernel's output is read

    const long n = g.points();
    BrickWalk walk(g, k1X, k1Y, k1Z, blockIdx.x, gridDim.x);
    const long ntiles = walk.count(g.nb);
    constexpr uint32_t idesc = umma_idesc_bf16(128, kNetCh, true, false);
    const uint64_t ad = umma_desc(smem_u32(sA), 128, k1Group), bd = umma_desc(smem_u32(sW), 128, 512);
    const int mx = tid % k1X, my = tid / k1X;                           // this thread's point of each plane
    const int half = tid & 1, hy = (tid >> 1) % (k1Y + 2), hz = (tid >> 1) / (k1Y + 2);  // and staged line

    // points x0 + 8 half - 1 .. + 8 of the line, zero outside the sample
    float v[10];
    auto load = [&] {
        const Brick bk = walk.at(k1X, k1Y, k1Z);
        const int x = bk.x0 + 8 * half - 1, y = bk.y0 + hy - 1, z = bk.z0 + hz - 1;
        const bool line = tid < k1Lines && (unsigned)y < (unsigned)g.ny && (unsigned)z < (unsigned)g.nz;
        const long at = (((long)bk.b * g.nz + z) * g.ny + y) * g.nx + x;
#pragma unroll
        for(int i = 0; i < 10; ++i)
            v[i] = line && (unsigned)(x + i) < (unsigned)g.nx ? in_value(in, at + i) : 0.f;
    };
    load();
    uint32_t phase = 0;
    bool ok = true;
    for(long tile = blockIdx.x; tile < ntiles; tile += gridDim.x)
    {
        if(tid < k1Lines)
        {
            uint32_t p[5], q[4];  // pairs (0,1) (2,3) .. and (1,2) (3,4) ..
#pragma unroll
            for(int i = 0; i < 5; ++i) p[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
#pragma unroll
            for(int i = 0; i < 4; ++i) q[i] = pack_bf16x2(v[2 * i + 1], v[2 * i + 2]);
#pragma unroll
            for(int dz = 0; dz < 3; ++dz)
#pragma unroll
                for(int dy = 0; dy < 3; ++dy)
                {
                    // the output plane and line whose tap (dz - 1, dy - 1) this line is
                    const int oz = hz - dz, oy = hy - dy;
                    if((unsigned)oz >= (unsigned)k1Z || (unsigned)oy >= (unsigned)k1Y) continue;
                    uint4* run = reinterpret_cast<uint4*>(sA + oz * k1PlaneBytes + (2 * oy + half) * k1Group) +
                                 dz * 9 + dy * 3;
                    run[0] = make_uint4(p[0], p[1], p[2], p[3]);
                    run[1] = make_uint4(q[0], q[1], q[2], q[3]);
                    run[2] = make_uint4(p[1], p[2], p[3], p[4]);
                }
        }
        fence_async_smem();  // the runs are read by the tensor cores
        tc_fence_before();
        if(__syncthreads_or(!ok)) break;
        tc_fence_after();
        if(warp == 0 && elect_one())
        {
#pragma unroll
            for(int z = 0; z < k1Z; ++z)
#pragma unroll
                for(int kh = 0; kh < 2; ++kh)
                    mma_bf16(tmem + z * kNetCh, ad + (uint64_t)((z * k1PlaneBytes + kh * 256) >> 4),
                             bd + (uint64_t)((kh * 256) >> 4), idesc, (uint32_t)kh);
            mma_commit(&mbar);
        }
        __syncwarp();
        const Brick bk = walk.at(k1X, k1Y, k1Z);
        walk.next();
        if(tile + gridDim.x < ntiles) load();
        ok = __all_sync(0xffffffffu, mbar_wait(&mbar, phase));
        if(!ok) continue;  // the block leaves together
        phase ^= 1u;
        tc_fence_after();
        const int x = bk.x0 + mx, y = bk.y0 + my;
        const long row = (((long)bk.b * g.nz + bk.z0) * g.ny + y) * g.nx + x;
#pragma unroll 1
        for(int z = 0; z < k1Z; ++z)
        {
            const bool inside = x < g.nx && y < g.ny && bk.z0 + z < g.nz;
            const long pt = row + (long)z * g.ny * g.nx;
            uint4 m[kMask ? 4 : 1];
            if constexpr(kMask)
            {
#pragma unroll
                for(int i = 0; i < (kPair ? 4 : 2); ++i)
                    m[i] = inside ? __ldg(reinterpret_cast<const uint4*>(act + (pt + (i >> 1) * n) * kNetCh) + (i & 1))
                                  : make_uint4(0, 0, 0, 0);
            }
            float s[16];
            tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(z * kNetCh), s);
            if(inside)
            {
#pragma unroll
                for(int br = 0; br < (kPair ? 2 : 1); ++br)
                {
                    float o[16];
                    __align__(16) __nv_bfloat16 h[kMask ? 16 : 8];
                    if constexpr(kMask)
                    {
                        *reinterpret_cast<uint4*>(h) = m[2 * br];
                        *reinterpret_cast<uint4*>(h + 8) = m[2 * br + 1];
                    }
#pragma unroll
                    for(int c = 0; c < 16; ++c)
                    {
                        const float v = br ? -s[c] : s[c];
                        if constexpr(kMask) o[c] = __bfloat162float(h[c]) > 0.f ? v : 0.f;
                        else o[c] = fmaxf(v, 0.f);
                    }
                    store_point(a1 + (pt + br * n) * kNetCh, pack_bf16x8(o), pack_bf16x8(o + 8));
                }
            }
            __syncwarp();
        }
    }
    tc_fence_before();
    const bool failed = __syncthreads_or(!ok);
    if(failed)
    {
        if(tid == 0) atomicExch(status, 7);
        if(!ok) mbar_wait(&mbar, phase);  // the MMAs in flight finish before TMEM is released
        __syncthreads();
    }
    tc_fence_after();
    if(warp == 0) tmem_free(tmem, k1Cols);
}

// 1 / (e.e) (kind 0) or 1 / (e.Ae) (kind 1) per sample: one block per sample.
__global__ void k_sample_norm(ConvGrid g, const float* __restrict__ e, int kind, float* __restrict__ out)
{
    __shared__ double red[32];
    const long per = (long)g.nz * g.ny * g.nx;
    const long base = (long)blockIdx.x * per;
    double s = 0.0;
    for(long i = threadIdx.x; i < per; i += blockDim.x)
    {
        const float ev = e[base + i];
        s += (double)ev * (kind ? stencil_at(g, e, base + i) : ev);
    }
    s = block_sum(s, red);
    if(threadIdx.x == 0) out[blockIdx.x] = (float)(1.0 / s);
}

// d = y - e, y the network output, one value a point (odd: already combined).
__global__ void k_loss_diff(long n, const float* __restrict__ y, const float* __restrict__ e, float* __restrict__ d)
{
    const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if(p < n) d[p] = y[p] - e[p];
}

constexpr int kLossBlocks = 1184;

// Loss terms d.Md * w (M = I for kind 0, the stencil A for kind 1, i.e. the
// error's energy norm) and the output gradient 2 M d w as BF16 channel 0 of
// G (odd: +/- half of it for the two branches), and of the first branch in gy.
__global__ void __launch_bounds__(256) k_loss_grad(ConvGrid g, const float* __restrict__ d,
                                                   const float* __restrict__ wnorm, float scale, int kind, int odd,
                                                   __nv_bfloat16* __restrict__ G, float* __restrict__ gy,
                                                   float* __restrict__ loss_partial)
{
    __shared__ float red[32];
    const long per = (long)g.nz * g.ny * g.nx;
    const long n = per * g.nb;
    float acc = 0.f;
    for(long p = (long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x)
    {
        const float w = wnorm[p / per] * scale;
        const float md = kind ? stencil_at(g, d, p) : d[p];
        acc += d[p] * md * w;
        const float gv = (odd ? 1.f : 2.f) * md * w;
        gy[p] = gv;
        store_embed(G, p, gv);
        if(odd) store_embed(G, p + n, -gv);
    }
    acc = block_sum(acc, red);
    if(threadIdx.x == 0) loss_partial[blockIdx.x] = acc;
}

// Projects the three layers' weights onto the odd-symmetric ("tied") form:
// hidden channels k and k+8 are a +/- pair, so that the network is an odd
// function of its input with one evaluation:
//   w1[t][0][k+8] = -w1[t][0][k]; w2[t][i][j] = w2[t][i^8][j^8]; w3[t][j^8][0] = -w3[t][j][0].
// Unused weights (layer 1 inputs >= 1, layer 3 outputs >= 1) are zeroed.
__global__ void k_tie_odd(float* __restrict__ w)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= kNetLayerWeights) return;
    const int t = i / 256, a = (i / 16) % 16, b = i % 16;
    float* w1 = w;
    float* w2 = w + kNetLayerWeights;
    float* w3 = w + 2 * kNetLayerWeights;
    // each pair/quad is handled by its lowest index
    if(a == 0 && b < 8)
    {
        const int k0 = (t * 16) * 16 + b, k1 = k0 + 8;
        const float v = 0.5f * (w1[k0] - w1[k1]);
        w1[k0] = v;
        w1[k1] = -v;
    }
    if(a != 0) w1[i] = 0.f;
    if(a < 8)
    {
        const int k0 = (t * 16 + a) * 16 + b, k1 = (t * 16 + (a ^ 8)) * 16 + (b ^ 8);
        const float v = 0.5f * (w2[k0] + w2[k1]);
        w2[k0] = v;
        w2[k1] = v;
    }
    if(b == 0 && a < 8)
    {
        const int k0 = (t * 16 + a) * 16, k1 = (t * 16 + (a ^ 8)) * 16;
        const float v = 0.5f * (w3[k0] - w3[k1]);
        w3[k0] = v;
        w3[k1] = -v;
    }
    if(b != 0) w3[i] = 0.f;
}

__global__ void k_adam(int n, float* __restrict__ w, const float* __restrict__ dw, float* __restrict__ m,
                       float* __restrict__ v, float lr, float beta1, float beta2, float eps, float c1, float c2)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const float gi = dw[i];
    const float mi = beta1 * m[i] + (1.f - beta1) * gi;
    const float vi = beta2 * v[i] + (1.f - beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
}

// ------------------------------------------------------------ launchers

static int sm_count()
{
    static int sms = 0;
    if(sms == 0)
    {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if(sms <= 0) sms = 148;
    }
    return sms;
}

// Tensor map of a channel-last BF16 tensor [nb][nz][ny][nx][16] with a box
// of 16 channels x bx x by x bz points x 1 sample, written in the 32-byte
// swizzle that the A descriptors declare; the driver entry point is looked up
// once through the runtime.
static int bf16_box_map(const ConvGrid& g, const void* in, int bx, int by, int bz, CUtensorMap* map)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if(!encode)
    {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        HB_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
        if(q != cudaDriverEntryPointSuccess || !fn)
            return record_error(HPCGB200_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    const cuuint64_t dims[5] = {(cuuint64_t)kNetCh, (cuuint64_t)g.nx, (cuuint64_t)g.ny, (cuuint64_t)g.nz,
                                (cuuint64_t)g.nb};
    const cuuint64_t row = (cuuint64_t)kNetCh * 2;
    const cuuint64_t strides[4] = {row, row * g.nx, row * g.nx * g.ny, row * g.nx * g.ny * g.nz};
    const cuuint32_t box[5] = {(cuuint32_t)kNetCh, (cuuint32_t)bx, (cuuint32_t)by, (cuuint32_t)bz, 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(in), dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if(r != CUDA_SUCCESS) return record_error(HPCGB200_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return 0;
}

// The conv brick box: 16 x 10 x 6 points (14 x 8 x 4 outputs and their halo).
static int conv_tensor_map(const ConvGrid& g, const void* in, CUtensorMap* map)
{
    return bf16_box_map(g, in, kTX, kHY, kHZ, map);
}

template <int kOut>
static int conv_launch(const ConvGrid& g, const void* in, const void* wB, void* out, const void* act, int* status,
                       cudaStream_t s)
{
    static bool attr = false;
    if(!attr)
    {
        HB_CUDA(cudaFuncSetAttribute(k_conv16<kOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmem));
        attr = true;
    }
    CUtensorMap map;
    HB_RETURN_IF(conv_tensor_map(g, in, &map));
    const long tiles = (long)g.nb * ((g.nx + kOX - 1) / kOX) * ((g.ny + kTY - 1) / kTY) * ((g.nz + kTZ - 1) / kTZ);
    const long cap = (long)HB_CONV_CTAS * sm_count();
    const int grid = (int)(tiles < cap ? tiles : cap);
    HB_CUDA(launch_pdl_net(k_conv16<kOut>, dim3(grid), dim3(kConvThreads), (size_t)kConvSmem, s, map, g,
                           (const __nv_bfloat16*)wB, out, (const __nv_bfloat16*)act, status));
    return 0;
}

int launch_conv16(const ConvGrid& g, const void* in, const void* wB, int out_mode, void* out, const void* act,
                  int* status, cudaStream_t s)
{
    switch(out_mode)
    {
        case kOutReluBf16: return conv_launch<kOutReluBf16>(g, in, wB, out, act, status, s);
        case kOutMaskBf16: return conv_launch<kOutMaskBf16>(g, in, wB, out, act, status, s);
        case kOutF32: return conv_launch<kOutF32>(g, in, wB, out, act, status, s);
        case kOutF32C0: return conv_launch<kOutF32C0>(g, in, wB, out, act, status, s);
        default: return record_error(HPCGB200_ERR_ARG, "conv16: unknown output mode %d", out_mode);
    }
}

template <int kOut, bool kPair>
static int layer3_launch(const ConvGrid& g, const void* a2, const float* w3, float* out, const PermMap& pm,
                         int* status, cudaStream_t s)
{
    static bool attr = false;
    if(!attr)
    {
        HB_CUDA(cudaFuncSetAttribute(k_layer3_tc<kOut, kPair>, cudaFuncAttributeMaxDynamicSharedMemorySize, k3Smem));
        attr = true;
    }
    CUtensorMap map;
    const ConvGrid gin{kPair ? 2 * g.nb : g.nb, g.nz, g.ny, g.nx};
    HB_RETURN_IF(bf16_box_map(gin, a2, kTX, kHY, kHZ, &map));
    const long tiles =
        (long)g.nb * ((g.nx + kOX - 1) / kOX) * ((g.ny + kTY - 1) / kTY) * ((g.nz + kTZ - 1) / kTZ);
    const long cap = sm_count();
    const int grid = (int)(tiles < cap ? tiles : cap);
    HB_CUDA(launch_pdl_net(k_layer3_tc<kOut, kPair>, dim3(grid), dim3(k3Threads), (size_t)k3Smem, s, map, g, w3,
                           out, pm, status));
    return 0;
}

int launch_layer3_tc(const ConvGrid& g, const PermMap* pm, const void* a2, const float* w3, int pair, int mode,
                     float* out, int* status, cudaStream_t s)
{
    if(mode < 0 || mode > 2) return record_error(HPCGB200_ERR_ARG, "layer 3: unknown output mode %d", mode);
    if(mode != 2 && (!pm || g.nb != 1)) return record_error(HPCGB200_ERR_ARG, "layer 3: level output needs one sample");
    const PermMap m = pm ? *pm : PermMap{};
    if(pair)
    {
        if(mode == 0) return layer3_launch<0, true>(g, a2, w3, out, m, status, s);
        if(mode == 1) return layer3_launch<1, true>(g, a2, w3, out, m, status, s);
        return layer3_launch<2, true>(g, a2, w3, out, m, status, s);
    }
    if(mode == 0) return layer3_launch<0, false>(g, a2, w3, out, m, status, s);
    if(mode == 1) return layer3_launch<1, false>(g, a2, w3, out, m, status, s);
    return layer3_launch<2, false>(g, a2, w3, out, m, status, s);
}

// CTAs of a weight gradient at most (the size of its workspace).
int conv16_wgrad_parts(long points)
{
    const long nblk = (points + 63) / 64;
    const long cap = sm_count();
    return (int)(nblk < cap ? nblk : cap);
}

int launch_conv16_wgrad(const ConvGrid& g, const void* x, const void* gr, float* partial, float* dw, int* status,
                        cudaStream_t s)
{
    static bool attr = false;
    if(!attr)
    {
        HB_CUDA(cudaFuncSetAttribute(k_conv16_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem));
        attr = true;
    }
    const long units = wg_units(g).count;
    const int most = conv16_wgrad_parts(g.points());
    const int parts = (int)(units < most ? units : most);
    k_conv16_wgrad<<<parts, kWgThreads + 32, kWgSmem, s>>>(g, (const __nv_bfloat16*)x, (const __nv_bfloat16*)gr, partial,
                                                      status);
    HB_LAUNCHED();
    k_wgrad_reduce<<<kNetLayerWeights / 32, 256, 0, s>>>(parts, partial, dw);
    HB_LAUNCHED();
    return 0;
}

int launch_prepare_weights(const float* w, void* wB, int flip, cudaStream_t s)
{
    k_prepare_weights<<<(kNetLayerWeights + 255) / 256, 256, 0, s>>>(w, (__nv_bfloat16*)wB, flip);
    HB_LAUNCHED();
    return 0;
}

int launch_embed_scalar_level(const PermMap& pm, int nz, int ny, int nx, const float* r, const float* x,
                              const float* diag32, void* s1, cudaStream_t s)
{
    const long n = (long)nz * ny * nx;
    HB_CUDA(launch_pdl_net(k_embed_scalar_level, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, s, pm, nz, ny, nx, r,
                           x, diag32, (__nv_bfloat16*)s1));
    return 0;
}


template <typename Tin, bool kPair, bool kMask = false>
static int layer1_launch(const ConvGrid& g, const Tin* in, const float* w1, void* a1, const void* act, int* status,
                         cudaStream_t s)
{
    static bool attr = false;
    if(!attr)
    {
        HB_CUDA(cudaFuncSetAttribute(k_layer1_tc<Tin, kPair, kMask>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     k1Smem));
        attr = true;
    }
    const long tiles = (long)g.nb * ((g.nx + k1X - 1) / k1X) * ((g.ny + k1Y - 1) / k1Y) * ((g.nz + k1Z - 1) / k1Z);
    const long cap = (long)k1CtasPerSm * sm_count();
    const int grid = (int)(tiles < cap ? tiles : cap);
    HB_CUDA(launch_pdl_net(k_layer1_tc<Tin, kPair, kMask>, dim3(grid), dim3(k1Threads), (size_t)k1Smem, s, g, in, w1,
                           (__nv_bfloat16*)a1, (const __nv_bfloat16*)act, status));
    return 0;
}

int launch_layer1_tc(const ConvGrid& g, const void* in, int in_f32, const float* w1, void* a1, int pair, int* status,
                     cudaStream_t s)
{
    if(in_f32)
        return pair ? layer1_launch<float, true>(g, (const float*)in, w1, a1, nullptr, status, s)
                    : layer1_launch<float, false>(g, (const float*)in, w1, a1, nullptr, status, s);
    return pair ? layer1_launch<__nv_bfloat16, true>(g, (const __nv_bfloat16*)in, w1, a1, nullptr, status, s)
                : layer1_launch<__nv_bfloat16, false>(g, (const __nv_bfloat16*)in, w1, a1, nullptr, status, s);
}

int launch_layer3_grad(const ConvGrid& g, const float* gy, const float* w3, const void* a2, void* out, int pair,
                       int* status, cudaStream_t s)
{
    return pair ? layer1_launch<float, true, true>(g, gy, w3, out, a2, status, s)
                : layer1_launch<float, false, true>(g, gy, w3, out, a2, status, s);
}

int launch_sample_norm(const ConvGrid& g, const float* e, int kind, float* out, cudaStream_t s)
{
    k_sample_norm<<<g.nb, 512, 0, s>>>(g, e, kind, out);
    HB_LAUNCHED();
    return 0;
}

int launch_natural_from_perm(const PermMap& pm, int nz, int ny, int nx, const float* in, float* out, cudaStream_t s)
{
    const long n = (long)nz * ny * nx;
    k_perm_copy<float, float, true><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(pm, nz, ny, nx, in, out);
    HB_LAUNCHED();
    return 0;
}

int launch_natural_from_perm(const PermMap& pm, int nz, int ny, int nx, const double* in, float* out, cudaStream_t s)
{
    const long n = (long)nz * ny * nx;
    k_perm_copy<double, float, true><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(pm, nz, ny, nx, in, out);
    HB_LAUNCHED();
    return 0;
}

int launch_perm_from_natural(const PermMap& pm, int nz, int ny, int nx, const float* in, double* out, cudaStream_t s)
{
    const long n = (long)nz * ny * nx;
    k_perm_copy<float, double, false><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(pm, nz, ny, nx, in, out);
    HB_LAUNCHED();
    return 0;
}

int launch_inv_sumsq(long n, const float* e, float* out, cudaStream_t s)
{
    k_inv_sumsq<<<1, 1024, 0, s>>>(n, e, out);
    HB_LAUNCHED();
    return 0;
}

int launch_loss_accumulate(const float* partial, double* acc, cudaStream_t s)
{
    k_loss_accumulate<<<1, 1024, 0, s>>>(kLossBlocks, partial, acc);
    HB_LAUNCHED();
    return 0;
}

int launch_normal_rhs(long long m, unsigned long long seed, const int* perm, double* out64, float* out32,
                      cudaStream_t s)
{
    k_normal_rhs<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(m, seed, perm, out64, out32);
    HB_LAUNCHED();
    return 0;
}

int launch_embed_f32(long n, const float* r, void* a, int pair, cudaStream_t s)
{
    k_embed_f32<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, r, (__nv_bfloat16*)a, pair);
    HB_LAUNCHED();
    return 0;
}

int loss_parts(long points)
{
    (void)points;
    return kLossBlocks;
}

int launch_loss_grad(const ConvGrid& g, float* y, const float* e, float* d, const float* wnorm, float scale,
                     int kind, int odd, void* G, float* loss_partial, cudaStream_t s)
{
    const long n = g.points();
    k_loss_diff<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, y, e, d);
    HB_LAUNCHED();
    k_loss_grad<<<kLossBlocks, 256, 0, s>>>(g, d, wnorm, scale, kind, odd, (__nv_bfloat16*)G, y, loss_partial);
    HB_LAUNCHED();
    return 0;
}

int launch_tie_odd(float* w, cudaStream_t s)
{
    k_tie_odd<<<(kNetLayerWeights + 255) / 256, 256, 0, s>>>(w);
    HB_LAUNCHED();
    return 0;
}

int launch_adam(int n, float* w, const float* dw, float* m, float* v, float lr, float beta1, float beta2, float eps,
                int t, cudaStream_t s)
{
    const float c1 = 1.f / (1.f - std::pow(beta1, (float)t));
    const float c2 = 1.f / (1.f - std::pow(beta2, (float)t));
    k_adam<<<(n + 255) / 256, 256, 0, s>>>(n, w, dw, m, v, lr, beta1, beta2, eps, c1, c2);
    HB_LAUNCHED();
    return 0;
}

}  // namespace hb

using namespace hb;

// ------------------------------------------------------------------ C ABI

extern "C" size_t hpcgb200_conv_weight_tile_bytes(void) { return kNetWeightTileBytes; }

extern "C" int hpcgb200_conv_prepare_weights(const float* w, void* wB, int flip, void* stream)
{
    HB_CHECK_ARG(w && wB, "bad arguments");
    HB_CHECK_ARG((reinterpret_cast<uintptr_t>(wB) & 15) == 0, "wB must be 16-byte aligned");
    return launch_prepare_weights(w, wB, flip, as_stream(stream));
}

extern "C" int hpcgb200_conv16(int nb, int nz, int ny, int nx, const void* in, const void* wB, int out_mode, void* out,
                               const void* act, int* status, void* stream)
{
    HB_CHECK_ARG(nb > 0 && nz > 0 && ny > 0 && nx > 0 && in && wB && out && status, "bad arguments");
    HB_CHECK_ARG(out_mode >= kOutReluBf16 && out_mode <= kOutF32C0, "out_mode must be 0..3");
    HB_CHECK_ARG(out_mode != kOutMaskBf16 || act, "the masked mode needs the activation tensor");
    HB_CHECK_ARG((reinterpret_cast<uintptr_t>(in) & 15) == 0 && (reinterpret_cast<uintptr_t>(wB) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (reinterpret_cast<uintptr_t>(act) & 15) == 0,
                 "tensors must be 16-byte aligned");
    const ConvGrid g{nb, nz, ny, nx};
    return launch_conv16(g, in, wB, out_mode, out, act, status, as_stream(stream));
}

extern "C" size_t hpcgb200_conv_wgrad_partial_bytes(int nb, int nz, int ny, int nx)
{
    return sizeof(float) * kNetLayerWeights * (size_t)conv16_wgrad_parts((long)nb * nz * ny * nx);
}

extern "C" int hpcgb200_conv16_wgrad(int nb, int nz, int ny, int nx, const void* x, const void* g, float* partial,
                                     float* dw, int* status, void* stream)
{
    HB_CHECK_ARG(nb > 0 && nz > 0 && ny > 0 && nx > 0 && x && g && partial && dw && status, "bad arguments");
    HB_CHECK_ARG((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(g) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(partial) & 15) == 0,
                 "tensors must be 16-byte aligned");
    const ConvGrid cg{nb, nz, ny, nx};
    return launch_conv16_wgrad(cg, x, g, partial, dw, status, as_stream(stream));
}

extern "C" int hpcgb200_normal_rhs(long long m, unsigned long long seed, double* out, void* stream)
{
    HB_CHECK_ARG(m >= 0 && (m == 0 || out), "bad arguments");
    if(m == 0) return 0;
    return launch_normal_rhs(m, seed, nullptr, out, nullptr, as_stream(stream));
}

extern "C" int hpcgb200_sample_norms(int nb, int nz, int ny, int nx, const float* e, int kind, float* out, void* stream)
{
    HB_CHECK_ARG(nb > 0 && nz > 0 && ny > 0 && nx > 0 && e && out && (kind == 0 || kind == 1), "bad arguments");
    return launch_sample_norm(ConvGrid{nb, nz, ny, nx}, e, kind, out, as_stream(stream));
}
