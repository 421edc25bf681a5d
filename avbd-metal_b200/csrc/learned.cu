// learned.cu — learned warm start: per-vertex features, a 32-128-128-128-16
// MLP (BF16 weights and activations, FP32 accumulation on the tensor cores)
// for inference and training, and the acceptance test that keeps a predicted
// warm start only when it is no worse than the plain gamma warm start.
//
// The MLP predicts the correction the solve applies to the plain warm start
// of every dynamic particle, in units of s = max(|g|, 1) dt^2:
//   x0 = x_plain + s * MLP(features)[0-2],
// and, when the model covers rigid bodies (Params::learnRigid), of every
// dynamic rigid body's pose, the rotation as the arc length it sweeps at the
// body's bounding radius r:
//   q0 = q_plain (+) (s / r) * MLP(features)[3-5]   (q_addw, tangent space).
// Learned rows list the particles first, then the rigid bodies.
// Features (32, normalised by per-feature mean and 1/std stored with the
// model): [0-2] inertial offset (x~ - x_start)/s, [3-5] plain warm-start
// offset (x_plain - x_start)/s, [6-8] previous-frame displacement
// v_prev dt / s, [9] incident contact count / 4, [10-12] summed oriented
// contact normal, [13] smallest contact gap / s (clipped), [14] log(1 +
// stiffness dt^2 / m) of the incident elements, [15] 1; rigid rows only
// (zeros for particles): [16] 1, [17-19] plain warm-start rotation
// q_sub(q_plain, q_start) r / s, [20-22] world up axis in the body frame,
// [23] log(1 + r / s) / 10, [24] incident position-PD hinge motors / 4,
// [28-30] the rotation those motors ask for at the plain warm start (sum
// of hinge axis x -(twist - target), as arc length at r in units of s),
// [31] log(1 + sum kp dt^2 / (m r^2)); 1-ring aggregates over the vertices sharing a tet or spring: [25]
// ring size / 10, [26] mean neighbour contact count / 4, [27] smallest
// neighbour contact gap / s (clipped).  Contacts are rigid manifolds and
// element contacts alike.
//
// Parameter block (fp32, also the layout of the gradients): W1[128][32], b1,
// W2[128][128], b2, W3[128][128], b3, W4[16][128], b4[16].  The weights are
// mirrored as BF16 for the tensor cores.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>

#include "../../include/avbd.h"
#include "dmath.cuh"
#include "kernels.h"
#include "pdl.cuh"

namespace avbd {

namespace mlp {
constexpr int DIN = 32, HID = 128, DOUT = 16, USED_OUT = 6;
constexpr uint32_t OW1 = 0, OB1 = OW1 + HID * DIN, OW2 = OB1 + HID, OB2 = OW2 + HID * HID, OW3 = OB2 + HID,
                   OB3 = OW3 + HID * HID, OW4 = OB3 + HID, OB4 = OW4 + DOUT * HID, NPARAM = OB4 + DOUT;
// bf16 weight mirror: W1 | W2 | W3 | W4
constexpr uint32_t HW1 = 0, HW2 = HW1 + HID * DIN, HW3 = HW2 + HID * HID, HW4 = HW3 + HID * HID,
                   NHALF = HW4 + DOUT * HID;
// normalisation block: xmean[32], xinvstd[32], ymean[16], ystd[16]
constexpr uint32_t NNORM = 96, NX_MEAN = 0, NX_INV = 32, NY_MEAN = 64, NY_STD = 80;
}  // namespace mlp

namespace {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}


// ---------------------------------------------------------------------------
// Fused inference on the Blackwell tensor cores (tcgen05): one CTA per SM
// whose two groups of eight warps each walk 128-row tiles of their own, so
// that one group's MMAs run beside the other's epilogues; the weights are
// shared.  Shared-memory operands are in the UMMA canonical K-major layout
// without swizzle (8-row x 16-byte core matrices: element (r, k) of an operand
// with row-group stride `sbo` at (r / 8) sbo + (k / 8) 128 + (r % 8) 16 +
// (k % 8) 2 bytes); the hidden activations never leave tensor memory.  A layer
// is 2 (K = 32) or 8 (K = 128) tcgen05.mma instructions of M = 128, K = 16,
// issued by one thread, accumulating in TMEM (128 lanes = the tile's rows).
// Two threads share a row: each reads 64 of its fp32 columns with tcgen05.ld,
// adds the bias (two fp32 additions an instruction), applies ReLU, rounds to
// BF16 and writes them back with tcgen05.st as the A operand of the next layer
// (two columns a 32-bit TMEM cell).  A warp reads feature rows whole (four
// 128-byte rows a load) one tile ahead, and the next tile's first layer is
// issued together with this tile's last, into columns of their own.
// Completion is signalled by tcgen05.commit on the group's mbarriers; every
// wait on them is bounded and a timeout sets *status (the CTA then frees its
// TMEM and stops).  Tiles go to group tile / gridDim of a CTA, so that up to
// 148 tiles spread over all SMs before any SM takes a second one.
//
// What bounds it: the chain of a layer, about 2,200 cycles of which the eight
// MMAs (512 cycles of arithmetic, shared with the other group's) take 1,300
// from their issue to the waiting threads and the epilogue 800; the call over
// 1,048,576 rows takes 122 us, the kernel 109 of them, the rest the launch, the
// status read-back and the wait for it (236 us with one tile in flight per CTA and
// two CTAs per SM; 150 us with four groups of 128 threads and the activations
// in shared memory; 159 us before the issuing lane was elected, see elect_one).
// ---------------------------------------------------------------------------
namespace tc {
constexpr uint32_t ROWS = 128;
constexpr uint32_t SBO_K128 = 2048, SBO_K32 = 512;      // row-group strides (K = 128, K = 32)
// shared memory: weight image | input tiles | biases b1 b2 b3 b4 (fp32) |
// normalisation block (fp32) | MMA barriers | staging barrier | TMEM address
constexpr uint32_t GROUPS = 2, GROUP_THREADS = 256;         // tiles in flight of a CTA, threads of each
// input tile: 16-byte chunks 160 B apart, so that the eight lanes writing two
// rows' chunks touch all banks once
constexpr uint32_t XLBO = 160, XSBO = 4 * XLBO, XBYTES = (ROWS / 8) * XSBO;
constexpr uint32_t W1 = 0, W2 = W1 + 128 * 32 * 2, W3 = W2 + 128 * 128 * 2, W4 = W3 + 128 * 128 * 2,
                   XT = W4 + 16 * 128 * 2, BIAS = XT + GROUPS * XBYTES, NORM = BIAS + (3 * 128 + 16) * 4,
                   BAR = NORM + 96 * 4, WBAR = BAR + 16 * GROUPS, TSLOT = WBAR + 8, SMEM = TSLOT + 8;
// TMEM columns of a group: layer outputs | A operand (BF16 pairs) | last layer's output
constexpr uint32_t TD = 0, TA = 128, TY = 192, TGROUP = 256;
constexpr uint32_t WBYTES = XT - W1;                     // the weight image: 77,824 bytes
constexpr uint32_t STAGED = WBYTES + (NORM - BIAS) + 96 * 4;   // every byte the staging barrier expects
constexpr uint32_t TMEM_COLS = TGROUP * GROUPS;
constexpr uint64_t WAIT_NS = 1000000000ull;              // a wait gives up after one second

__device__ __forceinline__ uint32_t off(uint32_t r, uint32_t k, uint32_t sbo) {
    return (r >> 3) * sbo + (k >> 3) * 128u + (r & 7u) * 16u + (k & 7u) * 2u;
}
// shared-memory matrix descriptor: start address, LBO (the second 8-element K
// chunk), SBO, descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t desc(uint32_t saddr, uint32_t sbo, uint32_t lbo = 128u) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}
// instruction descriptor of kind::f16: F32 accumulator, BF16 A and B, both
// K-major, N >> 3, M >> 4
__host__ __device__ constexpr uint32_t idesc(uint32_t m, uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        :
        : "r"(tmem), "l"(a), "l"(b), "r"(id), "r"(acc));
}
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}
__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// bounded wait for the mbarrier phase `parity`; false on timeout.  The global
// timer is first read after 64 polls: reading it costs more than most waits.
__device__ __forceinline__ bool wait(uint32_t bar, uint32_t parity) {
    uint64_t t0 = 0;
    for (uint32_t i = 0;; i++) {
        if ((i & 63u) == 63u) {
            const uint64_t t = now_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > WAIT_NS) return false;
        }
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// bulk asynchronous copy global -> this CTA's shared memory (no multicast),
// completing `bytes` of the barrier's transaction count
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// one lane of a converged warp; with warp-uniform operands (uniform()) the
// MMA instructions that follow need no per-lane to uniform register moves
// (eight MMAs took 1,150 cycles to issue from a lane that the compiler could
// not know to be alone)
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0u;
}
__device__ __forceinline__ uint32_t uniform(uint32_t x) { return __shfl_sync(0xffffffffu, x, 0); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// 32 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ void ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = __uint_as_float(r[j]);
}
}  // namespace tc

// eight consecutive floats, 16-byte loads where the address allows them
__device__ __forceinline__ void load8(const float* p, bool vec, float (&v)[8]) {
    if (vec) {
        const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = p[e];
    }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
    return make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
}
// position of the k-th bias (b1 | b2 | b3 | b4) in the parameter block
__device__ __forceinline__ uint32_t bias_at(uint32_t k) {
    using namespace mlp;
    return k < 128u ? OB1 + k : (k < 256u ? OB2 + k - 128u : (k < 384u ? OB3 + k - 256u : OB4 + k - 384u));
}
// fp32 weights -> the BF16 weight image at the head of shared memory, eight
// columns of a row at a time
__device__ __forceinline__ void stage_weights(const float* prm, bool vec, unsigned char* sm, uint32_t t,
                                              uint32_t threads) {
    using namespace mlp;
    for (uint32_t g = t; g < NHALF / 8; g += threads) {
        uint32_t src, base, cols, sbo, j = 8 * g;
        if (j < HW2) { src = OW1; base = tc::W1; cols = DIN; sbo = tc::SBO_K32; }
        else if (j < HW3) { j -= HW2; src = OW2; base = tc::W2; cols = HID; sbo = tc::SBO_K128; }
        else if (j < HW4) { j -= HW3; src = OW3; base = tc::W3; cols = HID; sbo = tc::SBO_K128; }
        else { j -= HW4; src = OW4; base = tc::W4; cols = HID; sbo = tc::SBO_K128; }
        float v[8];
        load8(prm + src + j, vec, v);
        *reinterpret_cast<uint4*>(sm + base + tc::off(j / cols, j % cols, sbo)) = pack8(v);
    }
}

namespace tc {
// 64 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void ld64(uint32_t taddr, float (&v)[64]) {
    uint32_t r[64];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x64.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32,%33,%34,%35,%36,%37,%38,%39,"
        "%40,%41,%42,%43,%44,%45,%46,%47,%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%64];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
          "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
          "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
          "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
          "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
        : "r"(taddr)
        : "memory");
#pragma unroll
    for (int j = 0; j < 64; j++) v[j] = __uint_as_float(r[j]);
}
// two fp32 additions in one instruction, each rounded as a scalar addition
__device__ __forceinline__ void add2(float& x, float& y, float a, float b) {
    asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\tadd.rn.f32x2 p, p, q;\n\t"
        "mov.b64 {%0, %1}, p;\n\t}"
        : "+f"(x), "+f"(y)
        : "f"(a), "f"(b));
}
// bf16(max(x, 0)) of two values: rounded first (rounding keeps the order), a NaN gives 0 as fmaxf does
__device__ __forceinline__ uint32_t relu_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __hmax2(__floats2bfloat162_rn(lo, hi), __float2bfloat162_rn(0.0f));
    return *reinterpret_cast<const uint32_t*>(&v);
}
// barrier of one group (ids 1, 2); true when no thread passed `failed`
__device__ __forceinline__ bool group_sync(uint32_t id, bool failed) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.or.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 0, 1, q;\n\t}\n"
        : "=r"(r)
        : "r"(failed ? 1u : 0u), "r"(id), "n"(GROUP_THREADS)
        : "memory");
    return r != 0u;
}
// A from TMEM (BF16 pairs, lane = row), B from shared memory
__device__ __forceinline__ void mma_ta(uint32_t tmem, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
        :
        : "r"(tmem), "r"(a), "l"(b), "r"(id), "r"(acc));
}
// 32 consecutive 32-bit columns of this thread's TMEM lane
__device__ __forceinline__ void st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]),
        "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]),
        "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
}  // namespace tc

// IMAGE: W is the weight image and arrives by bulk copies; otherwise every CTA
// converts the fp32 parameters itself (38,912 weights, about a microsecond,
// against the launch of a kernel that would write the image first).
template <bool IMAGE>
__global__ void __launch_bounds__(tc::GROUPS * tc::GROUP_THREADS, 1)
k_mlp_infer_tc(const bf16* __restrict__ W, const float* __restrict__ prm, const float* __restrict__ norm,
               const float* __restrict__ X, uint32_t n, float* __restrict__ Y, uint32_t* status, bool issue) {
    using namespace mlp;
    extern __shared__ __align__(128) unsigned char sm[];
    const uint32_t t = threadIdx.x, warp = tc::uniform(t >> 5), lane = t & 31u;
    const uint32_t group = warp / (tc::GROUP_THREADS / 32), row = t & 127u;
    const uint32_t half = (t >> 7) & 1u;                       // row and column half of this thread
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    const uint32_t bar = sbase + tc::BAR + 16u * group, bar4 = bar + 8u, wbar = sbase + tc::WBAR;
    if (t == 0) {
        for (uint32_t g = 0; g < 2 * tc::GROUPS; g++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbase + tc::BAR + 8u * g) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(wbar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (IMAGE) {
            // the weight image (already in the canonical layout), the biases
            // and the normalisation block: nine bulk copies on one barrier
            tc::expect_tx(wbar, tc::STAGED);
            const unsigned char* img = reinterpret_cast<const unsigned char*>(W);
            tc::bulk_load(sbase + tc::W1, img + tc::W1, tc::W2 - tc::W1, wbar);
            tc::bulk_load(sbase + tc::W2, img + tc::W2, tc::W3 - tc::W2, wbar);
            tc::bulk_load(sbase + tc::W3, img + tc::W3, tc::W4 - tc::W3, wbar);
            tc::bulk_load(sbase + tc::W4, img + tc::W4, tc::XT - tc::W4, wbar);
            tc::bulk_load(sbase + tc::BIAS, prm + OB1, 128 * 4, wbar);
            tc::bulk_load(sbase + tc::BIAS + 512, prm + OB2, 128 * 4, wbar);
            tc::bulk_load(sbase + tc::BIAS + 1024, prm + OB3, 128 * 4, wbar);
            tc::bulk_load(sbase + tc::BIAS + 1536, prm + OB4, 16 * 4, wbar);
            tc::bulk_load(sbase + tc::NORM, norm, 96 * 4, wbar);
        }
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + tc::TSLOT),
                     "r"(tc::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (!IMAGE) {
        stage_weights(prm, true, sm, t, tc::GROUPS * tc::GROUP_THREADS);
        float* sb = reinterpret_cast<float*>(sm + tc::BIAS);
        for (uint32_t i = t; i < 3 * HID + DOUT; i += tc::GROUPS * tc::GROUP_THREADS) sb[i] = prm[bias_at(i)];
        if (t < 96) reinterpret_cast<float*>(sm + tc::NORM)[t] = norm[t];
        tc::fence_proxy();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tbase = tc::uniform(*reinterpret_cast<volatile uint32_t*>(sm + tc::TSLOT));
    const uint32_t tmem = tbase + tc::TGROUP * group;
    const uint32_t lane_addr = tmem + (((warp & 3u) * 32u) << 16);   // this warp's 32 TMEM lanes
    unsigned char* xt = sm + tc::XT + tc::XBYTES * group;
    const uint32_t sxt = sbase + tc::XT + tc::XBYTES * group;
    bool ok = true;
    if (IMAGE) {
        // the weights have landed (bounded wait; block-uniform outcome)
        ok = __syncthreads_and(tc::wait(wbar, 0) ? 1 : 0) != 0;
        if (!ok) tc::wait(wbar, 0);    // give copies still in flight one more bounded wait
    }
    const float* sbias = reinterpret_cast<const float*>(sm + tc::BIAS);
    const float* snorm = reinterpret_cast<const float*>(sm + tc::NORM);
    const uint32_t tiles = n / tc::ROWS + (n % tc::ROWS ? 1u : 0u);
    const uint32_t stride = tc::GROUPS * gridDim.x;
    // A warp loads 16 feature rows four at a time, eight lanes a row: the
    // lane's four columns (and their normalisation) are the same in each.
    const uint32_t xr = (warp & 7u) * 16u + (lane >> 3), xc = (lane & 7u) * 4u;
    const float4 xmean = *reinterpret_cast<const float4*>(snorm + NX_MEAN + xc);
    const float4 xinv = *reinterpret_cast<const float4*>(snorm + NX_INV + xc);
    float4 x[4];
    auto fetch = [&](uint32_t tile) {
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const size_t r = (size_t)tile * tc::ROWS + xr + 4u * i;
            x[i] = tile < tiles && r < n ? __ldg(reinterpret_cast<const float4*>(X + r * DIN + xc))
                                         : make_float4(0, 0, 0, 0);
        }
    };
    // the fetched rows, normalised, as the BF16 operand of the first layer
    auto stage = [&](uint32_t tile) {
#pragma unroll
        for (uint32_t i = 0; i < 4; i++) {
            const uint32_t rr = xr + 4u * i;
            const bool in = tile < tiles && (size_t)tile * tc::ROWS + rr < n;
            const float4 v = x[i];
            const uint2 w = make_uint2(pack_bf16((v.x - xmean.x) * xinv.x, (v.y - xmean.y) * xinv.y),
                                       pack_bf16((v.z - xmean.z) * xinv.z, (v.w - xmean.w) * xinv.w));
            *reinterpret_cast<uint2*>(xt + (rr >> 3) * tc::XSBO + (xc >> 3) * tc::XLBO + (rr & 7u) * 16u +
                                      (xc & 7u) * 2u) = in ? w : make_uint2(0u, 0u);
        }
    };
    const bool issuer = warp % (tc::GROUP_THREADS / 32) == 0u && issue;   // a warp; issue = false only in the timeout test
    auto first_layer = [&]() {
        for (uint32_t s = 0; s < DIN / 16; s++)
            tc::mma(tmem + tc::TD, tc::desc(sxt + 2u * tc::XLBO * s, tc::XSBO, tc::XLBO),
                    tc::desc(sbase + tc::W1 + 256u * s, tc::SBO_K32), tc::idesc(128, HID), s > 0 ? 1u : 0u);
        tc::commit(bar);
    };
    // every thread's TMEM and shared-memory writes and TMEM reads are done;
    // false when a thread's wait gave up (the same answer for the group)
    bool failed = false;
    auto publish = [&]() {
        tc::fence_proxy();
        tc::fence_before();
        const bool all = tc::group_sync(1u + group, failed);
        tc::fence_after();
        return all;
    };
    auto wait = [&](uint32_t b, uint32_t parity) {
        if (!tc::wait(b, parity)) failed = true;
        tc::fence_after();
    };
    uint32_t tile = blockIdx.x + group * gridDim.x, phase = 0, phase4 = 0;
    if (tile < tiles && ok) {
        fetch(tile);
        stage(tile);
        fetch(tile + stride);
        ok = publish();
        if (issuer && tc::elect_one()) first_layer();
        for (; tile < tiles && ok; tile += stride) {
#pragma unroll 1
            for (int layer = 0; layer < 3 && ok; layer++) {
                wait(bar, phase);
                phase ^= 1u;
                // bias, ReLU, BF16 of this thread's 64 columns: the next layer's operand
                const float* bias = sbias + 128 * layer + 64u * half;
                float v[64];
                tc::ld64(lane_addr + tc::TD + 64u * half, v);
                uint32_t a[32];
#pragma unroll
                for (uint32_t q = 0; q < 16; q++) {
                    const float4 b = *reinterpret_cast<const float4*>(bias + 4 * q);
                    float* u = v + 4 * q;
                    tc::add2(u[0], u[1], b.x, b.y);
                    tc::add2(u[2], u[3], b.z, b.w);
                    a[2 * q] = tc::relu_bf16(u[0], u[1]);
                    a[2 * q + 1] = tc::relu_bf16(u[2], u[3]);
                }
                tc::st32(lane_addr + tc::TA + 32u * half, a);
                ok = publish();
                if (!ok) break;
                if (issuer && tc::elect_one()) {
                    const uint32_t wbase = sbase + (layer == 0 ? tc::W2 : (layer == 1 ? tc::W3 : tc::W4));
                    const uint32_t id = tc::idesc(128, layer == 2 ? DOUT : HID);
                    for (uint32_t s = 0; s < HID / 16; s++)
                        tc::mma_ta(tmem + (layer == 2 ? tc::TY : tc::TD), tmem + tc::TA + 8u * s,
                                   tc::desc(wbase + 256u * s, tc::SBO_K128), id, s > 0 ? 1u : 0u);
                    tc::commit(layer == 2 ? bar4 : bar);
                    if (layer == 2 && tile + stride < tiles) first_layer();
                }
                if (layer == 0) {       // the first layer has read its operand: write the next tile's
                    stage(tile + stride);
                    if (tile + stride < tiles) fetch(tile + 2u * stride);
                }
            }
            if (!ok) break;
            wait(bar4, phase4);
            phase4 ^= 1u;
            float v[16];
            tc::ld16(lane_addr + tc::TY, v);
            const size_t r = (size_t)tile * tc::ROWS + row;
            if (r < n && !failed) {
#pragma unroll
                for (uint32_t c = 0; c < (uint32_t)USED_OUT / 2; c++) {
                    const uint32_t k = c + half * (USED_OUT / 2);
                    const float y = (half ? v[c + USED_OUT / 2] : v[c]) + sbias[3 * 128 + k];
                    Y[r * USED_OUT + k] = y * snorm[NY_STD + k] + snorm[NY_MEAN + k];
                }
            }
        }
        ok = publish();
    }
    if (!ok) {
        if ((t & (tc::GROUP_THREADS - 1u)) == 0u) atomicCAS(status, 0u, (uint32_t)AVBD_FAIL_WAIT_TIMEOUT);
        if (issue) {                    // products still in flight (bounded)
            tc::wait(bar, phase ^ 1u);
            tc::wait(bar4, phase4 ^ 1u);
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(tc::TMEM_COLS)
                     : "memory");
}

// ---------------------------------------------------------------------------
// Training step on the tensor cores, two launches.
//
// k_train_tile: a CTA of eight warps takes 128-row tiles of the batch (tile
// blockIdx.x, + gridDim.x, ...) through the whole forward and backward pass
// without leaving the SM.  The BF16 weights, the tile's inputs and the three
// hidden activations stay in shared memory in the canonical K-major layout
// [row][column]; the same image serves both roles an operand has:
//   forward      Z_l  = H_{l-1} W_l^T    A, B K-major
//   input grads  G_l  = dH_{l+1} W_{l+1} A K-major, B = W MN-major (N = in)
//   weight grads dW_l = dH_l^T H_{l-1}   A, B MN-major (K = the tile's rows)
// (MN-major core matrices are the same 8 x 16-byte blocks: the stride over
// 8-row groups becomes the K stride.)  dW_4 is formed transposed, H_3^T dY,
// because M is 128.  The four weight gradients accumulate in their own TMEM
// columns over all tiles of the CTA; layer outputs and input gradients share
// 128 columns.  The weight-gradient MMAs are issued after the commit that the
// next epilogue waits for, so they run beside it; dH_3 goes to a spare tile
// and dH_2, dH_1 to the tiles of H_3 and H_2, whose last readers an earlier
// commit has covered.  Two threads share a row (64 columns each).
//
// Bias gradients are fp32 column sums of the unrounded dH: a warp folds its
// 32 rows by a shuffle exchange (lane j ends with column j), the warps of a
// column half are added in order at the end.
//
// k_train_reduce adds the CTAs' partial gradients in CTA order, and either
// stores the gradient or applies Adam.
//
// What bounds it: at the trainer's 8,192 rows a tile is a chain of eight
// dependent products with their epilogues (2.7 GFLOP in all), so latency, not
// the tensor pipe; one row tile per CTA keeps 64 SMs busy with one pass over
// the batch: 28.7 us a step at 8,192 rows, launches included (1,005 us as ~35
// launches with the activations in global memory and one thread per bias
// column, whose four serial sums over the rows were most of it).
// ---------------------------------------------------------------------------
namespace tt {
constexpr uint32_t THREADS = 256;
constexpr uint32_t SBO128 = 2048, SBO32 = 512, SBO16 = 256;   // row-group strides of 128-, 32-, 16-column images
constexpr uint32_t X = tc::WBYTES, H1 = X + 128 * 32 * 2, H2 = H1 + 128 * 128 * 2, H3 = H2 + 128 * 128 * 2,
                   SP = H3 + 128 * 128 * 2, DY = SP + 128 * 128 * 2, BIAS = DY + 128 * 16 * 2,
                   NORM = BIAS + (3 * 128 + 16) * 4, RED = NORM + 96 * 4, BAR = RED + 8 * 64 * 4, TSLOT = BAR + 8,
                   SMEM = TSLOT + 8;
static_assert(SMEM <= 227 * 1024, "shared memory of a training CTA");
// TMEM columns: D (layer outputs, input gradients) | dW3 | dW2 | dW1 | dW4^T
constexpr uint32_t TD = 0, TW3 = 128, TW2 = 256, TW1 = 384, TW4 = 416, TMEM_COLS = 512;
// a CTA's partial gradient (floats): dW3, dW2, dW1 as [in][out], dW4 as
// [out][in], the biases, the loss, 1 where all of this is valid; the lane of every
// TMEM row is contiguous
constexpr uint32_t P3 = 0, P2 = P3 + 128 * 128, P1 = P2 + 128 * 128, P4 = P1 + 32 * 128, PB1 = P4 + 16 * 128,
                   PB2 = PB1 + 128, PB3 = PB2 + 128, PB4 = PB3 + 128, PL = PB4 + 16, PV = PL + 1, PART = PL + 16;

// K-major descriptor (second 8-column K chunk 128 B on) and MN-major one of
// the same image: 8-column groups 128 B apart, 8-row (K) groups `sbo` apart
__device__ __forceinline__ uint64_t kmajor(uint32_t saddr, uint32_t sbo) { return tc::desc(saddr, sbo); }
__device__ __forceinline__ uint64_t mnmajor(uint32_t saddr, uint32_t sbo) {
    return tc::desc(saddr, 128u, sbo);
}
constexpr uint32_t MN_A = 1u << 15, MN_B = 1u << 16;          // instruction descriptor: operand is MN-major

// v[c] of 32 lanes -> lane j returns the sum of v[j] over the warp
__device__ __forceinline__ float column_sums(float (&v)[32], uint32_t lane) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const bool up = (lane & (uint32_t)o) != 0u;
#pragma unroll
        for (int j = 0; j < o; j++) {
            const float give = up ? v[j] : v[j + o], keep = up ? v[j + o] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    return v[0];
}
}  // namespace tt

__global__ void __launch_bounds__(tt::THREADS, 1)
k_train_tile(const float* __restrict__ prm, const float* __restrict__ norm, const float* __restrict__ Xg,
             const float* __restrict__ Tg, uint32_t n, float* __restrict__ part, uint32_t* status, bool issue) {
    using namespace mlp;
    extern __shared__ __align__(128) unsigned char sm[];
    const uint32_t t = threadIdx.x, warp = tc::uniform(t >> 5), lane = t & 31u;
    const uint32_t row = t & 127u, half = t >> 7;             // tile row and column half of this thread
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(sm);
    const uint32_t bar = sbase + tt::BAR;
    float* sbias = reinterpret_cast<float*>(sm + tt::BIAS);
    float* snorm = reinterpret_cast<float*>(sm + tt::NORM);
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + tt::TSLOT),
                     "r"(tt::TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the weights as BF16 images, biases and normalisation block
    const bool vecX = (reinterpret_cast<uintptr_t>(Xg) & 15u) == 0u;
    stage_weights(prm, (reinterpret_cast<uintptr_t>(prm) & 15u) == 0u, sm, t, tt::THREADS);
    for (uint32_t i = t; i < 3 * HID + DOUT; i += tt::THREADS) sbias[i] = prm[bias_at(i)];
    if (t < 96) snorm[t] = norm[t];
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tc::uniform(*reinterpret_cast<volatile uint32_t*>(sm + tt::TSLOT));
    const uint32_t lane_addr = tmem + (((warp & 3u) * 32u) << 16);  // this warp's 32 TMEM lanes
    uint32_t phase = 0;
    bool ok = true;
    // block-uniform outcome of the bounded wait for the last commit
    auto wait_mma = [&]() {
        ok = __syncthreads_and(tc::wait(bar, phase) ? 1 : 0) != 0;
        phase ^= 1u;
        tc::fence_after();
        return ok;
    };
    // shared-memory writes and TMEM reads of every thread are done
    auto publish = [&]() {
        tc::fence_proxy();
        tc::fence_before();
        __syncthreads();
        tc::fence_after();
    };
    // bias + ReLU + BF16 of this thread's 64 columns of D into the image at `dst`
    auto activate = [&](const float* bias, uint32_t dst) {
#pragma unroll
        for (uint32_t c = 0; c < 2; c++) {
            const uint32_t c0 = half * 64u + c * 32u;
            float v[32];
            tc::ld32(lane_addr + tt::TD + c0, v);
#pragma unroll
            for (uint32_t kg = 0; kg < 4; kg++) {
                float w[8];
#pragma unroll
                for (int e = 0; e < 8; e++) w[e] = fmaxf(v[kg * 8 + e] + bias[c0 + kg * 8 + e], 0.0f);
                *reinterpret_cast<uint4*>(sm + dst + tc::off(row, c0 + kg * 8, tt::SBO128)) = pack8(w);
            }
        }
    };
    float bsum[3][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}, {0.0f, 0.0f}};
    // dH = G where the activation at `act` is positive: BF16 into `dst`, fp32 column sums into bsum
    auto relu_back = [&](uint32_t act, uint32_t dst, float (&bs)[2]) {
#pragma unroll
        for (uint32_t c = 0; c < 2; c++) {
            const uint32_t c0 = half * 64u + c * 32u;
            float v[32];
            tc::ld32(lane_addr + tt::TD + c0, v);
#pragma unroll
            for (uint32_t kg = 0; kg < 4; kg++) {
                const uint4 a = *reinterpret_cast<const uint4*>(sm + act + tc::off(row, c0 + kg * 8, tt::SBO128));
                const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
                float w[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const float h = __uint_as_float((e & 1) ? (aw[e >> 1] & 0xFFFF0000u) : (aw[e >> 1] << 16));
                    w[e] = h > 0.0f ? v[kg * 8 + e] : 0.0f;
                    v[kg * 8 + e] = w[e];
                }
                *reinterpret_cast<uint4*>(sm + dst + tc::off(row, c0 + kg * 8, tt::SBO128)) = pack8(w);
            }
            bs[c] += tt::column_sums(v, lane);
        }
    };
    float b4sum[USED_OUT] = {}, lossSum = 0.0f;               // per row (half 0), folded over the rows at the end
    const uint32_t tiles = (n + 127u) / 128u;
    uint32_t accum = 0;                                       // the weight gradients hold earlier tiles
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t r = tile * 128u + row;
        const bool in = r < n;
        // normalised inputs, 16 columns a thread
#pragma unroll
        for (uint32_t kg = 0; kg < 2; kg++) {
            const uint32_t c = half * 16u + kg * 8u;
            float v[8] = {};
            if (in) {
                load8(Xg + (size_t)r * DIN + c, vecX, v);
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = (v[e] - snorm[NX_MEAN + c + e]) * snorm[NX_INV + c + e];
            }
            *reinterpret_cast<uint4*>(sm + tt::X + tc::off(row, c, tt::SBO32)) = pack8(v);
        }
        publish();
        // forward (issue = false only in the timeout test)
        if (warp == 0 && issue && tc::elect_one()) {
            for (uint32_t s = 0; s < DIN / 16; s++)
                tc::mma(tmem + tt::TD, tt::kmajor(sbase + tt::X + 256u * s, tt::SBO32),
                        tt::kmajor(sbase + tc::W1 + 256u * s, tc::SBO_K32), tc::idesc(128, 128), s > 0);
            tc::commit(bar);
        }
        if (!wait_mma()) break;
        activate(sbias, tt::H1);
        publish();
        if (warp == 0 && tc::elect_one()) {
            for (uint32_t s = 0; s < HID / 16; s++)
                tc::mma(tmem + tt::TD, tt::kmajor(sbase + tt::H1 + 256u * s, tt::SBO128),
                        tt::kmajor(sbase + tc::W2 + 256u * s, tc::SBO_K128), tc::idesc(128, 128), s > 0);
            tc::commit(bar);
        }
        if (!wait_mma()) break;
        activate(sbias + 128, tt::H2);
        publish();
        if (warp == 0 && tc::elect_one()) {
            for (uint32_t s = 0; s < HID / 16; s++)
                tc::mma(tmem + tt::TD, tt::kmajor(sbase + tt::H2 + 256u * s, tt::SBO128),
                        tt::kmajor(sbase + tc::W3 + 256u * s, tc::SBO_K128), tc::idesc(128, 128), s > 0);
            tc::commit(bar);
        }
        if (!wait_mma()) break;
        activate(sbias + 256, tt::H3);
        publish();
        if (warp == 0 && tc::elect_one()) {
            for (uint32_t s = 0; s < HID / 16; s++)
                tc::mma(tmem + tt::TD, tt::kmajor(sbase + tt::H3 + 256u * s, tt::SBO128),
                        tt::kmajor(sbase + tc::W4 + 256u * s, tc::SBO_K128), tc::idesc(128, 16), s > 0);
            tc::commit(bar);
        }
        if (!wait_mma()) break;
        // output layer, squared error and its gradient 2 (y - t) / n on the used columns
        if (half == 0) {
            float v[16], g[16] = {};
            tc::ld16(lane_addr + tt::TD, v);
            if (in) {
#pragma unroll
                for (int c = 0; c < USED_OUT; c++) {
                    const float y = v[c] + sbias[384 + c];
                    const float tn = (Tg[(size_t)r * USED_OUT + c] - snorm[NY_MEAN + c]) / snorm[NY_STD + c];
                    const float e = y - tn;
                    lossSum += e * e;
                    g[c] = 2.0f * e / (float)n;
                    b4sum[c] += g[c];
                }
            }
            const float lo[8] = {g[0], g[1], g[2], g[3], g[4], g[5], g[6], g[7]}, hi[8] = {};
            *reinterpret_cast<uint4*>(sm + tt::DY + tc::off(row, 0, tt::SBO16)) = pack8(lo);
            *reinterpret_cast<uint4*>(sm + tt::DY + tc::off(row, 8, tt::SBO16)) = pack8(hi);
        }
        publish();
        // backward: the input gradient is committed, then the layer's weight gradient follows it
        if (warp == 0 && tc::elect_one()) {
            tc::mma(tmem + tt::TD, tt::kmajor(sbase + tt::DY, tt::SBO16), tt::mnmajor(sbase + tc::W4, tc::SBO_K128),
                    tc::idesc(128, 128) | tt::MN_B, 0u);
            tc::commit(bar);
            for (uint32_t s = 0; s < 8; s++)
                tc::mma(tmem + tt::TW4, tt::mnmajor(sbase + tt::H3 + 2u * tt::SBO128 * s, tt::SBO128),
                        tt::mnmajor(sbase + tt::DY + 2u * tt::SBO16 * s, tt::SBO16),
                        tc::idesc(128, 16) | tt::MN_A | tt::MN_B, accum | (s > 0));
        }
        if (!wait_mma()) break;
        relu_back(tt::H3, tt::SP, bsum[2]);
        publish();
        if (warp == 0 && tc::elect_one()) {
            for (uint32_t s = 0; s < HID / 16; s++)
                tc::mma(tmem + tt::TD, tt::kmajor(sbase + tt::SP + 256u * s, tt::SBO128),
                        tt::mnmajor(sbase + tc::W3 + 2u * tc::SBO_K128 * s, tc::SBO_K128),
                        tc::idesc(128, 128) | tt::MN_B, s > 0);
            tc::commit(bar);
            for (uint32_t s = 0; s < 8; s++)
                tc::mma(tmem + tt::TW3, tt::mnmajor(sbase + tt::SP + 2u * tt::SBO128 * s, tt::SBO128),
                        tt::mnmajor(sbase + tt::H2 + 2u * tt::SBO128 * s, tt::SBO128),
                        tc::idesc(128, 128) | tt::MN_A | tt::MN_B, accum | (s > 0));
        }
        if (!wait_mma()) break;                               // dW4's products are complete as well
        relu_back(tt::H2, tt::H3, bsum[1]);
        publish();
        if (warp == 0 && tc::elect_one()) {
            for (uint32_t s = 0; s < HID / 16; s++)
                tc::mma(tmem + tt::TD, tt::kmajor(sbase + tt::H3 + 256u * s, tt::SBO128),
                        tt::mnmajor(sbase + tc::W2 + 2u * tc::SBO_K128 * s, tc::SBO_K128),
                        tc::idesc(128, 128) | tt::MN_B, s > 0);
            tc::commit(bar);
            for (uint32_t s = 0; s < 8; s++)
                tc::mma(tmem + tt::TW2, tt::mnmajor(sbase + tt::H3 + 2u * tt::SBO128 * s, tt::SBO128),
                        tt::mnmajor(sbase + tt::H1 + 2u * tt::SBO128 * s, tt::SBO128),
                        tc::idesc(128, 128) | tt::MN_A | tt::MN_B, accum | (s > 0));
        }
        if (!wait_mma()) break;                               // dW3's products are complete as well
        relu_back(tt::H1, tt::H2, bsum[0]);
        publish();
        if (warp == 0 && tc::elect_one()) {
            for (uint32_t s = 0; s < 8; s++)
                tc::mma(tmem + tt::TW1, tt::mnmajor(sbase + tt::H2 + 2u * tt::SBO128 * s, tt::SBO128),
                        tt::mnmajor(sbase + tt::X + 2u * tt::SBO32 * s, tt::SBO32),
                        tc::idesc(128, 32) | tt::MN_A | tt::MN_B, accum | (s > 0));
            tc::commit(bar);
        }
        if (!wait_mma()) break;                               // every product of the tile
        accum = 1u;
    }
    pdl_trigger();
    float* out = part + (size_t)blockIdx.x * tt::PART;
    if (ok) {
        // weight gradients: lane = output row (input row for dW4), contiguous over the warp
        float v[32];
        const uint32_t lr = (warp & 3u) * 32u + lane;
        for (uint32_t c0 = half * 64u; c0 < half * 64u + 64u; c0 += 32u) {
            tc::ld32(lane_addr + tt::TW3 + c0, v);
#pragma unroll
            for (int j = 0; j < 32; j++) out[tt::P3 + (c0 + j) * 128u + lr] = v[j];
            tc::ld32(lane_addr + tt::TW2 + c0, v);
#pragma unroll
            for (int j = 0; j < 32; j++) out[tt::P2 + (c0 + j) * 128u + lr] = v[j];
        }
        if (half == 0) {
            tc::ld32(lane_addr + tt::TW1, v);
#pragma unroll
            for (int j = 0; j < 32; j++) out[tt::P1 + j * 128u + lr] = v[j];
        } else {
            float w[16];
            tc::ld16(lane_addr + tt::TW4, w);
#pragma unroll
            for (int j = 0; j < 16; j++) out[tt::P4 + j * 128u + lr] = w[j];
        }
        // biases: the four warps of a column half, in order
        float* red = reinterpret_cast<float*>(sm + tt::RED);   // [8 warps][64]
        for (int l = 0; l < 3; l++) {
            __syncthreads();
            red[warp * 64u + lane] = bsum[l][0];
            red[warp * 64u + 32u + lane] = bsum[l][1];
            __syncthreads();
            if (t < 128) {
                const uint32_t w0 = (t >> 6) * 4u, c = t & 63u;
                const uint32_t at = l == 0 ? tt::PB1 : (l == 1 ? tt::PB2 : tt::PB3);
                out[at + t] = ((red[w0 * 64u + c] + red[(w0 + 1u) * 64u + c]) + red[(w0 + 2u) * 64u + c]) +
                              red[(w0 + 3u) * 64u + c];
            }
        }
        __syncthreads();
        if (half == 0) {
#pragma unroll
            for (int k = 0; k <= USED_OUT; k++) {
                float s = k < USED_OUT ? b4sum[k < USED_OUT ? k : 0] : lossSum;
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) red[warp * 8u + k] = s;
            }
        }
        __syncthreads();
        if (t < 16) {
            float s = 0.0f;
            if (t < USED_OUT) s = ((red[t] + red[8 + t]) + red[16 + t]) + red[24 + t];
            out[tt::PB4 + t] = s;
        }
        if (t == 32) {
            out[tt::PL] = ((red[USED_OUT] + red[8 + USED_OUT]) + red[16 + USED_OUT]) + red[24 + USED_OUT];
            out[tt::PV] = 1.0f;
        }
    } else {
        if (t == 0) {
            atomicCAS(status, 0u, (uint32_t)AVBD_FAIL_WAIT_TIMEOUT);
            out[tt::PV] = 0.0f;
        }
        if (issue) {                    // products still in flight, the weight gradients' included (bounded waits)
            if (t == 0) tc::commit(bar);
            if (tc::wait(bar, phase ^ 1u)) tc::wait(bar, phase);
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tt::TMEM_COLS)
                     : "memory");
}

struct AdamArgs { float *prm, *m, *v; uint32_t step; float lr, b1, b2, eps; };

// Adds `parts` partial gradients in CTA order and stores the gradient (ADAM =
// false) or applies Adam to the fp32 parameters.  Blocks of 256 elements: for
// the matrices held as [in][out], eight inputs x 32 outputs, read along the
// outputs and, after an exchange in shared memory, written along the inputs
// (whole 32-byte sectors both ways).
template <bool ADAM>
__global__ void __launch_bounds__(256) k_train_reduce(const float* part, uint32_t parts, uint32_t n, float* grad,
                                                      AdamArgs a, float* loss) {
    using namespace mlp;
    __shared__ float ex[8][33];
    constexpr uint32_t B3 = 64, B2 = B3 + 64, B1 = B2 + 16, B4 = B1 + 8;   // blocks of dW3, dW2, dW1, dW4
    const uint32_t t = threadIdx.x, b = blockIdx.x;
    uint32_t src, dst = 0xFFFFFFFFu;
    const bool turn = b < B1;
    bool idle = false;
    if (turn) {
        const uint32_t q = b < B3 ? b : (b < B2 ? b - B3 : b - B2);
        const uint32_t cols = b < B2 ? 128u : 32u, i0 = (q >> 2) * 8u, o0 = (q & 3u) * 32u;
        src = (b < B3 ? tt::P3 : (b < B2 ? tt::P2 : tt::P1)) + (i0 + (t >> 5)) * 128u + o0 + (t & 31u);
        dst = (b < B3 ? OW3 : (b < B2 ? OW2 : OW1)) + (o0 + (t >> 3)) * cols + i0 + (t & 7u);
    } else if (b < B4) {
        src = tt::P4 + (b - B1) * 256u + t;
        dst = OW4 + (b - B1) * 256u + t;
    } else {
        const uint32_t i = (b - B4) * 256u + t;               // biases, then the loss
        src = tt::PB1 + i;
        if (i < 128) dst = OB1 + i;
        else if (i < 256) dst = OB2 + i - 128u;
        else if (i < 384) dst = OB3 + i - 256u;
        else if (i < 400) dst = OB4 + i - 384u;
        else idle = i > 400;                                  // i == 400: the loss
    }
    pdl_wait();
    // a CTA that gave up a wait left no partial: nothing is stored
    if (__syncthreads_or(t < parts && part[(size_t)t * tt::PART + tt::PV] != 1.0f) || idle) return;
    float s = 0.0f;
    uint32_t z = 0;
    for (; z + 8 <= parts; z += 8) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = part[(size_t)(z + k) * tt::PART + src];
#pragma unroll
        for (int k = 0; k < 8; k++) s += v[k];
    }
    for (; z < parts; z++) s += part[(size_t)z * tt::PART + src];
    if (turn) {
        ex[t >> 5][t & 31u] = s;
        __syncthreads();
        s = ex[t & 7u][t >> 3];
    }
    if (dst == 0xFFFFFFFFu) {
        if (loss) *loss = s * (1.0f / (float)n);              // mean over the batch
        return;
    }
    if (ADAM) {
        const float mi = a.b1 * a.m[dst] + (1.0f - a.b1) * s;
        const float vi = a.b2 * a.v[dst] + (1.0f - a.b2) * s * s;
        a.m[dst] = mi;
        a.v[dst] = vi;
        const float mh = mi / (1.0f - powf(a.b1, (float)a.step));
        const float vh = vi / (1.0f - powf(a.b2, (float)a.step));
        a.prm[dst] = a.prm[dst] - a.lr * mh / (sqrtf(vh) + a.eps);
    } else if (grad) {
        grad[dst] = s;
    }
}
constexpr uint32_t kTrainReduceBlocks = 64 + 64 + 16 + 8 + 2;

// BF16 weight image of the inference kernel: W1..W4 in the UMMA canonical
// K-major layout, byte for byte the kernel's shared-memory weight region.
__global__ void k_mirror_umma(const float* prm, unsigned char* img) {
    using namespace mlp;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= NHALF) return;
    uint32_t src, base, cols, sbo, j;
    if (i < HW2) { j = i - HW1; src = OW1; base = tc::W1; cols = DIN; sbo = tc::SBO_K32; }
    else if (i < HW3) { j = i - HW2; src = OW2; base = tc::W2; cols = HID; sbo = tc::SBO_K128; }
    else if (i < HW4) { j = i - HW3; src = OW3; base = tc::W3; cols = HID; sbo = tc::SBO_K128; }
    else { j = i - HW4; src = OW4; base = tc::W4; cols = HID; sbo = tc::SBO_K128; }
    const uint32_t r = j / cols, k = j % cols;
    *reinterpret_cast<bf16*>(img + base + tc::off(r, k, sbo)) = __float2bfloat16(prm[src + j]);
}

}  // namespace

// ---------------------------------------------------------------------------
// Host side of training.  Workspace for a batch of B rows: the status words
// (256 bytes: training's at 0, an inference's at 128), then one partial
// gradient per CTA of k_train_tile.
// ---------------------------------------------------------------------------
namespace {
constexpr uint32_t kInferStatus = 32;   // words
inline uint32_t blocks(size_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }

// one 128-row tile per CTA while the batch has no more tiles than the device
// SMs (an SM holds one CTA: 220 KiB of shared memory, all of TMEM)
uint32_t train_ctas(uint32_t B) { return std::min<uint32_t>((B >> 7) + ((B & 127u) ? 1u : 0u), 148u); }

struct Work {
    uint32_t* status;        // nonzero when a tensor-core wait gave up
    float* part;
};
size_t work_layout(uint32_t B, char* base, Work* w) {
    if (w) {
        w->status = reinterpret_cast<uint32_t*>(base);
        w->part = reinterpret_cast<float*>(base + 256);
    }
    return 256 + sizeof(float) * (size_t)tt::PART * train_ctas(B);
}

// 220 KiB of dynamic shared memory (set once per device)
void train_attributes() {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load() & bit) return;
    cudaFuncSetAttribute(k_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tt::SMEM);
    done.fetch_or(bit);
}

// Forward, loss and partial gradients; then their sum into `grad` (a == null)
// or Adam on the parameters.
void forward_backward(const float* prm, const float* norm, const float* X, const float* T, uint32_t B, const Work& w,
                      float* grad, const AdamArgs* a, float* loss, bool issue, cudaStream_t st) {
    train_attributes();
    const uint32_t ctas = train_ctas(B);
    k_train_tile<<<ctas, tt::THREADS, tt::SMEM, st>>>(prm, norm, X, T, B, w.part, w.status, issue);
    if (a) launch_pdl(k_train_reduce<true>, kTrainReduceBlocks, 256, st, (const float*)w.part, ctas, B, (float*)nullptr, *a, loss);
    else if (grad || loss)
        launch_pdl(k_train_reduce<false>, kTrainReduceBlocks, 256, st, (const float*)w.part, ctas, B, grad, AdamArgs{}, loss);
}
}  // namespace

// ---------------------------------------------------------------------------
// Solver integration
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ float step_scale(const Params& P) { return fmaxf(fabsf(P.gravity), 1.0f) * P.dt * P.dt; }

// bounding radius of a rigid body (the rotation's length scale)
__device__ __forceinline__ float learn_radius(const DevPtrs& d, uint32_t v) { return fmaxf(d.shape[v].w, 1e-6f); }

// Pose of learned row i moved by its prediction y from the plain warm start
// (xp, qp).  A zero rotation prediction keeps qp bit for bit.
__device__ __forceinline__ void learn_pose(const Params& P, const DevPtrs& d, uint32_t i, uint32_t v, float4 xp,
                                           float4 qp, float4& x, float4& q) {
    const float s = step_scale(P);
    const float* y = d.learnPred + (size_t)i * mlp::USED_OUT;
    x = mk4(xyz(xp) + mk3(y[0], y[1], y[2]) * s, xp.w);
    q = qp;
    if (i >= P.learnParticles && (y[3] != 0.0f || y[4] != 0.0f || y[5] != 0.0f))
        q = q_addw(qp, mk3(y[3], y[4], y[5]) * (s / learn_radius(d, v)));
}

// Per-vertex features at the plain warm start (see the file comment).  The
// contact features walk the body's per-frame segment (manifolds, element
// contacts), the stiffness feature its static segments (springs; tets,
// membranes, bends).
// Contact state of every learned vertex: count of contact points, closest
// gap and summed oriented normal of its manifolds and element contacts.
__global__ void k_learn_contacts(const Params P, const DevPtrs d, uint32_t n) {
    pdl_prologue();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t v = d.learnIdx[i];
    float count = 0.0f, gap = 1e30f;
    float3 nsum = s3(0);
    const uint32_t ds = d.dynStart[v], dc = d.dynCount[v];
    for (uint32_t k = 0; k < dc; k++) {
        const uint32_t e = d.dynList[ds + k];
        const uint32_t kind = e >> ADJ_KIND_SHIFT;
        if (kind == FK_MANIFOLD) {
            const ManifoldGPU& m = d.manifolds[e & ADJ_INDEX_MASK];
            const float sg = m.header.x == v ? 1.0f : -1.0f;
            nsum += xyz(m.basisN) * sg;
            for (uint32_t c = 0; c < m.header.z; c++) {
                count += 1.0f;
                gap = fminf(gap, m.contacts[c].C0.x);
            }
        } else if (kind == FK_SOFT) {
            // element contact: the vertex's side of the stencil gives the sign
            const SoftContactGPU& sc = d.soft[e & ADJ_INDEX_MASK];
            const float w = sc.ids.x == v ? sc.weights.x : (sc.ids.y == v ? sc.weights.y
                                                            : (sc.ids.z == v ? sc.weights.z : sc.weights.w));
            nsum += xyz(sc.normal) * (w >= 0.0f ? 1.0f : -1.0f);
            count += 1.0f;
            gap = fminf(gap, sc.C0.x);
        }
    }
    d.learnStat[i] = mk4(nsum, count);
    d.learnGap[i] = gap;
}

// Features of every learned vertex.  The static parts (incident stiffness,
// the 1-ring of vertices sharing a tet or spring with its multiplicities)
// are precomputed at upload; the ring's contact state sums the neighbours'
// contact counts (times their multiplicity) and takes their closest gap.
__global__ void k_learn_features(const Params P, const DevPtrs d, uint32_t n) {
    pdl_prologue();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t v = d.learnIdx[i];
    const float s = step_scale(P);
    const float4 pl = d.posLin[v];
    const float3 x0 = xyz(d.initLin[v]);
    const float3 fi = (xyz(d.inertLin[v]) - x0) / s;
    const float3 fp = (xyz(pl) - x0) / s;
    const float3 fv = xyz(d.prevVelLin[v]) * (P.dt / s);
    const float4 st = d.learnStat[i];
    const float3 nsum = xyz(st);
    const float count = st.w, gap = d.learnGap[i];
    const float stiff = d.learnStiff[i];
    const float ringN = d.learnRingN[i];
    float ringContacts = 0.0f, ringGap = 1e30f;
    const uint32_t r1 = d.learnRingStart[i + 1];
    for (uint32_t k = d.learnRingStart[i]; k < r1; k++) {
        const uint2 e = d.learnRing[k];
        ringContacts += d.learnStat[e.x].w * (float)e.y;
        ringGap = fminf(ringGap, d.learnGap[e.x]);
    }
    const float inv = ringN > 0.0f ? 1.0f / ringN : 0.0f;
    float* f = d.learnFeat + (size_t)i * mlp::DIN;
    for (int k = 16; k < 25; k++) f[k] = 0.0f;          // rigid slots, reserved
    if (i >= P.learnParticles) {
        const float r = learn_radius(d, v);
        const float4 q = d.posAng[v];
        const float3 wq = q_sub(q, d.initAng[v]) * (r / s);
        const float3 up = q_rotate(q_conj(q), mk3(0, 0, 1));
        f[16] = 1.0f;
        f[17] = wq.x; f[18] = wq.y; f[19] = wq.z;
        f[20] = up.x; f[21] = up.y; f[22] = up.z;
        f[23] = 0.1f * log1pf(r / s);
    }
    f[25] = ringN * 0.1f;
    f[26] = ringContacts * inv * 0.25f;
    f[27] = ringContacts > 0.0f ? fminf(fmaxf(ringGap / s, -10.0f), 10.0f) : 10.0f;
    f[28] = 0.0f; f[29] = 0.0f; f[30] = 0.0f; f[31] = 0.0f;
    if (i >= P.learnParticles) {
        // position-PD hinge motors acting on the body (they are in its
        // static segment): the rotation each asks for, and their gains
        const float r = learn_radius(d, v);
        const uint4 sg = d.staticSeg[v];
        float motors = 0.0f, gain = 0.0f;
        float3 want = s3(0.0f);
        for (uint32_t k = 0; k < sg.y; k++) {
            const uint32_t e = d.preList[sg.x + k];
            if ((e >> ADJ_KIND_SHIFT) != FK_JOINT) continue;
            const JointGPU& j = d.joints[e & ADJ_INDEX_MASK];
            const uint32_t mode = j.header.w & MOTOR_MODE_MASK;
            if (!(j.motor.y > 0.0f) || j.hingeAxis.w == 0.0f || mode == MOTOR_EXPLICIT || mode == MOTOR_VELOCITY)
                continue;
            const uint32_t a = j.header.x, b = j.header.y;
            const float4 qA = a == WORLD_BODY ? make_float4(0, 0, 0, 1) : d.posAng[a];
            const float4 qB = d.posAng[b];
            const float3 axis = xyz(j.hingeAxis);
            const float Cm = wrap_pi(twist_angle(q_mul(qA, tof(j.restRel)), qB, axis) - j.motor.x);
            want += q_rotate(qB, axis) * (v == a ? Cm : -Cm);
            motors += 1.0f;
            gain += j.motor.w;
        }
        const float3 w = want * (r / s);
        f[24] = motors * 0.25f;
        f[28] = w.x; f[29] = w.y; f[30] = w.z;
        f[31] = log1pf(gain * P.dt * P.dt / fmaxf(pl.w * r * r, 1e-12f));
    }
    f[0] = fi.x; f[1] = fi.y; f[2] = fi.z;
    f[3] = fp.x; f[4] = fp.y; f[5] = fp.z;
    f[6] = fv.x; f[7] = fv.y; f[8] = fv.z;
    f[9] = count * 0.25f;
    f[10] = nsum.x; f[11] = nsum.y; f[12] = nsum.z;
    f[13] = count > 0.0f ? fminf(fmaxf(gap / s, -10.0f), 10.0f) : 10.0f;
    f[14] = log1pf(stiff * P.dt * P.dt / fmaxf(pl.w, 1e-12f));
    f[15] = 1.0f;
}

// x0 = x_plain + s * prediction for every learned row
__global__ void k_learn_apply(const Params P, const DevPtrs d, uint32_t n) {
    pdl_prologue();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t v = d.learnIdx[i];
    learn_pose(P, d, i, v, d.learnSaveLin[v], d.learnSaveAng[v], d.posLin[v], d.posAng[v]);
}

// keep the prediction when its residual after the trial sweeps is no worse
__global__ void k_learn_select(const Params P, const DevPtrs d, uint32_t n) {
    pdl_prologue();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool accept = d.learnResid[1] <= d.learnResid[0];
    if (i == 0 && accept) atomicAdd(d.learnAccepted, 1u);
    if (i >= n || !accept) return;
    const uint32_t v = d.learnIdx[i];
    learn_pose(P, d, i, v, d.learnSaveLin[v], d.learnSaveAng[v], d.posLin[v], d.posAng[v]);
}

// Pose buffers of the predicted branch: the solver's pose with every
// learned row (the first n slots) moved by its prediction.
__global__ void k_learn_branch(const Params P, const DevPtrs d, uint32_t nb, uint32_t n) {
    pdl_prologue();
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const uint32_t slot = d.learnSlot[b];
    if (slot < n) {
        learn_pose(P, d, slot, b, d.posLin[b], d.posAng[b], d.learnSweptLin[b], d.learnSweptAng[b]);
    } else {
        d.learnSweptLin[b] = d.posLin[b];
        d.learnSweptAng[b] = d.posAng[b];
    }
}

// After both trial sweeps: adopt the predicted branch's swept pose when its
// residual is no worse; otherwise the plain branch's pose stays.
__global__ void k_learn_adopt(const Params P, const DevPtrs d, uint32_t nb) {
    pdl_prologue();
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    const bool accept = d.learnResid[1] <= d.learnResid[0];
    if (b == 0 && accept) atomicAdd(d.learnAccepted, 1u);
    // the kept trial sweep is the first pass: its OGC bound-exceeder count
    // moves to the first pass's slot
    if (b == 0 && P.ogc) d.counters->ogcSlots[0] = d.counters->ogcSlots[accept ? 3 : 2];
    if (b >= nb || !accept) return;
    d.posLin[b] = d.learnSweptLin[b];
    d.posAng[b] = d.learnSweptAng[b];
}

// training target: the solve's correction of the plain warm start (the
// rotation part zero for particles)
__global__ void k_learn_target(const Params P, const DevPtrs d, uint32_t n) {
    pdl_prologue();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t v = d.learnIdx[i];
    const float s = step_scale(P);
    const float3 t = (xyz(d.posLin[v]) - xyz(d.learnSaveLin[v])) / s;
    const float3 w = i >= P.learnParticles ? q_sub(d.posAng[v], d.learnSaveAng[v]) * (learn_radius(d, v) / s)
                                           : s3(0.0f);
    float* y = d.learnTarget + (size_t)i * mlp::USED_OUT;
    y[0] = t.x; y[1] = t.y; y[2] = t.z;
    y[3] = w.x; y[4] = w.y; y[5] = w.z;
}

__global__ void k_copy_double(const double* src, double* dst) {
    pdl_prologue();
    if (threadIdx.x == 0 && blockIdx.x == 0) *dst = *src;
}

}  // namespace

void launch_learn_features(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    if (!z.numLearn) return;
    launch_pdl(k_learn_contacts, (z.numLearn + 127) / 128, 128, st, P, d, z.numLearn);
    launch_pdl(k_learn_features, (z.numLearn + 127) / 128, 128, st, P, d, z.numLearn);
}
void launch_learn_apply(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    if (z.numLearn) launch_pdl(k_learn_apply, (z.numLearn + 127) / 128, 128, st, P, d, z.numLearn);
}
void launch_learn_select(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    launch_pdl(k_learn_select, (z.numLearn + 128) / 128, 128, st, P, d, z.numLearn);
}
void launch_learn_branch(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    launch_pdl(k_learn_branch, (z.numBodies + 127) / 128, 128, st, P, d, z.numBodies, z.numLearn);
}
void launch_learn_adopt(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    launch_pdl(k_learn_adopt, (z.numBodies + 127) / 128, 128, st, P, d, z.numBodies);
}
void launch_learn_target(const Params& P, const DevPtrs& d, const Sizes& z, cudaStream_t st) {
    if (z.numLearn) launch_pdl(k_learn_target, (z.numLearn + 127) / 128, 128, st, P, d, z.numLearn);
}
void launch_copy_double(const double* src, double* dst, cudaStream_t st) { launch_pdl(k_copy_double, 1, 32, st, src, dst); }

// weights, two input tiles, biases and normalisation: 98 KiB of shared memory
// (set once per device)
static void mlp_infer_attributes() {
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const uint64_t bit = 1ull << (dev & 63);
    if (done.load() & bit) return;
    cudaFuncSetAttribute(k_mlp_infer_tc<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::SMEM);
    cudaFuncSetAttribute(k_mlp_infer_tc<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::SMEM);
    done.fetch_or(bit);
}

// halfW: the weight image of launch_mlp_mirror, or null to convert `prm` in
// the kernel (a call that would otherwise need the image written first)
void launch_mlp_infer(const void* halfW, const float* prm, const float* norm, const float* X, uint32_t n, float* Y,
                      uint32_t* status, cudaStream_t st) {
    if (n == 0) return;
    mlp_infer_attributes();
    const uint32_t tiles = n / tc::ROWS + (n % tc::ROWS ? 1u : 0u);
    const uint32_t blocks = std::min<uint32_t>(tiles, 148u);
    const bf16* W = static_cast<const bf16*>(halfW);
    if (W) k_mlp_infer_tc<true><<<blocks, tc::GROUPS * tc::GROUP_THREADS, tc::SMEM, st>>>(W, prm, norm, X, n, Y, status, true);
    else k_mlp_infer_tc<false><<<blocks, tc::GROUPS * tc::GROUP_THREADS, tc::SMEM, st>>>(W, prm, norm, X, n, Y, status, true);
}

void launch_mlp_mirror(const float* prm, void* halfW, cudaStream_t st) {
    k_mirror_umma<<<blocks(mlp::NHALF, 256), 256, 0, st>>>(prm, static_cast<unsigned char*>(halfW));
}

uint32_t mlp_param_count() { return mlp::NPARAM; }
uint32_t mlp_half_count() { return mlp::NHALF; }
uint32_t mlp_norm_count() { return mlp::NNORM; }

}  // namespace avbd

// ---------------------------------------------------------------------------
// C ABI of the training kernels (no counterpart in the reference: the learned
// warm start is new).  Every pointer is device memory; `stream` is a
// cudaStream_t or null.
// ---------------------------------------------------------------------------
using namespace avbd;
extern "C" {

uint32_t avbd_mlp_param_count(void) { return mlp::NPARAM; }

size_t avbd_mlp_workspace_bytes(uint32_t batch) { return work_layout(batch, nullptr, nullptr); }

// status word of a workspace: cleared, or read after a synchronisation
static int workspace_status(const Work& w, cudaStream_t st) {
    uint32_t h = 0;
    if (cudaMemcpyAsync(&h, w.status, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return AVBD_ERR_RUNTIME_FAILURE;
    return h == 0 ? AVBD_OK : AVBD_ERR_RUNTIME_FAILURE;
}

static int gradients(const float* params, const float* norm, const float* features, const float* targets,
                     uint32_t batch, void* workspace, float* grad_out, const AdamArgs* adam, float* loss_out,
                     bool issue, cudaStream_t st) {
    if (!params || !norm || !features || !targets || !workspace || batch == 0) return AVBD_ERR_INVALID_ARGUMENT;
    Work w{};
    work_layout(batch, static_cast<char*>(workspace), &w);
    if (!adam) cudaMemsetAsync(w.status, 0, sizeof(uint32_t), st);
    forward_backward(params, norm, features, targets, batch, w, grad_out, adam, loss_out, issue, st);
    if (cudaGetLastError() != cudaSuccess) return AVBD_ERR_RUNTIME_FAILURE;
    // a tensor-core wait that gave up fails the call (the kernel latches it
    // in the workspace's status word); the training step stays asynchronous
    return adam ? AVBD_OK : workspace_status(w, st);
}

int avbd_mlp_gradients(const float* params, const float* norm, const float* features, const float* targets,
                       uint32_t batch, void* workspace, float* grad_out, float* loss_out, void* stream) {
    return gradients(params, norm, features, targets, batch, workspace, grad_out, nullptr, loss_out, true,
                     static_cast<cudaStream_t>(stream));
}

int avbd_mlp_workspace_status(const void* workspace, uint32_t batch, void* stream) {
    if (!workspace || batch == 0) return AVBD_ERR_INVALID_ARGUMENT;
    Work w{};
    work_layout(batch, static_cast<char*>(const_cast<void*>(workspace)), &w);
    return workspace_status(w, static_cast<cudaStream_t>(stream));
}

static int train_step(float* params, const float* norm, const float* features, const float* targets, uint32_t batch,
                      float* adam_m, float* adam_v, uint32_t step, float lr, void* workspace, float* loss_out,
                      void* stream, bool issue) {
    if (!params || !adam_m || !adam_v || step == 0) return AVBD_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (workspace && batch && step == 1) {
        Work w{};
        work_layout(batch, static_cast<char*>(workspace), &w);
        cudaMemsetAsync(w.status, 0, sizeof(uint32_t), st);   // sticky from here on
    }
    const AdamArgs adam{params, adam_m, adam_v, step, lr, 0.9f, 0.999f, 1e-8f};
    return gradients(params, norm, features, targets, batch, workspace, nullptr, &adam, loss_out, issue, st);
}

int avbd_mlp_train_step(float* params, const float* norm, const float* features, const float* targets,
                        uint32_t batch, float* adam_m, float* adam_v, uint32_t step, float lr, void* workspace,
                        float* loss_out, void* stream) {
    return train_step(params, norm, features, targets, batch, adam_m, adam_v, step, lr, workspace, loss_out, stream,
                      true);
}

int avbd_mlp_train_step_wait_timeout_for_testing(float* params, const float* norm, const float* features,
                                                 const float* targets, uint32_t batch, float* adam_m, float* adam_v,
                                                 uint32_t step, float lr, void* workspace, float* loss_out,
                                                 void* stream) {
    return train_step(params, norm, features, targets, batch, adam_m, adam_v, step, lr, workspace, loss_out, stream,
                      false);
}

static int mlp_infer(const float* params, const float* norm, const float* features, uint32_t n, float* out,
                     void* workspace, void* stream, bool issue) {
    if (!params || !norm || !features || !out || !workspace) return AVBD_ERR_INVALID_ARGUMENT;
    // bulk copies and vector loads read the weight image, the biases, the
    // normalisation block and the feature rows in 16-byte units
    if ((reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(features) |
         reinterpret_cast<uintptr_t>(params) | reinterpret_cast<uintptr_t>(norm)) & 15u)
        return AVBD_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // not the training status word, which is sticky in a shared workspace
    uint32_t* status = static_cast<uint32_t*>(workspace) + kInferStatus;
    cudaMemsetAsync(status, 0, sizeof(uint32_t), st);
    if (issue) {
        launch_mlp_infer(nullptr, params, norm, features, n, out, status, st);
    } else if (n) {
        mlp_infer_attributes();
        k_mlp_infer_tc<false><<<1, tc::GROUPS * tc::GROUP_THREADS, tc::SMEM, st>>>(nullptr, params, norm, features, n, out, status,
                                                                     false);
    }
    uint32_t h = 0;
    if (cudaMemcpyAsync(&h, status, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return AVBD_ERR_RUNTIME_FAILURE;
    return h == 0 ? AVBD_OK : AVBD_ERR_RUNTIME_FAILURE;
}

int avbd_mlp_infer(const float* params, const float* norm, const float* features, uint32_t n, float* out,
                   void* workspace, void* stream) {
    return mlp_infer(params, norm, features, n, out, workspace, stream, true);
}

int avbd_mlp_infer_wait_timeout_for_testing(const float* params, const float* norm, const float* features,
                                            uint32_t n, float* out, void* workspace, void* stream) {
    return mlp_infer(params, norm, features, n, out, workspace, stream, false);
}

}  // extern "C"
