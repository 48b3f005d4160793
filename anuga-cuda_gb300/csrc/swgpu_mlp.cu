// swgpu_mlp.cu -- BF16 surrogate network of the solver's maximum depth and
// arrival time, on the 5th-generation tensor cores (tcgen05, TMEM).
//
// Rows are (scenario s, triangle k) pairs.  Each row's 16 input features
// are assembled on the fly: the scenario's 9 parameters, the triangle's
// centroid x and y, bed elevation and distance to the inflow, and 3 zeros,
// each normalised by a per-feature affine map.  The network is
//   16 -> 256 -> 256 -> 256 -> 3  (ReLU after each hidden layer)
// with weights and activations in BF16 and every product accumulated in
// FP32; its outputs are the normalised maximum depth, the normalised
// arrival time and the 90% quantile of the first output's absolute error.
//
// Every matrix is kept as core-matrix images (see "blocked images"), so the
// same bytes serve products over the features, the outputs and the rows; a
// kernel keeps the weights of its layer in shared memory and walks tiles of
// 128 rows, each a tcgen05.mma (kind::f16) into FP32 accumulators in tensor
// memory read back with tcgen05.ld:
//   mlp_predict         inference: the whole network (half of each matrix
//                       resident in each CTA of a pair)
//   mlp_layers12        training: features, layers 1 and 2 (W1, W2 resident)
//   mlp_layer3_train    layer 3 and the 256 -> 3 output layer, the loss, the
//                       output layer's gradients and the gradient back through
//                       layer 3 (W3 resident)
//   mlp_back2           the gradient back through layer 2 (W2 resident)
//   mlp_wgrad           the weight and bias gradients, split over the rows
//   mlp_finish          the splits' sums in a fixed order, Adam on the FP32
//                       master weights and the BF16 images
// Inference is the first, training the other five launches.  No sum
// depends on the order in which blocks finish.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "swgpu_internal.cuh"

namespace {

constexpr int kF = 16;       // input features (13 used)
constexpr int kH = 256;      // hidden units per layer
constexpr int kOut = 3;      // outputs: depth, arrival time, depth-error estimate
constexpr int kTargets = 2;  // targets per row: depth, arrival time
constexpr int kParams = 9;   // scenario parameters
constexpr int kTri = 4;      // per-triangle table: x, y, z, distance to the inflow
constexpr float kQuantile = 0.9f;  // quantile of the depth error the third output learns

// flat FP32 parameter vector, weights in-major ([in][out]):
// W1 [16][256], b1, W2 [256][256], b2, W3 [256][256], b3, W4 [256][3], b4
constexpr long kOffW1 = 0;
constexpr long kOffB1 = kOffW1 + kF * kH;
constexpr long kOffW2 = kOffB1 + kH;
constexpr long kOffB2 = kOffW2 + kH * kH;
constexpr long kOffW3 = kOffB2 + kH;
constexpr long kOffB3 = kOffW3 + kH * kH;
constexpr long kOffW4 = kOffB3 + kH;
constexpr long kOffB4 = kOffW4 + kH * kOut;
constexpr long kNumParams = kOffB4 + kOut;

// ---- blocked images ---------------------------------------------------------
//
// Every matrix that a tensor-core product reads is kept, in global and in
// shared memory alike, as 16-byte vectors of 8 BF16 in core-matrix order:
//   activations and their gradients: per tile of 128 rows
//     [feature / 8][row][8]          (64 kB for 256 features, 4 kB for 16)
//   weights: [in / 8][out][8 in]     (128 kB for 256 x 256, 8 kB for 16 x 256)
// Eight rows of one vector are a 128-byte core matrix, so one image serves a
// product that runs over the features (K-major: a layer forward) and one that
// runs over the rows (MN-major: a weight gradient) or over the outputs (a
// layer backward): only the two strides of the descriptor change places.  A
// tile is one contiguous bulk copy, and a warp that writes one vector per row
// writes 512 contiguous bytes.

constexpr int kTileM = 128;                      // rows per tile (TMEM lanes)
constexpr unsigned kActStride = kTileM * 16;     // bytes between 8-feature vectors
constexpr unsigned kActBytes = kTileM * kH * 2;  // one tile of activations
constexpr unsigned kXBytes = kTileM * kF * 2;    // one tile of features
constexpr unsigned kWStride = kH * 16;
constexpr unsigned kWBytes = kH * kH * 2;
constexpr unsigned kW1Bytes = kF * kH * 2;

struct __align__(128) BfWeights {
    __nv_bfloat16 w2[kH * kH];
    __nv_bfloat16 w3[kH * kH];
    __nv_bfloat16 w1[kF * kH];
    float4 w4[kH];  // the three BF16 weights of each hidden unit, widened
};
// place of weight (in, out) in its image
__host__ __device__ __forceinline__ int w_at(int in, int out) {
    return ((in >> 3) * kH + out) * 8 + (in & 7);
}

// ---- features --------------------------------------------------------------

struct FeatureTables {
    const float *scen;   // [S][9]
    const float *tri;    // [N][4]: x, y, z, distance to the inflow
    const float *mu;     // [16]
    const float *isd;    // [16]
    long long N;
};

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// The rows of a batch: given, drawn uniformly from all (scenario, triangle)
// pairs (seeded), or consecutive from row0 (inference).
struct Batch {
    const long long *rows;
    unsigned long long seed;
    long long total;  // > 0: drawn
    long long row0;
    long long nrows;
};
__device__ __forceinline__ long long batch_row(const Batch &b, long long r) {
    if (b.rows) return b.rows[r];
    if (b.total > 0)
        return (long long)(mix64(b.seed ^ (unsigned long long)r * 0xD1B54A32D192ED03ull) %
                           (unsigned long long)b.total);
    return b.row0 + r;
}

// Normalised BF16 features of batch row r (zero past the last row) into its
// two vectors of the tile at x; returns the data row.
__device__ __forceinline__ long long tile_features(const FeatureTables &F, const Batch &b,
                                                   const float *norm, long long r, int trow,
                                                   unsigned char *x) {
    __align__(16) __nv_bfloat162 o[kF / 2];
    long long q = 0;
    if (r < b.nrows) {
        q = batch_row(b, r);
        const long long s = q / F.N, k = q - s * F.N;
        const float4 tr = __ldg(reinterpret_cast<const float4 *>(F.tri) + k);
        float v[kF];
#pragma unroll
        for (int c = 0; c < kParams; c++) v[c] = __ldg(F.scen + s * kParams + c);
        v[9] = tr.z;   // bed
        v[10] = tr.x;
        v[11] = tr.y;
        v[12] = tr.w;  // distance to the inflow
        v[13] = v[14] = v[15] = 0.0f;
#pragma unroll
        for (int c = 0; c < kF; c++) v[c] = (v[c] - norm[c]) * norm[kF + c];
#pragma unroll
        for (int c = 0; c < kF / 2; c++) o[c] = __floats2bfloat162_rn(v[2 * c], v[2 * c + 1]);
    } else {
#pragma unroll
        for (int c = 0; c < kF / 2; c++) o[c] = __floats2bfloat162_rn(0.0f, 0.0f);
    }
    *reinterpret_cast<uint4 *>(x + trow * 16) = reinterpret_cast<const uint4 *>(o)[0];
    *reinterpret_cast<uint4 *>(x + kActStride + trow * 16) = reinterpret_cast<const uint4 *>(o)[1];
    return q;
}

// ---- tcgen05, mbarriers, bulk copies ---------------------------------------

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor: start, the byte offsets between core
// matrices along K (leading) and along M or N (stride), descriptor version 1
// (bit 46), no swizzle.
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned along_k,
                                                        unsigned along_mn) {
    return (unsigned long long)((addr >> 4) & 0x3FFFu) |
           ((unsigned long long)((along_k >> 4) & 0x3FFFu) << 16) |
           ((unsigned long long)((along_mn >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: FP32 accumulator, BF16 A and B (each
// K-major or MN-major), M = 128, N given.
__host__ __device__ constexpr unsigned tc_idesc(int n, bool a_mn, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)a_mn << 15) | ((unsigned)b_mn << 16) |
           ((unsigned)(n >> 3) << 17) | ((unsigned)(kTileM >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(unsigned d_tmem, unsigned long long a,
                                       unsigned long long b, unsigned idesc, bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"((unsigned)accumulate)
        : "memory");
}
__device__ __forceinline__ void tc_commit(unsigned long long *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void proxy_fence() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// A CTA's barrier after which the tensor core may read what its threads
// wrote to shared memory and overwrite what they read from tensor memory.
__device__ __forceinline__ void tc_sync() {
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}
// 32 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld32(unsigned taddr, float (&v)[32]) {
    unsigned r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
        "%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
          "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
// 8 consecutive FP32 columns at each of two places of this thread's lane
__device__ __forceinline__ void tc_ld8x2(unsigned a, unsigned b, float (&v)[8], float (&w)[8]) {
    unsigned r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                   "=r"(r[6]), "=r"(r[7])
                 : "r"(a));
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                   "=r"(r[14]), "=r"(r[15])
                 : "r"(b));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) {
        v[i] = __uint_as_float(r[i]);
        w[i] = __uint_as_float(r[8 + i]);
    }
}
// 8 consecutive FP32 columns of this thread's lane at each of 8 places, 32
// columns apart
__device__ __forceinline__ void tc_ld8x8(unsigned taddr, float (&v)[8][8]) {
    unsigned r[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[i][0]), "=r"(r[i][1]), "=r"(r[i][2]), "=r"(r[i][3]), "=r"(r[i][4]),
                       "=r"(r[i][5]), "=r"(r[i][6]), "=r"(r[i][7])
                     : "r"(taddr + 32 * i));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) v[i][j] = __uint_as_float(r[i][j]);
}
// 32 columns of 32 lanes (rows) by a warp, a thread's part being four rows of
// two neighbouring columns in every eight: v[b][i] is row 8 i + lane / 4 of
// columns 8 b + 2 (lane % 4) and the next.
__device__ __forceinline__ void tc_ld_quads(unsigned taddr, float2 (&v)[4][4]) {
    unsigned r[2][16];
#pragma unroll
    for (int i = 0; i < 2; i++)
        asm volatile(
            "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
            "%13,%14,%15}, [%16];"
            : "=r"(r[i][0]), "=r"(r[i][1]), "=r"(r[i][2]), "=r"(r[i][3]), "=r"(r[i][4]),
              "=r"(r[i][5]), "=r"(r[i][6]), "=r"(r[i][7]), "=r"(r[i][8]), "=r"(r[i][9]),
              "=r"(r[i][10]), "=r"(r[i][11]), "=r"(r[i][12]), "=r"(r[i][13]), "=r"(r[i][14]),
              "=r"(r[i][15])
            : "r"(taddr + ((unsigned)(16 * i) << 16)));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int b = 0; b < 4; b++)
#pragma unroll
        for (int i = 0; i < 4; i++)
            v[b][i] = make_float2(__uint_as_float(r[i >> 1][4 * b + 2 * (i & 1)]),
                                  __uint_as_float(r[i >> 1][4 * b + 2 * (i & 1) + 1]));
}
// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld16(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
        "%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_alloc(unsigned *base, unsigned columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(base)),
                 "r"(columns)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(unsigned base, unsigned columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns)
                 : "memory");
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
constexpr int kTcWaitLimit = 1 << 22;
// Bounded wait; on running out the status is set, what is in flight gets as
// long again to land before its memory is given up, and false is returned.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity, int *status) {
    for (int i = 0; i < kTcWaitLimit; i++)
        if (mbar_test(bar, parity)) return true;
    atomicExch(status, SWGPU_ETIMEOUT);
    for (int i = 0; i < kTcWaitLimit; i++)
        if (mbar_test(bar, parity)) break;
    return false;
}
// Arrives at the barrier that CTA `rank` of the cluster has where this one
// has `bar`.  It passes on that this CTA's own shared and tensor memory is
// ready for the tensor core (the caller's proxy_fence and tc_fence_before),
// no data that the other CTA's threads read.  It names no scope, so its release
// and the other CTA's wait are at CTA scope: that the product issued there sees
// this CTA's shared memory rests on the fence before it having completed here
// and on how pairs of CTAs are commonly handed their operands, not on the memory
// model's letter.  A release at cluster scope would also wait for the warp's
// stores to global memory (1,000 clocks and more: 1,441 us for 3.2 million rows
// instead of 740); inference equals the training forward, which needs no pair,
// bit for bit.
__device__ __forceinline__ void mbar_arrive_at(unsigned long long *bar, unsigned rank) {
    asm volatile(
        "{\n .reg .b32 a;\n mapa.shared::cluster.u32 a, %0, %1;\n"
        " mbarrier.arrive.shared::cluster.b64 _, [a];\n}" ::"r"(smem_u32(bar)),
        "r"(rank)
        : "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// The same by the whole CTA, which it also brings together: true when all
// saw the phase complete.
__device__ __forceinline__ bool cta_wait(unsigned long long *bar, unsigned parity, int *status) {
    return __syncthreads_and(mbar_wait(bar, parity, status)) != 0;
}
// bulk copies (addresses and size multiples of 16)
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes,
                                          unsigned long long *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void bulk_store(void *dst, const void *src, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(smem_u32(src)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_store_read() {  // the sources may be overwritten
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_store_done() {
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// D (128 x 256) = A (a tile of activations) x W: over the features, or
// backward over the outputs.
__device__ __forceinline__ void mma_layer(unsigned d, unsigned a, unsigned w, bool accumulate) {
    // 128 of the 256 features: a half that one bulk copy brings
#pragma unroll
    for (int kk = 0; kk < 8; kk++)
        tc_mma(d, smem_desc(a + 2 * kActStride * kk, kActStride, 128),
               smem_desc(w + 2 * kWStride * kk, kWStride, 128), tc_idesc(kH, false, false),
               accumulate || kk > 0);
}
__device__ __forceinline__ void mma_layer_back(unsigned d, unsigned a, unsigned w) {
#pragma unroll
    for (int kk = 0; kk < 16; kk++)
        tc_mma(d, smem_desc(a + 2 * kActStride * kk, kActStride, 128),
               smem_desc(w + 256 * kk, 128, kWStride), tc_idesc(kH, false, true), kk > 0);
}

// A thread's part of an epilogue: the tile row of its TMEM lane and one of
// `groups` equal parts of the columns.  Warp w reaches lanes 32 (w % 4) .. + 31
// only.
struct Part {
    int row, group, col0;
    unsigned tmem;  // its lane's first column
};
template <int groups>
__device__ __forceinline__ Part my_part(unsigned tmem) {
    const int warp = threadIdx.x >> 5;
    Part p;
    p.row = 32 * (warp & 3) + (threadIdx.x & 31);
    p.group = warp >> 2;
    p.col0 = kH / groups * p.group;
    p.tmem = tmem + ((unsigned)(32 * (warp & 3)) << 16);
    return p;
}
__device__ __forceinline__ uint4 pack8(const float *v) {
    __align__(16) __nv_bfloat162 o[4];
#pragma unroll
    for (int j = 0; j < 4; j++) o[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
    return *reinterpret_cast<const uint4 *>(o);
}
// two FP32 operations in one instruction
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("{\n .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
        " add.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
        " mov.b64 z, {%6, %7};\n fma.rn.f32x2 x, x, y, z;\n mov.b64 {%0, %1}, x;\n}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
// bias and ReLU of n columns from c0, in place
template <int n>
__device__ __forceinline__ void bias_relu(float (&v)[n], const float *bias, int c0) {
#pragma unroll
    for (int q = 0; q < n / 4; q++) {
        const float4 b = *reinterpret_cast<const float4 *>(bias + c0 + 4 * q);
        const float2 lo = add2(make_float2(v[4 * q], v[4 * q + 1]), make_float2(b.x, b.y));
        const float2 hi = add2(make_float2(v[4 * q + 2], v[4 * q + 3]), make_float2(b.z, b.w));
        v[4 * q] = fmaxf(lo.x, 0.0f);
        v[4 * q + 1] = fmaxf(lo.y, 0.0f);
        v[4 * q + 2] = fmaxf(hi.x, 0.0f);
        v[4 * q + 3] = fmaxf(hi.y, 0.0f);
    }
}
// A layer's epilogue is a chain of tensor memory read, arithmetic and store
// per 32 columns: sixteen warps, four on a scheduler, hide one another's.  (A
// training step of 32,768 rows: 108 us with eight, 104 with sixteen.)
constexpr int kGroups = 4;
constexpr int kThreads = 128 * kGroups;

// A hidden layer's epilogue: activations of the accumulator at column d into
// the tile images at global and, when asked for, smem.
template <bool SMEM>
__device__ __forceinline__ void hidden_epilogue(const Part &p, unsigned d, const float *bias,
                                                unsigned char *smem, unsigned char *global) {
#pragma unroll 1
    for (int c0 = p.col0; c0 < p.col0 + kH / kGroups; c0 += 32) {
        float v[32];
        tc_ld32(p.tmem + d + c0, v);
        bias_relu(v, bias, c0);
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint4 o = pack8(v + 8 * q);
            const size_t at = (size_t)(c0 / 8 + q) * kActStride + p.row * 16;
            if (SMEM) *reinterpret_cast<uint4 *>(smem + at) = o;
            *reinterpret_cast<uint4 *>(global + at) = o;
        }
    }
}
// Bits of the eight BF16 of a vector that are above zero (a ReLU's output).
__device__ __forceinline__ unsigned positive8(const uint4 &u) {
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        m |= ((short)(w[j] & 0xffffu) > 0 ? 1u : 0u) << (2 * j);
        m |= ((int)w[j] >> 16 > 0 ? 1u : 0u) << (2 * j + 1);
    }
    return m;
}
__device__ __forceinline__ void unpack8(const uint4 &u, float (&v)[8]) {
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
        v[2 * j] = __uint_as_float(w[j] << 16);
        v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
    }
}

// ---- layers 1 and 2 -----------------------------------------------------------

struct Layers12 {
    FeatureTables F;
    Batch batch;
    const BfWeights *W;
    const float *b1, *b2;
    unsigned char *h1, *h2;    // tile images
    unsigned char *x;
    long long *row_of;         // data row of each batch row
    int tiles;
    int *status;
};
struct __align__(1024) Smem12 {
    unsigned char w2[kWBytes];
    unsigned char h[kActBytes];
    unsigned char w1[kW1Bytes];
    unsigned char x[kXBytes];
    float b1[kH], b2[kH], norm[2 * kF];
    unsigned long long wbar, mbar;
    unsigned tmem;
};

// Training: features, layer 1 and layer 2 of the tiles blockIdx.x, + gridDim.x, ...;
// one CTA per SM with both weight matrices resident.  The two accumulators
// take turns: a tile's layer 1 and layer 2 use one, while the other holds the
// previous tile's layer 2 until its epilogue, which runs under this tile's
// layer 2 product, has read it.
__global__ void __launch_bounds__(kThreads, 1) mlp_layers12(Layers12 g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Smem12 &S = *reinterpret_cast<Smem12 *>(smem_raw +
                                            ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x;
    pdl_launch_dependents();
    if (tid < 32) tmem_alloc(&S.tmem, 512);
    if (tid == 0) {
        mbar_init(&S.wbar, 1);
        mbar_init(&S.mbar, 1);
    }
    pdl_wait();
    if (tid < kF) {
        S.norm[tid] = g.F.mu[tid];
        S.norm[kF + tid] = g.F.isd[tid];
    }
    if (tid < kH) {
        S.b1[tid] = g.b1[tid];
        S.b2[tid] = g.b2[tid];
    }
    tc_sync();
    const unsigned tmem = S.tmem;
    if (tid == 0) {
        mbar_expect(&S.wbar, kWBytes + kW1Bytes);
        bulk_load(S.w1, g.W->w1, kW1Bytes, &S.wbar);
        bulk_load(S.w2, g.W->w2, kWBytes, &S.wbar);
    }
    const Part p = my_part<kGroups>(tmem);
    const auto features = [&](int t) {
        if (tid < kTileM) {
            const long long r = (long long)t * kTileM + tid;
            const long long q = tile_features(g.F, g.batch, S.norm, r, tid, S.x);
            g.row_of[r] = q;
        }
    };
    const auto layer1 = [&](unsigned d) {
        tc_mma(tmem + d, smem_desc(smem_u32(S.x), kActStride, 128),
               smem_desc(smem_u32(S.w1), kWStride, 128), tc_idesc(kH, false, false), false);
        tc_commit(&S.mbar);
    };
    int t = blockIdx.x, last = -1;
    unsigned phase = 0, buf = 0;
    features(t);
    bool ok = cta_wait(&S.wbar, 0, g.status);
    tc_sync();
    if (ok && tid == 0) layer1(0);
    while (ok && t < g.tiles) {
        const unsigned d = buf * kH;
        ok = cta_wait(&S.mbar, phase, g.status);  // layer 1 of t, layer 2 of the last tile
        phase ^= 1;
        if (!ok) break;
        tc_fence_after();
        // (x's image leaves before the next tile's features replace it)
        if (tid < 2 * kTileM)
            reinterpret_cast<uint4 *>(g.x + (size_t)t * kXBytes)[tid] =
                reinterpret_cast<const uint4 *>(S.x)[tid];
        hidden_epilogue<true>(p, d, S.b1, S.h, g.h1 + (size_t)t * kActBytes);
        tc_sync();
        if (tid == 0) {
            mma_layer(tmem + d, smem_u32(S.h), smem_u32(S.w2), false);
            mma_layer(tmem + d, smem_u32(S.h) + 16 * kActStride, smem_u32(S.w2) + 16 * kWStride,
                      true);
        }
        const int next = t + gridDim.x;
        if (next < g.tiles) features(next);
        if (last >= 0)
            hidden_epilogue<false>(p, (buf ^ 1) * kH, S.b2, nullptr,
                                         g.h2 + (size_t)last * kActBytes);
        if (next < g.tiles) {
            tc_sync();
            if (tid == 0) layer1((buf ^ 1) * kH);
        } else if (tid == 0) {
            tc_commit(&S.mbar);
        }
        last = t;
        t = next;
        buf ^= 1;
    }
    if (ok) ok = cta_wait(&S.mbar, phase, g.status);
    if (ok) {
        tc_fence_after();
        hidden_epilogue<false>(p, (buf ^ 1) * kH, S.b2, nullptr,
                                     g.h2 + (size_t)last * kActBytes);
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_free(tmem, 512);
}

// ---- layer 3 and the output layer --------------------------------------------

struct Layer3 {
    const BfWeights *W;
    const float *b3, *b4;
    const unsigned char *h2;
    int tiles;
    long long nrows;
    float *y;                  // [nrows][3]
    int *status;
    const float *targets;
    const long long *row_of;
    unsigned char *d3, *d2;    // gradients of the layers' sums, tile images
    float *part4;              // per CTA: W4's gradient [256][3], b4's [3], the loss
    float w_d, w_a, w_e;
};
constexpr int kPart4 = kH * kOut + kOut + 1;

// One row's outputs over a quarter of layer 3's features: every fourth vector
// of eight from vector `quarter` on (the row's other threads have the rest),
// activations from the accumulator at lane address tmem, kept as BF16 in the
// tile image at `image`.  The sum's order: along the eight features
// of a vector, then pairwise over vectors 16, 8 and 4 apart (and 2 and 1
// apart in row_outputs).
__device__ __forceinline__ void head_quarter(unsigned tmem, int quarter, const float *b3,
                                             const float4 *w4, unsigned char *image,
                                             float (&out)[kOut]) {
    constexpr int order[4] = {0, 2, 1, 3};  // vectors 4 order + quarter, and 16 more
    float pair[kOut], sum[kOut];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float v[2][8], s[2][kOut];
        const int c0 = 32 * order[i] + 8 * quarter;
        tc_ld8x2(tmem + c0, tmem + c0 + 128, v[0], v[1]);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int c = c0 + 128 * q;
            bias_relu<8>(v[q], b3, c);
            const uint4 u = pack8(v[q]);
            *reinterpret_cast<uint4 *>(image + (c >> 3) * kActStride) = u;
            float h[8];
            unpack8(u, h);
#pragma unroll
            for (int o = 0; o < kOut; o++) s[q][o] = 0.f;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float4 w = w4[c + j];
                s[q][0] = fmaf(h[j], w.x, s[q][0]);
                s[q][1] = fmaf(h[j], w.y, s[q][1]);
                s[q][2] = fmaf(h[j], w.z, s[q][2]);
            }
        }
#pragma unroll
        for (int o = 0; o < kOut; o++) {
            const float a = s[0][o] + s[1][o];
            if (i % 2 == 0)
                pair[o] = a;
            else if (i == 1)
                sum[o] = pair[o] + a;
            else
                out[o] = sum[o] + (pair[o] + a);
        }
    }
}
// A row's outputs from its four quarters' sums.
__device__ __forceinline__ void row_outputs(const float4 (&part)[kGroups][kTileM], int row,
                                            const float *b4, float (&y)[kOut]) {
    const float4 a = part[0][row], b = part[1][row], c = part[2][row], d = part[3][row];
    y[0] = (a.x + c.x) + (b.x + d.x) + b4[0];
    y[1] = (a.y + c.y) + (b.y + d.y) + b4[1];
    y[2] = (a.z + c.z) + (b.z + d.z) + b4[2];
}

// Sums over a warp's lanes of n values each; this lane is left with those from
// index lanes_first on in v[0 ..] (32 values: one, 48: three, in both lanes of
// a pair).  Lanes half a warp apart share the values between them, each adding
// its half, then lanes a quarter apart: the additions are those of a butterfly
// over every value (48 values in 48 shuffles instead of 240, which took 6,000
// clocks at the end of mlp_layer3_train).
template <int n, int d = 16, int N>
__device__ __forceinline__ void lane_sums(float (&v)[N]) {
    if constexpr (n % 2 == 0) {
        const bool up = threadIdx.x & d;
#pragma unroll
        for (int i = 0; i < n / 2; i++) {
            const float mine = up ? v[n / 2 + i] : v[i], other = up ? v[i] : v[n / 2 + i];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, other, d);
        }
        if constexpr (d > 1) lane_sums<n / 2, d / 2>(v);
    } else {
#pragma unroll
        for (int i = 0; i < n; i++) v[i] += __shfl_xor_sync(0xffffffffu, v[i], d);
        if constexpr (d > 1) lane_sums<n, d / 2>(v);
    }
}
// The index of v[0] then, and whether this lane is the first to have it.
template <int n, int d = 16>
__device__ __forceinline__ int lanes_first(bool &own) {
    if constexpr (n % 2 == 0) {
        int i = threadIdx.x & d ? n / 2 : 0;
        if constexpr (d > 1) i += lanes_first<n / 2, d / 2>(own);
        return i;
    } else {
        own = own && !(threadIdx.x & d);
        if constexpr (d > 1) return lanes_first<n, d / 2>(own);
        return 0;
    }
}

struct __align__(1024) Smem3T {
    unsigned char w3[kWBytes];
    unsigned char a[kActBytes];        // h2, then h3, then its gradient
    float4 w4[kH];
    float b3[kH];
    float4 quarter[kGroups][kTileM];  // a row's outputs by parts
    float4 dy[kTileM];
    float sum4[4][kOut + 1];
    unsigned long long wbar, abar, mbar;
    unsigned tmem;
};

// Training: outputs, loss, the gradients of the output layer (summed per
// CTA), dz3 = (dy W4^T) * relu'(h3) and dz2 = (dz3 W3^T) * relu'(h2).  loss =
// mean over rows of w_d (y0 - t0)^2 + w_a (y1 - t1)^2 + w_e rho(|y0 - t0| - y2),
// rho the pinball loss of the kQuantile quantile, so that y2 learns that
// quantile of the depth output's absolute error (taken as a constant).  The
// tile's image in shared memory is h2 (layer 3's operand; its signs are kept
// in registers), then h3 (W4's gradient), then dz3 (the next product's
// operand and what is stored).
__global__ void __launch_bounds__(kThreads, 1) mlp_layer3_train(Layer3 g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Smem3T &S = *reinterpret_cast<Smem3T *>(smem_raw +
                                            ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (tid < 32) tmem_alloc(&S.tmem, 512);
    if (tid == 0) {
        mbar_init(&S.wbar, 1);
        mbar_init(&S.abar, 1);
        mbar_init(&S.mbar, 1);
    }
    pdl_wait();
    if (tid < kH) {
        S.w4[tid] = g.W->w4[tid];
        S.b3[tid] = g.b3[tid];
    }
    const float b4[kOut] = {g.b4[0], g.b4[1], g.b4[2]};
    tc_sync();
    const unsigned tmem = S.tmem;
    const auto load = [&](int t) {
        mbar_expect(&S.abar, kActBytes);
        bulk_load(S.a, g.h2 + (size_t)t * kActBytes, kActBytes, &S.abar);
    };
    if (tid == 0) {
        load(blockIdx.x);
        mbar_expect(&S.wbar, kWBytes);
        bulk_load(S.w3, g.W->w3, kWBytes, &S.wbar);
    }
    const Part p = my_part<kGroups>(tmem);
    // this thread's vectors of eight features: 4 i + p.group, i below kMine
    constexpr int kMine = kH / 8 / kGroups;
    const float inv_b = 1.0f / (float)g.nrows;
    // W4's gradient: this thread's rows lane + 32 i of every tile, the eight
    // features of each of the warp's two vectors
    constexpr int kWarpVecs = kH / 8 / (kThreads / 32);
    float gw[kWarpVecs][8][kOut], gb[kOut] = {0.f, 0.f, 0.f}, ls = 0.f;
#pragma unroll
    for (int q = 0; q < kWarpVecs; q++)
#pragma unroll
        for (int j = 0; j < 8; j++)
#pragma unroll
            for (int o = 0; o < kOut; o++) gw[q][j][o] = 0.f;
    bool ok = cta_wait(&S.wbar, 0, g.status);
    unsigned phase = 0, mphase = 0;
    for (int t = blockIdx.x; ok && t < g.tiles; t += gridDim.x) {
        ok = cta_wait(&S.abar, phase, g.status);
        phase ^= 1;
        if (!ok) break;
        if (tid == 0) {
            tc_fence_after();
            mma_layer(tmem, smem_u32(S.a), smem_u32(S.w3), false);
            mma_layer(tmem, smem_u32(S.a) + 16 * kActStride, smem_u32(S.w3) + 16 * kWStride, true);
            tc_commit(&S.mbar);
        }
        // the targets while the product runs
        const long long r = (long long)t * kTileM + p.row;
        float t0 = 0.f, t1 = 0.f;
        if (r < g.nrows) {
            const float2 tt = *reinterpret_cast<const float2 *>(g.targets + g.row_of[r] * kTargets);
            t0 = tt.x;
            t1 = tt.y;
        }
        // signs of this thread's features of h2
        unsigned char *image = S.a + p.row * 16;
        unsigned mask[kMine / 4];
#pragma unroll
        for (int q = 0; q < kMine / 4; q++) {
            mask[q] = 0;
#pragma unroll
            for (int j = 0; j < 4; j++)
                mask[q] |= positive8(*reinterpret_cast<const uint4 *>(
                               image + (4 * (4 * q + j) + p.group) * kActStride))
                           << (8 * j);
        }
        ok = cta_wait(&S.mbar, mphase, g.status);
        mphase ^= 1;
        if (!ok) break;
        tc_fence_after();
        float acc[kOut];
        head_quarter(p.tmem, p.group, S.b3, S.w4, image, acc);
        S.quarter[p.group][p.row] = make_float4(acc[0], acc[1], acc[2], 0.f);
        __syncthreads();
        float d0 = 0.f, d1 = 0.f, d2 = 0.f;
        if (r < g.nrows) {
            float y[kOut];
            row_outputs(S.quarter, p.row, b4, y);
            const float e0 = y[0] - t0, e1 = y[1] - t1;
            const float u = fabsf(e0) - y[2];
            d0 = 2.f * g.w_d * e0 * inv_b;
            d1 = 2.f * g.w_a * e1 * inv_b;
            d2 = g.w_e * (u < 0.f ? 1.f - kQuantile : -kQuantile) * inv_b;
            if (p.group == 0) {
                const float pin = u >= 0.f ? kQuantile * u : (kQuantile - 1.f) * u;
                ls += (g.w_d * e0 * e0 + g.w_a * e1 * e1 + g.w_e * pin) * inv_b;
                gb[0] += d0;
                gb[1] += d1;
                gb[2] += d2;
                g.y[r * kOut] = y[0];
                g.y[r * kOut + 1] = y[1];
                g.y[r * kOut + 2] = y[2];
            }
        }
        if (p.group == 0) S.dy[p.row] = make_float4(d0, d1, d2, 0.f);
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < kTileM; i += 32) {
            const float4 d = S.dy[i + lane];
#pragma unroll
            for (int q = 0; q < kWarpVecs; q++) {
                float h[8];
                unpack8(*reinterpret_cast<const uint4 *>(S.a + (kWarpVecs * warp + q) * kActStride +
                                                         (i + lane) * 16),
                        h);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    gw[q][j][0] = fmaf(h[j], d.x, gw[q][j][0]);
                    gw[q][j][1] = fmaf(h[j], d.y, gw[q][j][1]);
                    gw[q][j][2] = fmaf(h[j], d.z, gw[q][j][2]);
                }
            }
        }
        __syncthreads();
        // dz3 in h3's place
#pragma unroll 1
        for (int q = 0; q < kMine; q++) {
            uint4 *at = reinterpret_cast<uint4 *>(image + (4 * q + p.group) * kActStride);
            const unsigned m = positive8(*at);
            float dz[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float4 w = S.w4[32 * q + 8 * p.group + j];
                const float v = fmaf(d0, w.x, fmaf(d1, w.y, d2 * w.z));
                dz[j] = (m >> j) & 1u ? v : 0.f;
            }
            *at = pack8(dz);
        }
        tc_sync();
        if (tid == 0) {
            mma_layer_back(tmem + kH, smem_u32(S.a), smem_u32(S.w3));
            tc_commit(&S.mbar);
            bulk_store(g.d3 + (size_t)t * kActBytes, S.a, kActBytes);
        }
        ok = cta_wait(&S.mbar, mphase, g.status);
        mphase ^= 1;
        if (!ok) break;
        tc_fence_after();
        if (tid == 0) {
            bulk_store_read();
            if (t + (int)gridDim.x < g.tiles) load(t + gridDim.x);
        }
        unsigned char *d2_out = g.d2 + (size_t)t * kActBytes + p.row * 16;
#pragma unroll
        for (int i = 0; i < kMine / 2; i++) {
            const int c0 = 64 * i + 8 * p.group;
            float v[2][8];
            tc_ld8x2(p.tmem + kH + c0, p.tmem + kH + c0 + 32, v[0], v[1]);
#pragma unroll
            for (int q = 0; q < 2; q++) {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    v[q][j] = (mask[i >> 1] >> (16 * (i & 1) + 8 * q + j)) & 1u ? v[q][j] : 0.f;
                *reinterpret_cast<uint4 *>(d2_out + (size_t)(8 * i + 4 * q + p.group) * kActStride) =
                    pack8(v[q]);
            }
        }
        tc_fence_before();
    }
    if (tid == 0) bulk_store_done();
    // this CTA's sums, each over its lanes in a fixed order
    float *out = g.part4 + (size_t)blockIdx.x * kPart4;
    {
        constexpr int n = kWarpVecs * 8 * kOut;  // 48: three are left to a pair of lanes
        float v[n];
#pragma unroll
        for (int q = 0; q < kWarpVecs; q++)
#pragma unroll
            for (int j = 0; j < 8; j++)
#pragma unroll
                for (int o = 0; o < kOut; o++) v[(q * 8 + j) * kOut + o] = gw[q][j][o];
        lane_sums<n>(v);
        bool own = true;
        const int at = lanes_first<n>(own);
        if (own)
#pragma unroll
            for (int o = 0; o < kOut; o++) out[n * warp + at + o] = v[o];
    }
    const float tail[kOut + 1] = {gb[0], gb[1], gb[2], ls};
#pragma unroll
    for (int o = 0; o <= kOut; o++) {
        float s = tail[o];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
        if (lane == 0 && warp < 4) S.sum4[warp][o] = s;  // (the first group's rows)
    }
    tc_fence_before();
    __syncthreads();
    if (tid <= kOut) {
        float s = 0.f;
        for (int w = 0; w < 4; w++) s += S.sum4[w][tid];
        out[kH * kOut + tid] = s;
    }
    if (tid < 32) tmem_free(tmem, 512);
}

// ---- the gradient through layer 2 ----------------------------------------------

struct Back2 {
    const BfWeights *W;
    const unsigned char *d2, *h1;
    unsigned char *d1;
    int tiles;
    int *status;
};
struct __align__(1024) SmemB {
    unsigned char w2[kWBytes];
    unsigned char a[kActBytes];
    unsigned long long wbar, abar, mbar;
    unsigned tmem;
};

// dz1 = (dz2 W2^T) * relu'(h1) of the tiles blockIdx.x, + gridDim.x, ...
__global__ void __launch_bounds__(kThreads, 1) mlp_back2(Back2 g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    SmemB &S = *reinterpret_cast<SmemB *>(smem_raw +
                                          ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x;
    pdl_launch_dependents();
    if (tid < 32) tmem_alloc(&S.tmem, 256);
    if (tid == 0) {
        mbar_init(&S.wbar, 1);
        mbar_init(&S.abar, 1);
        mbar_init(&S.mbar, 1);
    }
    pdl_wait();
    tc_sync();
    const unsigned tmem = S.tmem;
    const auto load = [&](int t) {
        mbar_expect(&S.abar, kActBytes);
        bulk_load(S.a, g.d2 + (size_t)t * kActBytes, kActBytes, &S.abar);
    };
    if (tid == 0) {
        load(blockIdx.x);
        mbar_expect(&S.wbar, kWBytes);
        bulk_load(S.w2, g.W->w2, kWBytes, &S.wbar);
    }
    const Part p = my_part<kGroups>(tmem);
    bool ok = cta_wait(&S.wbar, 0, g.status);
    unsigned phase = 0;
    for (int t = blockIdx.x; ok && t < g.tiles; t += gridDim.x, phase ^= 1) {
        ok = cta_wait(&S.abar, phase, g.status);
        if (!ok) break;
        if (tid == 0) {
            tc_fence_after();
            mma_layer_back(tmem, smem_u32(S.a), smem_u32(S.w2));
            tc_commit(&S.mbar);
        }
        constexpr int kParts = kH / kGroups / 32;  // of 32 columns
        unsigned mask[kParts];
        const unsigned char *h = g.h1 + (size_t)t * kActBytes + p.row * 16;
#pragma unroll
        for (int q = 0; q < kParts; q++) {
            mask[q] = 0;
#pragma unroll
            for (int j = 0; j < 4; j++)
                mask[q] |= positive8(__ldg(reinterpret_cast<const uint4 *>(
                               h + (size_t)(p.col0 / 8 + 4 * q + j) * kActStride)))
                           << (8 * j);
        }
        ok = cta_wait(&S.mbar, phase, g.status);
        if (!ok) break;
        tc_fence_after();
        if (tid == 0 && t + (int)gridDim.x < g.tiles) load(t + gridDim.x);
#pragma unroll
        for (int i = 0; i < kParts; i++) {
            const int c0 = p.col0 + 32 * i;
            float v[32];
            tc_ld32(p.tmem + c0, v);
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] = (mask[i] >> j) & 1u ? v[j] : 0.f;
#pragma unroll
            for (int q = 0; q < 4; q++)
                *reinterpret_cast<uint4 *>(g.d1 + (size_t)t * kActBytes +
                                           (size_t)(c0 / 8 + q) * kActStride + p.row * 16) =
                    pack8(v + 8 * q);
        }
        tc_fence_before();
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_free(tmem, 256);
}

// ---- weight gradients --------------------------------------------------------

// gW3 = H2^T dZ3, gW2 = H1^T dZ2 (256 x 256: the whole of tensor memory) and
// gW1^T = dZ1^T X, every one over the rows, in splits of four tiles (512
// rows): an item is one split of one product, a CTA takes items in turn and
// leaves a partial sum of each.  With a product goes the sum over the rows of
// the layer's gradient (its bias).  The first `big` CTAs share the items of
// W3 and W2, the others those of W1 (a ninth of the products but half of the
// bytes).
constexpr int kSplitTiles = 4;
constexpr int kThreadsW = 256;  // eight warps sum and store; one more feeds the tensor core
struct Wgrad {
    const unsigned char *h1, *h2, *x, *d1, *d2, *d3;
    int tiles, splits, big;
    float *part;           // [2][splits][2][64][128][4] (W3, W2)
    float *part1;          // [splits][2][4][128][4] (W1)
    float *part_b;         // [3][splits][256] (b3, b2, b1)
    int *status;
};
struct __align__(1024) SmemW {
    unsigned char buf[3][kActBytes];
    unsigned char x[3][kXBytes];  // layer 1's features, with its gradient's buffer
    unsigned long long full[3], free_[3], done, drained;
    unsigned tmem;
};

__global__ void __launch_bounds__(kThreadsW + 32, 1) mlp_wgrad(Wgrad g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    SmemW &S = *reinterpret_cast<SmemW *>(smem_raw +
                                          ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_launch_dependents();
    if (tid < 32) tmem_alloc(&S.tmem, 512);
    if (tid == 0) {
        for (int i = 0; i < 3; i++) {
            mbar_init(&S.full[i], 1);
            mbar_init(&S.free_[i], 1 + 8);  // the products, and the eight summing warps
        }
        mbar_init(&S.done, 1);
        mbar_init(&S.drained, 8);
    }
    pdl_wait();
    tc_sync();
    const unsigned tmem = S.tmem;
    const bool first = (int)blockIdx.x >= g.big;  // layer 1
    const int item0 = first ? blockIdx.x - g.big : blockIdx.x;
    const int step = first ? gridDim.x - g.big : g.big;
    const int items = first ? g.splits : 2 * g.splits;
    const int per_tile = first ? 1 : 2;  // buffers
    bool ok = true;
    if (tid >= kThreadsW) {
        if (tid == kThreadsW) {
            // loads, into the three buffers in turn: of each tile the
            // activations, then the layer's gradient, a tile and a half ahead
            // of the products; of layer 1 its gradient with the tile's
            // features, three tiles ahead (with the features in a buffer of
            // their own, and so a tile and a half, an item of layer 1 took
            // 22,000 clocks and the launch 38 us; so 30)
            int load_item = item0, load_tile = 0, loads = 0;
            const auto load_next = [&] {
                const int prod = first ? 2 : load_item / g.splits;
                const int split = first ? load_item : load_item % g.splits;
                const int t = split * kSplitTiles + load_tile;
                const int i = loads % 3;
                const bool second = first || (loads & 1);
                if (loads >= 3) ok = mbar_wait(&S.free_[i], (loads / 3 - 1) & 1, g.status);
                if (!ok) return;
                mbar_expect(&S.full[i], first ? kXBytes + kActBytes : kActBytes);
                if (first) bulk_load(S.x[i], g.x + (size_t)t * kXBytes, kXBytes, &S.full[i]);
                const unsigned char *src = second ? (prod == 0 ? g.d3 : (prod == 1 ? g.d2 : g.d1))
                                                  : (prod == 0 ? g.h2 : g.h1);
                bulk_load(S.buf[i], src + (size_t)t * kActBytes, kActBytes, &S.full[i]);
                loads++;
                if (second) {
                    load_tile++;
                    if (load_tile == kSplitTiles || t + 1 == g.tiles) {
                        load_tile = 0;
                        load_item += step;
                    }
                }
            };
            const auto ahead = [&](int upto) {
                while (ok && load_item < items && loads < upto) load_next();
            };
            int used = 0, n = 0;
            ahead(3);
            for (int item = item0; ok && item < items; item += step, n++) {
                const int split = first ? item : item % g.splits;
                const int t1 = min(g.tiles, (split + 1) * kSplitTiles);
                // the accumulators' last reader
                if (n > 0) ok = mbar_wait(&S.drained, (n - 1) & 1, g.status);
                tc_fence_after();
                bool more = false;
                for (int t = split * kSplitTiles; ok && t < t1; t++) {
                    const int ia = used % 3, ib = (used + per_tile - 1) % 3;
                    ok = mbar_wait(&S.full[ia], (used / 3) & 1, g.status);
                    if (ok && !first)
                        ok = mbar_wait(&S.full[ib], ((used + 1) / 3) & 1, g.status);
                    if (!ok) break;
                    const unsigned a = smem_u32(first ? S.x[ia] : S.buf[ia]),
                                   b = smem_u32(S.buf[ib]);
                    for (int m = 0; m < 2; m++)
                        for (int kk = 0; kk < 8; kk++) {
                            if (!first)  // 128 inputs x 256 outputs
                                tc_mma(tmem + kH * m,
                                       smem_desc(a + 16 * m * kActStride + 256 * kk, 128,
                                                 kActStride),
                                       smem_desc(b + 256 * kk, 128, kActStride),
                                       tc_idesc(kH, true, true), more || kk > 0);
                            else  // 128 outputs x 16 inputs
                                tc_mma(tmem + kH * m,
                                       smem_desc(b + 16 * m * kActStride + 256 * kk, 128,
                                                 kActStride),
                                       smem_desc(a + 256 * kk, 128, kActStride),
                                       tc_idesc(kF, true, true), more || kk > 0);
                        }
                    more = true;
                    if (!first) tc_commit(&S.free_[ia]);
                    tc_commit(&S.free_[ib]);
                    if (t + 1 == t1) tc_commit(&S.done);
                    used += per_tile;
                    ahead(used + 3);
                }
            }
        }
    } else {
        const Part p = my_part<2>(tmem);
        int used = 0, n = 0;
        for (int item = item0; item < items; item += step, n++) {
            const int prod = first ? 2 : item / g.splits;
            const int split = first ? item : item % g.splits;
            const int t1 = min(g.tiles, (split + 1) * kSplitTiles);
            // the bias: rows lane + 32 i, the eight features of the warp's four vectors
            float gb[4][8];
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int j = 0; j < 8; j++) gb[q][j] = 0.f;
            for (int t = split * kSplitTiles; t < t1; t++, used += per_tile) {
                const int ia = used % 3, ib = (used + per_tile - 1) % 3;
                if (ok) ok = mbar_wait(&S.full[ia], (used / 3) & 1, g.status);
                if (!first) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&S.free_[ia]);
                    if (ok) ok = mbar_wait(&S.full[ib], ((used + 1) / 3) & 1, g.status);
                }
#pragma unroll 1
                for (int r = lane; ok && r < kTileM; r += 32)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        float v[8];
                        unpack8(*reinterpret_cast<const uint4 *>(
                                    S.buf[ib] + (4 * warp + q) * kActStride + r * 16),
                                v);
#pragma unroll
                        for (int j = 0; j < 8; j++) gb[q][j] += v[j];
                    }
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.free_[ib]);
            }
            float *out_b = g.part_b + (size_t)(prod * g.splits + split) * kH;
            float v[32];
#pragma unroll
            for (int q = 0; q < 4; q++)
#pragma unroll
                for (int j = 0; j < 8; j++) v[8 * q + j] = gb[q][j];
            lane_sums<32>(v);
            bool own = true;
            const int at = lanes_first<32>(own);
            out_b[32 * warp + at] = v[0];
            if (ok) ok = mbar_wait(&S.done, n & 1, g.status);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                tc_fence_after();
                const int half = p.col0 >> 7;
                if (!first) {
#pragma unroll 1
                    for (int m = 0; m < 2; m++) {
                        float4 *out = reinterpret_cast<float4 *>(g.part) +
                                      (size_t)((prod * g.splits + split) * 2 + m) * 64 * kTileM;
#pragma unroll 1
                        for (int c0 = p.col0; c0 < p.col0 + 128; c0 += 32) {
                            float v[32];
                            tc_ld32(p.tmem + kH * m + c0, v);
#pragma unroll
                            for (int q = 0; q < 8; q++)
                                out[(size_t)(c0 / 4 + q) * kTileM + p.row] = make_float4(
                                    v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                        }
                    }
                } else {
                    float4 *out = reinterpret_cast<float4 *>(g.part1) +
                                  (size_t)(split * 2 + half) * 4 * kTileM;
                    float v[16];
                    tc_ld16(p.tmem + kH * half, v);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        out[(size_t)q * kTileM + p.row] =
                            make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                tc_fence_before();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.drained);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (tid < 32) tmem_free(tmem, 512);
}

// ---- sums of the partials, Adam -------------------------------------------------

struct Adam {
    float *p, *m, *v;  // null p: gradients only
    float lr, b1, b2, eps, c1, c2;
};
struct Finish {
    const float *part, *part1, *part_b, *part4;
    int splits, ctas4;
    float *grad;       // null: not asked for
    float *loss;
    Adam adam;
    BfWeights *W;
};

// A gradient becomes a parameter's step; returns the new parameter.
__device__ __forceinline__ float adam_step(const Adam &a, long i, float gi) {
    const float mi = a.b1 * a.m[i] + (1.f - a.b1) * gi;
    const float vi = a.b2 * a.v[i] + (1.f - a.b2) * gi * gi;
    a.m[i] = mi;
    a.v[i] = vi;
    const float p = a.p[i] - a.lr * (mi * a.c1) / (sqrtf(vi * a.c2) + a.eps);
    a.p[i] = p;
    return p;
}

constexpr int kItemsW = 4 * 2 * 2 * 64 * kTileM;       // W3 and W2, one output each
constexpr int kItems1 = 4 * 2 * 4 * kTileM;            // W1, one input each
constexpr int kItemsB = 3 * kH;                        // b3, b2, b1
constexpr int kItems4 = kPart4;                        // W4, b4, the loss
constexpr int kItems = kItemsW + kItems1 + kItemsB + kItems4;

__device__ __forceinline__ float4 add4(const float4 &a, const float4 &b) {
    return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
// The sum over n splits of the float4 at p, step apart: four running sums over
// the splits k, k + 4, ... (what is left over four goes to the first), each by
// one lane of four, all its loads in flight together; every lane returns
// (s0 + s1) + (s2 + s3).
__device__ __forceinline__ float4 split_sum4(const float4 *p, size_t step, int n, int lane4) {
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    const int n4 = n & ~3;
#pragma unroll 16
    for (int k = lane4; k < n4; k += 4) s = add4(s, __ldcs(p + (size_t)k * step));
    if (lane4 == 0)
        for (int k = n4; k < n; k++) s = add4(s, p[(size_t)k * step]);
#pragma unroll
    for (int d = 1; d <= 2; d <<= 1)
        s = add4(s, make_float4(__shfl_xor_sync(0xffffffffu, s.x, d),
                                __shfl_xor_sync(0xffffffffu, s.y, d),
                                __shfl_xor_sync(0xffffffffu, s.z, d),
                                __shfl_xor_sync(0xffffffffu, s.w, d)));
    return s;
}
__device__ __forceinline__ float split_sum(const float *p, size_t step, int n) {
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
    int k = 0;
#pragma unroll 4
    for (; k + 4 <= n; k += 4) {
        s0 += p[(size_t)k * step];
        s1 += p[(size_t)(k + 1) * step];
        s2 += p[(size_t)(k + 2) * step];
        s3 += p[(size_t)(k + 3) * step];
    }
    for (; k < n; k++) s0 += p[(size_t)k * step];
    return (s0 + s1) + (s2 + s3);
}

// One thread per parameter: the partials of every split summed in a fixed
// order, then Adam and the BF16 image, or the gradient.  Reads 128 kB per
// split and product half: bound by the latency of those reads, which is why
// four lanes share the splits of four weights.
__global__ void __launch_bounds__(256) mlp_finish(Finish g) {
    pdl_launch_dependents();
    pdl_wait();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = i & 3;
    const auto put = [&](long at, float gi, __nv_bfloat16 *image) {
        if (g.grad) g.grad[at] = gi;
        if (g.adam.p) {
            const float p = adam_step(g.adam, at, gi);
            if (image) *image = __float2bfloat16(p);
        }
    };
    const auto pick = [&](const float4 &s) {
        return j == 0 ? s.x : (j == 1 ? s.y : (j == 2 ? s.z : s.w));
    };
    if (i < kItemsW) {
        i >>= 2;
        const int row = i & 127, c4 = (i >> 7) & 63, m = (i >> 13) & 1, layer2 = i >> 14;
        const float4 s = split_sum4(reinterpret_cast<const float4 *>(g.part) +
                                        (size_t)(layer2 * g.splits * 2 + m) * 64 * kTileM +
                                        (size_t)c4 * kTileM + row,
                                    (size_t)2 * 64 * kTileM, g.splits, j);
        const int in = m * kTileM + row, out = 4 * c4 + j;
        put((layer2 ? kOffW2 : kOffW3) + (long)in * kH + out, pick(s),
            (layer2 ? g.W->w2 : g.W->w3) + w_at(in, out));
        return;
    }
    i -= kItemsW;
    if (i < kItems1) {
        i >>= 2;
        const int row = i & 127, c4 = (i >> 7) & 3, m = i >> 9;
        const float4 s = split_sum4(reinterpret_cast<const float4 *>(g.part1) +
                                        (size_t)(m * 4 + c4) * kTileM + row,
                                    (size_t)8 * kTileM, g.splits, j);
        const int in = 4 * c4 + j, out = m * kTileM + row;
        put(kOffW1 + (long)in * kH + out, pick(s), g.W->w1 + w_at(in, out));
        return;
    }
    i -= kItems1;
    if (i < kItemsB) {
        const int layer = i >> 8, f = i & 255;  // 0: b3, 1: b2, 2: b1
        put((layer == 0 ? kOffB3 : (layer == 1 ? kOffB2 : kOffB1)) + f,
            split_sum(g.part_b + (size_t)layer * g.splits * kH + f, (size_t)kH, g.splits),
            nullptr);
        return;
    }
    i -= kItemsB;
    if (i < kItems4) {
        const float s = split_sum(g.part4 + i, (size_t)kPart4, g.ctas4);
        if (i == kPart4 - 1) {
            *g.loss = s;
        } else {
            const long at = kOffW4 + i;  // W4 [256][3], then b4
            put(at, s, nullptr);
            if (g.adam.p && i < kH * kOut)
                reinterpret_cast<float *>(g.W->w4 + i / kOut)[i % kOut] =
                    __bfloat162float(__float2bfloat16(g.adam.p[at]));
        }
    }
}

// ---- inference ---------------------------------------------------------------

// The whole network in one launch, activations never leaving the SM: no SM's
// shared memory holds W1, W2 and W3 (264 kB), so the two CTAs of a cluster
// hold half of the outputs' columns of each, and their products are of 256
// rows (cta_group::2): 128 rows of each CTA's own against both halves.
//
// X and Y are the two accumulators (256 columns each, all of tensor memory)
// and h the tile's activations in shared memory, whose halves (128 features)
// are written and multiplied one after the other.  Tile n has P = X and Q = Y
// for even n, the other way round for odd:
//   product warp (of the first CTA)      sixteen epilogue warps (of both)
//                                          P -> h half 0 (layer 1)
//     layer 2, half 0: h -> Q              Q -> registers (n - 1's layer 3)
//     layer 2, half 1                      P -> h half 1
//                                          outputs of n - 1, two of their
//                                            four parts
//     layer 1 of n + 1 -> Q, half 0        Q -> h half 0 (layer 2)
//     layer 3, half 0: h -> P              Q -> h half 1
//     layer 1 of n + 1 -> Q, half 1        outputs of n - 1, the other two
//     layer 3, half 1: h -> P
// The products hide the outputs of the tile before.  Two warps compute
// features a tile ahead.
//
// Clocks per tile and SM, of which the products are 4,200 (3.2 million rows):
//   12,800  layers 1 and 2, then layer 3 and the outputs, as launches of five
//           tiles an SM with layer 2's activations through L2: every launch
//           reloads the weights, and of a tile's 6,100 + 4,400 clocks its
//           features, the products' issue and layer 1's epilogue come one
//           after the other
//   15,000  one CTA of a pair layers 1 and 2, the other layer 3, through a
//           ring in L2: an SM stores 32 bytes a clock, 2,000 clocks a tile
//    8,700  this: 1,130 -> 740 us
// What is left is the chain of a tile's three products and the halves of
// epilogues between them (about 600 clocks each, and 300 for every hand-over
// between the CTAs); shared memory has no room for a second tile of h.
constexpr int kFeatureWarps = 2;
constexpr int kThreadsP = kThreads + 32 + 32 * kFeatureWarps;
constexpr int kPairRows = 2 * kTileM;

struct Predict {
    FeatureTables F;
    Batch batch;
    const BfWeights *W;
    const float *b1, *b2, *b3, *b4;
    float *y;   // [nrows][3]
    int pairs;  // of tiles
    int *status;
};
struct __align__(1024) SmemP {
    unsigned char w2[kWBytes / 2], w3[kWBytes / 2];  // [in / 8][this CTA's 128 outputs][8 in]
    unsigned char h[kActBytes];
    unsigned char w1[2][kW1Bytes / 4];  // the same of each half of layer 1's outputs
    unsigned char x[2][kXBytes];
    float4 w4xy[kH / 2];  // features c and c + 128: the weights of output 0, of output 1
    float2 w4z[kH / 2];   // and of output 2
    float b1[kH], b2[kH], b3[kH], norm[2 * kF];
    float4 quarter[kGroups][kTileM];  // a row's outputs by parts
    // the first CTA's: what the warps of both have done
    unsigned long long hfull[2], qfree, xfull[2], other_w;
    // products done (both CTAs'); this CTA's own
    unsigned long long l1done, l2done, h0free, l3done, xfree[2], wbar, parts;
    unsigned tmem;
};

template <int n>
__device__ __forceinline__ void tc_mma_pair(unsigned d_tmem, unsigned long long a,
                                            unsigned long long b, bool accumulate) {
    // as tc_idesc, M = 256
    constexpr unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) |
                               ((unsigned)(kPairRows >> 4) << 24);
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"((unsigned)accumulate)
        : "memory");
}
// Arrives at the barrier of both CTAs when the products so far are done.
__device__ __forceinline__ void tc_commit_pair(unsigned long long *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64"
        " [%0], %1;" ::"r"(smem_u32(bar)),
        "h"((unsigned short)3)
        : "memory");
}
// 128 of the 256 features of a layer; a, w: the first of each CTA's own
__device__ __forceinline__ void mma_half_pair(unsigned d, unsigned a, unsigned w,
                                              bool accumulate) {
#pragma unroll
    for (int kk = 0; kk < 8; kk++)
        tc_mma_pair<kH>(d, smem_desc(a + 2 * kActStride * kk, kActStride, 128),
                        smem_desc(w + kWStride * kk, kWStride / 2, 128), accumulate || kk > 0);
}
__device__ __forceinline__ void tmem_alloc_pair(unsigned *base) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
                     smem_u32(base))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free_pair(unsigned base) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(base) : "memory");
}

// relu(v + bias) of two features as BF16
__device__ __forceinline__ unsigned relu_pair(float2 v, float2 bias) {
    const float2 h = add2(v, bias);
    const __nv_bfloat162 o = __floats2bfloat162_rn(fmaxf(h.x, 0.0f), fmaxf(h.y, 0.0f));
    return *reinterpret_cast<const unsigned *>(&o);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreadsP, 1) mlp_predict(Predict g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    SmemP &S = *reinterpret_cast<SmemP *>(smem_raw +
                                          ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned rank = cluster_rank();
    const int first = blockIdx.x >> 1, stride = gridDim.x >> 1;
    constexpr int kWarps = kThreads / 32;  // of the epilogue
    pdl_launch_dependents();
    if (tid < 32) tmem_alloc_pair(&S.tmem);
    if (tid == 0) {
        mbar_init(&S.wbar, 1);
        mbar_init(&S.other_w, 1);
        mbar_init(&S.parts, kWarps);
        mbar_init(&S.qfree, 2 * kWarps);
        mbar_init(&S.l1done, 1);
        mbar_init(&S.l2done, 1);
        mbar_init(&S.l3done, 1);
        mbar_init(&S.h0free, 1);
        for (int i = 0; i < 2; i++) {
            mbar_init(&S.hfull[i], 2 * kWarps);
            mbar_init(&S.xfull[i], 2 * kFeatureWarps);
            mbar_init(&S.xfree[i], 1);
        }
    }
    pdl_wait();
    if (tid < kF) {
        S.norm[tid] = g.F.mu[tid];
        S.norm[kF + tid] = g.F.isd[tid];
    }
    if (tid < kH) {
        S.b1[tid] = g.b1[tid];
        S.b2[tid] = g.b2[tid];
        S.b3[tid] = g.b3[tid];
    }
    if (tid < kH / 2) {
        const float4 a = g.W->w4[tid], b = g.W->w4[tid + kH / 2];
        S.w4xy[tid] = make_float4(a.x, b.x, a.y, b.y);
        S.w4z[tid] = make_float2(a.z, b.z);
    }
    tc_sync();
    cluster_sync();
    const unsigned tmem = S.tmem;
    bool ok = true;
    if (warp == kWarps) {
        if (lane == 0) {
            // this CTA's columns of the weights
            mbar_expect(&S.wbar, kWBytes + kW1Bytes / 2);
            constexpr unsigned kCols = kWStride / 2;  // bytes of 128 outputs, 8 inputs
            const auto load = [&](unsigned char *dst, const void *src, int vecs, unsigned from,
                                  unsigned bytes) {
                for (int i = 0; i < vecs; i++)
                    bulk_load(dst + i * bytes,
                              static_cast<const unsigned char *>(src) + i * kWStride + from, bytes,
                              &S.wbar);
            };
            for (int half = 0; half < 2; half++)
                load(S.w1[half], g.W->w1, kF / 8, half * kCols + rank * (kCols / 2), kCols / 2);
            load(S.w2, g.W->w2, kH / 8, rank * kCols, kCols);
            load(S.w3, g.W->w3, kH / 8, rank * kCols, kCols);
            ok = mbar_wait(&S.wbar, 0, g.status);
            if (ok && rank != 0) mbar_arrive_at(&S.other_w, 0);
            const unsigned h = smem_u32(S.h), w2 = smem_u32(S.w2), w3 = smem_u32(S.w3);
            const auto wait = [&](unsigned long long *bar, unsigned parity) {
                ok = ok && mbar_wait(bar, parity, g.status);
                tc_fence_after();
            };
            const auto layer1 = [&](int n, int half) {
                wait(&S.xfull[n & 1], (n >> 1) & 1);
                if (!ok) return;
                tc_mma_pair<kH / 2>(tmem + (n & 1) * kH + half * (kH / 2),
                                    smem_desc(smem_u32(S.x[n & 1]), kActStride, 128),
                                    smem_desc(smem_u32(S.w1[half]), kCols / 2, 128), false);
                if (half) tc_commit_pair(&S.xfree[n & 1]);
            };
            int n = 0, t = first;
            if (rank != 0) t = g.pairs;
            if (ok && t < g.pairs) {
                wait(&S.other_w, 0);
                layer1(0, 0);
                layer1(0, 1);
                if (ok) tc_commit_pair(&S.l1done);
            }
            for (; ok && t < g.pairs; t += stride, n++) {
                const unsigned p = tmem + (n & 1) * kH, q = tmem + (~n & 1) * kH;
                const bool more = t + stride < g.pairs;
                wait(&S.hfull[0], 0);
                if (n) wait(&S.qfree, (n - 1) & 1);
                if (!ok) break;
                mma_half_pair(q, h, w2, false);
                wait(&S.hfull[1], 0);
                if (!ok) break;
                mma_half_pair(q, h + 16 * kActStride, w2 + 16 * kCols, true);
                tc_commit_pair(&S.l2done);
                wait(&S.hfull[0], 1);  // (Q's first half has been read)
                if (more) layer1(n + 1, 0);
                if (!ok) break;
                mma_half_pair(p, h, w3, false);
                tc_commit_pair(&S.h0free);
                wait(&S.hfull[1], 1);  // (and its second)
                if (more) layer1(n + 1, 1);
                if (!ok) break;
                mma_half_pair(p, h + 16 * kActStride, w3 + 16 * kCols, true);
                tc_commit_pair(&S.l3done);
            }
        }
    } else if (warp > kWarps) {
        const int row = tid - kThreads - 32;
        int n = 0;
        for (int t = first; ok && t < g.pairs; t += stride, n++) {
            const int b = n & 1;
            if (n >= 2) ok = __all_sync(~0u, mbar_wait(&S.xfree[b], ((n >> 1) - 1) & 1, g.status));
            if (!ok) break;
#pragma unroll
            for (int i = row; i < kTileM; i += 32 * kFeatureWarps)
                tile_features(g.F, g.batch, S.norm,
                              (long long)t * kPairRows + (int)rank * kTileM + i, i, S.x[b]);
            proxy_fence();
            __syncwarp();
            if (lane == 0) mbar_arrive_at(&S.xfull[b], 0);
        }
    } else {
        const Part p = my_part<kGroups>(tmem);
        const int c0 = 32 * p.group;  // this warp's columns of each half of a layer
        const int row0 = 32 * (warp & 3) + lane / 4;  // the first of this thread's four rows
        const float b4[kOut] = {g.b4[0], g.b4[1], g.b4[2]};
        const auto wait = [&](unsigned long long *bar, unsigned parity) {
            if (ok) ok = __all_sync(~0u, mbar_wait(bar, parity, g.status));
            tc_fence_after();
        };
        const int quad = lane & 3;
        const auto hidden_half = [&](unsigned acc, int half, const float *bias) {
            const int c = 128 * half + c0;
            float2 v[4][4];
            tc_ld_quads(p.tmem + acc + c, v);
            unsigned char *out = S.h + (c / 8) * kActStride + row0 * 16 + quad * 4;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const float2 bb = *reinterpret_cast<const float2 *>(bias + c + 8 * b + 2 * quad);
#pragma unroll
                for (int i = 0; i < 4; i++)
                    *reinterpret_cast<unsigned *>(out + b * kActStride + i * 128) =
                        relu_pair(v[b][i], bb);
            }
            proxy_fence();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_at(&S.hfull[half], 0);
        };
        // Layer 3 of tile n as BF16, which frees its accumulator: of the row of
        // this thread's lane, h3[m] is vector 4 m + group of eight features.
        uint4 h3[8];
        const auto read_layer3 = [&](int n) {
            wait(&S.l3done, n & 1);
            if (!ok) return;
            float v[8][8];
            tc_ld8x8(p.tmem + (n & 1) * kH + 8 * p.group, v);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_at(&S.qfree, 0);
#pragma unroll
            for (int m = 0; m < 8; m++) {
                bias_relu<8>(v[m], S.b3, 32 * m + 8 * p.group);
                h3[m] = pack8(v[m]);
            }
        };
        // Outputs of tile n: head_quarter's sums, those of two vectors 16 apart
        // side by side in the two halves of an instruction.
        const auto outputs = [&](int n) {
            constexpr int order[4] = {0, 2, 1, 3};
            float pair[kOut], sum[kOut], y[kOut];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int m = order[i], c = 32 * m + 8 * p.group;
                const unsigned lo[4] = {h3[m].x, h3[m].y, h3[m].z, h3[m].w};
                const unsigned hi[4] = {h3[m + 4].x, h3[m + 4].y, h3[m + 4].z, h3[m + 4].w};
                float2 s[kOut];
#pragma unroll
                for (int o = 0; o < kOut; o++) s[o] = make_float2(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const unsigned a = j & 1 ? lo[j / 2] & 0xffff0000u : lo[j / 2] << 16;
                    const unsigned b = j & 1 ? hi[j / 2] & 0xffff0000u : hi[j / 2] << 16;
                    const float2 h = make_float2(__uint_as_float(a), __uint_as_float(b));
                    const float4 w = S.w4xy[c + j];
                    s[0] = fma2(h, make_float2(w.x, w.y), s[0]);
                    s[1] = fma2(h, make_float2(w.z, w.w), s[1]);
                    s[2] = fma2(h, S.w4z[c + j], s[2]);
                }
#pragma unroll
                for (int o = 0; o < kOut; o++) {
                    const float a = s[o].x + s[o].y;
                    if (i % 2 == 0)
                        pair[o] = a;
                    else if (i == 1)
                        sum[o] = pair[o] + a;
                    else
                        y[o] = sum[o] + (pair[o] + a);
                }
            }
            S.quarter[p.group][p.row] = make_float4(y[0], y[1], y[2], 0.f);
            // (a part is written again after layer 3 of the next tile, for which
            // all of the warps have gone on)
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.parts);
            if (p.group != (n & (kGroups - 1))) return;
            wait(&S.parts, n & 1);
            const long long r = (long long)(first + n * stride) * kPairRows + (int)rank * kTileM +
                                p.row;
            if (ok && r < g.batch.nrows) {
                row_outputs(S.quarter, p.row, b4, y);
                g.y[r * kOut] = y[0];
                g.y[r * kOut + 1] = y[1];
                g.y[r * kOut + 2] = y[2];
            }
        };
        int n = 0;
        for (int t = first; ok && t < g.pairs; t += stride, n++) {
            const unsigned P = (n & 1) * kH, Q = (~n & 1) * kH;
            if (n)
                wait(&S.h0free, (n - 1) & 1);  // (and layer 1's first half)
            else
                wait(&S.l1done, 0);
            if (!ok) break;
            hidden_half(P, 0, S.b1);
            if (n) read_layer3(n - 1);  // (and so layer 1's second half)
            if (!ok) break;
            hidden_half(P, 1, S.b1);
            if (n) outputs(n - 1);
            wait(&S.l2done, n & 1);
            if (!ok) break;
            hidden_half(Q, 0, S.b2);
            hidden_half(Q, 1, S.b2);
        }
        if (ok && n) read_layer3(n - 1);
        if (ok && n) outputs(n - 1);
    }
    tc_fence_before();
    cluster_sync();  // both are done with tensor memory and with each other's barriers
    if (tid < 32) tmem_free_pair(tmem);
}

// ---- weights ----------------------------------------------------------------

__global__ void mlp_pack_weights(const float *__restrict__ p, BfWeights *W) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kH * kH) {
        const int in = i / kH, out = i % kH;
        W->w2[w_at(in, out)] = __float2bfloat16(p[kOffW2 + i]);
        W->w3[w_at(in, out)] = __float2bfloat16(p[kOffW3 + i]);
    }
    if (i < kF * kH) {
        const int in = i / kH, out = i % kH;
        W->w1[w_at(in, out)] = __float2bfloat16(p[kOffW1 + i]);
    }
    if (i < kH) {
        const float *w = p + kOffW4 + i * kOut;
        W->w4[i] = make_float4(__bfloat162float(__float2bfloat16(w[0])),
                               __bfloat162float(__float2bfloat16(w[1])),
                               __bfloat162float(__float2bfloat16(w[2])), 0.f);
    }
}

// ---- host side ----------------------------------------------------------------

struct Buffers {  // one batch of rows (training)
    int tiles = 0;
    unsigned char *h2 = nullptr;                    // tile images
    unsigned char *x = nullptr, *h1 = nullptr, *d3 = nullptr, *d2 = nullptr, *d1 = nullptr;
    long long *row_of = nullptr;
    float *y = nullptr;
    float *part = nullptr, *part1 = nullptr, *part_b = nullptr, *part4 = nullptr;  // partials
};

struct Mlp {
    int device = 0;
    int sms = 1;
    cudaStream_t stream = nullptr;
    float *params = nullptr, *grad = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    BfWeights *w = nullptr;
    float *mu = nullptr, *isd = nullptr;
    float *scen = nullptr, *tri = nullptr, *targets = nullptr;
    long long S = 0, N = 0;
    Buffers buf;
    long long *rows = nullptr;
    long long rows_cap = 0;
    float *loss = nullptr;
    int *status = nullptr;   // device-side failure of a tensor-core kernel
    bool unusable = false;   // a kernel reported SWGPU_ETIMEOUT
    long long adam_t = 0;
    std::vector<void *> allocs, data_allocs, buf_allocs;
    std::string err;
};

thread_local std::string g_mlp_error;

int mfail(Mlp *m, int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (m) m->err = buf;
    g_mlp_error = buf;
    return code;
}

#define MCK(x)                                                                         \
    do {                                                                               \
        cudaError_t e_ = (x);                                                          \
        if (e_ != cudaSuccess)                                                         \
            return mfail(m, SWGPU_ECUDA, "%s: %s", #x, cudaGetErrorString(e_));       \
    } while (0)

template <typename T>
int malloc_dev(Mlp *m, T **p, size_t count, std::vector<void *> *owner = nullptr) {
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, count * sizeof(T) + 16);
    if (e != cudaSuccess)
        return mfail(m, SWGPU_ENOMEM, "cudaMalloc %zu bytes: %s", count * sizeof(T),
                     cudaGetErrorString(e));
    (owner ? *owner : m->allocs).push_back(q);
    *p = static_cast<T *>(q);
    return SWGPU_OK;
}

void free_list(std::vector<void *> &v) {
    for (void *p : v) cudaFree(p);
    v.clear();
}

int wgrad_splits(int tiles) { return (tiles + kSplitTiles - 1) / kSplitTiles; }

// Buffers for `tiles` tiles of 128 rows, reallocated only when they grow or
// when training needs the gradients' images.
int ensure_buffers(Mlp *m, int tiles, std::vector<void *> &owned) {
    Buffers &B = m->buf;
    if (tiles <= B.tiles) return SWGPU_OK;
    MCK(cudaStreamSynchronize(m->stream));
    free_list(owned);
    B = Buffers{};
    int rc;
    const size_t act = (size_t)tiles * kActBytes, rows = (size_t)tiles * kTileM;
    const size_t s = wgrad_splits(tiles);
    if ((rc = malloc_dev(m, &B.h2, act, &owned)) ||
        (rc = malloc_dev(m, &B.x, (size_t)tiles * kXBytes, &owned)) ||
        (rc = malloc_dev(m, &B.h1, act, &owned)) || (rc = malloc_dev(m, &B.d3, act, &owned)) ||
        (rc = malloc_dev(m, &B.d2, act, &owned)) || (rc = malloc_dev(m, &B.d1, act, &owned)) ||
        (rc = malloc_dev(m, &B.row_of, rows, &owned)) ||
        (rc = malloc_dev(m, &B.y, rows * kOut, &owned)) ||
        (rc = malloc_dev(m, &B.part, s * 2 * kH * kH, &owned)) ||
        (rc = malloc_dev(m, &B.part1, s * kF * kH, &owned)) ||
        (rc = malloc_dev(m, &B.part_b, s * 3 * kH, &owned)) ||
        (rc = malloc_dev(m, &B.part4, (size_t)std::min(tiles, m->sms) * kPart4, &owned)))
        return rc;
    B.tiles = tiles;
    return SWGPU_OK;
}

template <typename Smem>
constexpr size_t smem_of() {
    return sizeof(Smem) + 1024;  // aligned up to 1024 in the kernel
}

// A launch as a programmatic dependent of the stream's previous kernel.
template <typename Args>
int launch(Mlp *m, void (*kernel)(Args), dim3 grid, int threads, size_t smem, const Args &args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = m->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    MCK(cudaLaunchKernelEx(&cfg, kernel, args));
    return SWGPU_OK;
}

template <typename F>
cudaError_t smem_attr(F *kernel, size_t bytes) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

FeatureTables tables(const Mlp *m) {
    return FeatureTables{m->scen, m->tri, m->mu, m->isd, m->N};
}

// Layers 1 and 2 of a batch into the buffers.
int layers12(Mlp *m, const Batch &batch, int tiles) {
    Buffers &B = m->buf;
    Layers12 g{};
    g.F = tables(m);
    g.batch = batch;
    g.W = m->w;
    g.b1 = m->params + kOffB1;
    g.b2 = m->params + kOffB2;
    g.h1 = B.h1;
    g.h2 = B.h2;
    g.x = B.x;
    g.row_of = B.row_of;
    g.tiles = tiles;
    g.status = m->status;
    return launch(m, mlp_layers12, dim3((unsigned)std::min(tiles, m->sms)), kThreads,
                  smem_of<Smem12>(), g);
}

Layer3 layer3(Mlp *m, int tiles, long long nrows, float *y) {
    Layer3 g{};
    g.W = m->w;
    g.b3 = m->params + kOffB3;
    g.b4 = m->params + kOffB4;
    g.h2 = m->buf.h2;
    g.tiles = tiles;
    g.nrows = nrows;
    g.y = y;
    g.status = m->status;
    return g;
}

// Forward and backward of nrows rows: five launches, the last of which leaves
// the gradient vector in m->grad or, with adam, takes the step.
int batch_gradients(Mlp *m, const long long *d_rows, unsigned long long seed, long long nrows,
                    float w_d, float w_a, float w_e, const Adam *adam) {
    const int tiles = (int)((nrows + kTileM - 1) / kTileM);
    int rc = ensure_buffers(m, tiles, m->buf_allocs);
    if (rc) return rc;
    Buffers &B = m->buf;
    const unsigned ctas = (unsigned)std::min(tiles, m->sms);
    Batch batch{d_rows, seed, d_rows ? 0 : m->S * m->N, 0, nrows};
    if ((rc = layers12(m, batch, tiles))) return rc;
    Layer3 g3 = layer3(m, tiles, nrows, B.y);
    g3.targets = m->targets;
    g3.row_of = B.row_of;
    g3.d3 = B.d3;
    g3.d2 = B.d2;
    g3.part4 = B.part4;
    g3.w_d = w_d;
    g3.w_a = w_a;
    g3.w_e = w_e;
    if ((rc = launch(m, mlp_layer3_train, dim3(ctas), kThreads, smem_of<Smem3T>(), g3))) return rc;
    Back2 g2{m->w, B.d2, B.h1, B.d1, tiles, m->status};
    if ((rc = launch(m, mlp_back2, dim3(ctas), kThreads, smem_of<SmemB>(), g2))) return rc;
    // CTAs of the weight gradients: an item each while the SMs suffice; a
    // seventh of them for layer 1
    const int s = wgrad_splits(tiles);
    const int big = std::max(1, std::min(2 * s, m->sms - m->sms / 7));
    const int small = std::max(1, std::min(s, m->sms - big));
    Wgrad gw{B.h1, B.h2, B.x, B.d1, B.d2, B.d3, tiles, s, big, B.part, B.part1, B.part_b,
             m->status};
    if ((rc = launch(m, mlp_wgrad, dim3((unsigned)(big + small)), kThreadsW + 32, smem_of<SmemW>(), gw)))
        return rc;
    Finish gf{B.part, B.part1, B.part_b, B.part4, s, (int)ctas, adam ? nullptr : m->grad, m->loss,
              adam ? *adam : Adam{}, m->w};
    return launch(m, mlp_finish, dim3((kItems + 255) / 256), 256, 0, gf);
}

int read_status(Mlp *m, const char *what) {
    int st = 0;
    MCK(cudaMemcpy(&st, m->status, sizeof(int), cudaMemcpyDeviceToHost));
    if (st) {
        if (st == SWGPU_ETIMEOUT) m->unusable = true;
        return mfail(m, st, "%s: a tensor-core wait ran out; destroy the handle", what);
    }
    return SWGPU_OK;
}

int usable(Mlp *m, const char *what) {
    if (m && m->unusable)
        return mfail(m, SWGPU_ETIMEOUT,
                     "%s: handle unusable after a tensor-core wait ran out; destroy it", what);
    return SWGPU_OK;
}

}  // namespace

extern "C" {

int swgpu_mlp_create(const float *params, const float *feature_mean,
                     const float *feature_inv_std, void **handle_out) {
    if (!params || !feature_mean || !feature_inv_std || !handle_out)
        return mfail(nullptr, SWGPU_EINVAL, "swgpu_mlp_create: null argument");
    *handle_out = nullptr;
    Mlp *m = new Mlp();
    int rc = SWGPU_OK;
    cudaError_t e = cudaGetDevice(&m->device);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, m->device);
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = smem_attr(mlp_predict, smem_of<SmemP>());
    if (e == cudaSuccess) e = smem_attr(mlp_layers12, smem_of<Smem12>());
    if (e == cudaSuccess) e = smem_attr(mlp_layer3_train, smem_of<Smem3T>());
    if (e == cudaSuccess) e = smem_attr(mlp_back2, smem_of<SmemB>());
    if (e == cudaSuccess) e = smem_attr(mlp_wgrad, smem_of<SmemW>());
    if (e != cudaSuccess) {
        rc = mfail(m, SWGPU_ECUDA, "swgpu_mlp_create: %s", cudaGetErrorString(e));
        delete m;
        return rc;
    }
    if ((rc = malloc_dev(m, &m->params, kNumParams)) || (rc = malloc_dev(m, &m->grad, kNumParams)) ||
        (rc = malloc_dev(m, &m->adam_m, kNumParams)) ||
        (rc = malloc_dev(m, &m->adam_v, kNumParams)) || (rc = malloc_dev(m, &m->w, 1)) ||
        (rc = malloc_dev(m, &m->mu, kF)) || (rc = malloc_dev(m, &m->isd, kF)) ||
        (rc = malloc_dev(m, &m->loss, 1)) || (rc = malloc_dev(m, &m->status, 1))) {
        free_list(m->allocs);
        delete m;
        return rc;
    }
    e = cudaMemcpy(m->params, params, sizeof(float) * kNumParams, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(m->mu, feature_mean, sizeof(float) * kF, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(m->isd, feature_inv_std, sizeof(float) * kF, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(m->adam_m, 0, sizeof(float) * kNumParams);
    if (e == cudaSuccess) e = cudaMemset(m->adam_v, 0, sizeof(float) * kNumParams);
    if (e == cudaSuccess) e = cudaMemset(m->status, 0, sizeof(int));
    if (e == cudaSuccess) {
        mlp_pack_weights<<<(kH * kH + 255) / 256, 256, 0, m->stream>>>(m->params, m->w);
        e = cudaStreamSynchronize(m->stream);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        rc = mfail(m, SWGPU_ECUDA, "swgpu_mlp_create: %s", cudaGetErrorString(e));
        free_list(m->allocs);
        delete m;
        return rc;
    }
    *handle_out = m;
    return SWGPU_OK;
}

int swgpu_mlp_destroy(void *handle) {
    Mlp *m = static_cast<Mlp *>(handle);
    if (!m) return SWGPU_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    free_list(m->data_allocs);
    free_list(m->buf_allocs);
    free_list(m->allocs);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return SWGPU_OK;
}

const char *swgpu_mlp_last_error(void *handle) {
    Mlp *m = static_cast<Mlp *>(handle);
    return m ? m->err.c_str() : g_mlp_error.c_str();
}

int swgpu_mlp_set_data(void *handle, const float *tri, int64_t ntri, const float *scen,
                       int64_t nscen, const float *targets) {
    Mlp *m = static_cast<Mlp *>(handle);
    if (!m || !tri || !scen || ntri <= 0 || nscen <= 0)
        return mfail(m, SWGPU_EINVAL, "swgpu_mlp_set_data: bad argument");
    if (int rc = usable(m, "swgpu_mlp_set_data")) return rc;
    if ((long long)ntri * nscen >= (1LL << 40))
        return mfail(m, SWGPU_EINVAL, "swgpu_mlp_set_data: too many rows");
    MCK(cudaStreamSynchronize(m->stream));
    free_list(m->data_allocs);
    m->tri = m->scen = m->targets = nullptr;
    m->N = m->S = 0;
    int rc;
    if ((rc = malloc_dev(m, &m->tri, (size_t)ntri * kTri, &m->data_allocs)) ||
        (rc = malloc_dev(m, &m->scen, (size_t)nscen * kParams, &m->data_allocs)))
        return rc;
    MCK(cudaMemcpy(m->tri, tri, sizeof(float) * kTri * ntri, cudaMemcpyHostToDevice));
    MCK(cudaMemcpy(m->scen, scen, sizeof(float) * kParams * nscen, cudaMemcpyHostToDevice));
    if (targets) {
        if ((rc = malloc_dev(m, &m->targets, (size_t)ntri * nscen * kTargets, &m->data_allocs)))
            return rc;
        MCK(cudaMemcpy(m->targets, targets, sizeof(float) * kTargets * ntri * nscen,
                       cudaMemcpyHostToDevice));
    }
    m->N = ntri;
    m->S = nscen;
    return SWGPU_OK;
}

int swgpu_mlp_predict(void *handle, int64_t row0, int64_t nrows, float *out_device,
                      float *elapsed_ms) {
    Mlp *m = static_cast<Mlp *>(handle);
    if (!m || !out_device || nrows <= 0 || row0 < 0 || row0 + nrows > m->S * m->N)
        return mfail(m, SWGPU_EINVAL, "swgpu_mlp_predict: bad rows");
    if (int rc = usable(m, "swgpu_mlp_predict")) return rc;
    const int most = std::max(1, m->sms / 2);  // pairs of CTAs
    int rc = SWGPU_OK;
    cudaEvent_t a, b;
    MCK(cudaEventCreate(&a));
    MCK(cudaEventCreate(&b));
    MCK(cudaEventRecord(a, m->stream));
    const long long chunk = (1LL << 24) * kTileM;  // (the tiles of a launch are counted in an int)
    for (long long r0 = 0; r0 < nrows; r0 += chunk) {
        const long long n = std::min(chunk, nrows - r0);
        const int pairs = (int)((n + kPairRows - 1) / kPairRows);
        const Predict g{tables(m), Batch{nullptr, 0, 0, row0 + r0, n}, m->w, m->params + kOffB1,
                        m->params + kOffB2, m->params + kOffB3, m->params + kOffB4,
                        out_device + r0 * kOut, pairs, m->status};
        if ((rc = launch(m, mlp_predict, dim3(2u * (unsigned)std::min(pairs, most)), kThreadsP,
                         smem_of<SmemP>(), g)))
            return rc;
    }
    MCK(cudaEventRecord(b, m->stream));
    MCK(cudaEventSynchronize(b));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if ((rc = read_status(m, "swgpu_mlp_predict"))) return rc;
    if (elapsed_ms) *elapsed_ms = ms;
    return SWGPU_OK;
}

int swgpu_mlp_gradients(void *handle, const int64_t *rows, int64_t nrows, float w_depth,
                        float w_arrival, float w_error, float *outputs, float *grad,
                        float *loss) {
    Mlp *m = static_cast<Mlp *>(handle);
    if (!m || !rows || nrows <= 0 || !m->targets)
        return mfail(m, SWGPU_EINVAL, "swgpu_mlp_gradients: bad argument or no targets");
    if (int rc = usable(m, "swgpu_mlp_gradients")) return rc;
    for (int64_t i = 0; i < nrows; i++)
        if (rows[i] < 0 || rows[i] >= m->S * m->N)
            return mfail(m, SWGPU_EINVAL, "swgpu_mlp_gradients: row %lld out of range",
                         (long long)rows[i]);
    int rc;
    if (nrows > m->rows_cap) {
        if ((rc = malloc_dev(m, &m->rows, (size_t)nrows))) return rc;
        m->rows_cap = nrows;
    }
    MCK(cudaMemcpyAsync(m->rows, rows, sizeof(long long) * nrows, cudaMemcpyHostToDevice,
                        m->stream));
    if ((rc = batch_gradients(m, m->rows, 0, nrows, w_depth, w_arrival, w_error, nullptr)))
        return rc;
    if (outputs)
        MCK(cudaMemcpyAsync(outputs, m->buf.y, sizeof(float) * kOut * nrows,
                            cudaMemcpyDeviceToHost, m->stream));
    if (grad)
        MCK(cudaMemcpyAsync(grad, m->grad, sizeof(float) * kNumParams, cudaMemcpyDeviceToHost,
                            m->stream));
    if (loss)
        MCK(cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    MCK(cudaStreamSynchronize(m->stream));
    return read_status(m, "swgpu_mlp_gradients");
}

int swgpu_mlp_train(void *handle, int steps, int64_t batch, uint64_t seed, float lr,
                    float w_depth, float w_arrival, float w_error, float *last_loss,
                    float *elapsed_ms) {
    Mlp *m = static_cast<Mlp *>(handle);
    if (!m || steps <= 0 || batch <= 0 || !m->targets)
        return mfail(m, SWGPU_EINVAL, "swgpu_mlp_train: bad argument or no targets");
    if (int rc = usable(m, "swgpu_mlp_train")) return rc;
    cudaEvent_t a, b;
    MCK(cudaEventCreate(&a));
    MCK(cudaEventCreate(&b));
    MCK(cudaEventRecord(a, m->stream));
    const float b1 = 0.9f, b2 = 0.999f;
    for (int s = 0; s < steps; s++) {
        const unsigned long long step_seed = seed * 0x9E3779B97F4A7C15ull + (unsigned)s;
        const float c1 = 1.f / (1.f - powf(b1, (float)(m->adam_t + 1)));
        const float c2 = 1.f / (1.f - powf(b2, (float)(m->adam_t + 1)));
        const Adam adam{m->params, m->adam_m, m->adam_v, lr, b1, b2, 1e-8f, c1, c2};
        int rc = batch_gradients(m, nullptr, step_seed, batch, w_depth, w_arrival, w_error, &adam);
        if (rc) return rc;
        m->adam_t++;
    }
    MCK(cudaGetLastError());
    MCK(cudaEventRecord(b, m->stream));
    MCK(cudaEventSynchronize(b));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, a, b);
    cudaEventDestroy(a);
    cudaEventDestroy(b);
    if (int rc = read_status(m, "swgpu_mlp_train")) return rc;
    if (elapsed_ms) *elapsed_ms = ms;
    if (last_loss) MCK(cudaMemcpy(last_loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost));
    return SWGPU_OK;
}

int swgpu_mlp_get_params(void *handle, float *params) {
    Mlp *m = static_cast<Mlp *>(handle);
    if (!m || !params) return mfail(m, SWGPU_EINVAL, "swgpu_mlp_get_params: null argument");
    MCK(cudaStreamSynchronize(m->stream));
    MCK(cudaMemcpy(params, m->params, sizeof(float) * kNumParams, cudaMemcpyDeviceToHost));
    return SWGPU_OK;
}

int swgpu_mlp_num_params(void) { return (int)kNumParams; }

}  // extern "C"
