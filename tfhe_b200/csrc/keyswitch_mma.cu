// keyswitch_mma.cu -- the LWE keyswitch (lweKeySwitch, lwe-keyswitch-functions.cpp:228-238, through
// lweKeySwitchTranslate_fromArray, :111-136) on the tensor cores, for t = 8 digits of 2 bits.
//
// The keyswitch subtracts, for every mask coefficient i and digit position j, the key sample
// ks[i][j][h] that digit j of abar_i = a_i + 2^(32-(1+2t)) selects; h = 0 is skipped.  That is a
// product of a one-hot matrix with the key:
//     A[s][(i, h, j)] = (digit j of sample s's abar_i == h),   B[(i, h, j)][col] = ks[i][j][h][col],  h = 1, 2, 3.
// Modulo 2^32 the key splits into four byte planes, B = sum_p 2^(8p) B_p, and each A x B_p is an exact
// product of u8 matrices with s32 sums: an entry adds at most t = 8 bytes per coefficient, kN * 8 * 255 < 2^23.  So
//     out[s][col] = (col == n ? b_s : 0) - sum_p 2^(8p) (A x B_p)[s][col]   (mod 2^32),
// the reference's result bit for bit.
//
// Tiling.  A unit of work is 256 samples (two accumulators of M = 128 rows) x 64 output columns, whose
// four byte planes make N = 256 (plane p of column c at n = 64 p + c).  K runs over the coefficients in quads:
// four of them, 8 digit positions each, make the 32 bytes of one K step per digit value h (byte 8c + position), so
// three tcgen05.mma.kind::i8 of M 128, N 256, K 32 per quad and accumulator; the two accumulators take all 512
// TMEM columns.  (With the 4 values of a digit side by side, h = 0 was a quarter of all bytes and products.)
//
// Split.  The units' quads are one line of work, cut into equal parts, one per CTA and SM: 160 units on 148 SMs
// otherwise take two waves, or five of quarter units.  A CTA's part spans a unit's end or two; each piece of a
// unit ends with its own epilogue, and the partial sums of a unit meet in the output through atomic adds, exact
// modulo 2^32 (a unit that one CTA does alone is stored).
//
// What bounds it: the products.  One of M 128, N 256, K 32 takes 267 cycles of an SM here (256 at 4096 multiply-adds per
// cycle); 4096 samples of the default set are 277 quads per SM, 6 products each: 0.217 ms, and 0.219 ms measured
// (0.305 ms with the h = 0 bytes and five waves of quarter units; one sample 0.021 ms, was 0.035).  Twice the row
// threads or 32-byte swizzled operands changed nothing.
//
// Roles (320 threads):
//   warps 0-7  one sample row each: write the row's one-hot A bytes (six 16-byte stores per quad) into the stage,
//              then, after a piece's last product, read the row's accumulators from TMEM, combine the planes
//              and store or add the 64 columns;
//   warp 8     lane 0 streams B: one bulk copy per stage from the device key, laid out offline in
//              the exact shared-memory image the descriptors describe;
//   warp 9     lane 0 issues the products and commits each stage back to the producers.
// A stage filled for the next piece by all 256 row threads implies that they have read the accumulators.
// Operands use the no-swizzle K-major layout: core matrices of 8 rows x 16 bytes, the two 16-byte K
// halves of a row 128 bytes apart, 8-row groups 256 bytes apart.
// Every mbarrier wait is bounded (async_copy.cuh).  After a wait runs out, each role stops, the copy
// issuer waits for its copies in flight, the issuing thread waits for its products, and warp 0
// frees the TMEM columns after the final barrier.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "async_copy.cuh"
#include "internal.h"
#include "tmem.cuh"

namespace tfheb {

namespace {

constexpr int kKmT = 8;                                   // digit positions
constexpr int kKmRows = 128;                              // samples per accumulator (M)
constexpr int kKmHalves = 2;                              // accumulators per CTA
constexpr int kKmTile = kKmRows * kKmHalves;              // samples per CTA
constexpr int kKmCols = 64;                               // output columns per CTA
constexpr int kKmN = 4 * kKmCols;                         // byte planes x columns (N)
constexpr int kKmQuad = 4;                                // coefficients per pipeline stage
constexpr int kKmSteps = 3;                               // K steps per stage: digit values 1, 2, 3
constexpr int kKmStages = 4;
constexpr int kKmABytes = kKmRows * 32;                   // one accumulator's A of one K step
constexpr int kKmBBytes = kKmN * 32;                      // B of one K step (8 KB)
constexpr int kKmStageA = kKmHalves * kKmSteps * kKmABytes;  // 24 KB
constexpr int kKmStageB = kKmSteps * kKmBBytes;              // 24 KB
constexpr int kKmStageBytes = kKmStageA + kKmStageB;
constexpr int kKmProducers = kKmTile;                     // one thread per sample row
constexpr int kKmThreads = kKmProducers + 64;
constexpr int kKmEpiCols = 16;                            // columns per pass of the epilogue
constexpr int kKmStageLd = kKmEpiCols + 1;                // its staging row length (words)
constexpr int kKmEpiOff = kKmStages * kKmStageBytes;      // 192 KB of stages, then the epilogue's staging
constexpr int kKmBarOff = kKmEpiOff + kKmProducers * kKmStageLd * 4;
constexpr int kKmMiscOff = kKmBarOff + (3 * kKmStages + 2) * 8;
constexpr int kKmSmem = kKmMiscOff + 16;
constexpr uint32_t kKmTmemCols = kKmHalves * kKmN;        // 512
constexpr int kKmLeast = 8;                               // least quads worth a CTA of their own
constexpr int kKmEpilogue = 3;                            // an epilogue's time in quads

static_assert(kKmSmem <= 227 * 1024, "shared memory");
static_assert(kKmTmemCols == 512, "two accumulators of N columns fill TMEM");

// byte of digit position j (0 = the most significant) of coefficient c of a quad, in a K step
__host__ __device__ constexpr int km_kbyte(int c, int j) { return 8 * c + (j < 4 ? 3 - j : 11 - j); }

// the four 2-bit digits of a byte (position 3 lowest) to one byte each
__device__ __forceinline__ uint32_t km_spread(uint32_t t) {
    const uint32_t y = (t * 4097u) & 0x000F000Fu;  // no two terms of either product overlap
    return (y * 65u) & 0x03030303u;
}

// byte offset of (row, k-byte) in an operand of the no-swizzle K-major layout
__host__ __device__ constexpr uint32_t km_offset(int row, int kb) {
    return (uint32_t)((row >> 3) * 256 + (kb >> 4) * 128 + (row & 7) * 16 + (kb & 15));
}

__global__ void __launch_bounds__(kKmThreads, 1)
    keyswitch_mma_kernel(const uint8_t *__restrict__ bkey, const uint32_t *__restrict__ in, int in_stride,
                         uint32_t *__restrict__ out, int count, int n, int kN, int groups, long total,
                         uint64_t timeout_ns, int32_t *err, int stall) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int quads = kN / kKmQuad;  // per unit
    const long begin = total * blockIdx.x / gridDim.x, end = total * (blockIdx.x + 1) / gridDim.x;

    const uint32_t sbase = smem_addr(smem);
    const uint32_t full_a = sbase + kKmBarOff, full_b = full_a + 8 * kKmStages, empty = full_b + 8 * kKmStages;
    const uint32_t done = empty + 8 * kKmStages, drained = done + 8;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + kKmMiscOff);
    volatile int32_t *abort_flag = reinterpret_cast<volatile int32_t *>(smem + kKmMiscOff + 4);
    if (tid == 0) {
        for (int s = 0; s < kKmStages; s++) {
            mbar_init(full_a + 8 * s, kKmProducers);
            mbar_init(full_b + 8 * s, 1);
            mbar_init(empty + 8 * s, 1);
        }
        mbar_init(done, 1);
        mbar_init(drained, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) tmem_alloc(smem_addr(tmem_slot), kKmTmemCols);
    tmem_fence_before_sync();
    __syncthreads();
    tmem_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (tid < kKmProducers) {
        // ---- one-hot rows, and per piece the epilogue ----
        const int h = tid / kKmRows, rr = tid % kKmRows;
        const uint32_t prec_offset = 1u << (32 - (1 + 2 * kKmT));  // lwe-keyswitch-functions.cpp:119
        unsigned char *a_row = smem + h * (kKmSteps * kKmABytes) + km_offset(rr, 0);
        uint32_t *stg = reinterpret_cast<uint32_t *>(smem + kKmEpiOff) + warp * 32 * kKmStageLd;
        const uint32_t t_row = tmem_base + ((uint32_t)((warp % 4) * 32) << 16) + (uint32_t)(h * kKmN);
        bool ok = true;
        int q0 = 0;  // stages filled before the piece
        uint32_t piece = 0;
        for (long w = begin; w < end && ok; piece++) {
            const int unit = (int)(w / quads), first = (int)(w - (long)unit * quads);
            const int len = (int)min((long)(quads - first), end - w);
            w += len;
            const int g = unit % groups, tile = unit / groups;
            const int sample = tile * kKmTile + tid;
            const bool live = sample < count;
            const uint32_t *src = in + (size_t)(live ? sample : 0) * in_stride + (size_t)first * kKmQuad;
            // the next two quads' inputs ahead: a row's eight words are one 32-byte sector
            constexpr int kPair = 2 * kKmQuad;
            uint32_t cur[kPair], nxt[kPair];
#pragma unroll
            for (int e = 0; e < kPair; e++) cur[e] = live && e < len * kKmQuad ? __ldg(src + e) : 0u;
            for (int i0 = 0; i0 < len && ok; i0 += 2) {
                const int ahead = (i0 + 2) * kKmQuad;
#pragma unroll
                for (int e = 0; e < kPair; e++) nxt[e] = live && ahead + e < len * kKmQuad ? __ldg(src + ahead + e) : 0u;
#pragma unroll
                for (int qq = 0; qq < 2; qq++) {
                    if (i0 + qq >= len) break;
                    const int q = q0 + i0 + qq, s = q % kKmStages;
                    if (q >= kKmStages && !wait_bounded(empty + 8 * s, ((q / kKmStages) - 1) & 1, abort_flag, timeout_ns, err)) {
                        ok = false;
                        break;
                    }
                    uint32_t v[kKmSteps][2 * kKmQuad];
#pragma unroll
                    for (int c = 0; c < kKmQuad; c++) {
                        const uint32_t x = cur[qq * kKmQuad + c] + prec_offset;
#pragma unroll
                        for (int b = 0; b < 2; b++) {  // digits 0-3, 4-7 from the top (:128-131)
                            const uint32_t y = live ? km_spread((x >> (24 - 8 * b)) & 255u) : 0u, z = y >> 1;
                            v[0][2 * c + b] = y & ~z & 0x01010101u;
                            v[1][2 * c + b] = ~y & z & 0x01010101u;
                            v[2][2 * c + b] = y & z & 0x01010101u;
                        }
                    }
                    unsigned char *a = a_row + s * kKmStageBytes;
#pragma unroll
                    for (int k = 0; k < kKmSteps; k++) {
                        *reinterpret_cast<uint4 *>(a + k * kKmABytes) = make_uint4(v[k][0], v[k][1], v[k][2], v[k][3]);
                        *reinterpret_cast<uint4 *>(a + k * kKmABytes + 128) = make_uint4(v[k][4], v[k][5], v[k][6], v[k][7]);
                    }
                    fence_proxy_async_smem();
                    mbar_arrive(full_a + 8 * s);
                }
#pragma unroll
                for (int e = 0; e < kPair; e++) cur[e] = nxt[e];
            }
            q0 += len;
            // accumulators -> columns
            ok = ok && wait_bounded(done, piece & 1u, abort_flag, timeout_ns, err);
            ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld is warp-collective
            if (!ok) break;
            tmem_fence_after_sync();
            const int ncols = n + 1, row0 = tile * kKmTile + warp * 32;
#pragma unroll 1
            for (int c0 = 0; c0 < kKmCols; c0 += kKmEpiCols) {
                uint32_t p0[16], p1[16], p2[16], p3[16];
                tmem_ld16(t_row + c0, p0);
                tmem_ld16(t_row + kKmCols + c0, p1);
                tmem_ld16(t_row + 2 * kKmCols + c0, p2);
                tmem_ld16(t_row + 3 * kKmCols + c0, p3);
                tmem_wait_ld16(p0);
                tmem_wait_ld16(p1);
                tmem_wait_ld16(p2);
                tmem_wait_ld16(p3);
#pragma unroll
                for (int e = 0; e < kKmEpiCols; e++)
                    stg[lane * kKmStageLd + e] = p0[e] + (p1[e] << 8) + (p2[e] << 16) + (p3[e] << 24);
                __syncwarp();
                // two rows of 16 columns per pass
                const int c = lane & 15, col = g * kKmCols + c0 + c;
                for (int r = lane >> 4; r < 32; r += 2) {
                    if (row0 + r >= count || col >= ncols) continue;
                    // result = (0, b) - sum  (lwe-keyswitch-functions.cpp:233-237)
                    uint32_t v = 0u - stg[r * kKmStageLd + c];
                    if (col == n && first == 0) v += in[(size_t)(row0 + r) * in_stride + kN];
                    uint32_t *o = out + (size_t)(row0 + r) * ncols + col;
                    if (len == quads) *o = v;
                    else atomicAdd(o, v);
                }
                __syncwarp();
            }
            tmem_fence_before_sync();  // before the arrivals that let the next piece's products start
        }
    } else if (warp == kKmProducers / 32 && lane == 0) {
        // ---- key stream ----
        int issued = 0;
        if (!stall) {  // stall: failure-detection test hook, no copy is ever issued
            for (long w = begin; w < end; w++) {
                const int s = issued % kKmStages, unit = (int)(w / quads);
                if (issued >= kKmStages &&
                    !wait_bounded(empty + 8 * s, ((issued / kKmStages) - 1) & 1, abort_flag, timeout_ns, err))
                    break;
                mbar_arrive_expect_tx(full_b + 8 * s, kKmStageB);
                bulk_copy_g2s(sbase + s * kKmStageBytes + kKmStageA,
                              bkey + ((size_t)(unit % groups) * quads + (size_t)(w - (long)unit * quads)) * kKmStageB,
                              kKmStageB, full_b + 8 * s);
                issued++;
            }
        }
        // copies still in flight land before the CTA exits (each wait bounded)
        volatile int32_t no_abort = 0;
        for (int q = std::max(0, issued - kKmStages); q < issued; q++)
            wait_bounded(full_b + 8 * (q % kKmStages), (q / kKmStages) & 1, &no_abort, timeout_ns, err);
    } else if (warp == kKmProducers / 32 + 1 && lane == 0) {
        // ---- products ----
        const uint32_t idesc = umma_idesc_u8_s32(kKmRows, kKmN);
        int q = 0;
        bool fresh = true;  // the piece's first products overwrite the accumulators
        for (long w = begin; w < end; w++, q++) {
            const int s = q % kKmStages, par = (q / kKmStages) & 1;
            if (!wait_bounded(full_a + 8 * s, par, abort_flag, timeout_ns, err) ||
                !wait_bounded(full_b + 8 * s, par, abort_flag, timeout_ns, err))
                break;
            tmem_fence_after_sync();
            const uint32_t stage = sbase + s * kKmStageBytes;
#pragma unroll
            for (int k = 0; k < kKmSteps; k++) {
                const uint64_t bdesc = umma_desc_kmajor(stage + kKmStageA + k * kKmBBytes, 128, 256);
#pragma unroll
                for (int hh = 0; hh < kKmHalves; hh++) {
                    const uint64_t adesc = umma_desc_kmajor(stage + (hh * kKmSteps + k) * kKmABytes, 128, 256);
                    umma_u8(tmem_base + (uint32_t)(hh * kKmN), adesc, bdesc, idesc, !fresh || k != 0);
                }
            }
            fresh = false;
            umma_commit(empty + 8 * s);
            if (w + 1 == end || (w + 1) % quads == 0) {
                umma_commit(done);
                fresh = true;
            }
        }
        // the products issued so far complete before the CTA exits (the wait is bounded)
        umma_commit(drained);
        volatile int32_t no_abort = 0;
        wait_bounded(drained, 0, &no_abort, timeout_ns, err);
    }

    tmem_fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        tmem_fence_after_sync();
        tmem_free(tmem_base, kKmTmemCols);
    }
}

}  // namespace

// ============================================================================================
// host side
// ============================================================================================

int km_groups(const tfheb_params &p) { return (p.n + 1 + kKmCols - 1) / kKmCols; }

// The key in the shared-memory image of the B operand: [group][quad][digit value h = 1, 2, 3][8 KB], byte plane p of
// ks[i][j][h][64 g + c] at (row 64 p + c, k-byte km_kbyte(i % 4, j)); columns past n stay zero.
cudaError_t upload_keyswitch_key_mma(CloudKey &ck) {
    const tfheb_params &p = ck.p;
    DeviceKsk &d = ck.dksk;
    if (d.mma || p.ks_t != kKmT || p.ks_basebit != 2 || p.k * p.N % kKmQuad != 0) return cudaSuccess;
    const int kN = p.k * p.N, t = p.ks_t, base = 1 << p.ks_basebit, ncols = p.n + 1;
    const int groups = km_groups(p);
    std::vector<uint8_t> img((size_t)groups * (kN / kKmQuad) * kKmStageB, 0);
    for (int g = 0; g < groups; g++)
        for (int i = 0; i < kN; i++) {
            for (int j = 0; j < t; j++)
                for (int h = 1; h < base; h++) {
                    uint8_t *blk = &img[((size_t)g * (kN / kKmQuad) + i / kKmQuad) * kKmStageB + (size_t)(h - 1) * kKmBBytes];
                    const int32_t *srow = &ck.ksk[(((size_t)i * t + j) * base + h) * ncols];
                    const int kb = km_kbyte(i % kKmQuad, j);
                    for (int c = 0; c < kKmCols && g * kKmCols + c < ncols; c++) {
                        const uint32_t v = (uint32_t)srow[g * kKmCols + c];
                        for (int pl = 0; pl < 4; pl++) blk[km_offset(pl * kKmCols + c, kb)] = (uint8_t)(v >> (8 * pl));
                    }
                }
        }
    cudaError_t e;
    if ((e = cudaMalloc((void **)&d.mma, img.size())) != cudaSuccess) return e;
    if ((e = cudaMemcpy(d.mma, img.data(), img.size(), cudaMemcpyHostToDevice)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute(keyswitch_mma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kKmSmem)) !=
        cudaSuccess)
        return e;
    d.mma_groups = groups;
    return cudaSuccess;
}

cudaError_t launch_keyswitch_mma(const CloudKey &ck, int count, const int32_t *in, int in_stride, int32_t *out,
                                 cudaStream_t s) {
    const tfheb_params &p = ck.p;
    const int kN = p.k * p.N;
    if (!ck.dksk.mma) return cudaErrorInvalidValue;
    int sms = 0;
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ck.device);
    if (e != cudaSuccess) return e;
    const int groups = ck.dksk.mma_groups, quads = kN / kKmQuad;
    const long units = (long)((count + kKmTile - 1) / kKmTile) * groups, total = units * quads;
    // one part per SM, or the same number of parts for each unit where that fits and costs no more: parts that do not
    // span a unit's end have one epilogue (about kKmEpilogue quads) instead of two
    long ctas = std::max(1, sms);
    const long each = std::min((long)quads / kKmLeast, ctas / units);
    if (each >= 1 && (quads + each - 1) / each + kKmEpilogue <= (total + ctas - 1) / ctas + 2 * kKmEpilogue)
        ctas = units * each;
    const bool whole = total % ctas == 0 && (total / ctas) % quads == 0;  // every unit in one CTA
    if (!whole && (e = cudaMemsetAsync(out, 0, (size_t)count * (p.n + 1) * sizeof(int32_t), s)) != cudaSuccess) return e;
    keyswitch_mma_kernel<<<(unsigned)ctas, kKmThreads, kKmSmem, s>>>(
        ck.dksk.mma, reinterpret_cast<const uint32_t *>(in), in_stride, reinterpret_cast<uint32_t *>(out), count, p.n,
        kN, groups, total, ck.wait_timeout_ns, ck.d_err, ck.stall_producer);
    return cudaGetLastError();
}

}  // namespace tfheb
