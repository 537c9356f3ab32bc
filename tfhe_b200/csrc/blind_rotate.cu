// blind_rotate.cu -- persistent blind rotation on sm_100a (tfhe_blindRotate_FFT,
// lwe-bootstrapping-functions-fft.cpp:88-112, with tfhe_MuxRotate_FFT :67-76 and the external
// product tGswFFTExternMulToTLwe, tgsw-fft-operations.cpp:89-114).
//
// One CTA = G "teams" (one bootstrap each, N/16 threads per team) + one producer warp.
//   * Each team keeps its accumulator TLWE (k+1 polynomials of N Torus32) in shared memory for all
//     n CMUX steps.  Per step: rotation (X^a - 1)*acc, gadget decomposition, a forward negacyclic FFT
//     per digit polynomial (fft.cuh), multiply-accumulate against the bootstrapping-key row in the
//     FFT domain, inverse FFTs, rounding back to Torus32 and accumulation.
//   * The bootstrapping key is streamed once per CTA: the producer warp copies each key row
//     ((k+1) x N/2 slots x 16 bytes = 16 KB at N=1024) with a bulk asynchronous copy (TMA engine,
//     cp.async.bulk, no multicast) into a D-stage shared-memory ring guarded by mbarriers; all G teams
//     read the same stage.  L2->SM key traffic is therefore 62 MB per G bootstraps instead of per
//     bootstrap.
//   * Every mbarrier wait is bounded (%globaltimer).  On expiry the CTA raises a shared abort flag,
//     every later wait returns at once (the FFT barriers stay uniform, so nothing hangs), the
//     producer drains its in-flight copies, and the host reads TFHEB_ERR_TIMEOUT from the error word.
//
// Precision forms:
//   FP64  (SPLIT=false): key row slot = double2 B_k / M; products rounded with the 1.5*2^52 addition
//          (exact round-to-nearest for |x| < 2^51), reduced mod 2^32.
//   split (SPLIT=true):  key coefficient c = hi * 2^S + lo (S from default_split_shift); per register
//          pair (2m, 2m+1) and limb, float4 {re(2m), re(2m+1), im(2m), im(2m+1)} / M, one 16-byte load
//          per packed multiply-accumulate.  The high-limb product sums round to their exact integers
//          (S keeps their FP32 error far below 1/2); the low-limb sums round to the nearest integer of
//          their FP32 value; the two recombine as hi * 2^S + lo mod 2^32.
#include <cuda_runtime.h>
#include <stdint.h>

#include "async_copy.cuh"
#include "br_common.cuh"
#include "fft.cuh"
#include "internal.h"

namespace tfheb {

// ---- shared-memory layout ---------------------------------------------------------------------

template <typename T, int N, int K, int G, int D, bool PW = true>
struct BrLayout {
    static constexpr int M = N / 2, NT = M / kR, KP1 = K + 1;
    static constexpr uint32_t chunk = (uint32_t)KP1 * M * 16;  // one key row (step, p): all v, all slots
    static constexpr size_t bars = 0;                           // full[D], empty[D], abort flag
    static constexpr size_t ring = (2 * D * 8 + 4 + 127) / 128 * 128;  // the barrier block, then the ring
    static constexpr size_t tables = ring + (size_t)D * chunk;
    static constexpr size_t tables_bytes = tw_table_bytes<T, M>();
    static constexpr size_t teams = tables + tables_bytes;
    static constexpr size_t team_acc = 4 * (size_t)KP1 * N;
    static constexpr size_t team_xbuf = ((size_t)Exch<T, M>::bytes + 15) / 16 * 16;  // one exchange buffer
    // two alternating exchange buffers: one barrier per exchange (at N = 2048 with the per-exchange
    // float2 maps: 69.5 ms per 2048 split bootstraps against 69.7-70.5 ms with one buffer)
    static constexpr int xbufs = 2;
    static constexpr size_t team_buf = xbufs * team_xbuf;
    // the rotated accumulator polynomial being decomposed (N words), read once per digit: kept in a
    // per-team shared scratch when registers are tight (more than 256 threads per CTA, so at most 168
    // registers each) and the scratch fits beside the key ring, else in registers.  A deeper ring
    // measured faster than the scratch (36.15 ms per 4096 split bootstraps at G = 7, D = 6 without it,
    // 36.6 ms at D = 4 with it), and a lone team with 255 registers runs slower with it.
    static constexpr size_t kMaxSmem = 227 * 1024;
    static constexpr int threads = G * (N / 16) + (PW ? 32 : 0);
    static constexpr bool rot_in_smem =
        threads > 256 && teams + G * (team_acc + team_buf + 4 * (size_t)N) <= kMaxSmem;
    static constexpr size_t team_rot = rot_in_smem ? 4 * (size_t)N : 0;
    __host__ __device__ static size_t team_bytes(int) { return team_acc + team_buf + team_rot; }
    __host__ __device__ static size_t bytes(int nsteps) { return teams + G * team_bytes(nsteps); }
    static_assert(2 * D * 8 + 4 <= ring, "barrier block");
    static_assert(teams + G * (team_acc + team_buf) <= kMaxSmem, "shared memory of the variant");
};



// PW: a key-streaming warp issues the row copies.  Without it (G teams only), thread 0 issues them:
// the first D at the start, then each row as soon as every team has released its slot, tested after
// each of its own rows and waited for only when thread 0 needs a row not yet issued.  That frees the
// producer warp's registers: 4 FP64 teams are 256 threads, which may use 255 registers each.
// EXT: the external product alone (tGswExternProduct, tgsw-functions.cpp:416-431): each step computes
// acc = bk_step (x) acc, without the rotation (X^a - 1) and without adding the old accumulator; the
// rotation amounts are not read.  Only a few one-bootstrap-per-CTA variants are compiled with it.
template <typename T, int N, int K, int L, bool SPLIT, int G, int D, bool PW = true, bool EXT = false>
__global__ void __launch_bounds__(G *(N / 16) + (PW ? 32 : 0), 1) blind_rotate_kernel(const BrArgs args) {
    using Lay = BrLayout<T, N, K, G, D, PW>;
    constexpr int M = N / 2, NT = M / kR, KP1 = K + 1, KPL = KP1 * L;
    using F = TeamFft<T, M, kR>;
    extern __shared__ __align__(128) unsigned char smem[];

    const int tid = threadIdx.x;
    const int consumers = G * NT;
    const int active_teams = min(G, args.boots - (int)blockIdx.x * G);
    const uint32_t bar0 = smem_addr(smem + Lay::bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (D + s); };
    volatile int32_t *abort_flag = reinterpret_cast<volatile int32_t *>(smem + Lay::bars + 16 * D);
    const uint32_t ring = smem_addr(smem + Lay::ring);

    if (tid == 0) {
        for (int s = 0; s < D; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), (uint32_t)(active_teams * NT));
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    cplx<T> *s_tab = reinterpret_cast<cplx<T> *>(smem + Lay::tables);
    {
        const int4 *g_tab = reinterpret_cast<const int4 *>(args.tables);
        int4 *s_tab4 = reinterpret_cast<int4 *>(smem + Lay::tables);
        for (int i = tid; i < (int)(Lay::tables_bytes / 16); i += blockDim.x) s_tab4[i] = g_tab[i];
    }
    __syncthreads();

    const int total_chunks = args.nsteps * KPL;
    // row c into its ring slot (the slot's previous row released by every team)
    auto issue_row = [&](int c) {
        const int s = c % D;
        mbar_arrive_expect_tx(full_bar(s), Lay::chunk);
        bulk_copy_g2s(ring + (uint32_t)s * Lay::chunk, args.bsk + (size_t)c * Lay::chunk, Lay::chunk, full_bar(s));
    };
    int issued = 0;        // !PW: rows issued by thread 0
    bool issuing = !PW && tid == 0 && !args.stall_producer;
    if (issuing)
        for (; issued < min(D, total_chunks); issued++) issue_row(issued);

    // ---------------- producer warp: stream the key rows ----------------
    if (tid >= consumers) {
        if (tid == consumers) {
            int sent = 0;
            if (!args.stall_producer) {
                for (int c = 0; c < total_chunks; c++) {
                    const int s = c % D;
                    if (c >= D && !wait_bounded(empty_bar(s), ((c / D) - 1) & 1, abort_flag, args.timeout_ns, args.err))
                        break;
                    mbar_arrive_expect_tx(full_bar(s), Lay::chunk);
                    bulk_copy_g2s(ring + (uint32_t)s * Lay::chunk, args.bsk + (size_t)c * Lay::chunk, Lay::chunk,
                                  full_bar(s));
                    sent = c + 1;
                }
            }
            // drain the copies still in flight before the CTA may exit (each wait bounded)
            volatile int32_t no_abort = 0;
            for (int c = (sent > D ? sent - D : 0); c < sent; c++)
                wait_bounded(full_bar(c % D), (c / D) & 1, &no_abort, args.timeout_ns, args.err);
        }
        return;
    }

    // ---------------- consumer teams ----------------
    const int team = tid / NT;
    const int t = tid - team * NT;
    if (team >= active_teams) return;  // not counted in the empty barriers; no CTA barrier follows
    const int boot = blockIdx.x * G + team;
    const int bar_id = 1 + team;

    unsigned char *tb = smem + Lay::teams + (size_t)team * Lay::team_bytes(args.nsteps);
    uint32_t *s_acc = reinterpret_cast<uint32_t *>(tb);
    ExchPair xp{tb + Lay::team_acc, Lay::xbufs == 2 ? (uint32_t)Lay::team_xbuf : 0u, 0u};
    uint32_t *s_rot = reinterpret_cast<uint32_t *>(tb + Lay::team_acc + Lay::team_buf);
    const cplx<T> *s_tw = s_tab;

    const int32_t *my_bara = EXT ? nullptr : args.bara + (size_t)boot * args.bara_stride;
    if (EXT || args.acc_in) {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(args.acc_in) + (size_t)boot * KP1 * N;
        for (int i = t; i < KP1 * N; i += NT) s_acc[i] = src[i];
    } else {
        // acc = (0, X^{2N-barb} * [mu,...,mu])  (lwe-bootstrapping-functions-fft.cpp:142-145)
        const int e = 2 * N - my_bara[args.nsteps];
        for (int i = t; i < K * N; i += NT) s_acc[i] = 0u;
        for (int j = t; j < N; j += NT) {
            int src = j - e;
            uint32_t neg = 0;
            while (src < 0) {
                src += N;
                neg ^= 1u;
            }
            s_acc[K * N + j] = neg ? 0u - (uint32_t)args.mu : (uint32_t)args.mu;
        }
    }
    team_sync(bar_id, NT);

    // gadget constants (tgsw.cpp:7-29)
    const int Bgbit = args.Bgbit;
    uint32_t offset = 0;
#pragma unroll
    for (int q = 0; q < L; q++) offset += 1u << (32 - (q + 1) * Bgbit);
    offset *= 1u << (Bgbit - 1);
    const uint32_t maskBg = (1u << Bgbit) - 1u;
    const T digit_bias = DigitConv<T>::base() + T(1 << (Bgbit - 1));

    int c = 0;  // key-row (chunk) counter, same sequence as the producer
    int a_next = (!EXT && args.nsteps > 0) ? my_bara[0] : 0;  // rotation amounts, loaded one step ahead
    // the new accumulator word: the old one plus the product, or (EXT) the product alone
    auto put = [](uint32_t &dst, uint32_t v) {
        if constexpr (EXT) dst = v;
        else dst += v;
    };
    for (int step = 0; step < args.nsteps; step++) {
        const int ai = a_next & (2 * N - 1);
        if (!EXT && step + 1 < args.nsteps) a_next = my_bara[step + 1];
        // FP64: one accumulator spectrum per output polynomial.  Split: hi- and lo-limb spectra as
        // packed register pairs over the slots (2m, 2m+1).
        cplx<T> acc_hi[SPLIT ? 1 : KP1][kR];
        cpair acc_h[SPLIT ? KP1 : 1][kR / 2], acc_l[SPLIT ? KP1 : 1][kR / 2];
        if constexpr (SPLIT) {
#pragma unroll
            for (int v = 0; v < KP1; v++)
#pragma unroll
                for (int m = 0; m < kR / 2; m++) {
                    acc_h[v][m] = {{0.f, 0.f}, {0.f, 0.f}};
                    acc_l[v][m] = {{0.f, 0.f}, {0.f, 0.f}};
                }
        } else {
#pragma unroll
            for (int v = 0; v < KP1; v++)
#pragma unroll
                for (int r = 0; r < kR; r++) acc_hi[v][r] = {T(0), T(0)};
        }

        // Two independent transforms side by side (two dependency chains for the scheduler) where
        // registers allow.  Inverse, at most 384 threads per CTA (168 registers each): the split form's
        // two limbs of one output (64.1 against 65.6 ms per 2048 bootstraps at N = 2048, G = 2), FP64's
        // two outputs.  At 128 registers the pair spills and ran 0.9 % slower (split, G = 7), so there
        // the transforms go one after the other.  Forward, FP64 at most 256 threads (255 registers):
        // the digits in chain order, two at a time, so every accumulator takes its products in the
        // same order as one at a time; the inverse that follows must be a pair (it begins with a
        // barrier).  One wave of 148 bootstraps at G = 1: 3.07 against 3.36 ms; at G = 3, 51.7 against
        // 53.6 ms per 4096.  The split form ran slower paired (3.97 against 3.20 ms at G = 1).
        constexpr bool kPairInverse = Lay::threads <= 384;
        constexpr bool kPairForward =
            !SPLIT && Lay::threads <= 256 && !Lay::rot_in_smem && KPL % 2 == 0 && kPairInverse && KP1 == 2;
        // one digit's spectrum times key row c into the accumulators; frees the row's ring slot
        auto accumulate = [&](const cplx<T> *z) {
            const int s = c % D;
            if constexpr (!PW) {
                // thread 0 issues every row before anyone waits for it
                while (issuing && issued <= c && issued < total_chunks) {
                    if (!wait_bounded(empty_bar(issued % D), ((issued / D) - 1) & 1, abort_flag, args.timeout_ns,
                                      args.err)) {
                        issuing = false;
                        break;
                    }
                    issue_row(issued++);
                }
            }
            wait_bounded(full_bar(s), (c / D) & 1, abort_flag, args.timeout_ns, args.err);
            const unsigned char *stage = smem + Lay::ring + (size_t)s * Lay::chunk;
            if constexpr (SPLIT) {
                // key row: [v][m][limb][t] x float4 {re(2m), re(2m+1), im(2m), im(2m+1)}
#pragma unroll
                for (int m = 0; m < kR / 2; m++) {
                    const cpair zp = make_cpair(z[2 * m], z[2 * m + 1]);
                    // the same bits; one team alone runs faster with the product (6.30 against 6.40 ms per wave of 148
                    // at N = 2048), five at N = 1024 with the sign flips (6.71 against 6.84 ms)
                    const float2 nzi = G == 1 ? mul2(zp.im, make_float2(-1.f, -1.f)) : neg2(zp.im);
#pragma unroll
                    for (int v = 0; v < KP1; v++) {
                        const float4 *kp = reinterpret_cast<const float4 *>(
                            stage + ((size_t)((v * (kR / 2) + m) * 2) * NT + t) * 16);
                        cmac_pair(acc_h[v][m], zp, nzi, kp[0]);
                        cmac_pair(acc_l[v][m], zp, nzi, kp[NT]);
                    }
                }
            } else {
#pragma unroll
                for (int v = 0; v < KP1; v++)
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        const size_t off = ((size_t)(v * kR + r) * NT + t) * 16;
                        const double2 b = *reinterpret_cast<const double2 *>(stage + off);
                        cmac(acc_hi[v][r], z[r], cplx<T>{(T)b.x, (T)b.y});
                    }
            }
            mbar_arrive(empty_bar(s));
            if constexpr (!PW) {
                while (issuing && issued < total_chunks && mbar_test_wait(empty_bar(issued % D), ((issued / D) - 1) & 1))
                    issue_row(issued++);
            }
            c++;
        };
        // digit q of the words x[r] (a_j) and x[kR + r] (a_{j+M}), j = t + NT * r
        auto decompose = [&](cplx<T> *z, const uint32_t *x, int q) {
            const int shift = 32 - (q + 1) * Bgbit;
#pragma unroll
            for (int r = 0; r < kR; r++) {
                const T d0 = DigitConv<T>::conv((x[r] >> shift) & maskBg, digit_bias);
                const T d1 = DigitConv<T>::conv((x[kR + r] >> shift) & maskBg, digit_bias);
                z[r] = cplx<T>{d0, -d1};  // a_j - i a_{j+M}; the twist is folded into the FFT
            }
        };

        if constexpr (kPairForward) {
            // every polynomial's (X^a - 1) * poly + offset in registers, then the digits two at a time
            uint32_t xr[KP1][2 * kR];
#pragma unroll
            for (int u = 0; u < KP1; u++)
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    const int j = t + NT * r;
                    xr[u][r] = (EXT ? s_acc[u * N + j] : rot_minus_one<N>(s_acc + u * N, j, ai)) + offset;
                    xr[u][kR + r] = (EXT ? s_acc[u * N + j + M] : rot_minus_one<N>(s_acc + u * N, j + M, ai)) + offset;
                }
#pragma unroll 1
            for (int d = 0; d < KPL; d += 2) {
                cplx<T> za[kR], zb[kR];
                uint32_t x[2 * kR];
#pragma unroll
                for (int i = 0; i < 2 * kR; i++) {  // polynomial d / L (selects, no local memory)
                    x[i] = xr[0][i];
#pragma unroll
                    for (int u = 1; u < KP1; u++)
                        if (d / L == u) x[i] = xr[u][i];
                }
                decompose(za, x, d % L);
#pragma unroll
                for (int i = 0; i < 2 * kR; i++) {  // polynomial (d + 1) / L
                    x[i] = xr[0][i];
#pragma unroll
                    for (int u = 1; u < KP1; u++)
                        if ((d + 1) / L == u) x[i] = xr[u][i];
                }
                decompose(zb, x, (d + 1) % L);
                F::forward_pair(za, zb, xp, s_tw, t, bar_id);
                accumulate(za);
                accumulate(zb);
            }
        } else {
#pragma unroll 1
            for (int u = 0; u < KP1; u++) {
                const uint32_t *poly = s_acc + u * N;
                // (X^a - 1) * poly + offset, kept for the L digits: in the team's scratch (each thread
                // its own words, so no barrier, and no registers held across the digits' transforms)
                // or, where that does not fit, in registers
                uint32_t x[Lay::rot_in_smem ? 1 : 2 * kR];
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    const int j = t + NT * r;
                    const uint32_t v0 = (EXT ? poly[j] : rot_minus_one<N>(poly, j, ai)) + offset;
                    const uint32_t v1 = (EXT ? poly[j + M] : rot_minus_one<N>(poly, j + M, ai)) + offset;
                    if constexpr (Lay::rot_in_smem) {
                        s_rot[r * NT + t] = v0;
                        s_rot[(kR + r) * NT + t] = v1;
                    } else {
                        x[r] = v0;
                        x[kR + r] = v1;
                    }
                }
#pragma unroll 1
                for (int q = 0; q < L; q++) {
                    const int shift = 32 - (q + 1) * Bgbit;
                    cplx<T> z[kR];
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        const uint32_t v0 = Lay::rot_in_smem ? s_rot[r * NT + t] : x[r];
                        const uint32_t v1 = Lay::rot_in_smem ? s_rot[(kR + r) * NT + t] : x[kR + r];
                        const T d0 = DigitConv<T>::conv((v0 >> shift) & maskBg, digit_bias);
                        const T d1 = DigitConv<T>::conv((v1 >> shift) & maskBg, digit_bias);
                        z[r] = cplx<T>{d0, -d1};  // a_j - i a_{j+M}; the twist is folded into the FFT
                    }
                    F::forward(z, xp, s_tw, t, bar_id);
                    accumulate(z);
                }
            }
        }

        // inverse transforms, exact rounding, accumulate (the key was pre-scaled by 1/M)
        if constexpr (!SPLIT && kPairInverse && KP1 == 2) {
            cplx<T> z0[kR], z1[kR];
#pragma unroll
            for (int r = 0; r < kR; r++) {
                z0[r] = acc_hi[0][r];
                z1[r] = acc_hi[1][r];
            }
            F::inverse_pair(z0, z1, xp, s_tw, t, bar_id);
#pragma unroll
            for (int r = 0; r < kR; r++) {
                const int j = t + NT * r;
                put(s_acc[j], round_f64_mod32(z0[r].re));  // (c_j - i c_{j+M})
                put(s_acc[j + M], round_f64_mod32(-z0[r].im));
                put(s_acc[N + j], round_f64_mod32(z1[r].re));
                put(s_acc[N + j + M], round_f64_mod32(-z1[r].im));
            }
        }
#pragma unroll
        for (int v = 0; v < KP1; v++) {
            if constexpr (!SPLIT && kPairInverse && KP1 == 2) break;  // done above
            uint32_t c0[kR], c1[kR];
            if constexpr (SPLIT && kPairInverse) {
                cplx<T> zh[kR], zl[kR];
#pragma unroll
                for (int m = 0; m < kR / 2; m++) {
                    zh[2 * m] = {acc_h[v][m].re.x, acc_h[v][m].im.x};
                    zh[2 * m + 1] = {acc_h[v][m].re.y, acc_h[v][m].im.y};
                    zl[2 * m] = {acc_l[v][m].re.x, acc_l[v][m].im.x};
                    zl[2 * m + 1] = {acc_l[v][m].re.y, acc_l[v][m].im.y};
                }
                F::inverse_pair(zh, zl, xp, s_tw, t, bar_id);
#pragma unroll
                for (int r = 0; r < kR; r++) {  // (c_j - i c_{j+M}) of each limb
                    c0[r] = (round_f32_mod32(zh[r].re) << args.split_shift) + (uint32_t)__float2ll_rn(zl[r].re);
                    c1[r] = (round_f32_mod32(-zh[r].im) << args.split_shift) + (uint32_t)__float2ll_rn(-zl[r].im);
                }
            } else if constexpr (SPLIT) {
                cplx<T> z[kR];
#pragma unroll
                for (int m = 0; m < kR / 2; m++) {
                    z[2 * m] = {acc_h[v][m].re.x, acc_h[v][m].im.x};
                    z[2 * m + 1] = {acc_h[v][m].re.y, acc_h[v][m].im.y};
                }
                F::inverse(z, xp, s_tw, t, bar_id);
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    c0[r] = round_f32_mod32(z[r].re) << args.split_shift;
                    c1[r] = round_f32_mod32(-z[r].im) << args.split_shift;
                }
#pragma unroll
                for (int m = 0; m < kR / 2; m++) {
                    z[2 * m] = {acc_l[v][m].re.x, acc_l[v][m].im.x};
                    z[2 * m + 1] = {acc_l[v][m].re.y, acc_l[v][m].im.y};
                }
                F::inverse(z, xp, s_tw, t, bar_id);
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    c0[r] += (uint32_t)__float2ll_rn(z[r].re);
                    c1[r] += (uint32_t)__float2ll_rn(-z[r].im);
                }
            } else {
                cplx<T> z[kR];
#pragma unroll
                for (int r = 0; r < kR; r++) z[r] = acc_hi[v][r];
                F::inverse(z, xp, s_tw, t, bar_id);
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    c0[r] = round_f64_mod32(z[r].re);  // (c_j - i c_{j+M})
                    c1[r] = round_f64_mod32(-z[r].im);
                }
            }
            uint32_t *poly = s_acc + v * N;
#pragma unroll
            for (int r = 0; r < kR; r++) {
                const int j = t + NT * r;
                put(poly[j], c0[r]);
                put(poly[j + M], c1[r]);
            }
        }
        team_sync(bar_id, NT);
    }

    uint32_t *dst = reinterpret_cast<uint32_t *>(args.acc_out) + (size_t)boot * KP1 * N;
    for (int i = t; i < KP1 * N; i += NT) dst[i] = s_acc[i];
    if constexpr (!PW) {
        // after an abort, drain the copies still in flight before the CTA may exit (bounded waits)
        if (tid == 0) {
            volatile int32_t no_abort = 0;
            for (int r = (issued > D ? issued - D : 0); r < issued; r++)
                wait_bounded(full_bar(r % D), (r / D) & 1, &no_abort, args.timeout_ns, args.err);
        }
    }
}

// ---- launch -------------------------------------------------------------------------------------

template <typename T, int N, int L, bool SPLIT, int G, int D, bool PW = true>
static cudaError_t launch_g(const BrArgs &a, cudaStream_t s) {
    using Lay = BrLayout<T, N, 1, G, D, PW>;
    const size_t smem = Lay::bytes(a.nsteps);
    auto kern = blind_rotate_kernel<T, N, 1, L, SPLIT, G, D, PW>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int grid = (a.boots + G - 1) / G;
    kern<<<grid, Lay::threads, smem, s>>>(a);
    return cudaGetLastError();
}

// External product only (EXT), one sample per CTA, thread 0 streaming the key rows.
template <typename T, int N, int L, bool SPLIT, int D>
static cudaError_t launch_ext(const BrArgs &a, cudaStream_t s) {
    using Lay = BrLayout<T, N, 1, 1, D, false>;
    const size_t smem = Lay::bytes(a.nsteps);
    auto kern = blind_rotate_kernel<T, N, 1, L, SPLIT, 1, D, false, true>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<a.boots, Lay::threads, smem, s>>>(a);
    return cudaGetLastError();
}

int blind_rotate_supported(const tfheb_params &p) {
    return br_variants(p.N, p.l, p.k == 1 ? TFHEB_FP64 : -1, nullptr, nullptr, 0) > 0;
}

// The warp kernel's split form keeps a word's digits in a float's mantissa: parameter sets with wider
// digits (l Bgbit > 23; the reference's sets have 21 and 20) run what was the default before it.
static cudaError_t launch_warp_split3(const BrArgs &a, cudaStream_t s) {
    return 3 * a.Bgbit <= 23 ? launch_warp<true, 3, 8, 6>(a, s) : launch_paired_il3<1024, 3, 7, 12, 1>(a, s);
}
template <int G>
static cudaError_t launch_warp_split2(const BrArgs &a, cudaStream_t s) {
    if (2 * a.Bgbit > 23) return launch_g<float, 1024, 2, true, 7, 4>(a, s);
    if constexpr (G == 8) return launch_warp<true, 2, 8, 8>(a, s);
    else return launch_warp_duo<true, 2, G, 8>(a, s);
}

// Compiled launch variants: (ring degree, gadget length, precision, bootstraps per CTA G, key-ring depth D).
// Every variant's shared memory stays within 227 KB, and every variant gives the same bits.  Tuned variants are
// the autotuner's candidates; small ones (few bootstraps per CTA) serve batches, and last waves of
// batches, with fewer bootstraps per SM than the chosen variant packs.  `us` is the time of a full wave
// (one CTA on each of 148 SMs at 1965 MHz) per step, by which launch_blind_rotate chooses without a tuned key: a
// kernel's time hardly depends on how many of its G bootstraps are there, so a batch is as fast as
// the waves it is cut into.
struct BrVariant {
    int N, l, precision, G, D;
    bool tuned;
    float us;  // measured time per step of a wave of SMs x G bootstraps, us (0: not measured)
    cudaError_t (*launch)(const BrArgs &, cudaStream_t);
    int plan = 0;  // 0: one transform per thread; 1: two per thread, spectra in TMEM (blind_rotate_paired.cu)
    int most_bits = 32;  // the variant serves l Bgbit up to this (a tuned one turns to another kernel by itself beyond)
    int ctas = 1;        // CTAs per bootstrap (a cluster); 2: for waves of at most SMs / 2 bootstraps, `us` of such a one
};
// FP64 with two warps (duo) or two CTAs per bootstrap adds a sum's products in another order than the other kernels.
// Their bits agree where every sum rounds to its exact integer: at l = 2 the sums' error has sigma 0.021 of a unit
// with 11 bits per digit (1/2 is 24 sigma away), 0.041 with 12 and 0.165 with 14; at l = 3 the widest digits, 10 bits, give 0.013
// (N = 2048: 0.018).  l = 2 with wider digits stays with the kernels of one order.
constexpr int kReorderBits = 22;  // l Bgbit at l = 2

static const BrVariant kBrVariants[] = {
    // the split default: two transforms per thread, spectra in TMEM, a 12-half-row key ring; the
    // step's rotated words wait in TMEM, the first two digit pairs' forward transforms run
    // interleaved, and so do both outputs' inverse transforms, output 0's input waiting in TMEM
    // meanwhile; the keys of a digit's first two slot pairs load during the previous digit's
    // multiply-accumulate (30.94 ms per 4096 bootstraps, no spills; on another box 31.50 against
    // 31.33 ms without it, so both stay candidates and the autotuner picks).  The same kernel
    // without that prefetch: 31.27 ms; loading 3 or 4 slot pairs ahead: 31.49 / 31.68 ms; with less interleaving: 31.59 ms (inverse input in registers, 20 B of
    // spills), 31.85 ms (forward only), 32.2 ms (none, rotated words in registers); 36.24 ms for the
    // plan-0 G = 7, D = 6 below.
    {1024, 3, TFHEB_SPLIT_FP32, 7, 12, true, 12.32, launch_paired_il7<1024, 3, 7, 12, 1>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 7, 12, true, 12.24, launch_paired_il3<1024, 3, 7, 12, 1>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 7, 12, true, 12.45, launch_paired_il2<1024, 3, 7, 12, 1>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 7, 12, true, 12.42, launch_paired_il<1024, 3, 7, 12, 1>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 7, 12, true, 12.71, launch_paired<1024, 3, 7, 12, 1, true>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 7, 6, true, 14.32, launch_g<float, 1024, 3, true, 7, 6>},
    {1024, 3, TFHEB_SPLIT_FP32, 7, 4, true, 14.40, launch_g<float, 1024, 3, true, 7, 4>},
    {1024, 3, TFHEB_SPLIT_FP32, 5, 4, true, 10.63, launch_g<float, 1024, 3, true, 5, 4>},
    {1024, 3, TFHEB_SPLIT_FP32, 4, 4, true, 8.94, launch_g<float, 1024, 3, true, 4, 4>},
    // plan 1: D counts half rows (8 KB) here; single or double exchange buffers per team
    {1024, 3, TFHEB_SPLIT_FP32, 7, 8, true, 13.24, launch_paired<1024, 3, 7, 8, 1, true>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 7, 4, true, 13.37, launch_paired<1024, 3, 7, 4, 2, true>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 6, 6, true, 10.50, launch_paired<1024, 3, 6, 6, 2, true>, 1},
    // one warp per bootstrap, exchanges in TMEM (blind_rotate_warp.cu; D counts 16 KB units): the split default
    {1024, 3, TFHEB_SPLIT_FP32, 8, 6, true, 10.94, launch_warp_split3, 1, 23},
    // the paired kernel with 3-6 teams, for waves of that many (3 to 5: for digits the warp kernel does not take)
    {1024, 3, TFHEB_SPLIT_FP32, 6, 12, false, 10.33, launch_paired_il3<1024, 3, 6, 12, 1>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 5, 12, false, 9.57, launch_paired_il3<1024, 3, 5, 12, 1>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 4, 12, false, 7.86, launch_paired_il3<1024, 3, 4, 12, 1>, 1},
    {1024, 3, TFHEB_SPLIT_FP32, 3, 12, false, 7.51, launch_paired_il3<1024, 3, 3, 12, 1>, 1},
    // the warp kernel with two warps per bootstrap: 3.91 ms per wave of four per SM, against 4.95 ms for the paired
    // kernel and 4.97 ms for one warp per bootstrap (FP64: 5.24 ms against 6.22 and 6.6)
    {1024, 3, TFHEB_SPLIT_FP32, 4, 6, false, 6.21, launch_warp_duo<true, 3, 4, 6>, 1, 23},
    {1024, 3, TFHEB_SPLIT_FP32, 3, 6, false, 6.14, launch_warp_duo<true, 3, 3, 6>, 1, 23},
    // few bootstraps (blind_rotate_latency.cu; D counts 48 KB stages): one per CTA, one per two CTAs
    {1024, 3, TFHEB_SPLIT_FP32, 1, 2, false, 2.65, launch_latency<float, 3, 1, 1024>},
    {1024, 3, TFHEB_SPLIT_FP32, 1, 2, false, 1.81, launch_latency<float, 3, 2, 1024>, 0, 32, 2},
    {1024, 3, TFHEB_FP64, 4, 5, true, 9.85, launch_g<double, 1024, 3, false, 4, 5, false>},
    {1024, 3, TFHEB_FP64, 4, 4, true, 10.18, launch_g<double, 1024, 3, false, 4, 4, false>},
    {1024, 3, TFHEB_FP64, 4, 6, true, 11.18, launch_g<double, 1024, 3, false, 4, 6>},
    {1024, 3, TFHEB_FP64, 4, 4, true, 11.04, launch_g<double, 1024, 3, false, 4, 4>},
    {1024, 3, TFHEB_FP64, 3, 4, true, 8.58, launch_g<double, 1024, 3, false, 3, 4>},
    {1024, 3, TFHEB_FP64, 2, 4, true, 5.86, launch_g<double, 1024, 3, false, 2, 4>},
    {1024, 3, TFHEB_FP64, 8, 6, true, 15.75, launch_warp<false, 3, 8, 6>},
    {1024, 3, TFHEB_FP64, 4, 6, false, 8.32, launch_warp_duo<false, 3, 4, 6>},
    {1024, 3, TFHEB_FP64, 3, 6, false, 8.34, launch_warp_duo<false, 3, 3, 6>},
    {1024, 3, TFHEB_FP64, 1, 2, false, 3.34, launch_latency<double, 3, 1, 1024>},
    {1024, 3, TFHEB_FP64, 1, 1, false, 2.35, launch_latency<double, 3, 2, 1024>, 0, 32, 2},
    // the split default at N = 2048: the N = 1024 default's structure with three teams and a 6-deep
    // ring of 16 KB half rows (51.3 ms per 2048 bootstraps; 51.7 ms with output 0's inverse input in
    // registers, 51.9 ms forward interleave only, 53.1 ms no interleave, 54.1 ms rotated words in
    // registers too, 56.5 ms 4 deep, 62.6 ms for the plan-0 G = 2 below)
    {2048, 3, TFHEB_SPLIT_FP32, 3, 6, true, 12.74, launch_paired_il3<2048, 3, 3, 6, 1>, 1},
    {2048, 3, TFHEB_SPLIT_FP32, 3, 6, true, 13.04, launch_paired_il2<2048, 3, 3, 6, 1>, 1},
    {2048, 3, TFHEB_SPLIT_FP32, 3, 6, true, 12.79, launch_paired_il<2048, 3, 3, 6, 1>, 1},
    {2048, 3, TFHEB_SPLIT_FP32, 3, 4, true, 14.11, launch_paired<2048, 3, 3, 4, 1, true>, 1},
    {2048, 3, TFHEB_SPLIT_FP32, 2, 4, true, 11.26, launch_g<float, 2048, 3, true, 2, 4, false>},
    {2048, 3, TFHEB_SPLIT_FP32, 2, 4, true, 11.45, launch_g<float, 2048, 3, true, 2, 4>},
    {2048, 3, TFHEB_SPLIT_FP32, 3, 3, true, 16.81, launch_g<float, 2048, 3, true, 3, 3>},
    {2048, 3, TFHEB_SPLIT_FP32, 2, 3, true, 11.56, launch_g<float, 2048, 3, true, 2, 3>},
    {2048, 3, TFHEB_SPLIT_FP32, 1, 3, false, 7.86, launch_g<float, 2048, 3, true, 1, 3>},
    // one bootstrap on two SMs, D counting 16 KB rows: 3.04 ms per wave of 74, where the entry above takes 5.9 (and two
    // of them 6.09 for 148, against its 6.29)
    {2048, 3, TFHEB_SPLIT_FP32, 1, 5, false, 3.80, launch_latency<float, 3, 2, 2048>, 0, 32, 2},
    {2048, 3, TFHEB_SPLIT_FP32, 2, 4, true, 12.86, launch_paired<2048, 3, 2, 4, 2, false>, 1},
    {2048, 3, TFHEB_SPLIT_FP32, 2, 4, true, 10.56, launch_paired<2048, 3, 2, 4, 2, true>, 1},
    // the warp kernel, D counting 32 KB units: 10.63 ms per wave of 592, against 10.19 ms per 444 for the first entry
    {2048, 3, TFHEB_SPLIT_FP32, 4, 3, true, 13.28, launch_warp_big<true, 3, 4>, 1},
    // FP64: the entry with G = 4 is the default (14.86 ms per wave of 592, against 10.35 ms per 296 for the first)
    {2048, 3, TFHEB_FP64, 2, 3, true, 12.94, launch_g<double, 2048, 3, false, 2, 3, false>},
    {2048, 3, TFHEB_FP64, 2, 3, true, 14.37, launch_g<double, 2048, 3, false, 2, 3>},
    {2048, 3, TFHEB_FP64, 1, 4, true, 7.66, launch_g<double, 2048, 3, false, 1, 4>},
    {2048, 3, TFHEB_FP64, 4, 3, true, 18.58, launch_warp_big<false, 3, 4>},
    {2048, 3, TFHEB_FP64, 1, 3, false, 5.90, launch_latency<double, 3, 2, 2048>, 0, 32, 2},  // 4.72 ms; 5.9 with G = 1 above
    {512, 3, TFHEB_SPLIT_FP32, 8, 4, true, 0, launch_g<float, 512, 3, true, 8, 4>},
    {512, 3, TFHEB_FP64, 8, 4, true, 0, launch_g<double, 512, 3, false, 8, 4>},
    // the 80-bit parameter set (n = 500, l = 2, Bgbit = 10; tfhe_gate_bootstrapping.cpp:23-48)
    {1024, 2, TFHEB_SPLIT_FP32, 7, 4, true, 11.49, launch_g<float, 1024, 2, true, 7, 4>},
    {1024, 2, TFHEB_SPLIT_FP32, 8, 8, true, 8.60, launch_warp_split2<8>, 1, 23},
    {1024, 2, TFHEB_SPLIT_FP32, 4, 8, false, 4.82, launch_warp_split2<4>, 1, 23},
    {1024, 2, TFHEB_SPLIT_FP32, 1, 2, false, 2.33, launch_latency<float, 2, 1, 1024>},
    {1024, 2, TFHEB_SPLIT_FP32, 1, 2, false, 1.67, launch_latency<float, 2, 2, 1024>, 0, 32, 2},
    {1024, 2, TFHEB_FP64, 4, 4, true, 7.90, launch_g<double, 1024, 2, false, 4, 4, false>},
    {1024, 2, TFHEB_FP64, 4, 4, true, 8.38, launch_g<double, 1024, 2, false, 4, 4>},
    {1024, 2, TFHEB_FP64, 8, 8, true, 11.66, launch_warp<false, 2, 8, 8>},
    {1024, 2, TFHEB_FP64, 4, 8, false, 6.35, launch_warp_duo<false, 2, 4, 8>, 0, kReorderBits},
    {1024, 2, TFHEB_FP64, 1, 2, false, 2.74, launch_latency<double, 2, 1, 1024>},
    {1024, 2, TFHEB_FP64, 1, 1, false, 2.04, launch_latency<double, 2, 2, 1024>, 0, kReorderBits, 2},
};

int br_variants(int N, int l, int precision, int *G, int *D, int cap) {
    int n = 0;
    for (const auto &v : kBrVariants)
        if (v.tuned && v.N == N && v.l == l && v.precision == precision) {
            if (n < cap) {
                if (G) G[n] = v.G;
                if (D) D[n] = v.D;
            }
            n++;
        }
    return n;
}

static BrArgs br_args(const tfheb_params &p, const DeviceBsk &bsk, const int32_t *bara, int bara_stride, int boots,
                      int nsteps, int32_t mu, const int32_t *acc_in, int32_t *acc_out, int32_t *d_err,
                      int stall_producer, uint64_t timeout_ns) {
    return BrArgs{bara,       bara_stride, reinterpret_cast<const uint8_t *>(bsk.bsk), reinterpret_cast<const uint8_t *>(bsk.bsk2), bsk.tables, bsk.tables2,
                  acc_in,     acc_out,    boots,       nsteps, mu, p.Bgbit, bsk.split_shift, d_err, timeout_ns, stall_producer, 0};
}

int br_variant_count() { return (int)(sizeof(kBrVariants) / sizeof(kBrVariants[0])); }

void br_variant_info(int g, int *N, int *l, int *precision, int *G, int *D, int *tuned) {
    const BrVariant &v = kBrVariants[g];
    if (N) *N = v.N;
    if (l) *l = v.l;
    if (precision) *precision = v.precision;
    if (G) *G = v.G;
    if (D) *D = v.D;
    if (tuned) *tuned = v.tuned;
}

int br_variant_plan(int g) { return kBrVariants[g].plan; }

int br_variant_ctas(int g) { return kBrVariants[g].ctas; }

int br_variant_plans(int N, int l, int precision, int *plan, int cap) {
    int n = 0;
    for (const auto &v : kBrVariants)
        if (v.tuned && v.N == N && v.l == l && v.precision == precision) {
            if (plan && n < cap) plan[n] = v.plan;
            n++;
        }
    return n;
}

int br_tuned_global(int N, int l, int precision, int tuned) {
    int seen = 0;
    for (int g = 0; g < br_variant_count(); g++) {
        const BrVariant &v = kBrVariants[g];
        if (v.tuned && v.N == N && v.l == l && v.precision == precision && seen++ == tuned) return g;
    }
    return -1;
}

// Whether a variant serves a parameter set.
static bool br_offered(const BrVariant &v, const tfheb_params &p, int precision) {
    return v.N == p.N && v.l == p.l && v.precision == precision && p.l * p.Bgbit <= v.most_bits;
}

bool br_variant_offered(int g, const tfheb_params &p, int precision) { return br_offered(kBrVariants[g], p, precision); }

cudaError_t launch_blind_rotate_exact(const tfheb_params &p, int precision, const DeviceBsk &bsk, const int32_t *bara,
                                      int bara_stride, int boots, int nsteps, int32_t mu, const int32_t *acc_in,
                                      int32_t *acc_out, cudaStream_t s, int32_t *d_err, int stall_producer,
                                      uint64_t timeout_ns, int global_index) {
    if (boots <= 0) return cudaSuccess;
    if (global_index < 0 || global_index >= br_variant_count()) return cudaErrorInvalidValue;
    const BrVariant &v = kBrVariants[global_index];
    if (v.N != p.N || v.l != p.l || v.precision != precision) return cudaErrorInvalidValue;
    if (!v.tuned && !br_offered(v, p, precision)) return cudaErrorInvalidValue;
    return v.launch(br_args(p, bsk, bara, bara_stride, boots, nsteps, mu, acc_in, acc_out, d_err, stall_producer,
                            timeout_ns), s);
}

int br_chosen_global(const tfheb_params &p, int precision, const BrChoice &choice) {
    if (choice.tuned >= 0) return br_tuned_global(p.N, p.l, precision, choice.tuned);
    int best = -1;
    for (int g = 0; g < br_variant_count(); g++) {
        const BrVariant &v = kBrVariants[g];
        if (!v.tuned || !br_offered(v, p, precision)) continue;
        if (best < 0 || (v.us > 0 && v.us * kBrVariants[best].G < kBrVariants[best].us * v.G)) best = g;
    }
    return best;
}

// The variant for one wave with `need` bootstraps per SM (0: at most one per two SMs), given the batch's
// variant `big`: the autotuner's choice, or else the one with the least measured time that has room for them.
static int wave_variant(const tfheb_params &p, int big, int need, const BrChoice &choice) {
    const BrVariant &b = kBrVariants[big];
    if (need >= b.G || need < 0) return big;
    if (need < kSmallNeeds && choice.small[need] != -2)
        return choice.small[need] >= 0 && choice.small[need] < br_variant_count() ? choice.small[need] : big;
    int pick = big;
    for (int g = 0; g < br_variant_count(); g++) {
        const BrVariant &v = kBrVariants[g];
        if (!br_offered(v, p, b.precision) || v.G < need || v.G >= b.G || v.us == 0 || (v.ctas > 1 && need > 0)) continue;
        if (kBrVariants[pick].us == 0 || v.us < kBrVariants[pick].us) pick = g;
    }
    return pick;
}

// What a launch takes beside its waves, us: the launch itself, the CTAs' setup and their last copies (5.0 to 10.4 by
// variant, 6.6 in the middle).  Rotations of one or a few steps are cut into fewer waves for it: 700 split bootstraps of one
// step run as one packed wave (20.7 us), not as 592 + 108 (12.8 + 8.3).
constexpr float kLaunchUs = 7.0f;

// The waves of a rest of `count` bootstraps, fewer than a wave of `big`, for nsteps steps: whole bootstraps per SM, by the
// least sum of measured times.  600 FP64 bootstraps run as 592 + 8 (5.2 + 1.5 ms; 9.9 ms in one wave of eight per SM),
// 296 split ones as two of 148 (1.67 ms each, against 3.68 two per SM).
// Level k = 1 .. need stands for the last k bootstraps per SM of the rest; its last one (k = 1) has `low` bootstraps,
// which two SMs each may serve, in one wave or in two (N = 2048 split, 148: 6.09 against 6.29 ms).
struct RestWaves {
    static constexpr int kMost = 16;  // bootstraps per SM of the largest variant, and one more wave
    int waves = 0;
    struct {
        int variant, count;
    } wave[kMost];
    float us = 0;  // 0: not known
};

static RestWaves rest_waves(const tfheb_params &p, int big, int count, int sms, int nsteps, const BrChoice &choice) {
    RestWaves out;
    const int need = (count + sms - 1) / sms, low = count - (need - 1) * sms, pairs = sms / 2;
    auto cost = [&](int g) { return kBrVariants[g].us > 0 ? kBrVariants[g].us * (float)nsteps + kLaunchUs : 0.f; };
    int variant[RestWaves::kMost], first[RestWaves::kMost];  // first[k]: bootstraps per SM of the next wave, -1: two of `pairs`
    float own[RestWaves::kMost], best[RestWaves::kMost];
    for (int k = 1; k <= need; k++) {
        variant[k] = wave_variant(p, big, k, choice);
        own[k] = cost(variant[k]);
        if (k == 1) {  // by itself the last bootstrap per SM may have two SMs
            const int two = wave_variant(p, big, 0, choice);
            const int g = low <= pairs ? two : variant[1];
            best[1] = cost(g);
            first[1] = 1;
            if (low > pairs && low <= 2 * pairs && cost(two) > 0 && 2 * cost(two) < best[1]) best[1] = 2 * cost(two), first[1] = -1;
            continue;
        }
        best[k] = own[k];
        first[k] = k;
        for (int a = 1; a < k && own[k] > 0; a++)
            if (own[a] > 0 && best[k - a] > 0 && own[a] + best[k - a] < best[k]) best[k] = own[a] + best[k - a], first[k] = a;
    }
    out.us = best[need];
    for (int k = need, left = count; k > 0;) {
        int n = first[k] < k ? first[k] * sms : left, g = variant[first[k] > 0 ? first[k] : 1];
        if (k == 1 && (first[1] < 0 || low <= pairs)) {
            g = wave_variant(p, big, 0, choice);
            if (first[1] < 0) n = pairs;
        }
        out.wave[out.waves++] = {g, n};
        left -= n;
        if (first[k] < 0 && left > 0) out.wave[out.waves++] = {g, left};
        k = first[k] < 0 ? 0 : k - first[k];
    }
    return out;
}

float br_rest_us(const tfheb_params &p, int precision, const BrChoice &choice, int sms, int count) {
    const int big = br_chosen_global(p, precision, choice);
    return big >= 0 && count > 0 ? rest_waves(p, big, count, sms, p.n, choice).us / (float)p.n : 0.f;
}

// Full waves of the chosen variant (SMs x G bootstraps each), then the rest in waves of whatever runs that many
// per CTA fastest: 4096 split bootstraps are 3 waves of 1184 and 544 spread over 4 per CTA (20.7 + 3.9 ms,
// where a fourth packed wave takes 6.9).  A lone bootstrap runs its 630 steps in 1.14 ms on two SMs, 1.67 ms
// on one.
cudaError_t launch_blind_rotate(const tfheb_params &p, int precision, const DeviceBsk &bsk, const int32_t *bara,
                                int bara_stride, int boots, int nsteps, int32_t mu, const int32_t *acc_in,
                                int32_t *acc_out, cudaStream_t s, int32_t *d_err, int stall_producer,
                                uint64_t timeout_ns, const BrChoice &choice, int *launches) {
    if (launches) *launches = 0;
    if (boots <= 0) return cudaSuccess;
    const int big = br_chosen_global(p, precision, choice);
    if (big < 0) return cudaErrorInvalidValue;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        sms = 0;
    auto launch = [&](int g, int first, int count) {
        const size_t at = (size_t)first * (p.k + 1) * p.N;
        if (launches) ++*launches;
        return launch_blind_rotate_exact(p, precision, bsk, bara + (size_t)first * bara_stride, bara_stride, count, nsteps,
                                         mu, acc_in ? acc_in + at : nullptr, acc_out + at, s, d_err, stall_producer,
                                         timeout_ns, g);
    };
    const int wave = sms * kBrVariants[big].G, rest = wave > 0 ? boots % wave : 0, full = boots - rest;
    if (rest == 0) return launch(big, 0, boots);
    const RestWaves tail = rest_waves(p, big, rest, sms, nsteps, choice);
    // after full waves the rest may be one more of them in the same launch
    if (full > 0 && !(tail.us < kBrVariants[big].us * (float)nsteps)) return launch(big, 0, boots);
    cudaError_t e = full > 0 ? launch(big, 0, full) : cudaSuccess;
    for (int w = 0, at = full; w < tail.waves && e == cudaSuccess; at += tail.wave[w++].count)
        e = launch(tail.wave[w].variant, at, tail.wave[w].count);
    return e;
}

struct ExtVariant {
    int N, l, precision;
    cudaError_t (*launch)(const BrArgs &, cudaStream_t);
};
static const ExtVariant kExtVariants[] = {
    {1024, 3, TFHEB_FP64, launch_ext<double, 1024, 3, false, 3>},
    {1024, 3, TFHEB_SPLIT_FP32, launch_ext<float, 1024, 3, true, 3>},
    {1024, 2, TFHEB_FP64, launch_ext<double, 1024, 2, false, 3>},
    {1024, 2, TFHEB_SPLIT_FP32, launch_ext<float, 1024, 2, true, 3>},
    {2048, 3, TFHEB_FP64, launch_ext<double, 2048, 3, false, 3>},
    {2048, 3, TFHEB_SPLIT_FP32, launch_ext<float, 2048, 3, true, 3>},
    {512, 3, TFHEB_FP64, launch_ext<double, 512, 3, false, 3>},
    {512, 3, TFHEB_SPLIT_FP32, launch_ext<float, 512, 3, true, 3>},
};

cudaError_t launch_extern_product(const tfheb_params &p, int precision, const DeviceBsk &bsk, int count,
                                  const int32_t *in, int32_t *out, cudaStream_t s, int32_t *d_err,
                                  uint64_t timeout_ns) {
    if (count <= 0) return cudaSuccess;
    if (!in || !out) return cudaErrorInvalidValue;
    for (const auto &v : kExtVariants)
        if (v.N == p.N && v.l == p.l && v.precision == precision)
            return v.launch(br_args(p, bsk, nullptr, 0, count, 1, 0, in, out, d_err, 0, timeout_ns), s);
    return cudaErrorInvalidValue;
}

}  // namespace tfheb
