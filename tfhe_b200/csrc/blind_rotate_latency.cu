// blind_rotate_latency.cu -- the blind rotation of few bootstraps (tfhe_blindRotate_FFT,
// lwe-bootstrapping-functions-fft.cpp:88-112): one bootstrap per CTA, or per cluster of two CTAs; N = 1024, and
// N = 2048 on two CTAs (split 3.04, FP64 4.72 ms per wave of 74, against 5.9 ms for one team of blind_rotate_kernel).
//
// A batch far below one wave (a single drop-in gate, a few dozen concurrent callers) waits for one bootstrap's
// serial chain of n steps, so a step is spread over as many warps as it has independent work:
//   1. all warps rotate: (X^a - 1) acc + offset into shared memory;
//   2. one team of 64 threads (N = 2048: 128) per gadget digit runs its forward transform; the spectra go to shared memory;
//   3. all warps multiply-accumulate: a thread takes two slots of an output polynomial (both key limbs as a
//      packed pair in the split form) over the digits in order.  Its keys are in registers before the
//      spectra are there: their shared-memory reads (two thirds of the phase's) are off the chain;
//   4. one team per (output polynomial, key limb) runs an inverse transform and adds its rounded words to
//      the accumulator, the two limbs' teams by shared-memory atomics (integer sums mod 2^32, in any order).
// A thread's twiddles stay in registers.  These last two took a wave of 148 from 1.84 to 1.67 ms, one of 74 from 1.23
// to 1.14 (split, l = 3): every phase waits for shared memory.  Slower: the rotation by each team for itself
// instead of once (1.24 against 1.14 ms), warps of their own for the multiply-accumulate (1.35).
// With C = 2 a cluster shares the bootstrap: CTA v keeps polynomial v of the accumulator, transforms its l digits
// and computes output v, so the only thing the two exchange is the spectra, once a step: each team also
// stores its spectrum into the other CTA's shared memory with st.async, which counts the bytes on the other
// CTA's mbarrier (plain remote stores and a releasing arrival cost the sender 900 cycles of a step's 5,000).
// The received half alternates between two buffers: a CTA writes step s + 2's half only after its own
// multiply-accumulate of step s + 1, hence after the other's sending of s + 1, hence after the other's
// multiply-accumulate of step s, which read the same buffer.
// Every accumulator takes the same products in the same order as in blind_rotate_kernel (but for FP64 with C = 2, see
// LatencyLayout::digit), and each transform runs the same operations, so the bits are the same.
//
// The key streams through a ring, issued by a warp of its own: two stages of 48 KB at l = 3 (a step's rows of one
// output with C = 2, three digits' rows of both with C = 1).  N = 2048 has room for five of one digit's row (16 KB;
// FP64: three, and that only with the spectra in the exchange buffers and each team rotating for itself, 5.16 against
// 5.64 ms with two), each given back as soon as its words are in registers (split, after the products instead: 3.70 ms).
// Waits are bounded as in blind_rotate_kernel.  After one that ran out, all threads of the CTA leave the loop at the
// end of the same step or of the next, and the other CTA's next wait for its spectra runs out too.  Each CTA tells the
// other how many steps it ran; after the last barrier (all threads of the cluster), which neither passes while it may
// still send, a CTA whose waits ran out waits for every spectrum that it was sent: a barrier does not order st.async,
// and a late one would land in the shared memory of the SM's next CTA (tests/test_cluster_exchange.py models this).
#include <cuda_runtime.h>
#include <stdint.h>

#include "async_copy.cuh"
#include "br_common.cuh"
#include "fft.cuh"
#include "internal.h"

namespace tfheb {

namespace {

template <typename T, int L, int C, int N_>
struct LatencyLayout {
    static constexpr int N = N_, M = N / 2, NT = M / kR, KP1 = 2, KPL = KP1 * L;
    static constexpr bool split = sizeof(T) == 4, big = N == 2048;
    static_assert(!big || (C == 2 && L == 3), "N = 2048: shared memory for two CTAs only");
    static constexpr bool spec_in_xbufs = big && !split;  // own spectra in the teams' exchange buffers, for room
    static constexpr bool direct = spec_in_xbufs;         // and each team rotates for itself
    static constexpr int polys = KP1 / C;                 // polynomials and outputs of a CTA
    static constexpr int fwd_teams = polys * L;           // NT threads each
    static constexpr int inv_teams = polys * (split ? 2 : 1);
    static constexpr int mac_warps = 8, pairs = 4 * NT / (32 * mac_warps);  // slot pairs of a thread per output
    static constexpr int team_warps = NT / 32;
    static constexpr int warps = team_warps * fwd_teams > mac_warps ? team_warps * fwd_teams : mac_warps;
    // whole warpgroups, for more registers in the consumers': 232 in two of three, 160 in three of four.  With the
    // twiddles in them: FP64, l = 3 2.32 -> 2.11 (C = 1) and 1.55 -> 1.48 ms (C = 2), N = 2048 split 3.42 -> 3.16.
    // Split, l = 3, C = 1 has room without and ran slower (1.77 against 1.67 ms).
    static constexpr bool wide = big || (!split && (C == 2 || L == 3));
    static constexpr int threads = wide ? 32 * (warps + 4) : 32 * (warps + 1), wide_regs = warps == 8 ? 232 : 160;
    static constexpr uint32_t half = (uint32_t)M * 16;    // one output's slots of one key row
    // ring: D stages of stage_digits digits' rows of the CTA's outputs; the first `early` digits' keys of a step go to
    // registers before the spectra have arrived
    static constexpr int stage_digits = big ? 1 : C == 2 ? KPL : L, early = big || C == 1 ? L : KPL;
    static constexpr int D = big ? (split ? 5 : 3) : !split && C == 2 ? 1 : 2;  // FP64 needs the room; a step outlasts a refill
    // stages whose twiddles a thread keeps (a last stage of radix 8 has none; FP64 at N = 2048 has no registers left)
    static constexpr int own_stages = big ? (split ? 3 : 0) : 2;
    static constexpr uint32_t stage = (uint32_t)stage_digits * polys * half;
    static constexpr size_t spec_bytes = sizeof(cplx<T>) * M;  // one digit's spectrum
    static constexpr size_t bars = 0;  // full[D], empty[D], remote[2], abort flag, stop, steps of this CTA and of the other
    static constexpr size_t ring = 128;
    static constexpr size_t tables = ring + D * (size_t)stage;
    static constexpr size_t acc = (tables + tw_table_bytes<T, M>() + 127) / 128 * 128;
    static constexpr size_t acc_bytes = 4 * (size_t)polys * N;
    static constexpr size_t rot = acc + acc_bytes;                                 // this step's rotated words
    static constexpr size_t own_spec = rot + (direct ? 0 : acc_bytes);             // [team] own digits
    // [parity][digit] the other CTA's
    static constexpr size_t spec_in = own_spec + (spec_in_xbufs ? 0 : fwd_teams * spec_bytes);
    static constexpr size_t after_spec = spec_in + (C == 2 ? 2 * L * spec_bytes : 0);
    static constexpr size_t xbuf_bytes = ((size_t)Exch<T, M>::bytes + 15) / 16 * 16;
    static constexpr int xbufs_of = !big && (split || C == 2) ? 2 : 1;  // per team; two save a barrier per exchange
    static constexpr int teams = fwd_teams > inv_teams ? fwd_teams : inv_teams;
    // [inverse team] the products' spectra: a region of their own, or where room is short the exchange buffers of
    // the teams that have no inverse transform, idle from the forward transforms on (FP64 in one CTA), or that of
    // the last team and the rotated words, which the digits were taken from (N = 2048 split), or that of the
    // second team with its digit's spectrum (N = 2048 FP64)
    static constexpr bool sums_in_xbufs = !split && C == 1;
    static constexpr size_t xbufs = after_spec + (sums_in_xbufs || big ? 0 : inv_teams * spec_bytes);
    __host__ __device__ static constexpr size_t sums(int team) {
        return spec_in_xbufs ? xbufs + xbuf_bytes  // each slot's digits are read by the thread that writes its sum
               : sums_in_xbufs ? xbufs + (size_t)(inv_teams + team) * xbuf_bytes
               : !big        ? after_spec + team * spec_bytes
               : team == 0   ? rot
                             : xbufs + (size_t)(teams - 1) * xbufs_of * xbuf_bytes;
    }
    static_assert(!sums_in_xbufs || (teams >= 2 * inv_teams && xbufs_of == 1), "idle exchange buffers");
    static constexpr size_t spec = spec_in_xbufs ? xbufs : own_spec, spec_stride = spec_in_xbufs ? xbuf_bytes : spec_bytes;
    static_assert(!spec_in_xbufs || (xbufs_of == 1 && inv_teams == 1 && xbuf_bytes >= spec_bytes), "spectra in exchange buffers");
    static_assert(!big || !split || (acc_bytes >= spec_bytes && xbuf_bytes >= spec_bytes && teams > inv_teams), "places of the sums");
    static constexpr size_t bytes = xbufs + (size_t)teams * xbufs_of * xbuf_bytes;
    static_assert((2 * D + 2) * 8 + 16 <= ring, "barrier block");
    static_assert(bytes <= 227 * 1024, "shared memory of the variant");
    static_assert(!wide || warps == 8 || warps == 12, "register split");
    static_assert(team_warps * inv_teams <= warps && KPL % stage_digits == 0, "every inverse transform has a team");
    // place (in 16-byte words) of row c of thread t in a spectrum: slots 2c, 2c + 1 (split) or slot c (FP64).  N = 2048: the
    // multiply-accumulate follows the key's second layout (key_transform.cu), whose lanes hold t's 8 apart; the XOR
    // lets it read 8 different bank groups, and keeps 8 consecutive t's, which a store to the other CTA sends
    // as one line, in one line (a place per t in the key's order: 2.1k cycles a step to send FP64's spectra)
    __host__ __device__ static constexpr int place(int c, int t) { return c * NT + (big ? t ^ (t >> 3 & 7) : t); }
    // the step's digit at turn dd.  FP64 sums round to the exact integers in any order (with the digits that this kernel
    // is given: kReorderBits in blind_rotate.cu): there a CTA's own digits go first, before the wait.  The split form's low limb keeps the digits' order.
    __host__ __device__ static constexpr int digit(int dd, int rank) {
        return split || C == 1 || rank == 0 ? dd : (dd + L) % KPL;
    }
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// asynchronous store of 16 bytes to the other CTA, counted on its mbarrier
__device__ __forceinline__ void store_remote(uint32_t addr, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t addr, double2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "d"(v.x), "d"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint32_t bar, uint32_t parity, uint32_t hint_ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
    return ok != 0;
}
// wait_bounded for the other CTA's stores
__device__ __forceinline__ bool wait_bounded_cluster(uint32_t bar, uint32_t parity, volatile int32_t *abort_flag,
                                                     uint64_t timeout_ns, int32_t *err) {
    if (mbar_try_wait_cluster(bar, parity, 0)) return true;
    const uint64_t t0 = global_timer_ns();
    for (;;) {
        if (*abort_flag) return false;
        if (mbar_try_wait_cluster(bar, parity, kWaitSleepNs)) return true;
        if (global_timer_ns() - t0 > timeout_ns) {
            *abort_flag = 1;
            atomicOr(err, 1);
            return false;
        }
    }
}

}  // namespace

template <typename T, int L, int C, int N>
__global__ void __launch_bounds__(LatencyLayout<T, L, C, N>::threads, 1) blind_rotate_latency_kernel(const BrArgs args) {
    using Lay = LatencyLayout<T, L, C, N>;
    constexpr int M = Lay::M, NT = Lay::NT, KP1 = 2, KPL = Lay::KPL, D = Lay::D;
    constexpr bool SPLIT = Lay::split;
    using F = TeamFft<T, M, kR>;
    extern __shared__ __align__(128) unsigned char smem[];

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = C == 2 ? (int)cluster_rank() : 0;
    const int boot = blockIdx.x / C;
    constexpr int consumers = 32 * Lay::warps;
    constexpr int kAllBar = 15;  // teams use 1..KPL
    const uint32_t bar0 = smem_addr(smem + Lay::bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (D + s); };
    auto remote_bar = [&](int s) { return bar0 + 8u * (2 * D + s); };
    volatile int32_t *abort_flag = reinterpret_cast<volatile int32_t *>(smem + Lay::bars + 8 * (2 * D + 2));
    volatile int32_t *stop = abort_flag + 1;  // one thread's reading of the flag, the same for all warps in a step
    volatile int32_t *ran = abort_flag + 2;  // steps that this CTA and the other ran, known after the last barrier

    if (threadIdx.x == 0) {
        for (int s = 0; s < D; s++) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), Lay::mac_warps);
        }
        for (int s = 0; s < 2; s++) mbar_init(remote_bar(s), 1);
        *abort_flag = 0;
        *stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {
        const int4 *g_tab = reinterpret_cast<const int4 *>(args.tables);
        int4 *s_tab = reinterpret_cast<int4 *>(smem + Lay::tables);
        for (int i = threadIdx.x; i < (int)(tw_table_bytes<T, M>() / 16); i += blockDim.x) s_tab[i] = g_tab[i];
    }
    __syncthreads();
    if constexpr (C == 2) cluster_sync();  // both CTAs' barriers exist before either signals

    if (Lay::wide ? warp >= Lay::warps : warp == Lay::warps) {  // ---- the key's stream ----
        if constexpr (Lay::wide) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Lay::wide_regs == 232 ? 40 : 32));
        if (lane == 0 && (!Lay::wide || warp == Lay::warps)) {
            const uint8_t *bsk = SPLIT || Lay::big ? args.bsk2 : args.bsk;
            const int total = args.nsteps * (KPL / Lay::stage_digits);
            int sent = 0;
            if (!args.stall_producer) {
                for (int c = 0; c < total; c++) {
                    const int s = c % D;
                    if (c >= D && !wait_bounded(empty_bar(s), ((c / D) - 1) & 1, abort_flag, args.timeout_ns, args.err))
                        break;
                    mbar_arrive_expect_tx(full_bar(s), Lay::stage);
                    const uint32_t dst = smem_addr(smem + Lay::ring) + (uint32_t)s * Lay::stage;
                    for (int d = 0; d < Lay::stage_digits; d++) {  // C = 2: output `rank` of each row
                        const size_t row = Lay::stage_digits > 1 ? (size_t)c * Lay::stage_digits + d
                                                                 : (size_t)(c - c % KPL + Lay::digit(c % KPL, rank));
                        bulk_copy_g2s(dst + (uint32_t)d * Lay::polys * Lay::half, bsk + (row * KP1 + rank) * Lay::half,
                                      Lay::polys * Lay::half, full_bar(s));
                    }
                    sent = c + 1;
                }
            }
            volatile int32_t no_abort = 0;
            for (int c = (sent > D ? sent - D : 0); c < sent; c++)
                wait_bounded(full_bar(c % D), (c / D) & 1, &no_abort, args.timeout_ns, args.err);
        }
        __syncwarp();
    } else {  // ---- consumer warps ----
        if constexpr (Lay::wide) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Lay::wide_regs));
        // spares the test whether a warp has a transform; at l = 3, N = 1024 the compiler then reads the keys later
        // (1.69 against 1.67 ms), elsewhere it is faster (N = 2048 6.6 against 6.8 ms per 148, l = 2 1.17 against 1.19)
        if constexpr (Lay::big || (SPLIT && L == 2)) __builtin_assume(warp < Lay::warps);
        const int tid = threadIdx.x, team = warp / Lay::team_warps, t = tid & (NT - 1);
        uint32_t *s_acc = reinterpret_cast<uint32_t *>(smem + Lay::acc);
        uint32_t *s_rot = reinterpret_cast<uint32_t *>(smem + Lay::rot);
        const cplx<T> *s_tw = reinterpret_cast<const cplx<T> *>(smem + Lay::tables);
        ExchPair xp{smem + Lay::xbufs + (size_t)(team < Lay::teams ? team : 0) * Lay::xbufs_of * Lay::xbuf_bytes,
                    Lay::xbufs_of == 2 ? (uint32_t)Lay::xbuf_bytes : 0u, 0u};
        const int32_t *my_bara = args.bara + (size_t)boot * args.bara_stride;

        // the CTA's polynomials: rank .. rank + polys - 1
        if (args.acc_in) {
            const uint32_t *src = reinterpret_cast<const uint32_t *>(args.acc_in) + ((size_t)boot * KP1 + rank) * N;
            for (int i = tid; i < Lay::polys * N; i += consumers) s_acc[i] = src[i];
        } else {
            // acc = (0, X^{2N-barb} * [mu,...,mu])  (lwe-bootstrapping-functions-fft.cpp:142-145)
            const int e = 2 * N - my_bara[args.nsteps];
            for (int i = tid; i < Lay::polys * N; i += consumers) {
                const int j = i & (N - 1);
                int src = j - e;
                uint32_t neg = 0;
                while (src < 0) {
                    src += N;
                    neg ^= 1u;
                }
                const bool last = rank + i / N == KP1 - 1;
                s_acc[i] = !last ? 0u : neg ? 0u - (uint32_t)args.mu : (uint32_t)args.mu;
            }
        }
        team_sync(kAllBar, consumers);

        // gadget constants (tgsw.cpp:7-29)
        const int Bgbit = args.Bgbit;
        uint32_t offset = 0;
#pragma unroll
        for (int q = 0; q < L; q++) offset += 1u << (32 - (q + 1) * Bgbit);
        offset *= 1u << (Bgbit - 1);
        const uint32_t maskBg = (1u << Bgbit) - 1u;
        const T digit_bias = DigitConv<T>::base() + T(1 << (Bgbit - 1));
        const int shift = 32 - (team % L + 1) * Bgbit;
        // |low-limb sum| <= (k+1) l N 2^(Bgbit-1) 2^(S-1), doubled for FP32's error
        const bool low_small = (KPL * N <= 8192) && 13 + Bgbit - 1 + args.split_shift - 1 + 1 <= 44;
        // this team's spectrum here and in the other CTA (per parity)
        unsigned char *my_spec = smem + Lay::spec + (size_t)(team < Lay::fwd_teams ? team : 0) * Lay::spec_stride;
        uint32_t far_spec = 0, far_bar = 0;
        if constexpr (C == 2) {
            far_spec = cluster_addr(smem_addr(smem + Lay::spec_in + (size_t)(team < L ? team : 0) * Lay::spec_bytes),
                                    (uint32_t)(rank ^ 1));
            far_bar = cluster_addr(remote_bar(0), (uint32_t)(rank ^ 1));
        }

        const typename F::template OwnTwiddles<Lay::own_stages> own_tw(s_tw, t);

        int a_next = args.nsteps > 0 ? my_bara[0] : 0;
        bool aborted = false;
        int step = 0;
        for (; step < args.nsteps && !aborted; step++) {
            const int ai = a_next & (2 * N - 1);
            if (step + 1 < args.nsteps) a_next = my_bara[step + 1];
            const int parity = step & 1;
            if (warp == Lay::mac_warps - 1 && lane == 0) {
                *stop = *abort_flag;
                if (C == 2) mbar_arrive_expect_tx(remote_bar(parity), (uint32_t)(L * Lay::spec_bytes));
            }

            // 1. (X^a - 1) acc + offset: coefficient e = j - a mod 2N is e mod N, negated when e has the N bit
            auto rotated = [&](int i) {
                const int e = (i & (N - 1)) - ai, src = (i & ~(N - 1)) + (e & (N - 1));
                const uint32_t neg = (uint32_t)((int32_t)((uint32_t)e << (N == 2048 ? 20 : 21)) >> 31), on = offset - neg;
                const uint32_t x = s_acc[src], y = s_acc[i];
                return (x ^ neg) + (on - y);
            };
            if constexpr (!Lay::direct) {
#pragma unroll
                for (int i0 = 0; i0 < Lay::polys * N; i0 += consumers) {
                    const int i = i0 + tid;
                    if (Lay::polys * N % consumers != 0 && i >= Lay::polys * N) break;
                    s_rot[i] = rotated(i);
                }
                team_sync(kAllBar, consumers);
            }

            // 2. digit, forward transform, spectrum out
            if (team < Lay::fwd_teams) {
                const int first = (team / L) * N + t;
                auto word = [&](int j) { return Lay::direct ? rotated(first + j) : s_rot[first + j]; };
                cplx<T> z[kR];
#pragma unroll
                for (int r = 0; r < kR; r++) {
                    const T d0 = DigitConv<T>::conv((word(NT * r) >> shift) & maskBg, digit_bias);
                    const T d1 = DigitConv<T>::conv((word(NT * r + M) >> shift) & maskBg, digit_bias);
                    z[r] = cplx<T>{d0, -d1};  // a_j - i a_{j+M}; the twist is folded into the FFT
                }
                F::forward(z, xp, own_tw, t, 1 + team);
                const uint32_t far = far_spec + (uint32_t)(parity * L * Lay::spec_bytes);
                const uint32_t bar = far_bar + 8u * (uint32_t)parity;
                if constexpr (SPLIT) {
                    // per register pair m {re(2m), im(2m), re(2m+1), im(2m+1)}
#pragma unroll
                    for (int m = 0; m < kR / 2; m++) {
                        const float4 v = make_float4(z[2 * m].re, z[2 * m].im, z[2 * m + 1].re, z[2 * m + 1].im);
                        if constexpr (C == 2) store_remote(far + 16u * (uint32_t)Lay::place(m, t), v, bar);
                        reinterpret_cast<float4 *>(my_spec)[Lay::place(m, t)] = v;
                    }
                } else {
                    // {re, im}
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        const double2 v = make_double2(z[r].re, z[r].im);
                        if constexpr (C == 2) store_remote(far + 16u * (uint32_t)Lay::place(r, t), v, bar);
                        reinterpret_cast<double2 *>(my_spec)[Lay::place(r, t)] = v;
                    }
                }
            }

            // 3. multiply-accumulate: a thread takes slots 2c, 2c + 1 of one virtual thread t (N = 2048: of two, c 2
            //    apart, in the order of the key's second layout).  The keys of the first digits come in while the
            //    spectra are on their way to the other CTA; read before the forward transform they delayed it
            //    (2.17 against 1.97 us per step).
            const int big_t = 64 * (lane >> 3 & 1) + 8 * (lane & 7) + ((warp ^ lane) & 7);  // N = 2048: t's part of its place
            auto pair = [&](int i) { return Lay::big ? (2 * i + (lane >> 4)) * NT + big_t : tid; };  // Lay::place of pair i
            auto key_at = [&](int i, int k) {  // slot 2c + k of pair i in a key row's half
                if constexpr (Lay::big) return i * 512 + k * 256 + tid;
                else return (2 * (tid / NT) + k) * NT + (tid & (NT - 1));
            };
            auto slot_of = [&](int i, int k) {  // Lay::place of slot k of pair i
                return Lay::big ? (4 * i + 2 * (lane >> 4) + k) * NT + big_t : key_at(i, k);
            };
            auto digit = [&](int dd) { return Lay::digit(dd, rank); };
            float4 key[Lay::early][Lay::polys][Lay::pairs][2];  // split {hi.re, lo.re, hi.im, lo.im}; FP64 {re, im}
            auto load_key = [&](int dd) {
                const int c = (step * KPL + dd) / Lay::stage_digits, s = c % D;
                if (dd % Lay::stage_digits == 0)
                    wait_bounded(full_bar(s), (c / D) & 1, abort_flag, args.timeout_ns, args.err);
                const unsigned char *row = smem + Lay::ring + (size_t)s * Lay::stage +
                                           (size_t)(digit(dd) % Lay::stage_digits) * Lay::polys * Lay::half;
#pragma unroll
                for (int v = 0; v < Lay::polys; v++)
#pragma unroll
                    for (int i = 0; i < Lay::pairs; i++)
#pragma unroll
                        for (int e = 0; e < 2; e++)
                            key[dd % Lay::early][v][i][e] = reinterpret_cast<const float4 *>(row + v * Lay::half)[key_at(i, e)];
            };
            auto release = [&](int dd) {  // after the last digit of a stage
                if ((dd + 1) % Lay::stage_digits != 0) return;
                __syncwarp();
                if (lane == 0) mbar_arrive(empty_bar((step * KPL + dd) / Lay::stage_digits % D));
            };
            if (warp < Lay::mac_warps) {
#pragma unroll
                for (int dd = 0; dd < Lay::early; dd++) {
                    load_key(dd);
                    if (Lay::big) release(dd);
                }
            }
            team_sync(kAllBar, consumers);
            if (warp < Lay::mac_warps) {
                auto wait_remote = [&] {
                    if constexpr (C == 2)
                        wait_bounded_cluster(remote_bar(parity), (uint32_t)(step >> 1) & 1u, abort_flag, args.timeout_ns, args.err);
                };
                if constexpr (SPLIT) wait_remote();
                cpair acc2[Lay::polys][Lay::pairs][2];
                cplx<double> accd[Lay::polys][Lay::pairs][2];
#pragma unroll
                for (int v = 0; v < Lay::polys; v++)
#pragma unroll
                    for (int i = 0; i < 2 * Lay::pairs; i++) {
                        acc2[v][i / 2][i % 2] = {{0.f, 0.f}, {0.f, 0.f}};
                        accd[v][i / 2][i % 2] = {0.0, 0.0};
                    }
#pragma unroll
                for (int dd = 0; dd < KPL; dd++) {
                    if (!SPLIT && C == 2 && dd == L) wait_remote();
                    if (dd > 0 && dd % Lay::early == 0)
#pragma unroll
                        for (int e = 0; e < Lay::early; e++) {
                            load_key(dd + e);
                            if (Lay::big) release(dd + e);
                        }
                    const int d = digit(dd), u = d / L, q = d - u * L;
                    const unsigned char *sp = smem + Lay::spec + (size_t)d * Lay::spec_stride;
                    if constexpr (C == 2)
                        sp = u == rank ? smem + Lay::spec + (size_t)q * Lay::spec_stride
                                       : smem + Lay::spec_in + (size_t)(parity * L + q) * Lay::spec_bytes;
#pragma unroll
                    for (int i = 0; i < Lay::pairs; i++) {
                        if constexpr (SPLIT) {
                            const float4 f = reinterpret_cast<const float4 *>(sp)[pair(i)];
#pragma unroll
                            for (int v = 0; v < Lay::polys; v++)
#pragma unroll
                                for (int e = 0; e < 2; e++) {
                                    const float4 k = key[dd % Lay::early][v][i][e];
                                    const float zr = e ? f.z : f.x, zi = e ? f.w : f.y;
                                    const float2 kr = make_float2(k.x, k.y), ki = make_float2(k.z, k.w);
                                    cpair &a = acc2[v][i][e];
                                    a.re = fma2(bc2(zr), kr, a.re);
                                    a.im = fma2(bc2(zr), ki, a.im);
                                    a.re = fma2(bc2(-zi), ki, a.re);
                                    a.im = fma2(bc2(zi), kr, a.im);
                                }
                        } else {
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                const double2 f = reinterpret_cast<const double2 *>(sp)[slot_of(i, e)];
#pragma unroll
                                for (int v = 0; v < Lay::polys; v++) {
                                    const float4 k = key[dd % Lay::early][v][i][e];
                                    const cplx<double> kd{
                                        __hiloint2double(__float_as_int(k.y), __float_as_int(k.x)),
                                        __hiloint2double(__float_as_int(k.w), __float_as_int(k.z))};
                                    cmac(accd[v][i][e], cplx<double>{f.x, f.y}, kd);
                                }
                            }
                        }
                    }
                    if (!Lay::big) release(dd);
                }
                // to the inverse teams: (output v, limb) in the layouts of the spectra
#pragma unroll
                for (int v = 0; v < Lay::polys; v++)
#pragma unroll
                    for (int i = 0; i < Lay::pairs; i++) {
                        if constexpr (SPLIT) {
                            const cpair &a = acc2[v][i][0], &b = acc2[v][i][1];
                            reinterpret_cast<float4 *>(smem + Lay::sums(2 * v))[pair(i)] =
                                make_float4(a.re.x, a.im.x, b.re.x, b.im.x);
                            reinterpret_cast<float4 *>(smem + Lay::sums(2 * v + 1))[pair(i)] =
                                make_float4(a.re.y, a.im.y, b.re.y, b.im.y);
                        } else {
                            double2 *o = reinterpret_cast<double2 *>(smem + Lay::sums(v));
#pragma unroll
                            for (int e = 0; e < 2; e++) o[slot_of(i, e)] = make_double2(accd[v][i][e].re, accd[v][i][e].im);
                        }
                    }
            }
            team_sync(kAllBar, consumers);

            // 4. inverse transforms, exact rounding, accumulate
            if (team < Lay::inv_teams) {
                const unsigned char *in = smem + Lay::sums(team);
                cplx<T> z[kR];
                if constexpr (SPLIT) {
#pragma unroll
                    for (int i = 0; i < kR / 2; i++) {
                        const float4 w = reinterpret_cast<const float4 *>(in)[Lay::place(i, t)];
                        z[2 * i] = {w.x, w.y};
                        z[2 * i + 1] = {w.z, w.w};
                    }
                    F::inverse(z, xp, own_tw, t, 1 + team);
                    // (c_j - i c_{j+M}) of this limb.  Where no low-limb sum can reach 2^44 it is rounded like the
                    // high limb's, on the FMA pipe (the same integer; the conversion instruction takes longer)
                    if ((team & 1) && !low_small) {
                        uint32_t *poly = s_acc + (team >> 1) * N + t;
#pragma unroll
                        for (int r = 0; r < kR; r++) {
                            atomicAdd(poly + NT * r, (uint32_t)__float2ll_rn(z[r].re));
                            atomicAdd(poly + NT * r + M, (uint32_t)__float2ll_rn(-z[r].im));
                        }
                    } else {
                        uint32_t *poly = s_acc + (team >> 1) * N + t;
                        const int weight = team & 1 ? 0 : args.split_shift;
#pragma unroll
                        for (int r = 0; r < kR; r++) {
                            atomicAdd(poly + NT * r, round_f32_mod32(z[r].re) << weight);
                            atomicAdd(poly + NT * r + M, round_f32_mod32(-z[r].im) << weight);
                        }
                    }
                } else {
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        const double2 w = reinterpret_cast<const double2 *>(in)[Lay::place(r, t)];
                        z[r] = {(T)w.x, (T)w.y};
                    }
                    F::inverse(z, xp, own_tw, t, 1 + team);
                    uint32_t *poly = s_acc + team * N + t;
#pragma unroll
                    for (int r = 0; r < kR; r++) {
                        poly[NT * r] += round_f64_mod32(z[r].re);  // (c_j - i c_{j+M})
                        poly[NT * r + M] += round_f64_mod32(-z[r].im);
                    }
                }
            }
            aborted = *stop != 0;
            team_sync(kAllBar, consumers);
        }

        uint32_t *dst = reinterpret_cast<uint32_t *>(args.acc_out) + ((size_t)boot * KP1 + rank) * N;
        for (int i = tid; i < Lay::polys * N; i += consumers) dst[i] = s_acc[i];
        if (C == 2 && tid == 0) {
            ran[0] = step;
            const uint32_t far_ran = cluster_addr(bar0 + 8u * (2 * D + 2) + 12u, (uint32_t)(rank ^ 1));  // its ran[1]
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(far_ran), "r"(step) : "memory");
        }
        __syncwarp();
    }
    if constexpr (C == 2) {
        cluster_sync();  // neither CTA sends any more
        // Without an abort here every step's wait saw its spectra land.  After one at most the last two steps' are
        // unseen, and the other CTA ran at most two steps more, for which nothing expects the bytes yet.
        if (threadIdx.x == 0 && *abort_flag) {
            const int step = ran[0], sent = ran[1];
            volatile int32_t no_abort = 0;
            for (int s = max(0, min(step, sent) - 2); s < sent; s++) {
                if (s >= step) mbar_arrive_expect_tx(remote_bar(s & 1), (uint32_t)(L * Lay::spec_bytes));
                if (!wait_bounded_cluster(remote_bar(s & 1), (uint32_t)(s >> 1) & 1u, &no_abort, args.timeout_ns, args.err)) break;
            }
        }
    }
}

template <typename T, int L, int C, int N>
cudaError_t launch_latency(const BrArgs &a, cudaStream_t s) {
    using Lay = LatencyLayout<T, L, C, N>;
    if ((Lay::split || Lay::big) && !a.bsk2) return cudaErrorInvalidValue;
    auto kern = blind_rotate_latency_kernel<T, L, C, N>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::bytes);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.boots * C));
    cfg.blockDim = dim3(Lay::threads);
    cfg.dynamicSmemBytes = Lay::bytes;
    cfg.stream = s;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = C;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = C > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

template cudaError_t launch_latency<float, 3, 1, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<float, 3, 2, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<double, 3, 1, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<double, 3, 2, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<float, 2, 1, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<float, 2, 2, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<double, 2, 1, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<double, 2, 2, 1024>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<float, 3, 2, 2048>(const BrArgs &, cudaStream_t);
template cudaError_t launch_latency<double, 3, 2, 2048>(const BrArgs &, cudaStream_t);

}  // namespace tfheb
