// qr_apply_rows.cu -- matrix-free Pauli-sum product y = H psi over rows:
// complex128, and complex64 calls of few rows.
//
//     y[r] = sum_g D_g(r) psi[r ^ x_g],
//     D_g(r) = (-1)^popc(r & z0) T_g[pi(r)],  pi(r)_i = popc(r & beta_i) & 1
// (row semantics of qrusty/src/accel.rs:171-210; replaces CSR build plus
// spmat_dot_densevec, :338-370).
//
// What bounds complex128: the FP64 pipe, 2 multiply-adds per SM and cycle on GB300,
// one 64th of the FP32 rate.  Everything else is nearly free beside it, so
// the design spends integer operations and L2 reads to save FP64 ones:
//   * a factor that is real (or imaginary) throughout a warp takes 2
//     multiply-adds per (row, group), not 4: every group of a spin chain and
//     almost every group of a random-letter operator.  The test is on the
//     table values themselves, so it follows coefficient updates, and rows
//     that meet an infinite or NaN amplitude take the full product, whose
//     0 * inf they must keep;
//   * signs are XORs on the sign bit, parities popc;
//   * partner amplitudes come straight from L2 (one coalesced 512-byte read
//     per warp: XOR permutes a warp's 32 rows among themselves), with no
//     tile staged, so a CTA is any set of rows: small problems split over
//     rows and, within a CTA, over groups (slices), until the chip is full.
// The group descriptors (64 bytes) pass through a two-stage shared-memory
// ring filled by 1-D TMA bulk copies, with bounded waits.
//
// Measured (us, before -> after; before: tiles of 4,096 amplitudes staged by
// TMA, 4 multiply-adds per (amplitude, group)):
//   random letters n = 12, 200 terms     848 ->  15   (was one CTA)
//   Jordan-Wigner n = 18, 2,000 terms, 3 states   1,660 -> 820
//   chain n = 22                       1,452 -> 623  (2 * 44 * 2^22
//     multiply-adds: 1.18 of 1.26 TFLOP/s, the FP64 peak at 2,070 MHz)
//   Jordan-Wigner n = 24, 4,000 terms 30,960 -> 29,940  (all factors complex:
//     98 % of the FP64 peak)
//
// complex64 takes the same route while a call has few rows (one tile of 4,096
// amplitudes is one SM's work in the tile kernels), with FP32 products, a
// compensated fold every 16 groups of a slice (Kahan: the error opens the next
// window) and the slices' compensated sums added in order.  Bound by latency
// and, from 2^16 rows on, by L2 reads.  Measured (us, tiles -> rows): random
// letters n = 10, 400 terms 28 -> 12; n = 11, 500 52 -> 15; Jordan-Wigner
// n = 14, 1,400 25 -> 9.4; n = 16, 1,600 33 -> 21; chain n = 16 13 -> 8.5.
#include <type_traits>

#include "qr_common.cuh"
#include "qr_device.cuh"

namespace qr {

namespace {

constexpr int kRowsThreads = 512;
constexpr uint32_t kRowsChunk = 32, kRowsStages = 2;

__device__ __forceinline__ uint32_t par(uint32_t v) { return (uint32_t)__popc(v) & 1u; }
__device__ __forceinline__ uint32_t par(uint64_t v) { return (uint32_t)__popcll(v) & 1u; }

}  // namespace

// parity of m & v for a register index m < 4
__device__ __forceinline__ uint32_t par2(uint32_t m, uint32_t v) {
    return ((m & v) ^ ((m & v) >> 1)) & 1u;
}

// acc += D p over the thread's rows.  re, im: zero iff every D.x (D.y) of the
// thread is +-0; big: the largest exponent field of p.  Warp-uniform branch.
template <int AMPS>
__device__ __forceinline__ void mac_rows(double2 (&acc)[AMPS], const double2 (&D)[AMPS],
                                         const double2 (&p)[AMPS], uint32_t re, uint32_t im,
                                         uint32_t big) {
    const bool fin = big != 0x7ff00000u;
    if (__all_sync(0xffffffffu, fin && im == 0)) {
#pragma unroll
        for (int m = 0; m < AMPS; ++m) {
            acc[m].x = fma(D[m].x, p[m].x, acc[m].x);
            acc[m].y = fma(D[m].x, p[m].y, acc[m].y);
        }
    } else if (__all_sync(0xffffffffu, fin && re == 0)) {
#pragma unroll
        for (int m = 0; m < AMPS; ++m) {
            acc[m].x = fma(-D[m].y, p[m].y, acc[m].x);
            acc[m].y = fma(D[m].y, p[m].x, acc[m].y);
        }
    } else {
#pragma unroll
        for (int m = 0; m < AMPS; ++m) {
            acc[m].x = fma(D[m].x, p[m].x, fma(-D[m].y, p[m].y, acc[m].x));
            acc[m].y = fma(D[m].x, p[m].y, fma(D[m].y, p[m].x, acc[m].y));
        }
    }
}

template <int AMPS>
__device__ __forceinline__ void mac_rows(float2 (&acc)[AMPS], const float2 (&D)[AMPS],
                                         const float2 (&p)[AMPS], uint32_t, uint32_t, uint32_t) {
#pragma unroll
    for (int m = 0; m < AMPS; ++m) {
        acc[m].x = fmaf(D[m].x, p[m].x, fmaf(-D[m].y, p[m].y, acc[m].x));
        acc[m].y = fmaf(D[m].x, p[m].y, fmaf(D[m].y, p[m].x, acc[m].y));
    }
}

// A CTA holds 2^lrw warps of 32 * AMPS consecutive rows (lane + 32 m) and as
// many slices of them as its warps allow: slice s takes groups s, s + slices,
// ... of each descriptor chunk.
template <typename Real, int AMPS, bool WIDE>
__global__ void __launch_bounds__(kRowsThreads) apply_rows(const ApplyArgs a, int lrw) {
    using W = typename std::conditional<WIDE, uint64_t, uint32_t>::type;
    constexpr bool F32 = sizeof(Real) == 4;
    using V = typename std::conditional<F32, float2, double2>::type;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(128) GroupDesc s_desc[kRowsStages][kRowsChunk];
    __shared__ uint64_t full[kRowsStages];
    // a slice's sums: double2, or (sum, error) of the compensated float2
    using P = typename std::conditional<F32, float4, double2>::type;
    P *part = reinterpret_cast<P *>(smem_raw);
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const uint32_t rw = warp & ((1u << lrw) - 1u), sl = warp >> lrw,
                   nsl = (blockDim.x >> 5) >> lrw;
    const uint32_t cta_rows = (32u * AMPS) << lrw;
    const uint64_t per_state = (a.N + cta_rows - 1) / cta_rows;
    const uint64_t st = blockIdx.x / per_state;
    const uint64_t r0 = (blockIdx.x - st * per_state) * cta_rows + (uint64_t)rw * (32u * AMPS) + lane;
    const V *psi = static_cast<const V *>(a.psi) + st * a.N;
    const V *tables = static_cast<const V *>(a.tables);
    const double2 *fat_c = static_cast<const double2 *>(a.fat_c);
    const V *diag = static_cast<const V *>(a.diag);
    const W nmask = (W)(a.N - 1);
    const uint32_t nchunk = (a.ngroups + kRowsChunk - 1) / kRowsChunk;

    uint32_t issued[kRowsStages] = {};  // copies into each stage (thread 0)
    auto issue = [&](uint32_t c) {
        if (blockIdx.x == 0 && (int64_t)c == a.withhold) return;  // test hook: never issued
        const uint32_t left = a.ngroups - c * kRowsChunk;
        const uint32_t bytes =
            (left < kRowsChunk ? left : kRowsChunk) * (uint32_t)sizeof(GroupDesc);
        ++issued[c % kRowsStages];
        mbar_expect_tx(&full[c % kRowsStages], bytes);
        bulk_g2s(s_desc[c % kRowsStages], a.groups + (size_t)c * kRowsChunk, bytes,
                 &full[c % kRowsStages]);
    };
    if (t == 0) {
        for (uint32_t s = 0; s < kRowsStages; ++s) mbar_init(&full[s], 1);
        mbar_fence_init();
        for (uint32_t c = 0; c < kRowsStages && c < nchunk; ++c) issue(c);
    }

    W row[AMPS];
    V acc[AMPS], hi[AMPS];  // hi: complex64 only
#pragma unroll
    for (int m = 0; m < AMPS; ++m) {
        row[m] = (W)(r0 + 32u * m) & nmask;  // n < 7: the spare lanes repeat rows
        acc[m].x = acc[m].y = hi[m].x = hi[m].y = Real(0);
    }
    if (diag != nullptr && sl == 0) {
        V p[AMPS], D[AMPS];
        uint32_t re = 0, im = 0, big = 0;
#pragma unroll
        for (int m = 0; m < AMPS; ++m) {
            D[m] = diag[row[m]];
            p[m] = psi[row[m]];
            if constexpr (!F32) {
                re |= mag_bits(D[m].x);
                im |= mag_bits(D[m].y);
                big = max(big, max(exp_bits(p[m].x), exp_bits(p[m].y)));
            }
        }
        mac_rows<AMPS>(acc, D, p, re, im, big);
    }
    __syncthreads();
    bool ok = true;
    uint32_t win = 0;
    for (uint32_t c = 0; c < nchunk; ++c) {
        const uint32_t s = c % kRowsStages;
        // an expired wait (the warp's vote) skips the chunk and ends the CTA
        const bool late = __any_sync(
            0xffffffffu, !mbar_wait_bounded(&full[s], (c / kRowsStages) & 1u, a.wait_ns));
        const uint32_t left = a.ngroups - c * kRowsChunk;
        const uint32_t ng = late ? 0u : (left < kRowsChunk ? left : kRowsChunk);
#pragma unroll 2
        for (uint32_t g = sl; g < ng; g += nsl) {
            const GroupDesc &gd = s_desc[s][g];
            const W x = (W)gd.x, z0 = (W)gd.z0;
            const uint32_t d = gd.d, off = gd.off;
            V p[AMPS], D[AMPS];
#pragma unroll
            for (int m = 0; m < AMPS; ++m) p[m] = __ldg(psi + (row[m] ^ x));
            const uint32_t s0 = par(row[0] & z0), zb = (uint32_t)(z0 >> 5);
            uint32_t re = 0, im = 0, big = 0;
            if (d != kFat) {
                uint32_t u = 0, any = 0;
                for (uint32_t i = 0; i < d; ++i) {
                    const W b = (W)gd.beta[i];
                    u |= par(row[0] & b) << i;
                    any |= (uint32_t)(b >> 5);
                }
                if ((any & (AMPS - 1)) == 0) {
                    const V e = __ldg(tables + off + u);
                    if constexpr (!F32) {
                        re = mag_bits(e.x);
                        im = mag_bits(e.y);
                    }
#pragma unroll
                    for (int m = 0; m < AMPS; ++m) {
                        const uint32_t sg = s0 ^ par2(m, zb);
                        D[m].x = flip(e.x, sg);
                        D[m].y = flip(e.y, sg);
                    }
                } else {
#pragma unroll
                    for (int m = 0; m < AMPS; ++m) {
                        uint32_t um = u;
                        for (uint32_t i = 0; i < d; ++i)
                            um ^= par2(m, (uint32_t)((W)gd.beta[i] >> 5)) << i;
                        const V e = __ldg(tables + off + um);
                        const uint32_t sg = s0 ^ par2(m, zb);
                        D[m].x = flip(e.x, sg);
                        D[m].y = flip(e.y, sg);
                        if constexpr (!F32) {
                            re |= mag_bits(e.x);
                            im |= mag_bits(e.y);
                        }
                    }
                }
            } else if constexpr (!F32) {  // complex64 plans have no rank above 4
                const uint32_t cnt = gd.cnt;
#pragma unroll
                for (int m = 0; m < AMPS; ++m) D[m] = make_double2(0.0, 0.0);
                for (uint32_t k = 0; k < cnt; ++k) {
                    const W zk = (W)a.fat_z[off + k];
                    const double2 ck = fat_c[off + k];
#pragma unroll
                    for (int m = 0; m < AMPS; ++m) {
                        const uint32_t sg = par(row[m] & zk);
                        D[m].x += flip(ck.x, sg);
                        D[m].y += flip(ck.y, sg);
                    }
                }
#pragma unroll
                for (int m = 0; m < AMPS; ++m) {
                    re |= mag_bits(D[m].x);
                    im |= mag_bits(D[m].y);
                }
            }
            if constexpr (!F32) {
#pragma unroll
                for (int m = 0; m < AMPS; ++m)
                    big = max(big, max(exp_bits(p[m].x), exp_bits(p[m].y)));
            }
            mac_rows<AMPS>(acc, D, p, re, im, big);
        }
        if constexpr (F32) {  // fold every 16 groups of the slice or more
            win += ng;
            if (win >= 16u * nsl) {
                win = 0;
#pragma unroll
                for (int m = 0; m < AMPS; ++m) acc[m] = two_sum_carry2(hi[m], acc[m]);
            }
        }
        // every warp is done with stage s
        if (__syncthreads_or(late)) {
            ok = false;
            break;
        }
        if (t == 0 && c + kRowsStages < nchunk) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(c + kRowsStages);
        }
    }
    if (!ok) {
        // no copy is in flight when the CTA exits: wait (2 s at most) for the
        // last one issued into each stage
        if (t == 0) {
            atomicExch(a.err, kErrMbarTimeout);
            for (uint32_t s = 0; s < kRowsStages; ++s)
                if (issued[s] != 0) mbar_wait_bounded(&full[s], (issued[s] - 1u) & 1u, kWaitLimitNs);
        }
        return;
    }
    if constexpr (F32) {
#pragma unroll
        for (int m = 0; m < AMPS; ++m) acc[m] = two_sum_carry2(hi[m], acc[m]);
    }
    if (nsl > 1) {
        // slice s > 0 hands its sums to slice 0, added there in slice order
        const uint32_t at = rw * (32u * AMPS) + lane;
        if (sl > 0) {
#pragma unroll
            for (int m = 0; m < AMPS; ++m) {
                P &q = part[(size_t)(sl - 1) * cta_rows + at + 32u * m];
                if constexpr (F32) q = make_float4(hi[m].x, hi[m].y, acc[m].x, acc[m].y);
                else q = acc[m];
            }
        }
        __syncthreads();
        if (sl > 0) return;
        for (uint32_t s = 0; s + 1 < nsl; ++s) {
#pragma unroll
            for (int m = 0; m < AMPS; ++m) {
                const P q = part[(size_t)s * cta_rows + at + 32u * m];
                if constexpr (F32) {
                    const float2 e = two_sum_carry2(hi[m], make_float2(q.x, q.y));
                    acc[m] = __fadd2_rn(acc[m], __fadd2_rn(e, make_float2(q.z, q.w)));
                } else {
                    acc[m].x += q.x;
                    acc[m].y += q.y;
                }
            }
        }
    }
    V *y = static_cast<V *>(a.y) + st * a.N;
    const V *v = a.v ? static_cast<const V *>(a.v) + st * a.N : nullptr;
#pragma unroll
    for (int m = 0; m < AMPS; ++m) {
        const uint64_t r = r0 + 32u * m;
        if (r >= a.N) continue;
        V o = acc[m];
        if constexpr (F32) {
            o = __fadd2_rn(hi[m], o);
            if (v) o = cx_axpby((float)a.ar, (float)a.ai, o, (float)a.br, (float)a.bi, v[r]);
        } else {
            if (v) o = cx_axpby(a.ar, a.ai, o, a.br, a.bi, v[r]);
        }
        y[r] = o;
    }
}

template <typename Real>
static cudaError_t launch_split(const ApplyArgs &a, int amps, int nsl, cudaStream_t st) {
    while (amps > 1 && 32ull * amps > a.N) amps >>= 1;
    const int lrw = nsl == 1 ? 2 : 0;
    const int warps = nsl << lrw;
    const uint64_t cta_rows = (32ull * amps) << lrw;
    const uint64_t per_state = (a.N + cta_rows - 1) / cta_rows;
    const uint64_t grid = per_state * (uint64_t)a.nstates;
    if (grid > 0x7fffffffull) return cudaErrorInvalidValue;
    const size_t smem = (size_t)(nsl - 1) * cta_rows * 16;
    const bool wide = a.n > 32 || a.wide;
    auto kern = amps == 4   ? (wide ? apply_rows<Real, 4, true> : apply_rows<Real, 4, false>)
                : amps == 2 ? (wide ? apply_rows<Real, 2, true> : apply_rows<Real, 2, false>)
                            : (wide ? apply_rows<Real, 1, true> : apply_rows<Real, 1, false>);
    kern<<<(unsigned)grid, warps * 32, smem, st>>>(a, lrw);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_rows(int dtype, const ApplyArgs &a, uint64_t call_rows, cudaStream_t st) {
    if (dtype == 0) {
        // Slices by the rows of the call: 16 warps share a row while the rows
        // give too few warps to hide the L2 reads, none from 2^21 on, where the
        // additions of the slices' sums are FP64 work like any other (us with
        // 16 / 8 / 4 / 2 / 1 slices: 300 random strings 2^13 rows 25 / 25 / 37 /
        // 60 / 107, 2^15 63 / 45 / 54 / 80 / 146, 2^17 209 / 149 / 130 / 135 /
        // 177, 2^20 1,577 / 1,051 / 915 / 889 / 923; chain n = 13 2^19 rows 218 /
        // 96 / 64 / 58 / 54, 2^21 856 / 361 / 234 / 199 / 189).  Without slices
        // a CTA holds 512 rows of a state, so smaller states keep two.  Rows
        // per thread by the number of rows of
        // all states: four share the parity and table work (1 or 2 are bound
        // by the instruction issue instead of FP64: Jordan-Wigner n = 24,
        // 49.9 ms against 29.9), so they are given up only below 2^14 rows,
        // where fewer than 128 CTAs would be left.
        const uint64_t rows = a.N * (uint64_t)a.nstates;
        const int nsl = call_rows <= (1ull << 14)   ? 16
                        : call_rows <= (1ull << 15) ? 8
                        : call_rows < (1ull << 20)  ? 4
                        : call_rows < (1ull << 21) || a.N < 512 ? 2 : 1;
        return launch_split<double>(a, rows < (1ull << 13) ? 1 : (rows < (1ull << 14) ? 2 : 4), nsl,
                                    st);
    }
    // complex64: slices and rows per thread by the rows of the call (best of
    // 1, 2, 4 rows x 1 ... 16 slices on random, chain and Jordan-Wigner
    // operators of 8-18 qubits, one and four states)
    if (call_rows <= (1ull << 13)) return launch_split<float>(a, 1, 16, st);
    if (call_rows <= (1ull << 14)) return launch_split<float>(a, 2, 16, st);
    if (call_rows <= (1ull << 15)) return launch_split<float>(a, 2, 8, st);
    if (call_rows <= (1ull << 16)) return launch_split<float>(a, 2, 4, st);
    return launch_split<float>(a, 4, 4, st);
}

}  // namespace qr
