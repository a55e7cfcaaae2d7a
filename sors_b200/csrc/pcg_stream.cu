// pcg_stream.cu -- a whole two-level PCG solve in one launch for meshes whose
// matrix does not fit on the SMs: the matrix streams through shared memory.
//
// Between the meshes whose matrix the SMs hold and those whose matrix HBM bounds,
// an iteration as separate launches (p, SpMV, update with restriction, coarse
// solve with prolongation) is bound by launches, cold starts and reductions, the
// matrix (52 MB of FP32 at 100,000 nodes) staying in L2.  A step, launches ->
// here: 77,841 FP32 nodes 11.2 -> 6.7 ms, 169,781 17.5 -> 12.9, FP64 24.1 -> 16.5,
// 291,870 25.3 -> 19.8; at 522,801 nodes, where HBM bounds both, 36.7 and 37.1.
// What bounds it now: the shared-memory wavefronts of the product (a block's nine
// values 2-way conflicting, p gathered: 30 per 32 blocks) and the sums' round trips.
//
// Here one block per SM owns a contiguous range of rows for the whole solve:
//   matrix   each warp takes every 16th group of eight rows (four lanes a row);
//            the group's CSR blocks are contiguous, so one thread fetches them
//            (and their column indices, and the rows' offsets) with bulk copies
//            (TMA) into the warp's ring of up to four groups, and the warp
//            multiplies from shared memory.  No load instruction of the product goes to global
//            memory; nothing waits for another warp.
//   p        the range's own and border columns in shared memory (p = z + beta p
//            formed by every range that reads it, from the same z)
//   x r z q  and the inverse diagonal blocks in global memory, component by
//            component (coalesced), touched once per iteration; with the matrix
//            read evict-first they stay in L2.
//   sums     p.q and r.z through mailboxes, as in the grid form of
//            pcg_resident.cu; the coarse unknowns' P^T q through a board that
//            every block posts to and reads whole (tagged words: no fence).
//   coarse   A aggregates per block; every block keeps y = P^T r (FP64) and forms
//            its own 6 A rows of Ac^-1 y.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fem_math.cuh"
#include "pcg_exchange.cuh"
#include "sors_internal.h"

namespace sors {

namespace {

constexpr int kMaxA = kStreamMaxAgg, kLPR = kStreamLanes;
constexpr int kGR = 32 / kLPR;  // rows per group
constexpr u64 kDrainNs = 1000000000ull;  // limit of the wait for a block's own copies

struct SOff {
    int zc, part, y, a, sp, srp, halo, bar, ring;
};
template <typename VT>
__host__ __device__ inline SOff soffsets(const StreamPlan& pl) {
    auto up = [](int b) { return (b + 15) & ~15; };
    SOff o;
    int at = kScratch;
    o.zc = at; at = up(at + 6 * kMaxA * 2 * 8);
    o.part = at; at = up(at + kMaxA * kWarps * 6 * 8);
    o.y = at; at = up(at + pl.ld * 8);
    o.a = at; at = up(at + (pl.a_shared ? 6 * pl.A * pl.ld * (int)sizeof(VT) : 0));
    o.sp = at; at = up(at + pl.max_cols * Lay<VT>::P * (int)sizeof(VT));
    o.srp = at; at = up(at + (pl.max_rows + 1) * 4);
    o.halo = at; at = up(at + pl.max_halo * 4);
    o.bar = at; at = up(at + kWarps * pl.depth * 8);
    o.ring = at;
    return o;
}

__device__ __forceinline__ unsigned sptr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Waits for phase `parity` of the barrier; false after the limit (a try_wait that
// fails has waited for some time itself).
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity, u64 limit_ns) {
    u64 t0 = 0;
    for (;;) {
        unsigned got;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(got)
            : "r"(bar), "r"(parity)
            : "memory");
        if (got) return true;
        const u64 t = clock_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 >= limit_ns) return false;
    }
}

__device__ __forceinline__ void bulk(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

template <typename VT>
__global__ void __launch_bounds__(kT, 1) k_pcg_stream(StreamPlan pl, StreamArgs<VT> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int P = Lay<VT>::P, Z = Lay<VT>::Z;
    constexpr int BB = 9 * (int)sizeof(VT);  // bytes of a matrix block
    double eta2, abs_tol2;
    if (!solve_tolerances(a, eta2, abs_tol2)) return;
    Scratch* sh = reinterpret_cast<Scratch*>(smem);
    const SOff o = soffsets<VT>(pl);
    double* zc = reinterpret_cast<double*>(smem + o.zc);      // 6 A rows, two partial sums each
    double* part = reinterpret_cast<double*>(smem + o.part);  // [aggregate][warp][6]
    double* y = reinterpret_cast<double*>(smem + o.y);
    VT* sa = reinterpret_cast<VT*>(smem + o.a);
    VT* sp = reinterpret_cast<VT*>(smem + o.sp);
    int* srp = reinterpret_cast<int*>(smem + o.srp);
    const int t = threadIdx.x, w = t >> 5, lane = t & 31, G = gridDim.x, me = blockIdx.x;
    const int r0 = pl.row0[me], nr = pl.row0[me + 1] - r0;
    const int h0 = pl.halo_ptr[me], nh = pl.halo_ptr[me + 1] - h0;
    int* halo = reinterpret_cast<int*>(smem + o.halo);
    const long long N = pl.N;
    const int nc = pl.nc, nagg = pl.A * G, na = 6 * pl.A;
    const int L = pl.agg_rows[me];  // rows per aggregate of this range, a multiple of 32
    const int b0 = a.row_ptr[r0];
    unsigned epoch = *(volatile const unsigned*)a.epoch;
    unsigned char* ring = smem + o.ring + (size_t)w * pl.depth * pl.group_bytes;
    const unsigned bars = sptr(smem + o.bar) + 8u * (unsigned)(w * pl.depth);
    if (t == 0) sh->abort = sh->late = 0;
    if (lane == 0)
        for (int k = 0; k < pl.depth; k++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + 8u * k) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    // bit k: the phase that slot k's next wait expects; a copy into it has not been waited for
    unsigned ring_phase = 0, ring_busy = 0;
    unsigned long long policy = 0;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
    for (int i = t; i <= nr; i += kT) srp[i] = a.row_ptr[r0 + i] - b0;
    for (int k = t; k < nh; k += kT) halo[k] = pl.halo[h0 + k];
    for (int k = t; k < (nr + nh) * P; k += kT) sp[k] = VT(0);
    if (t < kWarps)
#pragma unroll
        for (int k = 0; k < 8; k++) sh->part[t][k] = 0.0;
    for (int j = nc + t; j < pl.ld; j += kT) y[j] = 0.0;
    const VT* Arow = a.Ainv + (size_t)me * na * pl.ld;
    if (pl.a_shared)
        for (int k = t; k < na * pl.ld; k += kT) sa[k] = __ldg(Arow + k);

    VT *xs = a.ws, *rs = a.ws + 3 * N, *zs = a.ws + 6 * N, *qs = a.ws + 9 * N, *Ms = a.ws + 12 * N;
    // per row: inverse diagonal block (as k_block_jacobi; symmetric, six values), x, r, offset with flags
    for (int i = t; i < nr; i += kT) {
        const long long row = r0 + i;
        double d[9], c[9];
        const VT* hd = a.H + 9 * (size_t)a.diag_slot[row];
#pragma unroll
        for (int k = 0; k < 9; k++) d[k] = (double)hd[k];
        d[1] = d[3]; d[2] = d[6]; d[5] = d[7];
        cof3(d, c);
        const double det = d[0] * c[0] + d[1] * c[1] + d[2] * c[2];
        const bool inv = det != 0.0 && det == det;
        const double id = 1.0 / det;
        constexpr int S[6] = {0, 3, 6, 4, 7, 8};  // rows' entries 00 10 20 11 21 22
#pragma unroll
        for (int k = 0; k < 6; k++)
            Ms[k * N + row] = inv ? (VT)(c[S[k]] * id) : (VT)((k == 0 || k == 3 || k == 5) ? 1.0 : 0.0);
        const unsigned pf = a.pflag ? a.pflag[row] : 0u;
        VT r[3];
#pragma unroll
        for (int k = 0; k < 3; k++) r[k] = (VT)(-a.g[3 * row + k]);
        project<VT>(pf, a.pn + row, r);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            rs[k * N + row] = r[k];
            xs[k * N + row] = VT(0);
        }
        float4 v = pl.off[row];
        v.w = __uint_as_float((unsigned)a.fixed[row] | pf << 8 | (pl.border[row] ? 0x10000u : 0u));
        a.woff[row] = v;
    }
    // the bulk copies read woff
    asm volatile("fence.proxy.async;" ::: "memory");
    __syncthreads();

    // adds a warp's six sums for the range's aggregate ag (called as ag ascends)
    auto flush = [&](int ag, double (&c)[6], int from) {
#pragma unroll
        for (int m = 0; m < 6; m++) {
            for (int s = 16; s >= from; s >>= 1) c[m] += __shfl_xor_sync(0xffffffffu, c[m], s);
            if (lane == 0) part[(ag * kWarps + w) * 6 + m] = c[m];
            c[m] = 0.0;
        }
    };
    // posts the range's aggregates' six values (sums over the warps) on the board
    auto post = [&](u64* board, unsigned tag) {
        __syncthreads();
        for (int v = w; v < na; v += kWarps) {
            const int ag = v / 6, m = v - 6 * (v / 6);
            double x = part[(ag * kWarps + (lane & (kWarps - 1))) * 6 + m];
#pragma unroll
            for (int s = kWarps / 2; s > 0; s >>= 1) x += __shfl_xor_sync(0xffffffffu, x, s);
            if (lane == 0) {
                u64 lo, hi;
                split(x, tag, lo, hi);
                st_words(board + 2 * (size_t)(m * nagg + me * pl.A + ag), lo, hi);
            }
        }
    };
    auto clear_part = [&]() {
        for (int k = t; k < kMaxA * kWarps * 6; k += kT) part[k] = 0.0;
    };
    // y from the board (fresh: the posted values, else y - al posted), then the range's
    // rows of Ac^-1 y
    auto coarse = [&](const u64* board, unsigned tag, bool fresh, double al) {
        for (int j = t; j < nc; j += kT) {
            u64 lo, hi;
            Patience wait(a.wait_ns);
            bool here;
            do {
                ld_words(board + 2 * (size_t)j, lo, hi);
                here = has(lo, tag) && has(hi, tag);
            } while (!here && wait.more(a.wait_ns));
            if (!here) sh->late = 1;
            const double v = join(lo, hi);
            y[j] = fresh ? v : y[j] - al * v;
        }
        __syncwarp();
        __syncthreads();
        constexpr int W = 16 / (int)sizeof(VT);
        for (int task = w; task < 2 * na; task += kWarps) {
            const int m = task >> 1;
            double z = 0.0;
            const VT* A = (pl.a_shared ? sa : Arow) + (size_t)m * pl.ld;
            // y is padded with zeros to the leading dimension
#pragma unroll 8
            for (int j = ((task & 1) * 32 + lane) * W; j < pl.ld; j += 64 * W) {
                if constexpr (sizeof(VT) == 4) {
                    const float4 q = *reinterpret_cast<const float4*>(A + j);
                    const double2 y0 = *reinterpret_cast<const double2*>(y + j),
                                  y1 = *reinterpret_cast<const double2*>(y + j + 2);
                    z += (double)q.x * y0.x + (double)q.y * y0.y + (double)q.z * y1.x + (double)q.w * y1.y;
                } else {
                    const double2 q = *reinterpret_cast<const double2*>(A + j);
                    const double2 y0 = *reinterpret_cast<const double2*>(y + j);
                    z += q.x * y0.x + q.y * y0.y;
                }
            }
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) z += __shfl_xor_sync(0xffffffffu, z, s);
            if (lane == 0) zc[task] = z;
        }
        __syncthreads();
    };
    const size_t board_words = 2 * (size_t)nc;
    auto renew = [&]() {
        clear_part();
        __syncthreads();
        double c[6] = {0, 0, 0, 0, 0, 0};
        int ag = 0;
        for (int i = t; (i & ~31) < nr; i += kT) {
            const int an = (i & ~31) / L;
            if (an != ag) { flush(ag, c, 1); ag = an; }
            if (i < nr) {
                const long long row = r0 + i;
                const VT r[3] = {rs[row], rs[N + row], rs[2 * N + row]};
                const float4 d = a.woff[row];
                restrict_node<VT>(d, __float_as_uint(d.w), r, c);
            }
        }
        flush(ag, c, 1);
        ++epoch;
        post(a.board + 2 * board_words, epoch);
        coarse(a.board + 2 * board_words, epoch, true, 0.0);
        return sh->late == 0;  // set again only beyond the next exchange
    };
    // x += ax p, r -= ar q, z = M^-1 r + P zc published with the coming site-1 sum; r.z, r.r
    auto update = [&](VT ax, VT ar, bool with_z) {
        double acc[2] = {0.0, 0.0};
        constexpr int U = sizeof(VT) == 4 ? 2 : 1;  // rows a thread has in flight: their loads go before any store
        for (int ib = t; ib < nr; ib += U * kT) {
            VT r[U][3], q[U][3], x[U][3], M[U][6];
            float4 d[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const long long row = r0 + min(ib + u * kT, nr - 1);
                d[u] = a.woff[row];
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    r[u][k] = rs[k * N + row];
                    q[u][k] = qs[k * N + row];
                    x[u][k] = xs[k * N + row];
                }
#pragma unroll
                for (int k = 0; k < 6; k++) M[u][k] = Ms[k * N + row];
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int i = ib + u * kT;
                if (i >= nr) continue;
                const long long row = r0 + i;
                const unsigned f = __float_as_uint(d[u].w);
                if (ar != VT(0)) {
                    project<VT>((f >> 8) & 0xffu, a.pn + row, q[u]);
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        r[u][k] -= ar * q[u][k];
                        rs[k * N + row] = r[u][k];
                    }
                }
                if (ax != VT(0)) {
#pragma unroll
                    for (int k = 0; k < 3; k++) xs[k * N + row] = x[u][k] + ax * sp[P * i + k];
                }
                if (!with_z) continue;
                VT z[3] = {M[u][0] * r[u][0] + M[u][1] * r[u][1] + M[u][2] * r[u][2],
                           M[u][1] * r[u][0] + M[u][3] * r[u][1] + M[u][4] * r[u][2],
                           M[u][2] * r[u][0] + M[u][4] * r[u][1] + M[u][5] * r[u][2]};
                const double* cz = zc + 12 * (i / L);
                VT c[6];
#pragma unroll
                for (int m = 0; m < 6; m++) c[m] = (VT)(cz[2 * m] + cz[2 * m + 1]);
                const VT ox = (VT)d[u].x, oy = (VT)d[u].y, oz = (VT)d[u].z;
                if (!(f & 1u)) z[0] += c[0] + c[4] * oz - c[5] * oy;
                if (!(f & 2u)) z[1] += c[1] - c[3] * oz + c[5] * ox;
                if (!(f & 4u)) z[2] += c[2] + c[3] * oy - c[4] * ox;
                project<VT>((f >> 8) & 0xffu, a.pn + row, z);
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    zs[k * N + row] = z[k];
                    acc[0] += (double)r[u][k] * (double)z[k];
                    acc[1] += (double)r[u][k] * (double)r[u][k];
                }
                if (f & 0x10000u) {
                    u64 wd[Z];
                    if constexpr (sizeof(VT) == 4) {
#pragma unroll
                        for (int k = 0; k < 3; k++) wd[k] = tagged(__float_as_uint((float)z[k]), epoch + 1);
                        wd[3] = wd[2];
                    } else {
#pragma unroll
                        for (int k = 0; k < 3; k++) split((double)z[k], epoch + 1, wd[2 * k], wd[2 * k + 1]);
                    }
#pragma unroll
                    for (int k = 0; k < Z; k += 2) st_words(a.zg + Z * row + k, wd[k], wd[k + 1]);
                }
            }
        }
        __syncwarp();
        if (!with_z) return;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], s);
            acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], s);
        }
        if (lane == 0) { sh->part[w][0] = acc[0]; sh->part[w][1] = acc[1]; }
    };
    const int ngrp = (nr + kGR - 1) / kGR;
    const int sub = lane / kLPR, sl = lane % kLPR;
    // fetches group gi into slot k of the warp's ring: matrix blocks, column indices,
    // rows' offsets
    auto fetch = [&](int gi, int k) {
        const int i0 = gi * kGR, i1 = min(i0 + kGR, nr);
        const size_t n0 = (size_t)b0 + srp[i0], n1 = (size_t)b0 + srp[i1];
        const size_t g0 = n0 * BB & ~(size_t)15, g1 = (n1 * BB + 15) & ~(size_t)15;
        const size_t c0 = n0 * 2 & ~(size_t)15, c1 = (n1 * 2 + 15) & ~(size_t)15;
        const unsigned mb = (unsigned)(g1 - g0), cb = (unsigned)(c1 - c0), ob = 16u * (unsigned)(i1 - i0);
        const unsigned bar = bars + 8u * k, dst = sptr(ring + (size_t)k * pl.group_bytes);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(mb + cb + ob) : "memory");
        const char* src = reinterpret_cast<const char*>(a.H) + g0;
        if (pl.evict_first)
            asm volatile(
                "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
                    dst),
                "l"(src), "r"(mb), "r"(bar), "l"(policy)
                : "memory");
        else
            bulk(dst, src, mb, bar);
        bulk(dst + pl.slot_col, reinterpret_cast<const char*>(pl.lcol) + c0, cb, bar);
        bulk(dst + pl.slot_off, reinterpret_cast<const char*>(a.woff + r0 + i0), ob, bar);
    };
    // fills the ring for the next product (the matrix does not change: ahead of p)
    auto prefetch = [&]() {
        for (int k = 0; k < pl.depth; k++)
            if (w + k * kWarps < ngrp) {
                ring_busy |= 1u << k;
                if (lane == 0) fetch(w + k * kWarps, k);
            }
    };
    bool ok = renew();
    double acc[2], d1[1];
    update(VT(0), VT(0), true);
    prefetch();
    ok = exchange<1, 2, 2, false>(acc, sh, G, ++epoch, a.box, 0u, 0, nullptr, a.wait_ns) && ok;
    double rz = acc[0], rr = acc[1], pq = 0.0, alpha = 0.0, beta = 0.0;
    const double bnorm2 = rr;
    const double te = eta2 * rr, tol2 = te > abs_tol2 ? te : abs_tol2;
    int it = 0, breakdown = 0, flip = 0;
    bool done = !ok || rr <= tol2 || a.maxit <= 0;
    while (!done) {
        const VT bt = (VT)beta;
#pragma unroll 4
        for (int i = t; i < nr; i += kT) {
            VT* pc = sp + P * i;
            const VT z0 = zs[r0 + i], z1 = zs[N + r0 + i], z2 = zs[2 * N + r0 + i];
            pc[0] = z0 + bt * pc[0];
            pc[1] = z1 + bt * pc[1];
            pc[2] = z2 + bt * pc[2];
        }
        constexpr int HU = sizeof(VT) == 4 ? 3 : 2;  // border columns a thread has in flight
        for (int kb = t; kb < nh; kb += HU * kT) {
            u64 wd[HU][Z];
            bool here;
            Patience wait(a.wait_ns);
            do {
                here = true;
#pragma unroll
                for (int u = 0; u < HU; u++)
                    if (kb + u * kT < nh) {
                        const u64* q = a.zg + Z * (size_t)halo[kb + u * kT];
#pragma unroll
                        for (int m = 0; m < Z; m += 2) ld_words(q + m, wd[u][m], wd[u][m + 1]);
                    }
#pragma unroll
                for (int u = 0; u < HU; u++)
                    if (kb + u * kT < nh)
#pragma unroll
                        for (int m = 0; m < Z; m++) here = here && has(wd[u][m], epoch);
            } while (!here && wait.more(a.wait_ns));
            if (!here) sh->late = 1;
#pragma unroll
            for (int u = 0; u < HU; u++)
                if (kb + u * kT < nh) {
                    VT* pc = sp + P * (nr + kb + u * kT);
                    if constexpr (sizeof(VT) == 4) {
#pragma unroll
                        for (int m = 0; m < 3; m++) pc[m] = (VT)__uint_as_float((unsigned)wd[u][m]) + bt * pc[m];
                    } else {
#pragma unroll
                        for (int m = 0; m < 3; m++) pc[m] = (VT)join(wd[u][2 * m], wd[u][2 * m + 1]) + bt * pc[m];
                    }
                }
        }
        clear_part();
        __syncwarp();
        __syncthreads();
        // q = A p
        double pqw = 0.0, yw[6] = {0, 0, 0, 0, 0, 0};
        int ag = 0;
        int slot = 0;
        for (int gi = w; gi < ngrp; gi += kWarps) {
            const int i = gi * kGR + sub, an = gi * kGR / L;
            if (an != ag) { flush(ag, yw, kLPR); ag = an; }
            const int ii = min(i, nr - 1), k0 = srp[ii], k1 = i < nr ? srp[ii + 1] : k0, kg = srp[gi * kGR];
            // without its copy the group has no indices: the product ends here, and the
            // solve in the exchange behind it
            if (!__all_sync(0xffffffffu, bar_wait(bars + 8u * slot, (ring_phase >> slot) & 1u, a.wait_ns))) {
                sh->late = 1;
                break;
            }
            ring_phase ^= 1u << slot;
            const bool next = gi + pl.depth * kWarps < ngrp;
            if (!next) ring_busy &= ~(1u << slot);
            const unsigned char* rs_ = ring + (size_t)slot * pl.group_bytes;
            const VT* hg = reinterpret_cast<const VT*>(rs_ + (((size_t)b0 + kg) * BB & 15));
            const uint16_t* cg_ = reinterpret_cast<const uint16_t*>(rs_ + pl.slot_col + (((size_t)b0 + kg) * 2 & 15));
            const float4 d = *reinterpret_cast<const float4*>(rs_ + pl.slot_off + 16 * sub);
            VT a0 = VT(0), a1 = VT(0), a2 = VT(0), p0, p1, p2;
#pragma unroll 4
            for (int k = k0 + sl; k < k1; k += kLPR) {
                const VT* h = hg + 9 * (k - kg);
                ld_p<VT>(sp + P * (int)cg_[k - kg], p0, p1, p2);
                a0 += h[0] * p0 + h[1] * p1 + h[2] * p2;
                a1 += h[3] * p0 + h[4] * p1 + h[5] * p2;
                a2 += h[6] * p0 + h[7] * p1 + h[8] * p2;
            }
            __syncwarp();
            if (lane == 0 && next) fetch(gi + pl.depth * kWarps, slot);
            slot = slot + 1 == pl.depth ? 0 : slot + 1;
#pragma unroll
            for (int s = kLPR / 2; s > 0; s >>= 1) {
                a0 += __shfl_xor_sync(0xffffffffu, a0, s);
                a1 += __shfl_xor_sync(0xffffffffu, a1, s);
                a2 += __shfl_xor_sync(0xffffffffu, a2, s);
            }
            if (i < nr) {
                if (sl == 0) {
                    qs[r0 + i] = a0;
                    qs[N + r0 + i] = a1;
                    qs[2 * N + r0 + i] = a2;
                }
                ld_p<VT>(sp + P * i, p0, p1, p2);
                pqw += (double)p0 * (double)a0 + (double)p1 * (double)a1 + (double)p2 * (double)a2;
                const unsigned f = __float_as_uint(d.w);
                VT q[3] = {a0, a1, a2};
                project<VT>((f >> 8) & 0xffu, a.pn + r0 + i, q);
                restrict_node<VT>(d, f, q, yw);
            }
        }
        __syncwarp();
        flush(ag, yw, kLPR);
#pragma unroll
        for (int s = 16; s >= kLPR; s >>= 1) pqw += __shfl_xor_sync(0xffffffffu, pqw, s);
        if (lane == 0) sh->part[w][0] = pqw;
        ++epoch;
        u64* board = a.board + (flip ? board_words : 0);
        flip ^= 1;
        post(board, epoch);
        ok = exchange<0, 1, 1, false>(d1, sh, G, epoch, a.box, 0u, 0, nullptr, a.wait_ns);
        if (!ok) break;
        pq = d1[0];
        if (!(pq > 0.0)) {
            breakdown = 1;
            break;
        }
        alpha = rz / pq;
        const VT al = (VT)alpha;
        if (sizeof(VT) == 4 && (it & 7) == 7) {
            // y anew from the updated residual (see pcg_resident.cu)
            update(VT(0), al, false);
            __syncthreads();
            if (!renew()) { ok = false; break; }
            update(al, VT(0), true);
        } else {
            coarse(board, epoch, false, (double)al);
            update(al, al, true);
        }
        prefetch();
        ok = exchange<1, 2, 2, false>(acc, sh, G, ++epoch, a.box, 0u, 0, nullptr, a.wait_ns);
        if (!ok) break;
        beta = acc[0] / rz;
        rz = acc[0];
        rr = acc[1];
        it++;
        done = rr <= tol2 || it >= a.maxit || !(rr == rr);
    }
    // the bulk copies still in flight must land before the block leaves
    for (int k = 0; k < pl.depth; k++)
        if ((ring_busy >> k) & 1u) bar_wait(bars + 8u * k, (ring_phase >> k) & 1u, kDrainNs);
    for (int i = t; i < nr; i += kT) {
        const long long row = r0 + i;
#pragma unroll
        for (int k = 0; k < 3; k++) a.x[3 * row + k] = xs[k * N + row];
        if (breakdown) {
            VT* pb = ((it & 1) ? a.p0 : a.p1) + 4 * row;
#pragma unroll
            for (int k = 0; k < 3; k++) pb[k] = sp[P * i + k];
        }
    }
    __syncthreads();
    if (t == 0 && (sh->abort | sh->late)) atomicOr(&a.sc->status, kFlagTimeout);
    if (me == 0 && t == 0) {
        DevScalars* sc = a.sc;
        sc->rz = rz; sc->rr = rr; sc->bnorm2 = bnorm2; sc->tol2 = tol2; sc->pq = pq;
        sc->alpha = breakdown ? 0.0 : alpha; sc->beta = beta;
        sc->it = it; sc->maxit = a.maxit; sc->breakdown = breakdown; sc->done = 1; sc->skip = 0;
        *a.epoch = epoch;
    }
}

}  // namespace

size_t stream_smem(const StreamPlan& pl, int vsize) {
    const int at = vsize == 4 ? soffsets<float>(pl).ring : soffsets<double>(pl).ring;
    return (size_t)at + (size_t)kWarps * pl.depth * pl.group_bytes;
}

template <typename VT>
int launch_pcg_stream(const StreamPlan& pl, const StreamArgs<VT>& a, cudaStream_t st) {
    auto kern = k_pcg_stream<VT>;
    static std::atomic<int> done[kMaxDevices];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices || !done[dev].load(std::memory_order_relaxed)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentSmem);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < kMaxDevices) done[dev].store(1, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.G);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = stream_smem(pl, (int)sizeof(VT));
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, pl, a);
    if (e != cudaSuccess) return (int)e;
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return 0;
}
template int launch_pcg_stream<float>(const StreamPlan&, const StreamArgs<float>&, cudaStream_t);
template int launch_pcg_stream<double>(const StreamPlan&, const StreamArgs<double>&, cudaStream_t);

}  // namespace sors
