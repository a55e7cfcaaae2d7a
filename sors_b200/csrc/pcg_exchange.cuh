// pcg_exchange.cuh -- what the one-launch PCG kernels (pcg_resident.cu,
// pcg_stream.cu) share: sums and border values between the blocks of a launch,
// constraint projection, restriction to the coarse unknowns.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sors_internal.h"

namespace sors {
namespace {

constexpr int kT = kResidentThreads;
constexpr int kWarps = kT / 32;
constexpr int kBoxes = kResidentBoxEntries;  // mailbox entries: five per polling lane
constexpr int kScratch = 3328;
typedef unsigned long long u64;

__device__ __forceinline__ u64 clock_ns() {
    u64 t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// The limit of a wait, in elapsed time: one look at the clock in 256 at the value
// waited for, the first of which starts it.  Limit 0: a single look at the value.
struct Patience {
    u64 t0 = 0;
    unsigned n;
    __device__ __forceinline__ explicit Patience(u64 limit_ns) : n(limit_ns ? 0u : 255u) {}
    __device__ __forceinline__ bool clock(u64 limit_ns) {
        const u64 t = clock_ns();
        if (n == 256u) t0 = t;
        return t - t0 < limit_ns;
    }
    __device__ __forceinline__ bool more(u64 limit_ns) { return (++n & 255u) || clock(limit_ns); }
    // the same answer in every lane of the warp
    __device__ __forceinline__ bool more_warp(u64 limit_ns) {
        return (++n & 255u) || __shfl_sync(0xffffffffu, (int)clock(limit_ns), 0);
    }
};
static_assert(kResidentMaxBlocks <= kBoxes && kBoxes % 32 == 0, "a lane polls kBoxes / 32 entries");

// values per node of a column's p: one 16-byte load (FP32), three 8-byte loads (FP64)
template <typename VT>
struct Lay {
    static constexpr int P = sizeof(VT) == 4 ? 4 : 3;
    static constexpr int Z = sizeof(VT) == 4 ? 4 : 6;  // 64-bit words of a published z (grid form)
};

__device__ __forceinline__ void st_words(u64* p, u64 a, u64 b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_words(const u64* p, u64& a, u64& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ u64 tagged(unsigned v, unsigned epoch) { return ((u64)epoch << 32) | v; }
__device__ __forceinline__ bool has(u64 w, unsigned epoch) { return (unsigned)(w >> 32) == epoch; }
__device__ __forceinline__ double join(u64 lo, u64 hi) {
    return __longlong_as_double((long long)((hi << 32) | (lo & 0xffffffffull)));
}
__device__ __forceinline__ void split(double v, unsigned epoch, u64& lo, u64& hi) {
    const u64 b = (u64)__double_as_longlong(v);
    lo = tagged((unsigned)b, epoch);
    hi = tagged((unsigned)(b >> 32), epoch);
}

// cluster form: the address of `local` in block `rank`, and pushes that count
// their bytes on that block's mbarrier
__device__ __forceinline__ unsigned remote(const void* local, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
    return r;
}
__device__ __forceinline__ void push(unsigned dst, unsigned bar, double a) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(dst), "d"(a),
                 "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void push(unsigned dst, unsigned bar, double a, double b) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "d"(a), "d"(b), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void push(unsigned dst, unsigned bar, float a, float b, float c) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     dst),
                 "f"(a), "f"(b), "f"(c), "f"(0.0f), "r"(bar)
                 : "memory");
}

// Waits for phase `parity` of the block's own mbarrier; false after the limit (a
// try_wait that fails has waited for some time itself).
__device__ __forceinline__ bool cluster_wait(unsigned bar, unsigned parity, u64 limit_ns) {
    unsigned got;
    if (limit_ns == 0) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(got)
            : "r"(bar), "r"(parity)
            : "memory");
        return got != 0;
    }
    u64 t0 = 0;
    for (;;) {
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}"
            : "=r"(got)
            : "r"(bar), "r"(parity)
            : "memory");
        if (got) return true;
        const u64 t = clock_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 >= limit_ns) return false;
    }
}

// Exchange sites and their values: 0 p.q (and P^T q, six values, with the coarse
// correction), 1 r.z and r.r, 2 P^T r (six values, coarse correction).
constexpr int kMsg = 7;
__host__ __device__ constexpr int site_at(int site) { return site == 0 ? 0 : (site == 1 ? kMsg : kMsg + 2); }
constexpr int kVals = kMsg + 2 + 6;
static_assert(2 * kVals == kResidentBoxWords, "words of a mailbox entry");

// Fixed scratch at the start of the block's shared memory.
struct Scratch {
    u64 bar[4];                    // cluster form: one mbarrier per site
    double part[kWarps][8];        // warps' partial values
    double tot[2];
    double irz;                    // 1 / r.z
    double zc[6][2];               // the range's coarse correction, two partial sums each
    // A wait ran out.  Grid form: abort is set between the two barriers of an exchange
    // and read after the second, so the block's threads agree; late by the waits between
    // exchanges, and becomes abort in the next one.
    int abort, late;
    double slot[kVals][16];  // cluster form: the blocks' messages, by value
};
static_assert(sizeof(Scratch) <= kScratch, "fixed scratch");

// Exchanges the NV values whose per-warp sums are in sh->part: warp v < NV adds
// value v over the block's warps, sends it to every block, and collects all
// blocks' values.  The first NSUM values are summed (every thread gets the
// totals in v), the others are left per block: yq[(v - NSUM) G + b] in the grid
// form, sh->slot[site_at(SITE) + v][b] in the cluster form.  No site is used twice
// in a row, so a slot or mailbox entry is written again only after every block
// has read it.
// halo_bytes: border z the block receives with site 1 (cluster form).  False:
// something did not arrive within the limit; grid form: in every thread of the block
// alike, cluster form: in the threads that waited in vain.
template <int SITE, int NV, int NSUM, bool CL>
__device__ __forceinline__ bool exchange(double (&v)[NSUM ? NSUM : 1], Scratch* sh, int G, unsigned epoch, u64* box,
                                         unsigned parity, int halo_bytes, double* yq, u64 limit_ns) {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31, me = blockIdx.x;
    __syncthreads();
    if (w < NV) {
        double x = sh->part[l & (kWarps - 1)][w];
#pragma unroll
        for (int o = kWarps / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if constexpr (CL) {
            double* slot = sh->slot[site_at(SITE) + w];
            if (w == 0 && l == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                                 (unsigned)__cvta_generic_to_shared(&sh->bar[SITE])),
                             "r"(G * 8 * NV + halo_bytes)
                             : "memory");
            __syncwarp();
            if (l < G) push(remote(slot + me, l), remote(&sh->bar[SITE], l), x);
        } else {
            constexpr int J = kBoxes / 32;
            u64 lo, hi;
            split(x, epoch, lo, hi);
            const size_t at = (size_t)site_at(SITE) + w;  // this value's entries of a mailbox
#pragma unroll
            for (int j = 0; j < J; j++)
                if (l + 32 * j < G)
                    st_words(box + (((size_t)(l + 32 * j) * kVals + at) * G + me) * 2, lo, hi);
            // a lane's entries are loaded together, so a round of polls is one trip to L2
            const u64* q = box + (((size_t)me * kVals + at) * G + l) * 2;
            u64 a[J], b[J];
            bool ok;
            Patience wait(limit_ns);
            do {
                ok = true;
#pragma unroll
                for (int j = 0; j < J; j++)
                    if (l + 32 * j < G) ld_words(q + 64 * j, a[j], b[j]);
#pragma unroll
                for (int j = 0; j < J; j++)
                    if (l + 32 * j < G) ok = ok && has(a[j], epoch) && has(b[j], epoch);
                ok = __all_sync(0xffffffffu, ok);  // the warp stays together
            } while (!ok && wait.more_warp(limit_ns));
            if (w < NSUM) {
                double t = 0.0;
#pragma unroll
                for (int j = 0; j < J; j++)
                    if (l + 32 * j < G) t += join(a[j], b[j]);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (l == 0) sh->tot[w] = t;
            } else {
#pragma unroll
                for (int j = 0; j < J; j++)
                    if (l + 32 * j < G) yq[(w - NSUM) * G + l + 32 * j] = join(a[j], b[j]);
            }
            if (l == 0 && !ok) sh->abort = 1;
        }
    }
    if (!CL && threadIdx.x == kT - 1 && sh->late) sh->abort = 1;
    if constexpr (CL) {
        const bool got = cluster_wait((unsigned)__cvta_generic_to_shared(&sh->bar[SITE]), parity, limit_ns);
        if (!got) sh->abort = 1;
        // 16 values: a lane each (twice per warp), four shuffles
#pragma unroll
        for (int s = 0; s < NSUM; s++) v[s] = (l & 15) < G ? sh->slot[site_at(SITE) + s][l & 15] : 0.0;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int s = 0; s < NSUM; s++) v[s] += __shfl_xor_sync(0xffffffffu, v[s], o);
        return got;
    } else {
        __syncthreads();
#pragma unroll
        for (int s = 0; s < NSUM; s++) v[s] = sh->tot[s];
        return sh->abort == 0;
    }
}

// Tolerances of a solve; false when the Newton iteration ends before it (the
// whole grid agrees: the scalars read here are not written by this launch).
template <typename Args>
__device__ __forceinline__ bool solve_tolerances(const Args& a, double& eta2, double& abs2) {
    eta2 = a.eta2;
    abs2 = a.abs_tol2;
    if (!a.nf.on) return true;
    const double gn = sqrt(a.sc->gnorm2);
    if ((a.sc->status & kFlagInverted) || !(gn == gn) || (a.nf.res_tol > 0.0 && gn < a.nf.res_tol)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.sc->skip = 1;
            a.sc->it = 0;
            a.sc->breakdown = 0;
            a.sc->done = 1;
        }
        return false;
    }
    const double eta = newton_forcing(a.nf, gn);
    eta2 = eta * eta;
    abs2 = a.nf.res_tol > 0.0 ? 0.01 * a.nf.res_tol * a.nf.res_tol : 0.0;
    return true;
}

template <typename VT>
__device__ __forceinline__ void project(unsigned f, const double4* pn, VT (&y)[3]) {
    if (!f) return;
    if (f & 1u) y[0] = VT(0);
    if (f & 2u) y[1] = VT(0);
    if (f & 4u) y[2] = VT(0);
    if (f & 8u) {
        const double4 n = *pn;
        const VT d = (VT)n.x * y[0] + (VT)n.y * y[1] + (VT)n.z * y[2];
        y[0] -= d * (VT)n.x;
        y[1] -= d * (VT)n.y;
        y[2] -= d * (VT)n.z;
    }
}

template <typename VT>
__device__ __forceinline__ void ld_p(const VT* p, VT& a, VT& b, VT& c) {
    if constexpr (sizeof(VT) == 4) {
        const float4 t = *reinterpret_cast<const float4*>(p);
        a = t.x; b = t.y; c = t.z;
    } else {
        a = p[0]; b = p[1]; c = p[2];
    }
}

// P_i^T y (six values) at a node with offset o from its range's centre: three
// translations, three rotations; bits 0-2 of f: held DOFs.
template <typename VT>
__device__ __forceinline__ void restrict_node(const float4& o, unsigned f, const VT (&y)[3], double (&c)[6]) {
    const double w0 = f & 1u ? 0.0 : (double)y[0], w1 = f & 2u ? 0.0 : (double)y[1], w2 = f & 4u ? 0.0 : (double)y[2];
    const double dx = o.x, dy = o.y, dz = o.z;
    c[0] += w0;
    c[1] += w1;
    c[2] += w2;
    c[3] += dy * w2 - dz * w1;
    c[4] += dz * w0 - dx * w2;
    c[5] += dx * w1 - dy * w0;
}

}  // namespace
}  // namespace sors
