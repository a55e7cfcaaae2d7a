// pcg_resident.cu -- a whole block-Jacobi PCG solve in one launch, with the
// matrix resident in registers and shared memory.
//
// What bounds the solve of a mesh up to some tens of thousands of nodes is not
// its bytes: the matrix of 4,225 nodes is 4.3 MB in FP64 and sits in L2, but an
// iteration as three launches (p, SpMV with p.q, update with r.z) took 15-17 us
// of launch gaps, cold starts and two grid-wide reductions through a last
// block.  Here the thread blocks stay: each owns a contiguous range of rows
// (the locality numbering makes neighbouring rows neighbouring nodes), loads
// its CSR blocks once, and iterates until the solve ends.  An iteration
// exchanges z at the range's border and two sums, nothing else:
//
//   p = z + beta p     own and border columns (a border column's p is formed by
//                      every range that reads it, from the same z: same bits)
//   q = A p, p.q       lanes of a group share a row, shuffles add it
//   [sum]  alpha       x += alpha p, r -= alpha q, z = M^-1 r, publish z
//   [sum]  beta        r.z, r.r
//
// Matrix: a group of LPR lanes holds the first R * LPR blocks of its row in
// registers (the register file is the largest and fastest memory of an SM, and
// nine values per block from shared memory at 2-3 way bank conflicts were two
// thirds of an iteration); what does not fit, longer rows and the rows beyond
// one per group, is in shared memory, and past that is read through L2.
//
// Two forms of the exchange:
//   cluster  up to 16 blocks of one cluster: partial sums and border z are
//            pushed into the readers' shared memory (st.async), each site's
//            mbarrier counts the bytes.  A reader waits on its own mbarrier.
//   grid     a cooperative launch over the SMs: every block pushes its partial
//            sum into every block's mailbox in global memory and polls its own,
//            z goes through global memory.  Each 64-bit word carries 32 bits of
//            the value and the 32-bit epoch, so a word says by itself whether it
//            has arrived: no fence, no atomic, no flag.  (Polling one shared set
//            of slots instead took 4-5 us per sum: 148 readers on 37 lines.)
//
// All sums run in a fixed order, so a solve is bit-reproducible.
//
// Measured, whole iteration with block Jacobi (three launches before -> here):
// cluster, 1,728 FP32 nodes 15 -> 3.8 us; grid, 4,225 FP64 nodes 15 -> 6.4 us,
// 10,648 FP32 nodes 17 -> 6.2 us, 18,921 FP64 hex nodes (33 MB of matrix) 25 -> 10.8
// us.  With the two-level preconditioner, which takes two to five times fewer
// iterations, and a solve's loading shared out over them: cluster, 525 FP64 nodes
// 4.0 us; grid, 4,225 FP64 nodes 8.4, 9,856 FP32 nodes 9.8, 22,680 FP64 nodes 14.7,
// the hexes 14.6 us.  What bounds it now: the two sums' round trips through L2
// (1.4 us each over 64 blocks, 2.2 over 148, of which 1.2 us is one store and one
// load) or, in a cluster, latency of the dependent FP64 steps (about 1,000 cycles a
// sum, 1,100 a product).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "fem_math.cuh"
#include "pcg_exchange.cuh"
#include "sors_internal.h"

namespace cg = cooperative_groups;

namespace sors {

namespace {

constexpr u64 kStayNs = 20000;  // a push takes about a microsecond

// Byte offsets of a block's shared memory, the same in every block of a launch.
struct Off {
    int sp, sq, sm, sx, sz, soff, sa, syc, sov, sgb, shalo, spp, spush, scol, sval;
};
template <typename VT>
__host__ __device__ inline Off offsets(const ResidentPlan& pl) {
    auto up = [](int b) { return (b + 15) & ~15; };
    Off o;
    const int nc = pl.coarse ? 6 * pl.G : 0;
    int at = kScratch;
    o.sp = at; at = up(at + pl.max_cols * Lay<VT>::P * (int)sizeof(VT));
    o.sq = at; at = up(at + pl.max_rows * 3 * (int)sizeof(VT));
    o.sm = at; at = up(at + pl.max_rows * 9 * (int)sizeof(VT));
    o.sx = at; at = up(at + pl.max_rows * 9 * (int)sizeof(VT));
    o.sz = at; at = up(at + (pl.cluster ? pl.max_halo * 4 * (int)sizeof(VT) : 0));
    o.soff = at; at = up(at + (pl.coarse ? pl.max_rows * 16 : 0));
    o.sa = at; at = up(at + 6 * nc * (int)sizeof(VT));
    o.syc = at; at = up(at + 3 * nc * 8);
    o.sov = at; at = up(at + (pl.max_rows + 1) * 4);
    o.sgb = at; at = up(at + pl.max_rows * 4);
    o.shalo = at; at = up(at + (pl.cluster ? 0 : pl.max_halo * 4));
    o.spp = at; at = up(at + (pl.cluster ? pl.max_push * 2 : 0));
    o.spush = at; at = up(at + (pl.cluster ? pl.max_push * 4 : 0));
    o.scol = at; at = up(at + pl.max_over * 2);
    o.sval = at;
    return o;
}

// A loaded value stays in its register: the compiler may not load it again.
__device__ __forceinline__ void keep(float& v) { asm volatile("" : "+f"(v)); }
__device__ __forceinline__ void keep(double& v) { asm volatile("" : "+d"(v)); }

// TL: the two-level preconditioner M^-1 + P Ac^-1 P^T with one aggregate per
// range.  Every block keeps the whole y = P^T r (6 G values) and its own six
// rows of Ac^-1: P^T q travels with p.q, y -= alpha P^T q is formed by every
// block alike, and the correction costs no exchange of its own.
template <typename VT, int LPR, int R, bool CL, bool TL>
__global__ void __launch_bounds__(kT, 1) k_pcg_resident(ResidentPlan pl, ResidentArgs<VT> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int P = Lay<VT>::P, Z = Lay<VT>::Z;
    constexpr int NG = kT / LPR;  // groups of lanes
    double eta2, abs_tol2;
    if (!solve_tolerances(a, eta2, abs_tol2)) return;
    Scratch* sh = reinterpret_cast<Scratch*>(smem);
    const Off o = offsets<VT>(pl);
    VT* sp = reinterpret_cast<VT*>(smem + o.sp);
    VT* sq = reinterpret_cast<VT*>(smem + o.sq);
    VT* sm = reinterpret_cast<VT*>(smem + o.sm);
    VT* sz = reinterpret_cast<VT*>(smem + o.sz);
    int* sov = reinterpret_cast<int*>(smem + o.sov);
    int* sgb = reinterpret_cast<int*>(smem + o.sgb);
    int* shalo = reinterpret_cast<int*>(smem + o.shalo);
    uint16_t* spp = reinterpret_cast<uint16_t*>(smem + o.spp);
    int* spush = reinterpret_cast<int*>(smem + o.spush);
    uint16_t* scol = reinterpret_cast<uint16_t*>(smem + o.scol);
    VT* sval = reinterpret_cast<VT*>(smem + o.sval);
    float4* soff = reinterpret_cast<float4*>(smem + o.soff);
    VT* sa = reinterpret_cast<VT*>(smem + o.sa);
    double* syc = reinterpret_cast<double*>(smem + o.syc);  // y, its next value, P^T q
    const int t = threadIdx.x, lane = t & 31, G = gridDim.x, me = blockIdx.x;
    const int r0 = pl.row0[me], nr = pl.row0[me + 1] - r0;
    const int h0 = pl.halo_ptr[me], nh = pl.halo_ptr[me + 1] - h0;
    unsigned epoch = CL ? 0u : *(volatile const unsigned*)a.epoch;
    if (t == 0) {
        sh->abort = sh->late = 0;
        if constexpr (CL)
#pragma unroll
            for (int k = 0; k < 3; k++)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(&sh->bar[k]))
                             : "memory");
        if constexpr (CL) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // every block runs, its barriers set up, before any pushes into another's shared memory
    if constexpr (CL) cg::this_cluster().sync();

    // matrix: the group's first row in registers ...
    const int g = t / LPR, sl = t % LPR;
    VT hv[R][9];
    int hc[R];
    {
        const int gb = g < nr ? a.row_ptr[r0 + g] : 0, len = g < nr ? a.row_ptr[r0 + g + 1] - gb : 0;
#pragma unroll
        for (int j = 0; j < R; j++) {
            const int k = sl + LPR * j;
            hc[j] = k < len ? P * (int)pl.lcol[gb + k] : 0;
#pragma unroll
            for (int e = 0; e < 9; e++) {
                hv[j][e] = k < len ? __ldg(a.H + 9 * (size_t)(gb + k) + e) : VT(0);
                keep(hv[j][e]);
            }
        }
    }
    // ... the rest of its blocks and the rows beyond NG in shared memory, while it lasts
    for (int i = t; i <= nr; i += kT) sov[i] = pl.over[r0 + me + i];
    __syncthreads();
    for (int i = t >> 5; i < nr; i += kWarps) {
        const int gb = a.row_ptr[r0 + i + 1] - (sov[i + 1] - sov[i]);  // first block not in registers
        if (lane == 0) sgb[i] = gb;
        const int n = sov[i + 1] - sov[i], nres = min(max(pl.res_blocks - sov[i], 0), n);
        for (int k = lane; k < n; k += 32) scol[sov[i] + k] = pl.lcol[gb + k];
        for (int k = lane; k < 9 * nres; k += 32) sval[9 * sov[i] + k] = __ldg(a.H + 9 * (size_t)gb + k);
    }
    int np = 0;  // border z to push: row spp, to spush
    if constexpr (CL) {
        const int q0 = pl.push_ptr[r0];
        np = pl.push_ptr[r0 + nr] - q0;
        for (int k = t; k < np; k += kT) spush[k] = pl.push[q0 + k];
        for (int i = t; i < nr; i += kT)
            for (int k = pl.push_ptr[r0 + i] - q0; k < pl.push_ptr[r0 + i + 1] - q0; k++) spp[k] = (uint16_t)i;
    } else {
        for (int k = t; k < nh; k += kT) shalo[k] = pl.halo[h0 + k];
    }
    for (int k = t; k < (nr + nh) * P; k += kT) sp[k] = VT(0);
    const int nc = 6 * G;
    if constexpr (TL) {
        for (int k = t; k < 6 * nc; k += kT) sa[k] = __ldg(a.Ainv + (size_t)6 * me * nc + k);
        for (int i = t; i < nr; i += kT) {
            float4 v = pl.off[r0 + i];
            v.w = __uint_as_float((unsigned)a.fixed[r0 + i] | (a.pflag ? (unsigned)a.pflag[r0 + i] << 8 : 0u));
            soff[i] = v;
        }
    }
    if (t < kWarps)
#pragma unroll
        for (int k = 0; k < 8; k++) sh->part[t][k] = 0.0;

    // one thread per row: x, r, z and the inverse diagonal block (as k_block_jacobi), in
    // shared memory (a row's nine values are an odd stride: no bank conflicts), so that
    // the registers are left to the matrix
    VT* M = sm + 9 * t;
    VT* x = reinterpret_cast<VT*>(smem + o.sx) + 9 * t;
    VT *rs = x + 3, *zs = x + 6;
    unsigned pf = 0;
    const size_t row = (size_t)r0 + t;
    if (t < nr) {
        double d[9], c[9];
        const VT* hd = a.H + 9 * (size_t)a.diag_slot[row];
#pragma unroll
        for (int k = 0; k < 9; k++) d[k] = (double)hd[k];
        d[1] = d[3]; d[2] = d[6]; d[5] = d[7];
        cof3(d, c);
        const double det = d[0] * c[0] + d[1] * c[1] + d[2] * c[2];
        const bool inv = det != 0.0 && det == det;
        const double id = 1.0 / det;
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int m = 0; m < 3; m++)
                M[k * 3 + m] = inv ? (VT)(c[m * 3 + k] * id) : (VT)(k == m ? 1.0 : 0.0);
        if (a.pflag) pf = a.pflag[row];
        VT r[3];
#pragma unroll
        for (int k = 0; k < 3; k++) r[k] = (VT)(-a.g[3 * row + k]);
        project<VT>(pf, a.pn + row, r);
#pragma unroll
        for (int k = 0; k < 3; k++) { x[k] = VT(0); rs[k] = r[k]; }
    }
    __syncthreads();

    // z = M^-1 r (+ P zc), published with the coming site-1 sum; r.z and r.r of the warp
    auto precondition = [&]() {
        double acc[2] = {0.0, 0.0};
        if (t < nr) {
            VT z[3];
            const VT r[3] = {rs[0], rs[1], rs[2]};
#pragma unroll
            for (int k = 0; k < 3; k++) z[k] = M[k * 3] * r[0] + M[k * 3 + 1] * r[1] + M[k * 3 + 2] * r[2];
            if constexpr (TL) {
                VT c[6];
#pragma unroll
                for (int m = 0; m < 6; m++) c[m] = (VT)(sh->zc[m][0] + sh->zc[m][1]);
                const float4 d = soff[t];
                const unsigned f = __float_as_uint(d.w);
                const VT ox = (VT)d.x, oy = (VT)d.y, oz = (VT)d.z;
                if (!(f & 1u)) z[0] += c[0] + c[4] * oz - c[5] * oy;
                if (!(f & 2u)) z[1] += c[1] - c[3] * oz + c[5] * ox;
                if (!(f & 4u)) z[2] += c[2] + c[3] * oy - c[4] * ox;
            }
            project<VT>(pf, a.pn + row, z);
#pragma unroll
            for (int k = 0; k < 3; k++) zs[k] = z[k];
            if constexpr (!CL) {
                u64 w[Z];
                if constexpr (sizeof(VT) == 4) {
#pragma unroll
                    for (int k = 0; k < 3; k++) w[k] = tagged(__float_as_uint((float)z[k]), epoch + 1);
                    w[3] = w[2];
                } else {
#pragma unroll
                    for (int k = 0; k < 3; k++) split((double)z[k], epoch + 1, w[2 * k], w[2 * k + 1]);
                }
#pragma unroll
                for (int k = 0; k < Z; k += 2) st_words(a.zg + Z * row + k, w[k], w[k + 1]);
            }
#pragma unroll
            for (int k = 0; k < 3; k++) {
                acc[0] += (double)r[k] * (double)z[k];
                acc[1] += (double)r[k] * (double)r[k];
            }
        }
        if constexpr (CL) {
            // a thread per push (a row may have several readers)
            __syncthreads();
            for (int k = t; k < np; k += kT) {
                const int d = spush[k];
                const VT* z = reinterpret_cast<const VT*>(smem + o.sx) + 9 * (int)spp[k] + 6;
                const unsigned dst = remote(sz + 4 * (d & 0xffff), d >> 16), rb = remote(&sh->bar[1], d >> 16);
                if constexpr (sizeof(VT) == 4) {
                    push(dst, rb, z[0], z[1], z[2]);
                } else {
                    push(dst, rb, z[0], z[1]);
                    push(dst + 16, rb, z[2]);
                }
            }
            __syncwarp();
        }
        if ((t & ~31) < nr) {  // a warp with rows
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], s);
                acc[1] += __shfl_xor_sync(0xffffffffu, acc[1], s);
            }
        }
        if (lane == 0) {
            sh->part[t >> 5][0] = acc[0];
            sh->part[t >> 5][1] = acc[1];
        }
    };
    // zc = Ac^-1 y for the range's six coarse unknowns, two warps a row, with
    // y = ya - al P^T q (site 0's message), or the site-2 message itself (fresh); the
    // first row's warps keep y in yb.
    constexpr int kCW = 4;  // first of the twelve warps
    auto coarse = [&](bool fresh, double al, const double* ya, double* yb) {
        const int w = (t >> 5) - kCW;
        if (w >= 0) {
            const int m = w >> 1;
            double z = 0.0;
            for (int j = (w & 1) * 32 + lane; j < nc; j += 64) {
                double y;
                if constexpr (CL) y = sh->slot[site_at(fresh ? 2 : 0) + (fresh ? 0 : 1) + j / G][j % G];
                else y = syc[2 * nc + j];
                if (!fresh) y = ya[j] - al * y;
                if (m == 0) yb[j] = y;
                z += (double)sa[m * nc + j] * y;
            }
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) z += __shfl_xor_sync(0xffffffffu, z, s);
            if (lane == 0) sh->zc[m][w & 1] = z;
        }
        __syncthreads();
    };
    unsigned par0 = 0, par1 = 0, par2 = 0;  // the sites' phases
    int cur = 0;                            // which of the two y holds
    // y = P^T r anew from the residual: at the start, and in FP32 every eighth
    // iteration, so that y does not drift from the rounded r (y's own recurrence is FP64)
    auto renew = [&]() {
        double c[6] = {0, 0, 0, 0, 0, 0}, none[1];
        if (t < nr) {
            const VT r[3] = {rs[0], rs[1], rs[2]};
            restrict_node<VT>(soff[t], __float_as_uint(soff[t].w), r, c);
        }
#pragma unroll
        for (int m = 0; m < 6; m++) {
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) c[m] += __shfl_xor_sync(0xffffffffu, c[m], s);
            if (lane == 0) sh->part[t >> 5][m] = c[m];
        }
        const bool here = exchange<2, 6, 0, CL>(none, sh, G, ++epoch, a.box, par2, 0, syc + 2 * nc, a.wait_ns);
        par2 ^= 1u;
        coarse(true, 0.0, nullptr, syc + cur * nc);
        return here;
    };
    constexpr int kZBytes = sizeof(VT) == 4 ? 16 : 24;
    bool ok = true;
    double d1[1] = {0.0}, acc[2];
    if constexpr (TL) ok = renew();
    precondition();
    ok = exchange<1, 2, 2, CL>(acc, sh, G, ++epoch, a.box, par1, nh * kZBytes, nullptr, a.wait_ns) && ok;
    par1 ^= 1u;
    double rz = acc[0], rr = acc[1], pq = 0.0, alpha = 0.0, beta = 0.0;
    const double bnorm2 = rr;
    const double te = eta2 * rr, tol2 = te > abs_tol2 ? te : abs_tol2;
    int it = 0, breakdown = 0;
    bool done = !ok || rr <= tol2 || a.maxit <= 0;
    // Cluster form: no barrier lies between the sums and the threads that use them, and
    // where a wait ran out they may differ, so what ends the solve is agreed on at one
    // place, the barrier behind the border columns.
    // threads without a row take the border columns first
    const int nru = (nr + 31) & ~31;
    const int th = t >= nru ? t - nru : t + kT - nru;
    while (CL || !done) {
        // p at the range's own and border columns
        const VT bt = (VT)beta;
        if (t < nr && !(CL && done)) {
            VT* pc = sp + P * t;
#pragma unroll
            for (int k = 0; k < 3; k++) pc[k] = zs[k] + bt * pc[k];
        }
        for (int k = CL && done ? nh : th; k < nh; k += kT) {
            VT zz[3];
            if constexpr (CL) {
#pragma unroll
                for (int m = 0; m < 3; m++) zz[m] = sz[4 * k + m];
            } else {
                const u64* q = a.zg + Z * (size_t)shalo[k];
                u64 w[Z];
                bool here;
                Patience wait(a.wait_ns);
                do {
                    here = true;
#pragma unroll
                    for (int m = 0; m < Z; m += 2) ld_words(q + m, w[m], w[m + 1]);
#pragma unroll
                    for (int m = 0; m < Z; m++) here = here && has(w[m], epoch);
                } while (!here && wait.more(a.wait_ns));
                if (!here) sh->late = 1;
                if constexpr (sizeof(VT) == 4) {
#pragma unroll
                    for (int m = 0; m < 3; m++) zz[m] = (VT)__uint_as_float((unsigned)w[m]);
                } else {
#pragma unroll
                    for (int m = 0; m < 3; m++) zz[m] = (VT)join(w[2 * m], w[2 * m + 1]);
                }
            }
            VT* pc = sp + P * (nr + k);
#pragma unroll
            for (int m = 0; m < 3; m++) pc[m] = zz[m] + bt * pc[m];
        }
        // a block barrier does not bring lanes together that left the loop apart,
        // and a warp in pieces runs what follows once per piece
        __syncwarp();
        if constexpr (CL) {
            if (__syncthreads_or(done)) break;
        } else {
            __syncthreads();
        }
        // the coming beta's divisor, on a warp that has time: every thread has read the
        // last one before this barrier and reads this one after the sums' barriers
        if (t == kT - 1) sh->irz = 1.0 / rz;
        double pqw = 0.0, yw[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int base = 0; base + (t & ~31) / LPR < nr; base += NG) {
            const int i = base + g;
            VT a0 = VT(0), a1 = VT(0), a2 = VT(0), p0, p1, p2;
            if (base == 0) {
#pragma unroll
                for (int j = 0; j < R; j++) {
                    ld_p<VT>(sp + hc[j], p0, p1, p2);
                    a0 += hv[j][0] * p0 + hv[j][1] * p1 + hv[j][2] * p2;
                    a1 += hv[j][3] * p0 + hv[j][4] * p1 + hv[j][5] * p2;
                    a2 += hv[j][6] * p0 + hv[j][7] * p1 + hv[j][8] * p2;
                }
            }
            if (i < nr) {
                const int o0 = sov[i], n = sov[i + 1] - o0;
                for (int k = sl; k < n; k += LPR) {
                    VT h[9];
                    if (o0 + k < pl.res_blocks) {
#pragma unroll
                        for (int e = 0; e < 9; e++) h[e] = sval[9 * (o0 + k) + e];
                    } else {
#pragma unroll
                        for (int e = 0; e < 9; e++) h[e] = __ldg(a.H + 9 * (size_t)(sgb[i] + k) + e);
                    }
                    ld_p<VT>(sp + P * (int)scol[o0 + k], p0, p1, p2);
                    a0 += h[0] * p0 + h[1] * p1 + h[2] * p2;
                    a1 += h[3] * p0 + h[4] * p1 + h[5] * p2;
                    a2 += h[6] * p0 + h[7] * p1 + h[8] * p2;
                }
            }
#pragma unroll
            for (int s = LPR / 2; s > 0; s >>= 1) {
                a0 += __shfl_xor_sync(0xffffffffu, a0, s);
                a1 += __shfl_xor_sync(0xffffffffu, a1, s);
                a2 += __shfl_xor_sync(0xffffffffu, a2, s);
            }
            if (i < nr) {
                if (sl == 0) { sq[3 * i] = a0; sq[3 * i + 1] = a1; sq[3 * i + 2] = a2; }
                ld_p<VT>(sp + P * i, p0, p1, p2);
                pqw += (double)p0 * (double)a0 + (double)p1 * (double)a1 + (double)p2 * (double)a2;
                if constexpr (TL) {
                    const float4 d = soff[i];
                    const unsigned f = __float_as_uint(d.w);
                    VT q[3] = {a0, a1, a2};
                    project<VT>(f >> 8, a.pn + r0 + i, q);
                    restrict_node<VT>(d, f, q, yw);
                }
            }
        }
        // every lane of a group has its rows' share of the sums: add the warp's groups
#pragma unroll
        for (int s = 16; s >= LPR; s >>= 1) {
            pqw += __shfl_xor_sync(0xffffffffu, pqw, s);
            if constexpr (TL)
#pragma unroll
                for (int m = 0; m < 6; m++) yw[m] += __shfl_xor_sync(0xffffffffu, yw[m], s);
        }
        if (lane == 0) {
            sh->part[t >> 5][0] = pqw;
            if constexpr (TL)
#pragma unroll
                for (int m = 0; m < 6; m++) sh->part[t >> 5][1 + m] = yw[m];
        }
        ok = exchange<0, TL ? kMsg : 1, 1, CL>(d1, sh, G, ++epoch, a.box, par0, 0, syc + 2 * nc, a.wait_ns);
        par0 ^= 1u;
        if (!CL && !ok) break;
        pq = d1[0];
        breakdown = !(pq > 0.0);
        if (!CL && breakdown) break;
        alpha = rz / pq;
        const VT al = (VT)alpha;
        if (t < nr && !(CL && breakdown)) {
            VT q[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                x[k] += al * sp[P * t + k];
                q[k] = sq[3 * t + k];
            }
            project<VT>(pf, a.pn + row, q);
#pragma unroll
            for (int k = 0; k < 3; k++) rs[k] -= al * q[k];
        }
        if constexpr (TL) {
            if (sizeof(VT) == 4 && (it & 7) == 7) {
                ok = renew() && ok;
                if (!CL && !ok) break;
            } else {
                coarse(false, (double)al, syc + cur * nc, syc + (cur ^ 1) * nc);
                cur ^= 1;
            }
        }
        precondition();
        ok = exchange<1, 2, 2, CL>(acc, sh, G, ++epoch, a.box, par1, nh * kZBytes, nullptr, a.wait_ns) && ok;
        par1 ^= 1u;
        if (!CL && !ok) break;
        beta = acc[0] * sh->irz;
        rr = acc[1];
        it++;
        done = rr <= tol2 || it >= a.maxit || !(rr == rr);
        if (CL && (breakdown || !ok)) {
            it -= breakdown;
            done = true;
        } else {
            rz = acc[0];
        }
    }
    if (t < nr) {
#pragma unroll
        for (int k = 0; k < 3; k++) a.x[3 * row + k] = x[k];
        if (breakdown) {
            // the direction of non-positive curvature, where the caller looks for it
            VT* pb = ((it & 1) ? a.p0 : a.p1) + 4 * row;
#pragma unroll
            for (int k = 0; k < 3; k++) pb[k] = sp[P * t + k];
        }
    }
    // no block leaves while another may still push into its shared memory: a solve that
    // ends by its sums has received all that was sent to it, one that a wait ended stays
    // for what may be on its way
    if constexpr (CL) {
        cg::this_cluster().sync();
        if (t == 0 && sh->abort)
            for (const u64 t0 = clock_ns(); clock_ns() - t0 < kStayNs;) {}
    } else {
        __syncthreads();
    }
    // a wait of any block that ran out fails the solve
    if (t == 0 && (sh->abort | sh->late)) atomicOr(&a.sc->status, kFlagTimeout);
    if (me == 0 && t == 0) {
        DevScalars* sc = a.sc;
        sc->rz = rz; sc->rr = rr; sc->bnorm2 = bnorm2; sc->tol2 = tol2; sc->pq = pq;
        sc->alpha = breakdown ? 0.0 : alpha; sc->beta = beta;
        sc->it = it; sc->maxit = a.maxit; sc->breakdown = breakdown; sc->done = 1; sc->skip = 0;
        if (!CL) *a.epoch = epoch;
    }
}

template <typename VT, int LPR, int R, bool CL, bool TL>
int launch_one(const ResidentPlan& pl, const ResidentArgs<VT>& a, cudaStream_t st) {
    auto kern = k_pcg_resident<VT, LPR, R, CL, TL>;
    static std::atomic<int> done[kMaxDevices];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kMaxDevices || !done[dev].load(std::memory_order_relaxed)) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kResidentSmem);
        if (e == cudaSuccess && CL) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return (int)e;
        if (dev >= 0 && dev < kMaxDevices) done[dev].store(1, std::memory_order_relaxed);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.G);
    cfg.blockDim = dim3(kT);
    cfg.dynamicSmemBytes = pl.smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    if (CL) {
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = pl.G;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    } else {
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, pl, a);
    if (e != cudaSuccess) return (int)e;
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    return 0;
}

template <typename VT, bool CL, bool TL>
int launch_shape(const ResidentPlan& pl, const ResidentArgs<VT>& a, cudaStream_t st) {
    if (pl.lpr == 8)
        return pl.reg == 2 ? launch_one<VT, 8, 2, CL, TL>(pl, a, st) : launch_one<VT, 8, 4, CL, TL>(pl, a, st);
    if constexpr (sizeof(VT) == 4)
        if (pl.lpr == 2) return launch_one<VT, 2, 8, CL, TL>(pl, a, st);
    return launch_one<VT, 4, 4, CL, TL>(pl, a, st);
}

}  // namespace

// Shared memory of a plan's block with `res` matrix blocks in it.
size_t resident_smem(const ResidentPlan& pl, int vsize, int res) {
    const int at = vsize == 4 ? offsets<float>(pl).sval : offsets<double>(pl).sval;
    return (size_t)at + 9 * (size_t)res * vsize;
}

template <typename VT>
int launch_pcg_resident(const ResidentPlan& pl, const ResidentArgs<VT>& a, cudaStream_t st) {
    if (a.Ainv)
        return pl.cluster ? launch_shape<VT, true, true>(pl, a, st) : launch_shape<VT, false, true>(pl, a, st);
    return pl.cluster ? launch_shape<VT, true, false>(pl, a, st) : launch_shape<VT, false, false>(pl, a, st);
}
template int launch_pcg_resident<float>(const ResidentPlan&, const ResidentArgs<float>&, cudaStream_t);
template int launch_pcg_resident<double>(const ResidentPlan&, const ResidentArgs<double>&, cudaStream_t);

}  // namespace sors
