// Batched FP64 eigenvalues of complex Hermitian matrices (reduced density
// matrices), and the von Neumann entropy from them.
//
// Reference behaviour reproduced: the FP64 spectrum of rho_A and
// S_vN = -sum lambda log2 lambda over lambda > 1e-15, |S| < 1e-12 -> 0
// (cpp/src/cuda/tmi_cuda_svd.cu:663-798 with its FP64 retry :458-561, and
// cpp/include/mipt/tmi/linalg.hpp:125-132). The reference gets the spectrum
// from cuSOLVER (heevd / gesvd); here it is computed by two kernels of our
// own, written from the textbook algorithms:
//
//   k_tridiag_cluster  Householder reduction of the Hermitian matrix to a
//               real symmetric tridiagonal matrix, up to 256 rows: the matrix
//               stays in the shared memory of a cluster of CTAs. A step
//               reflects the vector x beside the diagonal onto alpha e_1 with
//               H = I - beta v v^H, v = x - alpha e_1,
//               alpha = -phase(x_0) |x|, beta = 2 / |v|^2, and updates the
//               block B that is left, B <- H B H, as B - v w^H - w v^H with
//               p = beta B v, K = beta/2 v^H p, w = p - K v. The off-diagonal
//               |alpha| is kept (a Hermitian tridiagonal matrix with complex
//               off-diagonals is unitarily similar to the real one with their
//               moduli).
//   k_tridiag   the same for up to 4096 rows, the matrix (row-major,
//               interleaved re/im, the lower triangle read and updated) in
//               global memory: one CTA per matrix, or several with barriers
//               between them.
//   k_tridiag_sturm  one thread or a few lanes per eigenvalue (tridiag.cuh),
//               then the entropy.
//
// All reductions run in a fixed order, so results are reproducible.
// FP64 throughout: GB300's FP64 rate bounds the reduction at about 16/3 d^3
// flops per matrix (full matrix-vector product, lower-triangle update).
#include "observables.cuh"
#include "tridiag.cuh"

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

namespace mg
{
namespace
{
constexpr int kTriThreads = 512;

// Block sum in a fixed order: per-warp shuffle trees, then warp 0 sums the
// warp totals. `red` holds at least 32 doubles. Every thread gets the sum.
__device__ double block_sum(double v, double *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads(); // red is free (previous readers are done)
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0)
    {
        double t = lane < nw ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

// Barrier among the `parts` CTAs of one matrix (multi-CTA reduction): a
// monotonic arrival counter, so epoch e is complete when it reaches
// (e + 1) * parts. The wait is bounded; a wait that runs out sets bit 2 of
// *err and makes every CTA of the matrix return.
__device__ bool parts_barrier(unsigned *ctr, unsigned parts, unsigned &epoch, int *err, int *s_ok)
{
    __syncthreads();
    if (threadIdx.x == 0)
    {
        int ok = 1;
        __threadfence();
        atomicAdd(ctr, 1u);
        const unsigned target = (epoch + 1) * parts;
        const std::uint64_t t0 = device_ns();
        for (unsigned it = 0; *reinterpret_cast<volatile unsigned *>(ctr) < target; ++it)
        {
            if (it > (1u << 24) || ((it & 15u) == 15u && device_ns() - t0 > 2000000000ull))
            {
                atomicOr(err, 2);
                ok = 0;
                break;
            }
            if (it > 32) __nanosleep(128);
        }
        __threadfence();
        *s_ok = ok;
    }
    ++epoch;
    __syncthreads();
    return *s_ok != 0;
}

// Householder tridiagonalisation. parts == 1: one CTA per matrix. parts > 1
// (cooperative launch, all CTAs resident): CTA `part` of a matrix owns the
// trailing-block rows i with i % parts == part; every CTA computes the
// reflector, |x| and K itself from the same data in the same order (so all
// agree bit for bit), the rows' p = beta B v go through pglob, and two
// barriers per step order the row updates against the next step's reads.
__global__ void __launch_bounds__(kTriThreads)
    k_tridiag(double2 *__restrict__ mats, int d, double *__restrict__ diag, double *__restrict__ off, int parts,
              double2 *__restrict__ pglob, unsigned *__restrict__ bars, int *__restrict__ err,
              const int *__restrict__ dims, int least)
{
    extern __shared__ double2 sh[];
    double2 *v = sh;     // Householder vector (length m)
    double2 *w = sh + d; // p, then w
    __shared__ double red[33];
    __shared__ int s_ok;
    const int mat = blockIdx.x / parts, part = blockIdx.x % parts;
    double2 *a = mats + static_cast<std::size_t>(mat) * d * d;
    double *dg = diag + static_cast<std::size_t>(mat) * d;
    double *of = off + static_cast<std::size_t>(mat) * d;
    double2 *pg = parts > 1 ? pglob + static_cast<std::size_t>(mat) * d : nullptr;
    unsigned *bar = parts > 1 ? bars + mat : nullptr;
    unsigned epoch = 0;
    const int tid = threadIdx.x, nt = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    // Rows that hold data (the rest of the d x d block is zero: their
    // eigenvalues are 0). The row stride stays d.
    const int dm = dims != nullptr ? dims[mat] : d;
    if (dm <= least) return; // k_tridiag_cluster's

    for (int j = 0; j + 1 < dm; ++j)
    {
        const int m = dm - 1 - j, r0 = j + 1;
        __syncthreads(); // the previous step's reads of v[] and w[] are done
        // x = column j below the diagonal (the lower triangle is the valid
        // half of the trailing block).
        double part_sum = 0.0;
        for (int i = tid; i < m; i += nt)
        {
            const double2 x = a[static_cast<std::size_t>(r0 + i) * d + j];
            v[i] = x;
            if (i > 0) part_sum += x.x * x.x + x.y * x.y;
        }
        const double sigma = block_sum(part_sum, red); // also orders the v[] writes
        const double2 x0 = v[0];
        const double ax0 = hypot(x0.x, x0.y);
        const double norm = sqrt(ax0 * ax0 + sigma);
        if (tid == 0 && part == 0)
        {
            dg[j] = a[static_cast<std::size_t>(j) * d + j].x;
            of[j] = norm;
        }
        if (m == 1 || sigma == 0.0) continue; // already tridiagonal in this column (a phase only)
        const double2 ph = ax0 > 0.0 ? make_double2(x0.x / ax0, x0.y / ax0) : make_double2(1.0, 0.0);
        const double beta = 2.0 / ((ax0 + norm) * (ax0 + norm) + sigma);
        __syncthreads(); // every thread has read v[0]
        if (tid == 0) v[0] = make_double2(ph.x * (ax0 + norm), ph.y * (ax0 + norm));
        __syncthreads();
        // p = beta * B v on this CTA's rows, one warp per row. Only the lower
        // triangle of B is kept: row i supplies B_ik for k <= i, column i
        // (conj(B_ki), a strided read) the rest. Four independent accumulator
        // pairs per lane keep the FP64 pipe busy.
        for (int i = part + warp * parts; i < m; i += nw * parts)
        {
            const double2 *row = a + static_cast<std::size_t>(r0 + i) * d + r0;
            const double2 *col = a + static_cast<std::size_t>(r0) * d + r0 + i;
            double sr[4] = {0.0, 0.0, 0.0, 0.0}, si[4] = {0.0, 0.0, 0.0, 0.0};
            auto acc = [&](int kk, double &ar, double &ai) {
                double2 bk;
                if (kk <= i)
                    bk = row[kk];
                else
                {
                    const double2 t = col[static_cast<std::size_t>(kk) * d];
                    bk = make_double2(t.x, -t.y);
                }
                const double2 x = v[kk];
                ar = fma(bk.x, x.x, ar);
                ar = fma(-bk.y, x.y, ar);
                ai = fma(bk.x, x.y, ai);
                ai = fma(bk.y, x.x, ai);
            };
            int k = lane;
            for (; k + 96 < m; k += 128)
            {
#pragma unroll
                for (int u = 0; u < 4; ++u) acc(k + 32 * u, sr[u], si[u]);
            }
#pragma unroll
            for (int u = 0; u < 3; ++u)
                if (k + 32 * u < m) acc(k + 32 * u, sr[u], si[u]);
            double tr = (sr[0] + sr[1]) + (sr[2] + sr[3]);
            double ti = (si[0] + si[1]) + (si[2] + si[3]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                tr += __shfl_xor_sync(0xffffffffu, tr, o);
                ti += __shfl_xor_sync(0xffffffffu, ti, o);
            }
            if (lane == 0)
            {
                const double2 pv = make_double2(beta * tr, beta * ti);
                if (pg)
                    pg[i] = pv;
                else
                    w[i] = pv;
            }
        }
        if (pg)
        {
            if (!parts_barrier(bar, parts, epoch, err, &s_ok)) return;
            for (int i = tid; i < m; i += nt) w[i] = pg[i];
        }
        __syncthreads();
        // K = beta/2 Re(v^H p) (real for Hermitian B).
        part_sum = 0.0;
        for (int i = tid; i < m; i += nt) part_sum += v[i].x * w[i].x + v[i].y * w[i].y;
        const double K = 0.5 * beta * block_sum(part_sum, red);
        for (int i = tid; i < m; i += nt) w[i] = make_double2(w[i].x - K * v[i].x, w[i].y - K * v[i].y);
        __syncthreads();
        // B <- B - v w^H - w v^H on this CTA's rows of the trailing block's
        // lower triangle: b -= v_i conj(w_k) + w_i conj(v_k), eight FMAs per
        // entry (the diagonal's imaginary parts cancel exactly).
        for (int i = part + warp * parts; i < m; i += nw * parts)
        {
            double2 *row = a + static_cast<std::size_t>(r0 + i) * d + r0;
            const double2 vi = v[i], wi = w[i];
#pragma unroll 4
            for (int k = lane; k <= i; k += 32)
            {
                const double2 wk = w[k], vk = v[k];
                double2 b = row[k];
                b.x = fma(-vi.x, wk.x, b.x);
                b.x = fma(-vi.y, wk.y, b.x);
                b.x = fma(-wi.x, vk.x, b.x);
                b.x = fma(-wi.y, vk.y, b.x);
                b.y = fma(-vi.y, wk.x, b.y);
                b.y = fma(vi.x, wk.y, b.y);
                b.y = fma(-wi.y, vk.x, b.y);
                b.y = fma(wi.x, vk.y, b.y);
                row[k] = b;
            }
        }
        if (pg && !parts_barrier(bar, parts, epoch, err, &s_ok)) return;
    }
    if (tid == 0 && part == 0)
    {
        dg[dm - 1] = a[static_cast<std::size_t>(dm - 1) * d + dm - 1].x;
        of[dm - 1] = 0.0;
        for (int i = dm; i < d; ++i) dg[i] = of[i] = 0.0;
    }
}

// The same reduction with the matrix resident in shared memory: one cluster
// of C CTAs per matrix, CTA r holding the lower-triangle rows i = r (mod C)
// packed. Rows are eliminated from the last one up, so the block that is left
// always starts at row and column 0 (aligned with the lanes) and the row that
// gives the next reflector lies in one CTA. One sweep over the lower triangle
// per step applies the previous step's rank-2 update and accumulates p = B v
// for this one, from each entry both as B_ik and as conj(B_ki): sixteen FP64
// FMAs per entry read and written once. A lane owns columns k = lane (mod 32):
// the column sums stay in registers over a warp's rows, and the row sums of
// two rows share one six-add shuffle tree.
// The partial p and the next pivot row go round the cluster in two steps, each
// behind a cluster barrier: every CTA sends each other one its part of a
// segment of the columns, and the segment's CTA sends the sums to all. Remote
// traffic is slow: sixteen CTAs that each sent everything to everyone spent
// 13k of a step's 31.5k clocks on it, and a remote load takes about 800.
// What bounds it is the FP64 pipe (a warp instruction takes 20 clocks of an
// SM, however many lanes are on), so whatever is not the sweep runs on as few
// warps as hold data: the reflector's roots and divisions on one warp, sums on
// the warps below row m. Of a step of a 256-row matrix on sixteen CTAs the
// sweep and its column sums take about half, the reflector a fifth, the
// exchange a fifth.
// With a work list, a cluster takes either one matrix of more than 128 rows,
// all its CTAs on it, or one smaller matrix per CTA: measured sites leave the
// spectra of one batch at different sizes, and the launch lasted as long as
// its few full-size ones took on four SMs each while most of the others idled
// (34 launches of 64 matrices of up to 256 rows 259 -> 251 ms: full-size ones
// are now one or two waves of clusters of eight).
// Measured against the reduction in global memory: 34 launches of 64 matrices
// of up to 256 rows 533 -> 228 ms, 48 launches of 800 of up to 64 rows
// 156 -> 57 ms, one of 256 rows 5.4 -> 3.4 ms. (Before the exchange by segments
// and the single instance of the block's code: 251, 62 and 3.8 ms.)
template <int NCB, int THREADS>
__global__ void __launch_bounds__(THREADS)
    k_tridiag_cluster(const double2 *__restrict__ mats, int d, double *__restrict__ diag, double *__restrict__ off,
                      const int *__restrict__ dims, const int *__restrict__ list, int nb)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    int C = static_cast<int>(cluster.num_blocks()), r = static_cast<int>(cluster.block_rank());
    int mat = blockIdx.x / C;
    if (list != nullptr)
    {
        // list[0], list[1]: large and small matrices; the large ones from
        // list[2] up, the small ones from list[nb + 1] down.
        if (mat < list[0])
            mat = list[2 + mat];
        else
        {
            const int i = (mat - list[0]) * C + r;
            if (i >= list[1]) return;
            mat = list[nb + 1 - i];
            C = 1;
            r = 0;
        }
    }
    constexpr int NW = THREADS / 32;
    constexpr int NP = (32 * NCB + THREADS - 1) / THREADS;
    extern __shared__ __align__(16) double2 csm[];
    constexpr int DS = 32 * NCB;                                  // >= d; every lane may read a vector
    double2 *v = csm, *vp = v + DS, *wp = vp + DS, *prow = wp + DS; // reflector, previous v and w, row sums
    double2 *pcw = prow + DS;                                     // [NW][DS] column sums per warp
    // C > 1: the pivot row, p, and this CTA's segment of both as it comes in
    // ([C][segment] partial p) and as it goes out.
    double2 *pivot = pcw + NW * DS, *pfull = pivot + DS, *part = pfull + DS, *rowseg = part + DS + 16;
    double2 *pseg = rowseg + DS / 2;
    double2 *rows = C > 1 ? pseg + DS / 2 : pcw + NW * DS;        // packed rows
    __shared__ double red[NW], s_nt, s_beta;
    const double2 *a = mats + static_cast<std::size_t>(mat) * d * d;
    double *dg = diag + static_cast<std::size_t>(mat) * d;
    double *of = off + static_cast<std::size_t>(mat) * d;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int dm = dims != nullptr ? dims[mat] : d;
    // Local row li is row li * C + r and starts at row_at(li, r).
    auto row_at = [C](int li, int rr) { return li * (rr + 1) + C * (li * (li - 1) / 2); };
    auto warp_sum = [](double x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    };
    // Sum of red[0 .. active) in every lane of a warp.
    auto red_sum = [&](int active) {
        double x = lane < active ? red[lane] : 0.0;
#pragma unroll
        for (int o = NW / 2; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return __shfl_sync(0xffffffffu, x, 0);
    };

    for (int li = warp; li * C + r < dm; li += NW)
    {
        const int i = li * C + r;
        for (int k = lane; k <= i; k += 32) rows[row_at(li, r) + k] = a[static_cast<std::size_t>(i) * d + k];
    }
    for (int k = tid; k < DS; k += THREADS) v[k] = vp[k] = wp[k] = make_double2(0.0, 0.0);
    if (C > 1)
    {
        // The first pivot row goes to every CTA.
        __syncthreads();
        if ((dm - 1) % C == r)
            for (int k = tid; k < dm; k += THREADS)
            {
                const double2 t = rows[row_at((dm - 1) / C, r) + k];
                for (int q = 0; q < C; ++q) cluster.map_shared_rank(pivot, q)[k] = t;
            }
        cluster.sync();
    }
    else
        __syncthreads();

    for (int m = dm - 1; m >= 1; --m)
    {
        // Row m with the previous update applied; x = its conjugate transpose.
        const double2 *rm = C > 1 ? pivot : rows + row_at(m, 0);
        const int aw = (m + 31) / 32 < NW ? (m + 31) / 32 : NW; // warps with an entry below m
        if (warp < aw)
        {
            const double2 vm = vp[m], wm = wp[m];
            double s = 0.0;
            for (int k = tid; k < m; k += THREADS)
            {
                const double2 b = rm[k], pv = vp[k], pw = wp[k];
                double2 x;
                x.x = b.x - (vm.x * pw.x + vm.y * pw.y) - (wm.x * pv.x + wm.y * pv.y);
                x.y = -(b.y - (vm.y * pw.x - vm.x * pw.y) - (wm.y * pv.x - wm.x * pv.y));
                v[k] = x;
                if (k < m - 1) s += x.x * x.x + x.y * x.y;
            }
            s = warp_sum(s);
            if (lane == 0) red[warp] = s;
        }
        __syncthreads();
        if (warp == 0)
        {
            const double sigma = red_sum(aw);
            const double2 x0 = v[m - 1];
            const double s0 = x0.x * x0.x + x0.y * x0.y;
            // Roots from reciprocal roots (440 clocks; a division takes 650);
            // hypot where the square is near underflow.
            double ax0, ir;
            if (s0 > 1e-280)
            {
                ir = rsqrt(s0);
                ax0 = s0 * ir;
            }
            else
            {
                ax0 = hypot(x0.x, x0.y);
                ir = ax0 > 0.0 ? 1.0 / ax0 : 0.0;
            }
            const bool reflect = !(sigma <= 1e-280); // else tridiagonal in this row already (NaN goes on)
            const double t2 = s0 + sigma;
            const double norm = reflect ? t2 * rsqrt(t2) : ax0;
            const double top = ax0 + norm;
            __syncwarp();
            if (lane == 0)
            {
                if (r == 0)
                {
                    const double2 vm = vp[m], wm = wp[m];
                    dg[m] = rm[m].x - 2.0 * (vm.x * wm.x + vm.y * wm.y);
                    of[m - 1] = norm;
                }
                v[m - 1] = ir > 0.0 ? make_double2(x0.x * ir * top, x0.y * ir * top) : make_double2(top, 0.0);
                s_nt = reflect ? norm * top : 0.0; // |v|^2 / 2
            }
        }
        __syncthreads();
        if (m == 1) break;
        const double nt = s_nt;
        // beta is needed after the sweep: one warp divides meanwhile.
        if (warp == NW - 1 && lane == 0) s_beta = nt > 0.0 ? 1.0 / nt : 0.0;
        if (!(nt > 0.0))
        {
            // No reflector, but the sweep still applies the previous update; a
            // NaN comes here too and stays one.
            for (int k = tid; k < m; k += THREADS) v[k] = make_double2(0.0 * nt, 0.0 * nt);
            __syncthreads();
        }

        // The sweep: pairs of local rows dealt to the warps in snake order.
        double2 pc[NCB];
#pragma unroll
        for (int c = 0; c < NCB; ++c) pc[c] = make_double2(0.0, 0.0);
        const int lrows = m > r ? (m - r + C - 1) / C : 0; // local rows below m
        const int pairs = (lrows + 1) / 2;
        for (int t = 0; t * NW < pairs; ++t)
        {
            const int g = (t & 1) ? t * NW + NW - 1 - warp : t * NW + warp;
            if (g >= pairs) continue;
            const int l0 = 2 * g, l1 = 2 * g + 1;
            const int i0 = l0 * C + r, i1 = l1 < lrows ? l1 * C + r : -1;
            double2 *q0 = rows + row_at(l0, r), *q1 = rows + row_at(l1, r);
            const double2 v0 = v[i0], vp0 = vp[i0], wp0 = wp[i0];
            const int ic = i1 < 0 ? i0 : i1;
            const double2 v1 = v[ic], vp1 = vp[ic], wp1 = wp[ic];
            double s0r = 0.0, s0i = 0.0, s1r = 0.0, s1i = 0.0;
            // One instance of the block's code per column block (a variant per
            // block count let more of them overlap, but the code outgrew the
            // instruction cache: 3.6 ms for one 256-row matrix against 3.4).
#pragma unroll
            for (int c = 0; c < NCB; ++c)
            {
                if (32 * c > ic) break;
                const int k = 32 * c + lane;
                const double2 vk = v[k], vpk = vp[k], wpk = wp[k];
                // Entries past the diagonal load and add zeros.
                auto entry = [&](double2 *q, int i, double2 vi, double2 vpi, double2 wpi, double &sr, double &si) {
                    double2 b = make_double2(0.0, 0.0);
                    if (k <= i) b = q[k];
                    b.x = fma(-vpi.x, wpk.x, b.x);
                    b.x = fma(-vpi.y, wpk.y, b.x);
                    b.x = fma(-wpi.x, vpk.x, b.x);
                    b.x = fma(-wpi.y, vpk.y, b.x);
                    b.y = fma(-vpi.y, wpk.x, b.y);
                    b.y = fma(vpi.x, wpk.y, b.y);
                    b.y = fma(-wpi.y, vpk.x, b.y);
                    b.y = fma(wpi.x, vpk.y, b.y);
                    b.x = k <= i ? b.x : 0.0;
                    b.y = k < i ? b.y : 0.0;
                    if (k <= i) q[k] = b;
                    sr = fma(b.x, vk.x, sr);
                    sr = fma(-b.y, vk.y, sr);
                    si = fma(b.x, vk.y, si);
                    si = fma(b.y, vk.x, si);
                    const double bx = k < i ? b.x : 0.0;
                    pc[c].x = fma(bx, vi.x, pc[c].x);
                    pc[c].x = fma(b.y, vi.y, pc[c].x);
                    pc[c].y = fma(bx, vi.y, pc[c].y);
                    pc[c].y = fma(-b.y, vi.x, pc[c].y);
                };
                entry(q0, i0, v0, vp0, wp0, s0r, s0i);
                entry(q1, i1, v1, vp1, wp1, s1r, s1i);
            }
            // Four sums over the warp: value (lane >> 3) ends in its lanes.
            const bool up = lane & 16, up2 = lane & 8;
            double x = up ? s1r : s0r, y = up ? s1i : s0i;
            x += __shfl_xor_sync(0xffffffffu, up ? s0r : s1r, 16);
            y += __shfl_xor_sync(0xffffffffu, up ? s0i : s1i, 16);
            double z = up2 ? y : x;
            z += __shfl_xor_sync(0xffffffffu, up2 ? x : y, 8);
            z += __shfl_xor_sync(0xffffffffu, z, 4);
            z += __shfl_xor_sync(0xffffffffu, z, 2);
            z += __shfl_xor_sync(0xffffffffu, z, 1);
            if ((lane & 7) == 0)
            {
                const int i = up ? i1 : i0;
                if (i >= 0) reinterpret_cast<double *>(prow + i)[up2 ? 1 : 0] = z;
            }
        }
        const int sw = pairs < NW ? pairs : NW; // warps that swept rows
        if (warp < sw)
        {
#pragma unroll
            for (int c = 0; c < NCB; ++c)
                if (32 * c + lane < m) pcw[warp * DS + 32 * c + lane] = pc[c];
        }
        __syncthreads();
        double2 p[NP];
        if (warp < aw)
        {
#pragma unroll
            for (int u = 0; u < NP; ++u)
            {
                const int k = u * THREADS + tid;
                p[u] = make_double2(0.0, 0.0);
                if (k >= m) continue;
                if (k % C == r) p[u] = prow[k];
#pragma unroll
                for (int q = 0; q < NW; ++q)
                {
                    if (q >= sw) break;
                    const double2 t = pcw[q * DS + k];
                    p[u].x += t.x;
                    p[u].y += t.y;
                }
            }
        }
        if (C > 1)
        {
            const int seg = (m + C - 1) / C; // columns r * seg .. of CTA r
            const bool owner = (m - 1) % C == r;
            const double2 *next = rows + row_at((m - 1) / C, r);
#pragma unroll
            for (int u = 0; u < NP; ++u)
            {
                const int k = u * THREADS + tid;
                if (k >= m) continue;
                const int q = k / seg, e = k - q * seg;
                cluster.map_shared_rank(part, q)[r * seg + e] = p[u];
                if (owner) cluster.map_shared_rank(rowseg, q)[e] = next[k];
            }
            cluster.sync();
            if (tid < seg && r * seg + tid < m)
            {
                double2 a0 = make_double2(0.0, 0.0), a1 = a0;
                for (int q = 0; q < C; q += 2)
                {
                    const double2 t0 = part[q * seg + tid], t1 = part[(q + 1) * seg + tid];
                    a0.x += t0.x;
                    a0.y += t0.y;
                    a1.x += t1.x;
                    a1.y += t1.y;
                }
                pseg[tid] = make_double2(a0.x + a1.x, a0.y + a1.y);
            }
            __syncthreads();
            for (int t = tid; t < seg * C; t += THREADS)
            {
                const int q = t / seg, e = t - q * seg, k = r * seg + e;
                if (k >= m) continue;
                cluster.map_shared_rank(pfull, q)[k] = pseg[e];
                cluster.map_shared_rank(pivot, q)[k] = rowseg[e];
            }
            cluster.sync();
#pragma unroll
            for (int u = 0; u < NP; ++u)
                if (u * THREADS + tid < m) p[u] = pfull[u * THREADS + tid];
        }
        const double beta = s_beta;
        // p = beta B v, K = beta/2 Re(v^H p) (real for Hermitian B), w = p - K v.
        if (warp < aw)
        {
            double s = 0.0;
#pragma unroll
            for (int u = 0; u < NP; ++u)
            {
                const int k = u * THREADS + tid;
                if (k >= m) continue;
                p[u].x *= beta;
                p[u].y *= beta;
                s += v[k].x * p[u].x + v[k].y * p[u].y;
            }
            s = warp_sum(s);
            if (lane == 0) red[warp] = s;
        }
        __syncthreads();
        if (warp < aw)
        {
            const double K = 0.5 * beta * red_sum(aw);
#pragma unroll
            for (int u = 0; u < NP; ++u)
            {
                const int k = u * THREADS + tid;
                if (k >= m) continue;
                const double2 vk = v[k];
                vp[k] = vk;
                wp[k] = make_double2(p[u].x - K * vk.x, p[u].y - K * vk.y);
            }
        }
        __syncthreads();
    }
    if (tid == 0 && r == 0)
    {
        // Row 0 (local row 0 of CTA 0) with the last update.
        dg[0] = rows[0].x - 2.0 * (vp[0].x * wp[0].x + vp[0].y * wp[0].y);
        of[dm - 1] = 0.0;
        for (int i = dm; i < d; ++i) dg[i] = of[i] = 0.0;
    }
    if (C > 1) cluster.sync(); // no CTA leaves while another may write to it
}

// Work list of k_tridiag_cluster: matrices of at most kSmallRows rows, those of
// up to kClusterRows, and (left out) larger ones. The order within a class is
// not fixed; every matrix is reduced the same way whatever its place.
constexpr int kSmallRows = 128, kClusterRows = 256;

__global__ void __launch_bounds__(256) k_eig_list(const int *__restrict__ dims, int d, int nb, int *__restrict__ list)
{
    __shared__ int count[2];
    if (threadIdx.x < 2) count[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += blockDim.x)
    {
        const int dm = dims != nullptr ? dims[i] : d;
        if (dm <= kSmallRows)
            list[nb + 1 - atomicAdd(&count[1], 1)] = i;
        else if (dm <= kClusterRows)
            list[2 + atomicAdd(&count[0], 1)] = i;
    }
    __syncthreads();
    if (threadIdx.x < 2) list[threadIdx.x] = count[threadIdx.x];
}

// Eigenvalues of every reduced matrix, 2^gl threads per eigenvalue (grid:
// matrices x chunks of blockDim threads), and the entropy terms
// -lambda log2 lambda over lambda > 1e-15; with one chunk per matrix the sum
// too. The implicit QL iteration that this replaces is one serial chain of
// about d^2 plane rotations per matrix at GB300's 64-clock FP64 latency. The 34
// launches of 64 matrices of up to 256 rows: QL 972 ms, this 43 ms; one matrix
// of 256 rows: 1.4 to 20 ms, this 0.33 ms.
constexpr double kEigCutoff = 1e-15;

__global__ void __launch_bounds__(128)
    k_tridiag_sturm(const double *__restrict__ diag, const double *__restrict__ off, int d, double *__restrict__ terms,
                    double *__restrict__ entropy, int *__restrict__ err, const int *__restrict__ dims, int gl)
{
    extern __shared__ __align__(16) double2 de[];
    float2 *df = reinterpret_cast<float2 *>(de + d);
    __shared__ double red[33];
    const int jb = blockIdx.x;
    const int dm = dims != nullptr ? dims[jb] : d;
    const double *dg = diag + static_cast<std::size_t>(jb) * d;
    const double *of = off + static_cast<std::size_t>(jb) * d;
    // |T| (largest row sum; a NaN or an infinity anywhere makes `sum` one). The
    // search runs on the matrix times a power of four that brings |T| into
    // [1/4, 1), so the counts' range does not depend on the state's norm; a
    // power of four also scales the search's geometric means exactly.
    double top = 0.0, sum = 0.0;
    for (int i = threadIdx.x; i < dm; i += blockDim.x)
    {
        const double e0 = i > 0 ? fabs(of[i - 1]) : 0.0, e1 = i + 1 < dm ? fabs(of[i]) : 0.0;
        const double t = fabs(dg[i]) + e0 + e1;
        top = fmax(top, t);
        sum += t;
    }
    sum = block_sum(sum, red);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = top;
    __syncthreads();
    top = red[0];
    for (int q = 1; q < static_cast<int>(blockDim.x >> 5); ++q) top = fmax(top, red[q]);
    const bool finite = sum - sum == 0.0;
    int shift = 0;
    if (finite && top > 0.0) frexp(top, &shift);
    shift = shift < -1000 ? -1000 : shift + (shift & 1); // below 2^-1000 every eigenvalue is under the cut-off
    const double scale = scalbn(1.0, -shift);
    top *= scale;
    const double floor2 = kTinyE2 * top * top, inv = top > 0.0 ? 1.0 / top : 0.0;
    for (int i = threadIdx.x; i < dm; i += blockDim.x)
    {
        const double e = i > 0 ? of[i - 1] * scale : 0.0;
        de[i] = make_double2(dg[i] * scale, i > 0 ? fmax(e * e, floor2) : 0.0);
        df[i] = sturm_entry32(de[i], inv, i);
    }
    __syncthreads();
    const int at = blockIdx.y * blockDim.x + threadIdx.x, idx = at >> gl;
    const bool writes = (at & ((1 << gl) - 1)) == 0;
    const double bound = top * (1.0 + 1e-14), cutoff = kEigCutoff * scale;
    double term = 0.0, l = 0.0;
    if (gl > 0 && finite && top > 0.0)
        l = sturm_eigenvalue_lanes(de, df, dm, idx < dm ? idx : dm - 1, top, bound, cutoff, gl, idx < dm);
    else if (finite && top > 0.0 && idx < dm)
        l = sturm_eigenvalue(de, df, dm, idx, top, bound, cutoff);
    if (finite && writes && idx < dm)
    {
        l = scalbn(l, shift);
        if (l > kEigCutoff) term = -l * log2(l);
    }
    if (!finite && blockIdx.y == 0 && threadIdx.x == 0) atomicOr(err, 1);
    if (gridDim.y == 1)
    {
        const double s = block_sum(term, red);
        if (threadIdx.x == 0) entropy[jb] = !finite ? NAN : (fabs(s) < 1e-12 ? 0.0 : s);
    }
    else if (writes && idx < d)
        terms[static_cast<std::size_t>(jb) * d + idx] = finite ? term : NAN;
}

// entropy[job] = the sum of its d terms (fixed order).
__global__ void __launch_bounds__(128) k_entropy_sum(const double *__restrict__ terms, int d, double *__restrict__ entropy)
{
    __shared__ double red[33];
    double s = 0.0;
    for (int i = threadIdx.x; i < d; i += blockDim.x) s += terms[static_cast<std::size_t>(blockIdx.x) * d + i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) entropy[blockIdx.x] = fabs(s) < 1e-12 ? 0.0 : s;
}

// Shared memory of k_tridiag_cluster for d rows over C CTAs.
std::size_t cluster_smem(int d, int C, int warps)
{
    const int lr = d / C, vectors = 4 + warps + (C > 1 ? 4 : 0);
    const std::size_t packed = static_cast<std::size_t>(lr) * C + static_cast<std::size_t>(C) * lr * (lr - 1) / 2;
    return sizeof(double2) * (packed + static_cast<std::size_t>(vectors) * std::max(d, 32) + (C > 1 ? 16 : 0));
}

template <int NCB, int THREADS>
cudaError_t launch_cluster(const double2 *rho, int d, int nb, int C, double *diag, double *off, cudaStream_t s,
                           const int *dims, const int *list = nullptr)
{
    // With a list, a CTA may also hold a small matrix by itself.
    const std::size_t smem = std::max(cluster_smem(32 * NCB, C, THREADS / 32),
                                      list ? cluster_smem(kSmallRows, 1, 0) + sizeof(double2) * (4 + THREADS / 32) * 32 * NCB
                                           : std::size_t{0});
    cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void *>(&k_tridiag_cluster<NCB, THREADS>), smem);
    if (e != cudaSuccess) return e;
    if (C > 8)
    {
        e = cudaFuncSetAttribute(k_tridiag_cluster<NCB, THREADS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(nb * C);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_tridiag_cluster<NCB, THREADS>, rho, d, diag, off, dims, list, nb);
}
} // namespace

std::size_t hermitian_eig_scratch_doubles(int d, int nb)
{
    // diag and off (d each), p vectors (2 d), barrier counters (1 double
    // each, used as unsigned), the work list (nb + 2 ints).
    return (4 * static_cast<std::size_t>(d) + 2) * nb + 1;
}

cudaError_t hermitian_eig_entropy(double *rho, int d, int nb, double *entropy_out, double *scratch,
                                  int *err, cudaStream_t s, const int *dims, int *launched)
{
    if (launched) *launched = 0;
    if (nb <= 0) return cudaSuccess;
    if (d < 2 || d > 4096) return cudaErrorInvalidValue;
    double *diag = scratch;
    double *off = scratch + static_cast<std::size_t>(d) * nb;
    double2 *pglob = reinterpret_cast<double2 *>(scratch + 2 * static_cast<std::size_t>(d) * nb);
    unsigned *bars = reinterpret_cast<unsigned *>(scratch + 4 * static_cast<std::size_t>(d) * nb);
    int *list = reinterpret_cast<int *>(scratch + (4 * static_cast<std::size_t>(d) + 1) * nb);
    int kernels = 0;
    int dev = 0, sms = 0;
    cudaError_t e = cudaSuccess;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 152;
    const double2 *r2 = reinterpret_cast<const double2 *>(rho);
    if (d <= 128)
    {
        // One CTA holds the matrix; more, down to 16 rows each, while SMs
        // would stay idle.
        int C = 1;
        while (C < 16 && nb * C * 2 <= sms && d / (2 * C) >= 16) C *= 2;
        e = d <= 32   ? launch_cluster<1, 32>(r2, d, nb, C, diag, off, s, dims)
            : d == 64 ? launch_cluster<2, 128>(r2, d, nb, C, diag, off, s, dims)
                      : launch_cluster<4, 256>(r2, d, nb, C, diag, off, s, dims);
        ++kernels;
    }
    else if (d == 256 && nb * 16 <= sms)
    {
        e = launch_cluster<8, 256>(r2, d, nb, 16, diag, off, s, dims);
        ++kernels;
    }
    else if (d == 256 || dims != nullptr)
    {
        k_eig_list<<<1, 256, 0, s>>>(dims, d, nb, list);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = launch_cluster<8, 256>(r2, d, nb, 8, diag, off, s, dims, list);
        kernels += 2;
    }
    if (e != cudaSuccess) return e;
    if (d > 256)
    {
        int least = dims != nullptr ? kClusterRows : 0;
        ++kernels;
        const std::size_t smem = 2 * sizeof(double2) * d;
        e = allow_dynamic_smem(reinterpret_cast<const void *>(&k_tridiag), smem);
        if (e != cudaSuccess) return e;
        // Fewer matrices than SMs: spread each matrix over `parts` resident CTAs
        // (cooperative launch), at least 16 trailing rows per CTA.
        int per_sm = 0, parts = 1;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tridiag, kTriThreads, smem) == cudaSuccess &&
            per_sm > 0)
        {
            const int resident = sms * per_sm;
            parts = std::max(1, std::min({resident / nb, d / 16, 64}));
        }
        cudaGetLastError();
        if (parts > 1)
        {
            e = cudaMemsetAsync(bars, 0, sizeof(unsigned) * nb, s);
            if (e != cudaSuccess) return e;
            int dd = d;
            void *args[] = {&rho, &dd, &diag, &off, &parts, &pglob, &bars, &err, &dims, &least};
            e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(&k_tridiag), dim3(nb * parts),
                                            dim3(kTriThreads), args, smem, s);
        }
        else
        {
            k_tridiag<<<nb, kTriThreads, smem, s>>>(reinterpret_cast<double2 *>(rho), d, diag, off, 1, nullptr, nullptr,
                                                    err, dims, least);
            e = cudaGetLastError();
        }
    }
    if (e != cudaSuccess) return e;
    // One thread per eigenvalue: CTAs of up to 128, or of one warp each while
    // that spreads a few matrices over idle SMs (two warps of one SM would
    // share its FP64 pipe). Four to 32 lanes per eigenvalue while the warps are
    // still no more than the SMs: one matrix of 256 rows (16 lanes, 128 warps)
    // 0.91 -> 0.33 ms. With more warps than that the FP64 pipes
    // are busy, and one lane's search needs the fewest counts in all; two lanes
    // would narrow a bracket only threefold per count.
    int gl = 0;
    while (gl < 5 && (static_cast<long long>(nb) * d << (gl + 1)) <= 32ll * sms) ++gl;
    if (gl < 2) gl = 0;
    const long long warps = static_cast<long long>(nb) * ((d + 31) / 32);
    const int tpb = gl > 0 || warps <= 2 * sms ? 32 : std::min(128, (d + 31) / 32 * 32);
    const int chunks = ((d << gl) + tpb - 1) / tpb;
    const std::size_t sm = (sizeof(double2) + sizeof(float2)) * d;
    e = allow_dynamic_smem(reinterpret_cast<const void *>(&k_tridiag_sturm), sm);
    if (e != cudaSuccess) return e;
    // The terms take the place of the p vectors, which the reduction is done with.
    double *terms = reinterpret_cast<double *>(pglob);
    k_tridiag_sturm<<<dim3(nb, chunks), tpb, sm, s>>>(diag, off, d, terms, entropy_out, err, dims, gl);
    e = cudaGetLastError();
    if (launched) *launched = kernels + (chunks == 1 ? 1 : 2);
    if (e != cudaSuccess || chunks == 1) return e;
    k_entropy_sum<<<nb, 128, 0, s>>>(terms, d, entropy_out);
    return cudaGetLastError();
}

} // namespace mg
