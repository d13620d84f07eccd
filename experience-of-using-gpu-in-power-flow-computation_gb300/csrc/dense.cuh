// dense.cuh -- the dense linear solve of metodo = denso: the Newton Jacobian as
// a dense FP64 matrix, LU with partial pivoting and the two triangular solves,
// in place of the dense Jacobian kernels (GPU/Jacobiano.cuh:33-222) and the
// cusolverDnXgetrf / getrs calls (GPU/newtonRaphson.cuh:507-530) of the
// reference.  Included by solver.cu after its Dev / Ctl definitions.
//
// The matrix has the sparse path's superset form: 2 x 2 blocks per non-slack
// bus in block order (rows P_j, Q_j; columns theta_j, V_j), a PV bus below its
// limits keeps an identity Q row and a zero V column.  Its solution equals that
// of the reference's reduced system (P rows of the non-slack buses, Q rows of
// the PQ list), so N = 2 (nB - 1) stays fixed while buses switch and the whole
// solve is one static CUDA graph.  Column-major, leading dimension N, with the
// right-hand side as column N, which the LU's interchanges, triangular solves
// and updates carry through the forward substitution.
//
// getrf here is right-looking and blocked by kDPanel columns, three launches a
// panel: the panel factorisation (pivot = first row of largest magnitude, as
// LAPACK's idamax) on a thread-block cluster (k_dpanel_cl), the panel's row
// interchanges on the other columns with U12 = L11^-1 A12 (k_dswap), and the
// Schur update A22 -= L21 U12 (k_dgemm).  Measured per Newton iteration on
// GB300, panel on one block, separate interchanges and forward substitution ->
// this form: N = 112 0.60 -> 0.31 ms, 234 1.38 -> 0.68 ms, 942 9.0 -> 3.2 ms,
// 1,886 38 -> 9.5 ms, 3,774 148 -> 43 ms; of the 9.2 ms of LU at N = 1,886 the
// Schur updates take about 4.6 (the FP64 pipes' floor is 4.2) and the panels 4.
#pragma once

constexpr int kDPanel = 32;
constexpr int kDPanelThreads = 1024;
constexpr int kDBackThreads = 512;

// Zero the matrix (fill-in positions of a previous pass) and the step's max|dx|.
__global__ void k_dzero(Dev d, int guard) {
    if (stopped(d, guard)) return;
    const long long total = (long long)d.N * d.N / 2;  // N is even
    double2 *A2 = reinterpret_cast<double2 *>(d.A);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x)
        A2[i] = make_double2(0.0, 0.0);
    if (blockIdx.x == 0 && threadIdx.x == 0) d.ctl->maxDx = 0ull;
}

// One thread per bus row: the 2 x 2 blocks of row k (k_jfill's formulas) at
// the dense positions of (block of k, block of m), and its right-hand side.
__global__ void k_dfill(Dev d, int guard) {
    if (stopped(d, guard)) return;
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= d.nB || k == d.slack) return;
    const int N = d.N, jr = d.blk_of_bus[k];
    const double Vk = d.V[k];
    const int ak = d.act[k];
    for (int p = d.yptr[k]; p < d.yptr[k + 1]; p++) {
        const int m = d.ycol[p];
        if (m == d.slack) continue;
        const int jc = d.blk_of_bus[m];
        const double2 y = d.yval[p];
        double H, Nn, M, L;
        if (m == k) {
            const double P = d.P[k], Q = d.Q[k], v2 = Vk * Vk;
            H = -Q - v2 * y.y;
            if (ak) { Nn = (P + v2 * y.x) / Vk; M = P - v2 * y.x; L = (Q - v2 * y.y) / Vk; }
            else { Nn = 0.0; M = 0.0; L = 1.0; }
        } else {
            const int am = d.act[m];
            const double ck = d.cs[k], sk = d.sn[k], cm = d.cs[m], sm = d.sn[m];
            const double tr = y.x * cm - y.y * sm, ti = y.x * sm + y.y * cm;
            const double wr = ck * tr + sk * ti, wi = sk * tr - ck * ti;
            const double Vm = d.V[m];
            H = Vk * Vm * wi;
            Nn = am ? Vk * wr : 0.0;
            M = ak ? -Vk * Vm * wr : 0.0;
            L = (ak && am) ? Vk * wi : 0.0;
        }
        double *c0 = d.A + (size_t)(2 * jc) * N, *c1 = c0 + N;
        c0[2 * jr] = H;
        c1[2 * jr] = Nn;
        c0[2 * jr + 1] = M;
        c1[2 * jr + 1] = L;
    }
    *(double2 *)(d.A + (size_t)N * N + 2 * jr) = d.rhs[jr];
}

// Panel factorisation of columns k0 .. k0 + nb - 1 over rows k0 .. N - 1, one
// block, for panels too tall for k_dpanel_cl: for each column the pivot search, the interchange inside the panel,
// the scaling of the column below the pivot and the rank-1 update of the
// panel's remaining columns.  A zero or non-finite pivot ends the solve with
// GBPF_E_SINGULAR.
__global__ void __launch_bounds__(kDPanelThreads) k_dpanel(Dev d, int k0, int guard) {
    if (stopped(d, guard)) return;
    __shared__ double sval[kDPanelThreads / 32];
    __shared__ int sidx[kDPanelThreads / 32];
    __shared__ int spiv;
    const int N = d.N, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nb = min(kDPanel, N - k0);
    double *A = d.A;
    for (int jj = 0; jj < nb; jj++) {
        const int j = k0 + jj;
        double *cj = A + (size_t)j * N;
        double best = -1.0;
        int bi = N;
        for (int r = j + tid; r < N; r += kDPanelThreads) {
            double v = fabs(cj[r]);
            if (v != v) v = INFINITY;
            if (v > best) { best = v; bi = r; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) { sval[warp] = best; sidx[warp] = bi; }
        __syncthreads();
        if (tid == 0) {
            double b = sval[0];
            int p = sidx[0];
            for (int w = 1; w < kDPanelThreads / 32; w++)
                if (sval[w] > b || (sval[w] == b && sidx[w] < p)) { b = sval[w]; p = sidx[w]; }
            if (!(b > 0.0) || !isfinite(b) || p >= N) {
                d.ctl->status = GBPF_E_SINGULAR;
                d.ctl->done = 1;
                p = j;
            }
            d.ipiv[j] = p;
            spiv = p;
        }
        __syncthreads();
        const int p = spiv;
        if (p != j)
            for (int c = k0 + tid; c < k0 + nb; c += kDPanelThreads) {
                double *col = A + (size_t)c * N;
                const double t = col[j];
                col[j] = col[p];
                col[p] = t;
            }
        __syncthreads();
        const double pv = cj[j];
        for (int r = j + 1 + tid; r < N; r += kDPanelThreads) cj[r] /= pv;
        __syncthreads();
        for (int c = j + 1; c < k0 + nb; c++) {
            double *col = A + (size_t)c * N;
            const double u = col[j];
            for (int r = j + 1 + tid; r < N; r += kDPanelThreads) col[r] -= cj[r] * u;
        }
        __syncthreads();
    }
}

// The same panel factorisation on a cluster, the panel's rows dealt in runs of
// rp >= kDPanel rows to the CTAs' shared memory.  What bounds it is the FP64
// pipe: R x 32 x 16 multiply-adds took one SM 0.5 ms of a 0.6 ms panel at R =
// 1,400; sixteen share them here.  A column costs one cluster barrier: each CTA
// pushes its candidate pivot row (and CTA 0 the row that trades places with
// the pivot) to all CTAs, which after the barrier all find the same winner,
// scale and update their rows, and find their candidate of the next column.
// About 4,400 cycles a column, most of it the chain search - push - barrier;
// pushing a candidate before the rest of the update was slower (N = 1,886: LU
// 9.1 -> 9.5 ms), since the extra multiply-adds of the pushed rows hold the
// FP64 pipe.
// The pivot search is an argmax on the integer order of |a| (NaN counted as
// +inf, the first row of the largest magnitude wins, as idamax); the scaling
// takes the pivot's reciprocal, or divides where the pivot is below the normal
// range and its reciprocal may not be finite (as LAPACK's dgetf2 does).  Four
// threads a row, columns interleaved over them.
constexpr int kDPanClT = 512, kDPanLd = 36;  // row stride in doubles: 8 rows x 4 threads meet each bank pair twice
constexpr int kDPanRows = 736;               // most rows of a CTA (212 KB)
struct DPanMsg {
    double cand[16][kDPanel], inv[16], rowj[kDPanel];
    unsigned long long key[16];
    int idx[16];
};
constexpr unsigned long long kMinNormal = 0x0010000000000000ull;  // key of 2^-1022
__device__ __forceinline__ unsigned long long dabs_key(double v) {
    unsigned long long k = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
    return k > 0x7ff0000000000000ull ? 0x7ff0000000000000ull : k;  // NaN -> +inf
}
__device__ __forceinline__ void cl_put_i(unsigned a, int v) {
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void cl_put_u64(unsigned a, unsigned long long v) {
    asm volatile("st.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
// largest key of the warp and the lowest row that has it
__device__ __forceinline__ void warp_argmax(unsigned long long &key, int &row) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
    const unsigned long long k = (unsigned long long)hi << 32 | lo;
    row = (int)__reduce_min_sync(0xffffffffu, key == k ? (unsigned)row : 0x7fffffffu);
    key = k;
}
__global__ void __launch_bounds__(kDPanClT, 1) k_dpanel_cl(Dev d, int k0, int rp, int guard) {
    extern __shared__ __align__(16) double P[];  // rp rows of kDPanLd
    __shared__ DPanMsg msg[2];
    __shared__ unsigned long long wkey[kDPanClT / 32];
    __shared__ int widx[kDPanClT / 32], s_stop;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5, rank = (int)cluster_rank(), C = gridDim.x;
    if (t == 0) s_stop = stopped(d, guard);
    __syncthreads();
    const int stop = s_stop;
    cluster_sync();  // every CTA has read the flag before a singular pivot may set it
    if (stop) return;
    const int N = d.N, R = N - k0, nb = min(kDPanel, R), lo = rank * rp, cnt = max(0, min(rp, R - lo));
    double *A = d.A + (size_t)k0 * N + k0 + lo;
    for (int c = wp; c < nb; c += kDPanClT / 32)
        for (int r = lane; r < cnt; r += 32) P[r * kDPanLd + c] = A[(size_t)c * N + r];
    __syncthreads();
    bool sing = false;
    // this CTA's candidate of column j from the threads' (key, row), its row and
    // row j to every CTA
    auto publish = [&](int j, unsigned long long key, int row) {
        DPanMsg &m = msg[j & 1];
        warp_argmax(key, row);
        if (lane == 0) { wkey[wp] = key; widx[wp] = row; }
        __syncthreads();
        key = lane < kDPanClT / 32 ? wkey[lane] : 0;
        row = lane < kDPanClT / 32 ? widx[lane] : 0x7fffffff;
        warp_argmax(key, row);
        const bool have = row < cnt;
        for (int q = wp; q < C; q += kDPanClT / 32) {
            if (have) cl_put(cl_map(&m.cand[rank][lane], q), P[row * kDPanLd + lane]);
            if (rank == 0) cl_put(cl_map(&m.rowj[lane], q), P[j * kDPanLd + lane]);
            if (lane == 0) {
                cl_put_u64(cl_map(&m.key[rank], q), have ? key : 0ull);
                cl_put_i(cl_map(&m.idx[rank], q), have ? lo + row : 0x7fffffff);
            }
        }
        if (wp == 0 && have) {
            const double inv = rcp_rn(P[row * kDPanLd + j]);
            if (lane < C) cl_put(cl_map(&m.inv[rank], lane), inv);
        }
        __syncwarp();
        cluster_sync();
    };
    {
        unsigned long long key = 0;
        int row = 0x7fffffff;
        for (int r = t; r < cnt; r += kDPanClT) {
            const unsigned long long k = dabs_key(P[r * kDPanLd]);
            if (row == 0x7fffffff || k > key) { key = k; row = r; }
        }
        publish(0, key, row);
    }
    const int ch = t & 3;
    for (int j = 0; j < nb; j++) {
        const DPanMsg &m = msg[j & 1];
        unsigned long long key = lane < C ? m.key[lane] : 0;
        int p = lane < C ? m.idx[lane] : 0x7fffffff;
        const unsigned long long mine = key;
        const int at = p;
        warp_argmax(key, p);
        const int w = __ffs(__ballot_sync(0xffffffffu, mine == key && at == p && lane < C)) - 1;
        if (key == 0 || key >= 0x7ff0000000000000ull) sing = true;
        if (rank == 0 && t == 0) d.ipiv[k0 + j] = k0 + p;
        const double *pr = m.cand[w], inv = m.inv[w];
        const bool tiny = key < kMinNormal;
        if (rank == 0 && wp == kDPanClT / 32 - 1) P[j * kDPanLd + lane] = pr[lane];  // row j is the pivot row now
        unsigned long long nkey = 0;
        int nrow = 0x7fffffff;
        for (int r = t >> 2; r - (lane >> 2) < cnt; r += kDPanClT / 4) {
            const int g = lo + r;
            const bool on = r < cnt && g > j, sw = g == p && p != j;  // row p takes row j's place
            double *row = P + r * kDPanLd;
            const double *src = sw ? m.rowj : row;
            double l = on ? src[j] * inv : 0.0;
            if (tiny && on) l = src[j] / pr[j];
            __syncwarp();
            if (on) {
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int c = 4 * u + ch;
                    if (4 * u + 3 > j && c > j && c < nb) {
                        const double v = __fma_rn(-l, pr[c], src[c]);
                        row[c] = v;
                        if (c == j + 1) {
                            const unsigned long long k = dabs_key(v);
                            if (nrow == 0x7fffffff || k > nkey) { nkey = k; nrow = r; }
                        }
                    }
                    if (c < j && sw) row[c] = src[c];
                    if (c == j) row[c] = l;
                }
            }
        }
        if (j + 1 < nb) publish(j + 1, nkey, nrow);
    }
    __syncthreads();
    if (sing && t == 0 && rank == 0) {
        d.ctl->status = GBPF_E_SINGULAR;
        d.ctl->done = 1;
    }
    for (int c = wp; c < nb; c += kDPanClT / 32)
        for (int r = lane; r < cnt; r += 32) A[(size_t)c * N + r] = P[r * kDPanLd + c];
}

// The panel's interchanges on every other column (the right-hand side with
// them) and, behind the panel, U12 = L11^-1 A12 (L11 unit lower triangular):
// one warp a column.  The interchanges are applied as one permutation of the
// at most 64 rows they touch, made from the pivot list by each block's first
// warp, so a column costs two loads and two stores a lane.
__global__ void __launch_bounds__(256) k_dswap(Dev d, int k0, int guard) {
    if (stopped(d, guard)) return;
    __shared__ double L11[kDPanel][kDPanel + 1];
    __shared__ int s_top[kDPanel], s_row[kDPanel], s_src[kDPanel];
    const int N = d.N, nb = min(kDPanel, N - k0), k1 = k0 + nb, t = threadIdx.x, lane = t & 31, wp = t >> 5;
    if (wp == 0) {
        // top: which row is in place `lane` of the panel's first nb; row / src:
        // a row below them that changes and which row it takes
        int top = lane, row = -1, src = -1, used = 0;
        const int piv = lane < nb ? d.ipiv[k0 + lane] - k0 : 0;
        for (int j = 0; j < nb; j++) {
            const int p = __shfl_sync(0xffffffffu, piv, j), tj = __shfl_sync(0xffffffffu, top, j);
            if (p < nb) {
                const int tp = __shfl_sync(0xffffffffu, top, p);
                if (lane == j) top = tp;
                else if (lane == p) top = tj;
            } else {
                const unsigned has = __ballot_sync(0xffffffffu, row == p);
                const int e = has ? __ffs(has) - 1 : used++;
                if (!has && lane == e) { row = p; src = p; }
                const int se = __shfl_sync(0xffffffffu, src, e);
                if (lane == j) top = se;
                if (lane == e) src = tj;
            }
        }
        s_top[lane] = top;
        s_row[lane] = row;
        s_src[lane] = src;
    }
    for (int i = t; i < nb * nb; i += 256) {
        const int r = i % nb, c = i / nb;
        L11[r][c] = d.A[(size_t)(k0 + c) * N + k0 + r];
    }
    __syncthreads();
    int c = blockIdx.x * 8 + wp;
    if (c >= k0) c += nb;
    if (c > N) return;
    double *col = d.A + (size_t)c * N + k0;
    const int row = s_row[lane];
    double x = lane < nb ? col[s_top[lane]] : 0.0;
    const double o = row >= 0 ? col[s_src[lane]] : 0.0;
    __syncwarp();
    if (c >= k1)
        for (int u = 0; u + 1 < nb; u++) {
            const double xu = __shfl_sync(0xffffffffu, x, u);
            if (lane > u) x = __fma_rn(-L11[lane][u], xu, x);
        }
    if (lane < nb) col[lane] = x;
    if (row >= 0) col[row] = o;
}

// A22 -= L21 U12 on 64 x 32 tiles of rows k1 .. N - 1 and columns k1 .. N (the
// right-hand side the last; K = nb <= 32): 256 threads, 4 x 2 outputs each, both
// operands staged in shared memory.  Bound by the FP64 pipe (a multiply-add of
// a warp holds it 19 cycles); tiles of half the size of 64 x 64 halve the
// last, partly filled round of the SMs.
__global__ void __launch_bounds__(256) k_dgemm(Dev d, int k0, int guard) {
    if (stopped(d, guard)) return;
    __shared__ double Ls[64][kDPanel + 1];
    __shared__ double Us[kDPanel][32 + 1];
    const int N = d.N, nb = min(kDPanel, N - k0), k1 = k0 + nb;
    const int r0 = k1 + blockIdx.y * 64, c0 = k1 + blockIdx.x * 32;
    const int tid = threadIdx.x, tr = (tid / 16) * 4, tc = (tid % 16) * 2;
    for (int i = tid; i < 64 * kDPanel; i += 256) {
        const int r = i % 64, t = i / 64;
        Ls[r][t] = (t < nb && r0 + r < N) ? d.A[(size_t)(k0 + t) * N + r0 + r] : 0.0;
    }
    for (int i = tid; i < kDPanel * 32; i += 256) {
        const int t = i % kDPanel, c = i / kDPanel;
        Us[t][c] = (t < nb && c0 + c <= N) ? d.A[(size_t)(c0 + c) * N + k0 + t] : 0.0;
    }
    double acc[4][2] = {}, old[4][2];
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int q = 0; q < 4; q++)
            old[q][s] = c0 + tc + s <= N && r0 + tr + q < N ? d.A[(size_t)(c0 + tc + s) * N + r0 + tr + q] : 0.0;
    __syncthreads();
    for (int t = 0; t < nb; t++) {
        double a[4], b[2];
#pragma unroll
        for (int q = 0; q < 4; q++) a[q] = Ls[tr + q][t];
#pragma unroll
        for (int s = 0; s < 2; s++) b[s] = Us[t][tc + s];
#pragma unroll
        for (int q = 0; q < 4; q++)
#pragma unroll
            for (int s = 0; s < 2; s++) acc[q][s] = __fma_rn(a[q], b[s], acc[q][s]);
    }
#pragma unroll
    for (int s = 0; s < 2; s++)
#pragma unroll
        for (int q = 0; q < 4; q++)
            if (c0 + tc + s <= N && r0 + tr + q < N)
                d.A[(size_t)(c0 + tc + s) * N + r0 + tr + q] = old[q][s] - acc[q][s];
}

// U x = y on a cluster, y = column N after the LU, x into d.xs: 32-row blocks
// round the CTAs.  For block b from the last: its CTA solves the diagonal block
// (one warp) and pushes the 32 values to all CTAs; behind the barrier every CTA
// takes them out of its blocks above, eight columns of a block to a warp, each
// warp with sums of its own (ys: per block y and four partial sums of 32).  One
// block alone read the factor at one SM's rate: 2.1 ms at N = 1,886.
__global__ void __launch_bounds__(kDBackThreads, 1) k_dback(Dev d, int guard) {
    extern __shared__ double ys[];
    __shared__ double U[kDPanel][kDPanel + 1], xb[2][kDPanel];
    __shared__ int s_stop;
    const int t = threadIdx.x, lane = t & 31, wp = t >> 5, rank = (int)cluster_rank(), C = gridDim.x;
    if (t == 0) s_stop = stopped(d, guard);
    __syncthreads();
    const int stop = s_stop;
    cluster_sync();
    if (stop) return;
    const int N = d.N, nbk = (N + kDPanel - 1) / kDPanel;
    const double *A = d.A;
    for (int b = rank, q = 0; b < nbk; b += C, q++)
        for (int i = t; i < 5 * kDPanel; i += kDBackThreads) {
            const int r = b * kDPanel + i;
            ys[q * 5 * kDPanel + i] = i < kDPanel && r < N ? A[(size_t)N * N + r] : 0.0;
        }
    __syncthreads();
    for (int b = nbk - 1; b >= 0; b--) {
        const int r0 = b * kDPanel, w = min(kDPanel, N - r0);
        if (rank == b % C) {
            for (int i = t; i < w * w; i += kDBackThreads) U[i % w][i / w] = A[(size_t)(r0 + i / w) * N + r0 + i % w];
            __syncthreads();
            if (wp == 0) {
                const double *y = ys + (b / C) * 5 * kDPanel + lane;
                double x = y[0] - ((y[kDPanel] + y[2 * kDPanel]) + (y[3 * kDPanel] + y[4 * kDPanel]));
                const double ud = lane < w ? U[lane][lane] : 1.0, rd = 1.0 / ud;
                auto rows = [&](auto over) {
                    for (int u = w - 1; u >= 0; u--) {
                        if (lane == u) x = over(x);
                        const double xu = __shfl_sync(0xffffffffu, x, u);
                        if (lane < u) x = __fma_rn(-U[lane][u], xu, x);
                    }
                };
                // (reciprocals may not be finite below the normal range: divide)
                if (__any_sync(0xffffffffu, dabs_key(ud) < kMinNormal)) rows([&](double v) { return v / ud; });
                else rows([&](double v) { return v * rd; });
                for (int q = 0; q < C; q++) cl_put(cl_map(&xb[b & 1][lane], q), x);
                if (lane < w) ((double *)d.xs)[r0 + lane] = x;
            }
        }
        cluster_sync();
        if (b == 0) break;
        // own blocks above b, the next one first
        const int last = b - 1 < rank ? -1 : (b - 1 - rank) / C;
        const double *x = xb[b & 1];
        for (int q = last - (wp >> 2); q >= 0; q -= kDBackThreads / 128) {
            const int r = (rank + q * C) * kDPanel + lane, s = wp & 3;
            double v[8], sum = 0.0;
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = 8 * s + u < w ? A[(size_t)(r0 + 8 * s + u) * N + r] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; u++) sum = __fma_rn(v[u], x[8 * s + u], sum);
            ys[(q * 5 + 1 + s) * kDPanel + lane] += sum;
        }
        __syncthreads();
    }
}
