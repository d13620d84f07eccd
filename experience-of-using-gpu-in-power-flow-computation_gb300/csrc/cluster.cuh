// cluster.cuh -- every elimination level of the block LU, the forward and the
// backward substitution of the single-grid solver in one launch of one
// thread-block cluster (in place of the cusolverSpDcsrlsvqr call of
// GPU/newtonRaphson.cuh:455-478).  Included by solver.cu after its Dev / SB
// definitions.
//
// What bounds the factorisation is the chain of levels: a 15,104-bus grid has
// 103 forward and 103 backward levels of a few microseconds' work in total, so
// a kernel per level pays 4-6 us of launch per level.  Here the levels of the
// elimination tree's bottom end in a hardware cluster barrier, and its top --
// long chains of one- or two-pivot levels -- is the segment: its blocks move
// into CTA 0's shared memory, where a level costs two block barriers and no trip
// to L2.  A dense trailing block, the tail, is factored right-looking in shared
// memory, one barrier a step, without gather lists: on CTA 0 in FP32, its
// columns round the cluster in FP64 (pivot columns pushed through distributed
// shared memory), whose work one SM's FP64 pipe cannot carry.  Each CTA reads
// its part of the schedule (gbpf::cluster_schedule: which pivots, entries and rows it
// computes, and their gather lists) from shared memory.
//
// Level equations (Crout, L scaled), k over earlier steps:
//   D_j     = A_jj - sum_k L(j,k) U(k,j),     y_j = b_j - sum_k L(j,k) y_k
//   U(j,i)  = A_ji - sum_k L(j,k) U(k,i),     L(i,j) = (A_ij - sum_k L(i,k) U(k,j)) D_j^-1
//   x_j     = D_j^-1 (y_j - sum_i U(j,i) x_i)
// Measured on GB300 (factorisation and both substitutions of one Newton step,
// kernel per level -> this kernel; a store, a cluster barrier and a load from
// L2 take 2,650 cycles, the barrier alone 480, which is what a cluster level
// cannot go below): 15,104 buses FP64 2.63 -> 0.46 ms, FP32 1.38 -> 0.26 ms;
// 7,552 buses FP64 2.98 -> 0.39 ms, FP32 1.65 -> 0.23 ms; 1,888 buses FP64 0.74
// -> 0.12 ms, FP32 0.37 -> 0.07 ms; a filled 472-bus grid FP64 2.26 -> 0.26 ms,
// FP32 1.23 -> 0.15 ms.  Clusters of 8 CTAs took 0.63 ms on 15,104 buses.
// The gathers of a level's pivots and entries run side by side and meet at a
// block barrier before the entries take D_j^-1; a CTA that has entries of a
// pivot computes that pivot too, so no inverse crosses CTAs within a level.
#pragma once

constexpr int kClT = gbpf::kClusterThreads;

__device__ __forceinline__ float cfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double cfma(double a, double b, double c) { return __fma_rn(a, b, c); }
// c - A B and v - A w, two fused multiply-adds a component
template <typename B4> __device__ __forceinline__ B4 cms(B4 c, B4 a, B4 b) {
    c.x = cfma(-a.y, b.z, cfma(-a.x, b.x, c.x)); c.y = cfma(-a.y, b.w, cfma(-a.x, b.y, c.y));
    c.z = cfma(-a.w, b.z, cfma(-a.z, b.x, c.z)); c.w = cfma(-a.w, b.w, cfma(-a.z, b.y, c.w));
    return c;
}
template <typename B4, typename B2> __device__ __forceinline__ B2 cmvs(B2 v, B4 a, B2 w) {
    v.x = cfma(-a.y, w.y, cfma(-a.x, w.x, v.x));
    v.y = cfma(-a.w, w.y, cfma(-a.z, w.x, v.y));
    return v;
}
template <typename B4> __device__ __forceinline__ B4 cbm(B4 a, B4 b) {
    B4 r;
    r.x = cfma(a.x, b.x, a.y * b.z); r.y = cfma(a.x, b.y, a.y * b.w);
    r.z = cfma(a.z, b.x, a.w * b.z); r.w = cfma(a.z, b.y, a.w * b.w);
    return r;
}
template <typename B4, typename B2> __device__ __forceinline__ B2 cmv(B4 a, B2 v) {
    B2 r;
    r.x = cfma(a.x, v.x, a.y * v.y);
    r.y = cfma(a.z, v.x, a.w * v.y);
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Inverse of a pivot block: in FP64 through one reciprocal (a division is a
// chain of dependent FP64 operations), in FP32 by four divisions, as
// pivot_done does.
__device__ __forceinline__ double4_32a pivot_inv(double4_32a D, double det) {
    const double rd = rcp_rn(det);
    return mk4(D.w * rd, -D.y * rd, -D.z * rd, D.x * rd);
}
__device__ __forceinline__ float4 pivot_inv(float4 D, float det) {
    return make_float4(D.w / det, -D.y / det, -D.z / det, D.x / det);
}

// Where a level's blocks and vectors are: the factor in global memory, or the
// segment's copy in shared memory (same indices: the bases are shifted).
template <typename TJ> struct ClMem {
    using B4 = typename SB<TJ>::b4;
    using B2 = typename SB<TJ>::b2;
    B4 *D;    // diagonal blocks in (segment: their inverses out)
    B4 *Lv, *Uv;
    B4 *inv;  // inverses as the entries' records name them
    B2 *ys;
};
// Whether a gather starts from the block it updates (FP64) or sums the updates
// by themselves and adds them to the block once, which rounds at the size of
// the updates rather than of the block (FP32; in FP64 the four to eight more
// instructions would cost 64 cycles each).
template <typename TJ> constexpr bool kFromBlock = sizeof(TJ) == 8;
// Element q of the schedule's lists (gbpf::ClusterSchedule::packed).
__device__ __forceinline__ int2 cl_pair(const int *sb, int q, int pk) {
    if (pk) {
        const unsigned v = (unsigned)sb[q];
        return make_int2((int)(v & 0xffffu), (int)(v >> 16));
    }
    return ((const int2 *)sb)[q];
}
// What a level does: kLevel = a cluster level (inverses to the CTA's table
// and, from the CTA that stores a pivot, to dinv; y from the right-hand side),
// kGather = the cluster's updates of the segment's blocks (no inverse),
// kSegment = a segment level.
enum ClKind { kLevel = 0, kGather = 1, kSegment = 2 };

// The pivots of a level, one lane a block: groups of 2^g lanes share a pivot,
// stride over its gather list and sum with shuffles.  A warp without a pivot
// skips the sums: an FP64 instruction holds GB300's pipe 16 cycles a warp.
template <typename TJ, int K>
__device__ __forceinline__ bool cl_pivots(const Dev &d, const ClMem<TJ> &m, const int *sb, const int4 *rec, int np,
                                          int g, int lw, int t, int pk) {
    using B4 = typename SB<TJ>::b4;
    using B2 = typename SB<TJ>::b2;
    bool sing = false;
    const int gl = t & ((1 << g) - 1), wf = t >> 5, slot = (t & 31) >> g;
    if (wf >> lw) return false;
    for (int b0 = 0; b0 + wf < np; b0 += (32 >> g) << lw) {
        const int w = b0 + (slot << lw) + wf;
        const bool on = w < np;
        const int4 r = on ? rec[w] : make_int4(0, 0, 0, 0);
        B4 D, D0;
        B2 y, y0;
        D.x = D.y = D.z = D.w = (TJ)0;
        y.x = y.y = (TJ)0;
        D0 = D;
        y0 = y;
        if (on && gl == 0) {
            D0 = m.D[r.x];
            if (K == kSegment) {
                y0 = m.ys[r.x];
            } else {
                const double2 b = d.rhs[r.x];
                y0.x = (TJ)b.x;
                y0.y = (TJ)b.y;
            }
            if (kFromBlock<TJ>) { D = D0; y = y0; }
        }
#pragma unroll 2
        for (int q = r.y + gl; q < r.z; q += 1 << g) {
            const int2 e = cl_pair(sb, q, pk);
            const B4 lj = m.Lv[e.x];
            D = cms(D, lj, m.Uv[e.x]);
            y = cmvs(y, lj, m.ys[e.y]);
        }
        for (int o = (1 << g) >> 1; o > 0; o >>= 1) {
            D.x += __shfl_xor_sync(0xffffffffu, D.x, o);
            D.y += __shfl_xor_sync(0xffffffffu, D.y, o);
            D.z += __shfl_xor_sync(0xffffffffu, D.z, o);
            D.w += __shfl_xor_sync(0xffffffffu, D.w, o);
            y.x += __shfl_xor_sync(0xffffffffu, y.x, o);
            y.y += __shfl_xor_sync(0xffffffffu, y.y, o);
        }
        if (on && gl == 0) {
            if (!kFromBlock<TJ>) {
                D = add4T(D0, D);
                y.x += y0.x;
                y.y += y0.y;
            }
            if (K == kGather) {
                m.D[r.x] = D;
                m.ys[r.x] = y;
            } else {
                const TJ det = D.x * D.w - D.y * D.z;
                sing |= (det == (TJ)0 || !isfinite(det));
                const B4 inv = pivot_inv(D, det);
                if (K == kSegment) {
                    m.D[r.x] = inv;
                    m.ys[r.x] = y;
                } else {
                    m.inv[w] = inv;
                    if (r.w) {
                        dinv_of<TJ>(d)[r.x] = inv;
                        m.ys[r.x] = y;
                    }
                }
            }
        }
    }
    return sing;
}

// The same in FP64 with each 2x2 block on a quad of four lanes (lane c = 2 r +
// s holds component (r, s)): a block product costs a lane two fused
// multiply-adds instead of eight.  One pass.
template <int K>
__device__ __forceinline__ bool cl_pivots_q(const Dev &d, const ClMem<double> &m, const int *sb, const int4 *rec,
                                            int np, int g, int lw, int t, int pk) {
    const int c = t & 3, r = c >> 1, s = c & 1, qb = (t & 31) & ~3;
    const unsigned qm = 0xfu << qb;  // the quad's lanes, which always run together
    const int sA0 = qb + 2 * r, sA1 = sA0 + 1, sB0 = qb + s, sB1 = qb + 2 + s;
    auto comp = [&](const blk4 *p) { return ((const double *)p)[c]; };
    const int gl = ((t & 31) >> 2) & ((1 << g) - 1), wf = t >> 5, w = ((t & 31) >> 2 >> g << lw) + wf;
    if (wf >> lw || wf >= np) return false;
    bool sing = false;
    const bool on = w < np;
    const int4 rc = on ? rec[w] : make_int4(0, 0, 0, 0);
    double D = 0.0, y = 0.0;  // component c of D_j, row r of y_j
    if (on && gl == 0) {
        D = comp(&m.D[rc.x]);
        y = K == kSegment ? ((const double *)&m.ys[rc.x])[r] : ((const double *)&d.rhs[rc.x])[r];
    }
#pragma unroll 2
    for (int q = rc.y + gl; q < rc.z; q += 1 << g) {
        const int2 e = cl_pair(sb, q, pk);
        const double l = comp(&m.Lv[e.x]), u = comp(&m.Uv[e.x]);
        const double2 yk = m.ys[e.y];
        const double l0 = __shfl_sync(qm, l, sA0), l1 = __shfl_sync(qm, l, sA1);
        const double u0 = __shfl_sync(qm, u, sB0), u1 = __shfl_sync(qm, u, sB1);
        D = __fma_rn(-l1, u1, __fma_rn(-l0, u0, D));
        y = __fma_rn(-l1, yk.y, __fma_rn(-l0, yk.x, y));
    }
    for (int o = (1 << g) >> 1; o > 0; o >>= 1) {
        D += __shfl_xor_sync(0xffffffffu, D, 4 * o);
        y += __shfl_xor_sync(0xffffffffu, y, 4 * o);
    }
    if (on && gl == 0) {
        if (K == kGather) {
            ((double *)&m.D[rc.x])[c] = D;
        } else {
            const double Dx = __shfl_sync(qm, D, qb), Dy = __shfl_sync(qm, D, qb + 1);
            const double Dz = __shfl_sync(qm, D, qb + 2), Dw = __shfl_sync(qm, D, qb + 3);
            const double det = Dx * Dw - Dy * Dz;
            sing = (det == 0.0 || !isfinite(det));
            const double inv = (c == 0 ? Dw : c == 1 ? -Dy : c == 2 ? -Dz : Dx) * rcp_rn(det);
            if (K == kSegment) {
                ((double *)&m.D[rc.x])[c] = inv;
            } else {
                ((double *)&m.inv[w])[c] = inv;
                if (rc.w) ((double *)&d.dinv[rc.x])[c] = inv;
            }
        }
        if (s == 0 && (K != kLevel || rc.w)) ((double *)&m.ys[rc.x])[r] = y;
    }
    return sing;
}

// The entries of a level: U(j,i) and the unscaled L(i,j), then L scaled by the
// pivot's inverse.  `one`: the entries fit one pass of the CTA, their sums
// stay in registers across the barrier behind which the inverses are there,
// and the gathers run beside the pivots'; otherwise the barrier comes first.
template <typename TJ, int K>
__device__ __forceinline__ void cl_entries(const ClMem<TJ> &m, const int *sb, const int4 *rec, int ne, int g, int lw,
                                           int t, bool one, int pk) {
    using B4 = typename SB<TJ>::b4;
    const int gl = t & ((1 << g) - 1), slot = (t & 31) >> g, wf = (t >> 5) >> lw ? ne : t >> 5;
    if (!one && K != kGather) __syncthreads();
    B4 aL, aU, L0, U0;
    int4 r = make_int4(0, 0, 0, 0);
    bool store = false;
    for (int b0 = 0; b0 + wf < ne; b0 += (32 >> g) << lw) {
        const int w = b0 + (slot << lw) + wf;
        const bool on = w < ne;
        r = on ? rec[w] : make_int4(0, 0, 0, 0);
        aL.x = aL.y = aL.z = aL.w = (TJ)0;
        aU = L0 = U0 = aL;
        store = on && gl == 0;
        if (store) { L0 = m.Lv[r.x]; U0 = m.Uv[r.x]; }
        if (kFromBlock<TJ>) { aL = L0; aU = U0; }
#pragma unroll 2
        for (int q = r.y + gl; q < r.z; q += 1 << g) {
            const int2 e = cl_pair(sb, q, pk);  // positions of L(j,k) / U(k,j) and of L(i,k) / U(k,i)
            aL = cms(aL, m.Lv[e.y], m.Uv[e.x]);
            aU = cms(aU, m.Lv[e.x], m.Uv[e.y]);
        }
        for (int o = (1 << g) >> 1; o > 0; o >>= 1) {
            aL.x += __shfl_xor_sync(0xffffffffu, aL.x, o);
            aL.y += __shfl_xor_sync(0xffffffffu, aL.y, o);
            aL.z += __shfl_xor_sync(0xffffffffu, aL.z, o);
            aL.w += __shfl_xor_sync(0xffffffffu, aL.w, o);
            aU.x += __shfl_xor_sync(0xffffffffu, aU.x, o);
            aU.y += __shfl_xor_sync(0xffffffffu, aU.y, o);
            aU.z += __shfl_xor_sync(0xffffffffu, aU.z, o);
            aU.w += __shfl_xor_sync(0xffffffffu, aU.w, o);
        }
        if (!kFromBlock<TJ>) { aL = add4T(L0, aL); aU = add4T(U0, aU); }
        if (store && (!one || K == kGather)) {
            m.Uv[r.x] = aU;
            m.Lv[r.x] = K == kGather ? aL : cbm(aL, m.inv[r.w]);
        }
    }
    if (one && K != kGather) {
        __syncthreads();
        if (store) {
            m.Uv[r.x] = aU;
            m.Lv[r.x] = cbm(aL, m.inv[r.w]);
        }
    }
}

// The same in FP64 on quads of lanes (always one pass).
template <int K>
__device__ __forceinline__ void cl_entries_q(const ClMem<double> &m, const int *sb, const int4 *rec, int ne, int g,
                                             int lw, int t, int pk) {
    const int c = t & 3, r = c >> 1, s = c & 1, qb = (t & 31) & ~3;
    const unsigned qm = 0xfu << qb;
    const int sA0 = qb + 2 * r, sA1 = sA0 + 1, sB0 = qb + s, sB1 = qb + 2 + s;
    auto comp = [&](const blk4 *p) { return ((const double *)p)[c]; };
    auto mul_sub = [&](double acc, double a, double b) {  // component c of acc - A B
        const double a0 = __shfl_sync(qm, a, sA0), a1 = __shfl_sync(qm, a, sA1);
        const double b0 = __shfl_sync(qm, b, sB0), b1 = __shfl_sync(qm, b, sB1);
        return __fma_rn(-a1, b1, __fma_rn(-a0, b0, acc));
    };
    const int gl = ((t & 31) >> 2) & ((1 << g) - 1), wf = t >> 5, w = ((t & 31) >> 2 >> g << lw) + wf;
    const bool any = wf < ne && !(wf >> lw), on = any && w < ne;
    const int4 rc = on ? rec[w] : make_int4(0, 0, 0, 0);
    double aL = 0.0, aU = 0.0;
    if (any) {
        if (on && gl == 0) { aL = comp(&m.Lv[rc.x]); aU = comp(&m.Uv[rc.x]); }
#pragma unroll 2
        for (int q = rc.y + gl; q < rc.z; q += 1 << g) {
            const int2 e = cl_pair(sb, q, pk);
            const double lx = comp(&m.Lv[e.x]), ux = comp(&m.Uv[e.x]), ly = comp(&m.Lv[e.y]), uy = comp(&m.Uv[e.y]);
            aL = mul_sub(aL, ly, ux);
            aU = mul_sub(aU, lx, uy);
        }
        for (int o = (1 << g) >> 1; o > 0; o >>= 1) {
            aL += __shfl_xor_sync(0xffffffffu, aL, 4 * o);
            aU += __shfl_xor_sync(0xffffffffu, aU, 4 * o);
        }
    }
    if (K != kGather) __syncthreads();
    if (on && gl == 0) {
        ((double *)&m.Uv[rc.x])[c] = aU;
        if (K != kGather) {
            const double iv = comp(&m.inv[rc.w]);
            const double a0 = __shfl_sync(qm, aL, sA0), a1 = __shfl_sync(qm, aL, sA1);
            const double b0 = __shfl_sync(qm, iv, sB0), b1 = __shfl_sync(qm, iv, sB1);
            aL = __fma_rn(a0, b0, a1 * b1);
        }
        ((double *)&m.Lv[rc.x])[c] = aL;
    }
}

// One CTA's part of a level (header h of its schedule sb).  One block barrier
// inside (none in the gather).
template <typename TJ, int K>
__device__ __forceinline__ bool cl_level(const Dev &d, const ClMem<TJ> &m, const int *sb, const int *h, int t, int pk) {
    const int4 hd = *(const int4 *)h;
    const int cfg = h[4], gp = cfg & 7, ge = (cfg >> 3) & 7, lp = (cfg >> 8) & 7, le = (cfg >> 11) & 7;
    const int te = (t + 32 * (cfg >> 16)) & (kClT - 1);
    const int4 *rp = (const int4 *)(sb + hd.z), *re = (const int4 *)(sb + hd.w);
    bool sing;
    if constexpr (sizeof(TJ) == 8) {
        if (cfg & 64) sing = cl_pivots_q<K>(d, m, sb, rp, hd.x, gp, lp, t, pk);
        else sing = cl_pivots<TJ, K>(d, m, sb, rp, hd.x, gp, lp, t, pk);
        if (cfg & 128) cl_entries_q<K>(m, sb, re, hd.y, ge, le, te, pk);
        else cl_entries<TJ, K>(m, sb, re, hd.y, ge, le, te, (cfg & 16384) != 0, pk);
    } else {
        sing = cl_pivots<TJ, K>(d, m, sb, rp, hd.x, gp, lp, t, pk);
        cl_entries<TJ, K>(m, sb, re, hd.y, ge, le, te, (cfg & 16384) != 0, pk);
    }
    return sing;
}

// One CTA's rows of a backward level: x_j = D_j^-1 (y_j - sum_i U(j,i) x_i);
// x in place of y (xs = ys) in the segment.
template <typename TJ>
__device__ __forceinline__ void cl_back(const typename SB<TJ>::b4 *dinv, const typename SB<TJ>::b4 *Uv,
                                        const typename SB<TJ>::b2 *ys, typename SB<TJ>::b2 *xs, const int *sb,
                                        const int *h, int t, int pk) {
    using B4 = typename SB<TJ>::b4;
    using B2 = typename SB<TJ>::b2;
    const int nr = h[0], g = h[2] & 7, lw = h[2] >> 8, slot = (t & 31) >> g;
    const int4 *rec = (const int4 *)(sb + h[1]);
    const int gl = t & ((1 << g) - 1), wf = t >> 5;
    if (wf >> lw) return;
    for (int b0 = 0; b0 + wf < nr; b0 += (32 >> g) << lw) {
        const int w = b0 + (slot << lw) + wf;
        const bool on = w < nr;
        const int4 r = on ? rec[w] : make_int4(0, 0, 0, 0);
        B4 inv;
        B2 acc;
        acc.x = acc.y = (TJ)0;
        if (on && gl == 0) {
            acc = ys[r.x];
            inv = dinv[r.x];
        }
#pragma unroll 2
        for (int q = r.y + gl; q < r.z; q += 1 << g) {
            const int2 e = cl_pair(sb, q, pk);
            acc = cmvs(acc, Uv[e.x], xs[e.y]);
        }
        for (int o = (1 << g) >> 1; o > 0; o >>= 1) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        }
        if (on && gl == 0) xs[r.x] = cmv(inv, acc);
    }
}

// The segment's updates (steps t0 .. td-1, in shared memory) of the tail's
// blocks and right-hand side, on CTA 0: into the tail's columns (tail != null)
// or into global memory.
template <typename TJ>
__device__ __forceinline__ void cl_seg_gather(const Dev &d, const ClMem<TJ> &m, typename SB<TJ>::b4 *tail, int mt,
                                              int td, const int *sb, const int *h, int t, int pk) {
    using B4 = typename SB<TJ>::b4;
    using B2 = typename SB<TJ>::b2;
    const int cfg = h[4], gp = cfg & 7, ge = (cfg >> 3) & 7, lp = (cfg >> 8) & 7, le = (cfg >> 11) & 7;
    B4 *fac = fac_of<TJ>(d);
    const int4 *rec = (const int4 *)(sb + h[2]);
    const int lane = t & 31, wp = t >> 5;
    for (int b0 = 0; !(wp >> lp) && b0 + wp < h[0]; b0 += (32 >> gp) << lp) {
        const int w = b0 + (lane >> gp << lp) + wp, gl = lane & ((1 << gp) - 1);
        const bool on = w < h[0];
        const int4 r = on ? rec[w] : make_int4(td, 0, 0, 0);
        const int a = r.x - td;
        B4 *D = tail ? tail + a * mt + a : fac + r.x;
        B4 v, v0;
        B2 y, y0;
        v.x = v.y = v.z = v.w = (TJ)0;
        y.x = y.y = (TJ)0;
        v0 = v;
        y0 = y;
        if (on && gl == 0) {
            v0 = *D;
            if (tail) { const B4 q = tail[mt * mt + a]; y0.x = q.x; y0.y = q.z; }
            else y0 = ys_of<TJ>(d)[r.x];
        }
        for (int q = r.y + gl; q < r.z; q += 1 << gp) {
            const int2 e = cl_pair(sb, q, pk);
            const B4 l = m.Lv[e.x];
            v = cms(v, l, m.Uv[e.x]);
            y = cmvs(y, l, m.ys[e.y]);
        }
        for (int o = (1 << gp) >> 1; o > 0; o >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
            v.z += __shfl_xor_sync(0xffffffffu, v.z, o);
            v.w += __shfl_xor_sync(0xffffffffu, v.w, o);
            y.x += __shfl_xor_sync(0xffffffffu, y.x, o);
            y.y += __shfl_xor_sync(0xffffffffu, y.y, o);
        }
        if (on && gl == 0) {
            *D = add4T(v0, v);
            y.x += y0.x;
            y.y += y0.y;
            if (tail) { tail[mt * mt + a].x = y.x; tail[mt * mt + a].z = y.y; }
            else ys_of<TJ>(d)[r.x] = y;
        }
    }
    rec = (const int4 *)(sb + h[3]);
    for (int b0 = 0; !(wp >> le) && b0 + wp < h[1]; b0 += (32 >> ge) << le) {
        const int w = b0 + (lane >> ge << le) + wp, gl = lane & ((1 << ge) - 1);
        const bool on = w < h[1];
        const int4 r = on ? rec[w] : make_int4(0, 0, 0, 0);
        const int i = r.w >> 16, j = r.w & 0xffff;  // block row and column of L, i > j
        B4 *Lt = tail ? tail + j * mt + i : fac + d.n + r.x;
        B4 *Ut = tail ? tail + i * mt + j : fac + d.n + d.nup + r.x;
        B4 aL, aU;
        aL.x = aL.y = aL.z = aL.w = (TJ)0;
        aU = aL;
        for (int q = r.y + gl; q < r.z; q += 1 << ge) {
            const int2 e = cl_pair(sb, q, pk);
            aL = cms(aL, m.Lv[e.y], m.Uv[e.x]);
            aU = cms(aU, m.Lv[e.x], m.Uv[e.y]);
        }
        for (int o = (1 << ge) >> 1; o > 0; o >>= 1) {
            aL.x += __shfl_xor_sync(0xffffffffu, aL.x, o);
            aL.y += __shfl_xor_sync(0xffffffffu, aL.y, o);
            aL.z += __shfl_xor_sync(0xffffffffu, aL.z, o);
            aL.w += __shfl_xor_sync(0xffffffffu, aL.w, o);
            aU.x += __shfl_xor_sync(0xffffffffu, aU.x, o);
            aU.y += __shfl_xor_sync(0xffffffffu, aU.y, o);
            aU.z += __shfl_xor_sync(0xffffffffu, aU.z, o);
            aU.w += __shfl_xor_sync(0xffffffffu, aU.w, o);
        }
        if (on && gl == 0) { *Lt = add4T(*Lt, aL); *Ut = add4T(*Ut, aU); }
    }
}

// --------------------------------------------------------------------- tail
// The tail of order m in shared memory: block column c, rows 0 .. m-1, on CTA
// c % nc at col[(c / nc) m + row]; column m holds the right-hand side (first
// components of two-row blocks).  dt[k] = D_k^-1 on every CTA.  With more than
// one CTA, lb[(k & 1) m + i] is the pivot column of step k and up (CTA 0) the
// strict upper triangle, column c at up[c (c - 1) / 2]; with one (FP32), lb
// holds the columns before the tail's own updates.
template <typename B4> struct ClTail {
    B4 *col, *dt, *lb, *up;
    int m, nc, rank;
};
__device__ __forceinline__ unsigned cl_map(const void *p, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(r)
                 : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void cl_put(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
// this CTA's columns of the tail from global memory
template <typename TJ>
__device__ __forceinline__ void cl_tail_load(const Dev &d, const ClTail<typename SB<TJ>::b4> &T, int td, int t) {
    using B4 = typename SB<TJ>::b4;
    const B4 *fac = fac_of<TJ>(d), *Lv = fac + d.n, *Uv = fac + d.n + d.nup;
    const int m = T.m, pu = d.up_ptr[td];
    if (T.rank >= T.nc) return;
    B4 *dst = T.nc == 1 ? T.lb : T.col;
    const int mine = (m - T.rank + T.nc - 1) / T.nc;
    for (int q = t; q < mine * m; q += kClT) {
        const int c = T.rank + q / m * T.nc, i = q % m;
        const int lo = min(i, c), p = pu + lo * (m - 1) - lo * (lo - 1) / 2 + (max(i, c) - lo - 1);
        dst[q] = i == c ? fac[td + i] : i < c ? Uv[p] : Lv[p];
    }
    if (T.rank == m % T.nc)
        for (int i = t; i < m; i += kClT) {
            const auto y = ys_of<TJ>(d)[td + i];
            B4 b;
            b.x = y.x;
            b.z = y.y;
            b.y = b.w = (TJ)0;
            dst[m / T.nc * m + i] = b;
        }
}
// The inverse of a 2x2 block held a component a lane by a quad; sets sing.
__device__ __forceinline__ double quad_inv(double v, int c, int qb, unsigned qm, bool &sing) {
    const double x = __shfl_sync(qm, v, qb), y = __shfl_sync(qm, v, qb + 1);
    const double z = __shfl_sync(qm, v, qb + 2), w = __shfl_sync(qm, v, qb + 3);
    const double det = x * w - y * z;
    sing |= (det == 0.0 || !isfinite(det));
    return (c == 0 ? w : c == 1 ? -y : c == 2 ? -z : x) * rcp_rn(det);
}
// Right-looking factorisation of the tail in FP64, its columns round the
// cluster.  Step k: every CTA updates its columns behind k with the pivot
// column (pushed to it before the barrier), A(i,j) -= A(i,k) (D_k^-1 A(k,j));
// the CTA with column k+1 takes that one first, inverts its pivot and pushes
// column and inverse to all CTAs while they update the rest, so a step is one
// pivot's chain and one cluster barrier.  A block is a component a lane.
__device__ __forceinline__ bool cl_tail_factor(const ClTail<blk4> &T, int t) {
    const int m = T.m, lane = t & 31, wp = t >> 5, c = lane & 3, r = c >> 1, s = c & 1, qb = lane & ~3, quad = lane >> 2;
    const unsigned qm = 0xfu << qb;
    bool sing = false;
    // W = D_k^-1 A(k,j) for the lane's component, then the two a block's update
    // takes: W(0,s), W(1,s)
    auto wcol = [&](const double *Di, const double *Ak, double &w0, double &w1) {
        const double w = __fma_rn(Di[2 * r], Ak[s], Di[2 * r + 1] * Ak[2 + s]);
        w0 = __shfl_sync(qm, w, qb + s);
        w1 = __shfl_sync(qm, w, qb + 2 + s);
    };
    auto push = [&](const double *p, double v) {  // the same place in every CTA
#pragma unroll 4
        for (int q = 0; q < T.nc; q++) cl_put(cl_map(p, q), v);
    };
    if (T.rank == 0) {
        double *col = (double *)T.col;
        for (int i = wp * 8 + quad; i < m; i += kClT / 4) {
            const double v = col[4 * i + c];
            if (i == 0) push((double *)T.dt + c, quad_inv(v, c, qb, qm, sing));
            else push((double *)T.lb + 4 * i + c, v);
        }
    }
    cluster_sync();
    const int cols = T.rank < T.nc ? (m - T.rank) / T.nc + 1 : 0;  // own columns, the right-hand side with them
    int jl = T.rank == 0 ? 1 : 0, next = T.nc > 1 ? 1 : 0;         // first own column behind k; the CTA with column k+1
    for (int k = 0; k + 1 < m; k++) {
        const double *L = (const double *)(T.lb + (k & 1) * m), *Di = (const double *)(T.dt + k);
        const int nx = k + 1;
        if (T.rank == next) {
            double *A = (double *)(T.col + (size_t)jl * m), w0, w1;
            double *nl = (double *)(T.lb + (nx & 1) * m);
            wcol(Di, A + 4 * k, w0, w1);
            for (int i = nx + wp * 8 + quad; i < m; i += kClT / 4) {
                const double2 l = *(const double2 *)(L + 4 * i + 2 * r);
                const double v = __fma_rn(-l.y, w1, __fma_rn(-l.x, w0, A[4 * i + c]));
                A[4 * i + c] = v;
                if (i == nx) push((double *)(T.dt + nx) + c, quad_inv(v, c, qb, qm, sing));
                else push(nl + 4 * i + c, v);
            }
            jl++;
        }
        // the other columns: 16 rows of one to a warp at a time, the warps
        // dealt over columns and rows alike
        const int chunks = (m - nx + 15) >> 4;
        for (int j = jl, q = wp; j < cols; j++, q -= chunks) {
            for (; q < chunks; q += kClT / 32) {
                double *A = (double *)(T.col + (size_t)j * m), w0, w1;
                wcol(Di, A + 4 * k, w0, w1);
                const int i0 = nx + q * 16 + quad;
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const int i = i0 + 8 * u;
                    if (i < m) {
                        const double2 l = *(const double2 *)(L + 4 * i + 2 * r);
                        A[4 * i + c] = __fma_rn(-l.y, w1, __fma_rn(-l.x, w0, A[4 * i + c]));
                    }
                }
            }
        }
        if (++next == T.nc) next = 0;
        cluster_sync();
    }
    return sing;
}
// The same in FP32 on one CTA: a block a lane, a block barrier a step.  The
// updates of a block are summed by themselves (col) and added to the block
// (lb) once, when its row or column is the next pivot's: updating in place
// would round at the block's size in every step (residual of a Newton step on
// filled 236- to 472-bus grids 1.3-1.5 times the level form's).
__device__ __forceinline__ bool cl_tail_factor(const ClTail<float4> &T, int t) {
    const int m = T.m, lane = t & 31, wp = t >> 5;
    bool sing = false;
    auto invert = [&](int k, float4 v) {
        const float det = v.x * v.w - v.y * v.z;
        sing |= (det == 0.f || !isfinite(det));
        T.dt[k] = pivot_inv(v, det);
    };
    for (int c = wp; c <= m; c += kClT / 32)
        for (int i = lane; i < m; i += 32)
            T.col[(size_t)c * m + i] = c == 0 || i == 0 ? T.lb[(size_t)c * m + i] : make_float4(0.f, 0.f, 0.f, 0.f);
    if (t == 0) invert(0, T.lb[0]);
    __syncthreads();
    for (int k = 0; k + 1 < m; k++) {
        const float4 *L = T.col + (size_t)k * m;
        const float4 Di = T.dt[k];
        const int nx = k + 1;
        // a column to a warp, column k+1 (its pivot's inverse with it) first
        for (int c = nx + wp; c <= m; c += kClT / 32) {
            float4 *S = T.col + (size_t)c * m;
            const float4 W = cbm(Di, S[k]);
#pragma unroll 2
            for (int i = nx + lane; i < m; i += 32) {
                float4 v = cms(S[i], L[i], W);
                if (c == nx || i == nx) v = add4T(T.lb[(size_t)c * m + i], v);
                S[i] = v;
                if (c == nx && i == nx) invert(nx, v);
            }
        }
        __syncthreads();
    }
    return sing;
}
// U and the right-hand side of the tail to CTA 0.
__device__ __forceinline__ void cl_tail_collect(const ClTail<blk4> &T, double2 *sx, int t) {
    const int m = T.m;
    for (int c = T.rank, jl = 0; T.rank < T.nc && c < m; c += T.nc, jl++) {
        const double *A = (const double *)(T.col + (size_t)jl * m);
        const unsigned u = cl_map(T.up + (size_t)c * (c - 1) / 2, 0);
        for (int q = t; q < 4 * c; q += kClT) cl_put(u + 8 * q, A[q]);
    }
    if (T.rank == m % T.nc) {
        const blk4 *b = T.col + (size_t)(m / T.nc) * m;
        const unsigned u = cl_map(sx, 0);
        for (int i = t; i < m; i += kClT) {
            cl_put(u + 16 * i, b[i].x);
            cl_put(u + 16 * i + 8, b[i].z);
        }
    }
    cluster_sync();
}
__device__ __forceinline__ void cl_tail_collect(const ClTail<float4> &T, float2 *sx, int t) {
    for (int i = t; i < T.m; i += kClT) {
        const float4 b = T.col[(size_t)T.m * T.m + i];
        sx[i] = make_float2(b.x, b.z);
    }
    __syncthreads();
}
// x of the tail in place of its right-hand side sx, on CTA 0: two threads a
// row, x_j published and then taken out of the rows above it.
template <typename TJ, typename B4, typename B2>
__device__ __forceinline__ void cl_tail_back(const ClTail<B4> &T, B2 *sx, int t) {
    constexpr int kBackT = 2 * gbpf::kTailMax;
    static_assert(kBackT % 32 == 0 && kBackT <= kClT, "whole warps");
    if (t < kBackT) {
        const int m = T.m, i = t >> 1, r = t & 1;
        TJ y = i < m ? ((const TJ *)&sx[i])[r] : (TJ)0;
        for (int j = m - 1; j >= 0; j--) {
            const TJ o = __shfl_xor_sync(0xffffffffu, y, 1);
            if (i == j) {
                const TJ *D = (const TJ *)&T.dt[j];
                ((TJ *)&sx[j])[r] = r ? cfma(D[2], o, D[3] * y) : cfma(D[0], y, D[1] * o);
            }
            TJ u0 = (TJ)0, u1 = (TJ)0;
            if (i < j) {
                const TJ *U = (const TJ *)(T.nc == 1 ? T.col + (size_t)j * m + i : T.up + (size_t)j * (j - 1) / 2 + i);
                u0 = U[2 * r];
                u1 = U[2 * r + 1];
            }
            asm volatile("bar.sync 1, %0;" ::"n"(kBackT) : "memory");
            const B2 x = sx[j];
            y = cfma(-u1, x.y, cfma(-u0, x.x, y));
        }
    }
    __syncthreads();
}

// What a launch needs of its schedule.
struct ClArgs {
    const int *sched, *off;
    int t0, td, tail_ctas;
    int p0, pd;  // first entry positions of the segment and of the tail
    int nf1, nfs, nbs, nb1, packed, in_smem;
    int seg_at, vec_at, tail_at, sched_at;  // bytes of dynamic shared memory before each region
};

// The whole factorisation and both substitutions.  Every CTA takes the same
// path through the cluster barriers: the stop flag is read before the first
// one, and nothing leaves the kernel between the first and the last.
template <typename TJ>
__global__ void __launch_bounds__(kClT, 1) k_lu_cluster(Dev d, ClArgs a, int guard) {
    using B4 = typename SB<TJ>::b4;
    using B2 = typename SB<TJ>::b2;
    extern __shared__ __align__(128) unsigned char csm[];
    __shared__ int s_stop;
    const int t = threadIdx.x, rank = (int)cluster_rank();
    if (t == 0) s_stop = stopped(d, guard);
    const int *sb = a.sched + a.off[rank];
    if (a.in_smem) {
        const int n4 = (a.off[rank + 1] - a.off[rank]) / 4;
        const int4 *src = (const int4 *)sb;
        int4 *dst = (int4 *)(csm + a.sched_at);
#pragma unroll 4
        for (int i = t; i < n4; i += kClT) dst[i] = src[i];
        sb = (const int *)dst;
    }
    __syncthreads();
    const int stop = s_stop;
    cluster_sync();  // every CTA has read the flag before a singular pivot may set it
    if (stop) return;
    B4 *fac = fac_of<TJ>(d), *Lv = fac + d.n, *Uv = fac + d.n + d.nup;
    const ClMem<TJ> G = {fac, Lv, Uv, (B4 *)csm, ys_of<TJ>(d)};
    B2 *xs = xs_of<TJ>(d);
    bool sing = false;
    for (int l = 0; l < a.nf1; l++) {
        sing |= cl_level<TJ, kLevel>(d, G, sb, sb + 8 * l, t, a.packed);
        cluster_sync();
    }
    const int *hseg = sb + 8 * (a.nf1 + 1), *hback = hseg + 8 * (a.nfs + 1);
    if (a.t0 < d.n) {
        (void)cl_level<TJ, kGather>(d, G, sb, sb + 8 * a.nf1, t, a.packed);
        cluster_sync();
        const int mt = d.n - a.td, ms = a.td - a.t0, mu = a.pd - a.p0;
        constexpr bool spread = sizeof(TJ) == 8;  // the tail's columns go round the cluster
        ClTail<B4> T;
        T.m = mt;
        T.nc = a.tail_ctas;
        T.rank = rank;
        T.col = (B4 *)(csm + a.tail_at);
        T.dt = T.col + (size_t)((mt + T.nc) / T.nc) * mt;
        T.lb = T.dt + mt;
        T.up = T.lb + 2 * mt;
        B4 *sD = (B4 *)(csm + a.seg_at), *sL = sD + ms, *sU = sL + mu;
        B2 *sy = (B2 *)(csm + a.vec_at);
        const ClMem<TJ> M = {sD - a.t0, sL - a.p0, sU - a.p0, sD - a.t0, sy - a.t0};
        if (rank == 0) {
            // the segment's blocks into shared memory and its levels
            for (int i = t; i < ms; i += kClT) {
                sD[i] = fac[a.t0 + i];
                sy[i] = G.ys[a.t0 + i];
            }
#pragma unroll 4
            for (int i = t; i < mu; i += kClT) {
                sL[i] = Lv[a.p0 + i];
                sU[i] = Uv[a.p0 + i];
            }
            if (!spread && mt) cl_tail_load<TJ>(d, T, a.td, t);
            __syncthreads();
            for (int l = 0; l < a.nfs; l++) {
                sing |= cl_level<TJ, kSegment>(d, M, sb, hseg + 8 * l, t, a.packed);
                __syncthreads();
            }
            if (mt && ms) {
                cl_seg_gather<TJ>(d, M, spread ? (B4 *)nullptr : T.lb, mt, a.td, sb, hseg + 8 * a.nfs, t, a.packed);
                __syncthreads();
            }
        }
        if (mt) {
            if (spread) {
                if (ms) cluster_sync();
                cl_tail_load<TJ>(d, T, a.td, t);
                cluster_sync();
            }
            if (spread || rank == 0) {
                sing |= cl_tail_factor(T, t);
                cl_tail_collect(T, sy + ms, t);
            }
        }
        if (rank == 0) {
            // x of the tail, then the segment's rows; x to global memory
            if (mt) cl_tail_back<TJ>(T, sy + ms, t);
            for (int l = 0; l < a.nbs; l++) {
                cl_back<TJ>(M.D, M.Uv, M.ys, M.ys, sb, hback + 4 * l, t, a.packed);
                __syncthreads();
            }
            for (int i = t; i < ms + mt; i += kClT) xs[a.t0 + i] = sy[i];
        }
        if (a.nb1) cluster_sync();
    }
    if (sing) {
        d.ctl->status = GBPF_E_SINGULAR;
        d.ctl->done = 1;
    }
    for (int l = 0; l < a.nb1; l++) {
        cl_back<TJ>(dinv_of<TJ>(d), Uv, G.ys, xs, sb, hback + 4 * (a.nbs + l), t, a.packed);
        if (l + 1 < a.nb1) cluster_sync();
    }
}
