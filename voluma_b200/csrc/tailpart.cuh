// The coarse tail of the V-cycle in the shared memory of a thread-block cluster (sm_100a).
//
// Levels first..coarsest of one system (GAMG.cpp:403-443) run in one launch of CL CTAs.  A level's
// 32-row slices are dealt to the CTAs in turn; each CTA holds its slices' matrix (values, 16-bit
// columns, transfer maps) in its own shared memory, and every CTA holds a copy of the two iterates,
// so a sweep gathers from its own shared memory only: a row's new value is stored to all CL copies
// (st.shared::cluster, coalesced) and the step ends at the cluster barrier.  A residual goes only
// to the CTA that owns its aggregate.  The row arithmetic is the per-level kernels' term for term
// (k_smooth_jacobi, k_smooth_gs, k_residual, k_restrict, k_coarse_apply), so the results are theirs
// bit for bit.
#pragma once

#include "dilu.cuh"
#include "kernels.cuh"

namespace vlm {

constexpr int kTailPartThreads = 512;  // 1024 threads leave 64 registers each: 600 bytes of spills in FP64

template <int CL>
__device__ __forceinline__ void part_sync() {
    if (CL == 1) {
        __syncthreads();
    } else {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

__device__ __forceinline__ void st_cluster(unsigned a, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(unsigned a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ unsigned map_rank(unsigned a, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

// *p of CTA `to` (p: the same location in this CTA) = v
template <int CL, class T>
__device__ __forceinline__ void part_store(T* p, int to, T v) {
    if (CL == 1)
        *p = v;
    else
        st_cluster(map_rank((unsigned)__cvta_generic_to_shared(p), (unsigned)to), v);
}

// *p of every CTA = v
template <int CL, class T>
__device__ __forceinline__ void part_publish(T* p, int rank, T v) {
    if (CL == 1) {
        *p = v;
        return;
    }
    const unsigned a = (unsigned)__cvta_generic_to_shared(p);
#pragma unroll
    for (int u = 0; u < CL; ++u) st_cluster(map_rank(a, unsigned((rank + u) & (CL - 1))), v);
}

// s -= a_ij v_j over a row's entries in entry order (entry q at e + 32 q), B entries' loads in flight
template <class T>
__device__ __forceinline__ T part_row_minus(const T* A, const uint16_t* col, int e, int len, const T* v, T s) {
    constexpr int B = sizeof(T) == 4 ? 8 : 4;
    for (; len > 0; len -= B, e += 32 * B) {
        T a[B], x[B];
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (u < len) {
                a[u] = A[e + 32 * u];
                x[u] = v[col[e + 32 * u]];
            }
#pragma unroll
        for (int u = 0; u < B; ++u)
            if (u < len) s -= a[u] * x[u];
    }
    return s;
}

// Grid: CL consecutive CTAs (one cluster) per system.  What bounds it: the chain of steps, each a
// shared-memory gather of ~15 entries per row and one cluster barrier.  One CTA held the FP64 images
// of levels up to about 700 rows; where the first small level was larger the tail read global memory,
// 82 us per V-cycle (56,000-cell FP64 corrector: 14.1 -> 8.8 ms with the cluster; a batch of 24 uneven
// systems of 16^3 to 48^3 cells 31.3 -> 25.6 ms; 96^3 FP64 solve 12.3 -> 11.2 ms).
template <class T, int CL>
__global__ void __launch_bounds__(kTailPartThreads, 1) k_vcycle_tail_parts(const TailPart* __restrict__ parts,
                                                                       const T* __restrict__ vimg,
                                                                       const uint16_t* __restrict__ simg,
                                                                       const TailLevel<T>* __restrict__ lev,
                                                                       const double* __restrict__ inv, const T* r0,
                                                                       T* x0, T omega, const SysState* st, int flag,
                                                                       int jacobi0) {
    pdl_launch();
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ __align__(16) TailPart I;
    {
        static_assert(sizeof(TailPart) % 4 == 0, "TailPart is copied as words");
        const int* src = reinterpret_cast<const int*>(parts + blockIdx.x);
        int* dst = reinterpret_cast<int*>(&I);
        for (int i = threadIdx.x; i < int(sizeof(TailPart) / 4); i += kTailPartThreads) dst[i] = __ldg(src + i);
    }
    __syncthreads();
    const int rank = CL == 1 ? 0 : int(blockIdx.x % CL);
    const int tid = threadIdx.x, nc = I.nc;
    T* t = reinterpret_cast<T*>(smraw);
    const int invRows = (nc + CL - 1) / CL;  // coarsest rows of a CTA: rank, rank + CL, ...
    double* sinv = reinterpret_cast<double*>(smraw + tail_align16(size_t(I.vecCount + I.valCount) * sizeof(T)));
    uint16_t* u = reinterpret_cast<uint16_t*>(reinterpret_cast<unsigned char*>(sinv) +
                                              tail_align16(size_t(nc) * invRows * sizeof(double)));
    // the images (fixed for the solve) while the predecessor drains: whole 16-byte words
    {
        const int4* vs = reinterpret_cast<const int4*>(vimg + I.valOff);
        int4* vd = reinterpret_cast<int4*>(t + I.vecCount);
        const int nv = int(size_t(I.valCount) * sizeof(T) / 16);
        for (int i = tid; i < nv; i += kTailPartThreads) cp_async16(vd + i, vs + i);
        const int4* ss = reinterpret_cast<const int4*>(simg + I.strOff);
        int4* sd = reinterpret_cast<int4*>(u);
        const int ns = int(size_t(I.strCount) * sizeof(uint16_t) / 16);
        for (int i = tid; i < ns; i += kTailPartThreads) cp_async16(sd + i, ss + i);
        // this CTA's rows of the coarsest inverse, transposed (a row's threads read consecutive words)
        const double* X = inv + I.invOffset;
        for (int i = tid; i < nc * invRows; i += kTailPartThreads) {
            const int il = i / nc, j = i - il * nc, row = il * CL + rank;
            sinv[j * invRows + il] = row < nc ? __ldg(X + (size_t)row * nc + j) : 0.0;
        }
        cp_async_commit();
        cp_async_wait<0>();
    }
    pdl_wait();
    if (st != nullptr && sys_idle(st[I.sys], flag)) return;  // uniform over the cluster
    const int f = I.first, c = I.coarsest;
    const bool gs0 = f == 0 && !jacobi0 && c > 0;
    const T* rg = (f == 0 ? r0 : lev[f].r) + I.rowStart[f];
    T* xg = (f == 0 ? x0 : lev[f].x) + I.rowStart[f];
    T* rC = t + I.tX2[c];  // the coarsest level's right-hand side
    auto rowOf = [&](int l) { return ((((l >> 5) * CL) + rank) << 5) | (l & 31); };
    auto relaxed = [&](T old, T v) { return omega == T(1) ? v : old + omega * (v - old); };
    if (gs0 && !I.two)  // multicolour sweeps with more than two colours start from zeros
        for (int i = tid; i < I.n[0]; i += kTailPartThreads) t[I.tX[0] + i] = T(0);
    part_sync<CL>();  // every CTA runs and holds its images: its shared memory may be written
    if (f == c) {
        for (int i = tid; i < I.n[c]; i += kTailPartThreads) rC[i] = __ldcg(rg + i);
        __syncthreads();
    } else {
        T* r = t + I.tR[f];
        const T* D = t + I.tDiag[f];
        T* x2 = t + I.tX2[f];
        for (int l = tid; l < I.nl[f]; l += kTailPartThreads) {
            const int i = rowOf(l);
            const T v = __ldcg(rg + i);
            r[l] = v;
            if (!gs0) {  // first pre-sweep from zero (k_smooth_jacobi MODE 1)
                const T q = v / D[l];
                part_publish<CL>(x2 + i, rank, omega == T(1) ? q : omega * q);
            }
        }
        if (gs0)
            __syncthreads();
        else
            part_sync<CL>();
    }
    // one colour step of level 0 (k_smooth_gs): this CTA's slices of the group
    auto gsStep = [&](int q, bool zero, bool last) {
        const T* A = t + I.tVal[0];
        const uint16_t *col = u + I.uCol[0], *rl = u + I.uRlen[0], *sl = u + I.uSlice[0];
        const T *D = t + I.tDiag[0], *r = t + I.tR[0];
        T* x = t + I.tX[0];
        const int s0 = I.grpStart[q] >> 5, s1 = (I.grpStart[q] + I.grpCount[q]) >> 5;
        const int ls0 = (s0 - rank + CL - 1) / CL, ls1 = (s1 - rank + CL - 1) / CL;  // local slices of [s0, s1)
        for (int l = ls0 * 32 + tid; l < ls1 * 32; l += kTailPartThreads) {
            const int i = rowOf(l);
            T s = r[l];
            if (!zero) s = part_row_minus<T>(A, col, int(sl[l >> 5]) * 32 + (l & 31), rl[l], x, s);
            s = s / D[l];
            if (last)
                x[i] = s;
            else
                part_publish<CL>(x + i, rank, s);
        }
    };
    for (int k = f; k < c; ++k) {
        const int nl = I.nl[k];
        const T* A = t + I.tVal[k];
        const uint16_t *col = u + I.uCol[k], *rl = u + I.uRlen[k], *sl = u + I.uSlice[k], *agg = u + I.uAgg[k];
        const T *D = t + I.tDiag[k], *r = t + I.tR[k];
        T *x = t + I.tX[k], *x2 = t + I.tX2[k];
        if (k == 0 && gs0) {
            for (int sweep = 0; sweep < 2; ++sweep)
                for (int q = 0; q < I.nColours; ++q) {
                    gsStep(q, I.two && sweep == 0 && q == 0, false);
                    part_sync<CL>();
                }
        } else {
            for (int l = tid; l < nl; l += kTailPartThreads) {  // second pre-sweep
                const int i = rowOf(l);
                const T v = part_row_minus<T>(A, col, int(sl[l >> 5]) * 32 + (l & 31), rl[l], x2, r[l]) / D[l];
                part_publish<CL>(x + i, rank, relaxed(x2[i], v));
            }
            part_sync<CL>();
        }
        // residuals (k_residual), each into the x2 copy of the CTA that sums it
        for (int l = tid; l < nl; l += kTailPartThreads) {
            const int i = rowOf(l), a = agg[l];
            const T v = part_row_minus<T>(A, col, int(sl[l >> 5]) * 32 + (l & 31), rl[l], x, r[l] - D[l] * x[i]);
            if (a != 0xffff) part_store<CL>(x2 + i, (a >> 5) & (CL - 1), v);
        }
        part_sync<CL>();
        // restriction (k_restrict) and the next level's first pre-sweep
        const uint16_t *cp = u + I.uCptr[k], *ch = u + I.uChild[k];
        for (int l = tid; l < I.nl[k + 1]; l += kTailPartThreads) {
            const int R = rowOf(l);
            T s = T(0);
            for (int q = cp[l]; q < cp[l + 1]; ++q) s += x2[ch[q]];
            if (k + 1 == c) {
                part_publish<CL>(rC + R, rank, s);
            } else {
                (t + I.tR[k + 1])[l] = s;
                const T v = s / (t + I.tDiag[k + 1])[l];
                part_publish<CL>(t + I.tX2[k + 1] + R, rank, omega == T(1) ? v : omega * v);
            }
        }
        part_sync<CL>();
    }
    {
        // coarsest level: x = inv * r (k_coarse_apply)
        T* x = t + I.tX[c];
        for (int il = tid; il < invRows; il += kTailPartThreads) {
            const int i = il * CL + rank;
            if (i >= nc) break;
            double g = 0.0;
#pragma unroll 8
            for (int j = 0; j < nc; ++j) g += sinv[j * invRows + il] * (double)rC[j];
            if (f == c)
                xg[i] = (T)g;
            else
                part_publish<CL>(x + i, rank, (T)g);
        }
        if (f == c) {
            if (rank == 0)
                for (int i = nc + tid; i < I.n[c]; i += kTailPartThreads) xg[i] = T(0);
            return;  // nothing was published: no CTA waits for or writes another's memory
        }
    }
    for (int k = c - 1; k >= f; --k) {
        part_sync<CL>();
        const int nl = I.nl[k];
        const T* A = t + I.tVal[k];
        const uint16_t *col = u + I.uCol[k], *rl = u + I.uRlen[k], *sl = u + I.uSlice[k], *agg = u + I.uAgg[k];
        const T *D = t + I.tDiag[k], *r = t + I.tR[k], *xc = t + I.tX[k + 1];
        T *x = t + I.tX[k], *x2 = t + I.tX2[k];
        // the coarse-grid correction, then the post-sweeps
        for (int l = tid; l < nl; l += kTailPartThreads) {
            const int i = rowOf(l), a = agg[l];
            if (a != 0xffff) part_publish<CL>(x + i, rank, x[i] + xc[a]);
        }
        part_sync<CL>();
        if (k == 0 && gs0) {
            for (int sweep = 0; sweep < 2; ++sweep)
                for (int q = I.nColours - 1; q >= 0; --q) {
                    const bool last = sweep == 1 && q == 0;
                    gsStep(q, false, last);
                    if (last)
                        __syncthreads();
                    else
                        part_sync<CL>();
                }
            for (int l = tid; l < nl; l += kTailPartThreads) {
                const int i = rowOf(l);
                xg[i] = x[i];
            }
            continue;
        }
        for (int l = tid; l < nl; l += kTailPartThreads) {
            const int i = rowOf(l);
            const T v = part_row_minus<T>(A, col, int(sl[l >> 5]) * 32 + (l & 31), rl[l], x, r[l]) / D[l];
            part_publish<CL>(x2 + i, rank, relaxed(x[i], v));
        }
        part_sync<CL>();
        for (int l = tid; l < nl; l += kTailPartThreads) {
            const int i = rowOf(l);
            const T v = part_row_minus<T>(A, col, int(sl[l >> 5]) * 32 + (l & 31), rl[l], x2, r[l]) / D[l];
            const T w = relaxed(x2[i], v);
            if (k == f)
                xg[i] = w;
            else
                part_publish<CL>(x + i, rank, w);
        }
    }
}

}  // namespace vlm
