// Pipelined DIC/DILU kernels of systems too wide for one CTA (dilu.h, DiluParts; LinearSolver.cpp:56-112).
//
// One CTA per part.  A sweep is bound by its chain of levels (nx + ny + nz - 2 of them on a box), so
// what counts is the time of one level.  A CTA-to-CTA barrier per level costs 2.5-5.7 us; here a part
// meets no barrier but its own: it streams its steps' rows and entries into a shared-memory ring with
// cp.async, keeps its swept vector in shared memory, and receives the values of other parts through
// mailboxes of 16 bytes {value, launch number}, written and read whole, which need neither a fence
// nor a flag.  A mailbox is polled two steps before its value is used, so a hand-over costs latency
// once per part (parts run staggered) and not once per level.  Measured: one PBiCGStab/DILU solve of
// 80 x 64 x 48 cells (a factorisation and six applications, 190 levels each way) 14.6 -> 5.2 ms; the
// Taylor-Green step at 64^3 15.1 -> 9.4 ms, the 96 x 72 x 48 LES channel step 39.9 -> 19.7 ms.
//
// Parts only wait for parts of an earlier ticket, and tickets are taken in the order in which CTAs
// start, so a sweep ends however few of its CTAs are resident; no cooperative launch.  Every wait
// gives up after kPartSpinLimit polls, leaves VLM_ERR_TIMEOUT in *err, and later waits then return at
// once.
//
// The operations are those of the reference in its order (bit for bit): factor rD[u] -= A_lu A_ul /
// rD[l], forward w[u] = rD[u] r[u] - sum rD[u] A_ul w[l], backward w[l] -= sum rD[l] A_lu w[u].
#pragma once

#include "dilu.cuh"

namespace vlm {

constexpr int kPartThreads = 256;
constexpr int kPartRing = 5;          // ring stages: a step's data is requested four steps ahead
constexpr int kPartEnt = 6;           // entries per slot staged in the ring (the rest are read in place)
constexpr int kPartSpinLimit = 1 << 21;  // polls of an L2 read each: about a second

struct __align__(16) DiluMail {
    double v;
    unsigned long long tag;
};

// Launch bookkeeping: ticket (part order), finished CTAs, launches so far.
struct DiluPartSync {
    unsigned ticket, done;
    unsigned long long epoch;
};

__device__ __forceinline__ void mail_put(DiluMail* m, double v, unsigned long long tag) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(m),
                 "l"(__double_as_longlong(v)), "l"(tag)
                 : "memory");
}
__device__ __forceinline__ void mail_get(const DiluMail* m, double& v, unsigned long long& tag) {
    long long a;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(tag)
                 : "l"(m)
                 : "memory");
    v = __longlong_as_double(a);
}
// Waits for the mailbox's value of this launch.
__device__ __forceinline__ double mail_wait(const DiluMail* m, double v, unsigned long long tag,
                                            unsigned long long want, int* err) {
    for (int it = 0; tag != want; ++it) {
        if ((it & 63) == 63 && *(volatile int*)err != 0) break;
        if (it > kPartSpinLimit) {
            atomicExch(err, int(VLM_ERR_TIMEOUT));
            break;
        }
        mail_get(m, v, tag);
    }
    return v;
}

// Ring stage of W slots with M staged entries each: a[W], b[W], v[M W] doubles; mail[W], row[W], col[M W].
__host__ __device__ constexpr size_t part_stage_bytes(int W, int M) {
    return dilu_align16(size_t(W) * ((M + 2) * sizeof(double) + (M + 2) * sizeof(int32_t)));
}
// localSlots: slots whose vector is kept in shared memory (0: it stays in global memory).
__host__ __device__ constexpr size_t part_smem(int localSlots, int W, int M, int maxRemote) {
    return dilu_align16(size_t(localSlots) * sizeof(double)) + dilu_align16(size_t(2) * maxRemote * sizeof(double)) +
           kPartRing * part_stage_bytes(W, M);
}

struct DiluPartArgs {
    const DiluPart* parts;
    const DiluStep* steps;
    int nParts, W, M, maxRemote;  // ring shape: slots, staged entries, remote entries per step
    const int32_t* slotRow;
    const int32_t *col, *remote, *mail;  // of the sweep's direction
    const double* coef;                  // per entry: A_lu A_ul (factor), A_ul (forward), A_lu (backward)
    DiluMail* box;                       // mailboxes of the direction
    double *rDs, *ws;                    // per slot: 1 / rD; the swept vector (scratch between sweeps)
    const double* src;                   // solver rows: the diagonal (factor), r (forward)
    double* w;                           // solver rows: the result (backward)
    DiluPartSync* sync;
    int* err;
    const SysState* st;
    int flag;
};

enum : int { kPartFactor = 0, kPartForward = 1, kPartBackward = 2 };

// SH: the part's vector lives in shared memory; else in ws, read through L2 (parts too large).
template <int KIND, bool SH>
__global__ void __launch_bounds__(kPartThreads, 1) k_dilu_part(const DiluPartArgs A) {
    pdl_entry();
    extern __shared__ __align__(16) char psm[];
    __shared__ int sPart;
    __shared__ unsigned long long sTag;
    const int tid = threadIdx.x;
    if (tid == 0) {
        const int t = int(atomicAdd(&A.sync->ticket, 1u));
        sPart = KIND == kPartBackward ? A.nParts - 1 - t : t;
        sTag = *(volatile unsigned long long*)&A.sync->epoch + 1;
    }
    __syncthreads();
    const DiluPart P = A.parts[sPart];
    const unsigned long long tag = sTag;
    if (A.st == nullptr || !sys_idle(A.st[P.sys], A.flag)) {  // uniform over the system's parts
        double* sh = reinterpret_cast<double*>(psm);
        double* rem = reinterpret_cast<double*>(psm + dilu_align16(size_t(SH ? P.nSlots : 0) * sizeof(double)));
        const int W = A.W, M = A.M, maxRem = A.maxRemote;
        char* ring = reinterpret_cast<char*>(rem) + dilu_align16(size_t(2) * maxRem * sizeof(double));
        const size_t SB = part_stage_bytes(W, M);
        auto stageA = [&](int q) { return reinterpret_cast<double*>(ring + size_t(q % kPartRing) * SB); };
        auto step = [&](int q) -> const DiluStep& {
            return A.steps[KIND == kPartBackward ? P.stepBegin + P.nSteps - 1 - q : P.stepBegin + q];
        };
        auto ent0 = [&](const DiluStep& S) { return KIND == kPartBackward ? S.up : S.lo; };
        auto entM = [&](const DiluStep& S) { return KIND == kPartBackward ? S.mup : S.mlo; };
        auto rem0 = [&](const DiluStep& S) { return KIND == kPartBackward ? S.rup : S.rlo; };
        auto remN = [&](const DiluStep& S) { return KIND == kPartBackward ? S.nrup : S.nrlo; };
        // this thread's row of step q (the gather of src needs it one step before the copy starts)
        auto rowOf = [&](int q) -> int {
            if (KIND == kPartBackward || q >= P.nSteps) return -1;
            const DiluStep& S = step(q);
            return tid < S.width ? __ldg(A.slotRow + S.s0 + tid) : -1;
        };
        auto issue = [&](int q, int row) {
            if (q < P.nSteps) {
                const DiluStep& S = step(q);
                double* a = stageA(q);
                double* b = a + W;
                double* v = b + W;
                int32_t* mail = reinterpret_cast<int32_t*>(v + size_t(M) * W);
                int32_t* rw = mail + W;
                int32_t* col = rw + W;
                if (tid < S.width) {
                    cp_async4(mail + tid, A.mail + S.s0 + tid);
                    if (KIND != kPartFactor) cp_async8(a + tid, A.rDs + S.s0 + tid);
                    if (KIND == kPartBackward) {
                        cp_async8(b + tid, A.ws + S.s0 + tid);
                        cp_async4(rw + tid, A.slotRow + S.s0 + tid);
                    } else {
                        cp_async8(b + tid, A.src + row);
                    }
                }
                const int n = min(entM(S), M) * S.width, e = ent0(S);
                for (int k = tid; k < n; k += kPartThreads) {
                    cp_async4(col + k, A.col + e + k);
                    cp_async8(v + k, A.coef + e + k);
                }
            }
            cp_async_commit();
        };
        // remote entry tid of step q: its mailbox, read without waiting
        const DiluMail* mCur = nullptr;  // of step q + 1, requested one step ago
        double vCur = 0.0;
        unsigned long long tCur = 0;
        auto request = [&](int q, const DiluMail*& m, double& v, unsigned long long& t) {
            m = nullptr;
            if (q >= P.nSteps) return;
            const DiluStep& S = step(q);
            if (tid < remN(S)) {
                m = A.box + __ldg(A.remote + rem0(S) + tid);
                mail_get(m, v, t);
            }
        };
        // the remote values of step q into their buffer
        auto deliver = [&](int q, const DiluMail* m, double v, unsigned long long t) {
            if (q >= P.nSteps) return;
            const DiluStep& S = step(q);
            double* rb = rem + (q & 1) * maxRem;
            if (m) rb[tid] = mail_wait(m, v, t, tag, A.err);
            for (int k = tid + kPartThreads; k < remN(S); k += kPartThreads) {
                const DiluMail* mk = A.box + __ldg(A.remote + rem0(S) + k);
                double vk;
                unsigned long long tk;
                mail_get(mk, vk, tk);
                rb[k] = mail_wait(mk, vk, tk, tag, A.err);
            }
        };
        for (int q = 0; q < kPartRing - 1; ++q) issue(q, rowOf(q));
        int rowNext = rowOf(kPartRing - 1);
        {
            request(0, mCur, vCur, tCur);
            deliver(0, mCur, vCur, tCur);
            request(1, mCur, vCur, tCur);
        }
        for (int q = 0; q < P.nSteps; ++q) {
            cp_async_wait<kPartRing - 2>();
            __syncthreads();  // step q staged, step q - 1's values and step q's remote values visible
            issue(q + kPartRing - 1, rowNext);
            rowNext = rowOf(q + kPartRing);
            const DiluMail* mNext;
            double vNext = 0.0;
            unsigned long long tNext = 0;
            request(q + 2, mNext, vNext, tNext);
            const DiluStep& S = step(q);
            if (tid < S.width) {
                const double* a = stageA(q);
                const double* b = a + W;
                const double* cv = b + W;
                const int32_t* mail = reinterpret_cast<const int32_t*>(cv + size_t(M) * W);
                const int32_t* rw = mail + W;
                const int32_t* col = rw + W;
                const double* rb = rem + (q & 1) * maxRem;
                const int wd = S.width, m = entM(S), e = ent0(S);
                auto value = [&](int l) -> double {
                    if (l <= -2) return rb[-2 - l];
                    return SH ? sh[l] : __ldcg(A.ws + P.slot0 + l);
                };
                const double rd = KIND == kPartFactor ? 0.0 : a[tid];
                double x = b[tid];
                if (KIND == kPartForward) x = rd * x;
                for (int j = 0; j < m; ++j) {
                    const int l = j < M ? col[j * wd + tid] : __ldg(A.col + e + j * wd + tid);
                    if (l == -1) break;
                    const double c = j < M ? cv[j * wd + tid] : __ldg(A.coef + e + j * wd + tid);
                    if (KIND == kPartFactor)
                        x -= c / value(l);
                    else
                        x -= rd * c * value(l);
                }
                const int slot = S.s0 + tid;
                if (SH) sh[slot - P.slot0] = x;
                if (!SH || KIND == kPartForward) A.ws[slot] = x;
                if (mail[tid] >= 0) mail_put(A.box + mail[tid], x, tag);
                if (KIND == kPartFactor) A.rDs[slot] = 1.0 / x;
                if (KIND == kPartBackward) A.w[rw[tid]] = x;
            }
            deliver(q + 1, mCur, vCur, tCur);
            mCur = mNext;
            vCur = vNext;
            tCur = tNext;
        }
        cp_async_wait<0>();
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&A.sync->done, 1u) == unsigned(A.nParts - 1)) {  // every CTA has read epoch and its ticket
            A.sync->ticket = 0;
            A.sync->done = 0;
            A.sync->epoch = tag;
        }
    }
}

}  // namespace vlm
