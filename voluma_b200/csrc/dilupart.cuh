// Pipelined DIC/DILU kernels of systems too wide for one CTA (dilu.h, DiluParts; LinearSolver.cpp:56-112).
//
// One CTA per part.  A sweep is bound by its chain of levels (nx + ny + nz - 2 of them on a box), so
// what counts is the time of one level.  A CTA-to-CTA barrier per level costs 2.5-5.7 us; here a part
// meets no barrier but its own: it streams its steps' rows and entries into a shared-memory ring with
// cp.async, keeps its swept vector in shared memory, and receives the values of other parts through
// mailboxes of 16 bytes {value, launch number}, written and read whole, which need neither a fence
// nor a flag.  A mailbox is read two steps before its value is used and polled again when it was empty.
// Measured: one PBiCGStab/DILU solve of 80 x 64 x 48 cells (a factorisation and six applications, 190
// levels each way) 13.8 ms with the barrier per level, 5.2 with k_dilu_part and 3.1 with k_dilu_pipe below,
// which takes such meshes; k_dilu_part alone: a column of 20,000 cells (two parts, one after the other)
// 0.85 us a level, 150 x 140 x 130 cells (418 levels, its vectors in global memory) 2.3 us a level.
//
// Parts only wait for parts of an earlier ticket, and tickets are taken in the order in which CTAs
// start, so a sweep ends however few of its CTAs are resident; no cooperative launch.  On a mesh that is
// one long chain the parts run one after another, so a wait may last as long as all the steps of the
// sweep: a wait gives up after kMailPolls polls and kMailStepPolls more for each such step (an L2 read
// each, 0.3 us at least, so 5 us a step against the 1.7 us a step takes), leaves VLM_ERR_TIMEOUT in *err,
// and later waits then return at once.  Both are looked at after every 64 polls, outside the polling loop:
// with a variable limit inside it a PBiCGStab iteration of 80 x 64 x 48 cells took 835 us instead of 826.
//
// The operations are those of the reference in its order (bit for bit): factor rD[u] -= A_lu A_ul /
// rD[l], forward w[u] = rD[u] r[u] - sum rD[u] A_ul w[l], backward w[l] -= sum rD[l] A_lu w[u].
#pragma once

#include "dilu.cuh"

namespace vlm {

constexpr int kPartThreads = 256;
constexpr int kPartRing = 5;          // ring stages: a step's data is requested four steps ahead
constexpr int kPartEnt = 6;           // entries per slot staged in the ring (the rest are read in place)
constexpr int kMailPolls = 1 << 21;   // about a second
constexpr int kMailStepPolls = 16;

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
// Waits for the mailbox's value of this launch, at most `limit` polls (rounded up to whole rounds of 64).
__device__ __forceinline__ double mail_wait(const DiluMail* m, double v, unsigned long long tag,
                                            unsigned long long want, int limit, int* err) {
    for (int it = 0; tag != want; it += 64) {
#pragma unroll 1
        for (int k = 0; k < 64; ++k) {
            mail_get(m, v, tag);
            if (tag == want) return v;
        }
        if (*(volatile int*)err != 0) break;
        if (it > limit) {
            atomicExch(err, int(VLM_ERR_TIMEOUT));
            break;
        }
    }
    return v;
}

// Ring stage of W slots with M staged entries each: a[W], b[W], v[M W] doubles; mail[W], row[W], col[M W].
__host__ __device__ constexpr size_t part_stage_bytes(int W, int M) {
    return dilu_align16(size_t(W) * ((M + 2) * sizeof(double) + (M + 2) * sizeof(int32_t)));
}
// localSlots: slots whose vector is kept in shared memory (0: it stays in global memory); steps: step
// descriptors kept there (0: read in place).
__host__ __device__ constexpr size_t part_smem(int localSlots, int W, int M, int maxRemote, int steps) {
    return dilu_align16(size_t(localSlots) * sizeof(double)) + dilu_align16(size_t(2) * maxRemote * sizeof(double)) +
           kPartRing * part_stage_bytes(W, M) + dilu_align16(size_t(steps) * sizeof(DiluStep));
}

struct DiluPartArgs {
    const DiluPart* parts;
    const DiluStep* steps;
    int nParts, W, M, maxRemote;  // ring shape: slots, staged entries, remote entries per step
    int stepsLocal;               // the part's step descriptors are copied to shared memory
    const int32_t *slotRow, *padRow;
    const int32_t *col, *remote, *mail;  // of the sweep's direction
    const double* coef;                  // per entry: A_lu A_ul (factor), A_ul (forward), A_lu (backward)
    DiluMail* box;                       // mailboxes of the direction
    double *rDs, *ws;                    // per slot: 1 / rD; the swept vector (scratch between sweeps)
    const double* src;                   // solver rows: the diagonal (factor), r (forward)
    double* w;                           // solver rows: the result (backward)
    DiluPartSync* sync;
    int limit;  // polls of a wait
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
        if (KIND == kPartBackward)
            for (int i = tid; i < P.nPad; i += kPartThreads) A.w[__ldg(A.padRow + P.pad0 + i)] = 0.0;
        double* sh = reinterpret_cast<double*>(psm);
        double* rem = reinterpret_cast<double*>(psm + dilu_align16(size_t(SH ? P.nSlots : 0) * sizeof(double)));
        const int W = A.W, M = A.M, maxRem = A.maxRemote;
        char* ring = reinterpret_cast<char*>(rem) + dilu_align16(size_t(2) * maxRem * sizeof(double));
        const size_t SB = part_stage_bytes(W, M);
        auto stageA = [&](int q) { return reinterpret_cast<double*>(ring + size_t(q % kPartRing) * SB); };
        const DiluStep* steps = A.steps + P.stepBegin;
        if (A.stepsLocal) {
            int* ls = reinterpret_cast<int*>(ring + kPartRing * SB);
            const int* gs = reinterpret_cast<const int*>(steps);
            for (int i = tid; i < P.nSteps * int(sizeof(DiluStep) / sizeof(int)); i += kPartThreads) ls[i] = __ldg(gs + i);
            __syncthreads();
            steps = reinterpret_cast<const DiluStep*>(ls);
        }
        auto step = [&](int q) -> const DiluStep& { return steps[KIND == kPartBackward ? P.nSteps - 1 - q : q]; };
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
        // remote entry tid of step q: its mailbox (looked up one step before), read without waiting
        const DiluMail* mCur = nullptr;  // of step q + 1, requested one step ago
        double vCur = 0.0;
        unsigned long long tCur = 0;
        auto boxOf = [&](int q) -> int {
            if (q >= P.nSteps) return -1;
            const DiluStep& S = step(q);
            return tid < remN(S) ? __ldg(A.remote + rem0(S) + tid) : -1;
        };
        auto request = [&](int box, const DiluMail*& m, double& v, unsigned long long& t) {
            m = nullptr;
            if (box >= 0) {
                m = A.box + box;
                mail_get(m, v, t);
            }
        };
        // the remote values of step q into their buffer
        auto deliver = [&](int q, const DiluMail* m, double v, unsigned long long t) {
            if (q >= P.nSteps) return;
            const DiluStep& S = step(q);
            double* rb = rem + (q & 1) * maxRem;
            if (m) rb[tid] = mail_wait(m, v, t, tag, A.limit, A.err);
            for (int k = tid + kPartThreads; k < remN(S); k += kPartThreads) {
                const DiluMail* mk = A.box + __ldg(A.remote + rem0(S) + k);
                double vk;
                unsigned long long tk;
                mail_get(mk, vk, tk);
                rb[k] = mail_wait(mk, vk, tk, tag, A.limit, A.err);
            }
        };
        for (int q = 0; q < kPartRing - 1; ++q) issue(q, rowOf(q));
        int rowNext = rowOf(kPartRing - 1);
        {
            request(boxOf(0), mCur, vCur, tCur);
            deliver(0, mCur, vCur, tCur);
            request(boxOf(1), mCur, vCur, tCur);
        }
        int boxNext = boxOf(2);
        for (int q = 0; q < P.nSteps; ++q) {
            cp_async_wait<kPartRing - 2>();
            __syncthreads();  // step q staged, step q - 1's values and step q's remote values visible
            issue(q + kPartRing - 1, rowNext);
            rowNext = rowOf(q + kPartRing);
            const DiluMail* mNext;
            double vNext = 0.0;
            unsigned long long tNext = 0;
            request(boxNext, mNext, vNext, tNext);
            boxNext = boxOf(q + 3);
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

// ---------------------------------------------------------------- records
// The same sweep for rows of at most six neighbours per direction (box meshes) whose parts' vectors fit in
// shared memory.  What bounds it is the latency of a level: 0.9-1.3 us in a solve (33 x 39 x 35 0.86, 80 x
// 64 x 48 1.03, 64^3 1.15, 96 x 72 x 48 1.27), with one issue slot in ten used and 44% of the warps' time at
// the step's barrier (ncu at 33 x 39 x 35: 1.2 us a level with cold caches, where the one-CTA kernels of
// dilu.cuh, which wait for nobody, take 0.47 at 64^2).  In k_dilu_part each entry is a dependent load of
// the column, a choice of source and a load of the value.  Here a row is
// one 16-byte word of columns, one 32-byte word of coefficients with 1 / rD, and three values at
// once; a few rows (periodic links) read a second record.  Everything a step needs from global
// memory is requested at least two steps before.
struct DiluPipeArgs {
    const DiluPart* parts;
    const DiluRecStep* steps;
    int nParts, W, E, maxRemote, ring;  // ring shape: slots, extensions; stages
    const int32_t *slotRow, *padRow;
    const int4* col;        // records of the sweep's direction
    const double* coef;     // four doubles per record: three coefficients, 1 / rD
    const int32_t* remote;  // mailbox of each remote entry
    DiluMail* box;
    double *rdLo, *rdUp;    // coefficient records of both directions: the factor writes their 1 / rD
    double* ws;
    const double* src;
    double* w;
    DiluPartSync* sync;
    int limit;  // polls of a wait
    int* err;
    const SysState* st;
    int flag;
};

// Ring stage: col[W] int4, ext col[E] int4, coef[4 W], ext coef[4 E], b[W] doubles, row[W] int.
__host__ __device__ constexpr size_t pipe_stage_bytes(int W, int E) {
    return dilu_align16(size_t(W + E) * (sizeof(int4) + 4 * sizeof(double)) + size_t(W) * (sizeof(double) + sizeof(int32_t)));
}
__host__ __device__ constexpr size_t pipe_smem(int slots, int W, int E, int maxRemote, int ring, int steps) {
    return dilu_align16((size_t(slots) + 2 * size_t(maxRemote)) * sizeof(double)) + ring * pipe_stage_bytes(W, E) +
           dilu_align16(size_t(steps) * sizeof(DiluRecStep));
}

__device__ __forceinline__ void cp_async_wait_n(int n) {
    switch (n) {  // all but the n newest groups
    case 1: cp_async_wait<1>(); break;
    case 2: cp_async_wait<2>(); break;
    case 3: cp_async_wait<3>(); break;
    default: cp_async_wait<4>(); break;
    }
}

// Coefficient records from the faces (DiluRecords): A_lu A_ul and A_ul of the lower entries, A_lu of the
// upper ones; the records' fourth word (1 / rD) is the factorisation's.
__global__ void k_dilu_record_values(int nLo, int nUp, const int4* __restrict__ loFace, const int4* __restrict__ upFace,
                                     const double* __restrict__ upper, const double* __restrict__ lower,
                                     double* __restrict__ prod, double* __restrict__ coefLo,
                                     double* __restrict__ coefUp) {
    pdl_entry();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nLo + nUp) return;
    const bool lo = k < nLo;
    const int4 f4 = lo ? loFace[k] : upFace[k - nLo];
    const int f[3] = {f4.x, f4.y, f4.z};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        double aul = 0.0, alu = 0.0;
        if (f[j] != DiluRecords::kNoFace) {
            const int a = f[j] & 0x7fffffff;
            const double u = upper[a], l = lower[a];
            aul = f[j] < 0 ? l : u;  // ownerIsL
            alu = f[j] < 0 ? u : l;
        }
        if (lo) {
            prod[4 * size_t(k) + j] = alu * aul;
            coefLo[4 * size_t(k) + j] = aul;
        } else {
            coefUp[4 * size_t(k - nLo) + j] = alu;
        }
    }
}

template <int KIND>
__global__ void __launch_bounds__(kPartThreads, 1) k_dilu_pipe(const DiluPipeArgs A) {
    pdl_entry();
    extern __shared__ __align__(16) char psm[];
    __shared__ int sPart;
    __shared__ unsigned long long sTag;
    constexpr bool back = KIND == kPartBackward;
    const int tid = threadIdx.x;
    if (tid == 0) {
        const int t = int(atomicAdd(&A.sync->ticket, 1u));
        sPart = back ? A.nParts - 1 - t : t;
        sTag = *(volatile unsigned long long*)&A.sync->epoch + 1;
    }
    __syncthreads();
    const DiluPart P = A.parts[sPart];
    const unsigned long long tag = sTag;
    if (A.st == nullptr || !sys_idle(A.st[P.sys], A.flag)) {  // uniform over the system's parts
        if (KIND == kPartBackward)
            for (int i = tid; i < P.nPad; i += kPartThreads) A.w[__ldg(A.padRow + P.pad0 + i)] = 0.0;
        const int W = A.W, E = A.E, maxRem = A.maxRemote, nSteps = P.nSteps, R = A.ring;
        double* sh = reinterpret_cast<double*>(psm);
        double* rem = sh + P.nSlots;
        char* ring = psm + dilu_align16((size_t(P.nSlots) + 2 * size_t(maxRem)) * sizeof(double));
        const size_t SB = pipe_stage_bytes(W, E);
        DiluRecStep* steps = reinterpret_cast<DiluRecStep*>(ring + R * SB);
        {
            const int* gs = reinterpret_cast<const int*>(A.steps + P.stepBegin);
            int* ls = reinterpret_cast<int*>(steps);
            for (int i = tid; i < nSteps * int(sizeof(DiluRecStep) / sizeof(int)); i += kPartThreads) ls[i] = __ldg(gs + i);
        }
        __syncthreads();
        auto step = [&](int q) -> const DiluRecStep& { return steps[back ? nSteps - 1 - q : q]; };
        auto rowOf = [&](int q) -> int {  // this thread's solver row of step q
            if (q >= nSteps) return 0;
            const DiluRecStep& S = step(q);
            return tid < S.width ? __ldg(A.slotRow + S.s0 + tid) : 0;
        };
        auto boxOf = [&](int q) -> int {  // this thread's remote entry of step q
            if (q >= nSteps) return -1;
            const DiluRecStep& S = step(q);
            return tid < (back ? S.nrup : S.nrlo) ? __ldg(A.remote + (back ? S.rup : S.rlo) + tid) : -1;
        };
        auto issue = [&](int q, char* stage, int row) {
            if (q < nSteps) {
                const DiluRecStep& S = step(q);
                int4* c = reinterpret_cast<int4*>(stage);
                double* v = reinterpret_cast<double*>(c + W + E);
                double* b = v + 4 * (W + E);
                int32_t* rw = reinterpret_cast<int32_t*>(b + W);
                if (tid < S.width) {
                    const int slot = S.s0 + tid;
                    cp_async16(c + tid, A.col + slot);
                    cp_async16(v + 4 * tid, A.coef + 4 * size_t(slot));
                    cp_async16(v + 4 * tid + 2, A.coef + 4 * size_t(slot) + 2);
                    if (back) {
                        cp_async8(b + tid, A.ws + slot);
                        cp_async4(rw + tid, A.slotRow + slot);
                    } else {
                        cp_async8(b + tid, A.src + row);
                    }
                }
                const int n = back ? S.nExtUp : S.nExtLo, x0 = back ? S.extUp : S.extLo;
                for (int k = tid; k < n; k += kPartThreads) {
                    cp_async16(c + W + k, A.col + x0 + k);
                    cp_async16(v + 4 * (W + k), A.coef + 4 * size_t(x0 + k));
                    cp_async16(v + 4 * (W + k) + 2, A.coef + 4 * size_t(x0 + k) + 2);
                }
            }
            cp_async_commit();
        };
        auto request = [&](int bx, const DiluMail*& m, double& v, unsigned long long& t) {
            m = nullptr;
            if (bx >= 0) {
                m = A.box + bx;
                mail_get(m, v, t);
            }
        };
        auto deliver = [&](int q, const DiluMail* m, double v, unsigned long long t) {
            if (q >= nSteps) return;
            const int i = back ? nSteps - 1 - q : q;
            double* rb = rem + (i & 1) * maxRem;
            if (m) rb[tid] = mail_wait(m, v, t, tag, A.limit, A.err);
            const DiluRecStep& S = steps[i];
            const int n = back ? S.nrup : S.nrlo;
            for (int k = tid + kPartThreads; k < n; k += kPartThreads) {
                const DiluMail* mk = A.box + __ldg(A.remote + (back ? S.rup : S.rlo) + k);
                double vk;
                unsigned long long tk;
                mail_get(mk, vk, tk);
                rb[k] = mail_wait(mk, vk, tk, tag, A.limit, A.err);
            }
        };
        for (int q = 0; q < R - 1; ++q) issue(q, ring + q * SB, back ? 0 : rowOf(q));
        int row1 = back ? 0 : rowOf(R - 1), row2 = back ? 0 : rowOf(R);  // of the next two steps to request
        const DiluMail *mCur, *mNext;
        double vCur = 0.0, vNext = 0.0;
        unsigned long long tCur = 0, tNext = 0;
        request(boxOf(0), mCur, vCur, tCur);
        deliver(0, mCur, vCur, tCur);
        request(boxOf(1), mCur, vCur, tCur);
        int box1 = boxOf(2), box2 = boxOf(3);
        int stage = 0, fill = R - 1;  // ring places of steps q and q + R - 1
        for (int q = 0; q < nSteps; ++q) {
            cp_async_wait_n(R - 2);
            __syncthreads();  // step q staged, step q - 1's values and step q's remote values visible
            issue(q + R - 1, ring + fill * SB, row1);
            row1 = row2;
            if (!back) row2 = rowOf(q + R + 1);
            request(box1, mNext, vNext, tNext);  // of step q + 2
            box1 = box2;
            box2 = boxOf(q + 4);
            const DiluRecStep& S = step(q);
            if (tid < S.width) {
                const char* sg = ring + stage * SB;
                const int4* c = reinterpret_cast<const int4*>(sg);
                const double* v = reinterpret_cast<const double*>(c + W + E);
                const double* b = v + 4 * (W + E);
                const int4 cc = c[tid];
                const double2 va = *reinterpret_cast<const double2*>(v + 4 * tid);
                const double2 vb = *reinterpret_cast<const double2*>(v + 4 * tid + 2);
                double x = b[tid];
                const double rd = vb.y;
                if (KIND == kPartForward) x = rd * x;
                // (an absent entry reads slot 0 and changes nothing)
                auto three = [&](const int4& k, double a0, double a1, double a2) {
                    const double y0 = sh[max(k.x, 0)], y1 = sh[max(k.y, 0)], y2 = sh[max(k.z, 0)];
                    if (KIND == kPartFactor) {
                        if (k.x >= 0) x -= a0 / y0;
                        if (k.y >= 0) x -= a1 / y1;
                        if (k.z >= 0) x -= a2 / y2;
                    } else {
                        const double z0 = x - rd * a0 * y0;
                        x = k.x >= 0 ? z0 : x;
                        const double z1 = x - rd * a1 * y1;
                        x = k.y >= 0 ? z1 : x;
                        const double z2 = x - rd * a2 * y2;
                        x = k.z >= 0 ? z2 : x;
                    }
                };
                three(cc, va.x, va.y, vb.x);
                const int e = (cc.w & 511) - 1;
                if (e >= 0) {
                    const double* ve = v + 4 * (W + e);
                    three(c[W + e], ve[0], ve[1], ve[2]);
                }
                const int slot = S.s0 + tid, mail = (cc.w >> 9) - 1;
                sh[slot - P.slot0] = x;
                if (mail >= 0) mail_put(A.box + mail, x, tag);
                if (KIND == kPartForward) A.ws[slot] = x;
                if (KIND == kPartBackward) A.w[reinterpret_cast<const int32_t*>(b + W)[tid]] = x;
                if (KIND == kPartFactor) {
                    const double inv = 1.0 / x;
                    A.rdLo[4 * size_t(slot) + 3] = inv;
                    A.rdUp[4 * size_t(slot) + 3] = inv;
                }
            }
            deliver(q + 1, mCur, vCur, tCur);
            mCur = mNext;
            vCur = vNext;
            tCur = tNext;
            stage = stage + 1 == R ? 0 : stage + 1;
            fill = fill + 1 == R ? 0 : fill + 1;
        }
        cp_async_wait<0>();
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&A.sync->done, 1u) == unsigned(A.nParts - 1)) {
            A.sync->ticket = 0;
            A.sync->done = 0;
            A.sync->epoch = tag;
        }
    }
}

}  // namespace vlm
