// Images of the shared-memory coarse tail: per system and CTA of its cluster, the CTA's 32-row slices
// of the levels first..coarsest-1 (values gathered per solve through `codes`, structure with 16-bit
// local indices); offsets as TailPart describes them.
#include "tailplan.h"

#include <algorithm>
#include <cstring>

namespace vlm {

namespace {

// One system's parts from level f on, appended to `out`; false (and nothing appended) when they do not fit.
bool appendSystem(const BatchPlan& plan, const TailSys& s, int f, int CL, size_t tsize, size_t budget, TailImages& out) {
    const int c = s.coarsest;
    if (c >= kTailMaxLevels || c > 31) return false;
    int vec = 0;
    int n[kTailMaxLevels], tX[kTailMaxLevels], tX2[kTailMaxLevels], tR[kTailMaxLevels] = {};
    for (int k = f; k <= c; ++k) {
        n[k] = s.rowCount[k];
        if (n[k] >= 0xffff || n[k] % kSlice != 0 || s.rowStart[k] % kSlice != 0) return false;
        tX[k] = vec;
        tX2[k] = vec + n[k];
        vec += 2 * n[k];
        if (k < c) {
            tR[k] = vec;
            vec += (n[k] / kSlice + CL - 1) / CL * kSlice;
        }
    }
    vec = (vec + 3) & ~3;  // whole 16-byte words in both precisions
    if (s.coarseN > n[c]) return false;
    if (size_t(vec) * tsize > budget) return false;
    for (int k = f; k < c; ++k) {
        const LevelPlan& P = plan.levels[k];
        if (P.col.empty() || P.rlen.size() < size_t(s.rowStart[k] + n[k])) return false;  // host structure released
    }
    const size_t nParts = out.parts.size(), nCodes = out.codes.size(), nStr = out.str.size();
    auto fail = [&] {
        out.parts.resize(nParts);
        out.codes.resize(nCodes);
        out.str.resize(nStr);
        return false;
    };
    const int invRows = (s.coarseN + CL - 1) / CL;
    size_t largest = out.bytes;
    for (int rank = 0; rank < CL; ++rank) {
        TailPart I;
        std::memset(&I, 0, sizeof I);
        I.sys = s.sys;
        I.first = f;
        I.coarsest = c;
        I.nc = s.coarseN;
        I.invOffset = s.invOffset;
        I.vecCount = vec;
        I.two = s.two;
        I.nColours = s.nColours;
        if (f == 0 && c > 0)
            for (int q = 0; q < s.nColours; ++q) {
                I.grpStart[q] = s.grpStart[q] - s.rowStart[0];
                I.grpCount[q] = s.grpCount[q];
                if (I.grpStart[q] % kSlice != 0 || I.grpCount[q] % kSlice != 0) return fail();
            }
        for (int k = f; k <= c; ++k) {
            I.n[k] = n[k];
            I.rowStart[k] = s.rowStart[k];
            const int ns = n[k] / kSlice;
            I.nl[k] = ns > rank ? (ns - rank + CL - 1) / CL * kSlice : 0;
            I.tX[k] = tX[k];
            I.tX2[k] = tX2[k];
            I.tR[k] = tR[k];
        }
        // value image: per level the diagonal of this CTA's rows, then its slices' entries
        I.valOff = int(out.codes.size());
        int tc = 0;
        for (int k = f; k < c; ++k) {
            const LevelPlan& P = plan.levels[k];
            const int slice0 = s.rowStart[k] / kSlice;
            I.tDiag[k] = vec + tc;
            for (int l = 0; l < I.nl[k]; l += kSlice)
                for (int i = 0; i < kSlice; ++i) {
                    const int row = s.rowStart[k] + (l / kSlice * CL + rank) * kSlice + i;
                    if (row >= (1 << 25)) return fail();
                    out.codes.push_back((k << 26) | (1 << 25) | row);
                }
            tc += I.nl[k];
            I.tVal[k] = vec + tc;
            for (int l = 0; l < I.nl[k]; l += kSlice) {
                const int sl = slice0 + l / kSlice * CL + rank;
                const int e0 = P.slPtr[size_t(sl)], e1 = P.slPtr[size_t(sl) + 1];
                if (e1 >= (1 << 25)) return fail();
                for (int e = e0; e < e1; ++e) {
                    const int q = (e - e0) / kSlice;
                    const bool real = q < P.rlen[size_t(sl * kSlice + (e - e0) % kSlice)];
                    out.codes.push_back(real ? (k << 26) | e : -1);
                }
                tc += e1 - e0;
            }
            if (size_t(vec + tc) * tsize > budget) return fail();
        }
        while (tc % 4) {
            out.codes.push_back(-1);
            ++tc;
        }
        I.valCount = tc;
        // structure image: row lengths, slice offsets, level-local columns, aggregates, children
        I.strOff = int(out.str.size());
        int su = 0;
        bool fits = true;
        auto push = [&](int v) {
            if (v < 0 || v > 0xffff) fits = false;
            out.str.push_back(uint16_t(v));
            ++su;
        };
        for (int k = f; k < c; ++k) {
            const LevelPlan& P = plan.levels[k];
            const int rs = s.rowStart[k], slice0 = rs / kSlice, rs1 = s.rowStart[k + 1];
            auto row = [&](int l) { return rs + (l / kSlice * CL + rank) * kSlice + l % kSlice; };
            I.uRlen[k] = su;
            for (int l = 0; l < I.nl[k]; ++l) push(P.rlen[size_t(row(l))]);
            I.uSlice[k] = su;
            int off = 0;
            for (int l = 0; l < I.nl[k]; l += kSlice) {
                push(off);
                const int sl = slice0 + l / kSlice * CL + rank;
                off += (P.slPtr[size_t(sl) + 1] - P.slPtr[size_t(sl)]) / kSlice;
            }
            I.uCol[k] = su;
            for (int l = 0; l < I.nl[k]; l += kSlice) {
                const int sl = slice0 + l / kSlice * CL + rank;
                const int e0 = P.slPtr[size_t(sl)], e1 = P.slPtr[size_t(sl) + 1];
                for (int e = e0; e < e1; ++e) {
                    int cl = 0;
                    if ((e - e0) / kSlice < P.rlen[size_t(sl * kSlice + (e - e0) % kSlice)]) {
                        cl = P.col[size_t(e)] - rs;
                        if (cl < 0 || cl >= n[k]) return fail();
                    }
                    push(cl);
                }
            }
            I.uAgg[k] = su;
            for (int l = 0; l < I.nl[k]; ++l) {
                const int a = P.agg[size_t(row(l))];
                if (a >= 0 && (a - rs1 < 0 || a - rs1 >= n[k + 1])) return fail();
                push(a < 0 ? 0xffff : a - rs1);
            }
            // children of this CTA's rows of the next level
            auto crow = [&](int l) { return rs1 + (l / kSlice * CL + rank) * kSlice + l % kSlice; };
            I.uCptr[k] = su;
            int cnt = 0;
            push(0);
            for (int l = 0; l < I.nl[k + 1]; ++l) {
                cnt += P.childPtr[size_t(crow(l)) + 1] - P.childPtr[size_t(crow(l))];
                push(cnt);
            }
            I.uChild[k] = su;
            for (int l = 0; l < I.nl[k + 1]; ++l)
                for (int q = P.childPtr[size_t(crow(l))]; q < P.childPtr[size_t(crow(l)) + 1]; ++q) {
                    const int v = P.child[size_t(q)] - rs;
                    if (v < 0 || v >= n[k]) return fail();
                    push(v);
                }
        }
        while (su % 8) push(0);
        I.strCount = su;
        const size_t bytes = tail_smem_bytes(tsize, vec + tc, s.coarseN * invRows, su);
        if (!fits || bytes > budget) return fail();
        largest = std::max(largest, bytes);
        out.parts.push_back(I);
    }
    out.bytes = largest;
    return true;
}

}  // namespace

bool buildTailImages(const BatchPlan& plan, const std::vector<TailSys>& ts, int cluster, size_t tsize, size_t budget,
                     TailImages& out) {
    out = TailImages();
    for (const TailSys& s : ts) {
        int f = s.first;
        while (f <= s.coarsest && !appendSystem(plan, s, f, cluster, tsize, budget, out)) ++f;
        if (f > s.coarsest) return false;
        out.first.push_back(f);
    }
    return !ts.empty();
}

}  // namespace vlm
