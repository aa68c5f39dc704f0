// Images of the shared-memory coarse tail: per system and CTA of its cluster, the CTA's 32-row slices
// of the levels first..coarsest-1 (values gathered per solve through `codes`, structure with 16-bit
// local indices); offsets as TailPart describes them.
#include "tailplan.h"

#include <algorithm>
#include <cstring>

namespace vlm {

namespace {

// Where one system's vectors lie in every part's shared memory, levels f on.
struct Vectors {
    int count = 0;
    int n[kTailMaxLevels] = {}, tX[kTailMaxLevels] = {}, tX2[kTailMaxLevels] = {}, tR[kTailMaxLevels] = {};

    Vectors(const TailSys& s, int f, int CL) {
        for (int k = f; k <= s.coarsest; ++k) {
            n[k] = s.rowCount[k];
            tX[k] = count;
            tX2[k] = count + n[k];
            count += 2 * n[k];
            if (k < s.coarsest) {
                tR[k] = count;
                count += (n[k] / kSlice + CL - 1) / CL * kSlice;
            }
        }
        count = (count + 3) & ~3;  // whole 16-byte words in both precisions
    }
    // rows of level k that part `rank` holds
    int rows(int k, int rank, int CL) const {
        const int ns = n[k] / kSlice;
        return ns > rank ? (ns - rank + CL - 1) / CL * kSlice : 0;
    }
};

// Largest part of system s from level f on, in bytes of shared memory; 0 when the parts do not fit `budget`
// or their indices 16 bits.  Nothing is built for a level that does not fit.
size_t partBytes(const BatchPlan& plan, const TailSys& s, int f, int CL, size_t tsize, size_t budget) {
    const int c = s.coarsest;
    if (c >= kTailMaxLevels || c > 31) return 0;
    for (int k = f; k <= c; ++k)
        if (s.rowCount[k] >= 0xffff || s.rowCount[k] % kSlice != 0 || s.rowStart[k] % kSlice != 0) return 0;
    if (s.coarseN > s.rowCount[c]) return 0;
    const Vectors v(s, f, CL);
    if (size_t(v.count) * tsize > budget) return 0;
    for (int k = f; k < c; ++k) {
        const LevelPlan& P = plan.levels[k];
        if (P.col.empty() || P.rlen.size() < size_t(s.rowStart[k] + v.n[k])) return 0;  // host structure released
        if (s.rowStart[k] + v.n[k] > (1 << 25) || P.slPtr[size_t((s.rowStart[k] + v.n[k]) / kSlice)] >= (1 << 25)) return 0;
    }
    if (f == 0 && c > 0)
        for (int q = 0; q < s.nColours; ++q)
            if ((s.grpStart[q] - s.rowStart[0]) % kSlice != 0 || s.grpCount[q] % kSlice != 0) return 0;
    size_t largest = 0;
    for (int rank = 0; rank < CL; ++rank) {
        size_t val = 0, str = 0;
        for (int k = f; k < c; ++k) {
            const LevelPlan& P = plan.levels[k];
            const int nl = v.rows(k, rank, CL), nl1 = v.rows(k + 1, rank, CL);
            size_t ent = 0, kids = 0;
            for (int l = 0; l < nl; l += kSlice) {
                const size_t sl = size_t(s.rowStart[k] / kSlice + l / kSlice * CL + rank);
                ent += size_t(P.slPtr[sl + 1] - P.slPtr[sl]);
            }
            for (int l = 0; l < nl1; l += kSlice) {
                const size_t R = size_t(s.rowStart[k + 1] + (l / kSlice * CL + rank) * kSlice);
                kids += size_t(P.childPtr[R + kSlice] - P.childPtr[R]);
            }
            if (ent / kSlice > 0xffff || kids > 0xffff) return 0;
            val += size_t(nl) + ent;
            str += 2 * size_t(nl) + size_t(nl / kSlice) + ent + size_t(nl1) + 1 + kids;
        }
        val = (val + 3) & ~size_t(3);
        str = (str + 7) & ~size_t(7);
        const size_t inv = size_t(s.coarseN) * size_t((s.coarseN + CL - 1) / CL);
        if ((size_t(v.count) + val) * tsize > budget || str * sizeof(uint16_t) > budget) return 0;
        const size_t bytes = tail_smem_bytes(tsize, int(size_t(v.count) + val), int(inv), int(str));
        if (bytes > budget) return 0;
        largest = std::max(largest, bytes);
    }
    return largest;
}

// One system's parts from level f on, appended to `out`; false when the plan's indices are inconsistent.
bool appendSystem(const BatchPlan& plan, const TailSys& s, int f, int CL, TailImages& out) {
    const int c = s.coarsest;
    const Vectors v(s, f, CL);
    for (int rank = 0; rank < CL; ++rank) {
        TailPart I;
        std::memset(&I, 0, sizeof I);
        I.sys = s.sys;
        I.first = f;
        I.coarsest = c;
        I.nc = s.coarseN;
        I.invOffset = s.invOffset;
        I.vecCount = v.count;
        I.two = s.two;
        I.nColours = s.nColours;
        if (f == 0 && c > 0)
            for (int q = 0; q < s.nColours; ++q) {
                I.grpStart[q] = s.grpStart[q] - s.rowStart[0];
                I.grpCount[q] = s.grpCount[q];
            }
        for (int k = f; k <= c; ++k) {
            I.n[k] = v.n[k];
            I.rowStart[k] = s.rowStart[k];
            I.nl[k] = v.rows(k, rank, CL);
            I.tX[k] = v.tX[k];
            I.tX2[k] = v.tX2[k];
            I.tR[k] = v.tR[k];
        }
        // value image: per level the diagonal of this CTA's rows, then its slices' entries
        I.valOff = int(out.codes.size());
        int tc = 0;
        for (int k = f; k < c; ++k) {
            const LevelPlan& P = plan.levels[k];
            const int slice0 = s.rowStart[k] / kSlice;
            I.tDiag[k] = v.count + tc;
            for (int l = 0; l < I.nl[k]; l += kSlice) {
                const int row = s.rowStart[k] + (l / kSlice * CL + rank) * kSlice;
                for (int i = 0; i < kSlice; ++i) out.codes.push_back((k << 26) | (1 << 25) | (row + i));
            }
            tc += I.nl[k];
            I.tVal[k] = v.count + tc;
            for (int l = 0; l < I.nl[k]; l += kSlice) {
                const int sl = slice0 + l / kSlice * CL + rank;
                const int e0 = P.slPtr[size_t(sl)], e1 = P.slPtr[size_t(sl) + 1];
                const int32_t* rlen = P.rlen.data() + size_t(sl) * kSlice;
                out.codes.resize(out.codes.size() + size_t(e1 - e0));
                int32_t* w = out.codes.data() + out.codes.size() - size_t(e1 - e0);
                for (int e = e0, q = 0; e < e1; e += kSlice, ++q, w += kSlice)
                    for (int i = 0; i < kSlice; ++i) w[i] = q < rlen[i] ? (k << 26) | (e + i) : -1;
                tc += e1 - e0;
            }
        }
        while (tc % 4) {
            out.codes.push_back(-1);
            ++tc;
        }
        I.valCount = tc;
        // structure image: row lengths, slice offsets, level-local columns, aggregates, children
        I.strOff = int(out.str.size());
        const size_t str0 = out.str.size();
        auto at = [&] { return int(out.str.size() - str0); };
        auto push = [&](int w) { out.str.push_back(uint16_t(w)); };
        for (int k = f; k < c; ++k) {
            const LevelPlan& P = plan.levels[k];
            const int rs = s.rowStart[k], slice0 = rs / kSlice, rs1 = s.rowStart[k + 1];
            auto row = [&](int l) { return rs + (l / kSlice * CL + rank) * kSlice + l % kSlice; };
            I.uRlen[k] = at();
            for (int l = 0; l < I.nl[k]; ++l) push(P.rlen[size_t(row(l))]);
            I.uSlice[k] = at();
            int off = 0;
            for (int l = 0; l < I.nl[k]; l += kSlice) {
                push(off);
                const int sl = slice0 + l / kSlice * CL + rank;
                off += (P.slPtr[size_t(sl) + 1] - P.slPtr[size_t(sl)]) / kSlice;
            }
            I.uCol[k] = at();
            for (int l = 0; l < I.nl[k]; l += kSlice) {
                const int sl = slice0 + l / kSlice * CL + rank;
                const int e0 = P.slPtr[size_t(sl)], e1 = P.slPtr[size_t(sl) + 1];
                const int32_t* rlen = P.rlen.data() + size_t(sl) * kSlice;
                out.str.resize(out.str.size() + size_t(e1 - e0));
                uint16_t* w = out.str.data() + out.str.size() - size_t(e1 - e0);
                const int32_t* col = P.col.data() + e0;
                bool ok = true;
                for (int e = e0, q = 0; e < e1; e += kSlice, ++q, w += kSlice, col += kSlice)
                    for (int i = 0; i < kSlice; ++i) {
                        const int cl = q < rlen[i] ? col[i] - rs : 0;
                        ok = ok && cl >= 0 && cl < v.n[k];
                        w[i] = uint16_t(cl);
                    }
                if (!ok) return false;
            }
            I.uAgg[k] = at();
            for (int l = 0; l < I.nl[k]; ++l) {
                const int a = P.agg[size_t(row(l))];
                if (a >= 0 && (a - rs1 < 0 || a - rs1 >= v.n[k + 1])) return false;
                push(a < 0 ? 0xffff : a - rs1);
            }
            // children of this CTA's rows of the next level
            auto crow = [&](int l) { return rs1 + (l / kSlice * CL + rank) * kSlice + l % kSlice; };
            I.uCptr[k] = at();
            int cnt = 0;
            push(0);
            for (int l = 0; l < I.nl[k + 1]; ++l) {
                cnt += P.childPtr[size_t(crow(l)) + 1] - P.childPtr[size_t(crow(l))];
                push(cnt);
            }
            I.uChild[k] = at();
            for (int l = 0; l < I.nl[k + 1]; ++l)
                for (int q = P.childPtr[size_t(crow(l))]; q < P.childPtr[size_t(crow(l)) + 1]; ++q) {
                    const int w = P.child[size_t(q)] - rs;
                    if (w < 0 || w >= v.n[k]) return false;
                    push(w);
                }
        }
        while (at() % 8) push(0);
        I.strCount = at();
        out.parts.push_back(I);
    }
    return true;
}

}  // namespace

bool tailStarts(const BatchPlan& plan, const std::vector<TailSys>& ts, int cluster, size_t tsize, size_t budget,
                std::vector<int>& first, size_t& bytes) {
    first.clear();
    bytes = 0;
    for (const TailSys& s : ts) {
        int f = s.first;
        size_t b = 0;
        while (f <= s.coarsest && (b = partBytes(plan, s, f, cluster, tsize, budget)) == 0) ++f;
        if (f > s.coarsest) return false;
        first.push_back(f);
        bytes = std::max(bytes, b);
    }
    return !ts.empty();
}

bool buildTailImages(const BatchPlan& plan, const std::vector<TailSys>& ts, const std::vector<int>& first, int cluster,
                     TailImages& out) {
    out = TailImages();
    for (size_t b = 0; b < ts.size(); ++b)
        if (!appendSystem(plan, ts[b], first[b], cluster, out)) return false;
    return true;
}

}  // namespace vlm
