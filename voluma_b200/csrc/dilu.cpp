// Host construction of the DIC/DILU level schedule (see dilu.h).
#include "dilu.h"

#include <algorithm>
#include <stdexcept>
#include <tuple>
#include <utility>

namespace vlm {

namespace {

// Stable sort of a row's entries by the cell each names (perm0), ascending or descending; rows are short
// and mostly in order.
void sortRow(int32_t* col, int32_t* face, int n, const std::vector<int32_t>& cell, bool descending) {
    auto after = [&](int32_t a, int32_t b) { return descending ? cell[a] < cell[b] : cell[a] > cell[b]; };
    if (n > 32) {
        std::vector<std::pair<int32_t, int32_t>> e(static_cast<size_t>(n));
        for (int k = 0; k < n; ++k) e[size_t(k)] = {col[k], face[k]};
        std::stable_sort(e.begin(), e.end(), [&](const auto& a, const auto& b) { return after(b.first, a.first); });
        for (int k = 0; k < n; ++k) std::tie(col[k], face[k]) = e[size_t(k)];
        return;
    }
    for (int k = 1; k < n; ++k) {
        const int32_t c = col[k], f = face[k];
        int m = k;
        for (; m > 0 && after(col[m - 1], c); --m) {
            col[m] = col[m - 1];
            face[m] = face[m - 1];
        }
        col[m] = c;
        face[m] = f;
    }
}

}  // namespace

// Counting passes over flat arrays.  (A vector per row and a sort of all faces took 185 ms on the host for
// 80 x 64 x 48 cells, 25 ms now.)
DiluPlan buildDiluPlan(const std::vector<SysTopo>& systems, const BatchPlan& P) {
    const LevelPlan& L0 = P.levels[0];
    const int nrows = L0.nrows;
    DiluPlan D;
    // user cell -> level-0 row
    std::vector<int32_t> rowOf(static_cast<size_t>(P.userCells), -1);
    for (int r = 0; r < nrows; ++r)
        if (P.perm0[r] >= 0) rowOf[P.perm0[r]] = r;
    // faces whose two cells are distinct cells of their system (LinearSolver.cpp:34-42), in face order:
    // use(row of the upper cell, row of the lower cell, face word)
    auto faces = [&](auto&& use) {
        for (int s : P.order) {
            const SysTopo& T = systems[s];
            const int32_t* row = rowOf.data() + P.userCellBase[s];
            for (int f = 0; f < T.nInternal; ++f) {
                const int o = T.own[f], n = T.nei[f];
                if (o >= T.nCells || n >= T.nCells || o == n) continue;
                const int32_t flag = o < n ? int32_t(1u << 31) : 0;
                use(row[std::max(o, n)], row[std::min(o, n)], int32_t(P.userFaceBase[s] + f) | flag);
            }
        }
    };
    D.loPtr.assign(size_t(nrows) + 1, 0);
    D.upPtr.assign(size_t(nrows) + 1, 0);
    faces([&](int ru, int rl, int32_t) {
        ++D.loPtr[ru + 1];
        ++D.upPtr[rl + 1];
    });
    for (int r = 0; r < nrows; ++r) {
        D.maxEnt = std::max({D.maxEnt, D.loPtr[r + 1], D.upPtr[r + 1]});
        D.loPtr[r + 1] += D.loPtr[r];
        D.upPtr[r + 1] += D.upPtr[r];
    }
    D.loCol.resize(size_t(D.loPtr[nrows]));
    D.loFace.resize(D.loCol.size());
    D.upCol.resize(size_t(D.upPtr[nrows]));
    D.upFace.resize(D.upCol.size());
    {
        // lower entries forwards, upper ones backwards: each row's by ascending / descending face
        std::vector<int32_t> lo(D.loPtr.begin(), D.loPtr.end() - 1), up(D.upPtr.begin() + 1, D.upPtr.end());
        faces([&](int ru, int rl, int32_t face) {
            const int a = lo[ru]++, b = --up[rl];
            D.loCol[a] = rl;
            D.loFace[a] = face;
            D.upCol[b] = ru;
            D.upFace[b] = face;
        });
    }
    for (int r = 0; r < nrows; ++r) {
        sortRow(D.loCol.data() + D.loPtr[r], D.loFace.data() + D.loPtr[r], D.loPtr[r + 1] - D.loPtr[r], P.perm0, false);
        sortRow(D.upCol.data() + D.upPtr[r], D.upFace.data() + D.upPtr[r], D.upPtr[r + 1] - D.upPtr[r], P.perm0, true);
    }
    // levels in natural order; padding rows (no neighbours, diag 1, r 0) stay on level 0
    std::vector<int32_t> level(static_cast<size_t>(nrows), 0);
    D.levPtr.push_back(0);
    D.levRows.resize(size_t(nrows));
    for (int b = 0; b < P.nsys; ++b) {
        const int s = P.order[b];
        int nLev = 1;
        for (int c = 0; c < systems[s].nCells; ++c) {
            const int r = rowOf[P.userCellBase[s] + c];
            int lv = 0;
            for (int k = D.loPtr[r]; k < D.loPtr[r + 1]; ++k) lv = std::max(lv, level[D.loCol[k]] + 1);
            level[r] = lv;
            nLev = std::max(nLev, lv + 1);
        }
        DiluSys ds{};
        ds.sys = b;
        ds.levBegin = int(D.levPtr.size()) - 1;
        ds.nLev = nLev;
        ds.rowBegin = L0.sysRow[b];
        ds.rowCount = L0.sysRow[b + 1] - L0.sysRow[b];
        // rows by level, ascending within one
        std::vector<int32_t> at(size_t(nLev) + 1, 0);
        for (int r = ds.rowBegin; r < ds.rowBegin + ds.rowCount; ++r) ++at[level[r] + 1];
        at[0] = D.levPtr.back();
        for (int t = 0; t < nLev; ++t) {
            D.maxWidth = std::max(D.maxWidth, at[t + 1]);
            at[t + 1] += at[t];
            D.levPtr.push_back(at[t + 1]);
        }
        for (int r = ds.rowBegin; r < ds.rowBegin + ds.rowCount; ++r) D.levRows[at[level[r]]++] = r;
        D.maxRows = std::max(D.maxRows, ds.rowCount);
        D.maxLevels = std::max(D.maxLevels, nLev);
        D.sys.push_back(ds);
    }
    return D;
}

void addDiluStream(DiluPlan& D) {
    for (DiluSys& ds : D.sys) {
        ds.slotBegin = D.levPtr[ds.levBegin];
        ds.slotEnd = D.levPtr[ds.levBegin + ds.nLev];
        ds.loBegin = int(D.sLoCol.size());
        ds.upBegin = int(D.sUpCol.size());
        for (int t = ds.levBegin; t < ds.levBegin + ds.nLev; ++t) {
            const int a = D.levPtr[t], e = D.levPtr[t + 1];
            DiluLevel lv{a, e - a, 0, 0, 0, 0};
            for (int i = a; i < e; ++i) {
                const int r = D.levRows[i];
                lv.mlo = std::max(lv.mlo, D.loPtr[r + 1] - D.loPtr[r]);
                lv.mup = std::max(lv.mup, D.upPtr[r + 1] - D.upPtr[r]);
                D.slotRow.push_back(r - ds.rowBegin);
            }
            auto entries = [&](int m, const std::vector<int32_t>& ptr, const std::vector<int32_t>& col,
                               const std::vector<int32_t>& face, std::vector<int32_t>& outCol,
                               std::vector<int32_t>& outFace) {
                const int first = int(outCol.size());
                for (int j = 0; j < m; ++j)
                    for (int i = a; i < e; ++i) {
                        const int k = ptr[D.levRows[i]] + j;
                        const bool has = k < ptr[D.levRows[i] + 1];
                        outCol.push_back(has ? col[k] - ds.rowBegin : -1);
                        outFace.push_back(has ? face[k] : 0);
                    }
                return first;
            };
            lv.lo = entries(lv.mlo, D.loPtr, D.loCol, D.loFace, D.sLoCol, D.sLoFace);
            lv.up = entries(lv.mup, D.upPtr, D.upCol, D.upFace, D.sUpCol, D.sUpFace);
            D.lev.push_back(lv);
        }
        ds.loEnd = int(D.sLoCol.size());
        ds.upEnd = int(D.sUpCol.size());
    }
}

int diluWidth(const DiluPlan& D, const DiluSys& ds, const BatchPlan& P) {
    int width = 0;
    for (int t = 0; t < ds.nLev; ++t) {
        const auto a = D.levRows.begin() + D.levPtr[ds.levBegin + t], e = D.levRows.begin() + D.levPtr[ds.levBegin + t + 1];
        const auto real = t == 0 ? std::count_if(a, e, [&](int r) { return P.perm0[r] >= 0; }) : e - a;
        width = std::max(width, int(real));
    }
    return width;
}

DiluParts buildDiluParts(const DiluPlan& D, const BatchPlan& P, const std::vector<int>& nParts, int maxWidth) {
    DiluParts R;
    const int nrows = int(P.perm0.size());
    std::vector<int32_t> partOf(size_t(nrows), -1), slotOf(size_t(nrows), -1);
    // slots: per part and level the rows of that level, in steps of at most maxWidth
    for (const DiluSys& ds : D.sys) {
        const int64_t n = P.sysCells[ds.sys], cb = P.userCellBase[P.order[ds.sys]];
        const int np = std::max(1, std::min<int>(nParts[ds.sys], int(std::max<int64_t>(n, 1))));
        const int part0 = int(R.parts.size());
        std::vector<std::vector<int32_t>> rows(static_cast<size_t>(np));  // level by level
        std::vector<std::vector<int32_t>> ends(static_cast<size_t>(np));  // end of each non-empty level's rows
        std::vector<int32_t> pads;
        for (int t = 0; t < ds.nLev; ++t) {
            for (int k = D.levPtr[ds.levBegin + t]; k < D.levPtr[ds.levBegin + t + 1]; ++k) {
                const int r = D.levRows[k];
                if (P.perm0[r] < 0) {  // padding: no neighbours, no step
                    pads.push_back(r);
                    continue;
                }
                const int q = int((P.perm0[r] - cb) * np / n);
                partOf[r] = part0 + q;
                rows[q].push_back(r);
            }
            for (int q = 0; q < np; ++q)
                if (int(rows[q].size()) > (ends[q].empty() ? 0 : ends[q].back())) ends[q].push_back(int(rows[q].size()));
        }
        for (int q = 0; q < np; ++q) {
            DiluPart part{ds.sys, int(R.steps.size()), 0, int(R.slotRow.size()), int(rows[q].size()), 0, 0};
            const size_t p0 = pads.size() * size_t(q) / size_t(np), p1 = pads.size() * size_t(q + 1) / size_t(np);
            part.pad0 = int(R.padRow.size());
            part.nPad = int(p1 - p0);
            R.padRow.insert(R.padRow.end(), pads.begin() + std::ptrdiff_t(p0), pads.begin() + std::ptrdiff_t(p1));
            int a = 0;
            for (int e : ends[q])
                while (a < e) {
                    const int w = std::min(maxWidth, e - a);
                    DiluStep st = {};
                    st.s0 = part.slot0 + a;
                    st.width = w;
                    R.steps.push_back(st);
                    R.maxWidth = std::max(R.maxWidth, w);
                    a += w;
                }
            part.nSteps = int(R.steps.size()) - part.stepBegin;
            for (int r : rows[q]) {
                slotOf[r] = int(R.slotRow.size());
                R.slotRow.push_back(r);
            }
            R.maxSlots = std::max(R.maxSlots, part.nSlots);
            R.parts.push_back(part);
        }
    }
    // mailboxes: one per row read by another part, per direction
    R.loMail.assign(R.slotRow.size(), -1);
    R.upMail.assign(R.slotRow.size(), -1);
    for (int r : R.slotRow) {
        for (int k = D.loPtr[r]; k < D.loPtr[r + 1]; ++k)
            if (partOf[D.loCol[k]] != partOf[r] && R.loMail[slotOf[D.loCol[k]]] < 0)
                R.loMail[slotOf[D.loCol[k]]] = R.nLoMail++;
        for (int k = D.upPtr[r]; k < D.upPtr[r + 1]; ++k)
            if (partOf[D.upCol[k]] != partOf[r] && R.upMail[slotOf[D.upCol[k]]] < 0)
                R.upMail[slotOf[D.upCol[k]]] = R.nUpMail++;
    }
    R.loCol.reserve(D.loCol.size() * 3 / 2);
    R.loFace.reserve(D.loCol.size() * 3 / 2);
    R.upCol.reserve(D.upCol.size() * 3 / 2);
    R.upFace.reserve(D.upCol.size() * 3 / 2);
    // entries, column-major per step
    auto fill = [&](const DiluPart& part, const DiluStep& st, const std::vector<int32_t>& ptr,
                    const std::vector<int32_t>& col, const std::vector<int32_t>& face,
                    const std::vector<int32_t>& mail, std::vector<int32_t>& outCol, std::vector<int32_t>& outFace,
                    std::vector<int32_t>& remote, int& e0, int& m, int& r0, int& nr) {
        e0 = int(outCol.size());
        r0 = int(remote.size());
        m = 0;
        for (int q = 0; q < st.width; ++q) {
            const int r = R.slotRow[st.s0 + q];
            m = std::max(m, int(ptr[r + 1] - ptr[r]));
        }
        outCol.resize(outCol.size() + size_t(m) * st.width, -1);
        outFace.resize(outCol.size(), 0);
        const int slot1 = part.slot0 + part.nSlots;
        for (int j = 0; j < m; ++j)
            for (int q = 0; q < st.width; ++q) {
                const int r = R.slotRow[st.s0 + q];
                const int k = ptr[r] + j;
                if (k >= ptr[r + 1]) continue;
                const int slot = slotOf[col[k]];
                int32_t& e = outCol[size_t(e0) + size_t(j) * st.width + q];
                if (slot >= part.slot0 && slot < slot1) {
                    e = slot - part.slot0;
                } else {
                    e = -2 - (int(remote.size()) - r0);
                    remote.push_back(mail[slot]);
                }
                outFace[size_t(e0) + size_t(j) * st.width + q] = face[k];
            }
        nr = int(remote.size()) - r0;
        R.maxRemote = std::max(R.maxRemote, nr);
    };
    for (const DiluPart& part : R.parts)
        for (int t = part.stepBegin; t < part.stepBegin + part.nSteps; ++t) {
            DiluStep& st = R.steps[t];
            fill(part, st, D.loPtr, D.loCol, D.loFace, R.loMail, R.loCol, R.loFace, R.loRemote, st.lo, st.mlo, st.rlo,
                 st.nrlo);
            fill(part, st, D.upPtr, D.upCol, D.upFace, R.upMail, R.upCol, R.upFace, R.upRemote, st.up, st.mup, st.rup,
                 st.nrup);
        }
    return R;
}

bool buildDiluRecords(const DiluParts& R, DiluRecords& out) {
    const size_t ns = R.slotRow.size();
    out = DiluRecords{};
    if (R.nLoMail >= (1 << 21) || R.nUpMail >= (1 << 21)) return false;
    out.steps.resize(R.steps.size());
    for (int dir = 0; dir < 2; ++dir) {
        const std::vector<int32_t>&col = dir ? R.upCol : R.loCol, &face = dir ? R.upFace : R.loFace,
                         &mail = dir ? R.upMail : R.loMail;
        std::vector<int32_t>&oc = dir ? out.upCol : out.loCol, &of = dir ? out.upFace : out.loFace;
        oc.assign(4 * ns, -1);
        of.assign(4 * ns, DiluRecords::kNoFace);
        for (const DiluPart& P : R.parts) {
            out.maxSteps = std::max(out.maxSteps, P.nSteps);
            for (int i = 0; i < P.nSteps; ++i) {
                const DiluStep& S = R.steps[size_t(P.stepBegin + i)];
                DiluRecStep& T = out.steps[size_t(P.stepBegin + i)];
                T.s0 = S.s0;
                T.width = S.width;
                T.rlo = S.rlo;
                T.nrlo = S.nrlo;
                T.rup = S.rup;
                T.nrup = S.nrup;
                const int e0 = dir ? S.up : S.lo, m = dir ? S.mup : S.mlo;
                if (m > 6) return false;
                const int ext0 = int(oc.size() / 4);
                int nExt = 0;
                for (int q = 0; q < S.width; ++q) {
                    const size_t slot = size_t(S.s0 + q);
                    int n = 0;
                    while (n < m && col[size_t(e0 + n * S.width + q)] != -1) ++n;
                    size_t ext = 0;
                    if (n > 3) {
                        ext = size_t(ext0 + nExt++);
                        oc.resize(4 * (ext + 1), -1);
                        of.resize(4 * (ext + 1), DiluRecords::kNoFace);
                    }
                    for (int j = 0; j < n; ++j) {
                        const size_t at = j < 3 ? 4 * slot + size_t(j) : 4 * ext + size_t(j - 3);
                        const int l = col[size_t(e0 + j * S.width + q)];
                        oc[at] = l >= 0 ? l : P.nSlots + (i & 1) * R.maxRemote + (-2 - l);
                        of[at] = face[size_t(e0 + j * S.width + q)];
                    }
                    oc[4 * slot + 3] = ((mail[slot] + 1) << 9) | (n > 3 ? int(ext) - ext0 + 1 : 0);
                }
                if (nExt >= 511) return false;
                (dir ? T.extUp : T.extLo) = ext0;
                (dir ? T.nExtUp : T.nExtLo) = nExt;
                out.maxExt = std::max(out.maxExt, nExt);
            }
        }
        (dir ? out.nUp : out.nLo) = int(oc.size() / 4);
    }
    return true;
}

}  // namespace vlm
