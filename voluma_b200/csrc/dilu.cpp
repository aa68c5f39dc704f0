// Host construction of the DIC/DILU level schedule (see dilu.h).
#include "dilu.h"

#include <algorithm>
#include <array>
#include <stdexcept>

namespace vlm {

DiluPlan buildDiluPlan(const std::vector<SysTopo>& systems, const BatchPlan& P) {
    const LevelPlan& L0 = P.levels[0];
    const int nrows = L0.nrows;
    DiluPlan D;
    // user cell -> level-0 row
    std::vector<int32_t> rowOf(static_cast<size_t>(P.userCells), -1);
    for (int r = 0; r < nrows; ++r)
        if (P.perm0[r] >= 0) rowOf[P.perm0[r]] = r;
    std::vector<std::vector<std::array<int32_t, 3>>> lo(static_cast<size_t>(nrows)), up(static_cast<size_t>(nrows));
    D.levPtr.push_back(0);
    for (int b = 0; b < P.nsys; ++b) {
        const int s = P.order[b];
        const SysTopo& T = systems[s];
        const int64_t cb = P.userCellBase[s], fb = P.userFaceBase[s];
        // faces whose two cells are distinct cells of this system (LinearSolver.cpp:34-42)
        std::vector<std::array<int32_t, 3>> faces;  // (u, l, f)
        faces.reserve(size_t(T.nInternal));
        for (int f = 0; f < T.nInternal; ++f) {
            const int o = T.own[f], n = T.nei[f];
            if (o >= T.nCells || n >= T.nCells || o == n) continue;
            faces.push_back({std::max(o, n), std::min(o, n), f});
        }
        std::sort(faces.begin(), faces.end());
        for (const auto& t : faces) {
            const int u = t[0], l = t[1], f = t[2];
            const int32_t flag = T.own[f] == l ? int32_t(1u << 31) : 0;
            const int32_t face = int32_t(fb + f) | flag;
            const int32_t ru = rowOf[cb + u], rl = rowOf[cb + l];
            lo[ru].push_back({ru, rl, face});  // appended in ascending (l, f) for this u
            up[rl].push_back({rl, ru, face});  // ascending (u, f) for this l: reversed below
        }
        // levels in natural order
        std::vector<int32_t> level(static_cast<size_t>(T.nCells), 0);
        int nLev = 1;
        for (int c = 0; c < T.nCells; ++c) {
            int lv = 0;
            for (const auto& e : lo[rowOf[cb + c]]) {
                // e[1] is a solver row; its natural cell is perm0 - cb
                lv = std::max(lv, level[P.perm0[e[1]] - cb] + 1);
            }
            level[c] = lv;
            nLev = std::max(nLev, lv + 1);
        }
        std::vector<std::vector<int32_t>> byLevel(static_cast<size_t>(nLev));
        for (int c = 0; c < T.nCells; ++c) byLevel[level[c]].push_back(rowOf[cb + c]);
        // padding rows of this system: level 0 (no neighbours, diag 1, r 0)
        for (int r = L0.sysRow[b]; r < L0.sysRow[b + 1]; ++r)
            if (P.perm0[r] < 0) byLevel[0].push_back(r);
        DiluSys ds;
        ds.sys = b;
        ds.levBegin = int(D.levPtr.size()) - 1;
        ds.nLev = nLev;
        ds.rowBegin = L0.sysRow[b];
        ds.rowCount = L0.sysRow[b + 1] - L0.sysRow[b];
        ds.slotBegin = int(D.levRows.size());
        ds.loBegin = int(D.sLoCol.size());
        ds.upBegin = int(D.sUpCol.size());
        D.maxRows = std::max(D.maxRows, ds.rowCount);
        for (auto& v : byLevel) {
            std::sort(v.begin(), v.end());
            const int width = int(v.size());
            D.maxWidth = std::max(D.maxWidth, width);
            DiluLevel lv;
            lv.s0 = int(D.levRows.size());
            lv.width = width;
            lv.mlo = lv.mup = 0;
            for (int r : v) {
                lv.mlo = std::max(lv.mlo, int(lo[r].size()));
                lv.mup = std::max(lv.mup, int(up[r].size()));
                D.slotRow.push_back(r - ds.rowBegin);
            }
            D.maxEnt = std::max({D.maxEnt, lv.mlo, lv.mup});
            lv.lo = int(D.sLoCol.size());
            for (int j = 0; j < lv.mlo; ++j)
                for (int r : v) {
                    const bool has = j < int(lo[r].size());
                    D.sLoCol.push_back(has ? lo[r][j][1] - ds.rowBegin : -1);
                    D.sLoFace.push_back(has ? lo[r][j][2] : 0);
                }
            lv.up = int(D.sUpCol.size());
            for (int j = 0; j < lv.mup; ++j)
                for (int r : v) {
                    const int nu = int(up[r].size());
                    const bool has = j < nu;  // backward order: descending (u, f)
                    D.sUpCol.push_back(has ? up[r][nu - 1 - j][1] - ds.rowBegin : -1);
                    D.sUpFace.push_back(has ? up[r][nu - 1 - j][2] : 0);
                }
            D.lev.push_back(lv);
            D.levRows.insert(D.levRows.end(), v.begin(), v.end());
            D.levPtr.push_back(int32_t(D.levRows.size()));
        }
        ds.slotEnd = int(D.levRows.size());
        ds.loEnd = int(D.sLoCol.size());
        ds.upEnd = int(D.sUpCol.size());
        D.maxLevels = std::max(D.maxLevels, nLev);
        D.sys.push_back(ds);
    }
    D.loPtr.assign(size_t(nrows) + 1, 0);
    D.upPtr.assign(size_t(nrows) + 1, 0);
    for (int r = 0; r < nrows; ++r) {
        D.loPtr[r + 1] = D.loPtr[r] + int32_t(lo[r].size());
        D.upPtr[r + 1] = D.upPtr[r] + int32_t(up[r].size());
        for (const auto& e : lo[r]) {
            D.loCol.push_back(e[1]);
            D.loFace.push_back(e[2]);
        }
        for (auto it = up[r].rbegin(); it != up[r].rend(); ++it) {
            D.upCol.push_back((*it)[1]);
            D.upFace.push_back((*it)[2]);
        }
    }
    return D;
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
        for (int j = 0; j < m; ++j)
            for (int q = 0; q < st.width; ++q) {
                const int r = R.slotRow[st.s0 + q];
                const int k = ptr[r] + j;
                if (k >= ptr[r + 1]) {
                    outCol.push_back(-1);
                    outFace.push_back(0);
                    continue;
                }
                const int c = col[k];
                if (partOf[c] == partOf[r]) {
                    outCol.push_back(slotOf[c] - part.slot0);
                } else {
                    outCol.push_back(-2 - (int(remote.size()) - r0));
                    remote.push_back(mail[slotOf[c]]);
                }
                outFace.push_back(face[k]);
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
