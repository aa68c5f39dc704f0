// Level schedule of the DIC/DILU preconditioner (LinearSolver.cpp:28-112) on the device.
//
// The reference factorises and applies DILU in natural cell order over the faces sorted by
// (upper cell, lower cell): rD[u] -= A_lu A_ul / rD[l], then a forward sweep
// w[u] -= rD[u] A_ul w[l] and a backward sweep w[l] -= rD[l] A_lu w[u].  Each is a recurrence
// along the natural-order dependency graph (l -> u for every face), so rows can be updated in
// parallel exactly when they sit on the same level of that graph: level[u] = 1 + max level[l]
// over its lower neighbours.  Inside a row the terms are applied in the reference's order
// (forward: lower neighbours by ascending (l, face); backward: upper neighbours by descending
// (u, face)), so the device result is the reference's, bit for bit.
#pragma once

#include <cstdint>
#include <vector>

#include "plan.h"

namespace vlm {

// One system's part of the schedule (batch position `sys`): levels [levBegin, levBegin + nLev) of
// the concatenated level table.
struct DiluSys {
    int sys, levBegin, nLev, rowBegin, rowCount;  // rows [rowBegin, rowBegin + rowCount) of level 0
    // streamed schedule (addDiluStream): its slots levRows[slotBegin .. slotEnd), its entries
    int slotBegin, slotEnd;
    int loBegin, loEnd, upBegin, upEnd;
};

// One level of the streamed schedule: slots [s0, s0 + width) of levRows; entry j of slot s0 + q at
// lo + j * width + q (j < mlo, lower neighbours in forward order) and up + j * width + q (j < mup,
// upper neighbours in backward order).  A row with fewer entries pads its column with -1.  A level's
// rows, scalars and entries are contiguous, so a CTA can stream them into shared memory levels ahead
// of the sweep without looking anything up.
struct DiluLevel {
    int s0, width, lo, mlo, up, mup;
};

struct DiluPlan {
    // per level-0 row (solver order): lower neighbours (forward order) and upper neighbours
    // (backward order); face = user face index | ownerIsL << 31
    std::vector<int32_t> loPtr, loCol, loFace;
    std::vector<int32_t> upPtr, upCol, upFace;
    // level schedule: levPtr[levBegin + t] .. levPtr[levBegin + t + 1] index levRows (solver rows);
    // padding rows are on level 0 of their system
    std::vector<int32_t> levPtr, levRows;
    std::vector<DiluSys> sys;
    // streamed schedule (addDiluStream; per level of levPtr): slot -> row - rowBegin, entries (local column or -1,
    // face as loFace)
    std::vector<DiluLevel> lev;
    std::vector<int32_t> slotRow;
    std::vector<int32_t> sLoCol, sLoFace, sUpCol, sUpFace;
    int maxEnt = 0;    // largest mlo / mup of any level
    int maxWidth = 0;  // widest level over all systems
    int maxLevels = 0;
    int maxRows = 0;   // largest system (level-0 rows incl. padding)
};

// Rows of a system's widest level, its padding rows (which sit on level 0 and are in no step) left out.
int diluWidth(const DiluPlan& D, const DiluSys& ds, const BatchPlan& P);

// systems: input order; P: the batch plan (solver order, perm0).
DiluPlan buildDiluPlan(const std::vector<SysTopo>& systems, const BatchPlan& P);

// Fills in the streamed schedule (systems whose sweeps run on one CTA each).
void addDiluStream(DiluPlan& D);

// Pipelined schedule of systems too wide for one CTA: the rows of a system are cut into parts of
// consecutive natural rows, one CTA each.  A lower neighbour precedes its row in natural order, so a
// part's forward sweep reads only its own rows and rows of earlier parts (its backward sweep, of
// later parts): each part walks its own rows level by level and takes the values of other parts from
// per-value mailboxes, so no two CTAs ever meet at a barrier.  Slots: every real row of a part, step by
// step; a step is at most maxWidth rows of one level.  A system's padding rows are dealt to its parts too:
// the backward sweep leaves 0 there, which the reductions over all rows rely on.
struct DiluPart {
    int sys, stepBegin, nSteps, slot0, nSlots;
    int pad0, nPad;  // its padding rows in padRow
};

// Slots [s0, s0 + width); entry j of slot s0 + q at lo + j * width + q (up likewise): a slot of the part
// relative to its slot0, -1 padding, or -2 - k: the step's remote entry k (mailbox loRemote[rlo + k]).
struct DiluStep {
    int s0, width, lo, mlo, up, mup, rlo, nrlo, rup, nrup;
};

struct DiluParts {
    std::vector<DiluPart> parts;  // forward order; the backward sweep takes them in reverse
    std::vector<DiluStep> steps;
    std::vector<int32_t> slotRow;                        // slot -> solver row
    std::vector<int32_t> padRow;                         // padding rows, part by part
    std::vector<int32_t> loCol, loFace, upCol, upFace;   // entries (faces as DiluPlan's)
    std::vector<int32_t> loRemote, upRemote;             // mailbox of each remote entry
    std::vector<int32_t> loMail, upMail;                 // per slot: the mailbox its value goes to, -1: none
    int nLoMail = 0, nUpMail = 0;
    int maxSlots = 0, maxWidth = 0, maxRemote = 0;
};

// The parts' entries as 16-byte records for rows of at most six lower and six upper neighbours (box
// meshes): record [slot] holds the first three columns and, in its fourth word, 1 + mailbox << 9 | 1 + the
// extension's place in the step (0: none); the extensions of a step's rows with more entries follow at
// extLo / extUp of the step.  Columns index the part's vector in shared memory: its slots, then two
// buffers of maxRemote remote values (step parity); -1: no entry.  faces: as DiluPlan's, kNoFace: none.
struct DiluRecStep {
    int s0, width, rlo, nrlo, rup, nrup, extLo, nExtLo, extUp, nExtUp;
};

struct DiluRecords {
    static constexpr int32_t kNoFace = 0x7fffffff;
    std::vector<DiluRecStep> steps;
    std::vector<int32_t> loCol, upCol, loFace, upFace;  // four words per record
    int nLo = 0, nUp = 0;                               // records (slots, then extensions)
    int maxExt = 0, maxSteps = 0;
};

// False when a row has more than six entries in a direction or a word overflows.
bool buildDiluRecords(const DiluParts& R, DiluRecords& out);

// nParts[b]: parts of the system at batch position b (at least 1).
DiluParts buildDiluParts(const DiluPlan& D, const BatchPlan& P, const std::vector<int>& nParts, int maxWidth);

}  // namespace vlm
