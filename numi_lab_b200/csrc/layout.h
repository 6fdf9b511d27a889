// Per-warp shared-memory carve-out of the microstep kernel.  Every section
// is sized from the compiled model, so a 7-DoF chain and a 29-DoF tree get
// exactly the scratch they need; sections start on 16-byte boundaries.
#pragma once

#include "device_model.h"

namespace numi {

// Words of one solver contact record in shared memory.
// Most environments (warps) one CTA of the FP32 temporalCone control-step
// kernel may carry; the other instances carry at most 4.
constexpr int kMaxStepWarpsPerBlock = 16;
// The solver's block and impulse change reuse the words of the geometry,
// which is dead once the Jacobian rows exist.
constexpr int kContactWords = 31;  // odd stride keeps lane-per-contact access conflict free
enum ContactWord : int {
    kCwPoint = 0,      // world contact point (3)
    kCwSeparation = 3,
    kCwNormal = 4,     // n, t, b directions (3 x 3)
    kCwTangent = 7,
    kCwBitangent = 10,
    kCwTarget = 13,    // evaluated target velocity per row (3)
    kCwReg = 16,       // regularisation per row (3)
    kCwMuU = 19,
    kCwMuV = 20,
    kCwLambda = 21,    // accumulated impulse (3)
    kCwPre = 0,        // 3x3 preconditioner, row-major (9)
    kCwRelax = 24,     // relaxation; the restitution until the row is evaluated
    kCwDelta = 9,      // last impulse change (3)
    kCwBody = 25,      // articulated body (int bits)
    kCwFlags = 26,     // bit0 new impact, bit8 articulated side is B (int bits)
    kCwSlot = 27,      // pair * 4 + manifold point (int bits)
    kCwUfree = 28      // contact-frame relative velocity at v_free (3); the
                       // restitution threshold until the row is evaluated
};

// Shared-memory strides (odd, so lane-per-body / per-DoF / per-pair access
// hits distinct banks).
constexpr int kPoseStride = 7;                    // COM position (3), orientation xyzw (4)
constexpr int kJStride = 7;                       // joint axis (3), origin (3), translation flag
constexpr int kSlotStride = kManifoldWords + 1;   // manifold slot

struct WarpLayout {
    int body_pose, dof_J;
    int q, v, vf, tgt;
    int tau, z, pair_stats;  // one section: drive efforts until the ABA has used them, then the narrowphase's, then the solver's
    int qdd, margins;        // one section: joint accelerations, then the narrowphase's margins
    int misc;
    int manifolds, contacts, G, L;
    int narrow;  // narrowphase scratch; aliases the contact records and rows
    int qcomp;   // compensation terms of q's running sums (compensated precision only)
    int quality; // FP64 workspace of the quality solver (quality.cuh; quality-solver instances only)
    int total;   // floats per warp
};

__host__ __device__ inline int align4(int x) { return (x + 3) & ~3; }

// Narrowphase scratch of one pair: four kept old points and up to
// `max_raw` raw contacts, 16 words each, plus 16 candidate-id bytes.
constexpr int kCandidateWords = 16;
__host__ __device__ inline int pair_scratch_words(int max_raw) { return (4 + max_raw) * kCandidateWords + 4; }

// Most raw contacts one pair class can produce before manifold reduction.
__host__ __device__ inline int pair_max_raw(int pair_class) {
    return pair_class == MR_COLLISION_PAIR_BOX_PLANE ? 8 : (pair_class == MR_COLLISION_PAIR_CAPSULE_PLANE ? 2 : 1);
}

// `narrow_words` is the sum of pair_scratch_words over the compiled pairs,
// `factor_words` DeviceTables::factor_words.
// `compensated` appends the q compensation section and `quality_doubles`
// (quality_workspace_doubles, or 0) the quality solver's FP64 workspace;
// the other sections keep their offsets.
__host__ __device__ inline WarpLayout make_layout(int nb, int nv, int nq, int np, int ncap, int max_anc, int narrow_words,
                                                  int factor_words, bool contact, bool compensated = false, int quality_doubles = 0) {
    WarpLayout L{};
    int o = 0;
    auto take = [&o](int words) { const int at = o; o += align4(words); return at; };
    L.body_pose = take(nb * kPoseStride);
    L.dof_J = take(nv * kJStride);
    const int shared = contact && nv < 32 ? 32 : nv;
    L.q = take(nq);
    L.v = take(nv);
    L.vf = take(nv);
    L.tau = L.z = L.pair_stats = take(shared);
    L.qdd = L.margins = take(shared);
    L.tgt = take(nv);
    L.misc = take(32);
    if (contact) {
        L.manifolds = take(np * kSlotStride);
        // Factor rows; past the root block (24 words) they later hold the
        // per-DoF contact lists (nv x ncap u16).
        const int lists = 24 + (nv * ncap + 1) / 2;
        L.L = take(factor_words > lists ? factor_words : lists);
        // Contact records and Jacobian rows are written only after the
        // narrowphase has finished with its scratch, so the three share words.
        L.contacts = take(ncap * kContactWords);
        const int rows = align4(ncap * 3 * (max_anc | 1));
        const int need = align4(narrow_words) - align4(ncap * kContactWords);
        L.G = take(rows > need ? rows : need);
        L.narrow = L.contacts;
    } else {
        L.manifolds = L.contacts = L.G = L.L = L.narrow = o;
    }
    L.qcomp = compensated ? take(nq) : o;
    L.quality = quality_doubles > 0 ? take(2 * quality_doubles) : o;
    L.total = align4(o);
    return L;
}

// misc words
enum MiscWord : int {
    kMiscP0 = 0,         // reference point (3)
    kMiscStatus = 4,     // step status code (int bits)
    kMiscFailIndex = 5,
    kMiscContactCount = 6,
    kMiscManifoldCount = 7,
    kMiscRawCount = 8,
    kMiscCandidatePairs = 9,
    kMiscIslands = 10,
    // Quality solver, over the control step's substeps: most Newton steps,
    // total line-search evaluations (int bits), largest scaled optimality,
    // cone violation and conic complementarity.
    kMiscQualityNewton = 16,
    kMiscQualityLineSearch = 17,
    kMiscQualityResidual = 18,
    kMiscQualityCone = 19,
    kMiscQualityComplementarity = 20
};

}  // namespace numi
