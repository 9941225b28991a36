// adjoint.cuh — reverse mode of one substep (adjoint.cu).
#pragma once
#include "common.cuh"

namespace seevr {

// Gradient buffers (device, FP64), indexed like the body / geom arrays.
struct Grads {
    double* pos;       // [N*3]  in: dL/d pos after the substep, out: before
    double* quat;      // [N*4]
    double* vel;       // [N*3]
    double* omega;     // [N*3]
    double* friction;  // [G]    accumulated: dL/d geom_friction
};

// Adjoint work arrays (device).
struct AdjScratch {
    float* tape;     // [max_contacts * iterations * 13] inputs of every contact update,
                     // per bundle [iteration][13][contact]
    uint4* ptape;    // [max_pairs * 2] supporting hull vertices per pair
    uint4* ctape;    // [max_contacts * 2] ... per contact
    uint4* side;     // [max_contacts] both sides' bundle-local body, rank and flags
    uint2* degree;   // [max_contacts] contacts at each side's body
    float* lam;      // [max_contacts] λ during the recomputed sweep
    // bundles above the shared-memory size
    float4* body4;   // [N*2] velocities during the recomputed sweep
    uint32_t* last;  // [N] update counts
    double* gvw;     // [N*6] running dL/d(v, ω)
    // reverse-pass accumulators, FP64
    double* gR;      // [N*9] dL/dR (rotation matrix, by columns)
    double* gp;      // [N*3] dL/d position
    double* gq;      // [N*4] dL/d quaternion
    double* gc;      // [max_contacts*12] dL/d (n, ra, rb, bias, kn, mu) per contact
    double* glam;    // [max_contacts] dL/dλ
    // contributions to the bodies' gradients, per contact and side:
    // v3 w3 p3 R9 friction1 (stride 20)
    double* fix;     // [max_contacts*40]
};

cudaError_t init_adjoint();
// max_bundle: bodies of the largest bundle
int launch_adjoint(const World& w, const Consts& k, const Scratch& s, const AdjScratch& a,
                   const Grads& g, float dt, uint32_t max_bundle, cudaStream_t st);

}  // namespace seevr
