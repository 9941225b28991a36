// solver.cu — PGS contact solver (step 5, physics.comp:500-583) and the
// impulse clear (step 4, physics.comp:494-497).
//
// Work is split into bundles: runs of whole consecutive scenes.  Scenes share
// no body, so a bundle is solved exactly like one scene whose contacts are
// the union of its scenes' (each scene's contacts keep their order, and the
// wavefront levels of different scenes simply merge); small scenes are
// bundled so that a warp's lanes have work.
//
// Per contact, the values the reference recomputes on every iteration but
// which cannot change during the solve are computed once: the lever arms ra, rb
// (positions and contact points are constant), the normal effective mass k, the
// friction coefficient and the restitution/Baumgarte bias (taken from the
// pre-solve velocities, as physics.comp:504-521 does).  Then the sweeps:
//  - SEQUENTIAL: one thread, contacts in index order (physics.comp:523-582);
//  - WAVEFRONT: an update runs as soon as the earlier updates that share one of
//    its dynamic bodies are done.  Each contact then sees exactly the body state
//    it sees in the sequential sweep, so the result is bit-identical;
//  - COLORED: the same with the contacts in the order of their greedy colours.
// Bundles of up to kWarpMaxBodies bodies: k_solver_flow.  Larger scenes are solved
// by islands (islands.cu), or without its work arrays by k_solver, one block over
// levels of contacts.
// A body is "fixed" when inv_mass == 0 and inv_inertia == 0: its velocities
// cannot change (the reference writes v - 0*impulse, the same value), so
// fixed bodies create no ordering constraint and are never written.
#include <algorithm>

#include "common.cuh"
#include "solver.cuh"

namespace seevr {

constexpr uint32_t kSolverThreads = 128;
constexpr uint32_t kBodySmemWords = 20;  // v3 w3 R9 invI3 invm1 last1

__global__ void __launch_bounds__(kSolverThreads)
    k_solver(World w, Consts k, Scratch s, uint32_t mode, float dt, uint32_t smem_bodies) {
    extern __shared__ float sm[];
    __shared__ uint32_t sh_levels;
    if (halted(w.status)) return;  // contacts from a scan that gave up
    const uint32_t scene = blockIdx.x;  // bundle index
    const uint32_t b0 = w.bundle_off[scene], b1 = w.bundle_off[scene + 1];
    const uint32_t nbs = b1 - b0;
    const uint32_t c0 = first_contact(w, s, b0), c1 = first_contact(w, s, b1);
    if (c0 >= c1) return;
    const uint32_t tid = threadIdx.x;

    // ---- phase 1: bodies ----
    const bool in_smem = nbs <= smem_bodies;
    BodyView B;
    uint32_t* last;
    if (in_smem) {
        float* p = sm;
        B.v = p; p += nbs * 3;
        B.w = p; p += nbs * 3;
        float* R = p; p += nbs * 9;
        float* invI = p; p += nbs * 3;
        float* invm = p; p += nbs;
        last = reinterpret_cast<uint32_t*>(p);
        for (uint32_t i = tid; i < nbs; i += blockDim.x) {
            const uint32_t g = b0 + i;
            st3(B.v, i, ld3(w.vel, g));
            st3(B.w, i, ld3(w.omega, g));
            st_m3(R, i, quat_to_mat(w.quat, g));
            st3(invI, i, ld3(w.inv_inertia, g));
            invm[i] = w.inv_mass[g];
            last[i] = 0;
        }
        B.R = R;
        B.invI = invI;
        B.invm = invm;
    } else {
        B.v = w.vel + size_t(b0) * 3;
        B.w = w.omega + size_t(b0) * 3;
        float* R = s.s_R + size_t(b0) * 9;
        for (uint32_t i = tid; i < nbs; i += blockDim.x) {
            st_m3(R, i, quat_to_mat(w.quat, b0 + i));
            s.s_last[b0 + i] = 0;
        }
        B.R = R;
        B.invI = w.inv_inertia + size_t(b0) * 3;
        B.invm = w.inv_mass + b0;
        last = s.s_last + b0;
        if (tid == 0) atomicOr(&s.status[0], kFlagSolverGlobal);
    }
    __syncthreads();

    // ---- phase 2: per-contact constants (physics.comp:504-521, 533-546) ----
    for (uint32_t c = c0 + tid; c < c1; c += blockDim.x) {
        const uint32_t ga = w.c_a[c], gb = w.c_b[c];
        const uint32_t a = w.geom_body[ga], b = w.geom_body[gb];
        const uint32_t la = a - b0, lb = b - b0;
        const f3 n = ld3(w.c_normal, c), cp = ld3(w.c_pos, c);
        const f3 ra = sub(cp, ld3(w.pos, a)), rb = sub(cp, ld3(w.pos, b));
        const f3 va = add(ld3(B.v, la), cross(ld3(B.w, la), ra));
        const f3 vb = add(ld3(B.v, lb), cross(ld3(B.w, lb), rb));
        const float vn = dot(sub(vb, va), n);
        const float e = gmax(w.restitution[ga], w.restitution[gb]);
        const float bias = k.baumgarte * gmax(w.c_pen[c] - k.slop, 0.0f) / dt + e * gmax(-vn, 0.0f);
        const float ima = B.invm[la], imb = B.invm[lb];
        const m3 Ra = ld_m3(B.R, la), Rb = ld_m3(B.R, lb);
        const f3 ran = cross(ra, n), rbn = cross(rb, n);
        const float kn = ima + imb + dot(ran, apply_inv_I(Ra, ld3(B.invI, la), ran)) +
                         dot(rbn, apply_inv_I(Rb, ld3(B.invI, lb), rbn));
        st3(s.s_ra, c, ra);
        st3(s.s_rb, c, rb);
        s.s_bias[c] = bias;
        s.s_kn[c] = kn;
        s.s_mu[c] = sqrtf(w.friction[ga] * w.friction[gb]);
        const bool skip = (ima == 0.0f && imb == 0.0f);  // physics.comp:531
        s.s_ab[size_t(c) * 2] = skip ? kNone : la;
        s.s_ab[size_t(c) * 2 + 1] = lb;
        w.lambda[c] = 0.0f;
    }
    __syncthreads();

    if (mode == 0) {
        // ---- SEQUENTIAL: the reference order on one thread ----
        if (tid == 0) {
            for (uint32_t it = 0; it < k.pgs_iterations; ++it)
                for (uint32_t c = c0; c < c1; ++c) {
                    const uint32_t la = s.s_ab[size_t(c) * 2];
                    if (la == kNone) continue;
                    solve_one(B, la, s.s_ab[size_t(c) * 2 + 1], ld3(w.c_normal, c), ld3(s.s_ra, c),
                              ld3(s.s_rb, c), s.s_bias[c], s.s_kn[c], s.s_mu[c], &w.lambda[c]);
                }
        }
    } else {
        // ---- WAVEFRONT: levels, counting sort by level, parallel sweeps ----
        uint32_t* lvl = s.s_lvl_start + c0 + scene;  // [levels+1], fits in [c0+scene, c1+scene]
        if (tid == 0) {
            uint32_t maxl = 0;
            for (uint32_t c = c0; c < c1; ++c) {
                const uint32_t la = s.s_ab[size_t(c) * 2];
                if (la == kNone) {
                    s.s_level[c] = kNone;
                    continue;
                }
                const uint32_t lb = s.s_ab[size_t(c) * 2 + 1];
                const bool fa = is_fixed(B, la), fb = is_fixed(B, lb);
                const uint32_t l = max(fa ? 0u : last[la], fb ? 0u : last[lb]) + 1u;
                if (!fa) last[la] = l;
                if (!fb) last[lb] = l;
                s.s_level[c] = l - 1u;
                maxl = max(maxl, l);
            }
            for (uint32_t l = 0; l <= maxl; ++l) lvl[l] = 0;
            for (uint32_t c = c0; c < c1; ++c)
                if (s.s_level[c] != kNone) lvl[s.s_level[c] + 1]++;
            for (uint32_t l = 1; l <= maxl; ++l) lvl[l] += lvl[l - 1];
            // stable fill: order[c0 + slot]; lvl[l] is used as a cursor and
            // restored afterwards
            for (uint32_t c = c0; c < c1; ++c) {
                const uint32_t l = s.s_level[c];
                if (l != kNone) s.s_order[c0 + lvl[l]++] = c;
            }
            for (uint32_t l = maxl; l > 0; --l) lvl[l] = lvl[l - 1];
            lvl[0] = 0;
            sh_levels = maxl;
        }
        __syncthreads();
        const uint32_t levels = sh_levels;
        for (uint32_t it = 0; it < k.pgs_iterations; ++it) {
            for (uint32_t l = 0; l < levels; ++l) {
                const uint32_t beg = lvl[l], end = lvl[l + 1];
                for (uint32_t i = beg + tid; i < end; i += blockDim.x) {
                    const uint32_t c = s.s_order[c0 + i];
                    solve_one(B, s.s_ab[size_t(c) * 2], s.s_ab[size_t(c) * 2 + 1],
                              ld3(w.c_normal, c), ld3(s.s_ra, c), ld3(s.s_rb, c), s.s_bias[c],
                              s.s_kn[c], s.s_mu[c], &w.lambda[c]);
                }
                __syncthreads();
            }
        }
    }
    __syncthreads();
    if (in_smem) {
        for (uint32_t i = tid; i < nbs; i += blockDim.x) {
            st3(w.vel, b0 + i, ld3(B.v, i));
            st3(w.omega, b0 + i, ld3(B.w, i));
        }
    }
}

// ---- block per bundle -------------------------------------------------------
// Bundles of up to kWarpMaxBodies bodies: one block of W warps each, in dataflow
// order.  In the sequential sweep the updates of one body's contacts follow each
// other in contact order, iteration after iteration, and nothing else orders two
// updates.  So every body counts the updates it has had, and the update of
// contact c in iteration k may run as soon as each of its two dynamic bodies has
// counted k d + r updates (d: the body's contacts, r: c's rank among them): it
// then reads exactly the state it reads in the sequential sweep, and results are
// bit for bit those of that sweep.  In every round the contacts that are ready
// run together, whatever their iterations.  A sweep takes about (largest d)
// rounds per iteration, where the levels of one iteration after another (7 to 11
// for a settled 512-body pile, in 32-wide passes) took 8 to 22.  Contacts that
// share no dynamic body with another (a third of a pile's) are taken apart: all
// their iterations at once, beside the rounds.
//
// A bundle's time is the dependent chain of its rounds, and a round is bound by one
// warp's latency and issue.  So a lane owns a contact for the whole solve, its
// constants in registers; velocities and counts live in shared memory, both in
// one 16-byte word per body; and the update's square root and divisions are
// the branch-free ones of vmath.cuh: a lane with an argument outside their
// ranges redoes the update with the built-in ones.
//
// A lane owns contacts i, i + 32 W, ... and takes them in order, iteration after
// iteration: the first unfinished update of the whole sequence is then at the
// head of its lane's list and ready, so every round makes progress.  (More than two
// contacts per lane in contact order go level by level instead: level_sweep.)

// a contact side's bundle-local body, flags and rank
// (Free: the body is not written and orders nothing; Skip: both masses infinite;
// Same, with Free, on side a: side b is the same dynamic body, whose velocities side a
// takes at every update and which b writes last)
constexpr uint32_t kSideBody = 0xFFFu, kSideFree = 1u << 12, kSideSkip = 1u << 13,
                   kSideSame = 1u << 14, kRankShift = 16, kMaxRank = 0xFFFFu;
static_assert(kWarpMaxBodies <= kSideBody, "body field too narrow");

// Shared memory of a block: per body its velocity with the count of its updates
// and its angular velocity (a float4 each); then, where they fit, the contacts'
// sides and positions (12 bytes each) and their records.
struct FlowBodies {
    float4* v;  // velocity, updates counted (bits of an integer)
    float4* w;  // angular velocity, latest level (zero but while contacts are ordered)
    __device__ __forceinline__ uint32_t* count(uint32_t l) const {
        return reinterpret_cast<uint32_t*>(&v[l].w);
    }
    __device__ __forceinline__ uint32_t* last(uint32_t l) const {
        return reinterpret_cast<uint32_t*>(&w[l].w);
    }
};

__device__ __forceinline__ float4 ld4(const float4* p) {  // shared memory
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(uint32_t(__cvta_generic_to_shared(p)))
                 : "memory");
    return v;
}
__device__ __forceinline__ void st4(float4* p, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(
                     uint32_t(__cvta_generic_to_shared(p))),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

// Barrier of the block's first `threads` threads.
template <uint32_t W>
__device__ __forceinline__ void part_sync(uint32_t threads) {
    if (W == 1 || threads == 32)
        __syncwarp();
    else
        __barrier_sync_count(1, threads);
}

// Ranks of the contact sides in info[0 .. 2 nc), contact order, by one warp:
// 16 contacts at a time.  The bodies' counts (zero before) end as their
// contacts.  False when a rank does not fit its field.
__device__ __forceinline__ bool rank_sides(uint32_t* info, const FlowBodies& B, uint32_t nc) {
    const uint32_t lane = threadIdx.x & 31u;
    bool fits = true;
    for (uint32_t e0 = 0; e0 < 2 * nc; e0 += 32) {
        const uint32_t e = e0 + lane;
        const uint32_t x = e < 2 * nc ? info[e] : kSideFree;
        const bool counts = !(x & kSideFree);
        const uint32_t body = x & kSideBody;
        const unsigned m = __match_any_sync(0xFFFFFFFFu, counts ? body : 0x80000000u | lane);
        if (counts) {
            const uint32_t r = *B.count(body) + __popc(m & ((1u << lane) - 1u));
            fits &= r < kMaxRank;
            info[e] = (x & 0xFFFFu) | (r << kRankShift);
        }
        __syncwarp();
        if (counts && lane == uint32_t(__ffs(m)) - 1u) *B.count(body) += __popc(m);
        __syncwarp();
    }
    return __all_sync(0xFFFFFFFFu, fits);
}

// COLORED order: greedy colours in contact order (the smallest colour not used
// by an earlier contact at either dynamic body; masks in the bodies' counts),
// contacts sorted by colour in order[0 .. nc), ranks by colour.  False when a
// body needs more than 32 colours.  One warp; level: scratch.
__device__ __forceinline__ bool colour_sides(uint32_t* info, const FlowBodies& B, uint32_t nc,
                                             uint32_t* level, uint32_t* order) {
    const unsigned full = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t ok = 1u, mx = 0u;
    if (lane == 0) {
        const uint2* sides = reinterpret_cast<const uint2*>(info);
        uint2 next = sides[0];
        for (uint32_t i = 0; i < nc && ok; ++i) {
            const uint32_t a = next.x, b = next.y;
            if (i + 1 < nc) next = sides[i + 1];
            if (a & kSideSkip) {
                level[i] = 0u;  // solved by nobody: any colour
                continue;
            }
            const uint32_t used = (a & kSideFree ? 0u : *B.count(a & kSideBody)) |
                                  (b & kSideFree ? 0u : *B.count(b & kSideBody));
            ok = used != 0xFFFFFFFFu;
            const uint32_t col = uint32_t(__ffs(int(~used))) - 1u;
            if (ok && !(a & kSideFree)) *B.count(a & kSideBody) |= 1u << col;
            if (ok && !(b & kSideFree)) *B.count(b & kSideBody) |= 1u << col;
            level[i] = col;
            mx = max(mx, col + 1u);
        }
    }
    ok = __shfl_sync(full, ok, 0);
    mx = __shfl_sync(full, mx, 0);
    __syncwarp();
    if (!ok) return false;
    for (uint32_t e = lane; e < 2 * nc; e += 32) {
        const uint32_t x = info[e];
        if (!(x & kSideFree))
            info[e] = (x & 0xFFFFu) |
                      (__popc(*B.count(x & kSideBody) & ((1u << level[e >> 1]) - 1u)) << kRankShift);
    }
    uint32_t pos = 0;
    for (uint32_t l = 0; l < max(mx, 1u); ++l)
        for (uint32_t i0 = 0; i0 < nc; i0 += 32) {
            const uint32_t i = i0 + lane;
            const bool hit = i < nc && level[i] == l;
            const unsigned m = __ballot_sync(full, hit);
            if (hit) order[pos + __popc(m & ((1u << lane) - 1u))] = i;
            pos += __popc(m);
        }
    __syncwarp();
    return true;
}

// Contacts per lane above which blocks of several warps sweep contact order level by
// level (level_sweep).  Lanes that own several take them in turn, and where contacts
// that follow each other wait for each other (boxes heaped row by row, columns) few
// lanes find theirs ready.  Solver time per substep in rounds / by levels (the former
// passes by level, 32 wide): 1,024 scenes of 8 to 500 boxes heaped, 1.4 contacts per body,
// 2,850 / 1,475 us (1,559); 300 heaps of 120 boxes 1,006 / 549 (874); 64 scenes of 10
// columns of 48 1,983 / 1,093 (1,406).  Up to two contacts per lane, rounds are the
// better where chains' iterations follow each other closely: two columns of 125 boxes
// 280 / 2,426 us, 13 of 10 121 / 249; at worst 20 of 10 314 / 239.  One warp takes as
// long for a level as for a round (heaps of 90 boxes 391 us in rounds, 507 by levels).
constexpr uint32_t kSweepFrom = 2;

// The larger of the numbers of contacts at contact i's dynamic bodies (after ranking).
__device__ __forceinline__ uint32_t degree_of(const uint32_t* info, const FlowBodies& B, uint32_t i) {
    const uint32_t a = info[2 * i], b = info[2 * i + 1];
    return max(a & kSideFree ? 0u : *B.count(a & kSideBody), b & kSideFree ? 0u : *B.count(b & kSideBody));
}
// Contacts that share a dynamic body with another one.  One warp.
__device__ __forceinline__ uint32_t count_chained(const uint32_t* info, const FlowBodies& B, uint32_t nc) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t chained = 0;
    for (uint32_t i0 = 0; i0 < nc; i0 += 32)
        chained += __popc(__ballot_sync(0xFFFFFFFFu, i0 + lane < nc &&
                                                         degree_of(info, B, min(i0 + lane, nc - 1)) > 1u));
    return chained;
}

// Positions: first the chained contacts, then the lone ones.  With a lane for each (at
// most `lanes`), the former go by falling degree (the larger of the two bodies'), so
// that the longest chains share few warps; lanes that own several need the
// sequence's order, which `seq` gives (NULL: contact order).  One warp.
__device__ __forceinline__ void order_contacts(const uint32_t* info, const FlowBodies& B, uint32_t nc,
                                               uint32_t chained, uint32_t lanes, const uint32_t* seq,
                                               uint32_t* order) {
    const uint32_t lane = threadIdx.x & 31u;
    // classes: degrees 4 and above, 3, 2, lone ones; or all chained ones, lone ones
    const bool one_each = chained <= lanes;
    uint32_t pos = 0;
    for (uint32_t cls = 4; cls > 0; --cls) {
        if (!one_each && (cls == 3u || cls == 2u)) continue;
        for (uint32_t i0 = 0; i0 < nc; i0 += 32) {
            const bool valid = i0 + lane < nc;
            const uint32_t i = valid ? (!one_each && seq ? seq[i0 + lane] : i0 + lane) : 0u;
            const uint32_t d = degree_of(info, B, i);
            const bool hit = valid && (cls == 1u   ? d <= 1u
                                       : !one_each ? d > 1u
                                       : cls == 4u ? d >= 4u
                                                   : d == cls);
            const unsigned m = __ballot_sync(0xFFFFFFFFu, hit);
            if (hit) order[pos + __popc(m & ((1u << lane) - 1u))] = i;
            pos += __popc(m);
        }
    }
}

// The chained contacts by levels (a contact's is the first after those of the earlier
// contacts at its dynamic bodies), then the lone ones, and the levels cut into chunks of
// up to 32.  The whole block; placed: nc words of scratch; counts: two words, zero
// before, as the bodies' `last` words are, which count the contacts placed at each.
// (The first contact not yet placed can be: every round places some.)
struct Chunks {
    uint32_t *first, *level;  // of each
    uint32_t n, levels;
};
template <uint32_t W>
__device__ __noinline__ Chunks build_levels(const uint32_t* info, const FlowBodies B, uint32_t nc,
                                               uint32_t chained, uint32_t* placed, uint32_t* order,
                                               Chunks chunks, uint32_t* counts) {
    // (A call of its own, and the sweep's two kinds of records apart: in one piece with
    // them the rounds' registers were allotted otherwise, 2% of a frame of 100 scenes.)
    __builtin_assume(__isShared(counts));
    __builtin_assume(__isShared(B.v));
    __builtin_assume(__isShared(B.w));
    __builtin_assume(__isGlobal(placed));
    __builtin_assume(__isGlobal(chunks.first));
    __builtin_assume(__isGlobal(chunks.level));
    const uint32_t t = threadIdx.x;
    for (uint32_t i = t; i < nc; i += 32 * W) {
        const bool lone = degree_of(info, B, i) <= 1u;
        if (lone) order[chained + atomicAdd(&counts[1], 1u)] = i;
        placed[i] = lone ? 1u : 0u;
    }
    uint32_t from = 0, l = 0;
    chunks.n = 0;
    for (; from < chained; ++l) {
        for (uint32_t i = t; i < nc; i += 32 * W) {
            if (placed[i]) continue;
            const uint32_t xa = info[2 * i], xb = info[2 * i + 1];
            if (!(xa & kSideFree) && *B.last(xa & kSideBody) != xa >> kRankShift) continue;
            if (!(xb & kSideFree) && *B.last(xb & kSideBody) != xb >> kRankShift) continue;
            order[atomicAdd(&counts[0], 1u)] = i;
            placed[i] = 2u + l;
        }
        __syncthreads();
        const uint32_t to = counts[0], n = (to - from + 31) / 32;
        for (uint32_t j = t; j < n; j += 32 * W) {
            chunks.first[chunks.n + j] = from + 32 * j;
            chunks.level[chunks.n + j] = l;
        }
        for (uint32_t i = t; i < nc; i += 32 * W) {  // no two of a level share a dynamic body
            if (placed[i] != 2u + l) continue;
            const uint32_t xa = info[2 * i], xb = info[2 * i + 1];
            if (!(xa & kSideFree)) ++*B.last(xa & kSideBody);
            if (!(xb & kSideFree)) ++*B.last(xb & kSideBody);
        }
        __syncthreads();
        from = to;
        chunks.n += n;
    }
    chunks.levels = l;
    return chunks;
}

// The records of a run.  In shared memory word k of all contacts lies together, even
// contacts apart from odd ones: lanes take neighbouring contacts (contact order) or
// every other one (a chain's colours), and read 16-byte words without bank conflicts
// either way; whole records of 160 bytes cost four-way ones, which bound runs with
// several contacts per lane.  Those that do not fit lie whole in s_rec, five sectors
// each, and `stage`, where there is room for it, holds `slots` of them at a time for the
// level sweep.
struct Recs {
    float4 *p, *stage;
    uint32_t half, stride, step, slots;
    bool fits;
    static constexpr uint32_t kPad = 7;  // contacts' worth of padding at most
    // room: float4s of shared memory; most: threads
    __device__ __forceinline__ Recs(float4* shared, uint32_t room, float4* global, uint32_t nc, uint32_t most) {
        fits = (nc + kPad) * kRecWords <= room;
        p = fits ? shared : global;
        half = (nc + 1) / 2;
        half = fits ? half + (12u - half % 8u) % 8u : kRecWords;  // 4 modulo 8
        stride = fits ? half + nc / 2 : 1u;
        step = fits ? 1u : 2 * kRecWords;
        slots = fits ? 0u : min(room / kRecWords & ~31u, most);
        stage = shared;
    }
    __device__ __forceinline__ float4* at(uint32_t i) const {
        return p + size_t(i >> 1) * step + (i & 1u) * half;
    }
};
__device__ __forceinline__ void copy_async(float4* to, const float4* from) {  // global to shared
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(uint32_t(__cvta_generic_to_shared(to))),
                 "l"(__cvta_generic_to_global(from))
                 : "memory");
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

struct FlowArgs {
    uint32_t nc, slot, width, threads, iters;  // nc: chained contacts
    const uint32_t* order;  // contact of each position
    const uint32_t* info;
    Recs rec;
    float* lam;         // impulses by contact
    uint32_t* deg;      // degrees of both bodies by contact (scratch)
    uint32_t* left;     // lanes that are not done
};

// The rounds of one bundle's chained contacts.  kSeveral: lanes own more than one.
template <uint32_t W, bool kSeveral>
__device__ __forceinline__ void flow_sweep(const FlowArgs& f, const FlowBodies& B) {
    const unsigned full = 0xFFFFFFFFu;
    uint32_t i = f.slot, it = 0, c = f.order[min(i, f.nc - 1)];
    Rec h = load_rec(f.rec.at(c), f.rec.stride);
    uint32_t xa = f.info[2 * c], xb = f.info[2 * c + 1];
    uint32_t da = 0, db = 0, ka = 0, kb = 0;  // degrees, counts to wait for
    State x{};
    bool live = i < f.nc && f.iters > 0 && !(xa & kSideSkip);
    auto degree = [&](uint32_t y) { return y & kSideFree ? 0u : *B.count(y & kSideBody); };
    // counts start at the body's contacts (the ranking's result)
    auto arm = [&] {
        if (kSeveral) {
            const uint32_t d = f.deg[c];
            da = d & 0xFFFFu;
            db = d >> 16;
        }
        ka = da * (it + 1) + (xa >> kRankShift);
        kb = db * (it + 1) + (xb >> kRankShift);
        // (the others are read in every round, and so is a body that is both sides)
        if ((!kSeveral || (xa & kSideFree)) && !(xa & kSideSame)) {
            const float4 v = ld4(B.v + (xa & kSideBody)), o = ld4(B.w + (xa & kSideBody));
            x.va = mk(v.x, v.y, v.z);
            x.wa = mk(o.x, o.y, o.z);
        }
        if (!kSeveral || (xb & kSideFree)) {
            const float4 v = ld4(B.v + (xb & kSideBody)), o = ld4(B.w + (xb & kSideBody));
            x.vb = mk(v.x, v.y, v.z);
            x.wb = mk(o.x, o.y, o.z);
        }
    };
    if (kSeveral) {
        // the degrees of the lane's contacts, before the counts move on
        for (uint32_t j = i; j < f.nc; j += f.width) {
            const uint32_t e = f.order[j];
            f.deg[e] = degree(f.info[2 * e]) | degree(f.info[2 * e + 1]) << 16;
        }
    } else {
        da = degree(xa);
        db = degree(xb);
    }
    if (live) {
        arm();
        atomicAdd(f.left, 1u);
    }
    part_sync<W>(f.threads);
    // the first unfinished update of the sequence is ready in every round, so
    // iters * nc rounds are enough
    for (uint64_t round = 0, cap = uint64_t(f.iters) * f.nc; round <= cap; ++round) {
        // a body that no other contact moves keeps its velocities in registers
        bool ready = live;
        const uint32_t la = xa & kSideBody, lb = xb & kSideBody;
        if (live && (kSeveral || da > 1u) && !(xa & kSideFree)) {
            const float4 v = ld4(B.v + la), o = ld4(B.w + la);
            ready = __float_as_uint(v.w) == ka;
            x.va = mk(v.x, v.y, v.z);
            x.wa = mk(o.x, o.y, o.z);
        }
        if (live && (kSeveral || db > 1u) && !(xb & kSideFree)) {
            const float4 v = ld4(B.v + lb), o = ld4(B.w + lb);
            ready = ready && __float_as_uint(v.w) == kb;
            x.vb = mk(v.x, v.y, v.z);
            x.wb = mk(o.x, o.y, o.z);
        }
        if (xa & kSideSame) {
            x.va = x.vb;
            x.wa = x.wb;
        }
        const uint32_t left = *f.left;
        part_sync<W>(f.threads);  // every read of the round before its writes
        if (left == 0u) break;
        if (__any_sync(full, ready)) {
            const State y = update(h, ready, x);
            if (ready) {
                x.lam = y.lam;
                if (!(xa & kSideFree)) {
                    x.va = y.va;
                    x.wa = y.wa;
                    st4(B.w + la, make_float4(y.wa.x, y.wa.y, y.wa.z, 0.0f));
                    st4(B.v + la, make_float4(y.va.x, y.va.y, y.va.z, __uint_as_float(ka + 1u)));
                }
                if (!(xb & kSideFree)) {
                    x.vb = y.vb;
                    x.wb = y.wb;
                    st4(B.w + lb, make_float4(y.wb.x, y.wb.y, y.wb.z, 0.0f));
                    st4(B.v + lb, make_float4(y.vb.x, y.vb.y, y.vb.z, __uint_as_float(kb + 1u)));
                }
                if (kSeveral) {  // on to the lane's next contact
                    f.lam[c] = x.lam;
                    i += f.width;
                    if (i >= f.nc) {
                        i = f.slot;
                        live = ++it < f.iters;
                    }
                    if (live) {
                        c = f.order[i];
                        h = load_rec(f.rec.at(c), f.rec.stride);
                        xa = f.info[2 * c];
                        xb = f.info[2 * c + 1];
                        x.lam = f.lam[c];
                        arm();
                    }
                } else {
                    live = ++it < f.iters;
                    ka += da;
                    kb += db;
                }
            }
            const unsigned done = __ballot_sync(full, ready && !live);
            if (done && (threadIdx.x & 31u) == 0u) atomicSub(f.left, uint32_t(__popc(done)));
        }
        part_sync<W>(f.threads);
    }
    if (!kSeveral && i < f.nc) f.lam[c] = x.lam;
}

// The chained contacts, a level at a time (a turn): its contacts touch different dynamic
// bodies and run together.  A turn takes 1,100 to 1,400 cycles: the bodies' velocities,
// the update's chain, the barrier.  The warps take the iterations' chunks in rotation, so
// that a warp prepares its next chunk (table, contact, sides, record: 400 cycles) while
// others solve theirs, behind the barrier that ended its own; only where that chunk's
// turn is this one or the next it starts the record's copy before it solves.
template <uint32_t W>
__device__ __forceinline__ void level_sweep(const FlowArgs& f, const FlowBodies& B, const Chunks& chunks) {
    const uint32_t lane = threadIdx.x & 31u;
    const bool staged = threadIdx.x < f.rec.slots;
    auto record = [&](uint32_t c) {
        const float4* p = f.rec.at(c);
        if (f.rec.fits) {
            __builtin_assume(__isShared(p));
            return load_rec(p, f.rec.stride);
        }
        __builtin_assume(__isGlobal(p));
        return load_rec(p);
    };
    float4* const slot = f.rec.stage + threadIdx.x;
    // a chunk of this warp's: its turn (kNone: none), this lane's contact and its sides
    struct Part {
        uint32_t turn, c, xa, xb;
    };
    // chunks this far along: the table's entries, then the contacts, then the sides
    uint32_t at = threadIdx.x >> 5, base = 0;  // chunk of the table read next; its iteration's first turn
    uint32_t first = 0, end = 0, turn = kNone;
    auto read_table = [&] {
        while (at >= chunks.n) {
            at -= chunks.n;
            base += chunks.levels;
        }
        turn = base + chunks.level[at];
        first = chunks.first[at];
        end = min(first + 32u, at + 1 < chunks.n ? chunks.first[at + 1] : f.nc);
        at += W;
    };
    auto read_part = [&] {
        Part p{turn, kNone, 0u, 0u};
        if (first + lane < end) p.c = f.order[first + lane];
        return p;
    };
    auto read_sides = [&](Part& p) {
        if (p.c == kNone) return;
        p.xa = f.info[2 * p.c];
        p.xb = f.info[2 * p.c + 1];
    };
    auto fetch = [&](uint32_t c) {
        if (c == kNone || !staged) return;
        const float4* from = f.rec.at(c);
#pragma unroll
        for (uint32_t j = 0; j < kRecWords; ++j) copy_async(slot + j * f.rec.slots, from + j);
    };
    const uint32_t turns = f.iters * chunks.levels;
    read_table();
    Part cur = read_part();
    read_table();
    Part next = read_part();
    read_table();
    read_sides(cur);
    read_sides(next);
    Rec h{};
    if (cur.c != kNone) h = record(cur.c);
    auto advance = [&] {  // cur <- next
        cur = next;
        next = read_part();
        read_sides(next);
        read_table();
    };
    for (uint32_t k = 0; k < turns; ++k) {
        bool later = false;  // the next chunk's record is still to be loaded
        while (cur.turn == k) {
            const bool soon = next.turn <= k + 1;
            if (soon) fetch(next.c);
            if (cur.c != kNone) {
                const uint32_t la = cur.xa & kSideBody, lb = cur.xb & kSideBody;
                const float4 va = ld4(B.v + la), wa = ld4(B.w + la), vb = ld4(B.v + lb), wb = ld4(B.w + lb);
                const State y = update(h, true,
                                       State{mk(va.x, va.y, va.z), mk(wa.x, wa.y, wa.z),
                                             mk(vb.x, vb.y, vb.z), mk(wb.x, wb.y, wb.z), f.lam[cur.c]});
                if (!(cur.xa & kSideFree)) {
                    st4(B.v + la, make_float4(y.va.x, y.va.y, y.va.z, 0.0f));
                    st4(B.w + la, make_float4(y.wa.x, y.wa.y, y.wa.z, 0.0f));
                }
                if (!(cur.xb & kSideFree)) {
                    st4(B.v + lb, make_float4(y.vb.x, y.vb.y, y.vb.z, 0.0f));
                    st4(B.w + lb, make_float4(y.wb.x, y.wb.y, y.wb.z, 0.0f));
                }
                f.lam[cur.c] = y.lam;
            }
            if (!soon) {
                later = true;
                break;
            }
            advance();
            copies_done();
            if (cur.c != kNone)
                h = staged ? load_rec(slot, f.rec.slots) : record(cur.c);
        }
        part_sync<W>(32 * W);
        if (later) {
            advance();
            if (cur.c != kNone) h = record(cur.c);
        }
    }
}

// The lone contacts (no other contact at their dynamic bodies): all their
// iterations at once, 32 contacts per warp, the batches by ticket.
__device__ __forceinline__ void lone_sweep(const FlowArgs& f, const FlowBodies& B, uint32_t total,
                                           uint32_t* ticket) {
    const uint32_t lane = threadIdx.x & 31u;
    for (;;) {
        uint32_t b = 0;
        if (lane == 0) b = atomicAdd(ticket, 1u);
        b = f.nc + 32 * __shfl_sync(0xFFFFFFFFu, b, 0);
        if (b >= total) return;
        if (b + lane >= total) continue;
        const uint32_t c = f.order[b + lane], xa = f.info[2 * c], xb = f.info[2 * c + 1];
        if (xa & kSideSkip) continue;
        const Rec h = load_rec(f.rec.at(c), f.rec.stride);
        const uint32_t la = xa & kSideBody, lb = xb & kSideBody;
        const float4 va = ld4(B.v + la), wa = ld4(B.w + la), vb = ld4(B.v + lb), wb = ld4(B.w + lb);
        State x{mk(va.x, va.y, va.z), mk(wa.x, wa.y, wa.z), mk(vb.x, vb.y, vb.z),
                mk(wb.x, wb.y, wb.z), 0.0f};
        for (uint32_t it = 0; it < f.iters; ++it) {
            if (xa & kSideSame) {
                x.va = x.vb;
                x.wa = x.wb;
            }
            const State y = update(h, true, x);
            x.lam = y.lam;
            if (!(xa & kSideFree)) {  // a fixed body keeps its velocities
                x.va = y.va;
                x.wa = y.wa;
            }
            if (!(xb & kSideFree)) {
                x.vb = y.vb;
                x.wb = y.wb;
            }
        }
        if (!(xa & kSideFree)) {
            st4(B.v + la, make_float4(x.va.x, x.va.y, x.va.z, 0.0f));
            st4(B.w + la, make_float4(x.wa.x, x.wa.y, x.wa.z, 0.0f));
        }
        if (!(xb & kSideFree)) {
            st4(B.v + lb, make_float4(x.vb.x, x.vb.y, x.vb.z, 0.0f));
            st4(B.w + lb, make_float4(x.wb.x, x.wb.y, x.wb.z, 0.0f));
        }
        f.lam[c] = x.lam;
    }
}

struct RunShared {
    uint32_t order, failed, left, chained, by_level, placed[2], ticket;
};

// The solve of a run of nc contacts by a block of W warps, the bodies' velocities and
// the sides' words in place, left and ticket zero.  c0: the run's place in the scratch
// lists; contact(i), body(l): the contact and body that i and l stand for; lam: the
// impulses, zero before; deg: nc words.  Mode COLORED where a body needs more than 32
// colours: contact order, or (fall_back false) nothing is done and the result is false.
// kLevels: there may be more than kSweepFrom contacts per lane in contact order.
template <uint32_t W, bool kLevels, class Contact, class Body>
__device__ __forceinline__ bool solve_run(const World& w, const Consts& k, const Scratch& s,
                                          uint32_t mode, float dt, uint32_t c0, uint32_t nc,
                                          uint32_t nbs, const FlowBodies& B, uint32_t* info,
                                          uint32_t* order, const Recs& rec, float* lam, uint32_t* deg,
                                          uint32_t salt,
                                          bool fall_back, RunShared& sh, Contact contact, Body body) {
    constexpr uint32_t kThreads = 32 * W;
    const uint32_t t = threadIdx.x, lane = t & 31u, wid = t >> 5;
    // ---- ranks and positions by the last warp, records by the others ----
    if (wid == W - 1) {
        bool coloured = mode == 2, ok = true;
        if (coloured && !colour_sides(info, B, nc, deg, s.s_order + c0)) {
            coloured = false;  // contact order instead
            for (uint32_t i = lane; i < nbs; i += 32) *B.count(i) = 0;
            __syncwarp();
        }
        if (mode != 0 && !coloured) ok = rank_sides(info, B, nc);
        if (coloured) {
            __syncwarp();
            for (uint32_t i = lane; i < nbs; i += 32) *B.count(i) = __popc(*B.count(i));
            __syncwarp();
        }
        uint32_t chained = nc;
        bool by_level = false;
        if (mode != 0) {
            __syncwarp();
            if (kThreads == 32u && nc <= kThreads) {  // the warp runs the lone ones in the same rounds
                if (lane < nc) order[lane] = lane;
            } else {
                chained = count_chained(info, B, nc);
                by_level = kLevels && ok && !coloured && chained > kSweepFrom * kThreads;
                if (!by_level)
                    order_contacts(info, B, nc, chained, kThreads, coloured ? s.s_order + c0 : nullptr, order);
            }
        }
        // contacts one by one, the reference's loop, when the ranks are too large
        if (lane == 0) {
            sh.order = mode != 0 && ok;
            sh.failed = mode == 2 && !coloured;
            sh.chained = chained;
            sh.by_level = by_level;
            sh.placed[0] = sh.placed[1] = 0;
        }
    }
    if (W == 1 || wid < W - 1)
        for (uint32_t i = t; i < nc; i += 32 * (W == 1 ? 1 : W - 1)) {
            const uint32_t la = info[2 * i] & kSideBody, lb = info[2 * i + 1] & kSideBody;
            const float4 va = B.v[la], wa = B.w[la], vb = B.v[lb], wb = B.w[lb];
            make_rec(w, k, contact(i), body(la), body(lb), mk(va.x, va.y, va.z), mk(wa.x, wa.y, wa.z),
                     mk(vb.x, vb.y, vb.z), mk(wb.x, wb.y, wb.z), dt, rec.at(i), rec.stride);
        }
    __syncthreads();
    if (sh.failed && !fall_back) return false;
    Chunks chunks{s.s_order + c0, s.s_lvl_start + c0, 0u, 0u};
    if (kLevels && sh.by_level) {
        chunks = build_levels<W>(info, B, nc, sh.chained, deg, order, chunks, sh.placed);
        __syncthreads();
    }

    if (!sh.order) {
        // ---- SEQUENTIAL: the reference order, one lane ----
        if (t == 0)
            for (uint32_t it = 0; it < k.pgs_iterations; ++it)
                for (uint32_t i = 0; i < nc; ++i) {
                    const uint32_t xa = info[2 * i], xb = info[2 * i + 1];
                    if (xa & kSideSkip) continue;
                    const uint32_t la = xa & kSideBody, lb = xb & kSideBody;
                    const float4 va = B.v[la], wa = B.w[la], vb = B.v[lb], wb = B.w[lb];
                    const State x = update(load_rec(rec.at(i), rec.stride), true,
                                           State{mk(va.x, va.y, va.z), mk(wa.x, wa.y, wa.z),
                                                 mk(vb.x, vb.y, vb.z), mk(wb.x, wb.y, wb.z),
                                                 lam[i]});
                    if (!(xa & kSideFree)) {
                        B.v[la] = make_float4(x.va.x, x.va.y, x.va.z, 0.0f);
                        B.w[la] = make_float4(x.wa.x, x.wa.y, x.wa.z, 0.0f);
                    }
                    if (!(xb & kSideFree)) {
                        B.v[lb] = make_float4(x.vb.x, x.vb.y, x.vb.z, 0.0f);
                        B.w[lb] = make_float4(x.wb.x, x.wb.y, x.wb.z, 0.0f);
                    }
                    lam[i] = x.lam;
                }
    } else {
        // contacts go to the warps from a different one on in each block, so that
        // the longest chains of an SM's blocks do not meet on one scheduler
        const uint32_t role = (wid + salt) % W, chained = sh.chained;
        const FlowArgs f{chained, role * 32 + lane, kThreads, 32u * min(W, (chained + 31) / 32),
                         k.pgs_iterations, order, info, rec, lam, deg, &sh.left};
        if (role * 32 < chained) {  // dataflow rounds, by the warps that own chained contacts
            if (kLevels && sh.by_level)
                level_sweep<W>(f, B, chunks);
            else if (chained > kThreads)
                flow_sweep<W, true>(f, B);
            else
                flow_sweep<W, false>(f, B);
        }
        lone_sweep(f, B, nc, &sh.ticket);
    }
    __syncthreads();
    return true;
}

// room: float4s of shared memory, two for every body of the largest bundle at least.
template <uint32_t W>
__global__ void __launch_bounds__(32 * W, 12 / W)
    k_solver_flow(World w, Consts k, Scratch s, uint32_t mode, float dt, uint32_t room) {
    constexpr uint32_t kThreads = 32 * W;
    extern __shared__ float4 sm4[];
    __shared__ RunShared sh;
    wait_for_previous();
    if (halted(w.status)) return;  // contacts from a scan that gave up
    const uint32_t t = threadIdx.x;
    const uint32_t bundle = blockIdx.x;
    if (bundle >= w.nbundles) return;
    const uint32_t b0 = w.bundle_off[bundle], b1 = w.bundle_off[bundle + 1];
    const uint32_t c0 = first_contact(w, s, b0), c1 = first_contact(w, s, b1);
    if (c0 >= c1) return;
    const uint32_t nbs = b1 - b0, nc = c1 - c0;
    const FlowBodies B{sm4, sm4 + nbs};
    uint32_t at = 2 * nbs;
    const uint32_t lists = (12 * nc + 15) / 16;
    const bool near = at + lists <= room;
    uint32_t* info = near ? reinterpret_cast<uint32_t*>(sm4 + at) : s.s_ab + size_t(c0) * 2;
    // (s_level: the colours of mode 2 are done with when the positions are made)
    uint32_t* order = near ? info + 2 * nc : s.s_level + c0;
    if (near) at += lists;
    const Recs rec(sm4 + at, room - at, s.s_rec + size_t(c0) * kRecWords, nc, kThreads);

    // ---- the bundle's bodies; every contact side's body and flags ----
    for (uint32_t i = t; i < nc; i += kThreads) {
        const uint32_t a = w.geom_body[w.c_a[c0 + i]], b = w.geom_body[w.c_b[c0 + i]];
        const float ma = w.inv_mass[a], mb = w.inv_mass[b];
        const f3 Ia = ld3(w.inv_inertia, a), Ib = ld3(w.inv_inertia, b);
        const bool fa = ma == 0.0f && Ia.x == 0.0f && Ia.y == 0.0f && Ia.z == 0.0f;
        const bool fb = mb == 0.0f && Ib.x == 0.0f && Ib.y == 0.0f && Ib.z == 0.0f;
        uint32_t xa = a - b0, xb = b - b0;
        if (ma == 0.0f && mb == 0.0f) {  // skipped (physics.comp:531)
            xa |= kSideSkip | kSideFree;
            xb |= kSideSkip | kSideFree;
        } else {
            if (fa) xa |= kSideFree;
            if (fb) xb |= kSideFree;
            if (a == b && !fb) xa |= kSideFree | kSideSame;
        }
        info[2 * i] = xa;
        info[2 * i + 1] = xb;
    }
    for (uint32_t i = t; i < nbs; i += kThreads) {
        const f3 v = ld3(w.vel, b0 + i), om = ld3(w.omega, b0 + i);
        B.v[i] = make_float4(v.x, v.y, v.z, 0.0f);
        B.w[i] = make_float4(om.x, om.y, om.z, 0.0f);
    }
    if (t == 0) sh.left = sh.ticket = 0;
    __syncthreads();
    solve_run<W, (W > 1)>(
        w, k, s, mode, dt, c0, nc, nbs, B, info, order, rec, w.lambda + c0, s.s_abp + c0, bundle,
        true, sh,
        [&](uint32_t i) { return c0 + i; }, [&](uint32_t l) { return b0 + l; });
    // ---- velocities back to the bound buffers ----
    for (uint32_t i = t; i < nbs; i += kThreads) {
        const float4 v = B.v[i], om = B.w[i];
        st3(w.vel, b0 + i, mk(v.x, v.y, v.z));
        st3(w.omega, b0 + i, mk(om.x, om.y, om.z));
    }
}

// ---- runs of islands --------------------------------------------------------
// Contacts sorted by island (islands.cu): a block takes the islands that start in a
// window of kIslandWindow sorted contacts and sweeps them as a bundle.  Their bodies
// are not consecutive: the first contact side that claims a body (s_last, zero before)
// gives it a slot; a fixed body, which several islands may share, gets one per side.
// Islands of more than kIslandMost contacts (in contact order kIslandWindow: a lane that
// owns several contacts takes them in turn, so a long chain's iterations no longer follow
// each other closely: 1,024 towers of 256 boxes 12.4 ms per substep, 10.7 ms by a warp
// each) and, in mode COLORED, runs with a body of more than 32 colours are marked in todo and counted in left[1] for the kernel that
// gives each island a warp (k_solver_island).  left[0]: the windows' ticket.
//
// Bound by issue (734 instructions per warp and round) where there are many islands:
// 1,024 towers of 256 boxes, 61 rounds each, 404 us per substep; a warp per island,
// swept level by level with the velocities in L2, took 651 us.  A settled pile of 2,601
// bodies (a chain of 91 rounds) 157 against 252 us.  Four warps, so that three blocks
// share an SM and a tower's colours of 128 contacts fill a round each.
constexpr uint32_t kIslandWarps = 4, kIslandSmem = 72 * 1024;
constexpr uint32_t kIslandWindow = 32 * kIslandWarps;
static_assert((kIslandMost + kIslandWindow) * 56 + kIslandWindow * 36 + 48 <= kIslandSmem,
              "a run's sides and bodies must fit");
static_assert(kIslandMost + 2 * kIslandWindow <= kSideBody, "body field too narrow");

__global__ void __launch_bounds__(32 * kIslandWarps, 12 / kIslandWarps)
    k_island_flow(World w, Consts k, Scratch s, uint32_t mode, float dt, uint32_t* todo, uint32_t* left) {
    constexpr uint32_t kThreads = 32 * kIslandWarps;
    extern __shared__ float4 sm4[];
    __shared__ RunShared sh;
    __shared__ uint32_t sh_window, sh_slots;
    wait_for_previous();
    if (halted(w.status)) return;
    const uint32_t t = threadIdx.x;
    const uint32_t count = *s.isl.count, total = s.isl.start[count];
    const uint32_t most_contacts = mode == 2 ? kIslandMost : kIslandWindow;
    const uint32_t* perm = s.isl.perm;
    // the first windows by block: few of them lie one to an SM
    for (bool first = true;; first = false) {
        if (t == 0) {
            sh_window = first ? blockIdx.x : gridDim.x + atomicAdd(&left[0], 1u);
            sh_slots = sh.left = sh.ticket = 0;
        }
        __syncthreads();
        const uint32_t from = sh_window * kIslandWindow;
        if (from >= total) return;
        const uint32_t ia = s.isl.idx[from];
        uint32_t ib = from + kIslandWindow < total ? s.isl.idx[from + kIslandWindow] : count;
        const uint32_t p0 = s.isl.start[ia];
        for (uint32_t i = ia + t; i < ib; i += kThreads) todo[i] = 0;
        // only the last island can reach past the window
        if (ib > ia && s.isl.start[ib] - s.isl.start[ib - 1] > most_contacts) {
            --ib;
            __syncthreads();
            if (t == 0) {
                todo[ib] = 1;
                atomicAdd(&left[1], 1u);
            }
        }
        const uint32_t nc = ib > ia ? s.isl.start[ib] - p0 : 0u;
        if (nc > 0) {
            uint32_t* info = reinterpret_cast<uint32_t*>(sm4);
            uint32_t *order = info + 2 * nc, *deg = info + 3 * nc;
            float* lam = reinterpret_cast<float*>(info + 4 * nc);
            const uint32_t most = nc + (ib - ia);  // bodies: a tree's, an island, at most
            float4* const bodies = sm4 + (5 * nc + 3) / 4;
            const FlowBodies B{bodies, bodies + most};
            uint32_t* list = reinterpret_cast<uint32_t*>(bodies + 2 * most);
            const uint32_t used = (5 * nc + 3) / 4 + 2 * most + (most + 3) / 4;
            const Recs rec(sm4 + used, kIslandSmem / 16 - used, s.s_rec + size_t(p0) * kRecWords, nc, kThreads);
            auto fixed = [&](uint32_t b) {
                const f3 I = ld3(w.inv_inertia, b);
                return w.inv_mass[b] == 0.0f && I.x == 0.0f && I.y == 0.0f && I.z == 0.0f;
            };
            auto claim = [&](uint32_t b, bool f) {
                if (!f && atomicCAS(&s.s_last[b], 0u, kNone) != 0u) return 0u;
                const uint32_t slot = atomicAdd(&sh_slots, 1u);
                const f3 v = ld3(w.vel, b), om = ld3(w.omega, b);
                B.v[slot] = make_float4(v.x, v.y, v.z, 0.0f);
                B.w[slot] = make_float4(om.x, om.y, om.z, 0.0f);
                list[slot] = f ? b | 0x80000000u : b;
                if (!f) atomicExch(&s.s_last[b], slot + 1u);
                return slot;
            };
            for (uint32_t i = t; i < nc; i += kThreads) {
                const uint32_t c = perm[p0 + i];
                const uint32_t a = w.geom_body[w.c_a[c]], b = w.geom_body[w.c_b[c]];
                info[2 * i] = claim(a, fixed(a));
                info[2 * i + 1] = claim(b, fixed(b));
                lam[i] = 0.0f;
            }
            __syncthreads();
            for (uint32_t i = t; i < nc; i += kThreads) {
                const uint32_t c = perm[p0 + i];
                const uint32_t a = w.geom_body[w.c_a[c]], b = w.geom_body[w.c_b[c]];
                const bool fa = fixed(a), fb = fixed(b);
                const uint32_t la = fa ? info[2 * i] : __ldcg(&s.s_last[a]) - 1u;
                const uint32_t lb = fb ? info[2 * i + 1] : __ldcg(&s.s_last[b]) - 1u;
                info[2 * i] = la | (fa ? kSideFree : 0u) | (a == b && !fb ? kSideFree | kSideSame : 0u);
                info[2 * i + 1] = lb | (fb ? kSideFree : 0u);
            }
            __syncthreads();
            const uint32_t slots = sh_slots;
            const bool done = solve_run<kIslandWarps, false>(
                w, k, s, mode, dt, p0, nc, slots, B, info, order, rec, lam, deg, sh_window, false,
                sh, [&](uint32_t i) { return perm[p0 + i]; },
                [&](uint32_t l) { return list[l] & 0x7FFFFFFFu; });
            for (uint32_t l = t; l < slots; l += kThreads) {
                const uint32_t b = list[l];
                if (b & 0x80000000u) continue;
                if (!done) {  // as the warp-per-island kernel expects it
                    s.s_last[b] = 0;
                    continue;
                }
                const float4 v = B.v[l], om = B.w[l];
                st3(w.vel, b, mk(v.x, v.y, v.z));
                st3(w.omega, b, mk(om.x, om.y, om.z));
            }
            if (done)
                for (uint32_t i = t; i < nc; i += kThreads) w.lambda[perm[p0 + i]] = lam[i];
            else
                for (uint32_t i = ia + t; i < ib; i += kThreads) {
                    todo[i] = 1;
                    atomicAdd(&left[1], 1u);
                }
        }
        __syncthreads();
    }
}

int launch_island_flow(const World& w, const Consts& k, const Scratch& s, uint32_t mode, float dt,
                       uint32_t sms, uint32_t* todo, uint32_t* left, cudaStream_t st) {
    const uint32_t windows = (w.max_contacts + kIslandWindow - 1) / kIslandWindow;
    launch_after(k_island_flow, std::min(windows, sms * (12 / kIslandWarps)), 32 * kIslandWarps,
                 kIslandSmem, st, w, k, s, mode, dt, todo, left);
    return 1;
}

constexpr uint32_t kSolverMaxSmem = 160 * 1024;
constexpr uint32_t kFlowMaxSmem = 120 * 1024, kFlowSmem = 192 * 1024,
                   kFlowSmemGroups = 150 * 1024, kFlowSmemTwo = 79 * 1024 - 128,
                   kTwoPerSm = 2 * 148 + 148 / 5;

cudaError_t init_solver() {
    for (const void* f : {reinterpret_cast<const void*>(k_solver_flow<1>),
                          reinterpret_cast<const void*>(k_solver_flow<2>),
                          reinterpret_cast<const void*>(k_solver_flow<4>),
                          reinterpret_cast<const void*>(k_solver_flow<8>)}) {
        const cudaError_t e =
            cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kFlowMaxSmem));
        if (e != cudaSuccess) return e;
    }
    const cudaError_t ei = cudaFuncSetAttribute(
        k_island_flow, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kIslandSmem));
    if (ei != cudaSuccess) return ei;
    // opt in to more than 48 KB of dynamic shared memory; done at handle
    // creation so that no attribute call happens during graph capture
    return cudaFuncSetAttribute(k_solver, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                int(kSolverMaxSmem));
}

// Warps per block by the largest bundle: a settled pile has about a quarter
// contact per body, two thirds of them chained, and the warps without chained
// contacts take the lone ones.  Solver time per substep with 1 / 2 / 4 warps:
// 1,024 scenes in 512-body bundles 274 / 226 / 183 us, one 512-body scene
// - / 162 / 124 us.  Above 512 bodies eight warps keep a lane for most chained
// contacts but take an SM each, so more bundles than SMs, or scene groups (whose other
// kernels run beside), get four: 4,096 scenes in 1,024-body bundles 471 us with eight,
// 341 with four, and with eight groups 11.7 and 10.5 ms per frame; one scene of 1,000
// bodies 1.92 ms per frame with eight, 2.13 with four.
//
// Blocks of up to four warps share an SM as its registers allow (twelve warps), with an
// equal part each of 192 KB of shared memory, of which the system takes a block's first
// KB.  With 228 KB two blocks of four warps fitted (77,824 bytes each, 454 us for 4,096
// scenes in 512-body bundles; 377 with three), and three of 76,700 bytes leave the SM's
// other kernels next to no L1: with eight groups 13.4 ms per frame, 11.2 with 192 KB.
// Scene groups' bundles of up to 512 bodies, whose records mostly fit, share 150 KB: 8
// groups of 128 scenes 4.29 ms per frame with 192 KB, 4.26 with 150.  Two blocks of four
// warps to an SM while that leaves few bundles over, which start as the first ones end: a
// third block beside the longest chain costs more, and more records fit (1,024 scenes, 306
// bundles: 4.30 ms per frame with two, 4.14 to 4.51 with three, by where the chain lies;
// 1,150 scenes 4.52 and 4.38).
static void launch_flow(const World& w, const Consts& k, const Scratch& s, uint32_t mode, float dt,
                        uint32_t nbmax, cudaStream_t st) {
    const uint32_t warps = nbmax <= 128                                            ? 1u
                           : nbmax <= 256                                          ? 2u
                           : nbmax <= 512 || w.nbundles > 148u || s.order_pairs != 0 ? 4u
                                                                                   : 8u;
    const uint32_t share = s.order_pairs != 0 && nbmax <= 512 ? kFlowSmemGroups : kFlowSmem;
    uint32_t part = warps <= 4 ? share / (12 / warps) - 1024u - 128u : kFlowMaxSmem;
    if (warps == 4 && s.order_pairs == 0 && w.nbundles <= kTwoPerSm) part = kFlowSmemTwo;
    const uint32_t smem = std::max(part, 32 * nbmax) & ~15u;
    switch (warps) {
        case 1: launch_after(k_solver_flow<1>, w.nbundles, 32, smem, st, w, k, s, mode, dt, smem / 16); break;
        case 2: launch_after(k_solver_flow<2>, w.nbundles, 64, smem, st, w, k, s, mode, dt, smem / 16); break;
        case 4: launch_after(k_solver_flow<4>, w.nbundles, 128, smem, st, w, k, s, mode, dt, smem / 16); break;
        default: launch_after(k_solver_flow<8>, w.nbundles, 256, smem, st, w, k, s, mode, dt, smem / 16);
    }
}

int launch_solver(const World& w, const Consts& k, const Scratch& s, uint32_t mode, float dt,
                  uint32_t max_scene_bodies, cudaStream_t st) {
    if (w.nbundles == 0 || w.max_contacts == 0) return 0;
    if (max_scene_bodies <= kWarpMaxBodies) {
        launch_flow(w, k, s, mode, dt, std::max(max_scene_bodies, 1u), st);
        return 1;
    }
    if (s.isl.parent) return launch_solver_islands(w, k, s, mode, dt, st);
    uint32_t cta_bodies = max_scene_bodies;
    if (cta_bodies * kBodySmemWords * 4 > kSolverMaxSmem)
        cta_bodies = kSolverMaxSmem / (kBodySmemWords * 4);
    const size_t smem = size_t(cta_bodies) * kBodySmemWords * 4;
    k_solver<<<w.nbundles, kSolverThreads, smem, st>>>(w, k, s, mode, dt, cta_bodies);
    return 1;
}

}  // namespace seevr
