// All iterations of a step in one launch for worlds whose colours leave the chip mostly idle:
// each body is solved by 8 or 32 lanes of one warp, and warps hand bodies to one another
// through stamped 16-byte words.
//
// What bounds such a world is the chain from one colour's bodies to the next colour's, not
// bandwidth or issue. k_iterations spends per link of that chain a release store (the body's
// pose must be visible before its count), an acquire poll (which also empties the SM's L1), a
// second trip to L2 for the data behind the count, ceil(rows / 4) rounds of rows, a barrier
// of 256 threads and a factorisation on one thread. Here:
//  - a body's pose, a contact's and a joint's multipliers travel in 16-byte words that carry
//    their version next to three floats, written and read as single 128-bit relaxed accesses
//    (one copy, never torn): the poll brings the data, no fence orders separate words, and
//    constant data (bases, anchors, row lists) stays in L1;
//  - the group of lanes is as wide as the colour leaves room for, so a body's rows take one
//    round (two for the fullest), and nothing waits outside the warp;
//  - the 6x6 factorisation takes one lane per matrix row (ldl_solve_team), the divisions of a
//    column side by side.
// Every float operation and the order of every sum are those of primal_batch and
// ldl_solve27, so the results are the same bits. Measured against k_iterations (us for the 10
// iterations of a step): a 20-link rope 172 -> 67, the 210-box pyramid 404 -> 85, 6,000 mixed
// bodies 303 -> 115, 4,096 boxes in stacks 202 -> 65, 20,000 poured spheres (3,950 solved) 385
// -> 120, 64 uneven worlds (13,700 solved) 292 -> 129.
//
// What is left is one warp's instruction latency: a body's own 1,100 instructions a pass take
// 5,000 to 6,000 cycles. A straight run of code costs 1.3 cycles an instruction while it fits
// the instruction cache next to the scheduler and 3.3 beyond about 2,000 instructions, so rare
// cases share code with common ones here rather than being unrolled.
//
// Versions. A body's words carry the iterations it has completed (0: the warm start's pose), a
// contact's and a joint's the dual updates made. Rows wait as in k_iterations: a partner of
// an earlier colour must have finished this iteration, one of a later colour the previous one;
// the owner of a contact or joint (the earlier colour, or the only dynamic body) makes its
// dual update of iteration k - 1 in iteration k, and the partner's row of iteration k waits for
// that update's words. A word is never overwritten before its readers are done: whoever
// writes version k + 1 has seen a stamp that each reader of version k set after its read.
// Each wait is for a strictly earlier (iteration, colour) and all blocks are resident, so the
// waits cannot cycle; on expiry of the poll limit the kernel records an error, as k_iterations
// does.
//
// contactFlow, two words per slot: (pen.xyz, C0.z) with the low bit of the version in the sign
// of pen.x (a penalty is at least PENALTY_MIN and its ramp not negative, choose_wide; a reader is
// at most one version behind), and (lambda.xyz, version << 1 | stick). jointFlow, four words per
// joint: (penLin, version << 1 | broken) (penAng, version) (lamLin, version) (lamAng, version).
// The contact and joint records themselves are written once, with the last update.
#pragma once

namespace avbd
{

// One block per SM of 12 warps: up to 168 registers a thread (the instances take 162 to 165, none
// spills), which the words in flight need.
constexpr int WIDE_BLOCK = 384, WIDE_WARPS = WIDE_BLOCK / 32, WIDE_MIN_GROUP = 8;

struct WideShared
{
    static constexpr int GROUPS = WIDE_BLOCK / WIDE_MIN_GROUP;
    float term[WIDE_BLOCK][E_COUNT]; // one row per lane (odd stride: no bank conflicts)
    float sys[GROUPS][E_COUNT];
    float4 self[GROUPS][FLOW_USED]; // the body's stamped words
};

AVBD_DEV float4 ld_flow(const float4 *p)
{
    unsigned long long a, b;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
    return make_float4(__uint_as_float((unsigned)a), __uint_as_float((unsigned)(a >> 32)),
                       __uint_as_float((unsigned)b), __uint_as_float((unsigned)(b >> 32)));
}

AVBD_DEV void st_flow(float4 *p, float4 v)
{
    const unsigned long long a = (unsigned long long)__float_as_uint(v.x) |
                                 ((unsigned long long)__float_as_uint(v.y) << 32);
    const unsigned long long b = (unsigned long long)__float_as_uint(v.z) |
                                 ((unsigned long long)__float_as_uint(v.w) << 32);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(a), "l"(b)
                 : "memory");
}

AVBD_DEV int stamp_of(float4 w) { return __float_as_int(w.w); }

struct WideFlow
{
    int it;
    int *error;
    unsigned spinLimit;
    float4 *poseTape, *lpNow, *lpNext; // a taped step's records (IterFlow), else null
    int tapeN;
};

AVBD_DEV Motion motion_of_words(float4 w0, float4 w1, float4 w2, float4 w3)
{
    Motion m;
    m.q = make_float4(w0.x, w0.y, w0.z, w1.x);
    m.dLin = f3(w1.y, w1.z, w2.x);
    m.dAng = f3(w2.y, w2.z, w3.x);
    return m;
}

AVBD_DEV BodyPose pose_of_words(float4 w0, float4 w1, float4 w4)
{
    BodyPose s;
    s.q = make_float4(w0.x, w0.y, w0.z, w1.x);
    s.p = xyz(w4);
    return s;
}

// Keeps a value computed where it stands: before the wait, beside it.
AVBD_DEV void here(float3 &v) { asm volatile("" : "+f"(v.x), "+f"(v.y), "+f"(v.z)); }

// What a contact row of `self` (its words S in shared memory) has of its own: its share of C
// (eval_contact_arms) needs nothing of the partner.
struct WideContact
{
    ContactRec c;
    M3 basis, jLin, jAng; // self's Jacobian rows
    float3 myLin, myAng;  // their products with self's pose difference
    float friction;
    bool round;
};

template <bool ROUND>
AVBD_DEV float3 wide_arm(const DevBodies &B, const WideContact &w, int body, bool isA, float4 q)
{
    const float3 r = isA ? w.c.rA : w.c.rB;
    return ROUND && w.round ? contact_offset(body_shape(B, body), q, r, w.basis, isA, w.c.key) : rotate(q, r);
}

// `key`: the feature key is needed (round bodies' arms need it too)
template <bool ROUND>
AVBD_DEV void wide_contact_begin(const DevBodies &B, const DevForces &F, unsigned m, int ci, bool isA, int self,
                                 const float4 *S, bool key, WideContact &w)
{
    const float4 *bs = F.man.basis + 3 * (size_t)m, *record = F.man.contact + (size_t)m * 32 + 4 * ci;
    const float4 b0 = bs[0], b1 = bs[1], b2 = bs[2], c0 = record[0], c1 = record[1];
    w.c.rA = f3(c0.x, c0.y, c0.z);
    w.c.rB = f3(c0.w, c1.x, c1.y);
    w.c.C0 = f3(c1.z, c1.w, 0.0f);
    w.c.key = ROUND || key ? (int)(__float_as_uint(record[3].w) & 0x7FFFFFFFu) : 0;
    w.friction = b0.w;
    w.basis = rows(xyz(b0), xyz(b1), xyz(b2));
    w.round = ROUND && b1.w != 0.0f;
    const Motion me = motion_of_words(S[0], S[1], S[2], S[3]);
    const float3 rW = wide_arm<ROUND>(B, w, self, isA, me.q);
    w.jLin = isA ? w.basis : mneg(w.basis);
    w.jAng = rows(cross(rW, w.jLin.r0), cross(rW, w.jLin.r1), cross(rW, w.jLin.r2));
    w.myLin = mv(w.jLin, me.dLin);
    w.myAng = mv(w.jAng, me.dAng);
}

// C with the partner's motion, and the contact's state from its words d0, d1.
template <bool ROUND>
AVBD_DEV float3 wide_contact_end(const DevBodies &B, const Params &P, bool isA, int partner, const Motion &other,
                                      float4 d0, float4 d1, WideContact &w)
{
    ContactRec &c = w.c;
    c.C0.z = d0.w;
    c.pen = f3(fabsf(d0.x), d0.y, d0.z);
    c.lam = xyz(d1);
    c.stick = (stamp_of(d1) & 1) != 0;
    const float3 rO = wide_arm<ROUND>(B, w, partner, !isA, other.q);
    const M3 oLin = isA ? mneg(w.basis) : w.basis;
    const M3 oAng = rows(cross(rO, oLin.r0), cross(rO, oLin.r1), cross(rO, oLin.r2));
    const float3 othLin = mv(oLin, other.dLin), othAng = mv(oAng, other.dAng);
    return add(add(add(add(mul(c.C0, 1.0f - P.alpha), isA ? w.myLin : othLin), isA ? othLin : w.myLin),
                   isA ? w.myAng : othAng),
               isA ? othAng : w.myAng);
}

AVBD_DEV JointState joint_of_words(float4 j0, float4 j1, float4 j2, float4 j3)
{
    JointState s;
    s.penLin = xyz(j0);
    s.penAng = xyz(j1);
    s.lamLin = xyz(j2);
    s.lamAng = xyz(j3);
    s.broken = (stamp_of(j0) & 1) ? 1.0f : 0.0f;
    return s;
}

// One listed row's contribution, with the previous iteration's dual update where this body
// owns the contact or joint. Every lane of the warp calls this, and the warp waits as one: the
// seven words a row can need have the same places for every kind of row, so the poll is one loop
// that all lanes leave together (lanes that left a loop of their own one by one stayed
// apart through the rest of the pass). `mine` false: a lane that only goes along, waits for
// nothing and stores nothing but its own `t`. jointOut / jointStore: an updated joint, to be
// stored by the caller once every lane of the warp has read the previous version.
template <bool ROUND, bool TAPE>
AVBD_DEV unsigned wide_row(const DevBodies &B, const DevForces &F, const Params &P, int2 row, int self,
                           const float4 *S, const WideFlow &flow, float *t, bool mine, JointState &jointOut,
                           int &jointStore)
{
    constexpr unsigned ALL = 0xFFFFFFFFu;
    const unsigned e = (unsigned)row.x;
    const unsigned i = adj_index(e), type = adj_type(e);
    const bool isA = adj_isA(e) != 0;
    const int sub = row_sub(row), partner = row_partner(row), it = flow.it;
    const bool owns = (row.y & ROW_OWNS_DUAL) != 0, dual = owns && it > 0;
    const int needBody = partner < 0 ? INT_MIN : (!owns ? it + 1 : ((row.y & ROW_PARTNER_LATER) ? it : 0));
    const int needDual = owns ? max(it - 1, 0) : it;
    const bool contact = type == ADJ_MANIFOLD, joint = type == ADJ_JOINT;
    WideContact w;
    if (contact)
    {
        wide_contact_begin<ROUND>(B, F, i, sub, isA, self, S, TAPE, w);
        here(w.jAng.r0);
        here(w.jAng.r1);
        here(w.jAng.r2);
        here(w.myLin);
        here(w.myAng);
    }
    // contact: w0 - w3 the partner's motion, w4 w5 the contact's words; joint: w0 - w2 the
    // partner's pose, w3 - w6 the joint's words; spring: w0 - w2. What is not needed is a copy.
    const float4 *pw = B.flow + (size_t)(partner >= 0 ? partner : self) * FLOW_STRIDE;
    float4 *fw = contact ? F.contactFlow + 16 * (size_t)i + 2 * sub : (joint ? F.jointFlow + 4 * (size_t)i : nullptr);
    const float4 *a2 = pw + (contact ? 2 : 4), *a3 = contact ? pw + 3 : (joint ? fw : pw);
    const float4 *a4 = joint ? fw + 1 : (contact ? fw : pw), *a5 = joint ? fw + 2 : (contact ? fw + 1 : pw);
    const float4 *a6 = joint ? fw + 3 : pw;
    float4 w0, w1, w2, w3, w4, w5, w6;
    unsigned spins = 0;
    for (;;)
    {
        w0 = ld_flow(pw);
        w1 = ld_flow(pw + 1);
        w2 = ld_flow(a2);
        w3 = ld_flow(a3);
        w4 = ld_flow(a4);
        w5 = ld_flow(a5);
        w6 = ld_flow(a6);
        bool ready = min(min(stamp_of(w0), stamp_of(w1)), stamp_of(w2)) >= needBody;
        if (contact)
            ready = ready && stamp_of(w3) >= needBody && (stamp_of(w5) >> 1) >= needDual &&
                    (int)(__float_as_uint(w4.x) >> 31) == (needDual & 1);
        if (joint) // one version in all four words: the owner's own update may be made already
        {
            const int v = stamp_of(w3) >> 1;
            ready = ready && v == stamp_of(w4) && v == stamp_of(w5) && v == stamp_of(w6) &&
                    (v == needDual || (dual && v == it));
        }
        if (!__any_sync(ALL, !ready && mine))
            break;
        if (++spins >= flow.spinLimit)
        {
            atomicExch(flow.error, 1);
            break;
        }
        if (spins > 64)
        {
            if (__any_sync(ALL, *(volatile int *)flow.error != 0)) // another wait expired
                break;
            __nanosleep(32);
        }
    }
    unsigned kind = KIND_NONE;
    if (contact)
    {
        ContactEval ev;
        ev.C = wide_contact_end<ROUND>(B, P, isA, partner, motion_of_words(w0, w1, w2, w3), w4, w5, w);
        // the force, the owner's dual update with it, and the force after the update (a lane
        // without an update forms the same force twice: one copy of the code, see above)
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass)
        {
            contact_force(ev, w.c, w.friction);
            if (pass == 0 && dual)
                contact_dual(w.c, ev, P.betaLin);
        }
        if (dual && mine)
        {
            const unsigned sign = (unsigned)(it & 1) << 31;
            st_flow(fw, make_float4(__uint_as_float((__float_as_uint(w.c.pen.x) & 0x7FFFFFFFu) | sign), w.c.pen.y,
                                    w.c.pen.z, w.c.C0.z));
            st_flow(fw + 1, f4(w.c.lam, __int_as_float((it << 1) | (w.c.stick ? 1 : 0))));
            if (TAPE)
                tape_contact_state(flow.lpNow, 8ll * i + sub, w.c);
        }
        contact_stamp(w.jLin, w.jAng, w.c.pen, ev.F, t);
        kind = KIND_FULL;
    }
    else if (type != ADJ_IGNORE)
    {
        BodyPose other = pose_of_words(w0, w1, w2);
        if (partner < 0)
        {
            other.p = f3(0, 0, 0);
            other.q = make_float4(0, 0, 0, 1);
        }
        const BodyPose me = pose_of_words(S[0], S[1], S[4]);
        const BodyPose A = isA ? me : other, Bb = isA ? other : me;
        if (joint)
        {
            const float4 *d = F.joint + 8 * (size_t)i;
            const bool hasA = isA || partner >= 0;
            JointState s = joint_of_words(w3, w4, w5, w6);
            if (dual && (stamp_of(w3) >> 1) < it)
            {
                joint_dual(d, hasA, A, Bb, P, s);
                if (sub == 0 && mine)
                {
                    jointOut = s;
                    jointStore = (int)i;
                }
            }
            const float3 pen = sub < 2 ? s.penLin : s.penAng;
            if (lensq(pen) > 0)
                kind = joint_rows(d, sub, isA, hasA, A, Bb, pen, sub < 2 ? s.lamLin : s.lamAng, P.alpha, t);
        }
        else
            kind = spring_rows(F.spring + 2 * (size_t)i, isA, A, Bb, t);
    }
    return kind;
}

// The last iteration's dual update of a force, by the body that moves last in it, on both
// final poses, into the force's record. The partner is static or of an earlier colour, so it
// is final, and this lane's row of this iteration has read the words used here: no wait.
template <bool ROUND, bool TAPE>
AVBD_DEV void wide_last_dual(const DevBodies &B, const DevForces &F, const Params &P, int2 row, int self,
                             const float4 *S, const WideFlow &flow)
{
    if (row.y & ROW_PARTNER_LATER)
        return;
    const unsigned e = (unsigned)row.x;
    const unsigned i = adj_index(e);
    const bool isA = adj_isA(e) != 0;
    const int sub = row_sub(row), partner = row_partner(row);
    const float4 *pw = B.flow + (size_t)(partner >= 0 ? partner : self) * FLOW_STRIDE;
    if (adj_type(e) == ADJ_MANIFOLD)
    {
        const float4 *fw = F.contactFlow + 16 * (size_t)i + 2 * sub;
        WideContact w;
        wide_contact_begin<ROUND>(B, F, i, sub, isA, self, S, true, w);
        const Motion other = motion_of_words(ld_flow(pw), ld_flow(pw + 1), ld_flow(pw + 2), ld_flow(pw + 3));
        ContactEval ev;
        ev.C = wide_contact_end<ROUND>(B, P, isA, partner, other, ld_flow(fw), ld_flow(fw + 1), w);
        contact_force(ev, w.c, w.friction);
        contact_dual(w.c, ev, P.betaLin);
        store_contact_state(F.man.contact + (size_t)i * 32 + 4 * sub, w.c);
        if (TAPE)
            tape_contact_state(flow.lpNext, 8ll * i + sub, w.c);
    }
    else if (adj_type(e) == ADJ_JOINT && sub == 0)
    {
        float4 *d = F.joint + 8 * (size_t)i;
        const float4 *fw = F.jointFlow + 4 * (size_t)i;
        BodyPose other = pose_of_words(ld_flow(pw), ld_flow(pw + 1), ld_flow(pw + 4));
        if (partner < 0)
        {
            other.p = f3(0, 0, 0);
            other.q = make_float4(0, 0, 0, 1);
        }
        const BodyPose me = pose_of_words(S[0], S[1], S[4]);
        JointState s = joint_of_words(ld_flow(fw), ld_flow(fw + 1), ld_flow(fw + 2), ld_flow(fw + 3));
        joint_dual(d, isA || partner >= 0, isA ? me : other, isA ? other : me, P, s);
        store_joint_state(d, s);
    }
}

// ldl_solve27 with lane i of the group (i < 6; further lanes repeat lane 5) holding row i of the
// matrix: per column, the pivot is formed by every lane, the column's entries and their
// divisions side by side, and the forward substitution goes along. Every entry sees the
// operations of ldl_solve27 in their order. All lanes of the warp call this; every lane
// receives the solution.
template <int G>
AVBD_DEV void ldl_solve_team(const float *s, int gl, float3 &xl, float3 &xa)
{
    constexpr unsigned ALL = 0xFFFFFFFFu;
    const int i = min(gl, 5);
    float a[6], diag[6], L[6], D[6];
#pragma unroll
    for (int j = 0; j < 6; ++j)
    {
        const int jj = min(j, i);
        const int at = i < 3 ? i * (i + 1) / 2 + jj
                             : (jj < 3 ? E_LC00 + 3 * (i - 3) + jj : E_LA00 + (i - 3) * (i - 2) / 2 + (jj - 3));
        a[j] = s[at];
        diag[j] = s[j < 3 ? j * (j + 1) / 2 + j : E_LA00 + (j - 3) * (j - 2) / 2 + (j - 3)];
        L[j] = 0.0f;
    }
    float y = -s[E_RL0 + i], dMine = 1.0f;
#pragma unroll
    for (int j = 0; j < 6; ++j)
    {
        float Lj[6];
#pragma unroll
        for (int k = 0; k < j; ++k)
            Lj[k] = __shfl_sync(ALL, L[k], j, G);
        const float yj = __shfl_sync(ALL, y, j, G);
        if (j == 0)
            D[0] = diag[0];
        else
        {
            float acc = Lj[0] * Lj[0] * D[0];
#pragma unroll
            for (int k = 1; k < j; ++k)
                acc = acc + Lj[k] * Lj[k] * D[k];
            D[j] = diag[j] - acc;
        }
        if (i == j)
            dMine = D[j];
        if (j < 5)
        {
            float v = a[j];
#pragma unroll
            for (int k = 0; k < j; ++k)
                v = v - Lj[k] * L[k] * D[k];
            const bool below = i > j;
            const float q = fdiv(below ? v : 1.0f, below ? D[j] : 1.0f);
            if (below)
            {
                L[j] = q;
                y = y - q * yj;
            }
        }
    }
    const float z = fdiv(y, dMine);
    float x[6];
#pragma unroll
    for (int r = 5; r >= 0; --r)
    {
        float v = __shfl_sync(ALL, z, r, G);
#pragma unroll
        for (int k = r + 1; k < 6; ++k)
            v = v - __shfl_sync(ALL, L[r], k, G) * x[k];
        x[r] = v;
    }
    xl = f3(x[0], x[1], x[2]);
    xa = f3(x[3], x[4], x[5]);
}

// One body per group of G lanes: rows, solve, publication and, in the last iteration, the dual
// updates of the forces in which it moves last. Every lane of the warp calls this. A lane
// without a row of its own goes through its group's first one and a group without a body (live
// false) through the chunk's last, storing nothing, so the warp never splits around the rows:
// lanes that had gone ahead stayed apart through the sum, the factorisation and the
// publication (8 of 32 active), which then ran twice.
template <int G, bool ROUND, bool TAPE>
AVBD_DEV void wide_body(const DevBodies &B, const DevForces &F, const Params &P, int4 ent, bool live, bool last,
                        const WideFlow &flow, WideShared &sh)
{
    constexpr unsigned ALL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, gl = lane % G;
    const int warp = threadIdx.x >> 5, gi = warp * (32 / WIDE_MIN_GROUP) + lane / G;
    const int b = ent.x, r0 = ent.y, nr = ent.z - ent.y;
    const int maxRows = __reduce_max_sync(ALL, nr);
    float4 *S = sh.self[gi];
    float *sys = sh.sys[gi];
    float(*term)[E_COUNT] = sh.term + (threadIdx.x - gl);
    if (gl < FLOW_USED)
        S[gl] = ld_flow(B.flow + (size_t)b * FLOW_STRIDE + gl);
    const float4 i0 = B.initLin[b], a0inv = B.initAngInv[b];
    __syncwarp();
    const float4 q0 = make_float4(S[0].x, S[0].y, S[0].z, S[1].x);
    const float3 p0 = xyz(S[4]);
    // entry gl + k G of the system in acc[k], from M/dt^2 on
    constexpr int OWN = (E_COUNT + G - 1) / G;
    float acc[OWN];
    {
        const float4 md = B.massDt2[b];
        const float z = zero_over(P.dt * P.dt);
        const float3 dl = sub(p0, xyz(B.inertLin[b])), da = qdiff_inv(q0, B.inertAngInv[b]);
        const float3 RL = f3(dot(f3(md.x, z, z), dl), dot(f3(z, md.x, z), dl), dot(f3(z, z, md.x), dl));
        const float3 RA = f3(dot(f3(md.y, z, z), da), dot(f3(z, md.z, z), da), dot(f3(z, z, md.w), da));
#pragma unroll
        for (int k = 0; k < OWN; ++k)
        {
            const int e = gl + k * G;
            float v = e < E_LC00 ? z : 0.0f;
            v = e == E_LL00 || e == E_LL11 || e == E_LL22 ? md.x : v;
            v = e == E_LA00 ? md.y : (e == E_LA11 ? md.z : (e == E_LA22 ? md.w : v));
            v = e == E_RL0 ? RL.x : (e == E_RL1 ? RL.y : (e == E_RL2 ? RL.z : v));
            acc[k] = e == E_RA0 ? RA.x : (e == E_RA1 ? RA.y : (e == E_RA2 ? RA.z : v));
        }
    }
    for (int base = 0; base < maxRows; base += G)
    {
        JointState js;
        int jointStore = -1;
        const bool has = live && base + gl < nr;
        const int2 row = nr > 0 ? F.rows[r0 + (has ? base + gl : 0)] : make_int2((int)make_adj(ADJ_IGNORE, 0, 0), 0);
        unsigned kind = wide_row<ROUND, TAPE>(B, F, P, row, b, S, flow, term[gl], has, js, jointStore);
        if (!has)
            kind = KIND_NONE;
        __syncwarp(); // every lane's row is in shared memory, and has read its joint's words
        if (jointStore >= 0)
        {
            float4 *jw = F.jointFlow + 4 * (size_t)jointStore;
            st_flow(jw, f4(js.penLin, __int_as_float((flow.it << 1) | (js.broken != 0.0f ? 1 : 0))));
            st_flow(jw + 1, f4(js.penAng, __int_as_float(flow.it)));
            st_flow(jw + 2, f4(js.lamLin, __int_as_float(flow.it)));
            st_flow(jw + 3, f4(js.lamAng, __int_as_float(flow.it)));
        }
        // The group's rows, in order: which of them stamp which of this lane's entries; the
        // others count as -0, which leaves every float as it is, so no row is branched over.
        const int at = lane & ~(G - 1);
        const unsigned full = __ballot_sync(ALL, kind == KIND_FULL) >> at;
        const unsigned lhsAng = __ballot_sync(ALL, kind == KIND_LHSANG) >> at;
        const unsigned ang = __ballot_sync(ALL, kind == KIND_ANG) >> at;
        unsigned rows[OWN];
#pragma unroll
        for (int k = 0; k < OWN; ++k)
        {
            const int e = min(gl + k * G, E_COUNT - 1);
            rows[k] = full | (((KIND_LHSANG >> e) & 1u) ? lhsAng : 0u) | (((KIND_ANG >> e) & 1u) ? ang : 0u);
        }
        const int count = min(G, maxRows - base);
#pragma unroll 1
        for (int rr = 0; rr < count; rr += 4) // four rows are read ahead of their additions
        {
            float v[4][OWN];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int k = 0; k < OWN; ++k)
                    v[u][k] = term[rr + u][min(gl + k * G, E_COUNT - 1)];
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int k = 0; k < OWN; ++k)
                    acc[k] = acc[k] + (((rows[k] >> (rr + u)) & 1u) ? v[u][k] : -0.0f);
        }
        __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < OWN; ++k)
        if (gl + k * G < E_COUNT)
            sys[gl + k * G] = acc[k];
    __syncwarp();
    float3 dxl, dxa;
    ldl_solve_team<G>(sys, gl, dxl, dxa);
    // qstep(q0, dxa) with its four divisions side by side
    const float4 r = qadd(q0, qscale(qmul(make_float4(dxa.x, dxa.y, dxa.z, 0.0f), q0), 0.5f));
    const int cq = gl & 3;
    const float comp4 = cq == 0 ? r.x : (cq == 1 ? r.y : (cq == 2 ? r.z : r.w));
    const float qc = fdiv(comp4, sqrtf(qlensq(r)));
    const float4 q = make_float4(__shfl_sync(ALL, qc, 0, G), __shfl_sync(ALL, qc, 1, G), __shfl_sync(ALL, qc, 2, G),
                                 __shfl_sync(ALL, qc, 3, G));
    const float3 p = add(p0, dxl);
    const float3 dl = sub(p, xyz(i0)), da = qdiff_inv(q, a0inv);
    if (live && gl < FLOW_USED)
    {
        const float4 w = flow_word(gl, p, q, dl, da, flow.it + 1);
        st_flow(B.flow + (size_t)b * FLOW_STRIDE + gl, w);
        S[gl] = w;
    }
    if (TAPE && live && gl >= 5 && gl < 7)
        flow.poseTape[(size_t)(flow.it + 1) * 2 * flow.tapeN + (gl == 5 ? 0 : flow.tapeN) + b] =
            gl == 5 ? f4(p, 0.0f) : q;
    if (last)
    {
        if (live && gl == 0)
            B.dqLin[b] = f4(dl, 0.0f);
        if (live && gl == 1)
            B.dqAng[b] = f4(da, 0.0f);
        if (live && gl == 2)
            B.pos[b] = f4(p, 0.0f);
        if (live && gl == 3)
            B.quat[b] = q;
        __syncwarp();
        for (int k = live ? gl : nr; k < nr; k += G)
            wide_last_dual<ROUND, TAPE>(B, F, P, F.rows[r0 + k], b, S, flow);
    }
    __syncwarp();
}

// Chunks of G-lane groups the colours make: a chunk is a warp's worth of one colour's bodies.
template <int G>
AVBD_DEV int wide_chunks(const int *colourStart, int c)
{
    return (colourStart[c + 1] - colourStart[c] + 32 / G - 1) / (32 / G);
}

// Every iteration with groups of G lanes. The chunks of all colours, in colour order, are
// dealt to the warps of the grid, neighbouring chunks to different SMs; a warp without more than
// one prepares its bodies' next iteration while it waits for the other colours. A body keeps
// its lanes through the launch, so a force's owner reads its own previous update back on the
// same lane.
template <int G, bool ROUND, bool TAPE>
AVBD_DEV void wide_iterate(const DevBodies &B, const DevForces &F, const Params &P, const int4 *entries,
                           const int *colourStart, int chunks, int iterations, int *error, unsigned spinLimit,
                           const IterTape &tape, WideShared &sh)
{
    WideFlow flow;
    flow.error = error;
    flow.spinLimit = spinLimit;
    flow.poseTape = flow.lpNow = flow.lpNext = nullptr;
    flow.tapeN = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int it = 0; it < iterations; ++it)
    {
        flow.it = it;
        if constexpr (TAPE)
        {
            flow.poseTape = tape.pose;
            flow.tapeN = tape.n;
            flow.lpNow = tape.lp + (size_t)it * 16 * tape.nMan;
            flow.lpNext = flow.lpNow + (size_t)16 * tape.nMan;
        }
        int c = 0, before = 0; // the chunk's colour and the chunks of the colours before it
        for (int k = warp * gridDim.x + blockIdx.x; k < chunks; k += gridDim.x * WIDE_WARPS)
        {
            for (int in; k >= before + (in = wide_chunks<G>(colourStart, c)); ++c)
                before += in;
            const int at = colourStart[c] + (k - before) * (32 / G) + lane / G, end = colourStart[c + 1];
            wide_body<G, ROUND, TAPE>(B, F, P, entries[min(at, end - 1)], at < end, it == iterations - 1, flow, sh);
        }
    }
}

// Solver::iteratePrimalDualCpu (solver.cpp:1177-1271) for every iteration of a step.
//
// Groups of 8 lanes where bodies have about a row per lane or fewer; 32 lanes where they have
// more (one round of rows instead of two or three) and every warp still gets at most one
// chunk. Measured, iterations of a step at 8 / 16 / 32 lanes: 210-box pyramid (14 rows a body)
// 134 / 106 / 85 us, 4,096 boxes in stacks (8 rows) 64 / 66 / 71, 64 uneven worlds with jointed
// chains (6 rows, 13,700 bodies) 128 / 143 / 161.
template <bool ROUND, bool TAPE>
__global__ void __launch_bounds__(WIDE_BLOCK, 1) k_iterations_wide(DevBodies B, DevForces F, Params P,
                                                                   const int4 *entries, const int *colourStart,
                                                                   int nColours, int iterations, int *error,
                                                                   unsigned spinLimit, const StepState *st,
                                                                   const int *orphanFlag, IterTape tape)
{
    if (st)
    {
        if (step_aborted(st))
            return;
        nColours = st->nColours;
        F.nMan = st->nMan;
    }
    extern __shared__ __align__(16) unsigned char smemRaw[];
    WideShared &sh = *reinterpret_cast<WideShared *>(smemRaw);
    const int solved = nColours > 0 ? colourStart[nColours] : 0, rows = nColours > 0 ? F.rowStart[B.n] : 0;
    int chunks8 = 0, chunks32 = 0;
    for (int c = 0; c < nColours; ++c)
    {
        chunks8 += wide_chunks<8>(colourStart, c);
        chunks32 += wide_chunks<32>(colourStart, c);
    }
    if (rows > 7ll * solved && chunks32 <= (int)gridDim.x * WIDE_WARPS)
        wide_iterate<32, ROUND, TAPE>(B, F, P, entries, colourStart, chunks32, iterations, error, spinLimit, tape, sh);
    else
        wide_iterate<8, ROUND, TAPE>(B, F, P, entries, colourStart, chunks8, iterations, error, spinLimit, tape, sh);
    if (!orphanFlag || *orphanFlag == 0)
        return;
    // forces between static bodies: nothing moves them, so no barrier and no version is needed
    const long long stride = (long long)gridDim.x * WIDE_BLOCK;
    for (long long t = (long long)blockIdx.x * WIDE_BLOCK + threadIdx.x; t < 8ll * F.nMan; t += stride)
        orphan_contact_duals<ROUND>(B, F, P, t, iterations,
                                    TAPE ? tape.lp : nullptr, tape.nMan);
    for (long long j = (long long)blockIdx.x * WIDE_BLOCK + threadIdx.x; j < F.nJoint; j += stride)
        orphan_joint_duals(B, F, P, (int)j, iterations);
}

} // namespace avbd
