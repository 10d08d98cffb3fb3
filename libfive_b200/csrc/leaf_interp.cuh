// Tape interpreters of the leaf stage (DCTree::evalLeaf, libfive/src/render/
// brep/dc/dc_tree.inl:131-552): the clauses of a leaf group's pruned tape
// evaluated by one warp at four points per lane (corners and edge search,
// ArrayEvaluator::values, eval_array.cpp:106-118) or at one point per lane
// with derivatives (DerivArrayEvaluator::derivs, eval_deriv_array.cpp:
// 101-117).
//
// Layout for throughput on an interpreter whose cost is per step:
//  * clauses are decoded before they are run.  Values: k_leaf_decode turns a
//    tape into fused steps once (ValOp, several clauses each) and a warp
//    fetches them into shared memory.  Derivatives: the warp decodes
//    kLeafOps clauses at a time into LeafOps in shared memory (one clause
//    per lane), where opcode and operand kinds have become one handler
//    number and a constant or free-variable operand an immediate value;
//  * the register file holds one float4 per (register, lane): the four
//    points of a lane (or value + gradient) move with one 128-bit shared
//    memory access per operand.
// Arithmetic is the per-opcode arithmetic of dev_point.cuh, operation for
// operation, so values are bit-identical to the other evaluators'.
#pragma once
#include "dc_features.cuh"
#include "dev_interval.cuh"
#include "dev_point.cuh"

namespace lfb {

/// One decoded clause.  a, b, o are register numbers; `imm` is the value
/// of the immediate operand (flags bit 0: a is immediate, bit 1: b is; an
/// operand kind of OPND_CONST or OPND_VAR).  A clause whose every operand is
/// immediate is folded into H_SET (imm = its result; flags bit 2: it is a
/// min / max whose arguments tie).
struct __align__(16) LeafOp {
    uint8_t h;
    uint8_t op;
    uint8_t flags;
    uint8_t pad0;
    uint16_t a, b, o;
    uint16_t pad1;
    float imm;
};
static_assert(sizeof(LeafOp) == 16, "LeafOp is one 16-byte word");

enum : uint8_t {
    H_ADD_RR, H_ADD_RI, H_MUL_RR, H_MUL_RI, H_SUB_RR, H_SUB_RI, H_SUB_IR,
    H_MIN_RR, H_MIN_RI, H_MIN_IR, H_MAX_RR, H_MAX_RI, H_MAX_IR,
    H_SQUARE, H_SQRT, H_NEG, H_ABS, H_COPY, H_SET, H_GENERIC,
};

constexpr uint32_t kLeafOps = 64;   // decoded clauses per warp and chunk

/// Decodes one register-tape clause.  ADD and MUL with an immediate first
/// operand are swapped (both are exactly commutative, values and
/// derivatives alike); MIN, MAX and SUB are not.  `prev_out` is the result
/// register of the clause before (or 0xffff): flags bit 3 / bit 4 say that
/// operand a / b is that result, which the interpreters then take from
/// their registers instead of the register file.
__device__ __forceinline__ LeafOp leaf_decode(const RegClause& c, const float* __restrict__ cpool,
                                              uint32_t prev_out)
{
    LeafOp L;
    L.op = c.op;
    L.pad0 = 0;
    L.pad1 = 0;
    L.a = c.a;
    L.b = c.b;
    L.o = c.out;
    const uint8_t ka = c.kinds & 3, kb = (c.kinds >> 2) & 3;
    const bool bin = dev_is_binary(c.op);
    const bool ai = ka != OPND_REG, bi = bin && kb != OPND_REG;
    const float va = ai ? __ldg(cpool + c.a) : 0.0f;
    const float vb = bi ? __ldg(cpool + c.b) : 0.0f;
    L.flags = (ai ? 1 : 0) | (bi ? 2 : 0);
    L.imm = ai ? va : vb;
    if (ai && (bi || !bin)) {
        L.h = H_SET;
        L.imm = dv_value(c.op, va, vb);
        if ((c.op == op::MIN || c.op == op::MAX) && va == vb) L.flags |= 4;
        return L;
    }
    uint8_t h = H_GENERIC;
    switch (c.op) {
        case op::ADD:
        case op::MUL: {
            const bool mul = c.op == op::MUL;
            if (!ai && !bi) {
                h = mul ? H_MUL_RR : H_ADD_RR;
            } else {
                h = mul ? H_MUL_RI : H_ADD_RI;
                if (ai) {   // swap: register first
                    L.a = c.b;
                    L.b = c.a;
                    L.flags = 2;
                }
            }
            break;
        }
        case op::SUB: h = ai ? H_SUB_IR : bi ? H_SUB_RI : H_SUB_RR; break;
        case op::MIN: h = ai ? H_MIN_IR : bi ? H_MIN_RI : H_MIN_RR; break;
        case op::MAX: h = ai ? H_MAX_IR : bi ? H_MAX_RI : H_MAX_RR; break;
        case op::SQUARE: h = H_SQUARE; break;
        case op::SQRT: h = H_SQRT; break;
        case op::NEG: h = H_NEG; break;
        case op::ABS: h = H_ABS; break;
        case op::CONST_VAR:
        case OP_COPY: h = H_COPY; break;
        default: h = H_GENERIC; break;
    }
    L.h = h;
    if (!(L.flags & 1) && L.a == prev_out) L.flags |= 8;
    if (!(L.flags & 2) && dev_is_binary(c.op) && L.b == prev_out) L.flags |= 16;
    return L;
}

__device__ __forceinline__ RegClause leaf_unpack(uint2 raw)
{
    RegClause c;
    c.op = raw.x & 0xff;
    c.kinds = (raw.x >> 8) & 0xff;
    c.out = raw.x >> 16;
    c.a = raw.y & 0xffff;
    c.b = raw.y >> 16;
    return c;
}

/// The raw words of clauses c0 + lane and c0 + 32 + lane (the lane's share
/// of one chunk), loaded ahead of leaf_decode_chunk.
struct LeafRaw {
    uint2 w[2];
};
__device__ __forceinline__ LeafRaw leaf_fetch(const RegClause* __restrict__ cl, uint32_t len,
                                              uint32_t c0, int lane)
{
    LeafRaw r;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t i = c0 + lane + 32 * k;
        r.w[k] = i < len ? __ldg(reinterpret_cast<const uint2*>(cl + i)) : make_uint2(0, 0);
    }
    return r;
}

/// Decodes clauses [c0, c0 + kLeafOps) of a tape, whose raw words this lane
/// fetched into `raw`, into `ops` (the warp together); returns how many
/// there were.
__device__ __forceinline__ uint32_t leaf_decode_chunk(LeafOp* ops, const LeafRaw& raw,
                                                      uint32_t len, uint32_t c0,
                                                      const float* __restrict__ cpool, int lane)
{
    static_assert(kLeafOps == 64, "two clauses per lane");
    const uint32_t n = min(kLeafOps, len - c0);
    // result register of the clause before each of this lane's two
    const uint32_t out0 = raw.w[0].x >> 16, out1 = raw.w[1].x >> 16;
    const uint32_t up0 = __shfl_up_sync(0xffffffffu, out0, 1);
    const uint32_t last0 = __shfl_sync(0xffffffffu, out0, 31);
    const uint32_t up1 = __shfl_up_sync(0xffffffffu, out1, 1);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const uint32_t i = lane + 32 * k;
        if (i < n) {
            // the interpreters' forwarded result does not outlive a chunk:
            // nothing is forwarded into a chunk's first clause
            const uint32_t prev = lane > 0 ? (k ? up1 : up0) : (k ? last0 : 0xffffu);
            ops[i] = leaf_decode(leaf_unpack(raw.w[k]), cpool, prev);
        }
    }
    __syncwarp();
    return n;
}

__device__ __forceinline__ float4 splat4(float v) { return make_float4(v, v, v, v); }

__device__ __forceinline__ float f_square(float a) { return __fmul_rn(a, a); }
__device__ __forceinline__ float f_neg(float a) { return -a; }
__device__ __forceinline__ float f_sqrt(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ float f_abs(float a) { return fabsf(a); }
__device__ __forceinline__ float f_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float f_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float f_mul(float a, float b) { return __fmul_rn(a, b); }

__device__ __forceinline__ uint32_t tie4(const float4& a, const float4& b)
{
    return (a.x == b.x ? 1u : 0u) | (a.y == b.y ? 2u : 0u) | (a.z == b.z ? 4u : 0u) |
           (a.w == b.w ? 8u : 0u);
}

/// Every other opcode on four points, out of line.
static __device__ __noinline__ float4 leaf_generic4(uint8_t o, float4 a, float4 b)
{
    return make_float4(dv_value(o, a.x, b.x), dv_value(o, a.y, b.y), dv_value(o, a.z, b.z),
                       dv_value(o, a.w, b.w));
}

////////////////////////////////////////////////////////////////////////////////
// Values: fused steps

/// One step of the value interpreter.  A step first makes t from operand a
/// (a "unit": a clause with one register operand, or a run of such clauses
/// each in place on the one before, in the order below), then may combine t
/// with a second register b (a "tail": the two-register clause that reads
/// the unit's result next).  Every clause's own operation is kept,
/// separately rounded and in order, so values are those of the clauses one
/// by one.
///
/// Why steps: the interpreter's cost is per step (fetch, dispatch, operand
/// loads and the result's store, each a 512-byte shared-memory access that
/// the four schedulers of an SM share), not per operation; a sphere is 4
/// steps instead of 10 clauses, a box 3 instead of 11, a smooth union 4
/// instead of 9.  And dispatch by switch took 20 branches a step, so a unit
/// is one straight line,
///     t = f(a) (VF_FN);  t = ((t - i) & andm) ^ xorm;
///     t *= (VF_SQ ? t : m);  t -= j;  t = -t (VF_NEG)
/// whose unused parts are exact identities (subtracting +0, multiplying by
/// 1, all bits kept); t + i is t - (-i), and additions and subtractions of
/// b are additions of t and b with their signs flipped.
///
/// a, b, o and o2 are byte offsets into the warp's register file
/// (kValRegBytes a register); o2 is where t itself goes when the tail
/// writes another register.  Bit 0 of a / b: the operand is the step
/// before's result, taken from hardware registers.
struct __align__(16) ValOp {
    uint16_t a, b, o, o2;
    uint32_t flags;
    float i;
    uint32_t andm, xorm;   // VF_RARE: form (RARE_*)
    float m, j;
};
static_assert(sizeof(ValOp) == 32, "ValOp is two 16-byte words");

enum : uint32_t {
    VF_PRE = 1,        // t is not just operand a
    VF_RARE = 2,       // by opcode, out of line
    VF_FN = 4,         // a function first: square root, exp or log
    VF_SQ = 8,         // multiply by itself
    VF_TAIL = 16,
    VF_MM = 32,        // the tail is a min / max: (b < t) != VF_FLIP picks b,
    VF_SWAP = 64,      // ... with VF_SWAP (t < b) != VF_FLIP
    VF_FLIP = 128,
    VF_MUL = 256,      // the tail is a multiplication; otherwise an addition
    VF_NEG_T = 512,    // ... of -t
    VF_NEG_B = 1024,   // ... and -b
    VF_TIE = 2048,     // a min / max of two immediate operands that tie
    VF_NEG = 4096,     // negated last
    VF_OP_SHIFT = 16,  // opcode of VF_FN and VF_RARE
};
enum : uint32_t { RARE_SET, RARE_RI, RARE_IR, RARE_RR };
constexpr uint32_t kValRegBytes = 512;   // one float4 per lane
constexpr uint32_t kValMaxRegs = 128;    // register offsets fit 16 bits

/// Raw clauses of a chunk, with three empty ones on either side.
constexpr uint32_t kValRaw = kLeafOps + 6;

struct ValClause {
    uint32_t op, out;
    uint32_t a, b;       // operands: registers or pool indexes
    uint32_t r;          // the register operand of a clause with only one
    bool ai, bi, valid;
    bool one;            // one register operand (or none)
};
__device__ __forceinline__ ValClause val_clause(const uint2* raw, int c)
{
    const uint2 w = raw[c + 3];
    ValClause v;
    v.op = w.x & 0xff;
    v.out = w.x >> 16;
    v.a = w.y & 0xffff;
    v.b = w.y >> 16;
    const bool bin = dev_is_binary(static_cast<uint8_t>(v.op));
    v.ai = ((w.x >> 8) & 3) != OPND_REG;
    v.bi = !bin || ((w.x >> 10) & 3) != OPND_REG;
    v.valid = w.x != 0xffffffffu;
    v.one = v.ai || v.bi;
    v.r = v.ai ? (v.bi ? 0xffffffffu : v.b) : v.a;
    return v;
}
/// Clause v is in place on the clause before it, both in one unit's reach.
__device__ __forceinline__ bool val_linked(const ValClause& v, const ValClause& before)
{
    return v.valid && before.valid && v.one && before.one && v.r == before.out &&
           v.out == before.out;
}
/// One clause of a unit: state is where the unit has got to (0 at its
/// start), and the result where it gets with this clause, or 0 when the
/// clause must start a unit of its own.
enum : uint32_t { VS_FN = 1, VS_I, VS_ABS, VS_SIGN, VS_MUL, VS_J, VS_END };
__device__ __forceinline__ uint32_t val_next(uint32_t state, const ValClause& v)
{
    if (v.ai && v.bi) return state == 0 ? VS_END : 0;
    switch (v.op) {
        case op::SQRT:
        case op::EXP:
        case op::LOG: return state == 0 ? VS_FN : 0;
        case op::SUB:
            if (v.ai) return state == 0 ? VS_END : 0;
            return state < VS_I ? VS_I : state < VS_J ? VS_J : 0;
        case op::ADD: return state < VS_I ? VS_I : state < VS_J ? VS_J : 0;
        case op::ABS: return state < VS_ABS ? VS_ABS : 0;
        case op::NEG: return state < VS_SIGN ? VS_SIGN : state < VS_END ? VS_END : 0;
        case op::SQUARE:
        case op::MUL: return state < VS_MUL ? VS_MUL : 0;
        default: return state == 0 ? VS_END : 0;
    }
}
/// Clause c is the tail of a step: a two-register clause that reads the
/// one-register clause just before it.
__device__ __forceinline__ bool val_is_tail(const ValClause& v, const ValClause& before)
{
    const bool rr = v.valid && !v.one &&
                    (v.op == op::ADD || v.op == op::MUL || v.op == op::SUB || v.op == op::MIN ||
                     v.op == op::MAX);
    return rr && before.valid && before.one && ((v.a == before.out) != (v.b == before.out));
}
/// Clause c starts a step.
__device__ __forceinline__ bool val_is_head(const uint2* raw, int c)
{
    const ValClause v = val_clause(raw, c);
    if (!v.valid || val_is_tail(v, val_clause(raw, c - 1))) return false;
    // Walk the run of linked clauses that c is in from its start.
    int c0 = c;
    while (c0 > 0 && val_linked(val_clause(raw, c0), val_clause(raw, c0 - 1))) --c0;
    uint32_t state = 0;
    for (int k = c0; k < c; ++k) {
        const ValClause u = val_clause(raw, k);
        const uint32_t s = val_next(state, u);
        state = s ? s : val_next(0, u);
    }
    return state == 0 || val_next(state, v) == 0;
}

__device__ __forceinline__ uint32_t val_tail_of(uint32_t o, bool t_first)
{
    switch (o) {
        case op::ADD: return VF_TAIL;
        case op::MUL: return VF_TAIL | VF_MUL;
        case op::SUB: return VF_TAIL | (t_first ? VF_NEG_B : VF_NEG_T);
        case op::MIN: return VF_TAIL | VF_MM | (t_first ? 0 : VF_SWAP | VF_FLIP);
        case op::MAX: return VF_TAIL | VF_MM | (t_first ? VF_SWAP : VF_FLIP);
        default: return 0;
    }
}

/// The step whose first clause is c.
__device__ __forceinline__ ValOp val_step(const uint2* raw, int c, const float* __restrict__ cpool)
{
    ValClause v = val_clause(raw, c);
    const ValClause before = val_clause(raw, c - 1);
    uint32_t a = v.r, b = 0;
    bool reads_a = true, reads_b = false;
    ValOp s;
    s.flags = VF_PRE;
    s.i = s.j = 0.0f;
    s.m = 1.0f;
    s.andm = 0xffffffffu;
    s.xorm = 0;
    if (!v.one) {
        s.flags = val_tail_of(v.op, true);
        a = v.a;
        b = v.b;
        reads_b = true;
        if (!s.flags) {
            s.flags = VF_PRE | VF_RARE | v.op << VF_OP_SHIFT;
            s.xorm = RARE_RR;
        }
    } else if (v.ai && v.bi) {
        const bool bin = dev_is_binary(static_cast<uint8_t>(v.op));
        const float va = __ldg(cpool + v.a), vb = bin ? __ldg(cpool + v.b) : 0.0f;
        s.flags = VF_PRE | VF_RARE;
        if ((v.op == op::MIN || v.op == op::MAX) && va == vb) s.flags |= VF_TIE;
        reads_a = false;
        s.i = dv_value(static_cast<uint8_t>(v.op), va, vb);
        s.xorm = RARE_SET;
    } else {
        uint32_t state = 0;
        for (;;) {
            const float i = dev_is_binary(static_cast<uint8_t>(v.op))
                                ? __ldg(cpool + (v.ai ? v.a : v.b)) : 0.0f;
            const uint32_t to = val_next(state, v);
            const bool add = v.op == op::ADD || (v.op == op::SUB && !v.ai);
            if (to == VS_FN) {
                s.flags |= VF_FN | v.op << VF_OP_SHIFT;
            } else if (add && to == VS_I) {
                s.i = v.op == op::ADD ? -i : i;
            } else if (add) {
                s.j = v.op == op::ADD ? -i : i;
            } else if (to == VS_ABS) {
                s.andm = 0x7fffffffu;
            } else if (to == VS_SIGN) {
                s.xorm = 0x80000000u;
            } else if (v.op == op::NEG) {
                s.flags |= VF_NEG;
            } else if (v.op == op::SQUARE) {
                s.flags |= VF_SQ;
            } else if (v.op == op::MUL) {
                s.m = i;
            } else if (v.op == op::CONST_VAR || v.op == OP_COPY) {
                s.flags = 0;
            } else {
                s.flags |= VF_RARE | v.op << VF_OP_SHIFT;
                s.i = i;
                s.xorm = v.ai ? RARE_IR : RARE_RI;
            }
            state = to;
            const ValClause next = val_clause(raw, c + 1);
            if (!val_linked(next, v) || val_next(state, next) == 0) break;
            v = next;
            ++c;
        }
    }
    // v, at c, is the unit's last clause
    uint32_t out = v.out;
    const ValClause t = val_clause(raw, c + 1);
    if (!reads_b && val_is_tail(t, v)) {
        const bool first = t.a == v.out;
        s.flags |= val_tail_of(t.op, first);
        b = first ? t.b : t.a;
        reads_b = true;
        out = t.out;
    }
    s.a = static_cast<uint16_t>(reads_a ? a * kValRegBytes | (before.valid && before.out == a) : 0);
    s.b = static_cast<uint16_t>(reads_b ? b * kValRegBytes | (before.valid && before.out == b) : 0);
    s.o = static_cast<uint16_t>(out * kValRegBytes);
    s.o2 = static_cast<uint16_t>(v.out * kValRegBytes);
    return s;
}

/// Decodes clauses [c0, c0 + kLeafOps) of a tape into steps (the warp
/// together, two clauses a lane) at `out`; returns how many there are.  raw:
/// kValRaw words of shared memory.
__device__ __forceinline__ uint32_t val_decode(ValOp* out, uint2* raw,
                                               const RegClause* __restrict__ cl, uint32_t len,
                                               uint32_t c0, const float* __restrict__ cpool,
                                               int lane)
{
    const uint2 none = make_uint2(0xffffffffu, 0xffffffffu);
    const LeafRaw r = leaf_fetch(cl, len, c0, lane);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        raw[3 + lane + 32 * k] = c0 + lane + 32 * k < len ? r.w[k] : none;
    }
    if (lane < 3) {
        raw[lane] = none;
        raw[kLeafOps + 3 + lane] = none;
    }
    __syncwarp();
    uint32_t n = 0;
#pragma unroll 1
    for (uint32_t k = 0; k < kLeafOps && c0 + k < len; k += 32) {
        const int c = lane + k;
        const bool head = val_is_head(raw, c);
        const uint32_t m = __ballot_sync(0xffffffffu, head);
        if (head) out[n + __popc(m & ((1u << lane) - 1))] = val_step(raw, c, cpool);
        n += __popc(m);
    }
    return n;
}

/// The rare steps' t (VF_RARE), out of line.
static __device__ __noinline__ float4 val_rare(uint32_t o, uint32_t form, float i, float4 t,
                                               float4 b)
{
    const float4 i4 = splat4(i);
    if (form == RARE_SET) return i4;
    if (form == RARE_RI) b = i4;
    const bool swap = form == RARE_IR;
    const float4 p = swap ? i4 : t, q = swap ? t : b;
    const float pv[4] = {p.x, p.y, p.z, p.w}, qv[4] = {q.x, q.y, q.z, q.w};
    float r[4];
    dv_value4(static_cast<uint8_t>(o), pv, qv, r);
    return make_float4(r[0], r[1], r[2], r[3]);
}

/// Runs n decoded steps over four points per lane; R is the lane's float4 of
/// register 0.  With ties, bit k of amb is set when a min / max has equal
/// arguments at point k.  `last` carries the last step's result to the next
/// run of the same tape.
__device__ __forceinline__ void val_run(const ValOp* __restrict__ ops, uint32_t n,
                                        unsigned char* R, bool ties, uint32_t& amb,
                                        float (&last)[4])
{
    const uint4* w = reinterpret_cast<const uint4*>(ops);
    uint4 h = w[0], u = w[1];
    auto load = [&](uint32_t off, float (&v)[4]) {
        const float4 f = *reinterpret_cast<const float4*>(R + off);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    };
    auto store = [&](uint32_t off, const float (&v)[4]) {
        *reinterpret_cast<float4*>(R + off) = make_float4(v[0], v[1], v[2], v[3]);
    };
#pragma unroll 1
    for (uint32_t c = 0; c < n; ++c) {
        w += 2;   // the next step, one ahead (past the last: unused)
        const uint4 h1 = w[0], u1 = w[1];
        float t[4];
        if (h.x & 1) {
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = last[k];
        } else {
            load(h.x & 0xfe00, t);
        }
        const uint32_t b_off = h.x >> 16, fl = h.z;
        const uint32_t o = h.y & 0xffff, o2 = h.y >> 16;
        const float i = __uint_as_float(h.w);
        float b[4];
        if (fl & (VF_TAIL | VF_RARE)) {
            if (b_off & 1) {
#pragma unroll
                for (int k = 0; k < 4; ++k) b[k] = last[k];
            } else {
                load(b_off & 0xfe00, b);
            }
        }
        if (fl & VF_PRE) {
            if (fl & VF_RARE) {
                const uint32_t o_ = fl >> VF_OP_SHIFT;
                if (fl & VF_TIE) amb |= 15u;
                else if (ties && (o_ == op::MIN || o_ == op::MAX)) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) amb |= (t[k] == i ? 1u : 0u) << k;
                }
                const float4 r = val_rare(o_, u.y, i, make_float4(t[0], t[1], t[2], t[3]),
                                          make_float4(b[0], b[1], b[2], b[3]));
                t[0] = r.x; t[1] = r.y; t[2] = r.z; t[3] = r.w;
            } else {
                if (fl & VF_FN) {
                    if (fl >> VF_OP_SHIFT == op::SQRT) {
#pragma unroll
                        for (int k = 0; k < 4; ++k) t[k] = f_sqrt(t[k]);
                    } else {
                        const float4 r = val_rare(fl >> VF_OP_SHIFT, RARE_RI, 0.0f,
                                                  make_float4(t[0], t[1], t[2], t[3]),
                                                  make_float4(0.0f, 0.0f, 0.0f, 0.0f));
                        t[0] = r.x; t[1] = r.y; t[2] = r.z; t[3] = r.w;
                    }
                }
                const float m = __uint_as_float(u.z), j = __uint_as_float(u.w);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    t[k] = f_sub(t[k], i);
                    t[k] = __uint_as_float((__float_as_uint(t[k]) & u.x) ^ u.y);
                    t[k] = f_mul(t[k], fl & VF_SQ ? t[k] : m);
                    t[k] = f_sub(t[k], j);
                }
                if (fl & VF_NEG) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) t[k] = -t[k];
                }
            }
        }
        if (fl & VF_TAIL) {
            if (o2 != o) store(o2, t);
            if (fl & VF_MM) {
                const bool flip = fl & VF_FLIP;
                if (ties) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) amb |= (t[k] == b[k] ? 1u : 0u) << k;
                }
                if (fl & VF_SWAP) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) t[k] = ((t[k] < b[k]) != flip) ? b[k] : t[k];
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) t[k] = ((b[k] < t[k]) != flip) ? b[k] : t[k];
                }
            } else if (fl & VF_MUL) {
#pragma unroll
                for (int k = 0; k < 4; ++k) t[k] = f_mul(t[k], b[k]);
            } else {
                const uint32_t st = (fl & VF_NEG_T) << 22, sb = (fl & VF_NEG_B) << 21;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    t[k] = f_add(__uint_as_float(__float_as_uint(t[k]) ^ st),
                                 __uint_as_float(__float_as_uint(b[k]) ^ sb));
                }
            }
        }
        store(o, t);
#pragma unroll
        for (int k = 0; k < 4; ++k) last[k] = t[k];
        h = h1;
        u = u1;
    }
}

__device__ __forceinline__ D4 d4_of(const float4& f) { return {f.x, f.y, f.z, f.w}; }

/// The derivative interpreter's clause loop (one point per lane, value and
/// d/dx, d/dy, d/dz per register as a float4) with the tie settling of the
/// feature rules: see leaf_deriv in dc_kernels.cu.  `taint` holds one bit per
/// register (registers above 63 share bits and are reported as lost).
__device__ __forceinline__ void leaf_run_deriv(const LeafOp* __restrict__ ops, uint32_t n,
                                               float4* R, uint64_t& taint, bool& amb,
                                               bool& lost, bool trackable)
{
    float4 last = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    LeafOp L = ops[0];
#pragma unroll 1
    for (uint32_t c = 0; c < n; ++c) {
        const LeafOp next = ops[c + 1 < n ? c + 1 : c];
        D4 r;
        bool t_out;
        if (L.h == H_SET) {
            if (L.flags & 4) {
                amb = true;
                lost |= !trackable;
            }
            r = D4{L.imm, 0.0f, 0.0f, 0.0f};
            t_out = false;
        } else {
            const uint8_t o = L.op;
            const bool ai = L.flags & 1, bi = L.flags & 2;
            const bool binary = dev_is_binary(o);
            const D4 a = ai ? D4{L.imm, 0.0f, 0.0f, 0.0f}
                            : d4_of(L.flags & 8 ? last : R[L.a * 32]);
            const D4 b = bi ? D4{L.imm, 0.0f, 0.0f, 0.0f}
                            : binary ? d4_of(L.flags & 16 ? last : R[L.b * 32])
                                     : D4{0.0f, 0.0f, 0.0f, 0.0f};
            const bool ta = !ai && ((taint >> (L.a & 63)) & 1);
            const bool tbb = binary && !bi && ((taint >> (L.b & 63)) & 1);
            if ((o == op::MIN || o == op::MAX) && a.v == b.v) {
                amb = true;
                lost |= !trackable;
                const bool is_min = o == op::MIN;
                const float e[3] = {is_min ? b.dx - a.dx : a.dx - b.dx,
                                    is_min ? b.dy - a.dy : a.dy - b.dy,
                                    is_min ? b.dz - a.dz : a.dz - b.dz};
                const float nrm = sqrtf(fdot(e, e));
                bool take_b = false;
                t_out = ta || tbb;
                if (!t_out && nrm != 0) {
                    const float dd[3] = {b.dx - a.dx, b.dy - a.dy, b.dz - a.dz};
                    if (!(static_cast<double>(fdot(dd, dd)) < 1e-10)) {
                        t_out = true;
                    } else {
                        const float en[3] = {e[0] / nrm, e[1] / nrm, e[2] / nrm};
                        const float ep[3] = {-en[0], -en[1], -en[2]};
                        const float ad[3] = {a.dx, a.dy, a.dz}, bd[3] = {b.dx, b.dy, b.dz};
                        // Candidate order: b's feature carries -e, a's carries e.
                        const int cmp = vcmp3(ep, en);
                        take_b = cmp != 0 ? cmp < 0 : vcmp3(bd, ad) < 0;
                    }
                }
                r = take_b ? D4{dv_value(o, a.v, b.v), b.dx, b.dy, b.dz}
                           : D4{dv_value(o, a.v, b.v), a.dx, a.dy, a.dz};
            } else {
                r = dv_deriv(o, a, b, false);
                if (o == op::MIN) t_out = (a.v < b.v) ? ta : tbb;
                else if (o == op::MAX) t_out = (a.v < b.v) ? tbb : ta;
                else t_out = ta || tbb;
            }
        }
        if (t_out) taint |= 1ull << (L.o & 63);
        else taint &= ~(1ull << (L.o & 63));
        last = make_float4(r.v, r.dx, r.dy, r.dz);
        R[L.o * 32] = last;
        L = next;
    }
}

}  // namespace lfb
