// Breadth-first dual contouring on the GPU.
//
// The reference builds its octree depth-first with a CPU thread pool
// (WorkerPool::run, libfive/src/render/brep/worker_pool.inl:93-255) and walks
// the dual grid with another pool (Dual<3>::walk, dual.hpp:126-385).  Here
// every stage is a level-synchronous pass over compacted arrays:
//
//   1. k_interval_block / _wide / _group   (one of them per depth d < L)
//        DCTree::evalInterval (dc_tree.inl:94-128): interval-evaluate every
//        cell of depth d with the tape of its parent, classify it
//        EMPTY / FILLED / AMBIGUOUS, and prune the tape for its children
//        (Tape::push, tape.cpp:23-160) as a backward liveness pass over the
//        register tape; decided min/max clauses become register copies.
//   2. k_leaf_decode, k_leaf_groups, k_leaf_qef, k_edge_rank,
//      k_leaf_vertices    (depth L)
//        DCTree::evalLeaf (dc_tree.inl:131-552) for the eight children of
//        each ambiguous depth L-1 cell, one warp per sibling group: the 27
//        shared corners, the crossing edges of the 3x3x3 lattice (each
//        searched once), the QEFs and the per-patch vertices.
//   3. k_collapse_level   (depths L-1 .. 0)
//        DCTree::collectChildren (dc_tree.inl:581-735).
//   4. k_dual_round       (one round per depth, launched without waiting)
//        Dual<3>::work / face3 / edge3 as a breadth-first task expansion and
//        DCMesher::load (dc_mesher.cpp:18-169) at minimal edges.
//
// Every numeric decision uses the same float32 / float64 operations as the
// reference's scalar code, so the octree and the mesh are reproducible.
#include <cub/cub.cuh>
#include <sys/mman.h>
#include <type_traits>
#include <thread>
#include <cstddef>
#include <cstdlib>
#include <cstring>

#include "dc_device.cuh"
#include "dc_features.cuh"
#include "eval_kernels.cuh"
#include "interval_lists.cuh"
#include "leaf_interp.cuh"

namespace lfb {

__constant__ DcTables c_tab;

////////////////////////////////////////////////////////////////////////////////
// 1. Interval classification and tape pruning

// One warp per cell.  The tape a cell inherits is held twice: as a register
// tape (for point evaluation) and as a list of its clauses sorted by
// dependency level whose operands name list slots (WideEntry), so the lanes
// of a warp evaluate the independent clauses of one level at once.  The
// per-slot state of a list of up to kWideSmemSlots entries lives in shared
// memory, that of longer lists in a per-warp global scratch slice.

constexpr uint32_t kWideSmemSlots = 512;
constexpr uint32_t kRenumberMax = kWideSmemSlots;   // tapes up to this length get compact registers
constexpr uint32_t kGroupModeCells = 8192;          // cells per level from which k_interval_group runs
constexpr uint32_t kBlockModeCells = 2048;          // cells per level up to which k_interval_block runs

struct WideSmem {
    float2 S[kWideSmemSlots + 3];      // slot intervals
    uint32_t newpos[kWideSmemSlots];   // entry -> position in the child list
    uint32_t mask[(kMaxTapeRegs + 31) / 32];   // register bitmask (renumbering)
    uint16_t regmap[kMaxTapeRegs];     // old -> new register (renumbering)
    uint8_t SN[kWideSmemSlots + 3];    // slot maybe-NaN flags
    uint8_t pst[kWideSmemSlots];       // entry state for the children
    uint8_t live[kWideSmemSlots];      // entry still needed by the children
};

__device__ __forceinline__ Iv wide_fetch(uint32_t kind, uint32_t idx, float c, const float2* S,
                                         const uint8_t* SN)
{
    if (kind == OPND_REG) {
        const float2 v = S[idx];
        return {v.x, v.y, SN[idx] != 0};
    }
    return iv_make(c, c);
}

/// The values of a list entry's constant and free-variable operands, loaded
/// with the entry so that they are at hand when its level comes.
struct WideConsts {
    float a, b;
};
__device__ __forceinline__ WideConsts wide_consts(const uint4& e, const float* __restrict__ cp)
{
    const uint32_t kinds = (e.x >> 8) & 0xf;
    WideConsts c{0.0f, 0.0f};
    if ((kinds & 3) != OPND_REG) c.a = __ldg(cp + e.y);
    if ((kinds >> 2) != OPND_REG) c.b = __ldg(cp + e.z);
    return c;
}

/// Interval of list entry k, stored in slot 3 + k, and the entry's state for
/// the cell's children; returns whether a min/max got decided
/// (IntervalEvaluator::eval + push, eval_interval.cpp:116-167); ENCLOSING:
/// intervals enclose what the point interpreters compute, and nothing is
/// decided between operands that may be NaN.
template <bool ENCLOSING = false>
__device__ __forceinline__ bool wide_forward(const uint4& e, const WideConsts& c, uint32_t k,
                                             float2* S, uint8_t* SN, uint8_t* pst)
{
    const uint8_t o = e.x & 0xff;
    const uint32_t kinds = (e.x >> 8) & 0xf;
    const uint32_t st = (e.x >> 12) & 3;
    Iv r;
    uint8_t ps = static_cast<uint8_t>(st);
    bool decided = false;
    if (st == WIDE_A) {
        r = wide_fetch(kinds & 3, e.y, c.a, S, SN);
    } else if (st == WIDE_B) {
        r = wide_fetch((kinds >> 2) & 3, e.z, c.b, S, SN);
    } else {
        const Iv a = wide_fetch(kinds & 3, e.y, c.a, S, SN);
        const Iv b = dev_is_binary(o) ? wide_fetch((kinds >> 2) & 3, e.z, c.b, S, SN) : a;
        r = iv_eval<ENCLOSING>(o, a, b);
        if (o == op::MIN || o == op::MAX) {
            uint8_t keep = 0;   // 0 both, 1 a, 2 b
            if (a.lo > b.hi) keep = (o == op::MAX) ? 1 : 2;
            else if (b.lo > a.hi) keep = (o == op::MAX) ? 2 : 1;
            if (keep && !(ENCLOSING && (a.nan || b.nan))) {
                ps = keep == 1 ? WIDE_A : WIDE_B;
                decided = true;
            }
        }
    }
    S[3 + k] = make_float2(r.lo, r.hi);
    SN[3 + k] = r.nan;
    pst[k] = ps;
    return decided;
}

/// Marks the operands a live entry still needs (Tape::push's remapping,
/// tape.cpp:23-160, as liveness).
__device__ __forceinline__ void wide_mark(const uint4& e, uint8_t ps, uint8_t* live)
{
    const uint8_t o = e.x & 0xff;
    const uint32_t kinds = (e.x >> 8) & 0xf;
    if (ps != WIDE_B && (kinds & 3) == OPND_REG && e.y >= 3) live[e.y - 3] = 1;
    if (ps != WIDE_A && dev_is_binary(o) && ((kinds >> 2) & 3) == OPND_REG && e.z >= 3) {
        live[e.z - 3] = 1;
    }
}

/// Register clauses emitted for one 16-clause word of 2-bit states.
__device__ __forceinline__ uint32_t wide_word_emits(uint32_t word, uint32_t w,
                                                    const RegClause* root)
{
    uint32_t emit = 0;
    while (word) {
        const int j = (__ffs(word) - 1) >> 1;
        const uint32_t ps = (word >> (2 * j)) & 3;
        word &= ~(3u << (2 * j));
        if (ps == WIDE_BOTH) {
            ++emit;
            continue;
        }
        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(root + w * 16 + j));
        const uint32_t kinds = (raw.x >> 8) & 0xff;
        const uint32_t k = ps == WIDE_A ? (kinds & 3) : ((kinds >> 2) & 3);
        const uint32_t src = ps == WIDE_A ? (raw.y & 0xffff) : (raw.y >> 16);
        emit += !(k == OPND_REG && src == (raw.x >> 16));
    }
    return emit;
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v, int lane)
{
    for (int sh = 1; sh < 32; sh <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, v, sh);
        if (lane >= sh) v += t;
    }
    return v;
}

/// Linear-scan register allocation of a pruned tape, in place (one thread):
/// a backward pass marks each operand's last use, a forward pass gives every
/// result the lowest free register (X, Y and Z keep registers 0-2 while they
/// are still to be read).  On straight-line code this uses as many registers
/// as values are live at once, which is at most the unpruned tape's count;
/// the leaf kernel then fits the register file of most leaf tapes in shared
/// memory.  A copy (a decided min / max) whose source is not read again is
/// dropped: its result takes over the source's register.  Union-heavy models
/// leave one copy per decided level of their tree, a fifth to a third of a
/// deep tape.  Values are unchanged: only storage moves.
static __device__ __noinline__ TapeRef renumber_tape(uint2* raw_t, TapeRef tr,
                                                     uint8_t* lastuse,
                                                     uint16_t* regmap,
                                                     uint32_t* mask,
                                                     uint32_t* status)
{
    const uint32_t nm = (tr.nregs + 31) / 32;
    const uint32_t rk = tr.root >> 16, rr = tr.root & 0xffff;
    for (uint32_t w = 0; w < nm; ++w) mask[w] = 0;   // live-after bits
    if (rk == OPND_REG) mask[rr >> 5] |= 1u << (rr & 31);
    for (int64_t c = static_cast<int64_t>(tr.len) - 1; c >= 0; --c) {
        const uint2 raw = raw_t[c];
        const uint32_t o = raw.x >> 16, kinds = (raw.x >> 8) & 0xff;
        const uint32_t a = raw.y & 0xffff, b = raw.y >> 16;
        mask[o >> 5] &= ~(1u << (o & 31));
        uint8_t f = 0;
        if ((kinds & 3) == OPND_REG) {
            if (!(mask[a >> 5] & (1u << (a & 31)))) f |= 1;
            mask[a >> 5] |= 1u << (a & 31);
        }
        if (dev_is_binary(raw.x & 0xff) && ((kinds >> 2) & 3) == OPND_REG) {
            if (!(mask[b >> 5] & (1u << (b & 31)))) f |= 2;
            mask[b >> 5] |= 1u << (b & 31);
        }
        lastuse[c] = f;
    }
    // X, Y, Z start in registers 0-2; those not read by the tape are free.
    const uint32_t xyz_live = mask[0] & 7u;
    constexpr uint32_t kWords = (kMaxTapeRegs + 31) / 32;
    for (uint32_t w = 0; w < kWords; ++w) mask[w] = ~0u;   // free bits
    if (kMaxTapeRegs % 32) mask[kWords - 1] = (1u << (kMaxTapeRegs % 32)) - 1;
    mask[0] &= ~xyz_live;
    for (uint32_t r = 0; r < 3; ++r) regmap[r] = static_cast<uint16_t>(r);
    uint32_t hi = 3, kept = 0;
    for (uint32_t c = 0; c < tr.len; ++c) {
        uint2 raw = raw_t[c];
        const uint32_t o = raw.x >> 16, kinds = (raw.x >> 8) & 0xff;
        const bool binary = dev_is_binary(raw.x & 0xff);
        uint32_t a = raw.y & 0xffff, b = raw.y >> 16;
        const uint8_t f = lastuse[c];
        if ((raw.x & 0xff) == OP_COPY && (f & 1)) {
            regmap[o] = regmap[a];
            continue;
        }
        if ((kinds & 3) == OPND_REG) a = regmap[a];
        if (binary && ((kinds >> 2) & 3) == OPND_REG) b = regmap[b];
        if (f & 1) mask[a >> 5] |= 1u << (a & 31);
        if (f & 2) mask[b >> 5] |= 1u << (b & 31);
        uint32_t r = 0xffffffffu;
        for (uint32_t w = 0; w < kWords; ++w) {
            if (mask[w]) {
                r = w * 32 + __ffs(mask[w]) - 1;
                break;
            }
        }
        if (r >= kMaxTapeRegs) {   // more live values than registers: cannot happen
            atomicOr(status, ST_REGS);
            return tr;
        }
        mask[r >> 5] &= ~(1u << (r & 31));
        regmap[o] = static_cast<uint16_t>(r);
        hi = max(hi, r + 1);
        raw.x = (raw.x & 0xffffu) | (r << 16);
        raw.y = a | (b << 16);
        raw_t[kept++] = raw;
    }
    const uint32_t root = rk == OPND_REG ? regmap[rr] : rr;
    return {tr.off, kept, hi, root | (rk << 16)};
}

__global__ void __launch_bounds__(256)
k_interval_wide(WideArgs A, int d)
{
    extern __shared__ __align__(16) unsigned char wsm[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t gw = blockIdx.x * (blockDim.x >> 5) + warp;
    WideSmem* SM = reinterpret_cast<WideSmem*>(wsm) + warp;
    const Octree& o = A.o;
    const LevelView& lv = o.lv[d];
    const DevTape& bt = A.bt;
    const uint32_t n = A.n;
    const uint32_t nw = (n + 15) / 16;
    const uint32_t nw1 = (nw + 31) / 32;
    float2* gS = A.S + static_cast<size_t>(gw) * (n + 3);
    uint8_t* gSN = A.SN + static_cast<size_t>(gw) * (n + 3);
    uint8_t* gP = A.pst + static_cast<size_t>(gw) * n;
    uint8_t* gL = A.live + static_cast<size_t>(gw) * n;
    uint32_t* gN = A.newpos + static_cast<size_t>(gw) * n;
    uint32_t* st2 = A.st2 + static_cast<size_t>(gw) * nw;
    uint32_t* l1 = A.l1 + static_cast<size_t>(gw) * nw1;
    uint32_t* wl = A.wl + static_cast<size_t>(gw) * nw;
    const unsigned full = 0xffffffffu;
    const uint32_t lt_mask = (1u << lane) - 1;

    while (true) {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(A.next_cell, 1u);
        i = __shfl_sync(full, i, 0);
        if (i >= lv.n_cells) break;
        ListRef P;
        TapeRef T;
        if (d == 0) {
            P = A.root_list;
            T = root_tape_ref(bt);
        } else {
            P = lv.group_list[i >> A.group_shift];
            T = lv.group_tape[i >> A.group_shift];
        }
        const uint4* PL = reinterpret_cast<const uint4*>(A.in_lists + P.off);
        const bool small = P.len <= kWideSmemSlots;
        float2* S = small ? SM->S : gS;
        uint8_t* SN = small ? SM->SN : gSN;
        uint8_t* pst = small ? SM->pst : gP;
        uint8_t* live = small ? SM->live : gL;
        uint32_t* newpos = small ? SM->newpos : gN;
        if (lane < 3) {
            double blo[3], bhi[3];
            cell_bounds(o, d, lv.coords[i], blo, bhi);
            const Iv v = iv_make(static_cast<float>(blo[lane]), static_cast<float>(bhi[lane]));
            S[lane] = make_float2(v.lo, v.hi);
            SN[lane] = v.nan;
        }
        for (uint32_t k = lane; k < P.len; k += 32) live[k] = 0;
        __syncwarp();

        // Forward pass, level by level (entries are sorted by level, so a
        // chunk of 32 spans few levels; the warp steps through them).
        const uint32_t nchunks = (P.len + 31) / 32;
        bool changed = false;
        for (uint32_t ch = 0; ch < nchunks; ++ch) {
            const uint32_t k = ch * 32 + lane;
            const bool valid = k < P.len;
            const uint4 e = valid ? PL[k] : make_uint4(0, 0, 0, 0);
            const WideConsts c = wide_consts(e, bt.cpool);
            const uint32_t lev = valid ? (e.x >> kWideLevelShift) : 0xffffffffu;
            const int last = static_cast<int>(min(31u, P.len - 1 - ch * 32));
            uint32_t l = __shfl_sync(full, lev, 0);
            const uint32_t lmax = __shfl_sync(full, lev, last);
            while (true) {
                if (lev == l) changed |= wide_forward(e, c, k, S, SN, pst);
                __syncwarp();
                if (l == lmax) break;
                const uint32_t m = __ballot_sync(full, valid && lev > l);
                l = __shfl_sync(full, lev, __ffs(m) - 1);
            }
        }
        changed = __any_sync(full, changed);
        const float root_c = bt.root_kind == OPND_REG ? 0.0f : __ldg(bt.cpool + P.root);
        const Iv root = wide_fetch(bt.root_kind, P.root, root_c, S, SN);
        const uint8_t state = iv_state(root);
        if (lane == 0) {
            lv.type[i] = state == ST_EMPTY ? CELL_EMPTY
                       : state == ST_FILLED ? CELL_FILLED : CELL_BRANCH;
        }
        if (state != ST_AMBIGUOUS) continue;

        if (root.nan || !changed) {
            // NaN-unsafe or nothing decided: the children keep this tape
            // (dc_tree.inl:107-111).  Its list moves to the next arena.
            uint32_t off = 0;
            if (A.write_lists) {
                unsigned long long o64 = 0;
                if (lane == 0) o64 = atomicAdd(A.out_top, static_cast<unsigned long long>(P.len));
                o64 = __shfl_sync(full, o64, 0);
                if (o64 + P.len <= A.out_cap) {
                    off = static_cast<uint32_t>(o64);
                    uint4* out = reinterpret_cast<uint4*>(A.out_lists + off);
                    for (uint32_t k = lane; k < P.len; k += 32) out[k] = PL[k];
                } else if (lane == 0) {
                    atomicOr(A.status, ST_LIST_OVERFLOW);
                }
            }
            if (lane == 0) {
                lv.cell_list[i] = {off, P.len, P.root, 0u};
                lv.cell_tape[i] = T;
            }
            continue;
        }

        // Backward liveness pass, levels in decreasing order.
        if (lane == 0 && bt.root_kind == OPND_REG && P.root >= 3) live[P.root - 3] = 1;
        __syncwarp();
        for (int ch = static_cast<int>(nchunks) - 1; ch >= 0; --ch) {
            const uint32_t k = ch * 32 + lane;
            const bool valid = k < P.len;
            const uint4 e = valid ? PL[k] : make_uint4(0, 0, 0, 0);
            const uint32_t lev = valid ? (e.x >> kWideLevelShift) : 0u;
            const int last = static_cast<int>(min(31u, P.len - 1 - ch * 32));
            const uint32_t lmin = __shfl_sync(full, lev, 0);
            uint32_t l = __shfl_sync(full, lev, last);
            while (true) {
                if (valid && lev == l && live[k]) wide_mark(e, pst[k], live);
                __syncwarp();
                if (l == lmin) break;
                const uint32_t m = __ballot_sync(full, valid && lev < l);
                l = __shfl_sync(full, lev, 31 - __clz(m));
            }
        }

        // Child positions of the live entries, and their 2-bit states by
        // clause index (for the register tape, which is in clause order).
        uint32_t cnt = 0;
        for (uint32_t ch = 0; ch < nchunks; ++ch) {
            const uint32_t k = ch * 32 + lane;
            const bool lv_ = k < P.len && live[k];
            const uint32_t m = __ballot_sync(full, lv_);
            if (lv_) {
                newpos[k] = cnt + __popc(m & lt_mask);
                const uint32_t c = PL[k].w;
                atomicOr(st2 + (c >> 4), static_cast<uint32_t>(pst[k]) << (2 * (c & 15)));
                atomicOr(l1 + (c >> 9), 1u << ((c >> 4) & 31));
            }
            cnt += __popc(m);
        }
        __syncwarp();
        const uint32_t new_root = (bt.root_kind == OPND_REG && P.root >= 3)
                                      ? newpos[P.root - 3] + 3 : P.root;
        uint32_t loff = 0;
        if (A.write_lists) {
            unsigned long long o64 = 0;
            if (lane == 0) o64 = atomicAdd(A.out_top, static_cast<unsigned long long>(cnt));
            o64 = __shfl_sync(full, o64, 0);
            const bool ok = o64 + cnt <= A.out_cap;
            if (!ok && lane == 0) atomicOr(A.status, ST_LIST_OVERFLOW);
            if (ok) {
                loff = static_cast<uint32_t>(o64);
                uint4* out = reinterpret_cast<uint4*>(A.out_lists + loff);
                for (uint32_t k = lane; k < P.len; k += 32) {
                    if (!live[k]) continue;
                    uint4 e = PL[k];
                    const uint32_t ps = pst[k];
                    const uint32_t kinds = (e.x >> 8) & 0xf;
                    const bool binary = dev_is_binary(e.x & 0xff);
                    if (ps == WIDE_B) e.y = 0;
                    else if ((kinds & 3) == OPND_REG && e.y >= 3) e.y = newpos[e.y - 3] + 3;
                    if (ps == WIDE_A) e.z = 0;
                    else if (binary && ((kinds >> 2) & 3) == OPND_REG && e.z >= 3) {
                        e.z = newpos[e.z - 3] + 3;
                    }
                    e.x = (e.x & ~(3u << 12)) | (ps << 12);
                    out[newpos[k]] = e;
                }
            }
        }

        // Register tape for this cell: the live clauses in clause order, with
        // decided min/max clauses as copies (dropped when the copy is onto
        // the same register).  First the non-zero state words, in order.
        uint32_t nwl = 0;
        for (uint32_t j0 = 0; j0 < nw1; j0 += 32) {
            const uint32_t j = j0 + lane;
            uint32_t bits = 0;
            if (j < nw1) {
                bits = l1[j];
                l1[j] = 0;
            }
            const uint32_t c_ = __popc(bits);
            const uint32_t incl = warp_incl_scan(c_, lane);
            uint32_t at = nwl + incl - c_;
            while (bits) {
                const int b = __ffs(bits) - 1;
                bits &= bits - 1;
                wl[at++] = j * 32 + b;
            }
            nwl += __shfl_sync(full, incl, 31);
        }
        __syncwarp();
        uint32_t emit = 0;
        for (uint32_t k0 = 0; k0 < nwl; k0 += 32) {
            const uint32_t k = k0 + lane;
            uint32_t e_ = 0;
            if (k < nwl) {
                const uint32_t w = wl[k];
                e_ = wide_word_emits(st2[w], w, bt.clauses);
            }
            emit += __reduce_add_sync(full, e_);
        }
        unsigned long long a64 = 0;
        if (lane == 0) a64 = atomicAdd(A.arena_top, static_cast<unsigned long long>(emit));
        a64 = __shfl_sync(full, a64, 0);
        const bool aok = a64 + emit <= A.arena_cap;
        if (!aok && lane == 0) atomicOr(A.status, ST_ARENA_OVERFLOW);
        uint32_t pos = static_cast<uint32_t>(a64);
        for (uint32_t k0 = 0; k0 < nwl; k0 += 32) {
            const uint32_t k = k0 + lane;
            uint32_t word = 0, w = 0, e_ = 0;
            if (k < nwl) {
                w = wl[k];
                word = st2[w];
                e_ = wide_word_emits(word, w, bt.clauses);
                st2[w] = 0;
            }
            const uint32_t incl = warp_incl_scan(e_, lane);
            uint32_t at = pos + incl - e_;
            if (aok) {
                while (word) {
                    const int j = (__ffs(word) - 1) >> 1;
                    const uint32_t ps = (word >> (2 * j)) & 3;
                    word &= ~(3u << (2 * j));
                    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(bt.clauses + w * 16 + j));
                    if (ps == WIDE_BOTH) {
                        *reinterpret_cast<uint2*>(A.arena + at++) = raw;
                        continue;
                    }
                    const uint32_t kinds = (raw.x >> 8) & 0xff;
                    const uint32_t kk = ps == WIDE_A ? (kinds & 3) : ((kinds >> 2) & 3);
                    const uint32_t src = ps == WIDE_A ? (raw.y & 0xffff) : (raw.y >> 16);
                    const uint32_t ro = raw.x >> 16;
                    if (kk == OPND_REG && src == ro) continue;
                    RegClause cc;
                    cc.op = OP_COPY;
                    cc.kinds = static_cast<uint8_t>(kk);
                    cc.out = static_cast<uint16_t>(ro);
                    cc.a = static_cast<uint16_t>(src);
                    cc.b = 0;
                    A.arena[at++] = cc;
                }
            }
            pos += __shfl_sync(full, incl, 31);
        }
        __syncwarp();
        TapeRef out_t = T;
        if (aok) {
            out_t = {static_cast<uint32_t>(a64), emit, bt.n_regs,
                     static_cast<uint32_t>(bt.root) | (static_cast<uint32_t>(bt.root_kind) << 16)};
            if (emit <= kRenumberMax) {
                // Short tapes get compact registers: staged through the
                // warp's shared slot area (free again at this point).
                uint2* buf = reinterpret_cast<uint2*>(SM->S);
                uint2* dst = reinterpret_cast<uint2*>(A.arena + a64);
                for (uint32_t k = lane; k < emit; k += 32) buf[k] = dst[k];
                __syncwarp();
                if (lane == 0) {
                    out_t = renumber_tape(buf, out_t, SM->live, SM->regmap, SM->mask, A.status);
                }
                __syncwarp();
                out_t.len = __shfl_sync(full, out_t.len, 0);
                for (uint32_t k = lane; k < out_t.len; k += 32) dst[k] = buf[k];
                out_t.nregs = __shfl_sync(full, out_t.nregs, 0);
                out_t.root = __shfl_sync(full, out_t.root, 0);
            }
        }
        if (lane == 0) {
            lv.cell_list[i] = {loff, cnt, new_root, 0u};
            lv.cell_tape[i] = out_t;
        }
        __syncwarp();
    }
}

// Top levels: one block per cell.  The first levels have few cells with
// long lists (the unpruned tape at depth 0), so all warps of a block work on
// one cell: a wave of kBlockThreads consecutive entries at a time, stepping
// through the levels the wave spans with a block barrier per level.  Same
// results as k_interval_wide (lists, register tapes); tapes are not
// renumbered (one thread renumbering 100 clauses took 40 us, longer than the
// rest of a cell).

constexpr int kBlockThreads = 512;
constexpr int kBlockWarps = kBlockThreads / 32;

/// Exclusive prefix over the block's warps of one count per warp, and the
/// total.
__device__ __forceinline__ uint32_t warp_counts_scan(uint32_t count, uint32_t* warp_tot,
                                                     uint32_t& total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) warp_tot[warp] = count;
    __syncthreads();
    const uint32_t v = lane < kBlockWarps ? warp_tot[lane] : 0;
    const uint32_t incl = warp_incl_scan(v, lane);
    total = __shfl_sync(0xffffffffu, incl, 31);
    return __shfl_sync(0xffffffffu, incl - v, warp);
}

/// boxes: the box form (WideArgs::boxes) is an instance of its own, so that
/// the levels' form carries nothing of it.  per_sm: blocks that share an SM;
/// where a list's state leaves room for one only, that one has 128 registers
/// a thread instead of 64, which spill in the box form (derivatives of a
/// 1,500-primitive CSG at 100,003 points 2.10 -> 1.92 ms, of a union of 1,200
/// spheres 3.01 -> 2.66 ms).
template <bool boxes, int per_sm>
__global__ void __launch_bounds__(kBlockThreads, per_sm)
k_interval_block(const __grid_constant__ WideArgs A, int d, uint32_t smem_slots)
{
    extern __shared__ __align__(16) unsigned char bsm[];
    __shared__ uint32_t lev_of[2][2];   // levels of a wave's first and last entry
    __shared__ uint32_t warp_tot[kBlockWarps];
    __shared__ unsigned long long bcast;
    __shared__ uint32_t cell;
    const int tid = threadIdx.x;
    const Octree& o = A.o;
    const LevelView& lv = o.lv[d];
    const DevTape& bt = A.bt;
    const uint32_t n_cells = boxes ? A.n_boxes : lv.n_cells;
    const uint32_t n = A.n;
    const size_t slot = blockIdx.x;

    while (true) {
        if (tid == 0) cell = atomicAdd(A.next_cell, 1u);
        __syncthreads();
        const uint32_t i = cell;
        __syncthreads();
        if (i >= n_cells) break;
        ListRef P;
        TapeRef T;
        if (boxes || d == 0) {
            P = A.root_list;
            T = root_tape_ref(bt);
        } else {
            P = lv.group_list[i >> A.group_shift];
            T = lv.group_tape[i >> A.group_shift];
        }
        const uint4* PL = reinterpret_cast<const uint4*>(A.in_lists + P.off);
        auto work = [&](auto in_smem) {
        constexpr bool SM = decltype(in_smem)::value;
        float2* S;
        uint8_t *SN, *pst, *live, *cstate;
        uint32_t* newpos;
        if constexpr (SM) {
            S = reinterpret_cast<float2*>(bsm);
            newpos = reinterpret_cast<uint32_t*>(bsm);   // once S has served
            cstate = bsm + 4 * smem_slots;
            SN = bsm + 8 * (smem_slots + 3);
            pst = SN + smem_slots + 3;
            live = pst + smem_slots;
        } else {
            S = A.S + slot * (n + 3);
            SN = A.SN + slot * (n + 3);
            pst = A.pst + slot * n;
            live = A.live + slot * n;
            newpos = A.newpos + slot * n;
            cstate = reinterpret_cast<uint8_t*>(S);
        }
        // The wave's entry of this thread, fetched while the wave before it
        // is at work, with its constants and (by the wave's first and last
        // entries) the levels that the wave spans.
        const uint32_t nwaves = (P.len + kBlockThreads - 1) / kBlockThreads;
        auto fetch = [&](uint32_t w, uint4& e) {
            const uint32_t k = w * kBlockThreads + tid;
            if (w >= nwaves || k >= P.len) return;
            e = __ldg(PL + k);
            if (tid == 0) lev_of[w & 1][0] = e.x >> kWideLevelShift;
            if (k + 1 == P.len || tid == kBlockThreads - 1) lev_of[w & 1][1] = e.x >> kWideLevelShift;
        };
        uint4 e{}, e_next{};
        fetch(0, e);
        if (tid < 3) {
            Iv v;
            if (boxes) {
                v = iv_not_empty(iv_make(A.boxes[6 * i + 2 * tid], A.boxes[6 * i + 2 * tid + 1]));
            } else {
                double blo[3], bhi[3];
                cell_bounds(o, d, lv.coords[i], blo, bhi);
                v = iv_make(static_cast<float>(blo[tid]), static_cast<float>(bhi[tid]));
            }
            S[tid] = make_float2(v.lo, v.hi);
            SN[tid] = v.nan;
        }
        for (uint32_t k = tid; k < P.len; k += kBlockThreads) live[k] = 0;
        __syncthreads();

        // Forward pass: waves of consecutive entries, levels in order.
        bool changed = false;
        WideConsts c = wide_consts(e, bt.cpool), c_next{};
        for (uint32_t w = 0; w < nwaves; ++w) {
            const uint32_t k = w * kBlockThreads + tid;
            const uint32_t lf = lev_of[w & 1][0], ll = lev_of[w & 1][1];
            const uint32_t lev = k < P.len ? (e.x >> kWideLevelShift) : 0xffffffffu;
            e_next = make_uint4(0, 0, 0, 0);
            fetch(w + 1, e_next);
            c_next = wide_consts(e_next, bt.cpool);
            for (uint32_t l = lf; l <= ll; ++l) {
                if (lev == l) changed |= wide_forward<boxes>(e, c, k, S, SN, pst);
                __syncthreads();
            }
            e = e_next;
            c = c_next;
        }
        changed = __syncthreads_or(changed) != 0;
        const float root_c = bt.root_kind == OPND_REG ? 0.0f : __ldg(bt.cpool + P.root);
        const Iv root = wide_fetch(bt.root_kind, P.root, root_c, S, SN);
        const uint8_t state = iv_state(root);
        if (tid == 0 && !boxes) {
            lv.type[i] = state == ST_EMPTY ? CELL_EMPTY
                       : state == ST_FILLED ? CELL_FILLED : CELL_BRANCH;
        }
        if (!boxes && state != ST_AMBIGUOUS) return;
        if (boxes && !changed) {
            if (tid == 0) A.box_tape[i] = T;
            return;
        }

        if (!boxes && (root.nan || !changed)) {
            // The children keep this tape; its list moves to the next arena.
            uint32_t off = 0;
            if (A.write_lists) {
                if (tid == 0) bcast = atomicAdd(A.out_top, static_cast<unsigned long long>(P.len));
                __syncthreads();
                const unsigned long long o64 = bcast;
                __syncthreads();
                if (o64 + P.len <= A.out_cap) {
                    off = static_cast<uint32_t>(o64);
                    uint4* out = reinterpret_cast<uint4*>(A.out_lists + off);
                    for (uint32_t k = tid; k < P.len; k += kBlockThreads) out[k] = PL[k];
                } else if (tid == 0) {
                    atomicOr(A.status, ST_LIST_OVERFLOW);
                }
            }
            if (tid == 0) {
                lv.cell_list[i] = {off, P.len, P.root, 0u};
                lv.cell_tape[i] = T;
            }
            return;
        }

        // Backward liveness pass: waves in reverse, levels decreasing.
        if (tid == 0 && bt.root_kind == OPND_REG && P.root >= 3) live[P.root - 3] = 1;
        fetch(nwaves - 1, e);
        __syncthreads();
        for (uint32_t w = nwaves; w-- > 0;) {
            const uint32_t k = w * kBlockThreads + tid;
            const uint32_t lf = lev_of[w & 1][0], ll = lev_of[w & 1][1];
            const bool valid = k < P.len;
            const uint32_t lev = valid ? (e.x >> kWideLevelShift) : 0xffffffffu;
            fetch(w - 1, e_next);   // wave -1 is past the last: nothing
            for (uint32_t l = ll + 1; l-- > lf;) {
                if (lev == l && live[k]) wide_mark(e, pst[k], live);
                __syncthreads();
            }
            e = e_next;
        }

        // Child positions of the live entries and, by clause, their states
        // (for the register tape, which is in clause order).  Each warp takes
        // a contiguous share of the entries: one block scan for all.
        for (uint32_t k = tid; k < (n + 3) / 4; k += kBlockThreads) {
            reinterpret_cast<uint32_t*>(cstate)[k] = 0;
        }
        const unsigned full = 0xffffffffu;
        const int lane = tid & 31, warp = tid >> 5;
        const uint32_t lt_mask = (1u << lane) - 1;
        const uint32_t share = (P.len + 32 * kBlockWarps - 1) / (32 * kBlockWarps) * 32;
        const uint32_t k_end = min(P.len, share * (warp + 1));
        uint32_t here = 0, cnt = 0;
        for (uint32_t k0 = share * warp; k0 < k_end; k0 += 32) {
            here += __popc(__ballot_sync(full, k0 + lane < k_end && live[k0 + lane]));
        }
        uint32_t at = warp_counts_scan(here, warp_tot, cnt);
        for (uint32_t k0 = share * warp; k0 < k_end; k0 += 32) {
            const uint32_t k = k0 + lane;
            const bool lv_ = k < k_end && live[k];
            const uint32_t m = __ballot_sync(full, lv_);
            if (lv_) {
                newpos[k] = at + __popc(m & lt_mask);
                cstate[__ldg(&PL[k].w)] = pst[k];
            }
            at += __popc(m);
        }
        if (tid == 0 && A.write_lists) bcast = atomicAdd(A.out_top, static_cast<unsigned long long>(cnt));
        __syncthreads();
        const uint32_t new_root = (bt.root_kind == OPND_REG && P.root >= 3)
                                      ? newpos[P.root - 3] + 3 : P.root;
        uint32_t loff = 0;
        if (A.write_lists) {
            const unsigned long long o64 = bcast;
            const bool ok = o64 + cnt <= A.out_cap;
            if (!ok && tid == 0) atomicOr(A.status, ST_LIST_OVERFLOW);
            if (ok) {
                loff = static_cast<uint32_t>(o64);
                uint4* out = reinterpret_cast<uint4*>(A.out_lists + loff);
#pragma unroll 2
                for (uint32_t k = tid; k < P.len; k += kBlockThreads) {
                    uint4 e = __ldg(PL + k);
                    if (!live[k]) continue;
                    const uint32_t ps = pst[k];
                    const uint32_t kinds = (e.x >> 8) & 0xf;
                    const bool binary = dev_is_binary(e.x & 0xff);
                    if (ps == WIDE_B) e.y = 0;
                    else if ((kinds & 3) == OPND_REG && e.y >= 3) e.y = newpos[e.y - 3] + 3;
                    if (ps == WIDE_A) e.z = 0;
                    else if (binary && ((kinds >> 2) & 3) == OPND_REG && e.z >= 3) {
                        e.z = newpos[e.z - 3] + 3;
                    }
                    e.x = (e.x & ~(3u << 12)) | (ps << 12);
                    out[newpos[k]] = e;
                }
            }
        }

        // Register tape: live clauses in clause order, a contiguous share of
        // the unpruned tape's clauses a warp.  A decided min / max is a copy,
        // dropped when it is onto the same register.
        const uint32_t cshare = (n + 32 * kBlockWarps - 1) / (32 * kBlockWarps) * 32;
        const uint32_t c_end = min(n, cshare * (warp + 1));
        auto clause_of = [&](uint32_t c, uint2& raw) -> bool {
            const uint32_t ps = c < c_end ? cstate[c] : 0;
            if (ps == 0) return false;
            raw = __ldg(reinterpret_cast<const uint2*>(bt.clauses + c));
            if (ps == WIDE_BOTH) return true;
            const uint32_t kinds = (raw.x >> 8) & 0xff;
            const uint32_t kk = ps == WIDE_A ? (kinds & 3) : ((kinds >> 2) & 3);
            const uint32_t src = ps == WIDE_A ? (raw.y & 0xffff) : (raw.y >> 16);
            const uint32_t ro = raw.x >> 16;
            raw = make_uint2(OP_COPY | (kk << 8) | (ro << 16), src);
            return !(kk == OPND_REG && src == ro);
        };
        uint32_t emit = 0, etot = 0;
#pragma unroll 4
        for (uint32_t c0 = cshare * warp; c0 < c_end; c0 += 32) {
            uint2 raw;
            emit += __popc(__ballot_sync(full, clause_of(c0 + lane, raw)));
        }
        uint32_t pos = warp_counts_scan(emit, warp_tot, etot);
        if (tid == 0) bcast = atomicAdd(A.arena_top, static_cast<unsigned long long>(etot));
        __syncthreads();
        const unsigned long long a64 = bcast + A.arena_base;
        const bool aok = a64 + etot <= A.arena_cap;
        if (!aok && tid == 0) atomicOr(A.status, ST_ARENA_OVERFLOW);
        uint2* to = reinterpret_cast<uint2*>(A.arena + a64);
        for (uint32_t c0 = cshare * warp; aok && c0 < c_end; c0 += 32) {
            uint2 raw;
            const bool emits = clause_of(c0 + lane, raw);
            const uint32_t m = __ballot_sync(full, emits);
            if (emits) to[pos + __popc(m & lt_mask)] = raw;
            pos += __popc(m);
        }
        TapeRef out_t = T;
        if (aok) {
            out_t = {static_cast<uint32_t>(a64), etot, bt.n_regs,
                     static_cast<uint32_t>(bt.root) | (static_cast<uint32_t>(bt.root_kind) << 16)};
        }
        if (tid == 0 && boxes) {
            A.box_tape[i] = out_t;
        } else if (tid == 0) {
            lv.cell_list[i] = {loff, cnt, new_root, 0u};
            lv.cell_tape[i] = out_t;
        }
        };
        if (P.len <= smem_slots && n <= 4 * smem_slots) work(std::true_type{});
        else work(std::false_type{});
        __syncthreads();
    }
}

// Deep levels: one warp per sibling group, one lane per cell.  The eight
// cells share their parent's register tape, so lanes 0-7 walk the same
// clause stream (no divergence) with the interval register file in shared
// memory, as IntervalEvaluator does, and prune with a backward liveness pass
// over registers (Tape::push, tape.cpp:23-160).  Used once cells are many
// and tapes short, where the per-cell overheads of the level-ordered form
// dominate; it writes register tapes only.

struct GroupArgs {
    Octree o;
    DevTape bt;
    RegClause* arena;
    unsigned long long* arena_top;
    uint64_t arena_cap;
    uint8_t* dec;                  // [warps][8][dec_cap] min/max decisions
    uint32_t dec_cap;
    uint8_t* lastuse;              // [warps][8][kRenumberMax] renumbering flags
    uint32_t nregs_max;            // register file size (this depth's largest group tape)
    uint32_t* status;
    uint32_t* next_group;          // work counter (zero at launch)
};

__host__ __device__ inline size_t group_smem_per_warp(uint32_t nregs_max)
{
    // L, H (float), regmap (u16) per register and lane; masks; N (u8).
    const size_t b = static_cast<size_t>(nregs_max) * 8 * (4 + 4 + 2) + 8 * 13 * 4 +
                     static_cast<size_t>(nregs_max) * 8;
    return (b + 15) / 16 * 16;
}

__global__ void __launch_bounds__(128)
k_interval_group(GroupArgs A, int d)
{
    extern __shared__ __align__(16) unsigned char gsm[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const uint32_t nr = A.nregs_max;
    unsigned char* base = gsm + group_smem_per_warp(nr) * warp;
    float* Lo = reinterpret_cast<float*>(base);
    float* Hi = Lo + nr * 8;
    uint16_t* RM = reinterpret_cast<uint16_t*>(Hi + nr * 8) + lane * nr;
    uint32_t* MK = reinterpret_cast<uint32_t*>(reinterpret_cast<uint16_t*>(Hi + nr * 8) + nr * 8) +
                   lane * 13;
    uint8_t* Nn = reinterpret_cast<uint8_t*>(reinterpret_cast<uint32_t*>(
                      reinterpret_cast<uint16_t*>(Hi + nr * 8) + nr * 8) + 8 * 13);
    const uint32_t gw = blockIdx.x * wpb + warp;
    uint8_t* dec = A.dec + (static_cast<size_t>(gw) * 8 + (lane & 7)) * A.dec_cap;
    uint8_t* lastuse = A.lastuse + (static_cast<size_t>(gw) * 8 + (lane & 7)) * kRenumberMax;
    const Octree& o = A.o;
    const LevelView& lv = o.lv[d];
    const DevTape& bt = A.bt;
    auto fetch = [&](uint32_t kind, uint32_t idx) -> Iv {
        if (kind == OPND_REG) return {Lo[idx * 8 + lane], Hi[idx * 8 + lane], Nn[idx * 8 + lane] != 0};
        const float v = __ldg(bt.cpool + idx);
        return iv_make(v, v);
    };

    while (true) {
        uint32_t g = 0;
        if (lane == 0) g = atomicAdd(A.next_group, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= lv.n_groups) break;
        if (lane >= 8) continue;
        const uint32_t i = 8 * g + lane;
        const TapeRef T = lv.group_tape[g];
        const RegClause* cl = A.arena + T.off;
        const uint32_t rk = T.root >> 16, rr = T.root & 0xffff;

        double blo[3], bhi[3];
        cell_bounds(o, d, lv.coords[i], blo, bhi);
        for (int a = 0; a < 3; ++a) {
            const Iv v = iv_make(static_cast<float>(blo[a]), static_cast<float>(bhi[a]));
            Lo[a * 8 + lane] = v.lo;
            Hi[a * 8 + lane] = v.hi;
            Nn[a * 8 + lane] = v.nan;
        }
        // Forward pass, recording the push decision of every min/max
        // (IntervalEvaluator::push, eval_interval.cpp:116-167).
        bool changed = false;
        uint32_t ch = 0;
        for (uint32_t c = 0; c < T.len; ++c) {
            const uint2 raw = __ldg(reinterpret_cast<const uint2*>(cl + c));
            const uint8_t o_ = raw.x & 0xff;
            const uint32_t kinds = (raw.x >> 8) & 0xff;
            const uint32_t ro = raw.x >> 16;
            const Iv a = fetch(kinds & 3, raw.y & 0xffff);
            const Iv b = fetch((kinds >> 2) & 3, raw.y >> 16);
            const Iv r = iv_eval(o_, a, b);
            if (o_ == op::MIN || o_ == op::MAX) {
                uint8_t keep = 0;   // 0 both, 1 a, 2 b
                if (a.lo > b.hi) keep = (o_ == op::MAX) ? 1 : 2;
                else if (b.lo > a.hi) keep = (o_ == op::MAX) ? 2 : 1;
                changed |= keep != 0;
                if (ch < A.dec_cap) dec[ch] = keep;
                ++ch;
            }
            Lo[ro * 8 + lane] = r.lo;
            Hi[ro * 8 + lane] = r.hi;
            Nn[ro * 8 + lane] = r.nan;
        }
        const Iv root = fetch(rk, rr);
        const uint8_t state = iv_state(root);
        lv.type[i] = state == ST_EMPTY ? CELL_EMPTY
                   : state == ST_FILLED ? CELL_FILLED : CELL_BRANCH;
        if (state != ST_AMBIGUOUS) continue;
        if (ch > A.dec_cap) {   // cannot happen: dec_cap is the unpruned tape's count
            atomicOr(A.status, ST_REGS);
            lv.cell_tape[i] = T;
            continue;
        }
        // NaN-unsafe results keep the unpruned tape (dc_tree.inl:107-111).
        if (root.nan || !changed) {
            lv.cell_tape[i] = T;
            continue;
        }
        // Backward liveness pass over registers: count, then allocate and
        // write the kept clauses from the back.
        uint32_t kept = 0;
        TapeRef out = T;
        for (int pass = 0; pass < 2; ++pass) {
            for (uint32_t r = 0; r < T.nregs; ++r) Nn[r * 8 + lane] = 0;
            if (rk == OPND_REG) Nn[rr * 8 + lane] = 1;
            uint32_t pos = kept;
            uint32_t chi = ch;
            unsigned long long off = 0;
            if (pass == 1) {
                off = atomicAdd(A.arena_top, static_cast<unsigned long long>(kept));
                if (off + kept > A.arena_cap) {
                    atomicOr(A.status, ST_ARENA_OVERFLOW);
                    break;
                }
            }
            for (int64_t c = static_cast<int64_t>(T.len) - 1; c >= 0; --c) {
                const uint2 raw = __ldg(reinterpret_cast<const uint2*>(cl + c));
                const uint8_t o_ = raw.x & 0xff;
                const uint32_t kinds = (raw.x >> 8) & 0xff;
                const uint32_t ro = raw.x >> 16;
                uint8_t keep = 0;
                if (o_ == op::MIN || o_ == op::MAX) keep = dec[--chi];
                if (!Nn[ro * 8 + lane]) continue;
                Nn[ro * 8 + lane] = 0;
                uint2 outc = raw;
                bool emit = true;
                if (keep) {
                    const uint32_t k = keep == 1 ? (kinds & 3) : ((kinds >> 2) & 3);
                    const uint32_t src = keep == 1 ? (raw.y & 0xffff) : (raw.y >> 16);
                    if (k == OPND_REG) {
                        Nn[src * 8 + lane] = 1;
                        emit = src != ro;
                    }
                    outc.x = OP_COPY | (k << 8) | (ro << 16);
                    outc.y = src;
                } else {
                    if ((kinds & 3) == OPND_REG) Nn[(raw.y & 0xffff) * 8 + lane] = 1;
                    if (dev_is_binary(o_) && ((kinds >> 2) & 3) == OPND_REG) {
                        Nn[(raw.y >> 16) * 8 + lane] = 1;
                    }
                }
                if (!emit) continue;
                if (pass == 0) {
                    ++kept;
                } else {
                    *reinterpret_cast<uint2*>(A.arena + off + (--pos)) = outc;
                }
            }
            if (pass == 1) {
                out = {static_cast<uint32_t>(off), kept, T.nregs, T.root};
                if (kept <= kRenumberMax) {
                    out = renumber_tape(reinterpret_cast<uint2*>(A.arena + off), out, lastuse,
                                        RM, MK, A.status);
                }
            }
        }
        lv.cell_tape[i] = out;
    }
}

////////////////////////////////////////////////////////////////////////////////
// 2. Leaves: one warp per group of eight sibling cells


struct EdgeSlot {
    float g0[4], g1[4];    // gradient + value at the bracket's ends
    uint8_t amb[2];        // tied min/max there
};

/// A lattice edge's search bracket: inside end (x, y, z), outside end.
struct EdgeBracket {
    double t[6];
};

/// Zero-valued samples of a group's edge search that its QEF pass checks.
constexpr uint32_t kLeafZeros = 48;

constexpr uint32_t kLeafSteps = 56;   // steps of a tape in shared memory at a time
constexpr uint32_t kLeafChunk = 4;    // groups taken at a time, with 16 or more a warp

/// Per-warp state of the corner and edge-search kernel, in shared memory
/// (24 warps an SM beside register files of kLeafSmemRegsMany registers, 16
/// beside kLeafSmemRegs).
struct __align__(16) LeafWarpShared {
    union {
        ValOp vops[kLeafSteps];    // the tape's steps (short tapes: once a group)
        LeafOp dops[kLeafOps];     // the derivative interpreter's clauses
    };
    EdgeBracket br[54];
    double lats[kLeafChunk][3][3]; // lattice coordinates along each axis, by group
    union {
        float zpt[kLeafZeros][3];  // samples with a zero value, to be checked
        uint8_t zlist[128];        // CAREFUL: their slots, to be settled here
    };
    uint32_t term[5];              // samples that are outside, by slot (one word more)
    uint32_t zero[4];              // samples with a zero value
    int8_t slot_of[54];            // lattice edge -> slot, -1 if not crossing
};

/// Per-warp state kept in global memory (L1-cached): the gradients at the
/// edges' final bracket ends and the feature evaluator's scratch, one slice
/// per resident warp.
struct LeafWarpScratch {
    FeatureScratch fs;
    EdgeSlot e[54];
    uint32_t check_status;   // of the feature searches at listed zeros
};

/// A crossing lattice edge's QEF, handed from the leaf kernel to the rank
/// and vertex kernels.
struct EdgeRec {
    double t[6];   // final search bracket: inside end, outside end
    Qef q;
    uint8_t exists;
    uint8_t rank;
};

/// Where a leaf group's edge records start, and which lattice edge has
/// which (-1: none).
struct GroupEdges {
    uint32_t base;          // 0xffffffff: the records did not fit
    uint32_t zbase;         // its zero-valued samples in LeafArgs::zeros
    uint8_t n_edges;
    uint8_t n_zeros;        // or kZerosRedo
    int8_t slot_of[54];
};
constexpr uint8_t kZerosRedo = 0xff;   // the group is on the redo list

/// The interpreters' register file (one float4 per register and lane): in
/// the block's dynamic shared memory at byte offset `soff` (S = true: the
/// compiler then emits shared-memory loads and stores, and knows they cannot
/// alias anything else), or in global memory at `g` (tapes with too many
/// registers).
template <bool S>
__device__ __forceinline__ float4* regfile4(uint32_t soff, float* g)
{
    if (S) {
        extern __shared__ __align__(16) unsigned char rf_smem[];
        return reinterpret_cast<float4*>(rf_smem + soff);
    }
    return reinterpret_cast<float4*>(g);
}

/// The warp's decoded-clause buffer (kLeafOps LeafOps) at byte offset `off`
/// of the block's dynamic shared memory.
__device__ __forceinline__ LeafOp* leaf_ops(uint32_t off)
{
    extern __shared__ __align__(16) unsigned char rf_smem[];
    return reinterpret_cast<LeafOp*>(rf_smem + off);
}

/// dv_value on four points (a float4 per operand), the value rules of
/// dev_point.cuh; the rare opcodes out of line.
__device__ __forceinline__ float4 dv_value4f(uint8_t o, const float4& a, const float4& b)
{
#define LFB_EACH2(F) make_float4(F(a.x, b.x), F(a.y, b.y), F(a.z, b.z), F(a.w, b.w))
#define LFB_EACH1(F) make_float4(F(a.x), F(a.y), F(a.z), F(a.w))
    switch (o) {
        case op::ADD: return LFB_EACH2(f_add);
        case op::MUL: return LFB_EACH2(f_mul);
        case op::MIN: return LFB_EACH2(sc_min);
        case op::MAX: return LFB_EACH2(sc_max);
        case op::SUB: return LFB_EACH2(f_sub);
        case op::SQUARE: return LFB_EACH1(f_square);
        case op::SQRT: return LFB_EACH1(f_sqrt);
        case op::NEG: return LFB_EACH1(f_neg);
        case op::ABS: return LFB_EACH1(f_abs);
        case op::CONST_VAR:
        case OP_COPY: return a;
        default: return leaf_generic4(o, a, b);
    }
#undef LFB_EACH1
#undef LFB_EACH2
}

/// Values of the tape at four points per lane (point k of this lane in
/// component k) for tapes with more registers than the shared-memory file
/// holds: the clauses are streamed (one fetched ahead), the register file R
/// (x, y, z in its first three) is in global memory.  With ties, bit k of
/// *amb reports a min / max with equal arguments at point k
/// (ArrayEvaluator::getAmbiguous, eval_array.cpp:197-217).
static __device__ __noinline__ float4 warp_value4(const float* __restrict__ cpool,
                                                  uint32_t root_kind, uint32_t root,
                                                  const RegClause* __restrict__ cl, uint32_t len,
                                                  float* Rg, int lane, bool ties, uint32_t* amb)
{
    float4* R = reinterpret_cast<float4*>(Rg) + lane;
    uint32_t t = 0;
    uint2 next = len ? __ldg(reinterpret_cast<const uint2*>(cl)) : make_uint2(0, 0);
#pragma unroll 1
    for (uint32_t c = 0; c < len; ++c) {
        const uint2 raw = next;
        if (c + 1 < len) next = __ldg(reinterpret_cast<const uint2*>(cl + c + 1));
        const uint8_t o = raw.x & 0xff;
        const uint32_t kinds = (raw.x >> 8) & 0xff;
        const uint32_t ra = raw.y & 0xffff, rb = raw.y >> 16, ro = raw.x >> 16;
        const float4 a = (kinds & 3) == OPND_REG ? R[ra * 32] : splat4(__ldg(cpool + ra));
        const float4 b = ((kinds >> 2) & 3) == OPND_REG ? R[rb * 32] : splat4(__ldg(cpool + rb));
        if (ties && (o == op::MIN || o == op::MAX)) t |= tie4(a, b);
        R[ro * 32] = dv_value4f(o, a, b);
    }
    *amb = t;
    if (root_kind == OPND_REG) return R[root * 32];
    return splat4(__ldg(cpool + root));
}

/// Value and gradient of the tape at one point per lane, plus, for most
/// points, FeatureEvaluator's feature list (eval_feature.cpp:171-372)
/// without building it.  Every register is either plain (one feature: its
/// gradient, no epsilons) or tainted (anything else).  A tied min/max of two
/// plain features is settled as the general feature path settles it
/// (Feature::push and operator<, feature.cpp:50-72, 247-284): a gradient
/// difference of zero length keeps the first argument; otherwise the two
/// candidates (each gradient with the normalised difference, or its
/// negation, as epsilon) are sorted and, when their gradients agree to
/// within 1e-10 (squared), collapse to the first, epsilons dropped.  Any
/// other tie taints the result; a min/max without a tie passes on the chosen
/// side, taint included; all other clauses are tainted when an operand is.
/// Values are always exact.  *plain says the root is untainted: its single
/// feature is then the returned gradient.  *ambig reports any tie
/// (ArrayEvaluator::getAmbiguous).  Tapes with more than 64 registers report
/// every tie as not plain.
template <bool S>
static __device__ __noinline__ D4 leaf_deriv(const float* __restrict__ cpool, uint32_t root_kind,
                                             uint32_t root, uint32_t n_regs,
                                             const RegClause* __restrict__ cl, uint32_t len,
                                             uint32_t soff, float* Rg, uint32_t ops_off, int lane,
                                             float x, float y, float z, bool* ambig, bool* plain,
                                             bool predecoded)
{
    float4* R = regfile4<S>(soff, Rg) + lane;
    LeafOp* ops = leaf_ops(ops_off);
    R[0] = make_float4(x, 1.0f, 0.0f, 0.0f);
    R[32] = make_float4(y, 0.0f, 1.0f, 0.0f);
    R[64] = make_float4(z, 0.0f, 0.0f, 1.0f);
    const bool trackable = n_regs <= 64;
    uint64_t taint = 0;
    bool amb = false, lost = false;
    if (len <= kLeafOps && predecoded) {
        if (len) leaf_run_deriv(ops, len, R, taint, amb, lost, trackable);
    } else {
        LeafRaw raw = leaf_fetch(cl, len, 0, lane);
        for (uint32_t c0 = 0; c0 < len; c0 += kLeafOps) {
            __syncwarp();
            const uint32_t n = leaf_decode_chunk(ops, raw, len, c0, cpool, lane);
            raw = leaf_fetch(cl, len, c0 + kLeafOps, lane);
            leaf_run_deriv(ops, n, R, taint, amb, lost, trackable);
        }
        __syncwarp();
    }
    *ambig = amb;
    *plain = !lost && !(root_kind == OPND_REG && ((taint >> (root & 63)) & 1));
    if (root_kind == OPND_REG) return d4_of(R[root * 32]);
    return {__ldg(cpool + root), 0.0f, 0.0f, 0.0f};
}

// Registers of the shared-memory register file per warp, 16 or 8 in
// k_leaf_groups (16 warps an SM or 24) and 16 in k_leaf_qef; longer tapes'
// groups run from global memory, clause by clause.
constexpr uint32_t kLeafSmemRegs = 16;
constexpr uint32_t kLeafSmemRegsMany = 8;
constexpr int kLeafWarps = 8, kLeafBlocks = 3;   // warps per block, blocks per SM
static_assert(kLeafSmemRegs <= kValMaxRegs, "register offsets of a step are 16 bits");

struct LeafArgs {
    Octree o;
    DevTape bt;
    const RegClause* arena;
    LeafRec* recs;
    uint32_t* rec_top;
    uint32_t rec_cap;
    uint32_t* status;
    unsigned long long* evals;
    LeafWarpScratch* scratch;   // gridDim.x * warps-per-block slices
    float* rd;                  // per warp: n_regs x 4 x 32 floats (long tapes)
    uint32_t smem_regs;         // registers of the shared-memory register file
    uint32_t* next_group;       // work counter (zero at launch)
    const uint32_t* order;      // processing order of the groups (or null)
    float* featws;              // per warp: n_regs x kRegBlock floats of feature lists
    EdgeRec* edges;             // crossing-edge QEFs of all groups
    unsigned long long* edge_top;
    uint32_t edge_cap;
    GroupEdges* group_edges;    // one per group
    uint32_t* rec_group;        // per leaf record: group * 8 + cell
    uint32_t* next_group2;      // work counter of k_leaf_qef (zero at launch)
    ValOp* vops;                // decoded steps of a tape, from its clause offset on
    uint32_t* n_steps;          // by clause offset: steps of the tape there
    uint32_t chunk;             // groups a warp of k_leaf_groups takes at a time
    float* zeros;               // zero-valued samples to check: x, y, z
    unsigned int* zero_top;
    uint32_t zero_cap;
    uint32_t* redo;             // groups to search again, carefully
    uint32_t* n_redo;
    uint32_t* next_redo;        // work counters of the two kernels of that
};

/// The value interpreter's steps (leaf_interp.cuh) of every tape that leaf
/// groups use, decoded once a tape: groups whose parents decided nothing
/// share theirs (six groups a tape on deep CSG meshes).  Steps go to
/// A.vops from the tape's own clause offset on (there are never more steps
/// than clauses), their number to A.n_steps, where the first group to come
/// claims the tape.  A kernel of its own: decoding in k_leaf_groups cost
/// 1,000 instructions a group and its code the instruction cache
/// (2,000-primitive CSG at depth 8: 1.95 ms with it, 1.38 ms without).
__global__ void __launch_bounds__(128)
k_leaf_decode(const __grid_constant__ LeafArgs A, const TapeRef* tapes, uint32_t n, uint32_t per_warp)
{
    __shared__ uint2 raws[4][kValRaw];
    const uint32_t lane = threadIdx.x & 31;
    uint2* raw = raws[threadIdx.x >> 5];
    const uint32_t i = (blockIdx.x * 4 + (threadIdx.x >> 5)) * per_warp + lane;
    uint32_t off = 0, len = 0;
    if (lane < per_warp && i < n) {
        const TapeRef t = tapes[i];
        if (t.nregs <= A.smem_regs && t.len && A.n_steps[t.off] == 0 &&
            atomicCAS(A.n_steps + t.off, 0u, 0xffffffffu) == 0) {
            off = t.off;
            len = t.len;
        }
    }
    uint32_t todo = __ballot_sync(0xffffffffu, len != 0);
    while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const uint32_t o = __shfl_sync(0xffffffffu, off, src);
        const uint32_t l = __shfl_sync(0xffffffffu, len, src);
        uint32_t steps = 0;
        for (uint32_t c0 = 0; c0 < l; c0 += kLeafOps) {
            steps += val_decode(A.vops + o + steps, raw, A.arena + o, l, c0, A.bt.cpool, lane);
        }
        if (lane == 0) A.n_steps[o] = steps;
    }
}

/// FeatureEvaluator::isInside at one point (all lanes the same), out of line
/// with its own contexts so that the leaf kernel's hot state stays in
/// registers.
static __device__ __noinline__ bool leaf_is_inside(const LeafArgs& A, TapeRef tr, uint32_t slice,
                                                   float x, float y, float z, int lane)
{
    const FeatCtx fc{A.featws + static_cast<size_t>(slice) * A.bt.n_regs * kRegBlock,
                     &A.scratch[slice].fs, A.status};
    return dev_is_inside(fc, with_tape(A.bt, tr), A.arena + tr.off, tr.len, x, y, z, lane);
}

/// DCTree::evalLeaf's corners, classification and edge search
/// (dc_tree.inl:156-410), one warp per sibling group.  SINGLE: the root cell
/// is the only leaf (a 2 x 2 x 2 lattice instead of 3 x 3 x 3).
///
/// A sample whose value is exactly zero is inside or not by its gradient
/// (FeatureEvaluator::isInside): for a point without tied min/max "gradient
/// is non-zero" (one feature), otherwise the full feature search.  Nearly
/// all are inside, and nearly every group has some in its last rounds.  So
/// the search takes them for inside and writes them down, and k_leaf_qef,
/// which evaluates gradients in any case and has lanes free, checks them; a
/// group with a sample that is not inside (or more of them than there is
/// room for) is listed in LeafArgs::redo and searched again by the CAREFUL
/// form, which settles each zero where it meets it.  Evaluating gradients
/// here instead took 2,500 of 10,000 instructions a group and, because the
/// two interpreters' code then alternates, 37 % of the time (64-sphere
/// union at depth 8: 1.71 ms against 1.08 ms).
template <bool SINGLE, bool CAREFUL>
__global__ void __launch_bounds__(32 * kLeafWarps, kLeafBlocks)
k_leaf_groups(const __grid_constant__ LeafArgs A, uint32_t n_groups)
{
    extern __shared__ __align__(16) unsigned char lsmem[];
    constexpr int n = SINGLE ? 2 : 3;        // lattice points per axis
    constexpr int seg = n - 1;
    constexpr int ncell = SINGLE ? 1 : 8;
    constexpr int npts = n * n * n;
    constexpr int n_lat_edges = 3 * seg * n * n;
    constexpr bool REDO = CAREFUL && !SINGLE;   // groups of the redo list
    // The edge search's sample fractions j / 15 and 1 - j / 15, computed
    // once per block (the same correctly rounded values as at every sample).
    __shared__ double2 frac_tab[16];
    if (threadIdx.x < 16) {
        const double frac = threadIdx.x / (16 - 1.0);
        frac_tab[threadIdx.x] = make_double2(frac, 1 - frac);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const unsigned full = 0xffffffffu;
    LeafWarpShared* S = reinterpret_cast<LeafWarpShared*>(lsmem) + warp;
    const uint32_t rsoff = static_cast<uint32_t>(sizeof(LeafWarpShared) * wpb +
                                                 size_t{kValRegBytes} * A.smem_regs * warp);
    const uint32_t ops_off = static_cast<uint32_t>(reinterpret_cast<unsigned char*>(S->dops) - lsmem);
    unsigned char* Rl = lsmem + rsoff + 16 * lane;
    const uint32_t slice = blockIdx.x * wpb + warp;   // of the per-warp global scratch
    float* Rgl = A.rd + static_cast<size_t>(slice) * A.bt.n_regs * 128;
    const Octree& o = A.o;
    const int Ld = o.levels;
    // Persistent warps take the next groups from a shared counter (group
    // costs vary by orders of magnitude with the tape length), a few at a
    // time, so that the loads that lead to a group's tape and region overlap
    // for all of them: one group a lane.
    const uint32_t n_todo = REDO ? min(*A.n_redo, n_groups) : n_groups;
    while (true) {
    uint32_t g0 = 0;
    if (lane == 0) g0 = atomicAdd(REDO ? A.next_redo : A.next_group, A.chunk);
    g0 = __shfl_sync(full, g0, 0);
    if (g0 >= n_todo) break;
    const uint32_t n_here = min(A.chunk, n_todo - g0);
    uint32_t lane_g = 0, lane_steps = 0;
    TapeRef lane_tr{};
    unsigned long long lane_pc = 0;
    if (lane < n_here) {
        lane_g = REDO ? A.redo[g0 + lane] : A.order ? A.order[g0 + lane] : g0 + lane;
        lane_tr = SINGLE ? root_tape_ref(A.bt) : o.lv[Ld].group_tape[lane_g];
        if (!SINGLE) lane_pc = o.lv[Ld - 1].coords[o.lv[Ld].group_parent[lane_g]];
        if (lane_tr.len && lane_tr.nregs <= A.smem_regs) lane_steps = A.n_steps[lane_tr.off];
    }
    {
        // Lattice coordinates along each axis (double), from the parent
        // region split at its centre exactly like Region::subdivide: lane 3
        // i + a computes group i's axis a.
        const int i = min(lane / 3, static_cast<int>(kLeafChunk) - 1), a = lane % 3;
        const uint64_t pc = __shfl_sync(full, lane_pc, i);
        if (lane < 3 * static_cast<int>(kLeafChunk)) {
            double l = o.lo[a], h = o.hi[a];
            double* lat = S->lats[i][a];
            if (SINGLE) {
                lat[0] = l;
                lat[1] = h;
            } else {
                const uint32_t idx = static_cast<uint32_t>(pc >> (21 * a)) & 0x1fffff;
                for (int b = Ld - 2; b >= 0; --b) {
                    const double m = (l + h) / 2;
                    if ((idx >> b) & 1) l = m; else h = m;
                }
                lat[0] = l;
                lat[1] = (l + h) / 2;
                lat[n - 1] = h;
            }
        }
    }
    __syncwarp();
#pragma unroll 1
    for (uint32_t gi = 0; gi < n_here; ++gi) {
    const uint32_t g = __shfl_sync(full, lane_g, gi);
    const TapeRef tr{__shfl_sync(full, lane_tr.off, gi), __shfl_sync(full, lane_tr.len, gi),
                     __shfl_sync(full, lane_tr.nregs, gi), __shfl_sync(full, lane_tr.root, gi)};
    const uint32_t n_steps = __shfl_sync(full, lane_steps, gi);
    if (REDO && A.group_edges[g].base == 0xffffffffu) continue;
    const double (*lat)[3] = S->lats[gi];
    const RegClause* cl = A.arena + tr.off;
    const float* cpool = A.bt.cpool;
    const uint32_t root_kind = tr.root >> 16, root = tr.root & 0xffff;
    const bool rs = tr.nregs <= A.smem_regs;
    // Tapes that fit the buffer are fetched once for the whole group (the
    // derivative interpreter's clauses share it: CAREFUL fetches every pass).
    auto fetch = [&](uint32_t s0) -> uint32_t {
        const uint32_t m = min(kLeafSteps, n_steps - s0);
        const uint4* src = reinterpret_cast<const uint4*>(A.vops + tr.off + s0);
        __syncwarp();
        for (uint32_t k = lane; k < 2 * m; k += 32) reinterpret_cast<uint4*>(S->vops)[k] = __ldg(src + k);
        __syncwarp();
        return m;
    };
    const bool once = !CAREFUL && n_steps <= kLeafSteps;
    if (once) fetch(0);

    // Value and gradient at one point per lane, as leaf_deriv.
    auto deriv = [&](float x, float y, float z, bool* amb, bool* plain) -> D4 {
        return rs ? leaf_deriv<true>(cpool, root_kind, root, tr.nregs, cl, tr.len, rsoff,
                                     Rgl, ops_off, lane, x, y, z, amb, plain, false)
                  : leaf_deriv<false>(cpool, root_kind, root, tr.nregs, cl, tr.len, rsoff,
                                      Rgl, ops_off, lane, x, y, z, amb, plain, false);
    };
    auto lat_edge_ends = [&](int e, int& p0, int& p1) {
        const int ax = e / (seg * n * n);
        const int r = e % (seg * n * n);
        const int s = r % seg;
        const int u = (r / seg) % n;
        const int w = r / (seg * n);
        const int step = ax == 0 ? 1 : ax == 1 ? n : n * n;
        const int su = ax == 0 ? n : 1;
        const int sw = ax == 2 ? n : n * n;
        p0 = s * step + u * su + w * sw;
        p1 = p0 + step;
    };
    // Sample j of an edge's bracket (dc_tree.inl:345-351).
    auto sample = [&](int slot, int j) -> double3 {
        const double2 f = frac_tab[j];
        const EdgeBracket& es = S->br[slot];
        return make_double3(es.t[0] * f.y + es.t[3] * f.x, es.t[1] * f.y + es.t[4] * f.x,
                            es.t[2] * f.y + es.t[5] * f.x);
    };
    // The loops below stay rolled where they can: 24 warps an SM in
    // different places of this kernel miss the instruction cache otherwise
    // (unrolled twice, the step loop ran 13 % fewer instructions in the same
    // time, with three times the stalls on instruction fetch).

    // --- passes: first the corners, then the edge search: 4 rounds of 16
    // points (dc_tree.inl:326-410).  Each round samples an edge's bracket
    // [t0, t1] at 16 evenly spaced points j = 0..15 and keeps
    // [s(j-1), s(j)] around the first sample j >= 1 that is outside;
    // failing that, the last one, unless it is an inside zero.  s(0) = t0
    // is never tested, and s(15) = t1 is the previous round's outside end
    // (round 1: the corner known to be outside), which is never an inside
    // zero, so the outcome is "first outside j in 1..14, else 15": only 14
    // samples per edge are evaluated.  One pass holds nine edges (126 of
    // the 4 x 32 sample slots): slot p = 32k + lane of sub-batch k is
    // sample 1 + p % 14 of edge base + p / 14.  Most groups have nine
    // crossing edges, one pass per round.
    constexpr int kEdgesPerPass = 9, kSamples = 14;
    int E = 0, base = 0;
    uint32_t n_zeros = 0;
    for (int round = -1; round < 4;) {
        // register file: x, y, z of the lane's four points
        float* P = reinterpret_cast<float*>(rs ? Rl : reinterpret_cast<unsigned char*>(Rgl) + 16 * lane);
        if (round < 0) {
            const int q = lane < npts ? lane : 0;
            const int c[3] = {q % n, (q / n) % n, q / (n * n)};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                reinterpret_cast<float4*>(P)[32 * a] = splat4(static_cast<float>(lat[a][c[a]]));
            }
        } else {
            // slots past the last sample repeat one, and are masked below
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                const int p = 32 * k + lane;
                const double3 q = sample(min(base + p / kSamples, E - 1), 1 + p % kSamples);
                P[k] = static_cast<float>(q.x);
                P[128 + k] = static_cast<float>(q.y);
                P[256 + k] = static_cast<float>(q.z);
            }
        }
        float4 v4;
        uint32_t amb4 = 0;
        if (rs) {
            float last[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            for (uint32_t s0 = 0; s0 < n_steps; s0 += kLeafSteps) {
                const uint32_t m = once ? n_steps : fetch(s0);
                val_run(S->vops, m, Rl, round < 0, amb4, last);
            }
            v4 = root_kind == OPND_REG
                     ? *reinterpret_cast<const float4*>(Rl + kValRegBytes * root)
                     : splat4(__ldg(cpool + root));
        } else {
            v4 = warp_value4(cpool, root_kind, root, cl, tr.len, Rgl, lane, round < 0, &amb4);
        }

        if (round < 0) {
            // --- corners (dc_tree.inl:156-239) -------------------------
            const float cv = v4.x;
            uint8_t cst = CELL_EMPTY;
            bool need_d = false, need_f = false;
            if (lane < npts) {
                if (cv > 0 || cv != cv) cst = CELL_EMPTY;
                else if (cv < 0) cst = CELL_FILLED;
                else if (!(amb4 & 1)) need_d = true;
                else need_f = true;
            }
            const uint32_t zeros = __ballot_sync(full, need_d || need_f);
            if (zeros) {
                bool amb = false, plain = false;
                const int q = lane < npts ? lane : 0;
                const float px = static_cast<float>(lat[0][q % n]);
                const float py = static_cast<float>(lat[1][(q / n) % n]);
                const float pz = static_cast<float>(lat[2][q / (n * n)]);
                const D4 d = deriv(px, py, pz, &amb, &plain);
                if (once) fetch(0);
                if (lane == 0) atomicAdd(A.evals + 1, static_cast<unsigned long long>(__popc(zeros)) * tr.len);
                if (need_d) {
                    cst = (d.dx != 0 || d.dy != 0 || d.dz != 0) ? CELL_FILLED : CELL_EMPTY;
                }
                if (need_f && plain) {
                    // FeatureEvaluator::isInside with one feature at a zero value.
                    const float gr[3] = {d.dx, d.dy, d.dz};
                    cst = sqrtf(fdot(gr, gr)) > 0 ? CELL_FILLED : CELL_EMPTY;
                    need_f = false;
                }
                uint32_t pending = __ballot_sync(full, need_f);
                while (pending) {
                    const int src = __ffs(pending) - 1;
                    pending &= pending - 1;
                    const float fx = __shfl_sync(full, px, src);
                    const float fy = __shfl_sync(full, py, src);
                    const float fz = __shfl_sync(full, pz, src);
                    const bool inside = leaf_is_inside(A, tr, slice, fx, fy, fz, lane);
                    if (lane == src) cst = inside ? CELL_FILLED : CELL_EMPTY;
                }
            }
            const uint32_t filled = __ballot_sync(full, lane < npts && cst == CELL_FILLED);

            // --- cell classification -----------------------------------
            const LevelView& lvL = o.lv[Ld];
            if (!REDO && lane < ncell) {
                const int cx = lane & 1, cy = (lane >> 1) & 1, cz = (lane >> 2) & 1;
                uint32_t mask = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int p = (cx + (k & 1)) + n * ((cy + ((k >> 1) & 1)) +
                                                        n * (cz + ((k >> 2) & 1)));
                    mask |= ((filled >> p) & 1) << k;
                }
                const uint32_t ci = SINGLE ? 0 : (g * 8 + lane);
                int32_t rec = -1;
                const uint8_t type = mask == 0 ? CELL_EMPTY : mask == 0xff ? CELL_FILLED : CELL_LEAF;
                if (type == CELL_LEAF) {
                    const uint32_t r = atomicAdd(A.rec_top, 1u);
                    if (r >= A.rec_cap) {
                        atomicOr(A.status, ST_RECORD_OVERFLOW);
                    } else {
                        rec = static_cast<int32_t>(r);
                        LeafRec& L = A.recs[r];
                        L.corner_mask = static_cast<uint8_t>(mask);
                        L.manifold = c_tab.manifold[mask];
                        L.vertex_count = c_tab.npatch[mask];
                        L.level = 0;
                        L.rank = 0;
                        A.rec_group[r] = (SINGLE ? 0u : g * 8u) + static_cast<uint32_t>(lane);
                    }
                }
                lvL.type[ci] = type;
                lvL.rec[ci] = rec;
            }

            // --- crossing lattice edges --------------------------------
#pragma unroll 1
            for (int e0 = 0; e0 < n_lat_edges; e0 += 32) {
                const int e = e0 + lane;
                bool crossing = false;
                int p0 = 0, p1 = 0;
                if (e < n_lat_edges) {
                    lat_edge_ends(e, p0, p1);
                    crossing = ((filled >> p0) ^ (filled >> p1)) & 1;
                }
                const uint32_t m = __ballot_sync(full, crossing);
                const int slot = E + __popc(m & ((1u << lane) - 1));
                if (e < n_lat_edges) S->slot_of[e] = crossing ? static_cast<int8_t>(slot) : -1;
                if (crossing) {
                    const bool f0 = (filled >> p0) & 1;
                    const int in = f0 ? p0 : p1, out = f0 ? p1 : p0;
                    EdgeBracket& es = S->br[slot];
                    es.t[0] = lat[0][in % n];
                    es.t[1] = lat[1][(in / n) % n];
                    es.t[2] = lat[2][in / (n * n)];
                    es.t[3] = lat[0][out % n];
                    es.t[4] = lat[1][(out / n) % n];
                    es.t[5] = lat[2][out / (n * n)];
                }
                E += __popc(m);
            }
            __syncwarp();
            if (E == 0) break;
            round = 0;
            continue;
        }

        // --- one pass of the edge search -------------------------------
        const float vs[4] = {v4.x, v4.y, v4.z, v4.w};
        const int n_act = kSamples * min(kEdgesPerPass, E - base);
        uint32_t any_zero = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t act = n_act >= 32 * (k + 1) ? full
                                 : n_act > 32 * k ? (1u << (n_act - 32 * k)) - 1 : 0u;
            const uint32_t t = __ballot_sync(full, vs[k] > 0) & act;
            const uint32_t z = __ballot_sync(full, vs[k] == 0) & act;
            if (lane == k) {
                S->term[k] = t;
                S->zero[k] = z;
            }
            any_zero |= z;
        }
        __syncwarp();
        // The 14 samples' bits of the pass's edge e.
        auto edge_bits = [&](int e) -> uint32_t {
            const int p0 = kSamples * e;
            return __funnelshift_r(S->term[p0 >> 5], S->term[(p0 >> 5) + 1], p0 & 31) &
                   ((1u << kSamples) - 1);
        };
        if (any_zero) {
            // Zeros before the edge's first positive sample, gathered one
            // per lane: CAREFUL settles them, otherwise they go on the list.
            uint32_t nz = CAREFUL ? 0 : n_zeros;
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
                if (!S->zero[k]) continue;
                const int p = 32 * k + lane;
                const uint32_t t = edge_bits(p / kSamples);
                const bool need = ((S->zero[k] >> lane) & 1) && (!t || p % kSamples < __ffs(t) - 1);
                const uint32_t m = __ballot_sync(full, need);
                const uint32_t at = nz + __popc(m & ((1u << lane) - 1));
                if (need) {
                    if (CAREFUL) {
                        S->zlist[at] = static_cast<uint8_t>(p);
                    } else if (at < kLeafZeros) {
                        const double3 q = sample(base + p / kSamples, 1 + p % kSamples);
                        S->zpt[at][0] = static_cast<float>(q.x);
                        S->zpt[at][1] = static_cast<float>(q.y);
                        S->zpt[at][2] = static_cast<float>(q.z);
                    }
                }
                nz += __popc(m);
            }
            __syncwarp();
            if (!CAREFUL) n_zeros = nz;
            if (CAREFUL && nz && lane == 0) {
                atomicAdd(A.evals + 1, static_cast<unsigned long long>(nz) * tr.len);
            }
            for (uint32_t i0 = 0; CAREFUL && i0 < nz; i0 += 32) {
                const bool on = i0 + lane < nz;
                const int p = S->zlist[on ? i0 + lane : 0];
                const double3 q = sample(base + p / kSamples, 1 + p % kSamples);
                const float zx = static_cast<float>(q.x);
                const float zy = static_cast<float>(q.y);
                const float zz = static_cast<float>(q.z);
                bool amb = false, plain = false;
                const D4 dg = deriv(zx, zy, zz, &amb, &plain);
                amb = amb && !plain;   // a settled tie leaves one plain feature
                const float gr[3] = {dg.dx, dg.dy, dg.dz};
                bool inside = !on || amb || sqrtf(fdot(gr, gr)) > 0;
                uint32_t pending = __ballot_sync(full, on && amb);
                while (pending) {
                    const int src = __ffs(pending) - 1;
                    pending &= pending - 1;
                    const float fx = __shfl_sync(full, zx, src);
                    const float fy = __shfl_sync(full, zy, src);
                    const float fz = __shfl_sync(full, zz, src);
                    const bool in = leaf_is_inside(A, tr, slice, fx, fy, fz, lane);
                    if (lane == src) inside = in;
                }
                if (!inside) atomicOr(&S->term[p >> 5], 1u << (p & 31));
                __syncwarp();
            }
        }
        // New brackets from the old ones: lanes 2 e and 2 e + 1 make edge e's
        // inside and outside end.
        const int e = min(min(lane >> 1, kEdgesPerPass - 1), E - 1 - base);
        const uint32_t t = edge_bits(e);
        const int pick = t ? __ffs(t) : 15;   // sample index of the outside end
        const double3 q = sample(base + e, pick - 1 + (lane & 1));
        __syncwarp();
        if (e == lane >> 1) {
            double* to = S->br[base + e].t + 3 * (lane & 1);
            to[0] = q.x;
            to[1] = q.y;
            to[2] = q.z;
        }
        __syncwarp();
        base += kEdgesPerPass;
        if (base >= E) {
            base = 0;
            ++round;
        }
    }

    // --- hand the final brackets and the lattice edge map to k_leaf_qef and
    //     the vertex kernel --------------------------------------------------
    GroupEdges& ge = A.group_edges[SINGLE ? 0 : g];
    unsigned long long first = 0;
    if (REDO) {
        first = ge.base;
    } else {
        if (lane == 0) first = atomicAdd(A.edge_top, static_cast<unsigned long long>(E));
        first = __shfl_sync(full, first, 0);
    }
    if (first + E > A.edge_cap) {
        if (lane == 0) {
            atomicOr(A.status, ST_EDGE_OVERFLOW);
            ge.base = 0xffffffffu;
            ge.n_edges = 0;
        }
    } else {
        for (int k = lane; k < 6 * E; k += 32) A.edges[first + k / 6].t[k % 6] = S->br[k / 6].t[k % 6];
        uint32_t zbase = 0;
        if (!CAREFUL && n_zeros) {
            if (n_zeros <= kLeafZeros) {
                if (lane == 0) zbase = atomicAdd(A.zero_top, n_zeros);
                zbase = __shfl_sync(full, zbase, 0);
            }
            if (n_zeros > kLeafZeros || zbase > A.zero_cap || n_zeros > A.zero_cap - zbase) {
                if (lane == 0) A.redo[atomicAdd(A.n_redo, 1u)] = g;
                n_zeros = kZerosRedo;
            }
            for (uint32_t k = lane; n_zeros != kZerosRedo && k < 3 * n_zeros; k += 32) {
                A.zeros[size_t{3} * zbase + k] = S->zpt[k / 3][k % 3];
            }
        }
        if (lane == 0) {
            ge.base = static_cast<uint32_t>(first);
            ge.n_edges = static_cast<uint8_t>(E);
            ge.zbase = zbase;
            ge.n_zeros = static_cast<uint8_t>(n_zeros);
        }
        for (int k = lane; k < n_lat_edges; k += 32) ge.slot_of[k] = S->slot_of[k];
    }
    if (lane == 0) {
        atomicAdd(A.evals, static_cast<unsigned long long>(npts + 4 * kSamples * E) * tr.len);
    }
    __syncwarp();
    }
    }   // groups
}

/// Gradients at the two ends of every crossing edge's final bracket and the
/// edge's QEF (dc_tree.inl:412-471): one warp per leaf group (the group's
/// tape), one bracket end per lane, then each lane pushes whole edges
/// (inside end first).  Points where a min / max is tied use every feature
/// gradient instead (eval_feature.cpp:125-169).  A launch of its own, so
/// that the derivative interpreter does not share the instruction cache
/// with the value interpreter of the edge search.
/// The group's zero-valued samples are checked along with them (REDO: not,
/// the groups of the redo list after their careful search).
template <bool REDO>
__global__ void __launch_bounds__(256, 3)
k_leaf_qef(LeafArgs A, uint32_t n_groups)
{
    extern __shared__ __align__(16) unsigned char lsmem[];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    float* Rs = reinterpret_cast<float*>(lsmem) + static_cast<size_t>(warp) * A.smem_regs * 128;
    float* Rgl = A.rd + (static_cast<size_t>(blockIdx.x) * wpb + warp) * A.bt.n_regs * 128;
    const uint32_t ops_off = static_cast<uint32_t>(static_cast<size_t>(wpb) * A.smem_regs * 128 * 4 +
                                                   static_cast<size_t>(warp) * kLeafOps * sizeof(LeafOp));
    LeafWarpScratch* W = A.scratch + static_cast<size_t>(blockIdx.x) * wpb + warp;
    const FeatCtx fc{A.featws + (static_cast<size_t>(blockIdx.x) * wpb + warp) *
                                    A.bt.n_regs * kRegBlock,
                     &W->fs, A.status};
    // A listed zero may lie where the careful search never comes (after one
    // that is not inside), so a feature search that overflows there sends the
    // group back instead of failing the mesh.
    const FeatCtx check_fc{fc.regs, fc.tmp, &W->check_status};
    if (!REDO && lane == 0) W->check_status = 0;
    uint64_t my_devals = 0;
    const Octree& o = A.o;
    const int Ld = o.levels;
    const bool single = (Ld == 0);
    while (true) {
        uint32_t g = 0;
        if (lane == 0) g = atomicAdd(REDO ? A.next_redo + 1 : A.next_group2, 1u);
        g = __shfl_sync(0xffffffffu, g, 0);
        if (g >= (REDO ? min(*A.n_redo, n_groups) : n_groups)) break;
        if (REDO) g = A.redo[g];
        else if (A.order) g = A.order[g];
        const GroupEdges& ge = A.group_edges[single ? 0 : g];
        const uint32_t gbase = ge.base;
        const int E = ge.n_edges;
        if (gbase == 0xffffffffu || E == 0 || (!REDO && ge.n_zeros == kZerosRedo)) continue;
        const TapeRef tr = single ? root_tape_ref(A.bt) : o.lv[Ld].group_tape[g];
        const RegClause* cl = A.arena + tr.off;
        const DevTape tb = with_tape(A.bt, tr);
        const bool rs = tb.n_regs <= A.smem_regs;
        float* R = rs ? Rs : Rgl;
        const uint32_t rsoff = static_cast<uint32_t>(reinterpret_cast<unsigned char*>(Rs) - lsmem);
        __syncwarp();
        if (tr.len <= kLeafOps) {
            leaf_decode_chunk(leaf_ops(ops_off), leaf_fetch(cl, tr.len, 0, lane), tr.len, 0,
                              tb.cpool, lane);
        }
        EdgeRec* er = A.edges + gbase;
        const float* zp = A.zeros + size_t{3} * ge.zbase;
        const int n_pts = 2 * E + (REDO ? 0 : ge.n_zeros);
        bool outside = false;   // a zero-valued sample that is not inside
        for (int base = 0; base < n_pts; base += 32) {
            const int p = base + lane;
            const bool active = p < 2 * E, check = !active && p < n_pts;
            float q[3] = {0, 0, 0};
            if (active) {
                const EdgeRec& e = er[p >> 1];
                for (int k = 0; k < 3; ++k) q[k] = static_cast<float>(e.t[(p & 1) * 3 + k]);
            } else if (check) {
                for (int k = 0; k < 3; ++k) q[k] = zp[3 * (p - 2 * E) + k];
            }
            bool amb = false, plain = false;
            const D4 d = rs ? leaf_deriv<true>(tb.cpool, tb.root_kind, tb.root, tb.n_regs, cl,
                                               tr.len, rsoff, R, ops_off, lane, q[0], q[1], q[2],
                                               &amb, &plain, true)
                            : leaf_deriv<false>(tb.cpool, tb.root_kind, tb.root, tb.n_regs, cl,
                                                tr.len, rsoff, R, ops_off, lane, q[0], q[1], q[2],
                                                &amb, &plain, true);
            if (lane == 0) my_devals += static_cast<uint64_t>(min(32, n_pts - base)) * tr.len;
            amb = amb && !plain;   // a settled tie leaves one plain feature
            const float gr[3] = {d.dx, d.dy, d.dz};
            outside |= check && !amb && !(sqrtf(fdot(gr, gr)) > 0);
            uint32_t pending = __ballot_sync(0xffffffffu, check && amb);
            const bool searched = pending != 0;
            while (pending) {
                const int src = __ffs(pending) - 1;
                pending &= pending - 1;
                const float fx = __shfl_sync(0xffffffffu, q[0], src);
                const float fy = __shfl_sync(0xffffffffu, q[1], src);
                const float fz = __shfl_sync(0xffffffffu, q[2], src);
                outside |= !dev_is_inside(check_fc, tb, cl, tr.len, fx, fy, fz, lane);
            }
            if (searched) {
                __syncwarp();
                uint32_t overflowed = 0;
                if (lane == 0) overflowed = atomicExch(&W->check_status, 0u);
                outside |= __shfl_sync(0xffffffffu, overflowed, 0) != 0;
            }
            if (active) {
                EdgeSlot& es = W->e[p >> 1];
                float* gg = (p & 1) ? es.g1 : es.g0;
                gg[0] = d.dx; gg[1] = d.dy; gg[2] = d.dz; gg[3] = d.v;
                es.amb[p & 1] = amb;
            }
        }
        __syncwarp();
        if (!REDO && __any_sync(0xffffffffu, outside)) {
            if (lane == 0) A.redo[atomicAdd(A.n_redo, 1u)] = g;
            continue;
        }
        const uint32_t any_amb = __ballot_sync(0xffffffffu, [&] {
            bool a = false;
            for (int s_ = lane; s_ < E; s_ += 32) a |= W->e[s_].amb[0] || W->e[s_].amb[1];
            return a;
        }());
        if (!any_amb) {
            for (int s_ = lane; s_ < E; s_ += 32) {
                const EdgeSlot& es = W->e[s_];
                EdgeRec& r = er[s_];
                Qef qf;
                qef_zero(qf);
                for (int side = 0; side < 2; ++side) {
                    const float* gg = side ? es.g1 : es.g0;
                    const double* pos = r.t + 3 * side;
                    const double gd[3] = {gg[0], gg[1], gg[2]};
                    qef_push(qf, pos, gd, static_cast<double>(gg[3]));
                }
                r.q = qf;
                r.exists = 1;
                r.rank = 0;
            }
        } else {
            for (int s_ = lane; s_ < E; s_ += 32) {
                qef_zero(er[s_].q);
                er[s_].exists = 0;
                er[s_].rank = 0;
            }
            __syncwarp();
            for (int s_ = 0; s_ < E; ++s_) {
                const EdgeSlot& es = W->e[s_];
                EdgeRec& r = er[s_];
                for (int side = 0; side < 2; ++side) {
                    const float* gg = side ? es.g1 : es.g0;
                    const double* pos = r.t + 3 * side;
                    if (es.amb[side]) {
                        dev_push_features(fc, tb, cl, tr.len, pos, static_cast<double>(gg[3]),
                                          &r.q, &r.exists, lane);
                    } else if (lane == 0) {
                        const double gd[3] = {gg[0], gg[1], gg[2]};
                        qef_push(r.q, pos, gd, static_cast<double>(gg[3]));
                        r.exists = 1;
                    }
                    __syncwarp();
                }
            }
        }
        __syncwarp();
    }
    if (lane == 0) atomicAdd(A.evals + 1, static_cast<unsigned long long>(my_devals));
}

/// Intersection::get_rank (intersection.hpp:67-88) of every crossing edge's
/// QEF, one thread per edge.
__global__ void __launch_bounds__(128)
k_edge_rank(EdgeRec* edges, const unsigned long long* edge_top, uint32_t cap)
{
    const uint64_t n = min(static_cast<unsigned long long>(cap), *edge_top);
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        edges[i].rank = static_cast<uint8_t>(qef_rank(edges[i].q));
    }
}

/// Per-patch vertices of the leaf records (dc_tree.inl:474-549), one thread
/// per record: the patch's crossing edges found through the group's lattice
/// edge map, the mass point over the edges of highest rank, the summed QEF
/// and DCTree::findVertex.  `single`: the root cell is the only leaf (a
/// 2 x 2 x 2 lattice instead of the 3 x 3 x 3 of a sibling group).
__global__ void __launch_bounds__(128)
k_leaf_vertices(LeafRec* recs, const uint32_t* rec_top, uint32_t rec_cap,
                const uint32_t* rec_group, const GroupEdges* group_edges, uint32_t n_groups,
                const EdgeRec* edges, uint32_t edge_cap, int single)
{
    const uint32_t n_recs = min(rec_cap, *rec_top);
    const int n = single ? 2 : 3;
    const int seg = n - 1;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n_recs;
         r += gridDim.x * blockDim.x) {
        const uint32_t gi = rec_group[r];
        // records of groups whose edges did not fit have none (the mesh is
        // rendered again with more room)
        if (gi == 0xffffffffu || (gi >> 3) >= n_groups) continue;
        const int cell = static_cast<int>(gi & 7);
        const GroupEdges& ge = group_edges[gi >> 3];
        if (ge.base == 0xffffffffu || ge.base + ge.n_edges > edge_cap) continue;
        LeafRec& L = recs[r];
        const uint8_t mask = L.corner_mask;
        auto lat_pt = [&](int corner) {
            const int cx = cell & 1, cy = (cell >> 1) & 1, cz = (cell >> 2) & 1;
            return (cx + (corner & 1)) + n * ((cy + ((corner >> 1) & 1)) +
                                              n * (cz + ((corner >> 2) & 1)));
        };
        const int np = c_tab.npatch[mask];
        for (int patch = 0; patch < np; ++patch) {
            const int ne = c_tab.nedge[mask][patch];
            int slots[12];
            for (int k = 0; k < ne; ++k) {
                const int ca = c_tab.v[mask][patch][k][0];
                const int cb = c_tab.v[mask][patch][k][1];
                // lattice edge between the two corners of this cell
                const int pa = lat_pt(ca), pb = lat_pt(cb);
                const int lo_p = pa < pb ? pa : pb;
                const int diff = (pa < pb ? pb - pa : pa - pb);
                const int ax = diff == 1 ? 0 : diff == n ? 1 : 2;
                const int c0 = lo_p % n, c1 = (lo_p / n) % n, c2 = lo_p / (n * n);
                int le;
                if (ax == 0) le = c0 + seg * (c1 + n * c2);
                else if (ax == 1) le = c1 + seg * (c0 + n * c2);
                else le = c2 + seg * (c0 + n * c1);
                le += ax * seg * n * n;
                const int sl = ge.slot_of[le];
                slots[k] = sl < 0 ? -1 : static_cast<int>(ge.base) + sl;
            }
            int max_rank = 0;
            for (int k = 0; k < ne; ++k) {
                if (slots[k] >= 0 && edges[slots[k]].exists && edges[slots[k]].rank > max_rank) {
                    max_rank = edges[slots[k]].rank;
                }
            }
            Qef q;
            qef_zero(q);
            for (int k = 0; k < ne; ++k) {
                if (slots[k] < 0 || !edges[slots[k]].exists) continue;
                const EdgeRec& es = edges[slots[k]];
                if (es.rank == max_rank) {
                    q.mass[0] += es.q.mass[0] / es.q.mass[3];
                    q.mass[1] += es.q.mass[1] / es.q.mass[3];
                    q.mass[2] += es.q.mass[2] / es.q.mass[3];
                    q.mass[3] += 1.0;
                }
            }
            for (int k = 0; k < ne; ++k) {
                if (slots[k] < 0 || !edges[slots[k]].exists) continue;
                qef_add(q, edges[slots[k]].q);
            }
            double v[3];
            int rank = 0;
            qef_vertex(q, v, &rank);
            for (int k = 0; k < 3; ++k) L.vert[patch][k] = v[k];
            if (patch == np - 1) {
                for (int k = 0; k < 4; ++k) L.mass[k] = q.mass[k];
                for (int k = 0; k < 6; ++k) L.ata[k] = q.ata[k];
                for (int k = 0; k < 3; ++k) L.atb[k] = q.atb[k];
                L.btb = q.btb;
                L.rank = static_cast<uint8_t>(rank);
            }
        }
    }
}

}  // namespace lfb

namespace lfb {

////////////////////////////////////////////////////////////////////////////////
// 3. Bottom-up collapse (DCTree::collectChildren, dc_tree.inl:581-735)

struct CollapseArgs {
    Octree o;
    DevTape bt;
    const RegClause* arena;
    LeafRec* recs;
    uint32_t* rec_top;
    uint32_t rec_cap;
    uint32_t* status;
    double max_err;
};

__device__ __forceinline__ uint8_t corner_state(uint8_t type, const LeafRec* r,
                                                int corner)
{
    if (type == CELL_LEAF) {
        return ((r->corner_mask >> corner) & 1) ? CELL_FILLED : CELL_EMPTY;
    }
    return type;
}

/// Serial value evaluation of one point by one thread (registers in R with
/// stride B), used for the collapse test at a candidate vertex.
__device__ float thread_value(const DevTape& bt, const RegClause* cl,
                              uint32_t len, float* R, int tid, int B, float x,
                              float y, float z)
{
    R[0 * B + tid] = x;
    R[1 * B + tid] = y;
    R[2 * B + tid] = z;
    for (uint32_t c = 0; c < len; ++c) {
        const uint2 raw = __ldg(reinterpret_cast<const uint2*>(cl + c));
        const uint8_t o = raw.x & 0xff;
        const uint8_t kinds = (raw.x >> 8) & 0xff;
        const uint16_t ra = raw.y & 0xffff, rb = raw.y >> 16;
        const float a = (kinds & 3) == OPND_REG ? R[ra * B + tid] : __ldg(bt.cpool + ra);
        const float b = ((kinds >> 2) & 3) == OPND_REG ? R[rb * B + tid] : __ldg(bt.cpool + rb);
        R[(raw.x >> 16) * B + tid] = dv_value(o, a, b);
    }
    return bt.root_kind == OPND_REG ? R[bt.root * B + tid] : __ldg(bt.cpool + bt.root);
}

__global__ void __launch_bounds__(128)
k_collapse_level(CollapseArgs A, int d)
{
    extern __shared__ float csmem[];
    const int B = blockDim.x, tid = threadIdx.x;
    const Octree& o = A.o;
    const LevelView& lv = o.lv[d];
    const uint32_t i = blockIdx.x * B + tid;
    if (i >= lv.n_cells || lv.type[i] != CELL_BRANCH) return;

    const LevelView& cv = o.lv[d + 1];
    const uint32_t k = static_cast<uint32_t>(lv.child_group[i]);
    uint8_t ct[8];
    const LeafRec* cr[8];
    bool any_branch = false, all_empty = true, all_filled = true;
    for (int j = 0; j < 8; ++j) {
        ct[j] = cv.type[8 * k + j];
        const int32_t r = cv.rec[8 * k + j];
        cr[j] = (ct[j] == CELL_LEAF && r >= 0) ? &A.recs[r] : nullptr;
        any_branch |= ct[j] == CELL_BRANCH;
        all_empty &= ct[j] == CELL_EMPTY;
        all_filled &= ct[j] == CELL_FILLED;
    }
    if (any_branch) return;
    if (all_empty || all_filled) {
        lv.type[i] = all_empty ? CELL_EMPTY : CELL_FILLED;
        return;
    }
    auto cs = [&](int child, int corner) { return corner_state(ct[child], cr[child], corner); };
    uint8_t corners[8];
    uint8_t mask = 0;
    for (int j = 0; j < 8; ++j) {
        corners[j] = cs(j, j);
        mask |= (corners[j] == CELL_FILLED ? 1 : 0) << j;
    }
    bool manifold = c_tab.manifold[mask];
    for (int j = 0; j < 8 && manifold; ++j) {
        if (ct[j] == CELL_LEAF) manifold = cr[j]->manifold;
    }
    if (manifold) {
        // Ju et al. 2002 sign checks at coarse edge, face and cube centres
        // (dc_tree3.cpp:16-109): the child at corner a holds the midpoint of
        // the coarse edge a -> a|bit as its corner a|bit.
        for (int a = 0; a < 8 && manifold; ++a) {
            for (int bit = 1; bit < 8 && manifold; bit <<= 1) {
                if (a & bit) continue;
                const uint8_t m = cs(a, a | bit);
                manifold = (m == corners[a] || m == corners[a | bit]);
            }
        }
        const int faces[6][5] = {
            {0, 5, 0, 1, 4}, {0, 6, 0, 2, 4}, {0, 3, 0, 2, 1},
            {7, 1, 1, 5, 3}, {7, 2, 2, 6, 3}, {7, 4, 4, 6, 5}};
        for (int f = 0; f < 6 && manifold; ++f) {
            const uint8_t m = cs(faces[f][0], faces[f][1]);
            const int c3 = faces[f][0] == 0 ? faces[f][1] : 7;
            manifold = m == corners[faces[f][2]] || m == corners[faces[f][3]] ||
                       m == corners[faces[f][4]] || m == corners[c3];
        }
        if (manifold) {
            const uint8_t m = cs(0, 7);
            bool ok = false;
            for (int j = 0; j < 8; ++j) ok |= m == corners[j];
            manifold = ok;
        }
    }
    if (!manifold) return;

    unsigned rank = 0;
    for (int j = 0; j < 8; ++j) {
        if (cr[j] && cr[j]->rank > rank) rank = cr[j]->rank;
    }
    Qef q;
    qef_zero(q);
    for (int j = 0; j < 8; ++j) {
        if (!cr[j]) continue;
        if (cr[j]->rank == rank) {
            for (int t = 0; t < 4; ++t) q.mass[t] += cr[j]->mass[t];
        }
        for (int t = 0; t < 6; ++t) q.ata[t] += cr[j]->ata[t];
        for (int t = 0; t < 3; ++t) q.atb[t] += cr[j]->atb[t];
        q.btb += cr[j]->btb;
    }
    double v[3];
    const double err = qef_vertex(q, v, nullptr);
    double lo[3], hi[3];
    cell_bounds(o, d, lv.coords[i], lo, hi);
    bool inside = true;
    for (int a = 0; a < 3; ++a) {
        inside &= (v[a] >= lo[a] - 1e-6) && (v[a] <= hi[a] + 1e-6);
    }
    if (!(err < A.max_err) || !inside) return;

    // Value at the vertex with a tape that is valid there: walk up from this
    // cell to the first ancestor whose (float) box contains the point
    // (Tape::getBase, tape.cpp:188-209); the unpruned tape otherwise.  Any
    // tape valid at the point gives the same value, so when this cell
    // contains the vertex, the shortest one is taken instead: that of the
    // deepest cell below it that contains the vertex and was ambiguous when
    // its interval was evaluated (so has a pruned tape).
    const float vf[3] = {static_cast<float>(v[0]), static_cast<float>(v[1]),
                         static_cast<float>(v[2])};
    auto contains = [&](int dd, uint32_t ii) {
        double blo[3], bhi[3];
        cell_bounds(o, dd, o.lv[dd].coords[ii], blo, bhi);
        bool in = true;
        for (int a = 0; a < 3; ++a) {
            in &= vf[a] >= static_cast<float>(blo[a]) && vf[a] <= static_cast<float>(bhi[a]);
        }
        return in;
    };
    TapeRef tr = root_tape_ref(A.bt);
    if (contains(d, i)) {
        int dd = d;
        uint32_t ii = i;
        while (dd + 1 < o.levels) {
            const int32_t k = o.lv[dd].child_group[ii];
            if (k < 0) break;
            bool found = false;
            for (uint32_t j = 0; j < 8 && !found; ++j) {
                const uint32_t c = 8 * static_cast<uint32_t>(k) + j;
                if (o.lv[dd + 1].child_group[c] >= 0 && contains(dd + 1, c)) {
                    ii = c;
                    found = true;
                }
            }
            if (!found) break;
            ++dd;
        }
        tr = o.lv[dd].cell_tape[ii];
    } else {
        int dd = d;
        uint32_t ii = i;
        while (dd > 0) {
            ii = o.lv[dd].group_parent[ii >> 3];
            --dd;
            if (contains(dd, ii)) {
                tr = o.lv[dd].cell_tape[ii];
                break;
            }
        }
    }
    const float value = thread_value(with_tape(A.bt, tr), A.arena + tr.off, tr.len, csmem, tid, B,
                                     vf[0], vf[1], vf[2]);
    if (!(fabsf(value) < A.max_err)) return;

    const uint32_t r = atomicAdd(A.rec_top, 1u);
    if (r >= A.rec_cap) {
        atomicOr(A.status, ST_RECORD_OVERFLOW);
        return;
    }
    LeafRec& L = A.recs[r];
    for (int t = 0; t < 3; ++t) L.vert[0][t] = v[t];
    for (int t = 0; t < 4; ++t) L.mass[t] = q.mass[t];
    for (int t = 0; t < 6; ++t) L.ata[t] = q.ata[t];
    for (int t = 0; t < 3; ++t) L.atb[t] = q.atb[t];
    L.btb = q.btb;
    L.level = o.levels - d;
    L.corner_mask = mask;
    L.vertex_count = 1;
    L.rank = static_cast<uint8_t>(rank);
    L.manifold = 1;
    lv.rec[i] = static_cast<int32_t>(r);
    lv.type[i] = CELL_LEAF;
}

////////////////////////////////////////////////////////////////////////////////
// 4. Dual walk (Dual<3>::work / face3 / edge3, dual.hpp:126-203) and
//    DCMesher::load (dc_mesher.cpp:18-169)

enum : uint8_t { TASK_CELL = 0, TASK_FACE = 1, TASK_EDGE = 2 };

struct DualTask {
    uint8_t kind;
    uint8_t axis;   // 1, 2, 4
    uint8_t pad[2];
    uint32_t ref[4];
};

__device__ __forceinline__ uint32_t make_ref(int depth, uint32_t idx)
{
    return (static_cast<uint32_t>(depth) << 27) | idx;
}
__device__ __forceinline__ int ref_depth(uint32_t r) { return r >> 27; }
__device__ __forceinline__ uint32_t ref_idx(uint32_t r) { return r & 0x7ffffff; }

__device__ __forceinline__ int axis_q(int a) { return a == 1 ? 2 : a == 2 ? 4 : 1; }
__device__ __forceinline__ int axis_r(int a) { return a == 1 ? 4 : a == 2 ? 1 : 2; }

struct DualArgs {
    Octree o;
    const LeafRec* recs;
    uint32_t* status;
    DualTask* out;
    uint32_t* n_out;
    uint32_t out_cap;
    uint32_t* tris;      // 3 vertex keys per triangle (record * 4 + vertex)
    uint32_t* n_tris;
    uint32_t tri_cap;
    uint8_t* used;       // per vertex key
};

__device__ __forceinline__ uint8_t ref_type(const Octree& o, uint32_t r)
{
    return o.lv[ref_depth(r)].type[ref_idx(r)];
}

__device__ __forceinline__ uint32_t ref_child(const Octree& o, uint32_t r, int k)
{
    const int d = ref_depth(r);
    const uint32_t i = ref_idx(r);
    if (o.lv[d].type[i] != CELL_BRANCH) return r;
    return make_ref(d + 1, 8u * static_cast<uint32_t>(o.lv[d].child_group[i]) + k);
}

__device__ __forceinline__ void push_task(const DualArgs& A, uint8_t kind,
                                          uint8_t axis, const uint32_t* refs,
                                          int nref)
{
    // A task holding an EMPTY / FILLED leaf can never produce a face: that
    // leaf stays in every task derived from it and DCMesher::load exits on
    // it (dc_mesher.cpp:23-28).
    bool branch = false;
    for (int k = 0; k < nref; ++k) {
        const uint8_t t = ref_type(A.o, refs[k]);
        if (t == CELL_EMPTY || t == CELL_FILLED) return;
        branch |= t == CELL_BRANCH;
    }
    if (kind == TASK_FACE && !branch) return;
    const uint32_t slot = atomicAdd(A.n_out, 1u);
    if (slot >= A.out_cap) {
        atomicOr(A.status, ST_QUEUE_OVERFLOW);
        return;
    }
    DualTask t;
    t.kind = kind;
    t.axis = axis;
    t.pad[0] = t.pad[1] = 0;
    for (int k = 0; k < 4; ++k) t.ref[k] = k < nref ? refs[k] : 0;
    A.out[slot] = t;
}

__device__ void emit_edge(const DualArgs& A, int ax, const uint32_t ts[4])
{
    const Octree& o = A.o;
    const LeafRec* R[4];
    int32_t ri[4];
    for (int k = 0; k < 4; ++k) {
        ri[k] = o.lv[ref_depth(ts[k])].rec[ref_idx(ts[k])];
        if (ri[k] < 0) return;
        R[k] = &A.recs[ri[k]];
    }
    int index = 0;
    for (int k = 1; k < 4; ++k) {
        if (R[k]->level < R[index]->level) index = k;
    }
    const int Q = axis_q(ax), Rr = axis_r(ax);
    const int corners[4] = {Q | Rr, Rr, Q, 0};
    const int ca = (R[index]->corner_mask >> corners[index]) & 1;
    const int cb = (R[index]->corner_mask >> (corners[index] | ax)) & 1;
    if (ca == cb) return;
    const bool D = ca != 0;   // a is FILLED
    const int ev[4][2] = {{Q | Rr, Q | Rr | ax}, {Rr, Rr | ax}, {Q, Q | ax}, {0, ax}};
    uint32_t vs[4];
    float P[4][3];
    for (int k = 0; k < 4; ++k) {
        const int e = D ? c_tab.e[ev[k][0]][ev[k][1]] : c_tab.e[ev[k][1]][ev[k][0]];
        const int vi = R[k]->level > 0 ? 0 : c_tab.p[R[k]->corner_mask][e];
        vs[k] = static_cast<uint32_t>(ri[k]) * 4u + static_cast<uint32_t>(vi < 0 ? 0 : vi);
        for (int t = 0; t < 3; ++t) P[k][t] = static_cast<float>(R[k]->vert[vi < 0 ? 0 : vi][t]);
    }
    if (!D) {
        const uint32_t tv = vs[1]; vs[1] = vs[2]; vs[2] = tv;
        for (int t = 0; t < 3; ++t) {
            const float tp = P[1][t]; P[1][t] = P[2][t]; P[2][t] = tp;
        }
    }
    float N[4][3];
    auto save_norm = [&](int a, int b, int c) {
        const float u[3] = {__fsub_rn(P[b][0], P[a][0]), __fsub_rn(P[b][1], P[a][1]),
                            __fsub_rn(P[b][2], P[a][2])};
        const float w[3] = {__fsub_rn(P[c][0], P[a][0]), __fsub_rn(P[c][1], P[a][1]),
                            __fsub_rn(P[c][2], P[a][2])};
        float n[3] = {__fsub_rn(__fmul_rn(u[1], w[2]), __fmul_rn(u[2], w[1])),
                      __fsub_rn(__fmul_rn(u[2], w[0]), __fmul_rn(u[0], w[2])),
                      __fsub_rn(__fmul_rn(u[0], w[1]), __fmul_rn(u[1], w[0]))};
        const float z = __fadd_rn(__fadd_rn(__fmul_rn(n[0], n[0]), __fmul_rn(n[1], n[1])),
                                  __fmul_rn(n[2], n[2]));
        if (z > 0) {
            const float s = __fsqrt_rn(z);
            n[0] = __fdiv_rn(n[0], s);
            n[1] = __fdiv_rn(n[1], s);
            n[2] = __fdiv_rn(n[2], s);
        }
        N[a][0] = n[0]; N[a][1] = n[1]; N[a][2] = n[2];
    };
    save_norm(0, 1, 2);
    save_norm(1, 3, 0);
    save_norm(2, 0, 3);
    save_norm(3, 2, 1);
    auto dot = [](const float* a, const float* b) {
        return __fadd_rn(__fadd_rn(__fmul_rn(a[0], b[0]), __fmul_rn(a[1], b[1])),
                         __fmul_rn(a[2], b[2]));
    };
    uint32_t tri[2][3];
    if (dot(N[0], N[3]) > dot(N[1], N[2])) {
        tri[0][0] = vs[0]; tri[0][1] = vs[1]; tri[0][2] = vs[2];
        tri[1][0] = vs[2]; tri[1][1] = vs[1]; tri[1][2] = vs[3];
    } else {
        tri[0][0] = vs[0]; tri[0][1] = vs[1]; tri[0][2] = vs[3];
        tri[1][0] = vs[0]; tri[1][1] = vs[3]; tri[1][2] = vs[2];
    }
    for (int t = 0; t < 2; ++t) {
        const uint32_t a = tri[t][0], b = tri[t][1], c = tri[t][2];
        if (a == b || b == c || a == c) continue;
        const uint32_t slot = atomicAdd(A.n_tris, 1u);
        if (slot >= A.tri_cap) {
            atomicOr(A.status, ST_QUEUE_OVERFLOW);
            return;
        }
        A.tris[3 * slot + 0] = a;
        A.tris[3 * slot + 1] = b;
        A.tris[3 * slot + 2] = c;
        A.used[a] = 1;
        A.used[b] = 1;
        A.used[c] = 1;
    }
}

__device__ __forceinline__ void dual_task(const DualArgs& A, const DualTask& task)
{
    const Octree& o = A.o;
    const int ax = task.axis;
    if (task.kind == TASK_CELL) {
        const uint32_t c = task.ref[0];
        uint32_t ch[8];
        for (int k = 0; k < 8; ++k) ch[k] = ref_child(o, c, k);
        for (int k = 0; k < 8; ++k) {
            if (ref_type(o, ch[k]) == CELL_BRANCH) {
                push_task(A, TASK_CELL, 0, &ch[k], 1);
            }
        }
        for (int a = 1; a <= 4; a <<= 1) {
            const int q = axis_q(a), r = axis_r(a);
            const int pairs[4][2] = {{0, a}, {q, q | a}, {r, r | a}, {q | r, q | r | a}};
            for (int p = 0; p < 4; ++p) {
                const uint32_t f[2] = {ch[pairs[p][0]], ch[pairs[p][1]]};
                push_task(A, TASK_FACE, static_cast<uint8_t>(a), f, 2);
            }
        }
        for (int a = 1; a <= 4; a <<= 1) {
            const int q = axis_q(a), r = axis_r(a);
            for (int s = 0; s < 2; ++s) {
                const int b = s ? a : 0;
                const uint32_t e[4] = {ch[b], ch[q | b], ch[r | b], ch[q | r | b]};
                push_task(A, TASK_EDGE, static_cast<uint8_t>(a), e, 4);
            }
        }
    } else if (task.kind == TASK_FACE) {
        const uint32_t t0 = task.ref[0], t1 = task.ref[1];
        const int Q = axis_q(ax), R = axis_r(ax);
        const int ks[4] = {0, Q, R, Q | R};
        for (int k = 0; k < 4; ++k) {
            const uint32_t f[2] = {ref_child(o, t0, ks[k] | ax), ref_child(o, t1, ks[k])};
            push_task(A, TASK_FACE, static_cast<uint8_t>(ax), f, 2);
        }
        const uint32_t e0[4] = {ref_child(o, t0, ax), ref_child(o, t0, R | ax),
                                ref_child(o, t1, 0), ref_child(o, t1, R)};
        push_task(A, TASK_EDGE, static_cast<uint8_t>(Q), e0, 4);
        const uint32_t e1[4] = {ref_child(o, t0, Q | ax), ref_child(o, t0, Q | R | ax),
                                ref_child(o, t1, Q), ref_child(o, t1, Q | R)};
        push_task(A, TASK_EDGE, static_cast<uint8_t>(Q), e1, 4);
        const uint32_t e2[4] = {ref_child(o, t0, ax), ref_child(o, t1, 0),
                                ref_child(o, t0, ax | Q), ref_child(o, t1, Q)};
        push_task(A, TASK_EDGE, static_cast<uint8_t>(R), e2, 4);
        const uint32_t e3[4] = {ref_child(o, t0, R | ax), ref_child(o, t1, R),
                                ref_child(o, t0, R | ax | Q), ref_child(o, t1, R | Q)};
        push_task(A, TASK_EDGE, static_cast<uint8_t>(R), e3, 4);
    } else {
        bool branch = false;
        for (int k = 0; k < 4; ++k) branch |= ref_type(o, task.ref[k]) == CELL_BRANCH;
        if (!branch) {
            emit_edge(A, ax, task.ref);
            return;
        }
        const int Q = axis_q(ax), R = axis_r(ax);
        const uint32_t a[4] = {ref_child(o, task.ref[0], Q | R), ref_child(o, task.ref[1], R),
                               ref_child(o, task.ref[2], Q), ref_child(o, task.ref[3], 0)};
        push_task(A, TASK_EDGE, static_cast<uint8_t>(ax), a, 4);
        const uint32_t b[4] = {ref_child(o, task.ref[0], Q | R | ax),
                               ref_child(o, task.ref[1], R | ax),
                               ref_child(o, task.ref[2], Q | ax),
                               ref_child(o, task.ref[3], ax)};
        push_task(A, TASK_EDGE, static_cast<uint8_t>(ax), b, 4);
    }
}

/// One round: the tasks that the round before it left (n_in; null: the root
/// cell), however many those are, so that the host need not wait between
/// rounds.
__global__ void __launch_bounds__(128)
k_dual_round(const __grid_constant__ DualArgs A, const DualTask* in, const uint32_t* n_in)
{
    const uint32_t n = n_in ? min(*n_in, A.out_cap) : 1u;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        DualTask task{};   // the root cell
        if (n_in) task = in[t];
        dual_task(A, task);
    }
}

////////////////////////////////////////////////////////////////////////////////
// Small helpers for the host driver

/// Sort keys for the leaf groups: tape length (longest first), so that the
/// persistent leaf kernel starts the expensive groups early.
__global__ void k_leaf_order_keys(const TapeRef* group_tape, uint32_t n,
                                  uint32_t* keys, uint32_t* vals)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    keys[i] = group_tape[i].len;
    vals[i] = i;
}

/// What the kernels of one mesh count on the device, read back as a whole.
struct MeshCounters {
    uint32_t status;
    uint32_t n_recs;
    unsigned long long arena_top;
    unsigned long long evals[2];
    unsigned long long edge_top;
    // zeroed before every octree level
    unsigned long long list_top;
    uint32_t next_cell;
    uint32_t n_groups;       // branch cells of the level
    uint32_t nregs;          // largest register count of their tapes
    uint32_t pad;
    // clauses of their tapes (the last level's): of up to 8 registers, of
    // 9 to 16 and of more
    unsigned long long clauses[3];
    // leaf stage
    uint32_t next_group, next_group2;
    uint32_t zero_top, n_redo;
    uint32_t next_redo[2];
    // dual walk
    uint32_t n_tris;
    uint32_t n_verts;
    uint32_t n_tasks[kMaxLevels + 8];   // by round
};
constexpr size_t kLevelCounters = offsetof(MeshCounters, next_group) - offsetof(MeshCounters, list_top);

__global__ void k_init_root(Octree o, MeshCounters* c, uint32_t n_clauses)
{
    o.lv[0].coords[0] = 0;
    o.lv[0].rec[0] = -1;
    o.lv[0].child_group[0] = -1;
    c->arena_top = n_clauses;
}

/// Flags of the branch cells (flags[n] = 0), how many there are and the
/// largest register count of their tapes (which sizes the group-mode
/// interval kernel's shared memory for the next depth); of the last level
/// also their clauses by register count (which size the leaf kernel's).
__global__ void k_branch_flags(const uint8_t* type, const TapeRef* cell_tape, uint32_t n,
                               uint32_t* flags, MeshCounters* c, bool last)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool branch = i < n && type[i] == CELL_BRANCH;
    if (i <= n) flags[i] = branch ? 1u : 0u;
    const uint32_t count = __popc(__ballot_sync(0xffffffffu, branch));
    const uint32_t nregs = branch ? cell_tape[i].nregs : 0u;
    const uint32_t most = __reduce_max_sync(0xffffffffu, nregs);
    if (last) {
        __shared__ unsigned long long sums[3];
        if (threadIdx.x < 3) sums[threadIdx.x] = 0;
        __syncthreads();
        if (branch) {
            atomicAdd(sums + (nregs <= kLeafSmemRegsMany ? 0 : nregs <= kLeafSmemRegs ? 1 : 2),
                      static_cast<unsigned long long>(cell_tape[i].len));
        }
        __syncthreads();
        if (threadIdx.x < 3 && sums[threadIdx.x]) atomicAdd(c->clauses + threadIdx.x, sums[threadIdx.x]);
    }
    if ((threadIdx.x & 31) == 0 && count) {
        atomicAdd(&c->n_groups, count);
        atomicMax(&c->nregs, most);
    }
}

/// For each branch cell at depth d: its group index at d + 1, and the
/// group's parent, tapes and child coordinates.
__global__ void k_build_groups(Octree o, int d, const uint32_t* scan)
{
    const LevelView& lv = o.lv[d];
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= lv.n_cells) return;
    if (lv.type[i] != CELL_BRANCH) {
        lv.child_group[i] = -1;
        return;
    }
    const uint32_t g = scan[i];
    lv.child_group[i] = static_cast<int32_t>(g);
    const LevelView& nv = o.lv[d + 1];
    nv.group_parent[g] = i;
    nv.group_tape[g] = lv.cell_tape[i];
    nv.group_list[g] = lv.cell_list[i];
    uint32_t x, y, z;
    unpack_coords(lv.coords[i], x, y, z);
    for (int k = 0; k < 8; ++k) {
        nv.coords[8 * g + k] = pack_coords(2 * x + (k & 1), 2 * y + ((k >> 1) & 1),
                                           2 * z + ((k >> 2) & 1));
        nv.rec[8 * g + k] = -1;
    }
}

__global__ void k_vertex_ids(const uint8_t* used, const uint32_t* scan,
                             uint32_t n_keys, const LeafRec* recs,
                             float* verts)
{
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n_keys || !used[k]) return;
    const LeafRec& r = recs[k >> 2];
    const uint32_t id = scan[k] + 1;   // index 0 is the placeholder vertex
    for (int t = 0; t < 3; ++t) verts[3 * id + t] = static_cast<float>(r.vert[k & 3][t]);
}

__global__ void k_u8_to_u32(const uint8_t* in, uint32_t* out, uint32_t n)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = in[i];
}

__global__ void k_remap_tris(uint32_t* tris, uint32_t n, const uint32_t* scan)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 3 * n) tris[i] = scan[tris[i]] + 1;
}

// Binary STL records (mesh.cpp:177-193): per triangle a zero normal, its
// three vertices and a zero attribute word, 50 bytes, little-endian like
// the host.  50-byte records are only 2-byte aligned, so a block packs its
// kStlBlock records in shared memory as 16-bit words and writes them out as
// one contiguous run of words.
constexpr uint32_t kStlBlock = 128;
constexpr uint32_t kStlWords = 25;

__global__ void __launch_bounds__(kStlBlock)
k_pack_stl(const float* __restrict__ verts, const uint32_t* __restrict__ tris, uint32_t n,
           uint16_t* __restrict__ out)
{
    __shared__ uint16_t rec[kStlBlock * kStlWords];
    const uint32_t first = blockIdx.x * kStlBlock;
    const uint32_t i = first + threadIdx.x;
    uint16_t* r = rec + threadIdx.x * kStlWords;
    if (i < n) {
        for (int k = 0; k < 6; ++k) r[k] = 0;
        for (int v = 0; v < 3; ++v) {
            const uint32_t id = tris[3 * static_cast<size_t>(i) + v];
            for (int a = 0; a < 3; ++a) {
                const uint32_t bits = __float_as_uint(verts[3 * static_cast<size_t>(id) + a]);
                r[6 + 6 * v + 2 * a] = static_cast<uint16_t>(bits & 0xffff);
                r[6 + 6 * v + 2 * a + 1] = static_cast<uint16_t>(bits >> 16);
            }
        }
        r[24] = 0;
    }
    __syncthreads();
    const uint32_t m = min(kStlBlock, n - first);
    uint16_t* dst = out + static_cast<size_t>(first) * kStlWords;
    for (uint32_t k = threadIdx.x; k < m * kStlWords; k += kStlBlock) dst[k] = rec[k];
}

// libfive_mesh_coords' index list (libfive.cpp:375-388): a, b, c, -1 per
// triangle.
__global__ void k_pack_coords(const uint32_t* __restrict__ tris, uint32_t n, int4* __restrict__ out)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const size_t t = 3 * static_cast<size_t>(i);
        out[i] = make_int4(static_cast<int>(tris[t]), static_cast<int>(tris[t + 1]),
                           static_cast<int>(tris[t + 2]), -1);
    }
}

}  // namespace lfb

////////////////////////////////////////////////////////////////////////////////
// Host driver

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <vector>

#include "mesher.hpp"

namespace lfb {

namespace {

/// What one mesh in flight owns on the host side: grow-only device buffers
/// keyed by purpose, the stream its work runs on and download()'s
/// page-locked staging buffer.  A context serves one mesh at a time (its
/// mutex) and keeps its buffers from call to call.
/// Freed scratch the device's memory pool keeps across synchronisations
/// (for the next mesh of any context) before it returns memory to the driver.
constexpr uint64_t kPoolKeepBytes = uint64_t(32) << 30;

struct Workspace {
    std::mutex mu;
    cudaStream_t s = 0;
    std::map<int, DevBuf> bufs;
    void* pinned = nullptr;
    size_t pinned_bytes = 0;
    MeshCounters* seen = nullptr;   // page-locked: the counters as last read
    // The mesh is rendered again after the device ran out of memory: it does
    // without what it can do without.
    bool lean = false;
    // Leaf edge records per leaf group (grows when a mesh needs more; the
    // mesh is then rendered again).
    uint32_t edges_per_group = 16;
    bool retry = false;

    template <class T>
    T* get(int key, size_t count)
    {
        DevBuf& b = bufs[key];
        if (!b.ordered) {
            // scratch lives in the device's memory pool, allocated in this
            // context's stream order
            b.ordered = true;
            b.stream = s;
        }
        if (!b.reserve(std::max<size_t>(count, 1) * sizeof(T))) return nullptr;
        return b.as<T>();
    }
};

/// The context of single-mesh calls: work on the legacy default stream, as
/// callers that time those calls with events on that stream expect.
Workspace& default_workspace()
{
    static Workspace* w = new Workspace;   // never destroyed: see pinned_pool()
    return *w;
}

/// Context k of the concurrent batch path, created on first use with its
/// own non-blocking stream (so that batched meshes overlap each other and
/// never wait on unrelated default-stream work).
struct StreamPool {
    std::mutex mu;
    std::vector<Workspace*> pool;
};

StreamPool& stream_pool()
{
    static StreamPool* p = new StreamPool;   // never destroyed, like the contexts
    return *p;
}

Workspace* stream_workspace(unsigned k)
{
    auto& sp = stream_pool();
    std::lock_guard<std::mutex> lock(sp.mu);
    auto& pool = sp.pool;
    while (pool.size() <= k) {
        auto* w = new Workspace;
        if (!cuda_ok(cudaStreamCreateWithFlags(&w->s, cudaStreamNonBlocking), "stream")) {
            delete w;
            return nullptr;
        }
        pool.push_back(w);
    }
    return pool[k];
}

enum BufKey {
    K_ARENA = 1, K_COUNTERS, K_RECS, K_FLAGS, K_SCAN,
    K_CUBTMP, K_TASK_A, K_TASK_B, K_TRIS, K_USED, K_VSCAN, K_VERTS, K_FEAT,
    K_LIST_A, K_LIST_B, K_WIDE_S, K_WIDE_SN, K_WIDE_P, K_WIDE_LIVE, K_WIDE_NEW,
    K_WIDE_ST2, K_WIDE_L1, K_WIDE_WL, K_LEAF_RD, K_ORDER_K0, K_ORDER_K1,
    K_ORDER_V0, K_ORDER_V1, K_SORTTMP, K_GDEC, K_GLAST, K_FEATWS,
    K_EDGES, K_GEDGES, K_RECGROUP, K_STL, K_COORDS, K_ZEROS, K_REDO,
    K_VOPS, K_NSTEPS, K_ROOTTAPE,
    K_LEVEL = 100,
};

bool upload_tables()
{
    static std::mutex mu;
    static bool ready = false;
    std::lock_guard<std::mutex> lock(mu);
    if (ready) return true;
    static DcTables t;
    build_dc_tables(t);
    if (!cuda_ok(cudaMemcpyToSymbol(c_tab, &t, sizeof(t)), "dc tables") ||
        !uploaded("dc tables")) {
        return false;
    }
    ready = true;
    return true;
}

int level_from_resolution(const double lo[3], const double hi[3], double min_feature)
{
    // Region::withResolution (region.hpp:226-231), including its float logf.
    double md = hi[0] - lo[0];
    for (int a = 1; a < 3; ++a) md = std::min(md, hi[a] - lo[a]);
    const float l = std::ceil(std::fmax(0.0f, logf(static_cast<float>(md / min_feature))) /
                              logf(2.0f));
    return static_cast<int>(l);
}

/// Cells per level up to which a whole block works on each cell
/// (kBlockModeCells; LFB_BLOCK_MODE_CELLS overrides it, for the parity tests).
uint32_t block_mode_cells()
{
    static const long v = [] {
        const char* e = std::getenv("LFB_BLOCK_MODE_CELLS");
        return e ? std::max(0L, std::atol(e)) : static_cast<long>(kBlockModeCells);
    }();
    return static_cast<uint32_t>(v);
}

/// Cells per level from which the interval stage switches to group mode
/// (kGroupModeCells; the LFB_GROUP_MODE_CELLS environment variable overrides
/// it, which the parity tests use to run both modes on small shapes).
uint32_t group_mode_cells()
{
    static const uint32_t v = [] {
        const char* e = std::getenv("LFB_GROUP_MODE_CELLS");
        return e ? static_cast<uint32_t>(std::max(1L, std::atol(e))) : kGroupModeCells;
    }();
    return v;
}

bool debug_levels()
{
    static const bool on = [] {
        const char* e = std::getenv("LFB_DEBUG_LEVELS");
        return e && e[0] == '1';
    }();
    return on;
}

}  // namespace

namespace {

/// Entries whose state fits the shared memory of a block when `per_sm`
/// blocks share an SM, and the bytes that takes.
uint32_t block_slots(uint32_t n, uint32_t per_sm)
{
    return std::min<uint32_t>((n + 3) / 4 * 4, (216u * 1024 / per_sm - 2048) / 11 / 4 * 4);
}
size_t block_smem(uint32_t slots) { return (11 * static_cast<size_t>(slots) + 27 + 15) / 16 * 16; }

}  // namespace

uint32_t interval_box_slots(uint32_t n, uint32_t n_boxes)
{
    // Two blocks an SM when a list's state then still fits, else one.
    const uint32_t sms = static_cast<uint32_t>(device_sm_count());
    return std::min(n_boxes, block_slots(n, 2) >= n ? 2 * sms : sms);
}

cudaError_t launch_interval_boxes(const WideArgs& W, uint32_t slots, cudaStream_t s)
{
    const uint32_t per_sm = block_slots(W.n, 2) >= W.n ? 2 : 1;
    const uint32_t n_slots = block_slots(W.n, per_sm);
    const size_t smem = block_smem(n_slots);
    auto* kernel = per_sm == 2 ? k_interval_block<true, 2> : k_interval_block<true, 1>;
    if (!raise_smem_limit(reinterpret_cast<const void*>(kernel), smem)) {
        return cudaErrorInvalidValue;
    }
    kernel<<<std::max<uint32_t>(slots, 1), kBlockThreads, smem, s>>>(W, 0, n_slots);
    return cudaGetLastError();
}

cudaError_t launch_interval_lists(const WideArgs& W, int d, uint32_t n_cells, uint32_t scratch_warps,
                                  cudaStream_t s)
{
    if (n_cells <= block_mode_cells()) {
        // Shared memory for the longest list a cell of this level can have
        // up to a whole SM's, half of it where there are more cells than SMs
        // (their lists are pruned): two blocks then share an SM.
        const uint32_t sms = static_cast<uint32_t>(device_sm_count());
        const uint32_t per_sm = n_cells <= sms ? 1 : 2;
        const uint32_t slots = block_slots(W.n, per_sm);
        const size_t smem = block_smem(slots);
        if (!raise_smem_limit(reinterpret_cast<const void*>(k_interval_block<false, 2>), smem)) {
            return cudaErrorInvalidValue;
        }
        const uint32_t blocks = std::min<uint32_t>(std::min<uint32_t>(scratch_warps, sms * per_sm),
                                                   n_cells);
        k_interval_block<false, 2><<<std::max<uint32_t>(blocks, 1), kBlockThreads, smem, s>>>(W, d, slots);
    } else {
        const size_t smem = sizeof(WideSmem) * 8;
        if (!raise_smem_limit(reinterpret_cast<const void*>(k_interval_wide), smem)) {
            return cudaErrorInvalidValue;
        }
        const uint32_t warps = std::min<uint32_t>(scratch_warps, (n_cells + 7) / 8 * 8);
        k_interval_wide<<<warps / 8, 256, smem, s>>>(W, d);
    }
    return cudaGetLastError();
}

namespace {

template <class T>
bool exclusive_scan(Workspace& ws, const T* in, T* out, uint32_t n, cudaStream_t s)
{
    size_t tmp = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp, in, out, n, s);
    void* t = ws.get<unsigned char>(K_CUBTMP, tmp);
    if (!t) return false;
    return cuda_ok(cub::DeviceScan::ExclusiveSum(t, tmp, in, out, n, s), "scan");
}

}  // namespace

namespace {

/// Page-locked host blocks for mesh arrays, recycled: a mesh freed by
/// libfive_mesh_delete gives its blocks back for the next one, so a render
/// loop pins memory once and every download is a single direct copy.
struct PinnedPool {
    std::mutex mu;
    std::multimap<size_t, void*> free_blocks;   // capacity -> block
    std::map<void*, size_t> owned;              // every pool block
    size_t free_bytes = 0;
    size_t owned_bytes = 0;
    static constexpr size_t kKeepBytes = size_t(1) << 30;   // cached when free
    // Page-locked memory in use or cached at most; beyond it (many large
    // meshes alive at once) blocks are pageable, since pinning is slow and
    // takes memory from the rest of the host.
    static constexpr size_t kMaxOwned = size_t(4) << 30;
};

PinnedPool& pinned_pool()
{
    static PinnedPool* p = new PinnedPool;   // never destroyed: meshes may outlive statics
    return *p;
}

}  // namespace

void* host_alloc(size_t bytes)
{
    constexpr size_t kGrain = size_t(2) << 20;
    const size_t n = std::max<size_t>((bytes + kGrain - 1) / kGrain * kGrain, kGrain);
    auto& P = pinned_pool();
    {
        std::lock_guard<std::mutex> lock(P.mu);
        auto it = P.free_blocks.lower_bound(n);
        if (it != P.free_blocks.end() && it->first <= 2 * n) {
            void* blk = it->second;
            P.free_bytes -= it->first;
            P.free_blocks.erase(it);
            return blk;
        }
    }
    {
        std::lock_guard<std::mutex> lock(P.mu);
        if (P.owned_bytes + n > PinnedPool::kMaxOwned) {
            return std::aligned_alloc(kGrain, n);   // pageable; same interface
        }
        P.owned_bytes += n;   // reserved before the (slow) pinning call
    }
    void* blk = nullptr;
    if (cudaMallocHost(&blk, n) != cudaSuccess || !blk) {
        cudaGetLastError();
        std::lock_guard<std::mutex> lock(P.mu);
        P.owned_bytes -= n;
        return std::aligned_alloc(kGrain, n);   // pageable fallback; same interface
    }
    std::lock_guard<std::mutex> lock(P.mu);
    P.owned[blk] = n;
    return blk;
}

void host_free(void* p)
{
    if (!p) return;
    auto& P = pinned_pool();
    std::lock_guard<std::mutex> lock(P.mu);
    auto it = P.owned.find(p);
    if (it == P.owned.end()) {
        std::free(p);
        return;
    }
    P.free_blocks.emplace(it->second, p);
    P.free_bytes += it->second;
    // Keep at most kKeepBytes of idle blocks, largest first out.
    while (P.free_bytes > PinnedPool::kKeepBytes && !P.free_blocks.empty()) {
        auto last = std::prev(P.free_blocks.end());
        P.free_bytes -= last->first;
        P.owned_bytes -= last->first;
        P.owned.erase(last->second);
        cudaFreeHost(last->second);
        P.free_blocks.erase(last);
    }
}

MeshOut::~MeshOut()
{
    host_free(verts);
    host_free(tris);
    host_free(coords);
}

libfive_mesh* MeshOut::release()
{
    auto m = new libfive_mesh;
    m->verts = verts;
    m->tris = tris;
    m->vert_count = vert_count;
    m->tri_count = tri_count;
    verts = nullptr;
    tris = nullptr;
    return m;
}

namespace {

/// Device -> pageable host copy: one transfer into a pinned staging buffer
/// (grow-only, kept between calls), then a host copy split over a few
/// threads (a single thread's memcpy is the slow part of a mesh download).
/// wait = false: the caller waits for the stream when the destination is
/// page-locked.
bool download(Workspace& ws, void* dst, const void* src, size_t bytes, cudaStream_t s,
              bool wait = true)
{
    if (bytes == 0) return true;
    bool page_locked = false;
    {
        auto& P = pinned_pool();
        std::lock_guard<std::mutex> lock(P.mu);
        page_locked = P.owned.count(dst) != 0;
    }
    if (page_locked) {
        // Page-locked destination: one direct transfer.
        return cuda_ok(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), "download") &&
               (!wait || cuda_ok(cudaStreamSynchronize(s), "download"));
    }
    void*& pinned = ws.pinned;
    if (bytes > ws.pinned_bytes) {
        if (pinned) cudaFreeHost(pinned);
        pinned = nullptr;
        ws.pinned_bytes = 0;
        const size_t want = std::max<size_t>(bytes + bytes / 4, size_t(8) << 20);
        if (!cuda_ok(cudaMallocHost(&pinned, want), "pinned staging")) return false;
        ws.pinned_bytes = want;
    }
    if (!cuda_ok(cudaMemcpyAsync(pinned, src, bytes, cudaMemcpyDeviceToHost, s), "download") ||
        !cuda_ok(cudaStreamSynchronize(s), "download")) {
        return false;
    }
    host_copy(dst, pinned, bytes);
    return true;
}

}  // namespace

namespace {

/// Stage-timing events, destroyed on every way out of a render.
struct StageEvents {
    cudaEvent_t ev[5] = {};
    bool on = false;
    void create()
    {
        for (auto& e : ev) cudaEventCreate(&e);
        on = true;
    }
    ~StageEvents()
    {
        if (on) {
            for (auto& e : ev) cudaEventDestroy(e);
        }
    }
};

/// Writes the STL file of a mesh whose vertices and triangles (indices from
/// 1, vertex 0 the placeholder) are on the device: header and count, then
/// the records, packed on the device kStlChunk triangles at a time into two
/// alternating device buffers and copied into two page-locked halves, so
/// that the file write of one chunk overlaps the packing and copy of the
/// next.
int stream_stl(Workspace& ws, const char* path, const float* verts, const uint32_t* tris,
               uint32_t n_tri, cudaStream_t s, uint64_t& n_launch)
{
    constexpr uint32_t kStlChunk = 1u << 20;
    const uint32_t chunk = std::min<uint32_t>(kStlChunk, std::max<uint32_t>(n_tri, 1));
    const size_t chunk_bytes = static_cast<size_t>(chunk) * 2 * kStlWords;
    uint16_t* dev = ws.get<uint16_t>(K_STL, 2 * chunk_bytes / 2);
    if (!dev) return LFB_E_CUDA;
    if (2 * chunk_bytes > ws.pinned_bytes) {
        if (ws.pinned) cudaFreeHost(ws.pinned);
        ws.pinned = nullptr;
        ws.pinned_bytes = 0;
        if (!cuda_ok(cudaMallocHost(&ws.pinned, 2 * chunk_bytes), "pinned staging")) {
            return LFB_E_CUDA;
        }
        ws.pinned_bytes = 2 * chunk_bytes;
    }
    std::FILE* f = stl_begin(path, n_tri);
    if (!f) return set_error(LFB_E_INVALID, std::string("could not open ") + path);
    cudaEvent_t done[2];
    if (!cuda_ok(cudaEventCreateWithFlags(&done[0], cudaEventDisableTiming), "event") ||
        !cuda_ok(cudaEventCreateWithFlags(&done[1], cudaEventDisableTiming), "event")) {
        std::fclose(f);
        return LFB_E_CUDA;
    }
    int rc = 0;
    const uint32_t n_chunks = (n_tri + chunk - 1) / chunk;
    for (uint32_t k = 0; k <= n_chunks && rc == 0; ++k) {
        if (k < n_chunks) {
            const uint32_t first = k * chunk;
            const uint32_t m = std::min(chunk, n_tri - first);
            uint16_t* d = dev + (k & 1) * (chunk_bytes / 2);
            char* h = static_cast<char*>(ws.pinned) + (k & 1) * chunk_bytes;
            k_pack_stl<<<(m + kStlBlock - 1) / kStlBlock, kStlBlock, 0, s>>>(
                verts, tris + 3 * static_cast<size_t>(first), m, d);
            ++n_launch;
            if (!cuda_ok(cudaGetLastError(), "STL kernel") ||
                !cuda_ok(cudaMemcpyAsync(h, d, static_cast<size_t>(m) * 50,
                                         cudaMemcpyDeviceToHost, s), "download") ||
                !cuda_ok(cudaEventRecord(done[k & 1], s), "event")) {
                rc = LFB_E_CUDA;
            }
        }
        if (rc == 0 && k > 0) {
            // the previous chunk: wait for its copy, then write it
            const uint32_t p = k - 1;
            const char* h = static_cast<const char*>(ws.pinned) + (p & 1) * chunk_bytes;
            const size_t bytes = static_cast<size_t>(std::min(chunk, n_tri - p * chunk)) * 50;
            if (!cuda_ok(cudaEventSynchronize(done[p & 1]), "download")) {
                rc = LFB_E_CUDA;
            } else if (std::fwrite(h, 1, bytes, f) != bytes) {
                rc = set_error(LFB_E_INVALID, std::string("could not write ") + path);
            }
        }
    }
    cudaStreamSynchronize(s);
    cudaEventDestroy(done[0]);
    cudaEventDestroy(done[1]);
    if (std::fclose(f) != 0 && rc == 0) {
        rc = set_error(LFB_E_INVALID, std::string("could not write ") + path);
    }
    return rc;
}

/// One mesh in the context `ws` (held by the caller), on its stream; one
/// attempt (render_in retries when a capacity estimate was too small).
int render_once(Workspace& ws, GpuTape& g, const libfive_region3& R, double min_feature,
                double max_err, MeshOut& out, lfb_mesh_stats* stats,
                const volatile int32_t* cancel, bool first_attempt)
{
    if (!upload_tables()) return LFB_E_CUDA;
    cudaStream_t s = ws.s;
    // Cancellation (BRepSettings::cancel, polled by WorkerPool::run,
    // worker_pool.inl:105, and the dual walk, dual.hpp:315): checked at
    // every point where the host waits for the stream anyway.
    auto cancelled = [&] {
        if (cancel && *cancel) {
            cudaStreamSynchronize(s);
            set_error(LFB_E_CANCELLED, "mesh cancelled");
            return true;
        }
        return false;
    };
    if (cancelled()) return LFB_E_CANCELLED;
    const bool small = debug_hooks().small_capacity.load() != 0;
    if (small) {
        // test hook: start from empty buffers and minimal capacities
        cudaStreamSynchronize(s);
        ws.bufs.clear();
        if (first_attempt) ws.edges_per_group = 1;
    }
    const auto t_start = std::chrono::steady_clock::now();

    Octree o{};
    o.lo[0] = R.X.lower; o.hi[0] = R.X.upper;
    o.lo[1] = R.Y.lower; o.hi[1] = R.Y.upper;
    o.lo[2] = R.Z.lower; o.hi[2] = R.Z.upper;
    const int L = level_from_resolution(o.lo, o.hi, min_feature);
    if (L > kMaxLevels) {
        return set_error(LFB_E_UNSUPPORTED, "octree deeper than 24 levels");
    }
    o.levels = L;
    const DevTape bt = g.dev();
    if (bt.n_regs > 400) {
        return set_error(LFB_E_UNSUPPORTED, "tape needs more than 400 registers");
    }

    MeshCounters* counters = ws.get<MeshCounters>(K_COUNTERS, 1);
    if (!counters) return LFB_E_CUDA;
    if (!ws.seen && !cuda_ok(cudaMallocHost(reinterpret_cast<void**>(&ws.seen), sizeof(MeshCounters)),
                             "page-locked counters")) {
        return LFB_E_CUDA;
    }
    MeshCounters& seen = *ws.seen;
    cudaMemsetAsync(counters, 0, sizeof(MeshCounters), s);
    uint32_t* status = &counters->status;
    unsigned long long* edge_top = &counters->edge_top;
    unsigned long long* arena_top = &counters->arena_top;
    uint32_t* rec_top = &counters->n_recs;
    unsigned long long* evals = counters->evals;
    unsigned long long* list_top = &counters->list_top;
    // Reads the counters back; the host waits for them only where it has to
    // know them to go on.
    auto fetch_counters = [&](const char* what) {
        return cuda_ok(cudaMemcpyAsync(&seen, counters, sizeof(MeshCounters), cudaMemcpyDeviceToHost, s),
                       what);
    };
    if (!g.ensure_wide()) return LFB_E_UNSUPPORTED;

    // Register-tape arena: the unpruned tape first, pruned tapes appended
    // (every depth's tapes stay: the collapse pass evaluates points with
    // them).  It keeps its size from call to call.
    auto cap_of = [&](int key, size_t elem) {
        return static_cast<uint64_t>(ws.bufs[key].bytes / elem);
    };
    RegClause* arena = ws.get<RegClause>(
        K_ARENA, std::max<uint64_t>(cap_of(K_ARENA, sizeof(RegClause)),
                                    small ? bt.n + 64
                                          : std::max<size_t>(bt.n * 64 + (1u << 20), 1u << 22)));
    if (!arena) return LFB_E_CUDA;
    uint64_t arena_cap = cap_of(K_ARENA, sizeof(RegClause));
    if (bt.n && !cuda_ok(cudaMemcpyAsync(arena, bt.clauses, bt.n * sizeof(RegClause),
                                         cudaMemcpyDeviceToDevice, s), "arena")) {
        return LFB_E_CUDA;
    }
    auto alloc_level = [&](int d, uint32_t n_cells, uint32_t n_groups) -> bool {
        LevelView& lv = o.lv[d];
        lv.n_cells = n_cells;
        lv.n_groups = n_groups;
        const int k = K_LEVEL + 16 * d;
        lv.coords = ws.get<uint64_t>(k + 0, n_cells);
        lv.type = ws.get<uint8_t>(k + 1, n_cells);
        lv.rec = ws.get<int32_t>(k + 2, n_cells);
        lv.child_group = ws.get<int32_t>(k + 3, n_cells);
        lv.cell_tape = ws.get<TapeRef>(k + 4, n_cells);
        lv.group_parent = ws.get<uint32_t>(k + 5, n_groups);
        lv.group_tape = ws.get<TapeRef>(k + 6, n_groups);
        lv.cell_list = ws.get<ListRef>(k + 7, n_cells);
        lv.group_list = ws.get<ListRef>(k + 8, n_groups);
        if (!lv.coords || !lv.type || !lv.rec || !lv.child_group || !lv.cell_tape ||
            !lv.group_parent || !lv.group_tape || !lv.cell_list || !lv.group_list) {
            return false;
        }
        return true;
    };
    // Level 0: the root cell.
    if (!alloc_level(0, 1, 0)) return LFB_E_CUDA;
    k_init_root<<<1, 1, 0, s>>>(o, counters, bt.n);
    if (L == 0) {
        // No interval pass: the root is evaluated as a leaf right away.
        cudaMemsetAsync(o.lv[0].type, CELL_BRANCH, 1, s);
    }

    // Stage timing with CUDA events on the pipeline's stream (only when the
    // caller asks for statistics).
    StageEvents events;
    cudaEvent_t* ev = events.ev;
    if (stats) {
        events.create();
        cudaEventRecord(ev[0], s);
    }
    uint64_t n_launch = 1;   // k_init_root
    uint64_t cells_evaluated = 0;

    // Per-warp global scratch of the interval kernel (see WideArgs).
    const uint64_t n = bt.n;
    const uint64_t nw16 = (n + 15) / 16;
    const uint64_t nw1 = (nw16 + 31) / 32;
    const uint64_t per_warp = 9 * (n + 3) + 6 * n + 8 * nw16 + 4 * nw1;
    const uint64_t max_warps = static_cast<uint64_t>(device_sm_count()) * 32;
    const uint64_t budget_warps = std::max<uint64_t>(8, (768ull << 20) / std::max<uint64_t>(per_warp, 1));
    const uint32_t scratch_warps =
        static_cast<uint32_t>(std::min(max_warps, budget_warps) / 8 * 8);
    float2* wS = ws.get<float2>(K_WIDE_S, scratch_warps * (n + 3));
    uint8_t* wSN = ws.get<uint8_t>(K_WIDE_SN, scratch_warps * (n + 3));
    uint8_t* wP = ws.get<uint8_t>(K_WIDE_P, scratch_warps * n);
    uint8_t* wLive = ws.get<uint8_t>(K_WIDE_LIVE, scratch_warps * n);
    uint32_t* wNew = ws.get<uint32_t>(K_WIDE_NEW, scratch_warps * n);
    uint32_t* wSt2 = ws.get<uint32_t>(K_WIDE_ST2, scratch_warps * nw16);
    uint32_t* wL1 = ws.get<uint32_t>(K_WIDE_L1, scratch_warps * nw1);
    uint32_t* wWl = ws.get<uint32_t>(K_WIDE_WL, scratch_warps * nw16);
    if (!wS || !wSN || !wP || !wLive || !wNew || !wSt2 || !wL1 || !wWl) return LFB_E_CUDA;
    bool wide_zeroed = false;   // the state words, which k_interval_wide leaves zero
    // Two list arenas, one per parity of depth: depth d reads the lists of
    // its groups from one and writes its children's lists to the other.
    const int list_key[2] = {K_LIST_A, K_LIST_B};
    for (int k = 0; k < 2; ++k) {
        if (!ws.get<WideEntry>(list_key[k], std::max<uint64_t>(cap_of(list_key[k], sizeof(WideEntry)),
                                                                small ? 64 : 4 * n + 1024))) {
            return LFB_E_CUDA;
        }
    }

    // Deep levels (many cells, short tapes) switch to one warp per sibling
    // group over register tapes; every level below stays in that mode.
    const uint32_t group_warps = static_cast<uint32_t>(device_sm_count()) * 32;
    const uint32_t gdec_cap = std::max<uint32_t>(bt.n_choices, 1);
    uint8_t* gdec = ws.get<uint8_t>(K_GDEC, static_cast<size_t>(group_warps) * 8 * gdec_cap);
    uint8_t* glast = ws.get<uint8_t>(K_GLAST, static_cast<size_t>(group_warps) * 8 * kRenumberMax);
    if (!gdec || !glast) return LFB_E_CUDA;
    bool group_mode = false;
    unsigned long long arena_used = bt.n;   // clauses in the arena

    for (int d = 0; d < L; ++d) {
        if (cancelled()) return LFB_E_CANCELLED;
        LevelView& lv = o.lv[d];
        cells_evaluated += lv.n_cells;
        const auto t_level = std::chrono::steady_clock::now();
        const unsigned long long arena_before = arena_used;
        // The group-mode register file holds this depth's largest tape (the
        // pruned tapes of deep levels need far fewer registers than the
        // unpruned tape, so more warps fit on an SM).
        const uint32_t nregs_d =
            d == 0 ? bt.n_regs : std::min<uint32_t>(std::max<uint32_t>(seen.nregs, 3), bt.n_regs);
        const size_t group_smem = group_smem_per_warp(nregs_d) * 4;
        group_mode = group_mode || (d > 0 && lv.n_cells >= group_mode_cells() &&
                                    group_smem <= 200 * 1024);
        if (group_mode && group_smem > 48 * 1024 &&
            !raise_smem_limit(reinterpret_cast<const void*>(k_interval_group), group_smem)) {
            return LFB_E_CUDA;
        }
        const bool write_lists = d + 1 < L && !group_mode;
        const int out_key = list_key[(d + 1) & 1];
        uint32_t* flags = ws.get<uint32_t>(K_FLAGS, lv.n_cells + 1);
        uint32_t* scan = ws.get<uint32_t>(K_SCAN, lv.n_cells + 1);
        if (!flags || !scan) return LFB_E_CUDA;
        for (int attempt = 0; attempt < 4; ++attempt) {
            WideArgs W;
            W.o = o;
            W.bt = bt;
            W.n = bt.n;
            W.in_lists = d == 0 ? g.d_wide : ws.bufs[list_key[d & 1]].as<WideEntry>();
            W.root_list = {0u, bt.n, g.wide_root, 0u};
            W.out_lists = ws.bufs[out_key].as<WideEntry>();
            W.out_top = list_top;
            W.out_cap = cap_of(out_key, sizeof(WideEntry));
            W.write_lists = write_lists ? 1 : 0;
            W.arena = arena;
            W.arena_top = arena_top;
            W.arena_cap = arena_cap;
            W.S = wS;
            W.SN = wSN;
            W.pst = wP;
            W.live = wLive;
            W.newpos = wNew;
            W.st2 = wSt2;
            W.l1 = wL1;
            W.wl = wWl;
            W.status = status;
            W.next_cell = &counters->next_cell;
            W.group_shift = 3;
            W.boxes = nullptr;
            W.n_boxes = W.arena_base = 0;
            W.box_tape = nullptr;
            cudaMemsetAsync(list_top, 0, kLevelCounters, s);
            if (!group_mode && lv.n_cells > block_mode_cells() && !wide_zeroed) {
                wide_zeroed = true;
                cudaMemsetAsync(wSt2, 0, scratch_warps * nw16 * 4, s);
                cudaMemsetAsync(wL1, 0, scratch_warps * nw1 * 4, s);
            }
            if (group_mode) {
                GroupArgs G{o, bt, arena, arena_top, arena_cap, gdec, gdec_cap, glast,
                            nregs_d, status, W.next_cell};
                const uint32_t blocks = std::min<uint32_t>(group_warps / 4, (lv.n_groups + 3) / 4);
                k_interval_group<<<std::max<uint32_t>(blocks, 1), 128, group_smem, s>>>(G, d);
            } else if (!cuda_ok(launch_interval_lists(W, d, lv.n_cells, scratch_warps, s),
                                "interval kernel")) {
                return LFB_E_CUDA;
            }
            ++n_launch;
            if (!cuda_ok(cudaGetLastError(), "interval kernel")) return LFB_E_CUDA;
            // The level's counts go back while the branch cells are scanned:
            // one wait per level.
            k_branch_flags<<<lv.n_cells / 256 + 1, 256, 0, s>>>(lv.type, lv.cell_tape, lv.n_cells,
                                                                flags, counters, d + 1 == L);
            ++n_launch;
            if (!fetch_counters("interval kernel") || !exclusive_scan(ws, flags, scan, lv.n_cells + 1, s) ||
                !cuda_ok(cudaStreamSynchronize(s), "interval kernel")) {
                return LFB_E_CUDA;
            }
            const uint32_t st = seen.status;
            const unsigned long long tops[2] = {seen.arena_top, seen.list_top};
            if (st & ST_REGS) {
                return set_error(LFB_E_UNSUPPORTED, "tape register renumbering failed");
            }
            arena_used = tops[0];
            if (!(st & (ST_ARENA_OVERFLOW | ST_LIST_OVERFLOW))) break;
            if (attempt == 3) return set_error(LFB_E_CAPACITY, "tape arena overflow");
            // The counters kept counting past the capacity: grow to what this
            // depth needs and run it again.
            if (st & ST_LIST_OVERFLOW) {
                // The output arena holds nothing yet: no copy needed.
                if (!ws.get<WideEntry>(out_key, tops[1] + tops[1] / 4 + 1024)) return LFB_E_CUDA;
            }
            if (st & ST_ARENA_OVERFLOW) {
                // The arena keeps its contents (the tapes of the levels
                // above): a larger buffer in the same stream order, the
                // used part copied over, the old one freed after the copy.
                const uint64_t new_cap = tops[0] + tops[0] / 4 + (1u << 20);
                DevBuf& b = ws.bufs[K_ARENA];
                RegClause* bigger = nullptr;
                const cudaError_t e =
                    b.ordered ? cudaMallocAsync(reinterpret_cast<void**>(&bigger),
                                                new_cap * sizeof(RegClause), b.stream)
                              : cudaMalloc(&bigger, new_cap * sizeof(RegClause));
                if (e == cudaErrorMemoryAllocation) note_device_oom();
                if (!cuda_ok(e, "arena grow")) return LFB_E_CUDA;
                cudaMemcpyAsync(bigger, arena, arena_before * sizeof(RegClause),
                                cudaMemcpyDeviceToDevice, s);
                if (b.ordered) {
                    cudaFreeAsync(b.ptr, b.stream);
                } else {
                    cudaStreamSynchronize(s);
                    cudaFree(b.ptr);
                }
                b.ptr = bigger;
                b.bytes = new_cap * sizeof(RegClause);
                arena = bigger;
                arena_cap = new_cap;
            }
            cudaMemcpyAsync(arena_top, &arena_before, sizeof(arena_before), cudaMemcpyHostToDevice, s);
            cudaMemsetAsync(status, 0, sizeof(uint32_t), s);
        }

        if (debug_levels()) {
            unsigned long long top_now = 0, lt = 0;
            cudaMemcpyAsync(&top_now, arena_top, sizeof(top_now), cudaMemcpyDeviceToHost, s);
            cudaMemcpyAsync(&lt, list_top, sizeof(lt), cudaMemcpyDeviceToHost, s);
            cudaStreamSynchronize(s);
            const double ms = std::chrono::duration<double, std::milli>(
                std::chrono::steady_clock::now() - t_level).count();
            std::fprintf(stderr, "[lfb] depth %d: %u cells, arena %llu clauses, lists %llu, %.3f ms\n",
                         d, lv.n_cells, top_now, lt, ms);
        }
        // Compact the branch cells into the groups of depth d + 1.
        const uint32_t n_groups = seen.n_groups;
        if (static_cast<uint64_t>(n_groups) * 8 >= (1u << 27)) {
            return set_error(LFB_E_CAPACITY, "more than 2^27 cells on one octree level");
        }
        if (!alloc_level(d + 1, n_groups * 8, n_groups)) return LFB_E_CUDA;
        k_build_groups<<<(lv.n_cells + 255) / 256, 256, 0, s>>>(o, d, scan);
        ++n_launch;
        if (n_groups == 0) {
            // Nothing ambiguous below this depth: no leaves, no faces.
            o.levels = L;
            for (int dd = d + 1; dd <= L; ++dd) {
                if (!alloc_level(dd, 0, 0)) return LFB_E_CUDA;
            }
            break;
        }
    }

    if (cancelled()) return LFB_E_CANCELLED;
    if (stats) cudaEventRecord(ev[1], s);
    // Leaves.
    const uint32_t n_leaf_groups = (L == 0) ? 1 : o.lv[L].n_groups;
    const size_t rec_cap = static_cast<size_t>(n_leaf_groups) * 8 + cells_evaluated + 16;
    LeafRec* recs = ws.get<LeafRec>(K_RECS, rec_cap);
    if (!recs) return LFB_E_CUDA;
    if (n_leaf_groups) {
        // Warps per block: eight, fewer while that leaves SMs without a block.
        const uint32_t sms = static_cast<uint32_t>(device_sm_count());
        uint32_t wpb = kLeafWarps;
        while (wpb > 1 && n_leaf_groups < sms * wpb) wpb /= 2;
        if (debug_levels() && L > 0) {
            std::vector<TapeRef> gt(n_leaf_groups);
            cudaMemcpyAsync(gt.data(), o.lv[L].group_tape, n_leaf_groups * sizeof(TapeRef),
                            cudaMemcpyDeviceToHost, s);
            cudaStreamSynchronize(s);
            std::map<uint32_t, uint64_t> hist, lhist;
            uint64_t len_sum = 0;
            for (const TapeRef& t : gt) {
                ++hist[t.nregs];
                len_sum += t.len;
                uint32_t b = 0;
                while ((1u << (b + 1)) <= t.len) ++b;
                lhist[b] += t.len;
            }
            std::fprintf(stderr, "[lfb] leaf tape clauses by log2(length):");
            for (const auto& h : lhist) {
                std::fprintf(stderr, " %u:%llu", h.first, static_cast<unsigned long long>(h.second));
            }
            std::fprintf(stderr, "\n");
            std::fprintf(stderr, "[lfb] leaf groups %u, mean tape %.1f, registers:",
                         n_leaf_groups, static_cast<double>(len_sum) / std::max<uint32_t>(n_leaf_groups, 1));
            for (const auto& h : hist) {
                std::fprintf(stderr, " %u:%llu", h.first, static_cast<unsigned long long>(h.second));
            }
            std::fprintf(stderr, "\n");
        }
        // Shared memory: per warp its state and a register file of smem_regs
        // float4s a lane; groups whose tape needs more registers use global
        // memory instead.  Sixteen registers where all warps then fit beside
        // each other anyway (16 an SM), and where the tapes of 9 to 16 gain
        // more than the others lose with fewer warps an SM.  Leaf stage with
        // 8 and 16 registers, ms: all clauses in tapes of 9 to 16 (16 and 64
        // smooth blends) 9.8 and 7.9, 81 and 67; of up to 8 (CSG of 1,000)
        // 5.7 and 6.1; of more than 16 (blends with min) 119 and 141.  CSG of
        // 2,000 with 67 % of the clauses in tapes of 9 to 16 24.4 and 23.5, of
        // 4,000 with 21 % 78 and 81: hence the weights.
        const unsigned long long* clauses = seen.clauses;
        const bool few = n_leaf_groups <= sms * 16;
        uint32_t group_regs = std::min<uint32_t>(
            bt.n_regs, few || 2 * clauses[1] > clauses[0] + 3 * clauses[2] ? kLeafSmemRegs
                                                                           : kLeafSmemRegsMany);
        // Steps by clause offset, so room for as many as the arena has
        // clauses: 36 bytes beside each clause's own 8.  Where no tape can be
        // decoded, or the device has no such room left even for a mesh that is
        // rendered again by itself, every group runs from global memory,
        // clause by clause.
        ValOp* vops = nullptr;
        uint32_t* n_steps = nullptr;
        const bool decodable = L == 0 ? bt.n_regs <= group_regs
                                      : clauses[0] + (group_regs > kLeafSmemRegsMany ? clauses[1] : 0) != 0;
        if (decodable) {
            vops = ws.get<ValOp>(K_VOPS, arena_used);
            n_steps = ws.get<uint32_t>(K_NSTEPS, arena_used);
        }
        if (!vops || !n_steps) {
            if (decodable && !ws.lean) return LFB_E_CUDA;
            take_device_oom();
            clear_error();
            group_regs = 0;
        } else {
            cudaMemsetAsync(n_steps, 0, arena_used * sizeof(uint32_t), s);
        }
        const uint32_t qef_regs = std::min<uint32_t>(bt.n_regs, kLeafSmemRegs);
        const size_t group_bytes = (sizeof(LeafWarpShared) + size_t{512} * group_regs) * wpb;
        const size_t qef_bytes = (sizeof(LeafOp) * kLeafOps + size_t{512} * qef_regs) * wpb;
        auto* groups_kernel = L == 0 ? k_leaf_groups<true, true> : k_leaf_groups<false, false>;
        auto* redo_kernel = k_leaf_groups<false, true>;
        if (!raise_smem_limit(reinterpret_cast<const void*>(groups_kernel), group_bytes) ||
            !raise_smem_limit(reinterpret_cast<const void*>(redo_kernel), group_bytes) ||
            !raise_smem_limit(reinterpret_cast<const void*>(k_leaf_qef<false>), qef_bytes) ||
            !raise_smem_limit(reinterpret_cast<const void*>(k_leaf_qef<true>), qef_bytes)) {
            return LFB_E_CUDA;
        }
        const uint32_t want = (n_leaf_groups + wpb - 1) / wpb;
        int per_sm = 0, qef_per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, groups_kernel, 32 * wpb, group_bytes);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&qef_per_sm, k_leaf_qef<false>, 32 * wpb, qef_bytes);
        const uint32_t grid = std::min<uint32_t>(want, sms * std::max(per_sm, 1));
        const uint32_t qef_grid = std::min<uint32_t>(want, sms * std::max(qef_per_sm, 1));
        const size_t slices = static_cast<size_t>(std::max(grid, qef_grid)) * wpb;
        LeafWarpScratch* scratch = ws.get<LeafWarpScratch>(K_FEAT, slices);
        if (!scratch) return LFB_E_CUDA;
        float* rd = ws.get<float>(K_LEAF_RD, slices * bt.n_regs * 128);
        if (!rd) return LFB_E_CUDA;
        uint32_t* next_group = &counters->next_group;
        // Longest tapes first, where not all groups run at once anyway.
        const uint32_t* order = nullptr;
        if (L > 0 && n_leaf_groups > grid * wpb) {
            uint32_t* k0 = ws.get<uint32_t>(K_ORDER_K0, n_leaf_groups);
            uint32_t* k1 = ws.get<uint32_t>(K_ORDER_K1, n_leaf_groups);
            uint32_t* v0 = ws.get<uint32_t>(K_ORDER_V0, n_leaf_groups);
            uint32_t* v1 = ws.get<uint32_t>(K_ORDER_V1, n_leaf_groups);
            if (!k0 || !k1 || !v0 || !v1) return LFB_E_CUDA;
            k_leaf_order_keys<<<(n_leaf_groups + 255) / 256, 256, 0, s>>>(
                o.lv[L].group_tape, n_leaf_groups, k0, v0);
            ++n_launch;
            size_t tmp = 0;
            int bits = 1;   // of a tape length
            while (bits < 32 && (bt.n >> bits)) ++bits;
            cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, k0, k1, v0, v1,
                                                      static_cast<int>(n_leaf_groups), 0, bits, s);
            void* t = ws.get<unsigned char>(K_SORTTMP, tmp);
            if (!t || !cuda_ok(cub::DeviceRadixSort::SortPairsDescending(
                                   t, tmp, k0, k1, v0, v1, static_cast<int>(n_leaf_groups), 0,
                                   bits, s), "leaf order")) {
                return LFB_E_CUDA;
            }
            order = v1;
        }
        float* featws = ws.get<float>(K_FEATWS, slices * bt.n_regs * kRegBlock);
        if (!featws) return LFB_E_CUDA;
        const uint64_t edge_cap64 = static_cast<uint64_t>(n_leaf_groups) * ws.edges_per_group +
                                    (small ? 0 : 1024);
        const uint32_t edge_cap = static_cast<uint32_t>(std::min<uint64_t>(edge_cap64, 1u << 31));
        EdgeRec* edges = ws.get<EdgeRec>(K_EDGES, edge_cap);
        GroupEdges* gedges = ws.get<GroupEdges>(K_GEDGES, n_leaf_groups);
        uint32_t* rec_group = ws.get<uint32_t>(K_RECGROUP, rec_cap);
        if (!edges || !gedges || !rec_group) return LFB_E_CUDA;
        // Zero-valued samples: room for 32 a group on average (none with the
        // small-capacity hook, so that every such group is searched again).
        const uint32_t zero_cap = small ? 0u : static_cast<uint32_t>(std::min<uint64_t>(
            static_cast<uint64_t>(n_leaf_groups) * 32 + 4096, 1u << 30));
        float* zeros = ws.get<float>(K_ZEROS, size_t{3} * zero_cap);
        uint32_t* redo = ws.get<uint32_t>(K_REDO, n_leaf_groups);
        if (!zeros || !redo) return LFB_E_CUDA;
        LeafArgs A{o, bt, arena, recs, rec_top, static_cast<uint32_t>(rec_cap), status,
                   evals, scratch, rd, group_regs, next_group, order, featws,
                   edges, edge_top, edge_cap, gedges, rec_group,
                   &counters->next_group2,
                   vops, n_steps, n_leaf_groups >= kLeafChunk * 4 * grid * wpb ? kLeafChunk : 1u,
                   zeros, &counters->zero_top, zero_cap, redo, &counters->n_redo,
                   counters->next_redo};
        const TapeRef* tapes = o.lv[L].group_tape;
        if (L == 0) {
            // the unpruned tape is the only one
            TapeRef* t = reinterpret_cast<TapeRef*>(ws.get<uint4>(K_ROOTTAPE, 1));
            const TapeRef root = root_tape_ref(bt);
            if (!t || !cuda_ok(cudaMemcpyAsync(t, &root, sizeof(root), cudaMemcpyHostToDevice, s),
                               "root tape")) {
                return LFB_E_CUDA;
            }
            tapes = t;
        }
        if (group_regs) {
            // groups per decoding warp: as few as fill the GPU
            const uint32_t per_warp = std::min(32u, n_leaf_groups / (sms * 32) + 1);
            k_leaf_decode<<<(n_leaf_groups + 4 * per_warp - 1) / (4 * per_warp), 128, 0, s>>>(
                A, tapes, n_leaf_groups, per_warp);
            ++n_launch;
        }
        groups_kernel<<<grid, 32 * wpb, group_bytes, s>>>(A, n_leaf_groups);
        if (!cuda_ok(cudaGetLastError(), "leaf kernel")) return LFB_E_CUDA;
        A.smem_regs = qef_regs;
        k_leaf_qef<false><<<qef_grid, 32 * wpb, qef_bytes, s>>>(A, n_leaf_groups);
        ++n_launch;
        if (L > 0) {
            // the groups a check sent back (usually none)
            const uint32_t few_blocks = std::min(grid, sms);
            A.smem_regs = group_regs;
            A.chunk = 1;
            redo_kernel<<<few_blocks, 32 * wpb, group_bytes, s>>>(A, n_leaf_groups);
            A.smem_regs = qef_regs;
            k_leaf_qef<true><<<std::min(qef_grid, sms), 32 * wpb, qef_bytes, s>>>(A, n_leaf_groups);
            n_launch += 2;
        }
        if (!cuda_ok(cudaGetLastError(), "leaf QEF kernel")) return LFB_E_CUDA;
        // Edge ranks, then the records' vertices: one thread per edge / record.
        k_edge_rank<<<std::min<uint32_t>(sms * 16, (edge_cap + 127) / 128), 128, 0, s>>>(
            edges, edge_top, edge_cap);
        k_leaf_vertices<<<std::min<uint32_t>(sms * 16, static_cast<uint32_t>((rec_cap + 127) / 128)),
                          128, 0, s>>>(recs, rec_top, static_cast<uint32_t>(rec_cap), rec_group,
                                       gedges, n_leaf_groups, edges, edge_cap, L == 0 ? 1 : 0);
        n_launch += 2;
        if (!cuda_ok(cudaGetLastError(), "leaf vertex kernels")) return LFB_E_CUDA;
        ++n_launch;
    }
    if (cancelled()) return LFB_E_CANCELLED;
    if (stats) cudaEventRecord(ev[2], s);

    // Bottom-up collapse.
    {
        CollapseArgs C{o, bt, arena, recs, rec_top, static_cast<uint32_t>(rec_cap), status,
                       max_err};
        int block = 128;
        while (block > 32 && static_cast<size_t>(bt.n_regs) * block * 4 > 96 * 1024) block /= 2;
        const size_t smem = static_cast<size_t>(bt.n_regs) * block * 4;
        if (smem > 48 * 1024) {
            if (!raise_smem_limit(reinterpret_cast<const void*>(k_collapse_level), smem)) {
                return LFB_E_CUDA;
            }
        }
        for (int d = L - 1; d >= 0; --d) {
            const uint32_t n = o.lv[d].n_cells;
            if (!n) continue;
            const auto t_c = std::chrono::steady_clock::now();
            k_collapse_level<<<(n + block - 1) / block, block, smem, s>>>(C, d);
            ++n_launch;
            if (debug_levels()) {
                cudaStreamSynchronize(s);
                std::fprintf(stderr, "[lfb] collapse depth %d: %u cells, %.3f ms\n", d, n,
                             std::chrono::duration<double, std::milli>(
                                 std::chrono::steady_clock::now() - t_c).count());
            }
        }
        if (!cuda_ok(cudaGetLastError(), "collapse kernel")) return LFB_E_CUDA;
    }

    if (stats) cudaEventRecord(ev[3], s);
    if (!fetch_counters("leaf/collapse") ||
        !cuda_ok(cudaMemcpyAsync(&seen.pad, o.lv[0].type, 1, cudaMemcpyDeviceToHost, s),
                 "leaf/collapse") ||
        !cuda_ok(cudaStreamSynchronize(s), "leaf/collapse")) {
        return LFB_E_CUDA;
    }
    const uint8_t root_type = static_cast<uint8_t>(seen.pad & 0xff);
    const uint32_t st = seen.status, n_recs = seen.n_recs;
    if (st & ST_RECORD_OVERFLOW) return set_error(LFB_E_CAPACITY, "leaf record overflow");
    if (st & ST_EDGE_OVERFLOW) {
        // more crossing edges than records were reserved for: grow, and the
        // caller renders the mesh again
        const unsigned long long need = seen.edge_top;
        const uint32_t groups = std::max<uint32_t>(n_leaf_groups, 1);
        ws.edges_per_group = static_cast<uint32_t>(std::min<unsigned long long>(
            54, need / groups + 2));
        ws.retry = true;
        return set_error(LFB_E_CAPACITY, "leaf edge records overflowed");
    }
    if (st & ST_FEATURE_OVERFLOW) {
        std::string why;
        if (st & ST_FEAT_EPS) {
            why += " (more than " + std::to_string(kMaxEps) + " epsilon directions in a feature)";
        }
        if (st & ST_FEAT_LIST) {
            why += " (more than " + std::to_string(kMaxFeat) + " features in a clause)";
        }
        if (st & ST_FEAT_TMP) {
            why += " (more than " + std::to_string(kTmpFeat) + " candidate features in a clause)";
        }
        return set_error(LFB_E_CAPACITY,
                         "feature list overflow at a non-smooth sample point" + why);
    }

    // Dual walk.
    host_free(out.verts);
    host_free(out.tris);
    out.verts = static_cast<libfive_vec3*>(host_alloc(sizeof(libfive_vec3)));
    out.tris = nullptr;
    out.vert_count = 1;
    out.tri_count = 0;
    if (!out.verts) return set_error(LFB_E_CAPACITY, "host allocation failed");
    out.verts[0] = {0.0f, 0.0f, 0.0f};
    const uint32_t n_keys = n_recs * 4;
    bool stl_written = false;
    if (root_type == CELL_BRANCH && n_recs) {
        size_t task_cap = small ? 1024 : std::max<size_t>(1u << 16, static_cast<size_t>(n_recs) * 24);
        size_t tri_cap = small ? 1024 : std::max<size_t>(1u << 16, static_cast<size_t>(n_recs) * 16);
        for (int attempt = 0; attempt < 5; ++attempt) {
            DualTask* qa = ws.get<DualTask>(K_TASK_A, task_cap);
            DualTask* qb = ws.get<DualTask>(K_TASK_B, task_cap);
            uint32_t* tris = ws.get<uint32_t>(K_TRIS, 3 * tri_cap);
            uint8_t* used = ws.get<uint8_t>(K_USED, n_keys + 1);
            if (!qa || !qb || !tris || !used) return LFB_E_CUDA;
            cudaMemsetAsync(used, 0, n_keys + 1, s);
            cudaMemsetAsync(&counters->n_tris, 0, sizeof(MeshCounters) - offsetof(MeshCounters, n_tris), s);
            cudaMemsetAsync(status, 0, sizeof(uint32_t), s);
            DualArgs D{o, recs, status, qb, nullptr, static_cast<uint32_t>(task_cap),
                       tris, &counters->n_tris, static_cast<uint32_t>(tri_cap), used};
            // A task's cells are one depth deeper every round, so L + 2
            // rounds leave none; each reads how many tasks there are itself.
            const uint32_t dual_blocks = std::min<uint32_t>(
                static_cast<uint32_t>(device_sm_count()) * 32, n_recs / 16 + 1);
            for (int r = 0; r < L + 2; ++r) {
                if (cancelled()) return LFB_E_CANCELLED;
                D.out = qb;
                D.n_out = counters->n_tasks + r;
                k_dual_round<<<r == 0 ? 1 : dual_blocks, 128, 0, s>>>(
                    D, qa, r == 0 ? nullptr : counters->n_tasks + r - 1);
                ++n_launch;
                std::swap(qa, qb);
            }
            // Vertex numbering: ids in record order, 0 is the placeholder.
            uint32_t* flags = ws.get<uint32_t>(K_FLAGS, n_keys + 1);
            uint32_t* vscan = ws.get<uint32_t>(K_VSCAN, n_keys + 1);
            if (!flags || !vscan) return LFB_E_CUDA;
            k_u8_to_u32<<<(n_keys + 1 + 255) / 256, 256, 0, s>>>(used, flags, n_keys + 1);
            if (!exclusive_scan(ws, flags, vscan, n_keys + 1, s) || !fetch_counters("dual walk") ||
                !cuda_ok(cudaMemcpyAsync(&seen.n_verts, vscan + n_keys, sizeof(uint32_t),
                                         cudaMemcpyDeviceToHost, s), "dual walk") ||
                !cuda_ok(cudaStreamSynchronize(s), "dual walk")) {
                return LFB_E_CUDA;
            }
            if (cancelled()) return LFB_E_CANCELLED;   // raised during the walk
            if (seen.status & ST_QUEUE_OVERFLOW) {
                task_cap *= 4;
                tri_cap *= 4;
                continue;
            }
            const uint32_t n_tri = seen.n_tris, n_verts = seen.n_verts;
            if (seen.n_tasks[L + 1] != 0) {   // cannot happen
                return set_error(LFB_E_CAPACITY, "dual walk did not end");
            }
            float* verts = ws.get<float>(K_VERTS, 3 * (static_cast<size_t>(n_verts) + 1));
            if (!verts) return LFB_E_CUDA;
            cudaMemsetAsync(verts, 0, 3 * sizeof(float), s);
            k_vertex_ids<<<(n_keys + 255) / 256, 256, 0, s>>>(used, vscan, n_keys, recs, verts);
            n_launch += 2;   // k_u8_to_u32 + k_vertex_ids
            if (n_tri) {
                k_remap_tris<<<(3 * n_tri + 255) / 256, 256, 0, s>>>(tris, n_tri, vscan);
                ++n_launch;
            }
            if (out.format == MeshFormat::Stl) {
                // records packed on the device, streamed to the file
                out.tri_count = n_tri;
                const int rc = stream_stl(ws, out.stl_path, verts, tris, n_tri, s, n_launch);
                if (rc) return rc;
                stl_written = true;
                break;
            }
            host_free(out.verts);
            out.verts = static_cast<libfive_vec3*>(
                host_alloc((static_cast<size_t>(n_verts) + 1) * sizeof(libfive_vec3)));
            if (!out.verts) return set_error(LFB_E_CAPACITY, "host allocation failed");
            out.vert_count = n_verts + 1;
            out.tri_count = n_tri;
            const bool coords = out.format == MeshFormat::Coords;
            int4* c = nullptr;
            if (coords) {
                c = ws.get<int4>(K_COORDS, std::max<uint32_t>(n_tri, 1));
                host_free(out.coords);
                out.coords = static_cast<int32_t*>(host_alloc(static_cast<size_t>(n_tri) * 16));
                if (!c) return LFB_E_CUDA;
            } else {
                out.tris = static_cast<libfive_tri*>(
                    host_alloc(static_cast<size_t>(n_tri) * sizeof(libfive_tri)));
            }
            if (coords ? !out.coords && n_tri : !out.tris) {
                return set_error(LFB_E_CAPACITY, "host allocation failed");
            }
            if (coords && n_tri) {
                k_pack_coords<<<(n_tri + 255) / 256, 256, 0, s>>>(tris, n_tri, c);
                ++n_launch;
            }
            // one wait for both downloads, when there is a second
            const bool ok =
                download(ws, out.verts, verts, out.vert_count * sizeof(libfive_vec3), s, n_tri == 0) &&
                (coords ? download(ws, out.coords, c, static_cast<size_t>(n_tri) * 16, s)
                        : download(ws, out.tris, tris, static_cast<size_t>(n_tri) * sizeof(libfive_tri), s));
            if (!ok) {
                cudaStreamSynchronize(s);   // nothing may still be writing to the arrays
                return LFB_E_CUDA;
            }
            break;
        }
    }

    if (out.format == MeshFormat::Stl && !stl_written) {
        // no surface: the file holds the header and a zero count
        std::FILE* f = stl_begin(out.stl_path, 0);
        if (!f) return set_error(LFB_E_INVALID, std::string("could not open ") + out.stl_path);
        const bool ok = std::ferror(f) == 0;
        if (std::fclose(f) != 0 || !ok) {
            return set_error(LFB_E_INVALID, std::string("could not write ") + out.stl_path);
        }
    }
    note_launches(n_launch);
    if (stats) {
        cudaEventRecord(ev[4], s);
        cudaEventSynchronize(ev[4]);
        unsigned long long ce[2] = {0, 0};
        cudaMemcpyAsync(ce, evals, sizeof(ce), cudaMemcpyDeviceToHost, s);
        cudaStreamSynchronize(s);
        stats->levels = static_cast<uint32_t>(L);
        stats->cells_evaluated = cells_evaluated;
        stats->leaf_groups = n_leaf_groups;
        stats->leaves_ambiguous = n_recs;
        stats->clause_evals = ce[0];
        stats->clause_evals_grad = ce[1];
        stats->triangles = out.tri_count;
        stats->vertices = out.vert_count - 1;
        stats->kernel_launches = n_launch;
        float ms[4];
        for (int k = 0; k < 4; ++k) cudaEventElapsedTime(&ms[k], ev[k], ev[k + 1]);
        stats->ms_interval = ms[0];
        stats->ms_leaf = ms[1];
        stats->ms_collapse = ms[2];
        stats->ms_dual = ms[3];
        stats->ms_total = std::chrono::duration<double, std::milli>(
                              std::chrono::steady_clock::now() - t_start).count();
    }
    return 0;
}

}  // namespace

/// One mesh in the context `ws`, rendered again (up to twice) when an
/// attempt reports that a capacity estimate was too small.
int render_in(Workspace& ws, GpuTape& g, const libfive_region3& R, double min_feature,
              double max_err, MeshOut& out, lfb_mesh_stats* stats,
              const volatile int32_t* cancel)
{
    int rc = 0;
    for (int attempt = 0; attempt < 3; ++attempt) {
        ws.retry = false;
        rc = render_once(ws, g, R, min_feature, max_err, out, stats, cancel, attempt == 0);
        if (rc == 0 || !ws.retry) break;
        clear_error();
    }
    return rc;
}

int render_dc_mesh(GpuTape& g, const libfive_region3& R, double min_feature,
                   double max_err, MeshOut& out, lfb_mesh_stats* stats,
                   const volatile int32_t* cancel)
{
    if (!require_device()) return LFB_E_CUDA;
    keep_pool_memory(kPoolKeepBytes);
    Workspace& ws = default_workspace();
    std::lock_guard<std::mutex> lock(ws.mu);
    take_device_oom();
    int rc = render_in(ws, g, R, min_feature, max_err, out, stats, cancel);
    if (rc == LFB_E_CUDA && take_device_oom()) {
        // The device ran out of memory: idle batch contexts give their
        // scratch back, this context starts from empty buffers, and the
        // mesh is rendered once more.
        cudaStreamSynchronize(ws.s);
        cudaGetLastError();
        {
            auto& sp = stream_pool();
            std::lock_guard<std::mutex> plock(sp.mu);
            for (Workspace* w : sp.pool) {
                std::unique_lock<std::mutex> wl(w->mu, std::try_to_lock);
                if (wl.owns_lock()) w->bufs.clear();
            }
        }
        ws.bufs.clear();
        clear_error();
        ws.lean = true;
        rc = render_in(ws, g, R, min_feature, max_err, out, stats, cancel);
        ws.lean = false;
    }
    return rc;
}

int render_dc_meshes(MeshJob* jobs, size_t n, unsigned workers)
{
    if (!require_device()) return LFB_E_CUDA;
    keep_pool_memory(kPoolKeepBytes);
    if (n == 0) return 0;
    for (size_t i = 0; i < n; ++i) {
        if (!jobs[i].g) return set_error(LFB_E_INVALID, "null tape in a mesh batch");
    }
    int dev = 0;
    if (!cuda_ok(cudaGetDevice(&dev), "device")) return LFB_E_CUDA;

    // Longest first, so that the last meshes to start are short ones.
    std::vector<double> cost(n);
    for (size_t i = 0; i < n; ++i) {
        const MeshJob& j = jobs[i];
        const double lo[3] = {j.R.X.lower, j.R.Y.lower, j.R.Z.lower};
        const double hi[3] = {j.R.X.upper, j.R.Y.upper, j.R.Z.upper};
        const int L = std::min(level_from_resolution(lo, hi, j.min_feature), 30);
        cost[i] = static_cast<double>(j.g->reg.clauses.size() + 1) * std::ldexp(1.0, 2 * L);
    }
    std::vector<size_t> order(n);
    for (size_t i = 0; i < n; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(),
                     [&](size_t a, size_t b) { return cost[a] > cost[b]; });

    workers = std::max(1u, std::min<unsigned>(workers, static_cast<unsigned>(
                                                           std::min<size_t>(n, 16))));
    // Large meshes (tape length x 4^depth above kBigCost) fill the GPU on
    // their own and need the most scratch memory: worker 0 renders them one
    // after another while the other workers render the small ones side by
    // side; worker 0 joins them when the large ones are done.
    constexpr double kBigCost = 2e9;
    std::vector<size_t> big, small;
    for (size_t i : order) (cost[i] >= kBigCost && workers > 1 ? big : small).push_back(i);
    std::atomic<size_t> next_big{0}, next_small{0};
    auto run_queue = [&](Workspace* ws, const std::vector<size_t>& q, std::atomic<size_t>& next) {
        for (;;) {
            const size_t i = next.fetch_add(1);
            if (i >= q.size()) break;
            MeshJob& j = jobs[q[i]];
            clear_error();
            j.rc = render_in(*ws, *j.g, j.R, j.min_feature, j.max_err, j.out,
                             j.want_stats ? &j.stats : nullptr, j.cancel);
            if (j.rc != 0) last_error(&j.err);
        }
    };
    auto work = [&](unsigned k) {
        cudaSetDevice(dev);
        Workspace* ws = stream_workspace(k);
        if (!ws) return;
        std::lock_guard<std::mutex> lock(ws->mu);
        if (k == 0) run_queue(ws, big, next_big);
        run_queue(ws, small, next_small);
    };
    std::vector<std::thread> pool;
    for (unsigned k = 1; k < workers; ++k) pool.emplace_back(work, k);
    work(0);
    for (auto& t : pool) t.join();

    // A mesh that ran out of device memory while others were in flight is
    // rendered again alone, after the other contexts (and the single-call
    // context, when idle) have given their buffers back.
    std::vector<size_t> retry;
    for (size_t i = 0; i < n; ++i) {
        if (jobs[i].rc == LFB_E_CUDA && jobs[i].err.find("out of memory") != std::string::npos) {
            retry.push_back(i);
        }
    }
    if (!retry.empty()) {
        cudaDeviceSynchronize();
        cudaGetLastError();
        for (unsigned k = 1; k < workers; ++k) {
            Workspace* w = stream_workspace(k);
            std::lock_guard<std::mutex> lock(w->mu);
            w->bufs.clear();
        }
        {
            Workspace& d = default_workspace();
            std::unique_lock<std::mutex> lock(d.mu, std::try_to_lock);
            if (lock.owns_lock()) d.bufs.clear();
        }
        Workspace* w = stream_workspace(0);
        std::lock_guard<std::mutex> lock(w->mu);
        w->lean = true;
        for (size_t i : retry) {
            MeshJob& j = jobs[i];
            clear_error();
            j.err.clear();
            j.rc = render_in(*w, *j.g, j.R, j.min_feature, j.max_err, j.out,
                             j.want_stats ? &j.stats : nullptr, j.cancel);
            if (j.rc != 0) last_error(&j.err);
        }
        w->lean = false;
    }

    clear_error();
    for (size_t i = 0; i < n; ++i) {
        const MeshJob& j = jobs[i];
        if (j.rc == 1) return set_error(LFB_E_CUDA, "no stream context for a mesh batch");
        if (j.rc != 0) return set_error(j.rc, j.err);
    }
    return 0;
}

}  // namespace lfb
