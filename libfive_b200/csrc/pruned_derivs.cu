// Derivatives of long tapes, pruned by place (DerivArrayEvaluator::derivs
// over Tape::push'ed tapes, libfive/src/eval/eval_deriv_array.cpp:101-117 and
// tape.cpp:23-160).
//
// A tape too long to be compiled is interpreted clause by clause, a serial
// chain of about 390 cycles a clause whatever the number of points.  Most of
// a CSG model's clauses do not matter at a given place, so for many points:
//
//   1. the points are sorted along a Hilbert curve over their bounding box
//      (30-bit keys; a run of a Morton curve can straddle the whole box, and
//      such a cell's tape set the length of the launch: 15,800 of 18,700
//      clauses) and cut into cells of consecutive points;
//   2. k_interval_block evaluates the tape's intervals over each cell's
//      bounding box and prunes the tape for it: a min / max is decided only
//      when its operands' intervals are disjoint and neither may be NaN, so
//      that at every point of the cell the kept operand is the one that the
//      full tape takes, value and partials alike;
//   3. a warp for every 32 points of a cell runs the derivative interpreter
//      over the cell's tape, the warps of the longest tapes first.
//
// Results are the full tape's, bit for bit.  Nothing here waits for the
// device: a pruned tape that does not fit the arena is replaced by the full
// one, and scratch is allocated and freed in stream order.
// 100,003 points over an 18,667-clause CSG tape: 1.92 ms (the whole tape
// 11.2; sorting 0.08, intervals 0.58, the interpreter 1.23); 256 points 2.70 ms
// (3.31), 10^6 points 6.86 ms (78.5).
#include <cub/cub.cuh>

#include <algorithm>

#include "eval_api.hpp"
#include "eval_kernels.cuh"
#include "interval_lists.cuh"
#include "libfive_b200.h"

namespace lfb {

namespace {

constexpr uint32_t kCellClauses = 4096;  // arena room per cell, on average

/// Float -> unsigned key with the same order.
__device__ __forceinline__ uint32_t order_key(float f)
{
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

/// Bounding box of the finite points as order keys: box[0..2] the smallest,
/// box[3..5] the complements of the largest (both by atomicMin from ~0).
__global__ void __launch_bounds__(256)
k_pd_bounds(uint32_t n, const float* __restrict__ x, const float* __restrict__ y,
            const float* __restrict__ z, uint32_t* box)
{
    const float* p[3] = {x, y, z};
    uint32_t lo[3] = {~0u, ~0u, ~0u}, hi[3] = {~0u, ~0u, ~0u};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float v = p[a][i];
            if (!isfinite(v)) continue;
            lo[a] = min(lo[a], order_key(v));
            hi[a] = min(hi[a], ~order_key(v));
        }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, lo[a]);
        const uint32_t h = __reduce_min_sync(0xffffffffu, hi[a]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(box + a, l);
            atomicMin(box + 3 + a, h);
        }
    }
}

__device__ __forceinline__ uint32_t spread10(uint32_t v)
{
    v = (v | v << 16) & 0x030000ffu;
    v = (v | v << 8) & 0x0300f00fu;
    v = (v | v << 4) & 0x030c30c3u;
    return (v | v << 2) & 0x09249249u;
}

/// Place along the Hilbert curve of a cell of a 1024^3 grid (J. Skilling,
/// "Programming the Hilbert curve", AIP Conf. Proc. 707, 2004: axes to
/// transpose, whose bits are then interleaved).
__device__ __forceinline__ uint32_t hilbert30(uint32_t x, uint32_t y, uint32_t z)
{
    uint32_t X[3] = {x, y, z};
#pragma unroll
    for (uint32_t q = 512; q > 1; q >>= 1) {
        const uint32_t p = q - 1;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            if (X[i] & q) {
                X[0] ^= p;
            } else {
                const uint32_t t = (X[0] ^ X[i]) & p;
                X[0] ^= t;
                X[i] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    uint32_t t = 0;
#pragma unroll
    for (uint32_t q = 512; q > 1; q >>= 1) {
        if (X[2] & q) t ^= q - 1;
    }
    return spread10(X[0] ^ t) << 2 | spread10(X[1] ^ t) << 1 | spread10(X[2] ^ t);
}

/// Curve key of every point; points with a coordinate that is not finite
/// come last.
__global__ void __launch_bounds__(256)
k_pd_keys(uint32_t n, const float* __restrict__ x, const float* __restrict__ y,
          const float* __restrict__ z, const uint32_t* __restrict__ box, uint32_t* keys,
          uint32_t* idx)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float p[3] = {x[i], y[i], z[i]};
    uint32_t c[3];
    bool finite = true;
    // one scale for the three axes: cells as near to cubes as the box allows
    float side = 1e-30f;
#pragma unroll
    for (int a = 0; a < 3; ++a) side = fmaxf(side, key_float(~box[3 + a]) - key_float(box[a]));
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float t = (p[a] - key_float(box[a])) / side * 1024.0f;
        finite = finite && isfinite(p[a]);
        c[a] = static_cast<uint32_t>(fminf(fmaxf(t, 0.0f), 1023.0f));
    }
    keys[i] = finite ? hilbert30(c[0], c[1], c[2]) : 0x3fffffffu;
    idx[i] = i;
}

/// Bounding box of each cell's points (one warp a cell): lower and upper
/// bound per axis, NaN where a coordinate is.
__global__ void __launch_bounds__(128)
k_pd_boxes(uint32_t n, uint32_t per_cell, uint32_t n_cells, const uint32_t* __restrict__ idx,
           const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
           float* boxes)
{
    const uint32_t c = blockIdx.x * 4 + (threadIdx.x >> 5);
    const uint32_t lane = threadIdx.x & 31;
    if (c >= n_cells) return;
    const float* p[3] = {x, y, z};
    uint32_t lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0, 0, 0};
    bool nan = false;
    const uint32_t end = min(n, (c + 1) * per_cell);
    for (uint32_t k = c * per_cell + lane; k < end; k += 32) {
        const uint32_t i = idx[k];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float v = p[a][i];
            nan |= v != v;
            lo[a] = min(lo[a], order_key(v));
            hi[a] = max(hi[a], order_key(v));
        }
    }
    nan = __any_sync(0xffffffffu, nan);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const uint32_t l = __reduce_min_sync(0xffffffffu, lo[a]);
        const uint32_t h = __reduce_max_sync(0xffffffffu, hi[a]);
        if (lane == 0) {
            boxes[6 * c + 2 * a] = nan ? LF_QNAN : key_float(l);
            boxes[6 * c + 2 * a + 1] = nan ? LF_QNAN : key_float(h);
        }
    }
}

/// A clause as the interpreter below reads it: one 16-byte word in shared
/// memory, constant and free-variable operands already fetched.
/// x: opcode | PD_* << 8 | result register << 16; y: operand registers a |
/// b << 16; z, w: the values of immediate operands.
enum : uint32_t {
    PD_A_IMM = 1, PD_B_IMM = 2,     // the operand is z / w
    PD_A_LAST = 4, PD_B_LAST = 8,   // ... is the clause before's result
    PD_UNARY = 16,
};
constexpr uint32_t kPdOps = 64;     // clauses a warp decodes at a time

__device__ __forceinline__ uint4 pd_decode(uint2 raw, uint32_t prev_out, const float* __restrict__ cp)
{
    const uint32_t o = raw.x & 0xff, kinds = (raw.x >> 8) & 0xf;
    const uint32_t a = raw.y & 0xffff, b = raw.y >> 16;
    uint32_t f = 0;
    float ia = 0.0f, ib = 0.0f;
    if ((kinds & 3) != OPND_REG) {
        f |= PD_A_IMM;
        ia = __ldg(cp + a);
    } else if (a == prev_out) {
        f |= PD_A_LAST;
    }
    if (!dev_is_binary(static_cast<uint8_t>(o))) {
        f |= PD_UNARY;
    } else if ((kinds >> 2) != OPND_REG) {
        f |= PD_B_IMM;
        ib = __ldg(cp + b);
    } else if (b == prev_out) {
        f |= PD_B_LAST;
    }
    return make_uint4(o | f << 8 | (raw.x & 0xffff0000u), raw.y, __float_as_uint(ia), __float_as_uint(ib));
}

/// dv_deriv with the square root inline, in dv_deriv_all's operations.
__device__ __forceinline__ D4 pd_deriv(uint8_t o, const D4& a, const D4& b)
{
    if (o != op::SQRT) return dv_deriv(o, a, b, false);
    const float v = __fsqrt_rn(a.v), den = __fmul_rn(2.0f, v);
    const bool none = a.v < 0;
    return {v, none || a.dx == 0 ? 0.0f : __fdiv_rn(a.dx, den),
            none || a.dy == 0 ? 0.0f : __fdiv_rn(a.dy, den),
            none || a.dz == 0 ? 0.0f : __fdiv_rn(a.dz, den)};
}

/// Sort keys of the cells: longest tape first.
__global__ void k_pd_lengths(const TapeRef* __restrict__ tapes, uint32_t n_cells, uint32_t* keys,
                             uint32_t* cells)
{
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n_cells) return;
    keys[c] = ~tapes[c].len;
    cells[c] = c;
}

/// The derivative interpreter over each cell's own tape: one warp for 32 of
/// its points, one float4 (value, partials) per register and lane.  Tapes'
/// lengths differ by orders of magnitude, so the warps are blocks of their
/// own, those of the longest tapes first (with a block a cell, in the
/// curve's order, the SMs were busy for half of the kernel: 1.45 ms, of
/// which the instructions need 0.46).  The warp first decodes kPdOps clauses
/// at a time, a clause a lane, with their constants (the raw words fetched a
/// chunk ahead), and a result read by the next clause stays in hardware
/// registers.
__global__ void __launch_bounds__(32)
k_pd_derivs(DevTape bt, const TapeRef* __restrict__ tapes, const RegClause* __restrict__ arena,
            const uint32_t* __restrict__ order, uint32_t n, uint32_t per_cell, const uint32_t* __restrict__ idx,
            const float* __restrict__ X, const float* __restrict__ Y, const float* __restrict__ Z,
            float* __restrict__ ov, float* __restrict__ odx, float* __restrict__ ody,
            float* __restrict__ odz)
{
    extern __shared__ __align__(16) float4 regs[];
    __shared__ uint4 ops[kPdOps];
    constexpr uint32_t B = 32;
    const uint32_t lane = threadIdx.x;
    float4* R = regs + lane;
    const uint32_t cell = order[blockIdx.x / (per_cell / 32)];
    const uint32_t k = cell * per_cell + blockIdx.x % (per_cell / 32) * 32 + lane;
    const uint32_t end = min(n, (cell + 1) * per_cell);
    if (k - lane >= end) return;
    const TapeRef t = tapes[cell];
    const uint2* cl = reinterpret_cast<const uint2*>(arena + t.off);
    const float* cp = bt.cpool;
    const uint2 none = make_uint2(0, 0);
    auto raw_of = [&](uint32_t c) { return c < t.len ? __ldg(cl + c) : none; };
    const uint32_t i = idx[min(k, end - 1)];
    R[0] = make_float4(X[i], 1.0f, 0.0f, 0.0f);
    R[B] = make_float4(Y[i], 0.0f, 1.0f, 0.0f);
    R[2 * B] = make_float4(Z[i], 0.0f, 0.0f, 1.0f);
    D4 last{0.0f, 0.0f, 0.0f, 0.0f};
    uint2 raw0 = raw_of(lane), raw1 = raw_of(lane + 32);
    uint32_t before = 0xffffffffu;   // result register of the chunk before's last clause
    for (uint32_t c0 = 0; c0 < t.len; c0 += kPdOps) {
        const uint32_t up0 = __shfl_up_sync(0xffffffffu, raw0.x >> 16, 1);
        const uint32_t mid = __shfl_sync(0xffffffffu, raw0.x >> 16, 31);
        const uint32_t up1 = __shfl_up_sync(0xffffffffu, raw1.x >> 16, 1);
        __syncwarp();
        ops[lane] = pd_decode(raw0, lane ? up0 : before, cp);
        ops[lane + 32] = pd_decode(raw1, lane ? up1 : mid, cp);
        before = __shfl_sync(0xffffffffu, raw1.x >> 16, 31);
        raw0 = raw_of(c0 + kPdOps + lane);
        raw1 = raw_of(c0 + kPdOps + lane + 32);
        __syncwarp();
        const uint32_t m = min(kPdOps, t.len - c0);
        uint4 next = ops[0];
#pragma unroll 1
        for (uint32_t c = 0; c < m; ++c) {
            const uint4 w = next;
            next = ops[min(c + 1, kPdOps - 1)];
            const uint32_t f = w.x >> 8;
            D4 a, b;
            if (f & PD_A_LAST) {
                a = last;
            } else if (f & PD_A_IMM) {
                a = {__uint_as_float(w.z), 0.0f, 0.0f, 0.0f};
            } else {
                const float4 v = R[(w.y & 0xffff) * B];
                a = {v.x, v.y, v.z, v.w};
            }
            if (f & PD_UNARY) {
                b = a;
            } else if (f & PD_B_LAST) {
                b = last;
            } else if (f & PD_B_IMM) {
                b = {__uint_as_float(w.w), 0.0f, 0.0f, 0.0f};
            } else {
                const float4 v = R[(w.y >> 16) * B];
                b = {v.x, v.y, v.z, v.w};
            }
            last = pd_deriv(static_cast<uint8_t>(w.x), a, b);
            R[(w.x >> 16) * B] = make_float4(last.v, last.dx, last.dy, last.dz);
        }
    }
    if (k < end) {
        const uint32_t root = t.root & 0xffff;
        D4 d;
        if (t.root >> 16 == OPND_REG) {
            const float4 v = R[root * B];
            d = {v.x, v.y, v.z, v.w};
        } else {
            d = {__ldg(cp + root), 0.0f, 0.0f, 0.0f};
        }
        ov[i] = d.v;
        if (odx) odx[i] = d.dx;
        if (ody) ody[i] = d.dy;
        if (odz) odz[i] = d.dz;
    }
}

/// Whether every clause's interval rule encloses what the derivative
/// interpreter computes: directed-rounding operations, and exp and log,
/// whose bounds are widened past their error; all of them as iv_enclose
/// (dev_interval.cuh) corrects them.
bool sound_ops(GpuTape& g)
{
    std::lock_guard<std::mutex> lock(g.mu);
    if (g.sound_ops < 0) {
        g.sound_ops = 1;
        for (const RegClause& c : g.reg.clauses) {
            switch (c.op) {
                case op::ADD: case op::SUB: case op::MUL: case op::DIV: case op::MIN:
                case op::MAX: case op::SQUARE: case op::SQRT: case op::NEG: case op::ABS:
                case op::RECIP: case op::EXP: case op::LOG: case op::CONST_VAR:
                    break;
                default:
                    g.sound_ops = 0;
            }
        }
    }
    return g.sound_ops == 1;
}

}  // namespace

bool pruned_derivs(GpuTape& g, uint64_t n, const float* x, const float* y, const float* z, float* v,
                   float* dx, float* dy, float* dz, cudaStream_t s)
{
    // Tapes with a min / max in at least every 64th clause, and enough
    // points for a few cells.  (A tape without any could only lose the time
    // of steps 1 and 2, a tenth of the interpreter's.)
    constexpr uint32_t kMinPoints = 256;
    constexpr uint32_t kMostRegs = 100;   // as the interpreter (launch_derivs)
    const DevTape bt = g.dev();
    if (n < kMinPoints || n >= (1u << 30) || bt.n < 1024 || bt.n_choices < bt.n / 64 ||
        bt.n_regs > kMostRegs || !sound_ops(g)) {
        return false;
    }
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &capturing) != cudaSuccess ||
        capturing != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;   // the general path allocates nothing
    }
    RelaxedCapture relaxed;   // another stream's capture may be open
    if (!g.ensure_wide()) {
        clear_error();
        return false;
    }
    const uint32_t sms = static_cast<uint32_t>(device_sm_count());
    const uint32_t m = static_cast<uint32_t>(n);
    // Points per cell: about four cells an SM, 32 to 1024 points.
    const uint32_t per_cell =
        std::min<uint32_t>(1024, std::max<uint32_t>(32, (m / (4 * sms) + 31) / 32 * 32));
    const uint32_t n_cells = (m + per_cell - 1) / per_cell;
    const size_t file = static_cast<size_t>(bt.n_regs) * 32 * sizeof(float4);
    if (!raise_smem_limit(reinterpret_cast<const void*>(k_pd_derivs), file)) {
        clear_error();
        return false;
    }
    const uint32_t slots = interval_box_slots(bt.n, n_cells);
    const uint64_t arena_cap =
        bt.n + std::min<uint64_t>(static_cast<uint64_t>(n_cells) * kCellClauses, 1u << 25);
    size_t sort_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, static_cast<uint32_t*>(nullptr),
                                    static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                    static_cast<uint32_t*>(nullptr), static_cast<int>(m), 0, 32, s);
    // One block of scratch in stream order (the pool keeps it, as the
    // mesher's).
    keep_pool_memory(uint64_t(32) << 30);
    size_t total = 0;
    auto part = [&](size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t o_head = part(256), o_keys = part(4 * n), o_keys2 = part(4 * n),
                 o_idx = part(4 * n), o_idx2 = part(4 * n), o_boxes = part(24 * n_cells),
                 o_tapes = part(sizeof(TapeRef) * n_cells), o_order = part(4 * n_cells), o_sort = part(sort_bytes),
                 o_arena = part(8 * arena_cap),
                 o_wide = part(wide_scratch_bytes(bt.n, std::max<uint32_t>(slots, 1)));
    unsigned char* p = nullptr;
    if (cudaMallocAsync(reinterpret_cast<void**>(&p), total, s) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    // head: bounding box (6 words), then arena top, work counter, status
    uint32_t* box = reinterpret_cast<uint32_t*>(p + o_head);
    unsigned long long* arena_top = reinterpret_cast<unsigned long long*>(p + o_head + 64);
    uint32_t* keys = reinterpret_cast<uint32_t*>(p + o_keys);
    uint32_t* keys2 = reinterpret_cast<uint32_t*>(p + o_keys2);
    uint32_t* idx = reinterpret_cast<uint32_t*>(p + o_idx);
    uint32_t* idx2 = reinterpret_cast<uint32_t*>(p + o_idx2);
    uint32_t* order = reinterpret_cast<uint32_t*>(p + o_order);
    RegClause* arena = reinterpret_cast<RegClause*>(p + o_arena);
    bool ok = cudaMemsetAsync(box, 0xff, 64, s) == cudaSuccess &&
              cudaMemsetAsync(arena_top, 0, 64, s) == cudaSuccess &&
              cudaMemcpyAsync(arena, bt.clauses, bt.n * sizeof(RegClause), cudaMemcpyDeviceToDevice,
                              s) == cudaSuccess;
    k_pd_bounds<<<std::min<uint32_t>(sms * 4, (m + 255) / 256), 256, 0, s>>>(m, x, y, z, box);
    k_pd_keys<<<(m + 255) / 256, 256, 0, s>>>(m, x, y, z, box, keys, idx);
    ok = ok && cub::DeviceRadixSort::SortPairs(p + o_sort, sort_bytes, keys, keys2, idx, idx2,
                                               static_cast<int>(m), 0, 30, s) == cudaSuccess;
    float* boxes = reinterpret_cast<float*>(p + o_boxes);
    k_pd_boxes<<<(n_cells + 3) / 4, 128, 0, s>>>(m, per_cell, n_cells, idx2, x, y, z, boxes);
    WideArgs W{};
    W.bt = bt;
    W.n = bt.n;
    W.in_lists = g.d_wide;
    W.root_list = {0u, bt.n, g.wide_root, 0u};
    W.arena = arena;
    W.arena_top = arena_top;
    W.arena_base = bt.n;
    W.arena_cap = arena_cap;
    wide_scratch_carve(W, p + o_wide, bt.n, std::max<uint32_t>(slots, 1));
    W.next_cell = reinterpret_cast<uint32_t*>(arena_top + 1);
    W.status = reinterpret_cast<uint32_t*>(arena_top + 2);
    W.boxes = boxes;
    W.n_boxes = n_cells;
    W.box_tape = reinterpret_cast<TapeRef*>(p + o_tapes);
    ok = ok && launch_interval_boxes(W, slots, s) == cudaSuccess;
    // the keys' buffers again, for the cells' order (n_cells <= n)
    if (ok) {
        k_pd_lengths<<<(n_cells + 255) / 256, 256, 0, s>>>(W.box_tape, n_cells, keys, idx);
        ok = cub::DeviceRadixSort::SortPairs(p + o_sort, sort_bytes, keys, keys2, idx, order,
                                             static_cast<int>(n_cells), 0, 32, s) == cudaSuccess;
    }
    if (ok) {
        k_pd_derivs<<<n_cells * (per_cell / 32), 32, file, s>>>(bt, W.box_tape, arena, order, m,
                                                                per_cell, idx2, x, y, z, v, dx, dy, dz);
        note_launches(6);
    }
    cudaFreeAsync(p, s);
    if (cudaGetLastError() != cudaSuccess) ok = false;
    return ok;
}

}  // namespace lfb
