// substep.cu — the per-substep stage kernels of the PBF path.
//
// Data layout in HBM (one handle, n particles):
//   x, v          float4[n]  id order; the drop-in state (SPH position/velocity buffers)
//   xstar         float4[n]  predicted positions, id order (predictpos output)
//   keys          u32[n]     cell key per id; sorted keys + perm after the sort
//   P0, P1        float4[n]  sorted-order Jacobi position buffers (w = 0)
//   L             float4[n]  sorted (x, y, z, lambda): one 16-byte load per neighbour in delta-p
//   VS            float4[n]  committed velocity, sorted order
//   VX, OM        float4[n]  velocity after XSPH / vorticity vector, sorted order
//   Q             float4[n]  sorted (x, y, z, |vorticity|) for the confinement pass
//   cell_start    i32[cells] first sorted index of each cell, -1 when empty
//   cell_end      i32[cells] one past the last sorted index (valid where start != -1)
//   scan copies   ScanPos    pair-interleaved copies of XP and the iterates (masked scans)
//   pair lists    u32[cap][n] in-range candidates per particle, SoA (PairLists)
//
// Every neighbour sweep visits, for sorted particle i, the 9 (dy, dz) rows of
// its 3x3x3 stencil in the reference's order (neighbourcells.glsl:37-47),
// each row's up-to-3-cell x-run in ascending sorted index, skipping i itself
// (foreachneighbour.glsl:1-10), and accumulates in that order.
#include <type_traits>

#include "substep.cuh"
#include "repeat_add.h"
#include "neighbours.cuh"

namespace pbf {

// Clears the cell-start entry that sorted particle i's cell got from the
// previous sort, so the dense table never needs a full memset.
__device__ __forceinline__ void unmark_cell(uint32_t i, const uint32_t* __restrict__ prev_sorted,
                                            uint32_t ncells, int32_t* __restrict__ cstart) {
    const uint32_t k = prev_sorted[i];
    if (k < ncells && (i == 0 || prev_sorted[i - 1] != k)) cstart[k] = -1;
}

// predictpos.glsl:18-38 fused with the cell key of GetHash (counting.glsl:53-57),
// and what the substep needs cleared: the previous sort's cells (its keys are
// still in prev_sorted) and the count of heavy particles (k_stencil_rows).  In
// launches of their own these took 2 to 3 us each of a small scene's substep.
template <class CP>
__global__ void __launch_bounds__(kBlock)
k_predict(const float4* __restrict__ x, const float4* __restrict__ v, float4* __restrict__ xstar,
          uint32_t* __restrict__ keys, uint32_t n, CP cp, uint32_t* status,
          const uint32_t* __restrict__ prev_sorted, uint32_t ncells, int32_t* __restrict__ cstart,
          uint32_t* __restrict__ heavy_count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *heavy_count = 0u;
    if (i >= n) return;
    unmark_cell(i, prev_sorted, ncells, cstart);
    const auto& c = cp.at(i);
    const float4 q = x[i];
    const float4 w = v[i];
    float wz = w.z;
    if (c.ext_force && q.z > c.half_gz) wz = fsub(wz, c.g2dt);  // :27-28
    const float wy = fsub(w.y, c.gdt);                             // :32
    const float3 s = make_float3(fadd(q.x, fmul(c.dt, w.x)), fadd(q.y, fmul(c.dt, wy)),
                                 fadd(q.z, fmul(c.dt, wz)));       // :34
    if (!finite3(s)) atomicOr(status, kDevNonFinite);
    xstar[i] = make_float4(s.x, s.y, s.z, 0.0f);
    keys[i] = cell_key(s, c);
}

// Cell keys of the current positions (no prediction), for diagnostics.
template <class CP>
__global__ void __launch_bounds__(kBlock)
k_keys_of(const float4* __restrict__ x, float4* __restrict__ xstar, uint32_t* __restrict__ keys,
          uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const auto& c = cp.at(i);
    const float4 q = x[i];
    xstar[i] = make_float4(q.x, q.y, q.z, 0.0f);
    keys[i] = cell_key(xyz(q), c);
}

// The same on its own, for the diagnostics.
__global__ void __launch_bounds__(kBlock)
k_unmark_cells(const uint32_t* __restrict__ prev_sorted, uint32_t n, uint32_t ncells,
               int32_t* __restrict__ cstart) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) unmark_cell(i, prev_sorted, ncells, cstart);
}

// The scene of every particle (id order): the last whose first particle is not
// after it.
__global__ void __launch_bounds__(kBlock)
k_scene_ids(const uint32_t* __restrict__ first, uint32_t scenes, uint32_t n,
            uint32_t* __restrict__ sid) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t lo = 0, hi = scenes;  // first[lo] <= i, and i < first[hi] or hi == scenes
    while (hi - lo > 1u) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (__ldg(first + mid) <= i)
            lo = mid;
        else
            hi = mid;
    }
    sid[i] = lo;
}
void launch_scene_ids(cudaStream_t st, const uint32_t* first, uint32_t scenes, uint32_t n,
                      uint32_t* sid) {
    k_scene_ids<<<grid_for(n), kBlock, 0, st>>>(first, scenes, n, sid);
}

// Marks every cell empty (-1 in both tables): one launch, 16-byte stores where
// both tables are aligned for them.
__global__ void __launch_bounds__(kBlock)
k_empty_cells(int32_t* __restrict__ start, int32_t* __restrict__ end, uint32_t ncells, bool wide) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t c = 4u * i;
    if (c >= ncells) return;
    if (wide && ncells - c >= 4u) {
        const int4 none = make_int4(-1, -1, -1, -1);
        reinterpret_cast<int4*>(start)[i] = none;
        reinterpret_cast<int4*>(end)[i] = none;
    } else {
        for (uint32_t k = c; k < ncells && k < c + 4u; ++k) start[k] = end[k] = -1;
    }
}
void launch_empty_cells(cudaStream_t st, int32_t* start, int32_t* end, uint32_t ncells) {
    const bool wide = (((uintptr_t)start | (uintptr_t)end) & 15u) == 0u;
    k_empty_cells<<<grid_for(ncells / 4u + 1u), kBlock, 0, st>>>(start, end, ncells, wide);
}

// The run-start bit of sorted particle j (neighbours.cuh: runs) from its
// position p and the previous particle's q, with the warp's 32 bits stored
// by its first lane.  Call with every lane of the warp.
__device__ __forceinline__ void store_run_bits(uint32_t j, uint32_t n, float3 p, float3 q,
                                               uint32_t* __restrict__ runs) {
    const bool start = j == 0u || j >= n || j % kRunStride == 0u ||
                       __float_as_uint(p.x) != __float_as_uint(q.x) ||
                       __float_as_uint(p.y) != __float_as_uint(q.y) ||
                       __float_as_uint(p.z) != __float_as_uint(q.z);
    const uint32_t word = __ballot_sync(0xFFFFFFFFu, start);
    // words 0 .. n / 32 exist (n / 32 + 2 are allocated); later warps write none
    if ((threadIdx.x & 31u) == 0u && (j >> 5) <= (n >> 5)) runs[j >> 5] = word;
}

// Run-start bits of a position set, indices 0..n (launch over n + 1 threads
// in whole warps).
__global__ void __launch_bounds__(kBlock)
k_run_flags(const float4* __restrict__ P, uint32_t n, uint32_t* __restrict__ runs) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    float3 p = make_float3(0.0f, 0.0f, 0.0f), q = p;
    if (j < n) {
        p = xyz(__ldg(P + j));
        if (j > 0) q = xyz(__ldg(P + j - 1));
    }
    store_run_bits(j, n, p, q, runs);
}

// Run-start bits over a sweep's whole per-particle input, for the direct
// sweeps' value runs: particle j starts a run when its position (A.xyz), or
// A.w (lambda or |vorticity|, with use_w), or B.xyz (the committed velocity,
// when B is given) differs bitwise from particle j - 1's, or at the stride
// and terminator marks of store_run_bits.  Inside such a run every candidate
// gives the same term, so a sweep adds it with repeat_step instead of a loop.
// Launch over n + 1 threads in whole warps.
__global__ void __launch_bounds__(kBlock)
k_run_flags_vals(const float4* __restrict__ A, const float4* __restrict__ B, int use_w,
                 uint32_t n, uint32_t* __restrict__ runs) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    bool start = j == 0u || j >= n || j % kRunStride == 0u;
    if (!start) {
        const float4 a = __ldg(A + j), a0 = __ldg(A + j - 1);
        start = __float_as_uint(a.x) != __float_as_uint(a0.x) ||
                __float_as_uint(a.y) != __float_as_uint(a0.y) ||
                __float_as_uint(a.z) != __float_as_uint(a0.z) ||
                (use_w && __float_as_uint(a.w) != __float_as_uint(a0.w));
        if (!start && B) {
            const float4 b = __ldg(B + j), b0 = __ldg(B + j - 1);
            start = __float_as_uint(b.x) != __float_as_uint(b0.x) ||
                    __float_as_uint(b.y) != __float_as_uint(b0.y) ||
                    __float_as_uint(b.z) != __float_as_uint(b0.z);
        }
    }
    const uint32_t word = __ballot_sync(0xFFFFFFFFu, start);
    if ((threadIdx.x & 31u) == 0u && (j >> 5) <= (n >> 5)) runs[j >> 5] = word;
}

// findcells.glsl:34-53 (start of cell(x_0) = 0 and end of cell(x_{n-1}) = n)
// fused with the gather of the predicted positions into sorted order.
// Keys >= ncells are skipped and reported through `status` (bad input only).
__global__ void __launch_bounds__(kBlock)
k_find_cells(const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ perm,
             const float4* __restrict__ xstar, float4* __restrict__ P0, uint32_t n, uint32_t ncells,
             int32_t* __restrict__ cstart, int32_t* __restrict__ cend, uint32_t* bad,
             const uint32_t* __restrict__ sid, uint32_t* __restrict__ sid_sorted, ScanPos sx,
             uint32_t* __restrict__ runs, uint32_t* status) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool valid = i < n;
    if (status) {
        // neighbourcells.glsl:83 packs a 3-cell run's count into 8 bits
        // (foreachneighbour.glsl:5 drops counts >= 128).  Particles i and
        // i + 127 at most two cells apart in key order lie in one 3-cell
        // window: flag it (conservatively: the window may span a row end).
        const bool over = valid && i + 127u < n && skeys[i + 127u] - skeys[i] <= 2u;
        if (__any_sync(0xFFFFFFFFu, over) && (threadIdx.x & 31u) == 0u &&
            !(*(volatile uint32_t*)status & kDevRunOver127))
            atomicOr(status, kDevRunOver127);
    }
    float4 p = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#ifdef PBF_CHECK
    // bounds-checked build: a bad permutation entry (the standalone cell finder
    // passes no permutation, and it and the diagnostics no status word)
    auto entry_ok = [&](uint32_t k) { return !perm || perm[k] < n; };
    if (valid && !entry_ok(i)) {
        if (status) atomicOr(status, kDevIndexFault);
        valid = false;  // (the lane stays for the warp's shuffles)
    }
#else
    auto entry_ok = [](uint32_t) { return true; };
#endif
    if (valid && P0) {
        p = __ldg(xstar + perm[i]);
        P0[i] = p;
        if (sx.xy) scanpos_store(sx, i, p.x, p.y, p.z);
    }
    if (runs && P0) {
        // run-start bits of the predicted positions (launched over n + 1
        // threads); the previous particle's position is the previous lane's,
        // or a load on a warp's first lane
        float3 q = make_float3(__shfl_up_sync(0xFFFFFFFFu, p.x, 1),
                               __shfl_up_sync(0xFFFFFFFFu, p.y, 1),
                               __shfl_up_sync(0xFFFFFFFFu, p.z, 1));
        if ((threadIdx.x & 31u) == 0u && valid && i > 0 && entry_ok(i - 1))
            q = xyz(__ldg(xstar + perm[i - 1]));
        store_run_bits(i, n, xyz(p), q, runs);
    }
    if (!valid) return;
    const uint32_t k = skeys[i];
    if (sid_sorted) sid_sorted[i] = __ldg(sid + perm[i]);
    if (k >= ncells) {
        atomicOr(bad, 1u);
        return;
    }
    if (i == 0 || skeys[i - 1] != k) cstart[k] = (int32_t)i;
    if (i + 1 == n || skeys[i + 1] != k) cend[k] = (int32_t)(i + 1);
}

// ---- neighbour visitors ------------------------------------------------------
//
// Two ways to enumerate the candidates of sorted particle i, both in the
// reference's order:
//  full  the 9 stencil rows, each row's run in ascending index, i skipped;
//  list  the candidates that were within h + skin at the substep's predicted
//        positions, stored by the first lambda sweep in that same order.
// A candidate left out of the list was farther than h + skin apart at the
// predicted positions; while every particle has moved less than
// (skin - margin) / 2 since (the guard below), it is still farther than h
// apart in floating point, so it would have contributed nothing.  Both
// visitors therefore produce the same sums, bit for bit.

template <class F>
__device__ __forceinline__ void visit_list(uint32_t i, const DevConsts& c, int32_t cnt,
                                           const NbrLists& nl, F&& f) {
    const uint32_t* __restrict__ p = nl.idx + i;
    for (int32_t k = 0; k < cnt; ++k) {
        const uint32_t j = __ldg(p + (size_t)k * nl.n);
        if (check_ok(c, j < c.n_total)) f(j);
    }
}

// Writer of particle i's exact pair list (PairLists): appends in visit order,
// counts past the capacity, and marks an overflowed list with -1.
struct PairRecorder {
    const PairLists& pl;
    uint32_t i;
    uint32_t k;
    __device__ __forceinline__ void operator()(uint32_t j) {
        if (k < pl.cap) pl.idx[(size_t)k * pl.n + i] = j;
        ++k;
    }
    __device__ __forceinline__ void finish() const {
        if (pl.cap) pl.cnt[i] = k <= pl.cap ? (int32_t)k : -1;
    }
};

// Replays particle i's exact pair list when one was recorded and fits.
template <class F>
__device__ __forceinline__ bool visit_pairs(uint32_t i, const DevConsts& c, const PairLists& pl,
                                            F&& f) {
    if (!pl.cap) return false;
    const int32_t cnt = pl.cnt[i];
    if (cnt < 0 || !check_ok(c, (uint32_t)cnt <= pl.cap)) return false;
    const uint32_t* __restrict__ p = pl.idx + i;
    if (cnt > 0) {  // the next index is loaded one entry ahead
        uint32_t jn = __ldg(p);
#pragma unroll 1
        for (int32_t k = 0; k < cnt; ++k) {
            const uint32_t j = jn;
            if (k + 1 < cnt) jn = __ldg(p + (size_t)(k + 1) * pl.n);
            if (check_ok(c, j < c.n_total)) f(j);
        }
    }
    return true;
}

// Guard: may particle i (current position pi, predicted position xi) use
// its list in a sweep whose positions have moved at most dmax from the
// predicted ones?  NaN anywhere makes the answer false.
__device__ __forceinline__ bool list_usable(const DevConsts& c, const NbrLists& nl, int32_t cnt,
                                            float3 pi, float3 xi, int dmax_slot) {
    if (!c.use_lists || cnt < 0 || dmax_slot < -1) return false;  // -2: no lists built
    const float3 dd = make_float3(pi.x - xi.x, pi.y - xi.y, pi.z - xi.z);
    const float di = sqrtf(dd.x * dd.x + dd.y * dd.y + dd.z * dd.z) * 1.0001f;
    const float dmax = dmax_slot < 0 ? 0.0f : __uint_as_float(nl.guard[dmax_slot]) * 1.0001f;
    const float coord = fmaxf(__uint_as_float(nl.guard[0]), c.wall_abs_max);
    const float margin = c.margin_h + 16.0f * 5.9604645e-8f * coord;  // 16 ulp(coord)
    return di + dmax + margin < c.skin;
}

__device__ __forceinline__ void warp_max_to(uint32_t* slot, float v) {
    // v >= 0 or NaN; non-negative floats order like their bit patterns
    uint32_t b = __float_as_uint(v);
    for (int o = 16; o > 0; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if ((threadIdx.x & 31) == 0) atomicMax(slot, b);
}

// The full-stencil visit of a sweep: direct, or scan-then-evaluate by chunks.
template <bool MASKED, class Ctr, class F>
__device__ __forceinline__ void sweep_visit(uint32_t i, Ctr&& ctr, const DevConsts& c,
                                            const int32_t* __restrict__ cstart,
                                            const int32_t* __restrict__ cend, const PairLists& pl,
                                            const ScanPos& X, float3 pi, F&& body) {
    if constexpr (MASKED)
        visit_masked<false>(i, c, pl.rows, pl.n, X, pi, [](int32_t, uint32_t) {}, body);
    else
        visit_full(i, ctr, c, cstart, cend, body);
}

// Masked stencil scan with the pair list recorded first and the pair bodies
// run from it afterwards: the scan writes the indices of the in-range
// candidates (visit order) to particle i's list, then `eval` runs on the list
// entries, read back by the same thread, so the bodies of a warp's lanes run
// together over their own list positions (the same shape as the replaying
// sweeps) instead of chunk by chunk.  A list longer than its capacity keeps
// its first `cap` entries (and is marked -1 for the replaying sweep); the
// candidates past them are found by walking the rows again from the last entry
// on (the visit order is that of the sorted indices: the rows ascend), `near(j)`
// being the in-range test, and evaluated in order.
template <bool LIST, class S, class N, class F>
__device__ __forceinline__ void scan_then_eval(uint32_t i, const DevConsts& c, const ScanPos& X,
                                               float3 pi, const PairLists& pw, S&& list, N&& near,
                                               F&& eval) {
    uint32_t* const out = pw.idx + i;
    const size_t stride = pw.n;
    uint32_t tot = 0;
    visit_masked<LIST>(i, c, pw.rows, pw.n, X, pi, list, [&](uint32_t j) {
        if (tot < pw.cap) out[(size_t)tot * stride] = j;
        ++tot;
    });
    pw.cnt[i] = tot <= pw.cap ? (int32_t)tot : -1;
    const uint32_t m = min(tot, pw.cap);
    if (m) {  // the next index is loaded one entry ahead
        uint32_t jn = out[0];
#pragma unroll 1
        for (uint32_t k = 0; k < m; ++k) {
            const uint32_t j = jn;
            if (k + 1 < m) jn = out[(size_t)(k + 1) * stride];
            eval(j);
        }
    }
    if (tot > pw.cap) {
        const int32_t from = (int32_t)out[(size_t)(pw.cap - 1u) * stride] + 1;
#pragma unroll 1
        for (int o = 0; o < 9; ++o) {
            const int2 be = __ldg(pw.rows + (size_t)o * pw.n + i);
#pragma unroll 1
            for (int32_t j = max(be.x, from); j < be.y; ++j)
                if ((uint32_t)j != i && near((uint32_t)j)) eval((uint32_t)j);
        }
    }
}

// ---- pair bodies (shared by both visitors) ---------------------------------------

struct LambdaAcc {
    float rho, sumk;
    float3 gi;
};

// calclambda.glsl:75-95 for one neighbour at offset d = p_i - p_j, r2 = |d|^2.
// (call only for r2 not above r2cut: len > h gives Wpoly6 = gradWspiky = 0)
__device__ __forceinline__ void lambda_pair(const DevConsts& c, float3 d, float r2, LambdaAcc& a) {
    const float len = fsqrt(r2);
    a.rho = fadd(a.rho, w_poly6(c, len));  // :80-82
    if (len == 0.0f) return;               // gradWspiky(0) = 0 (:60)
    const float3 g = scale3(d, grad_scale(c.kg_lambda, c.h, len));  // :86-87
    a.sumk = fadd(a.sumk, dot3(g, g));     // :89
    a.gi = add3(a.gi, g);                  // :93
}

// lambda_pair for m neighbours at the same offset d (a run of equal
// positions): each of the four sums receives its term m times, as m calls
// would add it (repeat_add: the same bits).
__device__ __forceinline__ void lambda_pair_run(const DevConsts& c, float3 d, float r2,
                                                uint32_t m, LambdaAcc& a) {
    if (r2 > c.r2cut) return;
    const float len = fsqrt(r2);
    a.rho = repeat_add(a.rho, w_poly6(c, len), m);  // :80-82
    if (len == 0.0f) return;
    const float3 g = scale3(d, grad_scale(c.kg_lambda, c.h, len));  // :86-87
    a.sumk = repeat_add(a.sumk, dot3(g, g), m);                      // :89
    a.gi = make_float3(repeat_add(a.gi.x, g.x, m), repeat_add(a.gi.y, g.y, m),
                       repeat_add(a.gi.z, g.z, m));  // :93
}

// What the adjoint needs of a lambda evaluation: sum_j grad_pj C_i (the
// gradient w.r.t. p_i, calclambda.glsl:93) and the full denominator sum
// before epsilon (:89,97).
__device__ __forceinline__ float4 lambda_aux(const LambdaAcc& a) {
    return make_float4(a.gi.x, a.gi.y, a.gi.z, fadd(a.sumk, dot3(a.gi, a.gi)));
}

// calclambda.glsl:97-101
__device__ __forceinline__ float lambda_finish(const DevConsts& c, const LambdaAcc& a) {
    const float sumk = fadd(a.sumk, dot3(a.gi, a.gi));  // :97
    const float Ci = ffma(a.rho, c.oorho, -1.0f);        // :100
    return fdiv(-Ci, fadd(sumk, c.eps));                 // :101
}

// ---- solver kernels --------------------------------------------------------------

// Resident 256-thread blocks per SM the sweep kernels are compiled for (caps
// them at 32 registers: full occupancy hides the gather and sqrt/div latency;
// 6 or 4 blocks with more registers measured slower).  One thread per sorted
// particle.
constexpr int kSweepBlocksPerSM = 8;
// The first vorticity pass carries more state than the other sweeps (the
// XSPH and vorticity sums, the velocity, the run path's repeated steps): 6
// blocks per SM (40 registers) keep it from spilling; measured 10% faster
// than 8 blocks with spills on the 2M window.
constexpr int kVortThreadsPerSM = 1536;

// Instantiations of the sweep kernels (pbf_tuning): MODE is the stencil scan
// (kDirect: the reference's loop shape; kMasked: masked scans; kPairs: masked
// scans recording the exact pair lists the next sweep replays), LISTS whether
// the skin-radius neighbour lists are compiled in.  Every instantiation gives
// the same bits.
constexpr int kDirect = 0, kMasked = 1, kPairs = 2;

// First lambda sweep of a substep (calclambda.glsl:66-102) at the predicted
// positions XP: a full stencil scan that also records, in visit order, every
// candidate within h + skin (the neighbour list of the later sweeps) and the
// largest coordinate magnitude (for the guard's rounding margin).
template <class CP, int MODE, bool LISTS>
__global__ void __launch_bounds__(kLambdaMaxBlock, 2048 / kLambdaMaxBlock)
k_lambda_build(const float4* __restrict__ XP, const uint32_t* __restrict__ skeys,
               const int32_t* __restrict__ cstart, const int32_t* __restrict__ cend,
               float4* __restrict__ L, float4* __restrict__ aux, NbrLists nl, PairLists pw,
               ScanPos sx, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < n && !(pw.heavy && pw.heavy[i]);
    float3 pi = make_float3(0.0f, 0.0f, 0.0f);
    if (live) {
        const auto& c = cp.at(i);
        pi = xyz(XP[i]);
        auto ctr = [&] { return stencil_centre(pi, c); };  // neighbourcells.glsl:57
        LambdaAcc a{0.0f, 0.0f, make_float3(0.0f, 0.0f, 0.0f)};
        int32_t cnt = 0;
        const uint32_t cap = (LISTS && c.use_lists) ? nl.cap : 0u;
        auto list_rec = [&](int32_t base, uint32_t lm) {
            while (lm) {
                const int t = __ffs(lm) - 1;
                lm &= lm - 1;
                if ((uint32_t)cnt < cap) nl.idx[(size_t)cnt * n + i] = (uint32_t)(base + t);
                ++cnt;
            }
        };
        auto eval = [&](uint32_t j) {
            const float3 d = sub3(pi, xyz(__ldg(XP + j)));
            lambda_pair(c, d, dot3(d, d), a);
        };
        auto near = [&](uint32_t j) {
            const float3 d = sub3(pi, xyz(__ldg(XP + j)));
            return !(dot3(d, d) > c.r2cut);
        };
        if constexpr (MODE == kPairs) {
            if (LISTS && cap)
                scan_then_eval<true>(i, c, sx, pi, pw, list_rec, near, eval);
            else
                scan_then_eval<false>(i, c, sx, pi, pw, [](int32_t, uint32_t) {}, near, eval);
        } else if constexpr (MODE == kMasked) {
            if (LISTS && cap)
                visit_masked<true>(i, c, pw.rows, n, sx, pi, list_rec, eval);
            else
                visit_masked<false>(i, c, pw.rows, n, sx, pi, [](int32_t, uint32_t) {}, eval);
        } else {
            bool piles = false;
            if constexpr (!LISTS) {
                if (pw.runs) {
                    // a coincident neighbour adds W(0) to the density (:80-82)
                    visit_direct_piles(
                        i, ctr, c, cstart, cend, pw.runs,
                        [&](uint32_t j) { return xyz(__ldg(XP + j)); }, pi,
                        [&](uint32_t j) {
                            const float3 d = sub3(pi, xyz(__ldg(XP + j)));
                            const float r2 = dot3(d, d);
                            if (r2 > c.r2cut) return;
                            lambda_pair(c, d, r2, a);
                        },
                        [&](uint32_t, uint32_t, uint32_t m) { a.rho = repeat_add(a.rho, w_poly6(c, 0.0f), m); },
                        [&](uint32_t j0, uint32_t r, float3 d, float r2) {
                            lambda_pair_run(c, d, r2, r - j0, a);
                        });
                    piles = true;
                }
            }
            if (!piles)
                visit_full(i, ctr, c, cstart, cend, [&](uint32_t j) {
                    const float3 d = sub3(pi, xyz(__ldg(XP + j)));
                    const float r2 = dot3(d, d);
                    if (LISTS && r2 <= c.r2list) {
                        if ((uint32_t)cnt < cap) nl.idx[(size_t)cnt * n + i] = j;
                        ++cnt;
                    }
                    if (r2 > c.r2cut) return;
                    lambda_pair(c, d, r2, a);
                });
        }
        if (LISTS) nl.cnt[i] = (uint32_t)cnt <= cap ? cnt : -1;
        L[i] = make_float4(pi.x, pi.y, pi.z, lambda_finish(c, a));
        if (aux) aux[i] = lambda_aux(a);
    }
    if (LISTS) {
        const float m = fmaxf(fmaxf(fabsf(pi.x), fabsf(pi.y)), fabsf(pi.z));
        warp_max_to(nl.guard, m);
    }
}

// calclambda.glsl:66-102 at positions P (iterations after the first).
// dmax_slot: guard slot holding the largest displacement of P from XP.
template <class CP, int MODE, bool LISTS>
__global__ void __launch_bounds__(kLambdaMaxBlock, 2048 / kLambdaMaxBlock)
k_lambda(const float4* __restrict__ P, const float4* __restrict__ XP,
         const uint32_t* __restrict__ skeys, const int32_t* __restrict__ cstart,
         const int32_t* __restrict__ cend, float4* __restrict__ L, float4* __restrict__ aux,
         NbrLists nl, PairLists pw, ScanPos sx, int dmax_slot, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (pw.heavy && pw.heavy[i])) return;
    const auto& c = cp.at(i);
    const float3 pi = xyz(P[i]);
    auto ctr = [&] { return stencil_centre(XP[i], c); };  // neighbourcells.glsl:57
    LambdaAcc a{0.0f, 0.0f, make_float3(0.0f, 0.0f, 0.0f)};
    // in_range: the candidate is known to pass the in-range test (the
    // masked scans computed the same r2 bit for bit), so the test is skipped
    auto eval_in = [&](uint32_t j) {
        const float3 d = sub3(pi, xyz(__ldg(P + j)));
        lambda_pair(c, d, dot3(d, d), a);
    };
    auto near = [&](uint32_t j) {
        const float3 d = sub3(pi, xyz(__ldg(P + j)));
        return !(dot3(d, d) > c.r2cut);
    };
    auto eval = [&](uint32_t j) {
        const float3 d = sub3(pi, xyz(__ldg(P + j)));
        const float r2 = dot3(d, d);
        if (r2 > c.r2cut) return;
        lambda_pair(c, d, r2, a);
    };
    bool listed = false;
    if constexpr (LISTS) {
        const int32_t cnt = nl.cnt[i];
        if (list_usable(c, nl, cnt, pi, xyz(XP[i]), dmax_slot)) {
            listed = true;
            if constexpr (MODE == kPairs) {
                PairRecorder rec{pw, i, 0u};
                visit_list(i, c, cnt, nl, [&](uint32_t j) {
                    const float3 d = sub3(pi, xyz(__ldg(P + j)));
                    if (!(dot3(d, d) > c.r2cut)) rec(j);
                    eval(j);
                });
                rec.finish();
            } else {
                visit_list(i, c, cnt, nl, eval);
            }
        }
    }
    if (!listed) {
        if constexpr (MODE == kPairs)
            scan_then_eval<false>(i, c, sx, pi, pw, [](int32_t, uint32_t) {}, near, eval_in);
        else if constexpr (MODE == kMasked)
            sweep_visit<true>(i, ctr, c, cstart, cend, pw, sx, pi, eval_in);
        else if (!LISTS && pw.runs)
            visit_direct_piles(
                i, ctr, c, cstart, cend, pw.runs,
                [&](uint32_t j) { return xyz(__ldg(P + j)); }, pi, eval,
                [&](uint32_t, uint32_t, uint32_t m) { a.rho = repeat_add(a.rho, w_poly6(c, 0.0f), m); },
                [&](uint32_t j0, uint32_t r, float3 d, float r2) {
                    lambda_pair_run(c, d, r2, r - j0, a);
                });
        else
            sweep_visit<false>(i, ctr, c, cstart, cend, pw, sx, pi, eval);
    }
    L[i] = make_float4(pi.x, pi.y, pi.z, lambda_finish(c, a));
    if (aux) aux[i] = lambda_aux(a);
}

// updatepos.glsl:42-104.  Reads L = (p, lambda), writes clamped positions Pn
// and the largest displacement of Pn from XP into guard slot `out_slot`.
template <class CP, int MODE, bool LISTS>
__global__ void __launch_bounds__(kBlock, kSweepBlocksPerSM)
k_delta_p(const float4* __restrict__ L, const float4* __restrict__ XP,
          const uint32_t* __restrict__ skeys, const int32_t* __restrict__ cstart,
          const int32_t* __restrict__ cend, float4* __restrict__ Pn, NbrLists nl, PairLists pr,
          ScanPos sx, ScanPos sx_out, int dmax_slot, int out_slot, uint32_t n, CP cp,
          uint32_t* status) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < n && !(pr.heavy && pr.heavy[i]);
    float disp = 0.0f;
    if (live) {
        const auto& c = cp.at(i);
        const float4 Li = L[i];
        const float3 pi = xyz(Li);
        const float li = Li.w;
        float3 dp = make_float3(0.0f, 0.0f, 0.0f);
        auto body = [&](uint32_t j) {
            const float4 Lj = __ldg(L + j);
            const float3 d = sub3(pi, xyz(Lj));
            const float r2 = dot3(d, d);
            if (r2 > c.r2cut) return;
            const float len = fsqrt(r2);
            if (len == 0.0f) return;
            float sc = fmul(c.scale, w_poly6(c, len));  // :57
            sc = fmul(sc, sc);                           // :58
            sc = fmul(sc, sc);                           // :59
            sc = fmul(c.negk, sc);                       // :60
            const float coef = fadd(fadd(li, Lj.w), sc); // :65
            const float3 g = scale3(d, grad_scale(c.kg, c.h, len));
            dp = fma3(coef, g, dp);                      // :65
        };
        const float3 xi = xyz(XP[i]);
        auto ctr = [&] { return stencil_centre(XP[i], c); };  // neighbourcells.glsl:57
        bool done = false;
        if constexpr (MODE == kPairs) done = visit_pairs(i, c, pr, body);
        if (!done) {
            bool listed = false;
            if constexpr (LISTS) {
                const int32_t cnt = nl.cnt[i];
                if (list_usable(c, nl, cnt, pi, xi, dmax_slot)) {
                    visit_list(i, c, cnt, nl, body);
                    listed = true;
                }
            }
            if (!listed) {
                if (MODE == kDirect && !LISTS && pr.runs)  // coincident: no term (:56)
                    visit_direct_piles(
                        i, ctr, c, cstart, cend, pr.runs,
                        [&](uint32_t j) { return xyz(__ldg(L + j)); }, pi, body, [](uint32_t, uint32_t, uint32_t) {},
                        [&](uint32_t j0, uint32_t r, float3 d, float r2) {
                            // one offset and, the run bits being over (p, lambda),
                            // one lambda_j: r - j0 equal terms in a row
                            if (r2 > c.r2cut) return;
                            const float len = fsqrt(r2);
                            float sc = fmul(c.scale, w_poly6(c, len));  // :57
                            sc = fmul(sc, sc);                           // :58
                            sc = fmul(sc, sc);                           // :59
                            sc = fmul(c.negk, sc);                       // :60
                            const float3 g = scale3(d, grad_scale(c.kg, c.h, len));
                            const float coef = fadd(fadd(li, __ldg(&L[j0].w)), sc);  // :65
                            dp = repeat_fma3(coef, g, dp, r - j0);
                        });
                else
                    sweep_visit<MODE != kDirect>(i, ctr, c, cstart, cend, pr, sx, pi, body);
            }
        }
        float3 q = fma3(c.oorho, dp, pi);  // :85
        // clamp (:100) as min(max(q, lo), hi) with explicit selects, so signed
        // zeros and NaN behave like the oracle's std::min/std::max
        q.x = (q.x < c.lo[0]) ? c.lo[0] : q.x;
        q.x = (c.hi[0] < q.x) ? c.hi[0] : q.x;
        q.y = (q.y < c.lo[1]) ? c.lo[1] : q.y;
        q.y = (c.hi[1] < q.y) ? c.hi[1] : q.y;
        q.z = (q.z < c.lo[2]) ? c.lo[2] : q.z;
        q.z = (c.hi[2] < q.z) ? c.hi[2] : q.z;
        if (!finite3(q)) atomicOr(status, kDevNonFinite);
        Pn[i] = make_float4(q.x, q.y, q.z, 0.0f);
        if (sx_out.xy) scanpos_store(sx_out, i, q.x, q.y, q.z);
        if (LISTS) {
            const float3 dd = make_float3(q.x - xi.x, q.y - xi.y, q.z - xi.z);
            disp = sqrtf(dd.x * dd.x + dd.y * dd.y + dd.z * dd.z);
        }
    }
    if (LISTS) warp_max_to(nl.guard + out_slot, disp);
}

// ---- warp-cooperative sweeps (sweep_mode PBF_SWEEP_COOP) ---------------------------
//
// One warp per sorted particle i, for scenes too small to fill the GPU with a
// thread per particle (and for clumped states, where each particle has
// thousands of neighbours).  The warp's 32 lanes walk the 9 stencil rows as
// one flattened candidate sequence (visit order), 32 candidates per step:
//  1. every lane tests its candidate; the in-range ones are appended, in
//     order, to a queue in shared memory (offset d and one payload word);
//  2. when 32 are queued, every lane evaluates one pair and stores its terms
//     in shared memory, one row per term component;
//  3. lane c folds component c of the 32 terms into the particle's sum, in
//     order, four terms per shared-memory load.
// The terms are the same functions and the folding order the same visit order
// as the one-thread sweeps, so the bits are the same.
//
// What bounds it: instruction issue.  Evaluating a pair on the lane that found
// it and folding it on all lanes from shuffles spends ~14 instructions per
// term for the fold and an evaluation per 32-candidate step whatever the number
// in range (5 of 32 in a lattice at rest); queued, a full batch costs ~80
// instructions of evaluation and ~45 of folding for 32 terms.  The stencil
// rows are found by 9 lanes at once instead of by every lane in turn.
// Measured per launch against the shuffled fold.  16,384 particles at rest:
// lambda 30.6 -> 17.9 us, delta-p 30.2 -> 18.2, vorticity 36.7 -> 22.2 and
// 28.0 -> 19.4; ncu: 900 warp instructions per particle, issue slots 65% busy
// (the grid is 2.7 waves).  The same scene collapsed (substep 96): lambda
// 2,043 -> 221 us, the first vorticity pass 2,368 -> 386.  The heavy particles
// of 2,097,152 (20 substeps): lambda 287 -> 81 us, delta-p 114 -> 60.  Blocks
// of 2 warps instead of 8 measured the same.
//
// Piles of coincident particles: a step whose 32 candidates all carry the same
// offset and payload is not queued but counted, and a counted stretch is added
// with repeat_step (repeat_add.h: the bits of the sequential sum).
constexpr int kCoop = 3;
constexpr uint32_t kFull = 0xFFFFFFFFu;
// A step looks for equal candidates from this many stencil candidates up: below,
// piles are too short to pay for the test (an interior particle of the lattice
// at rest has 216 candidates).
constexpr uint32_t kCoopRunsFrom = 256;

__device__ __forceinline__ float shf(float v, int src) { return __shfl_sync(kFull, v, src); }
__device__ __forceinline__ float3 shf3(float3 v, int src) {
    return make_float3(shf(v.x, src), shf(v.y, src), shf(v.z, src));
}
__device__ __forceinline__ bool same_bits(float a, float b) {
    return __float_as_uint(a) == __float_as_uint(b);
}
__device__ __forceinline__ bool same_bits3(float3 a, float3 b) {
    return same_bits(a.x, b.x) && same_bits(a.y, b.y) && same_bits(a.z, b.z);
}

// A warp's share of shared memory.  Term rows are 36 floats apart, so that the
// 16-byte loads of up to 8 rows at one column fall in different banks.
constexpr int kCoopRows = 8;
struct CoopShared {
    float4 queue[64];
    float t[kCoopRows][36];
    int2 run[10];
};

// The pair terms of each sweep.  kRows term rows; lane c < kSums keeps sum c,
// acc <- fma(row s_row(c), row a_row(c), acc), or acc + row a_row(c) where
// kAdd.  kSkipCoincident: a candidate at distance 0 has no term.  payload() is
// the word queued with a candidate, same() whether two payloads give the same
// term.
struct CoopLambda {
    static constexpr int kRows = 5, kSums = 5;
    static constexpr bool kAdd = true, kSkipCoincident = false;
    static __device__ __forceinline__ int s_row(int) { return 0; }
    static __device__ __forceinline__ int a_row(int c) { return c; }
    __device__ __forceinline__ float payload(uint32_t, float4) const { return 0.0f; }
    __device__ __forceinline__ bool same(float, float) const { return true; }
    __device__ __forceinline__ void terms(const DevConsts& c, float3 d, float r2, float,
                                          float* t) const {
        const float len = fsqrt(r2);
        t[0] = w_poly6(c, len);  // calclambda.glsl:80-82
        // a coincident candidate adds no gradient (:60); +0 leaves the other
        // four sums as they are (they start at +0, so none is ever -0)
        float3 g = make_float3(0.0f, 0.0f, 0.0f);
        if (len != 0.0f) g = scale3(d, grad_scale(c.kg_lambda, c.h, len));  // :86-87
        t[1] = dot3(g, g);                                                   // :89
        t[2] = g.x;                                                          // :93
        t[3] = g.y;
        t[4] = g.z;
    }
};
struct CoopDeltaP {
    static constexpr int kRows = 4, kSums = 3;
    static constexpr bool kAdd = false, kSkipCoincident = true;
    float li;
    static __device__ __forceinline__ int s_row(int) { return 0; }
    static __device__ __forceinline__ int a_row(int c) { return 1 + c; }
    __device__ __forceinline__ float payload(uint32_t, float4 Lj) const { return Lj.w; }
    __device__ __forceinline__ bool same(float a, float b) const { return same_bits(a, b); }
    __device__ __forceinline__ void terms(const DevConsts& c, float3 d, float r2, float lj,
                                          float* t) const {
        const float len = fsqrt(r2);
        float sc = fmul(c.scale, w_poly6(c, len));  // updatepos.glsl:57
        sc = fmul(sc, sc);                           // :58
        sc = fmul(sc, sc);                           // :59
        sc = fmul(c.negk, sc);                       // :60
        t[0] = fadd(fadd(li, lj), sc);               // :65
        const float3 g = scale3(d, grad_scale(c.kg, c.h, len));
        t[1] = g.x;
        t[2] = g.y;
        t[3] = g.z;
    }
};
struct CoopVortA {
    static constexpr int kRows = 8, kSums = 6;
    static constexpr bool kAdd = false, kSkipCoincident = false;
    const float4* __restrict__ VS;
    float3 vi;
    // sums 0-2 (XSPH) scale by row 0, sums 3-5 (vorticity) by row 1 (ones:
    // fma(1, a, acc) is the rounded acc + a)
    static __device__ __forceinline__ int s_row(int c) { return c < 3 ? 0 : 1; }
    static __device__ __forceinline__ int a_row(int c) { return 2 + c; }
    __device__ __forceinline__ float payload(uint32_t j, float4) const {
        return __uint_as_float(j);
    }
    __device__ __forceinline__ bool same(float a, float b) const {
        return same_bits3(xyz(__ldg(VS + __float_as_uint(a))), xyz(__ldg(VS + __float_as_uint(b))));
    }
    __device__ __forceinline__ void terms(const DevConsts& c, float3 d, float r2, float j,
                                          float* t) const {
        const float len = fsqrt(r2);
        const float3 v = sub3(xyz(__ldg(VS + __float_as_uint(j))), vi);  // vorticity.glsl:50
        t[0] = w_poly6(c, len);                                           // :52-54
        t[1] = 1.0f;
        t[2] = v.x;
        t[3] = v.y;
        t[4] = v.z;
        // (a coincident candidate adds no curl; +0 keeps a sum that starts at +0)
        float3 w = make_float3(0.0f, 0.0f, 0.0f);
        if (len != 0.0f) w = cross3(v, scale3(d, grad_scale(c.kg, c.h, len)));  // :55
        t[5] = w.x;
        t[6] = w.y;
        t[7] = w.z;
    }
};
struct CoopVortB {
    static constexpr int kRows = 4, kSums = 3;
    static constexpr bool kAdd = false, kSkipCoincident = true;
    static __device__ __forceinline__ int s_row(int) { return 0; }
    static __device__ __forceinline__ int a_row(int c) { return 1 + c; }
    __device__ __forceinline__ float payload(uint32_t, float4 Qj) const { return Qj.w; }
    __device__ __forceinline__ bool same(float a, float b) const { return same_bits(a, b); }
    __device__ __forceinline__ void terms(const DevConsts& c, float3 d, float r2, float qj,
                                          float* t) const {
        t[0] = qj;  // vorticity.glsl:72
        const float3 g = scale3(d, grad_scale(c.kg, c.h, fsqrt(r2)));
        t[1] = g.x;
        t[2] = g.y;
        t[3] = g.z;
    }
};

// Sweeps particle i's stencil with one warp (every lane calls);
// lane c < Op::kSums returns sum c, the other lanes sum 0.
template <class Op>
__device__ __forceinline__ float coop_visit(uint32_t i, const DevConsts& c,
                                            const int2* __restrict__ rows, uint32_t n,
                                            const float4* __restrict__ X, float3 pi,
                                            CoopShared& sm, const Op& op) {
    const int lane = (int)(threadIdx.x & 31u);
    const uint32_t before = (1u << lane) - 1u;
    int2 mine = make_int2(0, lane == 9 ? 0x7FFFFFFF : 0);  // row 9 ends the sequence
    if (lane < 9) {
        mine = __ldg(rows + (size_t)lane * n + i);
        if (!check_ok(c, mine.x >= 0 && mine.x <= mine.y && (uint32_t)mine.y <= n))
            mine = make_int2(0, 0);
    }
    if (lane < 10) sm.run[lane] = mine;
    const bool look = __reduce_add_sync(kFull, lane < 9 ? (uint32_t)(mine.y - mine.x) : 0u) >=
                      kCoopRunsFrom;
    const int sum = lane < Op::kSums ? lane : 0;
    const float* const arow = sm.t[Op::a_row(sum)];
    const float* const srow = sm.t[Op::s_row(sum)];
    float acc = 0.0f;
    uint32_t qn = 0, qh = 0;  // queued candidates; the queue's head (0 or 32)
    // a stretch of `pm` equal candidates waiting to be added (the queue is then empty)
    uint32_t pm = 0;
    float3 pd = make_float3(0.0f, 0.0f, 0.0f);
    float pp = 0.0f;
    __syncwarp();

    auto batch = [&](uint32_t cnt) {  // evaluate and fold the queue's first cnt (<= 32)
        if ((uint32_t)lane < cnt) {
            const float4 e = sm.queue[qh + lane];
            const float3 d = xyz(e);
            float t[Op::kRows];
            op.terms(c, d, dot3(d, d), e.w, t);
#pragma unroll
            for (int k = 0; k < Op::kRows; ++k) sm.t[k][lane] = t[k];
        }
        __syncwarp();
        uint32_t k = 0;
#pragma unroll 2
        for (; k + 4 <= cnt; k += 4) {
            const float4 a = *reinterpret_cast<const float4*>(arow + k);
            if constexpr (Op::kAdd) {
                acc = fadd(fadd(fadd(fadd(acc, a.x), a.y), a.z), a.w);
            } else {
                const float4 s = *reinterpret_cast<const float4*>(srow + k);
                acc = ffma(s.w, a.w, ffma(s.z, a.z, ffma(s.y, a.y, ffma(s.x, a.x, acc))));
            }
        }
        for (; k < cnt; ++k) acc = Op::kAdd ? fadd(acc, arow[k]) : ffma(srow[k], arow[k], acc);
        __syncwarp();
    };
    auto add_stretch = [&] {  // pm equal candidates in a row
        float t[Op::kRows];
        op.terms(c, pd, dot3(pd, pd), pp, t);
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < Op::kRows; ++k) sm.t[k][0] = t[k];
        }
        __syncwarp();
        const float a = arow[0], s = srow[0];
        if constexpr (Op::kAdd)
            acc = repeat_add(acc, a, pm);
        else
            acc = repeat_step(acc, pm, [s, a](float x) { return ffma(s, a, x); });
        pm = 0;
        __syncwarp();
    };

    int row = 0;
    int2 be = sm.run[0];
    int j = be.x + lane;
    for (;; j += 32) {
        while (j >= be.y && row < 9) {  // past its row: the lane goes on in the next one
            const int over = j - be.y;
            be = sm.run[++row];
            j = be.x + over;
        }
        const bool valid = row < 9;
        if (!__any_sync(kFull, valid)) break;
        float3 d = make_float3(0.0f, 0.0f, 0.0f);
        float r2 = 0.0f, pay = 0.0f;
        bool in = false;
        if (valid) {
            const float4 xj = __ldg(X + j);
            d = sub3(pi, xyz(xj));
            r2 = dot3(d, d);
            pay = op.payload((uint32_t)j, xj);
            in = !(r2 > c.r2cut) && (uint32_t)j != i && !(Op::kSkipCoincident && r2 == 0.0f);
        }
        const uint32_t m = __ballot_sync(kFull, in);
        if (m == 0u) continue;
        // all 32 candidates equal (the particle itself may be one of them)?
        if (look) {
            const float r20 = shf(r2, 0);
            if (__all_sync(kFull, valid && r2 == r20)) {
                const float3 d0 = shf3(d, 0);
                const float p0 = shf(pay, 0);
                if (__all_sync(kFull, same_bits3(d, d0) && op.same(pay, p0))) {
                    if (pm == 0u || !(same_bits3(pd, d0) && op.same(pp, p0))) {
                        if (pm) add_stretch();
                        if (qn) batch(qn);
                        qn = 0;
                        pd = d0;
                        pp = p0;
                    }
                    pm += (uint32_t)__popc(m);
                    continue;
                }
            }
        }
        if (pm) add_stretch();
        if (in) sm.queue[(qh + qn + (uint32_t)__popc(m & before)) & 63u] =
            make_float4(d.x, d.y, d.z, pay);
        qn += (uint32_t)__popc(m);
        __syncwarp();
        if (qn >= 32u) {
            batch(32u);
            qh ^= 32u;
            qn -= 32u;
        }
    }
    if (pm) add_stretch();
    if (qn) batch(qn);
    return acc;
}

// Particles a cooperative kernel processes: all n (list == nullptr, one warp
// per particle), or the `*count` entries of `list` (the heavy particles of a
// mixed sweep), taken by the grid's warps in turn.
struct CoopWork {
    const uint32_t* list;
    const uint32_t* count;
};

// What one lane does with a particle's sums.
// updatepos.glsl:100: the clamp as min(max(q, lo), hi) with explicit selects,
// so signed zeros and NaN behave like the oracle's std::min/std::max.
__device__ __forceinline__ void store_position(uint32_t i, float3 q, const DevConsts& c,
                                               float4* __restrict__ Pn, const ScanPos& sx_out,
                                               uint32_t* status) {
    q.x = (q.x < c.lo[0]) ? c.lo[0] : q.x;
    q.x = (c.hi[0] < q.x) ? c.hi[0] : q.x;
    q.y = (q.y < c.lo[1]) ? c.lo[1] : q.y;
    q.y = (c.hi[1] < q.y) ? c.hi[1] : q.y;
    q.z = (q.z < c.lo[2]) ? c.lo[2] : q.z;
    q.z = (c.hi[2] < q.z) ? c.hi[2] : q.z;
    if (!finite3(q)) atomicOr(status, kDevNonFinite);
    Pn[i] = make_float4(q.x, q.y, q.z, 0.0f);
    if (sx_out.xy) scanpos_store(sx_out, i, q.x, q.y, q.z);
}
__device__ __forceinline__ void store_vorticity(uint32_t i, float3 pi, float3 vi, float3 acc,
                                                float3 w, const DevConsts& c,
                                                float4* __restrict__ VX, float4* __restrict__ OM,
                                                float4* __restrict__ Q) {
    const float3 vx = fma3(c.cx, acc, vi);  // vorticity.glsl:58
    VX[i] = make_float4(vx.x, vx.y, vx.z, 0.0f);
    OM[i] = make_float4(w.x, w.y, w.z, 0.0f);
    Q[i] = make_float4(pi.x, pi.y, pi.z, fsqrt(dot3(w, w)));  // :60
}
__device__ __forceinline__ void store_velocity(uint32_t i, float3 eta, const DevConsts& c,
                                               const float4* __restrict__ VX,
                                               const float4* __restrict__ OM,
                                               const uint32_t* __restrict__ perm,
                                               float4* __restrict__ v,
                                               float4* __restrict__ eta_out) {
    if (eta_out) eta_out[i] = make_float4(eta.x, eta.y, eta.z, 0.0f);
    const float l = fsqrt(dot3(eta, eta));  // vorticity.glsl:76
    if (l > 0.0f) eta = make_float3(fdiv(eta.x, l), fdiv(eta.y, l), fdiv(eta.z, l));  // :77-78
    const float3 vf = fma3(c.dteps, cross3(eta, xyz(OM[i])), xyz(VX[i]));  // :82
    if (check_ok(c, perm[i] < c.n_total)) v[perm[i]] = make_float4(vf.x, vf.y, vf.z, 0.0f);  // :85
}

// One particle by one warp (every lane calls).
struct LambdaCoop {
    const float4* __restrict__ P;
    float4* __restrict__ L;
    float4* __restrict__ aux;
    const int2* __restrict__ rows;
    uint32_t n;
    __device__ __forceinline__ void operator()(uint32_t i, const DevConsts& c,
                                               CoopShared& sm) const {
        const float3 pi = xyz(P[i]);
        const float s = coop_visit(i, c, rows, n, P, pi, sm, CoopLambda{});
        const LambdaAcc a{shf(s, 0), shf(s, 1), make_float3(shf(s, 2), shf(s, 3), shf(s, 4))};
        if ((threadIdx.x & 31u) == 0u) {
            L[i] = make_float4(pi.x, pi.y, pi.z, lambda_finish(c, a));
            if (aux) aux[i] = lambda_aux(a);
        }
    }
};
struct DeltaPCoop {
    const float4* __restrict__ L;
    float4* __restrict__ Pn;
    ScanPos sx_out;
    const int2* __restrict__ rows;
    uint32_t n;
    uint32_t* status;
    __device__ __forceinline__ void operator()(uint32_t i, const DevConsts& c,
                                               CoopShared& sm) const {
        const float4 Li = L[i];
        const float3 pi = xyz(Li);
        const float s = coop_visit(i, c, rows, n, L, pi, sm, CoopDeltaP{Li.w});
        const float3 dp = make_float3(shf(s, 0), shf(s, 1), shf(s, 2));
        if ((threadIdx.x & 31u) == 0u)
            store_position(i, fma3(c.oorho, dp, pi), c, Pn, sx_out, status);  // :85
    }
};
struct VortACoop {
    const float4* __restrict__ P;
    const float4* __restrict__ VS;
    float4* __restrict__ VX;
    float4* __restrict__ OM;
    float4* __restrict__ Q;
    const int2* __restrict__ rows;
    uint32_t n;
    __device__ __forceinline__ void operator()(uint32_t i, const DevConsts& c,
                                               CoopShared& sm) const {
        const float3 pi = xyz(P[i]);
        const float3 vi = xyz(VS[i]);
        const float s = coop_visit(i, c, rows, n, P, pi, sm, CoopVortA{VS, vi});
        const float3 acc = make_float3(shf(s, 0), shf(s, 1), shf(s, 2));
        const float3 w = make_float3(shf(s, 3), shf(s, 4), shf(s, 5));
        if ((threadIdx.x & 31u) == 0u) store_vorticity(i, pi, vi, acc, w, c, VX, OM, Q);
    }
};
struct VortBCoop {
    const float4* __restrict__ Q;
    const float4* __restrict__ VX;
    const float4* __restrict__ OM;
    const uint32_t* __restrict__ perm;
    float4* __restrict__ v;
    float4* __restrict__ eta_out;
    const int2* __restrict__ rows;
    uint32_t n;
    __device__ __forceinline__ void operator()(uint32_t i, const DevConsts& c,
                                               CoopShared& sm) const {
        const float3 pi = xyz(Q[i]);
        const float s = coop_visit(i, c, rows, n, Q, pi, sm, CoopVortB{});
        const float3 eta = make_float3(shf(s, 0), shf(s, 1), shf(s, 2));
        if ((threadIdx.x & 31u) == 0u) store_velocity(i, eta, c, VX, OM, perm, v, eta_out);
    }
};

// The particles of `wk`, taken in turn by `warps` warps of which this is the
// w-th: `body` on each.
template <class CP, class Body>
__device__ __forceinline__ void coop_each(uint32_t w, uint32_t warps, const CoopWork& wk,
                                          uint32_t n, const CP& cp, CoopShared& sm,
                                          const Body& body) {
    const uint32_t total = wk.list ? *wk.count : n;
    for (; w < total; w += warps) {
        const uint32_t i = wk.list ? wk.list[w] : w;
        if (check_ok(cp.at(0), i < n)) body(i, cp.at(i), sm);
    }
}

template <class CP, class Body>
__global__ void __launch_bounds__(kBlock) k_coop(Body body, uint32_t n, CP cp, CoopWork wk) {
    __shared__ CoopShared shared[kBlock / 32];
    coop_each((blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5, wk, n,
              cp, shared[threadIdx.x >> 5], body);
}

// ---- quad sweeps: four or eight lanes per particle ------------------------------------------
//
// For scenes between the two: a thread per particle leaves each SM a few warps
// whose every step waits for the one before it (at 32,768 particles, 7 warps
// per SM and 26 us per lambda launch of 8 us worth of instructions), a warp per
// particle spends five times the instructions.  A group of G lanes shares a
// particle of at most kQuadCandidates stencil candidates; the scene's others are
// listed (k_stencil_rows) and take a warp each.  Lane q tests the q-th part of
// the particle's flattened candidate sequence, eight candidates at a time, and
// keeps those in range in its column of shared memory; the columns in turn are
// the particle's pair list.  The pair terms are evaluated G entries at a time,
// one per lane, and folded in list order by lane c (sums c and c + G), as in the
// cooperative sweeps: the same terms in the same order, so the same bits.  The
// second sweep over a position set replays the list the same way.
//
// Measured, us per launch, before and after (lambda / delta-p / vorticity A /
// B): 16,384 particles (a warp each before) 17.9 -> 13.6, 18.2 -> 5.1, 22.2 ->
// 14.5, 19.4 -> 5.2; 32,768 (a thread each) 26.0 -> 18.5, 14.8 -> 6.9, 29.7 ->
// 21.0, 15.1 -> 7.0; 65,536 (two blocks, 32 candidates per particle) delta-p
// 11.9 -> 10.0, but lambda 19.2 -> 23.9: there only the second sweeps are quads.
// With 216 candidates per particle, stage times with a thread and with four lanes:
// lambda 34.3 / 22.8 at 32,768 particles, 35.8 / 33.0 at 46,656, 36.2 / 36.7 at
// 47,652, 36.4 / 37.1 at 63,960, vorticity A 37.1 / 24.8, 38.9 / 37.1, 39.4 / 42.0,
// 39.4 / 42.2: hence kQuadScanBelow.
// What bounds it now: latency (scan of 16,384: 5.8 of 13.6 us, the pairs 4.4).
constexpr int kQuad = 4;  // SweepCfg mode
constexpr int kQuadBlock = 64;
// A lane's share of a particle's candidates.
template <int G>
constexpr int kQuadShare = (int)kQuadCandidates / G;
template <int G>
struct QuadTerms {
    // term rows of G entries, two rounds in turn (padded against bank conflicts)
    float t[2][32 / G][8 * G + 4];
};
template <int G>
struct QuadScan {
    uint16_t found[kQuadShare<G>][32];  // each lane's candidates in range, a column per lane
    int2 run[32 / G][10];               // the rows; the tenth ends the sequence
};
static_assert(kQuadScanBelow <= 65536, "QuadScan::found holds 16-bit indices");
template <int G>
struct QuadFirst {  // a first sweep's shared memory per warp; a second sweep's is QuadTerms
    QuadTerms<G> terms;
    QuadScan<G> scan;
};
// A warp is a quad warp or a cooperative one for the whole launch.
template <class T>
union QuadOrCoop {
    T quad;
    CoopShared coop;
};

// One of a few registers by index.
template <int N>
__device__ __forceinline__ float pick(const float (&t)[N], int k) {
    float v = t[0];
#pragma unroll
    for (int i = 1; i < N; ++i) v = k == i ? t[i] : v;
    return v;
}

// The sums of a group's particle: lane q keeps sum q in `a` and sum q + G in `b`.
template <int G>
struct QuadSums {
    float a = 0.0f, b = 0.0f;
    __device__ __forceinline__ float get(int k) const {  // every lane of the warp calls
        return __shfl_sync(kFull, k < G ? a : b, k & (G - 1), G);
    }
};

template <class Op, int G>
__device__ __forceinline__ float quad_fold(float acc, const float* t, int c, uint32_t valid) {
#pragma unroll
    for (int k = 0; k < G; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(t + G * Op::a_row(c) + k);
        const uint32_t v = valid >> k;
        if constexpr (Op::kAdd) {
            if (v & 1u) acc = fadd(acc, a.x);
            if (v & 2u) acc = fadd(acc, a.y);
            if (v & 4u) acc = fadd(acc, a.z);
            if (v & 8u) acc = fadd(acc, a.w);
        } else {
            const float4 s = *reinterpret_cast<const float4*>(t + G * Op::s_row(c) + k);
            if (v & 1u) acc = ffma(s.x, a.x, acc);
            if (v & 2u) acc = ffma(s.y, a.y, acc);
            if (v & 4u) acc = ffma(s.z, a.z, acc);
            if (v & 8u) acc = ffma(s.w, a.w, acc);
        }
    }
    return acc;
}

// Adds the pairs of the first m list entries (entry(k) is the candidate of
// entry k < m) to the particle's sums.  Every lane of the warp calls; m is the
// same on the lanes of a group.  The next round's record and the entry after it
// are loaded ahead: with a few warps per SM a round otherwise waits for both.
template <class Op, int G, class E>
__device__ __forceinline__ void quad_pairs(uint32_t m, const DevConsts& c,
                                           const float4* __restrict__ X, float3 pi,
                                           QuadTerms<G>& sm, const Op& op, QuadSums<G>& sums,
                                           E&& entry) {
    const uint32_t q = threadIdx.x & (G - 1), part = (threadIdx.x & 31u) / G;
    const uint32_t most = __reduce_max_sync(kFull, m);
    uint32_t j1 = 0u, j2 = 0u;
    float4 x1 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (q < m) j1 = entry(q);
    if (!check_ok(c, j1 < c.n_total)) j1 = 0u;
    if (q < m) x1 = __ldg(X + j1);
    if (q + G < m) j2 = entry(q + G);
    int turn = 0;
#pragma unroll 1
    for (uint32_t k = q; k - q < most; k += G, turn ^= 1) {
        const uint32_t j = j1;
        const float4 xj = x1;
        j1 = check_ok(c, j2 < c.n_total) ? j2 : 0u;
        if (k + G < m) x1 = __ldg(X + j1);
        if (k + 2 * G < m) j2 = entry(k + 2 * G);
        bool has = k < m;
        if (has) {
            const float3 d = sub3(pi, xyz(xj));
            const float r2 = dot3(d, d);
            has = !(r2 > c.r2cut) && !(Op::kSkipCoincident && r2 == 0.0f);
            if (has) {
                float t[Op::kRows];
                op.terms(c, d, r2, op.payload(j, xj), t);
#pragma unroll
                for (int r = 0; r < Op::kRows; ++r) sm.t[turn][part][G * r + q] = t[r];
            }
        }
        const uint32_t valid = __ballot_sync(kFull, has) >> (threadIdx.x & 31u & ~(G - 1u));
        __syncwarp();
        const float* const t = sm.t[turn][part];
        if (q < Op::kSums) sums.a = quad_fold<Op, G>(sums.a, t, (int)q, valid);
        if (q + G < Op::kSums) sums.b = quad_fold<Op, G>(sums.b, t, (int)q + G, valid);
    }
    __syncwarp();
}

// The pairs in visit order, one after the other on all lanes of the group: for a
// particle whose pair list was too short.
template <class Op, int G>
__device__ __forceinline__ void quad_walk(uint32_t i, const DevConsts& c,
                                          const PairLists& pl, const float4* __restrict__ X,
                                          float3 pi, const Op& op, QuadSums<G>& sums) {
    const int q = (int)(threadIdx.x & (G - 1));
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int2 be = __ldg(pl.rows + (size_t)o * pl.n + i);
#pragma unroll 1
        for (int32_t j = be.x; j < be.y; ++j) {
            const float4 xj = __ldg(X + j);
            const float3 d = sub3(pi, xyz(xj));
            const float r2 = dot3(d, d);
            if ((uint32_t)j == i || r2 > c.r2cut) continue;
            if (Op::kSkipCoincident && r2 == 0.0f) continue;
            float t[Op::kRows];
            op.terms(c, d, r2, op.payload((uint32_t)j, xj), t);
            auto add = [&](float acc, int k) {
                const float a = pick(t, Op::a_row(k));
                return Op::kAdd ? fadd(acc, a) : ffma(pick(t, Op::s_row(k)), a, acc);
            };
            if (q < Op::kSums) sums.a = add(sums.a, q);
            if (q + G < Op::kSums) sums.b = add(sums.b, q + G);
        }
    }
}

// First sweep over a position set X: scans, records particle
// i's pair list and sums its pairs.  Every lane of the warp calls.
template <int G, class Op>
__device__ __forceinline__ QuadSums<G> quad_scan(uint32_t i, bool live, const DevConsts& c,
                                                 const PairLists& pl,
                                                 const float4* __restrict__ X, float3 pi,
                                                 QuadTerms<G>& sm, QuadScan<G>& sc,
                                                 const Op& op) {
    const int lane = (int)(threadIdx.x & 31u), q = lane & (G - 1), part = lane / G;
    for (int o = q; o < 9; o += G) {
        int2 be = make_int2(0, 0);
        if (live) be = __ldg(pl.rows + (size_t)o * pl.n + i);
        if (!check_ok(c, be.x >= 0 && be.x <= be.y && (uint32_t)be.y <= pl.n))
            be = make_int2(0, 0);
        sc.run[part][o] = be;
    }
    if (q == 0) sc.run[part][9] = make_int2(0, 0x7FFFFFFF);
    __syncwarp();
    int total = 0;
#pragma unroll
    for (int o = 0; o < 9; ++o) total += sc.run[part][o].y - sc.run[part][o].x;
    if (!check_ok(c, total <= (int)kQuadCandidates)) total = 0;
    // this lane's share: `left` candidates from position `at` of row o
    int at = total * q / G, o = 0;
    int left = total * (q + 1) / G - at;
    int2 be = sc.run[part][0];
    while (at >= be.y - be.x) {
        at -= be.y - be.x;
        be = sc.run[part][++o];
    }
    int j = be.x + at;
    uint32_t count = 0;
    // eight candidates at a time, across rows: a scene this small waits for the
    // first touch of every line, so eight loads are in flight
#pragma unroll 1
    for (; left > 0; left -= 8) {
        int js[8];
        float4 x[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            js[k] = k < left ? j : -1;
            ++j;
            while (j >= be.y && o < 9) {  // into the next row that is not empty
                be = sc.run[part][++o];
                j = be.x;
            }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = __ldg(X + max(js[k], 0));
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const float3 d = sub3(pi, xyz(x[k]));
            if (js[k] >= 0 && !(dot3(d, d) > c.r2cut) && (uint32_t)js[k] != i)
                sc.found[count++][lane] = (uint16_t)js[k];
        }
    }
    // the group's entries in visit order: lane q's follow those of the lanes before
    uint32_t upto = count;
#pragma unroll
    for (int d = 1; d < G; d <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, upto, d, G);
        if (q >= d) upto += v;
    }
    const uint32_t tot = __shfl_sync(kFull, upto, G - 1, G);
    uint32_t ends[G];
#pragma unroll
    for (int g = 0; g < G; ++g) ends[g] = __shfl_sync(kFull, upto, g, G);
    uint32_t* const out = pl.idx + i;
    for (uint32_t k = 0, rank = upto - count; k < count && rank < pl.cap; ++k, ++rank)
        out[(size_t)rank * pl.n] = sc.found[k][lane];
    if (live && q == 0) pl.cnt[i] = tot <= pl.cap ? (int32_t)tot : -1;
    __syncwarp();
    QuadSums<G> sums;
    quad_pairs(tot, c, X, pi, sm, op, sums, [&](uint32_t k) {
        uint32_t before = 0u;
        int who = 0;
#pragma unroll
        for (int g = 0; g + 1 < G; ++g)
            if (k >= ends[g]) {
                before = ends[g];
                who = g + 1;
            }
        return (uint32_t)sc.found[k - before][part * G + who];
    });
    return sums;
}

// Second sweep: replays the list.  Every lane of the warp calls.
template <int G, class Op>
__device__ __forceinline__ QuadSums<G> quad_replay(uint32_t i, bool live, const DevConsts& c,
                                                   const PairLists& pl,
                                                   const float4* __restrict__ X, float3 pi,
                                                   QuadTerms<G>& sm, const Op& op) {
    const int32_t cnt = live ? pl.cnt[i] : 0;
    const uint32_t m = cnt > 0 && check_ok(c, (uint32_t)cnt <= pl.cap) ? (uint32_t)cnt : 0u;
    const uint32_t* const in = pl.idx + i;
    QuadSums<G> sums;
    quad_pairs(m, c, X, pi, sm, op, sums,
               [&](uint32_t k) { return __ldg(in + (size_t)k * pl.n); });
    if (cnt < 0) quad_walk(i, c, pl, X, pi, op, sums);
    __syncwarp();
    return sums;
}

// One sweep of a scene: the first `quads` blocks take the particles that are not
// listed, a group of G lanes each, the blocks after them the listed ones, a warp
// each (a launch of their own cost 2.5 us a sweep, mostly over an empty list).
// Particle, liveness and constants of a quad follow; the lanes past the end and
// those of listed particles run along with nothing to do.
#define PBF_QUAD_PARTICLE(SHARED, pl, ...)                                                    \
    __shared__ QuadOrCoop<SHARED> shared_[kQuadBlock / 32];                                   \
    if (blockIdx.x >= quads) {                                                                \
        coop_each(((blockIdx.x - quads) * blockDim.x + threadIdx.x) >> 5,                     \
                  ((gridDim.x - quads) * blockDim.x) >> 5,                                    \
                  CoopWork{pl.heavy_list, pl.heavy_count}, n, cp,                             \
                  shared_[threadIdx.x >> 5].coop, __VA_ARGS__);                               \
        return;                                                                               \
    }                                                                                         \
    SHARED& sm = shared_[threadIdx.x >> 5].quad;                                              \
    const uint32_t own_ = (blockIdx.x * blockDim.x + threadIdx.x) / G;                        \
    const bool live = own_ < n && !(pl.heavy && pl.heavy[own_]);                              \
    const uint32_t i = live ? own_ : 0u;                                                      \
    const auto& c = cp.at(i);                                                                 \
    const bool writes = live && (threadIdx.x & (G - 1)) == 0u

template <class CP, int G>
__global__ void __launch_bounds__(kQuadBlock, 16)
k_lambda_quad(uint32_t quads, const float4* __restrict__ P, float4* __restrict__ L,
              float4* __restrict__ aux, PairLists pw, uint32_t n, CP cp) {
    PBF_QUAD_PARTICLE(QuadFirst<G>, pw, LambdaCoop{P, L, aux, pw.rows, n});
    const float3 pi = xyz(P[i]);
    const QuadSums<G> s =
        quad_scan<G>(i, live, c, pw, P, pi, sm.terms, sm.scan, CoopLambda{});
    const LambdaAcc a{s.get(0), s.get(1), make_float3(s.get(2), s.get(3), s.get(4))};
    if (writes) {
        L[i] = make_float4(pi.x, pi.y, pi.z, lambda_finish(c, a));
        if (aux) aux[i] = lambda_aux(a);
    }
}

template <class CP, int G>
__global__ void __launch_bounds__(kQuadBlock)
k_delta_p_quad(uint32_t quads, const float4* __restrict__ L, float4* __restrict__ Pn, PairLists pr,
               ScanPos sx_out, uint32_t n, CP cp, uint32_t* status) {
    PBF_QUAD_PARTICLE(QuadTerms<G>, pr, DeltaPCoop{L, Pn, sx_out, pr.rows, n, status});
    const float4 Li = L[i];
    const float3 pi = xyz(Li);
    const QuadSums<G> s = quad_replay<G>(i, live, c, pr, L, pi, sm, CoopDeltaP{Li.w});
    const float3 dp = make_float3(s.get(0), s.get(1), s.get(2));
    if (writes) store_position(i, fma3(c.oorho, dp, pi), c, Pn, sx_out, status);  // :85
}

template <class CP, int G>
__global__ void __launch_bounds__(kQuadBlock, 16)
k_vorticity_a_quad(uint32_t quads, const float4* __restrict__ P, const float4* __restrict__ VS,
                   float4* __restrict__ VX, float4* __restrict__ OM, float4* __restrict__ Q,
                   PairLists pw, uint32_t n, CP cp) {
    PBF_QUAD_PARTICLE(QuadFirst<G>, pw, VortACoop{P, VS, VX, OM, Q, pw.rows, n});
    const float3 pi = xyz(P[i]);
    const float3 vi = xyz(VS[i]);
    const QuadSums<G> s =
        quad_scan<G>(i, live, c, pw, P, pi, sm.terms, sm.scan, CoopVortA{VS, vi});
    const float3 acc = make_float3(s.get(0), s.get(1), s.get(2));
    const float3 w = make_float3(s.get(3), s.get(4), s.get(5));
    if (writes) store_vorticity(i, pi, vi, acc, w, c, VX, OM, Q);
}

template <class CP, int G>
__global__ void __launch_bounds__(kQuadBlock)
k_vorticity_b_quad(uint32_t quads, const float4* __restrict__ Q, const float4* __restrict__ VX,
                   const float4* __restrict__ OM, const uint32_t* __restrict__ perm,
                   float4* __restrict__ v, float4* __restrict__ eta_out, PairLists pr, uint32_t n,
                   CP cp) {
    PBF_QUAD_PARTICLE(QuadTerms<G>, pr, VortBCoop{Q, VX, OM, perm, v, eta_out, pr.rows, n});
    const float3 pi = xyz(Q[i]);
    const QuadSums<G> s = quad_replay<G>(i, live, c, pr, Q, pi, sm, CoopVortB{});
    const float3 eta = make_float3(s.get(0), s.get(1), s.get(2));
    if (writes) store_velocity(i, eta, c, VX, OM, perm, v, eta_out);
}

// The substep's stencil rows: row o of sorted particle i, [x, y), at
// rows[o * n + i].  They depend on the cell tables and the predicted positions
// only, so they are found once after the cell pass and every sweep of the
// substep reads them (9 coalesced 8-byte loads) instead of repeating the 27
// cell lookups, the bounds tests and the merging (~500 instructions, and a
// 72-byte local array) in each of its scanning sweeps.
// kWide: one thread per particle and row, a warp per row of 32 particles.  The
// three cell lookups of a row wait for each other, so nine rows in one thread
// are slow where threads are few; where they are many, the nine-fold particle
// reads cost more.  Measured, us, a thread per particle / per row: 16,384
// particles 8.9 / 3.1, 65,536 8.5 / 5.9, 2,097,152 72 / 143.
// Mixed and quad sweeps (heavy != nullptr): the particles with more than
// `threshold` stencil candidates go to the cooperative kernels and are listed
// here; the other kernels skip them.  A warp appends its heavy particles in
// ascending order (one atomic), so consecutive warps of a cooperative launch
// work on neighbouring particles.
constexpr int kRowsBlock = 9 * 32;
constexpr uint32_t kWideRowsBelow = 131072;
template <class CP, bool kWide>
__global__ void __launch_bounds__(kRowsBlock)
k_stencil_rows(const float4* __restrict__ XP, const int32_t* __restrict__ cstart,
               const int32_t* __restrict__ cend, uint32_t threshold, uint32_t n, CP cp,
               int2* __restrict__ rows, uint8_t* __restrict__ heavy, uint32_t* __restrict__ list,
               uint32_t* __restrict__ count) {
    __shared__ uint32_t cand[kWide ? 9 : 1][32];
    const uint32_t lane = threadIdx.x & 31u, o = threadIdx.x >> 5;
    const uint32_t i = kWide ? blockIdx.x * 32u + lane : blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t total = 0;
    if (i < n) {
        const auto& c = cp.at(i);
        const int3 ctr = stencil_centre(XP[i], c);  // neighbourcells.glsl:57
#pragma unroll
        for (int r = 0; r < (kWide ? 1 : 9); ++r) {
            const int row = kWide ? (int)o : r;
            const int2 be = run_of_row(row, ctr, c, cstart, cend);
            rows[(size_t)row * n + i] = be;
            total += (uint32_t)(be.y - be.x);
        }
    }
    if (!heavy) return;
    if constexpr (kWide) {
        cand[o][lane] = total;
        __syncthreads();
        if (o != 0u) return;
        total = 0;
#pragma unroll
        for (int r = 0; r < 9; ++r) total += cand[r][lane];
    }
    const bool h = total > threshold;
    if (i < n) heavy[i] = h ? 1 : 0;
    const uint32_t m = __ballot_sync(0xffffffffu, h);
    if (m == 0u) return;
    uint32_t base = 0;
    if (lane == 0u) base = atomicAdd(count, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (h) list[base + __popc(m & ((1u << lane) - 1u))] = i;
}

// Grid of the cooperative kernels of a mixed sweep (the heavy list's length is
// only known on the device): 8 blocks of 8 warps per SM, and 20 for large scenes,
// whose listed particles differ more in work (the blocks that find no more than
// one entry each even it out; 2,097,152 particles, per launch: lambda 79 -> 71
// us, delta-p 58.5 -> 53.5).  An empty launch takes 1.7 and 2.6 us.  A ticket
// counter per launch instead was slower (lambda 87 us, 5.2 us empty).
inline unsigned heavy_grid(uint32_t n) { return 152u * (n < 1048576u ? 8u : 20u); }

// Grid and launch of a quad sweep: eight lanes per particle below kOctsBelow
// particles (shorter chains), four above (fewer instructions).  Four / eight
// lanes, us: 16,384 particles lambda 13.7 / 13.6, delta-p 6.2 / 5.1; 32,768
// lambda 18.5 / 27.6, delta-p 6.9 / 8.8.
constexpr uint32_t kOctsBelow = 24576;
inline unsigned quad_blocks(uint32_t n, uint32_t lanes) { return grid_for(lanes * n, kQuadBlock); }
// Blocks (of two warps) for the listed particles.
inline unsigned quad_heavy_blocks(uint32_t n) { return n / 2u < 4864u ? n / 2u + 1u : 4864u; }
#define PBF_QUAD_LAUNCH(KERNEL, ...)                                                      \
    do {                                                                                  \
        const unsigned lanes_ = n < kOctsBelow ? 8u : 4u, q_ = quad_blocks(n, lanes_);    \
        const unsigned g_ = q_ + quad_heavy_blocks(n);                                    \
        if (lanes_ == 8u)                                                                 \
            KERNEL<CP, 8><<<g_, kQuadBlock, 0, st>>>(q_, __VA_ARGS__);                    \
        else                                                                              \
            KERNEL<CP, 4><<<g_, kQuadBlock, 0, st>>>(q_, __VA_ARGS__);                    \
    } while (0)
// Grid of warps, one per particle.
inline unsigned coop_grid(uint32_t n) { return (unsigned)(((size_t)n * 32 + kBlock - 1) / kBlock); }

// update.glsl:16-28: v = (x* - x_old) / dt, x = x*, scattered back to id order.
// VS receives the committed velocity in sorted order; when `v_out` is set the
// velocity is also stored in id order (vorticity confinement disabled).
template <class CP>
__global__ void __launch_bounds__(kBlock)
k_commit(const float4* __restrict__ P, const uint32_t* __restrict__ perm, float4* __restrict__ x,
         float4* __restrict__ VS, float4* __restrict__ v_out, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const auto& c = cp.at(i);
    const uint32_t id = perm[i];
    if (!check_ok(c, id < c.n_total)) return;
    const float4 q = P[i];
    const float4 xo = x[id];
    const float4 w = make_float4(fdiv(fsub(q.x, xo.x), c.dt), fdiv(fsub(q.y, xo.y), c.dt),
                                 fdiv(fsub(q.z, xo.z), c.dt), 0.0f);  // :23
    VS[i] = w;
    x[id] = make_float4(q.x, q.y, q.z, 0.0f);  // :26
    if (v_out) v_out[id] = w;                  // :27
}

// vorticity.glsl:34-60: XSPH velocity and the vorticity vector, Jacobi
// (every read sees the committed velocities).
template <class CP, int MODE, bool LISTS>
__global__ void __launch_bounds__(kVortMaxBlock, kVortThreadsPerSM / kVortMaxBlock)
k_vorticity_a(const float4* __restrict__ P, const float4* __restrict__ XP,
              const float4* __restrict__ VS, const uint32_t* __restrict__ skeys,
              const int32_t* __restrict__ cstart, const int32_t* __restrict__ cend,
              float4* __restrict__ VX, float4* __restrict__ OM, float4* __restrict__ Q,
              NbrLists nl, PairLists pw, ScanPos sx, int dmax_slot, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (pw.heavy && pw.heavy[i])) return;
    const auto& c = cp.at(i);
    const float3 pi = xyz(P[i]);
    const float3 vi = xyz(VS[i]);
    auto ctr = [&] { return stencil_centre(XP[i], c); };  // neighbourcells.glsl:57
    float3 acc = make_float3(0.0f, 0.0f, 0.0f), w = make_float3(0.0f, 0.0f, 0.0f);
    // body of one candidate; IN: already known to pass the in-range test (the
    // masked scans computed the same r2 bit for bit)
    auto body = [&](uint32_t j, auto in) {
        const float3 d = sub3(pi, xyz(__ldg(P + j)));  // :51
        const float r2 = dot3(d, d);
        if (!decltype(in)::value && r2 > c.r2cut) return;
        const float len = fsqrt(r2);
        const float3 vij = sub3(xyz(__ldg(VS + j)), vi);  // :50
        acc = fma3(w_poly6(c, len), vij, acc);            // :52-54
        if (len == 0.0f) return;
        const float3 g = scale3(d, grad_scale(c.kg, c.h, len));
        w = add3(w, cross3(vij, g));  // :55
    };
    auto eval = [&](uint32_t j) { body(j, std::false_type{}); };
    auto eval_in = [&](uint32_t j) { body(j, std::true_type{}); };
    auto near = [&](uint32_t j) {
        const float3 d = sub3(pi, xyz(__ldg(P + j)));
        return !(dot3(d, d) > c.r2cut);
    };
    bool listed = false;
    if constexpr (LISTS) {
        const int32_t cnt = nl.cnt[i];
        if (list_usable(c, nl, cnt, pi, xyz(XP[i]), dmax_slot)) {
            listed = true;
            if constexpr (MODE == kPairs) {
                PairRecorder rec{pw, i, 0u};
                visit_list(i, c, cnt, nl, [&](uint32_t j) {
                    const float3 d = sub3(pi, xyz(__ldg(P + j)));
                    if (!(dot3(d, d) > c.r2cut)) rec(j);
                    eval(j);
                });
                rec.finish();
            } else {
                visit_list(i, c, cnt, nl, eval);
            }
        }
    }
    if (!listed) {
        if constexpr (MODE == kPairs)
            scan_then_eval<false>(i, c, sx, pi, pw, [](int32_t, uint32_t) {}, near, eval_in);
        else if constexpr (MODE == kMasked)
            sweep_visit<true>(i, ctr, c, cstart, cend, pw, sx, pi, eval_in);
        else if (!LISTS && pw.runs)
            visit_direct_piles(
                i, ctr, c, cstart, cend, pw.runs,
                [&](uint32_t j) { return xyz(__ldg(P + j)); }, pi, eval,
                // the run bits are over (p, committed v): a run holds one
                // position and one velocity, so its terms are all equal
                [&](uint32_t j0, uint32_t, uint32_t m) {  // len 0: W(0) (v_j - v_i), no curl
                    acc = repeat_fma3(w_poly6(c, 0.0f), sub3(xyz(__ldg(VS + j0)), vi), acc, m);
                },
                [&](uint32_t j0, uint32_t r, float3 d, float r2) {
                    if (r2 > c.r2cut) return;
                    const float len = fsqrt(r2);
                    const float3 g = scale3(d, grad_scale(c.kg, c.h, len));
                    const float3 vij = sub3(xyz(__ldg(VS + j0)), vi);  // :50
                    acc = repeat_fma3(w_poly6(c, len), vij, acc, r - j0);  // :52-54
                    w = repeat_add3(cross3(vij, g), w, r - j0);            // :55
                });
        else
            sweep_visit<false>(i, ctr, c, cstart, cend, pw, sx, pi, eval);
    }
    const float3 vx = fma3(c.cx, acc, vi);  // :58
    VX[i] = make_float4(vx.x, vx.y, vx.z, 0.0f);
    OM[i] = make_float4(w.x, w.y, w.z, 0.0f);
    Q[i] = make_float4(pi.x, pi.y, pi.z, fsqrt(dot3(w, w)));  // :60
}

// vorticity.glsl:65-85: confinement from the gradient of |vorticity|; writes
// the final velocity in id order.
template <class CP, int MODE, bool LISTS>
__global__ void __launch_bounds__(kBlock, kSweepBlocksPerSM)
k_vorticity_b(const float4* __restrict__ Q, const float4* __restrict__ XP,
              const float4* __restrict__ VX, const float4* __restrict__ OM,
              const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ perm,
              const int32_t* __restrict__ cstart, const int32_t* __restrict__ cend,
              float4* __restrict__ v, float4* __restrict__ eta_out, NbrLists nl, PairLists pr,
              ScanPos sx, int dmax_slot, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || (pr.heavy && pr.heavy[i])) return;
    const auto& c = cp.at(i);
    const float3 pi = xyz(Q[i]);
    auto ctr = [&] { return stencil_centre(XP[i], c); };  // neighbourcells.glsl:57
    float3 eta = make_float3(0.0f, 0.0f, 0.0f);
    auto body = [&](uint32_t j) {
        const float4 Qj = __ldg(Q + j);
        const float3 d = sub3(pi, xyz(Qj));  // :69
        const float r2 = dot3(d, d);
        if (r2 > c.r2cut) return;
        const float len = fsqrt(r2);
        if (len == 0.0f) return;
        eta = fma3(Qj.w, scale3(d, grad_scale(c.kg, c.h, len)), eta);  // :72
    };
    bool done = false;
    if constexpr (MODE == kPairs) done = visit_pairs(i, c, pr, body);
    if (!done) {
        bool listed = false;
        if constexpr (LISTS) {
            const int32_t cnt = nl.cnt[i];
            if (list_usable(c, nl, cnt, pi, xyz(XP[i]), dmax_slot)) {
                visit_list(i, c, cnt, nl, body);
                listed = true;
            }
        }
        if (!listed) {
            if (MODE == kDirect && !LISTS && pr.runs)  // coincident: no term (:71)
                visit_direct_piles(
                    i, ctr, c, cstart, cend, pr.runs,
                    [&](uint32_t j) { return xyz(__ldg(Q + j)); }, pi, body, [](uint32_t, uint32_t, uint32_t) {},
                    [&](uint32_t j0, uint32_t r, float3 d, float r2) {
                        // one offset and, the run bits being over (p, |omega|),
                        // one |omega_j|: r - j0 equal terms in a row
                        if (r2 > c.r2cut) return;
                        const float3 g = scale3(d, grad_scale(c.kg, c.h, fsqrt(r2)));
                        eta = repeat_fma3(__ldg(&Q[j0].w), g, eta, r - j0);  // :72
                    });
            else
                sweep_visit<MODE != kDirect>(i, ctr, c, cstart, cend, pr, sx, pi, body);
        }
    }
    if (eta_out) eta_out[i] = make_float4(eta.x, eta.y, eta.z, 0.0f);
    const float l = fsqrt(dot3(eta, eta));  // :76
    if (l > 0.0f) eta = make_float3(fdiv(eta.x, l), fdiv(eta.y, l), fdiv(eta.z, l));  // :77-78
    const float3 vf = fma3(c.dteps, cross3(eta, xyz(OM[i])), xyz(VX[i]));  // :82
    if (check_ok(c, perm[i] < c.n_total)) v[perm[i]] = make_float4(vf.x, vf.y, vf.z, 0.0f);  // :85
}

// Per-particle density error |rho/rho0 - 1| (self excluded) and kinetic
// energy of the state sorted into P (positions) with velocities v (id order).
template <class CP>
__global__ void __launch_bounds__(kBlock)
k_diagnostics(const float4* __restrict__ P, const float4* __restrict__ v,
              const uint32_t* __restrict__ skeys, const uint32_t* __restrict__ perm,
              const int32_t* __restrict__ cstart, const int32_t* __restrict__ cend,
              float4* __restrict__ out, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const auto& c = cp.at(i);
    const float3 pi = xyz(P[i]);
    Runs r;
    runs_of(stencil_centre(pi, c), c, cstart, cend, r);
    float rho = 0.0f;
    int32_t cand = -1;
    for (int o = 0; o < 9; ++o) {
        cand += r.e[o] - r.b[o];
        for (int32_t j = r.b[o]; j < r.e[o]; ++j) {
            if ((uint32_t)j == i) continue;
            const float3 d = sub3(pi, xyz(__ldg(P + j)));
            const float r2 = dot3(d, d);
            if (r2 > c.r2cut) continue;
            rho = fadd(rho, w_poly6(c, fsqrt(r2)));
        }
    }
    const float4 w = v[perm[i]];
    out[i] = make_float4(fabsf(ffma(rho, c.oorho, -1.0f)),
                         0.5f * (w.x * w.x + w.y * w.y + w.z * w.z), (float)cand, 0.0f);
}

// highlight.glsl:16-30 after clearhighlight.glsl: bit 1 of every particle is
// cleared, then set on all stencil candidates (not distance-filtered, as the
// reference's FOR_EACH_NEIGHBOUR) of each particle whose bit 0 is set.
// flags are in id order; the candidates come from the last substep's sort.
template <class CP>
__global__ void __launch_bounds__(kBlock)
k_highlight(const float4* __restrict__ XP, const uint32_t* __restrict__ perm,
            const int32_t* __restrict__ cstart, const int32_t* __restrict__ cend,
            uint32_t* flags, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = perm[i];
    if (id >= n || (flags[id] & 1u) == 0u) return;
    const auto& c = cp.at(i);
    visit_full(i, [&] { return stencil_centre(XP[i], c); }, c, cstart, cend, [&](uint32_t j) {
        const uint32_t pj = perm[j];
        if (pj < n) atomicOr(flags + pj, 2u);
    });
}

__global__ void __launch_bounds__(kBlock) k_clear_highlight(uint32_t* flags, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flags[i] &= 1u;  // clearhighlight.glsl:7
}

template <class CP>
void launch_highlight(unsigned g, cudaStream_t st, const float4* XP, const uint32_t* perm,
                      const int32_t* cstart, const int32_t* cend, uint32_t* flags, uint32_t n,
                      CP cp) {
    k_clear_highlight<<<g, kBlock, 0, st>>>(flags, n);
    k_highlight<CP><<<g, kBlock, 0, st>>>(XP, perm, cstart, cend, flags, n, cp);
}
template void launch_highlight<OneScene>(unsigned, cudaStream_t, const float4*, const uint32_t*,
                                         const int32_t*, const int32_t*, uint32_t*, uint32_t,
                                         OneScene);
template void launch_highlight<ManyScenes>(unsigned, cudaStream_t, const float4*,
                                           const uint32_t*, const int32_t*, const int32_t*,
                                           uint32_t*, uint32_t, ManyScenes);

// Host-side launchers: the template kernels are launched from this file
// (their host stubs are not visible to other translation units).
template <class CP>
void launch_predict(unsigned g, cudaStream_t st, const float4* x, const float4* v, float4* xstar,
                    uint32_t* keys, uint32_t n, CP cp, uint32_t* status,
                    const uint32_t* prev_sorted, uint32_t ncells, int32_t* cstart,
                    uint32_t* heavy_count) {
    k_predict<CP><<<g, kBlock, 0, st>>>(x, v, xstar, keys, n, cp, status, prev_sorted, ncells,
                                        cstart, heavy_count);
}
template <class CP>
void launch_keys_of(unsigned g, cudaStream_t st, const float4* x, float4* xstar, uint32_t* keys,
                    uint32_t n, CP cp) {
    k_keys_of<CP><<<g, kBlock, 0, st>>>(x, xstar, keys, n, cp);
}
// Launches KERNEL<CP, MODE, LISTS> for the tuning in `sw`.
#define PBF_SWEEP_LAUNCH(KERNEL, ...)                                                        \
    do {                                                                                     \
        const unsigned g_ = grid_for(n, (int)sw.block);                                      \
        switch (sw.mode * 2 + (sw.lists ? 1 : 0)) {                                          \
            case 0: KERNEL<CP, kDirect, false><<<g_, sw.block, 0, st>>>(__VA_ARGS__); break; \
            case 1: KERNEL<CP, kDirect, true><<<g_, sw.block, 0, st>>>(__VA_ARGS__); break;  \
            case 2: KERNEL<CP, kMasked, false><<<g_, sw.block, 0, st>>>(__VA_ARGS__); break; \
            case 3: KERNEL<CP, kMasked, true><<<g_, sw.block, 0, st>>>(__VA_ARGS__); break;  \
            case 4: KERNEL<CP, kPairs, false><<<g_, sw.block, 0, st>>>(__VA_ARGS__); break;  \
            default: KERNEL<CP, kPairs, true><<<g_, sw.block, 0, st>>>(__VA_ARGS__); break;  \
        }                                                                                    \
    } while (0)

template <class CP>
void launch_lambda_build(SweepCfg sw, cudaStream_t st, const float4* XP, const uint32_t* skeys,
                         const int32_t* cstart, const int32_t* cend, float4* L, float4* aux,
                         NbrLists nl, PairLists pw, ScanPos sx, uint32_t n, CP cp) {
    if (sw.mode == kCoop) {
        k_coop<CP><<<coop_grid(n), kBlock, 0, st>>>(LambdaCoop{XP, L, aux, pw.rows, n}, n, cp,
                                               CoopWork{nullptr, nullptr});
        return;
    }
    if (sw.mode == kQuad)
        PBF_QUAD_LAUNCH(k_lambda_quad, XP, L, aux, pw, n, cp);
    else
        PBF_SWEEP_LAUNCH(k_lambda_build, XP, skeys, cstart, cend, L, aux, nl, pw, sx, n, cp);
    if (pw.heavy && sw.mode != kQuad)
        k_coop<CP><<<heavy_grid(n), kBlock, 0, st>>>(LambdaCoop{XP, L, aux, pw.rows, n}, n, cp,
                                               CoopWork{pw.heavy_list, pw.heavy_count});
}
template <class CP>
void launch_lambda(SweepCfg sw, cudaStream_t st, const float4* P, const float4* XP,
                   const uint32_t* skeys, const int32_t* cstart, const int32_t* cend, float4* L,
                   float4* aux, NbrLists nl, PairLists pw, ScanPos sx, int dmax_slot, uint32_t n,
                   CP cp) {
    if (sw.mode == kCoop) {
        k_coop<CP><<<coop_grid(n), kBlock, 0, st>>>(LambdaCoop{P, L, aux, pw.rows, n}, n, cp,
                                               CoopWork{nullptr, nullptr});
        return;
    }
    if (sw.mode == kQuad)
        PBF_QUAD_LAUNCH(k_lambda_quad, P, L, aux, pw, n, cp);
    else
        PBF_SWEEP_LAUNCH(k_lambda, P, XP, skeys, cstart, cend, L, aux, nl, pw, sx, dmax_slot, n, cp);
    if (pw.heavy && sw.mode != kQuad)
        k_coop<CP><<<heavy_grid(n), kBlock, 0, st>>>(LambdaCoop{P, L, aux, pw.rows, n}, n, cp,
                                               CoopWork{pw.heavy_list, pw.heavy_count});
}
template <class CP>
void launch_delta_p(SweepCfg sw, cudaStream_t st, const float4* L, const float4* XP,
                    const uint32_t* skeys, const int32_t* cstart, const int32_t* cend, float4* Pn,
                    NbrLists nl, PairLists pr, ScanPos sx, ScanPos sx_out, int dmax_slot,
                    int out_slot, uint32_t n, CP cp, uint32_t* status) {
    if (sw.mode == kCoop) {
        // (with its scan copy where the vorticity passes scan it: they may run
        // under another configuration than the solver)
        k_coop<CP><<<coop_grid(n), kBlock, 0, st>>>(DeltaPCoop{L, Pn, sx_out, pr.rows, n, status}, n, cp,
                                               CoopWork{nullptr, nullptr});
        return;
    }
    if (sw.mode == kQuad)
        PBF_QUAD_LAUNCH(k_delta_p_quad, L, Pn, pr, sx_out, n, cp, status);
    else
        PBF_SWEEP_LAUNCH(k_delta_p, L, XP, skeys, cstart, cend, Pn, nl, pr, sx, sx_out, dmax_slot,
                     out_slot, n, cp, status);
    if (pr.heavy && sw.mode != kQuad)
        k_coop<CP><<<heavy_grid(n), kBlock, 0, st>>>(DeltaPCoop{L, Pn, sx_out, pr.rows, n, status}, n, cp,
                                               CoopWork{pr.heavy_list, pr.heavy_count});
}
template <class CP>
void launch_stencil_rows(cudaStream_t st, const float4* XP, const int32_t* cstart,
                         const int32_t* cend, uint32_t threshold, uint32_t n, CP cp, int2* rows,
                         uint8_t* heavy, uint32_t* list, uint32_t* count) {
    if (n < kWideRowsBelow)
        k_stencil_rows<CP, true><<<grid_for(n, 32), kRowsBlock, 0, st>>>(
            XP, cstart, cend, threshold, n, cp, rows, heavy, list, count);
    else
        k_stencil_rows<CP, false><<<grid_for(n, kBlock), kBlock, 0, st>>>(
            XP, cstart, cend, threshold, n, cp, rows, heavy, list, count);
}
template <class CP>
void launch_commit(unsigned g, cudaStream_t st, const float4* P, const uint32_t* perm, float4* x,
                   float4* VS, float4* v_out, uint32_t n, CP cp) {
    k_commit<CP><<<g, kBlock, 0, st>>>(P, perm, x, VS, v_out, n, cp);
}
template <class CP>
void launch_vorticity_a(SweepCfg sw, cudaStream_t st, const float4* P, const float4* XP,
                        const float4* VS, const uint32_t* skeys, const int32_t* cstart,
                        const int32_t* cend, float4* VX, float4* OM, float4* Q, NbrLists nl,
                        PairLists pw, ScanPos sx, int dmax_slot, uint32_t n, CP cp) {
    if (sw.mode == kCoop) {
        k_coop<CP><<<coop_grid(n), kBlock, 0, st>>>(VortACoop{P, VS, VX, OM, Q, pw.rows, n}, n, cp,
                                               CoopWork{nullptr, nullptr});
        return;
    }
    if (sw.mode == kQuad)
        PBF_QUAD_LAUNCH(k_vorticity_a_quad, P, VS, VX, OM, Q, pw, n, cp);
    else
        PBF_SWEEP_LAUNCH(k_vorticity_a, P, XP, VS, skeys, cstart, cend, VX, OM, Q, nl, pw, sx, dmax_slot,
                     n, cp);
    if (pw.heavy && sw.mode != kQuad)
        k_coop<CP><<<heavy_grid(n), kBlock, 0, st>>>(VortACoop{P, VS, VX, OM, Q, pw.rows, n}, n, cp,
                                               CoopWork{pw.heavy_list, pw.heavy_count});
}
template <class CP>
void launch_vorticity_b(SweepCfg sw, cudaStream_t st, const float4* Q, const float4* XP,
                        const float4* VX, const float4* OM, const uint32_t* skeys,
                        const uint32_t* perm, const int32_t* cstart, const int32_t* cend,
                        float4* v, float4* eta_out, NbrLists nl, PairLists pr, ScanPos sx,
                        int dmax_slot, uint32_t n, CP cp) {
    if (sw.mode == kCoop) {
        k_coop<CP><<<coop_grid(n), kBlock, 0, st>>>(VortBCoop{Q, VX, OM, perm, v, eta_out, pr.rows, n}, n, cp,
                                               CoopWork{nullptr, nullptr});
        return;
    }
    if (sw.mode == kQuad)
        PBF_QUAD_LAUNCH(k_vorticity_b_quad, Q, VX, OM, perm, v, eta_out, pr, n, cp);
    else
        PBF_SWEEP_LAUNCH(k_vorticity_b, Q, XP, VX, OM, skeys, perm, cstart, cend, v, eta_out, nl, pr, sx,
                     dmax_slot, n, cp);
    if (pr.heavy && sw.mode != kQuad)
        k_coop<CP><<<heavy_grid(n), kBlock, 0, st>>>(VortBCoop{Q, VX, OM, perm, v, eta_out, pr.rows, n}, n, cp,
                                               CoopWork{pr.heavy_list, pr.heavy_count});
}
template <class CP>
void launch_diagnostics(unsigned g, cudaStream_t st, const float4* P, const float4* v,
                        const uint32_t* skeys, const uint32_t* perm, const int32_t* cstart,
                        const int32_t* cend, float4* out, uint32_t n, CP cp) {
    k_diagnostics<CP><<<g, kBlock, 0, st>>>(P, v, skeys, perm, cstart, cend, out, n, cp);
}

#define PBF_INSTANTIATE(CP)                                                                     \
    template void launch_predict<CP>(unsigned, cudaStream_t, const float4*, const float4*,      \
                                     float4*, uint32_t*, uint32_t, CP, uint32_t*,               \
                                     const uint32_t*, uint32_t, int32_t*, uint32_t*);           \
    template void launch_keys_of<CP>(unsigned, cudaStream_t, const float4*, float4*, uint32_t*, \
                                     uint32_t, CP);                                             \
    template void launch_lambda_build<CP>(SweepCfg, cudaStream_t, const float4*, const uint32_t*, \
                                          const int32_t*, const int32_t*, float4*, float4*,     \
                                          NbrLists, PairLists, ScanPos, uint32_t, CP);          \
    template void launch_lambda<CP>(SweepCfg, cudaStream_t, const float4*, const float4*,       \
                                    const uint32_t*, const int32_t*, const int32_t*, float4*,   \
                                    float4*, NbrLists, PairLists, ScanPos, int, uint32_t, CP);  \
    template void launch_delta_p<CP>(SweepCfg, cudaStream_t, const float4*, const float4*,      \
                                     const uint32_t*, const int32_t*, const int32_t*, float4*,  \
                                     NbrLists, PairLists, ScanPos, ScanPos, int, int, uint32_t, \
                                     CP, uint32_t*);                                            \
    template void launch_stencil_rows<CP>(cudaStream_t, const float4*, const int32_t*,         \
                                          const int32_t*, uint32_t, uint32_t, CP, int2*,         \
                                          uint8_t*, uint32_t*, uint32_t*);                       \
    template void launch_commit<CP>(unsigned, cudaStream_t, const float4*, const uint32_t*,     \
                                    float4*, float4*, float4*, uint32_t, CP);                   \
    template void launch_vorticity_a<CP>(SweepCfg, cudaStream_t, const float4*, const float4*,  \
                                         const float4*, const uint32_t*, const int32_t*,        \
                                         const int32_t*, float4*, float4*, float4*, NbrLists,   \
                                         PairLists, ScanPos, int, uint32_t, CP);                \
    template void launch_vorticity_b<CP>(SweepCfg, cudaStream_t, const float4*, const float4*,  \
                                         const float4*, const float4*, const uint32_t*,         \
                                         const uint32_t*, const int32_t*, const int32_t*,       \
                                         float4*, float4*, NbrLists, PairLists, ScanPos, int,   \
                                         uint32_t, CP);                                         \
    template void launch_diagnostics<CP>(unsigned, cudaStream_t, const float4*, const float4*,  \
                                         const uint32_t*, const uint32_t*, const int32_t*,      \
                                         const int32_t*, float4*, uint32_t, CP);

PBF_INSTANTIATE(OneScene)
PBF_INSTANTIATE(ManyScenes)

// Loads every sweep kernel the automatic configuration may launch (the
// runtime loads a kernel on its first use otherwise, a few hundred
// microseconds each, which would land in the first trial's substeps).
template <class CP>
cudaError_t preload_sweeps() {
    cudaFuncAttributes a;
    cudaError_t e = cudaSuccess;
    auto load = [&](const void* f) {
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&a, f);
    };
    load((const void*)k_lambda_build<CP, kDirect, false>);
    load((const void*)k_lambda_build<CP, kMasked, false>);
    load((const void*)k_lambda_build<CP, kPairs, false>);
    load((const void*)k_lambda<CP, kDirect, false>);
    load((const void*)k_lambda<CP, kMasked, false>);
    load((const void*)k_lambda<CP, kPairs, false>);
    load((const void*)k_delta_p<CP, kDirect, false>);
    load((const void*)k_delta_p<CP, kMasked, false>);
    load((const void*)k_delta_p<CP, kPairs, false>);
    load((const void*)k_vorticity_a<CP, kDirect, false>);
    load((const void*)k_vorticity_a<CP, kMasked, false>);
    load((const void*)k_vorticity_a<CP, kPairs, false>);
    load((const void*)k_vorticity_b<CP, kDirect, false>);
    load((const void*)k_vorticity_b<CP, kMasked, false>);
    load((const void*)k_vorticity_b<CP, kPairs, false>);
    load((const void*)k_coop<CP, LambdaCoop>);
    load((const void*)k_coop<CP, DeltaPCoop>);
    load((const void*)k_coop<CP, VortACoop>);
    load((const void*)k_coop<CP, VortBCoop>);
    load((const void*)k_lambda_quad<CP, 4>);
    load((const void*)k_lambda_quad<CP, 8>);
    load((const void*)k_delta_p_quad<CP, 4>);
    load((const void*)k_delta_p_quad<CP, 8>);
    load((const void*)k_vorticity_a_quad<CP, 4>);
    load((const void*)k_vorticity_a_quad<CP, 8>);
    load((const void*)k_vorticity_b_quad<CP, 4>);
    load((const void*)k_vorticity_b_quad<CP, 8>);
    load((const void*)k_stencil_rows<CP, true>);
    load((const void*)k_stencil_rows<CP, false>);
    load((const void*)k_run_flags);
    load((const void*)k_run_flags_vals);
    return e;
}
template cudaError_t preload_sweeps<OneScene>();
template cudaError_t preload_sweeps<ManyScenes>();

}  // namespace pbf
