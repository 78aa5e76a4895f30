// adjoint.cu — reverse-mode gradients of whole substeps (no reference
// counterpart: the reference has no differentiation).
//
// The sort permutation, the cell tables and therefore every particle's
// neighbour candidates are frozen from the forward pass: they are piecewise
// constant in the positions, and the pair terms vanish with zero slope at
// r = h, so freezing them gives the exact derivative almost everywhere.  The
// wall clamp contributes its subgradient (zero along a clamped component).
//
// Every reverse sweep is written as a gather, not a scatter: the pair
// functions obey G(-d) = -G(d), H(-d) = H(d), W(-d) = W(d), so each particle
// sums the contributions of its own equation and of its neighbours'
// equations from per-particle adjoint quantities.  No atomic adds into any
// sum (the only atomics set a flag and append to a list whose order no result
// depends on): results are deterministic.  The candidate relation is
// symmetric except around particles
// predicted outside the grid: the forward centres a stencil on the unclamped
// predicted cell (neighbourcells.glsl:57) while the sort files the particle
// under its clamped cell, so such a particle i may be a candidate of j without
// j being one of i's.  The reverse sweeps therefore visit the stencil around
// the clamped (key) cell, which holds both directions, and, in a substep with
// such particles, weigh each pair's terms by two flags: `own` (j is i's
// candidate: the terms of i's equation) and `trans` (i is j's candidate: the
// terms of j's equation).
//
// Notation (sorted particle i, neighbour j, d = p_i - p_j, r = |d|):
//   W(r)  = k6 (h^2 - r^2)^3                 poly6 (calclambda.glsl:41-47)
//   What  = dW/dp_i = -6 k6 (h^2 - r^2)^2 d
//   G(d)  = f(r) d, f = kg (h - r)^2 / r     spiky gradient (calclambda.glsl:57-64)
//   H u   = dG/dd u = f u + (f'/r)(d.u) d,   f' = -kg (h - r)(h + r) / r^2
// Forward solver iteration (lambda then delta-p, Jacobi):
//   lambda_i = -C_i / (S_i + eps),  C_i = rho_i/rho0 - 1,  rho_i = sum W,
//   S_i = sum |g_ij|^2 + |g_i|^2,   g_ij = G_ij / rho0,  g_i = sum_j g_ij
//   q_i = p_i + sum_j a_ij G_ij,    a_ij = (lambda_i + lambda_j + s_ij) / rho0,
//   s_ij = -k (scale W_ij)^4,       p'_i = clamp(q_i)
// Reverse (q-bar = p'-bar with clamped components zeroed):
//   lambda-bar_i = (1/rho0) sum_j (qb_i - qb_j).G_ij
//   p-bar_i     += qb_i + sum_j [a_ij H_ij (qb_i - qb_j) + (s'_ij/(r rho0)) ((qb_i - qb_j).G_ij) d]
//   rho-bar_i = -lambda-bar_i / (rho0 D_i),  S-bar_i = -lambda-bar_i lambda_i / D_i,  D = S + eps
//   p-bar_i     += sum_j [(rhob_i + rhob_j) What_ij + (2/rho0) H_ij (Sb_i (g_ij + g_i) + Sb_j (g_ij - g_j))]
// Velocity update (update.glsl) and XSPH + vorticity (vorticity.glsl):
//   v_i = (p_i - x_i)/dt;  vs_i = v_i + c sum_j W_ij (v_j - v_i);  w_i = sum_j (v_j - v_i) x G_ij
//   eta_i = sum_j |w_j| G_ij;  N_i = eta_i/|eta_i|;  vf_i = vs_i + dt eps_v (N_i x w_i)
#include "neighbours.cuh"
#include "internal.h"
#include "sim.h"

#include <algorithm>
#include <cstring>
#include <mutex>

namespace pbf {

constexpr int kAdjBlock = 256;
constexpr int kParams = 4;  // epsilon, tensile k, XSPH c, vorticity epsilon

// Buffers and bookkeeping of a recorded run.  The buffers are one allocation,
// kept with the handle and reused by the next pbf_forward_record of the same
// shape (a training step records again and again: allocating and freeing them
// in pieces cost 4 ms of a 21 ms step with 32,768 particles and 14 ms of 165 ms
// with 1.2 million).  pbf_release_record and the handle's end give them back,
// and so does any allocation of the library that finds no memory, of any
// handle, while they hold no recorded run (IdleTapes).
struct Tape {
    int device = 0;
    uint32_t substeps = 0, every = 0, iters = 0, nslots = 0;
    bool vort = false;
    bool valid = false;    // holds a complete recorded run
    uint32_t held = kNone; // the segment whose substeps the slots hold
    static constexpr uint32_t kNone = 0xFFFFFFFFu;
    std::vector<float4*> ckpt_x, ckpt_v;  // states at substeps 0, every, 2 every, ... (id order)
    float4 *final_x = nullptr, *final_v = nullptr;
    struct Slot {
        uint32_t* perm = nullptr;
        int2* rows = nullptr;  // [9][n] stencil rows around each particle's key cell
        std::vector<float4*> L, AUX;
        float4 *PF = nullptr, *VS = nullptr, *OM = nullptr, *Q = nullptr, *ETA = nullptr;
        // the forward sweeps' pair lists, one per solver iteration and the
        // vorticity passes' last (cap 0: not recorded)
        std::vector<PairLists> lists;
    };
    std::vector<Slot> slots;
    // adjoint work buffers
    float4 *XB = nullptr, *VB = nullptr;    // x-bar, v-bar at a substep boundary (id order)
    float4 *XB2 = nullptr, *VB2 = nullptr;  // the next boundary
    float4 *QB = nullptr, *PDB = nullptr, *RS = nullptr, *PA = nullptr;  // sorted
    float4 *VSB = nullptr, *ETB = nullptr, *OMB = nullptr, *VCB = nullptr;  // sorted
    float4 *XSB = nullptr, *XOB = nullptr;  // x*-bar and x_old-bar (id order)
    double* acc = nullptr;                  // [kParams][n] per-particle parameter gradients (id order)
    uint8_t* irr = nullptr;                 // [n] stencil centre != key cell (sorted), per substep
    uint32_t* words = nullptr;              // [2]: any particle irregular; flagged particles
    uint8_t* heavy = nullptr;               // [n] swept by a warp (sorted), per substep
    uint32_t* heavy_list = nullptr;         // [n] those particles
    uint32_t warp_above = 0;                // candidates above which a particle gets a warp
    double* sums = nullptr;                 // [scenes][kParams] parameter gradients
    uint32_t* scene_first = nullptr;        // [scenes + 1] first particle of each scene
    uint32_t list_cap = 0;                  // capacity of the recorded pair lists (0: none)
    uint32_t list_pairs = 0;                // the handle's pair-list capacity at allocation
    void* mem = nullptr;                    // holds all of the above
};

namespace {

// ---- pair geometry ------------------------------------------------------------

struct Pair {
    float3 d;
    float r2, r;
};

__device__ __forceinline__ float3 f3(float4 a) { return make_float3(a.x, a.y, a.z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return make_float3(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return make_float3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator*(float s, float3 a) { return make_float3(s * a.x, s * a.y, s * a.z); }
__device__ __forceinline__ float dotf(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 crossf(float3 a, float3 b) {
    return make_float3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// Spiky-gradient pieces at r > 0: G = f d and
// H u = f u + (f'/r)(d.u) d = f u + f' r (rhat.u) rhat.
// The spiky gradient turns direction at r = 0, so H grows like 1/r; pairs
// closer than 1e-6 h (only in collapsed clumps) keep their first-order terms
// and drop H, which would otherwise overflow FP32.
struct Spiky {
    float f, fpr, inv_r;  // f(r), f'(r) r, 1/r
    bool near;
    __device__ __forceinline__ Spiky(const DevConsts& c, float r) {
        const float u = c.h - r;
        inv_r = 1.0f / r;
        f = c.kg * u * u * inv_r;
        fpr = -c.kg * u * (c.h + r) * inv_r;
        near = r < 1e-6f * c.h;
    }
    __device__ __forceinline__ float3 G(float3 d) const { return f * d; }
    __device__ __forceinline__ float3 H(float3 d, float3 v) const {
        if (near) return make_float3(0.0f, 0.0f, 0.0f);
        const float3 rh = inv_r * d;
        return f * v + (fpr * dotf(rh, v)) * rh;
    }
};

__device__ __forceinline__ float w6(const DevConsts& c, float r2) {
    const float t = c.h2 - r2;
    return c.k6 * t * t * t;
}
// dW/dp_i = -6 k6 (h^2 - r^2)^2 d
__device__ __forceinline__ float3 w6_grad(const DevConsts& c, float3 d, float r2) {
    const float t = c.h2 - r2;
    return (-6.0f * c.k6 * t * t) * d;
}

__device__ __forceinline__ float3 clamp_mask(float3 g, float3 p, const DevConsts& c) {
    // subgradient of clamp(): zero where the component sits on a wall
    if (p.x == c.lo[0] || p.x == c.hi[0]) g.x = 0.0f;
    if (p.y == c.lo[1] || p.y == c.hi[1]) g.y = 0.0f;
    if (p.z == c.lo[2] || p.z == c.hi[2]) g.z = 0.0f;
    return g;
}

// ---- candidate directions ---------------------------------------------------------

// The key (sorted) cell of a predicted position, the clamped counterpart of
// stencil_centre (counting.glsl:55 with the cap at G - 1).
__device__ __forceinline__ int3 key_cell(float4 q, const DevConsts& c) {
    return make_int3((int)cell_coord(q.x, c.G[0], c.Gi[0]), (int)cell_coord(q.y, c.G[1], c.Gi[1]),
                     (int)cell_coord(q.z, c.G[2], c.Gi[2]));
}

// Whether each direction of pair (i, j) is a forward candidate (see the top
// of this file).  `on` (the substep has irregular particles) is uniform.
struct PairDirs {
    const uint8_t* irr;
    const float4* XPc;
    const uint32_t* any;  // nonzero when the substep has irregular particles
    __device__ __forceinline__ void of(const DevConsts& c, uint32_t i, uint32_t j, float& own,
                                       float& trans) const {
        own = trans = 1.0f;
        if (!__ldg(any) || !(__ldg(irr + i) | __ldg(irr + j))) return;
        const float4 qi = __ldg(XPc + i), qj = __ldg(XPc + j);
        auto inside = [](int3 cell, int3 ctr) {
            return abs(cell.x - ctr.x) <= 1 && abs(cell.y - ctr.y) <= 1 && abs(cell.z - ctr.z) <= 1;
        };
        own = inside(key_cell(qj, c), stencil_centre(qi, c)) ? 1.0f : 0.0f;
        trans = inside(key_cell(qi, c), stencil_centre(qj, c)) ? 1.0f : 0.0f;
    }
};

// ---- neighbour visits of the reverse sweeps -----------------------------------
//
// Two reverse sweeps read each position set (delta-p then lambda at an
// iterate, vorticity pass B then pass A at the final positions), the sets
// whose in-range candidates the forward sweeps listed: the recorded run keeps
// those lists, and both reverse sweeps replay them.  The lanes of a warp then
// run their (heavy) pair terms together instead of each at its own point of
// the stencil, and nothing is scanned.  (1.2 million particles, per launch:
// the delta-p sweep took 562 us when it scanned the stencil itself, 318 us now.)
//
// A particle without a recorded list (longer than its capacity, swept by a
// warp in the forward run, or every one in a substep with particles predicted
// outside the grid, whose one-way candidates the forward lists lack) scans its
// stencil in the first of the two sweeps, writing its candidates to the
// handle's own pair-list buffer, and replays those in the second; without
// room there it visits the stencil both times.  The same pairs are added in the
// same order either way, but for pairs within rounding of the radius: the forward
// lists test r2 with fused multiply-adds, the reverse scans and terms without.
// There h - r rounds to 0, and what such a pair adds (dW of (h^2 - r^2)^2) is below
// 1e-13 of the others'.
//
// Every index stays in range: list entries are candidates of the rows, written
// and counted by the sweep that found them (a count above the capacity is stored
// as -1, and the recorded counts start at -1, so a list that no sweep wrote is not
// read); the rows come from the cell tables, whose bounds are sorted indices; and
// the own list's count is written by the first sweep for exactly the particles
// for which the second reads it.
struct AdjLists {
    PairLists rec;         // the forward run's list of this position set (cap 0: none)
    PairLists own;         // scratch list (cap 0: none)
    const int2* rows;      // [9][n] the key-cell stencil rows
    const uint32_t* any;   // nonzero when the substep has irregular particles
    __device__ __forceinline__ bool recorded(uint32_t i) const {
        return rec.cap && !__ldg(any) && __ldg(rec.cnt + i) >= 0;
    }
};

template <class F>
__device__ __forceinline__ void adj_replay(uint32_t i, const DevConsts& c, const PairLists& pl,
                                           F&& f) {
    const int32_t cnt = pl.cnt[i];
    const uint32_t* p = pl.idx + i;
    if (cnt > 0 && check_ok(c, (uint32_t)cnt <= pl.cap)) {  // the next index is loaded one entry ahead
        uint32_t jn = p[0];
#pragma unroll 1
        for (int32_t k = 0; k < cnt; ++k) {
            const uint32_t j = jn;
            if (k + 1 < cnt) jn = p[(size_t)(k + 1) * pl.n];
            if (check_ok(c, j < c.n_total)) f(j);
        }
    }
}

// Row o of particle i's key-cell stencil.
__device__ __forceinline__ int2 adj_row(int o, uint32_t i, const DevConsts& c,
                                        const AdjLists& al) {
    const int2 be = __ldg(al.rows + (size_t)o * al.own.n + i);
    if (!check_ok(c, be.x >= 0 && be.x <= be.y && (uint32_t)be.y <= c.n_total))
        return make_int2(0, 0);
    return be;
}

template <class F>
__device__ __forceinline__ void adj_visit_rows(uint32_t i, const DevConsts& c, const AdjLists& al,
                                               F&& f) {
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int2 be = adj_row(o, i, c, al);
        for (int32_t j = be.x; j < be.y; ++j)
            if ((uint32_t)j != i) f((uint32_t)j);
    }
}

// The first of the two sweeps over a position set.
template <class F>
__device__ __forceinline__ void adj_visit_first(uint32_t i, const DevConsts& c,
                                                const float4* __restrict__ X, float3 pi,
                                                const AdjLists& al, F&& f) {
    if (al.recorded(i)) {
        adj_replay(i, c, al.rec, f);
        return;
    }
    const PairLists& own = al.own;
    if (!own.cap) {
        adj_visit_rows(i, c, al, f);
        return;
    }
    uint32_t tot = 0;
    uint32_t* const out = own.idx + i;
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int2 be = adj_row(o, i, c, al);
        const int32_t e = be.y;
#pragma unroll 1
        for (int32_t base = be.x; base < e; base += 32) {
            const float4* __restrict__ p = X + base;
            const float4* const pe = p + min(e - base, 32);
            uint32_t m = 0, bit = 1;
#pragma unroll 1
            for (; p < pe; ++p) {
                const float4 xj = __ldg(p);
                const float3 d = make_float3(pi.x - xj.x, pi.y - xj.y, pi.z - xj.z);
                if (!(d.x * d.x + d.y * d.y + d.z * d.z > c.r2cut)) m |= bit;
                bit <<= 1;
            }
            const uint32_t self = i - (uint32_t)base;
            if (self < 32u) m &= ~(1u << self);
            while (m) {
                const int t = __ffs(m) - 1;
                m &= m - 1;
                if (tot < own.cap) out[(size_t)tot * own.n] = (uint32_t)(base + t);
                ++tot;
            }
        }
    }
    if (tot <= own.cap) {
        own.cnt[i] = (int32_t)tot;
        adj_replay(i, c, own, f);
    } else {
        own.cnt[i] = -1;
        adj_visit_rows(i, c, al, f);
    }
}

// The second one.
template <class F>
__device__ __forceinline__ void adj_visit_again(uint32_t i, const DevConsts& c,
                                                const AdjLists& al, F&& f) {
    if (al.recorded(i))
        adj_replay(i, c, al.rec, f);
    else if (al.own.cap && al.own.cnt[i] >= 0)
        adj_replay(i, c, al.own, f);
    else
        adj_visit_rows(i, c, al, f);
}

// ---- a warp per particle for dense stencils ---------------------------------------
//
// A thread per particle leaves a dense stencil to one thread's serial loop
// over thousands of candidates (collapsed states: the 32,768-particle
// epsilon = 0.01 run holds piles of up to ~11,000 particles by substep 40),
// and with few particles per SM the slowest such thread sets the launch time.
// Particles whose key-cell stencil holds more than `warp_above` candidates
// are flagged by k_adj_flags and swept by a warp each: lane l takes the
// candidates b + l, b + l + 32, ... of each stencil row, in order, and the
// lanes' partial sums are folded by a fixed butterfly; lane 0 writes.  The
// thread sweeps skip flagged particles.  The sums run in another order than
// the thread's, so the two agree to rounding, not bitwise; both are
// deterministic.

template <class F>
__device__ __forceinline__ void warp_visit(uint32_t i, const DevConsts& c, const AdjLists& al,
                                           uint32_t lane, F&& f) {
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int2 be = adj_row(o, i, c, al);
#pragma unroll 1
        for (int32_t j = be.x + (int32_t)lane; j < be.y; j += 32)
            if ((uint32_t)j != i) f((uint32_t)j);
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}
__device__ __forceinline__ float3 warp_sum(float3 v) {
    return make_float3(warp_sum(v.x), warp_sum(v.y), warp_sum(v.z));
}

// The particles of one substep swept by warps (flag == nullptr: none).
struct Heavy {
    const uint8_t* flag;    // [n] 1: flagged (sorted index)
    const uint32_t* list;   // the flagged particles, in no fixed order
    const uint32_t* count;  // how many
};

// Warps per launch of the warp sweeps (4 blocks of 8 warps on each of 152 SMs);
// each takes flagged particles in turn.
constexpr unsigned kAdjWarpBlocks = 608;
constexpr uint32_t kAdjNoWarps = 0xFFFFFFFFu;  // warp_above: no particle gets a warp
constexpr uint32_t kAdjWarpAbove = 512;        // warp_above when the tuning gives 0

// Constants of particle `id` (scene lookup by id for batches).
template <class CP>
__device__ __forceinline__ const DevConsts& consts_of(const CP& cp, uint32_t id) {
    return cp.at(id);
}

// ---- reverse kernels --------------------------------------------------------------

// Stencil rows around the key cell of every particle, from the cell tables of
// the substep just recorded (the reverse sweeps read the rows, so the tables
// need not be kept).
// kWide: one thread per particle and row, a warp per row of 32 particles (as in
// k_stencil_rows: where threads are few).
constexpr int kAdjRowsBlock = 9 * 32;
constexpr uint32_t kAdjWideRowsBelow = 131072;
template <bool kWide, class CP>
__global__ void __launch_bounds__(kAdjRowsBlock)
k_adj_rows(const uint32_t* __restrict__ perm, const float4* __restrict__ XPc,
           const int32_t* __restrict__ cstart, const int32_t* __restrict__ cend,
           int2* __restrict__ rows, uint32_t n, CP cp) {
    const uint32_t i = kWide ? blockIdx.x * 32u + (threadIdx.x & 31u)
                             : blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const DevConsts& c = consts_of(cp, perm[i]);
    const int3 cell = key_cell(XPc[i], c);
#pragma unroll
    for (int r = 0; r < (kWide ? 1 : 9); ++r) {
        const int o = kWide ? (int)(threadIdx.x >> 5) : r;
        rows[(size_t)o * n + i] = run_of_row(o, cell, c, cstart, cend);
    }
}
template <class CP>
void launch_adj_rows(cudaStream_t st, const uint32_t* perm, const float4* XPc,
                     const int32_t* cstart, const int32_t* cend, int2* rows, uint32_t n,
                     const CP& cp) {
    if (n < kAdjWideRowsBelow)
        k_adj_rows<true><<<grid_for(n, 32), kAdjRowsBlock, 0, st>>>(perm, XPc, cstart, cend, rows,
                                                                    n, cp);
    else
        k_adj_rows<false><<<grid_for(n, kAdjBlock), kAdjBlock, 0, st>>>(perm, XPc, cstart, cend,
                                                                        rows, n, cp);
}

// Per substep: irr[i] = 1 when particle i's stencil centre is not its key
// cell (predicted outside the grid), and word[0] set when some particle is;
// with `above` != kAdjNoWarps, heavy[i] = 1 when i's key-cell stencil holds
// more than `above` candidates, those particles listed (in no fixed order:
// each one's result does not depend on it) and counted in word[1].
template <class CP>
__global__ void __launch_bounds__(kAdjBlock)
k_adj_flags(const uint32_t* __restrict__ perm, const float4* __restrict__ XPc,
            const int2* __restrict__ rows, uint32_t above, uint8_t* __restrict__ irr,
            uint8_t* __restrict__ heavy, uint32_t* __restrict__ list, uint32_t* __restrict__ word,
            uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const DevConsts& c = consts_of(cp, perm[i]);
    const float4 q = XPc[i];
    const int3 a = stencil_centre(q, c), b = key_cell(q, c);
    const bool odd = a.x != b.x || a.y != b.y || a.z != b.z;
    irr[i] = odd ? 1 : 0;
    if (odd) atomicOr(word, 1u);
    if (above == kAdjNoWarps) return;
    uint32_t cand = 0;
#pragma unroll
    for (int o = 0; o < 9; ++o) {
        const int2 be = rows[(size_t)o * n + i];
        cand += (uint32_t)(be.y - be.x);
    }
    const bool h = cand > above;
    heavy[i] = h ? 1 : 0;
    if (h) {
        const uint32_t k = atomicAdd(word + 1, 1u);
        if (check_ok(c, k < n)) list[k] = i;
    }
}

// Blocks per SM each body is compiled for (Body::kBlocksPerSM): 4 (64 registers)
// fit every body without spills; the delta-p body alone would take 71 and run
// 3.  Measured, 1.2 million particles: delta-p 318 -> 250 us per launch.
//
// One neighbour reversal (Body::run<W>): blocks below `tblocks` take a
// thread per unflagged particle, the blocks after them a warp per flagged
// particle (in turn, from the list).
template <class Body>
__global__ void __launch_bounds__(kAdjBlock, Body::kBlocksPerSM)
k_adj_sweep(Body b, Heavy hv, uint32_t n, uint32_t tblocks) {
    if (blockIdx.x < tblocks) {
        const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
        if (i >= n || (hv.flag && hv.flag[i])) return;
        b.template run<false>(i, 0u);
        return;
    }
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t w = ((blockIdx.x - tblocks) * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = ((gridDim.x - tblocks) * blockDim.x) >> 5;
    const uint32_t cnt = min(*hv.count, n);
#pragma unroll 1
    for (uint32_t k = w; k < cnt; k += nw) {
        const uint32_t i = hv.list[k];
        if (check_ok(b.cp.at(0), i < n)) b.template run<true>(i, lane);
    }
}

// vorticity.glsl:76-85 reversed, pointwise: from vf-bar to vs-bar, eta-bar and
// the direct part of w-bar; accumulates d/d(eps_v).
template <class CP>
__global__ void __launch_bounds__(kAdjBlock)
k_adj_vort_b1(const uint32_t* __restrict__ perm, const float4* __restrict__ VB,
              const float4* __restrict__ OM, const float4* __restrict__ ETA,
              float4* __restrict__ VSB, float4* __restrict__ ETB, float4* __restrict__ OMB,
              double* __restrict__ acc_epsv, uint32_t n, CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = perm[i];
    const DevConsts& c = consts_of(cp, id);
    const float3 vfb = f3(VB[id]);
    const float3 w = f3(OM[i]);
    const float3 eta = f3(ETA[i]);
    const float le = sqrtf(dotf(eta, eta));
    const float3 N = le > 0.0f ? (1.0f / le) * eta : eta;
    const float3 u = c.dteps * vfb;
    const float3 Nb = crossf(w, u);
    const float3 wb = crossf(u, N);
    acc_epsv[id] += (double)(c.dt * dotf(crossf(N, w), vfb));
    // d(eta/|eta|)/d(eta) grows like 1/|eta|; below 1e-20 (a particle with no
    // vorticity gradient) the normalisation's derivative is dropped
    const float3 eb = le > 1e-20f ? (1.0f / le) * (Nb - dotf(N, Nb) * N)
                                  : (le > 0.0f ? make_float3(0.0f, 0.0f, 0.0f) : Nb);
    VSB[i] = make_float4(vfb.x, vfb.y, vfb.z, 0.0f);
    ETB[i] = make_float4(eb.x, eb.y, eb.z, 0.0f);
    OMB[i] = make_float4(wb.x, wb.y, wb.z, 0.0f);
}

// vorticity.glsl:65-74 reversed: eta_i = sum_j |w_j| G_ij.  Gathers |w|-bar
// and the position adjoint, then folds |w|-bar into w-bar.
template <class CP>
struct AdjVortB2 {
    static constexpr int kBlocksPerSM = 4;
    const uint32_t* __restrict__ perm;
    const float4* __restrict__ Q;
    const float4* __restrict__ OM;
    const float4* __restrict__ ETB;
    float4* __restrict__ OMB;
    float4* __restrict__ PA;
    AdjLists al;
    PairDirs dirs;
    CP cp;
    template <bool W>
    __device__ __forceinline__ void run(uint32_t i, uint32_t lane) const {
        const uint32_t id = perm[i];
        if (!check_ok(cp.at(0), id < cp.at(0).n_total)) return;
        const DevConsts& c = consts_of(cp, id);
        const float4 Qi = Q[i];
        const float3 pi = f3(Qi);
        const float mi = Qi.w;
        const float3 ebi = f3(ETB[i]);
        float mb = 0.0f;
        float3 pb = make_float3(0.0f, 0.0f, 0.0f);
        auto pair = [&](uint32_t j) {
            const float4 Qj = __ldg(Q + j);
            const float3 d = pi - f3(Qj);
            const float r2 = dotf(d, d);
            if (r2 > c.r2cut || r2 == 0.0f) return;
            const Spiky sp(c, sqrtf(r2));
            float own, trans;
            dirs.of(c, i, j, own, trans);
            const float3 ebj = trans * f3(__ldg(ETB + j));
            mb -= dotf(ebj, sp.G(d));
            pb = pb + sp.H(d, (own * Qj.w) * ebi - mi * ebj);
        };
        if constexpr (W) {
            warp_visit(i, c, al, lane, pair);
            mb = warp_sum(mb);
            pb = warp_sum(pb);
            if (lane) return;
        } else {
            adj_visit_first(i, c, Q, pi, al, pair);
        }
        float3 wb = f3(OMB[i]);
        if (mi > 0.0f) wb = wb + (mb / mi) * f3(OM[i]);
        OMB[i] = make_float4(wb.x, wb.y, wb.z, 0.0f);
        PA[i] = make_float4(pb.x, pb.y, pb.z, 0.0f);
    }
};

// vorticity.glsl:47-58 reversed (XSPH and the vorticity vector): gathers the
// committed-velocity adjoint and adds the position adjoint; accumulates d/dc.
template <class CP>
struct AdjVortA {
    static constexpr int kBlocksPerSM = 4;
    const uint32_t* __restrict__ perm;
    const float4* __restrict__ PF;
    const float4* __restrict__ VS;
    const float4* __restrict__ VSB;
    const float4* __restrict__ OMB;
    float4* __restrict__ VCB;
    float4* __restrict__ PA;
    double* __restrict__ acc_c;
    AdjLists al;
    PairDirs dirs;
    CP cp;
    template <bool W>
    __device__ __forceinline__ void run(uint32_t i, uint32_t lane) const {
        const uint32_t id = perm[i];
        if (!check_ok(cp.at(0), id < cp.at(0).n_total)) return;
        const DevConsts& c = consts_of(cp, id);
        const float3 pi = f3(PF[i]);
        const float3 vi = f3(VS[i]);
        const float3 sbi = f3(VSB[i]);
        const float3 wbi = f3(OMB[i]);
        const float3 zero = make_float3(0.0f, 0.0f, 0.0f);
        float3 vb = W ? zero : sbi;
        float3 pb = W ? zero : f3(PA[i]);
        float3 wsum = zero;
        auto pair = [&](uint32_t j) {
            const float3 d = pi - f3(__ldg(PF + j));
            const float r2 = dotf(d, d);
            if (r2 > c.r2cut) return;
            float own, trans;
            dirs.of(c, i, j, own, trans);
            const float3 vji = f3(__ldg(VS + j)) - vi;
            const float3 sbj = trans * f3(__ldg(VSB + j));
            const float3 sbo = own * sbi;
            const float W6 = w6(c, r2);
            vb = vb + (c.cx * W6) * (sbj - sbo);
            wsum = wsum + (own * W6) * vji;
            pb = pb + (c.cx * dotf(sbo - sbj, vji)) * w6_grad(c, d, r2);
            if (r2 == 0.0f) return;
            const Spiky sp(c, sqrtf(r2));
            const float3 wbs = own * wbi + trans * f3(__ldg(OMB + j));
            vb = vb - crossf(sp.G(d), wbs);
            pb = pb + sp.H(d, crossf(wbs, vji));
        };
        if constexpr (W) {
            warp_visit(i, c, al, lane, pair);
            vb = sbi + warp_sum(vb);
            pb = f3(PA[i]) + warp_sum(pb);
            wsum = warp_sum(wsum);
            if (lane) return;
        } else {
            adj_visit_again(i, c, al, pair);
        }
        acc_c[id] += (double)dotf(sbi, wsum);
        VCB[i] = make_float4(vb.x, vb.y, vb.z, 0.0f);
        PA[i] = make_float4(pb.x, pb.y, pb.z, 0.0f);
    }
};

// update.glsl:23-27 reversed: p-bar of the final positions, x_old-bar, and
// the clamp mask of the last solver iteration.
template <class CP>
__global__ void __launch_bounds__(kAdjBlock)
k_adj_commit(const uint32_t* __restrict__ perm, const float4* __restrict__ XB,
             const float4* __restrict__ VB, const float4* __restrict__ VCB,
             const float4* __restrict__ PA, const float4* __restrict__ PF, float4* __restrict__ QB,
             float4* __restrict__ XOB, float4* __restrict__ XSB, int vort, int iters, uint32_t n,
             CP cp) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t id = perm[i];
    const DevConsts& c = consts_of(cp, id);
    const float3 vc = vort ? f3(VCB[i]) : f3(VB[id]);
    const float inv_dt = 1.0f / c.dt;
    float3 pb = f3(XB[id]) + inv_dt * vc;
    if (vort) pb = pb + f3(PA[i]);
    const float3 xo = (-inv_dt) * vc;
    XOB[id] = make_float4(xo.x, xo.y, xo.z, 0.0f);
    if (iters > 0) {
        pb = clamp_mask(pb, f3(PF[i]), c);
        QB[i] = make_float4(pb.x, pb.y, pb.z, 0.0f);
    } else {
        XSB[id] = make_float4(pb.x, pb.y, pb.z, 0.0f);
    }
}

// updatepos.glsl:42-104 reversed (one iteration), plus the pointwise part of
// calclambda's reverse: writes p-bar of the delta-p terms and (rho-bar, S-bar);
// accumulates d/d(eps) and d/dk.
template <class CP>
struct AdjDeltaP {
    static constexpr int kBlocksPerSM = 4;
    const uint32_t* __restrict__ perm;
    const float4* __restrict__ L;
    const float4* __restrict__ AUX;
    const float4* __restrict__ QB;
    float4* __restrict__ PDB;
    float4* __restrict__ RS;
    double* __restrict__ acc_eps;
    double* __restrict__ acc_k;
    AdjLists al;
    PairDirs dirs;
    CP cp;
    template <bool W>
    __device__ __forceinline__ void run(uint32_t i, uint32_t lane) const {
        const uint32_t id = perm[i];
        if (!check_ok(cp.at(0), id < cp.at(0).n_total)) return;
        const DevConsts& c = consts_of(cp, id);
        const float4 Li = L[i];
        const float3 pi = f3(Li);
        const float li = Li.w;
        const float3 qbi = f3(QB[i]);
        float lb = 0.0f, kb = 0.0f;
        float3 pb = W ? make_float3(0.0f, 0.0f, 0.0f) : qbi;
        const float sc4 = c.scale * c.scale * c.scale * c.scale;
        auto pair = [&](uint32_t j) {
            const float4 Lj = __ldg(L + j);
            const float3 d = pi - f3(Lj);
            const float r2 = dotf(d, d);
            if (r2 > c.r2cut || r2 == 0.0f) return;
            const Spiky sp(c, sqrtf(r2));
            const float t = c.h2 - r2;
            const float W6 = c.k6 * t * t * t;
            const float W3 = W6 * W6 * W6;
            const float s = c.negk * sc4 * W3 * W6;
            const float a = (li + Lj.w + s) * c.oorho;
            const float3 G = sp.G(d);
            float own, trans;
            dirs.of(c, i, j, own, trans);
            const float3 dq = own * qbi - trans * f3(__ldg(QB + j));
            const float dqG = dotf(dq, G);
            lb += c.oorho * dqG;
            // (ds/dr)/r = 4 negk scale^4 W^3 (-6 k6 (h^2 - r^2)^2)
            const float sr = 4.0f * c.negk * sc4 * W3 * (-6.0f * c.k6 * t * t);
            pb = pb + sp.H(d, a * dq) + (c.oorho * sr * dqG) * d;
            kb -= own * c.oorho * dotf(qbi, G) * sc4 * W3 * W6;
        };
        if constexpr (W) {
            warp_visit(i, c, al, lane, pair);
            lb = warp_sum(lb);
            kb = warp_sum(kb);
            pb = qbi + warp_sum(pb);
            if (lane) return;
        } else {
            adj_visit_first(i, c, L, pi, al, pair);
        }
        const float4 aux = AUX[i];
        const float D = aux.w + c.eps;
        const float rb = -lb * c.oorho / D;
        const float Sb = -lb * li / D;
        acc_eps[id] += (double)Sb;
        acc_k[id] += (double)kb;
        PDB[i] = make_float4(pb.x, pb.y, pb.z, 0.0f);
        RS[i] = make_float4(rb, Sb, 0.0f, 0.0f);
    }
};

// calclambda.glsl:75-101 reversed (one iteration): gathers the density and
// denominator terms; masks the previous iteration's clamp, or un-sorts into
// the predicted-position adjoint after the first iteration.
template <class CP>
struct AdjLambda {
    static constexpr int kBlocksPerSM = 4;
    const uint32_t* __restrict__ perm;
    const float4* __restrict__ L;
    const float4* __restrict__ AUX;
    const float4* __restrict__ RS;
    const float4* __restrict__ PDB;
    float4* __restrict__ QB;
    float4* __restrict__ XSB;
    int first;
    AdjLists al;
    PairDirs dirs;
    CP cp;
    template <bool W>
    __device__ __forceinline__ void run(uint32_t i, uint32_t lane) const {
        const uint32_t id = perm[i];
        if (!check_ok(cp.at(0), id < cp.at(0).n_total)) return;
        const DevConsts& c = consts_of(cp, id);
        const float3 pi = f3(L[i]);
        const float4 RSi = RS[i];
        const float3 gi = f3(AUX[i]);
        float3 pb = W ? make_float3(0.0f, 0.0f, 0.0f) : f3(PDB[i]);
        auto pair = [&](uint32_t j) {
            const float3 d = pi - f3(__ldg(L + j));
            const float r2 = dotf(d, d);
            if (r2 > c.r2cut) return;
            float own, trans;
            dirs.of(c, i, j, own, trans);
            const float4 RSj = __ldg(RS + j);
            pb = pb + (own * RSi.x + trans * RSj.x) * w6_grad(c, d, r2);
            if (r2 == 0.0f) return;
            const Spiky sp(c, sqrtf(r2));
            const float3 gij = c.oorho * sp.G(d);
            const float3 gj = f3(__ldg(AUX + j));
            const float3 u = (own * RSi.y) * (gij + gi) + (trans * RSj.y) * (gij - gj);
            pb = pb + (2.0f * c.oorho) * sp.H(d, u);
        };
        if constexpr (W) {
            warp_visit(i, c, al, lane, pair);
            pb = f3(PDB[i]) + warp_sum(pb);
            if (lane) return;
        } else {
            adj_visit_again(i, c, al, pair);
        }
        if (first) {
            XSB[id] = make_float4(pb.x, pb.y, pb.z, 0.0f);
        } else {
            pb = clamp_mask(pb, pi, c);
            QB[i] = make_float4(pb.x, pb.y, pb.z, 0.0f);
        }
    }
};

// predictpos.glsl:32-34 reversed: x* = x + dt v'; plus the commit's x_old.
template <class CP>
__global__ void __launch_bounds__(kAdjBlock)
k_adj_predict(const float4* __restrict__ XSB, const float4* __restrict__ XOB,
              float4* __restrict__ XB, float4* __restrict__ VB, uint32_t n, CP cp) {
    const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n) return;
    const DevConsts& c = consts_of(cp, id);
    const float3 xs = f3(XSB[id]);
    const float3 xb = xs + f3(XOB[id]);
    const float3 vb = c.dt * xs;
    XB[id] = make_float4(xb.x, xb.y, xb.z, 0.0f);
    VB[id] = make_float4(vb.x, vb.y, vb.z, 0.0f);
}

// Parameter gradients of each scene: sums the per-particle gradients acc
// [kParams][n] over the scene's particles, one block per (scene, parameter),
// in a fixed order (a strided partial sum per thread, then a tree).
__global__ void __launch_bounds__(kAdjBlock)
k_adj_param_sums(const double* __restrict__ acc, const uint32_t* __restrict__ first, uint32_t n,
                 double* __restrict__ sums) {
    __shared__ double part[kAdjBlock];
    const uint32_t scene = blockIdx.x / kParams, p = blockIdx.x % kParams;
    const uint32_t e = first[scene + 1];
    const double* __restrict__ a = acc + (size_t)p * n;
    double s = 0.0;
    for (uint32_t i = first[scene] + threadIdx.x; i < e; i += kAdjBlock) s += a[i];
    part[threadIdx.x] = s;
    for (uint32_t h = kAdjBlock / 2; h > 0; h >>= 1) {
        __syncthreads();
        if (threadIdx.x < h) part[threadIdx.x] += part[threadIdx.x + h];
    }
    if (threadIdx.x == 0) sums[blockIdx.x] = part[0];
}

// ---- host side ------------------------------------------------------------------

// The tapes that hold no recorded run.  A tape is in this list or claimed by the
// thread that uses its handle, and `mem` of one in the list changes under the
// lock only, so handles in other threads may free it.  Nothing runs on a tape
// in the list (its stream was waited for).
struct IdleTapes {
    std::mutex mu;
    std::vector<Tape*> list;
};
IdleTapes& idle_tapes() {
    static IdleTapes* t = new IdleTapes;  // outlives every handle
    return *t;
}
void park(Tape* t) {
    IdleTapes& idle = idle_tapes();
    std::lock_guard<std::mutex> lock(idle.mu);
    if (std::find(idle.list.begin(), idle.list.end(), t) == idle.list.end())
        idle.list.push_back(t);
}
// Whether the tape still has its buffers.
bool claim(Tape* t) {
    IdleTapes& idle = idle_tapes();
    std::lock_guard<std::mutex> lock(idle.mu);
    idle.list.erase(std::remove(idle.list.begin(), idle.list.end(), t), idle.list.end());
    return t->mem != nullptr;
}
// A run that ends without a complete record leaves its tape idle.
struct ParkUnlessValid {
    pbf_sim* s;
    ~ParkUnlessValid() {
        if (!s->tape || s->tape->valid) return;
        cudaStreamSynchronize(s->stream);
        park(s->tape);
    }
};

// Hands out 256-byte aligned pieces of one allocation (base null: only counts).
struct Carver {
    uint8_t* base;
    size_t used = 0;
    template <class T>
    void take(T** p, size_t count) {
        if (base) *p = reinterpret_cast<T*>(base + used);
        used += (sizeof(T) * (count ? count : 1) + 255) & ~size_t(255);
    }
};

void carve_tape(const pbf_sim* s, Tape* t, Carver& a) {
    const size_t n = s->n;
    const uint32_t nck = (t->substeps + t->every - 1) / t->every;
    t->ckpt_x.resize(nck);
    t->ckpt_v.resize(nck);
    for (uint32_t k = 0; k < nck; ++k) {
        a.take(&t->ckpt_x[k], n);
        a.take(&t->ckpt_v[k], n);
    }
    a.take(&t->final_x, n);
    a.take(&t->final_v, n);
    t->slots.resize(t->nslots);
    for (auto& sl : t->slots) {
        a.take(&sl.perm, n);
        a.take(&sl.rows, 9 * n);
        sl.L.resize(t->iters);
        sl.AUX.resize(t->iters);
        for (uint32_t k = 0; k < t->iters; ++k) {
            a.take(&sl.L[k], n);
            a.take(&sl.AUX[k], n);
        }
        float4** one[] = {&sl.PF, &sl.VS, &sl.OM, &sl.Q, &sl.ETA};
        for (float4** w : one) a.take(w, n);
        sl.lists.assign(t->iters + 1, PairLists{nullptr, nullptr, 0, s->n});
        if (t->list_cap)
            for (uint32_t k = 0; k < t->iters + (t->vort ? 1u : 0u); ++k) {
                sl.lists[k].cap = t->list_cap;
                a.take(&sl.lists[k].idx, (size_t)t->list_cap * n);
                a.take(&sl.lists[k].cnt, n);
            }
    }
    float4** work[] = {&t->XB, &t->VB, &t->XB2, &t->VB2, &t->QB, &t->PDB, &t->RS, &t->PA,
                       &t->VSB, &t->ETB, &t->OMB, &t->VCB, &t->XSB, &t->XOB};
    for (float4** w : work) a.take(w, n);
    a.take(&t->acc, (size_t)kParams * n);
    a.take(&t->irr, n);
    a.take(&t->words, 2);
    a.take(&t->heavy, n);
    a.take(&t->heavy_list, n);
    a.take(&t->sums, (size_t)s->nscenes * kParams);
    a.take(&t->scene_first, (size_t)s->nscenes + 1);
}

// Capacity of the recorded pair lists: the handle's while the tape then stays
// below kAdjListBytes, otherwise kAdjListCap entries per particle (a fluid at
// its rest density has about 33 neighbours; a longer list is not kept), and none
// where the lists would take more than 1 / kAdjListShare of the free memory:
// they are four fifths of a tape, which the host program's own allocator cannot
// call back.
constexpr size_t kAdjListBytes = size_t(4) << 30;
constexpr uint32_t kAdjListCap = 48;
constexpr size_t kAdjListShare = 8;

cudaError_t alloc_tape(pbf_sim* s, Tape* t) {
    auto bytes = [&](uint32_t cap) {
        t->list_cap = cap;
        Carver a{nullptr};
        carve_tape(s, t, a);
        return a.used;
    };
    size_t free_b = 0, total_b = 0;
    cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    if (e != cudaSuccess) return e;
    const size_t bare = bytes(0), share = free_b / kAdjListShare;
    size_t need = bytes(s->pair_cap);
    if (need > kAdjListBytes || need - bare > share)
        need = bytes(std::min(s->pair_cap, kAdjListCap));
    if (need - bare > share) need = bytes(0);
    e = device_alloc(&t->mem, need);
    if (e == cudaErrorMemoryAllocation && t->list_cap) {
        cudaGetLastError();
        need = bytes(0);
        e = device_alloc(&t->mem, need);
    }
    if (e != cudaSuccess) {
        t->mem = nullptr;
        return e;
    }
    Carver a{(uint8_t*)t->mem};
    carve_tape(s, t, a);
    // (on the handle's stream, which does not wait for a copy on the legacy one)
    return cudaMemcpyAsync(t->scene_first, s->offsets.data(), sizeof(uint32_t) * (s->nscenes + 1),
                           cudaMemcpyHostToDevice, s->stream);
}

template <class CP>
cudaError_t reverse_substep(pbf_sim* s, Tape* t, const Tape::Slot& sl, const CP& cp) {
    const uint32_t n = s->n;
    const unsigned g = grid_for(n, kAdjBlock);
    cudaStream_t st = s->stream;
    const int iters = (int)t->iters;
    double* acc_eps = t->acc;
    double* acc_k = t->acc + n;
    double* acc_c = t->acc + 2 * (size_t)n;
    double* acc_ev = t->acc + 3 * (size_t)n;
    const PairLists own{s->pair_idx, s->pair_cnt, s->pair_cap, n};
    auto lists = [&](int k) { return AdjLists{sl.lists[k], own, sl.rows, t->words}; };
    // the substep's predicted positions (sorted), where every stencil is
    // centred (neighbourcells.glsl:57): the first lambda sweep's L holds them,
    // and PF does when there is no solver iteration
    const float4* XPc = iters > 0 ? sl.L[0] : sl.PF;
    cudaError_t fe = cudaMemsetAsync(t->words, 0, 2 * sizeof(uint32_t), st);
    if (fe != cudaSuccess) return fe;
    k_adj_flags<<<g, kAdjBlock, 0, st>>>(sl.perm, XPc, sl.rows, t->warp_above, t->irr, t->heavy,
                                         t->heavy_list, t->words, n, cp);
    const PairDirs dirs{t->irr, XPc, t->words};
    // the particles with dense stencils get a warp each
    const bool warps = t->warp_above != kAdjNoWarps;
    const Heavy hv{warps ? t->heavy : nullptr, t->heavy_list, t->words + 1};
    auto sweep = [&](const auto& body) {
        k_adj_sweep<<<g + (warps ? kAdjWarpBlocks : 0u), kAdjBlock, 0, st>>>(body, hv, n, g);
    };
    if (t->vort) {
        k_adj_vort_b1<<<g, kAdjBlock, 0, st>>>(sl.perm, t->VB, sl.OM, sl.ETA, t->VSB, t->ETB,
                                               t->OMB, acc_ev, n, cp);
        const AdjLists al = lists(iters);
        sweep(AdjVortB2<CP>{sl.perm, sl.Q, sl.OM, t->ETB, t->OMB, t->PA, al, dirs, cp});
        sweep(AdjVortA<CP>{sl.perm, sl.PF, sl.VS, t->VSB, t->OMB, t->VCB, t->PA, acc_c, al, dirs,
                           cp});
    }
    k_adj_commit<<<g, kAdjBlock, 0, st>>>(sl.perm, t->XB, t->VB, t->VCB, t->PA, sl.PF, t->QB,
                                          t->XOB, t->XSB, t->vort ? 1 : 0, iters, n, cp);
    for (int k = iters - 1; k >= 0; --k) {
        const AdjLists al = lists(k);
        sweep(AdjDeltaP<CP>{sl.perm, sl.L[k], sl.AUX[k], t->QB, t->PDB, t->RS, acc_eps, acc_k, al,
                            dirs, cp});
        sweep(AdjLambda<CP>{sl.perm, sl.L[k], sl.AUX[k], t->RS, t->PDB, t->QB, t->XSB,
                            k == 0 ? 1 : 0, al, dirs, cp});
    }
    k_adj_predict<<<g, kAdjBlock, 0, st>>>(t->XSB, t->XOB, t->XB2, t->VB2, n, cp);
    std::swap(t->XB, t->XB2);
    std::swap(t->VB, t->VB2);
    return cudaGetLastError();
}

cudaError_t reverse_dispatch(pbf_sim* s, Tape* t, const Tape::Slot& sl) {
    if (s->nscenes == 1) return reverse_substep(s, t, sl, OneScene{s->dc});
    return reverse_substep(s, t, sl, ManyScenes{s->d_consts, s->sid});
}

// Runs segment `seg` (`count` substeps) from the current state, recording each
// substep into a slot; with `step` they are the handle's next substeps
// (recorded_substep), otherwise a repetition of earlier ones.
pbf_status record_segment(pbf_sim* s, Tape* t, uint32_t seg, uint32_t count, bool step) {
    cudaStream_t st = s->stream;
    const size_t n = s->n;
    t->held = Tape::kNone;
    for (uint32_t k = 0; k < count; ++k) {
        Tape::Slot& sl = t->slots[k];
        Recording rec;
        rec.L = sl.L.data();
        rec.AUX = sl.AUX.data();
        rec.PF = sl.PF;
        rec.VS = sl.VS;
        rec.OM = sl.OM;
        rec.Q = sl.Q;
        rec.ETA = sl.ETA;
        if (t->list_cap) {
            rec.lists = sl.lists.data();
            // particles that a cooperative sweep takes write no list
            for (const PairLists& pl : sl.lists)
                if (pl.cap) PBF_CUDA(s, cudaMemsetAsync(pl.cnt, 0xFF, sizeof(int32_t) * n, st));
        }
        if (step) {
            pbf_status r = recorded_substep(s, rec);
            if (r != PBF_OK) return r;
        } else {
            PBF_CUDA(s, enqueue_substep(s, nullptr, &rec));
        }
        PBF_CUDA(s, cudaMemcpyAsync(sl.perm, s->perm, sizeof(uint32_t) * n,
                                    cudaMemcpyDeviceToDevice, st));
        const float4* XPc = t->iters > 0 ? sl.L[0] : sl.PF;
        if (s->nscenes == 1)
            launch_adj_rows(st, sl.perm, XPc, s->cstart, s->cend, sl.rows, s->n, OneScene{s->dc});
        else
            launch_adj_rows(st, sl.perm, XPc, s->cstart, s->cend, sl.rows, s->n,
                            ManyScenes{s->d_consts, s->sid});
        PBF_CUDA(s, cudaGetLastError());
    }
    t->held = seg;
    return PBF_OK;
}

}  // namespace

void free_tape(pbf_sim* s) {
    if (!s->tape) return;
    if (claim(s->tape)) cudaFree(s->tape->mem);
    delete s->tape;
    s->tape = nullptr;
}

void invalidate_tape(pbf_sim* s) {
    if (!s->tape || !s->tape->valid) return;
    s->tape->valid = false;
    cudaStreamSynchronize(s->stream);
    park(s->tape);
}

bool free_idle_tapes() {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return false;
    IdleTapes& idle = idle_tapes();
    std::lock_guard<std::mutex> lock(idle.mu);
    bool freed = false;
    for (Tape* t : idle.list)
        if (t->device == device && t->mem) {
            cudaFree(t->mem);
            t->mem = nullptr;  // (its handle allocates anew: claim)
            freed = true;
        }
    return freed;
}

}  // namespace pbf

using namespace pbf;

extern "C" {

pbf_status pbf_forward_record(pbf_sim* s, uint32_t substeps, uint32_t checkpoint_every) {
    NvtxRange nvtx_("pbf_forward_record");
    if (!s) return fail(nullptr, PBF_ERR_INVALID_ARGUMENT, "sim is NULL");
    if (substeps == 0 || checkpoint_every == 0)
        return fail(s, PBF_ERR_INVALID_ARGUMENT, "substeps and checkpoint_every must be positive");
    DeviceGuard dg(s->device);
    PBF_CUDA(s, cudaStreamSynchronize(s->stream));
    const uint32_t every = std::min(checkpoint_every, substeps);
    const uint32_t iters = s->params.num_solver_iterations;
    const bool vort = s->params.vorticity_confinement != 0;
    Tape* t = s->tape;
    // (the recorded lists' capacity follows the handle's)
    if (t && !(claim(t) && t->substeps == substeps && t->every == every && t->iters == iters &&
               t->vort == vort && t->list_pairs == s->pair_cap)) {
        free_tape(s);
        t = nullptr;
    }
    if (!t) {
        t = s->tape = new Tape();
        t->device = s->device;
        t->substeps = substeps;
        t->every = every;
        t->iters = iters;
        t->nslots = every;
        t->vort = vort;
        t->list_pairs = s->pair_cap;
        cudaError_t e = alloc_tape(s, t);
        if (e != cudaSuccess) {
            free_tape(s);
            return cuda_fail(s, e, "tape allocation");
        }
    }
    t->valid = false;
    t->held = Tape::kNone;
    const ParkUnlessValid unless_valid{s};
    const size_t b = sizeof(float4) * s->n;
    // every segment but the last is stepped as usual and recorded when the
    // reverse pass reaches it; the last is recorded at once (its slots are the
    // first that the reverse pass reads)
    const uint32_t last = (substeps - 1) / t->every;
    for (uint32_t seg = 0; seg <= last; ++seg) {
        PBF_CUDA(s, cudaMemcpyAsync(t->ckpt_x[seg], s->x, b, cudaMemcpyDeviceToDevice, s->stream));
        PBF_CUDA(s, cudaMemcpyAsync(t->ckpt_v[seg], s->v, b, cudaMemcpyDeviceToDevice, s->stream));
        const uint32_t cnt = std::min(t->every, substeps - seg * t->every);
        if (seg < last || s->timing) {
            pbf_status r = pbf_step(s, cnt);
            if (r != PBF_OK) return r;
        } else {
            pbf_status r = record_segment(s, t, seg, cnt, true);
            if (r != PBF_OK) return r;
            // (a recorded substep keeps its lambdas in its slot: pbf_get_solver
            // reads the handle's, beside the last substep's predicted positions)
            if (iters > 0)
                PBF_CUDA(s, cudaMemcpyAsync(s->L, t->slots[cnt - 1].L[iters - 1], b,
                                            cudaMemcpyDeviceToDevice, s->stream));
        }
    }
    PBF_CUDA(s, cudaMemcpyAsync(t->final_x, s->x, b, cudaMemcpyDeviceToDevice, s->stream));
    PBF_CUDA(s, cudaMemcpyAsync(t->final_v, s->v, b, cudaMemcpyDeviceToDevice, s->stream));
    t->valid = true;
    return check_status(s);
}

pbf_status pbf_backward(pbf_sim* s, const float* dL_dx4, const float* dL_dv4, int where,
                        float* dL_dx0_4, float* dL_dv0_4, pbf_param_grads* grads) {
    NvtxRange nvtx_("pbf_backward");
    if (!s) return fail(nullptr, PBF_ERR_INVALID_ARGUMENT, "sim is NULL");
    if (!s->tape || !s->tape->valid)
        return fail(s, PBF_ERR_INVALID_ARGUMENT, "no recorded forward run (pbf_forward_record)");
    if (where != PBF_HOST && where != PBF_DEVICE) return fail(s, PBF_ERR_INVALID_ARGUMENT, "bad where");
    Tape* t = s->tape;
    if (t->iters != s->params.num_solver_iterations ||
        t->vort != (s->params.vorticity_confinement != 0))
        return fail(s, PBF_ERR_INVALID_ARGUMENT, "parameters changed since the recorded run");
    DeviceGuard dg(s->device);
    cudaStream_t st = s->stream;
    const size_t n = s->n;
    const size_t b = sizeof(float4) * n;
    const cudaMemcpyKind in = where == PBF_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    const cudaMemcpyKind out = where == PBF_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    if (dL_dx4)
        PBF_CUDA(s, cudaMemcpyAsync(t->XB, dL_dx4, b, in, st));
    else
        PBF_CUDA(s, cudaMemsetAsync(t->XB, 0, b, st));
    if (dL_dv4)
        PBF_CUDA(s, cudaMemcpyAsync(t->VB, dL_dv4, b, in, st));
    else
        PBF_CUDA(s, cudaMemsetAsync(t->VB, 0, b, st));
    PBF_CUDA(s, cudaMemsetAsync(t->acc, 0, sizeof(double) * kParams * n, st));
    PBF_CUDA(s, cudaMemsetAsync(t->VCB, 0, b, st));
    PBF_CUDA(s, cudaMemsetAsync(t->PA, 0, b, st));
    t->warp_above = s->tuning.adjoint_warp_candidates ? s->tuning.adjoint_warp_candidates
                                                      : kAdjWarpAbove;
    const uint32_t nseg = (t->substeps + t->every - 1) / t->every;
    for (int seg = (int)nseg - 1; seg >= 0; --seg) {
        const uint32_t t0 = (uint32_t)seg * t->every;
        const uint32_t cnt = std::min(t->every, t->substeps - t0);
        if (t->held != (uint32_t)seg) {
            PBF_CUDA(s, cudaMemcpyAsync(s->x, t->ckpt_x[seg], b, cudaMemcpyDeviceToDevice, st));
            PBF_CUDA(s, cudaMemcpyAsync(s->v, t->ckpt_v[seg], b, cudaMemcpyDeviceToDevice, st));
            pbf_status r = record_segment(s, t, (uint32_t)seg, cnt, false);
            if (r != PBF_OK) return r;
        }
        for (int k = (int)cnt - 1; k >= 0; --k) PBF_CUDA(s, reverse_dispatch(s, t, t->slots[k]));
    }
    // the handle's state returns to the end of the recorded run
    PBF_CUDA(s, cudaMemcpyAsync(s->x, t->final_x, b, cudaMemcpyDeviceToDevice, st));
    PBF_CUDA(s, cudaMemcpyAsync(s->v, t->final_v, b, cudaMemcpyDeviceToDevice, st));
    if (dL_dx0_4) PBF_CUDA(s, cudaMemcpyAsync(dL_dx0_4, t->XB, b, out, st));
    if (dL_dv0_4) PBF_CUDA(s, cudaMemcpyAsync(dL_dv0_4, t->VB, b, out, st));
    std::vector<double> sums;
    if (grads) {
        sums.resize((size_t)s->nscenes * kParams);
        k_adj_param_sums<<<s->nscenes * kParams, kAdjBlock, 0, st>>>(t->acc, t->scene_first, s->n,
                                                                     t->sums);
        PBF_CUDA(s, cudaGetLastError());
        PBF_CUDA(s, cudaMemcpyAsync(sums.data(), t->sums, sizeof(double) * sums.size(),
                                    cudaMemcpyDeviceToHost, st));
    }
    pbf_status r = check_status(s);
    if (r != PBF_OK) return r;
    if (grads) {
        for (uint32_t sc = 0; sc < s->nscenes; ++sc) {
            const double* v = &sums[(size_t)sc * kParams];
            grads[sc].epsilon = v[0];
            grads[sc].tensile_instability_k = v[1];
            grads[sc].xsph_viscosity_c = v[2];
            grads[sc].vorticity_epsilon = v[3];
        }
    }
    return PBF_OK;
}

pbf_status pbf_release_record(pbf_sim* s) {
    if (!s) return fail(nullptr, PBF_ERR_INVALID_ARGUMENT, "sim is NULL");
    DeviceGuard dg(s->device);
    PBF_CUDA(s, cudaStreamSynchronize(s->stream));
    free_tape(s);
    return PBF_OK;
}

}  // extern "C"
