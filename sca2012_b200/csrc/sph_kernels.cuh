// sph_kernels.cuh — sm_100a kernels of one adaptive-SPH step.
//
// Layout in HBM (all SoA, 16-byte aligned):
//   canonical state, two buffers swapped every step, in the reference's
//   particle-index order (the order split/merge/compaction and the readback
//   depend on): pos4 = (x, y, z, level), vel4, ev4, acc4, dens, press,
//   energy, surface, interior, and when in use scene (batched scenes) and
//   pos_lo (compensated positions);
//   sorted working copies, in cell-key order, that the neighbour loops read
//   contiguously: spos/svel/sev (gathered), saux = (rho, p, p/rho^2, m/rho),
//   and the post-integration spos_n/svel_n/sev_n/sacc_n, ssurf, senergy;
//   a force neighbour's values in two 16-byte records fnb_a = (x, y, z,
//   p/rho^2) and fnb_b = (m/rho signed by level, ev), written by density;
//   per-particle neighbour candidate lists (nlist, rows of four-entry
//   chunks), written by the density pass and read by the force and energy
//   passes.
// Cell key = z*R*C + y*R + x with x = floor(pos / cell) in FP32, exactly the
// reference's calc_grid_pos/calc_grid_hash (SPH-3D-2/sph_system.cu:18-32).
// Neighbour search visits the 3 (2D) or 9 (3D) rows of x-adjacent cells; in
// key order each row is one contiguous slot range.
//
// Every decision that is an integer outcome of float arithmetic (cell keys,
// r^2 < h^2, h - r > 0, the split/merge scores) is evaluated with explicit
// round-to-nearest intrinsics in a fixed order, so the CPU oracle's FP32
// replica reproduces it bit for bit.  Every sum with a product operand in the
// step's bodies is written as an explicit __fmaf_rn / __fadd_rn too: the
// compiler then has no multiply-add to contract, so a body compiled into a
// standalone kernel and into the persistent step kernel (sph_persistent.cuh)
// rounds the same way and the two give the same bits.
#pragma once
#include <cstdint>
#include <type_traits>
#include "../../include/sph/sph.h"
#include "sph_scan.cuh"

namespace sph {

constexpr uint32_t kEmpty = 0xffffffffu;
constexpr int kThreads = 256;

// First statement of every kernel that the host launches as a programmatic
// dependent of the one before it (launch() in sph_api.cu): waits until that
// kernel has finished and its writes are visible, then lets the next kernel's
// blocks be scheduled while this one runs, where they wait in turn.  The launch
// and the ramp-up of a step's 7 to 10 kernels then overlap the kernel before:
// 131k adaptive step 155 -> 142 us, 32,768-particle rollout iteration of 60 steps
// 16.1 -> 14.2 ms, 2D reference frame 182 -> 164 us.
// Such a kernel is resident before its inputs are written, so it reads none of
// them through the read-only data path (no __ldg, no __restrict__).
__device__ __forceinline__ void dependent_entry()
{
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

// Device-side counters of one step parity.
struct Counters {
    uint32_t n;            // live particles at step start
    uint32_t n_split;      // split particles this step
    uint32_t n_removed;    // merged-away particles this step
    uint32_t error;        // SPH_ERR_* bit flags (1 << code)
    uint32_t split_off;    // 1: splits suppressed this step (capacity)
    uint32_t disp2_max;    // bits of the step's largest squared displacement (FP32 >= 0), by the force pass
    uint32_t split_flags;  // particles the energy pass flagged to split this step
    uint32_t removed_flags;  // particles the merge pass flagged as merged away this step
                           // (at 0 the ranks of a kind are not written: every reader tests the count)
    uint32_t merge_candidates;  // particles that may be merge-eligible this step, by the energy
                           // pass (at 0 the merge pass has nothing to do and returns at once)
};

// Counts of one taped step, for its adjoint.
struct StepCounts {
    uint32_t n, n_split, n_removed, split_on;
};

struct CanonPtrs {
    float4 *pos, *vel, *ev, *acc;
    float *dens, *press, *energy, *surface;
    uint32_t *interior;
    uint32_t *sibling;                   // next member of the particle's split group (kEmpty: none)
    uint32_t *scene;                     // scene index (batched scenes)
    float4 *pos_lo;                      // low part of the position (compensated positions)
};

struct WorkPtrs {
    uint32_t *key, *slot, *tmp;          // per canonical particle / slot
    uint32_t *cell_count, *cell_off;     // C, C+1
    uint32_t *sidx, *skey, *inv;         // sorted slot -> particle, key; particle -> slot
    float4 *spos, *svel, *sev, *saux;
    float4 *spos_n, *svel_n, *sev_n, *sacc_n;
    float *ssurf, *senergy;
    uint32_t *snbr, *sinter;
    float4 *stv;                         // debug: wavelet-transformed velocity
    uint32_t *split_c, *removed_c;       // per canonical particle
    uint32_t *split_rank, *removed_rank; // exclusive scans
    uint32_t *split_list;                // split rank -> particle
    uint32_t *leader;                    // per sorted slot: 1 if merge survivor
    float4 *mpos, *mvel, *mev, *macc;    // merged values at the leader's slot
    float *menergy;
    uint32_t *sscene;                    // scene index per sorted slot
    const float4 *scene_tab;             // per scene: (lo.xyz, viscosity), (hi.xyz, gas constant)
    uint32_t nscenes;                    // 0: one scene in [0, world]
    uint32_t *merge_to;                  // taped steps only: slot -> its merge leader's slot
    float *mvs;                          // taped steps only: leader slot -> summed member volume
    uint32_t *wall;                      // taped steps only: wall contacts per slot
    StepCounts *step_counts;             // taped steps only: where the write-out leaves the step's counts
    uint32_t skip_energy;                // taped steps only: nothing reads this step's energy
    float4 *spos_lo, *spos_lo_n;         // low position parts per slot (compensated positions)
    uint32_t pos_comp;                   // the config's compensated_positions
    // neighbour candidates, by the density pass.  Entries come in chunks of four
    // (one 16-byte load); chunk j of every slot is one row of nl_stride chunks, so
    // the chunk-j loads of a warp's 32 consecutive slots read 512 contiguous bytes:
    // entry k of slot s is nlist[((k >> 2) * nl_stride + s) * 4 + (k & 3)].
    uint32_t *nlist, *ncnt;
    uint32_t nl_stride;                  // slots per list chunk row (the capacity)
    float4 *fnb_a, *fnb_b;               // a force neighbour in two loads: (x, y, z, p/rho^2) and
                                         // (m/rho with the sign bit set for level 2, ev.xyz), by the density pass
    uint32_t *out_src;                   // deferred outputs: per output index its sorted slot and kOut* flags
                                         // (nullptr: the write-out writes acc, dens, press, energy, surface)
};

// Deferred outputs.  acc, dens, press, energy and surface are outputs only:
// no stage of the next step reads them.  With w.out_src set the write-out
// records, per output index, the sorted slot its values come from (and how:
// a split parent, a child, a merge leader), and k_materialize writes the five
// fields from the step's sorted arrays when something reads the state; the
// values are write_body's.
constexpr uint32_t kOutChild = 1u << 31, kOutSplit = 1u << 30, kOutLeader = 1u << 29;
constexpr uint32_t kOutSlot = (1u << 29) - 1u;

// Neighbour candidates the density pass records per particle: every stencil
// neighbour within (1 + kNbrListMargin) h_max of the start-of-step position,
// in stencil-walk order (more than kNbrListCap: the consumers walk).
//  - The force pass uses the same positions: filtering the list with its own
//    test (r^2 < max(h_i^2, h_j^2), r^2 >= close_r2) gives its walk's pairs
//    in its walk's order.
//  - The energy pass tests the particles' integrated positions against the
//    stale cell lists of the particle's NEW cell.  When that cell is the old
//    one and |d_i| + max_j |d_j| (d: the step's displacements) stays under
//    the margin, every pair it accepts has a start-of-step distance below
//    h + margin, so it is on the list: filtering the list gives the walk's
//    pairs in the walk's order.  Other particles walk the stencil.
// Either way the sums are those of the walk, bit for bit.
constexpr uint32_t kNbrListCap = 128;
constexpr float kNbrListMargin = 0.05f;

// Pulls a line into L2 ahead of its use (no register, no result).
__device__ __forceinline__ void prefetch_l2(const void *p)
{
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

__device__ __forceinline__ float energy_list_r2(const sph_config &c)
{
    const float r = 1.0f + kNbrListMargin;
    return fmaxf(c.kernel2[0], c.kernel2[1]) * (r * r);
}

// the displacement budget the list covers: 1% under the margin, far above
// the FP32 rounding of the distances involved (~1e-7 relative)
__device__ __forceinline__ float energy_list_budget(const sph_config &c)
{
    return 0.99f * kNbrListMargin * sqrtf(fmaxf(c.kernel2[0], c.kernel2[1]));
}

// hi + lo += d with hi, lo FP32 (Fast2Sum; |hi| >= |d + lo| holds for a
// position and one step's displacement).
__device__ __forceinline__ void comp_add(float &hi, float &lo, float d)
{
    const float y = __fadd_rn(d, lo);
    const float t = __fadd_rn(hi, y);
    lo = __fadd_rn(__fsub_rn(hi, t), y);
    hi = t;
}

// ------------------------------------------------------------ helpers
__device__ __forceinline__ int lv(float w) { return w == 1.0f ? 0 : 1; }

__device__ __forceinline__ uint32_t cell_coord(float x, float cs, uint32_t n)
{
    float f = floorf(__fdiv_rn(x, cs));
    if (!(f >= 0.0f)) return 0u;
    if (f >= (float)n) return n - 1u;
    return (uint32_t)f;
}

template <int DIM>
__device__ __forceinline__ uint3 cell_of(const sph_config &c, float4 p)
{
    uint3 q;
    q.x = cell_coord(p.x, c.cell_size, c.ncell[0]);
    q.y = cell_coord(p.y, c.cell_size, c.ncell[1]);
    q.z = DIM == 3 ? cell_coord(p.z, c.cell_size, c.ncell[2]) : 0u;
    return q;
}

__device__ __forceinline__ uint32_t key_of(const sph_config &c, uint32_t x, uint32_t y, uint32_t z)
{
    return z * c.ncell[0] * c.ncell[1] + y * c.ncell[0] + x;
}

// The cell coordinates of a key (two integer divisions).
template <int DIM> __device__ __forceinline__ uint3 cell_of_key(const sph_config &c, uint32_t k)
{
    uint3 q;
    const uint32_t yz = k / c.ncell[0];
    q.x = k - yz * c.ncell[0];
    q.z = DIM == 3 ? yz / c.ncell[1] : 0u;
    q.y = DIM == 3 ? yz - q.z * c.ncell[1] : yz;
    return q;
}

// fma(dz, dz, fma(dx, dx, dy*dy)) with d = a - b, all round-to-nearest.
template <int DIM>
__device__ __forceinline__ float r2_of(float4 a, float4 b, float &dx, float &dy, float &dz)
{
    dx = __fsub_rn(a.x, b.x);
    dy = __fsub_rn(a.y, b.y);
    float t = __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
    if (DIM == 3) {
        dz = __fsub_rn(a.z, b.z);
        t = __fmaf_rn(dz, dz, t);
    } else {
        dz = 0.0f;
    }
    return t;
}

// 1/sqrt(x) by the PTX instruction, whose .ftz takes a denormal x as zero (+inf).
__device__ __forceinline__ float rsqrt_normal(float x)
{
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// sqrt(x) from y = rsqrt_normal(x) by one Newton step with the residual in
// one fused multiply-add (Markstein, IBM J. Res. Dev. 34, 1990): no branch
// and no second special-function instruction.  The bits of __fsqrt_rn for every
// FP32 value in [2.7e-20, 4e37] (compared value by value).  Not for x = 0 (NaN).
__device__ __forceinline__ float sqrt_of(float x, float y)
{
    const float g = __fmul_rn(x, y);
    return __fmaf_rn(__fmaf_rn(-g, g, x), __fmul_rn(0.5f, y), g);
}

__device__ __forceinline__ float split_score(const sph_config &c, float e, float s)
{
    return __fmaf_rn(s, c.co_surface, __fmul_rn(e, c.co_energy));
}

__device__ __forceinline__ uint32_t grid_stride_start() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ uint32_t grid_stride() { return gridDim.x * blockDim.x; }

// Row ranges of the 3^DIM neighbourhood of cell q: rows (dy, dz); each row is
// the slot range [off[key(x0)], off[key(x1)+1]) of cells x0..x1.
template <int DIM>
__device__ __forceinline__ int row_range(const sph_config &c, const uint32_t *off, uint3 q,
                                         int dy, int dz, uint32_t &b, uint32_t &e)
{
    int y = (int)q.y + dy, z = (int)q.z + dz;
    if (y < 0 || y >= (int)c.ncell[1]) return 0;
    if (DIM == 3 && (z < 0 || z >= (int)c.ncell[2])) return 0;
    uint32_t x0 = q.x > 0 ? q.x - 1 : 0;
    uint32_t x1 = q.x + 1 < c.ncell[0] ? q.x + 1 : q.x;
    uint32_t k0 = key_of(c, x0, (uint32_t)y, (uint32_t)z);
    uint32_t k1 = key_of(c, x1, (uint32_t)y, (uint32_t)z);
    b = off[k0];
    e = off[k1 + 1];
    return 1;
}

// ------------------------------------------------------------ 1. hash
// Particle i at p: its cell key, and a slot among its cell's members from
// the cell's counter (which must start the step at zero).  One atomic per
// group of lanes in the same cell (consecutive particles often share one);
// any distinct slots do, k_reorder restores the order.
template <int DIM>
__device__ __forceinline__ void hash_one(const sph_config &c, const WorkPtrs &w, uint32_t i, float4 p)
{
    const uint3 q = cell_of<DIM>(c, p);
    const uint32_t k = key_of(c, q.x, q.y, q.z);
    w.key[i] = k;
    const unsigned grp = __match_any_sync(__activemask(), k);
    const int lead = __ffs(grp) - 1, lane = threadIdx.x & 31;
    uint32_t first = 0;
    if (lane == lead) first = atomicAdd(w.cell_count + k, (uint32_t)__popc(grp));
    first = __shfl_sync(grp, first, lead);
    w.slot[i] = first + __popc(grp & ((1u << lane) - 1u));
}

template <int DIM>
__device__ __forceinline__ void hash_body(const sph_config &c, const Counters *cnt, const CanonPtrs &st,
                                          const WorkPtrs &w)
{
    const uint32_t n = cnt->n;
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) hash_one<DIM>(c, w, i, st.pos[i]);
}

template <int DIM, int BS = kThreads>
__global__ void __launch_bounds__(BS) k_hash(sph_config c, const Counters *cnt,
                                                  CanonPtrs st, WorkPtrs w)
{
    dependent_entry();
    hash_body<DIM>(c, cnt, st, w);
}

// ------------------------------------------------------------ 3. scatter
__device__ __forceinline__ void scatter_body(const Counters *cnt, const WorkPtrs &w)
{
    const uint32_t n = cnt->n;
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        // always below n when the counts, keys and slots come from one hash;
        // the test keeps a state left inconsistent by an abandoned persistent
        // step (SPH_ERR_TIMEOUT, not yet replaced by sph_set_state) in bounds
        const uint32_t d = w.cell_off[w.key[i]] + w.slot[i];
        if (d < n) w.tmp[d] = i;
    }
}

template <int BS = kThreads>
__global__ void __launch_bounds__(BS) k_scatter(const Counters *cnt, WorkPtrs w)
{
    dependent_entry();
    scatter_body(cnt, w);
}

// ------------------------------------------------------------ 4. stable order + gather
// The atomic slot order inside a cell is arbitrary; the stable order (equal
// keys in ascending particle index, as thrust's radix sort_by_key leaves
// them, SPH-3D-2/sph_system.cu:119-129) is restored by ranking each particle
// among its cell's members.  Then the state is gathered into key order.
// EARLY loads the state before the rank is found instead of after it: one
// latency less in a chain that a few warps wait for, but 12 registers more
// live across it.  The persistent step takes it (4,096 particles in one
// cluster: 23.9 -> 23.2 us per step); the launched kernel does not (1.05M
// particles, where the memory system is busy either way: 29 -> 32 us).
template <bool EARLY>
__device__ __forceinline__ void reorder_body(const Counters *cnt, const CanonPtrs &st, const WorkPtrs &w)
{
    const uint32_t n = cnt->n;
    for (uint32_t s = grid_stride_start(); s < n; s += grid_stride()) {
        uint32_t i = w.tmp[s];
        uint32_t k = w.key[i];
        float4 pos, vel, ev;
        if (EARLY) { pos = st.pos[i]; vel = st.vel[i]; ev = st.ev[i]; }
        uint32_t b = w.cell_off[k], e = w.cell_off[k + 1];
        uint32_t r = 0;
        for (uint32_t t = b; t < e; ++t) r += w.tmp[t] < i;
        uint32_t d = b + r;
        w.sidx[d] = i;
        w.skey[d] = k;
        w.inv[i] = d;
        w.spos[d] = EARLY ? pos : st.pos[i];
        w.svel[d] = EARLY ? vel : st.vel[i];
        w.sev[d] = EARLY ? ev : st.ev[i];
        if (w.nscenes) w.sscene[d] = st.scene[i];
        if (w.pos_comp) w.spos_lo[d] = st.pos_lo[i];
    }
}

template <int BS = kThreads>
__global__ void __launch_bounds__(BS) k_reorder(const Counters *cnt, CanonPtrs st, WorkPtrs w)
{
    dependent_entry();
    reorder_body<false>(cnt, st, w);
}

// ------------------------------------------------------------ warp-lockstep pair loop
// The force and energy loops walk each particle's 3^DIM-cell stencil with the
// particle's whole warp in lockstep (up to 4 candidates per lane per step,
// their loads in flight together).  A lane appends the candidates it accepts
// to its list in shared memory; as soon as any lane's list holds kWarpCap
// entries, the whole warp runs the pair math over the lists in rounds (round
// k: every lane's k-th entry), each lane adding into its own sums in list
// order.  Flushing together keeps the expensive pair math converged (lists
// fill at similar rates, so few lanes idle in a round), and every particle's
// sums take the same order whichever particles share its warp.
// List fill that triggers a warp flush (24 x 32 x 4 B per warp).  The lists
// take shared memory from the L1 that serves the neighbour loads of the warps
// that read candidate lists: 40 entries held the L1 to 60-67 % hits there
// (energy 251 us on 1.24M particles), 20 allow 69-71 % (246); a pass that
// walks every stencil loses what 40 gained (2 %).
constexpr uint32_t kWarpCap = 20;
constexpr uint32_t kWarpSlot = kWarpCap + 4;  // a step can add 4 more before the check

struct NbrPV { float4 p, v; };       // position, velocity

// Bundles a fetch(t) and a use(fetched) callable for warp_pairs<.., AHEAD>.
template <class F, class U> struct FetchUse {
    F fetch;
    U use;
};
template <class F, class U> __device__ __forceinline__ FetchUse<F, U> fetch_use(F f, U u) { return {f, u}; }

struct WarpPairSmem {
    uint32_t lst[kWarpSlot][32];     // per-lane lists, entry-major (appends hit 32 banks)
};

// accept(t, pj): this lane's test of candidate slot t at position pj.
// pair(t): adds this lane's pair with neighbour slot t into its sums.
// AHEAD > 0: pair is instead a fetch(t) / use(fetched) pair of callables
// (FetchUse) and a flush fetches AHEAD pairs before their math (entries past
// the lane's list read slot `self`), for callers whose fetched data fits in
// registers.  Every lane of the warp must call it (active = false for a lane
// without a particle).
template <int DIM, int AHEAD = 0, class Accept, class Pair>
__device__ __forceinline__ void warp_pairs(const sph_config &c, const uint32_t *off,
                                           const float4 *pos, bool active, uint3 q,
                                           WarpPairSmem &sm, Accept accept, Pair pair, uint32_t self = 0)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    constexpr int nrows = DIM == 3 ? 9 : 3;   // rows (dy, dz), dz outer as in the reference loops
    int row = -1;
    uint32_t t = 0, e = 0;
    auto next_row = [&]() -> bool {
        while (++row < nrows) {
            const int dy = row % 3 - 1, dz = DIM == 3 ? row / 3 - 1 : 0;
            uint32_t b, ee;
            if (row_range<DIM>(c, off, q, dy, dz, b, ee) && ee > b) {
                t = b;
                e = ee;
                return true;
            }
        }
        return false;
    };
    uint32_t cnt = 0;
    auto flush = [&]() {
        const uint32_t m = __reduce_max_sync(full, cnt);
        if constexpr (AHEAD == 0) {
            for (uint32_t k = 0; k < m; ++k)
                if (k < cnt) pair(sm.lst[k][lane]);
        } else {
            uint32_t k = 0;
            for (; k + AHEAD <= m; k += AHEAD) {
                decltype(pair.fetch(self)) got[AHEAD];
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) got[u] = pair.fetch(k + u < cnt ? sm.lst[k + u][lane] : self);
#pragma unroll
                for (int u = 0; u < AHEAD; ++u)
                    if (k + u < cnt) pair.use(got[u]);
            }
            for (; k < m; ++k)
                if (k < cnt) pair.use(pair.fetch(sm.lst[k][lane]));
        }
        cnt = 0;
        __syncwarp();
    };
    bool more = active && next_row();
    while (__any_sync(full, more)) {
        if (more) {
            const uint32_t t0 = t, last = e - 1u;
            float4 pj[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) pj[u] = pos[min(t0 + u, last)];   // independent loads in flight
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (t0 + u < e && accept(t0 + u, pj[u])) sm.lst[cnt++][lane] = t0 + u;
            t = t0 + 4u;
            if (t >= e) more = next_row();
        }
        if (__any_sync(full, cnt >= kWarpCap)) flush();
    }
    if (__any_sync(full, cnt > 0)) flush();
}

// ------------------------------------------------------------ 5. density
// rho_i = m_i poly6_i h_i^6 + sum_{j != i, skip <= r^2 < h_i^2} m_j poly6_i (h_i^2 - r^2)^3
// p_i = k ((rho_i / rho0)^3 - 1)         (SPH-3D-2/sph_system.cu:338-677)
// The walk's inner loop is the distance test alone, on candidates staged in
// shared memory.  A warp's 32 particles lie in a few neighbouring cells, so
// their ranges of a stencil row overlap: the warp stages the row 64 slots at a
// time (each lane loads two, a chunk ahead of its use), laid out in pairs so
// that one packed FP32 instruction serves two candidates, and each lane tests
// its own range of it.  A candidate within (1 + margin) h_max goes, with its
// r^2, to the lane's column of a small buffer.  The warp drains its buffers
// together: each lane adds its buffered pairs into its own density sum in walk
// order (to the bit the sum of a walk that adds as it goes) and stores the
// slots to its candidate list in whole chunks of four.
// Bound: the L1 / shared-memory data pipe (77 % of its wavefronts) beside
// instruction issue (66 %).  A 16-byte global load costs the pipe at least 4
// wavefronts however many lanes share its address, a staged one 2 to 3; a
// walk that loaded each candidate from global memory, summed it at once and
// stored its slot with a 4-byte store of its own held the pipe at 83 %.
// 1.24M particles (four-way dam): 0.358 -> 0.287 ms; 1.05M without splits:
// 0.222 -> 0.177 ms.
constexpr uint32_t kDensLevel2 = 1u << 30;   // in a staged slot number: not level 1 (max_particle <= 2^30)

// CAP buffer entries per lane (entry-major: appends and reads hit distinct
// banks), and the staged chunk: pair p holds slots 2p and 2p + 1.
template <uint32_t CAP> struct DensSmem {
    uint2 ent[CAP][32];   // (r^2, tagged slot)
    float4 xy[34];        // (x0, x1, y0, y1); the last two are read past, never used
    uint4 zs[34];         // (z0, tagged slot 0, z1, tagged slot 1)
};

// SKIP = false: the config skips no close pairs (density_skip_r2 == 0), so
// the test !(r^2 < skip) is true for every r^2 and is left out.
// FLUSH: the buffer entries a warp keeps free for its next chunk.
// LISTS: only the candidate lists, of every neighbour within h_max (no margin),
// over n particles; cnt is not used.
template <int DIM, int BS, bool SKIP, uint32_t CAP, uint32_t FLUSH, bool LISTS = false>
__device__ __forceinline__ void density_walk(const sph_config &c, Counters *cnt, uint32_t n, const WorkPtrs &w,
                                             DensSmem<CAP> *smem)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    if (!LISTS && blockIdx.x == 0 && threadIdx.x == 0) {
        cnt->disp2_max = 0u;   // the force pass takes the max
        cnt->n_split = cnt->n_removed = cnt->split_off = 0u;   // set by the rank scans a step runs
    }
    DensSmem<CAP> &sm = smem[wib];
    uint2 *const col = &sm.ent[0][lane];
    // the append position as a shared-memory address (256 bytes per entry)
    const uint32_t col0 = (uint32_t)__cvta_generic_to_shared(col), col_lim = col0 + (CAP - 4) * 256u;
    constexpr int nrows = DIM == 3 ? 9 : 3, own = nrows / 2;
    // list entry k at lbase[(k >> 2) * row4 + (k & 3)] (the offset
    // fits 32 bits under the lists' 12 GB allocation limit)
    const bool rec = w.nlist != nullptr;
    const uint32_t row4 = w.nl_stride * 4u;
    // warp-uniform grid-stride loop: a warp takes 32 consecutive slots
    for (uint32_t base = blockIdx.x * BS + wib * 32u; base < n; base += gridDim.x * BS) {
        const uint32_t s_raw = base + lane;
        const bool valid = s_raw < n;
        const uint32_t s = valid ? s_raw : n - 1u;
        const float4 pi = w.spos[s];
        const int li = lv(pi.w);
        const float h2 = c.kernel2[li];
        const float poly6 = c.poly6[li];
        const uint32_t k = w.skey[s];
        const uint3 q = cell_of_key<DIM>(c, k);
        const float m0 = c.mass[0], m1 = c.mass[1], skip = c.density_skip_r2;
        // (m_j * poly6) once per level: the same product the sum takes first
        const float mp0 = m0 * poly6, mp1 = m1 * poly6;
        const float reach2 = LISTS ? fmaxf(c.kernel2[0], c.kernel2[1]) : rec ? energy_list_r2(c) : h2;
        const uint32_t self = s | (li ? kDensLevel2 : 0u);
        uint32_t *const lbase = rec ? w.nlist + (size_t)s * 4u : nullptr;
        float rho = 0.0f;
        uint32_t nb = 0, nl = 0;      // nl: entries drained so far (a multiple of 4 until the end)
        uint32_t at = col0;           // where the next buffer entry goes
        // one buffered pair into the sum: skip <= r^2 < h_i^2 (:394-417)
        auto take = [&](const uint2 ent) {
            if (LISTS) return;
            const float r2 = __uint_as_float(ent.x);
            const float x = h2 - r2;
            const float x3 = x * x * x;
            if ((!SKIP || !(r2 < skip)) && r2 < h2) {
                rho = __fmaf_rn(ent.y & kDensLevel2 ? mp1 : mp0, x3, rho);
                ++nb;
            }
        };
        // whole chunks of four, then (last) the rest; up to three entries stay
        // at the front of the buffer in between
        // (the appends in quad are opaque to the compiler: no load or store of
        // the buffer may move across either end of the drain)
        auto drain = [&](bool last) {
            asm volatile("" ::: "memory");
            const uint32_t fill = (at - col0) >> 8, whole = fill & ~3u;
            for (uint32_t g = 0; g < whole; g += 4) {
                const uint2 a0 = col[(g + 0) * 32], a1 = col[(g + 1) * 32], a2 = col[(g + 2) * 32],
                            a3 = col[(g + 3) * 32];
                take(a0);
                take(a1);
                take(a2);
                take(a3);
                if (rec && nl < kNbrListCap)
                    *reinterpret_cast<uint4 *>(lbase + (nl >> 2) * row4) =
                        make_uint4(a0.y & ~kDensLevel2, a1.y & ~kDensLevel2, a2.y & ~kDensLevel2,
                                   a3.y & ~kDensLevel2);
                nl += 4;
            }
            const uint32_t rest = fill - whole;
            if (last) {
                uint32_t t4[4] = {s, s, s, s};
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if ((uint32_t)u < rest) {
                        const uint2 a = col[(whole + u) * 32];
                        take(a);
                        t4[u] = a.y & ~kDensLevel2;
                    }
                if (rec && rest && nl < kNbrListCap)
                    *reinterpret_cast<uint4 *>(lbase + (nl >> 2) * row4) = make_uint4(t4[0], t4[1], t4[2], t4[3]);
                nl += rest;
            } else if (whole) {
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if ((uint32_t)u < rest) col[u * 32] = col[(whole + u) * 32];
            }
            at = col0 + rest * 256u;
            asm volatile("" ::: "memory");
        };
        const float2 nx = make_float2(-pi.x, -pi.x), ny = make_float2(-pi.y, -pi.y);
        // slots 2p .. 2p + 3 of the staged chunk: thr0: the bound of the first
        // (-1 when it lies before the lane's range); left: slots of the range
        // from 2p on.  r^2 is r2_of's to the bit, two candidates per
        // instruction (d = x_j + (-x_i) is the IEEE x_j - x_i).
        auto quad = [&](uint32_t i, float thr0, int left, auto OWN) {
            float r2[4];
            uint32_t id[4];
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
                const float4 a = sm.xy[(i + u) >> 1];
                const uint4 b = sm.zs[(i + u) >> 1];
                const float2 dx = __fadd2_rn(make_float2(a.x, a.y), nx), dy = __fadd2_rn(make_float2(a.z, a.w), ny);
                const float2 d2 = __ffma2_rn(dx, dx, __fmul2_rn(dy, dy));
                r2[u] = d2.x;
                r2[u + 1] = d2.y;
                if (DIM == 3) {
                    const float dz0 = __fsub_rn(__uint_as_float(b.x), pi.z), dz1 = __fsub_rn(__uint_as_float(b.z), pi.z);
                    r2[u] = __fmaf_rn(dz0, dz0, d2.x);
                    r2[u + 1] = __fmaf_rn(dz1, dz1, d2.y);
                }
                id[u] = b.y;
                id[u + 1] = b.w;
            }
            // predicated append: if (in range && r^2 < bound [&& not self])
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const float thr = u == 0 ? thr0 : reach2;
                if (OWN.value)
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %3, %5;\n\t"
                                 "setp.lt.and.f32 p, %1, %4, p;\n\tsetp.ne.and.u32 p, %2, %6, p;\n\t"
                                 "@p st.shared.v2.b32 [%0], {%1, %2};\n\t@p add.u32 %0, %0, 256;\n\t}"
                                 : "+r"(at) : "f"(r2[u]), "r"(id[u]), "r"(left), "f"(thr), "r"(u), "r"(self));
                else if (u == 0)
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, %3;\n\t"
                                 "@p st.shared.v2.b32 [%0], {%1, %2};\n\t@p add.u32 %0, %0, 256;\n\t}"
                                 : "+r"(at) : "f"(r2[u]), "r"(id[u]), "f"(thr));
                else
                    asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %3, %5;\n\t"
                                 "setp.lt.and.f32 p, %1, %4, p;\n\t"
                                 "@p st.shared.v2.b32 [%0], {%1, %2};\n\t@p add.u32 %0, %0, 256;\n\t}"
                                 : "+r"(at) : "f"(r2[u]), "r"(id[u]), "r"(left), "f"(thr), "r"(u));
            }
        };
        // the lane's slot range of row r: cells x - 1 .. x + 1 (inside the
        // grid) of row (dy, dz); rows outside the grid are empty
        const uint32_t key0 = k - (q.x > 0 ? 1u : 0u), key1 = k + (q.x + 1 < c.ncell[0] ? 2u : 1u);
        uint32_t rows_in = (q.y > 0 ? 1u : 0u) | 2u | (q.y + 1 < c.ncell[1] ? 4u : 0u);
        if (DIM == 3) rows_in = (q.z > 0 ? rows_in : 0u) | rows_in << 3 | (q.z + 1 < c.ncell[2] ? rows_in << 6 : 0u);
        if (!valid) rows_in = 0u;
        auto range = [&](int r, uint32_t &b, uint32_t &e) {
            b = e = 0u;
            if (rows_in >> r & 1u) {
                const uint32_t d = ((DIM == 3 ? r / 3 - 1 : 0) * (int)c.ncell[1] + r % 3 - 1) * (int)c.ncell[0];
                b = w.cell_off[key0 + d];
                e = w.cell_off[key1 + d];
            }
        };
        constexpr uint32_t none = 0xffffffffu;
        int row = 0;
        uint32_t b, e, b1, e1;
        range(0, b, e);
        range(1, b1, e1);
        uint32_t cb;              // first slot of the chunk to stage next (even)
        float4 st0, st1;          // its slots 2 lane and 2 lane + 1
        // the next chunk any lane needs, from `from` on in this row, else in
        // the rows that follow
        auto next_chunk = [&](uint32_t from) {
            for (;;) {
                const uint32_t lo = max(b, from);
                cb = __reduce_min_sync(full, lo < e ? lo : none);
                if (cb != none) break;
                if (++row >= nrows) return;
                b = b1;
                e = e1;
                range(row + 1, b1, e1);
                from = 0u;
            }
            cb &= ~1u;
            const uint32_t t = cb + 2u * lane;
            st0 = w.spos[min(t, n - 1u)];
            st1 = w.spos[min(t + 1u, n - 1u)];
        };
        next_chunk(0u);
#pragma unroll 1
        while (row < nrows) {
            const uint32_t t = cb + 2u * lane;
            __syncwarp();
            sm.xy[lane] = make_float4(st0.x, st1.x, st0.y, st1.y);
            sm.zs[lane] = make_uint4(__float_as_uint(st0.z), t | (st0.w == 1.0f ? 0u : kDensLevel2),
                                     __float_as_uint(st1.z), (t + 1u) | (st1.w == 1.0f ? 0u : kDensLevel2));
            __syncwarp();
            // this lane's part of the chunk, then the next chunk's loads
            const uint32_t lo = max(b, cb), hi = min(e, cb + 64u);
            int left = lo < hi ? (int)(hi - lo) : 0;
            uint32_t i = left ? lo - cb : 0u;
            float thr0 = i & 1u ? -1.0f : reach2;
            left += (int)(i & 1u);
            i &= ~1u;
            const bool own_row = row == own;
            next_chunk(cb + 64u);
            for (;;) {
                if (own_row) {
                    for (; left > 0 && at <= col_lim; i += 4, left -= 4, thr0 = reach2)
                        quad(i, thr0, left, std::true_type());
                } else {
                    for (; left > 0 && at <= col_lim; i += 4, left -= 4, thr0 = reach2)
                        quad(i, thr0, left, std::false_type());
                }
                const bool again = __any_sync(full, left > 0);   // a lane's buffer filled up
                if (again || __any_sync(full, at > col_lim - FLUSH * 256u)) drain(false);
                if (!again) break;
            }
        }
        drain(true);
        if (!valid) continue;
        if (LISTS) {
            w.ncnt[s] = nl;
            continue;
        }
        rho = __fadd_rn(rho, c.mass[li] * poly6 * c.kernel6[li]);   // self term
        float r = rho / c.rest_density;
        const float gas = w.nscenes ? w.scene_tab[2 * min(w.sscene[s], w.nscenes - 1u) + 1].w : c.gas_constant;
        float p = __fsub_rn(r * r * r, 1.0f) * gas;
        const float pr2 = p / (rho * rho), mr = c.mass[li] / rho;
        w.saux[s] = make_float4(rho, p, pr2, mr);
        const float4 evs = w.sev[s];
        w.fnb_a[s] = make_float4(pi.x, pi.y, pi.z, pr2);
        w.fnb_b[s] = make_float4(li ? -mr : mr, evs.x, evs.y, evs.z);
        w.snbr[s] = nb;
        if (rec) w.ncnt[s] = nl;
    }
}

template <int DIM, int BS, uint32_t CAP, uint32_t FLUSH>
__device__ __forceinline__ void density_body(const sph_config &c, Counters *cnt, const WorkPtrs &w,
                                             DensSmem<CAP> *smem)
{
    if (c.density_skip_r2 == 0.0f) density_walk<DIM, BS, false, CAP, FLUSH>(c, cnt, cnt->n, w, smem);
    else density_walk<DIM, BS, true, CAP, FLUSH>(c, cnt, cnt->n, w, smem);
}

// The standalone kernel is instantiated per SKIP (the host picks it): one
// walk per kernel keeps its registers at the walk's own need.  24 buffer
// entries per lane let seven 128-thread blocks reside (72 registers, 28 KB);
// 20 entries drain more often (304 against 294 us on 1.24M particles), 28
// leave less L1 (303).  Larger blocks take fewer entries to fit.
template <int BS> constexpr uint32_t kDensCap = BS <= 128 ? 24 : 18;
template <int BS> constexpr uint32_t kDensFlush = BS <= 128 ? 10 : 8;
template <int BS> constexpr size_t kDensSmemBytes = sizeof(DensSmem<kDensCap<BS>>) * (BS / 32);

template <int DIM, int BS = kThreads, bool SKIP = true>
__global__ void __launch_bounds__(BS) k_density(sph_config c, Counters *cnt, WorkPtrs w)
{
    extern __shared__ __align__(16) unsigned char dens_smem[];
    dependent_entry();
    density_walk<DIM, BS, SKIP, kDensCap<BS>, kDensFlush<BS>>(
        c, cnt, cnt->n, w, reinterpret_cast<DensSmem<kDensCap<BS>> *>(dens_smem));
}

// ------------------------------------------------------------ 6. force + integrate
// Pressure, viscosity and colour-field terms (SPH-3D-2/sph_system.cu:679-1137,
// 2D SPH-2D/sph_system.cu:462-790), then the integrator and walls
// (SPH-3D-2/sph_system.cu:204-322, SPH-2D/sph_system.cu:198-252).  The
// integrated state goes to the *_n arrays so the loop never sees it.
// Bound: the latency of the neighbour loads beside instruction issue (52 % of
// the slots).  Pairs that branch on their tests and take the IEEE square root
// (a branch and a second special-function instruction each) ran one after the
// other; computed without branches, the terms of four pairs overlap.  1.24M
// adaptive particles: 0.302 -> 0.223 ms; 1.05M plain: 0.193 -> 0.147 ms.
template <int DIM, int BS>
__device__ __forceinline__ void force_integrate_body(const sph_config &c, Counters *cnt, const WorkPtrs &w,
                                                     WarpPairSmem *smem)
{
    const uint32_t n = cnt->n;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    // warp-uniform grid-stride loop: a warp takes 32 consecutive slots
    for (uint32_t base = blockIdx.x * BS + wib * 32u; base < n; base += gridDim.x * BS) {
        const uint32_t s_raw = base + lane;
        const bool valid = s_raw < n;
        const uint32_t s = valid ? s_raw : n - 1u;
        const float4 pi = w.spos[s];
        const float4 evi = w.sev[s];
        const float4 ai = w.saux[s];   // rho, p, p/rho^2, m/rho
        const int li = lv(pi.w);
        const float hi = c.kernel[li], hi2 = c.kernel2[li];
        const float mi = c.mass[li];
        const float ispk = c.kernel_h6_twice ? c.spiky[li] / c.kernel6[li] : c.spiky[li];
        const float ivis = c.kernel_h6_twice ? c.visco[li] / c.kernel6[li] : c.visco[li];
        const float igrad = -c.grad_poly6[li];
        const float ilap = c.lapc_poly6[li];
        const uint32_t sid = w.nscenes ? min(w.sscene[s], w.nscenes - 1u) : 0u;
        const float visc = w.nscenes ? w.scene_tab[2 * sid].w : c.viscosity;
        float fx = 0.f, fy = 0.f, fz = 0.f, gx = 0.f, gy = 0.f, gz = 0.f, lap = 0.f;
        if (DIM == 2)   // self term, SPH-2D/sph_system.cu:599-603 (0 with the integer 3/4)
            lap = __fmaf_rn(ilap * ai.w * hi2, __fsub_rn(0.0f, c.lapc_three_quarters * hi2), lap);
        // pairs with r^2 < max(h_i^2, h_j^2) and r^2 >= close_r2 (:797-804)
        const float cut0 = fmaxf(hi2, c.kernel2[0]), cut1 = fmaxf(hi2, c.kernel2[1]);
        const float close = c.close_r2;
        // neighbour-level constants, once per particle instead of per pair
        const float jspk0 = c.kernel_h6_twice ? c.spiky[0] / c.kernel6[0] : c.spiky[0];
        const float jspk1 = c.kernel_h6_twice ? c.spiky[1] / c.kernel6[1] : c.spiky[1];
        const float jvis0 = c.kernel_h6_twice ? c.visco[0] / c.kernel6[0] : c.visco[0];
        const float jvis1 = c.kernel_h6_twice ? c.visco[1] / c.kernel6[1] : c.visco[1];
        const float hj0 = c.kernel[0], hj1 = c.kernel[1];
        // lap enters the force only through surface_coef
        const bool tension = c.surface_coef != 0.0f;
        const float mm0 = mi * c.mass[0], mm1 = mi * c.mass[1], mms = li ? mm1 : mm0;
        auto accept = [&](uint32_t t, const float4 &pj) {
            float rx, ry, rz;
            const float r2 = r2_of<DIM>(pi, pj, rx, ry, rz);
            const float cut = pj.w == 1.0f ? cut0 : cut1;
            return t != s && r2 < cut && !(r2 < close);
        };
        // Pressure, viscosity and colour-field terms of one neighbour (a, b: its
        // two records), added when `in` and r^2 passes the pair test.  The terms
        // are computed without a branch, so those of several pairs overlap in the
        // pipeline; only the sums are conditional.  SAME: the neighbour's level is
        // the particle's own, so the two kernels' terms are equal and half their
        // sum is either one, exactly.
        auto pair_ab = [&](bool in, const float4 a, const float4 b, auto SAME) {
            float rx, ry, rz;
            const float r2 = r2_of<DIM>(pi, a, rx, ry, rz);
            const bool lj = SAME.value ? li != 0 : signbit(b.x);
            const float mrj = fabsf(b.x);   // m_j/rho_j
            const bool ok = in && r2 < (SAME.value ? hi2 : lj ? cut1 : cut0) && !(r2 < close);
            const float ir = rsqrt_normal(r2), r = sqrt_of(r2, ir);
            const float ikr = __fsub_rn(hi, r);
            const bool iin = ikr > 0.0f;
            const float iq = iin ? ikr : 0.0f;
            const float ipk = ispk * iq * iq, ivk = ivis * iq;
            float pk = ipk, vk = ivk;   // half the two kernels' sums
            if (!SAME.value) {
                const float jkr = __fsub_rn(lj ? hj1 : hj0, r);
                const float jq = jkr > 0.0f ? jkr : 0.0f;
                pk = 0.5f * __fadd_rn(ipk, (lj ? jspk1 : jspk0) * jq * jq);
                vk = 0.5f * __fadd_rn(ivk, (lj ? jvis1 : jvis0) * jq);
            }
            const float x = hi2 - r2;
            const float tg = igrad * mrj * x * x;   // -grad_poly6 * m_j/rho_j * (h^2-r^2)^2
            const float tp = (SAME.value ? mms : lj ? mm1 : mm0) * __fadd_rn(ai.z, a.w) * pk * ir;
            const float tv = (ai.w * mrj) * visc * vk;
            const float dvx = __fsub_rn(b.y, evi.x), dvy = __fsub_rn(b.z, evi.y),
                        dvz = DIM == 3 ? __fsub_rn(b.w, evi.z) : 0.0f;
            auto sums = [&](float sg, float sp, float sv) {
                gx = __fmaf_rn(sg, rx, gx); gy = __fmaf_rn(sg, ry, gy);
                if (DIM == 3) gz = __fmaf_rn(sg, rz, gz);
                fx = __fmaf_rn(dvx, sv, __fmaf_rn(-rx, sp, fx));
                fy = __fmaf_rn(dvy, sv, __fmaf_rn(-ry, sp, fy));
                if (DIM == 3) fz = __fmaf_rn(dvz, sv, __fmaf_rn(-rz, sp, fz));
            };
            if (tension && ok && iin)
                lap = __fmaf_rn(ilap * mrj * x, __fsub_rn(r2, c.lapc_three_quarters * x), lap);
            if (SAME.value) {
                if (ok) sums(iin ? tg : 0.0f, tp, tv);
            } else {
                const float tgs = ok && iin ? tg : 0.0f;   // a zero term leaves a sum as it is
                if (ok) sums(tgs, tp, tv);
            }
        };
        auto pair = [&](uint32_t t) { pair_ab(true, w.fnb_a[t], w.fnb_b[t], std::false_type()); };
        const unsigned full = 0xffffffffu;
        const uint32_t nf = valid && w.nlist ? w.ncnt[s] : 0u;
        if (__all_sync(full, w.nlist != nullptr && nf <= kNbrListCap)) {
            // the density pass's candidates, filtered by the walk's test: same
            // neighbours, same order as the walk
            const uint32_t m = __reduce_max_sync(full, nf);
            // four entries per 16-byte load, a round ahead of their use; the
            // neighbours' loads issued before the math (entries past nf are
            // replaced by the particle itself)
            const uint4 *lp = reinterpret_cast<const uint4 *>(w.nlist) + s;   // chunk j at lp[j * nl_stride]
            uint4 nxt = m ? *lp : make_uint4(s, s, s, s);
            if (4 < m) prefetch_l2(lp + w.nl_stride);
            for (uint32_t kk = 0; kk < m; kk += 4) {
                const uint4 t4 = nxt;
                lp += w.nl_stride;
                if (kk + 8 < m) prefetch_l2(lp + w.nl_stride);   // 2 rounds ahead
                if (kk + 4 < m) nxt = *lp;
                const uint32_t tt[4] = {kk < nf ? t4.x : s, kk + 1 < nf ? t4.y : s, kk + 2 < nf ? t4.z : s,
                                        kk + 3 < nf ? t4.w : s};
                float4 na[4], nb[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    na[u] = w.fnb_a[tt[u]];
                    nb[u] = w.fnb_b[tt[u]];
                }
                // one level among the warp's pairs (most of the fluid): the shorter terms
                const uint32_t own = li ? 0x80000000u : 0u;
                const uint32_t other = (__float_as_uint(nb[0].x) ^ own) | (__float_as_uint(nb[1].x) ^ own) |
                                       (__float_as_uint(nb[2].x) ^ own) | (__float_as_uint(nb[3].x) ^ own);
                if (__any_sync(full, (int)other < 0)) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) pair_ab(kk + u < nf, na[u], nb[u], std::false_type());
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u) pair_ab(kk + u < nf, na[u], nb[u], std::true_type());
                }
            }
        } else {
            const uint3 q = cell_of_key<DIM>(c, w.skey[s]);
            warp_pairs<DIM>(c, w.cell_off, w.spos, valid, q, smem[wib], accept, pair);
        }
        if (!valid) continue;
        // surface tension switch (SPH-3D-2/sph_system.cu:1113-1136)
        const float nrm = sqrtf(__fmaf_rn(gz, gz, __fmaf_rn(gy, gy, __fmul_rn(gx, gx))));
        if (nrm > c.surface_threshold) {
            const float f = c.surface_coef * lap / nrm;
            fx = __fmaf_rn(f, gx, fx); fy = __fmaf_rn(f, gy, fy); fz = __fmaf_rn(f, gz, fz);
        }
        if (DIM == 2 && c.extern_force_on) {   // SPH-2D/sph_system.cu:781-789
            float xl = __fsub_rn(pi.x, c.extern_click[0]), yl = __fsub_rn(pi.y, c.extern_click[1]);
            if (__fmaf_rn(xl, xl, __fmul_rn(yl, yl)) <= __fmul_rn(c.extern_len, c.extern_len)) {
                fx = __fmaf_rn(c.extern_force[0], c.extern_coe, fx);
                fy = __fmaf_rn(c.extern_force[1], c.extern_coe, fy);
            }
        }
        w.ssurf[s] = nrm;

        // ---- integrate ----
        const float rho = ai.x, dt = c.time_step;
        float4 x = pi;
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f);   // low position part (compensated positions)
        float4 v = w.svel[s];
        float4 ev = evi;
        float4 a = make_float4(fx, fy, fz, 0.f);
        float rad;
        if (c.integrator == SPH_INTEGRATE_REF2D) {
            rad = c.radius[li] / 2.0f;
            a.x = __fmaf_rn(c.gravity[0], dt, a.x) / rho;
            a.y = __fmaf_rn(c.gravity[1], dt, a.y) / rho;
            v.x = __fmaf_rn(a.x, dt, v.x); v.y = __fmaf_rn(a.y, dt, v.y);
            ev.x = (ev.x + v.x) / 2.0f; ev.y = (ev.y + v.y) / 2.0f;
            x.x = __fmaf_rn(v.x, dt, x.x); x.y = __fmaf_rn(v.y, dt, x.y);
        } else {
            rad = c.radius[li];
            if (c.integrator == SPH_INTEGRATE_REF3D) {
                if (c.push_left && pi.x < __fdiv_rn(c.world[0], 3.0f) &&
                    pi.y > __fdiv_rn(c.world[1], (float)c.push_y_div))
                    a.x += 20.0f;
                if (c.push_right && pi.x > __fmul_rn(__fdiv_rn(c.world[0], 3.0f), 2.0f) &&
                    pi.y > __fdiv_rn(c.world[1], (float)c.push_y_div))
                    a.x -= 20.0f;
                v.x += a.x * dt / rho; v.y += a.y * dt / rho; v.z += a.z * dt / rho;
                v.x += c.gravity[0] * dt / rho; v.y += c.gravity[1] * dt / rho; v.z += c.gravity[2] * dt / rho;
            } else {
                const float im = 1.0f / mi;
                v.x = __fmaf_rn(__fmaf_rn(a.x, im, c.gravity[0]), dt, v.x);
                v.y = __fmaf_rn(__fmaf_rn(a.y, im, c.gravity[1]), dt, v.y);
                v.z = __fmaf_rn(__fmaf_rn(a.z, im, c.gravity[2]), dt, v.z);
            }
            if (w.pos_comp) {
                lo = w.spos_lo[s];
                comp_add(x.x, lo.x, __fmul_rn(v.x, dt));
                comp_add(x.y, lo.y, __fmul_rn(v.y, dt));
                if (DIM == 3) comp_add(x.z, lo.z, __fmul_rn(v.z, dt));
            } else {
                x.x = __fmaf_rn(v.x, dt, x.x); x.y = __fmaf_rn(v.y, dt, x.y); x.z = __fmaf_rn(v.z, dt, x.z);
            }
            if (DIM == 3 && c.use_cylinder) {   // SPH-3D-2/sph_system.cu:242-282
                for (int qq = 0; qq < 3; ++qq) {
                    const sph_sphere S = c.sphere[qq];
                    float dxs = x.x - S.pos[0], dys = x.y - S.pos[1], dzs = x.z - S.pos[2];
                    float dist = sqrtf(__fmaf_rn(dzs, dzs, __fmaf_rn(dys, dys, __fmul_rn(dxs, dxs))));
                    float R = S.radius + rad;
                    if (dist < R) {
                        float sx = dxs / dist * R, sy = dys / dist * R, sz = dzs / dist * R;
                        float il = rsqrtf(__fmaf_rn(sz, sz, __fmaf_rn(sy, sy, __fmul_rn(sx, sx))));
                        float nx = sx * il, ny = sy * il, nz = sz * il;
                        x.x = S.pos[0] + sx; x.y = S.pos[1] + sy; x.z = S.pos[2] + sz;
                        lo = make_float4(0.f, 0.f, 0.f, 0.f);
                        float vn = __fmaf_rn(v.z, nz, __fmaf_rn(v.y, ny, __fmul_rn(v.x, nx)));
                        const float dv = S.damping * vn;
                        v.x = __fmaf_rn(-dv, nx, v.x); v.y = __fmaf_rn(-dv, ny, v.y); v.z = __fmaf_rn(-dv, nz, v.z);
                    }
                }
            }
        }
        // walls x, y, z (SPH-3D-2/sph_system.cu:285-319); a batched scene
        // has its own box
        {
            const float4 blo = w.nscenes ? w.scene_tab[2 * sid] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 bhi = w.nscenes ? w.scene_tab[2 * sid + 1]
                                         : make_float4(c.world[0], c.world[1], c.world[2], 0.f);
            const float damp = c.wall_damping;
            uint32_t hit = 0;
            auto wall = [&](float &xd, float &vd, float &xl, float lo_b, float hi_b, int d) {
                const float hi_w = hi_b - rad, lo_w = lo_b + rad;
                if (xd >= hi_w) { vd *= damp; xd = hi_w; xl = 0.0f; hit |= 1u << (2 * d); }
                if (xd < lo_w) { vd *= damp; xd = lo_w; xl = 0.0f; hit |= 2u << (2 * d); }
            };
            wall(x.x, v.x, lo.x, blo.x, bhi.x, 0);
            wall(x.y, v.y, lo.y, blo.y, bhi.y, 1);
            if (DIM == 3) wall(x.z, v.z, lo.z, blo.z, bhi.z, 2);
            if (w.wall) w.wall[s] = hit;   // recorded for the adjoint
        }
        // a non-finite position is reported (the walls would hide +-inf); the
        // neighbour tests fail for it, so it interacts with nothing
        if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z)) || !isfinite(v.x + v.y + v.z))
            atomicOr(&cnt->error, 1u << SPH_ERR_NONFINITE);
        if (c.integrator != SPH_INTEGRATE_REF2D) {
            ev.x = (ev.x + v.x) / 2.0f; ev.y = (ev.y + v.y) / 2.0f; ev.z = (ev.z + v.z) / 2.0f;
        }
        w.spos_n[s] = x;        // .w keeps the level
        if (w.pos_comp) w.spos_lo_n[s] = lo;
        w.svel_n[s] = v;
        w.sev_n[s] = ev;
        w.sacc_n[s] = a;
        if (w.nlist) {   // the step's largest squared displacement, one atomic per group of lanes
            float ddx, ddy, ddz;
            const float d2 = r2_of<DIM>(x, pi, ddx, ddy, ddz);
            // non-negative floats order as their bits; a NaN position (which
            // passes no neighbour test) is left out
            const uint32_t bits = d2 == d2 ? __float_as_uint(d2) : 0u;
            const unsigned am = __activemask();
            const uint32_t m = __reduce_max_sync(am, bits);
            if (lane == __ffs(am) - 1) atomicMax(&cnt->disp2_max, m);
        }
    }
}

template <int DIM, int BS = kThreads, int MINB = 3>
__global__ void __launch_bounds__(BS, MINB) k_force_integrate(sph_config c, Counters *cnt,
                                                              WorkPtrs w)
{
    __shared__ WarpPairSmem smem[BS / 32];
    dependent_entry();
    force_integrate_body<DIM, BS>(c, cnt, w, smem);
}

// ------------------------------------------------------------ 7. energy + split decision
// Wavelet energy on the STALE cell lists (built at step start) with the NEW
// positions (SPH-3D-2/sph_system.cu:1169-1546), then the split decision
// (decide_adaptive_kernel, :1548-1574) written per particle index.
// Bound: the L1 cost of gathering 32 bytes per list entry (73 % of its data
// pipe; the gathers alone take 0.85 of the kernel's time).  The pair terms, x
// and y as packed FP32 and without branches, take 32M instead of 50M
// instructions on 387,000 particles.  1.24M adaptive particles: 0.252 ->
// 0.215 ms; 1.05M plain: 0.151 -> 0.134 ms.
// psi(x) = amp * (x^2/4 - 1) * EXP^(-x^2/8), EXP = 2.718281f (sigma = 2), for
// |x| < 30: x^2/4 is exact, so one fused multiply-add rounds as the difference
// does; the exponent's factor 1/8 is an exact scaling.
// 2^x by the PTX instruction, whose .ftz gives zero for a result below 2^-126;
// the bits of exp2f for every FP32 value in [-126, 0] (compared value by value;
// a pair inside the kernel has x >= -0.19).
__device__ __forceinline__ float ex2_normal(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

__device__ __forceinline__ float wavelet(float x, float amp)
{
    const float x2 = __fmul_rn(x, x);
    return __fmul_rn(__fmul_rn(amp, __fmaf_rn(x2, 0.25f, -1.0f)), ex2_normal(__fmul_rn(x2, -0.125f * 1.44269476f)));
}

// Two components at once (each half rounds as wavelet does).
__device__ __forceinline__ float2 wavelet2(float2 x, float amp)
{
    const float2 x2 = __fmul2_rn(x, x);
    const float2 e = __fmul2_rn(x2, make_float2(-0.125f * 1.44269476f, -0.125f * 1.44269476f));
    return __fmul2_rn(__fmul2_rn(make_float2(amp, amp), __ffma2_rn(x2, make_float2(0.25f, 0.25f),
                                                                   make_float2(-1.0f, -1.0f))),
                      make_float2(ex2_normal(e.x), ex2_normal(e.y)));
}

template <int DIM, int BS>
__device__ __forceinline__ void energy_split_body(const sph_config &c, Counters *cnt, const CanonPtrs &st,
                                                  const WorkPtrs &w, int want_tv, WarpPairSmem *smem)
{
    const uint32_t n = cnt->n;
    // 2/(PI^0.25 * sqrt(3 sigma)) with PI = 3.141592f, sigma = 2
    const float amp = 2.0f / (powf(3.141592f, 0.25f) * sqrtf(6.0f));
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    // displacement budget left for this particle's own move (the list covers
    // |d_i| + max_j |d_j| up to energy_list_budget)
    const float own_budget = w.nlist ? energy_list_budget(c) - sqrtf(__uint_as_float(cnt->disp2_max)) : -1.0f;
    for (uint32_t base = blockIdx.x * BS + wib * 32u; base < n; base += gridDim.x * BS) {
        const uint32_t s_raw = base + lane;
        const bool valid = s_raw < n;
        const uint32_t s = valid ? s_raw : n - 1u;
        const float4 pi = w.spos_n[s];
        const int li = lv(pi.w);
        const int lk = c.energy_large_kernel ? 0 : li;
        const float h = c.kernel[lk], h2 = c.kernel2[lk];
        const float ih = 1.0f / h, isq = 1.0f / sqrtf(h);
        const uint3 q = cell_of<DIM>(c, pi);
        float2 ts = make_float2(0.f, 0.f), tv = ts;   // x and y sums, z below
        float tsz = 0.f, tvz = 0.f;
        const float skip = c.energy_skip_close ? c.close_r2 : 0.0f;   // :1229-1232 (2D keeps close pairs)
        // j != i with skip <= r^2 < h^2 (:1222-1233), on the stale lists
        auto accept = [&](uint32_t t, const float4 &pj) {
            float rx, ry, rz;
            const float r2 = r2_of<DIM>(pi, pj, rx, ry, rz);
            return t != s && r2 < h2 && !(r2 < skip);
        };
        // the wavelet transform of one neighbour (its loads fetched ahead);
        // x and y as packed FP32, each half rounded as alone
        auto fetch = [&](uint32_t t) { return NbrPV{w.spos_n[t], w.svel_n[t]}; };
        auto add = [&](bool ok, const NbrPV &g, float2 rxy, float rz) {
            const float2 wxy = wavelet2(__fmul2_rn(rxy, make_float2(ih, ih)), amp);
            const float2 pxy = __fmul2_rn(make_float2(g.v.x, g.v.y), wxy);
            const float wz = DIM == 3 ? wavelet(__fmul_rn(rz, ih), amp) : 0.0f, pz = __fmul_rn(g.v.z, wz);
            if (ok) {
                ts = __fadd2_rn(ts, wxy);
                tv = __ffma2_rn(pxy, make_float2(isq, isq), tv);
                if (DIM == 3) {
                    tsz = __fadd_rn(tsz, wz);
                    tvz = __fmaf_rn(pz, isq, tvz);
                }
            }
        };
        auto use = [&](const NbrPV &g) {
            float rx, ry, rz;
            r2_of<DIM>(pi, g.p, rx, ry, rz);
            add(true, g, make_float2(rx, ry), rz);
        };
        // a list entry: the walk's test (a list never holds the particle itself)
        auto use_listed = [&](bool in, const NbrPV &g) {
            float rx, ry, rz;
            const float r2 = r2_of<DIM>(pi, g.p, rx, ry, rz);
            add(in && r2 < h2 && !(r2 < skip), g, make_float2(rx, ry), rz);
        };
        // the density pass's candidates when the particle kept its cell and the
        // step's moves fit the margin; the stencil walk otherwise
        // (every test is false for a NaN distance or budget: such a lane walks)
        // (no pairs at all in a taped step whose decisions do not read the energy)
        uint32_t ne = 0;
        bool walk = valid && !w.skip_energy;
        if (walk && own_budget >= 0.0f) {
            float ddx, ddy, ddz;
            const float d2 = r2_of<DIM>(pi, w.spos[s], ddx, ddy, ddz);
            const uint32_t cand = w.ncnt[s];
            if (cand <= kNbrListCap && key_of(c, q.x, q.y, q.z) == w.skey[s] && sqrtf(d2) <= own_budget) {
                ne = cand;
                walk = false;
            }
        }
        const uint32_t m = __reduce_max_sync(0xffffffffu, ne);
        if (m) {
            // four entries per 16-byte load, a round ahead of their use; their
            // neighbours fetched before the math (entries past ne are replaced
            // by the particle itself)
            const uint4 *lp = reinterpret_cast<const uint4 *>(w.nlist) + s;   // chunk j at lp[j * nl_stride]
            uint4 nxt = ne ? *lp : make_uint4(s, s, s, s);
            if (4 < m) prefetch_l2(lp + w.nl_stride);
            for (uint32_t kk = 0; kk < m; kk += 4) {
                const uint4 t4 = nxt;
                lp += w.nl_stride;
                if (kk + 8 < m) prefetch_l2(lp + w.nl_stride);   // 2 rounds ahead
                if (kk + 4 < ne) nxt = *lp;
                const uint32_t tt[4] = {kk < ne ? t4.x : s, kk + 1 < ne ? t4.y : s, kk + 2 < ne ? t4.z : s,
                                        kk + 3 < ne ? t4.w : s};
                NbrPV g[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) g[u] = fetch(tt[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    use_listed(kk + u < ne, g[u]);
            }
        }
        warp_pairs<DIM, 4>(c, w.cell_off, w.spos_n, walk, q, smem[wib], accept, fetch_use(fetch, use), s);
        if (!valid) continue;
        const float tvx = tv.x / ts.x, tvy = tv.y / ts.y;
        tvz = DIM == 3 ? tvz / tsz : 0.f;
        float energy = 0.5f * __fmaf_rn(tvx, tvx, __fmul_rn(tvy, tvy));
        if (c.energy_mass_weight) energy *= c.mass[li];
        w.senergy[s] = energy;
        if (want_tv) w.stv[s] = make_float4(tvx, tvy, tvz, 0.f);

        const uint32_t i = w.sidx[s];
        const float surf = w.ssurf[s];
        const float dens = w.saux[s].x;
        const uint32_t nb = w.snbr[s];
        uint32_t split = 0;
        if (c.use_split && pi.w == 1.0f) {
            if (c.split_rule == SPH_SPLIT_DEFICIT)
                split = (nb < c.split_min_neighbors || dens < c.split_density_ratio * c.rest_density) ? 1u : 0u;
            else
                split = split_score(c, energy, surf) > c.split_criteria ? 1u : 0u;
        }
        w.split_c[i] = split;
        if (split) atomicAdd(&cnt->split_flags, 1u);
        w.removed_c[i] = 0u;
        uint32_t inter = 0;
        if (c.merge_rule == SPH_MERGE_INTERIOR || c.merge_rule == SPH_MERGE_SIBLING) {
            const int flagged = nb < c.split_min_neighbors || dens < c.split_density_ratio * c.rest_density;
            inter = (flagged || split) ? 0u : st.interior[i] + 1u;
            w.sinter[s] = inter;
        }
        // a superset of merge_eligible's particles, whichever way the capacity
        // guard decides this step's splits (a split particle becomes level 2)
        if (c.use_merge && c.merge_rule != SPH_MERGE_WAVELET_CELL) {
            const bool l2 = pi.w != 1.0f;
            bool may;
            if (c.merge_rule == SPH_MERGE_WAVELET)
                may = (l2 && split_score(c, energy, surf) < c.merge_criteria) ||
                      (split && split_score(c, c.split_ways == 4 ? energy / 4.0f : energy, surf) < c.merge_criteria);
            else
                may = (l2 || split) && inter >= c.merge_interior_steps;
            if (may) atomicAdd(&cnt->merge_candidates, 1u);
        }
    }
}

template <int DIM, int BS = kThreads, int MINB = 3>
__global__ void __launch_bounds__(BS, MINB) k_energy_split(sph_config c, Counters *cnt,
                                                           CanonPtrs st, WorkPtrs w, int want_tv)
{
    __shared__ WarpPairSmem smem[BS / 32];
    dependent_entry();
    energy_split_body<DIM, BS>(c, cnt, st, w, want_tv, smem);
}

// Capacity guard after the split scan: if the children would not fit, this
// step runs without splits and reports SPH_ERR_CAPACITY (the reference writes
// past its buffer, SPH-3D-2/sph_system.cu:1645-1656).
__device__ __forceinline__ void split_guard_body(const sph_config &c, Counters *cnt, uint32_t n_split, uint32_t cap)
{
    uint64_t extra = c.split_ways == 4 ? 3u : 1u;
    uint64_t after = (uint64_t)cnt->n + (uint64_t)n_split * extra;
    if (after > cap) {
        cnt->split_off = 1u;
        cnt->error |= 1u << SPH_ERR_CAPACITY;
    } else {
        cnt->split_off = 0u;
    }
}

__global__ void __launch_bounds__(kClusterScanThreads) k_scan_cluster(ClusterScan j)
{
    dependent_entry();
    if (j.skip_if_zero && *j.skip_if_zero == 0u) {
        if (blockIdx.x == 0 && threadIdx.x == 0 && j.grand) *j.grand = 0u;
        return;
    }
    cluster_scan_body(j);
}

// The split rank scan as one cluster, with the guard on its total.
__global__ void __launch_bounds__(kClusterScanThreads) k_split_ranks(ClusterScan j, const sph_config c, Counters *cnt,
                                                                    uint32_t cap)
{
    dependent_entry();
    const uint32_t total = cnt->split_flags ? cluster_scan_body(j) : 0u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        cnt->n_split = total;
        split_guard_body(c, cnt, total, cap);
    }
}

// The ranks of a step's flags by a full grid of kScanBlocks, where 16 SMs are
// too few: chunk totals, then rescans.  Bound: the two reads and one write of
// the flags and the launches; 592 and 296 blocks save 2 us where there are no
// flags and lose 8 and 30 at 4.2M.  As ordinary launches with the guard a third
// one: 19.5 instead of 17.4 us at 1.05M particles, 12.3 instead of 9.2 without
// flags.  flags: their device count (at 0 only the total is written); guard:
// the flags are splits.
struct RankScan {
    uint32_t *in, *out, *list, *block_tot;
    const uint32_t *flags;
    uint32_t *total;
    int guard;
};

__global__ void __launch_bounds__(kScanThreads) k_rank_totals(RankScan j, const Counters *cnt)
{
    dependent_entry();
    if (*j.flags) scan_phase1_body<uint32_t>(j.in, cnt->n, j.block_tot);
}

__global__ void __launch_bounds__(kScanThreads) k_ranks(RankScan j, const sph_config c, Counters *cnt, uint32_t cap)
{
    dependent_entry();
    if (*j.flags) scan_phase23_body<uint32_t>(j.in, j.out, cnt->n, j.block_tot, j.total, 0, j.list);
    if (blockIdx.x == 0 && threadIdx.x == 0) {   // the thread that wrote the total
        if (*j.flags == 0u) *j.total = 0u;
        if (j.guard) split_guard_body(c, cnt, *j.total, cap);
    }
}

// ------------------------------------------------------------ 8. merge
// One warp per cell over its sorted members (merge_kernel,
// SPH-3D-2/sph_system.cu:1661-1789; 3D-4 :1702-1888; 2D :1177-1270).
// Eligible members (evaluated on the post-split values) are ranked by warp
// ballots in slot order; groups of `ways` consecutive eligible members merge
// into the first, with V = m/rho weights (level already set to 1 for the
// survivor, :1742-1777) or the plain mean in 2D.
constexpr int kMergeListMax = 256;   // eligible members held per warp in shared memory
// Cells per warp: as few as give every warp of the grid its share, from 2 to
// 32.  32 cells of a dense fluid (14 particles per cell) hold more eligible
// members than the list, and the warp then takes its cells one at a time; the
// 47,564-particle four-way frame (16,000 cells) spent 136 us so, and 73, 34, 20
// and 15 us with 16, 8, 4 and 2 cells.  A large empty grid keeps 32.
constexpr uint32_t kMergeCellsMin = 2, kMergeCellsMax = 32;

template <int DIM>
__device__ __forceinline__ int merge_eligible(const sph_config &c, const WorkPtrs &w, uint32_t t,
                                              uint32_t split_on, uint32_t ways, float cell_score)
{
    const uint32_t i = w.sidx[t];
    const uint32_t sp = split_on & w.split_c[i];
    const float lvl = sp ? 2.0f : w.spos_n[t].w;
    if (c.merge_rule == SPH_MERGE_WAVELET) {
        float en = w.senergy[t];
        if (sp && ways == 4) en = en / 4.0f;
        return lvl != 1.0f && split_score(c, en, w.ssurf[t]) < c.merge_criteria;
    }
    if (c.merge_rule == SPH_MERGE_WAVELET_CELL) return lvl == 2.0f && cell_score < c.merge_criteria;
    return lvl != 1.0f && w.sinter[t] >= c.merge_interior_steps;   // SPH_MERGE_INTERIOR, SPH_MERGE_SIBLING
}

// Merges the group g[0..ways) into g[0] (values on the post-split state).
template <int DIM>
__device__ __forceinline__ void merge_group(const sph_config &c, const WorkPtrs &w, const uint32_t *g,
                                            uint32_t ways, uint32_t split_on, float hs2, uint32_t *removed_flags)
{
    float V[4], Vs = 0.f;
    for (uint32_t k = 0; k < ways; ++k) {
        // eligible members are level 2; the survivor's level is set to 1
        // before its volume is taken (SPH-3D-2/sph_system.cu:1742-1756)
        V[k] = DIM == 2 ? 1.0f : (k == 0 ? c.mass[0] : c.mass[1]) / w.saux[g[k]].x;
        Vs += V[k];
    }
    float4 P = make_float4(0.f, 0.f, 0.f, 0.f), Vv = P, E = P, A = P;
    float en = 0.f;
    for (uint32_t k = 0; k < ways; ++k) {
        const uint32_t t = g[k];
        const uint32_t sp = split_on & w.split_c[w.sidx[t]];
        float4 p = w.spos_n[t];
        if (sp) p.x += hs2;
        const float4 vv = w.svel_n[t], ee = w.sev_n[t], aa = w.sacc_n[t];
        float ek = w.senergy[t];
        if (sp && ways == 4) ek = ek / 4.0f;
        P.x = __fmaf_rn(p.x, V[k], P.x); P.y = __fmaf_rn(p.y, V[k], P.y); P.z = __fmaf_rn(p.z, V[k], P.z);
        Vv.x = __fmaf_rn(vv.x, V[k], Vv.x); Vv.y = __fmaf_rn(vv.y, V[k], Vv.y); Vv.z = __fmaf_rn(vv.z, V[k], Vv.z);
        E.x = __fmaf_rn(ee.x, V[k], E.x); E.y = __fmaf_rn(ee.y, V[k], E.y); E.z = __fmaf_rn(ee.z, V[k], E.z);
        A.x = __fmaf_rn(aa.x, V[k], A.x); A.y = __fmaf_rn(aa.y, V[k], A.y); A.z = __fmaf_rn(aa.z, V[k], A.z);
        en += ek;
    }
    const uint32_t t1 = g[0];
    w.mpos[t1] = make_float4(P.x / Vs, P.y / Vs, P.z / Vs, 1.0f);
    w.mvel[t1] = make_float4(Vv.x / Vs, Vv.y / Vs, Vv.z / Vs, 0.f);
    w.mev[t1] = make_float4(E.x / Vs, E.y / Vs, E.z / Vs, 0.f);
    w.macc[t1] = make_float4(A.x / Vs, A.y / Vs, A.z / Vs, 0.f);
    w.menergy[t1] = en / (float)ways;
    w.leader[t1] = 1u;
    for (uint32_t k = 1; k < ways; ++k) w.removed_c[w.sidx[g[k]]] = 1u;
    atomicAdd(removed_flags, ways - 1u);
    if (w.merge_to) {   // recorded for the adjoint
        for (uint32_t k = 0; k < ways; ++k) w.merge_to[g[k]] = t1;
        w.mvs[t1] = Vs;
    }
}

// Shared memory of one warp of the merge pass.
struct MergeSmem {
    uint32_t list[kMergeListMax];    // eligible slots in slot order
    uint32_t lcell[kMergeListMax];   // their cells
    uint8_t lrank[kMergeListMax];    // their ranks among their cell's eligible members
};

template <int DIM>
__device__ __forceinline__ void merge_body(const sph_config &c, Counters *cnt, const CanonPtrs &st,
                                           const WorkPtrs &w, uint32_t ncells, uint32_t cap, MergeSmem *ms)
{
    // the energy pass found no candidate (the 2D cell rule is not counted there)
    if (c.merge_rule != SPH_MERGE_WAVELET_CELL && cnt->merge_candidates == 0u) return;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t warps_total = gridDim.x * (blockDim.x >> 5);
    const uint32_t n = cnt->n;
    const uint32_t split_on = cnt->split_off ? 0u : 1u;
    const uint32_t ways = c.split_ways == 4 ? 4u : 2u;
    const uint32_t extra = ways - 1u;
    const float hs2 = c.kernel[1] / 2.0f;
    // 2D rule: the criterion of the particle whose INDEX equals the cell
    // index, as memory holds it at merge time (SPH-2D/sph_system.cu:1207)
    auto cell_score_of = [&](uint32_t cell) -> float {
        if (c.merge_rule != SPH_MERGE_WAVELET_CELL) return 0.f;
        float eq, sq;
        const uint32_t n_after = n + (split_on ? cnt->n_split * extra : 0u);
        if (cell < n) {
            const uint32_t sl = w.inv[cell];
            eq = w.senergy[sl]; sq = w.ssurf[sl];
        } else if (cell < n_after) {
            const uint32_t sl = w.inv[w.split_list[(cell - n) / extra]];
            eq = w.senergy[sl]; sq = w.ssurf[sl];
        } else if (cell < cap) {
            eq = st.energy[cell]; sq = st.surface[cell];
        } else {
            eq = 0.f; sq = 0.f;   // beyond the allocation: treated as zeroed memory
        }
        return split_score(c, eq, sq);
    };
    // each warp takes `per` consecutive cells at a time; their members are one
    // contiguous slot range, tested 32 slots at a time
    const uint32_t per = min(max((ncells + warps_total - 1u) / warps_total, kMergeCellsMin), kMergeCellsMax);
    for (uint32_t base = (blockIdx.x * (blockDim.x >> 5) + wib) * per; base < ncells; base += warps_total * per) {
        const uint32_t cend = min(base + per, ncells);
        const uint32_t sb = w.cell_off[base], se = w.cell_off[cend];
        // every eligible member is listed with its cell and its rank among
        // the cell's eligible members (cells are contiguous in slot order; the
        // count of the chunk's last cell carries into the next chunk)
        uint32_t len = 0, carry_cell = kEmpty, carry_cnt = 0;
        for (uint32_t t0 = sb; t0 < se; t0 += 32) {
            const uint32_t t = t0 + lane;
            const bool in = t < se;
            const uint32_t cell = in ? w.skey[t] : kEmpty;
            const int el = in ? merge_eligible<DIM>(c, w, t, split_on, ways, cell_score_of(cell)) : 0;
            const unsigned same = __match_any_sync(full, cell);
            const unsigned eb = __ballot_sync(full, el);
            const uint32_t rank = __popc(eb & same & lt) + (cell == carry_cell ? carry_cnt : 0u);
            const uint32_t pos = len + __popc(eb & lt);
            if (el && pos < (uint32_t)kMergeListMax) {
                ms[wib].list[pos] = t;
                ms[wib].lcell[pos] = cell;
                ms[wib].lrank[pos] = (uint8_t)min(rank, 255u);   // a rank inside the list is below its length
            }
            len += __popc(eb);
            const int last = __popc(__ballot_sync(full, in)) - 1;
            const uint32_t lc = __shfl_sync(full, cell, last);
            const unsigned lsame = __shfl_sync(full, same, last);
            carry_cnt = (lc == carry_cell ? carry_cnt : 0u) + __popc(eb & lsame);
            carry_cell = lc;
        }
        __syncwarp();
        if (len <= (uint32_t)kMergeListMax) {
            // a group = `ways` consecutive eligible members of one cell, from
            // rank 0 on; its first member is the survivor
            for (uint32_t k = lane; k < len; k += 32)
                if (ms[wib].lrank[k] % ways == 0 && k + ways - 1 < len &&
                    ms[wib].lcell[k + ways - 1] == ms[wib].lcell[k])
                    merge_group<DIM>(c, w, &ms[wib].list[k], ways, split_on, hs2, &cnt->removed_flags);
            __syncwarp();
            continue;
        }
        // more eligible members than the list holds: the cells one at a time
        const uint32_t mine = base + lane;
        const uint32_t members = mine < cend ? w.cell_off[mine + 1] - w.cell_off[mine] : 0u;
        uint32_t todo = __ballot_sync(full, members >= ways);
        while (todo) {
            const uint32_t cell = base + (__ffs(todo) - 1);
            todo &= todo - 1;
            const uint32_t b = w.cell_off[cell], e = w.cell_off[cell + 1];
            const float cell_score = cell_score_of(cell);
            uint32_t count = 0;
            for (uint32_t t0 = b; t0 < e; t0 += 32) {
                const uint32_t t = t0 + lane;
                const int el = t < e ? merge_eligible<DIM>(c, w, t, split_on, ways, cell_score) : 0;
                const unsigned m = __ballot_sync(full, el);
                const uint32_t r = count + __popc(m & lt);
                if (el && r < (uint32_t)kMergeListMax) ms[wib].list[r] = t;
                count += __popc(m);
            }
            __syncwarp();
            const uint32_t groups = count / ways;
            if (count <= (uint32_t)kMergeListMax) {
                for (uint32_t g = lane; g < groups; g += 32)
                    merge_group<DIM>(c, w, &ms[wib].list[g * ways], ways, split_on, hs2, &cnt->removed_flags);
            } else if (lane == 0) {
                // more eligible members than the list holds: walk the cell
                // serially with the same group arithmetic
                uint32_t grp[4], got = 0, done = 0;
                for (uint32_t t = b; t < e && done < groups; ++t) {
                    if (!merge_eligible<DIM>(c, w, t, split_on, ways, cell_score)) continue;
                    grp[got++] = t;
                    if (got == ways) {
                        merge_group<DIM>(c, w, grp, ways, split_on, hs2, &cnt->removed_flags);
                        got = 0;
                        ++done;
                    }
                }
            }
            __syncwarp();
        }
    }
}

// SPH_MERGE_SIBLING: a split group (the parent and its children, linked in a
// ring by `sibling`) merges back into one particle when all its `ways`
// members are level 2 and have been interior for merge_interior_steps
// steps.  The member with the smallest particle index survives; the group
// is averaged in ring order from it, with merge_group's weights.  One thread
// per particle; only the survivor-to-be writes, so no group is merged twice.
template <int DIM>
__device__ __forceinline__ void merge_sibling_body(const sph_config &c, Counters *cnt, const CanonPtrs &st,
                                                   const WorkPtrs &w)
{
    if (cnt->merge_candidates == 0u) return;   // the energy pass found no candidate
    const uint32_t n = cnt->n;
    const uint32_t split_on = cnt->split_off ? 0u : 1u;
    const uint32_t ways = c.split_ways == 4 ? 4u : 2u;
    const float hs2 = c.kernel[1] / 2.0f;
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        const uint32_t si = w.inv[i];
        if (!merge_eligible<DIM>(c, w, si, split_on, ways, 0.f)) continue;
        uint32_t g[4];
        g[0] = si;
        uint32_t j = st.sibling[i];
        bool ok = true;
        for (uint32_t k = 1; k < ways && ok; ++k) {
            // a ring member of smaller index is the survivor-to-be; it merges
            ok = j < n && j > i;
            if (ok) {
                g[k] = w.inv[j];
                ok = merge_eligible<DIM>(c, w, g[k], split_on, ways, 0.f);
                j = st.sibling[j];
            }
        }
        if (ok && j == i) merge_group<DIM>(c, w, g, ways, split_on, hs2, &cnt->removed_flags);
    }
}

template <int DIM, int BS = kThreads>
__global__ void __launch_bounds__(BS) k_merge(sph_config c, Counters *cnt,
                                                   CanonPtrs st, WorkPtrs w, uint32_t ncells, uint32_t cap)
{
    __shared__ MergeSmem ms[BS / 32];
    dependent_entry();
    if (c.merge_rule == SPH_MERGE_SIBLING) merge_sibling_body<DIM>(c, cnt, st, w);
    else merge_body<DIM>(c, cnt, st, w, ncells, cap, ms);
}

// ------------------------------------------------------------ 10. write-out
// Stable partition by status (rearrange, SPH-3D-2/sph_system.cu:1818-1840):
// [surviving particles in index order][children in split order][removed].
// Children follow adaptive_particle_kernel (:1576-1615; 3D-4 :1583-1656;
// 2D :1133-1160).  Writes the other canonical buffer.
// The split and removal ranks (and the flags behind them) are read only where
// the step's counts of them are not zero.
// hash_next: also hash every particle it writes for the next step (hash_one
// at its new index; the cell counts were cleared after this step's scan), so
// the next step starts at the cell scan.
// Split groups: a parent and its children form a ring through `sibling`
// (parent -> child 0 -> ... -> last child -> parent); a surviving member's
// link follows the compaction; a merged survivor and everything else has none.
template <int DIM>
__device__ __forceinline__ void write_body(const sph_config &c, const Counters *cnt, Counters *cnt_next,
                                           const CanonPtrs &in, const CanonPtrs &out, const WorkPtrs &w,
                                           bool hash_next = false)
{
    const uint32_t n = cnt->n;
    const bool split_on = cnt->split_flags != 0u && !cnt->split_off;
    const bool merged = cnt->removed_flags != 0u;
    const uint32_t ways = c.split_ways == 4 ? 4u : 2u;
    const uint32_t extra = ways - 1u;
    const uint32_t n_split = split_on ? cnt->n_split : 0u;
    const uint32_t n_removed = merged ? cnt->n_removed : 0u;
    const uint32_t n_after = n + n_split * extra;
    const uint32_t n_live = n_after - n_removed;
    const float hs2 = c.kernel[1] / 2.0f;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        cnt_next->n = n_live;
        cnt_next->error = cnt->error;
        cnt_next->n_split = 0;
        cnt_next->n_removed = 0;
        cnt_next->split_off = 0;
        cnt_next->split_flags = 0;
        cnt_next->removed_flags = 0;
        cnt_next->merge_candidates = 0;
        if (w.step_counts) *w.step_counts = StepCounts{n, cnt->n_split, n_removed, cnt->split_off ? 0u : 1u};
    }
    // one thread per particle index: reads gather from the sorted slot, the
    // writes (survivors keep their order) stay coalesced
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        const uint32_t s = w.inv[i];
        const uint32_t sp = split_on ? w.split_c[i] : 0u;
        const uint32_t rm = merged ? w.removed_c[i] : 0u;
        const uint32_t rr = merged ? w.removed_rank[i] : 0u;
        const uint32_t dst = rm ? n_live + rr : i - rr;
        float4 p = w.spos_n[s], v = w.svel_n[s], e = w.sev_n[s];
        uint32_t inter = (c.merge_rule == SPH_MERGE_INTERIOR || c.merge_rule == SPH_MERGE_SIBLING) ? w.sinter[s] : 0u;
        const float4 p_pre = p;
        if (sp) {
            p.x += hs2;
            p.w = 2.0f;
            inter = 0u;
        }
        float4 plo = w.pos_comp ? w.spos_lo_n[s] : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 plo_pre = plo;
        uint32_t sib = kEmpty;
        const uint32_t leader = merged ? w.leader[s] : 0u;
        if (!rm && !leader) {
            const uint32_t j = in.sibling[i];
            if (j < n) sib = j - (merged ? w.removed_rank[j] : 0u);
        }
        if (sp) sib = n - n_removed + w.split_rank[i] * extra;   // the first child
        if (leader) {
            plo = make_float4(0.f, 0.f, 0.f, 0.f);   // a merged position is a fresh FP32 mean
            p = w.mpos[s]; v = w.mvel[s]; e = w.mev[s];
            inter = 0u;
            w.leader[s] = 0u;   // reset for the next step
        }
        out.pos[dst] = p; out.vel[dst] = v; out.ev[dst] = e;
        if (w.out_src) {
            if (!rm) w.out_src[dst] = s | (sp ? kOutSplit : 0u) | (leader ? kOutLeader : 0u);
        } else {
            const float4 aux = w.saux[s];
            float en = w.senergy[s];
            if (sp && ways == 4) en = en / 4.0f;
            float4 a = w.sacc_n[s];
            if (leader) {
                a = w.macc[s];
                if (DIM == 2) en = w.menergy[s];
            }
            out.acc[dst] = a; out.dens[dst] = aux.x; out.press[dst] = aux.y; out.energy[dst] = en;
            out.surface[dst] = w.ssurf[s];
        }
        out.interior[dst] = inter;
        out.sibling[dst] = sib;
        const uint32_t sid = w.nscenes ? w.sscene[s] : 0u;   // a merge group never spans scenes
        if (w.nscenes) out.scene[dst] = sid;
        if (w.pos_comp) out.pos_lo[dst] = plo;
        if (hash_next && !rm) hash_one<DIM>(c, w, dst, p);
        if (sp) {
            const uint32_t base = n - n_removed + w.split_rank[i] * extra;
            const float4 v0 = w.svel_n[s], e0 = w.sev_n[s];
            for (uint32_t k = 0; k < extra; ++k) {
                float4 pc = p_pre;
                pc.w = 2.0f;
                if (k == 0) pc.x = p_pre.x - hs2;
                else if (k == 1) pc.z = p_pre.z - hs2;
                else pc.z = p_pre.z + hs2;
                const uint32_t cd = base + k;
                out.pos[cd] = pc; out.vel[cd] = v0; out.ev[cd] = e0;
                if (w.out_src) {
                    w.out_src[cd] = s | kOutChild;
                } else {
                    const float4 aux = w.saux[s];
                    out.acc[cd] = w.sacc_n[s]; out.dens[cd] = aux.x; out.press[cd] = aux.y;
                    out.energy[cd] = ways == 4 ? w.senergy[s] / 4.0f : w.senergy[s]; out.surface[cd] = w.ssurf[s];
                }
                out.interior[cd] = 0u;
                out.sibling[cd] = k + 1 < extra ? cd + 1 : dst;
                if (w.nscenes) out.scene[cd] = sid;
                if (w.pos_comp) out.pos_lo[cd] = plo_pre;
                if (hash_next) hash_one<DIM>(c, w, cd, pc);
            }
        }
    }
}

// The deferred outputs of the state st (count cnt->n) from the sorted arrays
// of the step that wrote it, as write_body writes them.
template <int DIM>
__global__ void __launch_bounds__(kThreads) k_materialize(sph_config c, const Counters *cnt,
                                                         CanonPtrs st, WorkPtrs w)
{
    dependent_entry();
    const uint32_t n = cnt->n;
    const uint32_t ways = c.split_ways == 4 ? 4u : 2u;
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        const uint32_t code = w.out_src[i], s = code & kOutSlot;
        const float4 aux = w.saux[s];
        float en = w.senergy[s];
        float4 a = w.sacc_n[s];
        if (code & kOutChild) {
            en = ways == 4 ? en / 4.0f : en;
        } else {
            if ((code & kOutSplit) && ways == 4) en = en / 4.0f;
            if (code & kOutLeader) {
                a = w.macc[s];
                if (DIM == 2) en = w.menergy[s];
            }
        }
        st.acc[i] = a; st.dens[i] = aux.x; st.press[i] = aux.y; st.energy[i] = en; st.surface[i] = w.ssurf[s];
    }
}

template <int DIM, int BS = kThreads>
__global__ void __launch_bounds__(BS) k_write(sph_config c, const Counters *cnt,
                                                   Counters *cnt_next, CanonPtrs in, CanonPtrs out,
                                                   WorkPtrs w, int hash_next)
{
    dependent_entry();
    write_body<DIM>(c, cnt, cnt_next, in, out, w, hash_next != 0);
}

// ------------------------------------------------------------ reference-layout records
// 3D Particle (SPH-3D-2/sph_system.h:8-24), 18 words:
//   pos3 vel3 ev3 acc3 dens press energy surface tension level(u32)
// 2D Particle (SPH-2D/sph_system.h:7-22), 14 words (56 B, 8-byte aligned):
//   pos2 vel2 ev2 acc2 dens pres energy level(u32) surface_normal pad
template <int DIM> struct AosLayout;
template <> struct AosLayout<3> { static constexpr int words = 18; };
template <> struct AosLayout<2> { static constexpr int words = 14; };

template <int DIM>
__global__ void __launch_bounds__(kThreads) k_to_aos(const Counters *cnt, CanonPtrs st, float *aos)
{
    dependent_entry();
    const uint32_t n = cnt->n;
    constexpr int W = AosLayout<DIM>::words;
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        const float4 p = st.pos[i], v = st.vel[i], e = st.ev[i], a = st.acc[i];
        float *o = aos + (size_t)i * W;
        if (DIM == 3) {
            o[0] = p.x; o[1] = p.y; o[2] = p.z; o[3] = v.x; o[4] = v.y; o[5] = v.z;
            o[6] = e.x; o[7] = e.y; o[8] = e.z; o[9] = a.x; o[10] = a.y; o[11] = a.z;
            o[12] = st.dens[i]; o[13] = st.press[i]; o[14] = st.energy[i]; o[15] = st.surface[i];
            o[16] = 0.0f; o[17] = __uint_as_float((uint32_t)p.w);
        } else {
            o[0] = p.x; o[1] = p.y; o[2] = v.x; o[3] = v.y; o[4] = e.x; o[5] = e.y; o[6] = a.x; o[7] = a.y;
            o[8] = st.dens[i]; o[9] = st.press[i]; o[10] = st.energy[i];
            o[11] = __uint_as_float((uint32_t)p.w); o[12] = st.surface[i]; o[13] = 0.0f;
        }
    }
}

// Same records written straight into mapped page-locked host memory (at most
// max_rec of them) plus the live count.  Each block builds 256 records in
// shared memory and then stores them as one contiguous run, a warp writing
// 128 consecutive bytes per store, so the writes cross PCIe as full lines
// (a thread storing its own record would scatter 4-byte writes 72 bytes
// apart).  dst needs 4-byte alignment only.
template <int DIM>
__global__ void __launch_bounds__(kThreads) k_to_aos_mapped(const Counters *cnt, CanonPtrs st,
                                                           float *dst, uint32_t max_rec, uint32_t *count_dst)
{
    constexpr int W = AosLayout<DIM>::words;
    __shared__ float stage[kThreads * W];
    const uint32_t n = cnt->n;
    const uint32_t m = min(n, max_rec);
    if (blockIdx.x == 0 && threadIdx.x == 0) *count_dst = n;
    for (uint32_t base = blockIdx.x * kThreads; base < m; base += gridDim.x * kThreads) {
        const uint32_t i = base + threadIdx.x;
        if (i < m) {
            const float4 p = st.pos[i], v = st.vel[i], e = st.ev[i], a = st.acc[i];
            float *o = stage + threadIdx.x * W;
            if (DIM == 3) {
                o[0] = p.x; o[1] = p.y; o[2] = p.z; o[3] = v.x; o[4] = v.y; o[5] = v.z;
                o[6] = e.x; o[7] = e.y; o[8] = e.z; o[9] = a.x; o[10] = a.y; o[11] = a.z;
                o[12] = st.dens[i]; o[13] = st.press[i]; o[14] = st.energy[i]; o[15] = st.surface[i];
                o[16] = 0.0f; o[17] = __uint_as_float((uint32_t)p.w);
            } else {
                o[0] = p.x; o[1] = p.y; o[2] = v.x; o[3] = v.y; o[4] = e.x; o[5] = e.y; o[6] = a.x; o[7] = a.y;
                o[8] = st.dens[i]; o[9] = st.press[i]; o[10] = st.energy[i];
                o[11] = __uint_as_float((uint32_t)p.w); o[12] = st.surface[i]; o[13] = 0.0f;
            }
        }
        __syncthreads();
        const uint32_t words = min((uint32_t)kThreads, m - base) * W;
        float *out = dst + (size_t)base * W;
        for (uint32_t q = threadIdx.x; q < words; q += kThreads) out[q] = stage[q];
        __syncthreads();   // the stage is refilled next round
    }
}

template <int DIM>
__global__ void __launch_bounds__(kThreads) k_from_aos(uint32_t n, CanonPtrs st, const float *aos)
{
    dependent_entry();
    constexpr int W = AosLayout<DIM>::words;
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        const float *o = aos + (size_t)i * W;
        if (DIM == 3) {
            st.pos[i] = make_float4(o[0], o[1], o[2], (float)__float_as_uint(o[17]));
            st.vel[i] = make_float4(o[3], o[4], o[5], 0.f);
            st.ev[i] = make_float4(o[6], o[7], o[8], 0.f);
            st.acc[i] = make_float4(o[9], o[10], o[11], 0.f);
            st.dens[i] = o[12]; st.press[i] = o[13]; st.energy[i] = o[14]; st.surface[i] = o[15];
        } else {
            st.pos[i] = make_float4(o[0], o[1], 0.f, (float)__float_as_uint(o[11]));
            st.vel[i] = make_float4(o[2], o[3], 0.f, 0.f);
            st.ev[i] = make_float4(o[4], o[5], 0.f, 0.f);
            st.acc[i] = make_float4(o[6], o[7], 0.f, 0.f);
            st.dens[i] = o[8]; st.press[i] = o[9]; st.energy[i] = o[10]; st.surface[i] = o[12];
        }
        st.interior[i] = 0u;
        st.sibling[i] = kEmpty;   // nor split groups
        st.scene[i] = 0u;    // the record format carries no scene index
        st.pos_lo[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// ------------------------------------------------------------ state upload
// Particles first .. first + n of a state from the caller's arrays as uploaded
// (DIM floats per vector, null: zeros).
struct RawState {
    const float *pos, *vel, *ev, *acc;
    const uint32_t *level;
};

template <int DIM>
__global__ void __launch_bounds__(kThreads) k_unpack_state(uint32_t n, uint32_t first, RawState raw, CanonPtrs st)
{
    dependent_entry();
    auto vec = [](const float *a, uint32_t i, float w) {
        if (!a) return make_float4(0.f, 0.f, 0.f, w);
        a += (size_t)i * DIM;
        return make_float4(a[0], a[1], DIM == 3 ? a[2] : 0.f, w);
    };
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        const uint32_t o = first + i;
        st.pos[o] = vec(raw.pos, i, (float)raw.level[i]);
        st.vel[o] = vec(raw.vel, i, 0.f);
        st.ev[o] = vec(raw.ev, i, 0.f);
        st.acc[o] = vec(raw.acc, i, 0.f);
    }
}

// The count of a state the host has put in place.  A new state lets steps run
// again after a timeout, and both barrier states of the persistent step start
// clean (a timeout leaves its abort flag set): `words` u32 from gsync on.
__global__ void k_set_count(Counters *cnt, uint32_t n, uint32_t *gsync, uint32_t words)
{
    dependent_entry();
    if (threadIdx.x == 0) {
        cnt->n = n;
        cnt->error &= ~(1u << SPH_ERR_TIMEOUT);
    }
    if (threadIdx.x < words) gsync[threadIdx.x] = 0u;
}

// ------------------------------------------------------------ conserved quantities
// Per-block FP64 partial sums of mass, momentum (3), kinetic energy and
// gravitational potential energy (-m g.x) over the canonical state; a second
// single-block pass adds the partials in block order (deterministic).
constexpr int kConservedTerms = 6;

template <int DIM>
__global__ void __launch_bounds__(kThreads) k_conserved(sph_config c, const Counters *cnt, CanonPtrs st,
                                                        double *partial)
{
    const uint32_t n = cnt->n;
    double acc[kConservedTerms] = {0, 0, 0, 0, 0, 0};
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) {
        const float4 p = st.pos[i], v = st.vel[i];
        const double m = c.mass[lv(p.w)];
        const double vx = v.x, vy = v.y, vz = DIM == 3 ? v.z : 0.0;
        acc[0] += m;
        acc[1] += m * vx; acc[2] += m * vy; acc[3] += m * vz;
        acc[4] += 0.5 * m * (vx * vx + vy * vy + vz * vz);
        acc[5] -= m * ((double)c.gravity[0] * p.x + (double)c.gravity[1] * p.y +
                       (DIM == 3 ? (double)c.gravity[2] * p.z : 0.0));
    }
    __shared__ double red[kThreads / 32][kConservedTerms];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int k = 0; k < kConservedTerms; ++k) {
        double x = acc[k];
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) red[wid][k] = x;
    }
    __syncthreads();
    if (threadIdx.x < kConservedTerms) {
        double x = 0.0;
        for (int q = 0; q < kThreads / 32; ++q) x += red[q][threadIdx.x];
        partial[(size_t)blockIdx.x * kConservedTerms + threadIdx.x] = x;
    }
}

// Level-2 particles of the state (sph_last_step_stats): *out += the count.
__global__ void __launch_bounds__(kThreads) k_count_level2(const Counters *cnt,
                                                          const float4 *__restrict__ pos, uint32_t *out)
{
    const uint32_t n = cnt->n;
    uint32_t k = 0;
    for (uint32_t i = grid_stride_start(); i < n; i += grid_stride()) k += pos[i].w != 1.0f ? 1u : 0u;
    k = __reduce_add_sync(0xffffffffu, k);
    if ((threadIdx.x & 31) == 0 && k) atomicAdd(out, k);
}

__global__ void k_conserved_final(const double *partial, uint32_t blocks, double *out)
{
    if (threadIdx.x < kConservedTerms) {
        double x = 0.0;
        for (uint32_t b = 0; b < blocks; ++b) x += partial[(size_t)b * kConservedTerms + threadIdx.x];
        out[threadIdx.x] = x;
    }
}

// ------------------------------------------------------------ debug helpers
__global__ void k_cell_ranges(const uint32_t *__restrict__ off, uint32_t ncells, uint32_t *start, uint32_t *end)
{
    for (uint32_t q = grid_stride_start(); q < ncells; q += grid_stride()) {
        uint32_t b = off[q], e = off[q + 1];
        start[q] = e > b ? b : kEmpty;
        end[q] = e > b ? e : 0u;
    }
}

}  // namespace sph
