// Kernels of the FP32 split-precision step loop, shared by the
// single-scenario path and the batched / served paths. One step is
//   k_prep   (grid)    16 lanes per active tile: its 9 candidate ranges, its
//                      segment in the next buffer, node blocks of new grid tiles
//   k_p2g_tiles (grid) one CTA per active tile: P2G partial sums, tiles of
//                      more than split_min particles sorted by cell, the
//                      others in fixed point; k_p2g_cells in steps of many tiles
//   k_grid   (grid)    steps of many tiles: grid update + friction, a warp per
//                      half grid tile
//   k_g2p    (grid)    one CTA per active tile: (steps of few tiles: grid update
//                      of the tile's node window, then) G2P, advection,
//                      regrouping
//   k_end    (1 CTA)   per scenario: end of the step, then the next step's
//                      dt / stop rules and work-list prefix (k_arm_begin does
//                      the same at the start of an advance call)
// The CTAs share a flat list of work items of all scenarios (work_items,
// many_rounds), so one launch advances every running scenario by one step,
// each with its own dt and friction law.
//
// Every result is independent of the timing of the threads: the cell-sorted
// P2G sorts a tile's particles by cell in a stable, data-determined order and
// sums in that order; the sparse-tile P2G and the other fixed-point variants
// add integers, exact and associative; the grid update adds the partials of a node's tiles in a
// fixed order; G2P places particles by block prefix sums in candidate order;
// everything else is per particle or a max/min. So a step is bitwise
// reproducible, alone or inside a batch.
#pragma once

#include <type_traits>

#include "split32.cuh"
#include "tma.cuh"

namespace slab {
namespace k32 {

__device__ __forceinline__ int dir_i(int d) { return d / 3 - 1; }
__device__ __forceinline__ int dir_j(int d) { return d % 3 - 1; }

// flat work index -> (scenario, index in that scenario's list)
__device__ __forceinline__ bool find_work(const int32_t* pref, int nscn, int w, int& sid, int& loc) {
    if (w >= pref[nscn]) return false;
    int lo = 0, hi = nscn;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pref[mid] <= w) lo = mid; else hi = mid;
    }
    sid = lo;
    loc = w - pref[lo];
    return true;
}

// exclusive prefix over one value per thread (any blockDim <= 1024 that is a
// multiple of 32); s_warp needs blockDim/32 + 1 ints
__device__ int block_exclusive_scan(int v, int* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int t = lane < nw ? s_warp[lane] : 0;
        const int t0 = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += y;
        }
        if (lane < nw) s_warp[lane] = t - t0;
        if (lane == nw - 1) s_warp[nw] = t;
    }
    __syncthreads();
    const int r = s_warp[warp] + x - v;
    __syncthreads();
    return r;
}

// atomicAdd of `val` to *addr by the lanes in `mask`; lanes with the same
// address are combined into one atomic. Returns the lane's old value.
__device__ int warp_atomic_add(int* addr, int val, unsigned mask) {
    const unsigned peers = __match_any_sync(mask, (unsigned long long)addr);
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    int prefix = 0, total = 0;
    for (unsigned m = peers; m; m &= m - 1) {
        const int l = __ffs(m) - 1;
        const int v = __shfl_sync(peers, val, l);
        if (l < lane) prefix += v;
        total += v;
    }
    int base = 0;
    if (lane == leader) base = atomicAdd(addr, total);
    base = __shfl_sync(peers, base, leader);
    return base + prefix;
}

// candidate index -> particle index in the current buffer (range d)
__device__ __forceinline__ int cand_to_index(int q, const TileDesc& D, int& d) {
    d = 0;
    while (d < 8 && D.rpref[d + 1] <= q) ++d;
    return D.rstart[d] + (q - D.rpref[d]);
}

// candidate index -> particle index in the current buffer (range d). Most
// candidates are the tile's own stayers, range 4.
__device__ __forceinline__ int cand_index(int q, const TileDesc& D, int& d) {
    const int p4 = D.rpref[4], p5 = D.rpref[5];
    if (q >= p4 && q < p5) {
        d = 4;
        return D.rstart[4] + (q - p4);
    }
    d = q < p4 ? 0 : 5;
    while (d < 8 && D.rpref[d + 1] <= q) ++d;
    return D.rstart[d] + (q - D.rpref[d]);
}

// two-wide FP32 (one instruction each on sm_100), rounded as written
__device__ __forceinline__ float2 f2add(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 f2mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

constexpr int DESC_WORDS = (int)(sizeof(TileDesc) / 4);

// copy a descriptor to shared memory (its first threads)
__device__ __forceinline__ void load_desc(const TileDesc* g, TileDesc* s) {
    if (threadIdx.x < (int)(sizeof(TileDesc) / 4)) reinterpret_cast<int*>(s)[threadIdx.x] = reinterpret_cast<const int*>(g)[threadIdx.x];
}

__device__ __forceinline__ int tile_of_cell(int32_t cell, int TY) { return (cell_i(cell) / TILE) * TY + cell_j(cell) / TILE; }

// ---------------------------------------------------------------- control

// Step control of one scenario, one thread: what the step before left (its
// end), then the stop rules of the running advance call and
// Simulation::updateDt (ctl_begin), then the values that the step's kernels
// read. The control block and counters are read whole in one round and written
// back once: field by field, each branch waited for its own load (5.3 us for
// the kernel with one scenario, the time of about 12 dependent loads).
enum : int { CTL_T0, CTL_ARM, CTL_END };

__device__ __forceinline__ int step_control(const Shared& sh, int s, int what, int64_t steps_left, int stop_at_frame) {
    Ctl k = sh.ctl[s];
    SCnt n = sh.cnt[s];
    const int Np = sh.scn[s].Np;
    const float ood = sh.scn[s].ood;
    if (what == CTL_ARM) {  // start of an advance call: its step budget and frame-stop rule
        k.stop = 0;
        k.frame_hit = 0;
        k.steps_left = steps_left;
        k.stop_at_frame = stop_at_frame;
    }
    if (what == CTL_END && k.active) {
        if ((int32_t)n.cursor != Np) k.err |= ERR_CAPACITY;
        ctl_end(&k);
        n.seq += 1;
        n.vz_valid = n.outs;
    }
    if (what == CTL_T0) {  // simulate()'s t=0 pass for scenarios that still need it
        if (n.t0_pending) {
            ctl_begin_t0(&k, sh.Nx, sh.Ny);
            n.t0_pending = 0;
        } else {
            k.active = 0;
        }
    } else if (n.t0_pending) {
        k.active = 0;  // added after the last t=0 pass: waits for the next one
    } else {
        ctl_begin(&k, sh.Nx, sh.Ny);
    }
    int cnt = 0;
    if (k.active) {
        n.stepid += 1;
        n.act_count[0] = (n.seq & 1) ? 0 : n.act_count[0];  // the next step's list starts empty
        n.act_count[1] = (n.seq & 1) ? n.act_count[1] : 0;
        n.cursor = 0;
        if (n.heaviest) k.heaviest = n.heaviest;
        n.heaviest = 0;
        n.grid_mass = 0.0;
        n.outs = k.write_outputs;
        const int frame_after = k.frame + (k.frame_end ? 1 : 0);
        const double nft = __dmul_rn(k.output_dt, (double)(frame_after + 1));
        n.vz_next = (k.keep_outputs || __dadd_rn(k.new_time, k.dt_max) > nft - 1e-12) ? 1 : 0;
        cnt = (n.seq & 1) ? n.act_count[1] : n.act_count[0];
        k.tiles = cnt;
        SDyn y;
        y.seq = n.seq;
        y.stepid = n.stepid;
        y.outs = n.outs != 0;
        y.need_vz = n.outs || n.vz_next;
        y.dt = (float)k.dt;
        y.dt_ood = y.dt * ood;
        // Cells of the box's extreme particles at the start of the step. A
        // particle moves to a neighbour tile at most (farther raises
        // ERR_MOVE), less than 2 TILE cells, so after the step the box still
        // reaches to within that of its old faces; a tile whose particles all
        // end up further inside cannot change it.
        constexpr int D = 2 * TILE + 2;
        const int i0 = (int)(__longlong_as_double((long long)k.pos[0]) * k.one_over_dx);
        const int i1 = (int)(__longlong_as_double((long long)k.pos[1]) * k.one_over_dx);
        const int j0 = (int)(__longlong_as_double((long long)k.pos[2]) * k.one_over_dx);
        const int j1 = (int)(__longlong_as_double((long long)k.pos[3]) * k.one_over_dx);
        y.in_i0 = (i0 + D + TILE - 1) / TILE + 1;
        y.in_i1 = (i1 - D) / TILE - 2;
        y.in_j0 = (j0 + D + TILE - 1) / TILE + 1;
        y.in_j1 = (j1 - D) / TILE - 2;
        y.pad_[0] = y.pad_[1] = 0;
        sh.dyn[s] = y;
    }
    sh.ctl[s] = k;
    sh.cnt[s] = n;
    return cnt;
}

// K5, run by one CTA: the control of every scenario, then the prefix of
// active tiles over scenarios (the work list of the step).
__device__ __forceinline__ void control_scenarios(const Shared& sh, int what, int64_t steps_left = 0, int stop_at_frame = 0) {
    __shared__ int s_warp[33];
    __shared__ int s_tot;
    const int tid = threadIdx.x;
    int total = 0;
    for (int base = 0; base < sh.nscn; base += blockDim.x) {
        const int s = base + tid;
        const int cnt = s < sh.nscn ? step_control(sh, s, what, steps_left, stop_at_frame) : 0;
        if (sh.nscn == 1) {
            total = cnt;  // thread 0's, the only one that uses it
            if (tid == 0) sh.work_pref[0] = 0;
            break;
        }
        const int ex = block_exclusive_scan(cnt, s_warp);
        if (s < sh.nscn) sh.work_pref[s] = total + ex;
        if (tid == blockDim.x - 1) s_tot = ex + cnt;
        __syncthreads();
        total += s_tot;
        __syncthreads();
    }
    if (tid == 0) {
        sh.work_pref[sh.nscn] = min(total, sh.work_cap);
        for (int k = 0; k < NLISTCNT; ++k) sh.lists[k] = 0;
        if (total > sh.work_cap) atomicOr(&sh.ctl[0].err, ERR_CAPACITY);
    }
}

constexpr int CTL_THREADS = 256;  // one thread per scenario; enough registers for the control block

// Start of simulate()'s t=0 pass of the scenarios that still need it.
__global__ void __launch_bounds__(CTL_THREADS) k_begin_t0(Shared sh) {
    chain_wait<true>();
    control_scenarios(sh, CTL_T0);
}

// Start of an advance call: every scenario gets the step budget and the
// frame-stop rule, then the first step begins.
__global__ void __launch_bounds__(CTL_THREADS) k_arm_begin(Shared sh, int64_t steps_left, int stop_at_frame) {
    chain_wait<true>();
    control_scenarios(sh, CTL_ARM, steps_left, stop_at_frame);
}

// A scenario's static descriptor and step values in shared memory, loaded by
// the threads of a CTA (or warp) together: one round of loads, whatever a
// kernel reads of it afterwards. (One thread following the pointers field by
// field took four rounds at the start of every CTA.)
struct ScnSm {
    Scn s;
    SDyn y;
    int sid;
    int base;  // first work item of the scenario
    __device__ __forceinline__ PBuf cur() const { return s.buf[y.seq & 1]; }
    __device__ __forceinline__ PBuf next() const { return s.buf[(y.seq & 1) ^ 1]; }
};
static_assert(sizeof(Scn) % 16 == 0 && sizeof(SDyn) % 16 == 0, "loaded as 16-byte words");

__device__ __forceinline__ void load_scn_static(const Shared& sh, int sid, ScnSm& z, int t, int nt) {
    for (int k = t; k < (int)(sizeof(Scn) / 16); k += nt) reinterpret_cast<int4*>(&z.s)[k] = reinterpret_cast<const int4*>(sh.scn + sid)[k];
    if (t == 0) z.sid = sid;
}
__device__ __forceinline__ void load_scn_step(const Shared& sh, int sid, ScnSm& z, int t) {
    if (t == 0) z.base = sh.nscn == 1 ? 0 : sh.work_pref[sid];
    if (t < (int)(sizeof(SDyn) / 16)) reinterpret_cast<int4*>(&z.y)[t] = reinterpret_cast<const int4*>(sh.dyn + sid)[t];
}
__device__ __forceinline__ void load_scn(const Shared& sh, int sid, ScnSm& z, int t, int nt) {
    load_scn_static(sh, sid, z, t, nt);
    load_scn_step(sh, sid, z, t);
}

// Start of a kernel of the step chain. With one scenario (the small runs,
// where a step is a chain of dependent loads more than anything else) its
// descriptor, which no kernel of the chain writes, is in shared memory before
// the kernel before is over, and the step values are requested beside the
// work count and the first work item, which the caller guesses.

// The work items w0, w0 + step, ... < w1 of one of n workers. Of several
// scenarios a worker takes a contiguous run of the flat list, so that
// consecutive items mostly belong to the same scenario. Of one scenario it
// takes every n-th item: the list is roughly in the order of space, so runs of
// it are all dense tiles for one worker and all sparse ones for the next (300 k
// particles in a thin tongue: P2G 62 us with runs, 49 us with strides). P2G
// leaves this order in some steps, see many_rounds.
struct WorkItems {
    int w0, w1, step;
};
__device__ __forceinline__ WorkItems work_items(const Shared& sh, int nwork, int me, int n) {
    if (sh.nscn == 1) return {me, nwork, n};
    const int per = (nwork + n - 1) / n;
    const int w0 = min(me * per, nwork);
    return {w0, min(w0 + per, nwork), 1};
}

// Steps of one scenario whose descriptors k_prep orders by size: tiles with more
// than 5/4 of the mean particle count from the front, the others from the back.
// These are steps of a few tiles per P2G CTA (more than one, at most about 5),
// where the heaviest tiles decide when the last CTA is done: 637 k particles in
// 1 905 tiles of 1 to 980, P2G 44 us in list order, 39 us so. Longer steps keep
// the list order, which is that of space: ordered, 12 M particles (47 k tiles)
// took 72 us instead of 69 in the grid update and 25 instead of 21 in k_prep.
__device__ __forceinline__ bool ordered_by_size(const Shared& sh, int nwork) {
    return sh.nscn == 1 && !sh.use_xlist && nwork > sh.p2g_ctas && nwork < (1 << 16);
}

// Steps of one scenario in which a P2G CTA takes, after its first tile, the next
// one that no CTA has taken, instead of every gridDim.x-th: ordered ones, and
// those of many tiles per CTA, where CTAs drift apart and strided tiles that lie
// side by side run at different times. 12 M particles (40 tiles per CTA of
// k_p2g_cells): 235 -> 231 us. (G2P in turn: no gain.)
constexpr int TURN_ROUNDS = 16;
__device__ __forceinline__ bool many_rounds(const Shared& sh, int nwork) { return sh.nscn == 1 && nwork >= TURN_ROUNDS * (int)gridDim.x; }

// K1 (bookkeeping half): a tile's particles are the stayers of its own
// segment in the current buffer plus the movers of the 8 neighbour segments
// that moved to it (those are filtered by cell when read). The descriptor
// records these 9 candidate ranges and the exact count, reserves the tile's
// segment in the next buffer, and gives node blocks to the grid tiles of its
// node window that have none.
// Sixteen lanes (half a warp) per active tile, so that its independent
// global accesses go out together: lanes 0-8 read the 9 segment records,
// lanes 9-12 stamp the 4 grid tiles and see to their node blocks; the counts
// and range prefixes are half-warp shuffles, and the lanes write the
// descriptor's words side by side.
constexpr int PREP_LANES = 16;
constexpr int PREP_THREADS = 256;
constexpr int PREP_MAX_TILES = 1024 / PREP_LANES;  // tiles of one block pass (the persistent kernel runs larger blocks)
static_assert(offsetof(TileDesc, rstart) == 4 * 4 && offsetof(TileDesc, rpref) == 13 * 4 && offsetof(TileDesc, fresh) == 23 * 4 &&
                  offsetof(TileDesc, nb) == 28 * 4 && offsetof(TileDesc, tij) == 37 * 4 &&
                  offsetof(TileDesc, slot) == 38 * 4,
              "k_prep writes the descriptor word by word");

__device__ __forceinline__ void prep_body(const Shared& sh) {
    __shared__ int s_sid[PREP_MAX_TILES], s_cnt[PREP_MAX_TILES], s_off[PREP_MAX_TILES], s_pos[PREP_MAX_TILES];  // of the block's tiles
    __shared__ ScnSm s_one;
    const int lane = threadIdx.x & 31, r = lane & (PREP_LANES - 1);
    const int per_block = (int)blockDim.x / PREP_LANES, mine = threadIdx.x / PREP_LANES;
    const int stride = gridDim.x * per_block;
    const bool one = sh.nscn == 1;
    if (one) {
        load_scn_static(sh, 0, s_one, threadIdx.x, blockDim.x);
        __syncthreads();
    }
    chain_wait<false>();
    // one scenario: the tile's entry in both lists, before the step's parity and
    // the work count are known; later ones while the tile before is handled
    int e0 = 0, e1 = 0;
    auto entries = [&](int w) {
        if (one && w < s_one.s.act_cap) {
            e0 = s_one.s.act_list[0][w];
            e1 = s_one.s.act_list[1][w];
        }
    };
    entries((int)blockIdx.x * per_block + mine);
    const int nwork = sh.work_pref[sh.nscn];
    // whole blocks run every iteration (barriers and shuffles); a half warp
    // without a tile computes with valid = false
    for (int w0 = blockIdx.x * per_block; w0 < nwork; w0 += stride) {
        const int w = w0 + mine;
        const bool valid = w < nwork;
        int sid = 0, loc = 0;
        if (valid && !one) find_work(sh.work_pref, sh.nscn, w, sid, loc);
        const Scn& S = one ? s_one.s : sh.scn[sid];
        const SDyn& n = sh.dyn[sid];
        int seq = 0, stamp = 0, t = 0;
        if (valid) {
            seq = n.seq;
            stamp = n.stepid;
            if (one) {
                t = (seq & 1) ? e1 : e0;
            } else {
                const int32_t *l0 = S.act_list[0], *l1 = S.act_list[1];  // loaded beside seq
                t = ((seq & 1) ? l1 : l0)[loc];
            }
        }
        entries(w + stride);
        const int cur = seq & 1;
        const int ti = t / sh.TY, tj = t % sh.TY;
        // lanes 0-8: the record of neighbour d = r (its particles that moved to t);
        // lanes 9-12: the grid tiles of t's node window, stamped with this step.
        // All requests go out before the first answer is looked at.
        int4 g = make_int4(0, 0, 0, 0);
        int gc = 0, gst = -1, ast = -1, aslot = 0;
        if (valid && r < 9) {
            const int si = ti - dir_i(r), sj = tj - dir_j(r);
            if (si >= 0 && sj >= 0 && si < sh.TX && sj < sh.TY) {
                const int32_t* G = S.grp[cur] + (size_t)(si * sh.TY + sj) * GRP_STRIDE;
                g = *reinterpret_cast<const int4*>(G);
                gc = G[3 + r];
                gst = G[GRP_STAMP];
                const int2 ac = S.act[si * sh.TY + sj];
                ast = ac.x;
                aslot = ac.y;
            }
        }
        int gt = 0, was = 0x7fffffff, blk = -1;
        if (valid && r >= 9 && r < 13) {
            const int k = r - 9;
            const int gi = ti + (k >> 1), gj = tj + (k & 1);
            if (gi < sh.TX && gj < sh.TY) {
                gt = gi * sh.TY + gj;
                blk = S.blk_of[gt];
                was = atomicMax(&S.gt_stamp[gt], stamp);
            }
        }
        const bool live = gst == seq && r < 9 && valid;
        const int rs = live ? (r == 4 ? g.x : g.y) : 0, rl = live ? (r == 4 ? g.y - g.x : g.z - g.y) : 0, c = live ? gc : 0;
        const bool new_gt = was < stamp && valid;
        // that tile's partial window; one past the work list (ERR_CAPACITY) is not written
        const int sl = (one ? 0 : w - loc) + aslot;
        const int nb = ast == seq && sl < nwork && r < 9 && valid ? sl : -1;
        // half-warp shuffles: the tile's particle count and the range prefixes
        int incl = rl;
#pragma unroll
        for (int o = 1; o < PREP_LANES; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o, PREP_LANES);
            if (r >= o) incl += y;
        }
        int cnt = c;
#pragma unroll
        for (int o = PREP_LANES / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o, PREP_LANES);
        const int ncand = __shfl_sync(0xffffffffu, incl, 8, PREP_LANES);
        // a new grid tile's node block: the one it has, else one released by a
        // retired scenario, else a fresh one
        if (new_gt) {
            if (blk < 0) {
                const int f = atomicSub(sh.free_count, 1);
                if (f > 0) {
                    blk = sh.free_blocks[f - 1];
                } else {
                    atomicAdd(sh.free_count, 1);
                    blk = atomicAdd(sh.blk_count, 1);
                }
                if (blk >= sh.blk_cap) {
                    atomicOr(&S.ctl->err, ERR_CAPACITY);
                    blk = -1;
                } else {
                    S.blk_of[gt] = blk;
                    sh.blk_owner[blk] = sid;
                }
            }
            if (blk >= 0) sh.blk_stamp[blk] = stamp;
        } else if (blk < 0 && was != 0x7fffffff) {
            blk = BLK_LATER;  // another tile is giving it one
        }
        // grid tile k = r - 9 (its particle tile is neighbour t + (k >> 1, k & 1),
        // whose record lane 8 - direction read)
        const int gk = r - 9, from = (lane & ~(PREP_LANES - 1)) + 8 - (((gk >> 1) + 1) * 3 + (gk & 1) + 1);
        const int gnb = __shfl_sync(0xffffffffu, nb, r >= 9 && r < 13 ? from : lane);
        const bool fresh = new_gt && gnb < 0;
        const unsigned gmask = __ballot_sync(0xffffffffu, fresh);
        int xat = 0;
        if (gmask && sh.use_xlist) {  // the grid update's list of these
            int at = 0;
            if (lane == __ffs(gmask) - 1) at = atomicAdd(&sh.lists[LIST_X], __popc(gmask));
            xat = __shfl_sync(0xffffffffu, at, __ffs(gmask) - 1) + __popc(gmask & ((1u << lane) - 1u));
        }
        // the segment cursor: one atomic per scenario and block, by its first
        // warp (one per warp, with the counters of the step's lists, made 3
        // same-address atomics per two tiles: 44 us on 47 k tiles)
        if (r == 0) {
            s_sid[mine] = valid ? sid : -1;
            s_cnt[mine] = cnt;
            s_pos[mine] = w;
        }
        __syncthreads();
        if (one && threadIdx.x < 32) {
            const bool by_size = ordered_by_size(sh, nwork);
            const int heavy = by_size ? (int)__fdividef(1.25f * (float)s_one.s.Np, (float)nwork) : 0;
            for (int q0 = 0; q0 < per_block; q0 += 32) {
                const int q = q0 + lane;
                const bool has = q < per_block && s_sid[q] >= 0;
                const int qc = has ? s_cnt[q] : 0;
                int ic = qc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int yc = __shfl_up_sync(0xffffffffu, ic, o);
                    if (lane >= o) ic += yc;
                }
                const unsigned hm = __ballot_sync(0xffffffffu, by_size && has && qc > heavy), lm = __ballot_sync(0xffffffffu, by_size && has && qc <= heavy);
                if (nwork <= FUSED_MAX_TILES) {  // the host chooses the step's kernels by it
                    const unsigned top = __reduce_max_sync(0xffffffffu, (unsigned)qc);
                    if (lane == 0) atomicMax(&sh.cnt[0].heaviest, (int)top);
                }
                unsigned long long old = 0;
                if (lane == 31)
                    old = atomicAdd(reinterpret_cast<unsigned long long*>(&sh.cnt[0].cursor),
                                    (unsigned long long)ic + ((unsigned long long)__popc(hm) << 32) + ((unsigned long long)__popc(lm) << 48));
                old = __shfl_sync(0xffffffffu, old, 31);
                if (has) {
                    const unsigned lt = (1u << lane) - 1u;
                    s_off[q] = (int)(unsigned)old + ic - qc;
                    if (by_size)
                        s_pos[q] = qc > heavy ? (int)(old >> 32 & 0xffff) + __popc(hm & lt) : nwork - 1 - ((int)(old >> 48) + __popc(lm & lt));
                }
            }
        } else if (threadIdx.x < 32) {
            for (int q0 = 0; q0 < per_block; q0 += 32) {
                const int q = q0 + lane;
                const int qs = q < per_block ? s_sid[q] : -1;
                const unsigned m = __ballot_sync(0xffffffffu, qs >= 0);
                if (qs >= 0) s_off[q] = warp_atomic_add(reinterpret_cast<int*>(&sh.cnt[qs].cursor), s_cnt[q], m);  // its low word
            }
        }
        __syncthreads();
        const int nxt_off = s_off[mine], pos = s_pos[mine];
        if (fresh && sh.use_xlist) sh.xlist[xat] = pos << 2 | gk;
        // the descriptor, word by word (TileDesc: t, total, nxt_off, sid,
        // rstart[9], rpref[10], fresh, blk4[4], nb[9], tij, slot)
        if (valid) {
            int* D = reinterpret_cast<int*>(sh.desc + pos);
            if (r < 9) {
                D[4 + r] = rs;
                D[13 + r] = incl - rl;  // candidates before range r
                D[28 + 8 - r] = nb;     // (lane r read the tile at -direction r)
            } else if (r < 13) {
                D[24 + r - 9] = blk;
            } else if (r == 13) {
                D[22] = ncand;
            } else if (r == 14) {
                D[23] = (int)(gmask >> ((lane & ~(PREP_LANES - 1)) + 9)) & 0xf;
            } else {
                D[0] = t;
                D[1] = cnt;
                D[2] = nxt_off;
                D[3] = sid;
                D[37] = pack_cell(ti, tj);
                D[38] = w;
            }
        }
    }
}

__global__ void __launch_bounds__(PREP_THREADS) k_prep(Shared sh) { prep_body(sh); }

// ------------------------------------------------------------------- P2G

constexpr int NWIN = TN * TN;  // nodes of a tile's window
constexpr int NSLOT = 9;       // nodes a cell's particles reach (3 x 3)

// A tile's partial window (PART_STRIDE floats): {m, m h, m vx, m vy} per node,
// then {Fx, Fy} per node, then m vz per node (output steps): a node is one
// 16-byte and one 8-byte access, and the pairs are operands of the two-wide
// adds. Sum q (the order of NQ) and node of float k of it:
__device__ __forceinline__ void part_slot(int k, int& q, int& node) {
    if (k < 4 * NWIN) {
        const int c = k & 3;
        q = c == 0 ? 0 : (c == 1 ? 3 : c - 1);
        node = k >> 2;
    } else if (k < 6 * NWIN) {
        q = 4 + (k & 1);
        node = (k - 4 * NWIN) >> 1;
    } else {
        q = 6;
        node = k - 6 * NWIN;
    }
}

// A grid tile's node block, looked up where k_prep could not name it yet.
__device__ __forceinline__ int node_block(const Shared& sh, const Scn& S, const TileDesc& D, int k) {
    const int blk = D.blk4[k];
    return blk != BLK_LATER ? blk : S.blk_of[(cell_i(D.tij) + (k >> 1)) * sh.TY + cell_j(D.tij) + (k & 1)];
}

// Clears the nodes of the grid tiles that are no particle tiles of this step
// and that tile D touches first: their nodes are then written one by one by
// the tiles that reach them, the others keep zero. (t: thread of nt)
__device__ __forceinline__ void p2g_clear_fresh(const Shared& sh, const Scn& S, const TileDesc& D, bool outs, int t, int nt) {
    for (int k = 1; k < 4; ++k) {
        if (!(D.fresh >> k & 1)) continue;
        const int blk = node_block(sh, S, D, k);
        if (blk < 0) continue;
        for (int c = t; c < NCELL; c += nt) {
            const size_t bn = (size_t)blk * NCELL + c;
            sh.nv[bn] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (outs) sh.oh[bn] = sh.om[bn] = sh.ovz[bn] = sh.oFx[bn] = sh.oFy[bn] = 0.f;
        }
    }
}

constexpr int P2G_THREADS = NCELL;  // one thread per cell slot; the CTA strides over its tile's particles
constexpr int P2G_MIN_BLOCKS = NCELL == 64 ? 16 : 4;

// Fixed-point accumulation schemes of k_p2g:
//  ACC_I32   one int32 per sum, 2^-30 of the tile's bound
//  ACC_HILO  int32 pair: the rounded contribution and, 2^-20 finer, the
//            part below one quantum -- each contribution keeps about FP32
//            precision relative to itself; two plain (non-returning) atomics
//  ACC_I64   one int64 per sum at 2^-52 of the bound
//  ACC_CELL  no fixed point: every tile by k_p2g_tiles / k_p2g_cells, FP32
//            sums over cell-sorted particles
//  ACC_WARP  k_p2g_warp: ACC_HILO sums with one warp per tile
//  ACC_MIXED dense tiles (more than split_min particles) as ACC_CELL, the
//            others in fixed point (p2g_sparse_tile), in the same launch: a
//            tile's scheme depends only on its particle count, so results are
//            still reproducible
enum { ACC_I32 = 0, ACC_HILO = 1, ACC_I64 = 2, ACC_CELL = 3, ACC_WARP = 4, ACC_MIXED = 5 };

struct P2GSmem {
    long long node[NQ * TN * TN];  // fixed-point sums of the (TILE+2)^2 window (int32 pairs / int64)
    float4 dem[(TILE + 1) * (TILE + 1)];
    int ccnt[NCELL];
    unsigned bmax[NQ];             // per-quantity bound of one contribution (float bits)
    int mcc;                       // most particles in one cell of the tile
    float scale[NQ], iscale[NQ];
    TileDesc d;
};

// Per-particle P2G quantities (src/simulation.cpp:729-756): mass, momentum,
// m vz, m h, and for the force K = m g cos^2(theta) with the slope of the
// containing cell (src/complex_terrain.cpp:113-130) and the depth-averaged
// pressure sigma = -rho g cos^2 h / 2 with h A = m / rho.
struct PQ {
    float fx, fy, m, mvx, mvy, mh, mvz, Kgx, Kgy, Khh;
    int li, lj;
};

// from the particle's two words and vz, its cell (li, lj) in the tile and the
// tile's terrain window
__device__ __forceinline__ PQ make_pq(float4 a, float4 b, float vz, int li, int lj, const float4* dem, float g, float hod) {
    PQ p;
    const float4 dm = dem[(li + (a.x >= 1.f ? 1 : 0)) * (TILE + 1) + (lj + (a.y >= 1.f ? 1 : 0))];
    const float h = b.x, m = b.y;
    const float K = m * g * dm.z * dm.z;
    p.fx = a.x;
    p.fy = a.y;
    p.m = m;
    p.mvx = m * a.z;
    p.mvy = m * a.w;
    p.mh = m * h;
    p.mvz = m * vz;
    p.Kgx = K * dm.x;
    p.Kgy = K * dm.y;
    p.Khh = K * h * hod;
    p.li = li;
    p.lj = lj;
    return p;
}

__device__ __forceinline__ PQ load_pq(const PBuf& B, int src, int li, int lj, const float4* dem, float g, float hod, bool outs) {
    return make_pq(B.a[src], B.b[src], outs ? B.vz[src] : 0.f, li, lj, dem, g, hod);
}

// K2: P2G of one tile (src/simulation.cpp:726-798), one thread per particle,
// sums in 32-bit fixed point with shared-memory integer atomics. Integer
// addition is exact and associative, so the sums do not depend on the order
// in which particles arrive: the result is bitwise reproducible without
// sorting. Pass A finds, per quantity, a bound b on one contribution and the
// largest particle count of a cell; a node's sum then stays below
// 9 * cells_max * 0.75 * b, and the scale 2^e is the largest power of two
// that keeps that below 2^30. The resolution is 2^-30 of that bound, finer
// than FP32 relative to the largest contribution. Pass B adds the
// contributions; the window is converted back and written as the partials.
template <int ACC>
__global__ void __launch_bounds__(P2G_THREADS, P2G_MIN_BLOCKS) k_p2g(Shared sh) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    P2GSmem& sm = *reinterpret_cast<P2GSmem*>(smem_raw);
    chain_wait<true>();
    const int tid = threadIdx.x, lane = tid & 31;
    const WorkItems W = work_items(sh, sh.work_pref[sh.nscn], blockIdx.x, gridDim.x);
    for (int w = W.w0; w < W.w1; w += W.step) {
        load_desc(sh.desc + w, &sm.d);
        for (int k = tid; k < NQ * TN * TN; k += P2G_THREADS) sm.node[k] = 0;
        int* node32 = reinterpret_cast<int*>(sm.node);  // ACC_I32: [q][node]; ACC_HILO: hi at [q][node], lo at NQ*TN*TN + [q][node]
        for (int k = tid; k < NCELL; k += P2G_THREADS) sm.ccnt[k] = 0;
        if (tid < NQ) sm.bmax[tid] = 0u;
        if (tid == 0) sm.mcc = 0;
        __syncthreads();
        const Scn& S = sh.scn[sm.d.sid];
        const int t = sm.d.t;
        const int ti = t / sh.TY, tj = t % sh.TY;
        SCnt* n = S.cnt;
        p2g_clear_fresh(sh, S, sm.d, n->outs != 0, tid, P2G_THREADS);
        const int cur = n->seq & 1;
        const bool outs = n->outs != 0;
        for (int k = tid; k < (TILE + 1) * (TILE + 1); k += P2G_THREADS) {
            const int i = ti * TILE + k / (TILE + 1), j = tj * TILE + k % (TILE + 1);
            sm.dem[k] = (i < sh.Nx && j < sh.Ny) ? sh.dem[(int64_t)i * sh.Ny + j] : make_float4(0.f, 0.f, 1.f, 0.f);
        }
        __syncthreads();
        const int ncand = sm.d.rpref[9];
        const PBuf B = S.buf[cur];
        const float g = S.g, hod = 0.5f * S.ood;
        // pass A: bounds and cell counts
        float bm = 0.f, bvx = 0.f, bvy = 0.f, bh = 0.f, bvz = 0.f, bF = 0.f;
        for (int k = tid; k < ncand; k += P2G_THREADS) {
            int d;
            const int src = cand_to_index(k, sm.d, d);
            const int32_t cell = p_cell(B, src);
            const int li = cell_i(cell) - ti * TILE, lj = cell_j(cell) - tj * TILE;
            if ((unsigned)li >= TILE || (unsigned)lj >= TILE) {
                if (d == 4) atomicOr(&S.ctl->err, ERR_MOVE);  // a stayer outside its tile
                continue;
            }
            const PQ p = load_pq(B, src, li, lj, sm.dem, g, hod, outs);
            const int c = atomicAdd(&sm.ccnt[li * TILE + lj], 1) + 1;
            atomicMax(&sm.mcc, c);
            bm = fmaxf(bm, p.m);
            bvx = fmaxf(bvx, fabsf(p.mvx));
            bvy = fmaxf(bvy, fabsf(p.mvy));
            bh = fmaxf(bh, p.mh);
            bvz = fmaxf(bvz, fabsf(p.mvz));
            bF = fmaxf(bF, p.Khh + fmaxf(fabsf(p.Kgx), fabsf(p.Kgy)));
        }
        bm = warp_max(bm);
        bvx = warp_max(bvx);
        bvy = warp_max(bvy);
        bh = warp_max(bh);
        bvz = warp_max(bvz);
        bF = warp_max(bF);
        if (lane == 0) {
            atomicMax(&sm.bmax[0], __float_as_uint(bm));
            atomicMax(&sm.bmax[1], __float_as_uint(bvx));
            atomicMax(&sm.bmax[2], __float_as_uint(bvy));
            atomicMax(&sm.bmax[3], __float_as_uint(bh));
            atomicMax(&sm.bmax[4], __float_as_uint(bF));
            atomicMax(&sm.bmax[5], __float_as_uint(bF));
            atomicMax(&sm.bmax[6], __float_as_uint(bvz));
        }
        __syncthreads();
        if (tid < NQ) {
            const float bound = 9.f * (float)sm.mcc * 0.75f * __uint_as_float(sm.bmax[tid]);
            int e = 0;
            if (bound > 0.f) {
                int E;
                frexpf(bound, &E);  // bound < 2^E
                e = min(max((ACC == ACC_I64 ? 52 : 30) - E, -120), 120);
            }
            sm.scale[tid] = ldexpf(1.f, e);
            sm.iscale[tid] = ldexpf(1.f, -e);
        }
        __syncthreads();
        const float s0 = sm.scale[0], s1 = sm.scale[1], s2 = sm.scale[2], s3 = sm.scale[3], s4 = sm.scale[4], s5 = sm.scale[5],
                    s6 = sm.scale[6];
        const int lob = lo_bits_for(9 * sm.mcc);  // lo sums of a node stay below 2^30
        const float lo_mul = ldexpf(1.f, lob);
        const double lo_div = ldexp(1.0, -lob);
        // pass B: fixed-point contributions
        for (int k = tid; k < ncand; k += P2G_THREADS) {
            int d;
            const int src = cand_to_index(k, sm.d, d);
            const int32_t cell = p_cell(B, src);
            const int li = cell_i(cell) - ti * TILE, lj = cell_j(cell) - tj * TILE;
            if ((unsigned)li >= TILE || (unsigned)lj >= TILE) continue;
            const PQ p = load_pq(B, src, li, lj, sm.dem, g, hod, outs);
            float wx[3], wy[3], dwx[3], dwy[3];
            bspline3(p.fx, wx, dwx);
            bspline3(p.fy, wy, dwy);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const float wgt = wx[a] * wy[b];
                    if (wgt > 3e-3f) {  // the reference's weight cut-off (src/simulation.cpp:780)
                        const int nd = (li + a) * TN + (lj + b);
                        const float c[NQ] = {p.m * wgt, p.mvx * wgt, p.mvy * wgt, p.mh * wgt, p.Khh * (dwx[a] * wy[b]) - p.Kgx * wgt,
                                             p.Khh * (dwy[b] * wx[a]) - p.Kgy * wgt, p.mvz * wgt};
                        const float sc[NQ] = {s0, s1, s2, s3, s4, s5, s6};
#pragma unroll
                        for (int q = 0; q < NQ; ++q) {
                            if (q == 6 && !outs) continue;
                            if (ACC == ACC_I64) {
                                atomicAdd(reinterpret_cast<unsigned long long*>(sm.node + q * TN * TN + nd),
                                          (unsigned long long)__float2ll_rn(c[q] * sc[q]));
                            } else {
                                const float x = c[q] * sc[q];
                                const int hi = __float2int_rn(x);
                                atomicAdd(node32 + q * TN * TN + nd, hi);
                                if (ACC == ACC_HILO) {
                                    const int lo = __float2int_rn((x - (float)hi) * lo_mul);
                                    if (lo) atomicAdd(node32 + (NQ + q) * TN * TN + nd, lo);
                                }
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
        float* P = sh.part + (size_t)sm.d.slot * PART_STRIDE;
        for (int k = tid; k < PART_STRIDE; k += P2G_THREADS) {
            int q, nd;
            part_slot(k, q, nd);
            const int at = q * NWIN + nd;
            const float is = sm.iscale[q];
            float v;
            if (ACC == ACC_I64) v = (float)((double)sm.node[at] * (double)is);
            else if (ACC == ACC_HILO) v = (float)(((double)node32[at] + (double)node32[NQ * NWIN + at] * lo_div) * (double)is);
            else v = (float)node32[at] * is;
            P[k] = v;
        }
        __syncthreads();
    }
}

// --------------------------------------- P2G, one warp per tile (fixed point)

constexpr int P2W_WARPS = TILE == 8 ? 8 : 2;  // tiles in flight per CTA
constexpr int P2W_THREADS = 32 * P2W_WARPS;
constexpr int P2W_REG = 1;                     // chunks of 32 candidates a lane keeps between the passes

struct P2WWarp {
    int node[2 * NQ * TN * TN];  // fixed-point sums of the tile's node window: hi [q][node], then lo
    int ccnt[NCELL];             // particles per cell
    TileDesc d;
};

// P2G quantities of one candidate of tile (ti, tj), with the slope of its
// containing cell read from the FP32 terrain copy; valid = in the tile
__device__ __forceinline__ PQ warp_pq(const Shared& sh, const PBuf& B, const TileDesc& D, int k, int ti, int tj, float g, float hod, bool outs,
                                      bool& valid, bool& stayer) {
    int d;
    const int src = cand_to_index(k, D, d);
    const float4 pa = B.a[src], pb = B.b[src];
    const int32_t cell = __float_as_int(pb.z);
    const float2 f = make_float2(pa.x, pa.y), v = make_float2(pa.z, pa.w);
    const float h = pb.x, m = pb.y;
    const float vz = outs ? B.vz[src] : 0.f;
    const int ci = cell_i(cell), cj = cell_j(cell);
    const int li = ci - ti * TILE, lj = cj - tj * TILE;
    valid = (unsigned)li < TILE && (unsigned)lj < TILE;
    stayer = d == 4;
    PQ p;
    p.li = li;
    p.lj = lj;
    p.fx = f.x;
    p.fy = f.y;
    if (!valid) {
        p.m = p.mvx = p.mvy = p.mh = p.mvz = p.Kgx = p.Kgy = p.Khh = 0.f;
        return p;
    }
    const float4 dm = sh.dem[(int64_t)(ci + (f.x >= 1.f ? 1 : 0)) * sh.Ny + (cj + (f.y >= 1.f ? 1 : 0))];
    const float K = m * g * dm.z * dm.z;
    p.m = m;
    p.mvx = m * v.x;
    p.mvy = m * v.y;
    p.mh = m * h;
    p.mvz = m * vz;
    p.Kgx = K * dm.x;
    p.Kgy = K * dm.y;
    p.Khh = K * h * hod;
    return p;
}

// K2 variant: P2G of one tile (src/simulation.cpp:726-798) by one warp, so
// that many tiles are in flight on an SM with no block-wide barrier. The
// sums are 32-bit fixed-point pairs in the warp's shared-memory node window,
// added with integer atomics: exact and associative, so the result does not
// depend on the order of the particles (bitwise reproducible, the same alone
// or inside a batch). Pass A bounds one contribution per quantity (b) and the
// particles of one cell (mcc); a node's sum stays below 9 * mcc * 0.75 * b,
// and the scale is the largest power of two that keeps that below 2^30; the
// hi word is the rounded contribution, the lo word the rest at 2^-20.
__global__ void __launch_bounds__(P2W_THREADS, 3) k_p2g_warp(Shared sh) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    P2WWarp& sw = reinterpret_cast<P2WWarp*>(smem_raw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    chain_wait<true>();
    const int gw = blockIdx.x * P2W_WARPS + (threadIdx.x >> 5), nw = gridDim.x * P2W_WARPS;
    const int nwork = sh.work_pref[sh.nscn];
    const int per = (nwork + nw - 1) / nw;
    const int i0 = min(gw * per, nwork), i1 = min(i0 + per, nwork);
    int* hi = sw.node;
    int* lo = sw.node + NQ * TN * TN;
    for (int w = i0; w < i1; ++w) {
        for (int k = lane; k < DESC_WORDS; k += 32) reinterpret_cast<int*>(&sw.d)[k] = reinterpret_cast<const int*>(sh.desc + w)[k];
        for (int k = lane; k < 2 * NQ * TN * TN; k += 32) sw.node[k] = 0;
        for (int k = lane; k < NCELL; k += 32) sw.ccnt[k] = 0;
        __syncwarp();
        const TileDesc& D = sw.d;
        const Scn& S = sh.scn[D.sid];
        const SCnt* n = S.cnt;
        const int cur = n->seq & 1;
        const bool outs = n->outs != 0;
        p2g_clear_fresh(sh, S, D, outs, lane, 32);
        const int ti = D.t / sh.TY, tj = D.t % sh.TY;
        const int ncand = D.rpref[9];
        const PBuf B = S.buf[cur];
        const float g = S.g, hod = 0.5f * S.ood;
        // pass A: bounds and cell counts (the first chunks stay in registers)
        PQ keep[P2W_REG];
        bool kval[P2W_REG];
        float bm = 0.f, bvx = 0.f, bvy = 0.f, bh = 0.f, bvz = 0.f, bF = 0.f;
        int mcc = 0;
        for (int c = 0, k0 = 0; k0 < ncand; ++c, k0 += 32) {
            const int k = k0 + lane;
            bool valid = false, stayer = false;
            PQ p;
            if (k < ncand) p = warp_pq(sh, B, D, k, ti, tj, g, hod, outs, valid, stayer);
            if (k < ncand && !valid && stayer) atomicOr(&S.ctl->err, ERR_MOVE);  // a stayer outside its tile
#pragma unroll
            for (int r = 0; r < P2W_REG; ++r)
                if (c == r) {
                    keep[r] = p;
                    kval[r] = valid;
                }
            if (valid) {
                mcc = max(mcc, atomicAdd(&sw.ccnt[p.li * TILE + p.lj], 1) + 1);
                bm = fmaxf(bm, p.m);
                bvx = fmaxf(bvx, fabsf(p.mvx));
                bvy = fmaxf(bvy, fabsf(p.mvy));
                bh = fmaxf(bh, p.mh);
                bvz = fmaxf(bvz, fabsf(p.mvz));
                bF = fmaxf(bF, p.Khh + fmaxf(fabsf(p.Kgx), fabsf(p.Kgy)));
            }
        }
        bm = warp_max(bm);
        bvx = warp_max(bvx);
        bvy = warp_max(bvy);
        bh = warp_max(bh);
        bvz = warp_max(bvz);
        bF = warp_max(bF);
        for (int o = 16; o > 0; o >>= 1) mcc = max(mcc, __shfl_xor_sync(0xffffffffu, mcc, o));
        const float bq[NQ] = {bm, bvx, bvy, bh, bF, bF, bvz};
        float sc[NQ], isc[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float bound = 9.f * (float)mcc * 0.75f * bq[q];
            int e = 0;
            if (bound > 0.f) {
                int E;
                frexpf(bound, &E);  // bound < 2^E
                e = min(max(30 - E, -120), 120);
            }
            sc[q] = ldexpf(1.f, e);
            isc[q] = ldexpf(1.f, -e);
        }
        const int lob = lo_bits_for(9 * mcc);  // lo sums of a node stay below 2^30
        const float lo_mul = ldexpf(1.f, lob);
        const double lo_div = ldexp(1.0, -lob);
        // pass B: fixed-point contributions
        for (int c = 0, k0 = 0; k0 < ncand; ++c, k0 += 32) {
            const int k = k0 + lane;
            bool valid = false, stayer = false;
            PQ p;
            if (c < P2W_REG) {
#pragma unroll
                for (int r = 0; r < P2W_REG; ++r)
                    if (c == r) {
                        p = keep[r];
                        valid = kval[r];
                    }
            } else if (k < ncand) {
                p = warp_pq(sh, B, D, k, ti, tj, g, hod, outs, valid, stayer);
            }
            if (!valid) continue;
            float wx[3], wy[3], dwx[3], dwy[3];
            bspline3(p.fx, wx, dwx);
            bspline3(p.fy, wy, dwy);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const float wgt = wx[a] * wy[b];
                    if (wgt > 3e-3f) {  // the reference's weight cut-off (src/simulation.cpp:780)
                        const int nd = (p.li + a) * TN + (p.lj + b);
                        const float cq[NQ] = {p.m * wgt, p.mvx * wgt, p.mvy * wgt, p.mh * wgt, p.Khh * (dwx[a] * wy[b]) - p.Kgx * wgt,
                                              p.Khh * (dwy[b] * wx[a]) - p.Kgy * wgt, p.mvz * wgt};
#pragma unroll
                        for (int q = 0; q < NQ; ++q) {
                            if (q == 6 && !outs) continue;
                            const float x = cq[q] * sc[q];
                            const int h_ = __float2int_rn(x);
                            atomicAdd(hi + q * TN * TN + nd, h_);
                            const int l_ = __float2int_rn((x - (float)h_) * lo_mul);
                            if (l_) atomicAdd(lo + q * TN * TN + nd, l_);
                        }
                    }
                }
            }
        }
        __syncwarp();
        float* P = sh.part + (size_t)D.slot * PART_STRIDE;
        for (int k = lane; k < PART_STRIDE; k += 32) {
            int q, nd;
            part_slot(k, q, nd);
            float is = isc[0];
#pragma unroll
            for (int r = 1; r < NQ; ++r)
                if (q == r) is = isc[r];
            P[k] = (float)(((double)hi[q * NWIN + nd] + (double)lo[q * NWIN + nd] * lo_div) * (double)is);
        }
        __syncwarp();
    }
}

// Optional per-phase cycle counters of the P2G kernel (builds with
// -DSLAB_PHASE_CLOCKS only): thread 0 of each CTA adds the clock64 cycles of
// each phase of each tile to g_phase_clk[phase] (P2G 0-5, G2P 8-11);
// g_phase_clk[15] and [14] count their tiles.
#ifdef SLAB_PHASE_CLOCKS
__device__ unsigned long long g_phase_clk[16];
#define SLAB_PHASE_BEGIN long long t_prev_ = clock64()
#define SLAB_PHASE_MARK(k)                                                  \
    do {                                                                    \
        if (threadIdx.x == 0) {                                             \
            const long long c_ = clock64();                                 \
            atomicAdd(&g_phase_clk[k], (unsigned long long)(c_ - t_prev_)); \
            t_prev_ = c_;                                                   \
        }                                                                   \
    } while (0)
#define SLAB_PHASE_TILE()                                         \
    do {                                                          \
        if (threadIdx.x == 0) atomicAdd(&g_phase_clk[15], 1ull); \
    } while (0)
#define SLAB_PHASE_TILE_G2P()                                     \
    do {                                                          \
        if (threadIdx.x == 0) atomicAdd(&g_phase_clk[14], 1ull); \
    } while (0)
#else
#define SLAB_PHASE_BEGIN
#define SLAB_PHASE_MARK(k)
#define SLAB_PHASE_TILE()
#define SLAB_PHASE_TILE_G2P()
#endif

// --------------------------------------------------------- P2G over tiles

// K2: P2G of the active tiles (src/simulation.cpp:726-798), one CTA per tile, in
// two kernels with the same bits: k_p2g_tiles here, for steps of few tiles and for
// persistent steps, and k_p2g_cells below, for steps of many.
// A tile with more than split_min particles is summed in FP32 over its
// particles sorted by cell; one with fewer in exact fixed point (below). Which
// scheme a tile gets depends only on its own particle count.
//
// Dense tiles of k_p2g_tiles. Threads = 3 x cells, which keeps the chain of one
// tile short: thread (row, cell) owns stencil row `row`
// of its cell's 3 x 3 nodes, so the sums of a cell's particles stay in 18
// registers however many particles there are. Per pass of up to P2C_CAP
// candidates (one pass, but for very dense tiles):
//  1. the candidates (two float4 each) and the terrain window (one 2-D tensor
//     copy) are in shared memory: both were requested while the tile before
//     was summed, each thread the candidates that it reads itself. They are
//     counted per cell and chunk of 32 (lanes of one cell grouped by
//     __match_any_sync);
//  2. warp 0 turns the counts into each chunk's write cursors and the cells'
//     ranges: a stable counting sort by cell;
//  3. each thread writes its candidates' P2G quantities (mass, momentum, m h,
//     force terms) straight to their sorted places, so these are computed
//     once per particle and the sums read them in order. Places are XOR-
//     swizzled: 4 particles per cell, the common filling, put the 8 threads of
//     a 128-byte phase on 8 different 16-byte banks. The next pass's or
//     tile's candidates are requested into the places just read;
//  4. thread (row, cell) adds its cell's particles in sorted order over the 3
//     nodes of its row (packed two-wide FP32: mass and m h, the momentum, the
//     force). Every operation is rounded as written.
// Then the 9 row sums of every cell go to shared memory (over the stage), and
// one thread per node adds its <= 9 cells in (a, b) order and writes the
// tile's partial window: no zeroed node sums, no rounds between barriers.
// The candidates of a tile come in an order fixed by the previous step's G2P
// (ordered placement), so every sum has a fixed order: results are bitwise
// reproducible and the same alone or inside a batch.
constexpr int P2G_T = 3 * NCELL;        // threads of a CTA
constexpr int P2C_CAP = 6 * NCELL;      // candidates of one pass, two per thread (tiles of 1 to 980 particles: 40 us with 5 x 64
                                        // and 38 with 6 x 64; with 7 x 64 a third one per thread spills: 12 M particles 309 against 296)
constexpr int P2C_PER = (P2C_CAP + P2G_T - 1) / P2G_T;  // per thread
constexpr int P2C_CHUNKS = P2C_CAP / 32;
constexpr int P2C_HALVES = NCELL / 2;   // words of a chunk's 16-bit cell counts
#ifndef SLAB_P2G_MIN_BLOCKS
#define SLAB_P2G_MIN_BLOCKS (NCELL == 64 ? 6 : 1)
#endif

constexpr int P2S_CAP = NCELL;  // particles of a sparse tile (split_min is capped to it)

struct P2GSparseSmem {
    int hi[NQ * NWIN];  // fixed-point sums of the window, [q][node]: rounded part
    int lo[NQ * NWIN];  //                                         finer rest
    PQ pq[P2S_CAP];
    int ccnt[NCELL];
    unsigned bmax[NQ];
    int mcc, nv;
};

struct P2GTileSmem {
    union {
        struct {                // dense: a pass's particles in sorted, swizzled places
            float4 a[P2C_CAP];  // f.x, f.y, m vx, m vy
            float4 b[P2C_CAP];  // m, m h, -K gx, -K gy
            float k[P2C_CAP];   // K h / (2 dx); then, on output steps, m vz
        } st;
        struct {                         // dense: row sums [row * 3 + b][cell]
            float4 q4[NSLOT * NCELL];    // m, m h, m vx, m vy
            float2 q2[NSLOT * NCELL];    // F; then, on output steps, m vz
        } cs;
        P2GSparseSmem sp;
    };
    alignas(128) float4 dem[(TILE + 1) * (TILE + 1)];  // a tensor copy's destination: 128-byte aligned
    float4 ra[P2C_CAP], rb[P2C_CAP];                   // candidates as they lie in the particle buffer
    alignas(8) uint64_t dem_bar;                       // completion of the terrain window's copy
    uint32_t cnt[P2C_CHUNKS][P2C_HALVES];              // cell counts of a chunk, two 16-bit halves per word
    uint16_t cbeg[NCELL + 2];                          // first sorted place of each cell; [NCELL]: the pass's particles
    TileDesc d[2];                                     // this tile and the next
    int next_w;                                        // the next tile's place in the order of work
    ScnSm z;
};

__device__ __forceinline__ int p2c_place(int p) { return p ^ ((p >> 3) & 7); }

// node coordinates of a tile's first cell
struct TileOrigin {
    int i, j;
};

// Requests tile D's candidates base, base + 1, ... of one pass. Thread t copies
// the pass's candidates t, t + P2G_T, ... and is their only reader, so it may
// call this as soon as it has read the ones before.
__device__ __forceinline__ void p2g_request_cands(P2GTileSmem& sm, const TileDesc& D, int base) {
    const PBuf B = sm.z.cur();
    const int nc = min(D.rpref[9] - base, P2C_CAP);
    for (int k = threadIdx.x; k < nc; k += P2G_T) {
        int r;
        const int src = cand_index(base + k, D, r);
        cpa::copy16(&sm.ra[k], B.a + src);
        cpa::copy16(&sm.rb[k], B.b + src);
    }
}

// Requests tile D's first candidates and its terrain window (by thread 0, after
// a barrier that follows the last reads of the one before).
__device__ __forceinline__ void p2g_request(P2GTileSmem& sm, const Shared& sh, const TileDesc& D, int, int, const CUtensorMap* dem_map) {
    p2g_request_cands(sm, D, 0);
    if (threadIdx.x == 0) {
        // one 2-D tensor copy (TMA) of 9 x 9 nodes. The map sees the terrain as
        // [Nx][4 Ny] floats, so x = 4 tj TILE (a multiple of 16 bytes). Nodes
        // past the terrain's far edges read as zero; no valid particle uses
        // them (its stencil lies inside the terrain).
        tma::fence_proxy_async();
        tma::mbar_arrive_expect_tx(&sm.dem_bar, (TILE + 1) * (TILE + 1) * 16);
        tma::tensor_g2s_2d(sm.dem, dem_map, 4 * cell_j(D.tij) * TILE, cell_i(D.tij) * TILE, &sm.dem_bar);
    }
}

// The cells' sums into a partial window: thread (row, cell)'s row sums first,
// then one thread per node.
template <bool OUTS>
__device__ __forceinline__ void p2g_cells_to_window(P2GTileSmem& sm, float* part, const float2 (&am)[3], const float2 (&av)[3],
                                                    const float2 (&aF)[3], const float (&az)[3], int row, int cell) {
    __syncthreads();  // the stage is no longer read
#pragma unroll
    for (int b = 0; b < 3; ++b) {
        const int k = (row * 3 + b) * NCELL + cell;
        sm.cs.q4[k] = make_float4(am[b].x, am[b].y, av[b].x, av[b].y);
        sm.cs.q2[k] = aF[b];
    }
    __syncthreads();
    const int n = threadIdx.x, i = n / TN, j = n % TN;
    if (n < NWIN) {
        float2 m = make_float2(0.f, 0.f), v = m, F = m;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const int ci = i - a, cj = j - b;
                if ((unsigned)ci < TILE && (unsigned)cj < TILE) {
                    const int k = (a * 3 + b) * NCELL + ci * TILE + cj;
                    const float4 q = sm.cs.q4[k];
                    m = f2add(m, make_float2(q.x, q.y));
                    v = f2add(v, make_float2(q.z, q.w));
                    F = f2add(F, sm.cs.q2[k]);
                }
            }
        reinterpret_cast<float4*>(part)[n] = make_float4(m.x, m.y, v.x, v.y);
        reinterpret_cast<float2*>(part + 4 * NWIN)[n] = F;
    }
    if (OUTS) {
        __syncthreads();
#pragma unroll
        for (int b = 0; b < 3; ++b) sm.cs.q2[(row * 3 + b) * NCELL + cell].x = az[b];
        __syncthreads();
        if (n < NWIN) {
            float z = 0.f;
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const int ci = i - a, cj = j - b;
                    if ((unsigned)ci < TILE && (unsigned)cj < TILE) z = __fadd_rn(z, sm.cs.q2[(a * 3 + b) * NCELL + ci * TILE + cj].x);
                }
            part[6 * NWIN + n] = z;
        }
    }
}

// Weights of one particle offset along y for the 3 nodes of a row, both
// halves the same, and the row's along x: w = fma(sg, (hc t) t, w0), dw = dc t,
// t = f - s, the operations of bspline3 (for row 0 with the sign of both
// factors turned).
struct RowSpline {
    float s, hc, sg, w0, dc;
    __device__ __forceinline__ explicit RowSpline(int row)
        : s(row == 0 ? 1.5f : (row == 1 ? 1.0f : 0.5f)), hc(row == 1 ? 1.0f : 0.5f), sg(row == 1 ? -1.0f : 1.0f),
          w0(row == 1 ? 0.75f : 0.0f), dc(row == 1 ? -2.0f : 1.0f) {}
    __device__ __forceinline__ void x(float f, float& w, float& dw) const {
        const float t = __fsub_rn(f, s);
        w = __fmaf_rn(sg, __fmul_rn(__fmul_rn(hc, t), t), w0);
        dw = __fmul_rn(dc, t);
    }
};
__device__ __forceinline__ void spline_y(float f, float2 (&w)[3], float (&dw)[3]) {
    const float2 fy = make_float2(f, f);
    const float2 t0 = f2add(fy, make_float2(-1.5f, -1.5f)), t1 = f2add(fy, make_float2(-1.f, -1.f)), t2 = f2add(fy, make_float2(-0.5f, -0.5f));
    const float2 hf = make_float2(0.5f, 0.5f);
    w[0] = f2mul(f2mul(hf, t0), t0);
    w[1] = f2fma(f2mul(t1, t1), make_float2(-1.f, -1.f), make_float2(0.75f, 0.75f));
    w[2] = f2mul(f2mul(hf, t2), t2);
    dw[0] = t0.x;
    dw[1] = __fmul_rn(-2.0f, t1.x);
    dw[2] = t2.x;
}

template <bool OUTS, typename Next>
__device__ __forceinline__ void p2g_dense_tile(P2GTileSmem& sm, const TileDesc& D, float* part, uint32_t dem_phase, TileOrigin o,
                                               Next& next) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cell = tid % NCELL, row = tid / NCELL;  // row is the same in a whole warp
    Ctl* const ctl = sm.z.s.ctl;
    const int ncand = D.rpref[9];
    uint16_t* const cnt = reinterpret_cast<uint16_t*>(&sm.cnt[0][0]);  // zero here
    const float2 zero = make_float2(0.f, 0.f);
    float2 am[3] = {zero, zero, zero}, av[3] = {zero, zero, zero}, aF[3] = {zero, zero, zero};
    float az[3] = {0.f, 0.f, 0.f};
    int placed = 0;
    SLAB_PHASE_BEGIN;
    int base = 0;
    do {
        const int nc = min(P2C_CAP, ncand - base);
        if (base) {  // a later pass of a very dense tile
            cpa::wait_all();
            __syncthreads();  // the sums of the pass before are done with its places and ranges
        }
        SLAB_PHASE_MARK(0);
        // 1. count: this thread's candidates as local cell | rank << 16, -1: not in the tile
        int at[P2C_PER];
#pragma unroll
        for (int u = 0; u < P2C_PER; ++u) at[u] = -1;
#pragma unroll
        for (int u = 0; u < P2C_PER; ++u) {
            const int k = tid + u * P2G_T;
            if (k - lane >= nc) break;  // no candidate in the warp
            if (k < nc) {
                const int32_t c = __float_as_int(sm.rb[k].z);
                const int ci = cell_i(c) - o.i, cj = cell_j(c) - o.j;
                if ((unsigned)ci < TILE && (unsigned)cj < TILE) at[u] = ci * TILE + cj;
                else if (base + k >= D.rpref[4] && base + k < D.rpref[5]) atomicOr(&ctl->err, ERR_MOVE);  // a stayer outside its tile
            }
            const unsigned vm = __ballot_sync(0xffffffffu, at[u] >= 0);
            if (at[u] >= 0) {
                const unsigned peers = __match_any_sync(vm, at[u]);
                const int rank = __popc(peers & ((1u << lane) - 1u));
                if (rank == 0) cnt[(warp + u * (P2G_T / 32)) * NCELL + at[u]] = (uint16_t)__popc(peers);
                at[u] |= rank << 16;
            }
        }
        __syncthreads();
        if (base == 0) next.fetch();
        SLAB_PHASE_MARK(1);
        // 2. exclusive prefix over the chunks of every cell, then over the cells
        if (warp == 0) {
            constexpr int WPL = P2C_HALVES / 32;  // count words per lane
            uint32_t sum[WPL];
#pragma unroll
            for (int q = 0; q < WPL; ++q) sum[q] = 0;
#pragma unroll
            for (int c = 0; c < P2C_CHUNKS; ++c)
#pragma unroll
                for (int q = 0; q < WPL; ++q) {
                    const uint32_t x = sm.cnt[c][lane * WPL + q];
                    sm.cnt[c][lane * WPL + q] = sum[q];
                    sum[q] += x;  // halves stay below 2^16
                }
            int tot = 0;
#pragma unroll
            for (int q = 0; q < WPL; ++q) tot += (int)(sum[q] & 0xffffu) + (int)(sum[q] >> 16);
            int e = tot;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, e, s);
                if (lane >= s) e += y;
            }
            if (lane == 31) sm.cbeg[NCELL] = (uint16_t)e;
            e -= tot;
#pragma unroll
            for (int q = 0; q < WPL; ++q) {
                sm.cbeg[2 * (lane * WPL + q)] = (uint16_t)e;
                e += (int)(sum[q] & 0xffffu);
                sm.cbeg[2 * (lane * WPL + q) + 1] = (uint16_t)e;
                e += (int)(sum[q] >> 16);
            }
        }
        if (base == 0 && !tma::mbar_wait(&sm.dem_bar, dem_phase)) atomicOr(&ctl->err, ERR_TIMEOUT);  // the terrain window
        __syncthreads();
        SLAB_PHASE_MARK(2);
        // 3. quantities of every particle to its sorted place
        const float g = sm.z.s.g, hod = 0.5f * sm.z.s.ood;
#pragma unroll
        for (int u = 0; u < P2C_PER; ++u) {
            if (at[u] >= 0) {
                const int k = tid + u * P2G_T, lc = at[u] & 0xffff;
                const int p = p2c_place((int)sm.cbeg[lc] + (int)cnt[(warp + u * (P2G_T / 32)) * NCELL + lc] + (at[u] >> 16));
                const float4 qa = sm.ra[k], qb = sm.rb[k];
                const float4 qd = sm.dem[(lc / TILE + (qa.x >= 1.f ? 1 : 0)) * (TILE + 1) + (lc % TILE + (qa.y >= 1.f ? 1 : 0))];
                const float h = qb.x, m = qb.y;
                const float K = m * g * qd.z * qd.z;
                sm.st.a[p] = make_float4(qa.x, qa.y, m * qa.z, m * qa.w);
                sm.st.b[p] = make_float4(m, m * h, -(K * qd.x), -(K * qd.y));
                sm.st.k[p] = K * h * hod;
                at[u] = p;
            }
        }
        placed += sm.cbeg[NCELL];
        if (base == 0) next.store();
        __syncthreads();
        SLAB_PHASE_MARK(3);
        for (int k = tid; k < P2C_CHUNKS * P2C_HALVES; k += P2G_T) (&sm.cnt[0][0])[k] = 0;  // for the next pass or tile
        if (base + P2C_CAP >= ncand) next.request();
        else p2g_request_cands(sm, D, base + P2C_CAP);
        // 4. the cell's particles over the row's 3 nodes
        const RowSpline rs(row);
        const int r0 = sm.cbeg[cell], r1 = sm.cbeg[cell + 1];
        for (int r = r0; r < r1; ++r) {
            const int p = p2c_place(r);
            const float4 a = sm.st.a[p], b = sm.st.b[p];
            const float kh = sm.st.k[p];
            float wx, dwx, dwy[3];
            float2 wy[3];
            rs.x(a.x, wx, dwx);
            spline_y(a.y, wy, dwy);
            const float2 wx2 = make_float2(wx, wx), kh2 = make_float2(kh, kh);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float2 w = f2mul(wx2, wy[k]);
                if (w.x > 3e-3f) {  // the reference's weight cut-off (src/simulation.cpp:780)
                    am[k] = f2fma(make_float2(b.x, b.y), w, am[k]);
                    av[k] = f2fma(make_float2(a.z, a.w), w, av[k]);
                    const float2 gr = make_float2(__fmul_rn(dwx, wy[k].x), __fmul_rn(dwy[k], wx));
                    aF[k] = f2add(aF[k], f2fma(kh2, gr, f2mul(make_float2(b.z, b.w), w)));
                }
            }
        }
        if (OUTS) {  // m vz by a second walk, in the place of the force factor
            __syncthreads();
            const float* const gvz = sm.z.cur().vz;
            const float4* const gb = sm.z.cur().b;
#pragma unroll
            for (int u = 0; u < P2C_PER; ++u)
                if (at[u] >= 0) {
                    int d;
                    const int src = cand_index(base + tid + u * P2G_T, D, d);
                    sm.st.k[at[u]] = gb[src].y * gvz[src];
                }
            __syncthreads();
            for (int r = r0; r < r1; ++r) {
                const int p = p2c_place(r);
                const float4 a = sm.st.a[p];
                const float mz = sm.st.k[p];
                float wx, dwx, dwy[3];
                float2 wy[3];
                rs.x(a.x, wx, dwx);
                spline_y(a.y, wy, dwy);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const float w = __fmul_rn(wx, wy[k].x);
                    if (w > 3e-3f) az[k] = __fmaf_rn(mz, w, az[k]);
                }
            }
        }
        base += P2C_CAP;
        SLAB_PHASE_MARK(4);
    } while (base < ncand);
    if (tid == 0 && placed != D.total) atomicOr(&ctl->err, ERR_CAPACITY);
    p2g_cells_to_window<OUTS>(sm, part, am, av, aF, az, row, cell);
    SLAB_PHASE_MARK(5);
    SLAB_PHASE_TILE();
}

// A tile with at most split_min particles. Its time is latency, not
// arithmetic: pass A puts each particle's quantities in shared memory with the
// bound of one contribution per quantity (as k_p2g); pass B gives each thread
// one (particle, stencil row) item, three nodes each, added as the hi/lo
// 32-bit fixed-point pairs of k_p2g<ACC_HILO> with native shared-memory
// integer atomics. The integer sums are exact, so the result does not depend
// on arrival order.
// T threads; OVER: the sums lie over the candidates (ra, rb), which each thread
// reads first (its first two; of a tile with more than 2 T candidates, almost
// all of them other tiles' movers, the others come from the particle buffer).
template <int T, bool OVER, typename Next>
__device__ __forceinline__ void p2g_sparse_tile(P2GSparseSmem& sp, const float4* ra, const float4* rb, const float4* dem, uint64_t* dem_bar,
                                                uint32_t dem_phase, const ScnSm& Z, const TileDesc& D, float* part, TileOrigin o,
                                                Next& next) {
    constexpr int AHEAD = OVER ? 2 : 0;
    const int tid = threadIdx.x, lane = tid & 31;
    SLAB_PHASE_BEGIN;
    const PBuf B = Z.cur();
    Ctl* const ctl = Z.s.ctl;
    const bool outs = Z.y.outs != 0;
    const float g = Z.s.g, hod = 0.5f * Z.s.ood;
    const int ncand = D.rpref[9];
    float bm = 0.f, bvx = 0.f, bvy = 0.f, bh = 0.f, bvz = 0.f, bF = 0.f;
    float4 ca[2], cb[2];
    if (OVER) {
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
            const int k = tid + u * T;
            if (k < ncand) {
                ca[u] = ra[k];
                cb[u] = rb[k];
            }
        }
        __syncthreads();
    }
    for (int k = tid; k < 2 * NQ * NWIN / 4; k += T) reinterpret_cast<int4*>(sp.hi)[k] = make_int4(0, 0, 0, 0);  // hi and lo
    for (int k = tid; k < NCELL; k += T) sp.ccnt[k] = 0;
    if (tid < NQ) sp.bmax[tid] = 0u;
    if (tid == 0) {
        sp.mcc = 0;
        sp.nv = 0;
    }
    if (!tma::mbar_wait(dem_bar, dem_phase)) atomicOr(&ctl->err, ERR_TIMEOUT);
    __syncthreads();  // (the window of the tile before was read before the barrier of that tile's caller)
    next.fetch();
    // pass A: particle quantities, cell counts, bounds
    for (int k = tid; k < ncand; k += T) {
        int d;
        const int src = cand_index(k, D, d);
        float4 a, b;
        if (OVER && k < AHEAD * T) {
            a = k < T ? ca[0] : ca[1];
            b = k < T ? cb[0] : cb[1];
        } else if (!OVER && k < P2C_CAP) {
            a = ra[k];
            b = rb[k];
        } else {
            a = B.a[src];
            b = B.b[src];
        }
        const float vz = outs ? B.vz[src] : 0.f;
        const int32_t cell = __float_as_int(b.z);
        const int li = cell_i(cell) - o.i, lj = cell_j(cell) - o.j;
        if ((unsigned)li >= TILE || (unsigned)lj >= TILE) {
            if (d == 4) atomicOr(&ctl->err, ERR_MOVE);  // a stayer outside its tile
            continue;
        }
        const PQ p = make_pq(a, b, vz, li, lj, dem, g, hod);
        const int slot = atomicAdd(&sp.nv, 1);
        if (slot < P2S_CAP) sp.pq[slot] = p;
        else atomicOr(&ctl->err, ERR_CAPACITY);
        const int c = atomicAdd(&sp.ccnt[li * TILE + lj], 1) + 1;
        atomicMax(&sp.mcc, c);
        bm = fmaxf(bm, p.m);
        bvx = fmaxf(bvx, fabsf(p.mvx));
        bvy = fmaxf(bvy, fabsf(p.mvy));
        bh = fmaxf(bh, p.mh);
        bvz = fmaxf(bvz, fabsf(p.mvz));
        bF = fmaxf(bF, p.Khh + fmaxf(fabsf(p.Kgx), fabsf(p.Kgy)));
    }
    if ((tid & ~31) < ncand) {  // warps that hold a candidate; bounds are >= 0, so their bits order like the values
        const unsigned v[6] = {__float_as_uint(bm), __float_as_uint(bvx), __float_as_uint(bvy),
                               __float_as_uint(bh), __float_as_uint(bF), __float_as_uint(bvz)};
        unsigned r[6];
#pragma unroll
        for (int q = 0; q < 6; ++q) r[q] = __reduce_max_sync(0xffffffffu, v[q]);
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < 5; ++q) atomicMax(&sp.bmax[q], r[q]);
            atomicMax(&sp.bmax[5], r[4]);
            atomicMax(&sp.bmax[6], r[5]);
        }
    }
    next.store();
    __syncthreads();
    SLAB_PHASE_MARK(6);
    next.request();  // candidates and terrain window have been read
    // scales 2^e of the sums from the exponents of their bounds (bound < 2^E,
    // e = 30 - E, |e| <= 120), in every thread: integer operations instead of
    // frexp / ldexp by 7 threads between two barriers
    const int mcc = sp.mcc;
    int ex[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const float bound = 9.f * (float)mcc * 0.75f * __uint_as_float(sp.bmax[q]);
        const int E = (int)(__float_as_uint(bound) >> 23) - 126;
        ex[q] = bound > 0.f ? min(max(30 - E, -120), 120) : 0;
    }
    // pass B: (particle, stencil row) items. The atomics are unconditional: a
    // branch around an addition of zero kept the six sums' conversions from
    // overlapping (3100 cycles for the pass in an idle SM).
    const int nv = min(sp.nv, P2S_CAP);
    const int nmax = 9 * mcc, c2 = nmax <= 1 ? 0 : 32 - __clz(nmax - 1);
    const int lob = min(20, 31 - c2);  // lo_bits_for(nmax): lo sums of a node stay below 2^30 (20 bits for <= 64 particles)
    const float lo_mul = __int_as_float((127 + lob) << 23);
    for (int it = tid; it < 3 * nv; it += T) {
        const int pi = it / 3, a = it - 3 * pi;
        const PQ p = sp.pq[pi];
        float wx[3], wy[3], dwx[3], dwy[3];
        bspline3(p.fx, wx, dwx);
        bspline3(p.fy, wy, dwy);
        const float wxa = a == 0 ? wx[0] : (a == 1 ? wx[1] : wx[2]);
        const float dwxa = a == 0 ? dwx[0] : (a == 1 ? dwx[1] : dwx[2]);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const float wgt = wxa * wy[b];
            if (wgt > 3e-3f) {  // the reference's weight cut-off (src/simulation.cpp:780)
                const int nd = (p.li + a) * TN + (p.lj + b);
                const float cq[NQ] = {p.m * wgt, p.mvx * wgt, p.mvy * wgt, p.mh * wgt, p.Khh * (dwxa * wy[b]) - p.Kgx * wgt,
                                      p.Khh * (dwy[b] * wxa) - p.Kgy * wgt, p.mvz * wgt};
#pragma unroll
                for (int q = 0; q < NQ; ++q) {
                    if (q == 6 && !outs) continue;
                    const float x = cq[q] * __int_as_float((127 + ex[q]) << 23);
                    const int h_ = __float2int_rn(x);
                    atomicAdd(sp.hi + q * NWIN + nd, h_);
                    atomicAdd(sp.lo + q * NWIN + nd, __float2int_rn((x - (float)h_) * lo_mul));
                }
            }
        }
    }
    __syncthreads();
    SLAB_PHASE_MARK(12);
    // the window, one node per thread
    const double lo_div = __hiloint2double((1023 - lob) << 20, 0);
    for (int n = tid; n < NWIN; n += T) {
        float v[NQ];
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            v[q] = q < 6 || outs ? (float)(((double)sp.hi[q * NWIN + n] + (double)sp.lo[q * NWIN + n] * lo_div) *
                                           (double)__int_as_float((127 - ex[q]) << 23))
                                 : 0.f;
        reinterpret_cast<float4*>(part)[n] = make_float4(v[0], v[3], v[1], v[2]);
        reinterpret_cast<float2*>(part + 4 * NWIN)[n] = make_float2(v[4], v[5]);
        if (outs) part[6 * NWIN + n] = v[6];
    }
    SLAB_PHASE_MARK(13);
}

// The tile after the one that a P2G CTA sums. Its place in the order of work is
// known to thread 0 (wn: of one scenario, the next that no CTA has taken, the
// atomic issued a tile ahead) and shown to the others by the tile's first
// barrier; then come its descriptor and, when this tile's candidates have been
// read, its own candidates.
template <typename Sm> struct P2GNext {
    Sm& sm;
    const Shared& sh;
    const CUtensorMap* dem_map;
    int w, w1, step, cur, wn, dn;
    bool in_turn, requested;
    int buf;  // where the next pass's candidates go (P2GCellSmem)
    __device__ __forceinline__ void take() {  // thread 0
        if (in_turn) wn = (int)gridDim.x + atomicAdd(&sh.lists[LIST_P2G], 1);
    }
    __device__ __forceinline__ void fetch() {
        w = in_turn ? sm.next_w : w + step;
        if (threadIdx.x < DESC_WORDS && w < w1) dn = reinterpret_cast<const int*>(sh.desc + w)[threadIdx.x];
    }
    __device__ __forceinline__ void store() {
        if (threadIdx.x < DESC_WORDS && w < w1) reinterpret_cast<int*>(&sm.d[cur ^ 1])[threadIdx.x] = dn;
        if (threadIdx.x == 0 && w < w1) take();
    }
    __device__ __forceinline__ void request() {
        const TileDesc& N = sm.d[cur ^ 1];
        requested = w < w1 && N.sid == sm.z.sid;
        if (requested) p2g_request(sm, sh, N, cur ^ 1, buf, dem_map);
    }
};

// The active tiles of the step. Latency: the first descriptor is read beside
// the work count (the guess blockIdx.x is right for one scenario); a tile's
// candidates are requested while the tile before it is summed; the scenario's
// values stay in shared memory across a run of its tiles.
__device__ __forceinline__ void p2g_tiles_body(const Shared& sh, unsigned char* smem_raw, const CUtensorMap* dem_map) {
    P2GTileSmem& sm = *reinterpret_cast<P2GTileSmem*>(smem_raw);
    const int tid = threadIdx.x;
    int dn = 0;
    const bool words = tid < DESC_WORDS;
    if (sh.nscn == 1) load_scn_static(sh, 0, sm.z, tid, P2G_T);
    else if (tid == 0) sm.z.sid = -1;
    for (int k = tid; k < P2C_CHUNKS * P2C_HALVES; k += P2G_T) (&sm.cnt[0][0])[k] = 0;
    if (tid == 0) {
        tma::mbar_init(&sm.dem_bar, 1);
        tma::fence_mbar_init();
    }
    chain_wait<false>();
    if (words && (int)blockIdx.x < sh.work_cap) dn = reinterpret_cast<const int*>(sh.desc + blockIdx.x)[tid];
    if (sh.nscn == 1) load_scn_step(sh, 0, sm.z, tid);
    const int nwork = sh.work_pref[sh.nscn];
    const WorkItems W = work_items(sh, nwork, blockIdx.x, gridDim.x);
    P2GNext<P2GTileSmem> next{sm, sh, dem_map, W.w0, W.w1, W.step, 0, W.w1, 0, many_rounds(sh, nwork) || ordered_by_size(sh, nwork), false, 0};
    if (tid == 0 && next.w < next.w1) next.take();
    if (words && next.w < next.w1 && next.w != (int)blockIdx.x) dn = reinterpret_cast<const int*>(sh.desc + next.w)[tid];
    if (words) reinterpret_cast<int*>(&sm.d[0])[tid] = dn;
    __syncthreads();
    uint32_t dem_phase = 0;  // parity of the terrain window's next completion
    for (; next.w < next.w1; next.cur ^= 1) {
        const TileDesc& D = sm.d[next.cur];
        if (tid == 0) sm.next_w = next.wn;
        if (D.sid != sm.z.sid) {  // uniform: a new scenario in this CTA's run
            __syncthreads();
            load_scn(sh, D.sid, sm.z, tid, P2G_T);
            __syncthreads();
        }
        if (!next.requested) p2g_request(sm, sh, D, next.cur, 0, dem_map);
        if (D.fresh) p2g_clear_fresh(sh, sm.z.s, D, sm.z.y.outs != 0, tid, P2G_T);
        cpa::wait_all();
        float* part = sh.part + (size_t)D.slot * PART_STRIDE;
        const TileOrigin o{cell_i(D.tij) * TILE, cell_j(D.tij) * TILE};
        if (D.total <= sh.split_min) {
            __syncthreads();  // the sums share memory with the row sums of the tile before
            p2g_sparse_tile<P2G_T, false>(sm.sp, sm.ra, sm.rb, sm.dem, &sm.dem_bar, dem_phase, sm.z, D, part, o, next);
        } else if (sm.z.y.outs) {
            p2g_dense_tile<true>(sm, D, part, dem_phase, o, next);
        } else {
            p2g_dense_tile<false>(sm, D, part, dem_phase, o, next);
        }
        dem_phase ^= 1u;
    }
    __syncthreads();
    if (tid == 0) tma::mbar_inval(&sm.dem_bar);  // every copy was waited for; the memory may serve another purpose next
}

__global__ void __launch_bounds__(P2G_T, SLAB_P2G_MIN_BLOCKS) k_p2g_tiles(Shared sh, const __grid_constant__ CUtensorMap dem_map) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    p2g_tiles_body(sh, smem_raw, &dem_map);
}

// ---------------------------------------- P2G over tiles, a thread per cell

// K2 of steps of many tiles, where k_p2g_tiles is bound by how many instructions
// it issues (59 % of the slots, 4 200 warp instructions per tile of 253
// particles): its three threads per cell each read a particle's staged
// quantities and compute its weights along y, and 6 warps run the steps around
// the sums. Here a thread owns a cell and all 9 nodes it reaches (54 sums in
// registers), so
// a particle's quantities and weights are computed once, where they are used,
// and nothing is staged but the order of the candidates by cell. Per pass of up
// to P2X_CAP candidates:
//  1. count them per cell and chunk of 32 (as k_p2g_tiles);
//  2. each thread turns its cell's counts into the chunks' write cursors, each
//     warp the counts of its cells into places in its own list;
//  3. every candidate's offset goes to its place (a stable counting sort); the
//     next pass's or tile's candidates are requested into the other buffer;
//  4. each thread adds its cell's particles in that order.
// Then the 9 x 64 sums go to shared memory and 100 nodes add theirs in (a, b)
// order. The operations and their order are those of k_p2g_tiles.
// 3 000 warp instructions per tile; 8 CTAs of 2 warps per SM at 128 registers.
// 12 M particles: 297 -> 231 us, 2 M: 59.6 -> 50.2, 300 k in a thin flow: 46.2 ->
// 38.4. Fewer tiles are a matter of one tile's latency: 637 k in 1 900 uneven
// tiles 47 us against 38, 12 tiles 10.5 against 10.2. Not better: the next
// particle's values requested a turn ahead (249 us; registers), 9 CTAs (262;
// spills), two rounds of the node sums in the space of one (240).
constexpr int P2X_T = NCELL;                    // threads of a CTA
constexpr int P2X_CAP = NCELL * 9 / 2;          // candidates of one pass: two float4 each are as large as the cells' float4 sums
constexpr int P2X_PER = (P2X_CAP + P2X_T - 1) / P2X_T;
constexpr int P2X_CHUNKS = P2X_CAP / 32;
constexpr int P2X_DEM = ((TILE + 1) * (TILE + 1) + 7) / 8 * 8;  // a tensor copy's destination starts on 128 bytes
#ifndef SLAB_P2X_MIN_BLOCKS
#define SLAB_P2X_MIN_BLOCKS (NCELL == 64 ? 8 : 1)
#endif

struct P2GCellSmem {
    union Buf {
        struct {
            float4 a[P2X_CAP], b[P2X_CAP];  // candidates as they lie in the particle buffer
        } r;
        float4 q4[NSLOT * NCELL];           // sums [row * 3 + b][cell]: m, m h, m vx, m vy
        float q1[NSLOT * NCELL];            // then, on output steps, m vz
        P2GSparseSmem sp;
    };
    alignas(128) float4 dem[2][P2X_DEM];
    Buf buf[2];                                // this pass's candidates and the next one's
    alignas(8) uint64_t dem_bar[2];
    uint16_t cnt[P2X_CHUNKS][NCELL];           // cell counts of a chunk of 32 candidates
    union {
        uint16_t order[NCELL / 32][P2X_CAP];   // the pass's candidates by cell, for each warp's cells
        float2 q2[NSLOT * NCELL];              // sums F, as q4
    };
    uint16_t cbeg[NCELL];                      // first place of a cell in order
    int wtot[NCELL / 32];
    TileDesc d[2];
    int next_w;
    ScnSm z;
};

__device__ __forceinline__ void p2x_request_cands(P2GCellSmem& sm, const TileDesc& D, int base, int buf) {
    const PBuf B = sm.z.cur();
    const int nc = min(D.rpref[9] - base, P2X_CAP);
    for (int k = threadIdx.x; k < nc; k += P2X_T) {
        int r;
        const int src = cand_index(base + k, D, r);
        cpa::copy16(&sm.buf[buf].r.a[k], B.a + src);
        cpa::copy16(&sm.buf[buf].r.b[k], B.b + src);
    }
}

// Requests tile D's first candidates and its terrain window (descriptor slot q).
__device__ __forceinline__ void p2g_request(P2GCellSmem& sm, const Shared& sh, const TileDesc& D, int q, int buf, const CUtensorMap* dem_map) {
    p2x_request_cands(sm, D, 0, buf);
    if (threadIdx.x == 0) {
        tma::fence_proxy_async();
        tma::mbar_arrive_expect_tx(&sm.dem_bar[q], (TILE + 1) * (TILE + 1) * 16);
        tma::tensor_g2s_2d(sm.dem[q], dem_map, 4 * cell_j(D.tij) * TILE, cell_i(D.tij) * TILE, &sm.dem_bar[q]);
    }
}

template <bool OUTS, typename Next>
__device__ __forceinline__ void p2g_cell_tile(P2GCellSmem& sm, const TileDesc& D, float* part, uint32_t dem_phase, TileOrigin o, int& cb,
                                              Next& next) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int q = next.cur;
    Ctl* const ctl = sm.z.s.ctl;
    const int ncand = D.rpref[9];
    const float2 zero = make_float2(0.f, 0.f);
    float2 am[NSLOT], av[NSLOT], aF[NSLOT];
    float az[OUTS ? NSLOT : 1];
#pragma unroll
    for (int k = 0; k < NSLOT; ++k) {
        am[k] = av[k] = aF[k] = zero;
        if (OUTS) az[k] = 0.f;
    }
    const unsigned origin = (unsigned)pack_cell(o.i, o.j);
    int placed = 0;
    int base = 0;
    do {
        const int nc = min(P2X_CAP, ncand - base);
        if (base) {
            cpa::wait_all();
            __syncthreads();  // the pass before is done with its order and counts
        }
        const float4* const ra = sm.buf[cb].r.a;
        const float4* const rb = sm.buf[cb].r.b;
        // 1. count: this thread's candidates as local cell | rank << 16, -1: not in the tile
        int at[P2X_PER];
#pragma unroll
        for (int u = 0; u < P2X_PER; ++u) at[u] = -1;
#pragma unroll
        for (int u = 0; u < P2X_PER; ++u) {
            const int k = tid + u * P2X_T;
            if (k - lane >= nc) break;  // no candidate in the warp
            if (k < nc) {
                // both coordinates at once: a borrow leaves more than TILE - 1 in the lower half
                const unsigned c = (unsigned)__float_as_int(rb[k].z) - origin;
                if ((c & ~((TILE - 1u) << 16 | (TILE - 1u))) == 0u) at[u] = (int)((c >> 16) * TILE + (c & 0xffffu));
                else if (base + k >= D.rpref[4] && base + k < D.rpref[5]) atomicOr(&ctl->err, ERR_MOVE);  // a stayer outside its tile
            }
            const unsigned vm = __ballot_sync(0xffffffffu, at[u] >= 0);
            if (at[u] >= 0) {
                const unsigned peers = __match_any_sync(vm, at[u]);
                const int rank = __popc(peers & ((1u << lane) - 1u));
                if (rank == 0) sm.cnt[warp + u * (P2X_T / 32)][at[u]] = (uint16_t)__popc(peers);
                at[u] |= rank << 16;
            }
        }
        __syncthreads();
        if (base == 0) next.fetch();
        // 2. exclusive prefix over the chunks of the thread's cell, then over the warp's cells
        int num = 0;
#pragma unroll
        for (int c = 0; c < P2X_CHUNKS; ++c) {
            const int x = sm.cnt[c][tid];
            sm.cnt[c][tid] = (uint16_t)num;
            num += x;
        }
        int e = num;
#pragma unroll
        for (int s = 1; s < 32; s <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, e, s);
            if (lane >= s) e += y;
        }
        if (lane == 31) sm.wtot[warp] = e;
        e -= num;
        sm.cbeg[tid] = (uint16_t)e;
        if (base == 0 && !tma::mbar_wait(&sm.dem_bar[q], dem_phase)) atomicOr(&ctl->err, ERR_TIMEOUT);  // the terrain window
        __syncthreads();
        // 3. the candidates' order by cell, as byte offsets
#pragma unroll
        for (int u = 0; u < P2X_PER; ++u)
            if (at[u] >= 0) {
                const int lc = at[u] & 0xffff;
                const int p = (int)sm.cbeg[lc] + (int)sm.cnt[warp + u * (P2X_T / 32)][lc] + (at[u] >> 16);
                sm.order[lc >> 5][p] = (uint16_t)(16 * (tid + u * P2X_T));
            }
        if (tid == 0)
            for (int w = 0; w < NCELL / 32; ++w) placed += sm.wtot[w];
        if (base == 0) next.store();
        __syncthreads();
        for (int k = tid; k < P2X_CHUNKS * NCELL / 2; k += P2X_T) reinterpret_cast<uint32_t*>(&sm.cnt[0][0])[k] = 0;  // for the next pass or tile
        next.buf = cb ^ 1;
        if (base + P2X_CAP >= ncand) next.request();
        else p2x_request_cands(sm, D, base + P2X_CAP, cb ^ 1);
        // 4. the cell's particles over its 9 nodes
        const uint16_t* const ord = sm.order[warp] + e;
        const float4* const dem = sm.dem[q] + (tid / TILE) * (TILE + 1) + tid % TILE;
        const float g = sm.z.s.g, hod = 0.5f * sm.z.s.ood;
        for (int r = 0; r < num; ++r) {
            const int k16 = ord[r];
            const float4* const pa = reinterpret_cast<const float4*>(reinterpret_cast<const char*>(ra) + k16);
            const float4 a = pa[0], b = pa[P2X_CAP];
            const float4 qd = dem[(a.x >= 1.f ? TILE + 1 : 0) + (a.y >= 1.f ? 1 : 0)];
            const float h = b.x, m = b.y;
            const float K = m * g * qd.z * qd.z;
            const float2 pm = make_float2(m, m * h), pv = make_float2(m * a.z, m * a.w), pk = make_float2(-(K * qd.x), -(K * qd.y));
            const float khs = K * h * hod;
            const float2 kh = make_float2(khs, khs);
            float2 wx[3], wy[3];
            float dwx[3], dwy[3];
            spline_y(a.x, wx, dwx);
            spline_y(a.y, wy, dwy);
            float mz = 0.f;
            if (OUTS) {
                int d;
                const int src = cand_index(base + k16 / 16, D, d);
                mz = m * sm.z.cur().vz[src];
            }
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int k = 3 * i + j;
                    const float2 w = f2mul(wx[i], wy[j]);
                    if (w.x > 3e-3f) {  // the reference's weight cut-off (src/simulation.cpp:780)
                        am[k] = f2fma(pm, w, am[k]);
                        av[k] = f2fma(pv, w, av[k]);
                        const float2 gr = f2mul(make_float2(dwx[i], wx[i].x), make_float2(wy[j].x, dwy[j]));
                        aF[k] = f2add(aF[k], f2fma(kh, gr, f2mul(pk, w)));
                        if (OUTS) az[k] = __fmaf_rn(mz, w.x, az[k]);
                    }
                }
        }
        base += P2X_CAP;
        cb ^= 1;
    } while (base < ncand);
    if (tid == 0 && placed != D.total) atomicOr(&ctl->err, ERR_CAPACITY);
    // the cells' sums into the window, over the candidates just summed
    auto& cs = sm.buf[cb ^ 1];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NSLOT; ++k) {
        cs.q4[k * NCELL + tid] = make_float4(am[k].x, am[k].y, av[k].x, av[k].y);
        sm.q2[k * NCELL + tid] = aF[k];
    }
    __syncthreads();
    for (int n = tid; n < NWIN; n += P2X_T) {
        const int i = n / TN, j = n % TN;
        float2 m = zero, v = zero, F = zero;
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const int ci = i - a, cj = j - b;
                if ((unsigned)ci < TILE && (unsigned)cj < TILE) {
                    const int k = (a * 3 + b) * NCELL + ci * TILE + cj;
                    const float4 x = cs.q4[k];
                    m = f2add(m, make_float2(x.x, x.y));
                    v = f2add(v, make_float2(x.z, x.w));
                    F = f2add(F, sm.q2[k]);
                }
            }
        reinterpret_cast<float4*>(part)[n] = make_float4(m.x, m.y, v.x, v.y);
        reinterpret_cast<float2*>(part + 4 * NWIN)[n] = F;
    }
    if (OUTS) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NSLOT; ++k) cs.q1[k * NCELL + tid] = az[k];
        __syncthreads();
        for (int n = tid; n < NWIN; n += P2X_T) {
            const int i = n / TN, j = n % TN;
            float z = 0.f;
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int b = 0; b < 3; ++b) {
                    const int ci = i - a, cj = j - b;
                    if ((unsigned)ci < TILE && (unsigned)cj < TILE) z = __fadd_rn(z, cs.q1[(a * 3 + b) * NCELL + ci * TILE + cj]);
                }
            part[6 * NWIN + n] = z;
        }
    }
}

__device__ __forceinline__ void p2g_cells_body(const Shared& sh, unsigned char* smem_raw, const CUtensorMap* dem_map) {
    P2GCellSmem& sm = *reinterpret_cast<P2GCellSmem*>(smem_raw);
    const int tid = threadIdx.x;
    int dn = 0;
    const bool words = tid < DESC_WORDS;
    if (sh.nscn == 1) load_scn_static(sh, 0, sm.z, tid, P2X_T);
    else if (tid == 0) sm.z.sid = -1;
    for (int k = tid; k < P2X_CHUNKS * NCELL / 2; k += P2X_T) reinterpret_cast<uint32_t*>(&sm.cnt[0][0])[k] = 0;
    if (tid == 0) {
        tma::mbar_init(&sm.dem_bar[0], 1);
        tma::mbar_init(&sm.dem_bar[1], 1);
        tma::fence_mbar_init();
    }
    chain_wait<false>();
    if (words && (int)blockIdx.x < sh.work_cap) dn = reinterpret_cast<const int*>(sh.desc + blockIdx.x)[tid];
    if (sh.nscn == 1) load_scn_step(sh, 0, sm.z, tid);
    const int nwork = sh.work_pref[sh.nscn];
    const WorkItems W = work_items(sh, nwork, blockIdx.x, gridDim.x);
    P2GNext<P2GCellSmem> next{sm, sh, dem_map, W.w0, W.w1, W.step, 0, W.w1, 0, many_rounds(sh, nwork), false, 0};
    if (tid == 0 && next.w < next.w1) next.take();
    if (words && next.w < next.w1 && next.w != (int)blockIdx.x) dn = reinterpret_cast<const int*>(sh.desc + next.w)[tid];
    if (words) reinterpret_cast<int*>(&sm.d[0])[tid] = dn;
    __syncthreads();
    uint32_t phases = 0;  // bit q: parity of the next completion of terrain window q
    int cb = 0;           // buffer of the running pass
    for (; next.w < next.w1; next.cur ^= 1) {
        const int q = next.cur;
        const TileDesc& D = sm.d[q];
        if (tid == 0) sm.next_w = next.wn;
        if (D.sid != sm.z.sid) {  // uniform: a new scenario in this CTA's run
            __syncthreads();
            load_scn(sh, D.sid, sm.z, tid, P2X_T);
            __syncthreads();
        }
        if (!next.requested) p2g_request(sm, sh, D, q, cb, dem_map);
        if (D.fresh) p2g_clear_fresh(sh, sm.z.s, D, sm.z.y.outs != 0, tid, P2X_T);
        cpa::wait_all();
        float* part = sh.part + (size_t)D.slot * PART_STRIDE;
        const TileOrigin o{cell_i(D.tij) * TILE, cell_j(D.tij) * TILE};
        const uint32_t phase = phases >> q & 1u;
        if (D.total <= sh.split_min) {
            next.buf = cb ^ 1;
            p2g_sparse_tile<P2X_T, true>(sm.buf[cb].sp, sm.buf[cb].r.a, sm.buf[cb].r.b, sm.dem[q], &sm.dem_bar[q], phase, sm.z, D, part, o, next);
            cb ^= 1;
        } else if (sm.z.y.outs) {
            p2g_cell_tile<true>(sm, D, part, phase, o, cb, next);
        } else {
            p2g_cell_tile<false>(sm, D, part, phase, o, cb, next);
        }
        phases ^= 1u << q;
    }
    __syncthreads();
    if (tid == 0) {  // every copy was waited for
        tma::mbar_inval(&sm.dem_bar[0]);
        tma::mbar_inval(&sm.dem_bar[1]);
    }
}

__global__ void __launch_bounds__(P2X_T, SLAB_P2X_MIN_BLOCKS) k_p2g_cells(Shared sh, const __grid_constant__ CUtensorMap dem_map) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    p2g_cells_body(sh, smem_raw, &dem_map);
}

// ------------------------------------------------------------ grid update

// computeGridVelocity (src/simulation.cpp:800-875) for node (li, lj) of grid
// tile (gi, gj): velocity and FLIP increment. The P2G sum is the partials of
// the tiles whose window covers the node -- slot[k]: 0 own, 1 -y, 2 -x, 3 -xy
// tile of the grid tile, -1 if it has no particles this step -- added in the
// order own, -x, -y, -xy, so everyone who computes the node gets the same
// bits. blk >= 0: the caller owns the node and writes its maxima, its entry
// of the node block and the output fields, and counts its mass.
__device__ __forceinline__ float4 grid_node(const Shared& sh, const Scn& Z, const SDyn& Y, int gi, int gj, int li, int lj, const int (&slot)[4],
                                            int blk, double& macc, unsigned& nacc) {
    const int i = gi * TILE + li, j = gj * TILE + lj;
    const bool inside = i < sh.Nx && j < sh.Ny;
    // all partials requested before the first is added (a branch per tile made
    // them four rounds of loads); a tile that does not cover the node adds zero
    float4 pq[4];
    float2 pF[4];
    float pz[4];
    constexpr int order[4] = {0, 2, 1, 3};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int k = order[u];
        const bool covers = slot[k] >= 0;
        const float* P = sh.part + (size_t)(covers ? slot[k] : 0) * PART_STRIDE;
        const int pn = covers ? (li + (k >> 1) * TILE) * TN + lj + (k & 1) * TILE : 0;
        pq[u] = covers ? reinterpret_cast<const float4*>(P)[pn] : make_float4(0.f, 0.f, 0.f, 0.f);
        pF[u] = covers ? reinterpret_cast<const float2*>(P + 4 * NWIN)[pn] : make_float2(0.f, 0.f);
        pz[u] = covers && Y.outs ? P[6 * NWIN + pn] : 0.f;
    }
    const size_t bn = (size_t)max(blk, 0) * NCELL + li * TILE + lj;
    const float4 dm = inside ? sh.dem[(int64_t)i * sh.Ny + j] : make_float4(0.f, 0.f, 1.f, 0.f);
    const float hmax0 = blk >= 0 ? sh.hmax[bn] : 0.f, vmax0 = blk >= 0 ? sh.vmax2[bn] : 0.f;
    float2 m2 = make_float2(0.f, 0.f), v2 = m2, F2 = m2;  // m, m h; m v; F
    float qz = 0.f;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        m2 = f2add(m2, make_float2(pq[u].x, pq[u].y));
        v2 = f2add(v2, make_float2(pq[u].z, pq[u].w));
        F2 = f2add(F2, pF[u]);
        qz += pz[u];
    }
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
    float hn = 0.f, vzn = 0.f;
    const float mi = m2.x;
    if (mi > 1e-6f && inside) {
        const float vox = v2.x / mi, voy = v2.y / mi;
        if (Y.outs) vzn = qz / mi;
        hn = m2.y / mi;
        const float dt = Y.dt;
        const float vtx = vox + dt * (F2.x / mi), vty = voy + dt * (F2.y / mi);
        const float vsq = vtx * vtx + vty * vty;
        float nvx = 0.f, nvy = 0.f;
        if (vsq > 1e-16f) {
            const float ct = dm.z;
            const float vz = vtx * dm.x + vty * dm.y;
            const float v3sq = vsq + vz * vz;
            const float v3 = sqrtf(v3sq);
            const float g = Z.g;
            float af;
            if (Z.fric == SLAB_COULOMB) {
                af = Z.mu_c * g * ct;
            } else if (Z.fric == SLAB_VOELLMY) {
                af = Z.mu_v * g * ct + g * v3sq / (Z.xi * hn * ct);
            } else {
                const float I = 5.f * Z.d * v3 / (2.f * hn * ct * ct * sqrtf(g * hn * Z.phi));
                const float muI = Z.mu1 + (Z.mu2 - Z.mu1) / (1.f + Z.I0 / I);
                af = muI * g * ct;
            }
            const float dv = dt * af;
            if (dv < v3) {
                const float fct = 1.f - dv / v3;
                nvx = vtx * fct;
                nvy = vty * fct;
            }
        }
        out = make_float4(nvx, nvy, nvx - vox, nvy - voy);
        if (blk >= 0) {
            sh.hmax[bn] = fmaxf(hmax0, hn);
            sh.vmax2[bn] = fmaxf(vmax0, nvx * nvx + nvy * nvy);
            macc += (double)mi;
            nacc += 1u;
        }
    }
    if (blk >= 0) {
        sh.nv[bn] = out;
        if (Y.outs) {
            sh.oh[bn] = hn;
            sh.om[bn] = inside ? mi : 0.f;
            sh.ovz[bn] = vzn;
            sh.oFx[bn] = inside ? F2.x : 0.f;
            sh.oFy[bn] = inside ? F2.y : 0.f;
        }
    }
    return out;
}

// whether the window of tile k (grid_node) covers node (li, lj) of the grid tile
__device__ __forceinline__ bool covers_node(int k, int li, int lj) { return li + (k >> 1) * TILE < TN && lj + (k & 1) * TILE < TN; }

// Node n of tile D's window, for its G2P. Owner of a node is the first active
// tile, in the order of the sum, whose window covers it.
__device__ __forceinline__ float4 window_node(const Shared& sh, const Scn& Z, const SDyn& Y, const TileDesc& D, int n, double& macc,
                                              unsigned& nacc) {
    const int a = n / TN, b = n % TN, qi = a >= TILE ? 1 : 0, qj = b >= TILE ? 1 : 0, li = a - qi * TILE, lj = b - qj * TILE;
    int slot[4], first = -1;
    constexpr int order[4] = {0, 2, 1, 3};
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        const int k = order[u];
        slot[k] = covers_node(k, li, lj) ? D.nb[(qi - (k >> 1) + 1) * 3 + (qj - (k & 1) + 1)] : -1;
        if (slot[k] >= 0 && first < 0) first = k;
    }
    const int blk = first == 2 * qi + qj ? node_block(sh, Z, D, 2 * qi + qj) : -1;
    return grid_node(sh, Z, Y, cell_i(D.tij) + qi, cell_j(D.tij) + qj, li, lj, slot, blk, macc, nacc);
}

// K3 + K6 as a kernel of its own, for steps of many tiles: a warp per 32 nodes
// of a grid tile -- the particle tiles' own, then those without particles
// (xlist). The kernel is a round of loads after the descriptor's words (which
// the lanes hold, the next item's requested ahead) and the friction law's chain
// of divisions, so what counts is how many warps an SM has in flight. Mass and
// active nodes (diagnostics) are added up over a warp's run of one scenario.
constexpr int GRID_T = 128;

template <int T> __device__ __forceinline__ void grid_body(const Shared& sh) {  // T: threads of a CTA
    __shared__ ScnSm s_scn[T / 32];
    constexpr int PARTS = NCELL / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = T / 32;
    ScnSm& zs = s_scn[warp];
    const int gw = (int)blockIdx.x * nwarp + warp, gn = (int)gridDim.x * nwarp;
    if (sh.nscn == 1) load_scn_static(sh, 0, zs, lane, 32);
    chain_wait<false>();
    // lane's word of a descriptor: nb, blk4, then tij, sid
    const int word = lane < 9 ? 28 + lane : (lane < 13 ? 24 + lane - 9 : (lane == 13 ? 37 : 3));
    int v = 0, q_nxt = 0, csid = -1;
    if (sh.nscn == 1) {
        if (gw < sh.work_cap * PARTS) v = reinterpret_cast<const int*>(sh.desc + gw / PARTS)[word];  // a guess until the count is known
        load_scn_step(sh, 0, zs, lane);
        csid = 0;
        __syncwarp();
    }
    const int ntile = sh.work_pref[sh.nscn];
    const WorkItems W = work_items(sh, (ntile + sh.lists[LIST_X]) * PARTS, gw, gn);
    const int w0 = W.w0, w1 = W.w1, step = W.step;
    auto request = [&](int it) {
        int w = it / PARTS;
        q_nxt = 0;
        if (w >= ntile) {
            const int e = sh.xlist[w - ntile];
            w = e >> 2;
            q_nxt = e & 3;
        }
        v = reinterpret_cast<const int*>(sh.desc + w)[word];
    };
    if (w0 >= w1) return;  // warps run alone: no block barrier below
    if (sh.nscn != 1 || w0 / PARTS >= ntile) request(w0);
    double macc = 0.0;
    unsigned nacc = 0;
    auto flush = [&] {
        nacc = __reduce_add_sync(0xffffffffu, nacc);
        for (int o = 16; o > 0; o >>= 1) macc += __shfl_xor_sync(0xffffffffu, macc, o);
        if (lane == 0) {
            if (macc != 0.0) atomicAdd(&zs.s.cnt->grid_mass, macc);
            if (nacc) atomicAdd(&zs.s.ctl->node_steps, (unsigned long long)nacc);
        }
        macc = 0.0;
        nacc = 0;
    };
    for (int w = w0; w < w1; w += step) {
        const int cur = v, q = q_nxt, sid = __shfl_sync(0xffffffffu, cur, 14), tij = __shfl_sync(0xffffffffu, cur, 13);
        if (w + step < w1) request(w + step);
        if (sid != csid) {  // a new scenario in this warp's run
            if (csid >= 0) flush();
            csid = sid;
            __syncwarp();
            load_scn(sh, csid, zs, lane, 32);
            __syncwarp();
        }
        if (w / PARTS < ntile && w % PARTS == 0 && cur == BLK_LATER && lane >= 9 && lane < 13)  // named now, for G2P
            sh.desc[w / PARTS].blk4[lane - 9] = zs.s.blk_of[(cell_i(tij) + ((lane - 9) >> 1)) * sh.TY + cell_j(tij) + ((lane - 9) & 1)];
        const int c = (w % PARTS) * 32 + lane, li = c / TILE, lj = c % TILE;
        const int qi = q >> 1, qj = q & 1, gi = cell_i(tij) + qi, gj = cell_j(tij) + qj;
        int blk = __shfl_sync(0xffffffffu, cur, 9 + q);
        if (blk == BLK_LATER) blk = zs.s.blk_of[gi * sh.TY + gj];
        int slot[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int s = __shfl_sync(0xffffffffu, cur, (qi - (k >> 1) + 1) * 3 + (qj - (k & 1) + 1));
            slot[k] = covers_node(k, li, lj) ? s : -1;
        }
        if (blk >= 0) grid_node(sh, zs.s, zs.y, gi, gj, li, lj, slot, blk, macc, nacc);
    }
    flush();
}

#ifndef SLAB_GRID_MIN_BLOCKS
#define SLAB_GRID_MIN_BLOCKS 8
#endif
__global__ void __launch_bounds__(GRID_T, SLAB_GRID_MIN_BLOCKS) k_grid(Shared sh) { grid_body<GRID_T>(sh); }

// -------------------------------------------------------------------- G2P

__device__ __forceinline__ int dir_of(int ib, int jb, int ti, int tj) {
    int di = (ib >= 0 ? ib / TILE : -1) - ti, dj = (jb >= 0 ? jb / TILE : -1) - tj;
    if (di < -1 || di > 1 || dj < -1 || dj > 1) return -1;
    return (di + 1) * 3 + (dj + 1);
}

constexpr int G2P_T = 2 * NCELL;  // threads of a CTA with the grid update
#ifndef SLAB_G2P_MIN_BLOCKS
#define SLAB_G2P_MIN_BLOCKS (NCELL == 64 ? 32 : 8)
#endif
#ifndef SLAB_G2P_FUSED_MIN_BLOCKS
#define SLAB_G2P_FUSED_MIN_BLOCKS (NCELL == 64 ? 7 : 1)
#endif

// puts tile tt on the next step's active list, once; its place there is also
// the place of its partial window
__device__ __forceinline__ void g2p_activate(const ScnSm& z, int tt) {
    const int seq1 = z.y.seq + 1;
    if (atomicMax(&z.s.act[tt].x, seq1) < seq1) {
        const int kk = atomicAdd(&z.s.cnt->act_count[seq1 & 1], 1);
        z.s.act[tt].y = kk;
        if (kk < z.s.act_cap) z.s.act_list[seq1 & 1][kk] = tt;
        else atomicOr(&z.s.ctl->err, ERR_CAPACITY);
    }
}

// What a thread gathers over a run of tiles of one scenario: its particles'
// largest |v|^2, and mass and number of the active nodes it owns (the FP64 grid
// mass and the node count are diagnostics).
struct G2PRun {
    float vmax2 = 0.f;
    unsigned nodes = 0;
    double mass = 0.0;
    // into the scenario's control block: one atomic of each per warp, without
    // waiting for an answer (speeds squared are >= 0, so their bit patterns
    // order like the values)
    __device__ __forceinline__ void flush(const ScnSm& z) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(vmax2));
        nodes = __reduce_add_sync(0xffffffffu, nodes);
        for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
        if ((threadIdx.x & 31) == 0) {
            const double v = (double)__uint_as_float(m);
            if (m) atomicMax(reinterpret_cast<unsigned long long*>(&z.s.ctl->vmax2_acc), (unsigned long long)__double_as_longlong(v));
            if (nodes) atomicAdd(&z.s.ctl->node_steps, (unsigned long long)nodes);
            if (mass != 0.0) atomicAdd(&z.s.cnt->grid_mass, mass);
        }
        vmax2 = 0.f;
        nodes = 0;
        mass = 0.0;
    }
};

template <int T> struct G2PSmem {
    float4 nv[NWIN];
    float4 dem[(TILE + 1) * (TILE + 1)];
    int front, back;
    alignas(16) int wcnt[2][(T / 32 + 3) / 4 * 4];  // stayers | movers << 16 of each warp of a chunk (double buffered)
    int dcnt[9];
    TileDesc d;
    ScnSm z;
    double red[4][T / 32];
};

// one candidate of a tile: its two words, and whether it exists
struct G2PCand {
    float4 a, b;
    bool there;
};

__device__ __forceinline__ G2PCand load_g2p_cand(const TileDesc& D, const PBuf& B, int k, int ncand) {
    G2PCand q;
    q.there = k < ncand;
    q.a = make_float4(1.f, 1.f, 0.f, 0.f);
    q.b = make_float4(0.f, 0.f, 0.f, 0.f);
    if (q.there) {
        int r;
        const int src = cand_index(k, D, r);
        q.a = B.a[src];
        q.b = B.b[src];
    }
    return q;
}

// G2P's barrier: of the block, or of its only warp
template <int T> __device__ __forceinline__ void g2p_sync() {
    if (T == 32) __syncwarp();
    else __syncthreads();
}

// K4, one tile per CTA of T threads. Two kernels:
//
// k_g2p_fused (T = 128), for steps of few tiles: K3 and K6 first, the grid
// update of the tile's node window into shared memory (window_node). 100 nodes
// for 64 cells, nodes near an edge computed by up to 4 tiles, but no kernel of
// its own between P2G and G2P: per step 22 -> 18.5 us at 1 600 particles, 30 ->
// 27 at 180 k (734 tiles), 76 -> 63 at 637 k (1 900 tiles); at 2 M particles
// (8 000 tiles) the pass through memory is the cheaper one (Engine32::fused).
//
// k_g2p (T = 32), for steps of many: the window comes from the node blocks. One
// warp per CTA, because the rounds of a tile (descriptor, candidates and window,
// chunks, records) depend on one another and all warps of a larger CTA wait in
// the same place: with 128 / 96 / 64 / 32 threads and the same number of warps
// per SM, 12 M particles take 214 / 205 / 187 / 172 us, 2 M 44 / 42 / 40 / 37
// and 300 k in a thin flow 27 / 25 / 23 / 20. The stayers' and movers' places
// then need no block prefix either. (Several such warps in one CTA of 128 lose
// it again: the tile number is no longer the same in the whole CTA, so
// addresses that were uniform take registers, 250 us with the spills.)
//
// G2P itself (src/simulation.cpp:877-940): FLIP/PIC blend,
// advection, depth update, and the write of the particle into the tile's
// segment of the next buffer -- stayers from the front, particles that moved
// to a neighbour tile from the back, with per-direction counts. The max of
// |v|^2 and the particle bounding box feed the next step's dt and remesh box
// (K5). A particle is two 16-byte loads and two 16-byte stores; a thread
// holds its candidate of this chunk and of the next in registers, so the
// loads of a chunk go out with the node window's or while the chunk before it
// is computed. The scenario's values stay in shared memory across a run of its
// tiles, the next tile's descriptor is requested while this one runs, and a
// tile's neighbour activations (two dependent atomics) are issued while the
// next tile's loads are in flight.
template <int T, bool FUSED> __device__ __forceinline__ void g2p_body(const Shared& sh, const double* __restrict__ z64, G2PSmem<T>& sm) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int PER = (DESC_WORDS + T - 1) / T;  // descriptor words per thread
    int dn[PER] = {};
    auto load_words = [&](int w) {
#pragma unroll
        for (int u = 0; u < PER; ++u)
            if (tid + u * T < DESC_WORDS) dn[u] = reinterpret_cast<const int*>(sh.desc + w)[tid + u * T];
    };
    if (sh.nscn == 1) load_scn_static(sh, 0, sm.z, tid, T);
    else if (tid == 0) sm.z.sid = -1;
    chain_wait<true>();
    if ((int)blockIdx.x < sh.work_cap) load_words(blockIdx.x);
    if (sh.nscn == 1) load_scn_step(sh, 0, sm.z, tid);
    const WorkItems W = work_items(sh, sh.work_pref[sh.nscn], blockIdx.x, gridDim.x);
    const int w0 = W.w0, w1 = W.w1, step = W.step;
    if (w0 < w1 && w0 != (int)blockIdx.x) load_words(w0);
    int pend_tt = -1;    // threads 0..8: neighbour tile the previous tile activates
    G2PRun run;
    for (int w = w0; w < w1; w += step) {
        g2p_sync<T>();  // the tile before is done with the shared memory
#pragma unroll
        for (int u = 0; u < PER; ++u)
            if (tid + u * T < DESC_WORDS) reinterpret_cast<int*>(&sm.d)[tid + u * T] = dn[u];
        if (tid < 9) sm.dcnt[tid] = 0;
        g2p_sync<T>();
        if (w + step < w1) load_words(w + step);
        if (sm.d.sid != sm.z.sid) {  // uniform: a new scenario in this CTA's run
            if (pend_tt >= 0) g2p_activate(sm.z, pend_tt);
            pend_tt = -1;
            run.flush(sm.z);  // (nothing yet before the first)
            g2p_sync<T>();
            load_scn(sh, sm.d.sid, sm.z, tid, T);
            g2p_sync<T>();
        }
        const ScnSm& Z = sm.z;
        const TileDesc& D = sm.d;
        Ctl* c = Z.s.ctl;
        const int t = D.t, ti = cell_i(D.tij), tj = cell_j(D.tij);
        const bool outs = Z.y.outs != 0;
        const bool need_vz = Z.y.need_vz != 0;
        const int ncand = D.rpref[9];
        // the first candidates, the node window and the terrain in one round
        // (requested while the tile before ran, they took as long: the kernel is
        // bound by instruction issue, and the second window's shared memory and
        // the longer-lived registers cost what the wait did)
        SLAB_PHASE_BEGIN;
        G2PCand nxt = load_g2p_cand(D, Z.cur(), tid, ncand);
        if (need_vz) {
            for (int k = tid; k < (TILE + 1) * (TILE + 1); k += T) {
                const int i = ti * TILE + k / (TILE + 1), j = tj * TILE + k % (TILE + 1);
                if (i < sh.Nx && j < sh.Ny) cpa::copy16(&sm.dem[k], sh.dem + (int64_t)i * sh.Ny + j);
                else sm.dem[k] = make_float4(0.f, 0.f, 1.f, 0.f);
            }
        }
        if (pend_tt >= 0) g2p_activate(Z, pend_tt);  // the previous tile's, while the loads above are in flight
        pend_tt = -1;
        for (int k = tid; k < NWIN; k += T) {
            if constexpr (FUSED) {
                sm.nv[k] = window_node(sh, Z.s, Z.y, D, k, run.mass, run.nodes);
            } else {
                // a part of the window whose grid tile has no block (past the terrain edge) is zero
                const int a = k / TN, b = k % TN;
                const int blk = ti * TILE + a < sh.Nx && tj * TILE + b < sh.Ny ? D.blk4[(a >= TILE ? 2 : 0) + (b >= TILE ? 1 : 0)] : -1;
                if (blk >= 0) cpa::copy16(&sm.nv[k], &sh.nv[(size_t)blk * NCELL + (a % TILE) * TILE + (b % TILE)]);
                else sm.nv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        SLAB_PHASE_MARK(8);
        cpa::wait_all();
        g2p_sync<T>();
        SLAB_PHASE_MARK(9);
        const int total = D.total, base = D.nxt_off;
        const bool edge = ti < Z.y.in_i0 || ti > Z.y.in_i1 || tj < Z.y.in_j0 || tj > Z.y.in_j1;  // uniform: may change the particle box
        const bool inner = (ti + 1) * TILE + 1 <= sh.Nx - 1 && (tj + 1) * TILE + 1 <= sh.Ny - 1;  // uniform
        double mnx = INFINITY, mxx = 0.0, mny = INFINITY, mxy = 0.0;
        int front = 0, back = 0;  // stayers / movers placed so far (same in every thread)
        for (int k0 = 0; k0 < ncand; k0 += T) {
            // this chunk's candidate, and the next chunk's requested before this one is computed
            const G2PCand q = nxt;
            if (k0 + T < ncand) nxt = load_g2p_cand(D, Z.cur(), k0 + T + tid, ncand);
            const int32_t cell = __float_as_int(q.b.z);
            const int ci = cell_i(cell) - ti * TILE, cj = cell_j(cell) - tj * TILE;
            const bool valid = q.there && (unsigned)ci < TILE && (unsigned)cj < TILE;
            int d = 4, ib = 0, jb = 0;
            float2 fn = make_float2(1.f, 1.f), vn = make_float2(0.f, 0.f);
            float hn = 0.f, vzp = 0.f;
            double zp = 0.0;
            const float dt = Z.y.dt, dt_ood = Z.y.dt_ood;
            if (valid) {
                const float2 f = make_float2(q.a.x, q.a.y);
                const float2 v = make_float2(q.a.z, q.a.w);
                const float h = q.b.x;
                float wx[3], wy[3], dwx[3], dwy[3];
                bspline3(f.x, wx, dwx);
                bspline3(f.y, wy, dwy);
                float2 pic = make_float2(0.f, 0.f), fl = make_float2(0.f, 0.f);
                float div = 0.f;
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int b = 0; b < 3; ++b) {
                        const float wgt = wx[a] * wy[b];
                        const float4 nv = sm.nv[(ci + a) * TN + (cj + b)];
                        const float2 w2 = make_float2(wgt, wgt);
                        pic = f2fma(make_float2(nv.x, nv.y), w2, pic);
                        fl = f2fma(make_float2(nv.z, nv.w), w2, fl);
                        div += (dwx[a] * wy[b]) * nv.x + (dwy[b] * wx[a]) * nv.y;
                    }
                div *= Z.s.ood;
                const float fr = Z.s.fr;
                vn = make_float2(fr * (v.x + fl.x) + (1.f - fr) * pic.x, fr * (v.y + fl.y) + (1.f - fr) * pic.y);
                hn = h / (1.f + dt * div);
                if (need_vz) {
                    const float4 dm = sm.dem[(ci + (f.x >= 1.f ? 1 : 0)) * (TILE + 1) + (cj + (f.y >= 1.f ? 1 : 0))];
                    vzp = vn.x * dm.x + vn.y * dm.y;
                }
                if (outs) {
                    const int i0 = cell_i(cell), j0 = cell_j(cell);
#pragma unroll
                    for (int a = 0; a < 3; ++a)
#pragma unroll
                        for (int b = 0; b < 3; ++b) zp += (double)(wx[a] * wy[b]) * z64[(int64_t)(i0 + a) * sh.Ny + (j0 + b)];
                }
                // advection with the PIC velocity and re-anchoring of the offset
                const float ux = f.x + dt_ood * pic.x, uy = f.y + dt_ood * pic.y;
                const int ki = (int)floorf(ux - 0.5f), kj = (int)floorf(uy - 0.5f);
                ib = cell_i(cell) + ki;
                jb = cell_j(cell) + kj;
                fn = make_float2(ux - (float)ki, uy - (float)kj);
                // most particles stay in a tile whose stencils all lie inside the
                // terrain: nothing else to check
                if (!inner || (unsigned)(ci + ki) >= TILE || (unsigned)(cj + kj) >= TILE) {
                d = dir_of(ib, jb, ti, tj);
                if (d < 0) {
                    atomicOr(&c->err, ERR_MOVE);
                    d = 4;
                }
                if (ib < 0 || jb < 0 || ib + 2 > sh.Nx - 1 || jb + 2 > sh.Ny - 1) {
                    atomicOr(&c->err, ERR_DOMAIN);
                    ib = min(max(ib, 0), sh.Nx - 3);
                    jb = min(max(jb, 0), sh.Ny - 3);
                    d = dir_of(ib, jb, ti, tj);
                    if (d < 0) d = 4;
                }
                }
                if (edge) {
                    const double px = ((double)ib + (double)fn.x) * sh.dx, py = ((double)jb + (double)fn.y) * sh.dx;
                    mnx = fmin(mnx, px);
                    mxx = fmax(mxx, px);
                    mny = fmin(mny, py);
                    mxy = fmax(mxy, py);
                }
                run.vmax2 = fmaxf(run.vmax2, vn.x * vn.x + vn.y * vn.y);
                // 0 unless one of them is infinite or NaN
                const float bad = fmaf(vn.x, 0.f, fmaf(vn.y, 0.f, fmaf(hn, 0.f, fmaf(fn.x, 0.f, fn.y * 0.f))));
                if (bad != 0.f) atomicOr(&c->err, ERR_NONFINITE);
            }
            // stayers to the front of the segment, movers to the back, both in
            // candidate order (a block prefix of the warps' counts), so the next
            // step sees the tile's particles in an order fixed by the data
            const bool stay = valid && d == 4, move = valid && d != 4;
            const unsigned ms = __ballot_sync(0xffffffffu, stay), mm = __ballot_sync(0xffffffffu, move);
            int before = 0, all = __popc(ms) | __popc(mm) << 16;  // stayers | movers << 16: of the warps before this one, of all
            if (T > 32) {
                const int par = (k0 / T) & 1;
                if (lane == 0) sm.wcnt[par][warp] = all;
                g2p_sync<T>();
                all = 0;
#pragma unroll
                for (int q_ = 0; q_ < T / 32; ++q_) {
                    const int a = sm.wcnt[par][q_];
                    if (q_ < warp) before += a;
                    all += a;
                }
            }
            const int bs = front + (before & 0xffff), bm = back + (before >> 16);
            front += all & 0xffff;
            back += all >> 16;
            const unsigned lt = (1u << lane) - 1u;
            if (valid) {
                int pos;
                if (stay) {
                    pos = base + bs + __popc(ms & lt);
                } else {
                    pos = base + total - 1 - (bm + __popc(mm & lt));
                    atomicAdd(&sm.dcnt[d], 1);
                }
                const PBuf O = Z.next();
                O.a[pos] = make_float4(fn.x, fn.y, vn.x, vn.y);
                O.b[pos] = make_float4(hn, q.b.y, __int_as_float(pack_cell(ib, jb)), q.b.w);
                if (need_vz) O.vz[pos] = vzp;
                if (outs) O.z[pos] = (float)zp;
            }
        }
        SLAB_PHASE_MARK(10);
        if (tid == 0) {
            sm.front = front;
            sm.back = back;
        }
        g2p_sync<T>();
        if (tid < 9) {
            int32_t* G = Z.s.grp[(Z.y.seq & 1) ^ 1] + (size_t)t * GRP_STRIDE;
            const int cnt = tid == 4 ? sm.front : sm.dcnt[tid];
            G[3 + tid] = cnt;
            if (tid == 0) {
                G[0] = base;
                G[1] = base + sm.front;
                G[2] = base + sm.front + sm.back;
                G[GRP_STAMP] = Z.y.seq + 1;
                if (sm.front + sm.back != total) atomicOr(&c->err, ERR_CAPACITY);
            }
            if (cnt) pend_tt = (ti + dir_i(tid)) * sh.TY + (tj + dir_j(tid));
        }
        if (edge) {  // the tile's particle box into the scenario's control block
            mnx = warp_min(mnx);
            mxx = warp_max(mxx);
            mny = warp_min(mny);
            mxy = warp_max(mxy);
            if (lane == 0) {
                sm.red[0][warp] = mnx;
                sm.red[1][warp] = mxx;
                sm.red[2][warp] = mny;
                sm.red[3][warp] = mxy;
            }
            g2p_sync<T>();
            if (tid == 0 && total > 0) {
                for (int k = 1; k < T / 32; ++k) {
                    mnx = fmin(mnx, sm.red[0][k]);
                    mxx = fmax(mxx, sm.red[1][k]);
                    mny = fmin(mny, sm.red[2][k]);
                    mxy = fmax(mxy, sm.red[3][k]);
                }
                atomicMin(reinterpret_cast<unsigned long long*>(&c->pos_acc[0]), (unsigned long long)__double_as_longlong(mnx));
                atomicMax(reinterpret_cast<unsigned long long*>(&c->pos_acc[1]), (unsigned long long)__double_as_longlong(mxx));
                atomicMin(reinterpret_cast<unsigned long long*>(&c->pos_acc[2]), (unsigned long long)__double_as_longlong(mny));
                atomicMax(reinterpret_cast<unsigned long long*>(&c->pos_acc[3]), (unsigned long long)__double_as_longlong(mxy));
            }
        }
        SLAB_PHASE_MARK(11);
        SLAB_PHASE_TILE_G2P();
    }
    run.flush(sm.z);
    if (pend_tt >= 0) g2p_activate(sm.z, pend_tt);  // the last tile's
}

__global__ void __launch_bounds__(G2P_T, SLAB_G2P_FUSED_MIN_BLOCKS) k_g2p_fused(Shared sh, const double* __restrict__ z64) {
    __shared__ G2PSmem<G2P_T> sm;
    g2p_body<G2P_T, true>(sh, z64, sm);
}

__global__ void __launch_bounds__(32, SLAB_G2P_MIN_BLOCKS) k_g2p(Shared sh, const double* __restrict__ z64) {
    __shared__ G2PSmem<32> sm;
    g2p_body<32, false>(sh, z64, sm);
}

// K5: end of the step for every running scenario (the per-step reductions
// of G2P into dt, time and the remesh box), then the next step's dt, stop
// rules and work list. One CTA, after G2P.
__global__ void __launch_bounds__(CTL_THREADS) k_end(Shared sh) {
    chain_wait<true>();
    control_scenarios(sh, CTL_END);
}

// ------------------------------------------------------- persistent steps

// Barrier of the persistent step kernel: one cooperative launch, every CTA
// resident. Thread 0 of each CTA arrives on the counter; the last arrival
// resets it and advances the generation; the others wait for the generation
// to change -- at most `limit` clock cycles, after which the CTA records
// ERR_TIMEOUT in every scenario's control block and leaves the kernel. A CTA
// that left never arrives again, so every later wait of the launch runs out
// too: the launch always ends, and no phase runs on inputs that a phase
// before it did not finish (a phase starts only when every CTA arrived).
// The engine is then dead: its later persistent launches return at once.
struct GridBar {
    unsigned count;
    unsigned gen;
    int dead;  // a wait ran out: this engine's step state is incomplete, later launches do nothing
    int pad_;
};

__device__ __forceinline__ bool grid_sync(const Shared& sh, GridBar* bar, long long limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        volatile unsigned* vgen = &bar->gen;
        const unsigned g = *vgen;
        __threadfence();
        if (atomicAdd(&bar->count, 1u) == gridDim.x - 1) {
            *reinterpret_cast<volatile unsigned*>(&bar->count) = 0u;
            __threadfence();
            atomicAdd(&bar->gen, 1u);
        } else {
            const long long t0 = clock64();
            while (*vgen == g) {
                if (clock64() - t0 > limit) {
                    ok = 0;
                    break;
                }
                __nanosleep(64);
            }
            if (!ok) {
                atomicExch(&bar->dead, 1);
                for (int s = 0; s < sh.nscn; ++s) atomicOr(&sh.scn[s].ctl->err, ERR_TIMEOUT);
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Shared memory of the persistent kernels: the largest phase's, reused by
// every phase (each phase initialises what it reads).
constexpr size_t PERSIST_SMEM = sizeof(P2GTileSmem) > sizeof(G2PSmem<P2G_T>) ? sizeof(P2GTileSmem) : sizeof(G2PSmem<P2G_T>);
constexpr size_t PERSIST_MANY_SMEM = sizeof(P2GCellSmem) > sizeof(G2PSmem<P2X_T>) ? sizeof(P2GCellSmem) : sizeof(G2PSmem<P2X_T>);

// Up to nsteps whole steps (K1 tile bookkeeping, K2 P2G, K3 grid update and
// K4 G2P, K5 end of step) in one launch, the phases separated by grid_sync
// instead of kernel boundaries. The same phase bodies as the separate kernels,
// over the same work lists and in the same per-tile order, so a step gives
// the same bits either way. The launch ends early once no scenario has work
// (every one stopped at its frame, step budget or end).
// Two kernels by the same rule as the separate ones (Engine32::fused), each with
// the CTAs of its P2G. One register budget serves all phases of a kernel:
//   k_persist       4 CTAs per SM, 80 registers (100 bytes of spill stores). us per
//                   step at 878 / 56 k / 198 k particles 25.6 / 28 / 40; 5 CTAs 28 /
//                   31 / 44, 6 CTAs (484 bytes) 30 / 34 / 50, 3 CTAs 24.5 / 27.5 / 45.
//   k_persist_many  8 CTAs per SM, 128 registers (52 bytes). 2 M particles 154 us
//                   per step, 256 scenarios over 6 000 steps 19.8 s; 9 CTAs (268
//                   bytes) 170 and 22.1; these steps by k_persist 173 and 23.1.
template <bool MANY>
__device__ __forceinline__ void persist_steps(const Shared& sh, const double* __restrict__ z64, int nsteps, long long limit, GridBar* bar,
                                              const CUtensorMap* dem_map) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    // after a launch whose waits ran out, the tile bookkeeping of the step it
    // left is half done: no phase may run on it again
    if (*reinterpret_cast<volatile const int*>(&bar->dead)) return;
    for (int s = 0; s < nsteps; ++s) {
        prep_body(sh);
        if (!grid_sync(sh, bar, limit)) return;
        if constexpr (MANY) {
            p2g_cells_body(sh, smem_raw, dem_map);
            if (!grid_sync(sh, bar, limit)) return;
            grid_body<P2X_T>(sh);
            if (!grid_sync(sh, bar, limit)) return;
            g2p_body<P2X_T, false>(sh, z64, *reinterpret_cast<G2PSmem<P2X_T>*>(smem_raw));
        } else {
            p2g_tiles_body(sh, smem_raw, dem_map);
            if (!grid_sync(sh, bar, limit)) return;
            g2p_body<P2G_T, true>(sh, z64, *reinterpret_cast<G2PSmem<P2G_T>*>(smem_raw));
        }
        if (!grid_sync(sh, bar, limit)) return;
        if (blockIdx.x == 0) control_scenarios(sh, CTL_END);
        if (!grid_sync(sh, bar, limit)) return;
        if (*reinterpret_cast<volatile const int*>(sh.work_pref + sh.nscn) == 0) break;  // the same value in every CTA
    }
}

#ifndef SLAB_PERSIST_MIN_BLOCKS
#define SLAB_PERSIST_MIN_BLOCKS (NCELL == 64 ? 4 : 1)
#endif
__global__ void __launch_bounds__(P2G_T, SLAB_PERSIST_MIN_BLOCKS) k_persist(Shared sh, const double* __restrict__ z64, int nsteps, long long limit,
                                                                            GridBar* bar, const __grid_constant__ CUtensorMap dem_map) {
    persist_steps<false>(sh, z64, nsteps, limit, bar, &dem_map);
}
#ifndef SLAB_PERSIST_MANY_MIN_BLOCKS
#define SLAB_PERSIST_MANY_MIN_BLOCKS SLAB_P2X_MIN_BLOCKS
#endif
__global__ void __launch_bounds__(P2X_T, SLAB_PERSIST_MANY_MIN_BLOCKS)
    k_persist_many(Shared sh, const double* __restrict__ z64, int nsteps, long long limit, GridBar* bar, const __grid_constant__ CUtensorMap dem_map) {
    persist_steps<true>(sh, z64, nsteps, limit, bar, &dem_map);
}

// Particle z and vz at the current positions (for downloads between output
// frames, where the step loop does not keep them): vz = v . grad z of the
// containing cell, z from the quadratic stencil of FP64 terrain heights.
__global__ void k_refresh_vz_z(Shared sh, PBuf B, int Np, const double* __restrict__ z64) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < Np; q += gridDim.x * blockDim.x) {
        const int32_t cell = p_cell(B, q);
        const float4 pa = B.a[q];
        const float2 f = make_float2(pa.x, pa.y), v = make_float2(pa.z, pa.w);
        const int i0 = cell_i(cell), j0 = cell_j(cell);
        float wx[3], wy[3], dwx[3], dwy[3];
        bspline3(f.x, wx, dwx);
        bspline3(f.y, wy, dwy);
        const float4 dm = sh.dem[(int64_t)(i0 + (f.x >= 1.f ? 1 : 0)) * sh.Ny + (j0 + (f.y >= 1.f ? 1 : 0))];
        double zp = 0.0;
        for (int a = 0; a < 3; ++a)
            for (int b = 0; b < 3; ++b) zp += (double)(wx[a] * wy[b]) * z64[(int64_t)(i0 + a) * sh.Ny + (j0 + b)];
        B.vz[q] = v.x * dm.x + v.y * dm.y;
        B.z[q] = (float)zp;
    }
}

}  // namespace k32
}  // namespace slab
