// Particle-to-grid scatters by warps: runs of particles that share a stencil base are summed over
// the warp and the sums go straight to the L2 atomics.
//
// A warp splits its 32 particles into runs of equal stencil base. Each particle's own thread stores
// its 27 node weights (w_x w_y) w_z, as the reference rounds them, and its values in the warp's
// record in shared memory; the run is then summed over its particles and every node receives one
// atomic per run (one 16-byte vector atomic for momentum and mass). The transport fields, float64, go to the
// grid that way; the float32 momentum is summed over the block first (below).
//
// What bounds it, and why no warps share a tile: a shared-memory tile over the block's node box that every
// warp adds to needs three block barriers, the zeroing and flushing of the tile, and shared float atomics,
// which are compare-and-swap loops with bank conflicts; it held the LSU data pipe at 73% (momentum)
// and 71% (transport) of its peak. A run
// of ~18 particles already divides the atomics by 18, and L2 takes the rest without waiting. 1M
// particles, 128^3 grid, 40 particles a cell, fused P2G kernel: 102 us with the tile, 87 us with the
// same kernel writing straight to L2; transport scatter 68.5 against 62.1 us, 55 with the float64
// tensor cores; in tet order P2G of 41k particles 37 against 16 us, 8.6 with grouped lanes.
#pragma once

#include <climits>

#include "bk_device.cuh"

namespace bk {

constexpr unsigned kWarp = 0xffffffffu;

// The 128-byte lines of plane arrays that a warp's 32 particles read, requested into L2 by one
// instruction per 32 lines (lane c takes plane c) before the values are needed: the loads of a
// particle kernel fall into phases (position, node gather, state) and each phase otherwise waits for
// DRAM again.
BK_DEV void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Up to 32 planes of three arrays.
BK_DEV void prefetch_planes(int64_t i, int64_t n, int64_t pitch, const float* a, int na, const float* b, int nb,
                            const float* c, int nc) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = i - lane;
    if (w0 >= n || lane >= na + nb + nc) return;
    prefetch_l2((lane < na ? a + lane * pitch : lane < na + nb ? b + (lane - na) * pitch : c + (lane - na - nb) * pitch) + w0);
}

// ------------------------------------------------------------- node gathers
// sum_j w_j v_j and the moments sum_j w_j v_j o_jc over the stencil's nodes, with the offsets o_j in
// {0, 1, 2} known at compile time: what G2P forms v and C of (C_rc = 4/dx (M_rc - l_c S_r)).
BK_DEV void gather_velocity(const Stencil& st, const float4* node_v, int R32, float* nv, float* mo) {
#pragma unroll
    for (int r = 0; r < 3; ++r) nv[r] = 0.f;
#pragma unroll
    for (int e = 0; e < 9; ++e) mo[e] = 0.f;
    const float4* vbase = node_v + node_index(st.b[0], st.b[1], st.b[2], R32);
    const int64_t R = R32;
#pragma unroll
    for (int ox = 0; ox < 3; ++ox)
#pragma unroll
        for (int oy = 0; oy < 3; ++oy) {
            const float wxy = st.w[0][ox] * st.w[1][oy];
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) {
                float w = wxy * st.w[2][oz];
                float4 u = vbase[(ox * R + oy) * R + oz];
                float wu[3] = {w * u.x, w * u.y, w * u.z};
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    nv[r] += wu[r];
                    if (ox) mo[3 * r + 0] += (float)ox * wu[r];
                    if (oy) mo[3 * r + 1] += (float)oy * wu[r];
                    if (oz) mo[3 * r + 2] += (float)oz * wu[r];
                }
            }
        }
}

// sum_j w_j (dT, dW/W)_j of the diffused node fields in float64, with the weights as the scatter rounds them
// (put_weights): the heat and water that leave one particle then arrive at others to the last float64 place.
// Summed axis by axis from unrounded weights (a conversion and a product less a node) the energy of an
// insulated 40k cube drifted by 5.6e-11 of the heat moved in 100 substeps, with these by 2e-14.
BK_DEV void gather_scalars(const Stencil& st, const double2* dTr, int R32, double& dT, double& ratio) {
    const double2* nodes = dTr + node_index(st.b[0], st.b[1], st.b[2], R32);
    const int64_t R = R32;
    dT = ratio = 0.0;
#pragma unroll
    for (int ox = 0; ox < 3; ++ox)
#pragma unroll
        for (int oy = 0; oy < 3; ++oy) {
            const float wxy = st.w[0][ox] * st.w[1][oy];
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) {
                const double2 d = nodes[(ox * R + oy) * R + oz];
                const double w = (double)(wxy * st.w[2][oz]);
                dT = fma(w, d.x, dT);
                ratio = fma(w, d.y, ratio);
            }
        }
}

// a[k] for a run-time k in {0, 1, 2} without dynamic register indexing (which would move `a` to local
// memory): the outer loop of a long gather stays a loop, so that its 27 nodes' loads are not all hoisted
// and held at once.
BK_DEV float pick3(const float* a, int k) { return k == 0 ? a[0] : (k == 1 ? a[1] : a[2]); }

// Derivative of the quadratic weight of offset o by l (transfer.py:4-13).
BK_DEV float qweight_grad(float l, int o) {
    if (o == 0) return l - 1.5f;
    if (o == 1) return -2.f * (l - 1.f);
    return l - 0.5f;
}

// Stencil node j in 0..26 -> offsets (j / 9, (j / 3) % 3, j % 3), the reference's loop order.
BK_DEV void node_offset(int j, int& ox, int& oy, int& oz) {
    ox = j / 9;
    oy = (j / 3) % 3;
    oz = j - 9 * ox - 3 * oy;
}

// How a warp's particles are laid out in its record: this lane's column, and the columns that start a
// run (bit k: column k holds a valid particle whose stencil base differs from column k - 1's).
struct Runs {
    int column;
    unsigned starts;
};

// A warp with this many runs first groups its lanes by stencil base, in bodies of this many particles
// (grids up to 1024^3, whose bases fit 3 x 10 bits). Particles ordered by cell have 2 (40 a cell) to 5
// (8 a cell) runs a warp and gain nothing; particles in another order, as sampled tet by tet (up to 32
// runs a warp, about 10 bases), get a third of the atomics, and node sums of fewer and larger parts.
// P2G in tet order: 41k particles 16 -> 8.6 us, 5k 9.7 -> 8.3. Smaller bodies keep the order of their
// samples although grouping is faster there too (192 particles: 9.4 us, grouped 8.6): the finite differences
// that check the gradients over such bodies are differences of float32 roundings, and were resolved with
// the sums in that order (grouped, two of them miss their tolerance, by 9% and 74%).
constexpr int kGroupRuns = 8;
constexpr int64_t kGroupParticles = 256;

BK_DEV bool group_lanes(int64_t n, int R) { return n >= kGroupParticles && R <= 1024; }

// Momentum sums of a block's warps are merged before they reach the grid. A particle that has just crossed
// into another cell gives that cell's far nodes weights of 1e-6 and less; sent alone, such a sum is
// below half a unit of a node's last place and lost. Error against 64 bits of warps' sums sent
// alone over that of a node tile shared by 256 particles: grid mass of a strained 39k cube in sample order
// 2.5 +- 0.4, velocities of a pre-stressed 60k loaf 1.009 +- 0.001, its temperature gradient 1.05 (where
// the reverse scatter is not merged either); merged 0.94 +- 0.2, 1.000 and 1.003. Two forms:
// * bodies below kKeptParticles: every warp sums into a tile of its own (WarpTiles), which costs the fewest
//   steps but 24 KB a block: four blocks on an SM, one wave of up to 75,776 particles.
// * larger bodies, which need eight blocks on an SM: the warps keep their sums in their records and
//   add them up in the space of the values (merge_runs).
// us a substep with the tiles and with the kept sums: loaf of 30k particles 45.6 and 53.3, 65.6k 45.3 and 51.9,
// 90k 53.9 and 54.5, 302k 116.2 and 113.7; ball of 30k 52.6 and 58.0; 41k cube in sample order 22.2 and 24.8.
constexpr int64_t kKeptParticles = 65536;

BK_DEV Runs find_runs(bool valid, const int* b, bool group) {
    const int lane = threadIdx.x & 31;
    const int p0 = __shfl_up_sync(kWarp, b[0], 1), p1 = __shfl_up_sync(kWarp, b[1], 1),
              p2 = __shfl_up_sync(kWarp, b[2], 1);
    const bool before = __shfl_up_sync(kWarp, (int)valid, 1) != 0;
    Runs r;
    r.column = lane;
    r.starts = __ballot_sync(kWarp, valid && (lane == 0 || !before || p0 != b[0] || p1 != b[1] || p2 != b[2]));
    if (group && __popc(r.starts) >= kGroupRuns) {
        // An invalid particle is a group of its own (its stored weights are zero).
        const unsigned key = valid ? (unsigned)(b[0] << 20 | b[1] << 10 | b[2]) : 0x80000000u | (unsigned)lane;
        const unsigned peers = __match_any_sync(kWarp, key);
        const int rank = __popc(peers & ((1u << lane) - 1u)), first = __ffs(peers) - 1;
        // Groups of four or more first (each leaves room for a kept sum, merge_runs), then the others, in the
        // order of their first lanes: two prefix sums of the sizes in one word.
        const int peer_count = __popc(peers);
        const bool large = peer_count >= 4;
        int sum = rank == 0 ? (large ? peer_count : peer_count << 16) : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(kWarp, sum, o);
            if (lane >= o) sum += v;
        }
        const int all_large = __shfl_sync(kWarp, sum, 31) & 0xffff;
        const int start = (large ? sum & 0xffff : all_large + (sum >> 16)) - peer_count;  // of a first lane's group
        r.column = __shfl_sync(kWarp, start, first) + rank;
        r.starts = __reduce_or_sync(kWarp, valid && rank == 0 ? 1u << r.column : 0u);
    }
    return r;
}

// Column one past the run before the next start. (A run may include columns of invalid particles,
// whose stored weights are zero.)
BK_DEV int run_end(unsigned later_starts) { return later_starts ? __ffs(later_starts) - 1 : 32; }

// The 27 weights of this thread's particle into its column of the record's node-major rows.
template <int kPitch>
BK_DEV void put_weights(float (&w)[27][kPitch], int column, bool valid, const Stencil& st) {
#pragma unroll
    for (int ox = 0; ox < 3; ++ox)
#pragma unroll
        for (int oy = 0; oy < 3; ++oy) {
            const float wxy = valid ? st.w[0][ox] * st.w[1][oy] : 0.f;
#pragma unroll
            for (int oz = 0; oz < 3; ++oz) w[9 * ox + 3 * oy + oz][column] = valid ? wxy * st.w[2][oz] : 0.f;
        }
}

// Widens the node box `bounds` ([0..2] lowest, [3..5] highest node) over the block's valid stencils.
// Every thread of the block calls it, early, while the warps are still together: one test per warp
// in place of two barriers cost 4 us of 39 on a 41k-particle body, whose warps all start on an empty
// box and queue on its six addresses.
BK_DEV void widen_box(int* bounds, bool valid, const int* b) {
    __shared__ int s_box[6];
    if (threadIdx.x < 6) s_box[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int lo = __reduce_min_sync(kWarp, valid ? b[a] : INT_MAX);
        const int hi = __reduce_max_sync(kWarp, valid ? b[a] + 2 : INT_MIN);
        if ((threadIdx.x & 31) == 0 && lo != INT_MAX) {
            atomicMin(&s_box[a], lo);
            atomicMax(&s_box[3 + a], hi);
        }
    }
    __syncthreads();
    // The box only widens, so a value read through L2 that is older than the current one is never
    // narrower: a block whose box lies inside it skips the atomics.
    if (threadIdx.x < 6) {
        const int t = threadIdx.x, now = __ldcg(bounds + t);
        if (t < 3 && s_box[t] < now) atomicMin(bounds + t, s_box[t]);
        if (t >= 3 && s_box[t] > now) atomicMax(bounds + t, s_box[t]);
    }
}

// ------------------------------------------------------------- momentum form
// Node j of particle k receives w_jk (q + A o_j) in x, y, z and w_jk m in w, o_j the node's offsets
// in cells: the run's sums of w m, w q and w A (paired accumulators, one packed multiply-add per
// pair), with o_j applied once per run. Lane j < 27 owns node j; a lane reads its weight row at the
// particle's column (conflict-free) and the values as 128-bit broadcasts.
struct MomentumRecord {
    float4 val[32][3];  // {m q0 q1 q2} {A0 A1 A2 A3} {A4 A5 A6 A7}
    int64_t corner[32];  // the stencil's first node (a run reads its start's: one broadcast, no shuffles)
    float a8[32];
    float w[27][33];
    unsigned key[32];              // the stencil base, 10 bits an axis
    unsigned base[kGroupRuns];     // of the runs kept for the block
    int kept;
};

BK_DEV unsigned pack_base(int x, int y, int z) { return (unsigned)(x << 20 | y << 10 | z); }

// Nodes of a block's box that fit a tile. A block of 128 covers up to 300 in the sample order of a 41k cube, 85 to
// 95% of the blocks of a ball or sphere at 8 particles a cell have 384 or fewer; the others' sums go
// to the grid one by one.
constexpr int kMergeNodes = 384;

// Node t of a box with the extents ext (t < 384, so t * ext < 2^16: exact quotients).
BK_DEV int64_t box_node(int t, const int* lo, const int* ext, int R) {
    const unsigned by_z = (unsigned)__fdividef(65536.f, (float)ext[2]) + 1u, by_y = (unsigned)__fdividef(65536.f, (float)ext[1]) + 1u;
    const int yx = (int)((unsigned)t * by_z >> 16), x = (int)((unsigned)yx * by_y >> 16);
    return node_index(lo[0] + x, lo[1] + yx - x * ext[1], lo[2] + t - yx * ext[2], R);
}

// A tile over the block's node box for each of its four warps.
struct WarpTiles {
    float4 node[4][kMergeNodes];
    int low[4][3], high[4][3];  // each warp's bases
};
// (Declared in an inlined function, as warp_records of the substep's scatter.)
BK_DEV WarpTiles* warp_tiles() {
    __shared__ WarpTiles tiles;
    return &tiles;
}

// The block's kept runs, summed in a tile over their node box and sent to L2 as one atomic per node. Warp
// c sums component c, run by run in the order of the block's particles, in the space of its particles'
// values (no shared atomics: no two warps touch a word; with a thread per node looping over the runs 18 us).
BK_DEV void merge_runs(MomentumRecord* sm, float4* __restrict__ nodes, int R) {
    static_assert(sizeof(MomentumRecord::val) >= kMergeNodes * sizeof(float) && kGroupRuns == 8, "tile and slots");
    const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;
    __syncthreads();
    const int from = lane >> 3, slot = lane & 7;
    const bool kept = slot < sm[from].kept;
    const unsigned mask = __ballot_sync(kWarp, kept);
    if (!mask) return;  // the same for every warp
    const unsigned b = kept ? sm[from].base[slot] : 0u;
    int lo[3], ext[3], at[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        at[a] = (int)(b >> (20 - 10 * a)) & 1023;
        lo[a] = __reduce_min_sync(kWarp, kept ? at[a] : 1024);
        ext[a] = __reduce_max_sync(kWarp, kept ? at[a] : 0) + 3 - lo[a];
    }
    const int count = ext[0] * ext[1] * ext[2];
    int ox, oy, oz;
    node_offset(lane < 27 ? lane : 0, ox, oy, oz);
    if (count <= kMergeNodes) {
        float* const tile = reinterpret_cast<float*>(sm[c].val);
        for (int t = lane; t < count; t += 32) tile[t] = 0.f;
        const int corner = ((at[0] - lo[0]) * ext[1] + at[1] - lo[1]) * ext[2] + at[2] - lo[2];
        float* const mine = tile + (ox * ext[1] + oy) * ext[2] + oz;
        const int row = 33 * (lane < 27 ? lane : 0) + c;
        __syncwarp();
        for (unsigned left = mask; left; left &= left - 1) {
            const int l = __ffs(left) - 1;
            const int first = __shfl_sync(kWarp, corner, l);
            if (lane < 27) mine[first] += (&sm[l >> 3].w[0][0])[row + 4 * (l & 7)];
            __syncwarp();
        }
        __syncthreads();
        for (int t = threadIdx.x; t < count; t += 128) {
            const float4 sum = make_float4(reinterpret_cast<const float*>(sm[0].val)[t], reinterpret_cast<const float*>(sm[1].val)[t],
                                           reinterpret_cast<const float*>(sm[2].val)[t], reinterpret_cast<const float*>(sm[3].val)[t]);
            if (sum.x == 0.f && sum.y == 0.f && sum.z == 0.f && sum.w == 0.f) continue;
            atomicAdd(nodes + box_node(t, lo, ext, R), sum);
        }
    } else if (lane < 27) {  // far apart: each warp its own runs
        const MomentumRecord& rec = sm[c];
        for (int k = 0; k < rec.kept; ++k) {
            const unsigned a = rec.base[k];
            const float* v = rec.w[lane] + 4 * k;
            atomicAdd(nodes + node_index((int)(a >> 20) + ox, (int)(a >> 10 & 1023) + oy, (int)(a & 1023) + oz, R),
                      make_float4(v[0], v[1], v[2], v[3]));
        }
    }
}

// Sum of one run's particles, columns s to e - 1, at this lane's node (j < 27): momentum and mass.
BK_DEV float4 run_sum(const MomentumRecord& rec, const float* wj, const float* fo, int s, int e) {
    float2 mq0 = {0.f, 0.f}, q12 = {0.f, 0.f}, A01 = {0.f, 0.f}, A23 = {0.f, 0.f};
    float2 A45 = {0.f, 0.f}, A67 = {0.f, 0.f};
    float A8 = 0.f;
#pragma unroll 2
    for (int k = s; k < e; ++k) {
        const float w = wj[k];
        const float2 ww = make_float2(w, w);
        const float4 v0 = rec.val[k][0], v1 = rec.val[k][1], v2 = rec.val[k][2];
        mq0 = ffma2(ww, make_float2(v0.x, v0.y), mq0);
        q12 = ffma2(ww, make_float2(v0.z, v0.w), q12);
        A01 = ffma2(ww, make_float2(v1.x, v1.y), A01);
        A23 = ffma2(ww, make_float2(v1.z, v1.w), A23);
        A45 = ffma2(ww, make_float2(v2.x, v2.y), A45);
        A67 = ffma2(ww, make_float2(v2.z, v2.w), A67);
        A8 = fmaf(w, rec.a8[k], A8);
    }
    const float aq[3] = {mq0.y, q12.x, q12.y};
    const float aA[9] = {A01.x, A01.y, A23.x, A23.y, A45.x, A45.y, A67.x, A67.y, A8};
    float ap[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        ap[r] = aq[r] + (aA[3 * r] * fo[0] + aA[3 * r + 1] * fo[1] + aA[3 * r + 2] * fo[2]);
    return make_float4(ap[0], ap[1], ap[2], mq0.x);
}

// How a block's sums reach the grid.
enum class Sums { kAlone, kTiles, kKept };

// (The adjoint of G2P has the same form with m = 0.) kTiles and kKept: every warp of a block of 128 threads
// calls it; `tiles` is used by kTiles only. kKept keys bases by 10 bits an axis: on larger grids
// (`keyed` false) it sends the sums one by one. `group` and `keyed` are the same for all threads.
template <Sums kSums>
BK_DEV void scatter_momentum(MomentumRecord* sm, WarpTiles* tiles, bool valid, const Stencil& st, float m, const float* q,
                             const float* A, float4* __restrict__ nodes, int R, bool group, bool keyed = true) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    MomentumRecord& rec = sm[warp];
    const Runs runs = find_runs(valid, st.b, group);
    const bool keep = kSums == Sums::kKept && keyed;
    put_weights(rec.w, runs.column, valid, st);
    rec.val[runs.column][0] = make_float4(m, q[0], q[1], q[2]);
    rec.val[runs.column][1] = make_float4(A[0], A[1], A[2], A[3]);
    rec.val[runs.column][2] = make_float4(A[4], A[5], A[6], A[7]);
    rec.a8[runs.column] = A[8];
    rec.corner[runs.column] = node_index(st.b[0], st.b[1], st.b[2], R);
    if (keep) rec.key[runs.column] = pack_base(st.b[0], st.b[1], st.b[2]);
    int lo[3], ext[3], count = 0;  // the block's box (kTiles), count its nodes where they fit
    float4* tile = nullptr;
    if constexpr (kSums == Sums::kTiles) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int low = __reduce_min_sync(kWarp, valid ? st.b[a] : INT_MAX);
            const int high = __reduce_max_sync(kWarp, valid ? st.b[a] : INT_MIN);
            if (lane == 0) {
                tiles->low[warp][a] = low;
                tiles->high[warp][a] = high;
            }
        }
        __syncthreads();
        int64_t all = 1;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            lo[a] = min(min(tiles->low[0][a], tiles->low[1][a]), min(tiles->low[2][a], tiles->low[3][a]));
            const int high = max(max(tiles->high[0][a], tiles->high[1][a]), max(tiles->high[2][a], tiles->high[3][a]));
            if (lo[a] > high) return;  // no valid particle in the block (lo = INT_MAX): the same for all threads
            ext[a] = high + 3 - lo[a];
            all *= ext[a];
        }
        if (all <= kMergeNodes) count = (int)all;
        tile = tiles->node[warp];
        for (int t = lane; t < count; t += 32) tile[t] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (valid) rec.key[runs.column] = ((st.b[0] - lo[0]) * ext[1] + st.b[1] - lo[1]) * ext[2] + st.b[2] - lo[2];
    }
    __syncwarp();
    int ox, oy, oz;
    node_offset(lane < 27 ? lane : 0, ox, oy, oz);
    const float fo[3] = {(float)ox, (float)oy, (float)oz};
    float* const wj = rec.w[lane < 27 ? lane : 0];
    float4* const mine = nodes + ((int64_t)ox * R + oy) * R + oz;
    if constexpr (kSums == Sums::kTiles) tile += (ox * ext[1] + oy) * ext[2] + oz;
    int kept = 0;
    unsigned starts = runs.starts;
    while (starts) {
        const int s = __ffs(starts) - 1;
        starts &= starts - 1;
        const int e = run_end(starts);
        // A kept run's sums take the weights' place: row j is read by lane j only, columns below e no more.
        const bool here = keep && kept < kGroupRuns && 4 * (kept + 1) <= e;
        if (lane < 27) {
            const float4 sum = run_sum(rec, wj, fo, s, e);
            if (here) {
                wj[4 * kept] = sum.x;
                wj[4 * kept + 1] = sum.y;
                wj[4 * kept + 2] = sum.z;
                wj[4 * kept + 3] = sum.w;
            } else if (kSums == Sums::kTiles && count > 0) {
                float4& node = tile[rec.key[s]];
                const float4 old = node;
                node = make_float4(old.x + sum.x, old.y + sum.y, old.z + sum.z, old.w + sum.w);
            } else {
                atomicAdd(mine + rec.corner[s], sum);
            }
        }
        if (kSums == Sums::kTiles) __syncwarp();  // the next run's lanes meet these nodes
        if (here) {
            if (lane == 0) rec.base[kept] = rec.key[s];
            ++kept;
        }
    }
    if constexpr (kSums == Sums::kTiles) {
        __syncthreads();
        for (int t = threadIdx.x; t < count; t += 128) {
            const float4 a = tiles->node[0][t], b = tiles->node[1][t], c = tiles->node[2][t], d = tiles->node[3][t];
            const float4 sum = make_float4((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y), (a.z + b.z) + (c.z + d.z),
                                           (a.w + b.w) + (c.w + d.w));
            if (sum.x == 0.f && sum.y == 0.f && sum.z == 0.f && sum.w == 0.f) continue;
            atomicAdd(nodes + box_node(t, lo, ext, R), sum);
        }
    } else if (keep) {
        if (lane == 0) rec.kept = kept;
        merge_runs(sm, nodes, R);
    }
}

// ------------------------------------------------------------- float64 form
// kF float64 values per particle (the transport fields, the surface rates), node j receiving
// w_jk value_k: the contraction (27 nodes x particles) (particles x kF) on the float64 tensor cores,
// mma.m8n8k4 with four 8-node row tiles and the values in the columns, four particles a step. The
// products and sums are float64, as the reference's float64 atomics: float32 partial sums moved the
// node temperature E / C by ~3e-5 K, harmless to the trajectory but enough to make finite differences
// of the loss in the initial temperatures disagree with the adjoint by several percent.
// A scalar loop (lane j owns node j) reads five shared words and issues four float64 multiply-adds
// per particle; the mma form reads five words and issues four mma per FOUR particles. The row pitch
// of 36 puts the 32 words of a fragment (8 rows x 4 particles) in 32 banks.
template <int kF>
struct ScalarRecord {
    double val[kF][36];
    int64_t corner[32];  // the stencil's first node
    float w[27][36];
};

BK_DEV void dmma(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// Adds values val[0..kF) of the warp's particles to the node fields f[0..kF) (R^3 float64 each, kStride
// apart: 2 for the halves of a double2 field).
template <int kF, int kStride = 1>
BK_DEV void scatter_scalars(ScalarRecord<kF>& rec, bool valid, const Stencil& st, const double* val,
                            double* const (&f)[kF], int R, bool group) {
    static_assert(kF >= 1 && kF <= 4, "the values share one 8-column tile");
    const int lane = threadIdx.x & 31;
    const int row = lane >> 2, quad = lane & 3;  // fragment coordinates
    const Runs runs = find_runs(valid, st.b, group);
    put_weights(rec.w, runs.column, valid, st);
#pragma unroll
    for (int k = 0; k < kF; ++k) rec.val[k][runs.column] = valid ? val[k] : 0.0;
    rec.corner[runs.column] = node_index(st.b[0], st.b[1], st.b[2], R);
    __syncwarp();
    // Accumulator fragment: row 8 t + row, columns 2 quad and 2 quad + 1 (fields; quads 0 and 1).
    int offset[4];
    bool node[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        const int j = 8 * t + row;
        int ox, oy, oz;
        node_offset(j < 27 ? j : 0, ox, oy, oz);
        offset[t] = (ox * R + oy) * R + oz;
        node[t] = j < 27;
    }
    // (selects, not f[2 * quad]: a run-time index would copy the pointers to local memory)
    double* const f0 = kF > 2 && quad == 1 ? f[2] : f[0];
    double* const f1 = kF > 3 && quad == 1 ? f[3] : f[kF > 1 ? 1 : 0];
    unsigned starts = runs.starts;
    while (starts) {
        const int s = __ffs(starts) - 1;
        starts &= starts - 1;
        const int e = run_end(starts);
        double d[4][2] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
        for (int k0 = s; k0 < e; k0 += 4) {
            // Fragments: weight of node 8 t + row and value `row` of particle k0 + quad; particles past
            // the run are zero on both sides (their weights may belong to another run, or be NaN).
            const int k = k0 + quad;
            const bool in = k < e;
            double b = 0.0;
            if (in && row < kF) b = rec.val[row][k];
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                float w = 0.f;
                if (in && node[t]) w = rec.w[8 * t + row][k];
                dmma(d[t][0], d[t][1], (double)w, b);
            }
        }
        const int64_t corner = rec.corner[s];
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (node[t]) {
                if (2 * quad < kF) atomicAdd(f0 + kStride * (corner + offset[t]), d[t][0]);
                if (2 * quad + 1 < kF) atomicAdd(f1 + kStride * (corner + offset[t]), d[t][1]);
            }
    }
}

}  // namespace bk
