// Fused MLS-MPM baking substep for sm_100a (the simulator's hot path).
//
// The reference runs ~16 Warp launches per substep (physics/mpm.py:163-225,
// physics/thermal_water.py:296-367) with three host synchronisations and fresh
// dense-grid allocations. Here one substep is seven bodies in six launches (four without transport):
//
//   surface_vertices   rebuild only the boundary-face vertices (a block of 32-256 threads per
//                      vertex, sized by its mean particle bindings)
//   surface_owners     face areas -> boundary heat/loss/exchange of face-owning particles, scattered
//   transport_scatter  scalar P2G (volume, capacity, energy, water), warp-cooperative per stencil base;
//                      its blocks are spread among those of the vertices of a coarse mesh, or of the
//                      owners of a fine one (launch_substep)
//   diffuse            7-point finite-volume heat/water flux over the active node box only; its blocks
//                      also zero the last substep's momentum box (a launch of its own without transport)
//   p2g                scalar G2P + gas source + gas/water stress + momentum P2G, fused per particle
//   grid_update        momentum -> velocity with walls over the active box; zeroes the scatter fields
//   g2p_return         G2P (v, C, x, F) fused with the Ding return map (float64 SVD in registers)
//
// Scatter scheme (bk_scatter.cuh): a warp groups its 32 particles into runs of equal stencil base,
// sums each run and issues one atomic per run, node and field. With particles ordered by cell this
// turns 27 atomics per particle into 27 per run of ~tens of particles, and any order stays correct.
//
// The active node box (min/max stencil node of the current particles) bounds
// every dense grid pass; the grid passes leave the scatter fields zeroed behind
// them, so no dense memset is needed between substeps.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdio>
#include <type_traits>
#include <utility>
#include <vector>

#include "baking_b200.h"
#include "bk_common.h"
#include "bk_device.cuh"
#include "bk_launch.cuh"
#include "bk_mlp.cuh"
#include "bk_scatter.cuh"
#include "bk_profile.h"

using namespace bk;

namespace {

constexpr int kThreads = 256;

inline cudaStream_t S(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Kernel-side copy of the parameters (plain values only).
struct Params {
    int64_t n, pitch;
    int R, bc;
    float origin[3], dx, rec_dx, dt, gravity[3];
    int material;
    DingParamsDev ding;
    int transport, gas, settling;
    float oven, tray, tray_transfer, surface_loss, water_density, latent;
    int water_enabled;
    float conductivity, diffusivity, s0, water_stress;
    float ambient, density, elastic_modulus, cfl, peak, width;
    int keep_fields;
    int prescattered, prescatter_next, prescatter_stale;
    int box_widened;  // the launches before P2G in this call widen the node box over the same positions
    int32_t* status;
};

Params to_params(const BkSubstepParams& p) {
    Params k;
    k.n = p.n; k.pitch = p.pitch; k.R = p.resolution; k.bc = p.boundary_cells;
    for (int a = 0; a < 3; ++a) { k.origin[a] = p.origin[a]; k.gravity[a] = p.gravity[a]; }
    k.dx = p.spacing; k.rec_dx = 1.0f / p.spacing; k.dt = p.time_step;
    k.material = p.material;
    k.ding = ding_params_dev(p.ding);
    k.transport = p.transport; k.gas = p.gas; k.settling = p.settling;
    k.oven = p.scalar.oven_temperature; k.tray = p.scalar.tray_temperature;
    k.tray_transfer = p.scalar.tray_transfer; k.surface_loss = p.scalar.surface_loss;
    k.water_density = p.scalar.water_density; k.latent = p.scalar.latent_heat;
    k.water_enabled = p.scalar.water_enabled;
    k.conductivity = p.conductivity; k.diffusivity = p.diffusivity; k.s0 = p.initial_saturation;
    k.water_stress = p.water_stress;
    k.ambient = p.gas_ambient_pressure; k.density = p.density; k.elastic_modulus = p.elastic_modulus;
    k.cfl = p.cfl_limit; k.peak = p.gas_peak; k.width = p.gas_width;
    k.keep_fields = p.keep_transport_fields;
    k.prescattered = p.transport_prescattered;
    k.prescatter_next = p.transport_prescatter_next;
    k.prescatter_stale = p.transport_prescatter_stale;
    k.box_widened = 0;
    k.status = p.status;
    return k;
}

// The configuration of the loaf and dough bodies: Ding with temperature-dependent parameters, gas
// with the coupled porosity solve, thermal-water transport, no per-particle diagnostics and no
// harvest. The particle kernels have an instance for it in which these flags are compile-time
// constants, so the branches of the other configurations fold away (same arithmetic, less code).
bool loaf_mode(const BkSubstepParams& p, const BkDiagnostics& d) {
    return p.material == 1 && p.transport && p.gas && p.ding.coupled_porosity && p.ding.temperature_enabled &&
           !d.plastic_gradients && !d.return_residuals && !d.porosity_residuals &&
           !(p.surrogate && p.surrogate->samples);
}
__device__ __forceinline__ void fix_loaf_mode(Params& P) {
    P.material = 1;
    P.transport = 1;
    P.gas = 1;
    P.ding.coupled_porosity = 1;
    P.ding.temperature_enabled = 1;
}

struct GridPtrs {
    float4* pm;
    float4* v;
    double* f[7];
    double2* dTr;
    int* bounds;
};

GridPtrs grid_ptrs(const BkGrid& g) {
    GridPtrs r;
    r.pm = reinterpret_cast<float4*>(g.node_pm);
    r.v = reinterpret_cast<float4*>(g.node_v);
    for (int k = 0; k < 7; ++k) r.f[k] = g.fields[k];
    r.dTr = reinterpret_cast<double2*>(g.node_dT_ratio);
    r.bounds = g.bounds;
    return r;
}

// The block a kernel body runs as: its index among the blocks given to its simulator and their
// number. A plain launch gives one simulator the whole grid; a batched launch (below) splits its
// grid between the simulators of an instance table.
struct Slot {
    int block, blocks;
};
__device__ __forceinline__ Slot grid_slot() { return Slot{(int)blockIdx.x, (int)gridDim.x}; }

// How a kernel body takes its parameter structs: by value from a plain launch's parameter space
// (a reference to a kernel parameter would make the compiler copy it to local memory), by
// reference to the batched launch's shared-memory entry (a value copy would hold every field in
// registers).
template <class T, bool kRef>
using Arg = typename std::conditional<kRef, const T&, const T>::type;

// ------------------------------------------------------------------ surface
// geometry/mesh_tracking.py:13-38 restricted to the vertices of boundary faces. A vertex of a
// coarse mesh binds thousands of particles: one block of kBlock = 128 or 256 threads per vertex
// keeps enough gathers in flight. A vertex of a fine mesh binds tens: kBlock = 32 then means one
// warp per vertex, kVertexWarps vertices to a block.
constexpr int kVertexWarps = 4;

// Blocks of the surface vertex launch for `vertices` vertices at block size `threads`.
inline unsigned vertex_launch_blocks(int64_t vertices, int threads) {
    return (unsigned)(threads == 32 ? (vertices + kVertexWarps - 1) / kVertexWarps : vertices);
}
constexpr int vertex_launch_threads(int threads) { return threads == 32 ? 32 * kVertexWarps : threads; }

template <int kBlock, bool kRef = false, int kParts = 1>
__device__ __forceinline__ void surface_vertices_body(Arg<Params, kRef> P, const float* x,
                                                      const float* F, Arg<BkSurface, kRef> sf, Slot sl) {
    if constexpr (kBlock == 32) {
        const int64_t k = (int64_t)sl.block * kVertexWarps + (threadIdx.x >> 5);
        if (k >= sf.vertex_count) return;  // whole warps
        const int vid = sf.vertex_ids[k];
        const float v = vertex_warp(sf.binding_offsets, sf.binding_particles, sf.binding_weights,
                                    sf.reference_offsets, sf.binding_pitch, sf.reference_vertices, sf.vertex_pitch, x,
                                    F, P.pitch, vid);
        const int lane = threadIdx.x & 31;
        if (lane < 3) sf.vertices[lane * sf.vertex_pitch + vid] = v;
    } else {
        const int vid = sf.vertex_ids[sl.block];
        const float v = vertex_block<kBlock, kParts>(sf.binding_offsets, sf.binding_particles, sf.binding_weights,
                                               sf.reference_offsets, sf.binding_pitch, sf.reference_vertices,
                                               sf.vertex_pitch, x, F, P.pitch, vid);
        if (threadIdx.x < 3) sf.vertices[threadIdx.x * sf.vertex_pitch + vid] = v;
    }
}

template <int kBlock>
__global__ void __launch_bounds__(kBlock == 32 ? 32 * kVertexWarps : kBlock) k_surface_vertices(Params P, const float* x,
                                                          const float* F, BkSurface sf) {
    pdl_enter();
    surface_vertices_body<kBlock>(P, x, F, sf, grid_slot());
}

// ------------------------------------------------------- surface terms
// physics/thermal_water.py:77-92 (face areas, tray contact) and the surface terms of :108-122 for
// the face-owning particles, in two layouts chosen by how many particles own faces:
// * few owners, each with several faces (a coarse voxel mesh: about 3k owners of a 1M-particle
//   loaf): one warp per owner; lane 0 sums the owner's faces in order, every lane forms the rates,
//   lane j < 27 adds stencil node j's share (27 atomics in parallel);
// * many owners (a fine tetrahedral mesh: about a third of a dough ball's particles own faces): one
//   thread per owner, the node shares summed per stencil run like the transport scatter.
// With accumulators set in `sf`, the owner's water-loss and heat-exchange accumulators also advance
// by one substep (thermal_water.py:225-226), which bk_surface_accumulate does otherwise.
constexpr int kOwnerThreads = 128;  // also the block size of the transport scatter, which shares launches with it

// Area of boundary face f and whether it touches the tray.
template <class SF>
__device__ __forceinline__ double face_area(const SF& sf, int f, bool& tray) {
    const int64_t vp = sf.vertex_pitch;
    double q[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int vid = sf.faces[3 * f + k];
#pragma unroll
        for (int a = 0; a < 3; ++a) q[k][a] = (double)sf.vertices[a * vp + vid];
    }
    double e1[3] = {q[1][0] - q[0][0], q[1][1] - q[0][1], q[1][2] - q[0][2]};
    double e2[3] = {q[2][0] - q[0][0], q[2][1] - q[0][1], q[2][2] - q[0][2]};
    double nr[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    double len = sqrt(nr[0] * nr[0] + nr[1] * nr[1] + nr[2] * nr[2]);
    double cy = (q[0][1] + q[1][1] + q[2][1]) / 3.0;
    tray = cy <= (double)(sf.floor_height + sf.contact_distance) && nr[1] < -0.2 * len;
    return 0.5 * len;
}

// Exposed and tray-contact areas of owner o's faces, summed in face order.
template <class SF>
__device__ __forceinline__ void owner_areas(const SF& sf, int64_t o, double& exposed, double& contact) {
    exposed = 0.0;
    contact = 0.0;
    for (int f = sf.owner_face_offsets[o]; f < sf.owner_face_offsets[o + 1]; ++f) {
        bool tray;
        const double area = face_area(sf, f, tray);
        if (tray) contact += area;
        else exposed += area;
    }
}

// The same for a warp's 32 consecutive owners (or what is left of them): their faces are consecutive
// too, so the lanes take the faces, kFaceChunk at a time, and each owner then adds its own in face
// order. A thread walking its own faces waited for two dependent gathers per face, as often as the
// warp's busiest owner has faces.
constexpr int kFaceChunk = 64;
struct FaceChunk {
    double area[kFaceChunk];  // negative zero or below: tray contact
};
template <class SF>
__device__ __forceinline__ void owner_areas_warp(const SF& sf, FaceChunk& chunk, int64_t o, bool mine, double& exposed,
                                                 double& contact) {
    const int lane = threadIdx.x & 31;
    exposed = 0.0;
    contact = 0.0;
    const int f0 = mine ? sf.owner_face_offsets[o] : 0, f1 = mine ? sf.owner_face_offsets[o + 1] : 0;
    const unsigned owners = __ballot_sync(kWarp, mine);
    if (!owners) return;
    const int first = __shfl_sync(kWarp, f0, 0), last = __shfl_sync(kWarp, f1, 31 - __clz(owners));
    for (int base = first; base < last; base += kFaceChunk) {
#pragma unroll
        for (int k = 0; k < kFaceChunk; k += 32) {
            const int f = base + k + lane;
            if (f < last) {
                bool tray;
                const double area = face_area(sf, f, tray);
                chunk.area[k + lane] = tray ? -area : area;
            }
        }
        __syncwarp();
        for (int f = max(f0, base); f < min(f1, base + kFaceChunk); ++f) {
            const double area = chunk.area[f - base];
            if (signbit(area)) contact -= area;
            else exposed += area;
        }
        __syncwarp();
    }
}

// What owner particle p's rates and scatter read of the state, loaded before its face areas (a chain of
// three dependent gathers) so that the two chains run side by side.
struct OwnerState {
    V3 x;
    M3 F;
    double T, W;
    float volume;
};
template <class PP, class ST, class CS>
__device__ __forceinline__ OwnerState owner_state(const PP& P, const ST& in, const CS& cst, int p) {
    return OwnerState{load_v3(in.x, p, P.pitch), load_m3(in.F, p, P.pitch), in.temperature[p], in.water[p],
                      __ldg(cst.volume + p)};
}

// Heat, loss and exchange rates of an owner particle from its areas; rate[0..2].
template <class PP, class CS>
__device__ __forceinline__ void owner_rates(const PP& P, const OwnerState& o, const CS& cst, double exposed,
                                            double contact, double* rate) {
    const double vol = (double)o.volume * (double)det3(o.F);
    const double T = o.T, W = o.W;
    double sat = W / ((double)P.water_density * vol);
    double loss = 0.0;
    if (P.water_enabled) loss = (double)P.surface_loss * T * sat * exposed;
    double h = (double)cst.heat_parameter[0];
    double heat = h * exposed * ((double)P.oven - T) + (double)P.tray_transfer * contact * ((double)P.tray - T)
                - (double)P.latent * loss;
    double exch = h * exposed + (double)P.tray_transfer * contact;
    if (P.water_enabled) exch += (double)(P.latent * P.surface_loss) * sat * exposed;
    rate[0] = heat;
    rate[1] = loss;
    rate[2] = exch;
}

// Stores owner o's rates and advances its accumulators when `sf` names them.
template <class SF>
__device__ __forceinline__ void owner_store(const SF& sf, int64_t o, int p, const double* rate) {
    sf.owner_heat[o] = rate[0];
    sf.owner_loss[o] = rate[1];
    if (sf.accumulate_water_losses) {
        sf.accumulate_water_losses[p] += (double)sf.accumulate_time_step * rate[1];
        sf.accumulate_heat_exchanges[p] += (double)sf.accumulate_time_step * rate[0];
    }
}

template <bool kRef = false>
__device__ __forceinline__ void surface_owners_warp_body(Arg<Params, kRef> P, Arg<BkState, kRef> in,
                                                         Arg<BkConstants, kRef> cst, Arg<BkSurface, kRef> sf,
                                                         Arg<GridPtrs, kRef> g, int32_t* sim_flags, Slot sl) {
    const int lane = threadIdx.x & 31;
    const int64_t o = (sl.block * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (o >= sf.owner_count) return;  // whole warps
    const int p = sf.owners[o];
    const OwnerState os = owner_state(P, in, cst, p);
    double exposed = 0.0, contact = 0.0;
    if (lane == 0) owner_areas(sf, o, exposed, contact);
    exposed = __shfl_sync(kWarp, exposed, 0);
    contact = __shfl_sync(kWarp, contact, 0);
    double rate[3];
    owner_rates(P, os, cst, exposed, contact, rate);
    if (lane == 0) owner_store(sf, o, p, rate);
    Stencil st = make_stencil(os.x, P.origin, P.dx, P.R, P.rec_dx);
    if (!st.valid) {
        if (lane == 0) set_flag(sim_flags, 1);
        return;
    }
    if (lane < 27) {
        int ox, oy, oz;
        node_offset(lane, ox, oy, oz);
        double w = (double)(st.w[0][ox] * st.w[1][oy] * st.w[2][oz]);
        int64_t node = node_index(st.b[0] + ox, st.b[1] + oy, st.b[2] + oz, P.R);
        atomicAdd(g.f[4] + node, w * rate[0]);
        atomicAdd(g.f[5] + node, w * rate[1]);
        atomicAdd(g.f[6] + node, w * rate[2]);
    }
}

// The scatter records of a block's warps: one array per kernel, whichever bodies it holds. (Declared in
// an inlined function, not passed in: through a reference the compiler may not see that it is shared
// memory and issue generic loads, stores and atomics.)
template <int kWarps>
__device__ __forceinline__ ScalarRecord<4>* warp_records() {
    __shared__ ScalarRecord<4> records[kWarps];
    return records;
}

template <bool kRef = false, int kBlock = kOwnerThreads>
__device__ __forceinline__ void surface_owners_run_body(Arg<Params, kRef> P, Arg<BkState, kRef> in,
                                                         Arg<BkConstants, kRef> cst, Arg<BkSurface, kRef> sf,
                                                         Arg<GridPtrs, kRef> g, int32_t* sim_flags, Slot sl) {
    ScalarRecord<4>* sm = warp_records<kBlock / 32>();
    const int64_t o = sl.block * (int64_t)kBlock + threadIdx.x;
    const bool mine = o < sf.owner_count;
    bool valid = false;
    Stencil st;
    st.b[0] = st.b[1] = st.b[2] = 0;
    double rate[3] = {0.0, 0.0, 0.0}, exposed, contact;
    const int p = mine ? sf.owners[o] : 0;
    OwnerState os;
    if (mine) os = owner_state(P, in, cst, p);
    // (the faces' areas pass through the warp's scatter record before it is filled)
    owner_areas_warp(sf, reinterpret_cast<FaceChunk&>(sm[threadIdx.x >> 5]), o, mine, exposed, contact);
    if (mine) {
        owner_rates(P, os, cst, exposed, contact, rate);
        owner_store(sf, o, p, rate);
        st = make_stencil(os.x, P.origin, P.dx, P.R, P.rec_dx);
        valid = st.valid;
        if (!valid) set_flag(sim_flags, 1);
    }
    // the owners' nodes lie inside the particles' transport box: no box to widen
    scatter_scalars<3>(reinterpret_cast<ScalarRecord<3>&>(sm[threadIdx.x >> 5]), valid, st, rate, {g.f[4], g.f[5], g.f[6]}, P.R,
                       group_lanes(P.n, P.R));
}

// Many owners take the run form (one thread each), few the warp form (one warp each).
template <bool kRef = false>
__device__ __forceinline__ void surface_owners_body(Arg<Params, kRef> P, Arg<BkState, kRef> in, Arg<BkConstants, kRef> cst,
                                                    Arg<BkSurface, kRef> sf, Arg<GridPtrs, kRef> g, int32_t* sim_flags,
                                                    bool in_runs, Slot sl) {
    if (in_runs) surface_owners_run_body<kRef>(P, in, cst, sf, g, sim_flags, sl);
    else surface_owners_warp_body<kRef>(P, in, cst, sf, g, sim_flags, sl);
}

// Whether a body with `owners` face owners among `n` particles takes the run form, and its blocks.
inline bool owners_in_runs(int64_t owners, int64_t n) { return owners * 16 >= n; }
inline unsigned owner_blocks(int64_t owners, int64_t n) {
    const int64_t threads = owners_in_runs(owners, n) ? owners : owners * 32;
    return (unsigned)((threads + kOwnerThreads - 1) / kOwnerThreads);
}

__global__ void __launch_bounds__(kOwnerThreads) k_surface_owners(Params P, BkState in, BkConstants cst, BkSurface sf,
                                                                 GridPtrs g, int32_t* sim_flags, int in_runs) {
    pdl_enter();
    surface_owners_body(P, in, cst, sf, g, sim_flags, in_runs != 0, grid_slot());
}

// ---------------------------------------------------------- transport P2G
// physics/thermal_water.py:108-137 (volume, capacity, energy, water) by warp runs (bk_scatter.cuh),
// with the node box of the substep.
using ScatterRecord = ScalarRecord<4>;

// Asks L2 for the lines that the warp's particles read in the scatter.
__device__ __forceinline__ void scatter_prefetch(const Params& P, const BkState& in, const BkConstants& cst, int block) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = block * (int64_t)kOwnerThreads + (threadIdx.x & ~31);
    if (w0 >= P.n) return;
    if (lane < 12) prefetch_l2((lane < 3 ? in.x + lane * P.pitch : in.F + (lane - 3) * P.pitch) + w0);
    else if (lane == 12) prefetch_l2(cst.volume + w0);
    else if (lane < 19) {
        const double* a = lane < 15 ? cst.capacity : lane < 17 ? in.temperature : in.water;
        const int64_t half = w0 + 16 * ((lane - 13) & 1);
        prefetch_l2(a + (half < P.n ? half : w0));
    }
}

template <bool kRef = false>
__device__ __forceinline__ void transport_scatter_body(Arg<Params, kRef> P, Arg<BkState, kRef> in,
                                                       Arg<BkConstants, kRef> cst, Arg<GridPtrs, kRef> g, int32_t* sim_flags,
                                                       Slot sl) {
    ScatterRecord* sm = warp_records<kOwnerThreads / 32>();
    const int64_t i = sl.block * (int64_t)kOwnerThreads + threadIdx.x;
    const int64_t pitch = P.pitch;
    bool valid = false;
    Stencil st;
    st.b[0] = st.b[1] = st.b[2] = 0;
    double val[4] = {0.0, 0.0, 0.0, 0.0};
    if (i < P.n) {
        st = make_stencil(load_v3(in.x, i, pitch), P.origin, P.dx, P.R, P.rec_dx);
        valid = st.valid;
        if (!valid) set_flag(sim_flags, 1);
    }
    if (valid) {
        double cap = cst.capacity[i];
        val[0] = (double)cst.volume[i] * (double)det3(load_m3(in.F, i, pitch));
        val[1] = cap;
        val[2] = cap * in.temperature[i];
        val[3] = in.water[i];
    }
    widen_box(g.bounds, valid, st.b);
    scatter_scalars<4>(sm[threadIdx.x >> 5], valid, st, val, {g.f[0], g.f[1], g.f[2], g.f[3]}, P.R,
                       group_lanes(P.n, P.R));
}

__global__ void __launch_bounds__(kOwnerThreads, 8) k_transport_scatter(Params P, BkState in, BkConstants cst, GridPtrs g,
                                                               int32_t* sim_flags) {
    scatter_prefetch(P, in, cst, (int)blockIdx.x);
    pdl_enter();
    transport_scatter_body(P, in, cst, g, sim_flags, grid_slot());
}

// Two bodies in one launch: `first` blocks of one spread evenly among the blocks of the other, so that
// both are resident together from the start (placed in front, the surface vertices' blocks filled the
// SMs for 2.5 waves before the first scatter block ran, and nothing overlapped).
struct Mixed {
    bool is_first;
    int block;
};
__device__ __forceinline__ Mixed mixed_block(int first) {
    const long long b = blockIdx.x, total = gridDim.x;
    const int before = (int)(b * first / total), after = (int)((b + 1) * first / total);
    return after > before ? Mixed{true, before} : Mixed{false, (int)b - before};
}

// The surface vertices and the transport scatter of one substep: both read only the state. The
// vertices' blocks are chains of dependent gathers that leave the SMs' issue slots free. kBlock is the block
// of k_surface_vertices that sums the same bits; that of 256 threads is taken by half as many.
template <int kBlock>
__global__ void __launch_bounds__(kOwnerThreads, 8) k_vertices_scatter(Params P, BkState in, BkConstants cst, BkSurface sf,
                                                              GridPtrs g, int32_t* sim_flags, int vertex_blocks) {
    constexpr int kParts = kBlock / kOwnerThreads > 1 ? kBlock / kOwnerThreads : 1;
    static_assert(vertex_launch_threads(kBlock / kParts) == kOwnerThreads, "both bodies share the block size");
    const Mixed m = mixed_block(vertex_blocks);
    if (!m.is_first) scatter_prefetch(P, in, cst, m.block);
    pdl_enter();
    if (m.is_first) surface_vertices_body<kBlock / kParts, false, kParts>(P, in.x, in.F, sf, Slot{m.block, vertex_blocks});
    else transport_scatter_body(P, in, cst, g, sim_flags, Slot{m.block, (int)gridDim.x - vertex_blocks});
}

// The owners of a fine mesh and the transport scatter, after the vertices.
__global__ void __launch_bounds__(kOwnerThreads, 8) k_owners_scatter(Params P, BkState in, BkConstants cst, BkSurface sf,
                                                            GridPtrs g, int32_t* sim_flags, int owner_blocks) {
    const Mixed m = mixed_block(owner_blocks);
    if (!m.is_first) scatter_prefetch(P, in, cst, m.block);
    pdl_enter();
    if (m.is_first) surface_owners_run_body(P, in, cst, sf, g, sim_flags, Slot{m.block, owner_blocks});
    else transport_scatter_body(P, in, cst, g, sim_flags, Slot{m.block, (int)gridDim.x - owner_blocks});
}

// ------------------------------------------------------------ grid passes
// Node box [lo, hi] of `bounds` clipped to the grid; false when it is empty. The empty box is
// stored as lo = INT_MAX, hi = INT_MIN, so emptiness is tested before any subtraction.
__device__ __forceinline__ bool box_of(const int* bounds, int R, int lo[3], int ext[3], int64_t& count) {
    count = 1;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        int l = bounds[a], h = bounds[3 + a];
        if (l > h) return false;
        l = max(l, 0);
        h = min(h, R - 1);
        if (l > h) return false;
        lo[a] = l;
        ext[a] = h - l + 1;
        count *= ext[a];
    }
    return true;
}

// physics/thermal_water.py:140-190: node temperature/saturation (GridFields) and the 7-point flux
// (DiffuseGrid) over the active box, tiled through shared memory. A block takes a tile of
// kDiffX x kDiffY x kDiffZ nodes (z fastest, one warp per z row) and first stages the tile plus a
// one-node halo: for each staged node with capacity it forms T = E / C and s = W / (rho_w V) once,
// keeping V, T, s and the capacity test in shared memory. The six-neighbour stencil then reads only
// shared memory, so each node's fields are read from L2/HBM about (1 + halo) times instead of seven,
// and each node's two float64 divisions run once instead of once per neighbour.
constexpr int kDiffX = 2, kDiffY = 4, kDiffZ = 32;
constexpr int kDiffThreads = kDiffX * kDiffY * kDiffZ;
constexpr int kHaloX = kDiffX + 2, kHaloY = kDiffY + 2, kHaloZ = kDiffZ + 2;
constexpr int kHaloNodes = kHaloX * kHaloY * kHaloZ;

struct DiffuseSmem {
    double V[kHaloNodes], T[kHaloNodes], S[kHaloNodes];
    unsigned char ok[kHaloNodes];
};

template <bool kRef = false>
__device__ __forceinline__ void diffuse_body(Arg<Params, kRef> P, Arg<GridPtrs, kRef> g, int32_t* errors,
                                             Slot sl) {
    __shared__ DiffuseSmem sm;
    double* s_V = sm.V;
    double* s_T = sm.T;
    double* s_S = sm.S;
    unsigned char* s_ok = sm.ok;
    int lo[3], ext[3];
    int64_t count;
    // The node box of the transport fields: built by this substep's scalar P2G, or by the previous
    // substep's G2P when it scattered them ahead.
    if (!box_of(P.prescattered ? g.bounds + 12 : g.bounds, P.R, lo, ext, count)) return;
    const int R = P.R;
    const double rho_w = (double)P.water_density;
    const double rec_cell = 1.0 / (double)(P.dx * P.dx * P.dx);
    const double kc = (double)(P.conductivity * P.dx);
    const double kw = (double)(P.diffusivity * P.water_density * P.dx);
    const double dt = (double)P.dt;
    const int tiles_z = (ext[2] + kDiffZ - 1) / kDiffZ, tiles_y = (ext[1] + kDiffY - 1) / kDiffY;
    const int tiles_x = (ext[0] + kDiffX - 1) / kDiffX;
    const int tiles = tiles_x * tiles_y * tiles_z;
    const int tid = threadIdx.x;
    const int tz = tid % kDiffZ, ty = (tid / kDiffZ) % kDiffY, tx = tid / (kDiffZ * kDiffY);
    for (int tile = sl.block; tile < tiles; tile += sl.blocks) {
        const int t0[3] = {lo[0] + (tile / (tiles_z * tiles_y)) * kDiffX, lo[1] + ((tile / tiles_z) % tiles_y) * kDiffY,
                           lo[2] + (tile % tiles_z) * kDiffZ};
        // Stage the tile and its halo (nodes outside the grid are marked empty, like the reference's
        // range test; nodes outside the box but inside the grid hold zero fields).
        for (int h = tid; h < kHaloNodes; h += kDiffThreads) {
            const int hz = h % kHaloZ, hy = (h / kHaloZ) % kHaloY, hx = h / (kHaloZ * kHaloY);
            const int c0 = t0[0] + hx - 1, c1 = t0[1] + hy - 1, c2 = t0[2] + hz - 1;
            bool ok = c0 >= 0 && c0 < R && c1 >= 0 && c1 < R && c2 >= 0 && c2 < R;
            double V = 0.0, T = 0.0, S = 0.0;
            if (ok) {
                const int64_t j = node_index(c0, c1, c2, R);
                const double cj = g.f[1][j], Ej = g.f[2][j], Wj = g.f[3][j];  // independent loads
                V = g.f[0][j];
                ok = cj > 0.0;
                if (ok) {
                    T = Ej * reciprocal_newton(cj);
                    S = Wj * reciprocal_newton(rho_w * V);
                }
            }
            s_V[h] = V;
            s_T[h] = T;
            s_S[h] = S;
            s_ok[h] = ok;
        }
        __syncthreads();
        const int c[3] = {t0[0] + tx, t0[1] + ty, t0[2] + tz};
        const int h = ((tx + 1) * kHaloY + (ty + 1)) * kHaloZ + (tz + 1);
        if (c[0] < lo[0] + ext[0] && c[1] < lo[1] + ext[1] && c[2] < lo[2] + ext[2]) {
            const int64_t i = node_index(c[0], c[1], c[2], R);
            if (!s_ok[h]) {
                g.dTr[i] = make_double2(0.0, 0.0);
            } else {
                const double ci = g.f[1][i], Wi = g.f[3][i];
                const double vi = s_V[h], Ti = s_T[h], si = s_S[h];
                const double rec_water = P.water_enabled ? reciprocal_newton(rho_w * vi) : 0.0;
                double heat_rate = g.f[4][i], water_rate = -g.f[5][i], heat_diag = g.f[6][i], water_diag = 0.0;
                const int stride[3] = {kHaloY * kHaloZ, kHaloZ, 1};
#pragma unroll
                for (int axis = 0; axis < 3; ++axis)
#pragma unroll
                    for (int side = 0; side < 2; ++side) {
                        const int hj = h + (2 * side - 1) * stride[axis];
                        if (!s_ok[hj]) continue;
                        const double vj = s_V[hj], Tj = s_T[hj];
                        const double fill = 2.0 * vi * vj * reciprocal_newton(vi + vj) * rec_cell;
                        const double hc = kc * fill;
                        heat_rate += hc * (Tj - Ti);
                        heat_diag += hc;
                        if (P.water_enabled) {
                            const double sj = s_S[hj];
                            const double mob = kw * fill * 0.5 * (Ti + Tj) * 0.5 * (si + sj);
                            water_rate += mob * (sj - si);
                            water_diag += mob * rec_water;
                        }
                    }
                if (dt * heat_diag > ci) set_flag(errors, 0);
                const double change = dt * water_rate;
                if (Wi + change < 0.0 || dt * water_diag > 1.0) set_flag(errors, 1);
                const double dT = dt * heat_rate * reciprocal_newton(ci);
                g.dTr[i] = make_double2(dT, Wi > 0.0 ? change * reciprocal_newton(Wi) : 0.0);
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kDiffThreads) k_diffuse(Params P, GridPtrs g, int32_t* errors) {
    pdl_enter();
    diffuse_body(P, g, errors, grid_slot());
}

// Fields scattered ahead for a substep that runs its own scalar P2G instead (the state may have
// changed in between): zero the volume, capacity, energy and water fields over their box.
template <bool kRef = false>
__device__ __forceinline__ void clear_prescatter_body(Arg<Params, kRef> P, Arg<GridPtrs, kRef> g, Slot sl) {
    int lo[3], ext[3];
    int64_t count;
    if (!box_of(g.bounds + 12, P.R, lo, ext, count)) return;
    for (int64_t t = sl.block * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)sl.blocks * blockDim.x) {
        int c2 = lo[2] + (int)(t % ext[2]);
        int c1 = lo[1] + (int)((t / ext[2]) % ext[1]);
        int c0 = lo[0] + (int)(t / ((int64_t)ext[2] * ext[1]));
        int64_t i = node_index(c0, c1, c2, P.R);
#pragma unroll
        for (int k = 0; k < 4; ++k) g.f[k][i] = 0.0;
    }
}

__global__ void k_clear_prescatter(Params P, GridPtrs g) {
    pdl_enter();
    clear_prescatter_body(P, g, grid_slot());
}

// GridState.Clear (physics/grid.py:14-17) restricted to the previous substep's active box, the only
// nodes holding nonzero momentum, mass or velocity; the grid of the last substep stays readable
// until the next one starts.
template <bool kRef = false>
__device__ __forceinline__ void clear_previous_body(Arg<Params, kRef> P, Arg<GridPtrs, kRef> g, Slot sl) {
    int lo[3], ext[3];
    int64_t count;
    if (!box_of(g.bounds + 6, P.R, lo, ext, count)) return;
    for (int64_t t = sl.block * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)sl.blocks * blockDim.x) {
        int c2 = lo[2] + (int)(t % ext[2]);
        int c1 = lo[1] + (int)((t / ext[2]) % ext[1]);
        int c0 = lo[0] + (int)(t / ((int64_t)ext[2] * ext[1]));
        int64_t i = node_index(c0, c1, c2, P.R);
        g.pm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        g.v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

__global__ void k_clear_previous(Params P, GridPtrs g) {
    pdl_enter();
    clear_previous_body(P, g, grid_slot());
}

// Both node-box passes between the transport scatter and P2G in one launch (they touch different
// fields), when nothing on the host stands between the phases.
__global__ void __launch_bounds__(kDiffThreads) k_diffuse_clear(Params P, GridPtrs g, int32_t* errors) {
    pdl_enter();
    clear_previous_body(P, g, grid_slot());
    diffuse_body(P, g, errors, grid_slot());
}

// physics/grid.py:20-38 over the active box; clears the transport scatter fields behind it.
template <bool kRef = false>
__device__ __forceinline__ void grid_update_body(Arg<Params, kRef> P, Arg<GridPtrs, kRef> g, Slot sl) {
    int lo[3], ext[3];
    int64_t count;
    // The G2P that follows builds the next substep's transport box in bounds[12..17]: restart it
    // empty (this substep's diffusion, its only reader, has finished; no block here reads it).
    if (P.prescatter_next && sl.block == 0 && threadIdx.x < 6) g.bounds[12 + threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    if (!box_of(g.bounds, P.R, lo, ext, count)) return;
    const int R = P.R, bc = P.bc;
    for (int64_t t = sl.block * (int64_t)blockDim.x + threadIdx.x; t < count; t += (int64_t)sl.blocks * blockDim.x) {
        int c[3];
        c[2] = lo[2] + (int)(t % ext[2]);
        c[1] = lo[1] + (int)((t / ext[2]) % ext[1]);
        c[0] = lo[0] + (int)(t / ((int64_t)ext[2] * ext[1]));
        int64_t i = node_index(c[0], c[1], c[2], R);
        float4 pm = g.pm[i];
        float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
        if (pm.w > 0.0f) {
            float vel[3] = {pm.x / pm.w + P.dt * P.gravity[0], pm.y / pm.w + P.dt * P.gravity[1],
                            pm.z / pm.w + P.dt * P.gravity[2]};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (c[a] < bc && vel[a] < 0.0f) vel[a] = 0.0f;
                if (c[a] >= R - bc && vel[a] > 0.0f) vel[a] = 0.0f;
            }
            out = make_float4(vel[0], vel[1], vel[2], 0.f);
        }
        g.v[i] = out;
        if (P.transport && !P.keep_fields) {
#pragma unroll
            for (int k = 0; k < 7; ++k) g.f[k][i] = 0.0;
        }
    }
}

__global__ void k_grid_update(Params P, GridPtrs g) {
    pdl_enter();
    grid_update_body(P, g, grid_slot());
}

// ------------------------------------------------------------- fused P2G
// Scalar G2P (thermal_water.py:206-229), local gas source (:238-245), gas stress (gas.py:16-35),
// water stress (thermal_water.py:248-253) and momentum P2G (transfer.py:47-70) for one particle
// per thread, then the momentum scatter by warp runs (bk_scatter.cuh). Bound by the LSU data pipe
// (70% of its peak at 1M particles: the run loop's broadcasts and the node gather) and by the loads'
// latency behind it. Loads are plain: staging the block's planes by bulk copies (33 KB and two
// barriers a block) took 87.0 us where this form, with its L2 prefetch and no barrier, takes 82.
// Blocks of 128 against 256: 81.8 and 84.2 us at 1M particles (a finished block's slot is refilled
// earlier). The merge of a block's sums (bk_scatter.cuh) and its barriers come on top.
constexpr int kP2GThreads = 128;
// Bodies of at most this many particles are one block, whose warps send their sums in step after a
// barrier: the atomics of a node leave one SM in the same order each time, and a run repeats bit for bit
// (160 runs of a 192-particle body; with two blocks of 128, or without the barrier, 1 in 8 differed, and
// finite differences of such a body carried that noise). The time is the same (17 us).
constexpr int kP2GSmall = 256;

constexpr int p2g_threads(Sums sums) { return sums == Sums::kAlone ? kP2GSmall : kP2GThreads; }
inline Sums p2g_sums(int64_t n) { return n <= kP2GSmall ? Sums::kAlone : n < kKeptParticles ? Sums::kTiles : Sums::kKept; }

template <Sums kSums, bool kRef = false>
__device__ __forceinline__ void p2g_body(Arg<Params, kRef> P, Arg<BkState, kRef> in, Arg<BkState, kRef> out,
                                         Arg<BkConstants, kRef> cst, Arg<GridPtrs, kRef> g, Arg<BkFlags, kRef> flags,
                                         float* max_residuals, Slot sl) {
    constexpr int kBlock = p2g_threads(kSums);
    __shared__ MomentumRecord sm[kBlock / 32];
    WarpTiles* tiles = nullptr;
    if constexpr (kSums == Sums::kTiles) tiles = warp_tiles();
    const int64_t i = sl.block * (int64_t)kBlock + threadIdx.x;
    const int64_t pitch = P.pitch;
    {
        // v, C, F and tau planes by lane, then the scalars' lines (two per float64 array)
        const int lane = threadIdx.x & 31;
        const int64_t w0 = i - lane;
        if (w0 < P.n) {
            if (lane < (P.material == 1 ? 30 : 21)) {
                const float* a = lane < 3 ? in.v + lane * pitch : lane < 12 ? in.C + (lane - 3) * pitch
                                 : lane < 21 ? in.F + (lane - 12) * pitch : in.tau + (lane - 21) * pitch;
                prefetch_l2(a + w0);
            }
            if (P.transport && lane < 8) {
                const double* a = lane < 2 ? in.temperature : lane < 4 ? in.water : lane < 6 ? cst.dry_mass : in.gas_moles;
                if (lane < 6 || P.gas) prefetch_l2(a + (w0 + 16 * (lane & 1) < P.n ? w0 + 16 * (lane & 1) : w0));
            }
            if (lane == 8) prefetch_l2(cst.volume + w0);
            if (lane == 9 && P.material == 1 && P.gas) prefetch_l2(in.porosity + w0);
            if (lane == 10 && P.gas && cst.gas_rate_per_particle) prefetch_l2(cst.gas_rate + w0);
            if (lane >= 11 && lane < 14) prefetch_l2(in.x + (lane - 11) * pitch + w0);
        }
    }
    if constexpr (!kRef) pdl_enter();
    if (sl.block == 0 && threadIdx.x < 2) max_residuals[threadIdx.x] = 0.0f;
    bool valid = false;
    Stencil st;
    st.b[0] = st.b[1] = st.b[2] = 0;
    if (i < P.n) {
        st = make_stencil(load_v3(in.x, i, pitch), P.origin, P.dx, P.R, P.rec_dx);
        valid = st.valid;
        if (!valid) set_flag(flags.simulation, 1);
    }
    if (!P.box_widened) widen_box(g.bounds, valid, st.b);
    float mass = 0.f, q[3] = {0.f, 0.f, 0.f}, A[9] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (valid) {
        M3 F = load_m3(in.F, i, pitch);
        float J = det3(F);
        M3 tau;
        float T_mat = 0.f;
        float rho_ref = P.density;
        double sat = 0.0, N = 0.0, T_new = 0.0, W_new = 0.0;
        if (P.transport) {
            // The scalar G2P of the diffused node fields (thermal_water.py:206-215).
            double dTp, ratio;
            gather_scalars(st, g.dTr, P.R, dTp, ratio);
            double T_old = in.temperature[i];
            double Tn = T_old + dTp;
            double Wn = in.water[i] * (1.0 + ratio);
            double dry = cst.dry_mass[i];
            float V0 = cst.volume[i];
            T_new = Tn;
            W_new = Wn;
            mass = (float)(dry + Wn);
            rho_ref = (float)((dry + Wn) / (double)V0);
            sat = Wn / ((double)P.water_density * (double)V0 * (double)J);
            T_mat = (float)Tn;
            if (P.gas) {
                N = in.gas_moles[i];
                if (!P.settling) {
                    double Tm = 0.5 * (T_old + Tn);
                    double z = (Tm - (double)P.peak) / (double)P.width;
                    N += (double)(P.dt * P.density) * (double)cst.gas_rate[cst.gas_rate_per_particle ? i : 0] * exp(-(z * z));
                }
            }
        } else {
            mass = cst.mass[i];
            if (P.material == 1) T_mat = in.material_temperature[i];
        }
        if (P.material == 1) {
            tau = load_m3(in.tau, i, pitch);
            if (P.gas) {
                float n = in.porosity[i];
                if (n <= 0.0f || n >= 1.0f || !isfinite(n) || J <= 0.0f) {
                    set_flag(flags.ding, 0);
                } else {
                    float p = (float)gas_pressure(N, T_mat, J, n);
                    float iso = J * (P.ambient - p);
#pragma unroll
                    for (int e = 0; e < 9; ++e) tau.m[e] += (e % 4) == 0 ? iso : iso * 0.0f;
                    float bulk = p * (1.0f + (1.0f - P.ding.initial_porosity + n) / n);
                    float wave = sqrtf((P.elastic_modulus + bulk) * J / rho_ref);
                    if (!isfinite(p) || wave * P.dt / P.dx > P.cfl) set_flag(flags.ding, 2);
                }
            }
        } else {
            if (!isfinite(J) || J <= 0.0f) {
                set_flag(flags.simulation, 0);
#pragma unroll
                for (int e = 0; e < 9; ++e) tau.m[e] = 0.0f;
            } else {
                float lj = logf(J);
#pragma unroll
                for (int r = 0; r < 3; ++r)
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        float ffT = F.m[3 * r] * F.m[3 * c] + F.m[3 * r + 1] * F.m[3 * c + 1] + F.m[3 * r + 2] * F.m[3 * c + 2];
                        float id = r == c ? 1.0f : 0.0f;
                        tau.m[3 * r + c] = P.ding.mu * (ffT - id) + P.ding.lam * lj * id;
                    }
            }
        }
        if (P.transport) {
            float iso = J * P.water_stress * ((float)sat - P.s0);
#pragma unroll
            for (int e = 0; e < 9; ++e) tau.m[e] -= (e % 4) == 0 ? iso : iso * 0.0f;
        }
        float scale = P.dt * cst.volume[i] * 4.0f / (P.dx * P.dx);
        M3 Cm = load_m3(in.C, i, pitch);
        V3 vel = load_v3(in.v, i, pitch);
        if (P.transport) {  // after the loads, which the compiler may not move over a store
            out.temperature[i] = T_new;
            out.water[i] = W_new;
            if (P.gas) out.gas_moles[i] = N;
        }
#pragma unroll
        for (int e = 0; e < 9; ++e) A[e] = mass * Cm.m[e] - scale * tau.m[e];
        // w (m v + A (o - l) dx) = w (q + A dx o) with q = m v - A l dx.
#pragma unroll
        for (int r = 0; r < 3; ++r)
            q[r] = mass * vel.v[r] - (A[3 * r] * st.l[0] + A[3 * r + 1] * st.l[1] + A[3 * r + 2] * st.l[2]) * P.dx;
#pragma unroll
        for (int e = 0; e < 9; ++e) A[e] *= P.dx;
    }
    if constexpr (kSums == Sums::kAlone) __syncthreads();  // the warps send their sums in step (kP2GSmall)
    scatter_momentum<kSums>(sm, tiles, valid, st, mass, q, A, g.pm, P.R, group_lanes(P.n, P.R), P.R <= 1024);
}

template <Sums kSums, bool kLoaf = false>
__global__ void __launch_bounds__(p2g_threads(kSums), kSums == Sums::kKept ? 8 : 4) k_p2g(Params P, BkState in, BkState out, BkConstants cst, GridPtrs g,
                                                 BkFlags flags, float* max_residuals) {
    if constexpr (kLoaf) fix_loaf_mode(P);
    p2g_body<kSums>(P, in, out, cst, g, flags, max_residuals, grid_slot());
}

// ------------------------------------------------------ fused G2P + return
// The largest positive value over the warp's active lanes into *addr (nonnegative floats order as
// their bit patterns): one atomic per warp instead of one per lane on the same address.
__device__ __forceinline__ void atomic_max_nonneg(float* addr, float value) {
    const unsigned mask = __activemask();
    const int v = (int)__reduce_max_sync(mask, (unsigned)__float_as_int(value > 0.0f ? value : 0.0f));
    if (v > 0 && (int)(threadIdx.x & 31) == __ffs(mask) - 1) atomicMax(reinterpret_cast<int*>(addr), v);
}

// G2P of one particle (transfer.py:73-109): writes x', v', C', F' and returns F', C'. False (and the
// stencil flag) when the stencil leaves the grid.
// v = sum w v_i and C = 4/dx^2 sum w v_i (o_i - l) dx, accumulated as the moments
// S = sum w v_i and M_c = sum w v_i o_ic with the stencil offsets o_i in {0, 1, 2} known at compile
// time; C_rc = 4/dx (M_rc - l_c S_r).
__device__ __forceinline__ bool g2p_gather(const Params& P, const BkState& in, const BkState& out, const GridPtrs& g,
                                           const BkFlags& flags, int64_t i, M3& Fn, M3& Cn) {
    const int64_t pitch = P.pitch;
    V3 xi = load_v3(in.x, i, pitch);
    Stencil st = make_stencil(xi, P.origin, P.dx, P.R, P.rec_dx);
    if (!st.valid) { set_flag(flags.simulation, 1); return false; }
    float nv[3], mo[9];
    gather_velocity(st, g.v, P.R, nv, mo);
    float nc[9];
    const float kdx = 4.0f / P.dx;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) nc[3 * r + c] = kdx * (mo[3 * r + c] - st.l[c] * nv[r]);
    M3 F = load_m3(in.F, i, pitch);
    M3 G;
#pragma unroll
    for (int e = 0; e < 9; ++e) {
        Cn.m[e] = nc[e];
        G.m[e] = P.dt * nc[e] + ((e % 4) == 0 ? 1.0f : 0.0f);
    }
    Fn = matmul(G, F);
    V3 vo{{nv[0], nv[1], nv[2]}}, xo{{xi.v[0] + P.dt * nv[0], xi.v[1] + P.dt * nv[1], xi.v[2] + P.dt * nv[2]}};
    store_v3(out.v, i, pitch, vo);
    store_m3(out.C, i, pitch, Cn);
    store_v3(out.x, i, pitch, xo);
    store_m3(out.F, i, pitch, Fn);
    return true;
}

__device__ __forceinline__ void ding_store(const Params& P, const BkState& out, const BkDiagnostics& diag, int64_t i,
                                           float T, const DingParticleOut& o) {
    const int64_t pitch = P.pitch;
    store_m3(out.Fe, i, pitch, o.Fe);
    store_m3(out.tau, i, pitch, o.tau);
    out.porosity[i] = o.porosity;
    out.gelled[i] = o.gelled;
    if (!P.transport) out.material_temperature[i] = T;
    if (diag.plastic_gradients) store_m3(diag.plastic_gradients, i, pitch, o.Fp);
    if (diag.return_residuals) diag.return_residuals[i] = o.residual;
    if (diag.porosity_residuals) diag.porosity_residuals[i] = o.porosity_residual;
    atomic_max_nonneg(diag.max_residuals, o.residual);
    atomic_max_nonneg(diag.max_residuals + 1, o.porosity_residual);
}

// ------------------------------------------------------ return-map surrogate
struct SurrogateDev {
    const unsigned char* blob;
    float in_mean[8], in_scale[8], in_rec[8], in_low[8], in_high[8], out_scale[4];  // in_rec = 1 / in_scale
    float* samples;
    int32_t* sample_count;
    int sample_capacity, sample_stride, sample_offset;
    float* judge_error;
    int judge_stride;
    int32_t* path_counts;
};

SurrogateDev surrogate_dev(const BkReturnSurrogate* r) {
    SurrogateDev d{};
    if (!r) return d;
    d.blob = static_cast<const unsigned char*>(r->packed);
    for (int k = 0; k < 8; ++k) {
        d.in_mean[k] = r->norm.in_mean[k];
        d.in_scale[k] = r->norm.in_scale[k] != 0.0f ? r->norm.in_scale[k] : 1.0f;
        d.in_rec[k] = 1.0f / d.in_scale[k];
        d.in_low[k] = r->in_low[k];
        d.in_high[k] = r->in_high[k];
    }
    for (int k = 0; k < 4; ++k) d.out_scale[k] = r->norm.out_scale[k];
    d.samples = r->samples;
    d.sample_count = r->sample_count;
    d.sample_capacity = r->sample_capacity;
    d.sample_stride = r->sample_stride > 0 ? r->sample_stride : 1;
    d.sample_offset = r->sample_offset;
    d.judge_error = r->judge_error;
    d.judge_stride = r->judge_stride;
    d.path_counts = r->path_counts;
    return d;
}

// Singular-value order (descending) the network sees, from the values or their logs.
__device__ __forceinline__ void order3(const float* s, int* perm) {
    int a = 0, b = 1, c = 2, t;
    if (s[a] < s[b]) { t = a; a = b; b = t; }
    if (s[b] < s[c]) { t = b; b = c; c = t; }
    if (s[a] < s[b]) { t = a; a = b; b = t; }
    perm[0] = a; perm[1] = b; perm[2] = c;
}

// The 7 raw network inputs of a particle: sorted log singular values of the trial elastic
// gradient, effective temperature, water saturation, gas content, plastic volume strain.
__device__ __forceinline__ void surrogate_features(const Params& P, const BkState& out, const BkConstants& cst,
                                                   int64_t i, const DingPrelude& d, float por, float J,
                                                   const int* perm, float* f) {
#pragma unroll
    for (int k = 0; k < 3; ++k) f[k] = pick3(d.e, perm[k]);
    f[3] = d.T_eff;
    f[4] = P.transport ? (float)(out.water[i] * reciprocal_newton((double)P.water_density * (double)cst.volume[i] * (double)J))
                       : 0.0f;
    f[5] = P.gas ? (float)out.gas_moles[i] : 0.0f;
    f[6] = logf(1.0f - P.ding.initial_porosity + por);
}

// True when the exact return map leaves the particle elastic (no overstress solve): the cheap
// path for which the exact map runs unchanged.
__device__ __forceinline__ bool ding_elastic(const DingParamsDev& D, const DingPrelude& d, float por) {
    const float* st = d.e;
    float tr = st[0] + st[1] + st[2];
    float ts[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) ts[k] = 2.0f * D.mu * st[k] + D.lam * tr;
    float mean = (ts[0] + ts[1] + ts[2]) / 3.0f;
    float dev[3] = {ts[0] - mean, ts[1] - mean, ts[2] - mean};
    if (D.coupled_porosity) {
        const double trial = 1.0 - (double)D.initial_porosity + (double)por - 1.0 + (double)D.initial_porosity;
        const int side = particle_side(1.5f * (dev[0] * dev[0] + dev[1] * dev[1] + dev[2] * dev[2]), mean, d.ty, trial);
        if (side != 0) return side < 0;
    }
    float ty2 = d.ty * d.ty;
    float q = 1.5f * (dev[0] * dev[0] + dev[1] * dev[1] + dev[2] * dev[2]) / ty2;
    float p = mean * mean / ty2;
    if (D.coupled_porosity) {
        // elastic trial porosity Vp - 1 + n0 with Vp = 1 - n0 + n, as in solve_porosity's early exit
        double trial = 1.0 - (double)D.initial_porosity + (double)por - 1.0 + (double)D.initial_porosity;
        if (trial > 0.0 && trial < 1.0) return (double)q + pressure_coefficient64(trial) * (double)p <= 1.0;
        return false;
    }
    return q + porosity_coefficient(por) * p <= 1.0f;
}

// Close the return from predicted log principal strains e (SVD order, before volume corrections):
// tau = U diag(2 mu dev(e) + K mean(e)) U^T, Fe = U exp(e) V^T; in gas mode the end-state porosity
// is the plastic volume change Vp exp(tr eps_trial - tr e) - 1 + n0. False when that porosity
// leaves (0, 1), in which case the caller runs the exact map.
__device__ bool ding_surrogate(const DingParamsDev& D, const DingPrelude& d, float por, const M3& F_tot,
                               const float* e, int32_t* flags, DingParticleOut& out, bool need_fp) {
    const float mu = D.mu, bulk = 2.0f * D.mu + 3.0f * D.lam;
    float ret_por = por;
    if (D.coupled_porosity) {
        double dv = (double)d.e[0] + (double)d.e[1] + (double)d.e[2] - ((double)e[0] + e[1] + e[2]);
        double rp = (1.0 - (double)D.initial_porosity + (double)por) * exp_small(dv) - 1.0 + (double)D.initial_porosity;
        if (!(rp > 0.0 && rp < 1.0)) return false;
        ret_por = (float)rp;
    }
    const float eb = div_uniform(e[0] + e[1] + e[2], 3.0f, 1.0f / 3.0f);
    float cs[3], ex[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        cs[k] = 2.0f * mu * (e[k] - eb) + bulk * eb;
        ex[k] = expf(e[k]);
    }
    const float* U = d.U.m;
    const float* V = d.V.m;
    M3 Fe, tau;
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            Fe.m[3 * r + c] = (U[3 * r] * ex[0]) * V[3 * c] + (U[3 * r + 1] * ex[1]) * V[3 * c + 1] +
                              (U[3 * r + 2] * ex[2]) * V[3 * c + 2];
            tau.m[3 * r + c] = (U[3 * r] * cs[0]) * U[3 * c] + (U[3 * r + 1] * cs[1]) * U[3 * c + 1] +
                               (U[3 * r + 2] * cs[2]) * U[3 * c + 2];
        }
    if (!D.coupled_porosity && porosity_coefficient(por) == 0.0f) {
        float scale = cbrtf(d.det_trial / det3(Fe));
#pragma unroll
        for (int k = 0; k < 9; ++k) Fe.m[k] *= scale;
    }
    ding_close(D, por, FInRegs{F_tot}, ret_por, Fe, flags, out, need_fp);
    out.tau = tau;
    out.residual = 0.0f;
    out.porosity_residual = 0.0f;
    out.yield_stress = d.ty;
    out.viscosity = d.eta;
    out.gelled = d.gel;
#pragma unroll
    for (int k = 0; k < 3; ++k) out.e[k] = e[k];
    out.yielded = true;
    return true;
}

// Bound by instruction issue and fetch (1M elastic particles: 3,090 instructions a warp at 67% issue,
// the top stall no_instruction), so it is the instructions that every particle runs which count:
// divisions by launch constants are corrected products (div_uniform), an elastic particle is certified
// without the exact invariants, the plastic branch's float64 solve stands out of line, det F' is
// formed while F' is in registers, and the float64 special functions of the decomposition and the
// solves are Newton steps from float32 seeds. 1M elastic loaf 142 -> 120.5 us, 4M yielding 1037 -> 903.
// 8 blocks of 128 threads per SM (64 registers): the return map's dependent float64 chains are
// latency bound, so resident warps outweigh the spilled registers (measured at 3 to 12 blocks per
// SM: 8 is fastest for both elastic and yielding particles). With `sg.samples` set (harvest),
// yielding particles on the sampling stride append (features, return) rows.
__device__ __forceinline__ void g2p_return_particle(const Params& P, const BkState& in, const BkState& out,
                                                    const BkConstants& cst, const GridPtrs& g, const BkDiagnostics& diag,
                                                    const BkFlags& flags, const SurrogateDev& sg, int64_t i) {
    M3 Fn, Cn;
    if (!g2p_gather(P, in, out, g, flags, i, Fn, Cn)) return;
    if (P.material != 1) return;
    const int64_t pitch = P.pitch;
    const double det_F = P.ding.coupled_porosity ? det3_64(Fn) : 0.0;
    float T = P.transport ? (float)out.temperature[i] : in.material_temperature[i];
    const float por = in.porosity[i];
    DingPrelude d;
    if (!ding_prelude(P.ding, load_m3(in.Fe, i, pitch), por, in.gelled[i], Cn, T, __ldg(cst.viscosity_parameter),
                      flags.ding, d))
        return;
    DingParticleOut o;
    ding_exact(P.ding, d, por, FStored{out.F, i, pitch, det_F}, flags.ding, o, diag.plastic_gradients != nullptr);
    ding_store(P, out, diag, i, T, o);
    if (sg.samples && o.yielded && i % sg.sample_stride == sg.sample_offset) {
        int slot = atomicAdd(sg.sample_count, 1);
        if (slot < sg.sample_capacity) {
            int perm[3];
            order3(d.e, perm);
            float f[7];
            surrogate_features(P, out, cst, i, d, por, det3(FStored{out.F, i, pitch, 0.0}.get()), perm, f);
            float* row = sg.samples + (int64_t)slot * 12;
#pragma unroll
            for (int k = 0; k < 7; ++k) row[k] = f[k];
#pragma unroll
            for (int k = 0; k < 3; ++k) row[7 + k] = pick3(o.e, perm[k]) - f[k];
            row[10] = 0.0f;
            row[11] = 0.0f;
        }
    }
}

// Dynamic shared memory of the transport prescatter in k_g2p_return (128 particles per block).
constexpr size_t kG2PScatterBytes = 4 * sizeof(ScatterRecord);

template <bool kRef = false>
__device__ __forceinline__ void g2p_return_body(Arg<Params, kRef> P, Arg<BkState, kRef> in,
                                                Arg<BkState, kRef> out, Arg<BkConstants, kRef> cst, Arg<GridPtrs, kRef> g,
                                                Arg<BkDiagnostics, kRef> diag, Arg<BkFlags, kRef> flags, Arg<SurrogateDev, kRef> sg,
                                                Slot sl) {
    extern __shared__ __align__(16) unsigned char g2p_smem[];
    const int64_t i = sl.block * (int64_t)blockDim.x + threadIdx.x;
    {
        // F and Fe planes by lane, then the scalars' lines
        const int lane = threadIdx.x & 31;
        const int64_t w0 = i - lane;
        if (w0 < P.n) {
            if (lane < (P.material == 1 ? 18 : 9))
                prefetch_l2((lane < 9 ? in.F + lane * P.pitch : in.Fe + (lane - 9) * P.pitch) + w0);
            if (lane == 18 && P.material == 1) prefetch_l2(in.porosity + w0);
            if (lane == 19 && P.material == 1) prefetch_l2(in.gelled + w0);
            if (lane >= 20 && lane < 23) prefetch_l2(in.x + (lane - 20) * P.pitch + w0);
        }
    }
    if constexpr (!kRef) pdl_enter();
    if (sl.block == 0 && threadIdx.x < 6) {
        // This substep's box becomes the box the next substep clears; the active box restarts empty.
        g.bounds[6 + threadIdx.x] = g.bounds[threadIdx.x];
        g.bounds[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    }
    if (i < P.n) g2p_return_particle(P, in, out, cst, g, diag, flags, sg, i);
    if (P.prescatter_next) {
        // The next substep's scalar P2G (thermal_water.py:108-137) from the state just written:
        // x' and F' by this thread (read back with plain loads), T' and W' by this substep's P2G.
        // The grid update has zeroed the transport fields over this substep's box and restarted
        // the prescatter box bounds[12..17]. Uniform branch: every thread of the block scatters.
        ScatterRecord* sm = reinterpret_cast<ScatterRecord*>(g2p_smem);
        const int64_t pitch = P.pitch;
        bool valid = false;
        Stencil st;
        st.b[0] = st.b[1] = st.b[2] = 0;
        double val[4] = {0.0, 0.0, 0.0, 0.0};
        if (i < P.n) {
            const float* xs = out.x;
            const V3 x{{xs[i], xs[pitch + i], xs[2 * pitch + i]}};
            st = make_stencil(x, P.origin, P.dx, P.R, P.rec_dx);
            valid = st.valid;
            if (valid) {
                const double cap = cst.capacity[i];
                val[0] = (double)cst.volume[i] * (double)det3(FStored{out.F, i, pitch, 0.0}.get());
                val[1] = cap;
                val[2] = cap * out.temperature[i];
                val[3] = out.water[i];
            }
        }
        widen_box(g.bounds + 12, valid, st.b);
        scatter_scalars<4>(sm[threadIdx.x >> 5], valid, st, val, {g.f[0], g.f[1], g.f[2], g.f[3]}, P.R,
                       group_lanes(P.n, P.R));
    }
}

// kLoaf instances also fix whether the next substep's transport fields are scattered (kPrescatter).
template <bool kLoaf = false, bool kPrescatter = false>
__global__ void __launch_bounds__(128, 8) k_g2p_return(Params P, BkState in, BkState out, BkConstants cst, GridPtrs g,
                                                   BkDiagnostics diag, BkFlags flags, SurrogateDev sg) {
    if constexpr (kLoaf) {
        fix_loaf_mode(P);
        P.prescatter_next = kPrescatter;
        diag.plastic_gradients = diag.return_residuals = diag.porosity_residuals = nullptr;
        sg.samples = nullptr;
    }
    g2p_return_body(P, in, out, cst, g, diag, flags, sg, grid_slot());
}

// G2P + return map with the learned surrogate: a persistent CTA walks 128-particle tiles and
// evaluates the network for each on the tensor cores (bk_mlp.cuh), so the weights are staged,
// the tensor memory allocated and the mbarrier initialised once per CTA. Yielding particles inside
// the training range take the surrogate's return; all others (elastic, out of range, invalid
// porosity) the exact map. The trial gradient's SVD stops at float32 convergence (svd3f<false>):
// its float64 finishing sweep only matters at the reference's rounding level, far below the
// network's error.
template <bool kRef = false>
__device__ __forceinline__ void g2p_return_surrogate_body(Arg<Params, kRef> P, Arg<BkState, kRef> in, Arg<BkState, kRef> out,
                                                          Arg<BkConstants, kRef> cst, Arg<GridPtrs, kRef> g,
                                                          Arg<BkDiagnostics, kRef> diag, Arg<BkFlags, kRef> flags,
                                                          Arg<SurrogateDev, kRef> sg, Slot sl) {
    __shared__ mlp::TileSmem ts;
    __shared__ int s_counts[3];
    mlp::tile_setup(ts, sg.blob);
    if (threadIdx.x < 3) s_counts[threadIdx.x] = 0;
    if (sl.block == 0 && threadIdx.x < 6) {
        g.bounds[6 + threadIdx.x] = g.bounds[threadIdx.x];
        g.bounds[threadIdx.x] = threadIdx.x < 3 ? INT_MAX : INT_MIN;
    }
    __syncthreads();
    const int64_t pitch = P.pitch;
    uint32_t phase = 0;
    for (int64_t base = (int64_t)sl.block * 128; base < P.n; base += (int64_t)sl.blocks * 128) {
        const int64_t i = base + threadIdx.x;
        // the next tile's planes, while this one computes
        prefetch_planes(i + (int64_t)sl.blocks * 128, P.n, pitch, in.F, 9, in.Fe, P.material == 1 ? 9 : 0, in.x, 3);
        M3 Fn, Cn;
        bool ding = false, use_mlp = false;
        DingPrelude d;
        float T = 0.f, por = 0.f, x[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        int perm[3] = {0, 1, 2};
        if (i < P.n && g2p_gather(P, in, out, g, flags, i, Fn, Cn) && P.material == 1) {
            T = P.transport ? (float)out.temperature[i] : in.material_temperature[i];
            por = in.porosity[i];
            ding = ding_prelude<false>(P.ding, load_m3(in.Fe, i, pitch), por, in.gelled[i], Cn, T,
                                __ldg(cst.viscosity_parameter), flags.ding, d);
            if (ding && !ding_elastic(P.ding, d, por)) {
                order3(d.e, perm);
                float f[7];
                surrogate_features(P, out, cst, i, d, por, det3(Fn), perm, f);
                use_mlp = true;
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    use_mlp = use_mlp && f[k] >= sg.in_low[k] && f[k] <= sg.in_high[k];
                    x[k] = div_uniform(f[k] - sg.in_mean[k], sg.in_scale[k], sg.in_rec[k]);
                }
            }
        }
        float y[3] = {0.f, 0.f, 0.f};
        // A tile whose particles all take the exact map (elastic, or outside the training range)
        // skips the network; the barrier makes the decision uniform across the CTA.
        const bool any_mlp = __syncthreads_or(use_mlp) != 0;
        const bool tile_ok = any_mlp ? mlp::tile_eval(ts, x, use_mlp, y, phase) : true;
        int path = -1;
        if (ding) {
            DingParticleOut o;
            bool done = false;
            if (use_mlp && tile_ok) {
                // y is in the sorted order: singular value j has rank r_j with perm[r_j] = j.
                float e[3];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const int r = perm[0] == j ? 0 : (perm[1] == j ? 1 : 2);
                    e[j] = d.e[j] + pick3(y, r) * pick3(sg.out_scale, r);
                }
                done = ding_surrogate(P.ding, d, por, Fn, e, flags.ding, o, diag.plastic_gradients != nullptr);
                // Judged in whole warps, so that the exact map's cost falls on 1 warp in judge_stride.
                if (done && sg.judge_error && sg.judge_stride > 0 && (i >> 5) % sg.judge_stride == 0) {
                    DingParticleOut ex;
                    ding_exact(P.ding, d, por, FInRegs{Fn}, nullptr, ex, false);  // judge only: no flags
                    float err = 0.f;
#pragma unroll
                    for (int k = 0; k < 3; ++k) err = fmaxf(err, fabsf(ex.e[k] - e[k]));
                    atomic_max_nonneg(sg.judge_error, err);
                }
            }
            if (!done) ding_exact(P.ding, d, por, FInRegs{Fn}, flags.ding, o, diag.plastic_gradients != nullptr);
            path = done ? 1 : (o.yielded ? 2 : 0);
            ding_store(P, out, diag, i, T, o);
        }
        if (sg.path_counts && path >= 0) atomicAdd(&s_counts[path], 1);
        __syncthreads();
        if (ts.failed) {  // read after a barrier, so every thread takes the same branch
            if (threadIdx.x == 0 && P.status) atomicExch(P.status, 1);  // later tiles stay unprocessed
            break;
        }
    }
    mlp::tile_teardown(ts);
    if (sg.path_counts && threadIdx.x < 3 && s_counts[threadIdx.x]) atomicAdd(sg.path_counts + threadIdx.x, s_counts[threadIdx.x]);
}

template <bool kLoaf = false>
__global__ void __launch_bounds__(128, 4) k_g2p_return_surrogate(Params P, BkState in, BkState out, BkConstants cst,
                                                             GridPtrs g, BkDiagnostics diag, BkFlags flags,
                                                             SurrogateDev sg) {
    pdl_enter();
    if constexpr (kLoaf) {
        fix_loaf_mode(P);
        diag.plastic_gradients = diag.return_residuals = diag.porosity_residuals = nullptr;
        sg.samples = nullptr;
    }
    g2p_return_surrogate_body(P, in, out, cst, g, diag, flags, sg, grid_slot());
}

// ------------------------------------------------------------ materialize
__global__ void k_materialize(Params P, BkState s, BkConstants cst, float* Fp, float* T_mat, float* rho,
                              float* yield, float* visc, double* gas_p, double* sat, float* mass) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const int64_t pitch = P.pitch;
    M3 F = load_m3(s.F, i, pitch);
    float J = det3(F);
    float T = 0.f;
    if (P.transport) {
        double W = s.water[i], dry = cst.dry_mass[i];
        double V0 = (double)cst.volume[i];
        T = (float)s.temperature[i];
        if (rho) rho[i] = (float)((dry + W) / V0);
        if (sat) sat[i] = W / ((double)P.water_density * V0 * (double)J);
        if (mass) mass[i] = (float)(dry + W);
    } else if (P.material == 1) {
        T = s.material_temperature[i];
        if (rho) rho[i] = P.density;
    }
    if (P.material != 1) return;
    if (T_mat) T_mat[i] = T;
    if (Fp) store_m3(Fp, i, pitch, matmul(inverse3(load_m3(s.Fe, i, pitch)), F));
    const DingParamsDev& D = P.ding;
    float ty = D.yield_stress, eta = __ldg(cst.viscosity_parameter);
    if (D.temperature_enabled) {
        float Teff = s.gelled[i] ? D.knots[3] : T;
        ty = D.yield_stress * temperature_factor(Teff, D, D.yield_factors);
        eta = eta * temperature_factor(Teff, D, D.viscosity_factors);
    }
    if (yield) yield[i] = ty;
    if (visc) visc[i] = eta;
    if (gas_p && P.gas) {
        float n = s.porosity[i];
        if (n > 0.0f && n < 1.0f) gas_p[i] = gas_pressure(s.gas_moles[i], T, J, n);
    }
}

// physics/thermal_water.py:225-226 for the face-owning particles (the only ones whose loss or
// exchange changes): accumulators += dt * per-owner rate.
__global__ void k_surface_accumulate(int64_t owners_n, const int32_t* __restrict__ owners,
                                     const double* __restrict__ heat, const double* __restrict__ loss, double dt,
                                     double* __restrict__ water_losses, double* __restrict__ heat_exchanges) {
    int64_t o = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (o >= owners_n) return;
    int p = owners[o];
    water_losses[p] += dt * loss[o];
    heat_exchanges[p] += dt * heat[o];
}

unsigned blocks_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

#define BK_REQUIRE(cond, msg) do { if (!(cond)) return fail(BK_ERR_ARGUMENT, msg); } while (0)

// The argument checks of bk_substep (also applied to every instance of a batch).
int check_substep_args(const BkSubstepParams* params, const BkState* in, const BkState* out,
                       const BkConstants* constants, const BkGrid* grid, const BkSurface* surface,
                       const BkDiagnostics* diagnostics, const BkFlags* flags, int32_t phases) {
    BK_REQUIRE(params && in && out && constants && grid && diagnostics && flags, "bk_substep: null argument");
    const BkSubstepParams& p = *params;
    BK_REQUIRE(p.n >= 0 && p.pitch >= p.n, "bk_substep: bad particle count/pitch");
    BK_REQUIRE(p.resolution >= 4 && p.resolution < (1 << 20) && p.spacing > 0.0f, "bk_substep: bad grid");
    BK_REQUIRE(grid->node_pm && grid->node_v && grid->bounds, "bk_substep: missing grid arrays");
    BK_REQUIRE((((uintptr_t)grid->node_pm | (uintptr_t)grid->node_v) & 15) == 0, "bk_substep: grid not 16-byte aligned");
    BK_REQUIRE(in->x && in->v && in->C && in->F && out->x && out->v && out->C && out->F, "bk_substep: missing state");
    BK_REQUIRE(flags->simulation && flags->ding && flags->transport && diagnostics->max_residuals,
               "bk_substep: missing flags");
    if (p.material == 1)
        BK_REQUIRE(in->Fe && in->tau && in->porosity && in->gelled && out->Fe && out->tau && out->porosity &&
                   out->gelled && constants->viscosity_parameter, "bk_substep: missing Ding state");
    if (p.material == 1 && !p.transport)
        BK_REQUIRE(in->material_temperature && out->material_temperature, "bk_substep: missing Ding temperature");
    if (p.transport) {
        BK_REQUIRE(surface && in->temperature && in->water && out->temperature && out->water && constants->capacity &&
                   constants->dry_mass && constants->heat_parameter && grid->node_dT_ratio,
                   "bk_substep: missing transport arrays");
        for (int k = 0; k < 7; ++k) BK_REQUIRE(grid->fields[k] != nullptr, "bk_substep: missing node field");
        BK_REQUIRE(((uintptr_t)grid->node_dT_ratio & 15) == 0, "bk_substep: node_dT_ratio not 16-byte aligned");
    } else {
        BK_REQUIRE(constants->mass != nullptr, "bk_substep: missing particle masses");
    }
    if (p.gas)
        BK_REQUIRE(p.transport && p.material == 1 && in->gas_moles && out->gas_moles && constants->gas_rate,
                   "bk_substep: gas mode needs transport, the Ding model and gas arrays");
    if (p.transport_prescattered || p.transport_prescatter_next || p.transport_prescatter_stale)
        BK_REQUIRE(p.transport && !p.keep_transport_fields,
                   "bk_substep: the transport prescatter needs transport and a grid update that clears the fields");
    if (p.transport_prescatter_next)
        BK_REQUIRE(!(p.surrogate && p.surrogate->packed) && (phases & BK_PHASE_MECHANICS),
                   "bk_substep: the transport prescatter runs in the exact G2P kernel of a mechanics phase");
    return BK_OK;
}


// The launches of one substep (or of its phases); `with_flags` carries this substep's prescatter flags.
int launch_substep(const BkSubstepParams& p, const Params& with_flags, const GridPtrs& g, const BkState& in, const BkState& out,
                   const BkConstants& constants, const BkSurface* surface, const BkDiagnostics& diagnostics,
                   const BkFlags& flags, int32_t phases, int sms, cudaStream_t s) {
    const bool loaf = loaf_mode(p, diagnostics);
    const unsigned box_blocks = node_box_blocks(p.n, p.resolution, sms);
    const bool transport = (phases & BK_PHASE_TRANSPORT) && p.transport;
    // P2G leaves the node box to the transport scatter only where this call launches it: a mechanics phase
    // by itself, or one on fields scattered ahead (their box is another), finds the box empty.
    Params P = with_flags;
    P.box_widened = transport && !P.prescattered;
    cudaError_t e = cudaSuccess;
    if (transport) {
        const unsigned scatter_blocks = P.prescattered ? 0u : blocks_for(p.n, kOwnerThreads);
        const unsigned nv = (unsigned)surface->vertex_count;
        int vertex_threads = vertex_block_threads(surface->vertex_count, surface->binding_count);
        if (!P.prescattered && P.prescatter_stale) {
            e = launch_chained(k_clear_prescatter, box_blocks, kThreads, 0, s, P, g);
            if (int rc = check_chained(e, "bk_substep/clear_prescatter")) return rc;
        }
        // The scatter shares a launch with the longer of the two surface kernels before it: the vertices
        // of a coarse mesh (thousands of bindings each), the owners of a fine one (a third of the particles).
        const bool owners_first = surface->owner_count > 0 && owners_in_runs(surface->owner_count, p.n);
        const bool with_vertices = nv > 0 && scatter_blocks > 0 && !owners_first;
        const bool with_owners = scatter_blocks > 0 && owners_first;
        if (with_vertices) {
            const int rec = profile_begin("transport_scatter", s);
            const unsigned vb = vertex_threads == 32 ? vertex_launch_blocks(nv, 32) : nv;
            auto* kernel = vertex_threads == 32    ? k_vertices_scatter<32>
                           : vertex_threads == 128 ? k_vertices_scatter<128>
                                                   : k_vertices_scatter<256>;
            e = launch_chained(kernel, vb + scatter_blocks, kOwnerThreads, 0, s, P, in, constants, *surface, g, flags.simulation, (int)vb);
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/vertices_scatter")) return rc;
        } else if (nv > 0) {
            const int rec = profile_begin("surface_vertices", s);
            switch (vertex_threads) {
                case 256: e = launch_chained(k_surface_vertices<256>, nv, 256, 0, s, P, in.x, in.F, *surface); break;
                case 128: e = launch_chained(k_surface_vertices<128>, nv, 128, 0, s, P, in.x, in.F, *surface); break;
                default:
                    e = launch_chained(k_surface_vertices<32>, vertex_launch_blocks(nv, 32), vertex_launch_threads(32),
                                       0, s, P, in.x, in.F, *surface);
                    break;
            }
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/surface_vertices")) return rc;
        }
        if (with_owners) {
            const int rec = profile_begin("transport_scatter", s);
            const unsigned ob = blocks_for(surface->owner_count, kOwnerThreads);
            e = launch_chained(k_owners_scatter, ob + scatter_blocks, kOwnerThreads, 0, s, P, in, constants, *surface, g,
                               flags.simulation, (int)ob);
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/owners_scatter")) return rc;
        } else if (surface->owner_count > 0) {
            const int rec = profile_begin("surface_owners", s);
            e = launch_chained(k_surface_owners, owner_blocks(surface->owner_count, p.n), kOwnerThreads, 0, s, P, in,
                               constants, *surface, g, flags.simulation,
                               (int)owners_in_runs(surface->owner_count, p.n));
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/surface_owners")) return rc;
        }
        if (scatter_blocks > 0 && !with_vertices && !with_owners) {
            const int rec = profile_begin("transport_scatter", s);
            e = launch_chained(k_transport_scatter, scatter_blocks, kOwnerThreads, 0, s, P, in, constants, g, flags.simulation);
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/transport_scatter")) return rc;
        }
        {
            const int rec = profile_begin("diffuse", s);
            if (phases & BK_PHASE_MECHANICS) e = launch_chained(k_diffuse_clear, box_blocks, kDiffThreads, 0, s, P, g, flags.transport);
            else e = launch_chained(k_diffuse, box_blocks, kDiffThreads, 0, s, P, g, flags.transport);
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/diffuse")) return rc;
        }
    }
    if (phases & BK_PHASE_MECHANICS) {
        if (!transport) {
            const int rec = profile_begin("clear_previous", s);
            e = launch_chained(k_clear_previous, box_blocks, kThreads, 0, s, P, g);
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/clear_previous")) return rc;
        }
        {
            const int rec = profile_begin("p2g", s);
            const Sums sums = p2g_sums(p.n);
            const int threads = p2g_threads(sums);
            auto* kernel = sums == Sums::kAlone   ? (loaf ? k_p2g<Sums::kAlone, true> : k_p2g<Sums::kAlone>)
                           : sums == Sums::kTiles ? (loaf ? k_p2g<Sums::kTiles, true> : k_p2g<Sums::kTiles>)
                                                  : (loaf ? k_p2g<Sums::kKept, true> : k_p2g<Sums::kKept>);
            e = launch_chained(kernel, blocks_for(p.n, threads), threads, 0, s, P, in, out, constants, g, flags,
                               diagnostics.max_residuals);
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/p2g")) return rc;
        }
        {
            const int rec = profile_begin("grid_update", s);
            e = launch_chained(k_grid_update, box_blocks, kThreads, 0, s, P, g);
            profile_end(rec, s);
            if (int rc = check_chained(e, "bk_substep/grid_update")) return rc;
        }
        const SurrogateDev sg = surrogate_dev(p.surrogate);
        if (sg.blob && p.material == 1) {
            const int rec = profile_begin("g2p_return_surrogate", s);
            const unsigned tiles = blocks_for(p.n, 128);
            const unsigned persistent = (unsigned)sms * 4;
            e = launch_chained(loaf ? k_g2p_return_surrogate<true> : k_g2p_return_surrogate<false>,
                               tiles < persistent ? tiles : persistent, 128, 0, s, P, in, out, constants, g, diagnostics,
                               flags, sg);
            profile_end(rec, s);
        } else {
            const int rec = profile_begin("g2p_return", s);
            auto* kernel = !loaf ? k_g2p_return<false> : P.prescatter_next ? k_g2p_return<true, true> : k_g2p_return<true, false>;
            e = launch_chained(kernel, blocks_for(p.n, 128), 128, P.prescatter_next ? kG2PScatterBytes : 0, s, P, in, out,
                               constants, g, diagnostics, flags, sg);
            profile_end(rec, s);
        }
        if (int rc = check_chained(e, "bk_substep/g2p_return")) return rc;
    }
    return BK_OK;
}

thread_local int32_t substeps_launched = 0;  // by this thread's last bk_substeps call

int sm_count() {
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms;
}

}  // namespace

extern "C" {

int bk_substep(const BkSubstepParams* params, const BkState* in, BkState* out, const BkConstants* constants,
               BkGrid* grid, BkSurface* surface, BkDiagnostics* diagnostics, BkFlags* flags, int32_t phases,
               void* stream) {
    if (int rc = check_substep_args(params, in, out, constants, grid, surface, diagnostics, flags, phases)) return rc;
    if (params->n == 0) return BK_OK;
    return launch_substep(*params, to_params(*params), grid_ptrs(*grid), *in, *out, *constants, surface, *diagnostics,
                          *flags, phases, sm_count(), S(stream));
}

int bk_substeps(const BkSubstepParams* params, const BkState* states, double* const* water_losses,
                double* const* heat_exchanges, const BkConstants* constants, BkGrid* grid, const BkSurface* surface,
                const BkDiagnostics* diagnostics, BkFlags* flags, int32_t count, int32_t scatter_ahead, void* stream) {
    const int32_t phases = BK_PHASE_TRANSPORT | BK_PHASE_MECHANICS;
    substeps_launched = 0;
    BK_REQUIRE(states && diagnostics && count >= 0, "bk_substeps: null argument or negative count");
    BK_REQUIRE(params && !params->transport_prescattered && !params->transport_prescatter_next,
               "bk_substeps: the call sets the prescatter flags itself");
    for (int k = 0; k < 2; ++k)
        if (int rc = check_substep_args(params, states + k, states + 1 - k, constants, grid, surface, diagnostics + 1 - k,
                                        flags, phases))
            return rc;
    const BkSubstepParams& p = *params;
    if (p.transport) BK_REQUIRE(water_losses && heat_exchanges, "bk_substeps: missing surface accumulators");
    if (scatter_ahead)
        BK_REQUIRE(p.transport && !p.keep_transport_fields && !(p.surrogate && p.surrogate->packed),
                   "bk_substeps: the transport prescatter needs transport, cleared fields and the exact return map");
    if (p.n == 0) return BK_OK;
    Params P = to_params(p);
    const GridPtrs g = grid_ptrs(*grid);
    const int sms = sm_count();
    BkSurface sf{};
    if (p.transport) sf = *surface;
    for (int32_t k = 0; k < count; ++k) {
        const int from = k & 1, to = 1 - from;
        P.prescattered = scatter_ahead && k > 0;
        P.prescatter_next = scatter_ahead && k + 1 < count;
        P.prescatter_stale = k == 0 && p.transport_prescatter_stale;
        if (p.transport) {
            sf.accumulate_water_losses = water_losses[to];
            sf.accumulate_heat_exchanges = heat_exchanges[to];
            sf.accumulate_time_step = p.time_step;
        }
        if (int rc = launch_substep(p, P, g, states[from], states[to], *constants, &sf, diagnostics[to], *flags, phases, sms,
                                    S(stream)))
            return rc;
        ++substeps_launched;
    }
    return BK_OK;
}

int bk_substeps_launched(void) { return substeps_launched; }

int bk_surface_accumulate(const BkSurface* surface, float time_step, double* water_losses, double* heat_exchanges,
                          void* stream) {
    BK_REQUIRE(surface && water_losses && heat_exchanges, "bk_surface_accumulate: null argument");
    if (surface->owner_count == 0) return BK_OK;
    BK_REQUIRE(surface->owners && surface->owner_heat && surface->owner_loss, "bk_surface_accumulate: missing owners");
    k_surface_accumulate<<<blocks_for(surface->owner_count, kThreads), kThreads, 0, S(stream)>>>(
        surface->owner_count, surface->owners, surface->owner_heat, surface->owner_loss, (double)time_step,
        water_losses, heat_exchanges);
    return check_launch("bk_surface_accumulate");
}

int bk_materialize(const BkSubstepParams* params, const BkState* state, const BkConstants* constants,
                   float* plastic_gradients, float* material_temperature, float* reference_density,
                   float* yield_stress, float* viscosity, double* gas_pressure, double* saturation,
                   float* particle_mass, void* stream) {
    BK_REQUIRE(params && state && constants, "bk_materialize: null argument");
    const BkSubstepParams& p = *params;
    BK_REQUIRE(p.n >= 0 && p.pitch >= p.n, "bk_materialize: bad particle count/pitch");
    if (p.n == 0) return BK_OK;
    BK_REQUIRE(state->F != nullptr, "bk_materialize: missing F");
    if (p.transport)
        BK_REQUIRE(state->temperature && state->water && constants->dry_mass && constants->volume,
                   "bk_materialize: missing transport arrays");
    if (p.material == 1)
        BK_REQUIRE(state->Fe && state->gelled && state->porosity && constants->viscosity_parameter &&
                   (p.transport || state->material_temperature), "bk_materialize: missing Ding arrays");
    if (p.gas && gas_pressure) BK_REQUIRE(state->gas_moles != nullptr, "bk_materialize: missing gas moles");
    k_materialize<<<blocks_for(p.n, kThreads), kThreads, 0, S(stream)>>>(
        to_params(p), *state, *constants, plastic_gradients, material_temperature, reference_density, yield_stress,
        viscosity, gas_pressure, saturation, particle_mass);
    return check_launch("bk_materialize");
}

}  // extern "C"

// ===================================================================== batched substeps
// Many independent simulators advanced by one launch per stage: each block of a batched launch
// finds its instance in a device table (a binary search over the stage's first-block prefix),
// copies that instance's entry into shared memory and runs the same kernel body as a plain
// launch, with its index among the instance's blocks. The blocks an instance gets per stage are
// the ones its own launch would use (particles, vertices, owners), or for the node-box passes a
// share that grows with its particle count, so a batch of small bodies fills the GPU.
namespace {

enum BatchStage { kStVertices, kStOwners, kStScatter, kStDiffuse, kStClear, kStP2G, kStGrid, kStG2P, kStSurrogate,
                  kBatchStages };

struct BatchEntry {
    Params P;
    BkState in, out;
    BkConstants cst;
    GridPtrs g;
    BkSurface sf;
    BkDiagnostics diag;
    BkFlags flags;
    SurrogateDev sg;   // sf carries the surface accumulators of `out`
    int prescatter_ok;  // takes part in the transport prescatter
    int owners_in_runs;   // the surface terms take the run form (owners_in_runs)
};
static_assert(sizeof(BatchEntry) % 4 == 0, "entries are copied as 4-byte words");

struct BatchArgs {
    const BatchEntry* entries;  // [2][count]: parity 0 steps states[0] -> states[1], parity 1 back
    const uint32_t* first;      // [kBatchStages][count + 1]: first block of each instance per stage
    const int32_t* owner;       // the instance of every block of every stage, stage by stage
    uint32_t owner_offset[kBatchStages];  // where each stage's blocks start in `owner`
    int count, parity, prescattered, prescatter_next;
    int scatters;  // the call has a transport phase
};

// The instance that owns this block in `stage` (one load from the block map) and the block's slot
// within it.
__device__ __forceinline__ Slot batch_find(const BatchArgs& b, int stage, int& k) {
    k = __ldg(b.owner + b.owner_offset[stage] + blockIdx.x);
    const uint32_t* f = b.first + (size_t)stage * (b.count + 1);
    const uint32_t f0 = __ldg(f + k), f1 = __ldg(f + k + 1);
    return Slot{(int)(blockIdx.x - f0), (int)(f1 - f0)};
}

// Copies the block's entry into shared memory with this call's prescatter flags. Every thread of
// the block calls it (it synchronises the block).
__device__ __forceinline__ Slot batch_load(const BatchArgs& b, int stage, BatchEntry& e) {
    int k;
    const Slot sl = batch_find(b, stage, k);
    const int* src = reinterpret_cast<const int*>(b.entries + (size_t)b.parity * b.count + k);
    int* dst = reinterpret_cast<int*>(&e);
    for (int w = threadIdx.x; w < (int)(sizeof(BatchEntry) / 4); w += blockDim.x) dst[w] = __ldg(src + w);
    __syncthreads();
    if (threadIdx.x == 0) {
        e.P.prescattered = b.prescattered && e.prescatter_ok;
        e.P.prescatter_next = b.prescatter_next && e.prescatter_ok;
        e.P.prescatter_stale = 0;
        e.P.box_widened = b.scatters && e.P.transport && !e.P.prescattered;
    }
    __syncthreads();
    return sl;
}

// (Plain launches: chained by programmatic launch, waiting blocks of one table hold the SM slots that the
// other table's stream would use; 12 balls, 40 substeps, 6.77 ms against 6.51.)
template <int kBlock>
__global__ void __launch_bounds__(kBlock == 32 ? 32 * kVertexWarps : kBlock) kb_surface_vertices(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStVertices, e);
    surface_vertices_body<kBlock, true>(e.P, e.in.x, e.in.F, e.sf, sl);
}

__global__ void __launch_bounds__(kOwnerThreads) kb_surface_owners(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStOwners, e);
    surface_owners_body<true>(e.P, e.in, e.cst, e.sf, e.g, e.flags.simulation, e.owners_in_runs != 0, sl);
}

__global__ void __launch_bounds__(kOwnerThreads) kb_transport_scatter(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStScatter, e);
    if (e.P.prescattered) return;  // fields scattered ahead by this instance's previous G2P
    transport_scatter_body<true>(e.P, e.in, e.cst, e.g, e.flags.simulation, sl);
}

__global__ void __launch_bounds__(kDiffThreads) kb_diffuse(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStDiffuse, e);
    diffuse_body<true>(e.P, e.g, e.flags.transport, sl);
}

__global__ void __launch_bounds__(kThreads) kb_clear_previous(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStClear, e);
    clear_previous_body<true>(e.P, e.g, sl);
}

template <Sums kSums>
__global__ void __launch_bounds__(kP2GThreads, kSums == Sums::kKept ? 8 : 4) kb_p2g(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStP2G, e);
    p2g_body<kSums, true>(e.P, e.in, e.out, e.cst, e.g, e.flags, e.diag.max_residuals, sl);
}

__global__ void __launch_bounds__(kThreads) kb_grid_update(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStGrid, e);
    grid_update_body<true>(e.P, e.g, sl);
}

__global__ void __launch_bounds__(128, 8) kb_g2p_return(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStG2P, e);
    g2p_return_body<true>(e.P, e.in, e.out, e.cst, e.g, e.diag, e.flags, e.sg, sl);
}

__global__ void __launch_bounds__(128, 4) kb_g2p_return_surrogate(BatchArgs b) {
    __shared__ BatchEntry e;
    const Slot sl = batch_load(b, kStSurrogate, e);
    g2p_return_surrogate_body<true>(e.P, e.in, e.out, e.cst, e.g, e.diag, e.flags, e.sg, sl);
}

}  // namespace

struct BkBatch {
    int count = 0;
    BatchEntry* entries = nullptr;  // device [2][count]
    uint32_t* first = nullptr;      // device [kBatchStages][count + 1]
    int32_t* owner = nullptr;       // device: instance of each block, stage by stage
    uint32_t owner_offset[kBatchStages] = {};
    uint32_t total[kBatchStages] = {};
    int vertex_block = 32;
    bool all_prescatter = true;     // every transport instance takes part in the prescatter
    bool any_transport = false;
    bool tiles = true;              // every instance is small enough for P2G's tiles
};

extern "C" {

int bk_batch_create(const BkBatchInstance* instances, int32_t count, BkBatch** batch) {
    BK_REQUIRE(instances && batch && count > 0, "bk_batch_create: null argument or empty batch");
    *batch = nullptr;
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    std::vector<BatchEntry> entries(2 * (size_t)count);
    std::vector<uint32_t> first((size_t)kBatchStages * (count + 1), 0);
    int64_t particles = 0, vertices = 0, bindings = 0;
    for (int k = 0; k < count; ++k) {
        particles += instances[k].params.n;
        if (instances[k].params.transport && instances[k].params.n > 0) {
            vertices += instances[k].surface.vertex_count;
            bindings += instances[k].surface.binding_count;
        }
    }
    BkBatch host;
    host.count = count;
    host.vertex_block = vertex_block_threads(vertices, bindings);  // one block size for the whole launch
    for (int k = 0; k < count; ++k) {
        const BkBatchInstance& in = instances[k];
        const BkSubstepParams& p = in.params;
        const bool surrogate = p.surrogate && p.surrogate->packed && p.material == 1;
        for (int parity = 0; parity < 2; ++parity) {
            const BkState& a = in.states[parity];
            const BkState& b = in.states[1 - parity];
            BkSubstepParams q = p;
            q.transport_prescattered = q.transport_prescatter_next = q.transport_prescatter_stale = 0;
            if (int rc = check_substep_args(&q, &a, &b, &in.constants, &in.grid, &in.surface, &in.diagnostics,
                                            &in.flags, BK_PHASE_TRANSPORT | BK_PHASE_MECHANICS))
                return rc;
            if (p.transport)
                BK_REQUIRE(in.water_losses[1 - parity] && in.heat_exchanges[1 - parity],
                           "bk_batch_create: missing surface accumulators");
            BatchEntry& e = entries[(size_t)parity * count + k];
            e.P = to_params(q);
            e.in = a;
            e.out = b;
            e.cst = in.constants;
            e.g = grid_ptrs(in.grid);
            e.sf = in.surface;
            e.sf.accumulate_water_losses = p.transport ? in.water_losses[1 - parity] : nullptr;
            e.sf.accumulate_heat_exchanges = p.transport ? in.heat_exchanges[1 - parity] : nullptr;
            e.sf.accumulate_time_step = p.time_step;
            e.diag = in.diagnostics;
            e.flags = in.flags;
            e.sg = surrogate_dev(surrogate ? p.surrogate : nullptr);
            e.prescatter_ok = p.transport && !p.keep_transport_fields && !surrogate;
            e.owners_in_runs = owners_in_runs(in.surface.owner_count, p.n);
        }
        host.any_transport = host.any_transport || p.transport;
        host.tiles = host.tiles && p.n < kKeptParticles;
        if (p.transport && (p.keep_transport_fields || surrogate)) host.all_prescatter = false;
        uint32_t blocks[kBatchStages] = {};
        const int64_t n = p.n;
        if (n > 0) {
            if (p.transport) {
                blocks[kStVertices] = vertex_launch_blocks(in.surface.vertex_count, host.vertex_block);
                blocks[kStOwners] = owner_blocks(in.surface.owner_count, n);
                blocks[kStScatter] = blocks_for(n, kOwnerThreads);
            }
            // Node-box passes: the diffusion takes a block per 256 particles (a tile of 256 nodes costs it
            // ~3 us, and a ball's box holds about one node per particle: with a block per 2048 particles
            // 12 balls of 4.8-11.2k particles took 54 us, now 15), the clears one per 1024.
            const uint32_t box = (uint32_t)std::min<int64_t>((n + 1023) / 1024, 4 * sms);
            if (p.transport) blocks[kStDiffuse] = (uint32_t)std::min<int64_t>((n + 255) / 256, 4 * sms);
            blocks[kStClear] = box;
            blocks[kStP2G] = blocks_for(n, kP2GThreads);
            blocks[kStGrid] = box;
            if (surrogate) {
                // a persistent share of 4 CTAs per SM in proportion to the particles
                const int64_t share = std::max<int64_t>(1, (int64_t)(4.0 * sms * (double)n / (double)particles + 0.5));
                blocks[kStSurrogate] = (uint32_t)std::min<int64_t>(share, blocks_for(n, 128));
            } else {
                blocks[kStG2P] = blocks_for(n, 128);
            }
        }
        for (int st = 0; st < kBatchStages; ++st) {
            uint32_t* f = first.data() + (size_t)st * (count + 1);
            BK_REQUIRE((uint64_t)f[k] + blocks[st] < (1ull << 31), "bk_batch_create: too many blocks in one stage");
            f[k + 1] = f[k] + blocks[st];
        }
    }
    std::vector<int32_t> owner;
    for (int st = 0; st < kBatchStages; ++st) {
        host.total[st] = first[(size_t)st * (count + 1) + count];
        host.owner_offset[st] = (uint32_t)owner.size();
        for (int k = 0; k < count; ++k)
            owner.insert(owner.end(), first[(size_t)st * (count + 1) + k + 1] - first[(size_t)st * (count + 1) + k], k);
    }
    BK_REQUIRE(owner.size() < (1ull << 31), "bk_batch_create: too many blocks");
    if (owner.empty()) owner.push_back(0);
    BkBatch* out = new BkBatch(host);
    if (cudaMalloc(&out->entries, entries.size() * sizeof(BatchEntry)) != cudaSuccess ||
        cudaMalloc(&out->first, first.size() * sizeof(uint32_t)) != cudaSuccess ||
        cudaMalloc(&out->owner, owner.size() * sizeof(int32_t)) != cudaSuccess) {
        cudaFree(out->entries);
        cudaFree(out->first);
        cudaFree(out->owner);
        delete out;
        cudaGetLastError();
        return fail(BK_ERR_LAUNCH, "bk_batch_create: device allocation failed");
    }
    if (cudaMemcpy(out->entries, entries.data(), entries.size() * sizeof(BatchEntry), cudaMemcpyHostToDevice) !=
            cudaSuccess ||
        cudaMemcpy(out->first, first.data(), first.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(out->owner, owner.data(), owner.size() * sizeof(int32_t), cudaMemcpyHostToDevice) != cudaSuccess) {
        bk_batch_destroy(out);
        return fail(BK_ERR_LAUNCH, "bk_batch_create: table upload failed");
    }
    *batch = out;
    return BK_OK;
}

int bk_batch_substep(BkBatch* batch, int32_t parity, int32_t phases, int32_t prescattered, int32_t prescatter_next,
                     void* stream) {
    BK_REQUIRE(batch && (parity == 0 || parity == 1), "bk_batch_substep: bad batch or parity");
    BK_REQUIRE(!prescatter_next || (phases & BK_PHASE_MECHANICS),
               "bk_batch_substep: the transport prescatter runs in the G2P kernel of a mechanics phase");
    const BkBatch& B = *batch;
    BatchArgs a{};
    a.entries = B.entries;
    a.first = B.first;
    a.owner = B.owner;
    for (int st = 0; st < kBatchStages; ++st) a.owner_offset[st] = B.owner_offset[st];
    a.count = B.count;
    a.parity = parity;
    a.prescattered = prescattered ? 1 : 0;
    a.prescatter_next = prescatter_next ? 1 : 0;
    a.scatters = phases & BK_PHASE_TRANSPORT ? 1 : 0;
    const uint32_t* T = B.total;
    cudaStream_t s = S(stream);
    if ((phases & BK_PHASE_TRANSPORT) && B.any_transport) {
        if (T[kStVertices]) {
            int rec = profile_begin("batch_surface_vertices", s);
            switch (B.vertex_block) {
                case 256: kb_surface_vertices<256><<<T[kStVertices], 256, 0, s>>>(a); break;
                case 128: kb_surface_vertices<128><<<T[kStVertices], 128, 0, s>>>(a); break;
                default: kb_surface_vertices<32><<<T[kStVertices], vertex_launch_threads(32), 0, s>>>(a); break;
            }
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/surface_vertices")) return rc;
        }
        if (T[kStOwners]) {
            int rec = profile_begin("batch_surface_owners", s);
            kb_surface_owners<<<T[kStOwners], kOwnerThreads, 0, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/surface_owners")) return rc;
        }
        if (T[kStScatter] && !(prescattered && B.all_prescatter)) {
            int rec = profile_begin("batch_transport_scatter", s);
            kb_transport_scatter<<<T[kStScatter], kOwnerThreads, 0, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/transport_scatter")) return rc;
        }
        if (T[kStDiffuse]) {
            int rec = profile_begin("batch_diffuse", s);
            kb_diffuse<<<T[kStDiffuse], kDiffThreads, 0, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/diffuse")) return rc;
        }
    }
    if (phases & BK_PHASE_MECHANICS) {
        if (T[kStClear]) {
            int rec = profile_begin("batch_clear_previous", s);
            kb_clear_previous<<<T[kStClear], kThreads, 0, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/clear_previous")) return rc;
        }
        if (T[kStP2G]) {
            int rec = profile_begin("batch_p2g", s);
            if (B.tiles) kb_p2g<Sums::kTiles><<<T[kStP2G], kP2GThreads, 0, s>>>(a);
            else kb_p2g<Sums::kKept><<<T[kStP2G], kP2GThreads, 0, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/p2g")) return rc;
        }
        if (T[kStGrid]) {
            int rec = profile_begin("batch_grid_update", s);
            kb_grid_update<<<T[kStGrid], kThreads, 0, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/grid_update")) return rc;
        }
        if (T[kStG2P]) {
            int rec = profile_begin("batch_g2p_return", s);
            const size_t smem = prescatter_next ? kG2PScatterBytes : 0;
            kb_g2p_return<<<T[kStG2P], 128, smem, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/g2p_return")) return rc;
        }
        if (T[kStSurrogate]) {
            int rec = profile_begin("batch_g2p_return_surrogate", s);
            kb_g2p_return_surrogate<<<T[kStSurrogate], 128, 0, s>>>(a);
            profile_end(rec, s);
            if (int rc = check_launch("bk_batch_substep/g2p_return_surrogate")) return rc;
        }
    }
    return BK_OK;
}

int bk_batch_destroy(BkBatch* batch) {
    if (!batch) return BK_OK;
    cudaFree(batch->entries);
    cudaFree(batch->first);
    cudaFree(batch->owner);
    delete batch;
    return BK_OK;
}

}  // extern "C"
