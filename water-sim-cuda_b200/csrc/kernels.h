// Host-side launchers of the engine's CUDA kernels.  Each launcher enqueues
// its kernels on `st` and returns how many kernel launches it issued, so the
// engine can count the launches of a step.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "corrector.cuh"
#include "corrector_tc.cuh"
#include "device_math.cuh"

namespace mpm {

// ---------------------------------------------------------------- sort ----
// Stable LSD radix sort of 32-bit signed keys, 8-bit digits, 4 passes.
// Each pass is histogram -> per-digit spine scan -> scatter; no kernel waits
// on another CTA, so nothing can spin on the GPU.
struct SortScratch {
    int32_t* key_a = nullptr;
    int32_t* val_a = nullptr;
    int32_t* key_b = nullptr;
    int32_t* val_b = nullptr;
    uint32_t* hist = nullptr;    // [256][nb] per-CTA digit counts, scanned in place
    uint32_t* totals = nullptr;  // [256] digit totals of the pass
    uint32_t* diff = nullptr;    // [nb] bits in which a CTA's keys differ from key 0
    uint32_t* active = nullptr;  // bit k: pass k runs
    int n = 0;
    int nb = 0;       // CTAs per pass
    int per_cta = 0;  // keys per CTA (multiple of the 2048-key tile)
};

// Bytes of scratch for sorting n keys (256-byte aligned sub-buffers).
size_t sort_scratch_bytes(int n);
// Points the scratch sub-buffers into `base` (sort_scratch_bytes(n) bytes).
void sort_scratch_carve(void* base, int n, SortScratch* s);

// keys[i] = Morton key of (px[i], py[i], pz[i]) (setKeys, kernels.cu:361-371),
// i < s.n, and their sort permutation as launch_radix_sort writes it.
int launch_morton_sort(const float* px, const float* py, const float* pz, int32_t* keys, const SortScratch& s,
                       int32_t* sigma, cudaStream_t st);

// Sorts `keys` (n signed ints, left unchanged) with values 0..n-1, stable, and
// writes the permutation sigma[j] = index of the j-th smallest key, the
// result of thrust::sequence + thrust::sort_by_key (engine.cu:98-99).
// If rank_out is non-null it also writes rank_out[sigma[j]] = j, and if gidx
// is non-null gidx[j] = rank_in[sigma[j]] (rank_in null: sigma[j]).
int launch_radix_sort(const int32_t* keys, int n, const SortScratch& s, int32_t* sigma, int32_t* rank_out,
                      const int32_t* rank_in, int32_t* gidx, cudaStream_t st);

// ------------------------------------------------------------- substep ----
// The substep kernels work on all scenes of a SceneTable at once; particle
// slots, cells and bins are global (device_math.cuh).  P is the
// particle-major state, ordered by cell of the binning that produced it.
// pcell[j] is the global cell of slot j; ccur holds one slot cursor per
// cell, which the ordering's scatter draws the cell's slots from.  A counter
// set holds the cell counts (global cells) and the bin counts, which a G2P or
// an import fills, and the list of the bins that hold particles, as (scene,
// bin), with its length *nlist (zero until then), which the ordering by the
// set makes.  Two sets alternate: a substep orders the particles by one and
// its G2P fills the other, which that substep clears first, bin by bin of its
// list.
struct BinSet {
    uint32_t* ccount;
    int2* blist;
    uint32_t* bcount;
    uint32_t* nlist;
};

// Counters of one substep, zero before its ordering: P2G's work units taken
// and the length of the crowded-cell list.  The scatter resets work, G2P
// resets crowded; an ordering whose substep is abandoned needs it and its
// set's list length zeroed by the host.
struct OrderCtl {
    uint32_t* work;
    uint32_t* crowded;
};

// Node tiles of the grid update, one per bin: tile (bx, by, bz) of a scene
// holds the nodes x in [8 bx - 2, 8 bx + 6), y in [4 by - 2, 4 by + 2), z in
// [4 bz - 2, 4 bz + 2), so that the 10 x 6 x 6 nodes a bin's particles reach
// lie in tiles bx..bx+1 x by..by+1 x bz..bz+1.  stamp[0] counts orderings;
// mark[global bin] = the stamp of the last ordering whose listed bins reach
// the tile; dirty[global bin] = 1 while the tile's velocity nodes may hold
// values other than zero.
struct TileMarks {
    uint32_t* stamp;
    uint32_t* mark;
    uint8_t* dirty;
    long long count;  // global bin entries (nb + 2 per scene)
};

// Files the n particles of P (all scenes, slot order) into an empty set.
int launch_bin_count(const SceneTable& sc, long long n, const float* P, int32_t* pcell, const BinSet& set,
                     cudaStream_t st);
// Slots per entry of the ordering's `edge`: the cells of the first and the
// last of them.  G2P's CTAs take whole entries.
constexpr int kEdgeSlots = 128;
// Order by cell from set `cur`: gidx[new slot] = old slot, edge, desc (P2G's items:
// kBinZ per listed bin, indexed like the cells), crowd / *ctl.crowded (the
// crowded-cell list; crowd_cap entries of room, at least n / 4 + 64); clears
// `other`; with tiles.mark set, advances tiles.stamp and marks the tiles the
// listed bins of `cur` reach.  bstart: the bins' first slots; bpart: scenes x
// scan_chunks ints of scratch, scan_chunks = bin_scan_chunks(largest nb + 1).
// bins_total: sum over scenes of nb + 1.
// cell_cap: particles of a cell its own lane sums in P2G before the rest goes
// to the list (0 = chosen per work item from its cells' counts).
int launch_bin_order(const SceneTable& sc, long long n, long long bins_total, const BinSet& cur, const BinSet& other,
                     const OrderCtl& ctl, int32_t* bstart, int32_t* bpart, int scan_chunks, const int32_t* pcell,
                     int32_t* ccur, int32_t* gidx, int2* edge, int2* desc, int4* crowd, int crowd_cap, int cell_cap,
                     const TileMarks& tiles, uint32_t* status, cudaStream_t st);
// Chunks of the bin scan for a scene of `bins` bins.
int bin_scan_chunks(long long bins);
// P2G over the crowded-cell list and the items of `cur`; gidx maps slots of
// the new order to P.  ctas_per_sm: persistent single-warp CTAs per SM (0 =
// the default 12).
int launch_p2g(const SceneTable& sc, long long n, long long bins_total, const float* P, const int32_t* gidx,
               const BinSet& cur, const int2* desc, const int4* crowd, int crowd_cap, const OrderCtl& ctl,
               float4* accum, uint32_t* status, cudaStream_t st, int ctas_per_sm = 0);
// Most P2G CTAs that fit on one SM.
int p2g_max_ctas_per_sm();
// p0: the parameters of scene 0, used directly when the table holds one scene.
// With tiles.mark set: only the tiles marked by this substep's ordering are
// updated, and tiles updated before but not marked now are reset to zero;
// else every node.
int launch_grid_update(const SceneTable& sc, const SimParams& p0, long long g_total, float4* accum, float4* vgrid,
                       const float* sdf, const TileMarks& tiles, cudaStream_t st, int block = 256);
// Large-step G2P (one scene): particles advect with v_old + blend (v_new -
// v_old).  With mlp set: the corrector's correction is added to each
// particle's velocity and stat[0] += sum over particles of |1 / det(I + dt C)
// - 1| (the step's predicted relative density change).  With feat set
// (collection probe): feat[orig] receives the 16 features and vel[orig] the
// final velocity, by original index.  Neither: the uncorrected large step.
struct LearnArgs {
    const MlpPacked* mlp;
    float* feat;
    float* vel;
    float* stat;
    float blend;
    const MlpTc* mlp_tc;  // set: the MLP runs on tcgen05 (mlp unused)
    uint32_t* status;     // kStatusTimeout when a tcgen05 wait gives up
    uint32_t wait_test;   // test hooks of the first tcgen05 wait (kWaitTest*, corrector_tc.cuh)
};

// G2P: slot j of Pout = particle gidx[j] of Pin advanced one substep;
// sig_out[j] = sig_in[gidx[j]]; files slot j into `next`; zeroes *crowded
// (OrderCtl).  learn: a large step of one scene (LearnArgs), else null.
int launch_g2p(const SceneTable& sc, const SimParams& p0, long long n, const float* Pin, float* Pout,
               const int32_t* gidx, const int2* edge, const int32_t* sig_in, int32_t* sig_out, const float4* vgrid,
               const float* sdf, int32_t* pcell, const BinSet& next, uint32_t* crowded, uint32_t* health,
               cudaStream_t st, const LearnArgs* learn = nullptr, int block = 256);

// The kernels below take one scene's SimParams and pointers already offset to
// that scene's part of the arrays.
// ------------------------------------------------------ state transfer ----
// Loads a 26-plane host-layout state (already on the device, stride n) into
// P (original order) and sets sigma[i] = p.poff + i (global slots).
// init_rules applies initFMatrices (kernels.cu:349-358): F diagonal = 1.
int launch_state_import(const SimParams& p, const float* soa26, float* P, int32_t* sigma, bool init_rules,
                        cudaStream_t st);
// keys[sigma[j] - p.poff] = setKeys' Morton key of slot j of P (original order).
int launch_reference_keys(const SimParams& p, const float* P, const int32_t* sigma, int32_t* keys, cudaStream_t st);
// Writes the 26-plane state in original order: plane k of particle sigma[j]
// from slot j of P (VOL and MASS from the scalars).
int launch_state_export(const SimParams& p, const float* P, const int32_t* sigma, float* soa26, cudaStream_t st);
// Float3 positions in original order (changeFormat, kernels.cu:341-347), all
// scenes in one launch: xyz triple sigma[j] from slot j of P, j < n.  Also
// flags_host[0..1] = flags[0..1] (flags_host may be null).
int launch_positions_export(long long n, const float* P, const int32_t* sigma, float* xyz, const uint32_t* flags,
                            uint32_t* flags_host, cudaStream_t st);
// Node float4 (mass, x, y, z) -> 4 planes.
int launch_grid_export(const SimParams& p, const float4* grid, float* planes4, cudaStream_t st);

// ----------------------------------------------------------------- sdf ----
// tris: 9*t floats on the device, allocation padded by >= 16 bytes.  aux:
// sdf_aux_floats(t) floats on the device (16-byte aligned) holding what
// sdf_prepare_host wrote: the triangles sorted by the Morton code of their
// centroids, and the boxes of the triangles and of groups of them.  spread:
// what sdf_prepare_host returned, whether the sign is spread (a closed mesh,
// and enough nodes and triangles) or summed at every node.
// wait_test: test hooks of the first triangle tile's wait (kWaitTestGiveUp /
// kWaitTestExpire, corrector_tc.cuh), acted on after the real completion.
size_t sdf_aux_floats(int t);
bool sdf_prepare_host(const float* tris, int t, long long nodes, float* aux);
int launch_sdf_build(const SimParams& p, const float* tris, const float* aux, int t, bool spread, float* sdf,
                     uint32_t* status, cudaStream_t st, uint32_t wait_test = 0u);
int launch_fill(float* dst, long long count, float value, cudaStream_t st);
// The learned step's fallback decision (one thread): rule 0 / 1 / 2 =
// MPM_FALLBACK_DENSITY_CHANGE / REST_DENSITY / REST_DENSITY_EXCESS on the
// means of stat[0..2] over n particles; sets `fallback` to 1 to reject.
int launch_learned_decide(const float* stat, long long n, int rule, float threshold,
                          cudaGraphConditionalHandle fallback, long long* counters, float* last, cudaStream_t st);
// count 32-bit words from src to dst (device memory, not overlapping).
int launch_copy_words(void* dst, const void* src, long long count, cudaStream_t st);
// dst[i] = i for i < n.
int launch_identity(int32_t* dst, int n, cudaStream_t st);

// Device status bits written by kernels with bounded waits.
enum : uint32_t {
    kStatusTimeout = 1u << 0,  // a bounded wait gave up
    kStatusBinning = 1u << 1,  // P2G met a particle outside the cell it was filed under
    kStatusCrowdList = 1u << 2 // the crowded-cell list of P2G overflowed
};

// Sets the thread's mpm_global_last_error text (engine.cu).
void set_global_error(const std::string& msg);

}  // namespace mpm
