// gy_kernels.cuh -- launch interface between the host runtime (gy_api.cu) and the kernels.
#pragma once

#include <utility>

#include "gy_common.cuh"

namespace gy {

// Device view of one particle slab.
struct PView {
    float *base;
    long long cap;
    __device__ __forceinline__ float &f(int field, long long i) const { return base[(long long)field * cap + i]; }
    __device__ __forceinline__ int &ii(int field, long long i) const
    {
        return reinterpret_cast<int *>(base)[(long long)field * cap + i];
    }
};

// Single-body node buffers.  Accumulators (P2G target, zeroed by the solve):
//   acc0 = (m, px, py, pz), acc1 = (fx, fy, fz, -).
// Solved fields (read by G2P): gv = (m, v1x, v1y, v1z), ga = (a1x, a1y, a1z, -).
// Multi-body adds per-slot accumulators and solved fields.
struct NodeBufs {
    float4 *acc0, *acc1;
    float4 *gv, *ga;
    float4 *out_com;        // optional (vcom, -) for node getters
    float4 *out_force;      // optional COM force for node getters
    const unsigned char *bc_type;
    const float4 *bc_val;
    // multi-body
    float4 *bacc0[2], *bacc1[2];  // per body slot: (m, p), (f, -)
    float4 *bnrm[2];              // per body slot: (n, -)
    float4 *bgv[2], *bga[2];      // solved per slot: (m, v), (a, -); slot 0's are gv / ga
    float4 *nrm_out[2];           // normalised slot normals (only when normals are tracked)
    int2 *body;                   // body slot objects (dense ids) or -1
    int *flags;                   // per 4x4x4 node block: the epoch of the last step P2G or the fold wrote it in
    int *active_list;             // node blocks marked this step (when the solve is asked for the list)
    int *active_n;                // length of active_list
    unsigned char *has_rigid;     // bit0: slot 0 rigid, bit1: slot 1 rigid
    int *active_count;            // nodes with mass (stats)
    int *block_body;              // per 4x4x4 cell block: the one body of its 6x6x6 node tile, -1 none, -2 more
    int *nblk_two;                // per 4x4x4 node block: 1 if one of its nodes holds two bodies
};

// Hooks of the learned Drucker-Prager surrogate into the step (every pointer null when off).
// Logging: the exact return mapping records, for particles that yield and whose
// (insertion index + step) is a multiple of log_every, the MLP input (strain increment,
// previous stress, plastic strain, damage, cohesion, friction angle) and target (stress
// minus the elastic trial stress, plastic strain increment).  Deferral: a yielding particle
// without a BC goes to the pending list (slot and strain increment) with its stress left at
// the previous value; the surrogate pass finishes its return mapping and damage.
struct DpHooks {
    float *log_x, *log_y;         // [log_cap][16], [log_cap][7]
    unsigned int *log_n;          // records claimed (those past log_cap are dropped)
    unsigned int log_cap;
    int log_every;
    float4 *pend;                 // [pend_cap][2]: (slot bits, de0, de1, de2), (de3, de4, de5, -)
    unsigned int *pend_n;
    unsigned int pend_cap;
};

// The segments the particle kernels take, one CTA each: the particles [start, start + len) of one
// cell block, in cell order.  len null: a segment ends where the block of its run does.
struct Segs {
    const int *start, *len;
    const int *n;
    long long most;   // there are no more of them than this (0: not known)
    const int *blk = nullptr, *first = nullptr;  // with blk: whole cell blocks instead, [first[b], first[b + 1])
};

// How a cell block's particles are cut into segments: pieces of 2^shift, and a remainder of up to
// merge goes with the last of them.
struct Pieces {
    int shift, merge;
    __host__ __device__ int len() const { return 1 << shift; }
};

// Cell-block bookkeeping of the block merge sort (gy_blocks.cu); zeroed once at allocation.
struct BlockSort {
    int *cnt;             // particles per cell block by their current key, kept by G2P
    int *in_cnt;          // movers that entered each block since the last sort
    int *dirty;           // blocks in which a particle changed cell since the last sort
    int *first[2];        // first position of each block, of the last two sorts in turn
    int *in_off;          // first entry of each block in in_list
    int4 *mov;            // movers to another block: key, slot, arrival number at the block
    int *mov_n;
    int2 *in_list, *in_sorted;  // the movers (key, slot) grouped by new block, then also in slot order
    int *list, *list_n;   // the non-empty blocks
    int *seg_at;          // the first segment of each of them
    int nblk;
};

// The steps' scalars in pinned host memory, one slot per step in turn.  The first kernel of a step
// takes the next slot into `sc`, where the others read it: a copy
// ahead of the step's kernels cost a small step 3 of its 33 us.
struct ScalarRing {
    static constexpr int SLOTS = 32;
    const StepScalars *slots;
    int *taken;              // the slot the next step takes
    StepScalars *sc;
};
#ifdef __CUDACC__
// by one warp
__device__ __forceinline__ void take_scalars(const ScalarRing &r)
{
    const int lane = threadIdx.x & 31, t = *r.taken;
    static_assert(sizeof(StepScalars) <= 32 * sizeof(int), "a lane per word");
    if (lane < (int)(sizeof(StepScalars) / sizeof(int)))
        reinterpret_cast<int *>(r.sc)[lane] = __ldcv(reinterpret_cast<const int *>(r.slots + t) + lane);
    __syncwarp();
    if (lane == 0) *r.taken = (t + 1) % ScalarRing::SLOTS;
}
#endif

struct StepArgs {
    GridGeom g;
    const StepScalars *sc;   // the step's scalars in device memory, where its first kernel put them (ScalarRing)
    int multi_body;          // host-side launch choice, fixed per handle
    const DevMaterial *mats;
    const float4 *pbc_val;   // particle BC values by pid
    const float *flaw;       // Grady-Kipp activation strain scale by pid, or null (every scale 1)
    int *status;
    double *stats;           // STATS_SLOTS x 8 conservation partials written by G2P, or null
    DpHooks dp;              // learned-surrogate logging / deferral (zero when off)
    unsigned *mover_mask;    // G2P flags the slots whose key changed, one bit per slot (or null),
    int *mover_cnt;          //   with the flagged count per 32 slots, for the next re-sort
    int *blk_cnt, *blk_in, *blk_dirty;  // or, for the block merge sort, keeps its counts and its
    int4 *mov;                          //   list of movers (blk_cnt null: not)
    int *mov_n;
};

// partials of the conservation sums (mass, momentum, kinetic and strain energy); the host
// adds the slots
constexpr int STATS_SLOTS = 16;

// launch with programmatic stream serialization (the kernel starts with pdl_prologue), so the
// launch of a kernel overlaps the tail of the one before it in the stream or graph
template <typename... P, typename... A>
inline cudaError_t launch_pdl_smem(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A &&... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}
template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A &&... args)
{
    return launch_pdl_smem(kernel, grid, block, 0, s, std::forward<A>(args)...);
}

// The step's particle and grid kernels are launched plainly.  Launched ahead of their
// predecessor's end, a step took 41 us against 36 at 8,000 particles and 398 against 358 at 2.4
// million: the waiting CTAs hold the SMs' space while the running kernel finishes, and settle
// unevenly on them.
template <typename... P, typename... A>
inline cudaError_t launch_step(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A &&... args)
{
    kernel<<<grid, block, 0, s>>>(std::forward<A>(args)...);
    return cudaPeekAtLastError();
}

// a plain launch that answers for itself: what another call left pending in the runtime is not its
template <typename... P, typename... A>
inline cudaError_t launch_checked(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A &&... args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.stream = s;
    return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

// The status of an entry point whose CUDA call failed: the runtime keeps such an error for whoever
// asks it next (another handle's step or initialisation among them), so it is taken out with the answer.
template <class Status> inline Status cuda_failed(Status st)
{
    cudaGetLastError();
    return st;
}

// keeps the first failure of a sequence of launches (err may be null)
inline void keep_first(cudaError_t *err, cudaError_t e)
{
    if (err && e != cudaSuccess && *err == cudaSuccess) *err = e;
}

// process-wide count of kernel launches (for the benchmark's launch accounting)
void note_launch(int k);
long long launch_count();

// launchers (gy_kernels.cu)
// therm / tnode non-null: the single-body kernel also sums the heat conduction node fields
// (multi-body problems run launch_thermal_p2g instead).  lanes: 3 takes the warp kernel where the
// segments have lengths (steps sorted by block) and the z-plane kernel, three lanes per run of equal
// cell, elsewhere; 9 the x-column kernel, nine lanes per run (with several bodies the body-slot kernel
// throughout).  defer / ndefer: list and count of the segments left to the body-slot kernel.
void launch_p2g(const PView &p, const int *perm, const int *skey, long long n, const Segs &sg,
                int persist_grid, const NodeBufs &nb, const StepArgs &a, cudaStream_t s,
                const float4 *therm = nullptr, float2 *tnode = nullptr, int lanes = 3, int *defer = nullptr,
                int *ndefer = nullptr);
void launch_fold(const NodeBufs &nb, const StepArgs &a, cudaStream_t s);
void launch_block_body(const NodeBufs &nb, const GridGeom &g, cudaStream_t s);
// want_list: fill active_list / active_n (zeroed earlier in the step)
void launch_solve(const NodeBufs &nb, const StepArgs &a, bool keep_node_fields, bool want_list, cudaStream_t s);
// therm / tnode non-null: the single-body kernel also runs the heat conduction G2P and the
// temperature update (multi-body problems run launch_thermal_g2p instead)
void launch_g2p_update(const PView &src, const PView &dst, const int *perm, const int *skey, long long n,
                       const Segs &sg, int g2p_grid, const NodeBufs &nb, const StepArgs &a,
                       bool track_normals, bool check_finite, bool has_dp, cudaStream_t s, float4 *therm = nullptr,
                       const float2 *tnode = nullptr);
int g2p_blocks_per_sm(bool has_dp);
int p2g_blocks_per_sm();
// the learned surrogate's pass over the particles G2P deferred (gy_mlp.cu)
void launch_dp_surrogate(const PView &P, const float4 *pend, const unsigned int *pend_n, unsigned int cap,
                         const DevMaterial *mats, const float *prm, const StepScalars *scp, const float *flaw, float tol,
                         unsigned long long *counts, int *status, cudaStream_t s);
void launch_body_tables(const PView &p, long long n, const StepArgs &a, int *cell_min, int nbody,
                        const int *refkeys, cudaStream_t s);
void launch_body_assign(const NodeBufs &nb, const StepArgs &a, const int *cell_min, int nbody,
                        const int *nidx_x, const int *nidx_y, const int *nidx_z, cudaStream_t s);
void launch_stats(const PView &p, long long n, double *out8, cudaStream_t s);
void launch_gather_slab(const float *src, float *dst, const int *perm, long long n, long long cap, int nfields,
                        cudaStream_t s);

// heat conduction (gy_thermal.cu): therm = (T, grad T) per insertion index, tnode = (T, rate)
void launch_thermal_p2g(const PView &p, const float4 *therm, const int *perm, const int *skey, long long n,
                        const Segs &sg, float2 *tnode, const StepArgs &a, cudaStream_t s);
void launch_thermal_g2p(const PView &p, float4 *therm, const int *perm, const int *skey, long long n,
                        const Segs &sg, const float2 *tnode, const NodeBufs &nb,
                        const StepArgs &a, cudaStream_t s);
void launch_thermal_clear(const NodeBufs &nb, const StepArgs &a, float2 *tnode, cudaStream_t s);
void launch_thermal_set(float4 *therm, const int *ids, const float *T, int count, long long n, cudaStream_t s);

// sort (gy_sort.cu): stable LSD radix sort of (key, index) pairs
struct SortScratch {
    int *keys[2], *vals[2];
    int *hist;          // 2 * 256 * nblocks
    int *scan_tmp;      // scan workspace
    long long cap;
    int nblocks_cap;
};
size_t sort_scratch_bytes(long long n);

// Incremental re-sort (gy_resort.cu): scratch, zeroed once at allocation.
struct ResortScratch {
    unsigned *wmask;
    int *wcnt, *wpref, *wscan_tmp;
    int *bkey, *bidx, *gap, *bslot;       // the movers in slot order
    unsigned long long *stage;            // the movers grouped by key bucket, as (key, slot) words
    int *tval;                            // a buffer of the fallback sort
    int *gapcnt, *gwcnt, *gwpref, *gscan_tmp;
    int *big;                             // a bucket too crowded to rank by counting
    int *mlast;                           // the last re-sort's mover count
    long long cap, ngw;
};
size_t resort_scratch_ints(long long cap);
void resort_bind(ResortScratch &rs, int *mem, long long cap);
void resort_keys(const int *key, const int *prev_skey, int *skey_out, int *perm_out, long long n, int key_bits,
                 ResortScratch &rs, cudaStream_t s, bool mask_ready = false, const int *blk_first = nullptr);
// block merge sort (gy_blocks.cu)
size_t block_sort_ints(long long nblk, long long cap);
void block_sort_bind(BlockSort &b, int *mem, long long nblk, long long cap);
void launch_blocks_count(const BlockSort &b, const int *skey, long long n, cudaStream_t s);
void launch_blocks_scan(const BlockSort &b, const ScalarRing &ring, int which, Pieces piece, int *nseg, cudaStream_t s,
                        int *clear0 = nullptr, int *clear1 = nullptr, int *clear2 = nullptr, int *clear3 = nullptr);
void launch_take_scalars(const ScalarRing &ring, cudaStream_t s);
// key null: another sort has made the order, only the segments are written
void launch_blocks_place(const BlockSort &b, const int *key, int which, Pieces piece, int *seg_start, int *seg_len,
                         int *skey_out, int *perm_out, long long n, cudaStream_t s);
// particle fields in insertion order and FP64 (gy_export.cu)
struct ExportArgs {
    GridGeom g;
    const double *pos0;      // 3 per particle, by insertion index
    const int *key0;         // the cell key and the offsets (field by field) a particle was uploaded with
    const float *off0;
    double h, init_volume;
    bool has_dp, normals;
    int slot_obj[MAX_BODIES];
};
cudaError_t launch_export(const PView &p, long long n, int field, const ExportArgs &a, double *out, cudaStream_t s);
cudaError_t launch_export_int(const PView &p, long long n, int field, const ExportArgs &a, int *out, cudaStream_t s);
cudaError_t launch_export_therm(const float4 *therm, long long n, int field, double *out, cudaStream_t s);
// err (may be null) receives the first launch failure of the sort's kernels
const int *sort_pairs(const int *keys_in, int *perm_out, long long n, int key_bits, SortScratch &ws, cudaStream_t s,
                      cudaError_t *err = nullptr);
// nseg must be zero on entry; clear0..2 (may be null): counters the kernel zeroes on the way;
// blk_first (may be null, one int per cell block): each non-empty block's first position
void launch_block_heads(const int *skey, long long n, int *seg_start, int *nseg, cudaStream_t s,
                        int *clear0 = nullptr, int *clear1 = nullptr, int *clear2 = nullptr,
                        int *blk_first = nullptr);
void exclusive_scan_int(const int *in, int *out, long long n, int *tmp, cudaStream_t s, cudaError_t *err = nullptr);

// exclusive scan of ints: tiles of SCAN_TILE, scanned recursively over the tile sums
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 4;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

// ints of scratch exclusive_scan_int needs for n elements (constant-evaluable, so fixed
// scratch sizes can be checked at compile time)
constexpr size_t scan_tmp_ints(long long n)
{
    size_t total = 0;
    long long m = n;
    while (m > SCAN_TILE) {
        m = (m + SCAN_TILE - 1) / SCAN_TILE;
        total += (size_t)m * 2 + 32;
    }
    return total + 64;
}

}  // namespace gy
