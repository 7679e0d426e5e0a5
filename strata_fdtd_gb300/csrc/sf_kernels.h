// sf_kernels.h -- internal launcher declarations shared by the .cu files.
#pragma once
#include <cuda_runtime.h>

#include "sf_common.cuh"

// Step-kernel configuration indices used by sf_plan_set_kernel /
// sf_plan_autotune: 0 = automatic, 1 = per-cell kernel, 2 = slab march,
// SF_CFG_COL_FIRST + c = column kernel configuration c, then the warp-tile
// configurations.
enum { SF_CFG_AUTO = 0, SF_CFG_CELL = 1, SF_CFG_MARCH = 2, SF_CFG_COL_FIRST = 3 };

struct SfColConfig {
    int vec, by, minb, cs;
    const char* name;
};
extern const SfColConfig kSfColConfigs[];
extern const int kSfColConfigCount;

// Warp-tile kernel configurations follow the column ones:
// index SF_CFG_COL_FIRST + kSfColConfigCount + t.
struct SfTileConfig {
    int vec, rows, warps, minb, prefetch;
    const char* name;
};
extern const SfTileConfig kSfTileConfigs[];
extern const int kSfTileConfigCount;
// Whether a warp-tile kernel with `vec` cells per lane runs on this grid.
bool sf_tile_supported(const SfStepArgs& a, int vec);

// Multi-step pipeline configurations follow the warp-tile ones: index
// SF_CFG_COL_FIRST + kSfColConfigCount + kSfTileConfigCount + t.  One launch
// advances the state by `levels` steps (sf_step_pipe.cu).  Claimed-item
// pipelines (stream = 0): level s runs `lag` chunks behind level s-1 and the
// rings between levels hold `ring_chunks` chunks of planes each.  Streaming
// pipelines (stream = 1): one co-resident warp per (level, tile) walks the
// whole x extent; the rings hold `ring_chunks` planes (a power of two).
#define SF_PIPE_MAX_LEVELS 4
struct SfPipeConfig {
    int levels, warps, minb, lag, ring_chunks, stream;
    const char* name;
};
extern const SfPipeConfig kSfPipeConfigs[];
extern const int kSfPipeConfigCount;

// One launch of the pipeline: a.p.. is the input set, a.po.. the output
// set, a.src_val the first step's waveform values (level s uses row s-1),
// a.trace_prev the probe row of the input state.
struct SfPipeArgs {
    SfStepArgs a;
    int levels;   // steps per launch
    int S;        // planes per chunk
    int M;        // chunks per ring
    int nchunks;  // ceil(nx / S)
    int ntk;      // tiles along k (32 cells each)
    int ntiles;   // tiles per chunk
    int ngroups;  // (level, chunk) groups in claim order
    float* ring;        // (levels-1) rings x 4 fields x M*S planes
    const int* order;   // per group: (level << 24) | chunk, level 1-based
    int* ctrl;          // [0] next item; [1 + ((level-1)*nchunks + chunk)*ntiles + tile] done
    int* err;           // nonzero: a bounded wait expired (2)
    float* trace_lvl[SF_PIPE_MAX_LEVELS];  // probe row of level s+1's result, or null
    long long spin_limit;  // sleeps (64-256 ns each) before a wait gives up
    // Expiry test hook, normally null: a flag that nothing ever sets.  The
    // first claimed item (k_step_pipe) or the first warp (k_step_stream)
    // also waits on it, so its wait runs out and the launch fails cleanly.
    const int* hold;
};
// Default bound of every pipeline wait: 2^22 sleeps, about 1 s.
#define SF_PIPE_SPIN_DEFAULT (1LL << 22)
int sf_launch_step_pipe(const SfPipeArgs& P, const SfSources& src, bool geom, int cfg, int grid,
                        cudaStream_t st);
// Resident blocks of pipeline configuration cfg on this device (grid size).
int sf_pipe_grid(int cfg, bool geom, bool nu);
// Streaming pipeline: P.ctrl holds the per-(level, tile) plane progress
// (levels * ntiles ints, zeroed), P.S the publishing interval in planes,
// P.M the ring planes; probe_tile[u] / probe_plane[u] place the probes.
// Returns SF_PIPE_NOFIT (without launching) when its warps cannot all be
// resident at once.
#define SF_PIPE_NOFIT 77
int sf_launch_step_stream(const SfPipeArgs& P, const SfSources& src, bool geom, int cfg,
                          cudaStream_t st);

// Two-step configurations (sf_step_tb.cu) follow the pipeline ones: index
// SF_CFG_COL_FIRST + kSfColConfigCount + kSfTileConfigCount +
// kSfPipeConfigCount + t.  One launch advances the state by two steps;
// warps of 28 output k x `rows` output j, `warps` per block along j;
// trace1 receives the probe row of the state after the first step.
struct SfTbConfig {
    int rows, warps, minb;
    const char* name;
    int quads;  // 0: warp tiles; else windows of `rows` x `quads` (k_step_tbq)
};
extern const SfTbConfig kSfTbConfigs[];
extern const int kSfTbConfigCount;
bool sf_tb_supported(const SfStepArgs& a);
int sf_launch_step_tbq(const SfStepArgs& a, const SfSources& src, bool geom, int rows, int ich, float* trace1,
                       cudaStream_t st);
int sf_launch_step_tb(const SfStepArgs& a, const SfSources& src, bool geom, int cfg, int ich,
                      float* trace1, cudaStream_t st);

// Many steps of a small grid in one launch, its state on the chip
// (sf_step_resident.cu).  A cut says how the grid is divided into blocks.
// Shared memory of a block: offsets in floats (multiples of 4).
struct SfResLayout {
    int src;             // this step's source values (doubles)
    int ctl;             // [0] weighted cells, [1] probes, [2] a wait expired, [3] microphone corners
    int side;            // (decay, coefficient) of each side's faces
    int P, UX, UY, UZ;   // pressures; x faces at chunk ends, y faces, z faces
    int dx, dy, dz;      // PML decays of the block's planes, rows, cells
    int cx, cy, cz, sx, sy, sz;  // NU: face coefficients, cell scales
    int probe;           // (trace column, cell in P)
    int prev[SF_MAX_PLANE_OPS][2];  // plane boundaries: stored planes, low and high
    int wlist;           // weighted sources: (cell in P, source, weight) entries
    int mic;             // microphone corners (int4)
    int end;
    int plist;           // cells of the absorbing planes
};
// What acts between the steps: pressure-plane boundaries, weighted sources on
// the pressure, microphone corners.
struct SfResExtra {
    int n_plane;
    sf_plane_bc ops[SF_MAX_PLANE_OPS];
    float2 coeff[SF_MAX_PLANE_OPS];  // ops[].coeff as a sum of two floats (0, 0: not taken apart)
    float* prev[SF_MAX_PLANE_OPS][2];
    const long long* wcells[SF_MAX_SOURCES];  // by source
    const double* ww[SF_MAX_SOURCES];
    int wn[SF_MAX_SOURCES];
    int wbox[6];       // cells lo, hi (exclusive) per axis of all weighted sources, empty: none
    int w_slots;       // how many sources are weighted
    int n_mic;         // microphone rows
    const int* mic_field;
    const long long* mic_idx;
    float* corners;    // [step][row][8]
};
struct SfResCut {
    int kind;          // planes per thread and thread counts (kKinds), < 0: does not fit
    bool extra;        // for a plan with something between the steps
    int bi, bj, bk;    // blocks along x, y, z
    int chunks, quads; // chunks of planes and quads of k cells in the grid
    int threads;
    int side_max;      // message units of the largest block side that a cut crosses
    int units;         // message units of a block at most
    SfResLayout lay;
    size_t smem;
};
struct SfResArgs {
    SfStepArgs a;      // a.src_val, a.trace_prev: the first step's rows
    int n_steps;
    int bi, bj, bk, chunks, quads, side_max;
    SfResLayout lay;
    unsigned long long* mail;  // 2 x blocks x 6 x side_max x 4 words
    unsigned tag;      // the first step's tag
    int* err;          // set when a wait expired
    long long poll_limit;
    int hold;          // expiry test hook: block 0 waits for tags nothing sends
    SfResExtra x;
};
// Both sets of mailboxes of a launch, and the most that a cut may need.
constexpr size_t kSfResMailMax = size_t(64) << 20;
inline size_t sf_resident_mail_bytes(int blocks, int side_max) {
    return (size_t)2 * blocks * 6 * side_max * 4 * sizeof(unsigned long long);
}
SfResCut sf_resident_cut(int nx, int ny, int nz, int n_probe, bool nu, int sms, const SfResExtra* x);
int sf_launch_resident_mics(const float* corners, const float* w, int n_mic, long long n_steps,
                            float* mic_trace, cudaStream_t st);
int sf_launch_resident(SfResArgs& A, const SfSources& src, const SfResCut& c, cudaStream_t st);

int sf_launch_build_flags(const uint8_t* geom, uint8_t* flags, int nx, int ny, int nz,
                          cudaStream_t st);
int sf_launch_step(const SfStepArgs& a, const SfSources& src, const SfPoles& poles, bool geom,
                   cudaStream_t st);
int sf_launch_probe_gather(const float* p, const long long* cells, int n, float* out,
                           cudaStream_t st);
int sf_launch_step_march(const SfStepArgs& a, const SfSources& src, bool geom, int ich,
                         cudaStream_t st);
int sf_launch_step_col_cfg(const SfStepArgs& a, const SfSources& src, bool geom, int cfg, int ich,
                           cudaStream_t st);
int sf_launch_step_tile_cfg(const SfStepArgs& a, const SfSources& src, bool geom, int cfg, int ich,
                            cudaStream_t st);
int sf_launch_plane_bc(float* p, float* prev_lo, float* prev_hi, const sf_plane_bc& op, int nx,
                       int ny, int nz, cudaStream_t st);
int sf_launch_inject(float* p, const uint8_t* flags, const sf_source& s, const double* val, int nx,
                     int ny, int nz, cudaStream_t st);
int sf_launch_inject_weighted(float* f, const long long* cells, const double* w, long long n,
                              const double* val, cudaStream_t st);
int sf_launch_mic_gather(const float* p, const float* vx, const float* vy, const float* vz,
                         const int* field, const long long* idx, const float* w, int n, float* out,
                         cudaStream_t st);
// Blocks of the energy reduction over n cells on a device with `sms` SMs
// (at most 8 per SM); its scratch holds 2 partial sums per block + 2 totals.
long long sf_energy_blocks(long long n, int sms);
int sf_launch_energy(const float* p, const float* vx, const float* vy, const float* vz,
                     const uint8_t* flags, long long n, int sms, double* scratch, double* out2,
                     cudaStream_t st);
int sf_launch_voxelize(const sf_sdf_node* nodes, int n_nodes, int nx, int ny, int nz, double res,
                       const double* const* coords, int invert, uint8_t* out, cudaStream_t st);
void sf_voxel_release_kept();
int sf_launch_voxelize_materials(const sf_sdf_node* prog_dev, const int* off_dev,
                                 const uint8_t* ids_dev, int n_regions, int nx, int ny, int nz,
                                 double res, const double* coords_dev, uint8_t* geom,
                                 uint8_t* mat, int* err_dev, cudaStream_t st);
int sf_launch_sdf_points(const sf_sdf_node* prog_dev, int n_nodes, const double* pts, long long n,
                         double* out, int* err_dev, cudaStream_t st);
