// Stage kernels: one CTA advances one tile of one simulation by one substep of
// its scheme (the work of one block of a reference kernel launch, e.g.
// GPUSimulators/cuda/SWE2D_KP07_dimsplit.cu:123-205).  One launch covers any
// number of substeps: its CTAs take (substep, tile) tasks in order and wait for
// the tiles they read (stage_kernel).
//
// Tile: a CTA owns W x H interior cells.  One TMA box per variable brings the
// tile plus a 4-column / 2-row halo into shared memory ((H+4) x P floats with
// row pitch P = W+8, or wider for 8-segment tiles, split_pitch; box x aligned
// to 4 floats).  Ghost cells are then completed in shared memory
// (periodic wrap from global memory, reflective mirror in the reference's
// N, S, E, W order), the sweeps run in place, and the interior is written back
// with 128-bit stores.  The CFL minimum is reduced in the same pass; the CTA
// that finishes a launch's last substep last advances the simulation's control
// block (t, nt, dt, buffer parity).
//
// Sweep mapping:
//   x sweeps: a thread walks one row segment of W/4 cells (lanes = 8 rows x
//     4 segments; or W/8 cells, lanes = 4 rows x 8 segments).  With a shared
//     row pitch of an odd multiple of 4 floats (8 mod 32) and an odd segment
//     length the 32 lanes hit 32 distinct banks.
//   y sweeps: a thread walks one column segment (lanes = consecutive columns).
//   LPT = 2: a thread walks two lines side by side in packed f32x2
//     arithmetic (rows t and t + n/2, columns s and s + n/2).
// Each thread keeps a 3-cell window in registers and reconstructs every cell
// once; the halo cells of its segment are read before a barrier so that
// in-place updates by neighbouring segments cannot race with them.
#pragma once

#include <cuda.h>

#include <type_traits>

#include "fv_device.cuh"
#include "fv_tiles.h"

namespace fv {

enum Scheme { LXF = 0, FORCE = 1, HLL = 2, HLL2 = 3, WAF = 4, KP07 = 5, KP07_DIMSPLIT = 6, EE2D = 7 };

// Reference boundary codec (GPUSimulators/cuda/common.h:109-130).
enum BoundaryType { BC_DIRICHLET = 0, BC_NEUMANN = 1, BC_PERIODIC = 2, BC_REFLECTIVE = 3 };
__host__ __device__ inline int bc_north(int bc) { return (bc >> 24) & 0xF; }
__host__ __device__ inline int bc_south(int bc) { return (bc >> 16) & 0xF; }
__host__ __device__ inline int bc_east(int bc) { return (bc >> 8) & 0xF; }
__host__ __device__ inline int bc_west(int bc) { return bc & 0xF; }

// What a bounded wait that gave up was for.
constexpr int kTileLoadGaveUp = 1;   // the tensor copies of a tile
constexpr int kNeighbourGaveUp = 2;  // the tiles around it in the substep before

// Control block of one simulation, resident in device memory.
struct alignas(16) SimCtl {
    double t;          // simulation time (BaseSimulator.t, FP64)
    double t_end;      // end time of the current simulate() call
    long long nt;      // completed steps (BaseSimulator.nt)
    float dt;          // CFL step in use (BaseSimulator.dt)
    float cfl_min;     // min of the last CFL field (gpuarray.min(cfl_data))
    float factor;      // the scheme's computeDt factor
    float cfl_scale;   // Courant number
    int update_dt;     // recompute dt every 100 steps (simulate(t) without dt)
    int cur;           // buffer index holding u0
    unsigned int arrive;  // CTA arrival counter for the last-CTA epilogue
    int error;         // kTileLoadGaveUp, kNeighbourGaveUp: the bounded waits that gave up
    int bad;           // batched simulations: a step left a non-finite value or a non-positive depth
                       // (density); the simulation then stops (t_end is set to t)
};

// Steps of a launch that may take another time step than the control block's
// (the last steps of a simulate() call, shortened to end at its end time).
constexpr int kTailSteps = 4;

// Distance of the per-tile progress counters in 32-bit words: each has a
// 32-byte sector of its own, so that the CTAs that poll them are spread over the
// L2 (4 bytes apart, 256 x 256 cells took twice as long per substep).
constexpr int kDoneStride = 8;

// Launch arguments (passed as a __grid_constant__ parameter; the tensor maps
// must live in parameter, constant or global memory).
struct StageArgs {
    CUtensorMap tmap[2][4];  // [buffer][variable]
    float* buf[2][4];
    SimCtl* ctl;
    float* block_cfl;    // one float per tile
    unsigned* ticket;    // tasks taken (launches of several substeps); zero between launches
    unsigned* done;      // per tile, kDoneStride apart: substeps of this run completed; zero between runs
    int nx, ny, pitch;   // pitch in floats
    int tiles_x, tiles_y;
    float dx, dy, g, gamma, theta;
    float dt_scale;      // kernel dt = step dt * dt_scale (0.5 for split substeps)
    float variant_beta;  // parameter of the Osher and Sweby limiters (the variant itself is a kernel template)
    int bc;
    int order;           // RK order (KP07)
    int substeps;        // substeps (sweep orders of the split schemes, RK stages of KP07) per step
    int first_substep;   // substep of the step that the run starts with
    int n_sub;           // substeps of the run: of this launch, or of a chain of them (follows, followed)
    int steps;           // steps the run completes (0: a substep by itself, t and nt stay)
    int full_steps;      // steps that take the control block's dt; the ones after take tail[]
    float tail[kTailSteps];
    int explicit_dt;     // all steps take dt_step, whatever the control block says
    float dt_step;
    int want_cfl;        // compute the CFL minimum of the last substep's state
    int wait_limit;      // bounded waits for tile loads: 0 = kWaitPolls polls (the default, also for
                         // zero-filled arguments), n > 0 = n polls, negative = give up at once (tests)
    int neighbour_limit; // the same for the waits for neighbouring tiles
    int follows;         // this launch goes on where the one before stopped in the same run of substeps
    int followed;        // and the next one goes on where this one stops
    int tile_row0;       // first tile row of this launch (one substep may be split into launches by rows)
    int ntiles_total;    // tiles of the whole substep, 0 = this launch's; the last of them to
                         // arrive, over all launches, finishes the launch
};

// Polls of a bounded mbarrier wait before it gives up (each poll may suspend
// the thread for a short hardware-defined time; in all about a second).
constexpr uint32_t kWaitPolls = 1u << 20;
__host__ __device__ inline uint32_t wait_polls(int wait_limit) {
    return wait_limit == 0 ? kWaitPolls : (wait_limit < 0 ? 0u : (uint32_t)wait_limit);
}

// Storage: per variable, rows y = -2 .. ny+1 and columns x = -4 .. pitch-5,
// element (y, x) at [(y + 2) * pitch + (x + 4)].
__host__ __device__ inline long long cell_index(int y, int x, int pitch) {
    return (long long)(y + 2) * pitch + (x + 4);
}

// Split-scheme tiles: x-sweep segments per tile row and the shared-memory row
// pitch (the TMA box width) of a W-wide tile.  A warp's x-sweep lanes cover
// 32/NSEG rows x NSEG segments of W/NSEG cells; they hit 32 distinct banks
// when the segment length is odd and the pitch is an odd multiple of 4 for 4
// segments, 8 (mod 32) for 8.  W + 8 (4 halo columns each side) is an odd
// multiple of 4 for the 4-segment widths (124, 60, 28, 12); 8-segment widths
// (120) load a box padded on the right to the next pitch of 8 (mod 32).
__host__ __device__ constexpr int split_nseg_x(int W) { return ((W / 4) % 2 == 1) ? 4 : 8; }
__host__ __device__ constexpr int split_pitch(int W) {
    return split_nseg_x(W) == 4 ? W + 8 : W + 8 + (((8 - (W + 8)) % 32) + 32) % 32;
}

struct StepCtl {
    float dt;      // step dt (before dt_scale)
    double t_new;  // t after this step
    int cur;
    bool active;
    bool do_cfl;
};

// dt of the current step: float32(min(dt, t_end - t)) (GPUSimulators/Simulator.py:199),
// with Python's min() tie and NaN behaviour; a step runs while t < t_end and
// dt > 0 (Simulator.py:192, :202).
//
// The control block changes only between launches, or in this launch after
// every tile of the simulation has read it (the last tile's epilogue), so its
// first 48 bytes are read with three 16-byte relaxed loads issued together: one
// L2 round trip per warp instead of one per field.
__device__ __forceinline__ int4 ld_relaxed_v4(const void* p) {
    int4 r;
    asm volatile("ld.relaxed.gpu.global.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}

// The step of a control block from its first 48 bytes (w0, w1, w2).
__device__ __forceinline__ StepCtl step_from_words(const int4& w0, const int4& w1, const int4& w2, bool explicit_dt,
                                                   float dt_step, bool force_cfl, bool is_last) {
    StepCtl s;
    s.cur = w2.w;
    const double t = __hiloint2double(w0.y, w0.x);
    const double t_end = __hiloint2double(w0.w, w0.z);
    if (explicit_dt) {
        s.dt = dt_step;
        s.active = true;
    } else {
        const double rem = t_end - t;
        const double d = (double)__int_as_float(w1.z);
        s.dt = (float)((rem < d) ? rem : d);
        s.active = (t < t_end) && !(s.dt <= 0.0f);
    }
    s.t_new = t + (double)s.dt;
    const long long nt = (long long)(((unsigned long long)(unsigned)w1.y << 32) | (unsigned)w1.x);
    const bool sched = w2.z && ((nt + 1) % 100 == 0);
    s.do_cfl = force_cfl || (is_last && !explicit_dt && (sched || !(s.t_new < t_end)));
    return s;
}

static_assert(offsetof(SimCtl, t_end) == 8 && offsetof(SimCtl, nt) == 16 && offsetof(SimCtl, dt) == 24 &&
                  offsetof(SimCtl, update_dt) == 40 && offsetof(SimCtl, cur) == 44,
              "the vector loads of control blocks follow SimCtl's layout");

// A value that the compiler takes for a new one in every task of a looping
// kernel: what follows from it is computed per task instead of being kept in
// registers from task to task.
template <bool LOOP, class T>
__device__ __forceinline__ T per_task(T v) {
    if constexpr (LOOP && std::is_same<T, float>::value) asm volatile("" : "+f"(v));
    else if constexpr (LOOP) asm volatile("" : "+r"(v));
    return v;
}

// The thread's index in its CTA; tid, from per_task, in a looping kernel.
template <bool LOOP>
__device__ __forceinline__ unsigned thread_of(unsigned tid) {
    if constexpr (LOOP) return tid;
    else return threadIdx.x;
}

template <int NT, bool LOOP = false>
__device__ __forceinline__ float block_min(float v, float* red, unsigned tid) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int w = thread_of<LOOP>(tid) >> 5;
    __syncthreads();
    if ((thread_of<LOOP>(tid) & 31) == 0) red[w] = v;
    __syncthreads();
    float r = red[0];
#pragma unroll
    for (int i = 1; i < NT / 32; ++i) r = fminf(r, red[i]);
    return r;
}

template <int NT>
__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[w] = v;
    __syncthreads();
    double r = red[0];
#pragma unroll
    for (int i = 1; i < NT / 32; ++i) r += red[i];
    return r;
}

// ------------------------------------------------------------------ tile load + ghost cells

// One tile of one simulation: where its input comes from and where it goes.
struct TileJob {
    const CUtensorMap* tmap;  // NV tensor maps of the input planes (kernel parameters; unused by async loads)
    float* const* in;         // NV input planes
    float* const* out;        // NV output planes
    int nx, ny, pitch, bc;
    int x0, y0;               // first interior cell of the tile
    unsigned tid;             // thread of the CTA (per_task)
};

// Issues the TMA loads of the tile (thread 0) and waits for them with a bounded
// wait of `polls` polls on `phase` of the mbarrier (initialised here when
// `init`).  Returns false (uniformly across the CTA) if the wait gave up; *err
// is then set, after a second bounded wait has let the copies in flight land.
template <int NV, int SP, int TR, bool LOOP>
__device__ __forceinline__ bool load_tile(float* Qs, const CUtensorMap* tmap, int x0, int y0, uint64_t* bar,
                                          uint32_t phase, bool init, unsigned tid, int* err, uint32_t polls = kWaitPolls) {
    constexpr int PS = SP * TR;
    // Each variable's plane is the destination of a tensor copy, which must
    // start on a 128-byte boundary: tiles whose (W+8) x (H+4) plane is not a
    // multiple of 32 floats would misalign every plane after the first.
    static_assert((PS * sizeof(float)) % 128 == 0, "variable planes in shared memory must be 128-byte aligned");
    if (thread_of<LOOP>(tid) == 0) {
        if (init) {
            mbar_init(bar, 1);
            fence_barrier_init();
        }
        // The CTA's generic-proxy reads and writes of the previous tile in this
        // buffer (ordered before this point by the last barrier) must precede
        // the async-proxy writes of the new load.
        fence_proxy_async_shared();
        mbar_arrive_expect_tx(bar, NV * PS * (uint32_t)sizeof(float));
#pragma unroll
        for (int v = 0; v < NV; ++v) tma_load_2d(Qs + v * PS, tmap + v, x0, y0, bar);
    }
    __syncthreads();
    const bool ok = mbar_wait_bounded(bar, phase, polls);
    const int failed = __syncthreads_or(ok ? 0 : 1);
    if (failed) {
        if (thread_of<LOOP>(tid) == 0) atomicOr(err, kTileLoadGaveUp);
        mbar_wait_bounded(bar, phase, kWaitPolls);  // let copies in flight land before the CTA moves on
        return false;
    }
    return true;
}

// The same tile as load_tile, brought in by the CTA's threads with 16-byte
// asynchronous copies instead of a tensor map: the box of SP x TR floats at
// storage (x0, y0) of each input plane, with the tensor maps' extents
// (nx + 8 columns, ny + 4 rows) and their zero fill beyond them, so the shared
// tile holds the same values.  The batched kernels use it: their simulations
// are only known on the device, and a tensor map in global memory needs a
// proxy fence before every use, which measured about 10 us per tile.  Storage
// rows start on 16-byte boundaries and x0 is a multiple of 4, so every chunk
// is aligned; a chunk that straddles column nx + 8 copies its valid floats.
template <int NV, int SP, int TR, int NT>
__device__ __forceinline__ void load_tile_async(float* Qs, const TileJob& J) {
    constexpr int PS = SP * TR, CH = SP / 4, G = NT / CH;  // G rows of CH chunks at a time
    static_assert(SP % 4 == 0 && G >= 1, "shared rows of whole 16-byte chunks, one chunk per thread");
    // thread k copies chunk c = k % CH of tile rows g, g + G, g + 2G, ... (g = k / CH)
    const int c = threadIdx.x % CH, g = threadIdx.x / CH;
    if (g < G) {
        const float* in[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) in[v] = J.in[v];
        const int col = J.x0 + 4 * c;
        const uint32_t bytes = 4u * (uint32_t)max(0, min(4, J.nx + 8 - col));  // the tensor maps' nx + 8 columns
        const int rows = J.ny + 4 - J.y0;                                       // and ny + 4 rows
        long long gi = (long long)(J.y0 + g) * J.pitch + col;
        const long long gstep = (long long)G * J.pitch;
        float* dst = Qs + g * SP + 4 * c;
        for (int t = g; t < TR; t += G, gi += gstep, dst += G * SP) {
            const bool in_rows = t < rows;
#pragma unroll
            for (int v = 0; v < NV; ++v) cp_async16(dst + v * PS, in[v] + (in_rows ? gi : 0), in_rows ? bytes : 0u);
        }
    }
    cp_async_wait_all();
    __syncthreads();
}

__device__ __forceinline__ float sign_x(int v) { return v == 1 ? -1.0f : 1.0f; }
__device__ __forceinline__ float sign_y(int v) { return v == 2 ? -1.0f : 1.0f; }

// Ghost cells of a tile that reaches the domain boundary, with readBlock's
// semantics (GPUSimulators/cuda/common.h:248-351): periodic sides read the
// wrapped cell from global memory, then reflective sides mirror interior cells
// with the normal momentum negated, north, south, east, west in turn.
// Dirichlet ghosts keep the stored values the TMA load brought in.
template <int NV, int W, int H, int NT, int SP, bool LOOP, int UNROLL>
__device__ void apply_boundary(float* Qs, const TileJob& J) {
    constexpr int TR = H + 4, PS = SP * TR;
    const int nx = J.nx, ny = J.ny, bc = J.bc, x0 = J.x0, y0 = J.y0;
    const bool pw = bc_west(bc) == BC_PERIODIC, pe = bc_east(bc) == BC_PERIODIC;
    const bool ps = bc_south(bc) == BC_PERIODIC, pn = bc_north(bc) == BC_PERIODIC;
    if (pw || pe || ps || pn) {
        // The ghost rows and columns this tile holds, two of each side at most,
        // as one list of cells: whole rows first, then the columns' other
        // cells.  A thread has a few of them, whose loads are in flight
        // together.  Scanning the whole tile for them took one L2 round trip
        // after another, and the tiles at the walls held the others up.
        // Periodic walls, us per step before and after (reflective walls):
        // KP07_dimsplit 256 x 256 13.8, 10.6 (9.9), 777 x 1333 with 60 x 60
        // tiles 40.3, 28.1 (23.2); EE2D 2048 x 2048 113, 108 (104); FORCE
        // 777 x 1333 11.9, 8.9 (7.9).  UNROLL: loads of a variable in flight per
        // thread (batched_blocks has the reason for fewer).
        const int row_n = ny - y0 + 2, col_e = nx - x0 + 4;  // tile row of y = ny, tile column of x = nx
        const int lo_r = (ps && y0 == 0) ? 2 : 0, hi_r = pn ? max(0, min(2, TR - row_n)) : 0;
        const int lo_c = (pw && x0 == 0) ? 2 : 0, hi_c = pe ? max(0, min(2, SP - col_e)) : 0;
        const int in_rows = (lo_r + hi_r) * SP, all = in_rows + (lo_c + hi_c) * TR;
#pragma unroll UNROLL
        for (int i = thread_of<LOOP>(J.tid); i < all; i += NT) {
            int t, s;
            bool use = true;
            if (i < in_rows) {
                const int k = i / SP;
                s = i - k * SP;
                t = k < lo_r ? k : row_n + k - lo_r;
            } else {
                const int k = (i - in_rows) / TR;
                t = i - in_rows - k * TR;
                s = k < lo_c ? 2 + k : col_e + k - lo_c;
                use = t >= lo_r && !(hi_r > 0 && t >= row_n);  // not in a row above
            }
            const int x = x0 - 4 + s, y = y0 - 2 + t;
            use = use && x >= -2 && x < nx + 2 && y < ny + 2;
            if (use) {
                const int xs = (x < 0 && pw) ? x + nx : (x >= nx && pe) ? x - nx : x;
                const int ys = (y < 0 && ps) ? y + ny : (y >= ny && pn) ? y - ny : y;
                const long long gi = cell_index(ys, xs, J.pitch);
#pragma unroll
                for (int v = 0; v < NV; ++v) Qs[v * PS + t * SP + s] = __ldcg(J.in[v] + gi);
            }
        }
        __syncthreads();
    }
    // Tile row of domain row y: t = y - y0 + 2; tile column of x: s = x - x0 + 4.
    if (bc_north(bc) == BC_REFLECTIVE && y0 + H + 2 > ny) {
        for (int i = thread_of<LOOP>(J.tid); i < 2 * SP; i += NT) {
            const int m = i / SP, s = i - m * SP;
            const int t = ny + m - y0 + 2, ts = ny - 1 - m - y0 + 2;
            if (t < TR) {
#pragma unroll
                for (int v = 0; v < NV; ++v) Qs[v * PS + t * SP + s] = sign_y(v) * Qs[v * PS + ts * SP + s];
            }
        }
        __syncthreads();
    }
    if (bc_south(bc) == BC_REFLECTIVE && y0 == 0) {
        for (int i = thread_of<LOOP>(J.tid); i < 2 * SP; i += NT) {
            const int m = i / SP, s = i - m * SP;
            const int t = -1 - m + 2, ts = m + 2;
            if (ts < TR) {
#pragma unroll
                for (int v = 0; v < NV; ++v) Qs[v * PS + t * SP + s] = sign_y(v) * Qs[v * PS + ts * SP + s];
            }
        }
        __syncthreads();
    }
    if (bc_east(bc) == BC_REFLECTIVE && x0 + W + 2 > nx) {
        for (int i = thread_of<LOOP>(J.tid); i < 2 * TR; i += NT) {
            const int m = i / TR, t = i - m * TR;
            const int s = nx + m - x0 + 4, ss = nx - 1 - m - x0 + 4;
            if (s < SP) {
#pragma unroll
                for (int v = 0; v < NV; ++v) Qs[v * PS + t * SP + s] = sign_x(v) * Qs[v * PS + t * SP + ss];
            }
        }
        __syncthreads();
    }
    if (bc_west(bc) == BC_REFLECTIVE && x0 == 0) {
        for (int i = thread_of<LOOP>(J.tid); i < 2 * TR; i += NT) {
            const int m = i / TR, t = i - m * TR;
            const int s = -1 - m + 4, ss = m + 4;
            if (ss < SP) {
#pragma unroll
                for (int v = 0; v < NV; ++v) Qs[v * PS + t * SP + s] = sign_x(v) * Qs[v * PS + t * SP + ss];
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ line walkers

// Variable slot of logical component v along a line: y lines see (h, hv, hu)
// ("transposing" the domain, GPUSimulators/cuda/SWE2D_KP07_dimsplit.cu:81-107).
template <bool SWAP> __device__ __forceinline__ constexpr int vslot(int v) {
    return SWAP ? (v == 1 ? 2 : (v == 2 ? 1 : v)) : v;
}

template <int NV, bool SWAP, int PS>
__device__ __forceinline__ void ld_cell(const float* line, int k, int step, float (&q)[NV]) {
    const float* p = line + k * step;
#pragma unroll
    for (int v = 0; v < NV; ++v) q[v] = p[vslot<SWAP>(v) * PS];
}

template <int NV, bool SWAP, int PS>
__device__ __forceinline__ void st_cell(float* line, int k, int step, const float (&q)[NV]) {
    float* p = line + k * step;
#pragma unroll
    for (int v = 0; v < NV; ++v) p[vslot<SWAP>(v) * PS] = q[v];
}

// Two lines walked side by side: the second line starts d2 floats after the
// first; lane x of a pair is the first line, lane y the second.
template <int NV, bool SWAP, int PS>
__device__ __forceinline__ void ld_cell(const float* line, int k, int step, int d2, f2 (&q)[NV]) {
    const float* p = line + k * step;
#pragma unroll
    for (int v = 0; v < NV; ++v) q[v] = f2{p[vslot<SWAP>(v) * PS], p[vslot<SWAP>(v) * PS + d2]};
}

template <int NV, bool SWAP, int PS>
__device__ __forceinline__ void st_cell(float* line, int k, int step, int d2, const f2 (&q)[NV]) {
    float* p = line + k * step;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        p[vslot<SWAP>(v) * PS] = q[v].x;
        p[vslot<SWAP>(v) * PS + d2] = q[v].y;
    }
}

template <int NV, bool SWAP, int PS>
__device__ __forceinline__ void ld_cell(const float* line, int k, int step, int, float (&q)[NV]) {
    ld_cell<NV, SWAP, PS>(line, k, step, q);
}

template <int NV, bool SWAP, int PS>
__device__ __forceinline__ void st_cell(float* line, int k, int step, int, const float (&q)[NV]) {
    st_cell<NV, SWAP, PS>(line, k, step, q);
}

// Physics policies for the MUSCL-Hancock walker; N is float (one line per
// thread) or f2 (two lines per thread).
template <class N>
struct SwePhys {
    static constexpr int NV = 3;
    using Num = N;
    using Face = SweFaceT<N>;
    N theta2, g, half_g, k2;  // theta2 = 2 * theta (swe_muscl_hancock)
    __device__ __forceinline__ void recon(const N (&qm)[3], const N (&q0)[3], const N (&qp)[3], N (&bd)[3], Face& w,
                                          Face& e) const {
        swe_muscl_hancock(qm, q0, qp, bd, theta2, g, half_g, k2, w, e);
    }
    template <bool HLLF> __device__ __forceinline__ static void flux(const Face& l, const Face& r, N (&F)[3]) {
        if (HLLF) swe_hll(l, r, F);
        else swe_central_upwind(l, r, F);
    }
};

template <class N>
struct EulerPhys {
    static constexpr int NV = 4;
    using Num = N;
    using Face = EulerFaceT<N>;
    N theta2, gamma, gm1, k2;  // theta2 = 2 * theta, gm1 = gamma - 1
    __device__ __forceinline__ void recon(const N (&qm)[4], const N (&q0)[4], const N (&qp)[4], N (&bd)[4], Face& w,
                                          Face& e) const {
        euler_muscl_hancock(qm, q0, qp, bd, theta2, gamma, gm1, k2, w, e);
    }
    template <bool HLLF> __device__ __forceinline__ static void flux(const Face& l, const Face& r, N (&F)[4]) {
        if (HLLF) euler_hll(l, r, F);
        else euler_central_upwind(l, r, F);
    }
};

// One MUSCL-Hancock window step at cell c: shift in Q[c+1], reconstruct c,
// flux at c-1/2, update cell c-1 (GPUSimulators/cuda/common.h:444-475).
template <class Phys, bool HLLF, bool SWAP, int PS, class N = typename Phys::Num>
__device__ __forceinline__ void mh_step(float* line, int step, int d2, int c, N (&qm)[Phys::NV], N (&q0)[Phys::NV],
                                        N (&qp)[Phys::NV], const N (&qn)[Phys::NV], N (&bd)[Phys::NV],
                                        typename Phys::Face& eL, N (&Fprev)[Phys::NV], const Phys& P, N kdx,
                                        bool update) {
    constexpr int NV = Phys::NV;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        qm[v] = q0[v];
        q0[v] = qp[v];
        qp[v] = qn[v];
    }
    typename Phys::Face w, e;
    P.recon(qm, q0, qp, bd, w, e);
    N F[NV];
    Phys::template flux<HLLF>(eL, w, F);
    if (update) {
        N out[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) out[v] = ffma(fsub(Fprev[v], F[v]), kdx, qm[v]);
        st_cell<NV, SWAP, PS>(line, c - 1, step, d2, out);
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) Fprev[v] = F[v];
    eL = e;
}

// Updates cells [a, b) of a line (of two lines, d2 floats apart, for f2) in
// place.  pre holds Q[a-2], Q[a-1], Q[b], Q[b+1].
template <class Phys, bool HLLF, bool SWAP, int PS, class N = typename Phys::Num>
__device__ __forceinline__ void walk_mh(float* line, int step, int d2, int a, int b, const N (&pre)[4][Phys::NV],
                                        const Phys& P, N kdx) {
    constexpr int NV = Phys::NV;
    N qm[NV], q0[NV], qp[NV], qn[NV], Fprev[NV], bd[NV];
    typename Phys::Face eL;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
        q0[v] = pre[0][v];
        qp[v] = pre[1][v];
        Fprev[v] = splat<N>(0.0f);
    }
    // c = a-1: reconstruct only
    ld_cell<NV, SWAP, PS>(line, a, step, d2, qn);
    {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            qm[v] = q0[v];
            q0[v] = qp[v];
            qp[v] = qn[v];
            bd[v] = fmul(fsub(q0[v], qm[v]), P.theta2);
        }
        typename Phys::Face w;
        P.recon(qm, q0, qp, bd, w, eL);
    }
    // c = a: first face, no update
    ld_cell<NV, SWAP, PS>(line, a + 1, step, d2, qn);
    mh_step<Phys, HLLF, SWAP, PS>(line, step, d2, a, qm, q0, qp, qn, bd, eL, Fprev, P, kdx, false);
    // unrolled by the window's length, so the rotation of the three-cell
    // window becomes register renaming instead of moves
#pragma unroll 3
    for (int c = a + 1; c < b - 1; ++c) {
        ld_cell<NV, SWAP, PS>(line, c + 1, step, d2, qn);
        mh_step<Phys, HLLF, SWAP, PS>(line, step, d2, c, qm, q0, qp, qn, bd, eL, Fprev, P, kdx, true);
    }
    mh_step<Phys, HLLF, SWAP, PS>(line, step, d2, b - 1, qm, q0, qp, pre[2], bd, eL, Fprev, P, kdx, true);
    mh_step<Phys, HLLF, SWAP, PS>(line, step, d2, b, qm, q0, qp, pre[3], bd, eL, Fprev, P, kdx, true);
}

// Two-point flux walker (FORCE, HLL: GPUSimulators/cuda/SWE2D_FORCE.cu:29-81,
// SWE2D_HLL.cu:32-86).  pre holds Q[a-1] (slot 1) and Q[b] (slot 2).
// For HLL, VAR picks the flux: 0 HLL, 1 HLLC, 2 Godunov centred.
template <int SCHEME, bool SWAP, int PS, int VAR>
__device__ __forceinline__ void walk_2pt(float* line, int step, int a, int b, const float (&pre)[4][3], float g,
                                         float half_g, float kx, float kw, float kdx) {
    auto face_flux = [&](const SweFace& l, const SweFace& r, float (&F)[3]) {
        if constexpr (SCHEME == FORCE) swe_force(l, r, g, half_g, kx, kw, F);
        else if constexpr (VAR == 1) swe_hllc(l, r, F);
        else if constexpr (VAR == 2) swe_godc(l, r, g, half_g, kdx, F);
        else swe_hll(l, r, F);
    };
    SweFace sL = swe_face(pre[1][0], pre[1][1], pre[1][2], g, half_g);
    float qa[3];
    ld_cell<3, SWAP, PS>(line, a, step, qa);
    SweFace s = swe_face(qa[0], qa[1], qa[2], g, half_g);
    float Fprev[3];
    face_flux(sL, s, Fprev);
    float qprev[3] = {qa[0], qa[1], qa[2]};
    sL = s;
#pragma unroll 2
    for (int c = a + 1; c <= b; ++c) {
        float q[3];
        if (c < b) {
            ld_cell<3, SWAP, PS>(line, c, step, q);
        } else {
#pragma unroll
            for (int v = 0; v < 3; ++v) q[v] = pre[2][v];
        }
        s = swe_face(q[0], q[1], q[2], g, half_g);
        float F[3];
        face_flux(sL, s, F);
        float out[3];
#pragma unroll
        for (int v = 0; v < 3; ++v) out[v] = fmaf(Fprev[v] - F[v], kdx, qprev[v]);
        st_cell<3, SWAP, PS>(line, c - 1, step, out);
#pragma unroll
        for (int v = 0; v < 3; ++v) {
            Fprev[v] = F[v];
            qprev[v] = q[v];
        }
        sL = s;
    }
}

// WAF walker (GPUSimulators/cuda/SWE2D_WAF.cu:35-87): the flux at c-1/2 uses
// cells c-2 .. c+1; per-cell quantities and the star depths of neighbouring
// pairs are carried along the window.  N = f2 walks two lines d2 floats apart.
template <bool SWAP, int PS, int LIM, class N>
__device__ __forceinline__ void walk_waf(float* line, int step, int d2, int a, int b, const N (&pre)[4][3], N g,
                                         N half_g, N inv_g, N dtdx, N kdx, float beta) {
    constexpr int limiter = LIM;
    WafCellT<N> C0 = waf_cell(pre[0], g, half_g);
    WafCellT<N> C1 = waf_cell(pre[1], g, half_g);
    N q[3];
    ld_cell<3, SWAP, PS>(line, a, step, d2, q);
    WafCellT<N> C2 = waf_cell(q, g, half_g);
    ld_cell<3, SWAP, PS>(line, a + 1, step, d2, q);
    WafCellT<N> C3 = waf_cell(q, g, half_g);
    N hs01 = waf_h_star(C0, C1, inv_g), hs12 = waf_h_star(C1, C2, inv_g), hs23 = waf_h_star(C2, C3, inv_g);
    N Fprev[3];
    waf_flux(C0, C1, C2, C3, hs01, hs12, hs23, dtdx, Fprev, limiter, beta);  // face a-1/2
#pragma unroll 4
    for (int c = a + 1; c <= b; ++c) {
        if (c + 1 < b) {
            ld_cell<3, SWAP, PS>(line, c + 1, step, d2, q);
        } else {
            // a select, not pre[k]: a run-time index would put pre in local memory
            const bool first = (c + 1 == b);
#pragma unroll
            for (int v = 0; v < 3; ++v) q[v] = first ? pre[2][v] : pre[3][v];
        }
        C0 = C1;
        C1 = C2;
        C2 = C3;
        C3 = waf_cell(q, g, half_g);
        hs01 = hs12;
        hs12 = hs23;
        hs23 = waf_h_star(C2, C3, inv_g);
        N F[3];
        waf_flux(C0, C1, C2, C3, hs01, hs12, hs23, dtdx, F, limiter, beta);  // face c-1/2
        N out[3];
#pragma unroll
        for (int v = 0; v < 3; ++v) out[v] = ffma(fsub(Fprev[v], F[v]), kdx, C1.q[v]);
        st_cell<3, SWAP, PS>(line, c - 1, step, d2, out);
#pragma unroll
        for (int v = 0; v < 3; ++v) Fprev[v] = F[v];
    }
}

// Per-scheme parameters of one sweep direction.  The ratios of the time step
// to the cell size are formed once per sweep, here, for every walker (one
// line or two lines per thread), so each tile configuration uses the same
// bits.
struct SweepPar {
    float theta, g, half_g, inv_g, gamma;
    float kdt;   // kernel dt
    float dxx;   // cell size along the sweep
    float kdx;   // kdt / dxx
    float k2;    // kdt / (2 dxx)
    float beta;   // parameter of the Osher and Sweby limiters
    __device__ __forceinline__ void set_direction(float cell) {
        dxx = cell;
        kdx = fdiv_fast(kdt, cell);
        k2 = fmul(kdx, 0.5f);
    }
};

// VAR: HLL's flux variant or WAF's limiter (walk_2pt, flux_limiter); 0 is the
// reference's.  It is a template parameter so that each kernel inlines one.
template <int SCHEME, bool SWAP, int PS, int VAR>
__device__ __forceinline__ void walk_line(float* line, int step, int a, int b, const float (&pre)[4][(SCHEME == EE2D) ? 4 : 3],
                                          const SweepPar& p) {
    const float kdx = p.kdx;
    if constexpr (SCHEME == KP07_DIMSPLIT || SCHEME == HLL2) {
        const SwePhys<float> P{minmod_theta2(p.theta), p.g, p.half_g, p.k2};
        walk_mh<SwePhys<float>, SCHEME == HLL2, SWAP, PS>(line, step, 0, a, b, pre, P, kdx);
    } else if constexpr (SCHEME == EE2D) {
        const EulerPhys<float> P{minmod_theta2(p.theta), p.gamma, fsub(p.gamma, 1.0f), p.k2};
        // x sweeps use HLL, y sweeps central-upwind (GPUSimulators/cuda/EE2D_KP07_dimsplit.cu:62, :106)
        walk_mh<EulerPhys<float>, !SWAP, SWAP, PS>(line, step, 0, a, b, pre, P, kdx);
    } else if constexpr (SCHEME == WAF) {
        walk_waf<SWAP, PS, VAR>(line, step, 0, a, b, pre, p.g, p.half_g, p.inv_g, kdx, kdx, p.beta);
    } else {
        walk_2pt<SCHEME, SWAP, PS, VAR>(line, step, a, b, pre, p.g, p.half_g, fdiv_fast(p.dxx, fmul(2.0f, p.kdt)),
                                        p.k2, kdx);
    }
}

// Two lines, d2 floats apart, walked side by side in packed arithmetic
// (the MUSCL-Hancock schemes).  Each cell gets the same bits as walk_line.
template <int SCHEME, bool SWAP, int PS, int VAR>
__device__ __forceinline__ void walk_line2(float* line, int step, int d2, int a, int b,
                                           const f2 (&pre)[4][(SCHEME == EE2D) ? 4 : 3], const SweepPar& p) {
    static_assert(SCHEME == KP07_DIMSPLIT || SCHEME == HLL2 || SCHEME == EE2D || SCHEME == WAF,
                  "packed walkers: MUSCL-Hancock schemes and WAF");
    const f2 kdx = splat<f2>(p.kdx);
    if constexpr (SCHEME == WAF) {
        walk_waf<SWAP, PS, VAR>(line, step, d2, a, b, pre, splat<f2>(p.g), splat<f2>(p.half_g), splat<f2>(p.inv_g),
                                kdx, kdx, p.beta);
    } else if constexpr (SCHEME == EE2D) {
        const EulerPhys<f2> P{splat<f2>(minmod_theta2(p.theta)), splat<f2>(p.gamma), splat<f2>(fsub(p.gamma, 1.0f)),
                              splat<f2>(p.k2)};
        walk_mh<EulerPhys<f2>, !SWAP, SWAP, PS>(line, step, d2, a, b, pre, P, kdx);
    } else {
        const SwePhys<f2> P{splat<f2>(minmod_theta2(p.theta)), splat<f2>(p.g), splat<f2>(p.half_g), splat<f2>(p.k2)};
        walk_mh<SwePhys<f2>, SCHEME == HLL2, SWAP, PS>(line, step, d2, a, b, pre, P, kdx);
    }
}

// Sets a walker's prefetched cells where it has none.  In a looping kernel they
// would otherwise count as kept from the last task, a register each.
template <class N, int M, int NV>
__device__ __forceinline__ void clear(N (&pre)[M][NV]) {
#pragma unroll
    for (int m = 0; m < M; ++m)
#pragma unroll
        for (int v = 0; v < NV; ++v) pre[m][v] = splat<N>(0.0f);
}

// x sweep over tile rows [t0, t1): interior columns updated in place.
// LPT = 2: a thread walks rows t and t + (t1 - t0)/2 side by side.
template <int SCHEME, int NV, int W, int H, int NT, int VAR, int LPT, bool LOOP>
__device__ __forceinline__ void sweep_x(float* Qs, unsigned tid, int t0, int t1, const SweepPar& p) {
    constexpr int SP = split_pitch(W), PS = SP * (H + 4), NSEG = split_nseg_x(W), R = W / NSEG;
    const int item = thread_of<LOOP>(tid);
    const int nlines = (t1 - t0) / LPT;
    const bool has = item < nlines * NSEG;
    const int t = t0 + item / NSEG, seg = item % NSEG;
    const int a = 4 + seg * R, b = a + R;
    float* line = Qs + t * SP;
    if constexpr (LPT == 1) {
        float pre[4][NV];
        if (has) {
            ld_cell<NV, false, PS>(line, a - 2, 1, pre[0]);
            ld_cell<NV, false, PS>(line, a - 1, 1, pre[1]);
            ld_cell<NV, false, PS>(line, b, 1, pre[2]);
            ld_cell<NV, false, PS>(line, b + 1, 1, pre[3]);
        }
        if constexpr (LOOP) {
            if (!has) clear(pre);
        }
        __syncthreads();
        if (has) walk_line<SCHEME, false, PS, VAR>(line, 1, a, b, pre, p);
    } else {
        const int d2 = nlines * SP;
        f2 pre[4][NV];
        if (has) {
            ld_cell<NV, false, PS>(line, a - 2, 1, d2, pre[0]);
            ld_cell<NV, false, PS>(line, a - 1, 1, d2, pre[1]);
            ld_cell<NV, false, PS>(line, b, 1, d2, pre[2]);
            ld_cell<NV, false, PS>(line, b + 1, 1, d2, pre[3]);
        }
        if constexpr (LOOP) {
            if (!has) clear(pre);
        }
        __syncthreads();
        if (has) walk_line2<SCHEME, false, PS, VAR>(line, 1, d2, a, b, pre, p);
    }
    __syncthreads();
}

// y sweep over tile columns [s0, s1): interior rows updated in place.
// LPT = 2: a thread walks columns s and s + (s1 - s0)/2 side by side.
template <int SCHEME, int NV, int W, int H, int NT, int VAR, int LPT, bool LOOP>
__device__ __forceinline__ void sweep_y(float* Qs, unsigned tid, int s0, int s1, const SweepPar& p) {
    constexpr int SP = split_pitch(W), PS = SP * (H + 4);
    constexpr int NSEG = NT * LPT / (W + 4), R = H / NSEG;
    const int ncols = (s1 - s0) / LPT;
    const int item = thread_of<LOOP>(tid);
    const bool has = item < ncols * NSEG;
    const int s = s0 + item % ncols, seg = item / ncols;
    const int a = 2 + seg * R, b = a + R;
    float* line = Qs + s;
    if constexpr (LPT == 1) {
        float pre[4][NV];
        if (has) {
            ld_cell<NV, true, PS>(line, a - 2, SP, pre[0]);
            ld_cell<NV, true, PS>(line, a - 1, SP, pre[1]);
            ld_cell<NV, true, PS>(line, b, SP, pre[2]);
            ld_cell<NV, true, PS>(line, b + 1, SP, pre[3]);
        }
        if constexpr (LOOP) {
            if (!has) clear(pre);
        }
        __syncthreads();
        if (has) walk_line<SCHEME, true, PS, VAR>(line, SP, a, b, pre, p);
    } else {
        const int d2 = ncols;
        f2 pre[4][NV];
        if (has) {
            ld_cell<NV, true, PS>(line, a - 2, SP, d2, pre[0]);
            ld_cell<NV, true, PS>(line, a - 1, SP, d2, pre[1]);
            ld_cell<NV, true, PS>(line, b, SP, d2, pre[2]);
            ld_cell<NV, true, PS>(line, b + 1, SP, d2, pre[3]);
        }
        if constexpr (LOOP) {
            if (!has) clear(pre);
        }
        __syncthreads();
        if (has) walk_line2<SCHEME, true, PS, VAR>(line, SP, d2, a, b, pre, p);
    }
    __syncthreads();
}

// ------------------------------------------------------------------ tiles of the split schemes

// Scheme constants of a split-scheme tile.
struct SplitPar {
    float dx, dy, g, gamma, theta;
    float kdt;  // kernel dt of this substep
    int substep;
    float beta;  // parameter of the Osher and Sweby limiters
};

// Load, ghost cells, both sweeps and copy-out of one tile of a split scheme
// (FORCE, HLL, HLL2, WAF, KP07_dimsplit, EE2D).  Accumulates the tile's CFL
// minimum into the per-thread value.  Returns false if the tile load gave up
// (nothing was written).
// ASYNC_LOAD (batched kernels): the tile comes in through load_tile_async
// instead of the TMA (bar, phase, init_bar, err and polls are then unused).
// HEALTH (batched kernels): with `health` set, *unhealthy becomes true if any
// written cell holds a non-finite value or a non-positive depth (density).
template <int SCHEME, int W, int H, int NT, bool ASYNC_LOAD = false, int VAR = 0, int LPT = 1, bool HEALTH = false,
          bool LOOP = false>
__device__ bool process_tile_dimsplit(float* Qs, uint64_t* bar, uint32_t phase, bool init_bar, const TileJob& J,
                                      const SplitPar& P, bool do_cfl, int* err, float& my_cfl,
                                      uint32_t polls = kWaitPolls, bool health = false, bool* unhealthy = nullptr) {
    constexpr int NV = (SCHEME == EE2D) ? 4 : 3;
    constexpr int G = (SCHEME == FORCE || SCHEME == HLL) ? 1 : 2;
    constexpr int SP = split_pitch(W), TR = H + 4, PS = SP * TR, NSEG_X = split_nseg_x(W);
    static_assert(W % NSEG_X == 0 && (W / NSEG_X) % 2 == 1 && (NSEG_X == 4 ? SP % 8 == 4 : SP % 32 == 8),
                  "row segments must be odd and the pitch an odd multiple of 4 (8 mod 32) for conflict-free x sweeps");
    static_assert(TR * NSEG_X <= NT * LPT, "one x-sweep segment (LPT lines) per thread");
    static_assert((NT * LPT) / (W + 4) >= 1 && H % ((NT * LPT) / (W + 4)) == 0, "y-sweep segments must tile the block");
    static_assert(W / NSEG_X >= 2 && H / ((NT * LPT) / (W + 4)) >= 2,
                  "a walker reads its segment's second cell after its neighbours may have updated theirs");
    static_assert(LPT == 1 || (LPT == 2 && H % 2 == 0 &&
                               (SCHEME == KP07_DIMSPLIT || SCHEME == HLL2 || SCHEME == EE2D || SCHEME == WAF)),
                  "two lines per thread: MUSCL-Hancock schemes and WAF, with an even number of tile rows");
    if constexpr (ASYNC_LOAD) {
        load_tile_async<NV, SP, TR, NT>(Qs, J);
    } else {
        if (!load_tile<NV, SP, TR, LOOP>(Qs, J.tmap, J.x0, J.y0, bar, phase, init_bar, J.tid, err, polls)) return false;
    }
    const int x0 = J.x0, y0 = J.y0;
    if (x0 == 0 || x0 + W + 2 > J.nx || y0 == 0 || y0 + H + 2 > J.ny) apply_boundary<NV, W, H, NT, SP, LOOP, (SCHEME == WAF && ASYNC_LOAD) ? 1 : 4>(Qs, J);

    SweepPar p;
    p.theta = P.theta;
    p.g = P.g;
    p.half_g = fmul(0.5f, P.g);
    p.inv_g = frcp_fast(P.g);
    p.gamma = P.gamma;
    p.kdt = P.kdt;
    p.beta = P.beta;
    const bool x_first = (SCHEME == FORCE || SCHEME == HLL) ? true : (P.substep == 0);
    if (x_first) {
        p.set_direction(P.dx);
        sweep_x<SCHEME, NV, W, H, NT, VAR, LPT, LOOP>(Qs, J.tid, 2 - G, H + 2 + G, p);
        p.set_direction(P.dy);
        sweep_y<SCHEME, NV, W, H, NT, VAR, LPT, LOOP>(Qs, J.tid, 4, W + 4, p);
    } else {
        p.set_direction(P.dy);
        sweep_y<SCHEME, NV, W, H, NT, VAR, LPT, LOOP>(Qs, J.tid, 4 - G, W + 4 + G, p);
        p.set_direction(P.dx);
        sweep_x<SCHEME, NV, W, H, NT, VAR, LPT, LOOP>(Qs, J.tid, 2, H + 2, p);
    }

    // copy-out of the interior (+ gravity source, CFL); the output plane
    // pointers are read once (for batched kernels they live in global memory,
    // where a store through a float pointer could otherwise force a reload)
    constexpr int QW = W / 4;
    const float gg = (SCHEME == EE2D) ? P.gamma : P.g;
    float* outp[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) outp[v] = J.out[v];
    for (int i = thread_of<LOOP>(J.tid); i < H * QW; i += NT) {
        const int r = i / QW, q = i - r * QW;
        const int y = y0 + r, x = x0 + 4 * q;
        if (y >= J.ny || x >= J.nx) continue;
        float4 val[NV];
#pragma unroll
        for (int v = 0; v < NV; ++v) val[v] = *reinterpret_cast<const float4*>(Qs + v * PS + (r + 2) * SP + 4 + 4 * q);
        if (SCHEME == EE2D) {
            if (P.g > 0.0f) {
                // gravity source (GPUSimulators/cuda/EE2D_KP07_dimsplit.cu:197-205)
                const float gsrc = P.g;
                float* r0 = &val[0].x;
                float* r2 = &val[2].x;
                float* r3 = &val[3].x;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float rho_v = r2[j];
                    r2[j] = r2[j] - gsrc * r0[j] * P.kdt;
                    r3[j] = r3[j] - gsrc * rho_v * P.kdt;
                }
            }
        }
        const long long gi = cell_index(y, x, J.pitch);
        const int nvalid = min(4, J.nx - x);
        if (nvalid == 4) {
#pragma unroll
            for (int v = 0; v < NV; ++v) *reinterpret_cast<float4*>(outp[v] + gi) = val[v];
        } else {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const float* e = &val[v].x;
                for (int j = 0; j < nvalid; ++j) outp[v][gi + j] = e[j];
            }
        }
        if constexpr (HEALTH) {
            if (health) {
                bool bad = false;
                if (nvalid == 4) {
                    // NaN-propagating minimum of the depths (densities) and
                    // maximum of the other variables' magnitudes: the same
                    // verdict as the per-value tests below, in fewer instructions
                    const float hmin = vmin_nan(vmin3_nan(val[0].x, val[0].y, val[0].z), val[0].w);
                    float qmax = 0.0f;
#pragma unroll
                    for (int v = 1; v < NV; ++v)
                        qmax = vmax3_nan(qmax, vmax3_nan(fabsf(val[v].x), fabsf(val[v].y), fabsf(val[v].z)),
                                         fabsf(val[v].w));
                    bad = !(hmin > 0.0f) || !(qmax < __int_as_float(0x7f800000));
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (j < nvalid) {
                            bad |= !((&val[0].x)[j] > 0.0f);
#pragma unroll
                            for (int v = 1; v < NV; ++v)
                                bad |= !(fabsf((&val[v].x)[j]) < __int_as_float(0x7f800000));
                        }
                    }
                }
                if (bad) *unhealthy = true;
            }
        }
        if (do_cfl) {
            const float* h = &val[0].x;
            const float* hu = &val[1].x;
            const float* hv = &val[2].x;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < nvalid) my_cfl = fminf(my_cfl, cell_cfl(h[j], hu[j], hv[j], P.dx, P.dy, gg));
        }
    }
    return true;
}

// ------------------------------------------------------------------ tiles of the unsplit schemes (LxF, KP07)

__device__ __forceinline__ SweFace shfl_up_face(const SweFace& f, int d) {
    SweFace r;
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        r.q[v] = __shfl_up_sync(0xffffffffu, f.q[v], d);
        r.f[v] = __shfl_up_sync(0xffffffffu, f.f[v], d);
    }
    r.u = __shfl_up_sync(0xffffffffu, f.u, d);
    r.c = __shfl_up_sync(0xffffffffu, f.c, d);
    return r;
}

// Scheme constants of an unsplit tile.
struct UnsplitPar {
    float dx, dy, g, theta;
    float kdt;    // kernel dt of this stage
    int substep;  // RK stage (KP07)
    int order;    // RK order (KP07)
};

// One pass over the tile, as column walkers (GPUSimulators/cuda/SWE2D_LxF.cu:102-165,
// SWE2D_KP07.cu:136-232).  Lanes run along x: warp column wx of a row segment
// covers tile columns 3+30wx .. 34+30wx; lanes 1..30 update interior columns
// 30wx .. 30wx+29, lanes 0 and 31 supply the states of the columns beside
// them.  At each row a lane builds the west and east face states of its cell;
// the flux at its west face takes the east state of the lane to its left
// (warp shuffle), and its east-face flux is the west-face flux of the lane
// to its right, so each x face is computed once.  Along y each lane keeps a
// sliding window: the north face state of the row above and the flux at the
// south face carry over from the previous row.  The updated cells (KP07
// stage 2 blended with the old output) go straight to global memory.
//
// Load, ghost cells, the one-pass update and the stores of one tile of an
// unsplit scheme (LxF, KP07); the per-thread CFL minimum is
// accumulated.  Returns false if the tile load gave up (nothing was written).
// ASYNC_LOAD (batched kernels): the tile comes in through load_tile_async.
// HEALTH (batched kernels): with `health` set, *unhealthy becomes true if a
// written cell holds a non-finite value or a non-positive depth.
template <int SCHEME, int W, int H, int NT, bool ASYNC_LOAD = false, bool HEALTH = false, bool LOOP = false>
__device__ bool process_tile_unsplit(float* Qs, uint64_t* bar, uint32_t phase, bool init_bar, const TileJob& J,
                                     const UnsplitPar& P, bool do_cfl, int* err, float& my_cfl,
                                     uint32_t polls = kWaitPolls, bool health = false, bool* unhealthy = nullptr) {
    constexpr int SP = W + 8, TR = H + 4, PS = SP * TR;
    constexpr int WX = W / 30, NSEG = NT / (32 * WX), R = H / NSEG;
    static_assert(W % 30 == 0 && NT % (32 * WX) == 0 && NSEG >= 1 && H % NSEG == 0,
                  "warps of 30 updated columns must tile the block");
    const int x0 = J.x0, y0 = J.y0;
    bool bad = false;
    if constexpr (ASYNC_LOAD) {
        load_tile_async<3, SP, TR, NT>(Qs, J);
    } else {
        if (!load_tile<3, SP, TR, LOOP>(Qs, J.tmap, x0, y0, bar, phase, init_bar, thread_of<LOOP>(J.tid), err, polls)) return false;
    }
    {
        if (x0 == 0 || x0 + W + 2 > J.nx || y0 == 0 || y0 + H + 2 > J.ny) apply_boundary<3, W, H, NT, SP, LOOP, 4>(Qs, J);
        const float kdt = P.kdt;
        const float g = P.g, half_g = fmul(0.5f, g), theta2 = minmod_theta2(P.theta);
        const float k4x = fdiv_fast(P.dx, fmul(4.0f, kdt)), k4y = fdiv_fast(P.dy, fmul(4.0f, kdt));
        const float kdx = fdiv_fast(kdt, P.dx), kdy = fdiv_fast(kdt, P.dy);
        const bool blend = (SCHEME == KP07) && P.order == 2 && P.substep == 1;

        const int warp = thread_of<LOOP>(J.tid) >> 5, lane = thread_of<LOOP>(J.tid) & 31;
        const int wx = warp % WX, seg = warp / WX;
        const int s = 3 + 30 * wx + lane;  // tile column of this lane
        const int x = x0 + s - 4;          // domain column
        const bool owner = lane >= 1 && lane <= 30;
        const int a = 2 + seg * R, b = a + R;  // tile rows updated by this segment

        // q of tile cell (t, c), components in (h, hu, hv) order
        auto qat = [&](int t, int c, float (&q)[3]) {
#pragma unroll
            for (int v = 0; v < 3; ++v) q[v] = Qs[v * PS + t * SP + c];
        };
        // y-face states of row t (south, north) from rows t-1, t, t+1 of this
        // column, components swapped to (h, hv, hu) as computeFluxG does
        // (GPUSimulators/cuda/SWE2D_KP07.cu:117-131).  The slope is formed at
        // twice its size (minmod_slope2); bd carries theta2*(q0 - qm) in and
        // theta2*(qp - q0) out, in q's component order, since a row's forward
        // difference is the next row's backward one.
        auto ystates = [&](const float (&qm)[3], const float (&q0)[3], const float (&qp)[3], float (&bd)[3],
                           SweFace& sf, SweFace& nf) {
            float sv[3], nv[3];
#pragma unroll
            for (int v = 0; v < 3; ++v) {
                const int k = (v == 0) ? 0 : 3 - v;  // (h, hv, hu)
                if (SCHEME == LXF) {
                    sv[v] = nv[v] = q0[k];
                } else {
                    const float f = fmul(fsub(qp[k], q0[k]), theta2);
                    const float sl2 = minmod3(bd[k], fsub(qp[k], qm[k]), f);
                    bd[k] = f;
                    sv[v] = fmaf(-0.25f, sl2, q0[k]);
                    nv[v] = fmaf(0.25f, sl2, q0[k]);
                }
            }
            sf = swe_face(sv[0], sv[1], sv[2], g, half_g);
            nf = (SCHEME == LXF) ? sf : swe_face(nv[0], nv[1], nv[2], g, half_g);
        };
        auto yflux = [&](const SweFace& l, const SweFace& r, float (&G)[3]) {
            float tmp[3];
            if (SCHEME == LXF) swe_lxf_2d(l, r, k4y, tmp);
            else swe_central_upwind(l, r, tmp);
            G[0] = tmp[0];  // back to (h, hu, hv)
            G[1] = tmp[2];
            G[2] = tmp[1];
        };

        // window: rows a-1, a, a+1 of this column
        float qm[3], q0[3], qp[3];
        qat(a - 1, s, qm);
        qat(a, s, q0);
        qat(a + 1, s, qp);
        SweFace s_cur, n_cur, n_prev;
        float bdy[3];
        {
            float qmm[3];
            qat(a - 2, s, qmm);
#pragma unroll
            for (int v = 0; v < 3; ++v) bdy[v] = fmul(fsub(qm[v], qmm[v]), theta2);
            SweFace sd;
            ystates(qmm, qm, q0, bdy, sd, n_prev);  // row a-1
        }
        ystates(qm, q0, qp, bdy, s_cur, n_cur);  // row a
        float Gs[3];
        yflux(n_prev, s_cur, Gs);  // south face of row a
        // the lane's output column, from row a on; rows past the domain are not walked
        float* out[3];
#pragma unroll
        for (int v = 0; v < 3; ++v) out[v] = J.out[v] + cell_index(y0 + a - 2, x, J.pitch);
        const bool store = owner && x < J.nx;
        const int last = min(b, J.ny - y0 + 2);
        // KP07's second stage blends with the old output: a loop of its own, so
        // that the first one carries no selects.  With that, running output
        // pointers and one row bound instead of a test per row: 323 to 301 us
        // per step on 4096 x 4096, LxF 86.9 to 83.3 (the loop is bound by issue).
        auto walk = [&](auto blended) {
            // unrolled by the row window's length: its rotation becomes renaming
#pragma unroll 3
            for (int t = a; t < last; ++t) {
                float old[3];
                if constexpr (decltype(blended)::value) {
#pragma unroll
                    for (int v = 0; v < 3; ++v) old[v] = store ? __ldcg(out[v]) : 0.0f;
                }
                // x faces of (t, s): west and east states
                SweFace fw, fe;
                if (SCHEME == LXF) {
                    fw = fe = swe_face(q0[0], q0[1], q0[2], g, half_g);
                } else {
                    float ql[3], qr[3], wv[3], ev[3];
                    qat(t, s - 1, ql);
                    qat(t, s + 1, qr);
#pragma unroll
                    for (int v = 0; v < 3; ++v) {
                        const float sl2 = minmod_slope2(ql[v], q0[v], qr[v], theta2);
                        wv[v] = fmaf(-0.25f, sl2, q0[v]);
                        ev[v] = fmaf(0.25f, sl2, q0[v]);
                    }
                    fw = swe_face(wv[0], wv[1], wv[2], g, half_g);
                    fe = swe_face(ev[0], ev[1], ev[2], g, half_g);
                }
                const SweFace le = shfl_up_face(fe, 1);  // east state of the column to the left
                float Fw[3], Fe[3];
                if (SCHEME == LXF) swe_lxf_2d(le, fw, k4x, Fw);
                else swe_central_upwind(le, fw, Fw);
#pragma unroll
                for (int v = 0; v < 3; ++v) Fe[v] = __shfl_down_sync(0xffffffffu, Fw[v], 1);
                // y: states of row t+1, flux at the north face of row t
                float qn2[3];
                qat(t + 2, s, qn2);
                SweFace s_nxt, n_nxt;
                ystates(q0, qp, qn2, bdy, s_nxt, n_nxt);
                float Gn[3];
                yflux(n_cur, s_nxt, Gn);
                float qn[3], o[3];
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    qn[v] = q0[v] + fmaf(Fw[v] - Fe[v], kdx, (Gs[v] - Gn[v]) * kdy);
                    if constexpr (decltype(blended)::value) o[v] = 0.5f * (old[v] + qn[v]);
                    else o[v] = qn[v];
                }
                if (store) {
#pragma unroll
                    for (int v = 0; v < 3; ++v) {
                        *out[v] = o[v];
                        if constexpr (HEALTH) {
                            if (health) bad |= (v == 0) ? !(o[v] > 0.0f) : !(fabsf(o[v]) < __int_as_float(0x7f800000));
                        }
                    }
                    if (do_cfl) my_cfl = fminf(my_cfl, cell_cfl(qn[0], qn[1], qn[2], P.dx, P.dy, g));
                }
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    out[v] += J.pitch;
                    Gs[v] = Gn[v];
                    qm[v] = q0[v];
                    q0[v] = qp[v];
                    qp[v] = qn2[v];
                }
                s_cur = s_nxt;
                n_cur = n_nxt;
            }
        };
        if (SCHEME == KP07 && blend) walk(std::true_type{});
        else walk(std::false_type{});
    }
    if constexpr (HEALTH) {
        if (bad) *unhealthy = true;
    }
    return true;
}

// ------------------------------------------------------------------ stage kernel

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// CTAs per SM that a kernel is compiled for (0: the compiler's own choice).
//
// Packed kernels: as many as shared memory holds, at 128 registers or more per
// thread.  Told so, the compiler spends the registers that the shared tiles
// leave unused on overlapping more of a cell's arithmetic: EE2D 60 x 60 takes
// 164 instead of 127 at three CTAs per SM, 409 to 404 us per step on
// 4096 x 4096 and 34.0 to 30.6 on 1024 x 1024 (KP07_dimsplit 264.3 to 263.9,
// HLL2 335.4 to 334.3, WAF 505 to 506).
//
// The light schemes, and WAF on tiles whose shared memory keeps the threads per
// SM low: one, i.e. as many registers as the schedule likes: 4096 x 4096 HLL
// 134.5 to 124.7, FORCE 111.8 to 102.7, LxF 88.9 to 86.6; WAF 124 x 60 522 to
// 504.  The other one-line kernels lose the warps that hide their latencies:
// KP07 324 to 379, HLL2 60 x 60 374 to 442.  KP07 by 448 threads: two CTAs,
// 13.8 to 12.1 on 512 x 512.
__host__ __device__ constexpr int compiled_blocks(int scheme, int W, int H, int NT, int lpt) {
    if (lpt == 2) {
        const int tile = (scheme == EE2D ? 4 : 3) * split_pitch(W) * (H + 4) * (int)sizeof(float);
        const int by_smem = 228 * 1024 / (tile + 1024 + 256), by_regs = 65536 / (NT * 128);  // 228 KB per SM
        return by_smem < 1 ? 1 : by_smem < by_regs ? by_smem : by_regs;
    }
    if (scheme == KP07 && NT > 256) return 2;
    return scheme == LXF || scheme == FORCE || scheme == HLL || (scheme == WAF && W != 60) ? 1 : 0;
}

// Stage kernel of any scheme, with one CTA per task, a tile in one substep.
//
// A launch of one substep takes its tiles by block index.  A run of several
// substeps has no barrier between them: a CTA takes the next task, in the order
// substep by substep and row by row of tiles, and waits until the tiles within
// two cells of its own have completed the substep before, which is all that it
// reads and all that still reads what it overwrites.  Tasks are taken in the
// order in which CTAs start and depend on earlier ones only, so whatever part of
// the grid is resident makes progress; nothing needs the grid to be resident at
// once.  The waits are bounded: a CTA that gives up sets the error flag, and the
// run then goes on to its end with the state left undefined.
//
// A long run is a chain of launches, so that work of other streams gets its
// turn between them (chain_tasks).  They share the task and progress counters
// and start wherever in a substep the one before stopped.  A launch starts as
// soon as the one before has handed out its tasks; instead of the end of that
// one it waits for the tiles that it reads, as within a launch, so the chain has
// no gaps: KP07_dimsplit 4096 x 4096 in one launch per 100 steps, in a chain of
// 52, and in 17 launches that each wait for the end of the one before: 260.8,
// 261.6 and 265.6 us per step; LxF 84.4, 84.8 in 26, and 105.7 in 34.  Its CTAs
// end after the launch before has ended, so the end of the last launch is that of
// the run.
//
// LOOP: the form for GPUs shared with other simulations of the context.  The
// launch has fewer CTAs than tasks (loop_form) and each takes task after task,
// so that none is queued behind others and simulations run beside each other.
// us per step and simulation with 1, 2, 4 and 8 threads that each run one:
//                             a launch per substep    CTA per task            LOOP from 2 on
//   KP07_dimsplit 64 x 48     14.7  7.8  4.0  2.1     7.7  7.3  7.3  7.2      7.7  4.4  2.0  1.1
//   KP07_dimsplit 256 x 256   16.1  8.4  4.7  3.3     10.2 9.7  9.8  9.7      8.7  5.7  4.0  3.1
//   FORCE 777 x 1333          14.4  9.3  6.0  6.3     8.1  7.7  7.7  7.6      8.1  6.7  6.6  6.9
//   KP07_dimsplit 1024 x 1024 35.6 26.8 19.8 19.7     21.8 21.4 21.3 21.3     21.6 21.9 20.3 20.3
// A CTA keeps nothing but its task between two of them (per_task, clear): with
// what the compiler would keep, KP07_dimsplit's 28 x 28 tile takes 128 registers
// instead of 71.
//
// Against one launch per substep this fills the tail of a substep with the next
// one's tiles, lets tile loads overlap other tiles' sweeps where a substep is
// one wave or less, and has no launch, control-block read or arrival count per
// substep.  us per step on n x n cells, autotuned tiles: before (a launch per
// substep, replayed from graphs), with this alone, and as it is now, with the
// later launch bounds, column walks and small tiles:
//   n               256                1024               2048               4096
//   LxF             7.9   5.0   4.2    11.7   6.9   6.6   34.9  22.7  21.0    107    89    84
//   HLL             7.8   5.2   3.9    16.2  10.1   9.9   43.0  34.5  31.5    151   135   123
//   HLL2           16.9  12.3   9.1    41.4  27.5  27.5    115  89.4  85.6    376   349   334
//   WAF            18.7  14.7  10.4    52.2  37.4  37.7    157   132   128    545   514   504
//   KP07           18.7  15.4  10.7    36.6  21.9  19.8    103  81.3  74.6    348   324   301
//   KP07_dimsplit  15.1  10.5   8.2    34.5  22.0  21.5   84.7  67.3  66.7    282   264   261
//   EE2D           18.4  13.5  10.0    46.5  31.1  29.6    128   109   104    440   422   403
// (FORCE before and now: 6.5 3.4, 13.3 8.0, 35.3 26.6, 111 105).
template <int SCHEME, int W, int H, int NT, int VAR = 0, int LPT = 1, bool LOOP = false>
__global__ void __launch_bounds__(NT, compiled_blocks(SCHEME, W, H, NT, LPT)) stage_kernel(const __grid_constant__ StageArgs A) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* Qs = reinterpret_cast<float*>(smem_raw);
    __shared__ __align__(8) uint64_t bar;
    __shared__ unsigned taken;
    __shared__ float red[NT / 32];
    __shared__ int am_last;

    if (LOOP || !A.follows) grid_dependency_wait();  // the previous launch's state, control block and counters
    // The control block changes when the run's last task is complete.  A looping
    // CTA may start later than that: it takes its ticket after these loads, and
    // then finds no task left.
    const int4 w0 = ld_relaxed_v4(A.ctl);                                      // t, t_end
    const int4 w1 = ld_relaxed_v4(reinterpret_cast<const char*>(A.ctl) + 16);  // nt, dt, cfl_min
    const int4 w2 = ld_relaxed_v4(reinterpret_cast<const char*>(A.ctl) + 32);  // factor, cfl_scale, update_dt, cur
    const float dt0 = A.explicit_dt ? A.dt_step : __int_as_float(w1.z);
    const int cur0 = w2.w;
    int n_sub = A.n_sub, steps = A.steps;
    bool want_cfl = A.want_cfl != 0, active = true;
    if (!A.explicit_dt) {
        // a step runs while t < t_end and dt > 0 (GPUSimulators/Simulator.py:192, :202);
        // a dt that is not finite takes t past any end time in one step
        const double t = __hiloint2double(w0.y, w0.x), t_end = __hiloint2double(w0.w, w0.z);
        active = t < t_end && !(dt0 <= 0.0f);
        if (!LOOP && !active) return;
        if (A.full_steps > 0 && !(fabsf(dt0) < __int_as_float(0x7f800000))) {
            n_sub = A.substeps;
            steps = 1;
            want_cfl = true;
        }
    }
    const int ntiles = A.tiles_x * A.tiles_y;
    // Substeps that have tasks.  The looping form keeps those of substeps past
    // n_sub, without work: the control block changes after the last task only.
    const int n_all = LOOP ? A.n_sub : n_sub;
    unsigned task = blockIdx.x;
    if (A.n_sub > 1) {
        if (!LOOP && task >= (unsigned)ntiles * (unsigned)n_sub) return;
        if (threadIdx.x == 0) taken = atomicAdd(A.ticket, 1u);
        __syncthreads();
        task = taken;
        if (!LOOP && A.followed) grid_launch_dependents();
    }
    uint32_t loads = 0;   // tile loads of this CTA
    bool broken = false;  // one of them gave up

    while (!LOOP || (active && task < (unsigned)ntiles * (unsigned)n_all)) {
        const unsigned tid = per_task<LOOP>(threadIdx.x);
        if (LOOP) __builtin_assume(tid < NT);
        const unsigned row = task / (unsigned)A.tiles_x;
        const int tx = (int)(task - row * (unsigned)A.tiles_x);
        const int s = A.n_sub > 1 ? (int)(row / (unsigned)A.tiles_y) : 0;
        const int ty = (int)row - s * A.tiles_y + A.tile_row0;

        bool ok = true;
        if (s > 0 && tid < 16) {
            const int i = tid & 3, j = tid >> 2;
            const bool wrap_x = bc_west(A.bc) == BC_PERIODIC || bc_east(A.bc) == BC_PERIODIC;
            const bool wrap_y = bc_south(A.bc) == BC_PERIODIC || bc_north(A.bc) == BC_PERIODIC;
            const int nx = near_tile(tx, i, A.nx, A.tiles_x, W, wrap_x);
            const int ny = near_tile(ty, j, A.ny, A.tiles_y, H, wrap_y);
            if (tid == 15 || nx != tx || ny != ty) {  // thread 15 waits for the tile itself
                const unsigned* p = A.done + (size_t)kDoneStride * (ny * A.tiles_x + nx);
                const uint32_t polls = wait_polls(A.neighbour_limit);
                ok = false;
                for (uint32_t k = 0; k < polls; ++k) {
                    if (ld_acquire(p) >= (unsigned)s) {
                        ok = true;
                        break;
                    }
                    __nanosleep(20);
                }
            }
        }
        const bool run = !__syncthreads_or(ok && !(LOOP && broken) ? 0 : 1);
        const bool last = s == n_all - 1;
        const int sub = (A.first_substep + s) % A.substeps, step = s / A.substeps;
        const bool do_cfl = (LOOP ? s == n_sub - 1 : last) && want_cfl && SCHEME != WAF;  // WAFKernel has no CFL output (SWE2D_WAF.cu:103-119)
        float my_cfl = __int_as_float(0x7f800000);
        if (run && (!LOOP || s < n_sub)) {
            const int cur = cur0 ^ (s & 1);
            const float dt = (A.explicit_dt || step < A.full_steps) ? dt0 : A.tail[step - A.full_steps];
            const float kdt = dt * A.dt_scale;
            TileJob J;
            J.tmap = &A.tmap[cur][0];
            J.in = A.buf[cur];
            J.out = A.buf[cur ^ 1];
            J.nx = per_task<LOOP>(A.nx);
            J.ny = per_task<LOOP>(A.ny);
            J.pitch = per_task<LOOP>(A.pitch);
            J.bc = per_task<LOOP>(A.bc);
            J.x0 = tx * W;
            J.y0 = ty * H;
            J.tid = tid;
            // the other tiles' stores, which the wait above ordered before this
            // point, precede the tensor copies of the tile load
            if (tid == 0) fence_proxy_async_global();
            const float dx = per_task<LOOP>(A.dx), dy = per_task<LOOP>(A.dy), g = per_task<LOOP>(A.g),
                        theta = per_task<LOOP>(A.theta);
            const uint32_t phase = LOOP ? loads & 1u : 0u;
            const bool init = !LOOP || loads == 0;
            bool loaded;
            if constexpr (SCHEME == LXF || SCHEME == KP07) {
                const UnsplitPar P{dx, dy, g, theta, kdt, sub, A.order};
                loaded = process_tile_unsplit<SCHEME, W, H, NT, false, false, LOOP>(Qs, &bar, phase, init, J, P, do_cfl, &A.ctl->error,
                                                                my_cfl, wait_polls(A.wait_limit));
            } else {
                const SplitPar P{dx, dy, g, per_task<LOOP>(A.gamma), theta, kdt, sub, per_task<LOOP>(A.variant_beta)};
                loaded = process_tile_dimsplit<SCHEME, W, H, NT, false, VAR, LPT, false, LOOP>(
                    Qs, &bar, phase, init, J, P, do_cfl, &A.ctl->error, my_cfl, wait_polls(A.wait_limit));
            }
            if (LOOP) {
                ++loads;
                broken = !loaded;  // its barrier's phase is not known any more: no further load
            }
            fence_proxy_async_global();  // these stores precede other tiles' tensor copies
        } else if (!run && tid == 0 && !(LOOP && broken)) {
            atomicOr(&A.ctl->error, kNeighbourGaveUp);
        }
        const int tile = ty * A.tiles_x + tx;
        if constexpr (LOOP) {  // (below for the others)
            if (do_cfl) {
                const float m = block_min<NT, true>(my_cfl, red, tid);
                if (tid == 0) A.block_cfl[tile] = m;
            }
        }
        if (!last) {
            __syncthreads();
            if (tid == 0) st_release(A.done + (size_t)kDoneStride * tile, (unsigned)s + 1u);
            if constexpr (!LOOP) {
                if (A.follows) grid_dependency_wait();
                return;
            }
        } else {
            // The last substep: CFL minimum of the tile, arrival, and in the CTA that
            // arrives last the control-block update of Simulator.step / simulate
            // (GPUSimulators/Simulator.py:195-196, :227-228).  The tile is written: the
            // next launch's CTAs may start once every CTA of this one is here (they
            // wait in grid_dependency_wait for its end).
            if constexpr (!LOOP) {
                grid_launch_dependents();
                if (do_cfl) {
                    const float m = block_min<NT>(my_cfl, red, tid);
                    if (tid == 0) A.block_cfl[tile] = m;
                }
            }
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                am_last = atomicAdd(&A.ctl->arrive, 1u) == (unsigned)(A.ntiles_total ? A.ntiles_total : ntiles) - 1u;
            }
            __syncthreads();
            if constexpr (!LOOP) {
                if (A.follows) grid_dependency_wait();
                if (!am_last) return;
            }
            if (!LOOP || am_last) {
                __threadfence();
                float m = __int_as_float(0x7f800000);
                const bool new_cfl = LOOP ? want_cfl && SCHEME != WAF : do_cfl;
                if (new_cfl) {
                    for (int i = tid; i < ntiles; i += NT) m = fminf(m, __ldcg(&A.block_cfl[i]));
                    m = block_min<NT, LOOP>(m, red, tid);
                }
                if (!LOOP && A.n_sub > 1)  // every task is complete: no CTA takes or polls any more
                    for (int i = tid; i < ntiles; i += NT) A.done[(size_t)kDoneStride * i] = 0u;
                if (tid == 0) {
                    SimCtl* c = A.ctl;
                    c->cur = cur0 ^ (n_sub & 1);
                    if (new_cfl) c->cfl_min = m;
                    if (steps > 0) {
                        double t = c->t;
                        for (int k = 0; k < steps; ++k)
                            t += (double)((A.explicit_dt || k < A.full_steps) ? dt0 : A.tail[k - A.full_steps]);
                        c->t = t;
                        c->nt += steps;
                        if (!A.explicit_dt && c->update_dt && (c->nt % 100 == 0)) c->dt = (c->cfl_min * c->factor) * c->cfl_scale;
                    }
                    c->arrive = 0u;
                    if (!LOOP && A.n_sub > 1) *A.ticket = 0u;
                }
            }
        }
        if constexpr (!LOOP) return;
        if (threadIdx.x == 0) taken = atomicAdd(A.ticket, 1u);
        __syncthreads();
        task = taken;
    }

    if constexpr (LOOP) {
        // The last CTA to leave clears the counters: no CTA takes or polls any more.
        grid_launch_dependents();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            am_last = atomicAdd(A.ticket + 1, 1u) == gridDim.x - 1u;
        }
        __syncthreads();
        if (!am_last) return;
        __threadfence();
        for (int i = threadIdx.x; i < ntiles; i += NT) A.done[(size_t)kDoneStride * i] = 0u;
        if (threadIdx.x < 2) A.ticket[threadIdx.x] = 0u;
    }
}

// ------------------------------------------------------------------ batched stage kernel

// One simulation of a batch, resident in device memory.  Its tiles are loaded
// with load_tile_async, so it carries no tensor maps.
struct alignas(64) BatchInstance {
    float* buf[2][4];
    SimCtl* ctl;
    float* block_cfl;  // one float per tile of this simulation
    float2* scratch;   // partial minima of the initial CFL estimate
    int nx, ny, pitch, bc;
    int tiles_x, ntiles;
    float dx, dy, g, gamma, theta, dt_scale;
    float variant_beta;  // parameter of the Osher and Sweby limiters
};

struct BatchArgs {
    const BatchInstance* inst;
    SimCtl* ctl;        // control blocks, one per instance: inst[i].ctl == ctl + i
    const int2* work;   // (instance, tile within instance) per work item
    unsigned* ticket;   // tasks taken, zero before a run of several substeps
    unsigned* done;     // per instance, kDoneStride apart, zero before such a run: substeps of the run
                        // completed, or kStopped once the simulation takes no further steps
    int nwork;          // work items
    int substeps;       // substeps per step
    int first_substep;  // substep of the step that the run starts with
    int n_sub;          // substeps of the run: of this launch, or of a chain of them
    int follows;        // this launch goes on where the one before stopped in the same run (stage_kernel)
    int followed;       // and the next one goes on where this one stops
    int order;          // RK order (KP07)
    int* err;           // set when a wait gave up
    int wait_limit;     // polls of the bounded waits, as StageArgs' (0: the default)
};
constexpr unsigned kStopped = 0xffffffffu;

// Copies the instance record into shared memory (asynchronous, in 16-byte
// chunks by the CTA's first threads).
constexpr int kInstChunks = sizeof(BatchInstance) / 16;
__device__ __forceinline__ void prefetch_instance(BatchInstance* m, const BatchInstance* inst) {
    const int i = threadIdx.x;
    if (i < kInstChunks) cp_async16(reinterpret_cast<char*>(m) + 16 * i, reinterpret_cast<const char*>(inst) + 16 * i, 16);
}

// CTAs per SM that a batched kernel is compiled for: four of 128 threads (two
// of 256), i.e. at most 128 registers a thread.  The column walks of LxF and
// KP07, which shared memory holds eight times, would take 82 and 105 registers,
// and lose the warps that hide their latencies: bound to eight and six CTAs they
// take 64 and 80.  us per step, 128 grids of 64 to 1024 cells a side and one of
// 2048: LxF 139 to 115 and 34.6 to 30.6, KP07 513 to 408 and 123 to 99.7 (eight:
// 388 and 103, but spilling, and 64 grids of 64 to 128 take 27.6 instead of
// 23.9; six: 24.9).  WAF's 28-row tiles would take 101, which is one CTA less than
// five: bound to five 622 to 610 and 166 to 163, and with the periodic ghost
// cells' loads one after the other 594 and 160 (six CTAs: 64 small grids 47.8 to
// 54.3).
__host__ __device__ constexpr int batched_blocks(int scheme, int W, int H, int NT) {
    const int most = 65536 / (NT * 128);
    if (scheme == WAF && H == 28 && NT == 128) return 5;
    if (scheme != LXF && scheme != KP07) return most;
    const int by_smem = 228 * 1024 / (3 * (W + 8) * (H + 4) * (int)sizeof(float) + 1024 + 256);  // 228 KB per SM
    const int wanted = scheme == LXF ? 8 : 6;
    return by_smem < wanted ? (by_smem > most ? by_smem : most) : wanted;
}

// Stage kernel of any scheme over a batch: one CTA per work item and substep of
// a run.  A launch of one substep takes its items by block index.  The tasks of a
// run of several steps are taken in order, substep by substep along the work
// list, over a chain of launches if there are many, as in stage_kernel.  Each
// simulation keeps its own t, dt (its own CFL every 100 of its steps) and t_end:
// the last of its tiles to arrive in a substep updates its control block exactly
// as a launch of its own would, and then releases the simulation's next substep.
// So in a run a substep of one simulation overlaps those of the others, without a
// barrier.  A simulation that reached its t_end, or went bad, is released for
// good; its tasks return.
//
// us per step in runs of 16 steps, before (a launch per substep, replayed from
// graphs) and now (batch_in_runs chooses a launch per substep for the last):
//                 1 of 80 x 80  20 of 64 to 1024  128 of them  1 of 2048 x 2048
//   KP07_dimsplit   22.3  21.3     70.3  51.9      328   288      94.8  88.4
//   HLL2            26.1  25.3     86.1  66.0      418   363       119   110
//   EE2D            29.2  27.8      106  81.5      514   453       149   138
//   KP07            17.7  17.0     72.4  52.7      395   337       113  99.0
//   WAF             21.6  21.1      116   106      599   589       162   160
//   HLL              9.7   8.9     30.3  24.1      140   133      41.2  41.0
//   FORCE            8.1   7.5     25.1  19.8      117   109      34.5  34.0
//   LxF              7.9   7.3     22.7  15.3      108  93.2      32.1  28.9
// Slower than before: KP07 on a few grids of up to 300 x 300, 18.0 to 19.3 (its
// bound on registers, batched_blocks).
template <int SCHEME, int W, int H, int NT, int VAR = 0, int LPT = 1>
__global__ void __launch_bounds__(NT, batched_blocks(SCHEME, W, H, NT)) batched_stage_kernel(const __grid_constant__ BatchArgs B) {
    static_assert(NT >= kInstChunks && sizeof(BatchInstance) % 16 == 0, "one thread per copied 16-byte chunk");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float* Qs = reinterpret_cast<float*>(smem_raw);
    __shared__ BatchInstance I;
    __shared__ int4 words[3];  // the first 48 bytes of the control block
    __shared__ unsigned taken;
    __shared__ float red[NT / 32];
    __shared__ int flag;
    if (!B.follows) grid_dependency_wait();  // the previous launch's states, control blocks and counters
    unsigned item = blockIdx.x;
    int s = 0;
    if (B.n_sub > 1) {
        if (threadIdx.x == 0) taken = atomicAdd(B.ticket, 1u);
        __syncthreads();
        s = (int)(taken / (unsigned)B.nwork);
        item = taken - (unsigned)s * (unsigned)B.nwork;
        if (B.followed) grid_launch_dependents();
    }
    const int2 job = B.work[item];
    prefetch_instance(&I, B.inst + job.x);
    unsigned* const done = B.done + (size_t)kDoneStride * job.x;
    SimCtl* const ctl = B.ctl + job.x;
    if (threadIdx.x == 0) {
        unsigned seen = 0u;
        if (s > 0) {
            // bounded; one wait that gives up ends all of them
            for (uint32_t k = 0; k < wait_polls(B.wait_limit); ++k) {
                seen = ld_acquire(done);
                if (seen >= (unsigned)s || *(volatile int*)B.err) break;
                __nanosleep(20);
            }
            if (seen < (unsigned)s) {
                atomicExch(B.err, 1);
                seen = kStopped;
            }
        }
        flag = seen == kStopped;
        // one reader per CTA: the tiles of a simulation are released at once
        // and would queue at its control block
#pragma unroll
        for (int i = 0; i < 3; ++i) words[i] = ld_relaxed_v4(reinterpret_cast<const char*>(ctl) + 16 * i);
    }
    cp_async_wait_all();
    __syncthreads();
    if (flag) {
        if (B.follows) grid_dependency_wait();
        return;
    }
    const int sub = (B.first_substep + s) % B.substeps;
    const bool is_last = sub == B.substeps - 1;  // of its step
    StepCtl sc = step_from_words(words[0], words[1], words[2], false, 0.0f, false, is_last);
    if (!sc.active) {  // from the launch's start: later it is released as stopped
        if (B.n_sub > 1 && job.y == 0 && threadIdx.x == 0) st_release(done, kStopped);
        if (B.follows) grid_dependency_wait();
        return;
    }
    if (SCHEME == WAF) sc.do_cfl = false;  // WAFKernel has no CFL output (SWE2D_WAF.cu:103-119)
    float my_cfl = __int_as_float(0x7f800000);
    TileJob J;
    J.tmap = nullptr;
    J.in = I.buf[sc.cur];
    J.out = I.buf[sc.cur ^ 1];
    J.nx = I.nx;
    J.ny = I.ny;
    J.pitch = I.pitch;
    J.bc = I.bc;
    J.tid = threadIdx.x;
    const int ty = job.y / I.tiles_x;
    J.x0 = (job.y - ty * I.tiles_x) * W;
    J.y0 = ty * H;
    bool unhealthy = false;
    if constexpr (SCHEME == LXF || SCHEME == KP07) {
        const UnsplitPar P{I.dx, I.dy, I.g, I.theta, sc.dt * I.dt_scale, sub, B.order};
        process_tile_unsplit<SCHEME, W, H, NT, true, true>(Qs, nullptr, 0, false, J, P, sc.do_cfl, B.err, my_cfl,
                                                           kWaitPolls, is_last, &unhealthy);
    } else {
        const SplitPar P{I.dx, I.dy, I.g, I.gamma, I.theta, sc.dt * I.dt_scale, sub, I.variant_beta};
        process_tile_dimsplit<SCHEME, W, H, NT, true, VAR, LPT, true>(Qs, nullptr, 0, false, J, P, sc.do_cfl, B.err,
                                                                      my_cfl, kWaitPolls, is_last, &unhealthy);
    }
    // The tile's CFL minimum, its arrival, and in the last tile of the
    // simulation to arrive the control-block update of Simulator.step / simulate
    // (GPUSimulators/Simulator.py:195-196, :227-228).  The tile is written: the
    // next launch's CTAs may start, and wait for the end of this one.
    if (!B.followed) grid_launch_dependents();
    if (__syncthreads_or(unhealthy) && threadIdx.x == 0) atomicOr(&ctl->bad, 1);
    if (sc.do_cfl) {
        const float m = block_min<NT>(my_cfl, red, threadIdx.x);
        if (threadIdx.x == 0) I.block_cfl[job.y] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        flag = atomicAdd(&ctl->arrive, 1u) == (unsigned)I.ntiles - 1u;
    }
    __syncthreads();
    if (B.follows) grid_dependency_wait();
    if (!flag) return;
    __threadfence();
    float m = __int_as_float(0x7f800000);
    if (sc.do_cfl) {
        for (int i = threadIdx.x; i < I.ntiles; i += NT) m = fminf(m, __ldcg(&I.block_cfl[i]));
        m = block_min<NT>(m, red, threadIdx.x);
    }
    if (threadIdx.x == 0) {
        bool go = true;
        ctl->cur = sc.cur ^ 1;
        if (sc.do_cfl) ctl->cfl_min = m;
        if (is_last) {
            ctl->t = sc.t_new;
            ctl->nt = ctl->nt + 1;
            if (ctl->update_dt && (ctl->nt % 100 == 0)) ctl->dt = (ctl->cfl_min * ctl->factor) * ctl->cfl_scale;
            if (__ldcg(&ctl->bad)) ctl->t_end = ctl->t;  // a failed simulation takes no further steps
            const double rem = ctl->t_end - ctl->t, d = (double)ctl->dt;
            go = ctl->t < ctl->t_end && !((float)((rem < d) ? rem : d) <= 0.0f);  // step_from_words
        }
        ctl->arrive = 0u;
        if (B.n_sub > 1) st_release(done, go ? (unsigned)s + 1u : kStopped);
    }
}

}  // namespace fv
