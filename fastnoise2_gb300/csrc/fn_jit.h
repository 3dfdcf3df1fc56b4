// fn_jit.h -- run-time specialised kernels.
//
// The interpreter (fn_kernels.cu) evaluates any tree but pays for dispatch and
// for a register file in local memory.  For trees that will be evaluated many
// times, the same device program is turned into straight-line CUDA source --
// one call per instruction to the hand-written node functions of
// fn_device.cuh, positions and values in registers, parameters as literals --
// and compiled for sm_103a with NVRTC (-fmad=false, so results are identical
// to the interpreter's).  Each tree gets a module with its grid / position-array
// / tileable per-call kernels; one batch module holds a persistent batch kernel
// per tree, so the trees of a batch run as concurrent kernels, each with the
// register allocation its own code needs.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "fn_compile.h"
#include "fn_types.h"

namespace fn {

constexpr int kMaxColumnStates = 10;

struct ColumnRate {                   // of one column state
    float scale[4] = {};              // lattice cells per unit along the grid's axes
    float enter = 0, step = 0;        // issue slots of entering a cell (per neighbourhood if cellular), of a step,
    float point = 0;                  // and of the point function
    bool cellular = false;
};

struct JitKernels {
    cudaKernel_t grid = nullptr;      // GenUniformGrid for the program's dimensionality
    cudaKernel_t positions = nullptr; // GenPositionArray
    cudaKernel_t tileable = nullptr;  // GenTileable2D (4D programs only)
    cudaKernel_t solid = nullptr;     // chunk meshing (3D programs): classification bitmasks of a grid
    cudaKernel_t list = nullptr;      // chunk meshing (3D programs): grid values at listed point indices
    cudaKernel_t column = nullptr;    // grids walked along their last axis (trees with separable lattice noise)
    cudaKernel_t batch_column = nullptr;   // the same for a batch's grid requests
    ColumnRate column_rates[kMaxColumnStates];   // of its states
    int n_column_rates = 0;
    float column_step = 1.0f, point_cost = 1.0f;   // issue slots of a step of a column, of a point otherwise
    int column_resident = 1;          // its 256-thread blocks per SM at once
    int slot = -1;                    // index in the module's batch kernel
    int resident[3] = {1, 1, 1};      // 256-thread blocks per SM of grid / positions / tileable at once
};

// Variants of a tree's persistent batch kernel, among which the autotuner picks per
// tree: threads per block, the register bound (the blocks per SM the kernel must fit,
// __launch_bounds__) and how many points a thread has in flight per loop iteration.
// Variant 0 is the one fnJitCompile builds; the others are built when a tuning run
// (or a loaded tuning table) asks for them.
struct BatchVariant {
    int threads;
    int min_blocks;
    int points;
};
const std::vector<BatchVariant>& batch_variants();

struct BatchKernel {
    cudaKernel_t kernel = nullptr;
    int threads = 256;
};

// CUDA source of a module: a head, and parts that need the head but not each other, with the
// time each takes to compile (seconds, roughly).
struct ModuleSource {
    struct Part {
        std::string text;
        float seconds;
    };
    std::string head;
    std::vector<Part> parts;
};

// The batch kernels of `progs` (slot k = progs[k]) in one variant (variant 0: and the column kernels
// of the programs that have them), and one program's per-call module.
ModuleSource jit_batch_module(const std::vector<const CompiledProgram*>& progs, int variant);
ModuleSource jit_percall_module(const CompiledProgram& prog);

// NVRTC-compile modules, concurrently; those in the on-disk cache are taken from it.
// Host only, no GPU needed.
bool jit_compile_modules(const std::vector<ModuleSource>& modules, std::vector<std::vector<char>>& compiled,
                         std::string& error);
// The batch module and every per-call module: compiled[0] = batch, compiled[1 + k] = program k.
bool jit_compile_all(const std::vector<const CompiledProgram*>& progs, std::vector<std::vector<char>>& compiled,
                     std::string& error);

// Compile and load a module covering `progs`; on success every program gets
// per-call kernels and a batch kernel.  Thread safe.
bool jit_build(const std::vector<const CompiledProgram*>& progs, std::string& error);

// On-disk module cache (see fn_jit.cpp): the directory in use ("" = off, the default; the
// environment variable FASTNOISE_JIT_CACHE names one),
// its hit / miss counts in this process, and the tree's kernels loaded straight from the
// cache when an earlier process built them alone (the way automatic specialisation does):
// true when they are loaded now.  Looks once per program and process.
void jit_cache_set_dir(const char* dir);
std::string jit_cache_dir();
void jit_cache_stats(unsigned long long* hits, unsigned long long* misses);
bool jit_try_cached(const CompiledProgram* prog);

// Build variants 1.. of the batch kernels of `progs` (NVRTC, one module per variant,
// compiled concurrently); programs whose variants exist are skipped.  Thread safe.
bool jit_build_batch_variants(const std::vector<const CompiledProgram*>& progs, std::string& error);

// The batch kernel of `hash` in `variant`, or false when it is not built (or JIT is off).
bool jit_batch_kernel(uint64_t hash, int variant, BatchKernel& out);

// A grid walked in columns (PointArgs' col_ fields): points of the plane across the last axis
// (0: not walked in columns), steps along it and the index of the first, steps per unit, units.
struct ColumnShape {
    unsigned plane = 0, steps = 0, first = 0, len = 0, units = 0;
    // issue slots of a step, and of entering cells at a unit's first step and per step after it;
    // how long a step of one warp takes
    float step = 0, enter = 0, cross = 0, step_us = 0;
};

// The calling thread's route for grids of trees that have a column kernel (fnSetGridRoute): by
// estimate, or always through the point or the column kernel; steps per unit (0: by estimate).
struct GridRoute {
    int route = 0;                    // FN_GRID_ROUTE_*
    unsigned steps = 0;
    unsigned columns = 0;             // grids walked in columns since the route was last set
};
GridRoute& grid_route();

// Whether a request of a batch can be walked in columns by the kernels `jk` (fn_column.cuh); if so
// `shape` gets its plane and steps, and `point_us` and `column_us` the time that the GPU takes to issue
// it either way.  column_tiles cuts it into units of at most `len` steps and returns the batch's work
// items for it (eight units each).
bool jit_batch_columns(const PointArgs& args, const JitKernels& jk, ColumnShape& shape, float& point_us, float& column_us);
inline unsigned column_chunks(const ColumnShape& s) { return (s.plane + 31) / 32; }
unsigned column_tiles(ColumnShape& shape, unsigned len);
void column_args(PointArgs& args, const ColumnShape& shape);

// Queue a background build of the batch variants of `prog` (a tuning table loaded in this
// process may name variants that have not been built yet).
void jit_request_batch_variants(const CompiledProgram* prog);

// Kernels for a program hash, or false if none have been built.
bool jit_lookup(uint64_t hash, JitKernels& out);

// Where a kernel stores its output: device memory, or host memory that it writes directly.
enum OutputMemory { kDeviceMemory, kPageLocked, kPageable };

// Launch the specialised per-call kernel for `hash` if one is loaded (and JIT
// is enabled); returns false when the caller should use the interpreter.
// `err` carries the launch status when true is returned.
bool jit_launch(uint64_t hash, const PointArgs& args, float* out, MinMaxWork* work, float* dminmax, cudaStream_t stream,
                cudaError_t& err, OutputMemory memory = kDeviceMemory);

// Chunk meshing with a specialised 3D tree (false when none is loaded): bit i of `above` /
// `solid` = grid point i's value is > iso / <= iso (both 0 for NaN), and OutputMinMax into
// `dminmax`; and the values at the grid point indices idx[0 .. *count) into out (max_count
// bounds the launch).
bool jit_launch_solid(uint64_t hash, const PointArgs& args, unsigned* above, unsigned* solid, MinMaxWork* work, float* dminmax,
                      float iso, cudaStream_t stream, cudaError_t& err);
bool jit_launch_list(uint64_t hash, const PointArgs& args, const unsigned* idx, const unsigned* count, unsigned max_count,
                     float* out, cudaStream_t stream, cudaError_t& err);

// Programs the interpreter cannot run (CompiledProgram::needs_specialisation)
// get their specialised kernels built on first use; true if they exist now.
bool jit_ensure(const CompiledProgram* prog, std::string& error);

void jit_set_enabled(bool on);
bool jit_enabled();

// Automatic specialisation: the interpreter paths report each launch of a program
// here; once a program has run `threshold` times on the interpreter it is queued
// for a background NVRTC build (one worker thread), and later launches find its
// specialised kernels.  threshold 0 = off; the default comes from the environment
// variable FASTNOISE_AUTO_SPECIALISE (a number, 0 = off), else 4.
void jit_note_interpreted(const CompiledProgram* prog);
int jit_set_auto_threshold(int uses);              // returns the previous threshold
bool jit_auto_wait(int timeout_ms);                // true when no build is queued or running
bool jit_is_specialised(uint64_t hash);

}  // namespace fn
