// The streaming stage of the preconditioner: psi = L^{-1} q, L = streaming +
// removal, by an upwind transport sweep of every ordinate at once.
//
// UBOLT preconditions streaming with PCAIR (src/transport_solverk.kokkos.cxx:
// 238-260), an algebraic multigrid approximation of L^{-1}. Here L^{-1} is
// applied exactly wherever the per-ordinate upwind graph is acyclic.
//
// The plan (sweep_plan.cpp, host, once per mesh and ordinate set) cuts each
// ordinate's sweep into tasks - a piece of one patch of consecutive cells,
// its cells in level order - numbered so every task's upstream tasks come
// before it. Reflective inflow couples ordinates and is lagged (read as zero),
// as are the couplings a cycle break releases.
//
// Kernel: persistent, one warp per task, tasks taken in number order.
// Synchronisation is by the data itself: psi is filled with a sentinel bit
// pattern (all ones, a NaN the kernel never stores) before the launch, and a
// cell whose upwind neighbour lies in an earlier task polls that neighbour's
// psi values until none is the sentinel. So a task waits for exactly the
// values it reads, at the level that reads them, and can start while its
// upstream tasks are still walking: the chain of dependencies runs cell to
// cell through L2 with no flags, fences or task-granular barriers.
//
// Everything off that chain happens first, in a prologue: y0 = B^{-1} q and
// the couplings G_f = B^{-1} s_f face_up_f (one per gathered face) of every
// cell of the task go into the warp's shared-memory slice. The walk then runs
// level by level over a table of values in shared memory - the task's own
// cells and its ghosts, the cells of earlier tasks it reads: psi_c = y0 -
// sum_f G_f psi(up_f), one lane per row of a cell.
// Deadlock-free: a task polls only values of lower-numbered tasks, which were
// taken by warps already running. Every poll is bounded; a poll that gives up
// records a timeout, reads the value as zero and the sweep completes.
//
// What bounds it: the latency of the tasks and of the upwind chain, not bytes
// or flops (256^2 triangles, DG1, S8, FP64: 154 thousand tasks of 34 cells in 15
// levels). So the walk is built for few instructions and no divergence per
// level (a warp that splits on a branch loses about 100 cycles, as much as a
// level's arithmetic), and a wait asks for what the next levels wait for as
// well. Per sweep with an isotropic source and psi ordinate-major, before (a
// lane per cell, each level polling for itself) and now, FP64 / FP32: 256^2
// triangles 945 / 795 -> 593 / 489 us, 200^2 quadrilaterals 643 / 562 -> 308 /
// 275, 20^3 cubes of Kuhn tetrahedra 1453 / 1166 -> 905 / 496, 40^3 hexahedra
// 1188 / 687 -> 605 / 400.
#include "ctx.h"
#include "sweep_plan.h"
#include "wave.h"

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

// The task counter and the error words sit on separate 128-byte lines: every
// warp increments the counter, and a spinning lane must not contend with it.
// Words [kCtrlNever, kCtrlNever + 2) hold a sentinel nothing overwrites (the
// target of the bounded-wait test hook).
constexpr int kCtrlCounter = 0, kCtrlError = ubolt::kSweepCtrlError, kCtrlNever = 48, kCtrlWords = 64;
constexpr int kSweepWarpsPerSm = 32;
constexpr size_t kViaBytes = (size_t)8 << 20;
constexpr uint32_t kCopyTries = 1u << 22;  // bounded wait for a task's bulk copy

// Few cell-ordinates fill the device with tasks of either size
constexpr int64_t kFewCellOrdinates = (int64_t)1 << 20;

// The default patch, in cells. Larger patches make fewer and longer tasks
// with fewer waits between them, but their couplings take the shared memory of
// resident warps, and a task starts as late as its latest ghost. Measured per
// isotropic-source sweep at S8 (FP64 / FP32, us), a multiple or a part of the
// mesh builders' tiles (8 x 8 quads, 4^3 boxes) best:
//    256^2 triangles DG1     64: 591 / 485    128: 602 / 415    32: 921 / 813
//    100^2 quads DG1         64: 150 / 136    128: 139 / 124
//    101 x 77 triangles DG1  64: 154 / 142    128: 142 / 135
//    20^3 cubes of tets DG1  48: 901 / 492    24: 946 / 673     96: 1361 / 599
//    40^3 hexes DG1          64: 603 / 399    32: 683 / 350
// and DG0, whose couplings are one value each:
//    150^2 triangles         64: 256 / 237    256: 197 / 183
//    200^2 quads             64: 234 / 221    256: 225 / 212
//    20^3 cubes of tets      48: 386 / 351    192: 213 / 196
//    40^3 hexes              64: 150 / 136    128: 129 / 115    256: 155 / 125
// A mesh of one patch has no task that waits on another (125 hexahedra DG1 S8
// 24 -> 20; 162 tetrahedra without a factor store 36 -> 45, a patch of 48 36).
static int DefaultPatch(const ubolt_ctx *ctx)
{
   if (ctx->n_cells <= 128) return 128;
   const bool tets = ctx->dim == 3 && ctx->F == 4;
   if (ctx->nb == 1) return ctx->dim == 2 ? 256 : tets ? 192 : 128;
   if (ctx->dim == 3) return tets ? 48 : 64;
   return ctx->n_cells * (int64_t)ctx->A <= kFewCellOrdinates ? 128 : 64;
}

// Where AUTO takes the wave kernel. One block per ordinate leaves most of the
// device idle, and the task kernel was faster on the meshes measured (FP64,
// us, wave and tasks: 64^2 quads DG0 S4 68 / 41, 32^2 37 / 23, 24^2 triangles DG1
// S8 84 / 38, 16^3 hexes DG1 S2 72 / 53, 256^2 triangles DG1 S8 2220 / 703), but
// for small DG0 boxes of hexahedra, whose levels are many cells of one value and
// few: 10^3 S2 / S4 / S8 24 / 24 / 25 and 30 / 32 / 36, 16 x 15 x 17 S2 34 and 43, S4
// 35 and 47; 20^3 S2 50 and 45. A whole solve there 530 / 542 / 541 and 588 / 598 /
// 688 us at 10^3, 634 and 670 at 16 x 15 x 17, 786 and 691 at 20^3
static bool WaveByDefault(const ubolt_ctx *ctx)
{
   return ctx->dim == 3 && ctx->F == 6 && ctx->nb == 1 && ctx->n_cells <= 4096 &&
          ctx->n_cells * (int64_t)ctx->A <= (int64_t)1 << 17;
}

namespace ubolt {
struct Task;
}

struct ubolt_sweep_plan {
   int32_t P = 0, n_patches = 0, A = 0;
   int64_t n_tasks = 0, n_lagged = 0, n_split = 0, total_levels = 0;
   int32_t max_levels = 0, max_inflow = 0;
   // Device arrays (owned by the context's allocation list)
   const ubolt::Task *task = nullptr;   // [n_tasks]
   const int32_t *dep_ptr = nullptr;    // [n_tasks + 1]
   const int32_t *deps = nullptr;       // upstream task ids
   const uint16_t *sched = nullptr;     // per entry, SchedWords(F) words: the local cell, then per gathered face the
                                        // upwind cell's place in the task's value table (see SweepDev)
   const uint16_t *tmask = nullptr;     // upwind faces: in task (bit f) / earlier task (bit 8 + f)
   const uint16_t *pass = nullptr;      // end positions of every task's passes (levels cut at 32 / nb positions)
   const int32_t *ghost = nullptr;      // the cells of earlier tasks each task reads
   const int32_t *patch_ptr = nullptr;  // [n_patches + 1] each patch's tasks in patch_task
   const int32_t *patch_task = nullptr; // [n_tasks]
   int n_loc = 0;                       // most (positions + ghosts) of a task, plus one
   int n_ghost = 1;                     // most ghosts of a task
   uint32_t *ctrl = nullptr;            // [kCtrlCounter] task counter; [kCtrlError] error flag, [kCtrlError + 1] timeout count
   int grid = 0, slots = 1;
   uint32_t spin_limit = 1u << 22;
   int64_t unmet_task = -1;  // ubolt_sweep_test_wait: one task polls a value nothing writes
   // The factor store (B^{-1} and couplings per task entry) per precision,
   // valid for the group epoch it was built in; limit < 0: automatic
   void *fac[2] = {nullptr, nullptr};
   void *scratch = nullptr;  // one FP64 vector: a sweep between row vectors runs ordinate-major in it
   uint64_t fac_epoch[2] = {0, 0};
   int64_t fac_limit = -1;
   // The wave plan (one block per ordinate), where every ordinate's upwind
   // graph is acyclic and a level fits a block: wave[which].smem > 0 where
   // precision `which` (0 FP64, 1 FP32) can run it. fac_wave[which]: the
   // store reserved for that precision is in wave order (the wave kernel runs)
   bool wave_tried = false, wave_ok = false;  // built where the wave kernel is asked for or AUTO takes it
   int wave_threads = 256;
   int64_t wave_levels = 0;
   ubolt::WaveDev wave[2];
   int64_t wave_bytes[2] = {0, 0};
   bool fac_wave[2] = {false, false};
   int kernel_mode = UBOLT_SWEEP_AUTO;
   int64_t unmet_level = -1;  // ubolt_sweep_test_wait: one level's copy is never issued
   ~ubolt_sweep_plan()
   {
      for (void *f : {fac[0], fac[1], scratch})
         if (f) cudaFree(f);
   }
};

namespace ubolt {

namespace {

template <typename T>
int UploadVec(ubolt_ctx *ctx, const std::vector<T> &h, const T **d)
{
   void *p = nullptr;
   int rc = CtxAlloc(ctx, std::max<size_t>(h.size(), 1) * sizeof(T), &p);
   if (rc) return rc;
   if (!h.empty()) rc = CudaCheck(cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice), "sweep plan");
   *d = static_cast<const T *>(p);
   return rc;
}

}  // namespace

// psi values cross warps through L2 as single 4- or 8-byte relaxed accesses:
// a reader sees the sentinel or the final value, never a torn one
__device__ __forceinline__ double LoadRelaxed(const double *p)
{
   double v;
   asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
   return v;
}
__device__ __forceinline__ float LoadRelaxed(const float *p)
{
   float v;
   asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
   return v;
}
// Stores of psi, and the sweep's other one-lane operations, under a
// predicate instead of a branch (a branch that splits the warp costs about
// 100 cycles)
__device__ __forceinline__ void StoreRelaxedIf(bool yes, double *p, double v)
{
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.relaxed.gpu.global.f64 [%0], %1;\n\t}" ::"l"(p),
                "d"(v), "r"((int)yes)
                : "memory");
}
__device__ __forceinline__ void StoreRelaxedIf(bool yes, float *p, float v)
{
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.relaxed.gpu.global.f32 [%0], %1;\n\t}" ::"l"(p),
                "f"(v), "r"((int)yes)
                : "memory");
}
__device__ __forceinline__ void LoadRelaxedIf(bool yes, const double *p, double &v)
{
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.relaxed.gpu.global.f64 %0, [%1];\n\t}"
                : "+d"(v)
                : "l"(p), "r"((int)yes)
                : "memory");
}
__device__ __forceinline__ void LoadRelaxedIf(bool yes, const float *p, float &v)
{
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p ld.relaxed.gpu.global.f32 %0, [%1];\n\t}"
                : "+f"(v)
                : "l"(p), "r"((int)yes)
                : "memory");
}
__device__ __forceinline__ void StoreSharedIf(bool yes, double *p, double v)
{
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.f64 [%0], %1;\n\t}" ::"r"(SmemAddr(p)),
                "d"(v), "r"((int)yes)
                : "memory");
}
__device__ __forceinline__ void StoreSharedIf(bool yes, float *p, float v)
{
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.shared.f32 [%0], %1;\n\t}" ::"r"(SmemAddr(p)),
                "f"(v), "r"((int)yes)
                : "memory");
}
__device__ __forceinline__ uint32_t AtomicIncIf(bool yes, uint32_t *p)
{
   uint32_t v = 0;
   asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p atom.global.add.u32 %0, [%1], 1;\n\t}"
                : "+r"(v)
                : "l"(p), "r"((int)yes)
                : "memory");
   return v;
}
// mbarrier.arrive.expect_tx, then one bulk copy with an L2 policy completing on it
__device__ __forceinline__ void BulkLoadIf(bool yes, void *dst, const void *src, uint32_t bytes, uint64_t *bar,
                                           uint64_t policy)
{
   asm volatile(
       "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
       "@p mbarrier.arrive.expect_tx.shared::cta.b64 _, [%3], %2;\n\t"
       "@p cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
       "\n\t}" ::"r"(SmemAddr(dst)),
       "l"(src), "r"(bytes), "r"(SmemAddr(bar)), "l"(policy), "r"((int)yes)
       : "memory");
}
// N values from shared memory, as 16-byte words where they are aligned so
template <typename T, int N, bool WIDE>
__device__ __forceinline__ void LoadRow(const T *p, T (&v)[N])
{
   if constexpr (WIDE) {
#pragma unroll
      for (int u = 0; u < N * (int)sizeof(T) / 16; u++) {
         const int4 w = reinterpret_cast<const int4 *>(p)[u];
         memcpy(reinterpret_cast<char *>(v) + 16 * u, &w, 16);
      }
   } else {
#pragma unroll
      for (int e = 0; e < N; e++) v[e] = p[e];
   }
}
__device__ __forceinline__ uint32_t TopWord(double v) { return (uint32_t)__double2hiint(v); }
__device__ __forceinline__ uint32_t TopWord(float v) { return (uint32_t)__float_as_int(v); }
__device__ __forceinline__ bool IsSentinel(double v) { return __double_as_longlong(v) == -1LL; }
__device__ __forceinline__ bool IsSentinel(float v) { return __float_as_int(v) == -1; }
template <typename T>
__device__ __forceinline__ T Sentinel();
template <>
__device__ __forceinline__ double Sentinel<double>() { return __longlong_as_double(-1LL); }
template <>
__device__ __forceinline__ float Sentinel<float>() { return __int_as_float(-1); }
// A computed value equal to the sentinel (a NaN carrying its payload) is
// stored as another NaN, so a reader can never mistake a result for "not yet"
__device__ __forceinline__ double Publishable(double v) { return IsSentinel(v) ? __longlong_as_double(0x7ff8000000000001LL) : v; }
__device__ __forceinline__ float Publishable(float v) { return IsSentinel(v) ? __int_as_float(0x7fc00001) : v; }

// Words of an entry's schedule record: the local cell and up to F - 1 links
__host__ __device__ constexpr int SchedWords(int F) { return F <= 4 ? 4 : 8; }

// A task as one 32-byte record: cells, passes and ghosts in the first word,
// the patch, its first entry, first ghost and first pass, the ordinate
struct __align__(16) Task {
   uint32_t counts;
   int32_t patch;
   int64_t off;
   int64_t ghost0;
   int32_t pass0, ordinate;
   __host__ __device__ int ncell() const { return counts & 1023; }
   __host__ __device__ int npass() const { return (counts >> 10) & 1023; }
   __host__ __device__ int nghost() const { return (int)(counts >> 20); }
};
__device__ __forceinline__ Task LoadTask(const Task *p)
{
   Task t;
   const int4 *s = reinterpret_cast<const int4 *>(p);
   const int4 a = __ldg(s), b = __ldg(s + 1);
   memcpy(&t, &a, 16);
   memcpy(reinterpret_cast<char *>(&t) + 16, &b, 16);
   return t;
}

struct SweepDev {
   int32_t P, A;
   int64_t n_tasks;
   const Task *task;        // [n_tasks]
   const uint16_t *sched;   // per entry, SchedWords(F) words: the local cell, then per gathered face the upwind cell's
                            // place in the task's value table, in elements - nb times 1 + its position, or 1 + ncell +
                            // its place among the task's ghosts, or 0 (a zero: no such face)
   const uint16_t *tmask;   // [entries] gathered faces (factors built in the sweep, and the store)
   const int32_t *ghost;    // per task, the cells of earlier tasks it reads
   int32_t n_loc, n_ghost;
   const uint16_t *pass;    // end position of every pass of every task
   uint32_t *ctrl;
   uint32_t spin_limit;
   int32_t slots;
   int64_t unmet_task;
   // Affine input: when aff_phi is set the sweep reads
   // q(node, a) = alpha r0(node, a) + u_a (phi(node) - alpha rho(node)),
   // u_a = aff_u[a] or 1, with r0 passed as q (compressed GMRES's Arnoldi vector)
   const double *aff_alpha, *aff_phi, *aff_rho;
   const void *aff_u;
   int32_t aff_iso;  // r0 is isotropic (r0 = E rho): the input is u_a phi(node), q is not read
   int32_t aff_inv_volume;  // with aff_iso: the input is u_a phi(node) / V(cell) (the adjoint's P V^{-1} E_w phi)
   // psi(c, j, a) at psi[c os_c + j os_j + a os_a]: UBOLT's row layout
   // (NB A, A, 1), or ordinate-major (NB, 1, n_cells NB), where a task's
   // cells of one ordinate are contiguous and it writes whole sectors
   int64_t os_c, os_j, os_a;
   // q(c, j, a) at q[c qs_c + j qs_j + a qs_a], the same two layouts
   int64_t qs_c, qs_j, qs_a;
};

// Per-warp shared-memory slice, for P cells and S gathered faces per cell
// The stride between positions, in elements, where lanes write their own
// position's gc couplings into shared memory: a multiple of 64 bytes would put
// every lane on the same banks (the 4 x 4 blocks of 3D DG1), so one 16-byte
// unit is added there
__host__ __device__ constexpr int LaneStride(int gc, int elem) { return gc * elem % 64 == 0 ? gc + 16 / elem : gc; }

// The stride between staged class records, odd in 16-byte units
__host__ __device__ constexpr int RecordStride(int size, int elem) { return (size * elem / 16 | 1) * 16 / elem; }

struct SweepSlice {
   int loc, G, rec, pass, ghost, bar, bytes;
   __host__ __device__ constexpr SweepSlice(int P, int S, int F, int NB, int n_loc, int n_ghost, int elem, bool cached)
       : loc(0), G(0), rec(0), pass(0), ghost(0), bar(0), bytes(0)
   {
      G = 16;                                                     // after the copy's mbarrier: T [ncell][NB][S][NB],
                                                                  // and up to one 16-byte unit of lead-in
      loc = G + Pad16(P * (cached ? S * NB * NB : LaneStride(S * NB * NB, elem)) * elem, 1) + 16;
                                                                  // T [n_loc][NB]: a zero, the positions, the ghosts
      rec = Pad16(loc + n_loc * NB * elem, 1);                    // uint16 [P][SchedWords(F)]
      ghost = rec + P * SchedWords(F) * 2;                        // int32 [n_ghost]: the ghosts' cells
      pass = ghost + n_ghost * 4;                                 // uint16 [P + 2]
      bytes = Pad16(pass + (P + 2) * 2, 1);
   }
};


// The factor store, per task from element off R, R = NB^2 (1 + S): W = B^{-1}
// element-major over the task's positions (element e of position i at
// e ncell + i, the lanes of a prologue read consecutive words), then the
// couplings position by position, row-major over (row, slot, column): what one
// lane of the walk reads is one run. Unused slots are zero. Independent of the
// right-hand side: built once per group, read by every sweep. The couplings
// are laid out in shared memory and written 32 positions at a time.
// A block takes a patch: its cells' class records are staged in shared memory
// once (STAGED, where they fit) and read by the tasks of every ordinate, a warp
// per task or, where that leaves warps without one, per 32 positions of a task.
// Read by a lane per position straight from global memory, every load touched 32
// lines, which bound the kernel (and the factors built in the sweep itself). A
// group's factors, FP64 / FP32, a warp per task from global memory and this way:
// 256^2 triangles S8 724 / 415 -> 428 / 285 us, 20^3 cubes of tetrahedra 2088 /
// 1339 -> 1027 / 542, 40^3 hexahedra 2263 / 2033 -> 946 / 483, 125 hexahedra S8
// 10 / 10 -> 13 / 8. Slower on 2D meshes of a few hundred thousand cell-ordinates
// in FP64, whose larger patches are few blocks: 101 x 77 triangles S6 50 / 31 ->
// 60 / 35, 150^2 S4 71 / 41 -> 88 / 46; without staging there 65, a warp per 32
// positions 90, patches of 64 cells less, but a sweep takes 5 to 10 us longer then.
template <typename T, int NB, int F, bool STAGED>
__global__ void __launch_bounds__(256, sizeof(T) == 8 && NB == 4 ? 1 : 2) FactorKernel(const DevGeom<T> g, const SweepDev s, T *__restrict__ fac,
                                                    const int32_t *__restrict__ patch_ptr,
                                                    const int32_t *__restrict__ patch_task, int chunks)
{
   constexpr int RS = RecordLayout(NB, F, (int)sizeof(T)).size;
   constexpr int RP = RecordStride(RS, (int)sizeof(T));
   extern __shared__ __align__(16) unsigned char smem_raw[];
   const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n_warps = blockDim.x >> 5;
   const int S = s.slots, GC = S * NB * NB;
   const int GP = LaneStride(GC, (int)sizeof(T));
   T *recs = reinterpret_cast<T *>(smem_raw);
   T *stage = recs + (STAGED ? (size_t)s.P * RP : 0) + (size_t)warp * 32 * GP;
   const unsigned magic = ((1u << 20) + GC - 1) / GC;  // e / GC for e < 32 GC, GC <= 80 (exact: e * GC < 2^20)
   const size_t R = (size_t)NB * NB * (1 + S);
   const int64_t base = (int64_t)blockIdx.x * s.P;
   if constexpr (STAGED) {
      constexpr int UN = RS * (int)sizeof(T) / 16;
      const int nc = (int)min((int64_t)s.P, g.n_cells - base);
      // A warp per record, the class ids of four read at once (a lane per 16-byte
      // unit, each behind a class id of its own, took 10 us before the first task)
      for (int k0 = warp; k0 < nc; k0 += 4 * n_warps) {
         int32_t cl[4];
#pragma unroll
         for (int m = 0; m < 4; m++) cl[m] = g.cls[base + min(k0 + m * n_warps, nc - 1)];
#pragma unroll
         for (int m = 0; m < 4; m++) {
            const int k = k0 + m * n_warps;
            if (k < nc)
               for (int u = lane; u < UN; u += 32)
                  CpAsync<16>(recs + k * RP + u * (16 / (int)sizeof(T)),
                              g.rec + (int64_t)cl[m] * RS + u * (16 / (int)sizeof(T)));
         }
      }
      CpAsyncWaitAll();
      __syncthreads();
   }
   // A warp's unit of work: a task, or every `chunks`th 32 positions of one
   const int x0 = patch_ptr[blockIdx.x], n_units = (patch_ptr[blockIdx.x + 1] - x0) * chunks;
   for (int x = warp + n_warps * (int)blockIdx.y; x < n_units; x += n_warps * (int)gridDim.y) {
      const Task tk = LoadTask(s.task + patch_task[x0 + x / chunks]);
      const int ncell = tk.ncell(), a = tk.ordinate;
      const T om[3] = {g.omega[3 * a], g.omega[3 * a + 1], g.omega[3 * a + 2]};
      T *ft = fac + (size_t)tk.off * R;
      for (int i0 = 32 * (x % chunks); i0 < ncell; i0 += 32 * chunks) {
         // A lane past the end repeats the last position
         const int i = min(i0 + lane, ncell - 1);
         const int local = s.sched[(tk.off + i) * SchedWords(F)];
         const T *rec = STAGED ? recs + local * RP : g.rec + (int64_t)g.cls[base + local] * RS;
         T W[NB][NB];
         CellFactors<T, NB, F, STAGED>(rec, g.sigma_t[base + local], om, s.tmask[tk.off + i], S, W, stage + lane * GP, (size_t)NB,
                               (size_t)S * NB, 1);
#pragma unroll
         for (int ii = 0; ii < NB; ii++)
#pragma unroll
            for (int j = 0; j < NB; j++) ft[(size_t)(ii * NB + j) * ncell + i] = W[ii][j];
         __syncwarp();
         T *Gt = ft + (size_t)NB * NB * ncell + (size_t)i0 * GC;
         const int n = min(32, ncell - i0) * GC;
#pragma unroll 4
         for (int e = lane; e < n; e += 32) {
            const int q = (int)((e * magic) >> 20);
            Gt[e] = stage[q * GP + (e - q * GC)];
         }
         __syncwarp();
      }
   }
}

// Blocks of two warps the registers should leave room for per SM: eight (at
// most 128 registers), ten for FP32 tetrahedra, whose small tasks are bound by
// their number in flight (496 against 537 us per sweep of 20^3 cubes; the
// other shapes measured the same or slower), and no cap where the blocks would
// spill heavily and shared memory holds fewer anyway
template <typename T, int NB, int S, int KU>
constexpr int SweepMinBlocks()
{
   if (sizeof(T) == 8 && NB == 4 && (KU > 1 || S == 5)) return 1;
   return sizeof(T) == 4 && NB == 4 && KU == 1 ? 10 : 8;
}

// The sweep. A warp takes one task at a time.
//
// Prologue: one record says where the task's data are; then, all in flight at
// once, its couplings G come into shared memory by one bulk copy, and each
// lane reads, for its positions, the schedule record, W and q, and for its
// ghosts (cells of earlier tasks the task reads) the values stored so far. It
// leaves y0 = W q and the ghosts in the task's value table.
//
// Walk: pass by pass (a level, cut to the positions a warp holds at NB lanes
// each), one lane per row of a cell: psi_row = y0_row - sum_slots G_row .
// psi(up), the upwind values from the value table. What does not depend on
// other cells (y0, the G row, the links) is read one pass ahead, so a pass's
// critical path is the read of the upwind values, NB multiply-adds per slot
// and the store: about 240 cycles alone and 370 among 16 warps per SM (FP32
// triangles), against 520 for a lane per cell with all its rows. A task has
// 2 to 6 cells per level, so rows and not cells fill the lanes.
template <typename T, int NB, int F, int S, int KU, bool CACHED>
__global__ void __launch_bounds__(64, SweepMinBlocks<T, NB, S, KU>()) SweepKernel(const DevGeom<T> g, const SweepDev s,
                                                                                 const T *__restrict__ q,
                                                                                 T *__restrict__ psi,
                                                                                 const T *__restrict__ fac)
{
   extern __shared__ __align__(128) unsigned char smem_raw[];
   const int lane = threadIdx.x & 31;
   constexpr int EL = (int)sizeof(T);
   constexpr int IP = 32 / NB;        // positions of one pass
   constexpr int GC = S * NB * NB;    // coupling elements of a position
   constexpr int GP = CACHED ? GC : LaneStride(GC, EL);
   constexpr int SW = SchedWords(F);
   constexpr size_t R = (size_t)NB * NB * (1 + S);
   const SweepSlice L(s.P, S, F, NB, s.n_loc, s.n_ghost, EL, CACHED);
   unsigned char *slice = smem_raw + (size_t)(threadIdx.x >> 5) * L.bytes;
   uint64_t *bar = reinterpret_cast<uint64_t *>(slice + L.bar);
   T *table = reinterpret_cast<T *>(slice + L.loc), *loc = table + NB;
   uint16_t *pass = reinterpret_cast<uint16_t *>(slice + L.pass);
   int32_t *gcell = reinterpret_cast<int32_t *>(slice + L.ghost);
   const T *never = reinterpret_cast<const T *>(s.ctrl + kCtrlNever);
   // A lane's position within a pass and its row (a spare lane: a position
   // past every pass)
   const int li = lane < IP * NB ? lane / NB : 1 << 20, lr = lane % NB;
   // The factor store is read once per sweep: its lines go first from L2, so
   // that they do not push out psi and the schedule other warps are reading
   const uint64_t stream_once = EvictFirstPolicy();
   if (lane < NB) table[lane] = T(0);
   if (CACHED && lane == 0) {
      MbarInit(bar, 1);
      MbarInitFence();
   }
   __syncwarp();
   uint32_t phase = 0;
   for (;;) {
      // A task is claimed only when the warp is free: a task claimed while
      // the warp still walks (and waits in) another would sit idle behind it,
      // and the tasks downstream of it would wait too (claiming even two
      // levels before the walk ends measured slower)
      const int64_t t = __shfl_sync(0xffffffffu, AtomicIncIf(lane == 0, &s.ctrl[kCtrlCounter]), 0);
      if (t >= s.n_tasks) break;
      const Task tk = LoadTask(s.task + t);
      const int ncell = tk.ncell(), npass = tk.npass(), nghost = tk.nghost();
      const int64_t off = tk.off;
      const int a = tk.ordinate;
      const int64_t base = (int64_t)tk.patch * s.P;
      const bool hook = (t == s.unmet_task);
      T *G = reinterpret_cast<T *>(slice + L.G);
      const T *ft = fac + (size_t)off * R;
      if constexpr (CACHED) {
         // A bulk copy moves whole 16-byte units: from the unit the couplings
         // start in (the store has a spare unit at its end)
         const uintptr_t src = reinterpret_cast<uintptr_t>(ft + NB * NB * ncell);
         const int lead = (int)(src & 15);
         G += lead / EL;
         const uint32_t bytes = (uint32_t)(lead + GC * ncell * EL + 15) & ~15u;
         BulkLoadIf(lane == 0, slice + L.G, reinterpret_cast<const void *>(src - lead), bytes, bar, stream_once);
      }
      // No lane branches on its own below: a lane past the end repeats the last
      // position or ghost (the same values to the same place)
      const int32_t *gid = s.ghost + tk.ghost0;
      const T *psi_a = psi + a * s.os_a;
      const int glast = max(nghost - 1, 0);
      const int32_t gh[2] = {gid[min(lane, glast)], gid[min(lane + 32, glast)]};
      const uint16_t pass_word = s.pass[tk.pass0 + min(lane, npass - 1)];
#pragma unroll 1
      for (int i0 = 0; i0 < ncell; i0 += 32 * KU) {
         using Rec = typename std::conditional<SW == 4, uint2, uint4>::type;
         Rec rec[KU];
         T W[KU][NB][NB], r[KU][NB], gx[2][NB];
         int at[KU];
#pragma unroll
         for (int k = 0; k < KU; k++) {
            const int i = at[k] = min(i0 + 32 * k + lane, ncell - 1);
            rec[k] = __ldg(reinterpret_cast<const Rec *>(s.sched) + off + i);
            if constexpr (CACHED)
#pragma unroll
               for (int e = 0; e < NB * NB; e++) W[k][e / NB][e % NB] = LoadHint(ft + (e * ncell + i), stream_once);
         }
         if (i0 == 0 && nghost > 0) {
            // The ghosts' values where stored already, else the sentinel
#pragma unroll
            for (int k = 0; k < 2; k++) {
               if (k == 1 && nghost <= 32) break;
#pragma unroll
               for (int j = 0; j < NB; j++) gx[k][j] = LoadRelaxed(psi_a + gh[k] * s.os_c + j * s.os_j);
            }
         }
#pragma unroll
         for (int k = 0; k < KU; k++) {
            const int64_t c = base + (int)(rec[k].x & 0xffffu);
            if (!s.aff_phi) {
               const T *qc = q + c * s.qs_c + a * s.qs_a;
#pragma unroll
               for (int j = 0; j < NB; j++) r[k][j] = qc[j * s.qs_j];
            } else {
               const double ua = s.aff_u ? (double)static_cast<const T *>(s.aff_u)[a] : 1.0;
               const double *ph = s.aff_phi + c * NB;
               if (!s.aff_iso) {
                  const double al = *s.aff_alpha;
                  const T *qc = q + c * s.qs_c + a * s.qs_a;
                  const double *rh = s.aff_rho + c * NB;
#pragma unroll
                  for (int j = 0; j < NB; j++) r[k][j] = (T)(al * (double)qc[j * s.qs_j] + ua * (ph[j] - al * rh[j]));
               } else if (s.aff_inv_volume) {
                  const double v = (double)g.volume[c];
#pragma unroll
                  for (int j = 0; j < NB; j++) r[k][j] = (T)(ua * ph[j] / v);
               } else {
#pragma unroll
                  for (int j = 0; j < NB; j++) r[k][j] = (T)(ua * ph[j]);
               }
            }
         }
#pragma unroll
         for (int k = 0; k < KU; k++) {
            const int i = at[k];
            if constexpr (!CACHED) {
               if (i0 + 32 * k + lane >= ncell) continue;
               const T om[3] = {g.omega[3 * a], g.omega[3 * a + 1], g.omega[3 * a + 2]};
               T *Gi = G + i * GP;
               const int64_t c = base + (int)(rec[k].x & 0xffffu);
               CellFactors<T, NB, F, false>(g.rec + (int64_t)g.cls[c] * RecordLayout(NB, F, EL).size, g.sigma_t[c], om,
                                     s.tmask[off + i], S, W[k], Gi, (size_t)NB, (size_t)S * NB, 1);
            }
#pragma unroll
            for (int ii = 0; ii < NB; ii++) {
               T u = T(0);
#pragma unroll
               for (int j = 0; j < NB; j++) u += W[k][ii][j] * r[k][j];
               loc[i * NB + ii] = u;
            }
            reinterpret_cast<Rec *>(slice + L.rec)[i] = rec[k];
         }
         if (i0 == 0 && nghost > 0) {
#pragma unroll
            for (int k = 0; k < 2; k++) {
               if (k == 1 && nghost <= 32) break;
               const int i = min(lane + 32 * k, glast);
               gcell[i] = gh[k];
#pragma unroll
               for (int j = 0; j < NB; j++) loc[(ncell + i) * NB + j] = hook ? Sentinel<T>() : gx[k][j];
            }
         }
      }
      // Past the last pass the array repeats its end: two lookahead reads
      if (lane < 2) pass[npass + lane] = (uint16_t)ncell;
      pass[min(lane, npass - 1)] = pass_word;
      for (int i0 = 32; i0 < npass; i0 += 32) {
         const int i = min(i0 + lane, npass - 1);
         pass[i] = s.pass[tk.pass0 + i];
      }
      for (int i0 = 64; i0 < nghost; i0 += 32) {
         const int i = min(i0 + lane, glast);
         const T *up = psi_a + gid[i] * s.os_c;
         gcell[i] = gid[i];
#pragma unroll
         for (int j = 0; j < NB; j++) {
            const T v = LoadRelaxed(up + j * s.os_j);
            loc[(ncell + i) * NB + j] = hook ? Sentinel<T>() : v;
         }
      }
      if constexpr (CACHED) {
         // The couplings are in
         if (!MbarWaitBounded(bar, phase, kCopyTries)) {
            atomicOr(&s.ctrl[kCtrlError], 1u);
            atomicAdd(&s.ctrl[kCtrlError + 1], 1u);
            MbarWaitBounded(bar, phase, kCopyTries);
            return;
         }
      }
      phase ^= 1u;
      __syncwarp();

      // The walk. Every lane runs every pass (a branch that splits a warp cost
      // 100 cycles a pass and more, as much as the pass itself); a lane
      // without a row repeats position 0 and stores nothing
      unsigned char *out = reinterpret_cast<unsigned char *>(psi + base * s.os_c + lr * s.os_j + a * s.os_a);
      const int cell_bytes = (int)s.os_c * EL;
      const T *Gr = G + lr * (S * NB);
      const int ghost_from = (1 + ncell) * NB;
      struct Own {  // what a row needs besides the upwind values
         T y, g[S * NB];
         uint16_t rec[SW];
         int pos;
         bool act;
      };
      auto fetch = [&](Own &o, int p0, int p1) {
         o.act = p0 + li < p1;
         o.pos = o.act ? p0 + li : 0;
         memcpy(o.rec, slice + L.rec + o.pos * (SW * 2), SW * 2);
         o.y = loc[o.pos * NB + lr];
         LoadRow<T, S * NB, NB == 4>(Gr + o.pos * GP, o.g);
      };
      int p1 = pass[0], p2 = pass[1], l = 0;
      auto step = [&](Own &cur, Own &nxt) {
         T x[S][NB];
#pragma unroll
         for (int sl = 0; sl < S; sl++)
            LoadRow<T, NB, NB == 4>(table + cur.rec[1 + sl], x[sl]);
         // While those are on their way, the next pass's own data
         fetch(nxt, p1, p2);
         p1 = p2;
         p2 = pass[l + 2];
         // The row as if every ghost were there; then whether one may be
         // missing, by the sentinel's upper word alone
         auto row = [&]() {
            T v = cur.y;
#pragma unroll
            for (int sl = 0; sl < S; sl++) {
               T u = T(0);
#pragma unroll
               for (int j = 0; j < NB; j++) u += cur.g[sl * NB + j] * x[sl][j];
               v -= u;
            }
            return v;
         };
         T yr = row();
         uint32_t top = 0;
#pragma unroll
         for (int sl = 0; sl < S; sl++)
#pragma unroll
            for (int j = 0; j < NB; j++) top = max(top, TopWord(x[sl][j]));
         if (__any_sync(0xffffffffu, cur.act && top == 0xffffffffu)) {
            // Poll, one value per lane, a window of ghosts from the first
            // missing one this pass reads: the ghosts are numbered in the order
            // the passes read them, so the window holds what the next passes
            // wait for too, and they find it in the value table (polling
            // this pass's ghosts alone cost every later pass that reads a late
            // one a round trip of its own). Bounded: on giving up the sticky
            // error flag is set, the timeout counted, and this pass's missing
            // values read as zero
            for (uint32_t spins = 0;;) {
               int first = nghost;
#pragma unroll
               for (int sl = 0; sl < S; sl++) {
                  const int link = cur.rec[1 + sl];
                  const bool need = cur.act && link >= ghost_from &&
                                    IsSentinel(table[link + lr]);
                  first = need ? min(first, (link - ghost_from) / NB) : first;
               }
               const bool mine_missing = first < nghost;
               first = __reduce_min_sync(0xffffffffu, first);
               if (first == nghost) break;
               const int w = first + min(li, IP), i = min(w, glast), at = (ncell + i) * NB + lr;
               T v = loc[at];
               const bool ask = lane < IP * NB && w < nghost && IsSentinel(v);
               // (test hook: this wait can never be met)
               const T *src = hook ? never : psi_a + gcell[i] * s.os_c + lr * s.os_j;
               LoadRelaxedIf(ask, src, v);
               StoreSharedIf(ask, &loc[at], v);
               __syncwarp();
               // The error flag (another wait gave up) is read once per 1024
               // spins, so that waiting lanes stay off its line
               if (++spins > s.spin_limit ||
                   ((spins & 1023u) == 0 && __any_sync(0xffffffffu, *(volatile uint32_t *)&s.ctrl[kCtrlError]))) {
                  if (mine_missing) {
                     atomicOr(&s.ctrl[kCtrlError], 1u);
                     atomicAdd(&s.ctrl[kCtrlError + 1], 1u);
                  }
#pragma unroll
                  for (int sl = 0; sl < S; sl++) {
                     T *own = table + cur.rec[1 + sl] + lr;
                     StoreSharedIf(cur.act && cur.rec[1 + sl] >= ghost_from && IsSentinel(*own), own, T(0));
                  }
                  __syncwarp();
                  break;
               }
               if (spins > 64) __nanosleep(spins < 4096 ? 32 : 256);
            }
#pragma unroll
            for (int sl = 0; sl < S; sl++) LoadRow<T, NB, NB == 4>(table + cur.rec[1 + sl], x[sl]);
            yr = row();
         }
         StoreSharedIf(cur.act, &loc[cur.pos * NB + lr], yr);
         StoreRelaxedIf(cur.act, reinterpret_cast<T *>(out + cur.rec[0] * cell_bytes), Publishable(yr));
         __syncwarp();
      };
      Own own_a, own_b;
      fetch(own_a, 0, p1);
      while (true) {
         step(own_a, own_b);
         if (++l == npass) break;
         step(own_b, own_a);
         if (++l == npass) break;
      }
      __syncwarp();
   }
}

// ~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~~

static int ReserveFactors(ubolt_ctx *ctx, int64_t limit);

// Couplings kept per cell: the kernels are built for 2 on triangles, 2 or 3
// on quadrilaterals and tetrahedra, 3 or 5 on hexahedra
static int SweepSlots(int F, int max_inflow)
{
   const int least = F == 6 ? 3 : 2;
   return max_inflow <= least ? least : F - 1;
}

// The wave plan and both precisions' store layouts (host work and uploads;
// no store is reserved here). Leaves wave_ok false where the mesh has an
// upwind cycle or a level or front too large for one block.
static int BuildWavePlan(ubolt_ctx *ctx, ubolt_sweep_plan *plan)
{
   if (plan->wave_tried) return UBOLT_OK;
   plan->wave_tried = true;
   HostWavePlan h;
   BuildHostWavePlan(ctx->n_cells, ctx->F, ctx->A, ctx->h_omega.data(), ctx->h_nA.data(), ctx->h_code.data(), h);
   if (!h.acyclic || h.S > std::min(4, ctx->F - 1) || h.n_slots >= 0xffff || h.max_width > 512) return UBOLT_OK;
   const int S = std::max(1, h.S);
   int dev = 0, max_smem = 0;
   cudaGetDevice(&dev);
   if (cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
      cudaGetLastError();
      return UBOLT_OK;
   }
   const int A = ctx->A;
   const int64_t total = h.lvl_base[A];
   std::vector<int32_t> lvl_ord(total);
   for (int a = 0; a < A; a++)
      for (int32_t L = h.lvl_base[a]; L < h.lvl_base[a + 1]; L++) lvl_ord[L] = a;
   int rc = 0;
   ubolt::WaveDev base;
   base.A = A;
   base.S = S;
   base.n_slots = h.n_slots;
   base.max_levels = h.max_levels;
   base.n_cells = ctx->n_cells;
   const int32_t *meta = nullptr;
   if ((rc = UploadVec(ctx, h.lvl_base, &base.lvl_base)) || (rc = UploadVec(ctx, h.lvl_pos, &base.lvl_pos)) ||
       (rc = UploadVec(ctx, lvl_ord, &base.lvl_ord)) || (rc = UploadVec(ctx, h.meta, &meta)))
      return rc;
   base.meta = reinterpret_cast<const int4 *>(meta);
   bool any = false;
   for (int which = 0; which < 2; which++) {
      WaveLayout L;
      if (!BuildWaveLayout(h, ctx->nb, which ? 4 : 8, max_smem, L)) continue;
      ubolt::WaveDev w = base;
      if ((rc = UploadVec(ctx, L.region, &w.region)) || (rc = UploadVec(ctx, L.chunk_rel, &w.chunk_rel)) ||
          (rc = UploadVec(ctx, L.ring_off, &w.ring_off)))
         return rc;
      w.front_off = L.front_off;
      w.ring_base = L.ring_base;
      w.cap = L.cap;
      w.smem = L.smem;
      plan->wave[which] = w;
      plan->wave_bytes[which] = L.store_bytes;
      any = true;
   }
   plan->wave_ok = any;
   plan->wave_threads = h.max_width <= 256 ? 256 : 512;
   plan->wave_levels = total;
   return UBOLT_OK;
}

int BuildSweepPlan(ubolt_ctx *ctx, int patch_size)
{
   if (int rc = RequireDg(ctx, "the sweep")) return rc;
   const int64_t nc = ctx->n_cells;
   int P = patch_size > 0 ? patch_size : DefaultPatch(ctx);
   if (P > 256) P = 256;
   if (P > nc) P = (int)nc;
   if (((nc + P - 1) / P) * (int64_t)ctx->A * 4 >= INT32_MAX) return SetError(UBOLT_ERR_ARG, "too many sweep tasks");
   HostSweepPlan h;
   BuildHostSweepPlan(nc, ctx->F, ctx->A, P, ctx->h_omega.data(), ctx->h_nA.data(), ctx->h_code.data(), h);

   auto plan = new ubolt_sweep_plan();
   plan->P = h.P;
   plan->n_patches = h.n_patches;
   plan->A = h.A;
   plan->n_tasks = h.n_tasks;
   plan->n_lagged = h.n_lagged;
   plan->n_split = h.n_split;
   plan->max_levels = h.max_levels;
   plan->max_inflow = h.max_inflow;
   if (h.max_inflow > ctx->F - 1) {
      delete plan;
      return SetError(UBOLT_ERR_ARG, "a cell has %d upwind faces for one ordinate (at most %d)", h.max_inflow, ctx->F - 1);
   }
   plan->total_levels = (int64_t)h.lvl.size();
   plan->slots = SweepSlots(ctx->F, h.max_inflow);
   // Every entry's schedule record, with the upwind cells' places in the
   // task's value table in face order; the cells of earlier tasks a task reads
   // (its ghosts); and the passes, a level cut to the positions a warp walks
   // at nb lanes each. Each thread takes a run of tasks and appends to lists
   // of its own, joined in order
   const int per_pass = 32 / ctx->nb, SW = SchedWords(ctx->F), nb = ctx->nb;
   std::vector<uint16_t> sched(h.tcell.size() * SW, 0);
   std::vector<Task> task(h.n_tasks);
   const int n_parts = (int)std::min<int64_t>(std::max<int64_t>(1, h.n_tasks / 256), 256);
   struct Part {
      std::vector<uint16_t> pass;
      std::vector<int32_t> ghost;
      int n_loc = 0, n_ghost = 1;
   };
   std::vector<Part> part(n_parts);
#pragma omp parallel for schedule(dynamic, 1)
   for (int k = 0; k < n_parts; k++) {
      Part &out = part[k];
      std::vector<int32_t> pos_of(h.P, 0), mine;
      for (int64_t t = h.n_tasks * k / n_parts; t < h.n_tasks * (k + 1) / n_parts; t++) {
         const int64_t base = (int64_t)(h.task_pa[t] / h.A) * h.P, e0 = h.cell_ptr[t];
         const int ncell = (int)(h.cell_ptr[t + 1] - e0);
         mine.clear();
         for (int i = 0; i < ncell; i++) pos_of[h.tcell[e0 + i]] = i;
         for (int i = 0; i < ncell; i++) {
            const int64_t c = base + h.tcell[e0 + i];
            const uint32_t mask = h.tmask[e0 + i];
            uint16_t *rec = &sched[(e0 + i) * SW];
            rec[0] = h.tcell[e0 + i];
            int slot = 0;
            for (int f = 0; f < ctx->F; f++) {
               const bool here = (mask >> f) & 1u, earlier = (mask >> (8 + f)) & 1u;
               if (!(here || earlier)) continue;
               const int32_t code = ctx->h_code[c * ctx->F + f];
               int at = here ? pos_of[code - base] : 0;
               if (earlier) {
                  const auto it = std::find(mine.begin(), mine.end(), code);
                  at = ncell + (int)(it - mine.begin());
                  if (it == mine.end()) mine.push_back(code);
               }
               rec[1 + slot++] = (uint16_t)((1 + at) * nb);
            }
         }
         out.n_loc = std::max(out.n_loc, ncell + (int)mine.size() + 1);
         out.n_ghost = std::max(out.n_ghost, (int)mine.size());
         const size_t pass0 = out.pass.size();
         int p0 = 0;
         for (int32_t L = h.lvl_ptr[t]; L < h.lvl_ptr[t + 1]; L++) {
            for (; p0 + per_pass < (int)h.lvl[L]; p0 += per_pass) out.pass.push_back((uint16_t)(p0 + per_pass));
            p0 = h.lvl[L];
            out.pass.push_back((uint16_t)p0);
         }
         Task &tk = task[t];
         tk.counts = (uint32_t)ncell | (uint32_t)(out.pass.size() - pass0) << 10 | (uint32_t)mine.size() << 20;
         tk.patch = h.task_pa[t] / h.A;
         tk.ordinate = h.task_pa[t] % h.A;
         tk.off = e0;
         tk.ghost0 = (int64_t)out.ghost.size();
         tk.pass0 = (int32_t)pass0;
         out.ghost.insert(out.ghost.end(), mine.begin(), mine.end());
      }
   }
   std::vector<int64_t> pass_at(n_parts + 1, 0), ghost_at(n_parts + 1, 0);
   for (int k = 0; k < n_parts; k++) {
      pass_at[k + 1] = pass_at[k] + (int64_t)part[k].pass.size();
      ghost_at[k + 1] = ghost_at[k] + (int64_t)part[k].ghost.size();
      plan->n_loc = std::max(plan->n_loc, part[k].n_loc);
      plan->n_ghost = std::max(plan->n_ghost, part[k].n_ghost);
   }
   if (pass_at[n_parts] >= INT32_MAX) {
      delete plan;
      return SetError(UBOLT_ERR_ARG, "too many sweep levels");
   }
   std::vector<uint16_t> pass(pass_at[n_parts]);
   // A spare element, which a last task without ghosts reads (and does not use)
   std::vector<int32_t> ghost(ghost_at[n_parts] + 1, 0);
#pragma omp parallel for schedule(dynamic, 1)
   for (int k = 0; k < n_parts; k++) {
      std::copy(part[k].pass.begin(), part[k].pass.end(), pass.begin() + pass_at[k]);
      std::copy(part[k].ghost.begin(), part[k].ghost.end(), ghost.begin() + ghost_at[k]);
      for (int64_t t = h.n_tasks * k / n_parts; t < h.n_tasks * (k + 1) / n_parts; t++) {
         task[t].pass0 += (int32_t)pass_at[k];
         task[t].ghost0 += ghost_at[k];
      }
   }
   std::vector<int32_t> patch_ptr(h.n_patches + 1, 0), patch_task(h.n_tasks);
   for (int64_t t = 0; t < h.n_tasks; t++) patch_ptr[task[t].patch + 1]++;
   for (int32_t k = 0; k < h.n_patches; k++) patch_ptr[k + 1] += patch_ptr[k];
   {
      std::vector<int32_t> at(patch_ptr.begin(), patch_ptr.end() - 1);
      for (int64_t t = 0; t < h.n_tasks; t++) patch_task[at[task[t].patch]++] = (int32_t)t;
   }
   int rc = 0;
   if ((rc = UploadVec(ctx, patch_ptr, &plan->patch_ptr)) || (rc = UploadVec(ctx, patch_task, &plan->patch_task)) ||
       (rc = UploadVec(ctx, task, &plan->task)) || (rc = UploadVec(ctx, h.dep_ptr, &plan->dep_ptr)) ||
       (rc = UploadVec(ctx, h.deps, &plan->deps)) || (rc = UploadVec(ctx, sched, &plan->sched)) ||
       (rc = UploadVec(ctx, h.tmask, &plan->tmask)) || (rc = UploadVec(ctx, pass, &plan->pass)) ||
       (rc = UploadVec(ctx, ghost, &plan->ghost))) {
      delete plan;
      return rc;
   }
   void *p = nullptr;
   if ((rc = CtxAlloc(ctx, kCtrlWords * sizeof(uint32_t), &p))) { delete plan; return rc; }
   plan->ctrl = static_cast<uint32_t *>(p);
   cudaMemset(plan->ctrl, 0, kCtrlWords * sizeof(uint32_t));
   cudaMemset(plan->ctrl + kCtrlNever, 0xff, 2 * sizeof(uint32_t));
   if (ctx->sweep) {
      plan->fac_limit = ctx->sweep->fac_limit;
      plan->kernel_mode = ctx->sweep->kernel_mode;
   }
   if (plan->kernel_mode == UBOLT_SWEEP_WAVE || (plan->kernel_mode == UBOLT_SWEEP_AUTO && WaveByDefault(ctx))) {
      if ((rc = BuildWavePlan(ctx, plan))) { delete plan; return rc; }
      if (!plan->wave_ok) plan->kernel_mode = UBOLT_SWEEP_AUTO;
   }
   delete ctx->sweep;
   ctx->sweep = plan;
   if ((rc = CudaCheck(cudaDeviceSynchronize(), "sweep plan"))) return rc;
   return ReserveFactors(ctx, plan->fac_limit);
}

static SweepDev DevPlan(const ubolt_sweep_plan *pl)
{
   SweepDev s;
   s.P = pl->P;
   s.A = pl->A;
   s.n_tasks = pl->n_tasks;
   s.task = pl->task;
   s.sched = pl->sched;
   s.tmask = pl->tmask;
   s.ghost = pl->ghost;
   s.n_loc = pl->n_loc;
   s.n_ghost = pl->n_ghost;
   s.pass = pl->pass;
   s.ctrl = pl->ctrl;
   s.spin_limit = pl->spin_limit;
   s.unmet_task = -1;
   s.slots = pl->slots;
   s.aff_alpha = s.aff_phi = s.aff_rho = nullptr;
   s.aff_u = nullptr;
   s.aff_iso = 0;
   s.aff_inv_volume = 0;
   return s;
}

// The layouts of psi and of q for the task kernel
static void SetLayout(SweepDev &s, const ubolt_ctx *ctx, bool psi_om, bool q_om)
{
   const int64_t nb = ctx->nb, A = ctx->A;
   s.os_c = psi_om ? nb : nb * A;
   s.os_j = psi_om ? 1 : A;
   s.os_a = psi_om ? ctx->n_cells * nb : 1;
   s.qs_c = q_om ? nb : nb * A;
   s.qs_j = q_om ? 1 : A;
   s.qs_a = q_om ? ctx->n_cells * nb : 1;
}

// Between UBOLT's rows, x[node A + a], and ordinate-major, y[a n_nodes + node]:
// a block moves 64 nodes of up to 64 ordinates through shared memory, so that
// both its reads and its writes are runs of whole sectors. Bound by bandwidth.
constexpr int kTransNodes = 64, kTransOrds = 64;
template <typename T, bool TO_OM>
__global__ void __launch_bounds__(256) TransposeKernel(const T *__restrict__ in, T *__restrict__ out, int A, int chunk,
                                                       int64_t n_nodes)
{
   __shared__ T tile[kTransNodes][kTransOrds + 1];
   const int64_t node0 = (int64_t)blockIdx.x * kTransNodes;
   const int a0 = blockIdx.y * chunk, na = min(chunk, A - a0);
   const int nn = (int)min((int64_t)kTransNodes, n_nodes - node0);
   const int lane = threadIdx.x & 63, part = threadIdx.x >> 6;
   // e / na for e < 4096 and na <= 64 (exact: e * na < 2^20)
   const unsigned magic = ((1u << 20) + na - 1) / na;
   if (TO_OM) {
#pragma unroll 4
      for (int e = threadIdx.x; e < nn * na; e += 256) {
         const int n = (int)((e * magic) >> 20), a = e - n * na;
         tile[n][a] = in[(node0 + n) * A + a0 + a];
      }
      __syncthreads();
      if (lane < nn)
#pragma unroll 4
         for (int a = part; a < na; a += 4) out[(int64_t)(a0 + a) * n_nodes + node0 + lane] = tile[lane][a];
   } else {
      if (lane < nn)
#pragma unroll 4
         for (int a = part; a < na; a += 4) tile[lane][a] = in[(int64_t)(a0 + a) * n_nodes + node0 + lane];
      __syncthreads();
#pragma unroll 4
      for (int e = threadIdx.x; e < nn * na; e += 256) {
         const int n = (int)((e * magic) >> 20), a = e - n * na;
         out[(node0 + n) * A + a0 + a] = tile[n][a];
      }
   }
}

template <typename T>
static void Transpose2(const ubolt_ctx *ctx, const T *in, T *out, bool to_om, cudaStream_t st)
{
   const int parts = (ctx->A + kTransOrds - 1) / kTransOrds, chunk = (ctx->A + parts - 1) / parts;
   const dim3 grid((unsigned)((ctx->n_nodes + kTransNodes - 1) / kTransNodes), (unsigned)parts);
   if (to_om) TransposeKernel<T, true><<<grid, 256, 0, st>>>(in, out, ctx->A, chunk, ctx->n_nodes);
   else TransposeKernel<T, false><<<grid, 256, 0, st>>>(in, out, ctx->A, chunk, ctx->n_nodes);
   CountLaunch();
}

// x in UBOLT's rows to ordinate-major y
template <typename T>
void ToOrdinateMajor(ubolt_ctx *ctx, const T *x, T *y, cudaStream_t st)
{
   Transpose2<T>(ctx, x, y, true, st);
}
template void ToOrdinateMajor<double>(ubolt_ctx *, const double *, double *, cudaStream_t);
template void ToOrdinateMajor<float>(ubolt_ctx *, const float *, float *, cudaStream_t);

// Bytes of the factor store for one precision
static int64_t FactorBytes(const ubolt_ctx *ctx, const ubolt_sweep_plan *pl, size_t elem)
{
   return (int64_t)ctx->n_cells * ctx->A * ctx->nb * ctx->nb * (1 + pl->slots) * (int64_t)elem;
}

// Reserve the factor stores - at set-up (plan build, or an explicit limit),
// never inside a sweep. limit < 0: each store that fits, FP32 first, within
// half the free device memory at that moment (at most 96 GiB); 0: none;
// otherwise the byte limit for both together. A store not reserved means
// the sweep computes its factors as it goes: the result is the same.
static int ReserveFactors(ubolt_ctx *ctx, int64_t limit)
{
   ubolt_sweep_plan *pl = ctx->sweep;
   if (pl->fac[0] || pl->fac[1] || pl->scratch) cudaDeviceSynchronize();
   if (pl->scratch) cudaFree(pl->scratch);
   pl->scratch = nullptr;
   for (int which = 0; which < 2; which++) {
      if (pl->fac[which]) cudaFree(pl->fac[which]);
      pl->fac[which] = nullptr;
      pl->fac_epoch[which] = 0;
   }
   if (limit < 0) {
      size_t free_b = 0, total_b = 0;
      if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
         cudaGetLastError();
         return UBOLT_OK;
      }
      limit = std::min<int64_t>((int64_t)(free_b / 2), (int64_t)96 << 30);
   }
   int64_t left = limit;
   for (int which : {1, 0}) {
      // The wave kernel's store is in wave order
      const bool wave = pl->wave[which].smem > 0 &&
                        (pl->kernel_mode == UBOLT_SWEEP_WAVE ||
                         (pl->kernel_mode == UBOLT_SWEEP_AUTO && WaveByDefault(ctx)));
      pl->fac_wave[which] = false;
      const int64_t bytes = wave ? pl->wave_bytes[which] : FactorBytes(ctx, pl, which ? 4 : 8);
      if (bytes > left) continue;
      void *p = nullptr;
      if (cudaMalloc(&p, (size_t)bytes + 16) != cudaSuccess) {  // a copy of whole 16-byte units may end past the last factor
         cudaGetLastError();
         continue;
      }
      pl->fac[which] = p;
      pl->fac_wave[which] = wave;
      left -= bytes;
   }
   const int64_t vec = ctx->n_rows * (int64_t)sizeof(double);
   // (only where a sweep between row vectors goes through it, see LaunchSweep)
   if (ctx->nb > 1 && vec >= (int64_t)kViaBytes && vec <= left && !(pl->fac_wave[0] && pl->fac_wave[1])) {
      if (cudaMalloc(&pl->scratch, (size_t)vec) != cudaSuccess) {
         cudaGetLastError();
         pl->scratch = nullptr;
      }
   }
   return UBOLT_OK;
}

// The factor store for precision T, rebuilt by a kernel (no allocation) for
// the current group: ubolt_set_group starts a new one. nullptr where none
// is reserved: the sweep then computes its factors as it goes.
template <typename T, int NB, int F>
static T *EnsureFactors(ubolt_ctx *ctx, cudaStream_t st)
{
   ubolt_sweep_plan *pl = ctx->sweep;
   const int which = sizeof(T) == 8 ? 0 : 1;
   if (!pl->fac[which]) return nullptr;
   if (pl->fac_epoch[which] == ctx->group_epoch) return static_cast<T *>(pl->fac[which]);
   if (pl->fac_wave[which]) {
      if (WaveFactors(ctx, pl->wave[which], pl->fac[which], (int)sizeof(T), st, pl->wave_levels)) return nullptr;
      pl->fac_epoch[which] = ctx->group_epoch;
      return static_cast<T *>(pl->fac[which]);
   }
   int smem_max = 48 * 1024, n_sm = 1, dev = 0;
   cudaGetDevice(&dev);
   cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
   cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
   // Eight warps per patch, its class records in shared memory where they fit
   // beside the warps' staging
   const int warps = 8;
   const size_t stage = (size_t)warps * 32 * LaneStride(pl->slots * NB * NB, (int)sizeof(T)) * sizeof(T);
   const size_t recs = (size_t)pl->P * RecordStride(RecordLayout(NB, F, (int)sizeof(T)).size, (int)sizeof(T)) * sizeof(T);
   const bool staged = recs + stage <= (size_t)smem_max;
   const size_t smem = (staged ? recs : 0) + stage;
   auto kern = staged ? FactorKernel<T, NB, F, true> : FactorKernel<T, NB, F, false>;
   if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
   // Large patches make few blocks: then several share a patch's tasks. Where all
   // tasks' pieces of 32 positions are one for a warp at most, a warp takes a piece
   // (64^2 DG0 quadrilaterals S4 18 -> 8 us, 16 x 15 x 17 hexahedra S2 20 -> 14; with
   // more, 101 x 77 triangles S6 60 and 90: every block stages its patch's records)
   const int most_chunks = (pl->P + 31) / 32;
   const int chunks = !staged || pl->n_tasks * most_chunks <= (int64_t)n_sm * 16 ? most_chunks : 1;
   const int parts = std::max(1, std::min((n_sm * 8 + pl->n_patches - 1) / pl->n_patches, (ctx->A * chunks + warps - 1) / warps));
   kern<<<dim3(pl->n_patches, parts), 32 * warps, smem, st>>>(ctx->geom<T>(), DevPlan(pl), static_cast<T *>(pl->fac[which]),
                                                 pl->patch_ptr, pl->patch_task, chunks);
   if (CheckLaunch("sweep factors")) return nullptr;
   pl->fac_epoch[which] = ctx->group_epoch;
   return static_cast<T *>(pl->fac[which]);
}

template <typename T, int NB, int F>
static int LaunchSweep(ubolt_ctx *ctx, const T *q, T *psi, cudaStream_t st, const SweepDev *affine = nullptr,
                       bool ordinate_major = false, bool q_om = false)
{
   ubolt_sweep_plan *pl = ctx->sweep;
   const int which = sizeof(T) == 8 ? 0 : 1;
   // What the wave kernel cannot do the task kernel does where the
   // choice is automatic, its factors formed as it goes: the store is the wave's
   const bool not_wave = ordinate_major || q_om || (affine && affine->aff_inv_volume);
   const bool wave = pl->fac_wave[which] && !(not_wave && pl->kernel_mode == UBOLT_SWEEP_AUTO);
   const T *fac = pl->fac_wave[which] && !wave ? nullptr : EnsureFactors<T, NB, F>(ctx, st);
   if (wave) {
      // One block per ordinate over the store in wave order (no sentinel fill)
      if (!fac) return UBOLT_ERR_CUDA;  // the failed launch set the message
      if (ordinate_major) return SetError(UBOLT_ERR_STATE, "the wave sweep writes the row layout only");
      if (affine && affine->aff_inv_volume) return SetError(UBOLT_ERR_STATE, "the wave sweep takes no 1 / V source");
      WaveDev w = pl->wave[which];
      w.ctrl = pl->ctrl;
      w.spin_limit = pl->spin_limit;
      w.unmet_level = pl->unmet_level;
      pl->unmet_level = -1;
      pl->unmet_task = -1;
      pl->grid = ctx->A;
      WaveInput in;
      if (affine) {
         in.alpha = affine->aff_alpha;
         in.phi = affine->aff_phi;
         in.rho = affine->aff_rho;
         in.u = affine->aff_u;
         in.iso = affine->aff_iso;
      }
      return WaveSweep(ctx, w, q, psi, fac, (int)sizeof(T), affine ? &in : nullptr, pl->wave_threads, st);
   }
   // Two warps per block; one where the patch's couplings leave no room for two
   const size_t slice = (size_t)SweepSlice(pl->P, pl->slots, F, NB, pl->n_loc, pl->n_ghost, (int)sizeof(T), fac != nullptr).bytes;
   constexpr int S0 = F == 6 ? 3 : 2;
   // Two positions per lane in a prologue where the tasks hold more than a
   // warp's worth, one where they are small (jittered tetrahedra, whose patches'
   // cells are split over several tasks)
   const bool wide = ctx->n_cells * (int64_t)ctx->A > 24 * pl->n_tasks;
   auto kern = pl->slots == S0 ? (fac ? (wide ? SweepKernel<T, NB, F, S0, 2, true> : SweepKernel<T, NB, F, S0, 1, true>)
                                      : (wide ? SweepKernel<T, NB, F, S0, 2, false> : SweepKernel<T, NB, F, S0, 1, false>))
                               : (fac ? (wide ? SweepKernel<T, NB, F, F - 1, 2, true> : SweepKernel<T, NB, F, F - 1, 1, true>)
                                      : (wide ? SweepKernel<T, NB, F, F - 1, 2, false> : SweepKernel<T, NB, F, F - 1, 1, false>));
   int per_sm = 0, n_sm = 0, dev = 0, smem_max = 48 * 1024;
   cudaGetDevice(&dev);
   cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev);
   cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
   const int warps = 2 * slice <= (size_t)smem_max ? 2 : 1, threads = 32 * warps;
   const size_t smem = warps * slice;
   if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
   cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem);
   // At most 32 warps per SM (small DG0 tasks): beyond the throughput the
   // wavefront can use, more resident warps only take tasks early and wait
   per_sm = std::min(per_sm, kSweepWarpsPerSm / warps);
   const int64_t want = (pl->n_tasks + warps - 1) / warps;
   const int grid = (int)std::max<int64_t>(1, std::min<int64_t>((int64_t)std::max(per_sm, 1) * n_sm, want));
   pl->grid = grid;
   SweepDev s = DevPlan(pl);
   // Row vectors in and out: in UBOLT's rows a task's values of one ordinate
   // lie A apart, each its own sector in and out. Where there are several
   // rows per cell and more than a few MB, the sweep itself runs
   // ordinate-major, psi holding q's ordinate-major copy meanwhile and the
   // scratch vector the result: two passes at memory bandwidth against the
   // scattered words. Per sweep, FP64 / FP32, direct and this way: 256^2
   // triangles 916 / 586 -> 702 / 564 us, 40^3 hexahedra 1094 / 900 -> 775 /
   // 481, 20^3 cubes of tetrahedra 1278 / 890 -> 1054 / 576; DG0 quadrilaterals
   // 244 -> 247 and a 1.1 M-row FP32 vector 151 -> 154, which stay direct
   T *dst = psi;
   const bool via = !ordinate_major && !q_om && pl->scratch && NB > 1 && ctx->n_rows * sizeof(T) >= kViaBytes;
   if (via) {
      if (!affine || !affine->aff_iso) {
         Transpose2<T>(ctx, q, psi, true, st);
         q = psi;
      }
      dst = static_cast<T *>(pl->scratch);
   }
   SetLayout(s, ctx, ordinate_major || via, q_om || via);
   if (affine) {
      s.aff_alpha = affine->aff_alpha;
      s.aff_phi = affine->aff_phi;
      s.aff_rho = affine->aff_rho;
      s.aff_u = affine->aff_u;
      s.aff_iso = affine->aff_iso;
      s.aff_inv_volume = affine->aff_inv_volume;
   }
   s.unmet_task = pl->unmet_task;
   pl->unmet_task = -1;
   cudaMemsetAsync(pl->ctrl + kCtrlCounter, 0, sizeof(uint32_t), st);  // task counter; the error flag stays sticky
   // Every psi value starts as the sentinel: "not yet stored by its task"
   cudaMemsetAsync(dst, 0xff, (size_t)ctx->n_cells * NB * ctx->A * sizeof(T), st);
   kern<<<grid, threads, smem, st>>>(ctx->geom<T>(), s, q, dst, fac);
   const int rc = CheckLaunch("sweep");
   if (rc || !via) return rc;
   Transpose2<T>(ctx, dst, psi, false, st);
   return CudaCheck(cudaGetLastError(), "sweep");
}

template <typename T>
int Sweep(ubolt_ctx *ctx, const T *q, T *psi, void *stream, bool ordinate_major)
{
   int rc = CheckReady(ctx, true);
   if (rc) return rc;
   if (!ctx->sweep && (rc = BuildSweepPlan(ctx, 0))) return rc;
   if (!q || !psi || (const void *)q == (const void *)psi)
      return SetError(UBOLT_ERR_ARG, "sweep: q and psi must be distinct device arrays");
   UBOLT_DISPATCH(ctx->nb, ctx->F,
                  return (LaunchSweep<T, NB_, F_>(ctx, q, psi, (cudaStream_t)stream, nullptr, ordinate_major)));
   return SetError(UBOLT_ERR_STATE, "no sweep kernel for this shape");
}
template <typename T>
int Sweep(ubolt_ctx *ctx, const T *q, T *psi, void *stream)
{
   return Sweep<T>(ctx, q, psi, stream, false);
}

// True where the sweep is L^{-1} exactly: a plan with no lagged coupling and
// no reflective side (reflective inflow is lagged)
bool SweepIsExact(ubolt_ctx *ctx)
{
   if (!ctx->sweep && BuildSweepPlan(ctx, 0)) return false;
   return ctx->sweep->n_lagged == 0 && !ctx->has_reflect;
}

// psi = L^{-1} (alpha r0 + E_u (phi - alpha rho)) with the input formed as
// the sweep reads it (u = 1, or u_a = u[a]); alpha, phi, rho on the device.
// r0 == nullptr: r0 is isotropic, r0 = E_u rho, and the input is E_u phi.
// inv_volume (r0 == nullptr only): the input is u_a phi(node) / V(cell).
template <typename T>
int SweepAffine(ubolt_ctx *ctx, const T *r0, const double *alpha, const double *phi, const double *rho, const T *u,
                T *psi, void *stream, bool ordinate_major, bool inv_volume)
{
   int rc = CheckReady(ctx, true);
   if (rc) return rc;
   if (!ctx->sweep && (rc = BuildSweepPlan(ctx, 0))) return rc;
   if (inv_volume && r0) return SetError(UBOLT_ERR_ARG, "sweep: the 1 / V source is isotropic only");
   SweepDev aff{};
   aff.aff_alpha = alpha;
   aff.aff_phi = phi;
   aff.aff_rho = rho;
   aff.aff_u = u;
   aff.aff_iso = r0 == nullptr;
   aff.aff_inv_volume = inv_volume;
   UBOLT_DISPATCH(ctx->nb, ctx->F,
                  return (LaunchSweep<T, NB_, F_>(ctx, r0, psi, (cudaStream_t)stream, &aff, ordinate_major)));
   return SetError(UBOLT_ERR_STATE, "no sweep kernel for this shape");
}

// True where the next sweep in precision T runs the task kernel (which can
// write psi ordinate-major); false where the wave kernel runs
template <typename T>
bool SweepWritesOrdinateMajor(ubolt_ctx *ctx)
{
   if (!ctx->sweep && BuildSweepPlan(ctx, 0)) return false;
   const int which = sizeof(T) == 8 ? 0 : 1;
   return !(ctx->sweep->fac[which] && ctx->sweep->fac_wave[which]);
}

template int SweepAffine<double>(ubolt_ctx *, const double *, const double *, const double *, const double *,
                                 const double *, double *, void *, bool, bool);
template int SweepAffine<float>(ubolt_ctx *, const float *, const double *, const double *, const double *,
                                const float *, float *, void *, bool, bool);
template int Sweep<double>(ubolt_ctx *, const double *, double *, void *, bool);
template int Sweep<float>(ubolt_ctx *, const float *, float *, void *, bool);
template bool SweepWritesOrdinateMajor<double>(ubolt_ctx *);
template bool SweepWritesOrdinateMajor<float>(ubolt_ctx *);
template int Sweep<double>(ubolt_ctx *, const double *, double *, void *);
template int Sweep<float>(ubolt_ctx *, const float *, float *, void *);

}  // namespace ubolt

using namespace ubolt;

void UboltSweepFree(ubolt_ctx *ctx)
{
   delete ctx->sweep;
   ctx->sweep = nullptr;
}

extern "C" int ubolt_sweep_setup(ubolt_ctx *ctx, int patch_size)
{
   int rc = CheckReady(ctx, false);
   if (rc) return rc;
   if (patch_size < 0 || patch_size > 256) return SetError(UBOLT_ERR_ARG, "patch size %d (1..256, 0 = default)", patch_size);
   return BuildSweepPlan(ctx, patch_size);
}

extern "C" int ubolt_sweep_set_kernel(ubolt_ctx *ctx, int kernel)
{
   int rc = CheckReady(ctx, false);
   if (rc) return rc;
   if (kernel < UBOLT_SWEEP_AUTO || kernel > UBOLT_SWEEP_WAVE) return SetError(UBOLT_ERR_ARG, "sweep kernel %d", kernel);
   if (!ctx->sweep && (rc = BuildSweepPlan(ctx, 0))) return rc;
   ubolt_sweep_plan *pl = ctx->sweep;
   if ((kernel == UBOLT_SWEEP_WAVE || (kernel == UBOLT_SWEEP_AUTO && WaveByDefault(ctx))) && (rc = BuildWavePlan(ctx, pl)))
      return rc;
   if (kernel == UBOLT_SWEEP_WAVE && !pl->wave_ok)
      return SetError(UBOLT_ERR_STATE, "the wave sweep does not apply here (an upwind cycle, or a level or front too "
                                       "large for one block)");
   if (kernel == pl->kernel_mode) return UBOLT_OK;
   pl->kernel_mode = kernel;
   // The stores' layout follows the kernel: reserved again, rebuilt by the next sweep
   return ReserveFactors(ctx, pl->fac_limit);
}

extern "C" int ubolt_sweep(ubolt_ctx *ctx, const double *q, double *psi, void *stream)
{
   return Sweep<double>(ctx, q, psi, stream);
}

extern "C" int ubolt_sweep_f32(ubolt_ctx *ctx, const float *q, float *psi, void *stream)
{
   return Sweep<float>(ctx, q, psi, stream);
}

template <typename T>
static int SweepIso(ubolt_ctx *ctx, const double *phi, const T *u, T *psi, int ordinate_major, void *stream)
{
   int rc = CheckReady(ctx, true);
   if (rc) return rc;
   if (!phi || !psi) return SetError(UBOLT_ERR_ARG, "sweep_iso: NULL array");
   if (!ctx->sweep && (rc = BuildSweepPlan(ctx, 0))) return rc;
   if (ordinate_major && ctx->sweep->kernel_mode == UBOLT_SWEEP_WAVE && !SweepWritesOrdinateMajor<T>(ctx))
      return SetError(UBOLT_ERR_STATE, "sweep_iso: the wave kernel runs here, and it writes the row layout only");
   return SweepAffine<T>(ctx, nullptr, nullptr, phi, nullptr, u, psi, stream, ordinate_major != 0, false);
}

extern "C" int ubolt_sweep_iso(ubolt_ctx *ctx, const double *phi, const double *u, double *psi, int ordinate_major,
                               void *stream)
{
   return SweepIso<double>(ctx, phi, u, psi, ordinate_major, stream);
}

extern "C" int ubolt_sweep_iso_f32(ubolt_ctx *ctx, const double *phi, const float *u, float *psi, int ordinate_major,
                                   void *stream)
{
   return SweepIso<float>(ctx, phi, u, psi, ordinate_major, stream);
}

extern "C" int ubolt_sweep_set_factor_limit(ubolt_ctx *ctx, int64_t bytes)
{
   int rc = CheckReady(ctx, false);
   if (rc) return rc;
   if (!ctx->sweep) {
      if ((rc = BuildSweepPlan(ctx, 0))) return rc;
   }
   ctx->sweep->fac_limit = bytes;
   return ReserveFactors(ctx, bytes);
}

extern "C" int ubolt_sweep_status(ubolt_ctx *ctx, ubolt_sweep_info *info, void *stream)
{
   int rc = CheckReady(ctx, false);
   if (rc) return rc;
   if (!ctx->sweep) return SetError(UBOLT_ERR_STATE, "no sweep plan");
   ubolt_sweep_plan *pl = ctx->sweep;
   uint32_t h[2] = {0, 0};  // error flag, timeout count
   cudaStream_t s = (cudaStream_t)stream;
   cudaMemcpyAsync(h, pl->ctrl + kCtrlError, sizeof h, cudaMemcpyDeviceToHost, s);
   if ((rc = CudaCheck(cudaStreamSynchronize(s), "sweep_status"))) return rc;
   if (info) {
      info->patch_size = pl->P;
      info->n_patches = pl->n_patches;
      info->n_tasks = pl->n_tasks;
      info->n_lagged = pl->n_lagged;
      info->n_split = pl->n_split;
      info->max_levels = pl->max_levels;
      info->total_levels = pl->total_levels;
      info->grid = pl->grid;
      info->timeouts = h[1];
      info->kernel = (pl->fac[0] && pl->fac_wave[0]) ? UBOLT_SWEEP_WAVE : UBOLT_SWEEP_TASKS;
      info->factor_bytes = 0;
      info->factor_bytes_fp64 = 0;
      for (int which = 0; which < 2; which++)
         if (pl->fac[which]) {
            const int64_t b = pl->fac_wave[which] ? pl->wave_bytes[which] : FactorBytes(ctx, pl, which ? 4 : 8);
            info->factor_bytes += b;
            if (which == 0) info->factor_bytes_fp64 = b;
         }
   }
   if (h[0]) {
      cudaMemsetAsync(pl->ctrl + kCtrlError, 0, 2 * sizeof(uint32_t), s);
      cudaStreamSynchronize(s);
      return SetError(UBOLT_ERR_TIMEOUT, "a sweep wait gave up (%u timeouts); its result is not valid", h[1]);
   }
   return UBOLT_OK;
}

extern "C" int ubolt_sweep_test_wait(ubolt_ctx *ctx, uint32_t spin_limit, int make_one_wait_unmet)
{
   int rc = CheckReady(ctx, false);
   if (rc) return rc;
   if (!ctx->sweep && (rc = BuildSweepPlan(ctx, 0))) return rc;
   ubolt_sweep_plan *pl = ctx->sweep;
   if (spin_limit < 16) return SetError(UBOLT_ERR_ARG, "spin limit %u too small", spin_limit);
   pl->spin_limit = spin_limit;
   pl->unmet_task = -1;
   pl->unmet_level = -1;
   if (make_one_wait_unmet && pl->fac[0] && pl->fac_wave[0]) {
      // The wave kernel runs the next FP64 sweep: ordinate 0's first level
      // waits for a copy never issued
      pl->unmet_level = 0;
      return UBOLT_OK;
   }
   if (make_one_wait_unmet) {
      // The first task that has an upstream task polls, for its first
      // upwind value, a word that no task of the sweep stores
      std::vector<int32_t> dp(pl->n_tasks + 1);
      if ((rc = CudaCheck(cudaMemcpy(dp.data(), pl->dep_ptr, dp.size() * sizeof(int32_t), cudaMemcpyDeviceToHost),
                          "sweep_test_wait")))
         return rc;
      for (int64_t t = 0; t < pl->n_tasks; t++)
         if (dp[t + 1] > dp[t]) { pl->unmet_task = t; break; }
      if (pl->unmet_task < 0) return SetError(UBOLT_ERR_STATE, "no task of this plan waits on another");
   }
   return UBOLT_OK;
}
