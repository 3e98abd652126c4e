// Triangular sweeps with one CTA per component (sm_100a): the ILU and SSOR
// applies of component-diagonal matrices.
//
// What bounds a sweep is the hand-off from a level to the next one: about
// 0.85 us when the value travels through L2 from one SM to another
// (kernels_sweep.cu).  The components of a component-diagonal matrix never
// meet, so each can be solved by a CTA of its own, and inside a CTA a level
// ends with a barrier and its values travel through shared memory.  The price
// is that one SM does all the rows of a component, so this path is taken while
// the levels are narrow enough for that (local_sweep_warps).
//
// A level's rows are cut into steps of up to W tasks, a task being up to 32
// rows, one per lane; a team of W warps takes a step, and T teams take the
// steps in turn.  Step s waits for step s - 1 at a named barrier that team s - 1
// arrives at and team s waits at, so all a step leaves between two barriers is
// its shared-memory reads, its sums and one store.  A task's operands come by
// asynchronous copies, kDepth of the warp's tasks ahead, issued while the other
// teams have the barrier: loads into registers do not stay in flight that long
// (the same kernel with them took 0.95 us a level at 250 rows, however deep the
// pipeline).  Nothing polls: warps polling shared memory for a sentinel took
// 310 ns a level at 17 rows and 0.95 us at 250, the polls taking the issue
// slots.  One ILU(0) apply, FP64, before (all SMs, levels through L2) and now:
//   4,096 rows, 17 a level: 350 -> 47 us (W 1); 50,000 rows, 58 a level:
//   1,390 -> 235 us (W 2); 200,000 rows, 115 a level: 2,880 -> 700 us (W 4);
//   1,000,000 rows, 252 a level: 6,780 -> 3,270 us (W 4).
// A step of one warp costs 75 ns, of two 95, of four 145: the wide steps are
// bound by shared-memory wavefronts (about 80 a task: the gathers of the
// results, and the operands once in and once out), which is also why eight
// warps a team are slower than four.
//
// Results live in a shared-memory ring in step order, and a dependency is a
// 16-bit ring slot.  One further back than the ring reaches is final in global
// memory long before; it is copied into the task's stage like its operands (a
// row of a low level may be read thousands of levels later: at 490,000 rows,
// RCM order, 0.2% of the rows have such a dependency in the forward sweep).  Tasks with rows
// of more than kHold dependencies, or more than 32 far ones, read 32-bit codes
// and the far values in place instead.  Absent dependencies read
// a slot that holds zero with a zero coefficient, which leaves every y, -0 and
// NaN included, as it is.
//
// Per (row, component) the arithmetic is the reference's
// (preconditioner.hpp:165-247, :320-363), term by term in entry order with
// explicit rounding, so results equal the CPU path bit for bit.

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <future>
#include <memory>
#include <type_traits>
#include <utility>

#include <cuda_bf16.h>

#include "device_common.cuh"
#include "owtk_internal.h"

namespace owtk {
namespace {

using namespace dev;

constexpr int kHold = 8;              // dependencies held in registers
constexpr int kTaskEntries = 192;     // padded entries of a task that is staged
constexpr int kDepth = 2;             // tasks a warp has in flight (3 and 4: the same times)
constexpr int kSharedBytes = 226 * 1024;
// Teams by warps per team: as many as shared memory leaves a ring for and, at
// four warps, as registers allow (at 1,000,000 rows 4, 5 and 6 teams of four
// took 4,150, 3,730 and 3,260 us).
constexpr int kTeams1 = 12, kTeams2 = 12, kTeams4 = 6;
// Dense blocks: teams of one warp, as many as there are named barriers and as
// their stages leave a ring for.  A visit is some 500 instructions, so what a
// step costs is the visit over the number of teams (four warps a team, fewer
// teams: the same at 82 rows a level, two to three times slower below 32).
constexpr int block_teams(std::size_t stage)
{
    return static_cast<int>(std::min<std::size_t>(15, 170 * 1024 / (kDepth * stage)));
}

// A task's packed word: rows, width << 8, and
constexpr int kFarFlag = 1 << 24;     // some dependencies are staged from global memory
constexpr int kSlowFlag = 1 << 25;    // the slower form
constexpr int kFarSlot = 0xffe0;      // slots from here on: the task's far values
constexpr int kMaxEntries = 1 << 30;

template<class T> struct Bits;
template<> struct Bits<double> {
    static __device__ __forceinline__ double quiet_nan() { return __longlong_as_double(0x7ff8000000000000ll); }
};
template<> struct Bits<float> {
    static __device__ __forceinline__ float quiet_nan() { return __uint_as_float(0x7fc00000u); }
};

__device__ __forceinline__ void ld_ring(std::uint32_t a, double& v)
{
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void ld_ring(std::uint32_t a, float& v)
{
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
}
__device__ __forceinline__ void st_ring(std::uint32_t a, double v)
{
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_ring(std::uint32_t a, float v)
{
    asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
template<int THREADS> __device__ __forceinline__ void bar_wait(int id)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}
template<int THREADS> __device__ __forceinline__ void bar_signal(int id)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(THREADS) : "memory");
}

__device__ __forceinline__ void copy16(std::uint32_t to, const void* from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
template<class T> __device__ __forceinline__ void copy_value(std::uint32_t to, const T* from)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to), "l"(from), "n"(sizeof(T)) : "memory");
}

// One direction of a sweep; arrays as in LocalSweep.
template<class T>
struct Direction {
    const int4* task;        // [step][warp of the team]: first entry, first place, packed word, first ring slot
    const std::uint16_t* slots;   // per entry: ring slot, or kFarSlot + k for the task's k-th far value
    const int* far;          // [step][warp][32]: where the far values are (null: there are none)
    const int* code;         // per entry: ring slot, or -1 - index of a far dependency (null: no slow task)
    const int* to;           // per place: where its result goes (row, or place in the backward order)
    const T* coef;           // per component and entry
    const T* fin;            // per component and place: factor or divisor of the result
    const T* in;             // per component and place
    T* out;                  // forward: per component and place of the backward order; backward: the result
    std::size_t entries, places, out_places;
    int steps, ring, bs;
};

// A task's operands in shared memory.
template<class T>
struct __align__(16) Stage {
    T coef[kTaskEntries];                // [dependency][row]
    std::uint16_t slots[kTaskEntries];   // [dependency pair][row][2]
    int to[32];
    T own[32], fin[32], far[32];
    int4 task;
};

static_assert(sizeof(Stage<double>) % 16 == 0 && sizeof(Stage<float>) % 16 == 0, "stages are copied in 16-byte pieces");

// Where a lane copies a task's operands from, before the task's own offsets.
template<class T>
struct Source {
    const T* coef;
    const T* row;            // own (first lanes) or fin
    const char* index;       // slots (24 lanes) or to
    const T* far;            // result of the direction, for far values
    std::size_t far_step;
};

template<class T, bool BACK>
__device__ __forceinline__ Source<T> source_of(const Direction<T>& d, int lane, int c)
{
    constexpr int kPer = 16 / static_cast<int>(sizeof(T)), kRowLanes = 32 / kPer;
    Source<T> s;
    s.coef = d.coef + static_cast<std::size_t>(c) * d.entries + lane * kPer;
    const std::size_t q = static_cast<std::size_t>(c) * d.places;
    s.row = lane < kRowLanes ? d.in + q + lane * kPer : d.fin + q + (lane - kRowLanes) * kPer;
    s.index = lane < 24 ? reinterpret_cast<const char*>(d.slots) + lane * 16
                        : reinterpret_cast<const char*>(d.to) + (lane - 24) * 16;
    s.far = d.out + (BACK ? static_cast<std::size_t>(c) : static_cast<std::size_t>(c) * d.out_places);
    s.far_step = BACK ? d.bs : 1;
    return s;
}

// Up to six copies a lane: a task's entries are contiguous and padded to 8,
// its rows to 4.
template<class T, bool FIN>
__device__ __forceinline__ void load_operands(const Source<T>& s, int lane, int4 task, int far, std::uint32_t stage)
{
    constexpr int kSize = static_cast<int>(sizeof(T)), kPer = 16 / kSize, kRowLanes = 32 / kPer;
    constexpr std::uint32_t kSlots = kTaskEntries * kSize, kOwn = kSlots + kTaskEntries * 2 + 128;
    const int rows = task.z & 0xff;
    if (rows > 0) {
        const int entries = task.z & kSlowFlag ? 0 : rows * (task.z >> 8 & 0xff);
        const T* coef = s.coef + task.x;
        const std::uint32_t at = stage + lane * 16;
#pragma unroll
        for (int i = 0; i < kTaskEntries; i += 32 * kPer)
            if (i + lane * kPer < entries) copy16(at + i * kSize, coef + i);
        if (lane >= 24 || lane * 8 < entries)
            copy16(at + kSlots, s.index + (lane < 24 ? static_cast<std::size_t>(task.x) * 2
                                                     : static_cast<std::size_t>(task.y) * 4));
        if (lane < (FIN ? 2 * kRowLanes : kRowLanes)) copy16(at + kOwn, s.row + task.y);
        if (task.z & kFarFlag && far >= 0)
            copy_value(stage + kOwn + (64 + lane) * kSize, s.far + static_cast<std::size_t>(far) * s.far_step);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// The slower form: eight dependencies at a time, loaded when their turn comes.
template<class T, bool BACK>
__device__ __noinline__ T consume_slow(T y, const Direction<T>* dp, int lane, int c, int4 task, std::uint32_t ring)
{
    const Direction<T>& d = *dp;
    const T* far = d.out + (BACK ? c : static_cast<std::size_t>(c) * d.out_places);
    const std::size_t far_step = BACK ? d.bs : 1;
    const int rows = task.z & 0xff, width = task.z >> 8 & 0xff, at = task.x + min(lane, rows - 1);
    for (int j0 = 0; j0 < width; j0 += kHold) {
        T x[kHold], coef[kHold];
#pragma unroll
        for (int j = 0; j < kHold; ++j) {
            coef[j] = x[j] = T(0);
            if (j0 + j < width) {
                const std::size_t e = static_cast<std::size_t>(at) + (j0 + j) * rows;
                const int code = __ldg(d.code + e);
                coef[j] = __ldg(d.coef + static_cast<std::size_t>(c) * d.entries + e);
                if (code >= 0) ld_ring(ring + code * static_cast<int>(sizeof(T)), x[j]);
                else x[j] = __ldcg(far + static_cast<std::size_t>(-1 - code) * far_step);
            }
        }
#pragma unroll
        for (int j = 0; j < kHold; ++j) y = sub_rn(y, mul_rn(coef[j], x[j]));
    }
    return y;
}

// One task of `N` padded dependencies: the operands from the stage, the wait
// for the step before, the sums and the store that the next step waits for.
// Straight-line between the barriers, because every instruction there is paid
// once per step (uniform branches on the width there made a step of one warp
// 250 cycles).  Returns the result of the lane's row.
template<class T, int N, int PAIR, bool BACK, bool SSOR>
__device__ __forceinline__ T run_task(const Stage<T>& h, const int4& task, int lane, std::uint32_t ring,
                                      std::uint32_t slot, bool wait, bool signal, int wait_id, int signal_id)
{
    constexpr int kSize = static_cast<int>(sizeof(T));
    const int rows = task.z & 0xff, l = min(lane, rows - 1);
    const bool live = lane < rows;
    std::uint32_t at[N > 0 ? N : 1];
    T coef[N > 0 ? N : 1], x[N > 0 ? N : 1];
#pragma unroll
    for (int j = 0; j < N; j += 2) {
        const unsigned pair = *reinterpret_cast<const unsigned*>(h.slots + j * rows + 2 * l);
        const unsigned a0 = pair & 0xffffu, a1 = pair >> 16;
        at[j] = ring + a0 * kSize;
        at[j + 1] = ring + a1 * kSize;
        if (task.z & kFarFlag) {
            const std::uint32_t far = smem_u32(h.far) - kFarSlot * kSize;
            if (a0 >= kFarSlot) at[j] = far + a0 * kSize;
            if (a1 >= kFarSlot) at[j + 1] = far + a1 * kSize;
        }
        coef[j] = h.coef[j * rows + l];
        coef[j + 1] = h.coef[(j + 1) * rows + l];
    }
    T y = h.own[l];
    const T fin = BACK || SSOR ? h.fin[l] : T(1);
    if (BACK && SSOR) y = mul_rn(fin, y);
    if (wait) bar_wait<PAIR>(wait_id);
#pragma unroll
    for (int j = 0; j < N; ++j) ld_ring(at[j], x[j]);
#pragma unroll
    for (int j = 0; j < N; ++j) y = sub_rn(y, mul_rn(coef[j], x[j]));
    if (SSOR) y = div_rn(y, fin);
    else if (BACK) y = mul_rn(y, fin);
    if (live) st_ring(slot, y);
    if (signal) bar_signal<PAIR>(signal_id);
    return y;
}

// The shared memory holds a stage per warp and task in flight, then the ring
// and the slot of absent dependencies.
// SLOW: the schedule has tasks of the slower form (a call in the loop costs
// registers that the others need).
template<class T, int W, int TEAMS, bool BACK, bool SSOR, bool SLOW>
__global__ void __launch_bounds__(W * TEAMS * 32, 1) k_local_sweep(const __grid_constant__ Direction<T> d)
{
    constexpr int kSize = static_cast<int>(sizeof(T)), kStage = static_cast<int>(sizeof(Stage<T>));
    constexpr int kPair = 2 * W * 32;   // threads of a barrier: the team that signals and the one that waits
    extern __shared__ __align__(16) unsigned char shared[];
    const int lane = threadIdx.x & 31, c = blockIdx.x;
    const int w = threadIdx.x / 32 % W, team = threadIdx.x / (32 * W);
    Stage<T>* const stages = reinterpret_cast<Stage<T>*>(shared) + threadIdx.x / 32 * kDepth;
    const std::uint32_t first_stage = smem_u32(stages), ring = smem_u32(shared) + W * TEAMS * kDepth * kStage;
    if (threadIdx.x == 0) st_ring(ring + d.ring * kSize, T(0));
    __syncthreads();
    const Source<T> source = source_of<T, BACK>(d, lane, c);
    const int4* tasks = d.task + w;
    const int* fars = d.far ? d.far + w * 32 + lane : nullptr;
    auto task_of = [&](int s) { return s < d.steps ? __ldg(tasks + s * W) : make_int4(0, 0, 0, 0); };
    auto far_of = [&](int s) { return fars && s < d.steps ? __ldg(fars + static_cast<std::size_t>(s) * W * 32) : -1; };
    for (int u = 0; u < kDepth; ++u) {
        const int4 task = task_of(team + u * TEAMS);
        if (lane == 0) stages[u].task = task;
        load_operands<T, BACK || SSOR>(source, lane, task, far_of(team + u * TEAMS), first_stage + u * kStage);
    }
    int4 next = task_of(team + kDepth * TEAMS);
    int next_far = far_of(team + kDepth * TEAMS);
    const int wait_id = 1 + (team + TEAMS - 1) % TEAMS, signal_id = 1 + team;
    T* const out = d.out + (BACK ? static_cast<std::size_t>(c) : static_cast<std::size_t>(c) * d.out_places);
    int u = 0;
    for (int s = team; s < d.steps; s += TEAMS) {
        Stage<T>& h = stages[u];
        asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
        __syncwarp();
        const int4 task = h.task;
        const int rows = task.z & 0xff;
        const int place = task.w + lane;
        const std::uint32_t slot = ring + (place >= d.ring ? place - d.ring : place) * kSize;
        const bool wait = s > 0, signal = s + 1 < d.steps;
        T y = T(0);
        if (rows == 0) {
            if (wait) bar_wait<kPair>(wait_id);
            if (signal) bar_signal<kPair>(signal_id);
        } else if (SLOW && (task.z & kSlowFlag)) {
            y = h.own[min(lane, rows - 1)];
            const T fin = BACK || SSOR ? h.fin[min(lane, rows - 1)] : T(1);
            if (BACK && SSOR) y = mul_rn(fin, y);
            if (wait) bar_wait<kPair>(wait_id);
            y = consume_slow<T, BACK>(y, &d, lane, c, task, ring);
            if (SSOR) y = div_rn(y, fin);
            else if (BACK) y = mul_rn(y, fin);
            if (lane < rows) st_ring(slot, y);
            if (signal) bar_signal<kPair>(signal_id);
        } else {
            auto run = [&](auto n) {
                y = run_task<T, decltype(n)::value, kPair, BACK, SSOR>(h, task, lane, ring, slot, wait, signal, wait_id,
                                                                       signal_id);
            };
            const int width = task.z >> 8 & 0xff;
            if (width == 4) run(std::integral_constant<int, 4>());
            else if (width == 6) run(std::integral_constant<int, 6>());
            else if (width == 2) run(std::integral_constant<int, 2>());
            else if (width == 0) run(std::integral_constant<int, 0>());
            else run(std::integral_constant<int, 8>());
        }
        const int to = rows > 0 ? h.to[min(lane, rows - 1)] : 0;
        if (lane < rows) {
            if (y != y) y = Bits<T>::quiet_nan();
            out[BACK ? static_cast<std::size_t>(to) * d.bs : static_cast<std::size_t>(to)] = y;
        }
        __syncwarp();
        if (lane == 0) h.task = next;
        load_operands<T, BACK || SSOR>(source, lane, next, next_far, first_stage + u * kStage);
        next = task_of(s + (kDepth + 1) * TEAMS);
        next_far = far_of(s + (kDepth + 1) * TEAMS);
        u = u + 1 == kDepth ? 0 : u + 1;
    }
}

// ---------------------------------------------------------------- dense blocks
// The same for the dense-block ILU, whose components meet in every row: one
// CTA for all of them, a lane per row with its BS sums.  (A lane per block row,
// 32 / BS rows a task, took 1.86 ms where this takes 1.27: as many shared loads
// for a third of the rows.)  A task's blocks lie
// [dependency][element][row] in the factor's storage type, BF16 two elements
// to a word, so a lane's loads neither conflict nor split; a dependency's BS
// values lie side by side in the ring, padded to 2 or 4.
// 100,000 rows, bs 3, 82 rows a level, one apply: BF16 factors 2.94 -> 1.27 ms,
// FP32 2.94 -> 1.09, FP64 3.80 -> 3.04; 4,096 rows, BF16 0.50 -> 0.09.  Bound by
// the instructions of a visit (46% of the issue slots, shared-memory wavefronts
// 39%).
// Padded entries of a task, by the bytes of a block.
constexpr int block_entries(std::size_t bytes) { return bytes <= 40 ? 128 : 64; }

// Stored elements of a block (BF16: made even).
template<class F> constexpr int block_elements(int bs) { return sizeof(F) == 2 ? (bs * bs + 1) / 2 * 2 : bs * bs; }

template<class T, class F, int BS>
struct __align__(16) BlockStage {
    static constexpr int kEntries = block_entries(sizeof(F) * BS * BS);
    alignas(16) F coef[kEntries * block_elements<F>(BS)];
    alignas(16) std::uint16_t slots[kEntries];   // [dependency][row]
    alignas(16) T own[32 * BS];                       // [row][block row]
    alignas(16) F dinv[32 * block_elements<F>(BS)];   // [element][row]
    alignas(16) T far[32 * (BS == 3 ? 4 : BS)];
    alignas(16) int to[32];
    alignas(16) int4 task;
};

template<class T, class F>
struct BlockArgs {
    const int4* task;
    const std::uint16_t* slots;
    const int* far;
    const int* to;
    const F* coef;
    const F* dinv;           // backward, per task
    const T* in;             // per place
    T* out;                  // forward: per place of the backward order; backward: per row
    int steps, ring;
};

__device__ __forceinline__ void copy_run(std::uint32_t to, const void* from, int bytes, int lane)
{
    for (int o = lane * 16; o < bytes; o += 512) copy16(to + o, static_cast<const char*>(from) + o);
}

template<class T, class F, int BS, bool BACK>
__device__ __forceinline__ void load_block(const BlockArgs<T, F>& d, int lane, int4 task, int far,
                                           BlockStage<T, F, BS>& h)
{
    constexpr int kP = BS == 3 ? 4 : BS;
    const int rows = task.z & 0xff, entries = (rows * (task.z >> 8 & 0xff) + 7) & ~7;
    constexpr int kE = block_elements<F>(BS);
    if (lane == 0) h.task = task;
    if (rows > 0) {
        const int padded = (rows + 7) & ~7;   // places of a task are padded to 8, entries too
        copy_run(smem_u32(h.coef), d.coef + static_cast<std::size_t>(task.x) * kE,
                 entries * kE * static_cast<int>(sizeof(F)), lane);
        copy_run(smem_u32(h.slots), d.slots + task.x, entries * 2, lane);
        copy_run(smem_u32(h.own), d.in + static_cast<std::size_t>(task.y) * BS,
                 padded * BS * static_cast<int>(sizeof(T)), lane);
        if (BACK)
            copy_run(smem_u32(h.dinv), d.dinv + static_cast<std::size_t>(task.y) * kE,
                     padded * kE * static_cast<int>(sizeof(F)), lane);
        copy_run(smem_u32(h.to), d.to + task.y, padded * 4, lane);
        if (task.z & kFarFlag && far >= 0) {
#pragma unroll
            for (int j = 0; j < BS; ++j)
                copy_value(smem_u32(h.far) + (lane * kP + j) * static_cast<int>(sizeof(T)),
                           d.out + static_cast<std::size_t>(far) * BS + j);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template<int BS> __device__ __forceinline__ void ld_block(std::uint32_t a, float (&x)[BS])
{
    if constexpr (BS == 1) {
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x[0]) : "r"(a) : "memory");
    } else if constexpr (BS == 2) {
        asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(x[0]), "=f"(x[1]) : "r"(a) : "memory");
    } else {
        float y;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(y) : "r"(a) : "memory");
        if constexpr (BS == 4) x[3] = y;
    }
}
template<int BS> __device__ __forceinline__ void ld_block(std::uint32_t a, double (&x)[BS])
{
    if constexpr (BS == 1) {
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x[0]) : "r"(a) : "memory");
    } else {
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x[0]), "=d"(x[1]) : "r"(a) : "memory");
        if constexpr (BS == 3) {
            asm volatile("ld.shared.f64 %0, [%1];" : "=d"(x[2]) : "r"(a + 16) : "memory");
        } else if constexpr (BS == 4) {
            asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x[2]), "=d"(x[3]) : "r"(a + 16) : "memory");
        }
    }
}

template<class T> __device__ __forceinline__ T widen(double v) { return static_cast<T>(v); }
template<class T> __device__ __forceinline__ T widen(float v) { return static_cast<T>(v); }
template<class T> __device__ __forceinline__ T widen(__nv_bfloat16 v) { return static_cast<T>(__bfloat162float(v)); }

// Elements of a block of `at` (row l of a task of `rows`), widened.
template<class T, class F, int BS>
__device__ __forceinline__ void load_elements(const F* at, int rows, int l, T (&m)[BS * BS])
{
    if constexpr (sizeof(F) == 2) {
#pragma unroll
        for (int e = 0; e < block_elements<F>(BS); e += 2) {
            const unsigned pair = *reinterpret_cast<const unsigned*>(at + e * rows + 2 * l);
            m[e] = __uint_as_float(pair << 16);
            if (e + 1 < BS * BS) m[e + 1] = __uint_as_float(pair & 0xffff0000u);
        }
    } else {
#pragma unroll
        for (int e = 0; e < BS * BS; ++e) m[e] = at[e * rows + l];
    }
}

template<class T, class F, int BS, int N, int PAIR, bool BACK>
__device__ __forceinline__ void run_block_task(const BlockStage<T, F, BS>& h, const int4& task, int lane,
                                               std::uint32_t ring, std::uint32_t slot, bool wait, bool signal,
                                               int wait_id, int signal_id, T (&y)[BS])
{
    constexpr int kP = BS == 3 ? 4 : BS, kBytes = kP * static_cast<int>(sizeof(T)), kE = block_elements<F>(BS);
    const int rows = task.z & 0xff, l = min(lane, rows - 1);
    std::uint32_t at[N > 0 ? N : 1];
    T coef[N > 0 ? N : 1][BS * BS], acc[BS], dinv[BS * BS];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const unsigned a = h.slots[k * rows + l];
        at[k] = ring + a * kBytes;
        if (task.z & kFarFlag && a >= kFarSlot) at[k] = smem_u32(h.far) + (a - kFarSlot) * kBytes;
        load_elements<T, F, BS>(h.coef + k * kE * rows, rows, l, coef[k]);
    }
#pragma unroll
    for (int i = 0; i < BS; ++i) acc[i] = h.own[l * BS + i];
    if (BACK) load_elements<T, F, BS>(h.dinv, rows, l, dinv);
    if (wait) bar_wait<PAIR>(wait_id);
    T x[N > 0 ? N : 1][BS];
#pragma unroll
    for (int k = 0; k < N; ++k) ld_block<BS>(at[k], x[k]);
#pragma unroll
    for (int k = 0; k < N; ++k) {
#pragma unroll
        for (int i = 0; i < BS; ++i) {
            T sum = T(0);
#pragma unroll
            for (int j = 0; j < BS; ++j) sum = add_rn(sum, mul_rn(coef[k][i * BS + j], x[k][j]));
            acc[i] = sub_rn(acc[i], sum);
        }
    }
#pragma unroll
    for (int i = 0; i < BS; ++i) {
        if (BACK) {
            T z = T(0);
#pragma unroll
            for (int j = 0; j < BS; ++j) z = add_rn(z, mul_rn(dinv[i * BS + j], acc[j]));
            y[i] = z;
        } else {
            y[i] = acc[i];
        }
    }
    if (lane < rows) {
#pragma unroll
        for (int i = 0; i < BS; ++i) st_ring(slot + i * static_cast<int>(sizeof(T)), y[i]);
    }
    if (signal) bar_signal<PAIR>(signal_id);
}

template<class T, class F, int BS, int W, int TEAMS, bool BACK>
__global__ void __launch_bounds__(W * TEAMS * 32, 1) k_local_block(const __grid_constant__ BlockArgs<T, F> d)
{
    constexpr int kP = BS == 3 ? 4 : BS, kSize = static_cast<int>(sizeof(T)), kPair = 2 * W * 32;
    using Stages = BlockStage<T, F, BS>;
    extern __shared__ __align__(16) unsigned char shared[];
    const int lane = threadIdx.x & 31, w = threadIdx.x / 32 % W, team = threadIdx.x / (32 * W);
    Stages* const stages = reinterpret_cast<Stages*>(shared) + threadIdx.x / 32 * kDepth;
    const std::uint32_t ring = smem_u32(shared) + W * TEAMS * kDepth * static_cast<int>(sizeof(Stages));
    if (threadIdx.x < kP) st_ring(ring + (d.ring * kP + threadIdx.x) * kSize, T(0));
    __syncthreads();
    const int4* tasks = d.task + w;
    const int* fars = d.far ? d.far + w * 32 + lane : nullptr;
    auto task_of = [&](int s) { return s < d.steps ? __ldg(tasks + s * W) : make_int4(0, 0, 0, 0); };
    auto far_of = [&](int s) { return fars && s < d.steps ? __ldg(fars + static_cast<std::size_t>(s) * W * 32) : -1; };
    for (int u = 0; u < kDepth; ++u)
        load_block<T, F, BS, BACK>(d, lane, task_of(team + u * TEAMS), far_of(team + u * TEAMS), stages[u]);
    int4 next = task_of(team + kDepth * TEAMS);
    int next_far = far_of(team + kDepth * TEAMS);
    const int wait_id = 1 + (team + TEAMS - 1) % TEAMS, signal_id = 1 + team;
    int u = 0;
    for (int s = team; s < d.steps; s += TEAMS) {
        Stages& h = stages[u];
        asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
        __syncwarp();
        const int4 task = h.task;
        const int rows = task.z & 0xff, place = task.w + lane;
        const std::uint32_t slot = ring + (place >= d.ring ? place - d.ring : place) * kP * kSize;
        const bool wait = s > 0, signal = s + 1 < d.steps;
        T y[BS];
        if (rows == 0) {
            if (wait) bar_wait<kPair>(wait_id);
            if (signal) bar_signal<kPair>(signal_id);
        } else {
            auto run = [&](auto n) {
                run_block_task<T, F, BS, decltype(n)::value, kPair, BACK>(h, task, lane, ring, slot, wait, signal,
                                                                          wait_id, signal_id, y);
            };
            const int width = task.z >> 8 & 0xff;
            if (width == 4) run(std::integral_constant<int, 4>());
            else if (width == 6) run(std::integral_constant<int, 6>());
            else if (width == 2) run(std::integral_constant<int, 2>());
            else if (width == 0) run(std::integral_constant<int, 0>());
            else run(std::integral_constant<int, 8>());
        }
        if (lane < rows) {
            T* out = d.out + static_cast<std::size_t>(h.to[lane]) * BS;
#pragma unroll
            for (int i = 0; i < BS; ++i) out[i] = y[i] != y[i] ? Bits<T>::quiet_nan() : y[i];
        }
        __syncwarp();
        load_block<T, F, BS, BACK>(d, lane, next, next_far, h);
        next = task_of(s + (kDepth + 1) * TEAMS);
        next_far = far_of(s + (kDepth + 1) * TEAMS);
        u = u + 1 == kDepth ? 0 : u + 1;
    }
}

// Factor blocks, or inverse diagonal blocks (DIAG: one per place), into the
// order and layout of the tasks; a warp per task.
template<class F, bool DIAG>
__global__ void __launch_bounds__(kThreads) k_local_block_pack(std::size_t tasks, int bs, const int4* __restrict__ task,
                                                               const int* __restrict__ src, const F* __restrict__ from,
                                                               F* __restrict__ to)
{
    const std::size_t t = (static_cast<std::size_t>(blockIdx.x) * kThreads + threadIdx.x) / 32;
    if (t >= tasks) return;
    const int4 h = task[t];
    const int rows = h.z & 0xff, width = DIAG ? 1 : h.z >> 8 & 0xff, b2 = bs * bs;
    const int elements = sizeof(F) == 2 ? (b2 + 1) / 2 * 2 : b2;
    const std::size_t first = static_cast<std::size_t>(DIAG ? h.y : h.x);
    F* out = to + first * elements;
    for (int e = threadIdx.x % 32; e < rows * width; e += 32) {
        const int source = src[first + e], k = e / rows, l = e - k * rows;
        if (source < 0) continue;
        const F* block = from + static_cast<std::size_t>(source) * b2;
        for (int m = 0; m < b2; ++m)
            out[sizeof(F) == 2 ? (k * elements + (m & ~1)) * rows + 2 * l + (m & 1) : (k * elements + m) * rows + l] =
                block[m];
    }
}

// The right-hand side into the forward order.
template<class T>
__global__ void __launch_bounds__(kThreads) k_local_block_gather(std::size_t count, int bs, const int* __restrict__ rows,
                                                                 const T* __restrict__ in, T* __restrict__ to)
{
    const std::size_t i = static_cast<std::size_t>(blockIdx.x) * kThreads + threadIdx.x;
    const std::size_t p = i / bs;
    if (p < count && rows[p] >= 0) to[i] = in[static_cast<std::size_t>(rows[p]) * bs + i % bs];
}

// Into the sweep's layout (component-major, order of the steps): coefficients
// and diagonals of both directions, and the right-hand side.  One thread per
// entry or row, reading its bs values side by side; SCALE: coefficients times
// omega (SSOR).
template<class T, class F>
struct PackArgs {
    const int* src[2];
    T* coef[2];
    std::size_t entries[2];
    const int* rows[2];  // per place (-1: padding)
    T* fin[2];           // null: none
    const T* in;         // null: none
    T* in_to;
    std::size_t places[2];
    const F* vals;
    const F* diag;
    T omega;
    int bs;
};

template<class T, class F, bool SCALE>
__global__ void __launch_bounds__(kThreads) k_local_pack(PackArgs<T, F> a)
{
    std::size_t i = static_cast<std::size_t>(blockIdx.x) * kThreads + threadIdx.x;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        if (i < a.entries[s]) {
            const int e = a.src[s][i];
            if (e < 0) return;
            for (int c = 0; c < a.bs; ++c) {
                const T v = widen<T>(a.vals[static_cast<std::size_t>(e) * a.bs + c]);
                a.coef[s][static_cast<std::size_t>(c) * a.entries[s] + i] = SCALE ? mul_rn(a.omega, v) : v;
            }
            return;
        }
        i -= a.entries[s];
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        if (a.fin[s] == nullptr) continue;
        if (i < a.places[s]) {
            const int row = a.rows[s][i];
            if (row < 0) return;
            for (int c = 0; c < a.bs; ++c)
                a.fin[s][static_cast<std::size_t>(c) * a.places[s] + i] =
                    widen<T>(a.diag[static_cast<std::size_t>(row) * a.bs + c]);
            return;
        }
        i -= a.places[s];
    }
    if (a.in != nullptr && i < a.places[0]) {
        const int row = a.rows[0][i];
        if (row < 0) return;
        for (int c = 0; c < a.bs; ++c)
            a.in_to[static_cast<std::size_t>(c) * a.places[0] + i] = a.in[static_cast<std::size_t>(row) * a.bs + c];
    }
}

// values / in: null leaves the coefficients and diagonals, or the right-hand side, as they are.
template<class T, class F>
void pack(Context& c, Preconditioner& p, const F* values, const F* diag, const T* in, T omega, bool ssor)
{
    PackArgs<T, F> a{};
    LocalSweep* s[2] = {&p.lower_local, &p.upper_local};
    std::size_t total = in ? p.lower_local.places : 0;
    for (int k = 0; k < 2; ++k) {
        a.places[k] = s[k]->places;
        a.rows[k] = s[k]->rows.as<int>();
        if (values == nullptr) continue;
        a.src[k] = s[k]->src.as<int>();
        a.coef[k] = s[k]->coef.as<T>();
        a.entries[k] = s[k]->entries;
        a.fin[k] = ssor || k == 1 ? s[k]->fin.as<T>() : nullptr;
        total += s[k]->entries + (a.fin[k] ? s[k]->places : 0);
    }
    a.in = in;
    a.in_to = p.lower_local.in.as<T>();
    a.vals = values;
    a.diag = diag;
    a.omega = omega;
    a.bs = static_cast<int>(p.bs);
    const unsigned blocks = static_cast<unsigned>((total + kThreads - 1) / kThreads);
    if (ssor) k_local_pack<T, F, true><<<blocks, kThreads, 0, c.stream>>>(a);
    else k_local_pack<T, F, false><<<blocks, kThreads, 0, c.stream>>>(a);
    OWTK_CUDA(cudaGetLastError());
    c.launched();
}

template<class T, int W, int TEAMS, bool BACK, bool SSOR>
void launch_shape(Context& c, const Direction<T>& d)
{
    auto* kernel = d.code ? k_local_sweep<T, W, TEAMS, BACK, SSOR, true> : k_local_sweep<T, W, TEAMS, BACK, SSOR, false>;
    const int bytes = W * TEAMS * kDepth * static_cast<int>(sizeof(Stage<T>)) + (d.ring + 1) * static_cast<int>(sizeof(T));
    OWTK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedBytes));
    kernel<<<static_cast<unsigned>(d.bs), W * TEAMS * 32, bytes, c.stream>>>(d);
    OWTK_CUDA(cudaGetLastError());
    c.launched();
}

template<class T, bool BACK, bool SSOR>
void launch(Context& c, Preconditioner& p, T* out)
{
    const LocalSweep& s = BACK ? p.upper_local : p.lower_local;
    Direction<T> d{};
    d.task = s.task.as<int4>();
    d.slots = s.slots.as<std::uint16_t>();
    d.far = s.far.ptr ? s.far.as<int>() : nullptr;
    d.code = s.code.ptr ? s.code.as<int>() : nullptr;
    d.to = BACK ? s.rows.as<int>() : s.to.as<int>();
    d.coef = s.coef.as<T>();
    d.fin = s.fin.as<T>();
    d.in = s.in.as<T>();
    d.out = BACK ? out : p.upper_local.in.as<T>();
    d.entries = s.entries;
    d.places = s.places;
    d.out_places = p.upper_local.places;
    d.steps = s.steps;
    d.ring = s.ring;
    d.bs = static_cast<int>(p.bs);
    switch (s.warps) {
    case 1: launch_shape<T, 1, kTeams1, BACK, SSOR>(c, d); break;
    case 2: launch_shape<T, 2, kTeams2, BACK, SSOR>(c, d); break;
    default: launch_shape<T, 4, kTeams4, BACK, SSOR>(c, d); break;
    }
}

// [0, n) in ranges on up to four threads (each direction has its own four), the
// last one here; below `grain` a range is not worth a thread.
template<class F> void over_ranges(std::size_t n, std::size_t grain, F f)
{
    const std::size_t parts = std::min<std::size_t>(4, n / grain + 1);
    std::vector<std::future<void>> others;
    for (std::size_t k = 0; k + 1 < parts; ++k)
        others.push_back(std::async([&f, n, parts, k] { f(k, n * k / parts, n * (k + 1) / parts); }));
    f(parts - 1, n * (parts - 1) / parts, n);
    for (auto& o : others) o.get();
}

// Both directions side by side, the lower one on another thread where the rows
// are worth it and one can be had.
constexpr std::size_t kGrain = 4096;
template<class L, class U> bool both(std::size_t owned, L lower, U upper)
{
    if (owned < kGrain) return lower() && upper();
    std::future<bool> first = std::async(lower);
    const bool second = upper();
    return first.get() && second;
}

// Entries that the threads fill: not set to anything before.
template<class T> struct Table {
    std::unique_ptr<T[]> data;
    std::size_t size = 0;
    void allocate(std::size_t n)
    {
        data.reset(new T[n]);
        size = n;
    }
    T& operator[](std::size_t i) { return data[i]; }
};

// A direction's rows in step order, padded: each task starts at a multiple of
// four places.
struct Cut {
    struct Piece {
        std::int32_t first, rows, width;   // rows of one level in the sweep's order; their padded dependencies
        bool ends;                         // the last of its level
    };
    std::vector<Piece> pieces;
    std::vector<std::int32_t> task;    // per step and warp: first entry, first place, rows and width, first ring slot
    std::vector<std::int32_t> rows;    // per place (-1: padding)
    Table<std::int32_t> place;         // per row
    Table<std::int32_t> count;         // dependencies per row
};

// What a task holds: rows, padded entries, and the multiple its places are
// padded to; dense blocks have their slots [dependency][row] and no slower form.
struct Shape {
    int warps, rows, entries, pad;
    bool block;
    int teams;
};

// Steps that a far value must lie back.  The team that takes step s copies its
// task's far values when it is done with step s - kDepth * teams, whose wait put
// it behind all that was done before the signal of the step before; a result
// goes to global memory behind its own step's signal, so before the signal
// that its team gives `teams` steps later.
constexpr int far_reach(int teams) { return (kDepth + 1) * teams + 1; }

// Dependencies of every row: entries [begin, end) with a column below it, or
// for the backward sweep above it.
bool count_dependencies(Cut& cut, std::size_t owned, const std::int32_t* begin, const std::int32_t* end,
                        const std::int32_t* cols, bool backward)
{
    const auto n = static_cast<std::int32_t>(owned);
    cut.count.allocate(owned);
    over_ranges(owned, 8 * kGrain, [&](std::size_t, std::size_t r0, std::size_t r1) {
        for (auto r = static_cast<std::int32_t>(r0); r < static_cast<std::int32_t>(r1); ++r) {
            std::int32_t count = 0;
            for (std::int32_t e = begin[r]; e < end[r]; ++e)
                count += backward ? cols[e] > r && cols[e] < n : cols[e] < r;
            cut.count[r] = count;
        }
    });
    return true;
}

// Rows by level and row number, cut into tasks.  (Within a level by number of
// dependencies, for less padding: the same times.)  False for a row of more
// dependencies than a task's width holds.
bool cut_tasks(Cut& cut, const Sweep& sweep, std::size_t owned, const Shape& shape)
{
    const auto n = static_cast<std::int32_t>(owned);
    const std::vector<std::int32_t>&order = sweep.h_order, &level = sweep.h_level;
    cut.pieces.reserve(owned / static_cast<std::size_t>(shape.rows) + sweep.depth);
    for (std::int32_t b = 0; b < n;) {
        std::int32_t e = b;
        while (e < n && level[order[e]] == level[order[b]]) ++e;
        while (b < e) {
            // As many rows as their padded entries leave room for in a stage.
            std::int32_t rows = 0, width = 0;
            while (rows < shape.rows && b + rows < e) {
                const std::int32_t wider = std::max(width, (cut.count[order[b + rows]] + 1) / 2 * 2);
                if (rows > 0 && (rows + 1) * wider > shape.entries) break;
                width = wider;
                ++rows;
            }
            if (width > 0xff) return false;
            cut.pieces.push_back({b, rows, width, b + rows == e});
            b += rows;
        }
    }
    return true;
}

// The tasks into steps; a level's last step is filled up with tasks of no rows.
void cut_steps(Cut& cut, const Sweep& sweep, std::size_t owned, const Shape& shape)
{
    const std::size_t tasks = cut.pieces.size() + static_cast<std::size_t>(shape.warps - 1) * sweep.depth;
    cut.place.allocate(owned);
    cut.task.reserve(4 * tasks);
    cut.rows.reserve(owned + static_cast<std::size_t>(shape.pad) * tasks + 32);
    std::int32_t at = 0;
    auto add = [&](std::int32_t packed) {
        for (const std::int32_t word : {0, at, packed, 0}) cut.task.push_back(word);
    };
    for (const Cut::Piece& q : cut.pieces) {
        const std::int32_t padded = (q.rows + shape.pad - 1) / shape.pad * shape.pad;
        add(q.rows | q.width << 8);
        const auto first = sweep.h_order.begin() + q.first;
        for (std::int32_t l = 0; l < q.rows; ++l) cut.place[first[l]] = at + l;
        cut.rows.insert(cut.rows.end(), first, first + q.rows);
        cut.rows.insert(cut.rows.end(), static_cast<std::size_t>(padded - q.rows), -1);
        at += padded;
        while (q.ends && cut.task.size() / 4 % shape.warps != 0) add(0);
    }
    cut.rows.resize(cut.rows.size() + 32, -1);   // a task's copies always take 32 places
}

// A direction's tables on the host.
struct Plan {
    std::vector<std::int32_t> far, code;
    Table<std::int32_t> src, to;
    Table<std::uint16_t> slots;
};

// Fills the sizes of s, the tasks of cut and the plan; false where the
// direction does not suit the schedule.  Touches nothing of the other
// direction but its places, and no CUDA call.
bool plan_direction(Plan& plan, LocalSweep& s, std::size_t owned, const Sweep& sweep, Cut& cut, const Cut& other,
                    const std::int32_t* begin, const std::int32_t* end, const std::int32_t* cols, bool backward,
                    const Shape& shape, int shared_rows)
{
    const int warps = shape.warps;
    const auto n = static_cast<std::int32_t>(owned);
    const std::size_t tasks = cut.task.size() / 4;
    const std::int32_t* place = cut.place.data.get();
    s.warps = warps;
    s.places = cut.rows.size();
    s.steps = static_cast<int>(tasks) / warps;
    s.ring = std::min(static_cast<std::int32_t>(s.places), std::min(shared_rows, kFarSlot - 1));
    // A step's results may not overwrite what the same step still reads.
    const std::int32_t reach = static_cast<std::int32_t>(s.places) > s.ring ? s.ring - 32 * warps : s.ring;
    auto needed = [&](std::int32_t row, std::int32_t col) { return backward ? col > row && col < n : col < row; };
    auto far_index = [&](std::int32_t col) { return backward ? col : other.place.data[col]; };
    std::size_t first = 0, used = 0;
    for (std::size_t r = 0; r < owned; ++r) used += static_cast<std::size_t>(cut.count[r]);
    for (std::size_t t = 0; t < tasks; ++t) {
        std::int32_t* w = cut.task.data() + 4 * t;
        w[0] = static_cast<std::int32_t>(first);
        w[3] = w[1] % s.ring;
        first += (static_cast<std::size_t>(w[2] & 0xff) * (w[2] >> 8) + 7) / 8 * 8;
        if (first >= static_cast<std::size_t>(kMaxEntries)) return false;
    }
    s.entries = first;
    // A few rows much longer than the rest would pad their tasks' other rows.
    if (s.entries > 4 * used + 8 * owned + 4096) return false;

    plan.src.allocate(s.entries);
    plan.slots.allocate(s.entries);
    auto step_of = [&](std::int32_t p) {   // of a place: that of the last task starting at or before it
        std::size_t a = 0, b = tasks;
        while (b - a > 1) (cut.task[(a + b) / 2 * 4 + 1] <= p ? a : b) = (a + b) / 2;
        return static_cast<std::int32_t>(a) / warps;
    };
    struct Part {
        std::vector<std::pair<std::size_t, std::int32_t>> far;   // where in plan.far, and what
        std::size_t far_values = 0, slow_tasks = 0;
        int far_steps = INT32_MAX;
    } parts[4];
    over_ranges(tasks, kGrain / 8, [&](std::size_t part, std::size_t t0, std::size_t t1) {
        Part& out = parts[part];
        for (std::size_t t = t0; t < t1; ++t) {
            std::int32_t* w = cut.task.data() + 4 * t;
            const std::int32_t rows = w[2] & 0xff, width = w[2] >> 8;
            std::int32_t* src = plan.src.data.get() + w[0];
            std::uint16_t* slots = plan.slots.data.get() + w[0];
            std::size_t found = 0;
            for (std::int32_t l = 0; l < rows; ++l) {
                const std::int32_t p = w[1] + l, row = cut.rows[p], own = w[3] + l < s.ring ? w[3] + l : w[3] + l - s.ring;
                auto set = [&](std::int32_t j, std::int32_t slot, std::int32_t entry) {
                    slots[shape.block ? j * rows + l : (j & ~1) * rows + 2 * l + j % 2] = static_cast<std::uint16_t>(slot);
                    src[j * rows + l] = entry;
                };
                std::int32_t j = 0;
                for (std::int32_t e = begin[row]; e < end[row]; ++e) {
                    if (!needed(row, cols[e])) continue;
                    const std::int32_t back = p - place[cols[e]];
                    if (back <= reach) {
                        set(j++, back <= own ? own - back : own - back + s.ring, e);
                        continue;
                    }
                    if (found < 32) out.far.emplace_back(t * 32 + found, far_index(cols[e]));
                    set(j++, kFarSlot + static_cast<std::int32_t>(found++ % 32), e);
                    out.far_steps = std::min(out.far_steps, static_cast<std::int32_t>(t) / warps - step_of(p - back));
                }
                for (; j < width; ++j) set(j, s.ring, -1);
            }
            for (std::int32_t i = rows * width; i % 8 != 0; ++i) {
                slots[i] = static_cast<std::uint16_t>(s.ring);
                src[i] = -1;
            }
            const bool slow = width > kHold || found > 32;
            w[2] |= slow ? kSlowFlag : found > 0 ? kFarFlag : 0;
            out.far_values += found;
            out.slow_tasks += slow;
        }
    });
    std::size_t far_values = 0, slow_tasks = 0;
    s.far_steps = INT32_MAX;
    for (const Part& part : parts) {
        far_values += part.far_values;
        slow_tasks += part.slow_tasks;
        s.far_steps = std::min(s.far_steps, part.far_steps);
    }
    s.far_values = static_cast<int>(far_values);
    s.slow_tasks = static_cast<int>(slow_tasks);
    if (slow_tasks > 0 && shape.block) return false;
    // A copy could pass the result that it is to bring.  (With the rings that
    // shared memory holds the closest lie 67 steps back against 28, FP64 blocks
    // of 3; a ring of few rows, or more tasks in flight, end here.)
    if (s.far_steps < far_reach(shape.teams)) return false;
    // A task of the slower form costs its step about a microsecond, more than
    // a level of the level-scheduled sweep.
    if (slow_tasks > static_cast<std::size_t>(sweep.depth) / 4) return false;
    if (far_values > 0) plan.far.assign(tasks * 32, -1);
    for (const Part& part : parts)
        for (const auto& [at, value] : part.far) plan.far[at] = value;
    if (slow_tasks > 0) {
        // Every task's dependencies as the slower form reads them.
        plan.code.assign(s.entries, s.ring);
        for (std::size_t t = 0; t < tasks; ++t) {
            const std::int32_t* w = cut.task.data() + 4 * t;
            const std::int32_t rows = w[2] & 0xff;
            for (std::int32_t l = 0; l < rows; ++l) {
                const std::int32_t p = w[1] + l;
                for (std::int32_t k = w[0] + l; k < w[0] + rows * (w[2] >> 8 & 0xff); k += rows) {
                    if (plan.src[k] < 0) break;
                    const std::int32_t col = cols[plan.src[k]], from = place[col];
                    plan.code[k] = p - from <= reach ? from % s.ring : -1 - far_index(col);
                }
            }
        }
    }
    if (!backward) {
        plan.to.allocate(s.places);
        over_ranges(s.places, 16 * kGrain, [&](std::size_t, std::size_t p0, std::size_t p1) {
            for (std::size_t p = p0; p < p1; ++p) plan.to[p] = cut.rows[p] >= 0 ? other.place.data[cut.rows[p]] : 0;
        });
    }
    return true;
}

// What both directions of a component-diagonal sweep need, on the host.
struct Planned {
    Cut lower, upper;
    Plan lower_plan, upper_plan;
};

constexpr int teams_of(int warps) { return warps == 1 ? kTeams1 : warps == 2 ? kTeams2 : kTeams4; }
Shape component_shape(int warps) { return Shape{warps, 32, kTaskEntries, 4, false, teams_of(warps)}; }

// Warps per team of the cheapest shape, or 0 when the level-scheduled sweep is
// cheaper.  A shape costs the steps that it cuts the levels into, at their
// measured times on meshes (an ILU step of one, two and four tasks 75, 95 and
// 145 ns, an SSOR step, which divides, 95, 130 and 172 ns), 35 ns more for a
// step of tasks wider than six dependencies (which also hold 24 rows, not 32,
// so there are more of them), and in SSOR the copy of the values that precedes
// every apply, 4 ps a value beyond what the other sweep reads.  Against it stand
// 800 ns a level for ILU (0.71 to 0.86 us measured at 250 to 1,400 rows a level)
// and 870 ns for SSOR, once for every eight entries of a row, which that sweep
// reads in rounds of eight.  FP32 SSOR takes three quarters of these step times,
// and the figures for its copies and levels are in the same scale (6 ps; a level
// 575 ns with 3 entries a row, 710 to 760 with 7).  Levels of equal width,
// this / level-scheduled, ns a level on the two sides of the line:
//   ILU, 3 dependencies a row: 640 rows 636 / 774, 700 rows 789 / 788; 7 of
//   them: 384 rows 718 / 794, 512 rows 991 / 819;
//   SSOR, 3 of them, bs 1: 640 rows 858 / 890, 700 rows 6 steps / 891; bs 64:
//   128 rows 433 / 1,013, 512 rows 1,579 / 1,324; FP32, bs 1: 640 rows
//   667 / 696, 700 rows 6 steps / 721.
// FP32 and stored ILU factors cross where FP64 ones do, both sides a tenth to a
// fifth cheaper.
constexpr struct { int warps; double ilu, ssor; } kShapes[] = {{1, 75, 95}, {2, 95, 130}, {4, 145, 172}};

// What the level-scheduled sweep takes for a level, ns, by entries per row.
double level_ns(double per_row, std::size_t element_size, bool ssor)
{
    if (!ssor) return 800;
    return std::ceil(per_row / 8) * (element_size == 8 ? 870 : std::min(940.0, 618 + 45 * per_row));
}

int local_sweep_warps(const Cut& lower_cut, const Cut& upper_cut, const Sweep& lower, const Sweep& upper,
                      std::size_t owned, std::size_t bs, std::size_t element_size, int sm_count, bool ssor)
{
    constexpr double kWide = 35;
    if (bs > static_cast<std::size_t>(sm_count)) return 0;
    double cost[3] = {0, 0, 0}, entries = 0;
    for (const Cut* cut : {&lower_cut, &upper_cut}) {
        for (std::size_t r = 0; r < owned; ++r) entries += cut->count.data[r];
        std::int32_t tasks = 0, wide = 0;
        for (const Cut::Piece& q : cut->pieces) {
            ++tasks;
            wide += q.width > 6;
            if (!q.ends) continue;
            for (int k = 0; k < 3; ++k)
                cost[k] += (tasks + kShapes[k].warps - 1) / kShapes[k].warps
                    * ((ssor ? kShapes[k].ssor : kShapes[k].ilu) + kWide * wide / tasks);
            tasks = wide = 0;
        }
    }
    const double copy = ssor ? (element_size == 8 ? 0.004 : 0.006) * entries * static_cast<double>(bs) : 0;
    const double per_row = entries / static_cast<double>(owned) + 1;
    double least = level_ns(per_row, element_size, ssor) * (lower.depth + upper.depth) - copy;
    int best = 0;
    for (int k = 0; k < 3; ++k)
        if (cost[k] < least) {
            least = cost[k];
            best = kShapes[k].warps;
        }
    return best;
}

// False where the level-scheduled sweep is cheaper, or a direction does not suit
// the schedule.  ring_rows: 0 for as many as shared memory holds.
bool plan_local(Planned& x, LocalSweep& lo, LocalSweep& up, const Sweep& lower, const Sweep& upper, std::size_t owned,
                std::size_t bs, std::size_t element_size, int sm_count, int ring_rows, const std::int32_t* lower_begin,
                const std::int32_t* lower_end, const std::int32_t* upper_begin, const std::int32_t* upper_end,
                const std::int32_t* cols, bool ssor)
{
    if (owned == 0) return false;
    // Wide levels are told without cutting them: no cut is cheaper than full
    // steps of four tasks, no row longer than all its entries.
    const double rows = static_cast<double>(owned), full = 2 * rows / 128 * (ssor ? kShapes[2].ssor : kShapes[2].ilu);
    if (full >= level_ns((lower_end[owned - 1] - lower_begin[0]) / rows, element_size, ssor) * (lower.depth + upper.depth))
        return false;
    if (!both(owned, [&] { return count_dependencies(x.lower, owned, lower_begin, lower_end, cols, false)
                                && cut_tasks(x.lower, lower, owned, component_shape(1)); },
              [&] { return count_dependencies(x.upper, owned, upper_begin, upper_end, cols, true)
                        && cut_tasks(x.upper, upper, owned, component_shape(1)); })) return false;
    const int warps = local_sweep_warps(x.lower, x.upper, lower, upper, owned, bs, element_size, sm_count, ssor);
    if (warps == 0) return false;
    const Shape shape = component_shape(warps);
    if (ring_rows == 0) {
        const std::size_t stage = element_size == 8 ? sizeof(Stage<double>) : sizeof(Stage<float>);
        const std::size_t stages = static_cast<std::size_t>(warps * shape.teams * kDepth) * stage;
        ring_rows = static_cast<int>((kSharedBytes - stages) / element_size) - 2;
    }
    both(owned, [&] { return cut_steps(x.lower, lower, owned, shape), true; },
         [&] { return cut_steps(x.upper, upper, owned, shape), true; });
    return both(owned,
                [&] { return plan_direction(x.lower_plan, lo, owned, lower, x.lower, x.upper, lower_begin, lower_end,
                                            cols, false, shape, ring_rows); },
                [&] { return plan_direction(x.upper_plan, up, owned, upper, x.upper, x.lower, upper_begin, upper_end,
                                            cols, true, shape, ring_rows); });
}

// The plan on the device, in one allocation (with one for each of the twenty
// parts of both directions this took 4.2 of the 7 ms that the tables of 90,000
// rows take on the host).
// vector_size, value_size: bytes of a vector element and of a stored value.
void place_direction(Context& ctx, LocalSweep& s, const Plan& plan, const Cut& cut, std::size_t bs,
                     std::size_t vector_size, std::size_t value_size, bool with_fin, const Shape& shape)
{
    // Values of an entry, and of a row's diagonal.
    const std::size_t per = !shape.block ? bs : value_size == 2 ? (bs * bs + 1) / 2 * 2 : bs * bs;
    std::size_t total = 0;
    auto room = [&](std::size_t bytes) {   // a part's offset; a copy may read 16 bytes past its end
        const std::size_t at = total;
        total += (bytes + 16 + 255) / 256 * 256;
        return at;
    };
    struct Copy {
        DevicePart& part;
        const void* from;
        std::size_t bytes, at;
    };
    std::vector<Copy> copies;
    auto copied = [&](DevicePart& part, const void* from, std::size_t bytes) {
        if (bytes > 0) copies.push_back({part, from, bytes, room(bytes)});
    };
    copied(s.task, cut.task.data(), cut.task.size() * 4);
    copied(s.slots, plan.slots.data.get(), plan.slots.size * 2);
    copied(s.far, plan.far.data(), plan.far.size() * 4);
    copied(s.code, plan.code.data(), plan.code.size() * 4);
    copied(s.src, plan.src.data.get(), plan.src.size * 4);
    copied(s.rows, cut.rows.data(), cut.rows.size() * 4);
    copied(s.to, plan.to.data.get(), plan.to.size * 4);
    const std::size_t zeroed = total, coef = room(per * s.entries * value_size),   // padding: zero
                      fin = with_fin ? room(per * s.places * value_size) : 0,
                      in = room(bs * s.places * vector_size);
    s.store.allocate(total);
    char* base = s.store.as<char>();
    for (const Copy& c : copies) {
        c.part.ptr = base + c.at;
        OWTK_CUDA(cudaMemcpyAsync(c.part.ptr, c.from, c.bytes, cudaMemcpyHostToDevice, ctx.stream));
    }
    s.coef.ptr = base + coef;
    if (with_fin) s.fin.ptr = base + fin;
    s.in.ptr = base + in;
    OWTK_CUDA(cudaMemsetAsync(base + zeroed, 0, total - zeroed, ctx.stream));
    s.ready = true;
}

}  // namespace

// Dependencies of row r: entries [lower_begin[r], lower_end[r]) with a column
// below r, and [upper_begin[r], upper_end[r]) with one above it.
void build_local_sweep(Context& ctx, Preconditioner& p, std::size_t element_size, const std::int32_t* lower_begin,
                       const std::int32_t* lower_end, const std::int32_t* upper_begin, const std::int32_t* upper_end,
                       const std::int32_t* cols, bool ssor)
{
    const char* env = std::getenv("OWTK_LOCAL_SWEEP");   // 0: never
    if (env && std::atoi(env) == 0) return;
    Planned x;
    if (!plan_local(x, p.lower_local, p.upper_local, p.lower, p.upper, p.owned, p.bs, element_size, ctx.sm_count, 0,
                    lower_begin, lower_end, upper_begin, upper_end, cols, ssor)) {
        p.lower_local = LocalSweep();
        p.upper_local = LocalSweep();
        return;
    }
    const Shape shape = component_shape(p.lower_local.warps);
    place_direction(ctx, p.lower_local, x.lower_plan, x.lower, p.bs, element_size, element_size, ssor, shape);
    place_direction(ctx, p.upper_local, x.upper_plan, x.upper, p.bs, element_size, element_size, true, shape);
}

owtk_local_schedule local_schedule(const LocalSweep& lower, const LocalSweep& upper)
{
    owtk_local_schedule s{};
    s.warps = lower.warps;
    s.lower_steps = lower.steps;
    s.upper_steps = upper.steps;
    s.ring_rows = std::min(lower.ring, upper.ring);
    s.far_values = lower.far_values + upper.far_values;
    s.slow_tasks = lower.slow_tasks + upper.slow_tasks;
    s.far_steps = std::min(lower.far_steps, upper.far_steps);
    return s;
}

// No CUDA call.
owtk_local_schedule plan_local_schedule(std::size_t owned, std::size_t bs, const std::int32_t* rowptr,
                                        const std::int32_t* cols, std::size_t element_size, int sm_count, int ring_rows,
                                        bool ssor)
{
    std::vector<std::int32_t> lower_level, upper_level;
    levels_of(owned, rowptr, cols, lower_level, upper_level);
    Sweep lower, upper;
    order_by_level(lower, owned, bs, lower_level);
    order_by_level(upper, owned, bs, upper_level);
    LocalSweep lo, up;
    Planned x;
    if (!plan_local(x, lo, up, lower, upper, owned, bs, element_size, sm_count, ring_rows, rowptr, rowptr + 1, rowptr,
                    rowptr + 1, cols, ssor)) return {};
    return local_schedule(lo, up);
}

namespace {

template<class T, class F, int BS, bool BACK>
void launch_block_shape(Context& c, const BlockArgs<T, F>& d)
{
    constexpr int kTeams = block_teams(sizeof(BlockStage<T, F, BS>));
    auto* kernel = k_local_block<T, F, BS, 1, kTeams, BACK>;
    const int bytes = kTeams * kDepth * static_cast<int>(sizeof(BlockStage<T, F, BS>))
        + (d.ring + 1) * (BS == 3 ? 4 : BS) * static_cast<int>(sizeof(T));
    OWTK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedBytes));
    kernel<<<1, kTeams * 32, bytes, c.stream>>>(d);
    OWTK_CUDA(cudaGetLastError());
    c.launched();
}

template<class T, class F, bool BACK>
void launch_block(Context& c, Preconditioner& p, T* out)
{
    const LocalSweep& s = BACK ? p.upper_local : p.lower_local;
    BlockArgs<T, F> d{};
    d.task = s.task.as<int4>();
    d.slots = s.slots.as<std::uint16_t>();
    d.far = s.far.ptr ? s.far.as<int>() : nullptr;
    d.to = BACK ? s.rows.as<int>() : s.to.as<int>();
    d.coef = s.coef.as<F>();
    d.dinv = s.fin.as<F>();
    d.in = s.in.as<T>();
    d.out = BACK ? out : p.upper_local.in.as<T>();
    d.steps = s.steps;
    d.ring = s.ring;
    switch (p.bs) {
    case 1: launch_block_shape<T, F, 1, BACK>(c, d); break;
    case 2: launch_block_shape<T, F, 2, BACK>(c, d); break;
    case 3: launch_block_shape<T, F, 3, BACK>(c, d); break;
    default: launch_block_shape<T, F, 4, BACK>(c, d); break;
    }
}

template<class F, bool DIAG>
void pack_blocks(Context& c, const LocalSweep& s, std::size_t bs, const DevicePart& src, const F* from,
                 const DevicePart& to)
{
    const std::size_t tasks = static_cast<std::size_t>(s.steps) * s.warps;
    k_local_block_pack<F, DIAG><<<static_cast<unsigned>((tasks * 32 + kThreads - 1) / kThreads), kThreads, 0, c.stream>>>(
        tasks, static_cast<int>(bs), s.task.as<int4>(), src.as<int>(), from, to.as<F>());
    OWTK_CUDA(cudaGetLastError());
    c.launched();
}

template<class T, class F> std::size_t block_stage_bytes(std::size_t bs)
{
    return bs == 1 ? sizeof(BlockStage<T, F, 1>) : bs == 2 ? sizeof(BlockStage<T, F, 2>)
        : bs == 3 ? sizeof(BlockStage<T, F, 3>) : sizeof(BlockStage<T, F, 4>);
}

}  // namespace

// The dense-block ILU's schedule where it pays: its tasks at their cost (BF16,
// FP32 and FP64 factors, by block size; fitted at 82 rows a level, a step being
// one task) against what a level costs through L2 (1.1 us for FP32 vectors,
// 1.4 us for FP64).  At 1 to 320 rows a level of 1, 3 and 7 dependencies a row
// nothing taken is slower than the level-scheduled sweep (ns a level, this /
// that, BF16 bs 3: 32 rows 185 / 1,084, 192 rows 875 / 1,164; FP64 bs 3: 32 rows
// 396 / 1,381; FP64 bs 4: 32 rows 641 / 1,335).
constexpr double kBlockTaskNs[3][4] = {{105, 110, 160, 210}, {105, 110, 140, 310}, {105, 140, 390, 700}};
void build_local_block_sweep(Context& ctx, Preconditioner& p, owtk_dtype storage)
{
    const char* env = std::getenv("OWTK_LOCAL_SWEEP");   // 0: never
    if (env && std::atoi(env) == 0) return;
    const std::size_t n = p.owned, bs = p.bs, vector = storage == OWTK_F64 ? 8 : 4,
                      value = storage == OWTK_F64 ? 8 : storage == OWTK_F32 ? 4 : 2;
    const std::size_t stage = storage == OWTK_F64 ? block_stage_bytes<double, double>(bs)
        : storage == OWTK_F32 ? block_stage_bytes<float, float>(bs) : block_stage_bytes<float, __nv_bfloat16>(bs);
    const Shape shape{1, 32, block_entries(value * bs * bs), 8, true, block_teams(stage)};
    const std::size_t stages = shape.teams * kDepth * stage, row = (bs == 3 ? 4 : bs) * vector;
    if (n == 0 || stages + 1024 * row > kSharedBytes) return;
    const int shared_rows = static_cast<int>((kSharedBytes - stages) / row) - 2;
    const std::int32_t *rp = p.f_rowptr.data(), *dp = p.f_diagpos.data(), *ci = p.f_cols.data();
    std::vector<std::int32_t> after(n);   // first upper entry of each row
    for (std::size_t r = 0; r < n; ++r) after[r] = dp[r] + 1;
    Cut lower, upper;
    if (!both(n, [&] { return count_dependencies(lower, n, rp, dp, ci, false) && cut_tasks(lower, p.lower, n, shape); },
              [&] { return count_dependencies(upper, n, after.data(), rp + 1, ci, true)
                        && cut_tasks(upper, p.upper, n, shape); })) return;
    const std::size_t tasks = lower.pieces.size() + upper.pieces.size();
    const double task_ns = kBlockTaskNs[storage == OWTK_F64 ? 2 : storage == OWTK_F32 ? 1 : 0][bs - 1];
    const double level_ns = storage == OWTK_F64 ? 1400.0 : 1100.0;
    if (static_cast<double>(tasks) * task_ns > level_ns * (p.lower.depth + p.upper.depth)) return;
    both(n, [&] { return cut_steps(lower, p.lower, n, shape), true; },
         [&] { return cut_steps(upper, p.upper, n, shape), true; });
    Plan lower_plan, upper_plan;
    if (!both(n, [&] { return plan_direction(lower_plan, p.lower_local, n, p.lower, lower, upper, rp, dp, ci, false, shape,
                                          shared_rows); },
              [&] { return plan_direction(upper_plan, p.upper_local, n, p.upper, upper, lower, after.data(), rp + 1,
                                          ci, true, shape, shared_rows); })) {
        p.lower_local = LocalSweep();
        p.upper_local = LocalSweep();
        return;
    }
    place_direction(ctx, p.lower_local, lower_plan, lower, bs, vector, value, false, shape);
    place_direction(ctx, p.upper_local, upper_plan, upper, bs, vector, value, true, shape);
}

namespace kern {

template<class F> void local_block_pack(Context& c, Preconditioner& p, const F* factors, const F* inverse)
{
    pack_blocks<F, false>(c, p.lower_local, p.bs, p.lower_local.src, factors, p.lower_local.coef);
    pack_blocks<F, false>(c, p.upper_local, p.bs, p.upper_local.src, factors, p.upper_local.coef);
    pack_blocks<F, true>(c, p.upper_local, p.bs, p.upper_local.rows, inverse, p.upper_local.fin);
}

template<class T, class F> void local_block_apply(Context& c, Preconditioner& p, const T* in, T* out)
{
    const std::size_t count = p.lower_local.places;
    k_local_block_gather<T><<<static_cast<unsigned>((count * p.bs + kThreads - 1) / kThreads), kThreads, 0, c.stream>>>(
        count, static_cast<int>(p.bs), p.lower_local.rows.as<int>(), in, p.lower_local.in.as<T>());
    OWTK_CUDA(cudaGetLastError());
    c.launched();
    launch_block<T, F, false>(c, p, out);
    launch_block<T, F, true>(c, p, out);
}

template void local_block_pack<double>(Context&, Preconditioner&, const double*, const double*);
template void local_block_pack<float>(Context&, Preconditioner&, const float*, const float*);
template void local_block_pack<__nv_bfloat16>(Context&, Preconditioner&, const __nv_bfloat16*, const __nv_bfloat16*);
template void local_block_apply<double, double>(Context&, Preconditioner&, const double*, double*);
template void local_block_apply<float, float>(Context&, Preconditioner&, const float*, float*);
template void local_block_apply<float, __nv_bfloat16>(Context&, Preconditioner&, const float*, float*);

template<class T, class F>
void local_ilu_pack(Context& c, Preconditioner& p, const F* factors, const F* inverse)
{
    pack<T, F>(c, p, factors, inverse, nullptr, T(1), false);
}

template<class T> void local_ilu_apply(Context& c, Preconditioner& p, const T* in, T* out)
{
    pack<T, T>(c, p, nullptr, nullptr, in, T(1), false);
    launch<T, false, false>(c, p, out);
    launch<T, true, false>(c, p, out);
}

// The matrix's values are read at every apply, as the level-scheduled sweep
// reads them: they may have been written since the last one.
template<class T>
void local_ssor_apply(Context& c, Preconditioner& p, const T* values, const T* diag, const T* in, T* out)
{
    pack<T, T>(c, p, values, diag, in, static_cast<T>(p.parameter), true);
    launch<T, false, true>(c, p, out);
    launch<T, true, true>(c, p, out);
}

template void local_ilu_pack<double, double>(Context&, Preconditioner&, const double*, const double*);
template void local_ilu_pack<float, float>(Context&, Preconditioner&, const float*, const float*);
template void local_ilu_pack<float, __nv_bfloat16>(Context&, Preconditioner&, const __nv_bfloat16*,
                                                   const __nv_bfloat16*);
template void local_ilu_apply<double>(Context&, Preconditioner&, const double*, double*);
template void local_ilu_apply<float>(Context&, Preconditioner&, const float*, float*);
template void local_ssor_apply<double>(Context&, Preconditioner&, const double*, const double*, const double*,
                                       double*);
template void local_ssor_apply<float>(Context&, Preconditioner&, const float*, const float*, const float*, float*);

}  // namespace kern
}  // namespace owtk
