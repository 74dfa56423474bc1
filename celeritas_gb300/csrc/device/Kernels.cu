// CUDA kernels of the GB300 stepping loop.
//
// Each action kernel runs one thread per track slot and calls the same
// per-slot function as the reference's action executor (see gbx/Actions.hh
// and gbx/TrackInit.hh). Counters stay on the device: the number of new
// tracks, vacancies, secondaries and initializers are read and updated by
// kernels, so a whole step is a fixed sequence of launches that a CUDA graph
// can capture (the reference copies counters to the host several times per
// step, src/celeritas/track/detail/TrackInitAlgorithms.cu:34-78).
//
// End-of-step bookkeeping (src/celeritas/track/ExtendFromSecondariesAction.cc)
// is three kernels: per-slot flags with per-block totals, one block scanning
// the block totals and updating the counters, and a scatter that writes the
// stably compacted vacancy list and processes each slot's secondaries at its
// exclusive-scan offset.
#include "Kernels.cuh"

#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>

#include "../gbx/TrackInit.hh"

namespace gbx
{
namespace
{
__device__ __forceinline__ size_type thread_slot()
{
    return blockIdx.x * blockDim.x + threadIdx.x;
}

inline unsigned int num_blocks_for(size_type n)
{
    return static_cast<unsigned int>((n + block_size - 1) / block_size);
}

//---------------------------------------------------------------------------//
// Block-wide exclusive scan of one 32-bit value per thread (256 threads)
//---------------------------------------------------------------------------//
struct BlockScanStorage
{
    size_type warp_sums[block_size / 32];
    size_type total;
};

__device__ __forceinline__ size_type block_exclusive_scan(size_type value,
                                                          BlockScanStorage& tmp,
                                                          size_type* total)
{
    int const lane = threadIdx.x & 31;
    int const warp = threadIdx.x >> 5;
    // Inclusive warp scan
    size_type incl = value;
#pragma unroll
    for (int offset = 1; offset < 32; offset <<= 1)
    {
        size_type n = __shfl_up_sync(0xffffffffu, incl, offset);
        if (lane >= offset)
            incl += n;
    }
    if (lane == 31)
        tmp.warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        constexpr int nwarps = block_size / 32;
        size_type w = (lane < nwarps) ? tmp.warp_sums[lane] : 0;
        size_type wincl = w;
#pragma unroll
        for (int offset = 1; offset < nwarps; offset <<= 1)
        {
            size_type n = __shfl_up_sync(0xffffffffu, wincl, offset);
            if (lane >= offset)
                wincl += n;
        }
        if (lane < nwarps)
            tmp.warp_sums[lane] = wincl - w;  // exclusive warp offsets
        if (lane == nwarps - 1)
            tmp.total = wincl;
    }
    __syncthreads();
    size_type result = tmp.warp_sums[warp] + incl - value;
    *total = tmp.total;
    __syncthreads();
    return result;
}

//! Exclusive scan of one value per thread of a 1024-thread block: two warp
//! shuffle scans and three barriers
struct WideScanStorage
{
    size_type warp_sums[32];
    size_type total;
};

__device__ __forceinline__ size_type wide_exclusive_scan(size_type value, WideScanStorage& tmp)
{
    unsigned int const lane = threadIdx.x & 31u;
    unsigned int const warp = threadIdx.x >> 5;
    auto warp_inclusive = [lane](size_type v) {
#pragma unroll
        for (unsigned int offset = 1; offset < 32; offset <<= 1)
        {
            size_type const n = __shfl_up_sync(0xffffffffu, v, offset);
            if (lane >= offset)
                v += n;
        }
        return v;
    };
    size_type const incl = warp_inclusive(value);
    if (lane == 31)
        tmp.warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0)
    {
        size_type const w = tmp.warp_sums[lane];
        size_type const wincl = warp_inclusive(w);
        tmp.warp_sums[lane] = wincl - w;
        if (lane == 31)
            tmp.total = wincl;
    }
    __syncthreads();
    size_type const result = tmp.warp_sums[warp] + incl - value;
    __syncthreads();
    return result;
}

//! Exclusive scan in place of n values by one 1024-thread block, starting from
//! 'first'; returns the sum of all. Each thread takes a run of consecutive
//! values and the runs' sums are scanned once, where a pass of 1024 values at a
//! time would need its barriers for each.
__device__ __forceinline__ size_type scan_in_place(size_type* values,
                                                   size_type n,
                                                   size_type first,
                                                   WideScanStorage& tmp)
{
    size_type const per = (n + 1023) / 1024;
    size_type const begin = min_of(n, threadIdx.x * per);
    size_type const end = min_of(n, begin + per);
    size_type sum = 0;
    for (size_type i = begin; i < end; ++i)
        sum += values[i];
    size_type run = first + wide_exclusive_scan(sum, tmp);
    for (size_type i = begin; i < end; ++i)
    {
        size_type const v = values[i];
        values[i] = run;
        run += v;
    }
    return first + tmp.total;
}

//! First statement of every kernel that launch() starts: wait until the stream's
//! previous kernel is over and its writes are visible
__device__ __forceinline__ void begin_dependent()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

//---------------------------------------------------------------------------//
// Primaries and track initialization
//---------------------------------------------------------------------------//
__global__ void begin_primaries_kernel(StateData s, size_type num_primaries)
{
    Counters& c = *s.counters;
    if (num_primaries > s.initializer_capacity - c.num_initializers)
    {
        // The queue would overflow: drop the primaries, keep every queued
        // initializer valid, and let the host report the overflow
        c.error_flags |= error_initializer_overflow;
        c.num_generated = 0;
        c.num_pending_primaries = 0;
        return;
    }
    c.num_initializers += num_primaries;
    c.num_generated = num_primaries;
    c.num_pending_primaries = num_primaries;
}

__global__ void process_primaries_kernel(StateData s, size_type num_primaries)
{
    size_type tid = thread_slot();
    Counters const& c = *s.counters;
    if (tid < num_primaries && !(c.error_flags & error_initializer_overflow))
    {
        process_primary(s, c.num_initializers, num_primaries, tid);
    }
    // Primaries have no parents: clear the parent list
    for (size_type i = tid; i < s.size; i += gridDim.x * blockDim.x)
    {
        s.parents[i] = invalid_id;
    }
}

__global__ __launch_bounds__(block_size) void generate_primaries_kernel(
    PrimaryGeneratorData g, StateData s, size_type num)
{
    size_type const tid = thread_slot();
    if (tid < num)
        generate_primary(g, s.primaries, tid);
}

//! Counter update after the step's new tracks are initialized
__device__ __forceinline__ void finish_initialize(StateData const& s, StepLogRef const& log)
{
    Counters& c = *s.counters;
    size_type const num_new = min_of(c.num_vacancies, c.num_initializers);
    c.num_initializers -= num_new;
    c.num_vacancies -= num_new;
    c.num_taken_front = 0;
    c.num_taken_back = 0;
    c.num_active = s.size - c.num_vacancies;
    // pre-step clears the secondary stack
    c.secondary_stack_size = 0;
    StepRecord& r = log.records[*log.step_index % log.capacity];
    r.generated = c.num_generated;
    r.active = c.num_active;
    c.num_generated = 0;
}

//! Whether this block is the last of its grid to get here, for every thread of
//! the block; what the other blocks wrote before is then visible (through L2)
//! to its first thread, and after the barrier to all. The ticket is zero again
//! afterwards. No block waits for another.
__device__ __forceinline__ bool last_block(size_type* ticket)
{
    __shared__ bool last;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last = atomicAdd(ticket, size_type(1)) == gridDim.x - 1;
        if (last)
        {
            *ticket = 0;
            __threadfence();
        }
    }
    __syncthreads();
    return last;
}

__global__ __launch_bounds__(block_size) void initialize_tracks_kernel(
    ParamsData p, StateData s, StepLogRef log, size_type* ticket)
{
    begin_dependent();
    // Grid-stride over the new tracks, whose number is on the device
    Counters const c = *s.counters;
    size_type const num_new = min_of(c.num_vacancies, c.num_initializers);
    size_type const stride = gridDim.x * blockDim.x;
    for (size_type tid = thread_slot(); tid < num_new; tid += stride)
    {
        init_track(p, s, c, tid);
    }
    // Every block has read the counters when the last one gets here
    if (last_block(ticket) && threadIdx.x == 0)
        finish_initialize(s, log);
}

//! Track initialization with partitioned slots: the same initializers as
//! initialize_tracks_kernel, but a charged track takes the next vacancy from
//! the front of the (ascending) list and a neutral one the next from the
//! back. The front and back runs together cover num_new distinct vacancies;
//! the vacancies left between them are not read again before the end of the
//! step rebuilds the list. Which slot a track gets depends on the order in
//! which warps claim them, which is why this needs per-track random streams.
__global__ __launch_bounds__(block_size) void initialize_tracks_partitioned_kernel(
    ParamsData p, StateData s)
{
    begin_dependent();
    size_type tid = thread_slot();
    Counters const c = *s.counters;
    size_type num_new = min_of(c.num_vacancies, c.num_initializers);
    if (blockIdx.x * blockDim.x >= num_new)
        return;
    bool const valid = tid < num_new;
    bool charged = false;
    if (valid)
    {
        TrackInitializer const& init = s.initializers[c.num_initializers - tid - 1];
        charged = p.particles[init.particle_id].charge != 0;
    }
    // One atomic per warp and side: ranks within the warp by ballot
    unsigned int const lane = threadIdx.x & 31u;
    unsigned int const lt = (1u << lane) - 1u;
    unsigned int const front = __ballot_sync(0xffffffffu, valid && charged);
    unsigned int const back = __ballot_sync(0xffffffffu, valid && !charged);
    size_type front_base = 0;
    size_type back_base = 0;
    if (lane == 0)
    {
        if (front)
            front_base = atomicAdd(&s.counters->num_taken_front, __popc(front));
        if (back)
            back_base = atomicAdd(&s.counters->num_taken_back, __popc(back));
    }
    front_base = __shfl_sync(0xffffffffu, front_base, 0);
    back_base = __shfl_sync(0xffffffffu, back_base, 0);
    if (!valid)
        return;
    size_type const slot
        = charged ? s.vacancies[front_base + __popc(front & lt)]
                  : s.vacancies[c.num_vacancies - 1 - back_base - __popc(back & lt)];
    init_track_at(p, s, c, tid, slot);
}

//---------------------------------------------------------------------------//
// Charge partition of new tracks (TrackOrder init_charge): a stable
// partition of the last num_new initializers, neutral ones first
// (partition_initializers, src/celeritas/track/detail/
// TrackInitAlgorithms.cc:75-95), as a per-block count, a scan of the block
// counts and a scatter that ranks each initializer within its group. The
// end-of-step scan scratch is free at the start of the step: block_vacant
// holds the neutral count of each block, block_count[0] the total.
//---------------------------------------------------------------------------//
__device__ __forceinline__ bool new_track_is_neutral(ParamsData const& p,
                                                     StateData const& s,
                                                     Counters const& c,
                                                     size_type num_new,
                                                     size_type i)
{
    return i < num_new
           && is_neutral(p, s.initializers[c.num_initializers - num_new + i]);
}

__global__ __launch_bounds__(block_size) void charge_partition_count_kernel(
    ParamsData p, StateData s, ScanScratch scr)
{
    begin_dependent();
    Counters const c = *s.counters;
    size_type const num_new = min_of(c.num_vacancies, c.num_initializers);
    bool const neutral = new_track_is_neutral(p, s, c, num_new, thread_slot());
    int const n = __syncthreads_count(neutral);
    if (threadIdx.x == 0)
        scr.block_vacant[blockIdx.x] = static_cast<size_type>(n);
}

__global__ __launch_bounds__(1024) void charge_partition_scan_kernel(ScanScratch scr,
                                                                     size_type num_blocks)
{
    begin_dependent();
    // Exclusive scan of the per-block neutral counts by one block
    __shared__ WideScanStorage tmp;
    size_type const total = scan_in_place(scr.block_vacant, num_blocks, 0, tmp);
    if (threadIdx.x == 0)
        scr.block_count[0] = total;
}

__global__ __launch_bounds__(block_size) void charge_partition_scatter_kernel(
    ParamsData p, StateData s, ScanScratch scr)
{
    begin_dependent();
    __shared__ size_type warp_neutral[block_size / 32];
    Counters const c = *s.counters;
    size_type const num_new = min_of(c.num_vacancies, c.num_initializers);
    size_type const i = thread_slot();
    bool const neutral = new_track_is_neutral(p, s, c, num_new, i);
    unsigned int const lane = threadIdx.x & 31u;
    unsigned int const warp = threadIdx.x >> 5;
    unsigned int const ballot = __ballot_sync(0xffffffffu, neutral);
    if (lane == 0)
        warp_neutral[warp] = __popc(ballot);
    __syncthreads();
    size_type before = scr.block_vacant[blockIdx.x] + __popc(ballot & ((1u << lane) - 1u));
    for (unsigned int w = 0; w < warp; ++w)
        before += warp_neutral[w];
    if (i < num_new)
    {
        size_type const pos = neutral ? before : scr.block_count[0] + (i - before);
        s.init_indices[pos] = i;
    }
}

__global__ __launch_bounds__(block_size) void initialize_tracks_charge_kernel(
    ParamsData p, StateData s)
{
    begin_dependent();
    Counters const c = *s.counters;
    size_type const num_new = min_of(c.num_vacancies, c.num_initializers);
    size_type const stride = gridDim.x * blockDim.x;
    for (size_type tid = thread_slot(); tid < num_new; tid += stride)
        init_track_charge_partitioned(p, s, c, num_new, tid);
}

//! Clear stale parent slots after the charge-partitioned initialization
__global__ __launch_bounds__(block_size) void clear_parents_kernel(StateData s)
{
    begin_dependent();
    size_type const stride = gridDim.x * blockDim.x;
    for (size_type i = thread_slot(); i < s.size; i += stride)
        s.parents[i] = invalid_id;
}

__global__ void finish_initialize_kernel(StateData s, StepLogRef log)
{
    begin_dependent();
    finish_initialize(s, log);
}

//---------------------------------------------------------------------------//
// Physics actions
//---------------------------------------------------------------------------//
//! An idle slot is written only when that changes it: what pre-step would give
//! it, it has from its first idle step on. (The 17 to 21 bytes written for each idle
//! slot took most of this launch's 20.5 us over 2^21 slots with a few tracks.)
__global__ __launch_bounds__(block_size) void pre_step_kernel(ParamsData p, StateData s)
{
    begin_dependent();
    size_type slot = thread_slot();
    if (slot < s.size)
    {
        if (s.status[slot] == status_inactive && s.post_step_action[slot] == invalid_id
            && s.along_step_action[slot] == invalid_id
            && s.step_length[slot] == real_type(INFINITY) && s.detector[slot] == invalid_id)
        {
            return;
        }
        pre_step(p, s, slot);
        gather_pre(p, s, slot);
    }
}

__global__ __launch_bounds__(block_size) void discrete_select_kernel(
    ParamsData p, StateData s)
{
    begin_dependent();
    size_type slot = thread_slot();
    if (slot < s.size)
    {
        discrete_select(p, s, slot);
    }
}

//! Add each lane's value to bins[key] with one atomic per distinct key of
//! the warp: lanes with equal keys are grouped (__match_any_sync), each
//! group's values are summed in lane order, and the group's lowest lane adds
//! the sum. Lanes with an invalid key take part in the exchange only. Every
//! lane of the warp must call this.
__device__ __forceinline__ void warp_tally(double* bins, size_type key, double value)
{
    unsigned int const active = __activemask();
    if (__ballot_sync(active, key != invalid_id) == 0)
        return;
    unsigned int const lane = threadIdx.x & 31u;
    unsigned int const group = __match_any_sync(active, key);
    double sum = 0;
    for (unsigned int k = 0; k < 32; ++k)
    {
        if (!((active >> k) & 1u))
            continue;
        double const v = __shfl_sync(active, value, k);
        if ((group >> k) & 1u)
            sum += v;
    }
    if (key != invalid_id && lane == static_cast<unsigned int>(__ffs(group) - 1))
        atomicAdd(bins + key, sum);
}

//! SimpleCalo tally (SimpleCaloExecutor, src/celeritas/user/detail/
//! SimpleCaloExecutor.hh:48-67): the step's deposition of every track in a
//! detector volume. A zero deposit leaves the sums unchanged and is skipped,
//! as the reference's step filter does; the rest is aggregated per warp.
__global__ __launch_bounds__(block_size) void calo_kernel(ParamsData p, StateData s)
{
    begin_dependent();
    size_type const slot = thread_slot();
    size_type det = invalid_id;
    size_type event = invalid_id;
    double edep = 0;
    if (slot < s.size && s.status[slot] != status_inactive)
    {
        edep = s.energy_deposition[slot];
        if (edep != 0)
        {
            det = s.detector[slot];
            if (p.event_tallies && det != invalid_id)
                event = s.event_id[slot];
        }
    }
    warp_tally(s.calo_edep, det, edep);
    if (p.event_tallies)
    {
        warp_tally(s.event_edep, event, edep);
        warp_tally(s.event_det_edep,
                   event == invalid_id ? invalid_id : event * p.num_detectors + det,
                   edep);
    }
}

//---------------------------------------------------------------------------//
// Step output: each step's hits appended in slot order (DetectorSteps)
//---------------------------------------------------------------------------//
//! Hits of each block of slots
__global__ __launch_bounds__(block_size) void hits_count_kernel(StateData s,
                                                                StepHitsRef h,
                                                                size_type* block_hits)
{
    begin_dependent();
    size_type const slot = thread_slot();
    bool const hit = slot < s.size && has_step_hit(s, h, slot);
    int const count = __syncthreads_count(hit);
    if (threadIdx.x == 0)
        block_hits[blockIdx.x] = static_cast<size_type>(count);
}

//! Record offsets of the blocks: the hits already held plus an exclusive
//! scan of the block counts, by one block of 1024 threads. A step whose hits
//! do not fit sets the overflow flag and records none.
__global__ __launch_bounds__(1024) void hits_scan_kernel(StateData s,
                                                         size_type* block_hits,
                                                         size_type num_blocks,
                                                         size_type capacity)
{
    begin_dependent();
    __shared__ WideScanStorage tmp;
    Counters& c = *s.counters;
    size_type const total = scan_in_place(block_hits, num_blocks, c.num_hits, tmp);
    if (threadIdx.x == 0)
    {
        if (total > capacity)
            c.error_flags |= error_hit_overflow;
        else if (!(c.error_flags & error_hit_overflow))
            c.num_hits = total;
    }
}

//! Write each hit at its block offset plus its rank among the block's hits
__global__ __launch_bounds__(block_size) void hits_scatter_kernel(
    ParamsData p,
    StateData s,
    StepHitsRef h,
    size_type const* block_offsets,
    size_type const* step_index)
{
    begin_dependent();
    __shared__ size_type warp_hits[block_size / 32];
    size_type const slot = thread_slot();
    bool const hit = slot < s.size && has_step_hit(s, h, slot);
    unsigned int const ballot = __ballot_sync(0xffffffffu, hit);
    int const lane = threadIdx.x & 31;
    int const warp = threadIdx.x >> 5;
    if (lane == 0)
        warp_hits[warp] = __popc(ballot);
    __syncthreads();
    if (!hit || (s.counters->error_flags & error_hit_overflow))
        return;
    size_type index = block_offsets[blockIdx.x] + __popc(ballot & ((1u << lane) - 1u));
    for (int w = 0; w < warp; ++w)
        index += warp_hits[w];
    write_step_hit(p, s, h, slot, index, *step_index);
}

//! Live tracks per event: occupied slots plus queued initializers
__global__ void count_event_live_kernel(StateData s, size_type num_events)
{
    size_type const stride = gridDim.x * blockDim.x;
    size_type const tid = thread_slot();
    for (size_type i = tid; i < s.size; i += stride)
    {
        size_type const ev = s.event_id[i];
        if (s.status[i] != status_inactive && ev < num_events)
            atomicAdd(s.event_live + ev, size_type(1));
    }
    size_type const nq = s.counters->num_initializers;
    for (size_type i = tid; i < nq; i += stride)
    {
        size_type const ev = s.initializers[i].event_id;
        if (ev < num_events)
            atomicAdd(s.event_live + ev, size_type(1));
    }
}

//---------------------------------------------------------------------------//
// End of step: vacancies and secondaries
//---------------------------------------------------------------------------//
// A slot's flags byte says whether it is vacant, whether it has anything to
// process, and how many secondaries need a new slot.
constexpr std::uint8_t flag_vacant = 1;
constexpr std::uint8_t flag_process = 2;
constexpr int flag_count_shift = 2;

__global__ __launch_bounds__(block_size) void locate_alive_kernel(StateData s,
                                                                  ScanScratch scr,
                                                                  bool in_place)
{
    begin_dependent();
    size_type const slot = thread_slot();
    bool vacant = false;
    size_type count = 0;
    if (slot < s.size)
    {
        locate_alive(s, slot, &vacant, &count, in_place);
        scr.flags[slot] = static_cast<std::uint8_t>(
            (vacant ? flag_vacant : 0)
            | (s.status[slot] != status_inactive ? flag_process : 0)
            | (count << flag_count_shift));
    }
    // Vacancies and secondaries in the two halves of one word
    size_type const sum = __reduce_add_sync(0xffffffffu, size_type(vacant) | (count << 12));
    __shared__ size_type warp_sum[block_size / 32];
    if ((threadIdx.x & 31) == 0)
        warp_sum[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        size_type all = 0;
        for (int w = 0; w < block_size / 32; ++w)
            all += warp_sum[w];
        scr.block_vacant[blockIdx.x] = all & 0xfffu;
        scr.block_count[blockIdx.x] = all >> 12;
    }
}

__global__ __launch_bounds__(1024) void scan_blocks_kernel(StateData s,
                                                           ScanScratch scr,
                                                           StepLogRef log)
{
    begin_dependent();
    // Exclusive scan of the per-block totals by one block of 1024 threads
    __shared__ WideScanStorage tmp_vac;
    __shared__ WideScanStorage tmp_cnt;
    size_type const carry_vac = scan_in_place(scr.block_vacant, scr.num_blocks, 0, tmp_vac);
    size_type const carry_cnt = scan_in_place(scr.block_count, scr.num_blocks, 0, tmp_cnt);
    if (threadIdx.x == 0)
    {
        Counters& c = *s.counters;
        c.num_vacancies = carry_vac;
        if (carry_cnt > s.initializer_capacity - c.num_initializers)
        {
            // The queue would overflow: this step's secondaries are dropped
            // (the scatter skips them), the queued initializers stay valid
            // and the host reports the overflow
            c.error_flags |= error_initializer_overflow;
            c.num_secondaries = 0;
        }
        else
        {
            c.num_secondaries = carry_cnt;
            c.num_initializers += carry_cnt;
        }
        c.num_alive = s.size - c.num_vacancies;
        StepRecord& r = log.records[*log.step_index % log.capacity];
        r.queued = c.num_initializers;
        r.alive = c.num_alive;
        *log.step_index += 1;
    }
}

__global__ __launch_bounds__(block_size) void scatter_kernel(ParamsData p,
                                                             StateData s,
                                                             ScanScratch scr)
{
    begin_dependent();
    __shared__ BlockScanStorage tmp;
    size_type const slot = thread_slot();
    std::uint32_t const flags = slot < s.size ? scr.flags[slot] : 0;
    // Vacancies and secondaries before this slot in the block
    size_type all;
    size_type const before = block_exclusive_scan(
        (flags & flag_vacant) | (flags >> flag_count_shift << 12), tmp, &all);
    if (flags & flag_vacant)
        s.vacancies[scr.block_vacant[blockIdx.x] + (before & 0xfffu)] = slot;
    if (flags & flag_process)
    {
        Counters const c = *s.counters;
        if (!(c.error_flags & error_initializer_overflow))
        {
            process_secondaries(
                p, s, c, slot, scr.block_count[blockIdx.x] + (before >> 12));
        }
    }
}

__global__ void kill_active_kernel(ParamsData p, StateData s)
{
    size_type slot = thread_slot();
    if (slot < s.size && is_track_valid(s.status[slot]))
    {
        apply_errored(p, s, slot);
    }
}

//---------------------------------------------------------------------------//
// Action sort (SortTracksAction): stable counting sort of the track slots by
// action ID in three kernels. Blocks of sort_block_size slots count their
// keys with warp-aggregated shared-memory atomics (match_any + popc); one block
// per bin scans its row of the [bin][block] counts; the scatter ranks each slot
// among equal keys of its warp (match_any) and of the preceding warps, so
// slots of one action stay in increasing order.
//---------------------------------------------------------------------------//
__device__ __forceinline__ size_type sort_key(StateData const& s,
                                              SortScratch const& srt,
                                              SortKey key,
                                              size_type slot)
{
    size_type const invalid_bin = srt.num_bins - 1;
    if (key == SortKey::start)
    {
        // reindex_status: tracks that are not inactive first (IsNotInactive,
        // TrackSortUtils.cc:71-79); reindex_particle_type: by particle ID
        if (srt.track_order == track_order_reindex_status)
            return s.status[slot] != status_inactive ? 0 : 1;
        size_type const pid = s.particle_id[slot];
        return pid < invalid_bin ? pid : invalid_bin;
    }
    size_type a = (key == SortKey::along_step) ? s.along_step_action[slot]
                                               : s.post_step_action[slot];
    if (!(a < srt.num_actions))
        return invalid_bin;
    if (key == SortKey::along_step && srt.material_actions[0] != invalid_id)
    {
        // Tracks of a material-sorted action by material; later actions
        // after its bins
        size_type const mat = (a == srt.material_actions[0] || a == srt.material_actions[1])
                                  ? min_of(s.material[slot], srt.num_materials - 1)
                                  : 0;
        a = along_bin(srt, a, mat);
    }
    return a;
}

__global__ __launch_bounds__(sort_block_size) void sort_count_kernel(
    StateData s, SortScratch srt, SortKey key)
{
    begin_dependent();
    extern __shared__ size_type hist[];  // [num_bins]
    for (size_type i = threadIdx.x; i < srt.num_bins; i += blockDim.x)
        hist[i] = 0;
    __syncthreads();
    size_type const slot = blockIdx.x * sort_block_size + threadIdx.x;
    bool const valid = slot < s.size;
    size_type const k = valid ? sort_key(s, srt, key, slot) : srt.num_bins;
    unsigned int const peers = __match_any_sync(0xffffffffu, k);
    unsigned int const lane = threadIdx.x & 31u;
    if (valid && (peers & ((1u << lane) - 1u)) == 0)
        atomicAdd(hist + k, static_cast<size_type>(__popc(peers)));
    __syncthreads();
    for (size_type i = threadIdx.x; i < srt.num_bins; i += blockDim.x)
        srt.block_hist[i * srt.num_blocks + blockIdx.x] = hist[i];
}

//! One block per bin: exclusive scan of the bin's counts over the slot blocks
//! and the bin's total; the scatter adds the totals of the bins before. With a
//! single block over all bins, whose threads each read a run of their own, a sort
//! of 2^20 slots took 66 us (three launches, event times), with one bin per
//! block 22.
__global__ __launch_bounds__(1024) void sort_scan_kernel(SortScratch srt)
{
    begin_dependent();
    __shared__ WideScanStorage tmp;
    size_type const total = scan_in_place(
        srt.block_hist + std::size_t(blockIdx.x) * srt.num_blocks, srt.num_blocks, 0, tmp);
    if (threadIdx.x == 0)
        srt.bin_totals[blockIdx.x] = total;
}

__global__ __launch_bounds__(sort_block_size) void sort_scatter_kernel(
    StateData s, SortScratch srt, SortKey key, size_type* offsets)
{
    begin_dependent();
    constexpr unsigned int num_warps = sort_block_size / 32;
    extern __shared__ size_type warp_hist[];  // [num_warps][num_bins]
    size_type const nb = srt.num_bins;
    unsigned int const lane = threadIdx.x & 31u;
    unsigned int const warp = threadIdx.x >> 5;
    // First position of this thread's bin (there are no more bins than threads):
    // exclusive scan of the totals
    size_type bin_base = 0;
    if (warp * 32 < nb)
    {
        for (size_type b = lane; b < warp * 32; b += 32)
            bin_base += srt.bin_totals[b];
        bin_base = __reduce_add_sync(0xffffffffu, bin_base);
        size_type const v = threadIdx.x < nb ? srt.bin_totals[threadIdx.x] : 0;
        size_type incl = v;
        for (unsigned int off = 1; off < 32; off <<= 1)
        {
            size_type const n = __shfl_up_sync(0xffffffffu, incl, off);
            if (lane >= off)
                incl += n;
        }
        bin_base += incl - v;
        if (blockIdx.x == 0 && threadIdx.x < nb)
            offsets[threadIdx.x] = bin_base;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        offsets[nb] = s.size;
    for (size_type i = threadIdx.x; i < num_warps * nb; i += blockDim.x)
        warp_hist[i] = 0;
    __syncthreads();
    size_type const slot = blockIdx.x * sort_block_size + threadIdx.x;
    bool const valid = slot < s.size;
    size_type const k = valid ? sort_key(s, srt, key, slot) : nb;
    unsigned int const peers = __match_any_sync(0xffffffffu, k);
    unsigned int const lower = peers & ((1u << lane) - 1u);
    if (valid && lower == 0)
        warp_hist[warp * nb + k] = __popc(peers);
    __syncthreads();
    if (threadIdx.x < nb)
    {
        size_type acc = bin_base;
        for (unsigned int w = 0; w < num_warps; ++w)
        {
            size_type const c = warp_hist[w * nb + threadIdx.x];
            warp_hist[w * nb + threadIdx.x] = acc;
            acc += c;
        }
    }
    __syncthreads();
    if (valid)
    {
        size_type const pos = srt.block_hist[k * srt.num_blocks + blockIdx.x]
                              + warp_hist[warp * nb + k] + __popc(lower);
        s.track_slots[pos] = slot;
    }
}

//! Offsets and bins through which a sorted-range kernel visits its tracks:
//! the action's range of the key's sort; or, for the reindexing orders
//! (shuffle, status, particle type), every slot through the thread -> slot
//! permutation (the shuffle's is fixed when the state is made, the others'
//! are this step's start sort, when it runs)
struct SlotRange
{
    size_type const* slots;
    size_type const* offsets;
    size_type first_bin;
    size_type end_bin;
};

//! Call f(slot) for every slot of the sorted bins [first_bin, end_bin) (or,
//! without offsets, every slot) with a grid-stride loop: a grid of a few
//! blocks per SM covers a range of any length, where a grid sized for the
//! whole state would launch mostly blocks that find no track of the action
//! (the range lives on the device, so the host cannot size the grid to it)
template<class F>
__device__ __forceinline__ void for_each_sorted_slot(StateData const& s,
                                                     size_type const* offsets,
                                                     size_type first_bin,
                                                     size_type end_bin,
                                                     F&& f)
{
    size_type begin = 0;
    size_type end = s.size;
    if (offsets)
    {
        begin = offsets[first_bin];
        end = offsets[end_bin];
    }
    size_type const stride = gridDim.x * blockDim.x;
    for (size_type t = begin + blockIdx.x * blockDim.x + threadIdx.x; t < end; t += stride)
        f(offsets ? s.track_slots[t] : t);
}

// Minimum resident blocks per SM requested for the charged along-step kernel
// (1: the compiler may use up to 255 registers per thread)
#ifndef GBX_ALONG_MIN_BLOCKS
#    define GBX_ALONG_MIN_BLOCKS 1
#endif

// Register cap of the charged along-step kernels (0: none). An SM
// sub-partition holds 16,384 registers, so a cap of 168 per thread keeps 3
// warps resident on each (12 per SM) where 174 keeps 2.
#ifndef GBX_ALONG_MAXNREG
#    define GBX_ALONG_MAXNREG 0
#endif
// The charged kernels come in two instances: blocks of up to 256 threads
// (the kernel's natural register count), and blocks of 512, for which the
// launch bound caps registers at 65536 / 512 = 128 per thread (the compiler
// spills what does not fit)
#if GBX_ALONG_MAXNREG > 0
#    define GBX_ALONG_BOUNDS(THREADS, MINB) __maxnreg__(GBX_ALONG_MAXNREG)
#else
#    define GBX_ALONG_BOUNDS(THREADS, MINB) __launch_bounds__(THREADS, MINB)
#endif
constexpr int along_block_large = 512;

//! Threads on every SM over which few tracks are spread
constexpr int spread_threads = 256;

//! Whether 'count' tracks are few enough to be spread over the warps of the first
//! 'blocks' blocks (which all fit on the GPU), and the one that this thread gets.
//! Tracks in a field take paths and times of their own: one that curls up for a
//! million cycles alone took up to 1.9 million beside 31 others. A warp therefore
//! gets a second track only when every warp has one, neighbours in different SMs.
//! From 32 tracks a warp on, one after the other is the better order (coalesced
//! access). 650 particles in the CMS-like detector in 2^21 slots 377 -> 358 ms with
//! the launch settings found for it and 571 -> 393 ms with the default (persistent)
//! ones, an FP64 event of 20 there 477 -> 458 ms; with at most 4 or 16 tracks a warp
//! the first took 373 and 364 ms.
__device__ __forceinline__ bool
spread_track(size_type count, size_type blocks, size_type* index)
{
    size_type const warps = blocks * (blockDim.x >> 5);
    if (count > warps * 31)
        return false;
    size_type const lane = threadIdx.x & 31u;
    *index = blockIdx.x < blocks ? lane * warps + (threadIdx.x >> 5) * blocks + blockIdx.x
                                 : count;
    return true;
}

//! Spread: see spread_track(), over the first 'spread_blocks' blocks; up to
//! 'warp_tracks' tracks are left to along_charged_warp_kernel
template<AlongKind K, int Threads = block_size, bool Spread = false>
__global__ GBX_ALONG_BOUNDS(Threads, K == AlongKind::charged ? GBX_ALONG_MIN_BLOCKS : 1) void
along_step_sorted_kernel(ParamsData p,
                         StateData s,
                         SlotRange range,
                         size_type spread_blocks,
                         size_type warp_tracks)
{
    begin_dependent();
    size_type const first = range.offsets ? range.offsets[range.first_bin] : 0;
    size_type const count = range.offsets ? range.offsets[range.end_bin] - first : s.size;
    size_type stride = gridDim.x * blockDim.x;
    size_type index = thread_slot();
    if constexpr (Spread)
    {
        if (count <= warp_tracks)
            return;
        if (spread_track(count, spread_blocks, &index))
            stride = count;
    }
    for (; index < count; index += stride)
    {
        along_step_impl<K>(p, s, range.offsets ? range.slots[first + index] : index);
    }
}

//! FP64 charged along-step in a field of at most 'warp_tracks' tracks, the warps of
//! this grid: each runs one, lane 0 the track and the others its Runge-Kutta steps
//! with it (warp_step). Fewer warps than a block of 8 on every SM are worse also where
//! the FP64 units are shared (300 electrons in the calorimeter with at most 1, 2, 4, 8
//! tracks per SM: 239, 237, 234, 233 ms). A kernel of its own: in one with
//! along_step_sorted_kernel it makes that one 4% slower (233 against 224.5 ms).
//! Real: the build's real_type, for the launch that only the FP64 build has.
template<class Real>
__global__ __launch_bounds__(block_size, 1) void along_charged_warp_kernel(
    ParamsData p, StateData s, SlotRange range, size_type warp_tracks)
{
    begin_dependent();
    size_type const first = range.offsets[range.first_bin];
    size_type const count = range.offsets[range.end_bin] - first;
    if (count > warp_tracks)
        return;
    size_type const track = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    if (track >= count)
        return;
    if ((threadIdx.x & 31u) != 0)
    {
        help_field_warp();
        return;
    }
    along_step_impl<AlongKind::charged, true>(p, s, range.slots[first + track]);
    end_field_warp();
}

//! Before the list below or the persistent kernel: no track claimed, none listed
__global__ void clear_along_work_kernel(AlongWork work)
{
    begin_dependent();
    *work.counter = 0;
    work.offsets[1] = 0;
}

//! List the tracks of the charged along-step where the state is not sorted by
//! it, in no particular order
__global__ __launch_bounds__(block_size) void
list_charged_kernel(ParamsData p, StateData s, AlongWork work)
{
    begin_dependent();
    size_type const slot = thread_slot();
    bool const charged = slot < s.size && is_track_valid(s.status[slot])
                         && s.along_step_action[slot] == p.action_along_step;
    unsigned int const ballot = __ballot_sync(0xffffffffu, charged);
    if (!ballot)
        return;
    unsigned int const lane = threadIdx.x & 31u;
    size_type base = 0;
    if (lane == 0)
        base = atomicAdd(work.offsets + 1, size_type(__popc(ballot)));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (charged)
        work.slots[base + __popc(ballot & ((1u << lane) - 1u))] = slot;
}

//! Charged along-step in a uniform field over the sorted charged range, as
//! a persistent kernel: each thread takes tracks from a work counter
//! (warp-aggregated), keeps the track's propagation in registers, and runs
//! one field substep per loop iteration, taking the next track as soon as
//! its own finishes. Lanes of a warp thus stay busy on different tracks
//! instead of waiting for the one with the most substeps. Every track runs
//! the same sequence of operations as along_step_impl.
template<int Threads>
__global__ GBX_ALONG_BOUNDS(Threads, 1) void along_charged_persistent_kernel(
    ParamsData p, StateData s, SlotRange range, size_type* work_counter)
{
    begin_dependent();
    size_type const first = range.offsets[range.first_bin];
    size_type const count = range.offsets[range.end_bin] - first;
    size_type spread_index = count;
    bool const spread = spread_track(count, gridDim.x, &spread_index);
    unsigned int const lane = threadIdx.x & 31u;
    FieldOptions const& opt = p.field_options;
    FieldPropagation<false> fp(opt, UniformFieldEquation{});
    size_type slot = invalid_id;
    bool have = false;
    for (;;)
    {
        if (!have)
        {
            size_type idx = spread_index;
            spread_index = count;
            if (!spread)
            {
                // Claim the next track for every lane that needs one
                unsigned int const need = __activemask();
                unsigned int const rank = __popc(need & ((1u << lane) - 1u));
                unsigned int const leader = __ffs(need) - 1;
                size_type base = 0;
                if (lane == leader)
                    base = atomicAdd(work_counter, size_type(__popc(need)));
                base = __shfl_sync(need, base, leader);
                idx = base + rank;
            }
            if (idx >= count)
                break;
            slot = range.slots[first + idx];
            bool charged;
            double start_safety;
            if (!along_prologue<AlongKind::charged>(p, s, slot, &charged, &start_safety))
                continue;
            if (s.step_length[slot] == 0)
            {
                along_epilogue(p, s, slot, true);
                continue;
            }
            GeoTrackView geo(p.geo, s, slot);
            field_setup(p, s, slot, geo, &fp, start_safety);
            have = true;
        }
        GeoTrackView geo(p.geo, s, slot);
        fp.substep(geo);
        if (fp.done())
        {
            field_result(p, s, slot, fp.finish(geo));
            along_epilogue(p, s, slot, true);
            have = false;
        }
    }
}

__global__ __launch_bounds__(block_size) void interact_sorted_kernel(
    ParamsData p,
    StateData s,
    size_type const* offsets,
    size_type first_bin,
    size_type end_bin,
    size_type first_action,
    size_type end_action)
{
    begin_dependent();
    for_each_sorted_slot(s, offsets, first_bin, end_bin, [&](size_type slot) {
        size_type a = s.post_step_action[slot];
        if (a >= first_action && a < end_action)
            interact(p, s, slot, a);
    });
}

__global__ __launch_bounds__(block_size) void boundary_sorted_kernel(
    ParamsData p,
    StateData s,
    size_type const* offsets,
    size_type first_bin,
    size_type end_bin)
{
    begin_dependent();
    for_each_sorted_slot(
        s, offsets, first_bin, end_bin, [&](size_type slot) { boundary_cross(p, s, slot); });
}

__global__ __launch_bounds__(block_size) void tracking_cut_sorted_kernel(
    ParamsData p,
    StateData s,
    size_type const* offsets,
    size_type first_bin,
    size_type end_bin)
{
    begin_dependent();
    for_each_sorted_slot(
        s, offsets, first_bin, end_bin, [&](size_type slot) { tracking_cut(p, s, slot); });
}

//! geo-boundary and tracking-cut together: a track whose crossing fails is cut
//! in the same pass where the cut visits every slot, and left to the next step
//! where it visits the sorted range of its action, as when the two are launched
//! one after the other. Each is a few us of launch and first instructions when
//! there are few tracks: together with the counters' update in the last block of
//! the initialization, a step's two launches fewer take an FP64 calorimeter of 100
//! electrons from 36.3 to 36.05 ms and 2000 photons from 35.76 to 35.37 ms.
__global__ __launch_bounds__(block_size) void boundary_cut_sorted_kernel(
    ParamsData p, StateData s, SlotRange boundary, SlotRange cut)
{
    begin_dependent();
    bool const all = !boundary.offsets || boundary.first_bin == cut.first_bin;
    for_each_sorted_slot(
        s, boundary.offsets, boundary.first_bin, boundary.end_bin, [&](size_type slot) {
            boundary_cross(p, s, slot);
            if (all)
                tracking_cut(p, s, slot);
        });
    if (!all)
    {
        for_each_sorted_slot(s, cut.offsets, cut.first_bin, cut.end_bin, [&](size_type slot) {
            tracking_cut(p, s, slot);
        });
    }
}

//! Bin offsets written by the sort for a key
inline size_type* sort_offsets(LaunchContext const& ctx, SortKey key)
{
    std::size_t const table = std::size_t(ctx.sort.num_bins) + 1;
    return ctx.state.action_offsets + (key == SortKey::step_limit ? table : 0);
}

inline SlotRange
slot_range(LaunchContext const& ctx, SortKey key, size_type first_bin, size_type end_bin)
{
    unsigned int const order = ctx.params.track_order;
    if (reindexes_all(order))
    {
        bool const permuted = order == track_order_reindex_shuffle || ctx.sort_enabled;
        return {ctx.state.track_slots,
                permuted ? sort_offsets(ctx, SortKey::start) : nullptr,
                0,
                ctx.sort.num_bins};
    }
    bool const sorts = key == SortKey::along_step ? sorts_along_step(order)
                                                  : sorts_step_limit(order);
    return {ctx.state.track_slots,
            sorts && ctx.sort_enabled ? sort_offsets(ctx, key) : nullptr,
            first_bin,
            end_bin};
}

}  // namespace

//---------------------------------------------------------------------------//
// Launchers
//---------------------------------------------------------------------------//
//! Launch a kernel of the step, which may be scheduled as soon as the blocks of
//! the stream's previous kernel are through, while that one's writes are still being
//! flushed: it waits for them in begin_dependent(). A step of few tracks is a chain
//! of short kernels: one electron in 4096 slots 9.44 -> 9.12 ms, a two-particle event
//! in the CMS-like detector 17.8 -> 16.7 ms, 3000 electrons in 2^20 slots 177 -> 175.5
//! ms. Letting the next kernel's blocks in from the start of this one (an explicit
//! launch_dependents) is no better for those, and worse from 2^16 slots on (36.0 ->
//! 36.6 ms for 100 electrons, 377.7 -> 380.7 ms for the largest): they take the place
//! of running warps.
template<class... Params, class... Args>
void launch(void (*kernel)(Params...),
            unsigned int blocks,
            unsigned int threads,
            std::size_t shared,
            cudaStream_t stream,
            Args const&... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = shared;
    config.stream = stream;
    config.attrs = &attr;
    config.numAttrs = 1;
    cudaLaunchKernelEx(&config, kernel, Params(args)...);
}

void launch_process_primaries(LaunchContext const& ctx,
                              size_type num_primaries,
                              cudaStream_t stream)
{
    begin_primaries_kernel<<<1, 1, 0, stream>>>(ctx.state, num_primaries);
    size_type n = max_of(num_primaries, ctx.state.size);
    process_primaries_kernel<<<num_blocks_for(n), block_size, 0, stream>>>(
        ctx.state, num_primaries);
}

void launch_generate_primaries(LaunchContext const& ctx,
                               PrimaryGeneratorData const& gen,
                               cudaStream_t stream)
{
    size_type const n = gen.num_events * gen.primaries_per_event;
    generate_primaries_kernel<<<num_blocks_for(n), block_size, 0, stream>>>(
        gen, ctx.state, n);
}

void launch_initialize_tracks(LaunchContext const& ctx, cudaStream_t stream)
{
    if (partitions_by_charge(ctx.params.track_order))
    {
        // InitializeTracksAction with TrackOrder init_charge
        // (InitializeTracksAction.cc:55-95)
        unsigned int const nb = num_blocks_for(ctx.state.size);
        launch(charge_partition_count_kernel, nb, block_size, 0, stream, ctx.params,
               ctx.state, ctx.scratch);
        launch(charge_partition_scan_kernel, 1, 1024, 0, stream, ctx.scratch, nb);
        launch(charge_partition_scatter_kernel, nb, block_size, 0, stream, ctx.params,
               ctx.state, ctx.scratch);
        launch(initialize_tracks_charge_kernel, ctx.range_blocks, block_size, 0, stream,
               ctx.params, ctx.state);
        launch(finish_initialize_kernel, 1, 1, 0, stream, ctx.state, ctx.log);
        launch(clear_parents_kernel, ctx.range_blocks, block_size, 0, stream, ctx.state);
        return;
    }
    if (ctx.partition_slots)
    {
        launch(initialize_tracks_partitioned_kernel, num_blocks_for(ctx.state.size),
               block_size, 0, stream, ctx.params, ctx.state);
        launch(finish_initialize_kernel, 1, 1, 0, stream, ctx.state, ctx.log);
        return;
    }
    launch(initialize_tracks_kernel, ctx.range_blocks, block_size, 0, stream, ctx.params,
           ctx.state, ctx.log, ctx.scratch.ticket);
}

void launch_pre_step(LaunchContext const& ctx, cudaStream_t stream)
{
    launch(pre_step_kernel, num_blocks_for(ctx.state.size), block_size, 0, stream,
           ctx.params, ctx.state);
}


//! Charged along-step of few tracks by a warp each; returns up to how many (none in
//! the mixed build). One track per warp of a block on every SM; the persistent
//! kernel takes all its tracks itself.
template<class Real>
size_type launch_along_warps(LaunchContext const& ctx, SlotRange const& range, cudaStream_t stream)
{
    if constexpr (std::is_same_v<Real, double>)
    {
        if (ctx.persistent_blocks == 0)
        {
            size_type const warp_tracks = ctx.num_sms * (block_size / 32);
            launch(along_charged_warp_kernel<Real>, ctx.num_sms, block_size, 0, stream,
                   ctx.params, ctx.state, range, warp_tracks);
            return warp_tracks;
        }
    }
    return 0;
}

void launch_along_step(LaunchContext const& ctx,
                       size_type action,
                       cudaStream_t stream)
{
    // Each along-step action runs a kernel compiled for that action only,
    // over its sorted range or (sorting off) over all slots; the grid covers
    // the largest range. Sorted and unsorted orders thus run the same code,
    // and a track's result does not depend on the track order. (In the mixed build
    // it may on the kernel: the persistent one rounds one square of steps of at most the
    // minimum length differently, MixedFieldDriver's RoundX.)
    ParamsData const& p = ctx.params;
    unsigned int const nb = num_blocks_for(ctx.state.size);
    unsigned int const abs = static_cast<unsigned int>(ctx.along_block_size);
    unsigned int const anb = (ctx.state.size + abs - 1) / abs;
    // Charged along-step grid: up to 2^19 threads (grid-stride beyond), so
    // that a charged range well below the state size does not launch
    // thousands of blocks that find no track
    unsigned int const cnb = min_of(anb, max_of(1u, (1u << 19) / abs));
    size_type cfirst, cend, nfirst, nend;
    along_bins(ctx.sort, p.action_along_step, &cfirst, &cend);
    along_bins(ctx.sort, p.action_along_step_neutral, &nfirst, &nend);
    if (action == invalid_id || action == p.action_along_step)
    {
        SlotRange range = slot_range(ctx, SortKey::along_step, cfirst, cend);
        bool const large = abs > static_cast<unsigned int>(block_size);
        unsigned int blocks = cnb;
        size_type spread_blocks = 0;
        size_type warp_tracks = 0;
        if (p.has_field)
        {
            bool const list = !range.offsets || reindexes_all(p.track_order);
            if (list || ctx.persistent_blocks > 0)
                launch(clear_along_work_kernel, 1, 1, 0, stream, ctx.along_work);
            if (list)
            {
                launch(list_charged_kernel, nb, block_size, 0, stream, p, ctx.state,
                       ctx.along_work);
                range = {ctx.along_work.slots, ctx.along_work.offsets, 0, 1};
            }
            spread_blocks = ctx.num_sms * max_of(1u, spread_threads / abs);
            blocks = max_of<unsigned int>(blocks, spread_blocks);
            warp_tracks = launch_along_warps<real_type>(ctx, range, stream);
        }
        if (p.has_field && ctx.persistent_blocks > 0)
        {
            if (large)
                launch(along_charged_persistent_kernel<along_block_large>,
                       ctx.persistent_blocks, abs, 0, stream, p, ctx.state, range,
                       ctx.along_work.counter);
            else
                launch(along_charged_persistent_kernel<block_size>,
                       ctx.persistent_blocks, abs, 0, stream, p, ctx.state, range,
                       ctx.along_work.counter);
        }
        else
        {
            auto* kernel
                = large ? (p.has_field
                               ? along_step_sorted_kernel<AlongKind::charged, along_block_large, true>
                               : along_step_sorted_kernel<AlongKind::charged, along_block_large>)
                        : (p.has_field
                               ? along_step_sorted_kernel<AlongKind::charged, block_size, true>
                               : along_step_sorted_kernel<AlongKind::charged>);
            launch(kernel, blocks, abs, 0, stream, p, ctx.state, range, spread_blocks,
                   warp_tracks);
        }
    }
    if (action == invalid_id || action == p.action_along_step_neutral)
    {
        SlotRange const range = slot_range(ctx, SortKey::along_step, nfirst, nend);
        launch(along_step_sorted_kernel<AlongKind::neutral>, ctx.range_blocks, block_size, 0,
               stream, p, ctx.state, range, 0u, 0u);
    }
}

void launch_discrete_select(LaunchContext const& ctx, cudaStream_t stream)
{
    launch(discrete_select_kernel, num_blocks_for(ctx.state.size), block_size, 0, stream,
           ctx.params, ctx.state);
}

void launch_interact(LaunchContext const& ctx, size_type action, cudaStream_t stream)
{
    ParamsData const& p = ctx.params;
    size_type first = action, end = action + 1;
    if (action == invalid_id)
    {
        // All models at once: they are mutually exclusive per slot. A step's
        // seven launches become one: 100 electrons of 1 GeV in FP64 49 -> 37
        // ms, 3000 c2 electrons in the mixed build (with the sort's scan)
        // 207 -> 166 ms.
        first = p.model_to_action;
        end = p.model_to_action + p.num_models;
    }
    SlotRange const r = slot_range(ctx, SortKey::step_limit, first, end);
    launch(interact_sorted_kernel, ctx.range_blocks, block_size, 0, stream, p, ctx.state,
           r.offsets, r.first_bin, r.end_bin, first, end);
}

void launch_boundary(LaunchContext const& ctx, cudaStream_t stream)
{
    ParamsData const& p = ctx.params;
    SlotRange const r
        = slot_range(ctx, SortKey::step_limit, p.action_boundary, p.action_boundary + 1);
    launch(boundary_sorted_kernel, ctx.range_blocks, block_size, 0, stream, p, ctx.state,
           r.offsets, r.first_bin, r.end_bin);
}

void launch_tracking_cut(LaunchContext const& ctx, cudaStream_t stream)
{
    ParamsData const& p = ctx.params;
    SlotRange const r = slot_range(
        ctx, SortKey::step_limit, p.action_tracking_cut, p.action_tracking_cut + 1);
    launch(tracking_cut_sorted_kernel, ctx.range_blocks, block_size, 0, stream, p,
           ctx.state, r.offsets, r.first_bin, r.end_bin);
}

void launch_boundary_cut(LaunchContext const& ctx, cudaStream_t stream)
{
    ParamsData const& p = ctx.params;
    launch(boundary_cut_sorted_kernel, ctx.range_blocks, block_size, 0, stream, p,
        ctx.state,
        slot_range(ctx, SortKey::step_limit, p.action_boundary, p.action_boundary + 1),
        slot_range(ctx, SortKey::step_limit, p.action_tracking_cut, p.action_tracking_cut + 1));
}

void launch_calo_tally(LaunchContext const& ctx, cudaStream_t stream)
{
    unsigned int const nb = num_blocks_for(ctx.state.size);
    launch(calo_kernel, nb, block_size, 0, stream, ctx.params, ctx.state);
    if (ctx.hits.enabled())
    {
        launch(hits_count_kernel, nb, block_size, 0, stream, ctx.state, ctx.hits,
               ctx.hit_block_offsets);
        launch(hits_scan_kernel, 1, 1024, 0, stream, ctx.state, ctx.hit_block_offsets,
               nb, ctx.hits.capacity);
        launch(hits_scatter_kernel, nb, block_size, 0, stream, ctx.params, ctx.state,
               ctx.hits, ctx.hit_block_offsets, ctx.log.step_index);
    }
}

void launch_extend_from_secondaries(LaunchContext const& ctx, cudaStream_t stream)
{
    ScanScratch const& scr = ctx.scratch;
    launch(locate_alive_kernel, scr.num_blocks, block_size, 0, stream, ctx.state, scr,
           !partitions_by_charge(ctx.params.track_order));
    launch(scan_blocks_kernel, 1, 1024, 0, stream, ctx.state, scr, ctx.log);
    launch(scatter_kernel, scr.num_blocks, block_size, 0, stream, ctx.params, ctx.state,
           scr);
}

int persistent_along_blocks(int threads_per_block)
{
    int device = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&device) != cudaSuccess
        || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)
               != cudaSuccess
        || (threads_per_block > block_size
                ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                      &per_sm,
                      along_charged_persistent_kernel<along_block_large>,
                      threads_per_block,
                      0)
                : cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                      &per_sm,
                      along_charged_persistent_kernel<block_size>,
                      threads_per_block,
                      0))
               != cudaSuccess)
    {
        return 0;
    }
    return sms * per_sm;
}

void launch_count_event_live(LaunchContext const& ctx,
                             size_type num_events,
                             cudaStream_t stream)
{
    cudaMemsetAsync(ctx.state.event_live, 0, sizeof(size_type) * num_events, stream);
    // A grid-stride pass: four blocks per SM of the current device
    static thread_local int sms = 0;
    if (sms == 0)
    {
        int device = 0;
        if (cudaGetDevice(&device) != cudaSuccess
            || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)
                   != cudaSuccess
            || sms <= 0)
        {
            sms = 1;
        }
    }
    count_event_live_kernel<<<4 * sms, block_size, 0, stream>>>(ctx.state, num_events);
}

__global__ __launch_bounds__(block_size) void reseed_kernel(ParamsData p,
                                                            StateData s,
                                                            unsigned int seed,
                                                            unsigned long long event_id)
{
    size_type const slot = thread_slot();
    if (slot < s.size)
    {
        reseed_xorwow_slot(s.rng,
                           p.rng_jump + 32 * 5,
                           seed,
                           event_id * s.size + slot,
                           slot);
    }
}

void launch_reseed(LaunchContext const& ctx,
                   unsigned int seed,
                   unsigned long long event_id,
                   cudaStream_t stream)
{
    reseed_kernel<<<num_blocks_for(ctx.state.size), block_size, 0, stream>>>(
        ctx.params, ctx.state, seed, event_id);
}

void launch_kill_active(LaunchContext const& ctx, cudaStream_t stream)
{
    kill_active_kernel<<<num_blocks_for(ctx.state.size), block_size, 0, stream>>>(
        ctx.params, ctx.state);
}

void check_sort_bins(LaunchContext const& ctx)
{
    if (ctx.sort.num_bins > max_sort_bins)
        throw std::runtime_error("too many actions and materials for the track sort: "
                                 + std::to_string(ctx.sort.num_bins) + " bins, at most "
                                 + std::to_string(max_sort_bins));
}

void launch_sort_tracks(LaunchContext const& ctx, SortKey key, cudaStream_t stream)
{
    check_sort_bins(ctx);
    SortScratch const& srt = ctx.sort;
    launch(sort_count_kernel, srt.num_blocks, sort_block_size,
           srt.num_bins * sizeof(size_type), stream, ctx.state, srt, key);
    launch(sort_scan_kernel, srt.num_bins, 1024, 0, stream, srt);
    launch(sort_scatter_kernel, srt.num_blocks, sort_block_size,
           (sort_block_size / 32) * srt.num_bins * sizeof(size_type), stream,
           ctx.state, srt, key, sort_offsets(ctx, key));
}

//---------------------------------------------------------------------------//
// Extend-from-secondaries with library-owned scratch
//---------------------------------------------------------------------------//
// The three extend-from-secondaries kernels need a byte of scratch per track slot
// plus 8 bytes per block. This variant takes that scratch from one array compiled
// into the library instead of the stepper's allocation, for callers that may not
// allocate device memory at all. Layout for n slots and b = ceil(n / block_size)
// blocks, each part 256-byte aligned:
//   block_vacant[b] | block_count[b] | flags[n]
namespace
{
constexpr std::size_t align_256(std::size_t bytes)
{
    return (bytes + 255) & ~std::size_t(255);
}

constexpr std::size_t static_scratch_bytes(std::size_t n)
{
    std::size_t const b = (n + block_size - 1) / block_size;
    return 2 * align_256(b * sizeof(size_type)) + align_256(n);
}

// 135,168 bytes for 131,072 track slots
constexpr std::size_t static_scratch_capacity
    = static_scratch_bytes(static_scratch_max_slots);

__device__ __align__(256) unsigned char static_scan_scratch[static_scratch_capacity];

// Device address of static_scan_scratch, looked up once per device
constexpr int static_scratch_max_devices = 64;
std::mutex static_scratch_mutex;
void* static_scratch_address[static_scratch_max_devices] = {};

}  // namespace

unsigned char* static_scratch_for_current_device()
{
    int device = -1;
    if (cudaError_t err = cudaGetDevice(&device); err != cudaSuccess)
    {
        throw std::runtime_error(std::string("cudaGetDevice failed: ")
                                 + cudaGetErrorString(err));
    }
    if (device < 0 || device >= static_scratch_max_devices)
    {
        throw std::runtime_error("static scratch supports device ordinals below "
                                 + std::to_string(static_scratch_max_devices));
    }
    std::lock_guard<std::mutex> lock(static_scratch_mutex);
    if (!static_scratch_address[device])
    {
        void* ptr = nullptr;
        cudaError_t err = cudaGetSymbolAddress(&ptr, static_scan_scratch);
        if (err != cudaSuccess || !ptr)
        {
            throw std::runtime_error(
                std::string("cudaGetSymbolAddress of the static scratch failed: ")
                + cudaGetErrorString(err));
        }
        static_scratch_address[device] = ptr;
    }
    return static_cast<unsigned char*>(static_scratch_address[device]);
}

void launch_extend_from_secondaries_static(LaunchContext const& ctx,
                                           cudaStream_t stream)
{
    size_type const n = ctx.state.size;
    if (n > static_scratch_max_slots)
    {
        throw std::runtime_error(
            "the stepper has " + std::to_string(n)
            + " track slots but the static scratch of extend-from-secondaries "
              "holds at most "
            + std::to_string(static_scratch_max_slots));
    }
    unsigned char* base = static_scratch_for_current_device();
    unsigned int const nb = num_blocks_for(n);
    std::size_t const block_part = align_256(std::size_t(nb) * sizeof(size_type));

    // Nothing is cleared: locate_alive_kernel writes the flags of every slot
    // and both totals of every block before it and the scatter kernel read
    // them, so the previous call's contents are never used
    ScanScratch scr;
    scr.block_vacant = reinterpret_cast<size_type*>(base);
    scr.block_count = reinterpret_cast<size_type*>(base + block_part);
    scr.flags = base + 2 * block_part;
    scr.ticket = ctx.scratch.ticket;
    scr.num_blocks = nb;

    launch(locate_alive_kernel, nb, block_size, 0, stream, ctx.state, scr,
           !partitions_by_charge(ctx.params.track_order));
    launch(scan_blocks_kernel, 1, 1024, 0, stream, ctx.state, scr, ctx.log);
    launch(scatter_kernel, nb, block_size, 0, stream, ctx.params, ctx.state, scr);
}

}  // namespace gbx
