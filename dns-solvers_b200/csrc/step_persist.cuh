// The time loop of one or many channels in one launch.
//
// A launch advances every channel of its table through nsteps steps.  The
// work is one long sequence of items -- one row group (k rows) of one plane
// at one step -- that the blocks take in
// order from a counter.  Nothing separates the steps: an item starts when the
// row groups around it (the planes z-1 .. z+1, the groups next to it) are
// done with the step before, which each group announces in its own flag.
// In the AA scheme that is the whole dependency of a step: an even step
// touches only the cells' own rows, an odd step the rows around them, and
// every address is read and written by exactly one cell per step.  Nothing
// is left to a block by its number: items, and the planes to be summed, are
// taken in the order of the sequence by blocks that run, so the first
// unfinished one of either is always held by a running block, and what it
// waits for lies before it.  So the launch makes progress however many of
// its blocks are resident.
//
// Order of the sequence.  A channel's groups are numbered along the planes
// z = 0 .. nz-1; within a plane the periodic rows are folded (0, last, 1,
// last-1, ...), so that neighbours stay near each other.  `depth` steps run
// through the channel at once, each `lag` groups behind the step before it:
// what a step writes is read by the next one while it is still in L2, so
// DRAM sees the populations once per `depth` steps.
//
// A block has two special warps and the consumers:
//   load warp   takes items, waits until a stage is free and the item's
//               neighbours are done, and brings the 19 directions' rows into
//               the stage (bulk copies, as in step_tma.cuh);
//   consumers   collide the stage's cells in place (step_tma.cuh); each
//               warp leaves its sums of the cells in shared memory;
//   store warp  writes the rows back, adds up the warps' sums, and, when
//               the copies have landed, raises the group's flag and counts it
//               in its plane.  Between items it looks after one plane, the
//               next of the sequence of (step, plane) that no other block has
//               taken: once its groups are all counted it is summed, and
//               whoever sums the last plane of a step runs the step tail
//               (logs, next force), off the path of the following steps
//               unless their force depends on it (constant flow rate: the
//               consumers of a step wait for the tail before).
// Sums are per group and added in a fixed order, so logs and forces do not
// depend on which block took which item.  Steps in flight have their own
// sums and counters (kRing entries); a step starts only when the step kRing
// before it is logged.
//
// Planes with link masks (solids inside the flow): an even step moves them
// like any plane, and an odd step the rows whose cells are alike (RowInfo),
// each direction from the row its links lead to.  Of a mixed row an odd step
// brings in the rows of the regular address set; a link that bounces back or
// meets a wall reads its own address from global memory, and every result
// goes to global memory: a bounced link's address lies in a row of another
// cell row's set (that of the solid neighbour, which is never collided), so
// the rows are not stored back.
//
// Every wait is bounded by the GPU's global timer.  A wait that runs out
// raises the block's and the launch's abort flags; every warp then leaves,
// the load warp after the copies it has issued have landed, the store warp
// after its stores.
//
// Memory written by other SMs earlier in the launch is read through L2: bulk
// copies always are; the per-thread loads use ld.global.cg, and per-channel
// values are read with __ldcg.
#pragma once

#include <cuda.h>

#define DNSLBM_GROUPED_STAGE
#include "step_tma.cuh"

namespace dnslbm {

// The populations as a 5-D tensor of 8-byte words -- (word in a piece of the
// row, piece, y, z, array in lat_pos order) -- with boxes of a row group of
// all 19 arrays, of three, and of one.  A row is cut into equal pieces
// because a box has at most 256 words a side; its pieces follow each other
// in shared memory as in the row.
struct FlowMaps {
    CUtensorMap all, three, one;
};

// Sequence position r (0 .. depth * qmax - 1) of a channel's items: slot
// q = r / depth of stream r % depth; stream d is `lag` slots behind stream
// d - 1 and runs the steps d, d + depth, ... one after another.
struct ItemPos {
    int step;     // step within the launch; -1: the position holds no item
    int z, g;     // plane and row group within the plane
};

__host__ __device__ __forceinline__ unsigned flow_items(int depth, int lag, unsigned ngroups, int nsteps)
{
    // nsteps is a multiple of depth
    return (unsigned)depth * ((unsigned)(depth - 1) * (unsigned)lag + (unsigned)(nsteps / depth) * ngroups);
}

__host__ __device__ __forceinline__ ItemPos flow_item(unsigned r, int depth, int lag, unsigned ngroups, int gpp,
                                                      int nsteps)
{
    const unsigned q = depth == 1 ? r : r / (unsigned)depth, d = r - q * (unsigned)depth;
    ItemPos it{-1, 0, 0};
    if (q < d * (unsigned)lag) return it;
    const unsigned P = q - d * (unsigned)lag, w = P / ngroups, p = P - w * ngroups;
    const unsigned s = w * (unsigned)depth + d;
    if (s >= (unsigned)nsteps) return it;
    it.step = (int)s;
    it.z = (int)(p / (unsigned)gpp);
    const int pos = (int)(p - (unsigned)it.z * (unsigned)gpp);
    it.g = (pos & 1) ? gpp - 1 - (pos >> 1) : pos >> 1;
    return it;
}

// Neighbour i (0 .. 8) of group g of plane z whose previous step an item
// waits for; -1: none (beyond a wall).
__host__ __device__ __forceinline__ int flow_neighbour(int i, int z, int g, int nz, int gpp)
{
    const int zz = z + i / 3 - 1;
    if (zz < 0 || zz >= nz) return -1;
    int gg = g + i % 3 - 1;
    gg = gg < 0 ? gg + gpp : (gg >= gpp ? gg - gpp : gg);
    return zz * gpp + gg;
}

struct PersistArgs {
    const ChannelLaunch *chans;  // the launch table of a batch
    ChannelLaunch one;           // the channel of a launch of one
    const FlowMaps *maps;        // [nchan] the tensor maps of a batch
    FlowMaps one_maps;           // those of a launch of one
    int nchan, nsteps, stages;
    unsigned stage_bytes;        // bytes of one stage (the largest channel's)
    unsigned *counter;           // [2] items and planes taken (zero at launch)
    int *abort;                  // a bounded wait gave up: the launch stops
    unsigned long long wait_ns;  // limit of every bounded wait
    int eager;                   // announce each group as soon as its copies have landed
    int withhold;                // test switch (0 otherwise): the first item's load is withheld
};

constexpr int kMaxGroupRows = 16;

// Per-stage header, written by the load warp before it arms the stage.
struct StageHeader {
    int chan;        // -1: the end of the launch
    int step;        // step within the launch
    int odd;         // parity of the step
    int z, g, y0, k; // plane, row group, first row, rows
    int kind;        // 1: a plane with link masks
    long long abs_step;
    double sh[3];    // shift of the plane's energy sum
    unsigned long long rows[kMaxGroupRows];  // kind 1: RowInfo of the rows
};

constexpr int kMaxConsumerWarps = kTmaMaxThreads / 32 - 2;

// Where the warps read the channels' arguments: the kernel's parameters for
// one channel; for a batch, copies in shared memory of the table's entries in
// use -- one per stage, the load warp's, and the store warp's for the plane it
// looks after -- so that the number of channels costs none of it.  (The
// acquiring loads of the flags drop the SM's L1 contents again and again, so
// an entry in global memory would come from L2 every time.)
constexpr int kEntries = 2;  // besides the stages'
template <bool ONE>
struct FlowTable {
    const PersistArgs &a;
    ChannelLaunch *copies;  // the load warp's, the store warp's, [stages]
    __device__ __forceinline__ const ChannelLaunch &load() const { return at(0); }
    __device__ __forceinline__ const ChannelLaunch &duty() const { return at(1); }
    __device__ __forceinline__ const ChannelLaunch &stage(int st) const { return at(kEntries + st); }
    __device__ __forceinline__ const ChannelLaunch &at(int i) const
    {
        if constexpr (ONE) return a.one;
        else return copies[i];
    }
    __device__ __forceinline__ int count() const { return ONE ? 1 : a.nchan; }
    // entry c of the table in global memory
    __device__ __forceinline__ const ChannelLaunch &entry(int c) const
    {
        if constexpr (ONE) return a.one;
        else return a.chans[c];
    }
    __device__ __forceinline__ const FlowMaps &maps(int c) const
    {
        if constexpr (ONE) return a.one_maps;
        else return a.maps[c];
    }
    // Before the block's first use of channel c's tensor maps, which the host
    // has written to global memory (and may write anew between launches).
    __device__ __forceinline__ void fence_maps(int c, int lane) const
    {
        if constexpr (!ONE) {
            if (lane < (int)(sizeof(FlowMaps) / sizeof(CUtensorMap)))
                asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(
                                 reinterpret_cast<const CUtensorMap *>(a.maps + c) + lane)
                             : "memory");
            __syncwarp();
        }
    }
    // copy i of entry c, by the whole warp that uses it
    __device__ __forceinline__ void fetch(int i, int c, int lane) const
    {
        if constexpr (!ONE) {
            const int *src = reinterpret_cast<const int *>(a.chans + c);
            int *dst = reinterpret_cast<int *>(copies + i);
            __syncwarp();
            for (int w = lane; w < (int)(sizeof(ChannelLaunch) / sizeof(int)); w += 32) dst[w] = src[w];
            __syncwarp();
        }
    }
};

// Shared memory after the stages: full[S], empty[S], freed[S] (8 bytes
// each), per stage the consumer warps' sums, the stage headers, and a batch's
// entries in use.
__host__ __device__ constexpr size_t persist_smem(int stages, size_t stage_bytes, bool batch = false)
{
    return (size_t)stages * (stage_bytes + 24 + sizeof(StageHeader) + sizeof(double) * NP * kMaxConsumerWarps) +
           (batch ? (size_t)(stages + kEntries) * sizeof(ChannelLaunch) : 0);
}

__device__ __forceinline__ void fence_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
// a pause of the store warp longer than between two items of a busy block
constexpr long long kIdleClocks = 8000;

// whether phase `parity` is complete, without waiting (try_wait may suspend)
__device__ __forceinline__ bool mbar_test(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(sm_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ long long ld_acquire(const long long *p)
{
    long long v;
    asm volatile("ld.acquire.gpu.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned *p, unsigned v)
{
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release(long long *p, long long v)
{
    asm volatile("st.release.gpu.global.s64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void persist_raise(const PersistArgs &a, volatile int *s_abort)
{
    *s_abort = 1;
    atomicExch(a.abort, 1);
}

struct FlowShared {
    unsigned char *stages;
    uint64_t *full, *empty, *freed;
    StageHeader *hdr;
    double *sums;  // [S][kMaxConsumerWarps][NP]
    volatile int *abort;
};

// ------------------------------------------------------------------ copies
template <typename T>
__device__ __forceinline__ GroupRows flow_rows(bool odd, bool tex, const StepArgs &p, int A, int y0, int z, int wall)
{
    if (!odd) return group_rows<false, 0>(p, A, y0, z, wall);
    return tex ? group_rows<true, 1>(p, A, y0, z, wall) : group_rows<true, 0>(p, A, y0, z, wall);
}

template <bool LOAD>
__device__ __forceinline__ void tensor_copy(const CUtensorMap &m, unsigned char *stage, int y, int z, int array, uint64_t *bar)
{
    if (LOAD)
        asm volatile(
            "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3, %4, "
            "%5}], [%6];" ::"r"(sm_addr(stage)),
            "l"(&m), "r"(0), "r"(y), "r"(z), "r"(array), "r"(sm_addr(bar))
            : "memory");
    else
        asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.tile.bulk_group [%0, {%1, %1, %2, %3, %4}], [%5];" ::"l"(&m),
                     "r"(0), "r"(y), "r"(z), "r"(array), "r"(sm_addr(stage))
                     : "memory");
}

// Whether a row group moves by tensor copies: any of an even step, and of an
// odd step those whose rows neither wrap in y nor meet a wall.
__device__ __forceinline__ bool flow_plain(const ChannelLaunch &L, bool odd, int wall, int y0, int k)
{
    return !odd || (wall == 0 && y0 > 0 && y0 + k < L.p.ny);
}

// The copies of a row group's directions into (LOAD) or out of a stage, by
// the whole warp.  What bounds a block with few stages is the chain load ->
// collide -> store of a stage, and issuing 19 row copies costs it 1600 cycles
// for the loads and 2600 for the stores (measured, whatever their size);
// tensor copies are one for an even step and nine for an odd one.  Where the
// maps do not apply (rows that do not divide into aligned pieces) one thread
// issues the row copies in a row; 19 threads' copies in one instruction are
// issued one after another at three times the cost.  Groups at a wrap or a
// wall take one direction per thread.
template <typename T, bool LOAD>
__device__ __forceinline__ void flow_copies(const ChannelLaunch &L, const FlowMaps &maps, bool odd, bool tex, int z, int y0,
                                            int k, unsigned char *stage, uint64_t *bar, int lane)
{
    const StepArgs &p = L.p;
    const int wall = plane_wall(p, z);
    const int dir_bytes = L.t.dir_elems * (int)sizeof(T);
    if (flow_plain(L, odd, wall, y0, k)) {
        if (lane != 0) return;
        if (L.tensor) {
            if (!odd) {
                tensor_copy<LOAD>(maps.all, stage, y0, z, 0, bar);
                return;
            }
#pragma unroll
            for (int q = 0; q < 5; ++q) {
                const int a = q == 0 ? 0 : q + 2;  // directions 0, 3, 4, 5, 6 lead the groups of three
                tensor_copy<LOAD>(maps.three, stage + 3 * q * dir_bytes, y0 + lat_ey(a), z + lat_ez(a), 3 * q, bar);
            }
#pragma unroll
            for (int a = 15; a < Q; ++a)
                tensor_copy<LOAD>(maps.one, stage + a * dir_bytes, y0 + lat_ey(a), z + lat_ez(a), a, bar);
            return;
        }
        const uint32_t bytes = (uint32_t)(k * L.t.row_bytes);
        const ptrdiff_t rowb = odd ? L.t.row_bytes : 0, planeb = rowb * p.ny;
        unsigned char *g = static_cast<unsigned char *>(p.pop[0]) + (ptrdiff_t)(z * p.ny + y0) * L.t.row_bytes;
#pragma unroll
        for (int A = 0; A < Q; ++A) {
            unsigned char *ga = g + lat_pos(A) * (ptrdiff_t)L.pop_bytes + lat_ey(A) * rowb + lat_ez(A) * planeb;
            if (LOAD) bulk_g2s(stage + lat_pos(A) * dir_bytes, ga, bytes, bar);
            else bulk_s2g(ga, stage + lat_pos(A) * dir_bytes, bytes);
        }
        return;
    }
    if (lane >= Q) return;
    const GroupRows g = flow_rows<T>(odd, tex, p, lane, y0, z, wall);
    if (!g.bulk) return;
    copy_group<T>(p, L.t, g, k, stage + lat_pos(lane) * dir_bytes, LOAD, bar);
}

// The same for an odd step of a plane with link masks, row by row.  LOAD
// false: only the rows of cells alike are written back.
template <typename T>
__device__ __forceinline__ bool flow_row_source(const StepArgs &p, unsigned long long info, int A, int y, int z, int wall,
                                                int &slot, int &yy, int &zz)
{
    const int ez = lat_ez(A);
    int link = 0;
    if (info & RowInfo::kAlike) {
        if (info & RowInfo::kSolid) link = 3;
        else link = RowInfo::link(info, A);
    } else if (ez != 0 && ez == wall) {
        return false;  // moves per thread
    }
    slot = link == 1 ? lat_opp(A) : (link == 2 ? lat_mir(A) : A);
    yy = link == 0 || link == 2 ? y + lat_ey(A) : y;
    yy = yy < 0 ? yy + p.ny : (yy >= p.ny ? yy - p.ny : yy);
    zz = link == 0 ? z + ez : z;
    return true;
}

template <typename T, bool LOAD>
__device__ __forceinline__ void flow_copies_links(const ChannelLaunch &L, const StageHeader &H, unsigned char *stage,
                                                  uint64_t *bar, int lane)
{
    if (lane >= Q) return;
    const StepArgs &p = L.p;
    const int wall = plane_wall(p, H.z);
    unsigned char *sdir = stage + (size_t)lat_pos(lane) * L.t.dir_elems * sizeof(T);
    for (int j = 0; j < H.k; ++j) {
        const unsigned long long info = H.rows[j];
        if (!LOAD && (!(info & RowInfo::kAlike) || (info & RowInfo::kSolid))) continue;
        int slot, yy, zz;
        if (!flow_row_source<T>(p, info, lane, H.y0 + j, H.z, wall, slot, yy, zz)) continue;
        T *g = static_cast<T *>(p.pop[slot]) + (ptrdiff_t)(zz * p.ny + yy) * p.pitch;
        unsigned char *s = sdir + (size_t)j * L.t.row_bytes;
        if (LOAD) bulk_g2s(s, g, (uint32_t)L.t.row_bytes, bar);
        else bulk_s2g(g, s, (uint32_t)L.t.row_bytes);
    }
}

// ------------------------------------------------------------------ loads
// Wait until the neighbours of the item are done with the step before and
// the step kRing before it is logged.  Warp-uniform; false: gave up.
__device__ __forceinline__ bool flow_wait_item(const PersistArgs &a, const ChannelLaunch &L, const ItemPos &it,
                                               long long abs_step, int lane, volatile int *s_abort)
{
    const unsigned *flag = nullptr;
    const bool ring_lane = lane == 31 && it.step >= L.p.ring;
    if (it.step > 0 && lane < 9) {
        const int n = flow_neighbour(lane, it.z, it.g, L.p.nz, L.t.gpp);
        if (n >= 0) flag = L.flags + n;
    }
    bool ok = !flag && !ring_lane;
    auto poll = [&]() {
        if (flag) ok = ld_acquire(flag) >= (unsigned)it.step;
        else if (ring_lane) ok = ld_acquire(L.p.step_ctr) >= abs_step - L.p.ring + 1;
    };
    if (!ok) poll();
    if (__all_sync(0xffffffffu, ok)) return true;
    const unsigned long long t0 = globaltimer_ns();
    for (;;) {
        if (!ok) poll();
        if (__all_sync(0xffffffffu, ok)) return true;
        const bool late = globaltimer_ns() - t0 > a.wait_ns;
        const bool stop = *s_abort || *(volatile int *)a.abort;
        if (__any_sync(0xffffffffu, late || stop)) return false;
    }
}

// Wait until the steps before `step` are logged.  Warp-uniform; false: gave up.
__device__ __forceinline__ bool flow_wait_counter(const PersistArgs &a, const long long *ctr, long long step,
                                                  volatile int *s_abort)
{
    if (__all_sync(0xffffffffu, ld_acquire(ctr) >= step)) return true;
    const unsigned long long t0 = globaltimer_ns();
    for (;;) {
        if (__all_sync(0xffffffffu, ld_acquire(ctr) >= step)) return true;
        const bool late = globaltimer_ns() - t0 > a.wait_ns;
        if (__any_sync(0xffffffffu, late || *s_abort || *(volatile int *)a.abort)) return false;
    }
}

template <typename T, bool ONE>
__device__ __forceinline__ void flow_loads(const PersistArgs &a, const FlowTable<ONE> &chans, const FlowShared &sm,
                                           int lane)
{
    const int S = a.stages;
    volatile int *s_abort = sm.abort;
    unsigned loaded = 0;  // bit st: a load into stage st was issued (its phase is the last one armed)
    unsigned phase = 0;   // bit st: parity of that phase
    auto take = [&]() { return lane == 0 ? atomicAdd(a.counter, 1u) : 0u; };
    unsigned hn = take();
    int c = 0, st = 0, round = 0;
    bool run = true;
    unsigned citems = chans.entry(0).item_end;  // end of channel c's items
    chans.fetch(0, 0, lane);
    chans.fence_maps(0, lane);  // the store warp's uses follow the load warp's through the stage's barriers
    // the stage `st`, free for new contents
    auto stage_free = [&]() {
        if (round == 0) return true;
        return mbar_wait_bounded(sm.freed + st, (uint32_t)((round - 1) & 1), a.wait_ns, s_abort);
    };
    while (run) {
        const unsigned h = __shfl_sync(0xffffffffu, hn, 0);
        hn = take();  // the next item, fetched while this one is waited for and issued
        if (h >= citems) {
            do {
                if (++c >= chans.count()) break;
                citems = chans.entry(c).item_end;
            } while (h >= citems);
            if (c >= chans.count()) break;
            chans.fetch(0, c, lane);
            chans.fence_maps(c, lane);
        }
        const ChannelLaunch &L = chans.load();
        const ItemPos it = flow_item(h - L.item_first, L.depth, L.lag, L.flow_groups, L.t.gpp, a.nsteps);
        if (it.step < 0) continue;
        const long long abs_step = __ldcg(L.base) + it.step;
        const bool odd = abs_step & 1;
        const int y0 = it.g * L.t.k, k = min(L.t.k, L.p.ny - y0);
        const int wall = plane_wall(L.p, it.z);
        const int kind = L.p.band_of[it.z] >= 0;
        const bool tex = L.textured || kind;
        const int ncopies = odd && tex && wall != 0 ? Q - 5 : Q;  // a textured wall's five links move per thread
        // the neighbours first: usually long done, so their flags are read
        // while the stage is still in use
        bool ok = flow_wait_item(a, L, it, abs_step, lane, s_abort);
        const bool by_rows = odd && kind;
        unsigned long long info = 0;  // RowInfo of row y0 + lane
        // row copies of the item (a tensor copy counts the rows of its box
        // beyond the plane's last row too)
        int nrows = ncopies * (L.tensor && flow_plain(L, odd, wall, y0, k) ? L.t.k : k);
        if (kind) {
            if (lane < k) info = L.p.link_rows[(size_t)L.p.band_of[it.z] * L.p.ny + y0 + lane];
            if (odd) {
                nrows = 0;
                for (int j = 0; j < k; ++j)
                    nrows += (__shfl_sync(0xffffffffu, info, j) & RowInfo::kAlike) || wall == 0 ? Q : Q - 5;
            }
        }
        const double sh = ok && lane < 3 ? __ldcg(shift_entry(L.p, abs_step) + it.z * 3 + lane) : 0.0;
        if (ok) ok = __all_sync(0xffffffffu, stage_free());
        if (!ok) {
            if (lane == 0) persist_raise(a, s_abort);
            break;
        }
        // test switch: the first item is neither armed nor loaded, so its
        // consumers' wait runs out with no copy in flight
        if (!(a.withhold != 0 && h == 0)) {
            if (!ONE && (round == 0 || sm.hdr[st].chan != c)) chans.fetch(kEntries + st, c, lane);
            if (lane < 3) sm.hdr[st].sh[lane] = sh;
            if (lane < k) sm.hdr[st].rows[lane] = info;
            __syncwarp();
            const size_t bytes = (size_t)nrows * L.t.row_bytes;
            if (lane == 0) {
                StageHeader &H = sm.hdr[st];
                H.chan = c;
                H.step = it.step;
                H.odd = odd;
                H.z = it.z;
                H.g = it.g;
                H.y0 = y0;
                H.k = k;
                H.kind = kind;
                H.abs_step = abs_step;
                mbar_expect_tx(sm.full + st, (uint32_t)bytes);
            }
            __syncwarp();
            fence_async_global();  // the neighbours' stores, seen through their flags, before these loads
            unsigned char *stage = sm.stages + (size_t)st * a.stage_bytes;
            if (by_rows) flow_copies_links<T, true>(L, sm.hdr[st], stage, sm.full + st, lane);
            else flow_copies<T, true>(L, chans.maps(c), odd, tex, it.z, y0, k, stage, sm.full + st, lane);
            loaded |= 1u << st;
            phase = (phase & ~(1u << st)) | ((unsigned)(round & 1) << st);
        }
        if (++st == S) st = 0, ++round;
    }
    // the end of the launch
    if (!*s_abort && stage_free() && lane == 0) {
        sm.hdr[st].chan = -1;
        mbar_arrive(sm.full + st);
    }
    __syncwarp();
    if (*s_abort)  // loads still landing in shared memory (bounded; an issued load completes)
        for (int q = 0; q < S; ++q)
            if ((loaded >> q) & 1u) mbar_wait_bounded(sm.full + q, (phase >> q) & 1u, a.wait_ns, nullptr);
}

// ------------------------------------------------------------------ stores
// Sum of a plane whose groups are all counted, and for the last plane of the
// step the tail: the whole store warp.
__device__ __forceinline__ void flow_plane_done(const PersistArgs &a, const ChannelLaunch &L, long long abs_step, int z,
                                                int lane, volatile int *s_abort)
{
    const StepArgs &p = L.p;
    const int ring = (int)(abs_step & (p.ring - 1)), gpp = L.t.gpp;
    __threadfence();
    const int v = lane & 7;
    const double *part = L.fpart + ((size_t)ring * p.nz + z) * gpp * NP + v;
    double s = 0.0;
    int b = lane >> 3;
    for (; b + 28 < gpp; b += 32) {  // eight loads in flight
        double x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = __ldcg(part + (size_t)(b + 4 * i) * NP);
#pragma unroll
        for (int i = 0; i < 8; ++i) s += x[i];
    }
    for (; b < gpp; b += 4) s += __ldcg(part + (size_t)b * NP);
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    double *sums = L.fsums + (size_t)ring * p.nz * NP;
    if (lane < NP) sums[(size_t)z * NP + lane] = s;
    __syncwarp();
    unsigned ticket = 0;
    if (lane == 0) {
        L.fctr[(size_t)ring * p.nz + z] = 0;
        __threadfence();
        ticket = atomicAdd(L.ftotal + ring, 1u);
    }
    ticket = __shfl_sync(0xffffffffu, ticket, 0);
    if (ticket != (unsigned)p.nz - 1) return;
    __threadfence();
    // the tails run in the order of the steps
    if (!flow_wait_counter(a, p.step_ctr, abs_step, s_abort)) {
        if (lane == 0) persist_raise(a, s_abort);
        return;
    }
    // constant flow rate: the next step's force first, on its own counter;
    // the logs are off the path of the consumers that wait for it
    if (p.const_q) {
        double f[2] = {0.0, 0.0};
        for (int q = lane; q < p.nz; q += 32) {
            f[0] += __ldcg(sums + (size_t)q * NP + 6);
            f[1] += __ldcg(sums + (size_t)q * NP + 7);
        }
        warp_sum<2>(f);
        if (lane == 0) {
            p.force[(abs_step + 1) & 1] = tail_force<false>(p, f[0], f[1]);
            st_release(L.force_ctr, abs_step + 1);
        }
    }
    double t[6] = {0, 0, 0, 0, 0, 0};
    tail_planes(p, abs_step, 0, sums, lane, 32, t);
    warp_sum<6>(t);
    __syncwarp();
    if (lane == 0) {
        tail_record<false>(p, abs_step, p.const_q ? __ldcg(p.force + (abs_step & 1)) : p.gx, 0, sums, t, !p.const_q);
        L.ftotal[ring] = 0;
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) st_release(p.step_ctr, abs_step + 1);
}

template <typename T, bool ONE>
__device__ __forceinline__ void flow_stores(const PersistArgs &a, const FlowTable<ONE> &chans, const FlowShared &sm,
                                            int lane, int nwarps)
{
    const int S = a.stages;
    volatile int *s_abort = sm.abort;
    // the group whose stores were committed last, not yet announced
    bool pend = false;
    int pz = 0, pg = 0, pstep = 0;
    long long pabs = 0;
    unsigned *pflag = nullptr, *pcount = nullptr;
    // where it is announced: for one channel worked out then, which is off the
    // path of the stage; a batch's entry is gone by then
    auto address = [&](const ChannelLaunch &L) {
        pflag = L.flags + (size_t)pz * L.t.gpp + pg;
        pcount = L.fctr + (size_t)(pabs & (L.p.ring - 1)) * L.p.nz + pz;
    };
    // raise its flag (its copies have landed) and count it in its plane,
    // without waiting for either
    auto announce = [&]() {
        if (ONE) address(chans.at(0));
        if (lane < Q) fence_async_global();
        __syncwarp();
        if (lane == 0) {
            __threadfence();
            *reinterpret_cast<volatile unsigned *>(pflag) = (unsigned)pstep + 1u;
            asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(pcount) : "memory");
        }
    };
    // The plane to look after.  (The warp that counts a plane's last group
    // could sum it instead, but then every count needs its answer, and the sum
    // delays that block's stores: 628x314x200 FP64 7 % slower.)
    // One plane at a time, and none beside it: a warp in a step's tail waits for
    // the tail before, whose planes are all counted and each held by a warp
    // that holds no other, so nobody waits in a circle.  (With the next plane
    // taken ahead a batch of 450 channels ran into the wait limit: a warp's
    // first plane lacked a group whose block waited for the second.)
    int dc = 0, ds = 0, dz = 0;
    unsigned dfirst = 0;  // place in the sequence of channel dc's first plane
    bool dfree = false;   // the counter of the plane is this step's
    int dcopy = -1;       // channel of the copy
    auto take_duty = [&]() {
        unsigned d = 0;
        if (lane == 0) d = atomicAdd(a.counter + 1, 1u);
        d = __shfl_sync(0xffffffffu, d, 0);
        for (; dc < chans.count(); ++dc) {
            const unsigned nz = (unsigned)chans.entry(dc).p.nz, n = nz * (unsigned)a.nsteps;
            if (d - dfirst < n) {
                ds = (int)((d - dfirst) / nz);
                dz = (int)(d - dfirst - (unsigned)ds * nz);
                break;
            }
            dfirst += n;
        }
        if (!ONE && dc < chans.count() && dc != dcopy) chans.fetch(1, dcopy = dc, lane);
        dfree = false;
    };
    take_duty();
    // true: the plane is done, and the next one taken
    auto service = [&]() {
        if (dc >= chans.count()) return false;
        const ChannelLaunch &L = chans.duty();
        const long long abs_step = __ldcg(L.base) + ds;
        if (!dfree) {  // the step that had the counter before has cleared it when it is logged
            if (!__all_sync(0xffffffffu, ds < L.p.ring || ld_acquire(L.p.step_ctr) > abs_step - L.p.ring)) return false;
            dfree = true;
        }
        const unsigned n = ld_acquire(L.fctr + (size_t)(abs_step & (L.p.ring - 1)) * L.p.nz + dz);
        if (!__all_sync(0xffffffffu, n == (unsigned)L.t.gpp)) return false;
        flow_plane_done(a, L, abs_step, dz, lane, s_abort);
        take_duty();
        return true;
    };
    int st = 0;
    uint32_t par = 0;
    unsigned count = 0;
    for (;;) {
        // Wait for the stage's consumers.  Meanwhile announce the group
        // before: its copies land before the next stage is done, and a fence
        // behind newer copies would wait for those too.  The planes, whose
        // counters are a round trip to L2 away, only after a pause longer
        // than the usual one between two items, unless the next items depend
        // on them (eager).
        bool ok = true, end = false;
        unsigned long long t0 = 0;
        const long long c0 = clock64();
        for (bool first = true;;) {
            bool ready = mbar_test(sm.full + st, par);
            if (__all_sync(0xffffffffu, ready)) {
                end = sm.hdr[st].chan < 0;
                ready = end || mbar_test(sm.empty + st, par);
            }
            if (__all_sync(0xffffffffu, ready)) break;
            if (pend) {
                bulk_wait_all();
                announce();
                pend = false;
                continue;
            }
            if (!__all_sync(0xffffffffu, a.eager || clock64() - c0 > kIdleClocks)) continue;
            service();
            if (first) t0 = globaltimer_ns(), first = false;
            const bool late = globaltimer_ns() - t0 > a.wait_ns;
            if (__any_sync(0xffffffffu, late || *s_abort)) {
                ok = false;
                break;
            }
        }
        if (!ok) {
            if (lane == 0) persist_raise(a, s_abort);
            break;
        }
        if (end) break;
        if (pend) {
            bulk_wait_all();
            announce();
        }
        const StageHeader &H = sm.hdr[st];
        const ChannelLaunch &L = chans.stage(st);
        const int hc = H.chan, hz = H.z, hg = H.g, hs = H.step;
        const long long habs = H.abs_step;
        unsigned char *stage = sm.stages + (size_t)st * a.stage_bytes;
        if (!(H.odd && H.kind))
            flow_copies<T, false>(L, chans.maps(hc), H.odd != 0, L.textured, hz, H.y0, H.k, stage, nullptr, lane);
        else flow_copies_links<T, false>(L, H, stage, nullptr, lane);
        bulk_commit();
        // the warps' sums, in warp order
        {
            const double *w = sm.sums + (size_t)st * kMaxConsumerWarps * NP + (lane & 7);
            double s = 0.0;
            for (int q = lane >> 3; q < nwarps; q += 4) s += w[q * NP];
            s += __shfl_xor_sync(0xffffffffu, s, 8);
            s += __shfl_xor_sync(0xffffffffu, s, 16);
            const int ring = (int)(habs & (L.p.ring - 1));
            if (lane < NP) L.fpart[(((size_t)ring * L.p.nz + hz) * L.t.gpp + hg) * NP + lane] = s;
        }
        pz = hz;
        pg = hg;
        pstep = hs;
        pabs = habs;
        if (!ONE) address(L);
        bulk_wait_read_all();  // the stores have read the stage
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.freed + st);
        pend = true;
        if (++st == S) st = 0, par ^= 1u;
        if ((++count & 7u) == 0) service();  // also where the next stage is always ready
    }
    bulk_wait_all();
    if (pend && !__any_sync(0xffffffffu, *s_abort)) announce();
    // the rest of the planes
    unsigned long long t0 = globaltimer_ns();
    while (dc < chans.count()) {
        if (service()) t0 = globaltimer_ns();
        const bool late = globaltimer_ns() - t0 > a.wait_ns;
        if (__any_sync(0xffffffffu, late || *s_abort || *(volatile int *)a.abort)) {
            if (dc < chans.count() && lane == 0) persist_raise(a, s_abort);
            break;
        }
    }
}

// ------------------------------------------------------------------ cells
// A row group of a plane with link masks from the stage, one cell per thread
// (links_cell; the odd step's shifted elements at x-1 and x+1 wrap around
// the row).
template <typename T, bool ODD, bool CONSTQ>
__device__ __forceinline__ void persist_links(const StepArgs &p, const StageHeader &H, T *sb, int dstride, double G,
                                              const double (&sh)[3], double (&acc)[NP], int nc)
{
    const int nx = p.nx, y0 = H.y0, k = H.k, z = H.z;
    const int wall = plane_wall(p, z);
    for (int c = threadIdx.x; c < k * nx; c += nc) {
        const int j = c / nx, x = c - j * nx, y = y0 + j;
        float racc[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) racc[q] = 0.f;
        const Nbr n = make_nbr(x, y, z, nx, p.ny, p.pitch);
        const int om = x == 0 ? nx - 1 : -1, op = x == nx - 1 ? 1 - nx : 1;
        const unsigned long long info = H.rows[j];
        const bool alike = (info & RowInfo::kAlike) != 0;
        const unsigned lk = alike ? RowInfo::mask(info) : cell_links(p.band_of, p.links, nx, p.ny, x, y, z);
        links_cell<T, ODD, CONSTQ>(p, n, wall, lk, sb + (size_t)j * p.pitch + x, dstride, G, sh[0], sh[1], sh[2], acc,
                                   racc, om, op, alike);
#pragma unroll
        for (int q = 0; q < NP; ++q) acc[q] += (double)racc[q];
    }
}

// Sum of the warp's NP values by halving: the lanes exchange half of their
// values, then a quarter, an eighth; 9 exchanges instead of 40.  Lane l ends
// with the sum of value l >> 2, the same in its group of four.
__device__ __forceinline__ double warp_sum8(const double (&v)[NP], int lane)
{
    static_assert(NP == 8, "eight values");
    double a[4], b[2];
    const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double mine = h4 ? v[4 + i] : v[i], other = h4 ? v[i] : v[4 + i];
        a[i] = mine + __shfl_xor_sync(0xffffffffu, other, 16);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double mine = h3 ? a[2 + i] : a[i], other = h3 ? a[i] : a[2 + i];
        b[i] = mine + __shfl_xor_sync(0xffffffffu, other, 8);
    }
    const double mine = h2 ? b[1] : b[0], other = h2 ? b[0] : b[1];
    double c = mine + __shfl_xor_sync(0xffffffffu, other, 4);
    c += __shfl_xor_sync(0xffffffffu, c, 2);
    c += __shfl_xor_sync(0xffffffffu, c, 1);
    return c;
}

template <typename T, bool ODD, bool Q_, bool LINKS>
__device__ __forceinline__ void flow_cells(const ChannelLaunch &L, const StageHeader &H, T *sb, double G,
                                           const double (&sh)[3], double (&acc)[NP], int nc)
{
    using LpT = typename std::conditional<std::is_same<T, double>::value, float, T>::type;
    const StepArgs &p = L.p;
    const int dstride = L.t.dir_elems, z = H.z;
    if constexpr (LINKS) {
        if (H.kind) {
            persist_links<T, ODD, Q_>(p, H, sb, dstride, G, sh, acc, nc);
            return;
        }
    }
    [[maybe_unused]] const LpParams lk = lp_params<LpT>((float)p.omega, (float)G);
    if (L.textured) consume_group<T, ODD, Q_, true>(p, lk, sb, dstride, H.y0, H.k, z, G, sh, acc, nc);
    else consume_group<T, ODD, Q_, false>(p, lk, sb, dstride, H.y0, H.k, z, G, sh, acc, nc);
}

template <typename T, bool ANYQ, bool LINKS, bool ONE>
__device__ __forceinline__ void flow_consumers(const PersistArgs &a, const FlowTable<ONE> &chans, const FlowShared &sm,
                                               int nc)
{
    const int S = a.stages, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    volatile int *s_abort = sm.abort;
    int st = 0;
    uint32_t par = 0;
    for (;;) {
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(sm.full + st, par, a.wait_ns, s_abort))) {
            if (lane == 0) persist_raise(a, s_abort);
            return;
        }
        const StageHeader &H = sm.hdr[st];
        if (H.chan < 0) return;
        const ChannelLaunch &L = chans.stage(st);
        const StepArgs &p = L.p;
        const bool q = ANYQ && p.const_q != 0;  // a launch without constant-Q channels compiles no such path
        double G = p.gx;
        if (q) {  // the force of the step: after the tail of the step before
            if (!flow_wait_counter(a, L.force_ctr, H.abs_step, s_abort)) {
                if (lane == 0) persist_raise(a, s_abort);
                return;
            }
            G = __ldcg(p.force + (H.abs_step & 1));
        }
        const double sh[3] = {H.sh[0], H.sh[1], H.sh[2]};
        T *sb = reinterpret_cast<T *>(sm.stages + (size_t)st * a.stage_bytes);
        double acc[NP];
#pragma unroll
        for (int r = 0; r < NP; ++r) acc[r] = 0.0;
        if (H.odd) {
            if (q) flow_cells<T, true, ANYQ, LINKS>(L, H, sb, G, sh, acc, nc);
            else flow_cells<T, true, false, LINKS>(L, H, sb, G, sh, acc, nc);
            // results written by the threads themselves (wall links, link
            // masks) before other SMs' bulk loads of them
            if (H.kind || L.textured) fence_async_global();
        } else {
            if (q) flow_cells<T, false, ANYQ, LINKS>(L, H, sb, G, sh, acc, nc);
            else flow_cells<T, false, false, LINKS>(L, H, sb, G, sh, acc, nc);
        }
        const double s = warp_sum8(acc, lane);
        if ((lane & 3) == 0) sm.sums[((size_t)st * kMaxConsumerWarps + warp) * NP + (lane >> 2)] = s;
        fence_async_smem();  // this thread's shared-memory writes -> visible to the bulk stores
        __syncwarp();
        if (lane == 0) mbar_arrive(sm.empty + st);
        if (++st == S) st = 0, par ^= 1u;
    }
}

// ------------------------------------------------------------------ kernel
// Before each launch: the flags of every channel's groups and the item
// counter cleared, the channels' step counters noted.
static __device__ __forceinline__ void persist_reset(const ChannelLaunch &L, unsigned tid, unsigned n)
{
    for (unsigned i = tid; i < L.flow_groups; i += n) L.flags[i] = 0;
    if (tid == 0) *L.base = *L.force_ctr = *L.p.step_ctr;
}
static __global__ void persist_reset_kernel(const ChannelLaunch *__restrict__ chans, int nchan, unsigned *counter)
{
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, n = gridDim.x * blockDim.x;
    for (int c = 0; c < nchan; ++c) persist_reset(chans[c], tid, n);
    if (tid < 2) counter[tid] = 0;
}
static __global__ void persist_reset_one_kernel(const ChannelLaunch L, unsigned *counter)
{
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
    persist_reset(L, tid, gridDim.x * blockDim.x);
    if (tid < 2) counter[tid] = 0;
}

// ANYQ: some channel runs with a constant flow rate; LINKS: some plane has
// link masks; ONE: a launch of one channel; WIDE: the form for more threads
// than the dense step form's.
template <typename T, bool ANYQ, bool LINKS, bool ONE, bool WIDE>
__global__ void __launch_bounds__(WIDE ? kTmaMaxThreads : TmaBounds<T, ANYQ>::threads,
                                  WIDE ? 1 : TmaBounds<T, ANYQ>::min_blocks)
    persist_batch_kernel(const __grid_constant__ PersistArgs a)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    const int S = a.stages, nc = blockDim.x - 64;
    FlowShared sm;
    sm.stages = smem;
    sm.full = reinterpret_cast<uint64_t *>(smem + (size_t)S * a.stage_bytes);
    sm.empty = sm.full + S;
    sm.freed = sm.empty + S;
    sm.sums = reinterpret_cast<double *>(sm.freed + S);
    sm.hdr = reinterpret_cast<StageHeader *>(sm.sums + (size_t)S * kMaxConsumerWarps * NP);
    sm.abort = &s_abort;
    const FlowTable<ONE> chans{a, reinterpret_cast<ChannelLaunch *>(sm.hdr + S)};
    if (threadIdx.x == 0) {
        for (int st = 0; st < S; ++st) {
            mbar_init(sm.full + st, 1);
            mbar_init(sm.empty + st, nc / 32);
            mbar_init(sm.freed + st, 1);
        }
        fence_mbar_init();
        s_abort = 0;
    }
    __syncthreads();
    if ((int)threadIdx.x >= nc + 32) flow_stores<T, ONE>(a, chans, sm, threadIdx.x - nc - 32, nc / 32);
    else if ((int)threadIdx.x >= nc) flow_loads<T, ONE>(a, chans, sm, threadIdx.x - nc);
    else flow_consumers<T, ANYQ, LINKS, ONE>(a, chans, sm, nc);
}

template <typename T, bool ANYQ, bool LINKS, bool ONE>
const void *persist_form(int threads)
{
    if constexpr (TmaBounds<T, ANYQ>::has_dense)
        if (threads <= TmaBounds<T, ANYQ>::threads) return (const void *)persist_batch_kernel<T, ANYQ, LINKS, ONE, false>;
    return (const void *)persist_batch_kernel<T, ANYQ, LINKS, ONE, true>;
}

template <typename T, bool ONE>
const void *persist_kernel_of(bool any_q, bool links, int threads)
{
    if (any_q) return links ? persist_form<T, true, true, ONE>(threads) : persist_form<T, true, false, ONE>(threads);
    return links ? persist_form<T, false, true, ONE>(threads) : persist_form<T, false, false, ONE>(threads);
}

template <typename T, bool ONE>
int persist_set_smem_attr(int threads, size_t bytes, bool any_q, bool links)
{
    return cudaFuncSetAttribute(persist_kernel_of<T, ONE>(any_q, links, threads),
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess
               ? 0
               : -1;
}

template <typename T, bool ONE>
int persist_occupancy(int threads, size_t smem, bool any_q, bool links)
{
    int n = 0;
    if (threads > kTmaMaxThreads) return 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, persist_kernel_of<T, ONE>(any_q, links, threads), threads,
                                                         smem) == cudaSuccess
               ? n
               : 0;
}

// The reset and the launch of one chunk of steps.
template <typename T, bool ONE>
cudaError_t launch_persist(const PersistArgs &a, unsigned groups, int grid, int threads, size_t smem, bool any_q,
                           bool links, cudaStream_t s)
{
    const unsigned rb = (groups + 1023) / 1024, blocks = rb < 64 ? rb : 64;
    if (ONE) persist_reset_one_kernel<<<blocks, 256, 0, s>>>(a.one, a.counter);
    else persist_reset_kernel<<<blocks, 256, 0, s>>>(a.chans, a.nchan, a.counter);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    void *args[] = {const_cast<PersistArgs *>(&a)};
    return cudaLaunchKernel(persist_kernel_of<T, ONE>(any_q, links, threads), dim3(grid), dim3(threads), args, smem, s);
}

// The entry points of one precision, for one channel or a batch (one
// translation unit each).
#define DNSLBM_PERSIST_UNIT(T, ONE, SUFFIX)                                                                         \
    int persist_prepare_##SUFFIX(int threads, size_t smem, bool any_q, bool links)                                  \
    {                                                                                                               \
        return persist_set_smem_attr<T, ONE>(threads, smem, any_q, links);                                          \
    }                                                                                                               \
    int persist_occupancy_##SUFFIX(int threads, size_t smem, bool any_q, bool links)                                \
    {                                                                                                               \
        return persist_occupancy<T, ONE>(threads, smem, any_q, links);                                              \
    }                                                                                                               \
    cudaError_t launch_persist_##SUFFIX(const PersistArgs &a, unsigned groups, int grid, int threads, size_t smem,  \
                                        bool any_q, bool links, cudaStream_t s)                                     \
    {                                                                                                               \
        return launch_persist<T, ONE>(a, groups, grid, threads, smem, any_q, links, s);                             \
    }

}  // namespace dnslbm
