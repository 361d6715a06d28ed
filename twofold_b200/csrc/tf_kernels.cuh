// The step kernels. Each kernel walks whole worlds with thread groups: a group (one warp, or 64 to 512
// threads) steps one world at a time, and groups take worlds in largest-first order from a per-launch
// counter, so small worlds pack many to an SM and large ones get whole CTAs. Within a world a group's threads
// split bodies, candidates or one color's contacts, with a group barrier between dependent phases, over shared memory
// when the world fits the group's slice and over L1/L2-cached scratch otherwise. Worlds of more than 1024 bodies have a
// cluster of CTAs each. Work that the reference does in one sequential pass whose result depends on order (coloring,
// unions, joints, contacts solved one at a time) runs in rounds or levels that give each item what the pass gives it;
// the wake flood, which is rare, runs on the group's first thread in the reference's order.
//
// Kernel sequence of one step (src/world.cpp:1564-1727):
//   k_broadphase   growth, body-pair and half-space candidates, sorted unique keys (world.cpp:752-870)
//   k_narrowphase  reuse or collide each candidate, carry impulses, merge       (world.cpp:872-993)
//   k_wake         wake sleeping bodies touched by moving ones                  (world.cpp:705-735)
//   k_prepare      step state, active/fast/impact lists, prepare, axes, colors   (world.cpp:1589-1657)
//   k_refresh      fast pairs collided again before substeps 2..n               (world.cpp:1658-1668)
//   k_substep      integrate, warm start, solve, integrate, relax               (world.cpp:1669-1680)
//   k_finish       restitution, limits, refit bounds, sweep test, sleep         (world.cpp:1682-1726)
#pragma once

#include "tf_batch.cuh"
#include "tf_continuous.cuh"
#include "tf_joint.cuh"
#include "tf_planar.cuh"
#include "tf_solver.cuh"
#include "tf_tape.h"

namespace tfb {

constexpr int kMaxBlock = 512;
constexpr int kMaxGroups = kMaxBlock / 32;
constexpr uint32_t kMaxCluster = 16;  // CTAs of a cluster that steps a big world
constexpr uint32_t kDevPairOverflow = 1u << 0, kDevContactOverflow = 1u << 1, kDevNonFinite = 1u << 2,
                   kDevTimeout = 1u << 3, kDevUnsupported = 1u << 4, kDevListOverflow = 1u << 6;

// Where each launch of a step takes its worlds from (one counter each, zeroed when the step starts).
// Up to kMaxSubsteps substeps per step.
constexpr int kMaxSubsteps = 32;
enum WorkSlot : int {
    kSlotBroad = 0, kSlotNarrow = 1, kSlotWake = 2, kSlotPrepare = 3,
    kSlotRefresh = 4,                            // + substep index
    kSlotSubstep = kSlotRefresh + kMaxSubsteps,  // + substep index
    kSlotFinish = kSlotSubstep + kMaxSubsteps,
    kSlotBroadFinish = kSlotFinish + 1,                  // the big worlds' half of the broadphase
    kSlotCandItems = kSlotBroadFinish + 1,               // + pair class: candidate items of that class
    kSlotFastItems = kSlotCandItems + kPairClasses,       // + pair class: fast contacts of that class; + kPairClasses:
                                                          // the other active contacts of refreshed worlds
    kSlotTape = kSlotFastItems + kPairClasses + 1,      // the recording kernel's world counter
    // The flat solve of batches of many worlds (k_substep_flat): each color's contacts over every world, the
    // impact colors' likewise, the most colors, impact colors and levels of one-at-a-time contacts any world
    // has, and the grid barrier.
    kSlotFlatColor = kSlotTape + 1,                    // + color: contacts of that color in all worlds
    kSlotFlatImpact = kSlotFlatColor + kColors,        // + color
    kSlotFlatMaxColors = kSlotFlatImpact + kColors,
    kSlotFlatMaxImpact = kSlotFlatMaxColors + 1,
    kSlotFlatMaxRestLevels = kSlotFlatMaxImpact + 1,
    kSlotFlatMaxImpactRestLevels = kSlotFlatMaxRestLevels + 1,
    kSlotFlatBarrier = kSlotFlatMaxImpactRestLevels + 1,  // arrivals, then barriers passed
    kSlotRoomContacts = kSlotFlatBarrier + 2,  // active contacts of the worlds that rooms suit
    kSlotFast = kSlotRoomContacts + 1,  // whether any world has fast contacts (bit 0), any of solid bodies (bit 1)
    kSlotCount = kSlotFast + 1
};

// A group of threads that steps one world at a time: one warp, several warps, the whole CTA, or (Cluster) the CTAs
// of a thread-block cluster.
template <bool Cluster>
struct GroupOf {
    static constexpr bool kCluster = Cluster;
    uint32_t tid, size, id, count, lane, warp, warps;

    __device__ __forceinline__ void sync() const {
        if constexpr (Cluster) {
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        } else if (count == 1) {
            __syncthreads();
        } else if (size == 32) {
            __syncwarp();
        } else {
            asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "r"(size) : "memory");
        }
    }
    // The group's one copy of a shared variable: a cluster's lies in its first CTA's shared memory.
    template <class T>
    __device__ __forceinline__ T* shared(T* p) const {
        if constexpr (Cluster) {
            uint64_t out;
            asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"((uint64_t)p), "r"(0));
            return reinterpret_cast<T*>(out);
        } else {
            return p;
        }
    }
    // A barrier (as sync) that also tells every thread whether p held on any thread of the group. Clusters tell it
    // through flag, a word of the group's shared memory that is zero beforehand and left as it is.
    __device__ __forceinline__ bool any(bool p, uint32_t* flag) const {
        if constexpr (Cluster) {
            if (__any_sync(0xffffffffu, p) && lane == 0) { *(volatile uint32_t*)flag = 1u; }
            sync();
            return *(volatile uint32_t*)flag != 0u;
        }
        if (count == 1) { return __syncthreads_or(p) != 0; }
        if (size == 32) {
            __syncwarp();
            return __any_sync(0xffffffffu, p);
        }
        uint32_t r;
        asm volatile(
            "{\n\t.reg .pred in, out;\n\tsetp.ne.u32 in, %1, 0;\n\tbar.red.or.pred out, %2, %3, in;\n\t"
            "selp.u32 %0, 1, 0, out;\n\t}"
            : "=r"(r)
            : "r"((uint32_t)p), "r"(id + 1), "r"(size)
            : "memory");
        return r != 0;
    }
};
using Group = GroupOf<false>;

// blockDim.x is a multiple of size, size a multiple of 32, at most kMaxGroups groups.
__device__ __forceinline__ Group makeGroup(uint32_t size) {
    Group g;
    g.size = size;
    g.count = blockDim.x / size;
    g.id = threadIdx.x / size;
    g.tid = threadIdx.x % size;
    g.lane = threadIdx.x & 31;
    g.warp = g.tid >> 5;
    g.warps = size >> 5;
    return g;
}

__device__ __forceinline__ uint32_t clusterRank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t clusterSize() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

__device__ __forceinline__ GroupOf<true> makeClusterGroup() {
    GroupOf<true> g;
    g.size = blockDim.x * clusterSize();
    g.count = 1;
    g.id = 0;
    g.tid = clusterRank() * blockDim.x + threadIdx.x;
    g.lane = threadIdx.x & 31;
    g.warp = g.tid >> 5;
    g.warps = g.size >> 5;
    return g;
}

// How a launch hands out worlds. A CTA takes worlds in largest-first order (B.order) and steps a world with
// more than bigBodies bodies with all its threads; once it draws a world at or under that size every later
// world is too, and its warps go on alone, a world each. Each mode has its own shared-memory staging
// capacity: the whole dynamic allocation for a CTA-sized group, an equal share per warp otherwise.
struct StageSizes {
    uint32_t bodies, contacts;
};
struct Split {
    uint32_t bigBodies;
    StageSizes big, small;
    uint32_t smemBytes;
    uint32_t firstWorld;  // the worlds before it in largest-first order belong to another launch (forBigWorlds)
};

__device__ __forceinline__ uint32_t grabWarp(uint32_t* counter) {
    uint32_t v = 0;
    if ((threadIdx.x & 31) == 0) { v = atomicAdd(counter, 1u); }
    return __shfl_sync(0xffffffffu, v, 0);
}

// Takes one place from counters[c] for each calling thread and returns it: one atomic for the threads of a warp that
// share a counter (most contacts and pairs of a world are of one class, and a cluster's counters are another SM's
// shared memory).
__device__ __forceinline__ uint32_t takePlace(uint32_t* counters, uint32_t c) {
    const uint32_t active = __activemask(), lane = threadIdx.x & 31;
    const uint32_t same = __match_any_sync(active, c);
    const int leader = __ffs(same) - 1;
    uint32_t at = 0;
    if ((int)lane == leader) { at = atomicAdd(&counters[c], (uint32_t)__popc(same)); }
    return __shfl_sync(same, at, leader) + __popc(same & ((1u << lane) - 1u));
}

// Calls body(group, world, slice, stage sizes) for every world of the batch, each exactly once. The body has
// one call site, so it is inlined and reads the kernel's parameters in place.
template <class Body>
__device__ __forceinline__ void forWorlds(const Batch& B, int slotIndex, const Split& sp, unsigned char* smem,
                                          Body&& body) {
    __shared__ uint32_t s_world, s_big;
    const uint32_t nw = (uint32_t)B.nWorlds;
    uint32_t* counter = B.work + slotIndex;
    bool warpMode = false;
    for (;;) {
        uint32_t o;
        if (!warpMode) {
            if (threadIdx.x == 0) {
                const uint32_t t = sp.firstWorld + atomicAdd(counter, 1u);
                s_world = t;
                s_big = (t < nw && B.info[B.order[t]].bodyCount > sp.bigBodies) ? 1u : 0u;
            }
            __syncthreads();
            o = s_world;
            const uint32_t big = s_big;
            __syncthreads();
            if (o >= nw) { return; }
            if (!big) {
                // Every later world is small too: from here on each warp takes worlds on its own.
                warpMode = true;
                if ((threadIdx.x >> 5) != 0) { o = sp.firstWorld + grabWarp(counter); }
            }
        } else {
            o = sp.firstWorld + grabWarp(counter);
        }
        if (o >= nw) { return; }
        const Group g = makeGroup(warpMode ? 32u : blockDim.x);
        unsigned char* slice = warpMode && smem ? smem + (size_t)g.id * (sp.smemBytes / g.count) : smem;
        body(g, B.order[o], slice, warpMode ? sp.small : sp.big);
    }
}

// Calls body(group, world, no slice, no stage sizes) for each big world (B.bigWorlds), a cluster a world: the CTAs of
// a cluster are one group, apart by the cluster's hardware barrier. One CTA a world left 147 of 148 SMs idle in the
// step of one large world.
template <class Body>
__device__ __forceinline__ void forBigWorlds(const Batch& B, Body&& body) {
    const GroupOf<true> g = makeClusterGroup();
    const uint32_t clusters = gridDim.x / clusterSize();
    for (uint32_t k = blockIdx.x / clusterSize(); k < B.nBigWorlds; k += clusters) {
        body(g, B.bigWorlds[k], (unsigned char*)nullptr, StageSizes{ 0u, 0u });
        g.sync();
    }
    g.sync();  // no CTA leaves while another may still reach its shared memory
}

// Exclusive prefix sum over the group; every thread of the group calls it.
template <class G>
__device__ __forceinline__ uint32_t groupScan(const G& g, uint32_t v, uint32_t& total) {
    __shared__ uint32_t sums[kMaxGroups][kMaxBlock / 32];
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if ((int)g.lane >= o) { x += y; }
    }
    if constexpr (G::kCluster) {
        // The warps of each CTA, then the CTAs' totals, every CTA's in the first one's shared memory.
        __shared__ uint32_t s_ctas[kMaxCluster];
        const uint32_t warp = threadIdx.x >> 5, warps = blockDim.x >> 5, rank = clusterRank(), ctas = clusterSize();
        if (g.lane == 31) { sums[0][warp] = x; }
        __syncthreads();
        if (warp == 0) {
            uint32_t s = g.lane < warps ? sums[0][g.lane] : 0u;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
                if ((int)g.lane >= o) { s += y; }
            }
            if (g.lane < warps) { sums[0][g.lane] = s; }
            if (g.lane == warps - 1) { g.shared(s_ctas)[rank] = s; }
        }
        g.sync();
        const uint32_t mine = g.lane < ctas ? g.shared(s_ctas)[g.lane] : 0u;
        total = __reduce_add_sync(0xffffffffu, mine);
        const uint32_t before = __reduce_add_sync(0xffffffffu, g.lane < rank ? mine : 0u);
        const uint32_t prefix = before + (warp > 0 ? sums[0][warp - 1] : 0u) + x - v;
        g.sync();
        return prefix;
    } else {
        if (g.warps == 1) {
            total = __shfl_sync(0xffffffffu, x, 31);
            return x - v;
        }
        if (g.lane == 31) { sums[g.id][g.warp] = x; }
        g.sync();
        if (g.warp == 0) {
            uint32_t s = g.lane < g.warps ? sums[g.id][g.lane] : 0u;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
                if ((int)g.lane >= o) { s += y; }
            }
            if (g.lane < g.warps) { sums[g.id][g.lane] = s; }
        }
        g.sync();
        const uint32_t prefix = (g.warp > 0 ? sums[g.id][g.warp - 1] : 0u) + x - v;
        total = sums[g.id][g.warps - 1];
        g.sync();
        return prefix;
    }
}

// Exclusive prefix sums of the n words at v, in place; ends with a group barrier.
template <class G>
__device__ void groupScanWords(const G& g, uint32_t* v, uint32_t n) {
    uint32_t base = 0;
    for (uint32_t first = 0; first < n; first += g.size) {
        const uint32_t k = first + g.tid;
        const uint32_t x = k < n ? v[k] : 0u;
        uint32_t tot;
        const uint32_t pre = groupScan(g, x, tot);
        if (k < n) { v[k] = base + pre; }
        base += tot;
    }
    g.sync();
}

// Calls emit(i, position) for every i < n where pred(i) holds, positions dense and in index order. Ends with
// a group barrier, so everything emit wrote is visible to the whole group on return.
template <class G, class Pred, class Emit>
__device__ uint32_t groupCompact(const G& g, uint32_t n, Pred pred, Emit emit) {
    uint32_t base = 0;
    for (uint32_t start = 0; start < n; start += g.size) {
        const uint32_t i = start + g.tid;
        const bool f = i < n && pred(i);
        uint32_t tot;
        const uint32_t pos = groupScan(g, f ? 1u : 0u, tot);
        if (f) { emit(i, base + pos); }
        base += tot;
    }
    g.sync();
    return base;
}

// Calls emit(i, position, k) for k < count(i) of every i < n, positions dense and in (i, k) order. Ends with a
// group barrier.
template <class G, class Count, class Emit>
__device__ uint32_t groupExpand(const G& g, uint32_t n, Count count, Emit emit) {
    uint32_t base = 0;
    for (uint32_t start = 0; start < n; start += g.size) {
        const uint32_t i = start + g.tid;
        const uint32_t c = i < n ? count(i) : 0u;
        uint32_t tot;
        const uint32_t pos = groupScan(g, c, tot);
        for (uint32_t k = 0; k < c; ++k) { emit(i, base + pos + k, k); }
        base += tot;
    }
    g.sync();
    return base;
}

// What every kernel of a step does first. The kernel behind it in the step may be brought onto the device from now on,
// and nothing goes on before the kernels ahead of it are over and their writes can be seen. Then the abort word is read
// once per CTA (with Cluster, once per cluster: its CTAs have to agree): true when an earlier step of this launch
// sequence overflowed a list, or this step did in an earlier kernel.
template <bool Cluster = false>
__device__ __forceinline__ bool stepAborted(const Batch& B, int serial) {
    __shared__ int s_skip;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if constexpr (Cluster) {
        const GroupOf<true> g = makeClusterGroup();
        if (g.tid == 0) { s_skip = *(volatile uint32_t*)B.abortStep <= (uint32_t)serial; }
        g.sync();
        const bool skip = *g.shared(&s_skip) != 0;
        g.sync();
        return skip;
    }
    if (threadIdx.x == 0) { s_skip = *(volatile uint32_t*)B.abortStep <= (uint32_t)serial; }
    __syncthreads();
    const bool skip = s_skip != 0;
    __syncthreads();
    return skip;
}

// The flat list a pair of shapes (global indices) is collided from: the planar class when its bodies are
// solved in a plane (src/world.cpp:514), else the class of its shape kinds.
__device__ __forceinline__ int pairClassOf(const Batch& B, uint32_t a, uint32_t b) {
    const DShape& sa = B.shapes[a];
    const DShape& sb = B.shapes[b];
    if (sa.kind == kMesh || sb.kind == kMesh) { return kClassMesh; }
    Vec3 n;
    if (usePlanar(B.bodies[sa.body], B.bodies[sb.body], n)) { return kClassPlanar; }
    return pairClass(sa.kind, sb.kind);
}

__device__ __forceinline__ uint64_t pairKey(uint32_t a, uint32_t b) {
    return ((uint64_t)(a < b ? a : b) << 32) | (uint64_t)(a < b ? b : a);
}

__device__ __forceinline__ void emitCandidate(const Batch& B, const WorldInfo& wi, uint32_t* count, uint64_t key) {
    const uint32_t pos = takePlace(count, 0u);
    if (pos < wi.candCap) { B.cand[wi.candFirst + pos] = key; }
}

// ---------------------------------------------------------------------------------------------------------
// Joints outside the solve: the pairs they keep from colliding and the links they add for waking.

// Whether a joint that does not collide its bodies holds bodies ga and gb (src/world.cpp:375-388).
__device__ __forceinline__ bool joinedBodies(const Batch& B, const WorldInfo& wi, uint32_t ga, uint32_t gb) {
    if (wi.joinedCount == 0) { return false; }
    const uint32_t a = ga - wi.bodyFirst, b = gb - wi.bodyFirst;
    const uint64_t key = ((uint64_t)(a < b ? a : b) << 32) | (uint64_t)(a < b ? b : a);
    const uint64_t* keys = B.joined + wi.jointFirst;
    uint32_t l = 0, h = wi.joinedCount;
    while (l < h) {
        const uint32_t mid = (l + h) >> 1;
        if (keys[mid] < key) {
            l = mid + 1;
        } else {
            h = mid;
        }
    }
    return l < wi.joinedCount && keys[l] == key;
}

// Pushes onto a wake stack the sleeping dynamic bodies linked to body gb: by a pair whose contacts have points,
// or by a joint that holds and is not joined to the world (src/world.cpp:655-700). Marks what it pushes.
static __device__ void pushLinked(const Batch& B, const WorldInfo& wi, uint32_t gb, const DContact* cs, uint32_t nc,
                           uint32_t* stack, uint32_t& top) {
    for (uint32_t ci = 0; ci < nc; ++ci) {
        const DContact& c = cs[ci];
        if (c.bodyA != gb && c.bodyB != gb) { continue; }
        if (ci > 0 && cs[ci - 1].key == c.key) { continue; }  // one link per pair
        const uint32_t other = c.bodyA == gb ? c.bodyB : c.bodyA;
        const DBody& ob = B.bodies[other];
        if (ob.type != kDynamic || ob.awake || B.wakeMark[other]) { continue; }
        bool linked = false;
        for (uint32_t k = ci; k < nc && cs[k].key == c.key; ++k) { linked = linked || cs[k].count > 0; }
        if (linked && top < wi.bodyCount) {
            B.wakeMark[other] = 1;
            stack[top++] = other;
        }
    }
    const DJoint* js = B.joints + wi.jointFirst;
    for (uint32_t x = 0; x < wi.jointCount; ++x) {
        const DJoint& j = js[x];
        if (!j.alive || j.broken || j.bodyA == kWorldEnd || (j.bodyA != gb && j.bodyB != gb)) { continue; }
        const uint32_t other = j.bodyA == gb ? j.bodyB : j.bodyA;
        const DBody& ob = B.bodies[other];
        if (ob.type != kDynamic || ob.awake || B.wakeMark[other]) { continue; }
        if (top < wi.bodyCount) {
            B.wakeMark[other] = 1;
            stack[top++] = other;
        }
    }
}

// Wakes what a wake stack holds and everything linked to it (src/world.cpp:703-735).
static __device__ void wakeStack(const Batch& B, const WorldInfo& wi, const DContact* cs, uint32_t nc, uint32_t* stack,
                          uint32_t top) {
    while (top > 0) {
        const uint32_t gb = stack[--top];
        DBody& b = B.bodies[gb];
        B.wakeMark[gb] = 0;
        if (b.awake) { continue; }
        b.awake = 1;
        b.sleepTime = 0.0f;
        updateInverseMass(b);
        pushLinked(B, wi, gb, cs, nc, stack, top);
    }
}

// At the start of a step a joint pulls its sleeping dynamic end awake when the other end moves
// (src/world.cpp:1578-1585), over the last step's contacts. The group looks for such a joint; one thread wakes.
// flag: a word of the group's shared memory (clusters).
template <class G>
static __device__ void wakeJointPulled(const Batch& B, const G& g, const WorldInfo& wi, const WorldCounts& wc, uint32_t* flag) {
    const DJoint* js = B.joints + wi.jointFirst;
    auto moving = [&](uint32_t gb) { return gb != kWorldEnd && movingAwake(B.bodies[gb]); };
    auto pulled = [&](uint32_t gb) {
        if (gb == kWorldEnd) { return false; }
        const DBody& b = B.bodies[gb];
        return b.alive && b.type == kDynamic && !b.awake && !B.wakeMark[gb];
    };
    if constexpr (G::kCluster) {
        if (g.tid == 0) { *flag = 0; }
        g.sync();
    }
    bool found = false;
    for (uint32_t x = g.tid; x < wi.jointCount; x += g.size) {
        const DJoint& j = js[x];
        if (!j.alive || j.broken) { continue; }
        found = found || (moving(j.bodyB) && pulled(j.bodyA)) || (moving(j.bodyA) && pulled(j.bodyB));
    }
    if (!g.any(found, flag)) { return; }
    if (g.tid == 0) {
        uint32_t* stack = B.unionParent + wi.bodyFirst;
        uint32_t top = 0;
        auto pull = [&](uint32_t gb) {
            if (pulled(gb) && top < wi.bodyCount) {
                B.wakeMark[gb] = 1;
                stack[top++] = gb;
            }
        };
        for (uint32_t x = 0; x < wi.jointCount; ++x) {
            const DJoint& j = js[x];
            if (!j.alive || j.broken) { continue; }
            if (moving(j.bodyB)) { pull(j.bodyA); }
            if (moving(j.bodyA)) { pull(j.bodyB); }
        }
        wakeStack(B, wi, B.previous + wi.contactFirst, min(wc.contactCount, wi.contactCap), stack, top);
    }
    g.sync();
}

// Calls f(joint index) for a world's joints, level by level (B.jointOrder): joints of a level share no dynamic body,
// and every dynamic body meets its joints in index order, which is what the reference's pass in index order gives it;
// other ends take nothing from a joint. A warp takes the joints of one kind among 32 of a level, which keeps it on one
// code path. Bounded by the longest chain of joint solves: 256 worlds of 22 joints of every kind, chains of 6 at most,
// take 601 us of substeps and 119 of end of step, against 868 and 202 with a world's joints on one thread. A world that
// is nearly all one chain (WorldInfo::jointLevels is 0) has its joints on one thread, in index order: a level costs its
// barrier and the reads that find its joints. Substeps and end of step by levels and on one thread, us a step: a chain of
// 64, 2234 + 336 and 1677 + 289; with one of 16 beside it 2340 + 353 and 2167 + 357, with one of 32 2332 + 366 and 2676 +
// 419; 300 worlds with chains of 6 and 2 499 + 96 and 470 + 97, of 6 and 3 478 + 95 and 519 + 105.
template <class G, class F>
__device__ __forceinline__ void forEachJoint(const Batch& B, const G& g, const WorldInfo& wi, F&& f) {
    // One loop for both, with one call of f: a second copy of the joints' code put a tenth on the levels.
    const bool chain = wi.jointLevels == 0;
    const uint32_t levels = chain ? 1u : wi.jointLevels, stride = chain ? 1u : 32u;
    uint32_t begin = 0;
    for (uint32_t l = 0; l < levels; ++l) {
        const uint32_t end = chain ? (g.tid == 0 ? wi.jointCount : 0u) : B.jointLevel[wi.jointFirst + l];
        for (uint32_t i = begin + (chain ? 0u : g.lane), k = 0; i < end; i += stride, ++k) {
            const uint32_t x = chain ? i : B.jointOrder[wi.jointFirst + i];
            if (chain || (k + B.joints[wi.jointFirst + x].type) % g.warps == g.warp) { f(x); }
        }
        g.sync();
        begin = end;
    }
}

// ---------------------------------------------------------------------------------------------------------
// Broadphase (src/world.cpp:752-870).
// A half-space against one body's shapes (src/world.cpp:844-867).
static __device__ void pairPlane(const Batch& B, const WorldInfo& wi, uint32_t gp, uint32_t gb, uint32_t* count) {
    const DShape& sp = B.shapes[gp];
    const DBody& pb = B.bodies[sp.body];
    const DBody& b = B.bodies[gb];
    const bool planeMoving = movingAwake(pb);
    if (!b.alive || gb == sp.body || (!planeMoving && !movingAwake(b))) { return; }
    const float gp_ = B.grow[sp.body];
    const Transform xp = pb.xf * sp.local;
    const Vec3 n = rotate(xp.q, Vec3{ 0, 0, 1 });
    const float offset = dot(n, xp.p);
    const float g = gp_ + B.grow[gb];
    auto reaches = [&](const Vec3& lo, const Vec3& hi) {
        const Vec3 c = (lo + hi) * 0.5f, e = (hi - lo) * 0.5f + Vec3{ g, g, g };
        return dot(c, n) - offset <= e.x * fabsf(n.x) + e.y * fabsf(n.y) + e.z * fabsf(n.z);
    };
    if (b.hasBounds && !reaches(b.lo, b.hi)) { return; }
    for (uint32_t x = 0; x < b.shapeCount; ++x) {
        const uint32_t gs = B.shapeList[b.shapeFirst + x];
        const DShape& s = B.shapes[gs];
        if (s.kind != kHalfSpace && !reaches(s.lo, s.hi)) { continue; }
        // pairable(sp, s): neither a sensor, different bodies, one of them dynamic.
        if (sp.sensor || s.sensor || sp.body == s.body) { continue; }
        if (pb.type != kDynamic && b.type != kDynamic) { continue; }
        // test(pi, si) (src/world.cpp:798-808).
        const float ga = B.grow[sp.body], gbb = B.grow[s.body];
        const Vec3 g3a{ ga, ga, ga }, g3b{ gbb, gbb, gbb };
        if (!boxesOverlap(sp.lo - g3a, sp.hi + g3a, s.lo - g3b, s.hi + g3b)) { continue; }
        if (!(sp.category & s.mask) || !(s.category & sp.mask)) { continue; }
        if (joinedBodies(B, wi, sp.body, s.body)) { continue; }
        emitCandidate(B, wi, count, pairKey(sp.index, s.index));
    }
}

// The shapes of two bodies whose grown bounds overlap, paired by their own grown bounds
// (src/world.cpp:819-842).
static __device__ void pairShapes(const Batch& B, const WorldInfo& wi, const DBody& ba, const DBody& bb, float gA, float gB,
                           const Vec3& loA, const Vec3& hiA, const Vec3& loB, const Vec3& hiB, const Vec3& reach,
                           uint32_t* count) {
    if (joinedBodies(B, wi, (uint32_t)(&ba - B.bodies), (uint32_t)(&bb - B.bodies))) { return; }
    const Vec3 nearLoA = loB - reach, nearHiA = hiB + reach;
    const Vec3 nearLoB = loA - reach, nearHiB = hiA + reach;
    const Vec3 grownA{ gA, gA, gA }, grownB{ gB, gB, gB };
    for (uint32_t x = 0; x < ba.shapeCount; ++x) {
        const DShape& s = B.shapes[B.shapeList[ba.shapeFirst + x]];
        if (s.kind == kHalfSpace || s.sensor || !boxesOverlap(s.lo, s.hi, nearLoA, nearHiA)) { continue; }
        const Vec3 xlo = s.lo - grownA, xhi = s.hi + grownA;
        for (uint32_t y = 0; y < bb.shapeCount; ++y) {
            const DShape& t = B.shapes[B.shapeList[bb.shapeFirst + y]];
            if (t.kind == kHalfSpace || t.sensor || !boxesOverlap(t.lo, t.hi, nearLoB, nearHiB)) { continue; }
            if (!boxesOverlap(xlo, xhi, t.lo - grownB, t.hi + grownB)) { continue; }
            if (!(s.category & t.mask) || !(t.category & s.mask)) { continue; }
            emitCandidate(B, wi, count, pairKey(s.index, t.index));
        }
    }
}

constexpr uint32_t kBodyLive = 1u, kBodyDynamic = 2u, kBodyMoving = 4u;
// Largest worlds whose bodies the broadphase and the substep stage in shared memory.

// A body as the pair test sees it: bounds, growth and the three flags above.
struct PairBody {
    Vec3 lo, hi;
    float grow;
    uint32_t flags;
};

__device__ __forceinline__ PairBody pairBodyOf(const Batch& B, uint32_t g) {
    const DBody b = readBody<kBodySolve | kBodyBounds>(B.bodies[g]);
    PairBody p;
    p.lo = b.lo;
    p.hi = b.hi;
    p.grow = B.grow[g];
    p.flags = ((b.alive && b.hasBounds) ? kBodyLive : 0u) | (b.type == kDynamic ? kBodyDynamic : 0u) |
              (movingAwake(b) ? kBodyMoving : 0u);
    return p;
}

// Worlds with more bodies than this find their body pairs with a sweep along x over the whole grid instead of
// testing every pair on one group.
constexpr uint32_t kSweepBodies = 1024;

// Floats as unsigned keys in the same order, for atomicMin and atomicMax.
__device__ __forceinline__ uint32_t orderedKey(float f) {
    const uint32_t b = __float_as_uint(f);
    return b ^ ((b >> 31) ? 0xffffffffu : 0x80000000u);
}
__device__ __forceinline__ float fromOrderedKey(uint32_t k) {
    return __uint_as_float((k >> 31) ? (k ^ 0x80000000u) : ~k);
}

// How far a body's interval along x is widened beyond its grown bounds, so that two bodies the pair test
// accepts always have overlapping intervals whatever the rounding of the test's sums: a millimetre plus a
// millionth of the coordinate.
__device__ __forceinline__ float sweepSlack(float x) { return 1e-3f + 1e-6f * fabsf(x); }

// A big world's bodies lie in a grid of cells by where their intervals along x and along a second axis (the longer of
// y and z) start, at most a cell a body, x-major: the cells of one x column from a low to a high second coordinate
// are one contiguous run of bodies. A body whose interval covers an eighth of the second axis or more is wide: it can
// start far from what it meets, so it stands in a list of its own as well. Where more than a sixteenth of the bodies
// are wide (a single layer of bodies), the grid has x columns only and no body counts as wide. (Along x alone, a
// body of the terrain's 32 x 32 columns met the 1,500 bodies of its x range: 65 million tests, 1.9 ms.)
constexpr uint32_t kBodyWide = 8u;

// The range of a big world's intervals along x and along its second axis, from the keys alone.
struct SweepRange {
    float lo[2], hi[2];
    int axis;  // the second axis
};

__device__ __forceinline__ SweepRange sweepRange(const WorldCounts& wc) {
    float lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        lo[k] = fromOrderedKey(wc.sweepMinKey[k]);
        hi[k] = fromOrderedKey(wc.sweepMaxKey[k]);
    }
    SweepRange r;
    r.axis = hi[2] - lo[2] > hi[1] - lo[1] ? 2 : 1;
    r.lo[0] = lo[0], r.hi[0] = hi[0];
    r.lo[1] = r.axis == 2 ? lo[2] : lo[1], r.hi[1] = r.axis == 2 ? hi[2] : hi[1];
    return r;
}

struct SweepGrid {
    float lo[2], scale[2];
    uint32_t cells[2];
    int axis;     // the second axis
    float width;  // no body that is not wide is wider along it
};

// The grid of a world whose wide bodies are counted.
__device__ __forceinline__ SweepGrid sweepGrid(const WorldInfo& wi, const WorldCounts& wc) {
    const SweepRange r = sweepRange(wc);
    SweepGrid s;
    s.axis = r.axis;
    const bool flat = wc.sweepWide > wi.bodyCount / 16;
    const uint32_t side = (uint32_t)sqrtf((float)(wi.bodyCount / 4 + 1));
    s.cells[0] = flat ? wi.bodyCount / 4 + 1 : side;
    s.cells[1] = flat ? 1u : side;
    for (int k = 0; k < 2; ++k) {
        s.lo[k] = r.lo[k];
        s.scale[k] = r.hi[k] > r.lo[k] ? (float)s.cells[k] / (r.hi[k] - r.lo[k]) : 0.0f;
    }
    s.width = __uint_as_float(wc.sweepWidth);
    return s;
}

__device__ __forceinline__ uint32_t sweepCell(const SweepGrid& s, int k, float x) {
    const float f = (x - s.lo[k]) * s.scale[k];
    if (!(f > 0.0f)) { return 0u; }
    return f >= (float)(s.cells[k] - 1) ? s.cells[k] - 1 : (uint32_t)f;
}

// A body's grown interval along an axis, widened so that rounding never loses a pair.
__device__ __forceinline__ void sweepInterval(float lo, float hi, float grow, float& from, float& to) {
    from = lo - grow - sweepSlack(lo);
    to = hi + grow + sweepSlack(hi);
}

// The first half of a big world's broadphase, after the growth: each live body's interval along x, the ranges of the
// intervals along every axis, and the bodies counted into cells. Cell c then holds the records from start[c - 1] to
// start[c], start[-1] being 0.
template <class G>
static __device__ void prepareSweep(const Batch& B, const G& g, const WorldInfo& wi, WorldCounts& wc, uint32_t w) {
    const uint32_t n = wi.bodyCount;
    if (g.tid == 0) {
        for (int k = 0; k < 3; ++k) {
            wc.sweepMinKey[k] = 0xffffffffu;
            wc.sweepMaxKey[k] = 0u;
        }
        wc.candRaw = 0;
        wc.sweepWide = 0;
        wc.sweepWidth = 0;
    }
    g.sync();
    uint32_t least[3] = { 0xffffffffu, 0xffffffffu, 0xffffffffu }, most[3] = { 0u, 0u, 0u };
    for (uint32_t i = g.tid; i < n; i += g.size) {
        const uint32_t gb = wi.bodyFirst + i;
        const DBody& b = B.bodies[gb];
        float lo = FLT_MAX, hi = -FLT_MAX;
        if (b.alive && b.hasBounds) {
            const float gr = B.grow[gb];
            const Vec3 bl = b.lo, bh = b.hi;
            for (int k = 2; k >= 0; --k) {
                sweepInterval(comp(bl, k), comp(bh, k), gr, lo, hi);
                least[k] = min(least[k], orderedKey(lo));
                most[k] = max(most[k], orderedKey(hi));
            }
        }
        B.sweepLo[gb] = lo;
        B.sweepHi[gb] = hi;
    }
    for (int k = 0; k < 3; ++k) {
        least[k] = __reduce_min_sync(0xffffffffu, least[k]);
        most[k] = __reduce_max_sync(0xffffffffu, most[k]);
        if (g.lane == 0) {
            atomicMin(&wc.sweepMinKey[k], least[k]);
            atomicMax(&wc.sweepMaxKey[k], most[k]);
        }
    }
    g.sync();
    // Every thread takes the axis and what counts as wide from the keys, which stand: faster threads add to the count of
    // wide bodies, and with it to what the grid will be, while others are still here.
    const SweepRange span = sweepRange(wc);
    auto second = [&](uint32_t i, float& lo, float& hi) {
        const uint32_t gb = wi.bodyFirst + i;
        const DBody& b = B.bodies[gb];
        lo = FLT_MAX, hi = -FLT_MAX;
        if (!b.alive || !b.hasBounds) { return; }
        const Vec3 bl = b.lo, bh = b.hi;
        sweepInterval(span.axis == 2 ? bl.z : bl.y, span.axis == 2 ? bh.z : bh.y, B.grow[gb], lo, hi);
    };
    const float range = span.hi[1] - span.lo[1];
    auto wideAt = [&](float lo, float hi) { return !((hi - lo) * 8.0f < range); };
    uint32_t wide = 0, width = 0;
    for (uint32_t i = g.tid; i < n; i += g.size) {
        float lo, hi;
        second(i, lo, hi);
        if (!(hi >= lo)) { continue; }
        if (wideAt(lo, hi)) {
            ++wide;
        } else {
            width = max(width, __float_as_uint(hi - lo));
        }
    }
    wide = __reduce_add_sync(0xffffffffu, wide);
    width = __reduce_max_sync(0xffffffffu, width);
    if (g.lane == 0) {
        atomicAdd(&wc.sweepWide, wide);
        atomicMax(&wc.sweepWidth, width);
    }
    g.sync();
    const SweepGrid grid = sweepGrid(wi, wc);
    const uint32_t cells = grid.cells[0] * grid.cells[1];
    uint32_t* start = B.sweepStart + wi.bodyFirst + w;
    auto cellOf = [&](uint32_t i) {
        float lo, hi;
        second(i, lo, hi);
        return sweepCell(grid, 0, B.sweepLo[wi.bodyFirst + i]) * grid.cells[1] + sweepCell(grid, 1, lo);
    };
    for (uint32_t k = g.tid; k < cells; k += g.size) { start[k] = 0; }
    g.sync();
    for (uint32_t i = g.tid; i < n; i += g.size) { atomicAdd(&start[cellOf(i)], 1u); }
    g.sync();
    groupScanWords(g, start, cells);
    // Scattering advances each cell's start to its end.
    for (uint32_t i = g.tid; i < n; i += g.size) { B.sweepOrder[wi.bodyFirst + atomicAdd(&start[cellOf(i)], 1u)] = i; }
    g.sync();
    // The records in cell order, so a scan over neighbouring cells reads one contiguous run.
    for (uint32_t q = g.tid; q < n; q += g.size) {
        const uint32_t i = B.sweepOrder[wi.bodyFirst + q];
        PairBody p = pairBodyOf(B, wi.bodyFirst + i);
        float lo, hi;
        second(i, lo, hi);
        if (grid.cells[1] > 1 && hi >= lo && wideAt(lo, hi)) { p.flags |= kBodyWide; }
        B.sweepRecs[wi.bodyFirst + q] = SweepRec{ p.lo, p.hi, p.grow, p.flags, B.sweepLo[wi.bodyFirst + i], i };
    }
    g.sync();
    // The wide bodies' records, by position; the order has served.
    groupCompact(g, n, [&](uint32_t q) { return (B.sweepRecs[wi.bodyFirst + q].flags & kBodyWide) != 0; },
                 [&](uint32_t q, uint32_t pos) { B.sweepOrder[wi.bodyFirst + pos] = q; });
}

// sortKeys with the rows and the keys by row in the group's shared slice, where they fit it: each key's place is its
// row's start plus the keys of the row before it, which every thread counts for its own keys at once. (One thread
// sorts each row in place in global memory otherwise; with the pair tests below, the box pyramid's broadphase of 211
// bodies and 590 keys went from 102 to 44 us.)
template <class G>
static __device__ uint32_t sortKeysShared(const G& g, const Batch& B, const WorldInfo& wi, uint32_t count, unsigned char* slice,
                                          uint32_t* repeats) {
    uint64_t* keys = B.cand + wi.candFirst;
    uint64_t* byRow = reinterpret_cast<uint64_t*>(slice);
    uint32_t* row = reinterpret_cast<uint32_t*>(byRow + count);
    const uint32_t rows = wi.shapeCount;
    for (uint32_t r = g.tid; r < rows; r += g.size) { row[r] = 0; }
    if (g.tid == 0) { *repeats = 0; }
    g.sync();
    for (uint32_t i = g.tid; i < count; i += g.size) { atomicAdd(&row[(uint32_t)(keys[i] >> 32)], 1u); }
    g.sync();
    groupScanWords(g, row, rows);
    // Scattering advances each row's start to its end.
    for (uint32_t i = g.tid; i < count; i += g.size) {
        const uint64_t k = keys[i];
        byRow[atomicAdd(&row[(uint32_t)(k >> 32)], 1u)] = k;
    }
    g.sync();
    for (uint32_t i = g.tid; i < count; i += g.size) {
        const uint64_t k = byRow[i];
        const uint32_t r = (uint32_t)(k >> 32), s = r > 0 ? row[r - 1] : 0u, e = row[r];
        uint32_t before = 0;
        bool repeat = false;
        for (uint32_t j = s; j < e; ++j) {
            const uint64_t other = byRow[j];
            before += other < k || (other == k && j < i) ? 1u : 0u;
            repeat = repeat || (other == k && j != i);
        }
        keys[s + before] = k;
        if (repeat) { *(volatile uint32_t*)repeats = 1; }
    }
    g.sync();
    if (*(volatile uint32_t*)repeats == 0) { return count; }
    for (uint32_t i = g.tid; i < count; i += g.size) { byRow[i] = keys[i]; }
    g.sync();
    return groupCompact(g, count, [&](uint32_t i) { return i == 0 || byRow[i] != byRow[i - 1]; },
                        [&](uint32_t i, uint32_t pos) { keys[pos] = byRow[i]; });
}

// Sorts the world's count keys (minShape << 32 | maxShape, at B.cand) ascending and removes repeats: a
// counting sort by the first shape, then each row sorted on its own (rows are short), then compaction back
// into B.cand. Returns the unique count.
constexpr uint32_t kShortRow = 48;  // rows of keys at most this long are sorted by one thread

template <class G>
static __device__ uint32_t sortKeys(const G& g, const Batch& B, const WorldInfo& wi, uint32_t count) {
    uint32_t* row = B.rowScratch + wi.shapeFirst;
    uint64_t* tmp = B.mergeKeyA + wi.contactFirst;
    uint64_t* keys = B.cand + wi.candFirst;
    const uint32_t rows = wi.shapeCount;
    for (uint32_t r = g.tid; r < rows; r += g.size) { row[r] = 0; }
    g.sync();
    for (uint32_t i = g.tid; i < count; i += g.size) { atomicAdd(&row[(uint32_t)(keys[i] >> 32)], 1u); }
    g.sync();
    groupScanWords(g, row, rows);
    // Scattering advances each row's start to its end.
    for (uint32_t i = g.tid; i < count; i += g.size) {
        const uint64_t k = keys[i];
        tmp[atomicAdd(&row[(uint32_t)(k >> 32)], 1u)] = k;
    }
    g.sync();
    // Short rows: one thread each, by insertion.
    for (uint32_t r = g.tid; r < rows; r += g.size) {
        const uint32_t s = r > 0 ? row[r - 1] : 0u, e = row[r];
        if (e - s > kShortRow) { continue; }
        for (uint32_t i = s + 1; i < e; ++i) {
            const uint64_t k = tmp[i];
            uint32_t j = i;
            while (j > s && tmp[j - 1] > k) {
                tmp[j] = tmp[j - 1];
                --j;
            }
            tmp[j] = k;
        }
    }
    // Long rows (a half-space's or a mesh's pairs): one at a time by the whole group, counted by the second
    // shape. Equal keys may land in any order among themselves, which leaves the same sequence.
    uint32_t* longRows = B.rowLong + wi.shapeFirst;
    const uint32_t nLong = groupCompact(
        g, rows, [&](uint32_t r) { return row[r] - (r > 0 ? row[r - 1] : 0u) > kShortRow; },
        [&](uint32_t r, uint32_t pos) { longRows[pos] = r; });
    uint32_t* hist = B.rowCount + wi.shapeFirst;
    for (uint32_t x = 0; x < nLong; ++x) {
        const uint32_t r = longRows[x];
        const uint32_t s = r > 0 ? row[r - 1] : 0u, e = row[r];
        for (uint32_t c = g.tid; c < rows; c += g.size) { hist[c] = 0; }
        g.sync();
        for (uint32_t i = s + g.tid; i < e; i += g.size) { atomicAdd(&hist[(uint32_t)tmp[i]], 1u); }
        g.sync();
        uint32_t base = s;
        for (uint32_t first = 0; first < rows; first += g.size) {
            const uint32_t c = first + g.tid;
            const uint32_t v = c < rows ? hist[c] : 0u;
            uint32_t tot;
            const uint32_t pre = groupScan(g, v, tot);
            if (c < rows) { hist[c] = base + pre; }
            base += tot;
        }
        g.sync();
        for (uint32_t i = s + g.tid; i < e; i += g.size) {
            const uint64_t k = tmp[i];
            keys[atomicAdd(&hist[(uint32_t)k], 1u)] = k;
        }
        g.sync();
        for (uint32_t i = s + g.tid; i < e; i += g.size) { tmp[i] = keys[i]; }
        g.sync();
    }
    g.sync();
    return groupCompact(
        g, count, [&](uint32_t i) { return i == 0 || tmp[i] != tmp[i - 1]; }, [&](uint32_t i, uint32_t pos) { keys[pos] = tmp[i]; });
}

// Body pairs whose grown bounds overlap, then their shapes (src/world.cpp:788-842), and half-space pairs
// (:844-867); the keys are sorted and made unique (:868-869). Bodies are staged in the group's shared slice when at
// most stageN of them.
template <class G>
static __device__ void finishCandidates(const Batch& B, const G& g, const WorldInfo& wi, WorldCounts& wc, uint32_t w,
                                 uint32_t total, int serial, uint32_t* cls, uint32_t* classBase,
                                 unsigned char* slice = nullptr, uint32_t sliceBytes = 0);

// Growth by the speculative distance and the travel over the step (src/world.cpp:754-765).
__device__ __forceinline__ float growthOf(const DBody& b, const StepParams& P) {
    float gr = P.tol.speculative;
    if (b.alive && b.type != kStatic && !(lengthSquared(b.v) == 0.0f && lengthSquared(b.w) == 0.0f)) {
        gr += (length(b.v) + length(b.w) * b.extent) * P.dt;
    }
    return gr;
}

// The first half of the big worlds' broadphase, a cluster a world.
template <int Unused = 0>
__global__ void __launch_bounds__(kMaxBlock) k_broad_big(const __grid_constant__ Batch B, const __grid_constant__ StepParams P, int serial) {
    __shared__ uint32_t s_pulled;
    if (stepAborted<true>(B, serial)) { return; }
    forBigWorlds(B, [&](const GroupOf<true>& g, uint32_t w, unsigned char*, const StageSizes&) {
        const WorldInfo wi = B.info[w];
        WorldCounts& wc = B.counts[w];
        if (wi.jointCount > 0) { wakeJointPulled(B, g, wi, wc, g.shared(&s_pulled)); }
        for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
            B.grow[wi.bodyFirst + i] = growthOf(B.bodies[wi.bodyFirst + i], P);
        }
        g.sync();
        prepareSweep(B, g, wi, wc, w);
    });
}

template <int Unused = 0>
__global__ void __launch_bounds__(kMaxBlock, 1) k_broadphase(const __grid_constant__ Batch B, const __grid_constant__ StepParams P, const __grid_constant__ Split sp, int serial) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint32_t s_count[kMaxGroups];
    __shared__ uint32_t s_queue[kMaxGroups][64];
    __shared__ uint32_t s_class[kMaxGroups][kPairClasses], s_classBase[kMaxGroups][kPairClasses];
    if (stepAborted(B, serial)) { return; }
    forWorlds(B, kSlotBroad, sp, s_raw, [&](const Group& g, uint32_t w, unsigned char* slice, const StageSizes& ss) {
        PairBody* staged = reinterpret_cast<PairBody*>(slice);
        const uint32_t stageN = ss.bodies;
        const WorldInfo wi = B.info[w];
        WorldCounts& wc = B.counts[w];
        const uint32_t n = wi.bodyCount;
        const bool useStage = n <= stageN;
        if (wi.jointCount > 0) { wakeJointPulled(B, g, wi, wc, nullptr); }
        if (g.tid == 0) { s_count[g.id] = 0; }
        for (uint32_t i = g.tid; i < n; i += g.size) {
            const DBody b = readBody<kBodySolve | kBodyPose | kBodyBounds>(B.bodies[wi.bodyFirst + i]);
            const float gr = growthOf(b, P);
            B.grow[wi.bodyFirst + i] = gr;
            if (useStage) {
                PairBody p;
                p.lo = b.lo;
                p.hi = b.hi;
                p.grow = gr;
                p.flags = ((b.alive && b.hasBounds) ? kBodyLive : 0u) | (b.type == kDynamic ? kBodyDynamic : 0u) |
                          (movingAwake(b) ? kBodyMoving : 0u);
                staged[i] = p;
            }
        }
        g.sync();
        if (n > kSweepBodies) {
            prepareSweep(B, g, wi, wc, w);
            return;
        }
        uint32_t* count = &s_count[g.id];
        // The body pairs: a warp holds 32 second bodies, a lane each, and tests them against every first body before
        // them. The bodies of a block that are near each other in index usually are in space as well, so 32 first
        // bodies at a time are held against the block's common bounds, and only those that reach them are tested. The
        // pairs found wait in the warp's queue until a lane each can work on them. (A warp per first body, its lanes
        // over the second ones, read both from shared memory for each test and followed a found pair's shapes with
        // its other lanes waiting: 741 us of broadphase for the 4096 uneven worlds and 187 for 64 of them, 274 and 56 with
        // blocks at the same launch shape, 210 for the 4096 at the default one.)
        uint32_t* queue = s_queue[threadIdx.x >> 5];
        uint32_t queued = 0;
        auto work = [&](uint32_t items) {  // the queue's first items
            if (g.lane < items) {
                const uint32_t ab = queue[g.lane], a = ab & 0xffffu, b = ab >> 16;
                const PairBody A = useStage ? staged[a] : pairBodyOf(B, wi.bodyFirst + a);
                const PairBody Bb = useStage ? staged[b] : pairBodyOf(B, wi.bodyFirst + b);
                const float gg = A.grow + Bb.grow;
                pairShapes(B, wi, B.bodies[wi.bodyFirst + a], B.bodies[wi.bodyFirst + b], A.grow, Bb.grow, A.lo, A.hi, Bb.lo,
                           Bb.hi, Vec3{ gg, gg, gg }, count);
            }
            __syncwarp();
        };
        const uint32_t blocks = (n + 31) / 32;
        for (uint32_t k = 0; k * g.warps < blocks; ++k) {
            // A later block has more first bodies: the warps take them to and fro.
            const uint32_t block = k * g.warps + (k & 1 ? g.warps - 1 - g.warp : g.warp);
            if (block >= blocks) { continue; }
            const uint32_t b = block * 32 + g.lane;
            PairBody Bb{};
            if (b < n) { Bb = useStage ? staged[b] : pairBodyOf(B, wi.bodyFirst + b); }
            const bool live = (Bb.flags & kBodyLive) != 0;
            // The keys of the infinities stand for bodies that do not count: those without bounds, and NaNs, which
            // overlap nothing.
            auto least = [&](float x) { return fromOrderedKey(__reduce_min_sync(0xffffffffu, live && x == x ? orderedKey(x) : 0xff800000u)); };
            auto most = [&](float x) { return fromOrderedKey(__reduce_max_sync(0xffffffffu, live && x == x ? orderedKey(x) : 0x007fffffu)); };
            const Vec3 lo{ least(Bb.lo.x), least(Bb.lo.y), least(Bb.lo.z) }, hi{ most(Bb.hi.x), most(Bb.hi.y), most(Bb.hi.z) };
            const float grow = most(Bb.grow);
            if (!__any_sync(0xffffffffu, live)) { continue; }
            for (uint32_t first = 0; first < block * 32 + 32; first += 32) {
                const uint32_t mine = first + g.lane;
                PairBody A{};
                if (mine < n) { A = useStage ? staged[mine] : pairBodyOf(B, wi.bodyFirst + mine); }
                bool near = (A.flags & kBodyLive) != 0;
                if (near) {
                    const float gg = A.grow + grow;
                    const Vec3 reach{ gg, gg, gg };
                    near = !(gg < FLT_MAX) || boxesOverlap(A.lo - reach, A.hi + reach, lo, hi);
                }
                for (uint32_t left = __ballot_sync(0xffffffffu, near); left; left &= left - 1) {
                    const int from = __ffs(left) - 1;
                    const uint32_t a = first + (uint32_t)from;
                    const PairBody Aa = useStage ? staged[a] : pairBodyOf(B, wi.bodyFirst + a);
                    bool hit = live && a < b && ((Aa.flags | Bb.flags) & kBodyDynamic) && ((Aa.flags | Bb.flags) & kBodyMoving);
                    const float gg = Aa.grow + Bb.grow;
                    const Vec3 reach{ gg, gg, gg };
                    hit = hit && boxesOverlap(Aa.lo - reach, Aa.hi + reach, Bb.lo, Bb.hi);
                    const uint32_t hits = __ballot_sync(0xffffffffu, hit);
                    if (!hits) { continue; }
                    if (hit) { queue[queued + __popc(hits & ((1u << g.lane) - 1u))] = a | b << 16; }
                    __syncwarp();
                    queued += __popc(hits);
                    if (queued < 32) { continue; }
                    work(32);
                    queued -= 32;
                    const uint32_t rest = g.lane < queued ? queue[32 + g.lane] : 0u;
                    __syncwarp();
                    queue[g.lane] = rest;
                    __syncwarp();
                }
            }
        }
        work(queued);
        for (uint32_t pl = 0; pl < wi.planeCount; ++pl) {
            const uint32_t gp = B.planeList[wi.planeFirst + pl];
            for (uint32_t b = g.tid; b < n; b += g.size) { pairPlane(B, wi, gp, wi.bodyFirst + b, count); }
        }
        g.sync();
        finishCandidates(B, g, wi, wc, w, *count, serial, s_class[g.id], s_classBase[g.id], slice,
                         sp.smemBytes / g.count);
    });
}

// The end of a world's broadphase: the raw keys sorted and made unique (src/world.cpp:868-869), then the
// pairs join the flat list of their class: counted per class, a block of each list reserved for the
// world, then scattered into it. A list that did not fit stops this step, and the host grows it.
template <class G>
static __device__ void finishCandidates(const Batch& B, const G& g, const WorldInfo& wi, WorldCounts& wc, uint32_t w,
                                 uint32_t total, int serial, uint32_t* cls, uint32_t* classBase, unsigned char* slice,
                                 uint32_t sliceBytes) {
    {
        if (total > wi.candCap) {
            // The list did not fit: this step stops here and the host grows the world's lists.
            if (g.tid == 0) {
                wc.flags |= kDevPairOverflow;
                wc.candNeeded = max(wc.candNeeded, total);
                atomicMin(B.abortStep, (uint32_t)serial);
            }
            g.sync();
            return;
        }
        const bool fits = (uint64_t)total * 8 + (uint64_t)wi.shapeCount * 4 <= sliceBytes;
        const uint32_t unique = slice && fits ? sortKeysShared(g, B, wi, total, slice, &cls[0]) : sortKeys(g, B, wi, total);
        if (g.tid == 0) {
            wc.candCount = unique;
            wc.candNeeded = max(wc.candNeeded, total);
            wc.partCount = 0;
            wc.boundsCount = 0;
        }
        if (g.tid < kPairClasses) { cls[g.tid] = 0; }
        g.sync();
        auto classOf = [&](uint32_t i) {
            const uint64_t key = B.cand[wi.candFirst + i];
            return pairClassOf(B, wi.shapeFirst + (uint32_t)(key >> 32), wi.shapeFirst + (uint32_t)(key & 0xffffffffu));
        };
        for (uint32_t i = g.tid; i < unique; i += g.size) { takePlace(cls, (uint32_t)classOf(i)); }
        g.sync();
        if (g.tid < kPairClasses) {
            classBase[g.tid] = atomicAdd(B.work + kSlotCandItems + g.tid, cls[g.tid]);
            cls[g.tid] = 0;
        }
        g.sync();
        for (uint32_t i = g.tid; i < unique; i += g.size) {
            const int c = classOf(i);
            const uint32_t pos = classBase[c] + takePlace(cls, (uint32_t)c);
            B.candItems[(size_t)c * B.candItemStride + pos] = make_uint2(w, i);
        }
        g.sync();
    }
}

// The pair half of a big world's broadphase: each body takes the bodies whose intervals along x start within its own
// (the one starting first takes a pair, so each pair is taken once) among the wide ones and those of the cells whose
// bodies can reach it along the second axis, and applies the same pair test as the small worlds, in the pair's
// lower-body-first order. A warp per body, its lanes across the contiguous run of records of each x column; a wide
// body's run is the whole of its x range, a warp a part of it (kSweepPart). The worlds' items are one list that the
// warps take in turn. (Each world's items started at warp 0 once, so that 76 worlds queued on the same ninth of the
// device: 1029 us of broadphase a step for 76 planar worlds of 1119 bodies and 558 for 40, 164 and 128 as one list; 712
// and 295 for 76 pyramids of 1036.)
constexpr uint32_t kSweepPart = 1024;  // records of a wide body's run a warp takes

// A big world's wide bodies, none when its grid has x columns only, and what its pairs are taken by: its records, then
// the wide ones' parts.
__device__ __forceinline__ uint32_t sweepWides(const WorldInfo& wi, const WorldCounts& wc) {
    return wc.sweepWide > wi.bodyCount / 16 ? 0u : wc.sweepWide;
}
__device__ __forceinline__ uint32_t sweepParts(const WorldInfo& wi) { return (wi.bodyCount + kSweepPart - 1) / kSweepPart; }

// The items from first on, every step-th one, of one world.
static __device__ __forceinline__ void pairsOfWorld(const Batch& B, uint32_t w, uint32_t first, uint32_t items, uint32_t step,
                                                    uint32_t lane) {
    const WorldInfo wi = B.info[w];
    WorldCounts& wc = B.counts[w];
    const uint32_t n = wi.bodyCount, parts = sweepParts(wi), wide = sweepWides(wi, wc);
    const SweepRec* recs = B.sweepRecs + wi.bodyFirst;
    const uint32_t* start = B.sweepStart + wi.bodyFirst + w;
    const uint32_t* wides = B.sweepOrder + wi.bodyFirst;
    const SweepGrid grid = sweepGrid(wi, wc);
    for (uint32_t item = first; item < items; item += step) {
        const bool part = item >= n;
        const SweepRec ri = recs[part ? wides[(item - n) / parts] : item];
        if (!(ri.flags & kBodyLive)) { continue; }
        const float lo = ri.start, hi = B.sweepHi[wi.bodyFirst + ri.body];
        auto test = [&](const SweepRec& rj) {
            const uint32_t i = ri.body, j = rj.body;
            if (j == i || !(rj.start > lo || (rj.start == lo && j > i)) || rj.start > hi) { return; }
            const SweepRec& A = i < j ? ri : rj;
            const SweepRec& Bb = i < j ? rj : ri;
            if (!(A.flags & kBodyLive) || !(Bb.flags & kBodyLive)) { return; }
            if (!((A.flags | Bb.flags) & kBodyDynamic)) { return; }
            if (!((A.flags | Bb.flags) & kBodyMoving)) { return; }
            const float gg = A.grow + Bb.grow;
            const Vec3 reach{ gg, gg, gg };
            if (!boxesOverlap(A.lo - reach, A.hi + reach, Bb.lo, Bb.hi)) { return; }
            pairShapes(B, wi, B.bodies[wi.bodyFirst + A.body], B.bodies[wi.bodyFirst + Bb.body], A.grow, Bb.grow, A.lo,
                       A.hi, Bb.lo, Bb.hi, reach, &wc.candRaw);
        };
        const uint32_t x0 = sweepCell(grid, 0, lo), x1 = sweepCell(grid, 0, hi);
        if (part) {
            const uint32_t c0 = x0 * grid.cells[1], c1 = (x1 + 1) * grid.cells[1] - 1;
            const uint32_t from = (item - n) % parts * kSweepPart;
            const uint32_t q0 = max(from, c0 ? start[c0 - 1] : 0u), q1 = min(from + kSweepPart, start[c1]);
            for (uint32_t q = q0 + lane; q < q1; q += 32) {
                const SweepRec rj = recs[q];
                if (!(rj.flags & kBodyWide)) { test(rj); }
            }
            continue;
        }
        for (uint32_t q = lane; q < wide; q += 32) { test(recs[wides[q]]); }
        if (ri.flags & kBodyWide) { continue; }  // its parts take the others
        float from, to;
        sweepInterval(grid.axis == 2 ? ri.lo.z : ri.lo.y, grid.axis == 2 ? ri.hi.z : ri.hi.y, ri.grow, from, to);
        const uint32_t y0 = grid.cells[1] > 1 ? sweepCell(grid, 1, from - grid.width * 1.001f) : 0u;
        const uint32_t y1 = grid.cells[1] > 1 ? sweepCell(grid, 1, to) : 0u;
        for (uint32_t x = x0; x <= x1; ++x) {
            const uint32_t c0 = x * grid.cells[1] + y0, c1 = x * grid.cells[1] + y1;
            const uint32_t q1 = start[c1];
            for (uint32_t q = (c0 ? start[c0 - 1] : 0u) + lane; q < q1; q += 32) {
                const SweepRec rj = recs[q];
                if (!(rj.flags & kBodyWide)) { test(rj); }
            }
        }
    }
}

template <int Unused = 0>
__global__ void __launch_bounds__(256) k_broad_pairs(const __grid_constant__ Batch B, int serial) {
    if (stepAborted(B, serial)) { return; }
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t before = 0;  // items of the worlds before
    for (uint32_t k0 = 0; k0 < B.nBigWorlds; k0 += 32) {
        // A lane a world: its items, and this warp's first among them.
        uint32_t items = 0;
        if (k0 + lane < B.nBigWorlds) {
            const uint32_t w = B.bigWorlds[k0 + lane];
            const WorldInfo& wi = B.info[w];
            items = wi.bodyCount + sweepWides(wi, B.counts[w]) * sweepParts(wi);
        }
        uint32_t upTo = items;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, upTo, o);
            if ((int)lane >= o) { upTo += y; }
        }
        const uint32_t first = (warp + warps - (before + upTo - items) % warps) % warps;
        before += __shfl_sync(0xffffffffu, upTo, 31);
        for (uint32_t left = __ballot_sync(0xffffffffu, first < items); left; left &= left - 1) {
            const int k = __ffs(left) - 1;
            pairsOfWorld(B, B.bigWorlds[k0 + k], __shfl_sync(0xffffffffu, first, k), __shfl_sync(0xffffffffu, items, k), warps, lane);
        }
    }
}

// Calls body for every world of a launch: the big ones by cluster, or the others by CTA and warp.
template <bool Cluster, class Body>
__device__ __forceinline__ void forSomeWorlds(const Batch& B, int slotIndex, const Split& sp, unsigned char* smem, Body&& body) {
    if constexpr (Cluster) {
        forBigWorlds(B, body);
    } else {
        forWorlds(B, slotIndex, sp, smem, body);
    }
}

// The rest of a big world's broadphase: half-space pairs, then the keys sorted and sent to their lists.
template <bool Cluster>
__global__ void __launch_bounds__(kMaxBlock) k_broad_finish(const __grid_constant__ Batch B, const __grid_constant__ Split sp, int serial) {
    __shared__ uint32_t s_class[kMaxGroups][kPairClasses], s_classBase[kMaxGroups][kPairClasses];
    if (stepAborted<Cluster>(B, serial)) { return; }
    forSomeWorlds<Cluster>(B, kSlotBroadFinish, sp, nullptr, [&](const auto& g, uint32_t w, unsigned char*, const StageSizes&) {
        const WorldInfo wi = B.info[w];
        if (wi.bodyCount <= kSweepBodies) { return; }
        WorldCounts& wc = B.counts[w];
        for (uint32_t pl = 0; pl < wi.planeCount; ++pl) {
            const uint32_t gp = B.planeList[wi.planeFirst + pl];
            for (uint32_t b = g.tid; b < wi.bodyCount; b += g.size) { pairPlane(B, wi, gp, wi.bodyFirst + b, &wc.candRaw); }
        }
        g.sync();
        const uint32_t total = *(volatile uint32_t*)&wc.candRaw;
        finishCandidates(B, g, wi, wc, w, total, serial, g.shared(s_class[g.id]), g.shared(s_classBase[g.id]));
    });
}

// ---------------------------------------------------------------------------------------------------------
// Narrowphase and contact bookkeeping (src/world.cpp:872-1025).

__device__ __forceinline__ Vec3 lift(const DBody& a, const DBody& b, const Vec3& normal, float separation, float spec) {
    if (isPlanar(a) || isPlanar(b)) { return zero3(); }
    return separation > spec ? normal * (0.5f * separation) : zero3();
}

// src/world.cpp:1002-1009.
__device__ __forceinline__ bool stillFits(const DContact& c, const DBody& a, const DBody& b, const StepParams& P) {
    if (!(c.flags & kCReusable)) { return false; }
    const float reach = P.reuseDistance;
    if (lengthSquared(unrotate(a.xf.q, b.com - a.com) - c.baseOffset) > reach * reach) { return false; }
    const Quat turn = conjugate(a.xf.q) * b.xf.q;
    return fabsf(dot(turn, c.baseTurn)) >= P.reuseCos;
}

// src/world.cpp:1012-1025.
__device__ __forceinline__ void measurePoint(const DBody& a, const DBody& b, const Vec3& normal, DPoint& p, const StepParams& P) {
    const Vec3 pa = apply(a.xf, p.surfaceA), pb = apply(b.xf, p.surfaceB);
    const Vec3 mid = (pa + pb) * 0.5f;
    p.separation = dot(pb - pa, normal);
    const Vec3 up = lift(a, b, normal, p.separation, P.tol.speculative);
    p.anchorA = mid - up - a.com;
    p.anchorB = mid + up - b.com;
    p.tangentImpulse = p.tangentImpulse - normal * dot(normal, p.tangentImpulse);
}

static __device__ void measureAgain(const DBody& a, const DBody& b, DContact& c, const StepParams& P) {
    c.normal = rotate(a.xf.q, c.localNormal);
    c.tangent1 = perpendicular(c.normal);
    c.tangent2 = cross(c.normal, c.tangent1);
    for (int i = 0; i < c.count; ++i) { measurePoint(a, b, c.normal, c.points[i], P); }
}

// Each new point continues the nearest old point in reach; an old point continued by several new points
// splits its impulse among them (src/world.cpp:102-124).
static __device__ void carryImpulses(const DContact& old, DContact& c, float matchSq) {
    int from[4], claims[4] = { 0, 0, 0, 0 };
    for (int i = 0; i < c.count; ++i) {
        from[i] = -1;
        float bestSq = matchSq;
        for (int k = 0; k < old.count; ++k) {
            const float d = lengthSquared(old.points[k].localA - c.points[i].localA);
            if (d <= bestSq) {
                from[i] = k;
                bestSq = d;
            }
        }
        if (from[i] >= 0) { ++claims[from[i]]; }
    }
    for (int i = 0; i < c.count; ++i) {
        if (from[i] < 0) { continue; }
        const DPoint& o = old.points[from[i]];
        const float share = 1.0f / (float)claims[from[i]];
        c.points[i].normalImpulse = o.normalImpulse * share;
        c.points[i].tangentImpulse = (o.tangentImpulse - c.normal * dot(c.normal, o.tangentImpulse)) * share;
    }
    c.rollingImpulse = old.rollingImpulse;
}

__device__ __forceinline__ int nearestPoint(const DContact& old, const Vec3& localA) {
    int best = -1;
    float bestSq = FLT_MAX;
    for (int k = 0; k < old.count; ++k) {
        const float d = lengthSquared(old.points[k].localA - localA);
        if (d < bestSq) {
            best = k;
            bestSq = d;
        }
    }
    return best;
}

// A pair whose dynamic bodies are locked to the plane n (src/world.cpp:514-518): both bodies are placed in
// the plane, whatever the profiles turn out to be, and marked so the round's placements are kept once every
// pair is done. Returns collidePlanar's answer. Kept out of line: the 3D paths around it need its registers.
static __device__ __noinline__ int collidePlanarPair(const Batch& B, const StepParams& P, const DShape& sa, const DShape& sb,
                                              const Vec3& n, float margin, Manifold& m) {
    DBody& ba = B.bodies[sa.body];
    DBody& bb = B.bodies[sb.body];
    const PlanePose pa = placeInPlane(ba, n);
    const PlanePose pb = placeInPlane(bb, n);
    ba.posePending = 1;
    bb.posePending = 1;
    m.featKind = kFeatNone;
    m.featA = m.featB = -1;
    m.normal = zero3();
    return collidePlanar(B.cx.pt, sa, pa, sb, pb, margin, P.tol.linearSlop, m);
}

// Stores the placements of the round of collisions that just ended for the bodies of one world that were
// placed in it; nothing reads a body's pose while its world is here.
template <class G>
static __device__ void keepPlacements(const Batch& B, const G& g, const WorldInfo& wi) {
    if (wi.planeBody == UINT32_MAX) { return; }
    if (!TF_OK_INDEX(B, wi.planeBody < B.totalBodies, 31, wi.bodyFirst, wi.planeBody)) { return; }
    const Vec3 n = planeNormal(B.bodies[wi.planeBody]);
    for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
        DBody& b = B.bodies[wi.bodyFirst + i];
        if (!b.posePending) { continue; }
        keepPose(b, placeInPlane(b, n));
        b.posePending = 0;
    }
}

// Collides one shape pair over dt as Impl::collidePair does for non-mesh pairs (src/world.cpp:505-533).
// Returns false for a pair this build cannot collide.
template <int Cls = kClassAny>
__device__ bool collidePair(const Batch& B, const StepParams& P, const DShape& sa, const DShape& sb, float dt,
                            Manifold& m, int reuseKind, int reuseA, int reuseB) {
    if (!TF_OK_INDEX(B, (sa.poly < 0 || (uint32_t)sa.poly < B.nPolys) && (sb.poly < 0 || (uint32_t)sb.poly < B.nPolys) &&
                            sa.body < B.totalBodies && sb.body < B.totalBodies,
                     30, sa.body, sb.body)) {
        m.count = 0;
        return true;
    }
    const DBody& ba = B.bodies[sa.body];
    const DBody& bb = B.bodies[sb.body];
    const float travel = relativeTravel(ba, bb, dt);
    const float margin = P.tol.speculative + travel;
    if constexpr (Cls == kClassAny || Cls == kClassPlanar) {
        Vec3 n;
        if (sa.kind != kMesh && sb.kind != kMesh && usePlanar(ba, bb, n)) {
            const int r = collidePlanarPair(B, P, sa, sb, n, margin, m);
            if (r > 0) { return true; }
            if (r < 0) {
                m.count = 0;
                return false;
            }
        }
    }
    const Transform xa = ba.xf * sa.local;
    const Transform xb = bb.xf * sb.local;
    const Motion mo{ ba.v, ba.w, ba.com, bb.v, bb.w, bb.com, dt, travel > P.tol.speculative };
    constexpr int Shapes = Cls == kClassPlanar ? kClassAny : Cls;
    return collideShapes<Shapes>(B.cx, sa, xa, sb, xb, margin, mo, m, reuseKind, reuseA, reuseB);
}

// First index in [0, n) whose key is not below key.
__device__ __forceinline__ uint32_t lowerKey(const DContact* c, uint32_t n, uint64_t key) {
    uint32_t lo = 0, hi = n;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (c[mid].key < key) {
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    return lo;
}

// One candidate (src/world.cpp:883-959), in two halves. narrowKeep finds the pair's old contacts [lo, hi) and keeps and
// measures the old contact when the pair barely moved; narrowAnew collides a pair it did not keep and carries the old
// impulses over.
__device__ __forceinline__ void narrowWakes(const Batch& B, const DShape& sa, const DShape& sb, const DBody& ba, const DBody& bb,
                                            WorldCounts& wc) {
    if (ba.type == kDynamic && !ba.awake && movingAwake(bb)) {
        B.wakeMark[sa.body] = 1;
        wc.wakePending = 1;
    }
    if (bb.type == kDynamic && !bb.awake && movingAwake(ba)) {
        B.wakeMark[sb.body] = 1;
        wc.wakePending = 1;
    }
}

// measureAgain and the shapes' surface from the old contact into the new one, a point at a time in registers.
__device__ __forceinline__ void keepContact(const DBody& a, const DBody& b, const DShape& sa, const DShape& sb, const DContact& old,
                                            DContact& out, const StepParams& P) {
    constexpr int kHead = offsetof(DContact, points) / 16;
    DContact c;
    const float4* from = reinterpret_cast<const float4*>(&old);
#pragma unroll
    for (int k = 0; k < kHead; ++k) {
        const float4 piece = from[k];
        memcpy(reinterpret_cast<unsigned char*>(&c) + 16 * k, &piece, 16);
    }
    c.normal = rotate(a.xf.q, c.localNormal);
    c.tangent1 = perpendicular(c.normal);
    c.tangent2 = cross(c.normal, c.tangent1);
    c.boundsFirst = c.boundsCount = 0;
    c.friction = sqrtf(sa.friction * sb.friction);
    c.restitution = maxf(sa.restitution, sb.restitution);
    c.rollingResistance = maxf(sa.rollingResistance, sb.rollingResistance);
    float4* to = reinterpret_cast<float4*>(&out);
#pragma unroll
    for (int k = 0; k < kHead; ++k) {
        float4 piece;
        memcpy(&piece, reinterpret_cast<const unsigned char*>(&c) + 16 * k, 16);
        to[k] = piece;
    }
    for (int i = 0; i < 4; ++i) {
        DPoint p = old.points[i];
        if (i < c.count) { measurePoint(a, b, c.normal, p, P); }
        out.points[i] = p;
    }
}

// Whether nothing is left to do.
__device__ __forceinline__ bool narrowKeep(const Batch& B, const StepParams& P, const WorldInfo& wi, WorldCounts& wc, uint32_t i,
                                           const DContact* old, uint32_t oldCount, uint32_t& lo, uint32_t& hi) {
    const uint64_t key = B.cand[wi.candFirst + i];
    const uint32_t ia = (uint32_t)(key >> 32), ib = (uint32_t)(key & 0xffffffffu);
    if (!TF_OK_INDEX(B, ia < wi.shapeCount && ib < wi.shapeCount, 1, wi.bodyFirst, ia)) {
        B.stageUsed[wi.candFirst + i] = 0;
        return true;
    }
    const DShape& sa = B.shapes[wi.shapeFirst + ia];
    const DShape& sb = B.shapes[wi.shapeFirst + ib];
    if (!TF_OK_INDEX(B, sa.body - wi.bodyFirst < wi.bodyCount && sb.body - wi.bodyFirst < wi.bodyCount, 2,
                     wi.bodyFirst, sa.body)) {
        B.stageUsed[wi.candFirst + i] = 0;
        return true;
    }
    if (!TF_OK_INDEX(B, oldCount <= wi.contactCap, 3, wi.bodyFirst, oldCount)) {
        B.stageUsed[wi.candFirst + i] = 0;
        return true;
    }
    lo = lowerKey(old, oldCount, key);
    hi = lo;
    while (hi < oldCount && old[hi].key == key) { ++hi; }
    if (lo == hi) { return false; }
    const DBody ba = readBody<kBodySolve | kBodyPose | kBodyCom | kBodyInertia>(B.bodies[sa.body]);
    const DBody bb = readBody<kBodySolve | kBodyPose | kBodyCom | kBodyInertia>(B.bodies[sb.body]);
    for (uint32_t it = lo; it < hi; ++it) {
        if (!stillFits(old[it], ba, bb, P)) { return false; }
    }
    DContact& out = B.stage[wi.candFirst + i];
    if (hi - lo > 1) { atomicOr(&wc.flags, kDevUnsupported); }
    keepContact(ba, bb, sa, sb, old[lo], out, P);
    narrowWakes(B, sa, sb, ba, bb, wc);
    B.stageUsed[wi.candFirst + i] = 1;
    return true;
}

template <int Cls>
__device__ __forceinline__ void narrowAnew(const Batch& B, const StepParams& P, const WorldInfo& wi, WorldCounts& wc, uint32_t i,
                                           const DContact* old, uint32_t lo, uint32_t hi) {
    const uint64_t key = B.cand[wi.candFirst + i];
    const uint32_t gsa = wi.shapeFirst + (uint32_t)(key >> 32), gsb = wi.shapeFirst + (uint32_t)(key & 0xffffffffu);
    const DShape sa = B.shapes[gsa];
    const DShape sb = B.shapes[gsb];
    const DBody& ba = B.bodies[sa.body];
    const DBody& bb = B.bodies[sb.body];
    const bool touched = lo < hi && (old[lo].flags & kCTouched);
    DContact& out = B.stage[wi.candFirst + i];
    uint8_t used = 0;
    {
        Manifold m;
        if (!collidePair<Cls>(B, P, sa, sb, P.dt, m, kFeatNone, -1, -1)) { atomicOr(&wc.flags, kDevUnsupported); }
        if (m.count > 0) {
            DContact c{};
            c.key = key;
            c.part = 0;
            c.shapeA = gsa;
            c.shapeB = gsb;
            c.bodyA = sa.body;
            c.bodyB = sb.body;
            c.flags = touched ? kCTouched : 0u;
            c.featKind = m.featKind;
            c.featA = m.featA;
            c.featB = m.featB;
            c.boundsFirst = c.boundsCount = 0;
            c.normal = m.normal;
            c.tangent1 = perpendicular(m.normal);
            c.tangent2 = cross(m.normal, c.tangent1);
            c.count = m.count;
            for (int k = 0; k < m.count; ++k) {
                DPoint& p = c.points[k];
                const Vec3 pos = m.points[k].position;
                const float sep = m.points[k].separation;
                const Vec3 half = m.normal * (0.5f * sep);
                p.surfaceA = applyInverse(ba.xf, pos - half);
                p.surfaceB = applyInverse(bb.xf, pos + half);
                p.localA = applyInverse(ba.xf, pos);
                p.separation = sep;
                const Vec3 up = lift(ba, bb, m.normal, sep, P.tol.speculative);
                p.anchorA = pos - up - ba.com;
                p.anchorB = pos + up - bb.com;
            }
            // remember (src/world.cpp:995-1000).
            c.localNormal = unrotate(ba.xf.q, c.normal);
            c.baseOffset = unrotate(ba.xf.q, bb.com - ba.com);
            c.baseTurn = conjugate(ba.xf.q) * bb.xf.q;
            c.flags |= kCReusable;
            // The old contact of the pair whose normal is closest (src/world.cpp:543-549).
            int best = -1;
            for (uint32_t it = lo; it < hi; ++it) {
                if (old[it].count > 0 && (best < 0 || dot(old[it].normal, c.normal) > dot(old[best].normal, c.normal))) {
                    best = (int)it;
                }
            }
            if (best >= 0) { carryImpulses(old[best], c, P.tol.speculative * P.tol.speculative); }
            out = c;
            used = 1;
        }
    }
    if (used) {
        out.friction = sqrtf(sa.friction * sb.friction);
        out.restitution = maxf(sa.restitution, sb.restitution);
        out.rollingResistance = maxf(sa.rollingResistance, sb.rollingResistance);
        narrowWakes(B, sa, sb, ba, bb, wc);
    }
    B.stageUsed[wi.candFirst + i] = used;
}

// A pair with a mesh over dt (src/world.cpp:505-533): manifolds with normals from sa to sb, into out. Warp: the
// warp's lanes collide the triangles together (collideMeshWarp, warpFound its shared room); else one thread.
template <bool Warp>
static __device__ int collideMeshPair(const Batch& B, const StepParams& P, const DShape& sa, const DShape& sb, float dt,
                               Manifold* out, int& outCount, MeshBounds* bounds, Manifold* warpFound = nullptr,
                               uint32_t lane = 0) {
    const DBody& ba = B.bodies[sa.body];
    const DBody& bb = B.bodies[sb.body];
    const float travel = relativeTravel(ba, bb, dt);
    const float margin = P.tol.speculative + travel;
    const Transform xa = ba.xf * sa.local;
    const Transform xb = bb.xf * sb.local;
    const Motion mo{ ba.v, ba.w, ba.com, bb.v, bb.w, bb.com, dt, travel > P.tol.speculative };
    const bool meshFirst = sa.kind == kMesh;
    const DShape& mesh = meshFirst ? sa : sb;
    const DShape& other = meshFirst ? sb : sa;
    const Transform& xm = meshFirst ? xa : xb;
    const Transform& xo = meshFirst ? xb : xa;
    const Motion m = meshFirst ? mo : mo.swapped();
    int status;
    if constexpr (Warp) {
        status = collideMeshWarp(B.cx, mesh, xm, other, xo, margin, m, out, outCount, bounds, warpFound, lane);
    } else {
        status = collideMesh(B.cx, mesh, xm, other, xo, margin, m, out, outCount, bounds);
    }
    if (!meshFirst) {
        for (int i = 0; i < outCount; ++i) { out[i].normal = -out[i].normal; }
    }
    return status;
}

// A warp's shared room for one mesh pair: its triangle manifolds and the triangles it rules out. The mesh pair
// kernels run 4 warps to a CTA.
struct MeshWarpRoom {
    Manifold found[kMaxMeshFound];
    TriangleBound ruled[kMaxMeshBounds];
};
constexpr int kMeshWarps = 4;

// A contact of pair (sa, sb) from one manifold (src/world.cpp:912-939): points on both surfaces, anchors,
// tangents and the reuse record.
static __device__ void contactFromManifold(const StepParams& P, const DBody& ba, const DBody& bb, const Manifold& m, DContact& c) {
    c.featKind = m.featKind;
    c.featA = m.featA;
    c.featB = m.featB;
    c.normal = m.normal;
    c.tangent1 = perpendicular(m.normal);
    c.tangent2 = cross(m.normal, c.tangent1);
    c.count = m.count;
    for (int k = 0; k < m.count; ++k) {
        DPoint& p = c.points[k];
        const Vec3 pos = m.points[k].position;
        const float sep = m.points[k].separation;
        const Vec3 half = m.normal * (0.5f * sep);
        p.surfaceA = applyInverse(ba.xf, pos - half);
        p.surfaceB = applyInverse(bb.xf, pos + half);
        p.localA = applyInverse(ba.xf, pos);
        p.separation = sep;
        const Vec3 up = lift(ba, bb, m.normal, sep, P.tol.speculative);
        p.anchorA = pos - up - ba.com;
        p.anchorB = pos + up - bb.com;
    }
    c.localNormal = unrotate(ba.xf.q, c.normal);
    c.baseOffset = unrotate(ba.xf.q, bb.com - ba.com);
    c.baseTurn = conjugate(ba.xf.q) * bb.xf.q;
    c.flags |= kCReusable;
}

// Stops this step (the host grows the world's lists and runs it again) when a mesh pair's parts or triangle
// bounds do not fit the world's room for them.
static __device__ void meshRoomOverflow(const Batch& B, const WorldInfo& wi, WorldCounts& wc, int serial) {
    atomicOr(&wc.flags, kDevPairOverflow);
    atomicMax(&wc.candNeeded, 2 * wi.candCap);
    atomicMin(B.abortStep, (uint32_t)serial);
}

// One mesh candidate (src/world.cpp:883-959): the old contacts kept and measured again when the pair barely
// moved, else one contact per manifold the mesh collision makes, each carrying the impulses of the old
// contact whose normal is closest. The first contact goes to the candidate's staging slot, the others to
// the world's extra parts. A fast pair records the triangles it ruled out, for the refresh within the step.
// Warp: every lane of the warp calls it alike with the warp's room; the lanes collide the triangles together and
// lane 0 writes the results.
template <bool Warp>
static __device__ void narrowMesh(const Batch& B, const StepParams& P, const WorldInfo& wi, WorldCounts& wc, uint32_t i,
                           const DContact* old, uint32_t oldCount, int serial, MeshWarpRoom* room = nullptr,
                           uint32_t lane = 0) {
    const bool lead = !Warp || lane == 0;
    if (lead) { B.stageUsed[wi.candFirst + i] = 0; }
    const uint64_t key = B.cand[wi.candFirst + i];
    const uint32_t ia = (uint32_t)(key >> 32), ib = (uint32_t)(key & 0xffffffffu);
    if (!TF_OK_INDEX(B, ia < wi.shapeCount && ib < wi.shapeCount, 34, wi.bodyFirst, ia)) { return; }
    const uint32_t gsa = wi.shapeFirst + ia, gsb = wi.shapeFirst + ib;
    const DShape sa = B.shapes[gsa];
    const DShape sb = B.shapes[gsb];
    if (!TF_OK_INDEX(B, oldCount <= wi.contactCap, 35, wi.bodyFirst, oldCount)) { return; }
    const DBody& ba = B.bodies[sa.body];
    const DBody& bb = B.bodies[sb.body];
    const uint32_t lo = lowerKey(old, oldCount, key);
    uint32_t hi = lo;
    while (hi < oldCount && old[hi].key == key) { ++hi; }
    const bool hasOld = lo < hi;
    bool keep = hasOld;
    for (uint32_t it = lo; it < hi && keep; ++it) { keep = stillFits(old[it], ba, bb, P); }
    const bool touched = hasOld && (old[lo].flags & kCTouched);

    Manifold found[kMaxMeshParts];
    int n = 0;
    uint32_t boundsFirst = 0, boundsCount = 0;
    if (keep) {
        if (!lead) { return; }
        n = (int)(hi - lo);
        if (n > kMaxMeshParts) {
            atomicOr(&wc.flags, kDevUnsupported);
            return;
        }
    } else {
        const bool record = relativeTravel(ba, bb, P.dt) > P.tol.speculative;
        TriangleBound own[Warp ? 1 : kMaxMeshBounds];
        TriangleBound* ruled = Warp ? room->ruled : own;
        MeshBounds mb{ record ? ruled : nullptr, 0, nullptr, 0, 0.0f };
        const int status = collideMeshPair<Warp>(B, P, sa, sb, P.dt, found, n, &mb, Warp ? room->found : nullptr, lane);
        if (!lead) { return; }
        if (status != kMeshOk) {
            atomicOr(&wc.flags, kDevUnsupported);
            return;
        }
        if (mb.foundCount > 0) {
            // By triangle, as the reference sorts each pair's run.
            for (int x = 1; x < mb.foundCount; ++x) {
                const TriangleBound t = ruled[x];
                int y = x - 1;
                while (y >= 0 && ruled[y].triangle > t.triangle) {
                    ruled[y + 1] = ruled[y];
                    --y;
                }
                ruled[y + 1] = t;
            }
            boundsFirst = atomicAdd(&wc.boundsCount, (uint32_t)mb.foundCount);
            boundsCount = (uint32_t)mb.foundCount;
            if (boundsFirst + boundsCount > wi.boundsCap) {
                meshRoomOverflow(B, wi, wc, serial);
                return;
            }
            for (int x = 0; x < mb.foundCount; ++x) { B.triBounds[wi.boundsFirst + boundsFirst + x] = ruled[x]; }
        }
    }
    if (n == 0) { return; }
    uint32_t extra = 0;
    if (n > 1) {
        extra = atomicAdd(&wc.partCount, (uint32_t)(n - 1));
        if (extra + (uint32_t)(n - 1) > wi.partCap) {
            meshRoomOverflow(B, wi, wc, serial);
            return;
        }
    }
    for (int k = 0; k < n; ++k) {
        DContact& out = k == 0 ? B.stage[wi.candFirst + i] : B.stageExtra[wi.partFirst + extra + (uint32_t)(k - 1)];
        if (keep) {
            out = old[lo + (uint32_t)k];
            measureAgain(ba, bb, out, P);
            out.boundsFirst = out.boundsCount = 0;
        } else {
            DContact c{};
            c.key = key;
            c.part = (uint32_t)k;
            c.shapeA = gsa;
            c.shapeB = gsb;
            c.bodyA = sa.body;
            c.bodyB = sb.body;
            c.flags = touched ? kCTouched : 0u;
            contactFromManifold(P, ba, bb, found[k], c);
            c.boundsFirst = boundsFirst;
            c.boundsCount = boundsCount;
            int best = -1;
            for (uint32_t it = lo; it < hi; ++it) {
                if (old[it].count > 0 && (best < 0 || dot(old[it].normal, c.normal) > dot(old[best].normal, c.normal))) {
                    best = (int)it;
                }
            }
            if (best >= 0) { carryImpulses(old[best], c, P.tol.speculative * P.tol.speculative); }
            out = c;
        }
        out.friction = sqrtf(sa.friction * sb.friction);
        out.restitution = maxf(sa.restitution, sb.restitution);
        out.rollingResistance = maxf(sa.rollingResistance, sb.rollingResistance);
    }
    if (ba.type == kDynamic && !ba.awake && movingAwake(bb)) {
        B.wakeMark[sa.body] = 1;
        wc.wakePending = 1;
    }
    if (bb.type == kDynamic && !bb.awake && movingAwake(ba)) {
        B.wakeMark[sb.body] = 1;
        wc.wakePending = 1;
    }
    B.stagePart[wi.candFirst + i] = extra;
    B.stageUsed[wi.candFirst + i] = (uint8_t)n;
}

// Calls f(item, whether it is one of the list's) for the items of a list spread over the whole grid, a warp's lanes at
// once: a lane each when the list has items for every lane, and only as many lanes of a warp as it takes when it is
// shorter, down to one. The pairs of a list take different paths through the same code, which a warp walks one after the
// other: of few pairs, each gets a warp to itself. (28 pairs of boxes: 40 us of collisions a step on one warp, 26 spread;
// 64 uneven worlds: 85 and 54, their refreshes 230 and 165.) `turn` of `turns` lists that one launch works on moves a
// list's first warp, so that short lists do not queue on the same warps.
template <class F>
__device__ __forceinline__ void forSpreadItems(uint32_t n, uint32_t turn, uint32_t turns, F f) {
    const uint32_t lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t lanes = min(32u, (n + warps - 1) / warps);
    // Consecutive warps lie on different CTAs while the list is short, and in one, whose items share bodies, when it is
    // not.
    const uint32_t at = lanes < 32 ? (threadIdx.x >> 5) * gridDim.x + blockIdx.x : blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t warp = (at + warps - warps / turns * turn) % warps;
    for (uint32_t first = warp * lanes; first < n; first += warps * lanes) {
        const uint32_t item = first + lane;
        f(item, lane < lanes && item < n, first + warps * lanes >= n);
    }
}

// A convex pair that was not kept, waiting for its warp to have a pair for every lane.
struct AnewPair {
    uint32_t world, candidate, lo, hi;
};

// The candidate pairs of one class, over every world, one thread per pair (src/world.cpp:874-960); each
// result lands in the pair's own staging slot, so pairs need no order among themselves.
//
// Of convex pairs, which cost the most to collide, a warp first keeps those that can be kept and queues the others, and
// collides them once there is one for every lane. (Collided where they were met, the pairs of 1024 impact worlds, three
// quarters of them kept, left 6.4 of 32 lanes at work: 1644 us of pair collisions a step, and 920 this way.)
template <int Cls>
__device__ __forceinline__ void collideClass(const Batch& B, const StepParams& P, int serial, uint32_t turn = 0, uint32_t turns = 1) {
    const uint32_t n = *(volatile uint32_t*)(B.work + kSlotCandItems + Cls);
    const uint2* items = B.candItems + (size_t)Cls * B.candItemStride;
    if constexpr (Cls == kClassConvex) {
        __shared__ AnewPair s_anew[256 / 32][64];
        AnewPair* queue = s_anew[threadIdx.x >> 5];
        const uint32_t lane = threadIdx.x & 31;
        uint32_t queued = 0;
        forSpreadItems(n, turn, turns, [&](uint32_t item, bool mine, bool last) {
            bool anew = false;
            AnewPair pair;
            if (mine) {
                const uint2 it = items[item];
                const WorldInfo& wi = B.info[it.x];
                WorldCounts& wc = B.counts[it.x];
                pair = { it.x, it.y, 0, 0 };
                anew = !narrowKeep(B, P, wi, wc, it.y, B.previous + wi.contactFirst, wc.contactCount, pair.lo, pair.hi);
            }
            const uint32_t found = __ballot_sync(0xffffffffu, anew);
            if (anew) { queue[queued + __popc(found & ((1u << lane) - 1u))] = pair; }
            queued += __popc(found);
            __syncwarp();
            while (queued >= 32 || (last && queued > 0)) {
                const uint32_t now = min(queued, 32u);
                queued -= now;
                if (lane < now) {
                    const AnewPair p = queue[queued + lane];
                    const WorldInfo wi = B.info[p.world];
                    narrowAnew<Cls>(B, P, wi, B.counts[p.world], p.candidate, B.previous + wi.contactFirst, p.lo, p.hi);
                }
                __syncwarp();
            }
        });
        return;
    }
    forSpreadItems(n, turn, turns, [&](uint32_t item, bool mine, bool) {
        if (!mine) { return; }
        const uint2 it = items[item];
        const WorldInfo wi = B.info[it.x];
        WorldCounts& wc = B.counts[it.x];
        const DContact* old = B.previous + wi.contactFirst;
        if constexpr (Cls == kClassMesh) {
            narrowMesh<false>(B, P, wi, wc, it.y, old, wc.contactCount, serial);
        } else {
            uint32_t lo, hi;
            if (!narrowKeep(B, P, wi, wc, it.y, old, wc.contactCount, lo, hi)) { narrowAnew<Cls>(B, P, wi, wc, it.y, old, lo, hi); }
        }
    });
}

// The mesh candidates over every world, a warp per pair, the warp's lanes over the pair's triangles: a pair
// near many triangles (a large or fast shape on a fine mesh) no longer holds a whole launch on one thread.
// Launched with at most kMeshWarps warps to a CTA.
__device__ __forceinline__ void collideMeshPairs(const Batch& B, const StepParams& P, int serial) {
    __shared__ MeshWarpRoom s_rooms[kMeshWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t perCta = min(blockDim.x >> 5, (uint32_t)kMeshWarps);  // warps past the rooms stay idle
    if (warp >= perCta) { return; }
    const uint32_t n = *(volatile uint32_t*)(B.work + kSlotCandItems + kClassMesh);
    const uint2* items = B.candItems + (size_t)kClassMesh * B.candItemStride;
    const uint32_t warps = gridDim.x * perCta;
    for (uint32_t item = blockIdx.x * perCta + warp; item < n; item += warps) {
        const uint2 it = items[item];
        const WorldInfo wi = B.info[it.x];
        WorldCounts& wc = B.counts[it.x];
        narrowMesh<true>(B, P, wi, wc, it.y, B.previous + wi.contactFirst, wc.contactCount, serial, &s_rooms[warp], lane);
        __syncwarp();
    }
}

template <int Cls>
__global__ void __launch_bounds__(256) k_collide(const __grid_constant__ Batch B, const __grid_constant__ StepParams P,
                                                 int serial) {
    if (stepAborted(B, serial)) { return; }
    if constexpr (Cls == kClassMesh) {
        collideMeshPairs(B, P, serial);
    } else {
        collideClass<Cls>(B, P, serial);
    }
}

// Small batches collide every pair class in one launch, each class's list in turn over the whole grid (the
// classes' pairs are disjoint); large batches launch a kernel per class, which keeps a warp on one code path.
template <int Unused = 0>
__global__ void __launch_bounds__(256) k_collide_all(const __grid_constant__ Batch B, const __grid_constant__ StepParams P,
                                                     int serial) {
    if (stepAborted(B, serial)) { return; }
    collideClass<kClassSpheres>(B, P, serial, 0, 6);
    collideClass<kClassSpherePoly>(B, P, serial, 1, 6);
    collideClass<kClassPlane>(B, P, serial, 2, 6);
    collideClass<kClassConvex>(B, P, serial, 3, 6);
    collideClass<kClassPlanar>(B, P, serial, 4, 6);
    collideClass<kClassMesh>(B, P, serial, 5, 6);
}

__device__ __forceinline__ bool keyLess(uint64_t ka, uint32_t pa, uint64_t kb, uint32_t pb) {
    return ka != kb ? ka < kb : pa < pb;
}

// Copies the contacts of a warp's first n lanes, each lane's from and to, the warp over one contact's consecutive bytes
// after another's. (A lane each, a load of the warp touched 32 contacts' lines for 16 bytes of each: 492 us of the
// narrowphase a step for 1024 impact worlds of 487 contacts each, 322 this way.)
static __device__ void copyContacts(uint32_t lane, uint32_t n, const DContact* from, DContact* to) {
    constexpr uint32_t kPieces = sizeof(DContact) / 16, kAtOnce = 5;
    static_assert(sizeof(DContact) % 16 == 0, "a contact is whole pieces");
    const uint32_t total = n * kPieces;
    for (uint32_t base = 0; base < total; base += 32 * kAtOnce) {
        float4 piece[kAtOnce];
        float4* out[kAtOnce];
#pragma unroll
        for (uint32_t u = 0; u < kAtOnce; ++u) {
            const uint32_t q = base + 32 * u + lane, who = q < total ? q / kPieces : 0u;
            const float4* src = reinterpret_cast<const float4*>(
                __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(from), (int)who));
            float4* dst = reinterpret_cast<float4*>(
                __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(to), (int)who));
            out[u] = q < total ? dst + (q - who * kPieces) : nullptr;
            if (out[u]) { piece[u] = src[q - who * kPieces]; }
        }
#pragma unroll
        for (uint32_t u = 0; u < kAtOnce; ++u) {
            if (out[u]) { *out[u] = piece[u]; }
        }
    }
}

template <bool Cluster>
__global__ void __launch_bounds__(kMaxBlock) k_narrowphase(const __grid_constant__ Batch B, const __grid_constant__ StepParams P, const __grid_constant__ Split sp, int serial) {
    if (stepAborted<Cluster>(B, serial)) { return; }
    forSomeWorlds<Cluster>(B, kSlotNarrow, sp, nullptr, [&](const auto& g, uint32_t w, unsigned char*, const StageSizes&) {
        const WorldInfo wi = B.info[w];
        WorldCounts& wc = B.counts[w];
        if (g.tid == 0) {
            wc.touchEvents = 0;
            wc.hitEvents = 0;
            wc.touching = 0;
        }
        keepPlacements(B, g, wi);
        const uint32_t nc = wc.candCount;
        const uint32_t oldCount = wc.contactCount;
        const DContact* old = B.previous + wi.contactFirst;
        const uint32_t cf = wi.contactFirst;
        // Every candidate's contacts in part order: the first in its staging slot, the others (mesh pairs) in
        // the world's extra parts, named with the high bit set.
        const uint32_t nC = groupExpand(
            g, nc, [&](uint32_t i) { return (uint32_t)B.stageUsed[wi.candFirst + i]; },
            [&](uint32_t i, uint32_t pos, uint32_t k) {
                const uint32_t x = k == 0 ? i : (0x80000000u | (B.stagePart[wi.candFirst + i] + k - 1));
                const DContact* c = k == 0 ? B.stage + wi.candFirst + i : B.stageExtra + wi.partFirst + (x & 0x7fffffffu);
                B.mergeKeyA[cf + pos] = c->key;
                B.mergePartA[cf + pos] = c->part;
                B.mergeIdxA[cf + pos] = x;
            });
        // Contacts of pairs where nothing moves and one body is dynamic (asleep) stay as they were
        // (src/world.cpp:961-988).
        auto keepOld = [&](uint32_t j) {
            const DContact& c = old[j];
            if (!TF_OK_INDEX(B, c.bodyA - wi.bodyFirst < wi.bodyCount && c.bodyB - wi.bodyFirst < wi.bodyCount, 4,
                             wi.bodyFirst, j)) {
                return false;
            }
            const DBody& a = B.bodies[c.bodyA];
            const DBody& b = B.bodies[c.bodyB];
            if ((c.flags & kCRemoved) || movingAwake(a) || movingAwake(b)) { return false; }
            return !(a.type != kDynamic && b.type != kDynamic);
        };
        const uint32_t nK = groupCompact(
            g, oldCount, keepOld,
            [&](uint32_t j, uint32_t pos) {
                B.mergeKeyB[cf + pos] = old[j].key;
                B.mergePartB[cf + pos] = old[j].part;
                B.mergeIdxB[cf + pos] = j;
            });
        const uint32_t total = nC + nK;
        if (total > wi.contactCap) {
            if (g.tid == 0) {
                wc.flags |= kDevContactOverflow;
                wc.contactNeeded = max(wc.contactNeeded, total);
                atomicMin(B.abortStep, (uint32_t)serial);
            }
            g.sync();
            return;
        }
        // Stable merge by (key, part): collided contacts first among equals, as std::inplace_merge keeps them.
        for (uint32_t x = g.tid; x - g.lane < nC; x += g.size) {
            const uint64_t k = x < nC ? B.mergeKeyA[cf + x] : 0;
            const uint32_t p = x < nC ? B.mergePartA[cf + x] : 0;
            uint32_t l = 0, h = x < nC ? nK : 0;
            while (l < h) {
                const uint32_t mid = (l + h) >> 1;
                if (keyLess(B.mergeKeyB[cf + mid], B.mergePartB[cf + mid], k, p)) {
                    l = mid + 1;
                } else {
                    h = mid;
                }
            }
            const uint32_t src = x < nC ? B.mergeIdxA[cf + x] : 0;
            const DContact* from = (src & 0x80000000u) ? B.stageExtra + wi.partFirst + (src & 0x7fffffffu)
                                                        : B.stage + wi.candFirst + src;
            copyContacts(g.lane, min(nC - (x - g.lane), 32u), from, B.contacts + cf + x + l);
        }
        for (uint32_t y = g.tid; y - g.lane < nK; y += g.size) {
            const uint64_t k = y < nK ? B.mergeKeyB[cf + y] : 0;
            const uint32_t p = y < nK ? B.mergePartB[cf + y] : 0;
            uint32_t l = 0, h = y < nK ? nC : 0;
            while (l < h) {
                const uint32_t mid = (l + h) >> 1;
                if (!keyLess(k, p, B.mergeKeyA[cf + mid], B.mergePartA[cf + mid])) {
                    l = mid + 1;
                } else {
                    h = mid;
                }
            }
            const uint32_t src = y < nK ? B.mergeIdxB[cf + y] : 0;
            copyContacts(g.lane, min(nK - (y - g.lane), 32u), old + src, B.contacts + cf + y + l);
        }
        // A touching pair whose old contacts were dropped and that was not collided again has ended
        // (src/world.cpp:963-981): one event per pair, from its first such contact.
        for (uint32_t j = g.tid; j < oldCount; j += g.size) {
            const uint64_t key = old[j].key;
            if (!(old[j].flags & kCTouched) || keepOld(j)) { continue; }
            bool first = true;
            for (uint32_t k = j; k > 0 && old[k - 1].key == key && first; --k) {
                first = !((old[k - 1].flags & kCTouched) && !keepOld(k - 1));
            }
            if (!first) { continue; }
            uint32_t l = 0, h = nC;
            while (l < h) {
                const uint32_t mid = (l + h) >> 1;
                if (B.mergeKeyA[cf + mid] < key) {
                    l = mid + 1;
                } else {
                    h = mid;
                }
            }
            if (l < nC && B.mergeKeyA[cf + l] == key) { continue; }
            const uint32_t at = atomicAdd(&wc.touchEvents, 1u);
            B.touchEvents[2 * (size_t)cf + at] = TouchEvent{ key, 0u, 0u };
        }
        g.sync();
        if (g.tid == 0) {
            wc.nextContactCount = total;
            wc.contactNeeded = max(wc.contactNeeded, total);
        }
        g.sync();
    });
}

// ---------------------------------------------------------------------------------------------------------
// Waking (src/world.cpp:705-735): sleeping bodies a moving body reached wake, and so does everything linked
// to them by a contact with points. Runs on the group's first thread; it is rare.

template <int Unused = 0>
__global__ void __launch_bounds__(kMaxBlock) k_wake(const __grid_constant__ Batch B, const __grid_constant__ Split sp, int serial) {
    if (stepAborted(B, serial)) { return; }
    forWorlds(B, kSlotWake, sp, nullptr, [&](const Group& g, uint32_t w, unsigned char*, const StageSizes&) {
        if (g.tid != 0) { return; }
        const WorldInfo wi = B.info[w];
        WorldCounts& wc = B.counts[w];
        if (!wc.wakePending) { return; }
        wc.wakePending = 0;
        uint32_t* stack = B.unionParent + wi.bodyFirst;
        uint32_t top = 0;
        for (uint32_t i = 0; i < wi.bodyCount; ++i) {
            const uint32_t gb = wi.bodyFirst + i;
            if (!B.wakeMark[gb]) { continue; }
            const DBody& b = B.bodies[gb];
            if (b.alive && b.type == kDynamic && !b.awake && top < wi.bodyCount) {
                stack[top++] = gb;
            } else {
                B.wakeMark[gb] = 0;
            }
        }
        wakeStack(B, wi, B.contacts + wi.contactFirst, wc.nextContactCount, stack, top);
    });
}

// ---------------------------------------------------------------------------------------------------------
// Step state, lists, preparation and coloring (src/world.cpp:1589-1657, src/lanes.cpp:356-407).

constexpr uint32_t kNone = 0x7fffffffu;
constexpr uint32_t kNotColorable = 0x80000000u;

// ---------------------------------------------------------------------------------------------------------
// The laned contacts' solver record.
//
// The reference solves a color's contacts from a packed per-batch record rather than from its Contact
// (ContactLanes, src/internal.h:579-621, built by prepareBatch, src/lanes.cpp:66-110). Here each laned contact
// has one at its slot (contactFirst + its position in the world's colored list), component-major within tiles of
// kRowTile slots: component k of a tile's slots is 128 consecutive bytes, so the lanes of a color read consecutive
// 16-byte words, and every component of a record lies at a constant offset from its first. It holds what the
// substep's passes read of a contact and its points, and the impulses, which stay in it from k_prepare to
// k_finish (k_finish writes them back into the contact; a mid-step refresh takes them back first and builds
// the record again). Of each axis (makeAxis, src/solver.cpp:5-17) it keeps the velocity changes per unit
// impulse and the effective mass; the linear ones are the same for every point of a contact and are kept once;
// the lever arms, a cross product each, are formed again by every pass, with makeAxis's own arithmetic, so each
// pass sees the bits of the axes as built. 144 bytes a point and 144 a contact, against 240 bytes a point of
// stored axes plus the lines of the 560-byte contact a pass read before.
enum RowWord : int {
    kRowHead = 0,    // bodyA, bodyB (global), point count, contact index within the world (as integer bits)
    kRowNormal = 1,  // normal, friction
    kRowT1 = 2,      // tangent1, unused
    kRowT2 = 3,      // tangent2, unused
    kRowLinear = 4,  // 5 words: linearA, linearB of the normal, tangent1 and tangent2 axes (18 floats, 2 unused)
    kRowPoint = 9,   // point i, 9 words from kRowPoint + 9 i: anchorA and adjusted separation; anchorB and normal
                     // mass; tangent masses, normal impulse, largest normal impulse; tangent impulse; then 5
                     // words: angularA, angularB of the normal, tangent1 and tangent2 axes (2 floats unused)
    kRowPointWords = 9,
    kRowWords = kRowPoint + 4 * kRowPointWords
};
constexpr uint32_t kNoSlot = 0xffffffffu;
constexpr uint32_t kRowTile = 8;  // slots of a tile; a record's next component is this many float4 on

__device__ __forceinline__ float4* rowOf(const Batch& B, uint32_t slot) {
    return B.rows + (size_t)(slot / kRowTile) * (kRowTile * kRowWords) + slot % kRowTile;
}

__device__ __forceinline__ float4 f4(const Vec3& v, float w) { return make_float4(v.x, v.y, v.z, w); }
__device__ __forceinline__ Vec3 xyz(const float4& v) { return Vec3{ v.x, v.y, v.z }; }

// Six vectors (18 floats) into 5 consecutive components of a record, from component `first`, and back.
__device__ __forceinline__ void putSix(float4* R, int first, const Vec3 (&v)[6]) {
    constexpr int S = kRowTile;
    R[first * S] = make_float4(v[0].x, v[0].y, v[0].z, v[1].x);
    R[(first + 1) * S] = make_float4(v[1].y, v[1].z, v[2].x, v[2].y);
    R[(first + 2) * S] = make_float4(v[2].z, v[3].x, v[3].y, v[3].z);
    R[(first + 3) * S] = make_float4(v[4].x, v[4].y, v[4].z, v[5].x);
    R[(first + 4) * S] = make_float4(v[5].y, v[5].z, 0.0f, 0.0f);
}

struct SixVec {
    Vec3 v[6];
};

template <int S = kRowTile>
__device__ __forceinline__ SixVec getSix(const float4* R, int first) {
    const float4 a = R[first * S], b = R[(first + 1) * S], c = R[(first + 2) * S], d = R[(first + 3) * S],
                 e = R[(first + 4) * S];
    SixVec x;
    x.v[0] = { a.x, a.y, a.z };
    x.v[1] = { a.w, b.x, b.y };
    x.v[2] = { b.z, b.w, c.x };
    x.v[3] = { c.y, c.z, c.w };
    x.v[4] = { d.x, d.y, d.z };
    x.v[5] = { d.w, e.x, e.y };
    return x;
}

// The 16-byte pieces [First, End) of a contact or a point as one copy, as readBody's; the other fields are not set.
template <int First, int End, class T>
__device__ __forceinline__ T readPieces(const T& x) {
    T out;
#if defined(TF_DEVICE_CHECKS)
    memset(&out, 0x3f, sizeof(out));
#endif
    const float4* from = reinterpret_cast<const float4*>(&x);
#pragma unroll
    for (int k = First; k < End; ++k) {
        const float4 piece = from[k];
        memcpy(reinterpret_cast<unsigned char*>(&out) + 16 * k, &piece, 16);
    }
    return out;
}
// A contact's pieces from the bodies to the rolling resistance, and a point's up to the separation.
constexpr int kContactHead = 1, kContactHeadEnd = 6, kPointSolve = 0, kPointSolveEnd = 4;
static_assert(offsetof(DContact, bodyA) >= 16 * kContactHead && offsetof(DContact, rollingResistance) + 4 <= 16 * kContactHeadEnd &&
                  offsetof(DPoint, separation) + 4 <= 16 * kPointSolveEnd, "the pieces hold the fields");

// Builds the record of laned contact ci (world-local) at global slot `slot`, from the contact as prepared and
// its bodies' current world inverse mass and inertia (the axes are makeAxis's). The contact's head, the bodies and each
// point are read whole before the stores, past which the compiler moves no load: prepare of 1024 impact worlds 566 to 511
// us a step, of the box pyramid 168 to 151. (Preparing the contacts before from whole pieces too took 17 us off the
// pyramid's and put 500 on the impact worlds'.)
static __device__ void buildRow(const Batch& B, const WorldInfo& wi, uint32_t slot, uint32_t ci) {
    const DContact& from = B.contacts[wi.contactFirst + ci];
    const DContact c = readPieces<kContactHead, kContactHeadEnd>(from);
    const AxisBody xa = axisBodyOf(readBody<kBodyInvInertia | kBodyInvMass>(B.bodies[c.bodyA]));
    const AxisBody xb = axisBodyOf(readBody<kBodyInvInertia | kBodyInvMass>(B.bodies[c.bodyB]));
    constexpr int S = kRowTile;
    float4* R = rowOf(B, slot);
    const int n = c.count;
    R[kRowHead * S] = make_float4(__uint_as_float(c.bodyA), __uint_as_float(c.bodyB), __uint_as_float((uint32_t)n),
                                  __uint_as_float(ci));
    R[kRowNormal * S] = f4(c.normal, c.friction);
    R[kRowT1 * S] = f4(c.tangent1, 0.0f);
    R[kRowT2 * S] = f4(c.tangent2, 0.0f);
    const Vec3 linear[6] = { xa.invMassWorld * c.normal, xb.invMassWorld * c.normal, xa.invMassWorld * c.tangent1,
                             xb.invMassWorld * c.tangent1, xa.invMassWorld * c.tangent2, xb.invMassWorld * c.tangent2 };
    putSix(R, kRowLinear, linear);
    for (int i = 0; i < n; ++i) {
        const DPoint p = readPieces<kPointSolve, kPointSolveEnd>(from.points[i]);
        const Axis xn = makeAxis(xa, xb, p.anchorA, p.anchorB, c.normal);
        const Axis x1 = makeAxis(xa, xb, p.anchorA, p.anchorB, c.tangent1);
        const Axis x2 = makeAxis(xa, xb, p.anchorA, p.anchorB, c.tangent2);
        const int at = kRowPoint + kRowPointWords * i;
        R[at * S] = f4(p.anchorA, p.adjustedSeparation);
        R[(at + 1) * S] = f4(p.anchorB, xn.mass);
        R[(at + 2) * S] = make_float4(x1.mass, x2.mass, p.normalImpulse, p.maxNormalImpulse);
        R[(at + 3) * S] = f4(p.tangentImpulse, 0.0f);
        const Vec3 angular[6] = { xn.angularA, xn.angularB, x1.angularA, x1.angularB, x2.angularA, x2.angularB };
        putSix(R, at + 4, angular);
    }
}

// What the solve and the refreshes changed in a laned contact's record, back into the contact: the impulses, and the
// lever arms and separations a refresh expressed anew. A point's first 12 words, whole pieces at a time.
__device__ __forceinline__ void returnImpulses(const Batch& B, uint32_t slot, DContact& c) {
    static_assert(offsetof(DPoint, adjustedSeparation) == 24 && offsetof(DPoint, tangentImpulse) == 32 &&
                      offsetof(DPoint, relativeVelocity) == 48, "the order of a point's first words");
    constexpr int S = kRowTile;
    const float4* R = rowOf(B, slot);
    const int n = c.count;
    for (int i = 0; i < n; ++i) {
        const int at = kRowPoint + kRowPointWords * i;
        const float4 a = R[at * S], b = R[(at + 1) * S], m = R[(at + 2) * S], t = R[(at + 3) * S];
        float4* p = reinterpret_cast<float4*>(&c.points[i]);
        p[0] = make_float4(a.x, a.y, a.z, b.x);
        p[1] = make_float4(b.y, b.z, a.w, m.z);
        p[2] = make_float4(t.x, t.y, t.z, m.w);
    }
}

// A laned contact's record at a refresh that does not collide its pair again: rebaseContact and the axes of buildRow,
// from the record itself. Its normal and the bodies' inverse masses are what they were, so the head and the linear
// terms stay; the contact takes the lever arms back with the impulses (returnImpulses). (Through the contact, its
// impulses and its points first and then the whole record built again, the refreshes of 1024 impact worlds, which
// collide few pairs again, took 1255 us a step, nearly all of it waiting for scattered four-byte loads; 418 this way.)
static __device__ void rebaseRow(const Batch& B, uint32_t slot) {
    constexpr int S = kRowTile;
    float4* R = rowOf(B, slot);
    const float4 h = R[kRowHead * S], normal = R[kRowNormal * S], tangent1 = R[kRowT1 * S], tangent2 = R[kRowT2 * S];
    const SixVec lin = getSix<S>(R, kRowLinear);
    const DBody a = readBody<kBodySolve | kBodyInvInertia>(B.bodies[__float_as_uint(h.x)]);
    const DBody b = readBody<kBodySolve | kBodyInvInertia>(B.bodies[__float_as_uint(h.y)]);
    const int n = (int)__float_as_uint(h.z);
    const float shift = dot(b.dp - a.dp, xyz(normal));
    const Vec3 d[3] = { xyz(normal), xyz(tangent1), xyz(tangent2) };
    for (int i = 0; i < n; ++i) {
        const int at = kRowPoint + kRowPointWords * i;
        const float4 pa = R[at * S], pb = R[(at + 1) * S], m = R[(at + 2) * S];
        const Vec3 ra = rotate(a.dq, xyz(pa)), rb = rotate(b.dq, xyz(pb));
        Vec3 angular[6];
        float mass[3];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            // makeAxis's operations, the linear terms taken from the record.
            const Vec3 armA = cross(ra, d[x]), armB = cross(rb, d[x]);
            angular[2 * x] = a.invInertiaWorld * armA;
            angular[2 * x + 1] = b.invInertiaWorld * armB;
            const float k = dot(d[x], lin.v[2 * x]) + dot(d[x], lin.v[2 * x + 1]) + dot(armA, angular[2 * x]) + dot(armB, angular[2 * x + 1]);
            mass[x] = k > 1e-6f * (a.invMass + b.invMass) ? 1.0f / k : 0.0f;
        }
        R[at * S] = f4(ra, pa.w + shift);
        R[(at + 1) * S] = f4(rb, mass[0]);
        R[(at + 2) * S] = make_float4(mass[1], mass[2], m.z, m.w);
        putSix(R, at + 4, angular);
    }
}

constexpr uint32_t kOrderRounds = 64;       // rounds of visitInBodyOrder at most before one thread takes the rest
constexpr uint32_t kOrderRoundsMin = 64;    // shorter lists go to one thread at once
constexpr uint8_t kColorPending = 0xff;

// Visits the n entries of a contact list so that, at every moving body, its contacts are visited in list
// order: in each round every pending entry that is the first pending one at each of its bodies is visited
// (round r marks a body with (tag of r, its first pending entry) by atomicMin, tags falling from round to
// round so a round's marks replace the last one's). Entries visited in one round share no body, so visit(x)
// may read and write its own bodies' state without atomics. A result that depends, per body, only on the
// entries before x at that body (a greedy color, a level) therefore comes out as a pass in list order gives
// it. Once a round visits too few entries to pay for its two passes over the list (a long chain of contacts
// through a stack), or after kOrderRounds rounds, one thread visits what is left in list order, which keeps
// that property: the entries visited so far include every entry before them at a shared body. ends(x, a, b)
// gives an entry's bodies (kNone for one that does not count); firstAt holds a word per body, set to kNone
// beforehand.
template <class G, class Ends, class Pending, class Visit>
static __device__ void visitInBodyOrder(const G& g, uint32_t n, uint32_t* firstAt, Ends ends, Pending pending,
                                        Visit visit) {
    __shared__ uint32_t s_visits[kMaxGroups][2], s_left[3];
    if (n >= kOrderRoundsMin && n < (1u << 24)) {
        // A round costs two passes of n / size entries per thread; one thread takes an entry in about as long.
        const uint32_t worth = (n + g.size - 1) / g.size + 4;
        uint32_t* visits = g.shared(s_visits[g.id]);
        uint32_t* leftFlag = g.shared(s_left);
        if (g.tid == 0) { visits[0] = 0; }
        if constexpr (G::kCluster) {
            if (g.tid == 0) { leftFlag[0] = 0; }
            g.sync();
        }
        for (uint32_t r = 0; r < kOrderRounds; ++r) {
            const uint32_t tag = (kOrderRounds - 1 - r) << 24;
            bool left = false;
            for (uint32_t x = g.tid; x < n; x += g.size) {
                if (!pending(x)) { continue; }
                left = true;
                uint32_t a, b;
                ends(x, a, b);
                if (a != kNone) { atomicMin(&firstAt[a], tag | x); }
                if (b != kNone) { atomicMin(&firstAt[b], tag | x); }
            }
            if (!g.any(left, leftFlag + r % 3)) { return; }
            if (g.tid == 0) {
                visits[(r + 1) & 1] = 0;
                if constexpr (G::kCluster) { leftFlag[(r + 1) % 3] = 0; }
            }
            uint32_t visited = 0;
            for (uint32_t x = g.tid; x < n; x += g.size) {
                if (!pending(x)) { continue; }
                uint32_t a, b;
                ends(x, a, b);
                if ((a == kNone || firstAt[a] == (tag | x)) && (b == kNone || firstAt[b] == (tag | x))) {
                    visit(x);
                    ++visited;
                }
            }
            if (visited) { atomicAdd(&visits[r & 1], visited); }
            g.sync();
            if (*(volatile uint32_t*)&visits[r & 1] < worth) { break; }
        }
    }
    if (g.tid == 0) {
        for (uint32_t x = 0; x < n; ++x) {
            if (pending(x)) { visit(x); }
        }
    }
    g.sync();
}

// Greedy lowest free color of 32 over the moving bodies, in list order (src/lanes.cpp:356-374). endA/endB
// hold each contact's moving bodies (kNone for one that does not move); endA carries kNotColorable for a
// planar or rolling contact, which takes no color. masks (a word per body) start at 0, firstAt at kNone.
template <class G>
static __device__ void colorInOrder(const G& g, uint32_t n, const uint32_t* endA, const uint32_t* endB,
                                    uint32_t* masks, uint32_t* firstAt, uint8_t* color) {
    for (uint32_t x = g.tid; x < n; x += g.size) { color[x] = (endA[x] & kNotColorable) ? kNoColor : kColorPending; }
    g.sync();
    visitInBodyOrder(
        g, n, firstAt, [&](uint32_t x, uint32_t& a, uint32_t& b) { a = endA[x], b = endB[x]; },
        [&](uint32_t x) { return color[x] == kColorPending; },
        [&](uint32_t x) {
            const uint32_t a = endA[x], b = endB[x];
            const uint32_t taken = (a != kNone ? masks[a] : 0u) | (b != kNone ? masks[b] : 0u);
            uint8_t k = kNoColor;
            if (taken != 0xffffffffu) {
                const int f = __ffs(~taken) - 1;
                if (a != kNone) { masks[a] |= 1u << f; }
                if (b != kNone) { masks[b] |= 1u << f; }
                k = (uint8_t)f;
            }
            color[x] = k;
        });
}

// Groups a contact list by color: every color's contacts (any order within a color, which solves the same)
// into colored, colors in ascending order, the uncolored ones into rest in list order.
template <class G>
static __device__ void bucketByColor(const G& g, uint32_t n, const uint32_t* list, const uint8_t* colorOf, uint32_t* colored,
                              uint32_t* rest, uint32_t* startOut, uint32_t& colorsUsed, uint32_t& restCount) {
    __shared__ uint32_t s_size[kMaxGroups][kColors + 1];
    __shared__ uint32_t s_fill[kMaxGroups][kColors + 1];
    uint32_t* size = g.shared(s_size[g.id]);
    uint32_t* fill = g.shared(s_fill[g.id]);
    for (uint32_t k = g.tid; k <= kColors; k += g.size) { size[k] = 0; }
    g.sync();
    for (uint32_t x = g.tid; x < n; x += g.size) { takePlace(size, colorOf[list[x]]); }
    g.sync();
    if (g.tid == 0) {
        uint32_t sum = 0, used = 0;
        for (int k = 0; k <= kColors; ++k) {
            startOut[k] = sum;
            fill[k] = sum;
            sum += size[k];
            if (k < kColors && size[k] > 0) { used = (uint32_t)k + 1; }
        }
        colorsUsed = used;
    }
    g.sync();
    for (uint32_t x = g.tid; x < n; x += g.size) {
        const uint8_t k = colorOf[list[x]];
        if (k != kNoColor) {
            const uint32_t at = takePlace(fill, k);
#if defined(TF_DEVICE_CHECKS)
            if (at >= n) { continue; }
#endif
            colored[at] = list[x];
        }
    }
    const uint32_t r = groupCompact(g, n, [&](uint32_t x) { return colorOf[list[x]] == kNoColor; },
                                    [&](uint32_t x, uint32_t pos) { rest[pos] = list[x]; });
    if (g.tid == 0) { restCount = r; }
    g.sync();
}

// The contacts solved one at a time (planar, rolling, those past the colors) are swept in list order. Only
// contacts that share a moving body depend on that order: each takes a level one past the last earlier
// contact on either of its moving bodies, so that the contacts of a level share no moving body and run
// together while every body still meets its contacts in list order, which gives the sweep's own bits. The
// levels come from visitInBodyOrder; one warp then reorders list by level (stably, within the level in list
// order) and writes each level's end. last and firstAt (one word per body, zero and kNone on entry), tmp and
// out (one word per entry) are scratch. Returns the levels.
template <class G>
static __device__ uint32_t levelList(const G& g, const Batch& B, const WorldInfo& wi, const DContact* cs,
                                     uint32_t* list, uint32_t n, uint32_t* levelEnd, uint32_t* last,
                                     uint32_t* firstAt, uint32_t* tmp, uint32_t* out) {
    __shared__ uint32_t s_levels[kMaxGroups];
    // Each entry's moving bodies (tmp, out) and its level (levelEnd, kNone until set).
    for (uint32_t x = g.tid; x < n; x += g.size) {
        const DContact& c = cs[list[x]];
        const uint32_t a = c.bodyA - wi.bodyFirst, b = c.bodyB - wi.bodyFirst;
        tmp[x] = a < wi.bodyCount && movingBody(B.bodies[c.bodyA]) ? a : kNone;
        out[x] = b < wi.bodyCount && movingBody(B.bodies[c.bodyB]) ? b : kNone;
        levelEnd[x] = kNone;
    }
    uint32_t* deepest = g.shared(&s_levels[g.id]);
    if (g.tid == 0) { *deepest = 0; }
    g.sync();
    visitInBodyOrder(
        g, n, firstAt, [&](uint32_t x, uint32_t& a, uint32_t& b) { a = tmp[x], b = out[x]; },
        [&](uint32_t x) { return levelEnd[x] == kNone; },
        [&](uint32_t x) {
            const uint32_t a = tmp[x], b = out[x];
            uint32_t lev = 0;
            if (a != kNone) { lev = max(lev, last[a]); }
            if (b != kNone) { lev = max(lev, last[b]); }
            if (a != kNone) { last[a] = lev + 1; }
            if (b != kNone) { last[b] = lev + 1; }
            levelEnd[x] = lev;
            atomicMax(deepest, lev + 1);
        });
    for (uint32_t x = g.tid; x < n; x += g.size) { tmp[x] = levelEnd[x]; }
    g.sync();
    const uint32_t levels = *(volatile uint32_t*)deepest;
    for (uint32_t l = g.tid; l < levels; l += g.size) { levelEnd[l] = 0; }
    g.sync();
    for (uint32_t x = g.tid; x < n; x += g.size) { atomicAdd(&levelEnd[tmp[x]], 1u); }
    g.sync();
    groupScanWords(g, levelEnd, levels);
    // One warp fills the levels, 32 entries of the list at a time: an entry's place is its level's fill position
    // plus the entries of that level before it among the 32. A level's fill position is its end once filled.
    if (g.warp == 0) {
        for (uint32_t first = 0; first < n; first += 32) {
            const uint32_t x = first + g.lane;
            const uint32_t lev = x < n ? tmp[x] : kNone;
            const uint32_t same = __match_any_sync(0xffffffffu, lev);
            if (x < n) { out[levelEnd[lev] + __popc(same & ((1u << g.lane) - 1u))] = list[x]; }
            __syncwarp();
            if (x < n && (same >> g.lane) == 1u) { levelEnd[lev] += __popc(same); }
            __syncwarp();
        }
    }
    g.sync();
    for (uint32_t x = g.tid; x < n; x += g.size) { list[x] = out[x]; }
    g.sync();
    return levels;
}

// Runs f on every entry of a leveled list, a level at a time.
template <class G, class F>
__device__ void forEachLevel(const G& g, const uint32_t* list, const uint32_t* levelEnd, uint32_t levels, F f) {
    uint32_t begin = 0;
    for (uint32_t l = 0; l < levels; ++l) {
        const uint32_t end = levelEnd[l];
        for (uint32_t x = begin + g.tid; x < end; x += g.size) { f(list[x]); }
        g.sync();
        begin = end;
    }
}

// Whether a world's contacts are better solved with rooms (kRoomWarps), as far as the world itself goes: it has five
// contact points a body (a room holds four points of a contact whether it has them or not), no more contacts a color
// than its group has lanes (a second round waits for its records), and no more bodies than roomBodies (past it a CTA
// without rooms shares its SM with others). Measured, us of substeps a step with rooms and without. One world: 208 boxes
// in a pyramid (11.2 points a body, 98 contacts a color) 324 and 387, 497 (11.5 and 238) 480 and 497, 562 (270) 597 and
// 467, 991 (480) 1150 and 601; 512 boxes in a block (27 and 197) 1534 and 1676; balls on a box, 400 (2.7 and 215) 303 and
// 214, in a block, 216 (2.7) 207 and 185, packed tight, 343 (4.8) 422 and 390. 100 worlds of bullets and boxes (14 points
// a body, later 5) 1407 and 1664. 1200 worlds: 79 boxes 1189 and 1473, 137 boxes 2459 and 1881, 216 in a block 10568 and
// 7654.
__device__ __forceinline__ bool roomsSuit(const Batch& B, const WorldInfo& wi, uint32_t points, uint32_t colored,
                                          uint32_t colors) {
    return points >= 5 * wi.bodyCount && wi.bodyCount <= B.roomBodies &&
           (wi.bodyCount <= B.roomWarpBodies || colored <= (uint64_t)colors * B.roomThreads);
}

// Whether the contacts of the worlds that rooms suit outweigh the batch's bodies: the batch is solved with rooms then.
// By how much they have to (roomContacts) depends on the launch. The lines measured lie at 7.4 contacts a body (impact
// walls) and 2.8 (the pyramid) on one side, 0.5 and less on the other (the uneven batch's worlds: 3312 us with rooms and
// 1952 without).
__device__ __forceinline__ bool contactsOutweigh(const Batch& B) {
    return *(volatile uint32_t*)(B.work + kSlotRoomContacts) >= (uint64_t)B.roomContacts * B.totalBodies;
}

// Coloring is staged in the group's shared slice (masks by body, endpoints by active contact) when the world
// fits stageBodies bodies and stageContacts active contacts, else in the world's global scratch.
template <bool Cluster>
__global__ void __launch_bounds__(kMaxBlock) k_prepare(const __grid_constant__ Batch B, const __grid_constant__ StepParams P, const __grid_constant__ Split sp, int serial) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint32_t s_fast[kMaxGroups], s_fastSolid[kMaxGroups], s_points[kMaxGroups];
    __shared__ uint32_t s_class[kMaxGroups][kPairClasses + 1], s_classBase[kMaxGroups][kPairClasses + 1];
    if (stepAborted<Cluster>(B, serial)) { return; }
    forSomeWorlds<Cluster>(B, kSlotPrepare, sp, s_raw, [&](const auto& g, uint32_t w, unsigned char* slice, const StageSizes& ss) {
        const uint32_t stageBodies = ss.bodies, stageContacts = ss.contacts;
        const WorldInfo wi = B.info[w];
        WorldCounts& wc = B.counts[w];
        uint32_t nc = wc.nextContactCount;
        if (!TF_OK_INDEX(B, nc <= wi.contactCap, 6, w, nc)) { nc = 0; }
        uint32_t* fast = g.shared(&s_fast[g.id]);
        uint32_t* fastSolid = g.shared(&s_fastSolid[g.id]);
        uint32_t* pointSum = g.shared(&s_points[g.id]);
        if (g.tid == 0) {
            wc.contactCount = nc;
            *fast = 0;
            *fastSolid = 0;
            *pointSum = 0;
        }
        for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
            const uint32_t gb = wi.bodyFirst + i;
            DBody b = readBody<kBodySolve | kBodyMassReads | kBodyCom>(B.bodies[gb]);
            B.struck[gb] = 0;
            if (!b.alive) { continue; }
            b.q0 = b.xf.q;
            b.qBase = b.xf.q;
            b.com0 = b.com;
            b.expectedTravel = (length(b.v) + length(b.w) * b.extent) * P.dt;
            b.dp = zero3();
            b.dq = qid();
            updateInverseMass(b);
            writeBody<kBodySolve | kBodyMassWrites | kBodyBase | kBodyStart>(B.bodies[gb], b);
        }
        g.sync();
        // Joints: what the step will report for them starts over (src/world.cpp:1647).
        for (uint32_t x = g.tid; x < wi.jointCount; x += g.size) {
            DJoint& j = B.joints[wi.jointFirst + x];
            j.brokeNow = 0;
            const JBody a = j.bodyA == kWorldEnd ? worldEnd() : jointBodyOf(B.bodies[j.bodyA]);
            const JBody b = jointBodyOf(B.bodies[j.bodyB]);
            if (jointActive(j, a, b)) {
                j.force = zero3();
                j.torque = zero3();
            }
        }
        const uint32_t cf = wi.contactFirst;
        DContact* cs = B.contacts + cf;
        const uint32_t nActive = groupCompact(
            g, nc,
            [&](uint32_t i) {
                if (!TF_OK_INDEX(B, cs[i].bodyA - wi.bodyFirst < wi.bodyCount && cs[i].bodyB - wi.bodyFirst < wi.bodyCount &&
                                    cs[i].count >= 0 && cs[i].count <= 4, 5, wi.bodyFirst, i)) {
                    B.cflags[cf + i] = 0;
                    return false;
                }
                const DBody a = readBody<kBodySolve | kBodyPose | kBodyInertia>(B.bodies[cs[i].bodyA]);
                const DBody b = readBody<kBodySolve | kBodyPose | kBodyInertia>(B.bodies[cs[i].bodyB]);
                const bool on = (a.type == kDynamic && a.awake) || (b.type == kDynamic && b.awake);
                uint8_t f = 0;
                if (on && relativeTravel(a, b, P.dt) > P.tol.speculative) {
                    f |= kFlagFast;
                    atomicAdd(fast, 1u);
                    if (!isPlanar(a) && !isPlanar(b)) {
                        f |= kFlagFastSolid;
                        atomicAdd(fastSolid, 1u);
                    }
                }
                B.cflags[cf + i] = f | (on ? kFlagActive : 0);
                return on;
            },
            [&](uint32_t i, uint32_t pos) { B.active[cf + pos] = i; });
        const uint32_t* act = B.active + cf;
        const bool staged = wi.bodyCount <= stageBodies && nActive <= stageContacts;
        uint32_t* masks = staged ? reinterpret_cast<uint32_t*>(slice) : B.bodyColors + wi.bodyFirst;
        uint32_t* endA = staged ? masks + stageBodies : B.mergeIdxA + cf;
        uint32_t* endB = staged ? endA + stageContacts : B.mergeIdxB + cf;
        // Each body's first pending contact while coloring and leveling (the island scratch is free here).
        uint32_t* firstAt = staged ? endB + stageContacts : B.unionParent + wi.bodyFirst;
        // Colors by active position; moved to contact order below. The merge scratch is free by now.
        uint8_t* colorTmp = reinterpret_cast<uint8_t*>(B.mergePartA + cf);
        for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
            masks[i] = 0;
            firstAt[i] = kNone;
        }
        uint32_t points = 0;
        for (uint32_t x = g.tid; x < nActive; x += g.size) {
            if (!TF_OK_INDEX(B, act[x] < nc, 7, w, x)) { continue; }
            DContact& c = cs[act[x]];
            const DBody& a = B.bodies[c.bodyA];
            const DBody& b = B.bodies[c.bodyB];
            prepareContact(a, b, c);
            c.flags &= ~kCLaned;
            points += (uint32_t)c.count;
            const bool can = !(c.flags & kCPlanar) && !(c.rollingResistance > 0.0f);
            endA[x] = (movingBody(a) ? c.bodyA - wi.bodyFirst : kNone) | (can ? 0u : kNotColorable);
            endB[x] = movingBody(b) ? c.bodyB - wi.bodyFirst : kNone;
            // Bodies of pairs closing faster than the restitution threshold are struck (src/world.cpp:1029-1049).
            for (int i = 0; i < c.count; ++i) {
                if (c.points[i].relativeVelocity >= -P.restitutionThreshold) { continue; }
                if (a.type == kDynamic) { B.struck[c.bodyA] = 1; }
                if (b.type == kDynamic) { B.struck[c.bodyB] = 1; }
                break;
            }
        }
        points = __reduce_add_sync(0xffffffffu, points);
        if (g.lane == 0) { atomicAdd(pointSum, points); }
        g.sync();
        colorInOrder(g, nActive, endA, endB, masks, firstAt, colorTmp);
        uint8_t* colorOf = B.color + cf;
        for (uint32_t x = g.tid; x < nActive; x += g.size) {
            const uint8_t k = colorTmp[x];
            colorOf[act[x]] = k;
            if (k != kNoColor) { cs[act[x]].flags |= kCLaned; }
        }
        g.sync();
        const uint32_t nImpact = groupCompact(
            g, nActive,
            [&](uint32_t x) {
                const DContact& c = cs[act[x]];
                const uint32_t ia = c.bodyA, ib = c.bodyB;
                return (B.struck[ia] | B.struck[ib]) != 0;
            },
            [&](uint32_t x, uint32_t pos) { B.impact[cf + pos] = act[x]; });
        bucketByColor(g, nActive, act, colorOf, B.colored + cf, B.rest + cf, wc.colorStart, wc.colorCount, wc.restCount);
        bucketByColor(g, nImpact, B.impact + cf, colorOf, B.impactColored + cf, B.impactRest + cf, wc.impactColorStart,
                      wc.impactColorCount, wc.impactRestCount);
        // The laned contacts' records, in color order; the axes of the contacts solved one at a time.
        const uint32_t nColored = wc.colorStart[kColors];
        for (uint32_t x = g.tid; x < nColored; x += g.size) {
            const uint32_t ci = B.colored[cf + x];
            if (!TF_OK_INDEX(B, ci < nc, 7, w, x)) { continue; }
            B.slotOf[cf + ci] = cf + x;
            buildRow(B, wi, cf + x, ci);
        }
        for (uint32_t x = g.tid; x < wc.restCount; x += g.size) {
            const uint32_t ci = B.rest[cf + x];
            if (!TF_OK_INDEX(B, ci < nc, 7, w, x)) { continue; }
            B.slotOf[cf + ci] = kNoSlot;
            const DContact& c = cs[ci];
            makeContactAxes(axisBodyOf(B.bodies[c.bodyA]), axisBodyOf(B.bodies[c.bodyB]), c,
                            B.axes + (size_t)(cf + ci) * kAxesPerContact);
        }
        // A world with fast contacts is refreshed between substeps: its fast contacts join the flat list of
        // their pair class, its other active contacts the light list, in the order of their records.
        if (*(volatile uint32_t*)fast > 0) {
            uint32_t* cls = g.shared(s_class[g.id]);
            uint32_t* classBase = g.shared(s_classBase[g.id]);
            if (g.tid <= kPairClasses) { cls[g.tid] = 0; }
            g.sync();
            const uint32_t nListed = nColored + wc.restCount;
            auto contactAt = [&](uint32_t x) { return x < nColored ? B.colored[cf + x] : B.rest[cf + x - nColored]; };
            auto listOf = [&](uint32_t ci) {
                if (!(B.cflags[cf + ci] & kFlagFast)) { return kPairClasses; }
                return pairClassOf(B, cs[ci].shapeA, cs[ci].shapeB);
            };
            for (uint32_t x = g.tid; x < nListed; x += g.size) { takePlace(cls, (uint32_t)listOf(contactAt(x))); }
            g.sync();
            if (g.tid <= kPairClasses) {
                classBase[g.tid] = atomicAdd(B.work + kSlotFastItems + g.tid, cls[g.tid]);
                cls[g.tid] = 0;
            }
            g.sync();
            for (uint32_t x = g.tid; x < nListed; x += g.size) {
                const uint32_t ci = contactAt(x);
                const int l = listOf(ci);
                const uint32_t pos = classBase[l] + takePlace(cls, (uint32_t)l);
                B.contactItems[(size_t)l * B.contactItemStride + pos] = make_uint2(w, ci);
            }
            g.sync();
        }
        // The one-at-a-time lists by level; the coloring's scratch is free by now.
        for (int which = 0; which < 2; ++which) {
            const uint32_t n = which == 0 ? wc.restCount : wc.impactRestCount;
            if (n == 0) {
                if (g.tid == 0) { (which == 0 ? wc.restLevels : wc.impactRestLevels) = 0; }
                continue;
            }
            for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
                masks[i] = 0;
                firstAt[i] = kNone;
            }
            g.sync();
            uint32_t* list = (which == 0 ? B.rest : B.impactRest) + cf;
            uint32_t* ends = (which == 0 ? B.restLevel : B.impactRestLevel) + cf;
            const uint32_t levels = levelList(g, B, wi, cs, list, n, ends, masks, firstAt, endA, endB);
            if (g.tid == 0) { (which == 0 ? wc.restLevels : wc.impactRestLevels) = levels; }
            g.sync();
        }
        if (g.tid == 0) {
            if (roomsSuit(B, wi, *pointSum, nColored, wc.colorCount)) { atomicAdd(B.work + kSlotRoomContacts, nActive); }
            if (*fast > 0) { atomicOr(B.work + kSlotFast, *fastSolid > 0 ? 3u : 1u); }
            wc.activeCount = nActive;
            wc.impactCount = nImpact;
            wc.fastCount = *fast;
            wc.fastSolidCount = *fastSolid;
            wc.activePoints = *pointSum;
        }
        g.sync();
    });
}
// ---------------------------------------------------------------------------------------------------------
// The substep (src/world.cpp:1658-1681).

// Calls f(contact index) for every contact of each color in turn, the colors apart by a group barrier.
template <class G, class F>
__device__ void forEachColor(const G& g, const uint32_t* list, const uint32_t* start, uint32_t colors, F f) {
    for (uint32_t k = 0; k < colors; ++k) {
        const uint32_t end = start[k + 1];
        for (uint32_t x = start[k] + g.tid; x < end; x += g.size) { f(list[x]); }
        g.sync();
    }
}

// In checked builds, whether contact ci of a world can be read: in the list, with bodies in the world.
__device__ __forceinline__ bool contactOk(const Batch& B, const WorldInfo& wi, const WorldCounts& wc,
                                          uint32_t ci, int code) {
#if defined(TF_DEVICE_CHECKS)
    if (!TF_OK_INDEX(B, ci < wc.contactCount, code, wi.bodyFirst, ci)) { return false; }
    const DContact& c = B.contacts[wi.contactFirst + ci];
    return TF_OK_INDEX(B, c.bodyA - wi.bodyFirst < wi.bodyCount && c.bodyB - wi.bodyFirst < wi.bodyCount &&
                              c.shapeA - wi.shapeFirst < wi.shapeCount && c.shapeB - wi.shapeFirst < wi.shapeCount &&
                              c.count >= 0 && c.count <= 4,
                       code + 1, wi.bodyFirst, ci);
#else
    return true;
#endif
}

// A contact takes a manifold of its pair collided again mid-step: new points on body A, the approach speed
// and largest impulse of the nearest old point, and the old impulses carried (src/world.cpp:1106-1137).
static __device__ void takeRefreshed(const Batch& B, const StepParams& P, const DBody& a, const DBody& b, DContact& c,
                              const Manifold& m) {
    const DContact old = c;
    c.flags &= ~kCReusable;
    c.featKind = m.featKind;
    c.featA = m.featA;
    c.featB = m.featB;
    c.normal = m.normal;
    c.tangent1 = perpendicular(m.normal);
    c.tangent2 = cross(m.normal, c.tangent1);
    c.count = m.count;
    for (int i = 0; i < m.count; ++i) {
        DPoint& p = c.points[i];
        p = DPoint{};
        p.localA = applyInverse(a.xf, m.points[i].position);
        p.separation = m.points[i].separation;
        const Vec3 up = lift(a, b, m.normal, p.separation, P.tol.speculative);
        p.anchorA = m.points[i].position - up - a.com;
        p.anchorB = m.points[i].position + up - b.com;
    }
    prepareContact(a, b, c);
    for (int i = 0; i < c.count; ++i) {
        DPoint& p = c.points[i];
        const int k = nearestPoint(old, p.localA);
        if (k < 0) { continue; }
        p.relativeVelocity = old.points[k].relativeVelocity;
        p.maxNormalImpulse = old.points[k].maxNormalImpulse;
    }
    carryImpulses(old, c, P.tol.speculative * P.tol.speculative);
}

// A fast pair collided again with the remaining time (src/world.cpp:1074-1138).
template <int Cls = kClassAny>
__device__ void refreshContact(const Batch& B, const StepParams& P, DContact& c, float remaining) {
    const DBody& a = B.bodies[c.bodyA];
    const DBody& b = B.bodies[c.bodyB];
    const DShape sa = B.shapes[c.shapeA];
    const DShape sb = B.shapes[c.shapeB];
    // Polyhedra that turned little against each other keep the edge pair they met on (src/world.cpp:1051-1055).
    const Quat now = conjugate(a.xf.q) * b.xf.q, then = conjugate(a.q0) * b.q0;
    const bool little = fabsf(dot(now, then)) >= P.featureTurnCos;
    Manifold m;
    collidePair<Cls>(B, P, sa, sb, remaining, m, little ? c.featKind : kFeatNone, c.featA, c.featB);
    if (m.count == 0) {
        c.count = 0;
        return;
    }
    takeRefreshed(B, P, a, b, c, m);
}

// How far any point of the body moved since the step started (src/world.cpp:484-488).
__device__ __forceinline__ float movedThisStep(const DBody& b) {
    const Quat turn = conjugate(b.q0) * b.xf.q;
    const float s = minf(sqrtf(turn.x * turn.x + turn.y * turn.y + turn.z * turn.z), 1.0f);
    return length(b.com - b.com0) + 2.0f * asinRounded(s) * b.extent;
}

// The contacts of a fast mesh pair, one key run, collided again with the remaining time: the pair is
// collided once, skipping the triangles its collision at the step's start ruled out while they stay out of
// reach, and each contact in turn takes the new manifold whose normal is closest to its own; a contact left
// without one keeps no points (src/world.cpp:1078-1137).
// Warp: every lane of the warp calls it alike with the warp's room; the lanes collide the triangles together and
// lane 0 hands the manifolds to the contacts.
template <bool Warp>
static __device__ void refreshMeshRun(const Batch& B, const StepParams& P, const WorldInfo& wi, WorldCounts& wc, DContact* run,
                               int count, float remaining, MeshWarpRoom* room = nullptr, uint32_t lane = 0) {
    const DBody& a = B.bodies[run[0].bodyA];
    const DBody& b = B.bodies[run[0].bodyB];
    const DShape sa = B.shapes[run[0].shapeA];
    const DShape sb = B.shapes[run[0].shapeB];
    MeshBounds mb{ nullptr, 0, nullptr, 0, 0.0f };
    if (run[0].boundsCount > 0 && TF_OK_INDEX(B, run[0].boundsFirst + run[0].boundsCount <= wi.boundsCap, 36, wi.bodyFirst, 0)) {
        mb.known = B.triBounds + wi.boundsFirst + run[0].boundsFirst;
        mb.knownCount = (int)run[0].boundsCount;
        mb.moved = movedThisStep(a) + movedThisStep(b);
    }
    Manifold found[kMaxMeshParts];
    int n = 0;
    const int status = collideMeshPair<Warp>(B, P, sa, sb, remaining, found, n, &mb, Warp ? room->found : nullptr, lane);
    if (Warp && lane != 0) { return; }
    if (status != kMeshOk) {
        atomicOr(&wc.flags, kDevUnsupported);
        n = 0;
    }
    bool taken[kMaxMeshParts];
    for (int k = 0; k < n; ++k) { taken[k] = false; }
    for (int x = 0; x < count; ++x) {
        DContact& c = run[x];
        int pick = -1;
        for (int k = 0; k < n; ++k) {
            if (taken[k]) { continue; }
            if (pick < 0 || dot(found[k].normal, c.normal) > dot(found[pick].normal, c.normal)) { pick = k; }
        }
        if (pick < 0) {
            c.count = 0;
            continue;
        }
        taken[pick] = true;
        takeRefreshed(B, P, a, b, c, found[pick]);
    }
}

// The solver state of one body as a contact solved on its own (planar, rolling or past the last color) reads
// and writes it. Field names match DBody so the same solver templates run on either.
struct SBody {
    Vec3 v, w, dp;
    Quat dq;
    Mat3 invInertiaWorld;
    float planeInvMass, planeInvInertia;
    uint32_t type, awake;
};

// Staged words per body: v 0-2, w 3-5, dp 6-8, dq 9-12, type | awake << 8 in 13: what a laned solve reads
// and writes. The inverse world inertia (torques, contacts solved on their own) stays in global memory, so
// more bodies fit a slice.
constexpr int kSBodyWords = 14;

// Where one world's solver state lives during a substep: shared memory (structure of arrays, stride words
// apart) for worlds that fit, else the bodies in global memory.
struct SolverStore {
    float* s;
    uint32_t stride;
    bool staged;
    DBody* g;

    __device__ __forceinline__ float& at(int word, uint32_t i) const { return s[word * stride + i]; }

    __device__ LanedBody loadLaned(uint32_t i) const {
        LanedBody b;
        if (!staged) {
            const DBody& d = g[i];
            b.v = d.v;
            b.w = d.w;
            b.dp = d.dp;
            b.dq = d.dq;
            b.type = d.type;
            b.awake = d.awake;
            return b;
        }
        b.v = { at(0, i), at(1, i), at(2, i) };
        b.w = { at(3, i), at(4, i), at(5, i) };
        b.dp = { at(6, i), at(7, i), at(8, i) };
        b.dq = { at(9, i), at(10, i), at(11, i), at(12, i) };
        const uint32_t f = __float_as_uint(at(13, i));
        b.type = f & 0xffu;
        b.awake = f >> 8;
        return b;
    }

    __device__ SBody load(uint32_t i) const {
        SBody b;
        if (!staged) {
            const DBody& d = g[i];
            b.v = d.v;
            b.w = d.w;
            b.dp = d.dp;
            b.dq = d.dq;
            b.invInertiaWorld = d.invInertiaWorld;
            b.planeInvMass = d.planeInvMass;
            b.planeInvInertia = d.planeInvInertia;
            b.type = d.type;
            b.awake = d.awake;
            return b;
        }
        const LanedBody l = loadLaned(i);
        b.v = l.v;
        b.w = l.w;
        b.dp = l.dp;
        b.dq = l.dq;
        b.type = l.type;
        b.awake = l.awake;
        b.invInertiaWorld = g[i].invInertiaWorld;
        b.planeInvMass = g[i].planeInvMass;
        b.planeInvInertia = g[i].planeInvInertia;
        return b;
    }

    template <class BodyT>
    __device__ void storeVW(uint32_t i, const BodyT& b) const {
        if (!staged) {
            g[i].v = b.v;
            g[i].w = b.w;
            return;
        }
        at(0, i) = b.v.x;
        at(1, i) = b.v.y;
        at(2, i) = b.v.z;
        at(3, i) = b.w.x;
        at(4, i) = b.w.y;
        at(5, i) = b.w.z;
    }

    // Copies a body's solver fields from global memory into the store.
    __device__ void stage(uint32_t i) const {
        const DBody d = readBody<kBodySolve>(g[i]);
        at(0, i) = d.v.x, at(1, i) = d.v.y, at(2, i) = d.v.z;
        at(3, i) = d.w.x, at(4, i) = d.w.y, at(5, i) = d.w.z;
        at(6, i) = d.dp.x, at(7, i) = d.dp.y, at(8, i) = d.dp.z;
        at(9, i) = d.dq.x, at(10, i) = d.dq.y, at(11, i) = d.dq.z, at(12, i) = d.dq.w;
        at(13, i) = __uint_as_float(d.type | (d.awake << 8));
    }

    // Writes the fields a substep changes back to global memory.
    __device__ void unstage(uint32_t i) const {
        DBody& d = g[i];
        const LanedBody l = loadLaned(i);
        DBody b;
        b.v = l.v;
        b.w = l.w;
        b.dp = l.dp;
        b.dq = l.dq;
        writeBody<(kBodySolve & ~kBodyState)>(d, b);
        d.dq.w = l.dq.w;
    }

    __device__ void integrateVelocityAt(uint32_t i, const StepParams& P) const {
        DBody& d = g[i];
        DBody b = readBody<kBodySolve | kBodyInvInertia | kBodyForce | kBodyProj>(d);
        if (!b.alive || b.type != kDynamic || !b.awake) { return; }
        if (staged) {
            b.v = { at(0, i), at(1, i), at(2, i) };
            b.w = { at(3, i), at(4, i), at(5, i) };
        }
        const float kept = b.kept;
        integrateVelocity(b, P);
        storeVW(i, b);
        if (b.kept != kept) { d.kept = b.kept; }
    }

    __device__ void integratePositionAt(uint32_t i, const StepParams& P) const {
        DBody& d = g[i];
        DBody b = readBody<kBodySolve | kBodyForce | kBodyPose | kBodyCom | kBodyLocal | kBodyBase>(d);
        if (staged) {
            b.v = { at(0, i), at(1, i), at(2, i) };
            b.w = { at(3, i), at(4, i), at(5, i) };
            b.dp = { at(6, i), at(7, i), at(8, i) };
            b.dq = { at(9, i), at(10, i), at(11, i), at(12, i) };
        }
        if (!b.alive || b.type == kStatic || (b.type == kDynamic && !b.awake)) { return; }
        const float kept = b.kept;
        integratePosition(b, P);
        if (staged) {
            storeVW(i, b);
            at(6, i) = b.dp.x, at(7, i) = b.dp.y, at(8, i) = b.dp.z;
            at(9, i) = b.dq.x, at(10, i) = b.dq.y, at(11, i) = b.dq.z, at(12, i) = b.dq.w;
        } else {
            writeBody<kBodySolve>(d, b);
        }
        writeBody<kBodyPose | kBodyCom>(d, b);
        if (b.kept != kept) { d.kept = b.kept; }
    }
};

// One direction's axis at a point of a laned contact from its record: the lever arms formed as makeAxis forms
// them, the velocity changes and the effective mass as stored.
__device__ __forceinline__ Axis rowAxis(const Vec3& ra, const Vec3& rb, const Vec3& d, const Vec3& linA, const Vec3& angA,
                                        const Vec3& linB, const Vec3& angB, float mass) {
    Axis x;
    x.armA = cross(ra, d);
    x.armB = cross(rb, d);
    x.linearA = linA;
    x.angularA = angA;
    x.linearB = linB;
    x.angularB = angB;
    x.mass = mass;
    return x;
}

// A warp's room in shared memory for the records of the contacts it is about to solve, a lane's own record words a
// lane apart (word k of lane l at [k * 32 + l]). The copies are asynchronous and each lane waits for its own, so a
// color's records arrive while the group is still at the color before it. They leave an SM eight warps, so they pay
// where the contacts outweigh the bodies by far and each color's records fit the group's rooms at once.
constexpr uint32_t kRoomWarps = 8;  // warps of a CTA with rooms
constexpr uint32_t kRoomBytes = kRowWords * 32 * (uint32_t)sizeof(float4);

__device__ __forceinline__ void roomLoad(float4* mine, const float4* R) {
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(mine);
#pragma unroll
    for (int k = 0; k < kRowWords; ++k) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + k * 32 * 16), "l"(R + k * kRowTile) : "memory");
    }
}
__device__ __forceinline__ void roomWait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One contact's passes, for either store, with body indices counted from the store's first body (`base`: the same
// first body). The record's words are read at W, S apart: from a lane's room, or from the record itself (W = R); the
// impulses go to the record. A laned contact's bodies are stored only where they move, so a static body shared by a
// color's contacts is never written concurrently. The points' loops stay rolled: unrolled, a pass is 1,600
// instructions of straight code, and a world with few warps waited for them 1.8 of every 8.4 cycles it was not at a
// barrier (0.3 of 5.9 now; box pyramid).
//
// warmStartLaned: each point's normal and tangent impulses pushed in point order (src/lanes.cpp:195-217).
template <int S, class Store>
__device__ __forceinline__ void warmRecord(const Batch& B, const Store& st, uint32_t base, uint32_t limit, const float4* W) {
    const float4 h = W[kRowHead * S];
    const uint32_t ia = __float_as_uint(h.x) - base, ib = __float_as_uint(h.y) - base;
    const int n = (int)__float_as_uint(h.z);
#if defined(TF_DEVICE_CHECKS)
    if (!TF_OK_INDEX(B, ia < limit && ib < limit && n >= 0 && n <= 4, 10, base, ia)) { return; }
#endif
    if (n == 0) { return; }
    LanedBody a = st.loadLaned(ia), b = st.loadLaned(ib);
    const bool moveA = !anchored(a), moveB = !anchored(b);
    const Vec3 t1 = xyz(W[kRowT1 * S]), t2 = xyz(W[kRowT2 * S]);
    const SixVec lin = getSix<S>(W, kRowLinear);
    const float4* pt = W + kRowPoint * S;
#pragma unroll 1
    for (int i = 0; i < n; ++i, pt += kRowPointWords * S) {
        const float in = pt[2 * S].z;
        const Vec3 ti = xyz(pt[3 * S]);
        const SixVec ang = getSix<S>(pt, 4);
        auto push = [&](int k, float impulse) {
            if (moveA) {
                a.v -= lin.v[k] * impulse;
                a.w -= ang.v[k] * impulse;
            }
            if (moveB) {
                b.v += lin.v[k + 1] * impulse;
                b.w += ang.v[k + 1] * impulse;
            }
        };
        push(0, in);
        push(2, dot(ti, t1));
        push(4, dot(ti, t2));
    }
    if (moveA) { st.storeVW(ia, a); }
    if (moveB) { st.storeVW(ib, b); }
}

// solveLaned: the soft normal rows, then friction forward in the biased pass and in reverse in relax, with the
// operations and order of solveContact (src/solver.cpp:360-421, src/lanes.cpp:220-315).
template <int S, class Store>
__device__ __forceinline__ void solveRecord(const Batch& B, const StepParams& P, const Store& st, uint32_t base,
                                            uint32_t limit, float4* W, float4* R, bool useBias) {
    const float4 h = W[kRowHead * S];
    const uint32_t ia = __float_as_uint(h.x) - base, ib = __float_as_uint(h.y) - base;
    const int n = (int)__float_as_uint(h.z);
#if defined(TF_DEVICE_CHECKS)
    if (!TF_OK_INDEX(B, ia < limit && ib < limit && n >= 0 && n <= 4, 12, base, ia)) { return; }
#endif
    if (n == 0) { return; }
    LanedBody a = st.loadLaned(ia), b = st.loadLaned(ib);
    const bool moveA = !anchored(a), moveB = !anchored(b);
    const Softness soft = (!moveA || !moveB) ? P.staticSoft : P.contactSoft;
    const float4 nf = W[kRowNormal * S];
    const Vec3 normal = xyz(nf);
    const SixVec lin = getSix<S>(W, kRowLinear);
    const Vec3 dp = b.dp - a.dp;
    float4* pt = W + kRowPoint * S;
#pragma unroll 1
    for (int i = 0; i < n; ++i, pt += kRowPointWords * S) {
        const float4 pa = pt[0], pb = pt[S];
        const float2 im = reinterpret_cast<const float2*>(pt + 2 * S)[1];
        const float4 g0 = pt[4 * S], g1 = pt[5 * S];
        const Vec3 ra = xyz(pa), rb = xyz(pb);
        const Vec3 d = dp + turned(b, rb) - turned(a, ra);
        const float sep = dot(d, normal) + pa.w;
        float bias = 0.0f, massScale = 1.0f, impulseScale = 0.0f;
        if (sep > 0.0f) {
            bias = sep * P.invH;
        } else if (useBias) {
            bias = maxf(soft.biasRate * sep, -P.maxPushout);
            massScale = soft.massScale;
            impulseScale = soft.impulseScale;
        }
        const Axis x = rowAxis(ra, rb, normal, lin.v[0], Vec3{ g0.x, g0.y, g0.z }, lin.v[1], Vec3{ g0.w, g1.x, g1.y }, pb.w);
        const float vn = speedAlong(a, b, normal, x);
        float impulse = -x.mass * massScale * (vn + bias) - impulseScale * im.x;
        const float total = maxf(im.x + impulse, 0.0f);
        impulse = total - im.x;
        reinterpret_cast<float2*>(pt + 2 * S)[1] = make_float2(total, maxf(im.y, impulse));
        pushMoving(a, b, x, impulse, moveA, moveB);
    }
    const Vec3 t1 = xyz(W[kRowT1 * S]), t2 = xyz(W[kRowT2 * S]);
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const int i = useBias ? k : n - 1 - k;
        const float4* q = W + (kRowPoint + kRowPointWords * i) * S;
        float4* out = R + (kRowPoint + kRowPointWords * i) * kRowTile;
        const Vec3 ra = xyz(q[0]), rb = xyz(q[S]), old = xyz(q[3 * S]);
        const float4 pm = q[2 * S];
        const SixVec ang = getSix<S>(q, 4);
        const Axis x1 = rowAxis(ra, rb, t1, lin.v[2], ang.v[2], lin.v[3], ang.v[3], pm.x);
        const Axis x2 = rowAxis(ra, rb, t2, lin.v[4], ang.v[4], lin.v[5], ang.v[5], pm.y);
        const float old1 = dot(old, t1), old2 = dot(old, t2);
        float f1 = old1 - x1.mass * speedAlong(a, b, t1, x1);
        float f2 = old2 - x2.mass * speedAlong(a, b, t2, x2);
        const float most = nf.w * pm.z;
        const float mag = sqrtf(f1 * f1 + f2 * f2);
        if (mag > most) {
            const float scale = mag > 0.0f ? most / mag : 0.0f;
            f1 *= scale;
            f2 *= scale;
        }
        pushMoving(a, b, x1, f1 - old1, moveA, moveB);
        pushMoving(a, b, x2, f2 - old2, moveA, moveB);
        // The tangent masses stay; only the impulses are written.
        if (S != kRowTile) { reinterpret_cast<float2*>(out + 2 * kRowTile)[1] = make_float2(pm.z, pm.w); }
        out[3 * kRowTile] = f4(t1 * f1 + t2 * f2, 0.0f);
    }
    if (moveA) { st.storeVW(ia, a); }
    if (moveB) { st.storeVW(ib, b); }
}

// Runs f(words, record) on every contact of each color, a color at a time; slotAt gives the record slot of a
// position. With rooms, the records are solved from the lane's room (mine) and a color's first ones are asked for
// before the barrier that ends the color before it: contacts of a pass write only their own records, each in one
// color.
template <bool Rooms, class Slot, class F>
__device__ __forceinline__ void forEachColorRecord(const Batch& B, const Group& g, const uint32_t* start, uint32_t colors,
                                                   float4* mine, Slot slotAt, F f) {
    auto ask = [&](uint32_t x, uint32_t end) {
        if (Rooms && x < end) { roomLoad(mine, rowOf(B, slotAt(x))); }
    };
    if (colors > 0) { ask(start[0] + g.tid, start[1]); }
    for (uint32_t k = 0; k < colors; ++k) {
        const uint32_t end = start[k + 1];
        for (uint32_t x = start[k] + g.tid; x < end; x += g.size) {
            float4* R = rowOf(B, slotAt(x));
            if constexpr (Rooms) { roomWait(); }
            f(Rooms ? mine : R, R);
            ask(x + g.size, end);
        }
        if (k + 1 < colors) { ask(end + g.tid, start[k + 2]); }
        g.sync();
    }
}

// A refresh works on the contact itself: a laned contact first takes its impulses back from its record, and
// afterwards gets its record built again; a contact solved on its own gets its axes built again.
__device__ __forceinline__ void takeImpulsesBack(const Batch& B, const WorldInfo& wi, uint32_t ci, DContact& c) {
    if (c.flags & kCLaned) { returnImpulses(B, B.slotOf[wi.contactFirst + ci], c); }
}

__device__ __forceinline__ void rebuildSolverData(const Batch& B, const WorldInfo& wi, uint32_t ci, const DContact& c) {
    if (c.flags & kCLaned) {
        buildRow(B, wi, B.slotOf[wi.contactFirst + ci], ci);
        return;
    }
    makeContactAxes(axisBodyOf(B.bodies[c.bodyA]), axisBodyOf(B.bodies[c.bodyB]), c,
                    B.axes + (size_t)(wi.contactFirst + ci) * kAxesPerContact);
}

// The flat solve's store: the solver state of every body in global memory, kFlatBodyWords float4 a body
// (velocity and spin, the substep's displacement and turn, type | awake << 8 | alive << 16), small enough that
// a batch's bodies stay in L2 while its contacts are solved, indexed from a first body (a world's, or 0 for
// global indices). The same loads and stores as SolverStore's, over that array. For whole-batch views it also
// holds each body's pose (kFlatPoseWords) and the step's velocity-update terms (kFlatMotionWords), so that the
// body phases of a substep read a few coalesced words instead of the body's whole record.
constexpr int kFlatBodyWords = 4;
constexpr int kFlatPoseWords = 5;    // com, sleepTime; xf.p, extent; xf.q; qBase; localCenter
constexpr int kFlatMotionWords = 7;  // gravity-and-force term, linear damping factor; torque term, angular
                                     // damping factor; linear then angular projection (18 floats, 2 unused)

struct FlatStore {
    float4* s;
    DBody* g;
    float4* pose = nullptr;
    float4* motion = nullptr;
    static constexpr bool staged = true;

    __device__ __forceinline__ uint32_t flags(uint32_t i) const { return __float_as_uint(s[kFlatBodyWords * i + 3].y); }

    __device__ __forceinline__ LanedBody loadLaned(uint32_t i) const {
        const float4 a = s[kFlatBodyWords * i], b = s[kFlatBodyWords * i + 1], c = s[kFlatBodyWords * i + 2],
                     d = s[kFlatBodyWords * i + 3];
        LanedBody x;
        x.v = { a.x, a.y, a.z };
        x.w = { a.w, b.x, b.y };
        x.dp = { b.z, b.w, c.x };
        x.dq = { c.y, c.z, c.w, d.x };
        const uint32_t f = __float_as_uint(d.y);
        x.type = f & 0xffu;
        x.awake = (f >> 8) & 0xffu;
        return x;
    }

    __device__ SBody load(uint32_t i) const {
        const LanedBody l = loadLaned(i);
        SBody b;
        b.v = l.v;
        b.w = l.w;
        b.dp = l.dp;
        b.dq = l.dq;
        b.type = l.type;
        b.awake = l.awake;
        b.invInertiaWorld = g[i].invInertiaWorld;
        b.planeInvMass = g[i].planeInvMass;
        b.planeInvInertia = g[i].planeInvInertia;
        return b;
    }

    template <class BodyT>
    __device__ __forceinline__ void storeVW(uint32_t i, const BodyT& b) const {
        s[kFlatBodyWords * i] = make_float4(b.v.x, b.v.y, b.v.z, b.w.x);
        reinterpret_cast<float2*>(s + kFlatBodyWords * i + 1)[0] = make_float2(b.w.y, b.w.z);
    }

    __device__ __forceinline__ void put(uint32_t i, const Vec3& v, const Vec3& w, const Vec3& dp, const Quat& dq,
                                        uint32_t f) const {
        s[kFlatBodyWords * i] = make_float4(v.x, v.y, v.z, w.x);
        s[kFlatBodyWords * i + 1] = make_float4(w.y, w.z, dp.x, dp.y);
        s[kFlatBodyWords * i + 2] = make_float4(dp.z, dq.x, dq.y, dq.z);
        s[kFlatBodyWords * i + 3] = make_float4(dq.w, __uint_as_float(f), 0.0f, 0.0f);
    }
};

__device__ __forceinline__ float4 q4(const Quat& q) { return make_float4(q.x, q.y, q.z, q.w); }
__device__ __forceinline__ Quat quatOf(const float4& v) { return Quat{ v.x, v.y, v.z, v.w }; }

// integrateVelocity's terms that stay fixed over a step (gravity and force, the damping factors, the
// projections) and the torque term, which changes only with the world inverse inertia. Stored as the very
// values integrateVelocity forms from them (src/world.cpp:1141-1151), so adding them gives its bits.
__device__ __forceinline__ void storeTorqueTerm(const FlatStore& f, uint32_t i, const DBody& d, const StepParams& P) {
    float4* m = f.motion + (size_t)kFlatMotionWords * i;
    const Vec3 t = d.invInertiaWorld * d.torque * P.h;
    m[1] = make_float4(t.x, t.y, t.z, m[1].w);
}

__device__ __forceinline__ void storeMotion(const FlatStore& f, uint32_t i, const DBody& d, const StepParams& P) {
    float4* m = f.motion + (size_t)kFlatMotionWords * i;
    const float h = P.h;
    const Vec3 gv = (P.gravity * d.gravityScale + d.force * d.invMass) * h;
    const Vec3 t = d.invInertiaWorld * d.torque * h;
    m[0] = f4(gv, 1.0f / (1.0f + h * d.linearDamping));
    m[1] = f4(t, 1.0f / (1.0f + h * d.angularDamping));
    const Mat3& L = d.linearProj;
    const Mat3& A = d.angularProj;
    m[2] = make_float4(L.r[0].x, L.r[0].y, L.r[0].z, L.r[1].x);
    m[3] = make_float4(L.r[1].y, L.r[1].z, L.r[2].x, L.r[2].y);
    m[4] = make_float4(L.r[2].z, A.r[0].x, A.r[0].y, A.r[0].z);
    m[5] = make_float4(A.r[1].x, A.r[1].y, A.r[1].z, A.r[2].x);
    m[6] = make_float4(A.r[2].y, A.r[2].z, 0.0f, 0.0f);
}

// The first substep's staging: the body's solver state, pose and velocity terms from its record.
static __device__ void flatBegin(const FlatStore& f, uint32_t i, const StepParams& P) {
    const DBody d = readBody<kBodySolve | kBodyInvInertia | kBodyForce | kBodyProj | kBodyPose | kBodyCom | kBodyLocal | kBodyBase>(f.g[i]);
    f.put(i, d.v, d.w, d.dp, d.dq, d.type | (d.awake << 8) | (d.alive << 16));
    float4* q = f.pose + (size_t)kFlatPoseWords * i;
    q[0] = f4(d.com, d.sleepTime);
    q[1] = f4(d.xf.p, d.extent);
    q[2] = q4(d.xf.q);
    q[3] = q4(d.qBase);
    q[4] = f4(d.localCenter, 0.0f);
    if (d.alive && d.type == kDynamic && d.awake) { storeMotion(f, i, d, P); }
}

// What limitSpeed reads and writes.
struct SpeedBody {
    Vec3 v, w;
    float kept;
    uint32_t type, awake;
};

// integrateVelocity from the store and the step's terms: the same operations on the same values.
static __device__ void flatVelocity(const FlatStore& f, uint32_t i, const StepParams& P) {
    const uint32_t fl = f.flags(i);
    const uint32_t type = fl & 0xffu, awake = (fl >> 8) & 0xffu, alive = fl >> 16;
    if (!alive || type != kDynamic || !awake) { return; }
    const LanedBody l = f.loadLaned(i);
    const float4* m = f.motion + (size_t)kFlatMotionWords * i;
    const float4 m0 = m[0], m1 = m[1], a = m[2], b = m[3], c = m[4], d = m[5], e = m[6];
    Mat3 L, A;
    L.r[0] = { a.x, a.y, a.z };
    L.r[1] = { a.w, b.x, b.y };
    L.r[2] = { b.z, b.w, c.x };
    A.r[0] = { c.y, c.z, c.w };
    A.r[1] = { d.x, d.y, d.z };
    A.r[2] = { d.w, e.x, e.y };
    SpeedBody s;
    s.type = type;
    s.awake = awake;
    const float kept = s.kept = f.g[i].kept;
    s.v = l.v + xyz(m0);
    s.v = L * (s.v * m0.w);
    s.w = l.w + xyz(m1);
    s.w = A * (s.w * m1.w);
    limitSpeed(s, P.maxLinearSpeed, P.maxAngularSpeed);
    f.storeVW(i, s);
    if (s.kept != kept) { f.g[i].kept = s.kept; }
}

// The pose in the store, into a body.
__device__ __forceinline__ void flatPoseOf(const FlatStore& f, uint32_t i, DBody& b) {
    const float4* q = f.pose + (size_t)kFlatPoseWords * i;
    const float4 com = q[0], at = q[1];
    b.com = xyz(com);
    b.sleepTime = com.w;
    b.xf.p = xyz(at);
    b.extent = at.w;
    b.xf.q = quatOf(q[2]);
    b.qBase = quatOf(q[3]);
}

// integratePosition from the store and the pose: the new pose goes to the store, and with joints to the body's record
// as well (those of the relaxing pass read it there).
template <bool Joints>
static __device__ void flatPosition(const FlatStore& f, uint32_t i, const StepParams& P) {
    const uint32_t fl = f.flags(i);
    const LanedBody l = f.loadLaned(i);
    float4* q = f.pose + (size_t)kFlatPoseWords * i;
    DBody& d = f.g[i];
    DBody b;
    flatPoseOf(f, i, b);
    b.alive = fl >> 16;
    b.type = l.type;
    b.awake = l.awake;
    b.v = l.v;
    b.w = l.w;
    b.dp = l.dp;
    b.dq = l.dq;
    b.localCenter = xyz(q[4]);
    const float kept = b.kept = d.kept;
    integratePosition(b, P);
    f.put(i, b.v, b.w, b.dp, b.dq, fl);
    q[0] = f4(b.com, b.sleepTime);
    q[1] = f4(b.xf.p, b.extent);
    q[2] = q4(b.xf.q);
    if constexpr (Joints) { writeBody<kBodyPose | kBodyCom>(d, b); }
    if (b.kept != kept) { d.kept = b.kept; }
}

// The passes of a contact solved on its own, for either store, from the contact and its stored axes; both bodies are
// stored, as the reference does.
template <class Store>
__device__ __forceinline__ void warmOne(const Batch& B, const WorldInfo& wi, const WorldCounts& wc, const Store& st,
                                        uint32_t ci) {
    if (!contactOk(B, wi, wc, ci, 10)) { return; }
    DContact& c = B.contacts[wi.contactFirst + ci];
    const uint32_t ia = c.bodyA - wi.bodyFirst, ib = c.bodyB - wi.bodyFirst;
    SBody a = st.load(ia), b = st.load(ib);
    warmStartContact(a, b, c, false, B.axes + (size_t)(wi.contactFirst + ci) * kAxesPerContact);
    st.storeVW(ia, a);
    st.storeVW(ib, b);
}

template <class Store>
__device__ __forceinline__ void solveOne(const Batch& B, const StepParams& P, const WorldInfo& wi, const WorldCounts& wc,
                                         const Store& st, uint32_t ci, bool bias) {
    if (!contactOk(B, wi, wc, ci, 12)) { return; }
    DContact& c = B.contacts[wi.contactFirst + ci];
    const uint32_t ia = c.bodyA - wi.bodyFirst, ib = c.bodyB - wi.bodyFirst;
    SBody a = st.load(ia), b = st.load(ib);
    solveContact(a, b, c, P, bias, B.axes + (size_t)(wi.contactFirst + ci) * kAxesPerContact);
    st.storeVW(ia, a);
    st.storeVW(ib, b);
}

// Whether the substep `sub` starts with a refresh of world wc: fast pairs are collided again at the middle
// substep, pairs of solid bodies also at every other substep but the first (src/world.cpp:1658-1668).
__device__ __forceinline__ bool refreshedAt(const WorldCounts& wc, int sub, int n) {
    return sub > 0 && (sub == n / 2 ? wc.fastCount : wc.fastSolidCount) > 0;
}

// Whether any world of the batch is.
__device__ __forceinline__ bool batchRefreshedAt(const Batch& B, int sub, int n) {
    return sub > 0 && (*(volatile uint32_t*)(B.work + kSlotFast) & (sub == n / 2 ? 1u : 2u)) != 0;
}

// The contact half of a refresh, over the worlds refreshed at this substep: other contacts are rebased,
// fast ones collided again with the time left, and every active contact's axes built again. One thread per
// contact; the contacts come from one flat list, a pair class of fast contacts (refreshClass) or the other active
// contacts (refreshLight, listed in the order of their records). The body half runs in the substeps around it: the
// substep before updates the world inverse inertia at its end, the substep after resets dp and dq before anything
// reads them.
__device__ __forceinline__ void refreshLight(const Batch& B, const StepParams& P, int sub) {
    const uint32_t items = *(volatile uint32_t*)(B.work + kSlotFastItems + kPairClasses);
    const uint2* its = B.contactItems + (size_t)kPairClasses * B.contactItemStride;
    for (uint32_t item = blockIdx.x * blockDim.x + threadIdx.x; item < items; item += gridDim.x * blockDim.x) {
        const uint2 it = its[item];
        const WorldCounts& wc = B.counts[it.x];
        if (!refreshedAt(wc, sub, P.substeps)) { continue; }
        const WorldInfo& wi = B.info[it.x];
        if (!contactOk(B, wi, wc, it.y, 16)) { continue; }
        const uint32_t slot = B.slotOf[wi.contactFirst + it.y];
        if (slot != kNoSlot) {
            rebaseRow(B, slot);
            continue;
        }
        DContact& c = B.contacts[wi.contactFirst + it.y];
        const DBody& a = B.bodies[c.bodyA];
        const DBody& b = B.bodies[c.bodyB];
        rebaseContact(a, b, c);
        makeContactAxes(axisBodyOf(a), axisBodyOf(b), c, B.axes + (size_t)(wi.contactFirst + it.y) * kAxesPerContact);
    }
}

template <int Cls>
__device__ __forceinline__ void refreshClass(const Batch& B, const StepParams& P, int sub, uint32_t turn = 0, uint32_t turns = 1) {
    const int n = P.substeps;
    const uint8_t againFlag = sub == n / 2 ? kFlagFast : kFlagFastSolid;
    const float remaining = (float)(n - sub) * P.h;
    const uint32_t items = *(volatile uint32_t*)(B.work + kSlotFastItems + Cls);
    const uint2* its = B.contactItems + (size_t)Cls * B.contactItemStride;
    forSpreadItems(items, turn, turns, [&](uint32_t item, bool mine, bool) {
        if (!mine) { return; }
        const uint2 it = its[item];
        const WorldCounts& wc = B.counts[it.x];
        if (!refreshedAt(wc, sub, n)) { return; }
        const WorldInfo wi = B.info[it.x];
        const uint32_t ci = it.y;
        if (!contactOk(B, wi, wc, ci, 16)) { return; }
        DContact& c = B.contacts[wi.contactFirst + ci];
        const bool again = (B.cflags[wi.contactFirst + ci] & againFlag) != 0;
        if constexpr (Cls == kClassMesh) {
            // The contacts of a mesh pair share a key and sit together; the first takes the whole run.
            const DContact* cs = B.contacts + wi.contactFirst;
            if (ci > 0 && cs[ci - 1].key == c.key) { return; }
            uint32_t end = ci + 1;
            while (end < wc.contactCount && cs[end].key == c.key) { ++end; }
            DContact* run = B.contacts + wi.contactFirst + ci;
            const int count = (int)(end - ci);
            for (int x = 0; x < count; ++x) { takeImpulsesBack(B, wi, ci + x, run[x]); }
            if (again) {
                refreshMeshRun<false>(B, P, wi, B.counts[it.x], run, count, remaining);
            } else {
                for (int x = 0; x < count; ++x) { rebaseContact(B.bodies[run[x].bodyA], B.bodies[run[x].bodyB], run[x]); }
            }
            for (int x = 0; x < count; ++x) { rebuildSolverData(B, wi, ci + x, run[x]); }
            return;
        }
        takeImpulsesBack(B, wi, ci, c);
        if (again) {
            refreshContact<Cls>(B, P, c, remaining);
        } else {
            rebaseContact(B.bodies[c.bodyA], B.bodies[c.bodyB], c);
        }
        rebuildSolverData(B, wi, ci, c);
    });
}

// The fast mesh pairs' contacts, a warp per item (the first contact of a pair's run takes the run), the warp's
// lanes over the pair's triangles when it is collided again. Launched with at most kMeshWarps warps to a CTA.
__device__ __forceinline__ void refreshMeshPairs(const Batch& B, const StepParams& P, int sub) {
    __shared__ MeshWarpRoom s_rooms[kMeshWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t perCta = min(blockDim.x >> 5, (uint32_t)kMeshWarps);  // warps past the rooms stay idle
    if (warp >= perCta) { return; }
    const int n = P.substeps;
    const uint8_t againFlag = sub == n / 2 ? kFlagFast : kFlagFastSolid;
    const float remaining = (float)(n - sub) * P.h;
    const uint32_t items = *(volatile uint32_t*)(B.work + kSlotFastItems + kClassMesh);
    const uint2* its = B.contactItems + (size_t)kClassMesh * B.contactItemStride;
    const uint32_t warps = gridDim.x * perCta;
    for (uint32_t item = blockIdx.x * perCta + warp; item < items; item += warps) {
        const uint2 it = its[item];
        const WorldCounts& wc = B.counts[it.x];
        if (!refreshedAt(wc, sub, n)) { continue; }
        const WorldInfo wi = B.info[it.x];
        const uint32_t ci = it.y;
        if (!contactOk(B, wi, wc, ci, 16)) { continue; }
        const DContact* cs = B.contacts + wi.contactFirst;
        // The contacts of a mesh pair share a key and sit together; the first takes the whole run.
        if (ci > 0 && cs[ci - 1].key == cs[ci].key) { continue; }
        uint32_t end = ci + 1;
        while (end < wc.contactCount && cs[end].key == cs[ci].key) { ++end; }
        DContact* run = B.contacts + wi.contactFirst + ci;
        const int count = (int)(end - ci);
        const bool again = (B.cflags[wi.contactFirst + ci] & againFlag) != 0;
        if (lane == 0) {
            for (int x = 0; x < count; ++x) { takeImpulsesBack(B, wi, ci + x, run[x]); }
        }
        __syncwarp();
        if (again) {
            refreshMeshRun<true>(B, P, wi, B.counts[it.x], run, count, remaining, &s_rooms[warp], lane);
        } else if (lane == 0) {
            for (int x = 0; x < count; ++x) { rebaseContact(B.bodies[run[x].bodyA], B.bodies[run[x].bodyB], run[x]); }
        }
        if (lane == 0) {
            for (int x = 0; x < count; ++x) { rebuildSolverData(B, wi, ci + x, run[x]); }
        }
        __syncwarp();
    }
}

template <int Cls>
__global__ void __launch_bounds__(256) k_refresh(const __grid_constant__ Batch B, const __grid_constant__ StepParams P,
                                                 int sub, int serial) {
    if (stepAborted(B, serial) || !batchRefreshedAt(B, sub, P.substeps)) { return; }
    if constexpr (Cls == kClassMesh) {
        refreshMeshPairs(B, P, sub);
    } else if constexpr (Cls == kClassAny) {
        refreshLight(B, P, sub);
    } else {
        refreshClass<Cls>(B, P, sub);
    }
}

// Small batches refresh every list in one launch (the lists hold disjoint contacts: a pair's contacts are fast
// or not together); large batches launch a kernel per list.
template <int Unused = 0>
__global__ void __launch_bounds__(256) k_refresh_all(const __grid_constant__ Batch B, const __grid_constant__ StepParams P,
                                                     int sub, int serial) {
    if (stepAborted(B, serial) || !batchRefreshedAt(B, sub, P.substeps)) { return; }
    refreshLight(B, P, sub);
    refreshClass<kClassSpheres>(B, P, sub, 1, 7);
    refreshClass<kClassSpherePoly>(B, P, sub, 2, 7);
    refreshClass<kClassPlane>(B, P, sub, 3, 7);
    refreshClass<kClassConvex>(B, P, sub, 4, 7);
    refreshClass<kClassPlanar>(B, P, sub, 5, 7);
    refreshClass<kClassMesh>(B, P, sub, 6, 7);
}

// One pass over a world's joints, before the contacts of that pass (src/world.cpp:1670-1680,
// src/joint.cpp:568-590): kind 0 scales warm starts by the speed the ends kept under the speed limits
// (src/joint.cpp:570-593) and warm starts, 1 is the biased solve, 2 the relaxing solve with its reaction. The
// ends' velocities come from the substep's store.
template <class G, class Store>
__device__ void runJoints(const Batch& B, const StepParams& P, const G& g, const WorldInfo& wi, const Store& st, int kind) {
    const uint32_t nj = wi.jointCount;
    DJoint* js = B.joints + wi.jointFirst;
    auto endOf = [&](uint32_t gbody) {
        if (gbody == kWorldEnd) { return worldEnd(); }
        JBody e = jointBodyOf(B.bodies[gbody]);
        if (st.staged) {
            const LanedBody l = st.loadLaned(gbody - wi.bodyFirst);
            e.v = l.v;
            e.w = l.w;
        }
        return e;
    };
    auto putEnd = [&](uint32_t gbody, const JBody& e) {
        if (gbody == kWorldEnd || e.type != kDynamic || !e.awake) { return; }
        st.storeVW(gbody - wi.bodyFirst, e);
    };
    if (kind == 0) {
        for (uint32_t x = g.tid; x < nj; x += g.size) {
            DJoint& j = js[x];
            const JBody a = endOf(j.bodyA), b = endOf(j.bodyB);
            if (!jointActive(j, a, b)) { continue; }
            const float f = minf(a.kept, b.kept);
            if (f >= 1.0f) { continue; }
            j.linearImpulse = j.linearImpulse * f;
            j.angularImpulse = j.angularImpulse * f;
            j.frictionTurn = j.frictionTurn * f;
            j.axialImpulse *= f;
            j.motorImpulse *= f;
            j.lowerImpulse *= f;
            j.upperImpulse *= f;
            j.frictionImpulse *= f;
            j.swingImpulse *= f;
        }
        g.sync();
        for (uint32_t x = g.tid; x < nj; x += g.size) {
            const DJoint& j = js[x];
            if (!jointActive(j, endOf(j.bodyA), endOf(j.bodyB))) { continue; }
            if (j.bodyA != kWorldEnd) { B.bodies[j.bodyA].kept = 1.0f; }
            B.bodies[j.bodyB].kept = 1.0f;
        }
        g.sync();
    }
    forEachJoint(B, g, wi, [&](uint32_t x) {
        DJoint& j = js[x];
        JBody a = endOf(j.bodyA), b = endOf(j.bodyB);
        if (!jointActive(j, a, b)) { return; }
        if (kind == 0) {
            warmStartJoint(a, b, j);
        } else {
            solveJoint(a, b, j, P, P.jointSoft, kind == 1);
            if (kind == 2) { addReaction(j); }
        }
        putEnd(j.bodyA, a);
        putEnd(j.bodyB, b);
    });
}

// Integrate velocities, warm start, biased solve, integrate positions, relax (src/world.cpp:1669-1680). The
// world's solver state is staged in the group's shared slice when it has at most stageN bodies.
// Joints is false for batches without joints: that instantiation carries no joint code, which would cost the
// contact solve registers.
template <bool Joints, bool Rooms>
__global__ void __launch_bounds__(Rooms ? kRoomWarps * 32 : kMaxBlock) k_substep(const __grid_constant__ Batch B, const __grid_constant__ StepParams P, const __grid_constant__ Split sp, int sub, int serial) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    if (stepAborted(B, serial)) { return; }
    // A launch runs every world's substeps up to the next one that starts with a refresh of any world, their solver state
    // staged throughout; the launches of the substeps it ran return. (Worlds without fast contacts once ran on to the
    // step's end while the others waited for the launch: 1024 impact worlds spent 1374 us of a step's 2690 in the first
    // launch; 1744 together this way.)
    if (sub > 0 && !batchRefreshedAt(B, sub, P.substeps)) { return; }
    // The launches with rooms and without take turns by step: which of them steps the batch is decided when its
    // contacts are known.
    if (Rooms != contactsOutweigh(B)) { return; }
    // The warps' rooms for records lie after the staging slices.
    float4* room = reinterpret_cast<float4*>(s_raw + sp.smemBytes + (Rooms ? threadIdx.x >> 5 : 0u) * kRoomBytes) +
                   (threadIdx.x & 31);
    forWorlds(B, kSlotSubstep + sub, sp, s_raw, [&](const Group& g, uint32_t w, unsigned char* sliceRaw, const StageSizes& ss) {
        float* slice = reinterpret_cast<float*>(sliceRaw);
        const uint32_t stageN = ss.bodies;
        const WorldInfo wi = B.info[w];
        const WorldCounts& wc = B.counts[w];
        const uint32_t cf = wi.contactFirst;
        const uint32_t nb = wi.bodyCount;
        const SolverStore st{ slice, stageN, nb <= stageN, B.bodies + wi.bodyFirst };
        if (refreshedAt(wc, sub, P.substeps)) {
            // The body half of this substep's refresh: the planar placements of its collisions are kept, and
            // every body takes a new base pose (src/world.cpp:1663-1666).
            keepPlacements(B, g, wi);
            for (uint32_t i = g.tid; i < nb; i += g.size) {
                DBody b = readBody<kBodySolve | kBodyPose>(st.g[i]);
                b.dp = zero3();
                b.dq = qid();
                b.qBase = b.xf.q;
                writeBody<kBodySolve | kBodyBase>(st.g[i], b);
            }
            g.sync();
        }
        if (st.staged) {
            for (uint32_t i = g.tid; i < nb; i += g.size) { st.stage(i); }
            g.sync();
        }
        const uint32_t nj = wi.jointCount;
        const uint32_t base = wi.bodyFirst;
        const uint32_t* rest = B.rest + cf;
        const uint32_t* icolored = B.impactColored + cf;
        const uint32_t* irest = B.impactRest + cf;
        const uint32_t* slotOf = B.slotOf + cf;
        constexpr int kStride = Rooms ? 32 : kRowTile;
        int s = sub;
        for (;; ++s) {
            for (uint32_t i = g.tid; i < nb; i += g.size) { st.integrateVelocityAt(i, P); }
            g.sync();
            if constexpr (Joints) {
                if (nj > 0) { runJoints(B, P, g, wi, st, 0); }
            }
            forEachColorRecord<Rooms>(B, g, wc.colorStart, wc.colorCount, room, [&](uint32_t x) { return cf + x; },
                                      [&](float4* W, float4*) { warmRecord<kStride>(B, st, base, nb, W); });
            forEachLevel(g, rest, B.restLevel + cf, wc.restLevels, [&](uint32_t ci) { warmOne(B, wi, wc, st, ci); });
            for (int pass = 0; pass < 2; ++pass) {
                const bool bias = pass == 0;
                if constexpr (Joints) {
                    if (nj > 0) { runJoints(B, P, g, wi, st, bias ? 1 : 2); }
                }
                // The active contacts, then the struck ones again (one call site: the solve is inlined once).
                for (int struck = 0; struck < (wc.impactCount > 0 ? 2 : 1); ++struck) {
                    forEachColorRecord<Rooms>(
                        B, g, struck ? wc.impactColorStart : wc.colorStart, struck ? wc.impactColorCount : wc.colorCount,
                        room, [&](uint32_t x) { return struck ? slotOf[icolored[x]] : cf + x; },
                        [&](float4* W, float4* R) { solveRecord<kStride>(B, P, st, base, nb, W, R, bias); });
                    forEachLevel(g, struck ? irest : rest, (struck ? B.impactRestLevel : B.restLevel) + cf,
                                 struck ? wc.impactRestLevels : wc.restLevels,
                                 [&](uint32_t ci) { solveOne(B, P, wi, wc, st, ci, bias); });
                }
                if (bias) {
                    for (uint32_t i = g.tid; i < nb; i += g.size) { st.integratePositionAt(i, P); }
                    g.sync();
                }
            }
            if (s + 1 >= P.substeps || batchRefreshedAt(B, s + 1, P.substeps)) { break; }
        }
        if (st.staged) {
            for (uint32_t i = g.tid; i < nb; i += g.size) { st.unstage(i); }
            g.sync();
        }
        if (s + 1 < P.substeps && refreshedAt(wc, s + 1, P.substeps)) {
            // The next substep starts with a refresh, whose axes use the inverse inertia at the new pose
            // (src/world.cpp:1660-1662).
            for (uint32_t i = g.tid; i < nb; i += g.size) {
                DBody b = readBody<kBodyMassReads>(st.g[i]);
                if (!b.alive || b.type != kDynamic || !b.awake) { continue; }
                updateInverseInertia(b);
                writeBody<kBodyInvInertia>(st.g[i], b);
            }
        }
    });
}

// ---------------------------------------------------------------------------------------------------------
// The flat solve: one substep of every world of a batch of many small worlds as one cooperative launch.
//
// The world kernels above walk a world's colors with the world's own thread group, so a batch of thousands of
// worlds runs as thousands of short dependent chains, each waiting on its own barriers. Here the barrier is the
// grid's instead: each color's contacts of every world run at once across the device (contacts of one color
// move no body in common, in any world), then the next color, and the body phases run over every body of the
// batch. Contacts solved one at a time (by level), joints and a world's uncolored contacts keep their order
// inside their world, each world's on one warp or thread. Every contact and body sees exactly the operations,
// in the order, of the world kernel, so the results are the same bits.
//
// The grid barrier needs every CTA resident: the kernel is launched cooperatively, with at most as many CTAs
// as fit at once. Its wait is bounded: a CTA that has waited kBarrierSpins polls records kDevTimeout in world
// 0's flags and goes on (the host reports the step as failed), so a fault here cannot hang the device.
constexpr uint32_t kBarrierSpins = 1u << 24;

__device__ __forceinline__ uint32_t loadAcquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void storeRelease(uint32_t* p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t addAcqRel(uint32_t* p, uint32_t v) {
    uint32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Arrivals only grow within a step (the step's work slots start at zero and every flat launch of a step has
// the same grid), so arrival t is at barrier t / gridDim of the step. The last arrival of a barrier publishes
// the number of barriers passed with a release store; the other CTAs wait for it with acquire loads. Nothing
// is reset between barriers, so a barrier costs one atomic round trip, a store and the waiters' polls.
static __device__ void gridBarrier(const Batch& B) {
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t* arrive = B.work + kSlotFlatBarrier;
        uint32_t* passed = B.work + kSlotFlatBarrier + 1;
        __threadfence();  // the CTA's writes before the barrier, ahead of its arrival
        const uint32_t ticket = addAcqRel(arrive, 1u);
        const uint32_t after = ticket / gridDim.x + 1;  // barriers passed once this one is
        if (ticket % gridDim.x == gridDim.x - 1) {
            storeRelease(passed, after);
        } else {
            uint32_t spins = 0;
            while ((int32_t)(loadAcquire(passed) - after) < 0) {
                if (++spins > kBarrierSpins) {
                    atomicOr(&B.counts[0].flags, kDevTimeout);
                    break;
                }
                __nanosleep(32);
            }
        }
    }
    __syncthreads();
}

// The substep `sub` of every world (src/world.cpp:1669-1680), in the world kernel's order. At the first
// substep the step's per-color lists over all worlds are built from the worlds' color ranges.
template <bool Joints>
__global__ void __launch_bounds__(256, 2) k_substep_flat(const __grid_constant__ Batch B, const __grid_constant__ StepParams P,
                                                      int sub, int serial) {
    const bool skip = stepAborted(B, serial);  // the same for every CTA: nothing changes it during the launch
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
    const uint32_t lane = threadIdx.x & 31, warp = tid >> 5, warps = threads >> 5;
    const uint32_t nw = (uint32_t)B.nWorlds, nb = B.totalBodies;
    uint32_t* colorTotal = B.work + kSlotFlatColor;
    uint32_t* impactTotal = B.work + kSlotFlatImpact;
    const FlatStore all{ B.flatBodies, B.bodies, B.flatPose, B.flatMotion };
    if (sub == 0) {
        // Every world's share of each color list, and the most colors any world has.
        if (!skip) {
            for (uint32_t w = tid; w < nw; w += threads) {
                WorldCounts& wc = B.counts[w];
                atomicMax(B.work + kSlotFlatMaxColors, wc.colorCount);
                atomicMax(B.work + kSlotFlatMaxImpact, wc.impactColorCount);
                if (wc.restLevels) { atomicMax(B.work + kSlotFlatMaxRestLevels, wc.restLevels); }
                if (wc.impactRestLevels) { atomicMax(B.work + kSlotFlatMaxImpactRestLevels, wc.impactRestLevels); }
                for (uint32_t k = 0; k < wc.colorCount; ++k) {
                    const uint32_t n = wc.colorStart[k + 1] - wc.colorStart[k];
                    wc.flatColorAt[k] = n ? atomicAdd(colorTotal + k, n) : 0u;
                }
                for (uint32_t k = 0; k < wc.impactColorCount; ++k) {
                    const uint32_t n = wc.impactColorStart[k + 1] - wc.impactColorStart[k];
                    wc.flatImpactAt[k] = n ? atomicAdd(impactTotal + k, n) : 0u;
                }
            }
        }
        gridBarrier(B);
        // The record slots, a warp per world: color k of every world from the sum of the colors before it.
        if (!skip) {
            for (uint32_t w = warp; w < nw; w += warps) {
                const WorldInfo& wi = B.info[w];
                const WorldCounts& wc = B.counts[w];
                const uint32_t cf = wi.contactFirst;
                uint32_t before = 0;
                for (uint32_t k = 0; k < wc.colorCount; ++k) {
                    const uint32_t from = before + wc.flatColorAt[k], s0 = wc.colorStart[k], s1 = wc.colorStart[k + 1];
                    for (uint32_t x = s0 + lane; x < s1; x += 32) { B.flatColored[from + (x - s0)] = cf + x; }
                    before += colorTotal[k];
                }
                before = 0;
                for (uint32_t k = 0; k < wc.impactColorCount; ++k) {
                    const uint32_t from = before + wc.flatImpactAt[k], s0 = wc.impactColorStart[k];
                    const uint32_t s1 = wc.impactColorStart[k + 1];
                    for (uint32_t x = s0 + lane; x < s1; x += 32) {
                        B.flatImpact[from + (x - s0)] = B.slotOf[cf + B.impactColored[cf + x]];
                    }
                    before += impactTotal[k];
                }
            }
        }
        gridBarrier(B);
    }
    const uint32_t colors = B.work[kSlotFlatMaxColors], impactColors = B.work[kSlotFlatMaxImpact];
    // Whether any world has contacts solved one at a time (the same for every CTA: set before a barrier).
    const bool anyRest = B.work[kSlotFlatMaxRestLevels] != 0, anyImpactRest = B.work[kSlotFlatMaxImpactRestLevels] != 0;

    // At the first substep every body's state, pose and velocity terms are staged; at a later one, the body half
    // of a refresh (planar placements kept, a new base pose) for the worlds refreshed there. Then the velocity
    // update.
    if (!skip) {
        for (uint32_t gb = tid; gb < nb; gb += threads) {
            if (sub == 0) {
                flatBegin(all, gb, P);
            } else {
                DBody& d = B.bodies[gb];
                const uint32_t w = d.world;
                if (refreshedAt(B.counts[w], sub, P.substeps)) {
                    const uint32_t pb = B.info[w].planeBody;
                    if (pb != UINT32_MAX && d.posePending) {
                        keepPose(d, placeInPlane(d, planeNormal(B.bodies[pb])));
                        d.posePending = 0;
                    }
                    const LanedBody l = all.loadLaned(gb);
                    all.put(gb, l.v, l.w, zero3(), qid(), all.flags(gb));
                    float4* q = B.flatPose + (size_t)kFlatPoseWords * gb;
                    q[3] = q[2];
                }
            }
            flatVelocity(all, gb, P);
        }
    }
    gridBarrier(B);
    auto jointsPass = [&](int kind) {
        if constexpr (Joints) {
            if (!skip) {
                const Group g = makeGroup(32);
                for (uint32_t w = warp; w < nw; w += warps) {
                    const WorldInfo& wi = B.info[w];
                    if (wi.jointCount == 0) { continue; }
                    runJoints(B, P, g, wi, FlatStore{ B.flatBodies + (size_t)kFlatBodyWords * wi.bodyFirst, B.bodies + wi.bodyFirst },
                              kind);
                }
            }
            gridBarrier(B);
        }
    };
    // Each color's contacts of every world, a color at a time; the warps take them in turn over the CTAs, so that a
    // color of few contacts still spreads over every SM.
    const uint32_t spread = ((threadIdx.x >> 5) * gridDim.x + blockIdx.x) * 32 + lane;
    auto colorsPass = [&](const uint32_t* list, const uint32_t* totals, uint32_t count, auto&& f) {
        uint32_t from = 0;
        for (uint32_t k = 0; k < count; ++k) {
            const uint32_t n = totals[k];
            if (!skip) {
                for (uint32_t i = spread; i < n; i += threads) { f(list[from + i]); }
            }
            from += n;
            gridBarrier(B);
        }
    };
    // A world's contacts solved on their own, level by level on one warp of the world; nothing, not even the
    // barrier, when no world has any.
    auto restPass = [&](bool impact, auto&& f) {
        if (!(impact ? anyImpactRest : anyRest)) { return; }
        if (!skip) {
            const Group g = makeGroup(32);
            for (uint32_t w = warp; w < nw; w += warps) {
                const WorldInfo& wi = B.info[w];
                const WorldCounts& wc = B.counts[w];
                const uint32_t levels = impact ? wc.impactRestLevels : wc.restLevels;
                if (levels == 0) { continue; }
                const uint32_t cf = wi.contactFirst;
                const FlatStore st{ B.flatBodies + (size_t)kFlatBodyWords * wi.bodyFirst, B.bodies + wi.bodyFirst };
                forEachLevel(g, (impact ? B.impactRest : B.rest) + cf, (impact ? B.impactRestLevel : B.restLevel) + cf,
                             levels, [&](uint32_t ci) { f(wi, wc, st, ci); });
            }
        }
        gridBarrier(B);
    };
    const uint32_t limit = nb;
    jointsPass(0);
    colorsPass(B.flatColored, colorTotal, colors, [&](uint32_t slot) { warmRecord<kRowTile>(B, all, 0u, limit, rowOf(B, slot)); });
    restPass(false, [&](const WorldInfo& wi, const WorldCounts& wc, const FlatStore& st, uint32_t ci) {
        warmOne(B, wi, wc, st, ci);
    });
    for (int pass = 0; pass < 2; ++pass) {
        const bool bias = pass == 0;
        jointsPass(bias ? 1 : 2);
        for (int struck = 0; struck < 2; ++struck) {
            colorsPass(struck ? B.flatImpact : B.flatColored, struck ? impactTotal : colorTotal,
                       struck ? impactColors : colors,
                       [&](uint32_t slot) {
                           float4* R = rowOf(B, slot);
                           solveRecord<kRowTile>(B, P, all, 0u, limit, R, R, bias);
                       });
            restPass(struck != 0, [&](const WorldInfo& wi, const WorldCounts& wc, const FlatStore& st, uint32_t ci) {
                solveOne(B, P, wi, wc, st, ci, bias);
            });
        }
        if (bias) {
            if (!skip) {
                for (uint32_t gb = tid; gb < nb; gb += threads) { flatPosition<Joints>(all, gb, P); }
            }
            gridBarrier(B);
        }
    }
    // Back into the records of the bodies that something reads before the store is used again: after the last substep
    // all of them; before, those of the worlds whose next substep starts with a refresh, which takes the inverse
    // inertia at the new pose (src/world.cpp:1660-1662), and the torque term with it.
    if (!skip) {
        const bool last = sub + 1 >= P.substeps;
        for (uint32_t gb = tid; gb < nb; gb += threads) {
            DBody& d = B.bodies[gb];
            if (!last && !refreshedAt(B.counts[d.world], sub + 1, P.substeps)) { continue; }
            DBody b = readBody<kBodyInvInertia | kBodyForce | kBodyInertia>(d);
            const LanedBody l = all.loadLaned(gb);
            b.v = l.v;
            b.w = l.w;
            b.dp = l.dp;
            b.dq = l.dq;
            b.type = l.type;
            b.awake = l.awake;
            b.alive = all.flags(gb) >> 16;
            flatPoseOf(all, gb, b);
            writeBody<kBodySolve | kBodyPose | kBodyCom | kBodyBase>(d, b);
            if (!last && b.alive && b.type == kDynamic && b.awake) {
                updateInverseInertia(b);
                writeBody<kBodyInvInertia>(d, b);
                storeTorqueTerm(all, gb, b, P);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// After the substeps (src/world.cpp:1682-1726).

__device__ __forceinline__ uint32_t findRoot(uint32_t* parent, uint32_t x) {
    while (parent[x] != x) {
        parent[x] = parent[parent[x]];
        x = parent[x];
    }
    return x;
}

__device__ __forceinline__ uint32_t rootOf(const uint32_t* parent, uint32_t x) {
    while (parent[x] != x) { x = parent[x]; }
    return x;
}

// bound(): every shape's bounds at the body's pose, and the union of those that are not half-spaces
// (src/world.cpp:240-253).
static __device__ void boundBody(const Batch& B, DBody& b) {
    bool any = false;
    for (uint32_t x = 0; x < b.shapeCount; ++x) {
        DShape& s = B.shapes[B.shapeList[b.shapeFirst + x]];
        Vec3 lo, hi;
        shapeBounds(s, B.cx.pt, b.xf * s.local, lo, hi);
        s.lo = lo;
        s.hi = hi;
        if (s.kind == kHalfSpace) { continue; }
        b.lo = any ? minVec(b.lo, lo) : lo;
        b.hi = any ? maxVec(b.hi, hi) : hi;
        any = true;
    }
}

constexpr unsigned long long kNoHit = ~0ull;

// The root of x among bodies whose unions may still be running: parents only ever point to lower bodies.
__device__ __forceinline__ uint32_t hitRoot(const uint32_t* parent, uint32_t x) {
    for (;;) {
        const uint32_t y = ((const volatile uint32_t*)parent)[x];
        if (y == x) { return x; }
        x = y;
    }
}

// Joins the groups of a and b, the higher root under the lower, so each group's root is its lowest body
// whatever order the unions run in. A link that loses a race to another is tried again, a bounded number
// of times.
static __device__ bool uniteHits(uint32_t* parent, uint32_t a, uint32_t b) {
    for (int attempt = 0; attempt < 4096; ++attempt) {
        a = hitRoot(parent, a);
        b = hitRoot(parent, b);
        if (a == b) { return true; }
        if (a > b) {
            const uint32_t t = a;
            a = b;
            b = t;
        }
        if (atomicCAS(&parent[b], b, a) == b) { return true; }
    }
    return false;
}

// The continuous pass of one world after the leaf refit (src/world.cpp:1271-1418). Each fast shape is swept
// against every shape whose bounds over the step meet its own; a body keeps its earliest hit (time, then pair
// order: fast shape, then other shape); dynamic bodies that hit each other form groups, and each awake
// dynamic body of a group with a hit moves back to the group's earliest hit (time, then lowest body),
// carried along by the kinematic body that hit, if one did.
// Shapes wider than this along x (and half-spaces and meshes) are tested against every fast shape.
constexpr float kWideSweep = 16.0f;

// The continuous pass of a large world: the swept bounds of shapes that are not wide are bucketed by their low
// x (a counting sort into the world's per-shape scratch), and each fast shape, a warp at a time, runs test on
// the shapes of the buckets its bounds can overlap (low x within the widest narrow shape's extent below its
// own low x, up to its high x) and on every wide shape. Each pair is visited once, as the full scan would.
template <class G, class Test>
__device__ void sweepCandidates(const Batch& B, const G& g, const WorldInfo& wi, uint32_t nf, Test& test) {
    __shared__ uint32_t s_range[kMaxGroups][4];  // lowest and highest x, widest extent, wide shapes
    uint32_t* range = g.shared(s_range[g.id]);
    const uint32_t sf = wi.shapeFirst, ns = wi.shapeCount;
    uint32_t* order = B.rowScratch + sf;
    uint32_t* ends = B.rowLong + sf;
    uint32_t* wide = B.rowCount + sf;
    if (g.tid == 0) {
        range[0] = orderedKey(FLT_MAX);
        range[1] = orderedKey(-FLT_MAX);
        range[2] = 0;
        range[3] = 0;
    }
    g.sync();
    auto kindOf = [&](uint32_t i) {  // 0 skipped, 1 narrow, 2 wide
        const DShape& s = B.shapes[sf + i];
        if (!s.alive || s.sensor) { return 0; }
        const float w = B.sweptHi[sf + i].x - B.sweptLo[sf + i].x;
        return (s.kind == kHalfSpace || s.kind == kMesh || !(w <= kWideSweep)) ? 2 : 1;
    };
    uint32_t least = orderedKey(FLT_MAX), most = orderedKey(-FLT_MAX), widest = 0;
    for (uint32_t i = g.tid; i < ns; i += g.size) {
        const int k = kindOf(i);
        if (k == 2) { wide[atomicAdd(&range[3], 1u)] = i; }
        if (k != 1) { continue; }
        least = min(least, orderedKey(B.sweptLo[sf + i].x));
        most = max(most, orderedKey(B.sweptHi[sf + i].x));
        widest = max(widest, __float_as_uint(B.sweptHi[sf + i].x - B.sweptLo[sf + i].x));
    }
    least = __reduce_min_sync(0xffffffffu, least);
    most = __reduce_max_sync(0xffffffffu, most);
    widest = __reduce_max_sync(0xffffffffu, widest);
    if (g.lane == 0) {
        atomicMin(&range[0], least);
        atomicMax(&range[1], most);
        atomicMax(&range[2], widest);
    }
    g.sync();
    const uint32_t buckets = max(1u, ns / 4);
    const float minX = fromOrderedKey(range[0]), maxX = fromOrderedKey(range[1]);
    const float scale = (float)buckets / fmaxf(maxX - minX, 1e-6f);
    auto bucketOf = [&](float x) {
        const float t = fminf(fmaxf((x - minX) * scale, 0.0f), (float)(buckets - 1));
        return (uint32_t)t;
    };
    for (uint32_t b = g.tid; b < buckets; b += g.size) { ends[b] = 0; }
    g.sync();
    for (uint32_t i = g.tid; i < ns; i += g.size) {
        if (kindOf(i) == 1) { atomicAdd(&ends[bucketOf(B.sweptLo[sf + i].x)], 1u); }
    }
    g.sync();
    groupScanWords(g, ends, buckets);  // each bucket's fill position, its end once filled
    for (uint32_t i = g.tid; i < ns; i += g.size) {
        if (kindOf(i) == 1) { order[atomicAdd(&ends[bucketOf(B.sweptLo[sf + i].x)], 1u)] = i; }
    }
    g.sync();
    // Padded, so that rounding in the widths and the subtraction below never drops a pair.
    const float ext = __uint_as_float(range[2]) * 1.001f + 1e-3f;
    const uint32_t nWide = range[3];
    for (uint32_t k = g.warp; k < nf; k += g.warps) {
        const uint32_t fi = B.sweepList[sf + k];
        const uint32_t b0 = bucketOf(B.sweptLo[sf + fi].x - ext), b1 = bucketOf(B.sweptHi[sf + fi].x);
        const uint32_t from = b0 > 0 ? ends[b0 - 1] : 0u, to = ends[b1];
        for (uint32_t p = from + g.lane; p < to; p += 32) { test(k, order[p]); }
        for (uint32_t p = g.lane; p < nWide; p += 32) { test(k, wide[p]); }
    }
}

template <class G>
static __device__ void sweepWorld(const Batch& B, const StepParams& P, const G& g, const WorldInfo& wi, WorldCounts& wc,
                           uint32_t* pairs, uint32_t* impacts) {
    const uint32_t sf = wi.shapeFirst, ns = wi.shapeCount, bf = wi.bodyFirst, nb = wi.bodyCount;
    uint32_t* parent = B.hitParent + bf;
    for (uint32_t i = g.tid; i < ns; i += g.size) {
        const DShape& s = B.shapes[sf + i];
        Vec3 lo = s.lo, hi = s.hi;
        if (s.alive && B.bodies[s.body].type != kStatic) {
            Vec3 l, h;
            shapeBounds(s, B.cx.pt, sweepAt(sweepOf(B.bodies[s.body]), 0.0f) * s.local, l, h);
            lo = minVec(lo, l);
            hi = maxVec(hi, h);
        }
        B.sweptLo[sf + i] = lo;
        B.sweptHi[sf + i] = hi;
    }
    for (uint32_t i = g.tid; i < nb; i += g.size) {
        B.hitKey[bf + i] = kNoHit;
        B.groupKey[bf + i] = kNoHit;
        parent[i] = i;
    }
    const uint32_t nf = groupCompact(
        g, ns,
        [&](uint32_t i) {
            const DShape& s = B.shapes[sf + i];
            if (!s.alive || !TF_OK_INDEX(B, s.body - bf < nb, 32, bf, i)) { return false; }
            const DBody& b = B.bodies[s.body];
            if (!b.alive || b.type != kDynamic || !b.awake) { return false; }
            return sweepsShape(B.cx.pt, s, b, length(b.com - b.com0), sweepOf(b).angle);
        },
        [&](uint32_t i, uint32_t pos) { B.sweepList[sf + pos] = i; });
    const float target = P.tol.linearSlop;
    // Fast shape k against shape oi; x = k ns + oi orders equal hit times, whatever order the pairs run in.
    auto testPair = [&](uint32_t k, uint32_t oi) {
        const unsigned long long x = (unsigned long long)k * ns + oi;
        const uint32_t fi = B.sweepList[sf + k];
        const DShape& f = B.shapes[sf + fi];
        const DShape& o = B.shapes[sf + oi];
        if (!o.alive || o.sensor || o.body == f.body) { return; }
        if (!TF_OK_INDEX(B, o.body - bf < nb, 33, bf, oi)) { return; }
        if (joinedBodies(B, wi, o.body, f.body)) { return; }
        if (!boxesOverlap(B.sweptLo[sf + fi], B.sweptHi[sf + fi], B.sweptLo[sf + oi], B.sweptHi[sf + oi])) { return; }
        if (!(f.category & o.mask) || !(o.category & f.mask)) { return; }
        atomicAdd(pairs, 1u);
        const DBody& bo = B.bodies[o.body];
        float t = 1.0f;
        bool ok = true;
        const bool hit = sweepPair(B.cx, f, B.bodies[f.body], o, bo, B.sweptLo[sf + fi], B.sweptHi[sf + fi], target, t, ok);
        if (!ok) { atomicOr(&wc.flags, kDevUnsupported); }
        if (!hit) { return; }
        const unsigned long long order = x < 0xffffffffull ? x : 0xfffffffeull;
        atomicMin(&B.hitKey[f.body], ((unsigned long long)__float_as_uint(t) << 32) | order);
        if (bo.type == kDynamic && !uniteHits(parent, f.body - bf, o.body - bf)) { atomicOr(&wc.flags, kDevTimeout); }
    };
    if (ns <= kSweepBodies || nf <= 32) {
        const unsigned long long total = (unsigned long long)nf * ns;
        for (unsigned long long x = g.tid; x < total; x += g.size) { testPair((uint32_t)(x / ns), (uint32_t)(x % ns)); }
    } else {
        sweepCandidates(B, g, wi, nf, testPair);
    }
    g.sync();
    for (uint32_t i = g.tid; i < nb; i += g.size) {
        const unsigned long long hk = B.hitKey[bf + i];
        if (hk == kNoHit) { continue; }
        atomicMin(&B.groupKey[bf + rootOf(parent, i)], (hk & 0xffffffff00000000ull) | i);
    }
    g.sync();
    for (uint32_t i = g.tid; i < nb; i += g.size) {
        const unsigned long long gk = B.groupKey[bf + rootOf(parent, i)];
        if (gk == kNoHit) { continue; }
        const float t = __uint_as_float((uint32_t)(gk >> 32));
        DBody& b = B.bodies[bf + i];
        if (t >= 1.0f || !b.alive || b.type != kDynamic || !b.awake) { continue; }
        // The member whose hit came first, and what it hit.
        const unsigned long long first = B.hitKey[bf + (uint32_t)gk];
        const uint32_t oi = (uint32_t)((first & 0xffffffffull) % ns);
        const DBody& other = B.bodies[B.shapes[sf + oi].body];
        b.xf = sweepAt(sweepOf(b), t);
        if (other.type == kKinematic) {
            // A kinematic body keeps moving after the hit, so what hit it rides along to the end of the step.
            const Transform k = sweepAt(sweepOf(other), t);
            const Transform ride{ applyInverse(k, b.xf.p), normalize(conjugate(k.q) * b.xf.q) };
            b.xf = other.xf * ride;
        }
        b.com = apply(b.xf, b.localCenter);
        updateInverseMass(b);
        boundBody(B, b);
        atomicAdd(impacts, 1u);
    }
    g.sync();
}

// What the islands ask of a body, a byte each beside one another (Batch::struck, free after the solve): reading it from
// the bodies cost a scattered load for each end of each contact and for each body, three times over.
constexpr uint32_t kEndMoves = 1u, kEndDriven = 2u, kEndAlive = 4u;  // awake and dynamic; kinematic and moving

// Union-find is staged in the group's shared slice (parent and island time by body, union pairs by contact)
// when the world fits, else in its global scratch.
// After the solve (src/world.cpp:1685-1691): active joints turn the step's impulses into a force and torque
// and break past their limits (src/world.cpp:1543-1560), the rest settle positions in order, twice over, and
// every awake dynamic body's world inverse mass is built again at its settled pose. Every thread first finds
// whether any joint was active.
template <class G>
static __device__ void finishJoints(const Batch& B, const StepParams& P, const G& g, const WorldInfo& wi) {
    DJoint* js = B.joints + wi.jointFirst;
    auto endOf = [&](uint32_t gbody) { return gbody == kWorldEnd ? worldEnd() : jointBodyOf(B.bodies[gbody]); };
    bool anyActive = false;
    for (uint32_t x = 0; x < wi.jointCount && !anyActive; ++x) {
        anyActive = jointActive(js[x], endOf(js[x].bodyA), endOf(js[x].bodyB));
    }
    g.sync();
    if (!anyActive) { return; }
    for (uint32_t x = g.tid; x < wi.jointCount; x += g.size) {
        DJoint& j = js[x];
        if (!jointActive(j, endOf(j.bodyA), endOf(j.bodyB))) { continue; }
        j.force = j.force / P.dt;
        j.torque = j.torque / P.dt;
        if (length(j.force) > j.breakForce || length(j.torque) > j.breakTorque) {
            j.broken = 1;
            j.brokeNow = 1;
            j.linearImpulse = zero3();
            j.angularImpulse = zero3();
            j.frictionTurn = zero3();
            j.axialImpulse = j.motorImpulse = j.lowerImpulse = j.upperImpulse = 0.0f;
            j.frictionImpulse = j.swingImpulse = 0.0f;
        }
    }
    g.sync();
    auto putPose = [&](uint32_t gbody, const JBody& e) {
        if (gbody == kWorldEnd || e.type != kDynamic || !e.awake) { return; }
        B.bodies[gbody].com = e.com;
        B.bodies[gbody].xf = e.xf;
    };
    for (int it = 0; it < kSettleIterations; ++it) {
        forEachJoint(B, g, wi, [&](uint32_t x) {
            const DJoint& j = js[x];
            JBody a = endOf(j.bodyA), b = endOf(j.bodyB);
            if (!jointActive(j, a, b)) { return; }
            settleJoint(a, b, j);
            putPose(j.bodyA, a);
            putPose(j.bodyB, b);
        });
    }
    for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
        DBody& b = B.bodies[wi.bodyFirst + i];
        if (b.alive && b.type == kDynamic && b.awake) { updateInverseMass(b); }
    }
    g.sync();
}

// Counts the touching contacts, reports the pairs that began or stopped touching and the fastest struck point
// of each touching pair (src/world.cpp:1424-1468). The first contact of each pair walks the pair's contacts:
// a pair touches where the solver pushed on a point or a point overlaps (by more than the linear slop once it
// touched); a hit is a pushed point approaching faster than the threshold in a contact solved this step.
// Runs after restitution, on the poses the solve left, before kinematic bodies snap to their targets.
template <class G>
static __device__ void reportTouches(const Batch& B, const StepParams& P, const G& g, const WorldInfo& wi, WorldCounts& wc) {
    const uint32_t nc = wc.contactCount;
    DContact* cs = B.contacts + wi.contactFirst;
    uint32_t touchingHere = 0;
    for (uint32_t first = g.tid; first < nc; first += g.size) {
        const uint64_t key = cs[first].key;
        if (first > 0 && cs[first - 1].key == key) { continue; }
        const bool was = (cs[first].flags & kCTouched) != 0;
        const float apart = was ? P.tol.linearSlop : 0.0f;
        bool touching = false;
        float fastest = P.hitThreshold;
        uint32_t struck = UINT32_MAX;
        int point = 0;
        uint32_t last = first;
        for (; last < nc && cs[last].key == key; ++last) {
            const DContact& c = cs[last];
            const int count = c.count;
            // Every point's pieces that are asked for, before any is looked at.
            DPoint seen[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i < count) { seen[i] = readPieces<1, kPointSolveEnd>(c.points[i]); }
            }
            bool pressed = false;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                pressed = pressed || (i < count && (seen[i].separation < 0.0f || seen[i].normalImpulse > 0.0f));
            }
            touchingHere += pressed ? 1u : 0u;
            if (!TF_OK_INDEX(B, c.bodyA - wi.bodyFirst < wi.bodyCount && c.bodyB - wi.bodyFirst < wi.bodyCount, 22,
                             wi.bodyFirst, last)) {
                continue;
            }
            auto solved = [&] { return movingBody(B.bodies[c.bodyA]) || movingBody(B.bodies[c.bodyB]); };
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (i >= count) { break; }
                const DPoint& p = seen[i];
                if (p.maxNormalImpulse > 0.0f) {
                    touching = true;
                    if (-p.relativeVelocity > fastest && solved()) {
                        fastest = -p.relativeVelocity;
                        struck = last;
                        point = i;
                    }
                } else if (p.separation < apart) {
                    touching = true;
                }
            }
        }
        if (touching != was) {
            const uint32_t at = atomicAdd(&wc.touchEvents, 1u);
            B.touchEvents[2 * (size_t)wi.contactFirst + at] = TouchEvent{ key, touching ? 1u : 0u, 1u };
            for (uint32_t k = first; k < last; ++k) {
                cs[k].flags = touching ? (cs[k].flags | kCTouched) : (cs[k].flags & ~kCTouched);
            }
        }
        if (struck != UINT32_MAX) {
            const DContact& c = cs[struck];
            const uint32_t at = atomicAdd(&wc.hitEvents, 1u);
            B.hitEvents[(size_t)wi.contactFirst + at] =
                HitRecord{ key, apply(B.bodies[c.bodyA].xf, c.points[point].localA), c.normal, fastest, 0u };
        }
    }
    if (touchingHere > 0) { atomicAdd(&wc.touching, touchingHere); }
}

template <bool Joints, bool Cluster>
__global__ void __launch_bounds__(kMaxBlock) k_finish(const __grid_constant__ Batch B, const __grid_constant__ StepParams P, const __grid_constant__ Split sp, int serial) {
    extern __shared__ __align__(16) unsigned char s_raw[];
    __shared__ uint32_t s_awake[kMaxGroups], s_islands[kMaxGroups], s_sweep[kMaxGroups], s_pairs[kMaxGroups],
        s_impacts[kMaxGroups], s_linked[kMaxGroups];
    if (stepAborted<Cluster>(B, serial)) { return; }
    forSomeWorlds<Cluster>(B, kSlotFinish, sp, s_raw, [&](const auto& g, uint32_t w, unsigned char* slice, const StageSizes& ss) {
        const uint32_t stageBodies = ss.bodies, stageContacts = ss.contacts;
        const WorldInfo wi = B.info[w];
        WorldCounts& wc = B.counts[w];
        const uint32_t cf = wi.contactFirst;
        DContact* cs = B.contacts + cf;
        const Axis* axes = B.axes + (size_t)cf * kAxesPerContact;
        uint32_t* awakeSum = g.shared(&s_awake[g.id]);
        uint32_t* islandSum = g.shared(&s_islands[g.id]);
        uint32_t* sweepSum = g.shared(&s_sweep[g.id]);
        uint32_t* pairSum = g.shared(&s_pairs[g.id]);
        uint32_t* impactSum = g.shared(&s_impacts[g.id]);
        uint32_t* linked = g.shared(&s_linked[g.id]);
        if (g.tid == 0) {
            *awakeSum = 0;
            *islandSum = 0;
            *sweepSum = 0;
        }
        // The laned contacts' impulses come back from their records.
        const uint32_t nColored = wc.colorStart[kColors];
        for (uint32_t x = g.tid; x < nColored; x += g.size) {
            const uint32_t ci = __float_as_uint(rowOf(B, cf + x)[kRowHead * kRowTile].w);
            if (!contactOk(B, wi, wc, ci, 18)) { continue; }
            returnImpulses(B, cf + x, cs[ci]);
        }
        g.sync();
        // Restitution: colored contacts by color (their normal axes built again as the record's passes build
        // them), then the rest in active order.
        forEachColor(g, B.colored + cf, wc.colorStart, wc.colorCount, [&](uint32_t ci) {
            if (!contactOk(B, wi, wc, ci, 18)) { return; }
            DContact& c = cs[ci];
            restituteLaned(B.bodies[c.bodyA], B.bodies[c.bodyB], c, P);
        });
        forEachLevel(g, B.rest + cf, B.restLevel + cf, wc.restLevels, [&](uint32_t ci) {
            if (!contactOk(B, wi, wc, ci, 20)) { return; }
            DContact& c = cs[ci];
            restituteContact(B.bodies[c.bodyA], B.bodies[c.bodyB], c, P, false, axes + (size_t)ci * kAxesPerContact);
        });
        if constexpr (Joints) {
            if (wi.jointCount > 0) { finishJoints(B, P, g, wi); }
        }
        reportTouches(B, P, g, wi, wc);
        g.sync();
        const uint32_t nc = wc.contactCount;
        const bool staged = wi.bodyCount <= stageBodies && nc <= stageContacts;
        uint32_t* parent = staged ? reinterpret_cast<uint32_t*>(slice) : B.unionParent + wi.bodyFirst;
        uint32_t* islandTime = staged ? parent + stageBodies : reinterpret_cast<uint32_t*>(B.islandTime + wi.bodyFirst);
        uint32_t* uA = staged ? islandTime + stageBodies : B.mergeIdxA + cf;
        uint32_t* uB = staged ? uA + stageContacts : B.mergeIdxB + cf;
        const float threshold = P.sleepThreshold;
        for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
            const uint32_t gb = wi.bodyFirst + i;
            DBody& d = B.bodies[gb];
            DBody b = readBody<kBodySolve | kBodyForce | kBodyPose | kBodyCom | kBodyLocal | kBodyInvMass | kBodyLocks |
                               kBodyStart | kBodyBounds | kBodyShapes>(d);
            parent[i] = i;
            islandTime[i] = __float_as_uint(FLT_MAX);
            B.struck[gb] = (uint8_t)((movingBody(b) ? kEndMoves : 0u) |
                                     (b.type == kKinematic && movingAwake(b) ? kEndDriven : 0u) | (b.alive ? kEndAlive : 0u));
            if (!b.alive) { continue; }
            limitSpeed(b, P.maxLinearSpeed, P.maxAngularSpeed);
            b.force = zero3();
            b.torque = zero3();
            if (b.hasTarget) {
                b.xf = d.target;
                b.com = apply(b.xf, b.localCenter);
                b.hasTarget = 0;
                writeBody<kBodyPose | kBodyLocal>(d, b);
            }
            if (b.type != kStatic && !(b.type == kDynamic && !b.awake)) {
                // Leaf refit over the new pose (src/world.cpp:1713-1718).
                boundBody(B, b);
                // Shapes that moved well past what the speculative contacts covered are swept against their
                // surroundings below (src/world.cpp:1280-1292).
                if (P.continuous && b.type == kDynamic && b.awake) {
                    const float moved = length(b.com - b.com0);
                    const float angle = sweepOf(b).angle;
                    for (uint32_t x = 0; x < b.shapeCount; ++x) {
                        const DShape& s = B.shapes[B.shapeList[b.shapeFirst + x]];
                        if (sweepsShape(B.cx.pt, s, b, moved, angle)) { atomicAdd(sweepSum, 1u); }
                    }
                }
            }
            // Sleep timers (src/world.cpp:1176-1185).
            const bool moves = b.type == kDynamic && b.awake;
            const float speed = maxf(length(b.v), length(b.w) * b.extent);
            if (moves) { b.sleepTime = !b.canSleep || speed > threshold ? 0.0f : b.sleepTime + P.dt; }
            writeBody<kBodyVelocity | kBodyForce | kBodyCom | kBodyBounds>(d, b);
            if (!moves) { continue; }
            if (!(isfinite(b.v.x) && isfinite(b.v.y) && isfinite(b.v.z) && isfinite(b.xf.p.x) && isfinite(b.xf.p.y) &&
                  isfinite(b.xf.p.z))) {
                atomicOr(&wc.flags, kDevNonFinite);
            }
        }
        g.sync();
        if (g.tid == 0) {
            *pairSum = 0;
            *impactSum = 0;
        }
        if (P.continuous && *(volatile uint32_t*)sweepSum > 0) { sweepWorld(B, P, g, wi, wc, pairSum, impactSum); }
        // Islands over contacts with points (src/world.cpp:1187-1233). The roots are each component's lowest
        // body whatever order the unions run in, so only the unions themselves run on one thread.
        const uint32_t nu = groupCompact(
            g, nc,
            [&](uint32_t ci) {
                if (!contactOk(B, wi, wc, ci, 22)) { return false; }
                const DContact& c = cs[ci];
                const uint32_t ia = c.bodyA, ib = c.bodyB;
                const uint32_t a = B.struck[ia], b = B.struck[ib];
                if (c.count == 0) { return false; }
                if (a & b & kEndMoves) { return true; }
                if ((a & kEndMoves) && (b & kEndDriven)) {
                    B.bodies[ia].sleepTime = 0.0f;
                } else if ((b & kEndMoves) && (a & kEndDriven)) {
                    B.bodies[ib].sleepTime = 0.0f;
                }
                return false;
            },
            [&](uint32_t ci, uint32_t pos) {
                uA[pos] = cs[ci].bodyA - wi.bodyFirst;
                uB[pos] = cs[ci].bodyB - wi.bodyFirst;
            });
        // The unions run in parallel: each round links the higher of a pair's roots under the lower (parents
        // only ever point to lower bodies, so an atomicMin keeps the lowest link), then points every body at
        // its root, until a round links nothing. Each component ends rooted at its lowest body, which is what
        // the reference's sequential unions give.
        for (;;) {
            if (g.tid == 0) { *linked = 0; }
            g.sync();
            for (uint32_t x = g.tid; x < nu; x += g.size) {
                if (!TF_OK_INDEX(B, uA[x] < wi.bodyCount && uB[x] < wi.bodyCount, 24, w, x)) { continue; }
                const uint32_t ra = rootOf(parent, uA[x]), rb = rootOf(parent, uB[x]);
                if (ra != rb) {
                    atomicMin(&parent[ra > rb ? ra : rb], ra < rb ? ra : rb);
                    *(volatile uint32_t*)linked = 1;
                }
            }
            g.sync();
            const bool again = *(volatile uint32_t*)linked != 0;
            for (uint32_t i = g.tid; again && i < wi.bodyCount; i += g.size) { parent[i] = rootOf(parent, i); }
            g.sync();
            if (!again) { break; }
        }
        if (g.tid == 0) {
            // Joints that hold link their bodies too (src/world.cpp:1210-1222).
            const DJoint* js = B.joints + wi.jointFirst;
            for (uint32_t x = 0; x < wi.jointCount; ++x) {
                const DJoint& j = js[x];
                if (!j.alive || j.broken) { continue; }
                const uint32_t a = j.bodyA == kWorldEnd ? 0u : B.struck[j.bodyA], b = B.struck[j.bodyB];
                if (a & b & kEndMoves) {
                    const uint32_t ra = findRoot(parent, j.bodyA - wi.bodyFirst), rb = findRoot(parent, j.bodyB - wi.bodyFirst);
                    if (ra != rb) { parent[ra > rb ? ra : rb] = ra < rb ? ra : rb; }
                } else if ((a & kEndMoves) && (b & kEndDriven)) {
                    B.bodies[j.bodyA].sleepTime = 0.0f;
                } else if ((b & kEndMoves) && (a & kEndDriven)) {
                    B.bodies[j.bodyB].sleepTime = 0.0f;
                }
            }
        }
        g.sync();
        uint32_t awakeHere = 0, islandsHere = 0;
        for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
            DBody& b = B.bodies[wi.bodyFirst + i];
            const uint32_t state = B.struck[wi.bodyFirst + i];
            const float sleepTime = b.sleepTime;
            if ((state & (kEndAlive | kEndMoves)) != (kEndAlive | kEndMoves)) { continue; }
            const uint32_t r = rootOf(parent, i);
            b.island = r;
            ++awakeHere;
            if (r == i) { ++islandsHere; }
            atomicMin(&islandTime[r], __float_as_uint(sleepTime));
        }
        awakeHere = __reduce_add_sync(0xffffffffu, awakeHere);
        islandsHere = __reduce_add_sync(0xffffffffu, islandsHere);
        if (g.lane == 0) {
            atomicAdd(awakeSum, awakeHere);
            atomicAdd(islandSum, islandsHere);
        }
        g.sync();
        for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
            DBody& b = B.bodies[wi.bodyFirst + i];
            if ((B.struck[wi.bodyFirst + i] & (kEndAlive | kEndMoves)) != (kEndAlive | kEndMoves)) { continue; }
            if (__uint_as_float(islandTime[rootOf(parent, i)]) < P.timeToSleep) { continue; }
            b.awake = 0;
            b.v = zero3();
            b.w = zero3();
            updateInverseMass(b);
        }
        g.sync();
        if (g.tid == 0) {
            wc.awakeBodies = *awakeSum;
            wc.awakeIslands = *islandSum;
            wc.bodySteps += *awakeSum;
            wc.sweepShapes += *sweepSum;
            wc.sweptPairs = *pairSum;
            wc.impacts = *impactSum;
        }
        g.sync();
    });
}
// ---------------------------------------------------------------------------------------------------------
// Host traffic of a running batch: per-step forces in, poses out.

// World::addForce / addTorque with wake = false on every body (src/world.cpp:2118-2142).
// Records what this step's solve will see, right after preparation: every contact of every world with its
// lists and the awake dynamic bodies. One group per world.
template <int Unused = 0>
__global__ void __launch_bounds__(kMaxBlock) k_tape_record(const __grid_constant__ Batch B, const __grid_constant__ Split sp,
                                                           TapeStep T, int serial) {
    if (stepAborted(B, serial)) { return; }
    forWorlds(B, kSlotTape, sp, nullptr, [&](const Group& g, uint32_t w, unsigned char*, const StageSizes&) {
        const WorldInfo wi = B.info[w];
        const WorldCounts& wc = B.counts[w];
        const uint32_t cf = wi.contactFirst;
        if (g.tid == 0) {
            TapeWorld& tw = T.worlds[w];
            tw.contactFirst = cf;
            tw.contactCount = wc.contactCount;
            tw.colorCount = wc.colorCount;
            tw.impactColorCount = wc.impactColorCount;
            tw.restCount = wc.restCount;
            tw.impactRestCount = wc.impactRestCount;
            for (int k = 0; k < kTapeColors; ++k) {
                tw.colorStart[k] = wc.colorStart[k];
                tw.impactColorStart[k] = wc.impactColorStart[k];
            }
        }
        for (uint32_t i = g.tid; i < wc.contactCount; i += g.size) {
            const DContact& c = B.contacts[cf + i];
            TapeContact t;
            t.a = c.bodyA - wi.bodyFirst;
            t.b = c.bodyB - wi.bodyFirst;
            t.shapeA = c.shapeA - wi.shapeFirst;
            t.shapeB = c.shapeB - wi.shapeFirst;
            t.count = c.count;
            t.restitution = c.restitution;
            const Vec3 dirs[3] = { c.normal, c.tangent1, c.tangent2 };
            float* out[3] = { t.normal, t.t1, t.t2 };
            for (int d = 0; d < 3; ++d) {
                out[d][0] = dirs[d].x;
                out[d][1] = dirs[d].y;
                out[d][2] = dirs[d].z;
            }
            for (int k = 0; k < 4; ++k) {
                const DPoint& p = c.points[k];
                const bool on = k < c.count;
                t.anchorA[k][0] = on ? p.anchorA.x : 0.0f, t.anchorA[k][1] = on ? p.anchorA.y : 0.0f;
                t.anchorA[k][2] = on ? p.anchorA.z : 0.0f;
                t.anchorB[k][0] = on ? p.anchorB.x : 0.0f, t.anchorB[k][1] = on ? p.anchorB.y : 0.0f;
                t.anchorB[k][2] = on ? p.anchorB.z : 0.0f;
                t.adjSep[k] = on ? p.adjustedSeparation : 0.0f;
                t.relVel[k] = on ? p.relativeVelocity : 0.0f;
                t.normalImpulse[k] = on ? p.normalImpulse : 0.0f;
                t.tangentImpulse[k][0] = on ? p.tangentImpulse.x : 0.0f;
                t.tangentImpulse[k][1] = on ? p.tangentImpulse.y : 0.0f;
                t.tangentImpulse[k][2] = on ? p.tangentImpulse.z : 0.0f;
            }
            T.contacts[cf + i] = t;
        }
        const uint32_t nColored = wc.colorStart[wc.colorCount], nImpact = wc.impactColorStart[wc.impactColorCount];
        for (uint32_t x = g.tid; x < nColored; x += g.size) { T.colored[cf + x] = B.colored[cf + x]; }
        for (uint32_t x = g.tid; x < nImpact; x += g.size) { T.impactColored[cf + x] = B.impactColored[cf + x]; }
        for (uint32_t x = g.tid; x < wc.restCount; x += g.size) { T.rest[cf + x] = B.rest[cf + x]; }
        for (uint32_t x = g.tid; x < wc.impactRestCount; x += g.size) { T.impactRest[cf + x] = B.impactRest[cf + x]; }
        for (uint32_t i = g.tid; i < wi.bodyCount; i += g.size) {
            T.awake[wi.bodyFirst + i] = movingBody(B.bodies[wi.bodyFirst + i]) ? 1 : 0;
        }
        g.sync();
    });
}

template <int Unused = 0>
__global__ void k_add_forces(DBody* bodies, uint32_t n, const float* __restrict__ f, const float* __restrict__ t) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) { return; }
    DBody& b = bodies[i];
    if (!b.alive || b.type != kDynamic || !b.awake) { return; }
    if (f) { b.force += Vec3{ f[3 * i], f[3 * i + 1], f[3 * i + 2] }; }
    if (t) { b.torque += Vec3{ t[3 * i], t[3 * i + 1], t[3 * i + 2] }; }
}

// What the host checks after every step, from every world's counts in one CTA: the OR of the worlds' flags
// and the sum of their body steps (out[0] flags, out[1..2] the sum's low and high words).
template <int Unused = 0>
__global__ void __launch_bounds__(1024) k_step_summary(const WorldCounts* counts, uint32_t nWorlds, uint32_t* out) {
    __shared__ uint32_t s_flags;
    __shared__ unsigned long long s_steps;
    if (threadIdx.x == 0) {
        s_flags = 0;
        s_steps = 0;
    }
    __syncthreads();
    uint32_t flags = 0;
    unsigned long long steps = 0;
    for (uint32_t w = threadIdx.x; w < nWorlds; w += blockDim.x) {
        flags |= counts[w].flags;
        steps += counts[w].bodySteps;
    }
    atomicOr(&s_flags, flags);
    atomicAdd(&s_steps, steps);
    __syncthreads();
    if (threadIdx.x == 0) {
        out[0] = s_flags;
        out[1] = (uint32_t)s_steps;
        out[2] = (uint32_t)(s_steps >> 32);
    }
}

// Copies the contacts every world holds (counts[w].contactCount of its slots), `parts` CTAs a world. (A snapshot of 4096
// uneven worlds that copied every slot took 0.74 ms to put back, most of it empty slots; 0.17 this way.)
template <int Unused = 0>
__global__ void __launch_bounds__(256) k_copy_contacts(const DContact* from, DContact* to, const WorldInfo* info,
                                                       const WorldCounts* counts, uint32_t nWorlds, uint32_t parts) {
    constexpr uint32_t kPieces = sizeof(DContact) / 16, kAtOnce = 4;
    for (uint32_t t = blockIdx.x; t < nWorlds * parts; t += gridDim.x) {
        const uint32_t w = t / parts, part = t % parts, cap = info[w].contactCap;
        const uint32_t n = min(counts[w].contactCount, cap) * kPieces, share = (n + parts - 1) / parts;
        const uint32_t end = min(n, (part + 1) * share);
        const float4* src = reinterpret_cast<const float4*>(from + info[w].contactFirst);
        float4* dst = reinterpret_cast<float4*>(to + info[w].contactFirst);
        for (uint32_t i = part * share + threadIdx.x; i < end; i += kAtOnce * blockDim.x) {
            float4 piece[kAtOnce];
#pragma unroll
            for (uint32_t u = 0; u < kAtOnce; ++u) {
                if (i + u * blockDim.x < end) { piece[u] = src[i + u * blockDim.x]; }
            }
#pragma unroll
            for (uint32_t u = 0; u < kAtOnce; ++u) {
                if (i + u * blockDim.x < end) { dst[i + u * blockDim.x] = piece[u]; }
            }
        }
    }
}

template <int Unused = 0>
__global__ void k_pack_poses(const DBody* bodies, uint32_t n, float* __restrict__ p, float* __restrict__ q) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) { return; }
    const Transform xf = readBody<kBodyPose>(bodies[i]).xf;
    p[3 * i] = xf.p.x;
    p[3 * i + 1] = xf.p.y;
    p[3 * i + 2] = xf.p.z;
    q[4 * i] = xf.q.x;
    q[4 * i + 1] = xf.q.y;
    q[4 * i + 2] = xf.q.z;
    q[4 * i + 3] = xf.q.w;
}

}

