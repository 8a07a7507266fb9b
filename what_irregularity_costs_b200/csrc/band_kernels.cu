// The band walk: allocate, and count-and-sum (the first half of update,
// fused with allocation in integrate).
//
// Reference: cpp/src/volume.cpp:147-198 and :200-299 (one sample at a time:
// find_or_insert / find_block per sample) and cpp/src/volume_cuda.cu:160-192,
// :259-269, :302-337 (one thread per point, one hash probe sequence per
// sample).
//
// One thread walks one point's band (2*steps+1 samples, kChunk at a time, in its
// columns of shared memory); a persistent grid of CTAs strides over tiles of 128
// consecutive points (neighbouring pixels of a frame). The blocks of a warp's
// samples are resolved through a small table in shared memory (band_point):
// every distinct block of the 32 points is probed once, by one lane, with all
// of the warp's probes (the first two slots of each key's sequence) in flight
// together, so the global table sees a fraction of the per-sample probes and
// far fewer contending CAS attempts on a new block. Points that are no
// neighbours (unordered clouds, spinning lidars, depth edges) leave samples that
// the table cannot hold; those are resolved by the runs of equal blocks along
// each ray (resolve_runs), so that their cost grows with the blocks they meet.
//
// What bounds it (four 640x480 frames a call): L1 throughput of the scattered
// weight gathers and reductions (about 21 M sectors, one a cycle per SM: 75
// us) and instruction issue (57 M warp instructions: 50 us); 104 us measured.
// 143 before the table (67 M instructions, and values spilled around calls);
// 121 with the samples in registers, whose columns left room for fewer loads in
// flight than shared memory does.
//
// Update tail. The resolving lane also tags the block as touched by this update
// (one atomic exchange on the spare word of its table slot, unless the probe
// already showed the tag; the first tagger appends it to the touched list).
// Every band sample whose voxel can still accept a contribution adds one to
// the voxel's batch count and its normalised SDF, in 2^-40 fixed point, to
// the voxel's 64-bit sum: fire-and-forget L2 reductions, whose order does not
// matter. Every band slot (point i, step s) also gets a 4-byte record at
// records[(s + steps) * n + i] -- step-major, so each store of a warp is one
// contiguous 128-byte line -- holding the voxel's global index or kNoVoxel;
// only voxels that cross the cap read them again (their canonical order is
// the record position).
//
// Samples whose voxel already holds the cap's weight are left out: under
// "accept while weight before < cap" they cannot be accepted in any order,
// so leaving them out changes no result.
//
// Several frames per call (band_frames_kernel, band_depth_frames_kernel): the
// same walk, each point seen from the camera of its frame (a table among the
// kernel's parameters; depth images also carry their poses). The points
// of frame k precede those of frame k+1, so the canonical (point, step) order
// is (frame, point, step) order and the cap keeps what per-frame calls keep.
#include <algorithm>
#include <climits>
#include <mutex>

#include "volume.h"

namespace osn_b200 {
namespace {

constexpr int kBandThreads = kBatchTilePoints;
static_assert(kBandThreads >= kMaxBatchScenes, "one thread per scene builds the item prefix");
#ifndef OSN_BAND_CHUNK
#define OSN_BAND_CHUNK 9
#endif
constexpr int kChunk = OSN_BAND_CHUNK;  // samples per ray walked together (9: the whole band at 4 voxels)
// Resident CTAs per SM the register budget is sized for. Four 640x480 frames
// per call took 104.4 us at 7 (72 registers), 103.0 at 8, 110 at 6, and on a mapped
// room (all samples at the cap) 65.0 at 7 and 66.5 at 8; one frame 39.0 us at 8
// (64 registers), 41.6 at 7.
#ifndef OSN_BAND_MIN_BLOCKS
#define OSN_BAND_MIN_BLOCKS 8
#endif
#ifndef OSN_BAND_FRAMES_MIN_BLOCKS
#define OSN_BAND_FRAMES_MIN_BLOCKS 7
#endif
// Several depth images per call: the double-precision unprojection needs more
// (four images 123.7 us at 6, 123.4 at 7; one image is best at 8).
#ifndef OSN_BAND_DEPTH_MIN_BLOCKS
#define OSN_BAND_DEPTH_MIN_BLOCKS 6
#endif
constexpr int kBandDepthMinBlocks = OSN_BAND_DEPTH_MIN_BLOCKS;
constexpr int kBandMinBlocks = OSN_BAND_MIN_BLOCKS;
constexpr int kBandFramesMinBlocks = OSN_BAND_FRAMES_MIN_BLOCKS;

// Band records and slot values are read once more, by the group pass of the
// same update: stored with the streaming hint (1, evict-first) or as
// ordinary write-back stores that may stay in L2 (0; no difference measured).
#ifndef OSN_BAND_STREAM_RECORDS
#define OSN_BAND_STREAM_RECORDS 1
#endif

template <typename T>
__device__ __forceinline__ void store_slot(T* p, T x) {
    if (OSN_BAND_STREAM_RECORDS) __stcs(p, x);
    else *p = x;
}

// A block's pool index (-1: absent or dropped) and the slot that holds its key.
struct Resolved {
    int32_t bi;
    uint32_t slot;
};

template <int MODE>
__device__ __forceinline__ Resolved resolve(const DevVolume& v, long long key,
                                            unsigned long long* hist, int n_bins) {
    const int bx = unpack_axis(key, 2 * kCoordBits);
    const int by = unpack_axis(key, kCoordBits);
    const int bz = unpack_axis(key, 0);
    const uint32_t home = hash_slot(bx, by, bz, v.hash_mask);
    if (MODE == kLookupOnly) {
        uint32_t probes = 0;
        const int32_t bi = find_block(v, bx, by, bz, key, probes);
        return Resolved{bi, (home + probes - 1u) & v.hash_mask};
    }
    const InsertResult r = find_or_insert<MODE>(v, bx, by, bz, key);
    if (MODE == kAllocProbeHist && n_bins > 0)
        atomicAdd(&hist[min(r.probes, (uint32_t)(n_bins - 1))], 1ull);
    return Resolved{r.idx, (home + r.probes - 1u) & v.hash_mask};
}

// Modes whose first probe may be answered from the block's home slot alone.
template <int MODE>
__device__ __forceinline__ constexpr bool has_fast_probe() {
    return MODE == kAllocInsert || MODE == kLookupOnly;
}

constexpr int32_t kUnsettled = -2;  // the full probe is needed

// The home slot of a packed key, from the key's words (x: low, y: high).
__device__ __forceinline__ uint32_t home_slot(const DevVolume& v, uint2 key) {
    constexpr uint32_t kMask = (1u << kCoordBits) - 1u, kBias = (uint32_t)kCoordBias;
    const uint32_t bz = (key.x & kMask) - kBias;
    const uint32_t by = (__funnelshift_r(key.x, key.y, kCoordBits) & kMask) - kBias;
    const uint32_t bx = (key.y >> (2 * kCoordBits - 32)) - kBias;
    return (bx * 73856093u ^ by * 19349663u ^ bz * 83492791u) & v.hash_mask;
}

// The first two slots of a key's probe sequence, both loads in flight
// together, and what they settle: the pool index (and slot) of the key, -1
// when it is absent (lookups), else kUnsettled. A slot goes empty -> claimed
// (key, -1) -> published (key, index) and its key and index never change again
// within an update, so an entry read through L1 that shows this key with a
// valid index is final, wherever it is; and with no concurrent insertion
// (lookup) an empty slot ends the sequence. The hash sends 16 % of a room's
// blocks to their second slot: nearly every warp meets one of them.
struct Probe {
    int4 e0, e1;
};
template <int MODE>
__device__ __forceinline__ Probe probe_start(const DevVolume& v, uint32_t home) {
    Probe p{make_int4(0, 0, -1, 0), make_int4(0, 0, -1, 0)};
    if (has_fast_probe<MODE>()) {
        p.e0 = __ldca(reinterpret_cast<const int4*>(&v.table[home]));
        p.e1 = __ldca(reinterpret_cast<const int4*>(&v.table[(home + 1u) & v.hash_mask]));
    }
    return p;
}
// Sets out (slot: the home slot on entry); returns the touch tag seen.
template <int MODE>
__device__ __forceinline__ uint32_t probe_settle(const DevVolume& v, const Probe& p, uint2 key, Resolved& out) {
    out.bi = kUnsettled;
    if (!has_fast_probe<MODE>()) return 0u;
    const bool at0 = (uint32_t)p.e0.x == key.x && (uint32_t)p.e0.y == key.y;
    const bool at1 = !at0 && (uint32_t)p.e1.x == key.x && (uint32_t)p.e1.y == key.y;
    const int32_t idx = at1 ? p.e1.z : p.e0.z;
    if ((at0 || at1) && (uint32_t)idx < (uint32_t)v.pool_capacity) {
        out.bi = idx;
        if (at1) out.slot = (out.slot + 1u) & v.hash_mask;
    } else if (MODE == kLookupOnly && ((p.e0.x & p.e0.y) == -1 || (!at0 && (p.e1.x & p.e1.y) == -1))) {
        out.bi = -1;  // kEmptyKey before the key
    }
    return (uint32_t)(at1 ? p.e1.w : p.e0.w);
}

// The full probe for the lanes with `need` set (called by the whole warp):
// equal keys are grouped across the warp and one leader per key probes.
template <int MODE>
__device__ __forceinline__ void resolve_grouped(const DevVolume& v, bool need, long long key, Resolved& out,
                                                unsigned long long* hist, int n_bins) {
    const unsigned want = __ballot_sync(0xffffffffu, need);
    if (want == 0u) return;
    if (need) {
        const int leader = __ffs(__match_any_sync(want, key)) - 1;
        Resolved r{-1, 0u};
        if (leader == (int)(threadIdx.x & 31)) r = resolve<MODE>(v, key, hist, n_bins);
        out.bi = __shfl_sync(want, r.bi, leader);
        out.slot = __shfl_sync(want, r.slot, leader);
    }
    __syncwarp();
}

// Tag the blocks of the lanes with `need` set as touched by this update (the
// tag is the spare word of the block's table slot); the first tagger of a
// block appends it to the touched list. Called by the whole warp where any
// lane saw an older tag: one lane per block exchanges (SHARED: lanes may hold
// the same block), and the appends of the warp take their places with one
// atomic on the list's counter.
template <bool SHARED>
__device__ __forceinline__ void tag_touched(const DevVolume& v, const UpdateScratch& u, bool need, int32_t bi,
                                            uint32_t slot) {
    const unsigned want = __ballot_sync(0xffffffffu, need);
    if (want == 0u) return;
    const int lane = (int)(threadIdx.x & 31);
    bool add = false;
    if (need && (!SHARED || __ffs(__match_any_sync(want, bi)) - 1 == lane))
        add = (uint32_t)atomicExch(&v.table[slot].pad, (int)u.tag) != u.tag;
    const unsigned adds = __ballot_sync(0xffffffffu, add);
    if (adds == 0u) return;
    int base = 0;
    if (lane == __ffs(adds) - 1) base = atomicAdd(&u.ctl->n_touched, __popc(adds));
    base = __shfl_sync(0xffffffffu, base, __ffs(adds) - 1);
    if (add) u.touched[base + __popc(adds & lanemask_lt())] = bi;
}

// Fire-and-forget L2 reductions (no value comes back, nothing waits).
__device__ __forceinline__ void red_add(uint32_t* p, uint32_t x) {
    asm volatile("red.global.add.u32 [%0], %1;" ::"l"(p), "r"(x));
}
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long x) {
    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(p), "l"(x));
}

// Shared memory of one band CTA.
//   table    per warp: the blocks of its samples (x: key within the warp, y:
//            pool index), then the runs the table did not settle (full keys)
//   vox      per thread: its samples' voxel offsets, then their voxels
//   dsq      per thread: its samples' squared distances
//   run_key  measurement modes: per-thread columns of run keys (x: low word),
//            run q of thread t at [q][t] (no bank conflicts)
constexpr int kTableEntries = 64;  // two per lane
union BandSmem {
    struct {
        uint2 table[kBandThreads / 32][kTableEntries];
        uint32_t vox[kChunk][kBandThreads];
        float dsq[kChunk][kBandThreads];
    };
    uint2 run_key[kChunk][kBandThreads];
};

// N consecutive band samples of a ray once their blocks are resolved: the
// voxels' weights gathered together, then the saturation gate, counts, sums
// and records. vox, dsq: this thread's columns of the samples' voxels (or
// kNoVoxel) and squared distances of camera and voxel centre (unfused float
// arithmetic, as the reference's), from which the signed distance is taken only
// where a lane counts; f64: the FP64 oracle's value of sample j. n_steps:
// samples in use (warp-uniform). writes: this lane's records are stored.
template <int S, int N, typename F64>
__device__ __forceinline__ void count_samples(const DevVolume& v, const UpdateScratch& u, bool writes,
                                              uint32_t stride, float dist, const uint32_t* vox, const float* dsq,
                                              int n_steps, uint32_t& slot, uint32_t& counted, const F64& f64) {
    // Without a cap no voxel can be full or cross it: no weight is looked at,
    // and no record is kept for the cap selection.
    const bool capped = v.weight_cap > 0.0f;
    uint32_t at[N];
#pragma unroll
    for (int j = 0; j < N; ++j) at[j] = j < n_steps ? vox[j * kBandThreads] : kNoVoxel;
    if (capped) {
        float w0[N];
#pragma unroll
        for (int j = 0; j < N; ++j) w0[j] = weight_in_update<S>(v.weight, at[j] == kNoVoxel ? 0u : at[j]);
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (w0[j] >= v.weight_cap) at[j] = kNoVoxel;  // takes no contribution
    }
#pragma unroll
    for (int j = 0; j < N; ++j) {
        if (j >= n_steps) break;
        const bool counts = at[j] != kNoVoxel;
        if (__any_sync(0xffffffffu, counts)) {
            long long fix;
            float sdf_n = 0.0f;
            if constexpr (S == kStoreF64) {
                fix = counts ? f64(j) : 0ll;
            } else {
                const float sdf = __fsub_rn(dist, __fsqrt_rn(dsq[j * kBandThreads]));
                sdf_n = fminf(fmaxf(__fmul_rn(sdf, v.inv_trunc), -1.0f), 1.0f);
                fix = to_fix(sdf_n);
            }
            if (counts) {
                // Kept for the records of voxels that cross the cap, so the
                // update tail never reads the batch's points again.
                if (S != kStoreF64 && capped) store_slot(u.slot_val + slot, sdf_n);
                red_add(&u.vcnt[at[j]], 1u);
                red_add(&u.vacc[at[j]], (unsigned long long)fix);
                ++counted;
            }
        }
        if (capped && writes) store_slot(u.records + slot, at[j]);  // read again by the group pass
        slot += stride;
    }
}

// The FP64 oracle's normalised SDF of voxel (vx, vy, vz), 2^-40 fixed point.
__device__ __forceinline__ long long oracle_fix(const DevVolume& v, const BatchArgs& a, const Ray& r, int vx,
                                                int vy, int vz) {
    return to_fix(clamp_sdf_n_f64(sdf_f64(v, a, r.px, r.py, r.pz, vx, vy, vz), v.trunc));
}

// The allocate-only walk of the measurement modes: every lane keeps the runs
// of equal blocks of a chunk of its samples (their keys in a column of shared
// memory), and each run index of the warp's lanes is resolved by the full
// probe, one leader per distinct key. Returns the samples dropped.
template <int MODE>
__device__ __forceinline__ uint32_t measure_point(const DevVolume& v, const Ray& r, bool live, uint2 (*run_key)[kBandThreads],
                                                  unsigned long long* hist, int n_bins) {
    const int t = threadIdx.x;
    uint32_t drops = 0u;
    for (int c0 = -v.steps; c0 <= v.steps; c0 += kChunk) {
        int n_run = 0, n_of[kChunk];  // samples of each run
        int ox = 0, oy = 0, oz = 0;   // the last valid sample's voxel
#pragma unroll
        for (int j = 0; j < kChunk; ++j) n_of[j] = 0;
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
            int vx, vy, vz;
            float dsq;
            if (live && c0 + j <= v.steps && band_sample_ray(v, r, c0 + j, vx, vy, vz, dsq)) {
                // A straight ray leaves a block (a convex box) for good, so
                // equal consecutive blocks are the only repeats.
                if (n_run == 0 || (((vx ^ ox) | (vy ^ oy) | (vz ^ oz)) >> 3) != 0) {
                    const unsigned long long k = (unsigned long long)pack_key(vx >> 3, vy >> 3, vz >> 3);
                    run_key[n_run][t] = make_uint2((uint32_t)k, (uint32_t)(k >> 32));
                    ++n_run;
                }
                ox = vx;
                oy = vy;
                oz = vz;
#pragma unroll
                for (int q = 0; q < kChunk; ++q) n_of[q] += q == n_run - 1 ? 1 : 0;
            }
        }
#pragma unroll
        for (int q = 0; q < kChunk; ++q) {
            if (!__any_sync(0xffffffffu, q < n_run)) break;
            const uint2 k2 = q < n_run ? run_key[q][t] : make_uint2(0u, 0u);
            Resolved res{0, 0u};
            resolve_grouped<MODE>(v, q < n_run, (long long)((unsigned long long)k2.y << 32 | k2.x), res, hist, n_bins);
            if (res.bi < 0) drops += (uint32_t)n_of[q];
        }
        __syncwarp();  // the run columns are rewritten by the next chunk
    }
    return drops;
}

// Limits of the fast walk, in voxels. Coordinates below kReach: the floor is
// exact and block coordinates fit a key. Below kSureReach, rounding errors
// are small against a voxel, and beyond kSureDist from the camera the samples
// behind it are not occluded either: the occlusion shortcut needs both. Samples
// within kSpreadXY and kSpreadZ of the warp's first point share its table: as far
// as offsets of 11 and 10 bits reach, since pixels on both sides of a depth edge
// still share blocks (at 128, the walk of a mapped 640x480 room took 10 % longer;
// at 480, a band of 100 voxels 137 us instead of 84; shuffled clouds were the same
// to 2 %).
constexpr float kReach = 4194000.0f;  // 2^22 and rounding
constexpr float kSureReach = 32768.0f;
constexpr float kSureDist = 2.0f;
constexpr float kSpreadXY = 990.0f;
constexpr float kSpreadZ = 480.0f;
constexpr float kFloorMagic = 12582912.0f;  // 1.5 * 2^23
constexpr uint32_t kFloorBits = 0x4B400000u;  // its bits
constexpr uint32_t kNoOffset = 0xFFFFFFFFu;  // no sample; no block
constexpr uint32_t kBackXY = 1024u, kBackZ = 512u;  // voxels from the origin to its point's block
static_assert(kNoOffset == kNoVoxel, "a sample's column holds its offset, then its voxel");
static_assert(kSpreadXY + 16.0f < (float)kBackXY && kSpreadZ + 16.0f < (float)kBackZ, "offsets of 11 and 10 bits");

// Raw floor bits of the origin `back` voxels before the block at x.
__device__ __forceinline__ uint32_t origin_bits(float x, float inv_voxel, uint32_t back) {
    return (__float_as_uint(__fadd_rd(__fmul_rn(x, inv_voxel), kFloorMagic)) & ~7u) - back;
}
// A voxel's offset from an origin: x (11 bits), y << 11 (11 bits), z << 22 (10
// bits). An offset without the low three bits of its fields is its block's key
// within the warp.
__device__ __forceinline__ uint32_t pack_offset(uint32_t x, uint32_t y, uint32_t z) {
    return x + (y << 11) + (z << 22);
}
constexpr uint32_t kOffsetBlock = ~(7u | 7u << 11 | 7u << 22);
// The entry of a block (an offset's block bits) in the warp's table: about
// 8 x + 26 y - z of its coordinates, modulo 64, by one product. Found by a search
// over the warps of room scans (0.5 to 4 cm voxels, 160 to 1280 pixels a row)
// and of randomly tilted planes: two blocks of a warp share an entry in 15 % and
// 33 % of them; the coordinates modulo 4 did in 53 % and 35 %.
__device__ __forceinline__ uint32_t table_entry(uint32_t block) { return (block * 0x04019FFEu) >> 26; }
static_assert(kTableEntries == 64, "entries of 6 bits");
// The offset's voxel within its block, (lz * 8 + ly) * 8 + lx, in the nine
// high bits: one product brings the fields together (no two of its partial
// products meet).
__device__ __forceinline__ uint32_t voxel_high(uint32_t w) {
    return (w & (7u | 7u << 11 | 7u << 22)) * (1u << 23 | 1u << 15 | 1u << 7);
}
// The voxel of offset w in block bi (none where the block is absent).
__device__ __forceinline__ uint32_t voxel_index(int32_t bi, uint32_t w) {
    return bi < 0 ? kNoVoxel : __funnelshift_l(voxel_high(w), (uint32_t)bi, 9);
}

// The samples of a chunk that lie too far away for offsets, one by one: their
// columns hold the voxel within its block and, in the block's place, the number
// of the run of equal blocks.
__device__ __forceinline__ void odd_samples(const DevVolume& v, const Ray& r, int c0, int n_steps, uint32_t* vox,
                                            float* dsq) {
    int ox = 0, oy = 0, oz = 0, vx = 0, vy = 0, vz = 0;
    float d2 = 0.0f;
    bool ok = false;
    uint32_t run = 0u;
#pragma unroll 1
    for (int j = 0; j < n_steps; ++j) {
        // At an infinite distance the unit vector is zero (or not a number):
        // every sample is the first.
        if (j == 0 || r.dist < INFINITY) ok = band_sample_ray(v, r, c0 + j, vx, vy, vz, d2);
        if (ok) {
            if ((((vx ^ ox) | (vy ^ oy) | (vz ^ oz)) >> 3) != 0) ++run;
            ox = vx;
            oy = vy;
            oz = vz;
        }
        vox[j * kBandThreads] = ok ? pack_offset((uint32_t)(vx & 7) + (run << 3), vy & 7, vz & 7) : kNoOffset;
        dsq[j * kBandThreads] = d2;
    }
}

// Queue the runs of equal blocks among the samples left (bits of left; a
// straight ray leaves a block, a convex box, for good) in the warp's table, by
// their full keys, taken from the sample again: every lane's next run, while
// there is room. The samples' columns get their entry in the block's place.
// Returns the samples queued; queued: the entries in use. Called by the whole
// warp.
__device__ __forceinline__ uint32_t queue_runs(const DevVolume& v, const Ray& r, int c0, uint32_t left, uint32_t* vox,
                                               uint2* table, int& queued) {
    uint32_t open = left;
    queued = 0;
    for (;;) {
        const unsigned who = __ballot_sync(0xffffffffu, open != 0u);
        if (who == 0u || queued + __popc(who) > kTableEntries) break;
        if (open != 0u) {
            const int entry = queued + __popc(who & lanemask_lt());
            int j = __ffs(open) - 1;
            int vx, vy, vz;
            float d2;
            band_sample_ray(v, r, c0 + j, vx, vy, vz, d2);
            const unsigned long long key = (unsigned long long)pack_key(vx >> 3, vy >> 3, vz >> 3);
            table[entry] = make_uint2((uint32_t)key, (uint32_t)(key >> 32));
            const uint32_t block = vox[j * kBandThreads] & kOffsetBlock;
            for (; (open >> j) & 1u; ++j) {
                const uint32_t w = vox[j * kBandThreads];
                if ((w & kOffsetBlock) != block) break;
                vox[j * kBandThreads] = (w & ~kOffsetBlock) | (uint32_t)entry << 3;
                open &= ~(1u << j);
            }
        }
        queued += __popc(who);
    }
    return left & ~open;
}

// The samples of a chunk whose blocks the table did not settle (bits of left):
// their runs, queued in the table 64 at a time and probed like its entries, each
// by one lane. A second round of the table for them, and whole rounds for lanes
// apart from the first (the walk before this one), took 57 us where this takes
// 34 (292,000 shuffled points of a room, 2 cm voxels, all at the cap; grouping
// every lane's runs by matches across the warp: 55) and 113 against 95 for random
// directions up to 20 m.
template <int MODE, bool RECORDS>
__device__ __forceinline__ void resolve_runs(const DevVolume& v, const UpdateScratch& u, const Ray& r, int c0,
                                             uint32_t left, uint32_t* vox, uint2* table, bool counts_drops,
                                             uint32_t& drops) {
    const int lane = threadIdx.x & 31;
    do {
        __syncwarp();  // the table is rewritten
        int queued;
        uint32_t batch = queue_runs(v, r, c0, left, vox, table, queued);
        left &= ~batch;
        __syncwarp();
#pragma unroll 1
        for (int e = lane; e - lane < queued; e += 32) {
            const bool need = e < queued;
            const uint2 key = table[e];
            Resolved res{-1, 0u};
            bool rest = false;
            uint32_t seen = 0u;
            if (need) {
                res.slot = home_slot(v, key);
                seen = probe_settle<MODE>(v, probe_start<MODE>(v, res.slot), key, res);
                rest = res.bi == kUnsettled;
            }
            // Runs of several lanes may share a block.
            resolve_grouped<MODE>(v, rest, (long long)((unsigned long long)key.y << 32 | key.x), res, nullptr, 0);
            if (RECORDS) tag_touched<true>(v, u, res.bi >= 0 && (rest || seen != u.tag), res.bi, res.slot);
            if (need) table[e].y = (uint32_t)res.bi;
        }
        __syncwarp();
        for (; batch != 0u; batch &= batch - 1u) {
            const int j = __ffs(batch) - 1;
            const uint32_t w = vox[j * kBandThreads];
            const int32_t bi = (int32_t)table[(w >> 3) & (kTableEntries - 1)].y;
            if (counts_drops && bi < 0) ++drops;
            if (RECORDS) vox[j * kBandThreads] = voxel_index(bi, w);
        }
    } while (__any_sync(0xffffffffu, left != 0u));
}

// Walk point i (already loaded into px, py, pz; i >= a.n for lanes without a
// point) through its band. Called by every thread of the CTA,
// warp-synchronously.
//
// Where the 32 points of a warp are neighbouring pixels, a chunk of their bands
// lies in a few blocks (9 in the median 640x480 frame). Each sample writes its
// block's key into the warp's table in shared memory; the lanes then resolve the
// blocks found there, one each, all in one round trip: every distinct block of
// the warp is probed once, and no key is matched across lanes. Samples that find
// another block's key in their entry, and those of lanes apart from the warp's
// first, are left to resolve_runs. Nothing is called out of line: values that
// live across a call were spilled at every use (148 local loads a tile, a third
// of the walk's time).
//
// Samples round exactly as band_sample's: floor(x) is taken by adding
// 1.5 * 2^23 with rounding toward -infinity (exact for |x| < 2^22; the low
// bits are then the voxel coordinate), and (vf + 0.5) * size is the single
// fused rounding of vf * size + size / 2 (vf + 0.5 is exact). Within
// kSureReach and beyond kSureDist, a sample up to step trunc / voxel - 1
// (v.sure_step) cannot be occluded. Its voxel's centre lies within 0.87 voxels
// of it and rounding errors stay below 0.1 voxels, so in front of the camera
// sdf > -(s + 0.97) voxels. A sample behind the camera (s < 0, the point closer
// than |s| voxels) has sdf > 2 dist - (|s| + 0.97) voxels, and |s| is less than
// trunc / voxel + 1: above -trunc from a distance of 0.99 voxels on.
//
// FRAMES: the batch holds several frames; (cx, cy, cz) is the camera of
// point i's frame (otherwise the batch's one camera is used).
template <int MODE, bool RECORDS, int S, bool FRAMES = false>
__device__ __forceinline__ void band_point(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                                           int i, bool has, float px, float py, float pz,
                                           BandSmem& sm, uint32_t& drops, uint32_t& counted,
                                           unsigned long long* hist, int n_bins, float cx = 0.0f,
                                           float cy = 0.0f, float cz = 0.0f) {
    static_assert(!(FRAMES && S == kStoreF64), "the FP64 oracle integrates one frame per batch");
    const bool counts_drops = MODE != kLookupOnly && MODE != kAllocNoCas && MODE != kAllocCountingCas;
    if (!FRAMES) {
        cx = a.cam_x;
        cy = a.cam_y;
        cz = a.cam_z;
    }
    Ray r;
    const bool in_batch = i < a.n;
    const bool live = in_batch && has && ray_setup_cam(a.radius_sq, cx, cy, cz, px, py, pz, r);

    if constexpr (!has_fast_probe<MODE>()) {
        const uint32_t d = measure_point<MODE>(v, r, live, sm.run_key, hist, n_bins);
        if (counts_drops) drops += d;
        return;
    }

    const int lane = threadIdx.x & 31;
    uint2* const table = sm.table[threadIdx.x >> 5];
    const float half = __fmul_rn(0.5f, v.voxel_size);
    const float reach = v.inv_voxel * fmaxf(fmaxf(fabsf(px), fabsf(py)), fabsf(pz));
    const float far = reach + v.inv_voxel * fmaxf(fmaxf(fabsf(cx), fabsf(cy)), fabsf(cz));
    const float band = (float)v.steps + 2.0f;
    // A lane's samples are offsets from a block-aligned origin: the warp's, near
    // its first such point, where they may use the warp's table; its own, for
    // points too far from that one. Samples beyond kReach (and infinite ones) are
    // taken one by one.
    const bool fits = live && reach + band < kReach;
    const unsigned fit = __ballot_sync(0xffffffffu, fits);
    const int first = fit ? __ffs(fit) - 1 : 0;
    const float fx = __shfl_sync(0xffffffffu, px, first), fy = __shfl_sync(0xffffffffu, py, first),
                fz = __shfl_sync(0xffffffffu, pz, first);
    const bool tabled = fits && v.inv_voxel * fmaxf(fabsf(px - fx), fabsf(py - fy)) + band < kSpreadXY &&
                        v.inv_voxel * fabsf(pz - fz) + band < kSpreadZ;
    // Steps up to this one need no occlusion test.
    const bool sure = far < kSureReach && r.dist >= kSureDist * v.voxel_size;
    const int sure_step = __all_sync(0xffffffffu, sure || !fits) ? v.sure_step : INT_MIN;
    // The warp's origin as raw floor bits.
    const uint32_t ox = origin_bits(fx, v.inv_voxel, kBackXY), oy = origin_bits(fy, v.inv_voxel, kBackXY),
                   oz = origin_bits(fz, v.inv_voxel, kBackZ);
    uint32_t base = pack_offset(ox, oy, oz);
    uint32_t slot = (uint32_t)i;  // band slot (s = -steps, i)
    uint32_t* const vox = &sm.vox[0][threadIdx.x];  // voxel offset, then the voxel's index
    float* const dsq = &sm.dsq[0][threadIdx.x];

    for (int c0 = -v.steps; c0 <= v.steps; c0 += kChunk) {
        const int n_steps = min(kChunk, v.steps - c0 + 1);  // samples of this chunk
        table[lane].x = kNoOffset;
        table[lane + 32].x = kNoOffset;
        __syncwarp();
        if (fits && !tabled) {  // this lane's origin: by the chunk's first sample
            const float t = __fmul_rn((float)c0, v.voxel_size);
            base = pack_offset(origin_bits(__fadd_rn(px, __fmul_rn(r.ux, t)), v.inv_voxel, kBackXY),
                               origin_bits(__fadd_rn(py, __fmul_rn(r.uy, t)), v.inv_voxel, kBackXY),
                               origin_bits(__fadd_rn(pz, __fmul_rn(r.uz, t)), v.inv_voxel, kBackZ));
        }
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
            if (j >= n_steps) break;
            const float t = __fmul_rn((float)(c0 + j), v.voxel_size);
            const float yx = __fadd_rd(__fmul_rn(__fadd_rn(px, __fmul_rn(r.ux, t)), v.inv_voxel), kFloorMagic);
            const float yy = __fadd_rd(__fmul_rn(__fadd_rn(py, __fmul_rn(r.uy, t)), v.inv_voxel), kFloorMagic);
            const float yz = __fadd_rd(__fmul_rn(__fadd_rn(pz, __fmul_rn(r.uz, t)), v.inv_voxel), kFloorMagic);
            const float ex = __fsub_rn(__fmaf_rn(__fsub_rn(yx, kFloorMagic), v.voxel_size, half), cx);
            const float ey = __fsub_rn(__fmaf_rn(__fsub_rn(yy, kFloorMagic), v.voxel_size, half), cy);
            const float ez = __fsub_rn(__fmaf_rn(__fsub_rn(yz, kFloorMagic), v.voxel_size, half), cz);
            const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
            const uint32_t w = pack_offset(__float_as_uint(yx), __float_as_uint(yy), __float_as_uint(yz)) - base;
            bool hidden = false;
            if (c0 + j > sure_step) hidden = __fsub_rn(r.dist, __fsqrt_rn(d2)) < -v.trunc;
            vox[j * kBandThreads] = fits && !hidden ? w : kNoOffset;
            dsq[j * kBandThreads] = d2;
            if (tabled && !hidden) table[table_entry(w & kOffsetBlock)].x = w & kOffsetBlock;
        }
        if (live && !fits) odd_samples(v, r, c0, n_steps, vox, dsq);
        __syncwarp();

        // The blocks in the table, packed so that lane l takes the l-th (and the
        // 32nd after it): their entries are listed in the index words. Taking
        // entries l and l + 32 as they are makes two round trips for most warps
        // (107.4 us on four frames against 104.4).
        const bool in0 = table[lane].x != kNoOffset, in1 = table[lane + 32].x != kNoOffset;
        const unsigned b0 = __ballot_sync(0xffffffffu, in0), b1 = __ballot_sync(0xffffffffu, in1);
        if (in0) table[__popc(b0 & lanemask_lt())].y = (uint32_t)lane;
        if (in1) table[__popc(b0) + __popc(b1 & lanemask_lt())].y = (uint32_t)lane + 32u;
        __syncwarp();
        const int n_blocks = __popc(b0) + __popc(b1);
        uint32_t at = table[lane].y;
        const uint32_t at_next = table[lane + 32].y;
        __syncwarp();
        // A slot's 16 bytes hold the key, the index and the touch tag.
#pragma unroll 1
        for (int k = lane; k - lane < n_blocks; k += 32, at = at_next) {
            const bool need = k < n_blocks;
            const uint32_t b = need ? table[at].x : 0u;
            const uint32_t kx = (uint32_t)((int)(ox - kFloorBits) >> 3) + (uint32_t)kCoordBias + ((b >> 3) & 255u);
            const uint32_t ky = (uint32_t)((int)(oy - kFloorBits) >> 3) + (uint32_t)kCoordBias + ((b >> 14) & 255u);
            const uint32_t kz = (uint32_t)((int)(oz - kFloorBits) >> 3) + (uint32_t)kCoordBias + (b >> 25);
            const uint2 key = make_uint2(kz | ky << kCoordBits, ky >> (32 - kCoordBits) | kx << (2 * kCoordBits - 32));
            Resolved res{-1, home_slot(v, key)};
            bool rest = false;
            uint32_t seen = 0u;
            if (need) {
                seen = probe_settle<MODE>(v, probe_start<MODE>(v, res.slot), key, res);
                rest = res.bi == kUnsettled;
            }
            // The lanes' keys are distinct: each probes for itself.
            if (rest) res = resolve<MODE>(v, (long long)((unsigned long long)key.y << 32 | key.x), nullptr, 0);
            __syncwarp();
            if (RECORDS) tag_touched<false>(v, u, res.bi >= 0 && (rest || seen != u.tag), res.bi, res.slot);
            if (need) table[at].y = (uint32_t)res.bi;
        }
        __syncwarp();
        uint32_t left = 0u;  // bit j: sample j's block is not in the table
        const uint32_t apart = tabled ? 0u : 1u;  // matches no key
#pragma unroll
        for (int j = 0; j < kChunk; ++j) {
            const uint32_t w = j < n_steps ? vox[j * kBandThreads] : kNoOffset;
            const uint2 e = table[table_entry(w & kOffsetBlock)];
            if (e.x == ((w & kOffsetBlock) | apart)) {
                if (counts_drops && (int)e.y < 0) ++drops;
                vox[j * kBandThreads] = voxel_index((int32_t)e.y, w);
            } else if (w != kNoOffset) {
                left |= 1u << j;
            }
        }
        if (__any_sync(0xffffffffu, left != 0u))
            resolve_runs<MODE, RECORDS>(v, u, r, c0, left, vox, table, counts_drops, drops);
        if (RECORDS)
            count_samples<S, kChunk>(v, u, in_batch, (uint32_t)a.n, r.dist, vox, dsq, n_steps, slot, counted, [&](int j) {
                int vx, vy, vz;
                float d2;
                band_sample_ray(v, r, c0 + j, vx, vy, vz, d2);
                return oracle_fix(v, a, r, vx, vy, vz);
            });
        __syncwarp();  // the table is rewritten by the next chunk
    }
}

// The camera of every point of a batch with one camera: nothing to track.
struct OneCamera {
    float cx = 0.0f, cy = 0.0f, cz = 0.0f;
    __device__ __forceinline__ void at(int) {}
};

// The camera of each point of a batch of several frames. A thread's points
// only move forward (tile += grid size), so its frame does too: one
// comparison per tile, and a table read only where the frame changes.
struct FrameCursor {
    const FrameTable& table;  // kernel parameter
    int32_t f, next;
    float cx, cy, cz;
    __device__ __forceinline__ explicit FrameCursor(const FrameTable& t) : table(t), f(0) { load(); }
    __device__ __forceinline__ void load() {
        cx = table.f[f].x;
        cy = table.f[f].y;
        cz = table.f[f].z;
        next = f + 1 < table.n ? table.f[f + 1].begin : INT_MAX;
    }
    __device__ __forceinline__ void at(int i) {
        while (i >= next) {  // the last frame's bound is INT_MAX
            ++f;
            load();
        }
    }
};

// Where a batch's points come from: xyz positions or one depth image.
template <int SOURCE>
struct BatchPoints {
    const BatchArgs& a;
    __device__ __forceinline__ bool load(int i, float& px, float& py, float& pz) const {
        return load_point<SOURCE>(a, i, px, py, pz);
    }
};

// Several depth images of npix pixels back to back: pixel i belongs to image
// i / npix, unprojected with that image's pose (staged in shared memory).
struct DepthFramesPoints {
    const BatchArgs& a;
    const FramePose* pose;
    int32_t npix;
    __device__ __forceinline__ bool load(int i, float& px, float& py, float& pz) const {
        const int f = i / npix;
        return unproject_pixel(a.depth, pose[f].R, pose[f].t, i, i - f * npix, px, py, pz);
    }
};

// A persistent CTA's share of a batch: tiles of 128 points, strided by the
// grid, then the CTA's drop and record counts.
template <int MODE, bool RECORDS, int S, bool FRAMES, typename Points, typename Camera>
__device__ __forceinline__ void band_tiles(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                                           unsigned long long* hist, int n_bins, const Points pts,
                                           Camera cam) {
    __shared__ BandSmem sm;
    const int t = threadIdx.x;
    const int lane = t & 31;
    const bool counts_drops = MODE != kLookupOnly && MODE != kAllocNoCas && MODE != kAllocCountingCas;
    const int n_tiles = (a.n + kBandThreads - 1) / kBandThreads;
    uint32_t drops = 0, counted = 0;
    __shared__ unsigned s_drops, s_counted;
    if (t == 0) {
        s_drops = 0u;
        s_counted = 0u;
    }
    __syncthreads();
    launch_dependents();  // the finish pass may be scheduled as CTAs retire

    // The point of the next tile is loaded one tile ahead.
    float nx = 0.0f, ny = 0.0f, nz = 0.0f;
    bool nhas = false;
    {
        const int i0 = blockIdx.x * kBandThreads + t;
        if (blockIdx.x < n_tiles && i0 < a.n) nhas = pts.load(i0, nx, ny, nz);
    }
    for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const int i = tile * kBandThreads + t;
        const float px = nx, py = ny, pz = nz;
        const bool has = nhas;
        const int inext = i + gridDim.x * kBandThreads;
        nhas = false;
        if (inext < a.n) nhas = pts.load(inext, nx, ny, nz);
        cam.at(i);
        band_point<MODE, RECORDS, S, FRAMES>(v, a, u, i, has, px, py, pz, sm, drops, counted,
                                                         hist, n_bins, cam.cx, cam.cy, cam.cz);
    }

    // Counters: one global atomic per CTA (per-warp atomics on one line serialise).
    const unsigned wd = counts_drops ? __reduce_add_sync(0xffffffffu, drops) : 0u;
    const unsigned wc = RECORDS ? __reduce_add_sync(0xffffffffu, counted) : 0u;
    if (lane == 0 && wd) atomicAdd(&s_drops, wd);
    if (lane == 0 && wc) atomicAdd(&s_counted, wc);
    __syncthreads();
    if (t == 0 && s_drops) atomicAdd(v.drop_count, (unsigned long long)s_drops);
    if (t == 0 && s_counted) atomicAdd(&u.ctl->n_records, (int)s_counted);
}

// Every walk is launched with programmatic stream serialisation: its CTAs take
// their places while the previous call's last pass drains, and wait here for
// what that call wrote.
template <int MODE, bool RECORDS, int S, bool DEPTH = false>
__global__ void __launch_bounds__(kBandThreads, kBandMinBlocks)
band_kernel(DevVolume v, BatchArgs a, UpdateScratch u, unsigned long long* hist, int n_bins) {
    grid_dependency_wait();
    band_tiles<MODE, RECORDS, S, false>(v, a, u, hist, n_bins, BatchPoints<DEPTH ? 1 : 0>{a}, OneCamera{});
}

// Integrate (allocate + count-and-sum) of a batch of several frames: the
// single-frame walk with each point's camera taken from the frame table.
template <int S>
__global__ void __launch_bounds__(kBandThreads, kBandFramesMinBlocks)
band_frames_kernel(DevVolume v, BatchArgs a, UpdateScratch u, const __grid_constant__ FrameTable frames) {
    grid_dependency_wait();
    band_tiles<kAllocInsert, true, S, true>(v, a, u, nullptr, 0, BatchPoints<0>{a}, FrameCursor(frames));
}

// The same for several depth images of equal size: each CTA stages the
// images' poses in shared memory first.
template <int S>
__global__ void __launch_bounds__(kBandThreads, kBandDepthMinBlocks)
band_depth_frames_kernel(DevVolume v, BatchArgs a, UpdateScratch u, const __grid_constant__ FrameTable frames,
                         const __grid_constant__ PoseTable poses) {
    __shared__ FramePose s_pose[kMaxDepthFrames];
    constexpr int kWords = (int)(sizeof(FramePose) / sizeof(double));
    for (int k = threadIdx.x; k < poses.n * kWords; k += blockDim.x)
        reinterpret_cast<double*>(s_pose)[k] = reinterpret_cast<const double*>(poses.p)[k];
    grid_dependency_wait();
    __syncthreads();
    band_tiles<kAllocInsert, true, S, true>(v, a, u, nullptr, 0, DepthFramesPoints{a, s_pose, a.n / poses.n},
                                            FrameCursor(frames));
}

// ---- batched steps -----------------------------------------------------

// Copy a POD descriptor into shared memory with the whole CTA.
template <typename T>
__device__ __forceinline__ void cta_copy(T* dst, const T* src) {
    static_assert(sizeof(T) % 4 == 0, "descriptor copies go by words");
    const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d = reinterpret_cast<uint32_t*>(dst);
    for (int k = threadIdx.x; k < (int)(sizeof(T) / 4); k += blockDim.x) d[k] = s[k];
}

// Scene of global work item `item` given the per-scene item prefix `begin`
// (n + 1 entries, begin[0] = 0): the last scene whose range starts at or
// before it.
__device__ __forceinline__ int scene_of(const int* begin, int n, int item) {
    int lo = 0, hi = n;  // begin[lo] <= item < begin[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (begin[mid] <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Allocate + count-and-sum walk of every scene of a step. Work items are
// runs of tiles_per_item consecutive 128-point tiles of one scene, handed
// out by an atomic queue to a persistent grid; the CTA keeps the current
// item's scene descriptor in shared memory and flushes its per-scene
// counters whenever it moves to another scene.
template <int S>
__global__ void __launch_bounds__(kBandThreads, kBandFramesMinBlocks)
band_multi_kernel(StepWork w) {
    __shared__ BandSmem sm;
    __shared__ SceneWork sw;
    __shared__ int s_begin[kMaxBatchScenes + 1];
    __shared__ int s_item;
    __shared__ unsigned s_drops, s_counted;
    const int t = threadIdx.x, lane = t & 31;
    launch_dependents();
    grid_dependency_wait();
    // Item prefix: one thread per scene, then a scan (n <= 64 <= blockDim.x).
    if (t < w.n_scenes)
        s_begin[t + 1] = (w.scenes[t].band_tiles + w.band_tiles_per_item - 1) / w.band_tiles_per_item;
    if (t == 0) {
        s_begin[0] = 0;
        s_drops = 0u;
        s_counted = 0u;
    }
    __syncthreads();
    if (t == 0)
        for (int k = 1; k <= w.n_scenes; ++k) s_begin[k] += s_begin[k - 1];
    __syncthreads();
    const int total = s_begin[w.n_scenes];
    int cur = -1;
    uint32_t drops = 0u, counted = 0u;
    for (;;) {
        if (t == 0) s_item = (int)atomicAdd(&w.queues[kQBand], 1u);
        __syncthreads();
        const int item = s_item;
        const bool done = item >= total;  // also on a CTA's first pull when items are few
        const int sc = done ? -1 : scene_of(s_begin, w.n_scenes, item);
        if (sc != cur || done) {
            // Flush the counters of the scene left behind, then load the next one.
            const unsigned wd = __reduce_add_sync(0xffffffffu, drops);
            const unsigned wc = __reduce_add_sync(0xffffffffu, counted);
            if (lane == 0 && wd) atomicAdd(&s_drops, wd);
            if (lane == 0 && wc) atomicAdd(&s_counted, wc);
            __syncthreads();
            if (t == 0 && cur >= 0) {
                if (s_drops) atomicAdd(sw.v.drop_count, (unsigned long long)s_drops);
                if (s_counted) atomicAdd(&sw.u.ctl->n_records, (int)s_counted);
            }
            __syncthreads();
            if (t == 0) {
                s_drops = 0u;
                s_counted = 0u;
            }
            drops = counted = 0u;
            if (done) break;
            cta_copy(&sw, &w.scenes[sc]);
            __syncthreads();
            cur = sc;
        }
        const int first = (item - s_begin[sc]) * w.band_tiles_per_item;
        const int last = min(first + w.band_tiles_per_item, sw.band_tiles);
        for (int tile = first; tile < last; ++tile) {
            const int i = tile * kBandThreads + t;
            float px = 0.0f, py = 0.0f, pz = 0.0f;
            const bool has = i < sw.a.n && load_point(sw.a, i, px, py, pz);
            band_point<kAllocInsert, true, S>(sw.v, sw.a, sw.u, i, has, px, py, pz, sm, drops,
                                                    counted, nullptr, 0);
        }
        __syncthreads();  // s_item and the descriptor are rewritten next
    }
}

template <int MODE, bool RECORDS, int S = kStoreF32, bool DEPTH = false>
cudaError_t launch(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                   unsigned long long* hist, int n_bins, int sm_count, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    // Persistent grid: as many CTAs as are resident at once (queried once
    // per instantiation), striding over the point tiles.
    static int per_sm = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, band_kernel<MODE, RECORDS, S, DEPTH>,
                                                          kBandThreads, 0) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
    });
    const int tiles = (a.n + kBandThreads - 1) / kBandThreads;
    const int grid = std::min(tiles, per_sm * sm_count);
    return launch_after(band_kernel<MODE, RECORDS, S, DEPTH>, grid, kBandThreads, s, v, a, u, hist, n_bins);
}

}  // namespace

cudaError_t launch_allocate(const DevVolume& v, const BatchArgs& a, int mode,
                            unsigned long long* hist, int n_bins, int sm_count, cudaStream_t s) {
    const UpdateScratch none{};
    switch (mode) {
        case kAllocInsert: return launch<kAllocInsert, false>(v, a, none, nullptr, 0, sm_count, s);
        case kAllocCountingCas:
            return launch<kAllocCountingCas, false>(v, a, none, nullptr, 0, sm_count, s);
        case kAllocNoCas: return launch<kAllocNoCas, false>(v, a, none, nullptr, 0, sm_count, s);
        case kAllocProbeHist:
            return launch<kAllocProbeHist, false>(v, a, none, hist, n_bins, sm_count, s);
        case kAllocSlotIndex: return launch<kAllocSlotIndex, false>(v, a, none, nullptr, 0, sm_count, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_band_records(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                                bool insert, int sm_count, cudaStream_t s) {
    if (a.depth.depth != nullptr) {  // integrate from a depth image (allocates)
        if (!insert) return cudaErrorInvalidValue;
        switch (v.storage) {
            case kStoreF16U16:
                return launch<kAllocInsert, true, kStoreF16U16, true>(v, a, u, nullptr, 0, sm_count, s);
            case kStoreF64:
                return launch<kAllocInsert, true, kStoreF64, true>(v, a, u, nullptr, 0, sm_count, s);
            default:
                return launch<kAllocInsert, true, kStoreF32, true>(v, a, u, nullptr, 0, sm_count, s);
        }
    }
    switch (v.storage) {
        case kStoreF16U16:
            return insert ? launch<kAllocInsert, true, kStoreF16U16>(v, a, u, nullptr, 0, sm_count, s)
                          : launch<kLookupOnly, true, kStoreF16U16>(v, a, u, nullptr, 0, sm_count, s);
        case kStoreF64:
            return insert ? launch<kAllocInsert, true, kStoreF64>(v, a, u, nullptr, 0, sm_count, s)
                          : launch<kLookupOnly, true, kStoreF64>(v, a, u, nullptr, 0, sm_count, s);
        default:
            return insert ? launch<kAllocInsert, true>(v, a, u, nullptr, 0, sm_count, s)
                          : launch<kLookupOnly, true>(v, a, u, nullptr, 0, sm_count, s);
    }
}

namespace {
template <int S>
cudaError_t launch_band_frames_t(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                                 const FrameTable& frames, int sm_count, cudaStream_t s) {
    static int per_sm = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, band_frames_kernel<S>, kBandThreads, 0) !=
                cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
    });
    const int tiles = (a.n + kBandThreads - 1) / kBandThreads;
    const int grid = std::min(tiles, per_sm * sm_count);
    return launch_after(band_frames_kernel<S>, grid, kBandThreads, s, v, a, u, frames);
}
template <int S>
cudaError_t launch_band_depth_frames_t(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                                       const FrameTable& frames, const PoseTable& poses, int sm_count,
                                       cudaStream_t s) {
    static int per_sm = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, band_depth_frames_kernel<S>, kBandThreads,
                                                          0) != cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
    });
    const int tiles = (a.n + kBandThreads - 1) / kBandThreads;
    const int grid = std::min(tiles, per_sm * sm_count);
    return launch_after(band_depth_frames_kernel<S>, grid, kBandThreads, s, v, a, u, frames, poses);
}
}  // namespace

cudaError_t launch_band_depth_frames(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                                     const FrameTable& frames, const PoseTable& poses, int sm_count, cudaStream_t s) {
    if (a.n <= 0 || poses.n < 1 || poses.n > kMaxDepthFrames || a.n % poses.n != 0) return cudaErrorInvalidValue;
    switch (v.storage) {
        case kStoreF32: return launch_band_depth_frames_t<kStoreF32>(v, a, u, frames, poses, sm_count, s);
        case kStoreF16U16: return launch_band_depth_frames_t<kStoreF16U16>(v, a, u, frames, poses, sm_count, s);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_band_frames(const DevVolume& v, const BatchArgs& a, const UpdateScratch& u,
                               const FrameTable& frames, int sm_count, cudaStream_t s) {
    if (a.n <= 0) return cudaSuccess;
    switch (v.storage) {
        case kStoreF32: return launch_band_frames_t<kStoreF32>(v, a, u, frames, sm_count, s);
        case kStoreF16U16: return launch_band_frames_t<kStoreF16U16>(v, a, u, frames, sm_count, s);
        default: return cudaErrorInvalidValue;  // the FP64 oracle integrates one frame per batch
    }
}

namespace {
template <int S>
cudaError_t launch_band_multi_t(const StepWork& w, int sm_count, cudaStream_t s) {
    static int per_sm = 0;
    static std::once_flag once;
    std::call_once(once, [] {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, band_multi_kernel<S>, kBandThreads, 0) !=
                cudaSuccess ||
            per_sm < 1)
            per_sm = 1;
    });
    return launch_after(band_multi_kernel<S>, per_sm * sm_count, kBandThreads, s, w);
}
}  // namespace

cudaError_t launch_band_multi(const StepWork& w, int storage, int sm_count, cudaStream_t s) {
    switch (storage) {
        case kStoreF16U16: return launch_band_multi_t<kStoreF16U16>(w, sm_count, s);
        case kStoreF64: return launch_band_multi_t<kStoreF64>(w, sm_count, s);
        default: return launch_band_multi_t<kStoreF32>(w, sm_count, s);
    }
}

}  // namespace osn_b200
