// SPDX-License-Identifier: MIT
// The master's partition and bubble partition of one world over a park's rows, as one sequential program a world
// (exact_ballpark/space.py's SpaceBallpark on the master, the layer exact_ballpark/vec_space.py's VecSpace runs over
// a batched park): the partition's boxes, made on demand with their parents and released when empty, BoxAllocator's
// kept count and the reads of a released box (Partition's GetBox, CheckBox and the allocator, space.py:596-676); each
// ball's filing (Ball::InsertInBoxes and DeleteFromBoxes, space.py:683-818); the top boxes' bubbles, a neighbour's or
// a new id (Ballpark::InsertInBoxes, NearbyBubbles, Traverse), the bubble dictionaries (+1, 0, -1 in insertion
// order), the interactive and keep-alive sets (AddToBubble), InitializeBubbles, CopyBubbles, InDeadBubble
// (space.py:896-1056); AddBall's filing, the setters' re-filings and RemoveBall (space.py:1097-1319); the tick's
// dead-bubble flags and its re-filings (a warp's drop-out, the commits of the balls that moved).
//
// Layout: W worlds of N slots, in one of two arrangements (EbbSpaceState.pitch). Interleaved (pitch 0): every
// per-slot array is [N][W] and every per-entry array [cap][W] (world w's entry e at e W + w), so that the threads of
// a warp, one world each, touch consecutive words. World-major (pitch > 0): world w's copy of every array starts
// w pitch bytes past world 0's and holds its entries consecutively, so that a warp running one world reads its
// slots in one transaction and the world's state shares cache lines. A world's boxes live in a
// table of `boxes` entries (level -1 for a free entry, the free ones on a stack), found through a hash index of
// 2 `boxes` slots (linear probing, deletion by moving the run back). Exactness: the filing's double
// arithmetic through ebb_arith.cuh (correctly rounded single operations), compiled with -fmad=false.
#pragma once

#include <cstdint>

#include "../../include/ebb.h"
#include "ebb_arith.cuh"
#include "ebb_rand.cuh"   // LGPL-2.1-or-later: the C library's rand(), a shuffled sensor's draw

namespace ebb {
namespace space {

// The counting build's tally of CheckSensor's paths (EBB_COUNT_OPS, a measurement of the algorithm as it runs): the
// checks, those whose two re-filings were skipped (sensor_fast), and of those the ones whose filing did not change
#ifdef EBB_COUNT_OPS
#ifdef __CUDACC__
static __device__ unsigned long long sensor_paths[3];
#endif
#ifdef __CUDA_ARCH__
#define EBB_SENSOR_PATH(k)                                        \
    do {                                                          \
        if (lane <= 0) atomicAdd(&::ebb::space::sensor_paths[k], 1ull); \
    } while (0)
#else
#define EBB_SENSOR_PATH(k) ((void)0)
#endif
#else
#define EBB_SENSOR_PATH(k) ((void)0)
#endif

constexpr int NUM_LEVELS = 8;
constexpr int64_t BOX_KEEP = 256;                          // BoxAllocator's kept boxes
constexpr int64_t F_EDGE = EBB_SPACE_FLAG_EDGE, F_BOXES = EBB_SPACE_FLAG_BOXES, F_DICTS = EBB_SPACE_FLAG_DICTS,
                  F_ENTRIES = EBB_SPACE_FLAG_ENTRIES, F_BAD_OP = EBB_SPACE_FLAG_BAD_OP,
                  F_SETS = EBB_SPACE_FLAG_SETS, F_UNDEFINED = EBB_SPACE_FLAG_UNDEFINED,
                  F_EVENTS = EBB_SPACE_FLAG_EVENTS, F_PROXIMITY = EBB_SPACE_FLAG_PROXIMITY,
                  F_SENSOR_LIST = EBB_SPACE_FLAG_SENSOR_LIST, F_HUGE = EBB_SPACE_FLAG_HUGE;
constexpr int64_t GOTO = 0, FOLLOW = 1, WARP = 3, ORBIT = 4;
constexpr double TRACKING_MIN = 0.00001;                   // Ball.cpp:598's least tracking range
constexpr double RAND_MAX_D = 2147483647.0;                // floatrand's RAND_MAX (Ball.cpp:19)
// GetNearbyBalls' walk as a sort key (the reference's per-pair statement of the walk, vec_collide.py:825): one digit
// base 65 a level below the sensing ball's (64 children a box, then "past the candidate's level")
constexpr int64_t CODE_BASE = 65;
constexpr int64_t NOT_A_CANDIDATE = int64_t(1) << 62;
// The bucket counts of a std::unordered_map<int64_t, ...> under libstdc++'s prime rehash policy (max load factor 1)
// as it grows from its first insertion (13 buckets, room asked for 11 keys) past its bucket count each time: the
// first entry of the library's prime list at or above twice the old count. A map of at most 256 keys reaches 257.
EBB_HD constexpr int32_t umap_next_buckets(int32_t b) {
    return b <= 1 ? 13 : b == 13 ? 29 : b == 29 ? 59 : b == 59 ? 127 : b == 127 ? 257 : -1;
}

// a box's width at level i (Partition.h's constants: 2^16 grid units of 480 m a quarter at the top)
// The widths are powers of two times 480 m, so each value below is exact; the reciprocal is the correctly rounded
// 1 / width and the half-span 0.5 width 2^(2 level + 23) is exact, all folded at compile time to the values the
// formulas give at run time (level_width: 2^16 x 480 x 0.25 / 4^i; key_for's 1 / width and 0.5 width grid).
constexpr double level_width_c(int i) { return 65536.0 * 480.0 * 0.25 / (double)(int64_t(1) << (2 * i)); }
constexpr double level_inv_c(int i) { return 1.0 / level_width_c(i); }
constexpr double level_half_c(int i) {
    return 0.5 * level_width_c(i) * (double)(int64_t(1) << (2 * i - 2 * NUM_LEVELS + 39));
}
#define EBB_LEVEL_TABLE(f, i)                                                                                     \
    ((i) == 0 ? f(0) : (i) == 1 ? f(1) : (i) == 2 ? f(2) : (i) == 3 ? f(3) : (i) == 4 ? f(4) : (i) == 5 ? f(5)   \
     : (i) == 6 ? f(6) : f(7))
EBB_HD double level_width(int i) { return EBB_LEVEL_TABLE(level_width_c, i); }
EBB_HD double level_inv(int i) { return EBB_LEVEL_TABLE(level_inv_c, i); }
EBB_HD double level_half(int i) { return EBB_LEVEL_TABLE(level_half_c, i); }
EBB_HD int64_t level_grid(int i) { return int64_t(1) << (2 * i - 2 * NUM_LEVELS + 39); }
EBB_HD int64_t clamp_key(int64_t i, int64_t n) { return i < 0 ? int64_t(0) : (i >= n ? n - 1 : i); }

// the filing level of an inflated radius: the deepest level whose width is at least three radii
EBB_HD int level_for(double radius) {
    int level = 0;
    for (int i = 0; i < NUM_LEVELS; ++i) {
        if (dmul(3.0, radius) > level_width(i)) break;
        level = i;
    }
    return level;
}

// A sensor of a warp's batch as the scan over the slots reads it (World::scan_batch): its inflated filing's key ranges in
// the deepest level's units, its position, bubble, range and radius; `how`: bit 0 scanned, bit 1 fixed balls left out,
// bit 2 only interactive ones, its slot from bit 8
struct SensorRow {
    int64_t lo[3], hi[3];
    double x[3];
    int64_t bub;
    float range, radius;
    int32_t how, pad;
};

// A warp's scratch when a warp runs a world (EbbSpaceState.lanes = 32): the candidates' walk keys and ids by slot, and
// their slots in the walk's order; or the rows of the batch of sensors whose candidates are being found
struct Coop {
    union {
        struct {
            int64_t key[EBB_SPACE_MAX_SLOTS];
            int64_t id[EBB_SPACE_MAX_SLOTS];
            uint8_t out[EBB_SPACE_MAX_SLOTS];
        };
        SensorRow row[32];
    };
};

// One world's program. A thread runs it alone (lane -1), or the 32 lanes of a warp run it together (lane 0 .. 31):
// every lane then takes every step on the same data, so they stay converged and write the same values (one
// transaction a load or store), and GetNearbyBalls' scan and sort are split over the lanes (nearby_warp).
// WM: the world-major arrangement (the state's pitch > 0), else the interleaved one. COOP: a warp runs the world
// (the lanes' paths compiled in, the single thread's left out), else a thread. (WARP is the flight mode.)
template <bool WM, bool COOP = false>
struct World {
    const EbbFlightState* p;
    const EbbSpaceState* s;
    int64_t w, W, N, B;
    int lane = -1;
    Coop* sh = nullptr;
    static constexpr bool world_major = WM;
    // the slots whose filing this operation made from their current position, velocity and radius (the tick's
    // re-filings and a sensor's re-filing back): CheckSensor's fast path then knows the ball comes back to it
    uint64_t fresh[2] = {0, 0};
    int occupied = EBB_SPACE_MAX_SLOTS;                    // one past the last slot in the park (AFTER_EVOLVE's count)
    EBB_HD bool is_fresh(int64_t j) const { return (fresh[j >> 6] >> (j & 63)) & 1; }
    EBB_HD void set_fresh(int64_t j, bool on) {
        if (on)
            fresh[j >> 6] |= uint64_t(1) << (j & 63);
        else
            fresh[j >> 6] &= ~(uint64_t(1) << (j & 63));
    }

    // ---- accessors: entry e of a per-world array ([cap][W], or world w's run of cap entries), component c of a
    // [3][cap] one ----
    template <class T>
    EBB_HD T& at(T* a, int64_t e) const {
        if constexpr (WM)
            return ((T*)((const char*)a + w * s->pitch))[e];
        else
            return a[e * W + w];
    }
    EBB_HD int64_t step() const { return WM ? 1 : W; }     // the distance of consecutive entries, in elements
    EBB_HD int64_t& I(int64_t* a, int64_t e) const { return at(a, e); }
    EBB_HD int64_t& I3(int64_t* a, int64_t c, int64_t e, int64_t cap) const { return at(a, c * cap + e); }
    EBB_HD uint8_t& U(uint8_t* a, int64_t e) const { return at(a, e); }
    EBB_HD int64_t& one(int64_t* a) const { return at(a, 0); }
    // the box table's per-entry fields: interleaved [cap][W] arrays, or (world-major) records of BOX_RECORD words an
    // entry, each field's pointer naming it in world 0's entry 0, so that an entry's fields share a cache line
    EBB_HD int64_t& BX(int64_t* a, int64_t e) const {
        if constexpr (WM)
            return ((int64_t*)((const char*)a + w * s->pitch))[e * EBB_SPACE_BOX_RECORD];
        else
            return a[e * W + w];
    }
    EBB_HD int64_t& BK(int64_t c, int64_t e) const {
        if constexpr (WM)
            return ((int64_t*)((const char*)s->box_key + w * s->pitch))[e * EBB_SPACE_BOX_RECORD + c];
        else
            return s->box_key[(c * B + e) * W + w];
    }
    EBB_HD void flag(int64_t f) const { one(s->flags) |= f; }

    // ---- the park's row of a slot ----
    EBB_HD int64_t row(int64_t j) const { return at(s->rows, j); }
    EBB_HD double pos(int64_t j, int c) const { return p->pos[c * p->n + row(j)]; }
    EBB_HD double vel(int64_t j, int c) const { return p->vel[c * p->n + row(j)]; }
    EBB_HD int64_t id(int64_t j) const { return p->ids[row(j)]; }
    EBB_HD bool interactive(int64_t j) const { return p->interactive[row(j)] != 0; }

    // ---- the box table and its index (linear probing over 2 B slots, each entry + 1, 0 for an empty slot) ----
    EBB_HD int64_t home(int level, int64_t kx, int64_t ky, int64_t kz) const {
        uint64_t h = (uint64_t)kx * 0x9E3779B97F4A7C15ull;
        h ^= (uint64_t)ky * 0xC2B2AE3D27D4EB4Full + (h << 6) + (h >> 2);
        h ^= (uint64_t)kz * 0x165667B19E3779F9ull + (h << 6) + (h >> 2);
        h ^= (uint64_t)level * 0x27D4EB2F165667C5ull;
        h ^= h >> 29;
        // the slot: the high word of h x 2B (a multiply in place of a 64-bit remainder: the same spread over [0, 2B))
#ifdef __CUDA_ARCH__
        return (int64_t)__umul64hi(h, (uint64_t)(2 * B));
#else
        return (int64_t)(((unsigned __int128)h * (uint64_t)(2 * B)) >> 64);
#endif
    }
    EBB_HD bool is_box(int64_t e, int level, int64_t kx, int64_t ky, int64_t kz) const {
        return BX(s->box_level, e) == level && BK(0, e) == kx && BK(1, e) == ky &&
               BK(2, e) == kz;
    }
    EBB_HD int64_t box_find(int level, int64_t kx, int64_t ky, int64_t kz) const {
        const int64_t H = 2 * B;
        int64_t i = home(level, kx, ky, kz);
        for (int64_t probe = 0; probe < H; ++probe) {
            const int64_t v = I(s->box_hash, i);
            if (v == 0) return -1;
            if (is_box(v - 1, level, kx, ky, kz)) return v - 1;
            i = i + 1 == H ? 0 : i + 1;
        }
        return -1;
    }
    // (each entry keeps its home slot and the slot it sits in, so that its removal starts there without a probe)
    EBB_HD void hash_insert(int64_t e) {
        const int64_t H = 2 * B;
        int64_t i = home((int)BX(s->box_level, e), BK(0, e), BK(1, e),
                         BK(2, e));
        BX(s->box_home, e) = i;
        for (int64_t probe = 0; probe < H; ++probe) {
            if (I(s->box_hash, i) == 0) {
                I(s->box_hash, i) = e + 1;
                BX(s->box_slot, e) = i;
                return;
            }
            i = i + 1 == H ? 0 : i + 1;
        }
        flag(F_BOXES);                                     // (never: at most B entries in 2 B slots)
    }
    // the entry leaves the index; the entries after it in its run move back so that every probe still finds them
    EBB_HD void hash_erase(int64_t e) {
        const int64_t H = 2 * B;
        int64_t i = BX(s->box_slot, e);
        if (I(s->box_hash, i) != e + 1) return;            // (never: the slot is kept as entries move)
        int64_t j = i;
        for (int64_t step = 0; step < H; ++step) {
            j = j + 1 == H ? 0 : j + 1;
            const int64_t v = I(s->box_hash, j);
            if (v == 0) break;
            const int64_t k = BX(s->box_home, v - 1);
            const bool stays = i <= j ? (i < k && k <= j) : (i < k || k <= j);
            if (stays) continue;
            I(s->box_hash, i) = v;
            BX(s->box_slot, v - 1) = i;
            i = j;
        }
        I(s->box_hash, i) = 0;
    }
    // a key at the grid's edge, where Partition clamps (two neighbours would be one box): outside this layer
    EBB_HD bool edge(int64_t ix, int64_t iy, int64_t iz, int level) const {
        const int64_t g = level_grid(level);
        if (ix >= 0 && ix < g && iy >= 0 && iy < g && iz >= 0 && iz < g) return false;
        flag(F_EDGE);
        return true;
    }
    EBB_HD int64_t check_box(int64_t ix, int64_t iy, int64_t iz, int level) const {
        if (edge(ix, iy, iz, level)) return -1;
        return box_find(level, ix, iy, iz);
    }
    // a new box-table entry (a free one, else the next), which takes one of BoxAllocator's kept boxes
    EBB_HD int64_t new_box(int level, int64_t kx, int64_t ky, int64_t kz) {
        int64_t e = -1;
        const int64_t n = one(s->box_n);
        if (one(s->box_free_n) > 0) e = I(s->box_free, --one(s->box_free_n));   // a released entry again
        if (e < 0) {
            if (n >= B) {
                flag(F_BOXES);
                return -1;
            }
            e = n;
            one(s->box_n) = n + 1;
        }
        if (one(s->free_boxes) > 0) --one(s->free_boxes);
        BX(s->box_level, e) = level;
        BK(0, e) = kx;
        BK(1, e) = ky;
        BK(2, e) = kz;
        BX(s->box_balls, e) = 0;
        BX(s->box_kids, e) = 0;
        BX(s->box_bubble, e) = -1;
        hash_insert(e);
        return e;
    }
    // GetBox: the box, made with its missing ancestors when missing (a parent's key is its child's over 4)
    EBB_HDNI int64_t get_box(int64_t ix, int64_t iy, int64_t iz, int level) {
        if (edge(ix, iy, iz, level)) return -1;
        const int64_t found = box_find(level, ix, iy, iz);
        if (found >= 0) return found;
        int first = level;                                 // the shallowest missing level of the chain
        int64_t parent = -1;
        while (first > 0) {
            const int sh = 2 * (level - first + 1);
            parent = box_find(first - 1, ix >> sh, iy >> sh, iz >> sh);
            if (parent >= 0) break;
            --first;
        }
        for (int L = first; L <= level; ++L) {
            const int sh = 2 * (level - L);
            const int64_t e = new_box(L, ix >> sh, iy >> sh, iz >> sh);
            if (e < 0) return -1;
            BX(s->box_parent, e) = parent;                  // (a box's parent and top box outlive it: kids > 0)
            BX(s->box_top, e) = parent >= 0 ? BX(s->box_top, parent) : e;
            if (parent >= 0) ++BX(s->box_kids, parent);
            parent = e;
        }
        return parent;
    }
    // Release of an empty box, then of each ancestor it leaves empty: every box of the chain kept while BoxAllocator
    // held fewer than 256 when the chain began, else deleted. `watch` records the fate of two boxes the caller reads
    // afterwards (0 live, 1 released and kept, 2 released and deleted).
    EBB_HDNI void release(int64_t e, const int64_t* watch, int* fate) {
        const bool keep = one(s->free_boxes) < BOX_KEEP;
        int64_t cur = e;
        for (int guard = 0; guard < NUM_LEVELS && cur >= 0; ++guard) {
            const int64_t parent = BX(s->box_parent, cur);
            if (parent >= 0) --BX(s->box_kids, parent);
            hash_erase(cur);
            BX(s->box_level, cur) = -1;
            I(s->box_free, one(s->box_free_n)++) = cur;
            for (int k = 0; k < 2; ++k)
                if (watch[k] == cur) fate[k] = keep ? 1 : 2;
            if (keep) ++one(s->free_boxes);
            if (parent >= 0 && BX(s->box_kids, parent) == 0 && BX(s->box_balls, parent) == 0)
                cur = parent;
            else
                cur = -1;
        }
    }

    // ---- a ball's filing: level, key, sides, the active neighbours (bit 13 + x + 3 y + 9 z) ----
    EBB_HD int64_t& lvl(int64_t j) const { return I(s->level, j); }
    EBB_HD int64_t& key(int64_t j, int c) const { return I3(s->key, c, j, N); }
    EBB_HD int64_t& mod(int64_t j, int c) const { return I3(s->mod, c, j, N); }
    EBB_HD int64_t& active(int64_t j) const { return I(s->active, j); }
    // a filed ball's box entries by side (bit c set: the box beside its own on axis c), so that leaving them takes no
    // lookup; a huge ball's 27 boxes are looked up
    EBB_HD int64_t& fbox(int64_t j, int bits) const { return I3(s->fbox, bits, j, N); }

    // the ball's boxes in key order (the map DeleteFromBoxes walks), as table entries; returns their count
    EBB_HD int ball_boxes(int64_t j, int64_t* out) const {
        if (lvl(j) < 0) return 0;
        int64_t keys[27][3];
        int n = 0;
        const int64_t a = active(j);
        for (int z = -1; z <= 1; ++z)
            for (int y = -1; y <= 1; ++y)
                for (int x = -1; x <= 1; ++x) {
                    if (!((a >> (13 + x + 3 * y + 9 * z)) & 1)) continue;
                    const int64_t g = level_grid((int)lvl(j));
                    keys[n][0] = clamp_key(key(j, 0) + x, g);
                    keys[n][1] = clamp_key(key(j, 1) + y, g);
                    keys[n][2] = clamp_key(key(j, 2) + z, g);
                    ++n;
                }
        for (int i = 1; i < n; ++i)                        // insertion sort by (x, y, z)
            for (int k = i; k > 0; --k) {
                const bool less = keys[k][0] != keys[k - 1][0] ? keys[k][0] < keys[k - 1][0]
                                  : keys[k][1] != keys[k - 1][1] ? keys[k][1] < keys[k - 1][1]
                                                                 : keys[k][2] < keys[k - 1][2];
                if (!less) break;
                for (int c = 0; c < 3; ++c) {
                    const int64_t t = keys[k][c];
                    keys[k][c] = keys[k - 1][c];
                    keys[k - 1][c] = t;
                }
            }
        int m = 0;
        for (int i = 0; i < n; ++i) {
            if (i > 0 && keys[i][0] == keys[i - 1][0] && keys[i][1] == keys[i - 1][1] && keys[i][2] == keys[i - 1][2])
                continue;                                  // a clamped duplicate is one map entry
            out[m++] = box_find((int)lvl(j), keys[i][0], keys[i][1], keys[i][2]);
        }
        return m;
    }
    EBB_HD void clear_filing(int64_t j) const {
        lvl(j) = -1;
        I(s->my_box, j) = -1;
        I(s->my_top, j) = -1;
        active(j) = 0;
        for (int c = 0; c < 3; ++c) mod(j, c) = -2;
    }
    EBB_HD void leave_box(int64_t e, const int64_t* watch, int* fate) {
        if (e < 0) return;
        --BX(s->box_balls, e);
        if (BX(s->box_balls, e) == 0 && BX(s->box_kids, e) == 0) release(e, watch, fate);
    }
    // DeleteFromBoxes: the ball leaves each of its boxes in key order, each box released when left empty. The
    // entries come from the ball's record of them (key order: on each axis the lower key first, so the side box first
    // where the sphere reaches below); a huge ball, or a world past its table or the grid's edge (where keys clamp
    // and a box may be missing), looks its boxes up.
    EBB_HDNI void delete_from_boxes(int64_t j, const int64_t* watch, int* fate) {
        if (lvl(j) >= 0 && !huge(j) && !(one(s->flags) & (F_EDGE | F_BOXES))) {
            const int64_t mx = mod(j, 0), my = mod(j, 1), mz = mod(j, 2);
            for (int ox = 0; ox < 2; ++ox) {
                const int bx = mx < 0 ? 1 - ox : ox;
                if (bx && !mx) continue;
                for (int oy = 0; oy < 2; ++oy) {
                    const int by = my < 0 ? 1 - oy : oy;
                    if (by && !my) continue;
                    for (int oz = 0; oz < 2; ++oz) {
                        const int bz = mz < 0 ? 1 - oz : oz;
                        if (bz && !mz) continue;
                        leave_box(fbox(j, bx | (by << 1) | (bz << 2)), watch, fate);
                    }
                }
            }
        } else {
            int64_t boxes[27];
            const int n = ball_boxes(j, boxes);
            for (int i = 0; i < n; ++i) leave_box(boxes[i], watch, fate);
        }
        clear_filing(j);
    }
    EBB_HD void delete_from_boxes(int64_t j) {
        const int64_t watch[2] = {-1, -1};
        int fate[2] = {0, 0};
        delete_from_boxes(j, watch, fate);
    }
    EBB_HD int64_t topmost_of(int64_t e) const { return BX(s->box_top, e); }
    // a free ball's radius plus a tick at full thrust (Ball::GetInflatedRadius)
    EBB_HD double inflated_radius(int64_t j, const double* v) const {
        return inflated_radius_of(j, p->radius[row(j)], v);
    }
    // the same for a radius `rf` in place of the ball's own (a sensor's inflated one)
    EBB_HD double inflated_radius_of(int64_t j, float rf, const double* v) const {
        const int64_t r = row(j);
        const double radius = (double)rf;
        if (!p->free_[r]) return radius;
        const double m = dmul(p->mass[r], (double)p->agility[r]);
        const double k = p->friction;
        const double a = ddiv(dmul(dmul(k, (double)p->speed_fraction[r]), (double)p->max_vel[r]), m);
        const double speed = dsqrt(dadd(dadd(dmul(v[0], v[0]), dmul(v[1], v[1])), dmul(v[2], v[2])));
        const double ma = dmul(m, a);
        const double max_speed = ddiv(dsub(ma, dmul(dsub(ma, dmul(speed, k)), p->time_factor[r])), k);
        return dadd(radius, dmul(p->dt, max_speed));
    }
    EBB_HD static void key_for(int level, const double* x, int64_t* k) {
        const double fac = level_inv(level), half = level_half(level);
        for (int c = 0; c < 3; ++c) k[c] = to_i64(dmul(dadd(x[c], half), fac));
    }
    // the sides a sphere of radius `inflated` at x reaches out of its box (key `key0` at level0): -1, 0 or 1 an axis
    EBB_HD static void side_mods(int level0, const int64_t* key0, double inflated, const double* x, int64_t* m) {
        const double wd = level_width(level0);
        const double center = dmul(dmul(wd, (double)level_grid(level0)), 0.5);
        for (int q = 0; q < 3; ++q) {
            m[q] = 0;
            const double lo = dsub(dmul((double)key0[q], wd), center);
            const double hi = dsub(dmul((double)(key0[q] + 1), wd), center);
            if (dsub(dadd(lo, inflated), x[q]) > 0.0)
                m[q] = -1;
            else if (dsub(dsub(hi, inflated), x[q]) < 0.0)
                m[q] = 1;
        }
    }

    // ---- bubbles ----
    EBB_HD int64_t nearby_bubbles(int64_t kx, int64_t ky, int64_t kz) const {
        for (int i = -1; i <= 1; ++i)
            for (int j = -1; j <= 1; ++j)
                for (int k = -1; k <= 1; ++k) {
                    if (i == 0 && j == 0 && k == 0) continue;
                    const int64_t o = check_box(kx + i, ky + j, kz + k, 0);
                    if (o >= 0 && BX(s->box_bubble, o) != -1) return BX(s->box_bubble, o);
                }
        return -1;
    }
    // Traverse: the seed given to every top box reachable through neighbours without a bubble (a fill; the stack
    // holds each box once, marked as it is pushed)
    EBB_HD void traverse(int64_t top, int64_t seed) {
        if (BX(s->box_bubble, top) != -1) return;
        BX(s->box_bubble, top) = seed;
        int64_t sp = 0;
        I(s->stack, sp++) = top;
        while (sp > 0) {
            const int64_t e = I(s->stack, --sp);
            const int64_t kx = BK(0, e), ky = BK(1, e), kz = BK(2, e);
            for (int i = -1; i <= 1; ++i)
                for (int j = -1; j <= 1; ++j)
                    for (int k = -1; k <= 1; ++k) {
                        if (i == 0 && j == 0 && k == 0) continue;
                        const int64_t o = check_box(kx + i, ky + j, kz + k, 0);
                        if (o < 0 || BX(s->box_bubble, o) != -1) continue;
                        BX(s->box_bubble, o) = seed;
                        if (sp >= B) {
                            flag(F_BOXES);
                            return;
                        }
                        I(s->stack, sp++) = o;
                    }
        }
    }
    // the dictionary of bubble `bub`: whether it exists; its entry for ball `bid` (-1 none)
    EBB_HD int64_t dict_index(int64_t bub) const {
        const int64_t n = one(s->dict_n);
        for (int64_t d = 0; d < n; ++d)
            if (I(s->dict_bubble, d) == bub) return d;
        return -1;
    }
    EBB_HD int64_t entry_index(int64_t bub, int64_t bid) const {
        const int64_t n = one(s->entry_n);
        for (int64_t e = 0; e < n; ++e)
            if (I(s->entry_bubble, e) == bub && I(s->entry_id, e) == bid) return e;
        return -1;
    }
    EBB_HD void entry_erase(int64_t e) {
        const int64_t n = one(s->entry_n);
        for (int64_t i = e; i + 1 < n; ++i) {
            I(s->entry_bubble, i) = I(s->entry_bubble, i + 1);
            I(s->entry_id, i) = I(s->entry_id, i + 1);
            I(s->entry_value, i) = I(s->entry_value, i + 1);
        }
        one(s->entry_n) = n - 1;
    }
    // the interactive (which = 0) or keep-alive (1) set of a bubble: membership, insertion, removal
    EBB_HD int64_t* set_bub(int which) const { return which ? s->keep_bubble : s->inter_bubble; }
    EBB_HD int64_t* set_id(int which) const { return which ? s->keep_id : s->inter_id; }
    EBB_HD int64_t* set_n(int which) const { return which ? s->keep_n : s->inter_n; }
    EBB_HD bool set_any(int which, int64_t bub) const {
        const int64_t n = one(set_n(which));
        for (int64_t e = 0; e < n; ++e)
            if (I(set_bub(which), e) == bub) return true;
        return false;
    }
    EBB_HD void set_insert(int which, int64_t bub, int64_t bid) {
        const int64_t n = one(set_n(which));
        for (int64_t e = 0; e < n; ++e)
            if (I(set_bub(which), e) == bub && I(set_id(which), e) == bid) return;
        if (n >= s->sets) {
            flag(F_SETS);
            return;
        }
        I(set_bub(which), n) = bub;
        I(set_id(which), n) = bid;
        one(set_n(which)) = n + 1;
    }
    EBB_HD void set_erase(int which, int64_t bub, int64_t bid) {
        const int64_t n = one(set_n(which));
        for (int64_t e = 0; e < n; ++e)
            if (I(set_bub(which), e) == bub && I(set_id(which), e) == bid) {
                I(set_bub(which), e) = I(set_bub(which), n - 1);
                I(set_id(which), e) = I(set_id(which), n - 1);
                one(set_n(which)) = n - 1;
                return;
            }
    }
    // AddToBubble: the ball entered (+1, or 0 again after leaving) its bubble's dictionary and left (-1, or gone if it
    // had only entered) its old one's; its interactive and keep-alive memberships follow
    EBB_HDNI void add_to_bubble(int64_t j) {
        const int64_t bid = id(j), bub = I(s->bubble, j), old = I(s->old_bubble, j);
        if (bub != -1) {
            if (dict_index(bub) < 0) {
                const int64_t n = one(s->dict_n);
                if (n >= s->dicts) {
                    flag(F_DICTS);
                } else {
                    I(s->dict_bubble, n) = bub;
                    one(s->dict_n) = n + 1;
                }
            }
            const int64_t e = entry_index(bub, bid);
            if (e < 0) {
                const int64_t n = one(s->entry_n);
                if (n >= s->entries) {
                    flag(F_ENTRIES);
                } else {
                    I(s->entry_bubble, n) = bub;
                    I(s->entry_id, n) = bid;
                    I(s->entry_value, n) = 1;
                    one(s->entry_n) = n + 1;
                }
            } else if (I(s->entry_value, e) == -1) {
                I(s->entry_value, e) = 0;
            }
        }
        if (old != -1 && dict_index(old) >= 0) {
            const int64_t e = entry_index(old, bid);
            if (e >= 0) {
                if (I(s->entry_value, e) == 0)
                    I(s->entry_value, e) = -1;
                else if (I(s->entry_value, e) == 1)
                    entry_erase(e);
            }
        }
        if (interactive(j)) {
            if (bub != -1) set_insert(0, bub, bid);
            if (old != -1) set_erase(0, old, bid);
        }
        if (U(s->keep_alive, j)) {
            if (bub != -1) set_insert(1, bub, bid);
            if (old != -1) set_erase(1, old, bid);
        }
    }
    // InDeadBubble: no interactive and no keep-alive ball in the ball's bubble, and the ball not in WARP
    EBB_HD bool in_dead_bubble(int64_t j) const {
        if (p->mode[row(j)] == WARP) return false;
        const int64_t bub = I(s->bubble, j);
        return !set_any(0, bub) && !set_any(1, bub);
    }

    // ---- filing ----
    EBB_HD void insert_in_box(int64_t j, int64_t e) const {
        (void)j;
        if (e >= 0) ++BX(s->box_balls, e);
    }
    // Ball::InsertInBoxes: the ball's box at the level of its inflated radius and the neighbours its sphere reaches
    // (every neighbour for a huge ball), unless box and sides are as they were; the top box takes the bubble
    // (`inflated`: the ball's inflated radius; `box0`: its box at level0, live unless fate_box1 says it was released)
    EBB_HDNI void ball_insert_in_boxes(int64_t j, const double* x, double inflated, int level0, const int64_t* key0,
                                     int64_t box0, int fate_box1, int64_t new_bubble) {
        if (fate_box1 == 2) flag(F_UNDEFINED);             // a deleted box's memory read
        int64_t m[3];
        side_mods(level0, key0, inflated, x, m);
        if (lvl(j) >= 0 && lvl(j) == level0 && key(j, 0) == key0[0] && key(j, 1) == key0[1] && key(j, 2) == key0[2] &&
            mod(j, 0) == m[0] && mod(j, 1) == m[1] && mod(j, 2) == m[2])
            return;
        if (fate_box1 == 0 && refile_near(j, level0, key0, m, box0, new_bubble)) return;
        const int64_t watch[2] = {fate_box1 == 0 ? box0 : -1, -1};
        int fate[2] = {0, 0};
        delete_from_boxes(j, watch, fate);
        const int level = level0;                          // (level_for(inflated): the same radius)
        // the box found before, still live, or GetBox again (made anew when the leaving released it)
        const int64_t box1 = watch[0] >= 0 && fate[0] == 0 ? box0 : get_box(key0[0], key0[1], key0[2], level);
        if (box1 < 0) return;
        for (int c = 0; c < 3; ++c) {
            mod(j, c) = m[c];
            key(j, c) = BK(c, box1);
        }
        lvl(j) = level;
        insert_in_box(j, box1);
        const int64_t top = topmost_of(box1);
        if (top >= 0) BX(s->box_bubble, top) = new_bubble;
        I(s->my_box, j) = box1;                            // (entries stay put while the ball is filed in them)
        I(s->my_top, j) = top;
        int64_t act = int64_t(1) << 13;
        const int64_t ix = key(j, 0), iy = key(j, 1), iz = key(j, 2);
        const int64_t row_j = row(j);
        if (level == 0 && (double)fmul(p->radius[row_j], 2.0f) > level_width(0)) {   // a huge ball: every neighbour
            for (int a = -1; a <= 1; ++a)
                for (int b = -1; b <= 1; ++b)
                    for (int c = -1; c <= 1; ++c) {
                        if (a == 0 && b == 0 && c == 0) continue;
                        insert_in_box(j, get_box(ix + a, iy + b, iz + c, 0));
                        act |= int64_t(1) << (13 + a + 3 * b + 9 * c);
                    }
            active(j) = act;
            return;
        }
        const int64_t mx = m[0], my = m[1], mz = m[2];
        fbox(j, 0) = box1;
        // a warp finds the side boxes that exist at once, a lane a side (no side's making makes another side's box,
        // and making moves no entry); the others are made in order
        int64_t found = -1;
#ifdef __CUDA_ARCH__
        if constexpr (COOP) {
            const int bits = lane & 7;
            const bool on = lane >= 1 && lane <= 7 && !((bits & 1) && !mx) && !((bits & 2) && !my) && !((bits & 4) && !mz);
            if (on && (mx | my | mz)) {
                const int64_t kx = ix + ((bits & 1) ? mx : 0), ky = iy + ((bits & 2) ? my : 0),
                              kz = iz + ((bits & 4) ? mz : 0);
                const int64_t g = level_grid(level);
                if (kx >= 0 && kx < g && ky >= 0 && ky < g && kz >= 0 && kz < g) found = box_find(level, kx, ky, kz);
            }
        }
#endif
        auto side = [&](int64_t a, int64_t b, int64_t c) {
            const int bits = (a != 0) | ((b != 0) << 1) | ((c != 0) << 2);
            int64_t e = -1;
#ifdef __CUDA_ARCH__
            if constexpr (COOP) e = __shfl_sync(0xffffffffu, found, bits);
#endif
            if (e < 0) e = get_box(ix + a, iy + b, iz + c, level);
            insert_in_box(j, e);
            fbox(j, (a != 0) | ((b != 0) << 1) | ((c != 0) << 2)) = e;
            act |= int64_t(1) << (13 + a + 3 * b + 9 * c);
        };
        if (mx) side(mx, 0, 0);
        if (my) side(0, my, 0);
        if (mz) side(0, 0, mz);
        if (mx && my) side(mx, my, 0);
        if (mx && mz) side(mx, 0, mz);
        if (my && mz) side(0, my, mz);
        if (mx && my && mz) side(mx, my, mz);
        active(j) = act;
    }
    // A re-filing at the ball's own level under its own top box: the boxes it keeps are left alone, those it no longer reaches
    // left, the new ones entered. The whole one leaves every box first and makes again those it emptied, chains of
    // ancestors with them (a ball alone in its boxes, as most are): the same boxes, balls and children in the end, and the
    // same kept count, which its releases and makings move by their difference while every release is kept (the count far
    // enough below 256) and no making comes before a release (so a floor at 0 is met alike); its top's bubble is the ball's
    // either way. Conditions checked, else false and nothing done. 16,384 worlds of 4 ships a thread each 1.37 -> 1.25 ms a
    // tick, 8,000 partition worlds 4.1 -> 3.9.
    EBB_HD bool refile_near(int64_t j, int level, const int64_t* k, const int64_t* m, int64_t box0, int64_t new_bubble) {
        if (lvl(j) != level || huge(j) || box0 < 0 || one(s->flags) != 0 || one(s->free_boxes) >= BOX_KEEP - 64) return false;
        if (level == 0 && (double)fmul(p->radius[row(j)], 2.0f) > level_width(0)) return false;
        int64_t ok[3], om[3];
        unsigned oside = 0, nside = 0;                     // the axes with a side, before and now
        int kept_old = 0, kept_new = 0;                    // bit 2 q + i: on axis q the key i (1 the side's) is also the other's
        for (int q = 0; q < 3; ++q) {
            ok[q] = key(j, q);
            om[q] = mod(j, q);
            const int64_t a[2] = {ok[q], ok[q] + om[q]}, b[2] = {k[q], k[q] + m[q]};
            const int up = 2 * level;
            if ((a[0] >> up) != (b[0] >> up) || (a[1] >> up) != (b[0] >> up) || (b[1] >> up) != (b[0] >> up)) return false;
            oside |= (om[q] != 0) << q;
            nside |= (m[q] != 0) << q;
            for (int i = 0; i < 2; ++i) {
                kept_old |= (a[i] == b[0] || a[i] == b[1]) << (2 * q + i);
                kept_new |= (b[i] == a[0] || b[i] == a[1]) << (2 * q + i);
            }
        }
        auto kept = [](int on, unsigned c) {
            return (((on >> (c & 1)) & (on >> (2 + ((c >> 1) & 1))) & (on >> (4 + (c >> 2)))) & 1) != 0;
        };
        int32_t was[8];
        const int64_t none[2] = {-1, -1};
        int fate[2] = {0, 0};
        for (unsigned c = 0; c < 8; ++c)
            if (!(c & ~oside)) was[c] = (int32_t)fbox(j, (int)c);
        for (unsigned c = 0; c < 8; ++c)
            if (!(c & ~oside) && !kept(kept_old, c)) leave_box(was[c], none, fate);
        for (int q = 0; q < 3; ++q) {
            key(j, q) = k[q];
            mod(j, q) = m[q];
        }
        const int64_t top = topmost_of(box0);
        if (top >= 0) BX(s->box_bubble, top) = new_bubble;
        I(s->my_box, j) = box0;
        I(s->my_top, j) = top;
        // (a warp finds the sides that exist at once, a lane a side)
        int64_t found = -1;
#ifdef __CUDA_ARCH__
        if constexpr (COOP) {
            const unsigned c = lane & 7;
            if (lane >= 1 && lane <= 7 && !(c & ~nside) && !kept(kept_new, c)) {
                const int64_t kx = k[0] + ((c & 1) ? m[0] : 0), ky = k[1] + ((c & 2) ? m[1] : 0),
                              kz = k[2] + ((c & 4) ? m[2] : 0);
                const int64_t g = level_grid(level);
                if (kx >= 0 && kx < g && ky >= 0 && ky < g && kz >= 0 && kz < g) found = box_find(level, kx, ky, kz);
            }
        }
#endif
        int64_t act = 0;
        for (unsigned c = 0; c < 8; ++c) {
            if (c & ~nside) continue;
            int64_t e = c == 0 ? box0 : -1;
            const int64_t d[3] = {(c & 1) ? m[0] : 0, (c & 2) ? m[1] : 0, (c & 4) ? m[2] : 0};
            if (kept(kept_new, c)) {
                unsigned o = 0;                            // the corner it was
                for (int q = 0; q < 3; ++q) o |= (k[q] + d[q] != ok[q]) << q;
                e = was[o];
            } else {
#ifdef __CUDA_ARCH__
                if constexpr (COOP) {
                    const int64_t f = __shfl_sync(0xffffffffu, found, (int)c);
                    if (c != 0) e = f;
                }
#endif
                if (e < 0) e = get_box(k[0] + d[0], k[1] + d[1], k[2] + d[2], level);
                insert_in_box(j, e);
            }
            fbox(j, (int)c) = e;
            act |= int64_t(1) << (13 + d[0] + 3 * d[1] + 9 * d[2]);
        }
        active(j) = act;
        return true;
    }
    // Ballpark::InsertInBoxes on the master: the ball's new top box, its bubble or, for a top without one, a
    // neighbour's or a new id; AddToBubble when the ball's bubble changes; then its filing
    EBB_HDNI void insert_in_boxes(int64_t j, const double* x, const double* v) {
        const double inflated = inflated_radius(j, v);
        const int level0 = level_for(inflated);
        int64_t k[3];
        key_for(level0, x, k);
        // the ball's own box when it stays in it (the common re-filing): its entry and its top's, without a scan
        const bool same = lvl(j) == level0 && key(j, 0) == k[0] && key(j, 1) == k[1] && key(j, 2) == k[2] &&
                          I(s->my_box, j) >= 0 && I(s->my_top, j) >= 0;
        const int64_t box1 = same ? I(s->my_box, j) : get_box(k[0], k[1], k[2], level0);
        if (box1 < 0) return;
        int64_t key0[3];
        for (int c = 0; c < 3; ++c) key0[c] = BK(c, box1);
        const int64_t top = same ? I(s->my_top, j) : topmost_of(box1);
        int64_t new_bubble = BX(s->box_bubble, top);
        int fate[2] = {0, 0};
        if (new_bubble == -1) {
            const int64_t tk[3] = {BK(0, top), BK(1, top), BK(2, top)};
            const int64_t watch[2] = {box1, top};
            delete_from_boxes(j, watch, fate);             // may release box1 and its top: both are still read
            if (fate[1] == 2) flag(F_UNDEFINED);
            new_bubble = nearby_bubbles(tk[0], tk[1], tk[2]);
            if (new_bubble == -1) new_bubble = one(s->bubble_id)++;
            if (fate[1] == 0) BX(s->box_bubble, top) = new_bubble;   // (a released top's write is lost)
        }
        if (I(s->bubble, j) != new_bubble) {
            I(s->old_bubble, j) = I(s->bubble, j);
            I(s->bubble, j) = new_bubble;
            add_to_bubble(j);
        }
        ball_insert_in_boxes(j, x, inflated, level0, key0, box1, fate[0], new_bubble);
    }
    EBB_HD void insert_in_boxes(int64_t j) {
        const double x[3] = {pos(j, 0), pos(j, 1), pos(j, 2)}, v[3] = {vel(j, 0), vel(j, 1), vel(j, 2)};
        insert_in_boxes(j, x, v);
    }


    // ---- GetNearbyBalls' walk (Partition.cpp:344), as a sort key per pair ----
    // A ball's boxes are a product of one key range an axis: its box's key and the side its sphere reaches (mod), or
    // for a huge ball the three keys around its own (its 27 top boxes).
    EBB_HD bool huge(int64_t j) const { return active(j) == int64_t(0x7FFFFFF); }
    EBB_HD void key_range(int64_t j, int q, int64_t* lo, int64_t* hi) const {
        const int64_t k = key(j, q), m = mod(j, q);
        if (huge(j)) {
            *lo = k - 1;
            *hi = k + 1;
        } else {
            *lo = k + (m < 0 ? m : 0);
            *hi = k + (m > 0 ? m : 0);
        }
    }
    // A filing as the walk reads it: the level and each axis's key range
    struct Filing {
        int64_t L;
        int64_t lo[3], hi[3];
    };
    EBB_HD Filing filing_of(int64_t j) const {
        Filing f;
        f.L = lvl(j);
        for (int q = 0; q < 3; ++q) key_range(j, q, &f.lo[q], &f.hi[q]);
        return f;
    }
    // The position of slot o's first box in slot b's walk, or NOT_A_CANDIDATE when no box of o is one of b's, an
    // ancestor of one or below one. b's boxes are walked in key order; at each, its ancestors holding balls bottom-up
    // (those not met before), its descendants in post-order (children by key), then the box itself. The key: the
    // index of the first of b's boxes o's box relates to, the part (0 an ancestor, 1 below, 2 the box itself), then
    // the ancestor's distance or the box's post-order code (path digits below b's level, 64 past o's level).
    // Relatedness factors over the axes: the finer filing's key range, shifted to the coarser level, meets the
    // coarser's.
    // whether slot o's filing meets b's walk (walk_key's first test: it then has a key)
    EBB_HD bool related(const Filing& fb, int64_t o) const {
        const Filing fo = filing_of(o);
        const bool coarse = fo.L <= fb.L;
        const int64_t sh = 2 * (coarse ? fb.L - fo.L : fo.L - fb.L);
        for (int q = 0; q < 3; ++q) {
            const int64_t xl = (coarse ? fb.lo[q] : fo.lo[q]) >> sh, xh = (coarse ? fb.hi[q] : fo.hi[q]) >> sh;
            const int64_t yl = coarse ? fo.lo[q] : fb.lo[q], yh = coarse ? fo.hi[q] : fb.hi[q];
            if ((xl > yl ? xl : yl) > (xh < yh ? xh : yh)) return false;
        }
        return true;
    }
    EBB_HD int64_t walk_key(const Filing& fb, int64_t o) const {
        const Filing fo = filing_of(o);
        const int64_t Lb = fb.L, Ln = fo.L;
        int64_t cb[3];
        for (int q = 0; q < 3; ++q) cb[q] = fb.hi[q] - fb.lo[q] + 1;
        const bool coarse = Ln <= Lb;
        const int64_t sh = 2 * (coarse ? Lb - Ln : Ln - Lb);
        for (int q = 0; q < 3; ++q) {
            const int64_t xl = (coarse ? fb.lo[q] : fo.lo[q]) >> sh, xh = (coarse ? fb.hi[q] : fo.hi[q]) >> sh;
            const int64_t yl = coarse ? fo.lo[q] : fb.lo[q], yh = coarse ? fo.hi[q] : fb.hi[q];
            if ((xl > yl ? xl : yl) > (xh < yh ? xh : yh)) return NOT_A_CANDIDATE;
        }
        int64_t span = 1;
        for (int l = 0; l < NUM_LEVELS - 1; ++l) span *= CODE_BASE;
        if (coarse) {                                      // an ancestor or a box of b's level: b's first box under it
            int64_t idx[3];
            for (int q = 0; q < 3; ++q) {
                idx[q] = 0;
                while (idx[q] + 1 < cb[q]) {
                    const int64_t v = (fb.lo[q] + idx[q]) >> sh;
                    if (v >= fo.lo[q] && v <= fo.hi[q]) break;
                    ++idx[q];
                }
            }
            const int64_t seg = (idx[0] * cb[1] + idx[1]) * cb[2] + idx[2];
            return Ln < Lb ? (seg * 3) * span + (Lb - Ln) : (seg * 3 + 2) * span;
        }
        // below: the least key over o's boxes under b's. o's boxes are the product of its axes' keys, and the key is
        // the index of b's box (lexicographic in the axes' indices), then the post-order code, whose digit at a level
        // is 16 x + 4 y + z of the box's path (0 above b's level, 64 past o's): a sum of one term an axis. So the least
        // key takes on each axis the least index, and among the keys with it the least path term.
        int64_t jmin[3], pmin[3];
        for (int q = 0; q < 3; ++q) {
            jmin[q] = INT64_MAX;
            pmin[q] = INT64_MAX;
            for (int64_t v = fo.lo[q]; v <= fo.hi[q]; ++v) {
                const int64_t anc = v >> sh;
                if (anc < fb.lo[q] || anc > fb.hi[q]) continue;
                const int64_t jq = anc - fb.lo[q];
                int64_t path = 0;                          // the path's digits on this axis, base 65, levels Lb+1..Ln
                for (int64_t li = Lb + 1; li <= Ln; ++li) path = path * CODE_BASE + ((v >> (2 * (Ln - li))) & 3);
                if (jq < jmin[q] || (jq == jmin[q] && path < pmin[q])) {
                    jmin[q] = jq;
                    pmin[q] = path;
                }
            }
            if (jmin[q] == INT64_MAX) return NOT_A_CANDIDATE;
        }
        int64_t tail = 1;                                  // 65 ^ (levels past o's)
        for (int64_t li = Ln + 1; li < NUM_LEVELS; ++li) tail *= CODE_BASE;
        const int64_t seg = (jmin[0] * cb[1] + jmin[1]) * cb[2] + jmin[2];
        const int64_t code = tail * (16 * pmin[0] + 4 * pmin[1] + pmin[2] + 1) - 1;   // the 64s past o's level: tail - 1
        return (seg * 3 + 1) * span + code;
    }
    // GetNearbyBalls from slot b (no missiles, fields or global balls here): the balls filed in related boxes that
    // pass the filter, in the walk's order (its key, then id), into out; returns their count
    // (`as`: b's filing for the walk in place of its own, the sensor's inflated one when it is not re-filed)
    EBB_HDNI int nearby(int64_t b, bool exclude_fixed, bool exclude_inert, bool exclude_cloaked, uint8_t* out,
                        const Filing* as = nullptr) const {
        const int64_t bub = I(s->bubble, b);
        if (exclude_inert && !set_any(0, bub)) return 0;
        if (lvl(b) < 0) return 0;
        const Filing fb = as ? *as : filing_of(b);
#ifdef __CUDA_ARCH__
        if constexpr (COOP) {
            return nearby_warp(b, bub, exclude_fixed, exclude_inert, exclude_cloaked, out, fb);
        } else
#endif
        {
            return nearby_serial(b, bub, exclude_fixed, exclude_inert, exclude_cloaked, out, fb);
        }
    }
    // nearby's single-thread form: an insertion by (key, id) as each candidate is met
    EBB_HDNI int nearby_serial(int64_t b, int64_t bub, bool exclude_fixed, bool exclude_inert, bool exclude_cloaked,
                             uint8_t* out, const Filing& fb) const {
        int64_t keys[EBB_SPACE_MAX_SLOTS], oid[EBB_SPACE_MAX_SLOTS];
        int n = 0;
        for (int64_t o = 0; o < N; ++o) {
            if (o == b || !slot_ok(o) || !U(s->in_park, o) || lvl(o) < 0) continue;
            const int64_t k = walk_key(fb, o);
            if (k == NOT_A_CANDIDATE) continue;
            const int64_t r = row(o);
            if (exclude_cloaked && (at(s->cloaked, o) != 0 || !p->massive[r])) continue;
            if (exclude_inert) {
                if (!p->interactive[r]) continue;
            } else {
                if (I(s->bubble, o) != bub) continue;
                if (exclude_fixed && !p->free_[r]) continue;
            }
            const int64_t i = p->ids[r];
            int m = n;
            for (; m > 0 && (keys[m - 1] > k || (keys[m - 1] == k && oid[m - 1] > i)); --m) {
                keys[m] = keys[m - 1];
                oid[m] = oid[m - 1];
                out[m] = out[m - 1];
            }
            keys[m] = k;
            oid[m] = i;
            out[m] = (uint8_t)o;
            ++n;
        }
        return n;
    }

#ifdef __CUDA_ARCH__
    // The slots the warp's sorts cover: the world's N rounded up to a power of two, 32 at least
    __device__ int sort_span() const {
        int S = 32;
        while (S < N) S <<= 1;
        return S;
    }
    // A bitonic sort of the warp's scratch (sh->key, sh->id, carrying sh->out) by (key, id) over its first S entries
    // (S a power of two), the lanes taking the pairs of each stage
    __device__ void warp_sort(int S) const {
        for (int k = 2; k <= S; k <<= 1)
            for (int jj = k >> 1; jj > 0; jj >>= 1) {
                for (int i = lane; i < S; i += 32) {
                    const int x = i ^ jj;
                    if (x <= i) continue;
                    const int64_t ki = sh->key[i], kx = sh->key[x], ii = sh->id[i], ix = sh->id[x];
                    const bool x_less = kx < ki || (kx == ki && ix < ii);
                    const bool x_more = kx > ki || (kx == ki && ix > ii);
                    if (((i & k) == 0) ? x_less : x_more) {
                        sh->key[i] = kx;
                        sh->key[x] = ki;
                        sh->id[i] = ix;
                        sh->id[x] = ii;
                        const uint8_t t = sh->out[i];
                        sh->out[i] = sh->out[x];
                        sh->out[x] = t;
                    }
                }
                __syncwarp();
            }
    }

    // nearby's warp form: each lane takes the slots lane, lane + 32, ...: the filter and the walk key (NOT_A_CANDIDATE
    // for a ball that is none); the candidates are packed to the front of the scratch (a ballot a round) and sorted
    // by (key, id) over the lanes, a bitonic sort of their count rounded up to a power of two (ids are distinct, so
    // the order is the serial insertion's); every lane reads the order back
    __device__ int nearby_warp(int64_t b, int64_t bub, bool exclude_fixed, bool exclude_inert, bool exclude_cloaked,
                               uint8_t* out, const Filing& fb) const {
        int n = 0;
        const int S = sort_span() < occupied ? sort_span() : occupied;   // (no candidate past the last slot in the park)
        for (int64_t base = 0; base < S; base += 32) {     // the candidates packed to the front, in slot order
            const int64_t o = base + lane;
            int64_t k = NOT_A_CANDIDATE, i = INT64_MAX;
            if (o < N && o != b && slot_ok(o) && U(s->in_park, o) && lvl(o) >= 0) {
                k = walk_key(fb, o);
                const int64_t r = row(o);
                if (k != NOT_A_CANDIDATE) {
                    bool keep = !(exclude_cloaked && (at(s->cloaked, o) != 0 || !p->massive[r]));
                    if (exclude_inert)
                        keep = keep && p->interactive[r];
                    else
                        keep = keep && I(s->bubble, o) == bub && !(exclude_fixed && !p->free_[r]);
                    if (!keep) k = NOT_A_CANDIDATE;
                    else i = p->ids[r];
                }
            }
            const bool is = k != NOT_A_CANDIDATE;
            const unsigned in = __ballot_sync(0xffffffffu, is);
            if (is) {
                const int at_ = n + __popc(in & ((1u << lane) - 1u));
                sh->key[at_] = k;
                sh->id[at_] = i;
                sh->out[at_] = (uint8_t)o;
            }
            n += __popc(in);
        }
        int P = 1;                                         // the sort's span: the candidates, to a power of two
        while (P < n) P <<= 1;
        for (int e = n + lane; e < P; e += 32) {
            sh->key[e] = NOT_A_CANDIDATE;
            sh->id[e] = INT64_MAX;
        }
        __syncwarp();
        warp_sort(P);
        for (int i = 0; i < n; ++i) out[i] = sh->out[i];
        __syncwarp();
        return n;
    }
#endif

    // ---- std::unordered_map<int64_t, ...> in libstdc++'s iteration order (space.py:193-322) ----
    // A map's keys are slots (their balls' ids the keys' values): k[e step] for e < len, in iteration order, with
    // the map's bucket count (1 for a fresh map).
    // Beside the order, the keys as a set of slots: 128 bits, word c at m[c mstep] (membership without a scan).
    struct UMap {
        uint8_t* k;
        int64_t step;
        int32_t* len;
        int32_t* bkt;
        uint64_t* m;
        int64_t mstep;
    };
    EBB_HD UMap sensor_map(int64_t j) const {
        return UMap{&at(s->slist, j), N * step(), &at(s->slen, j), &at(s->sbkt, j), &at(s->smask, j), N * step()};
    }
    EBB_HD UMap proximity_map() const {
        return UMap{&at(s->pmap, 0), step(), &at(s->pn, 0), &at(s->pbkt, 0), &at(s->pmask, 0), step()};
    }
    EBB_HD bool umap_has(const UMap& m, int64_t slot) const {
        return ((m.m[(slot >> 6) * m.mstep] >> (slot & 63)) & 1) != 0;
    }
    EBB_HD void umap_clear(const UMap& m) const {
        *m.len = 0;
        m.m[0] = 0;
        m.m[m.mstep] = 0;
    }
    EBB_HD uint64_t bucket_of(int64_t slot, int32_t bkt) const {
        const uint64_t k = (uint64_t)id(slot);             // (a 32-bit remainder for the ids that fit in one)
        return (k >> 32) == 0 ? (uint64_t)((uint32_t)k % (uint32_t)bkt) : k % (uint64_t)bkt;
    }
    EBB_HD int32_t umap_find(const UMap& m, int64_t slot) const {
        const int32_t n = *m.len;
        for (int32_t e = 0; e < n; ++e)
            if (m.k[e * m.step] == (uint8_t)slot) return e;
        return -1;
    }
    // the linking rule: just before the first key of the order in the key's bucket, else at the front
    EBB_HD void umap_link(const UMap& m, int64_t slot) const {
        const int32_t n = *m.len, bkt = *m.bkt;
        const uint64_t b = bucket_of(slot, bkt);
        int32_t at0 = 0;
        for (int32_t e = 0; e < n; ++e)
            if (bucket_of(m.k[e * m.step], bkt) == b) {
                at0 = e;
                break;
            }
        for (int32_t e = n; e > at0; --e) m.k[e * m.step] = m.k[(e - 1) * m.step];
        m.k[at0 * m.step] = (uint8_t)slot;
        *m.len = n + 1;
        m.m[(slot >> 6) * m.mstep] |= uint64_t(1) << (slot & 63);
    }
    // insert(): an absent key linked; before it, a fresh map takes 13 buckets and a key past the bucket count grows
    // the table, every key re-linked in its old order. A map past umap_cap keys flags the world.
    EBB_HDNI bool umap_insert(const UMap& m, int64_t slot, int64_t flag_bit) const {
        if (umap_has(m, slot)) return false;
        const int32_t n = *m.len;
        if (n >= s->umap_cap) {
            flag(flag_bit);
            return false;
        }
        if (*m.bkt <= 1 || n + 1 > *m.bkt) {
            const int32_t nb = umap_next_buckets(*m.bkt);
            if (nb < 0) {
                flag(flag_bit);
                return false;
            }
            uint8_t old[EBB_SPACE_MAX_SLOTS];
            for (int32_t e = 0; e < n; ++e) old[e] = m.k[e * m.step];
            *m.bkt = nb;
            *m.len = 0;
            for (int32_t e = 0; e < n; ++e) umap_link(m, old[e]);
        }
        umap_link(m, slot);
        return true;
    }
    EBB_HD void umap_erase_at(const UMap& m, int32_t e0) const {
        const int32_t n = *m.len;
        const int64_t slot = m.k[e0 * m.step];
        m.m[(slot >> 6) * m.mstep] &= ~(uint64_t(1) << (slot & 63));
        for (int32_t e = e0; e + 1 < n; ++e) m.k[e * m.step] = m.k[(e + 1) * m.step];
        *m.len = n - 1;
    }
    EBB_HD void umap_erase(const UMap& m, int64_t slot) const {
        if (!umap_has(m, slot)) return;
        const int32_t e = umap_find(m, slot);
        if (e >= 0) umap_erase_at(m, e);
    }

    // ---- the proximity sensors, notification ranges and target tracking (space.py:1345-1477) ----
    EBB_HD void event(int kind, int64_t ball, int64_t other, int value) const {
        const int64_t n = one(s->evn);
        if (n < s->events)
            at(s->ev, n) = (int32_t)(kind | (value << 4) | ((int32_t)ball << 8) | ((int32_t)other << 16));
        else
            flag(F_EVENTS);
        one(s->evn) = n + 1;
    }
    EBB_HD double dist2(int64_t a, const double* x) const {
        const double d0 = dsub(pos(a, 0), x[0]), d1 = dsub(pos(a, 1), x[1]), d2 = dsub(pos(a, 2), x[2]);
        return dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
    }
    EBB_HD double dist2_slots(int64_t a, int64_t b) const {
        const double x[3] = {pos(b, 0), pos(b, 1), pos(b, 2)};
        return dist2(a, x);
    }
    // Ball::UpdateProximityStatus: a ball with a tracking range, a notification range or an active sensor is in the
    // proximity map, else out of it
    EBB_HD void update_proximity_status(int64_t j) const {
        const bool on = at(s->trk_range, j) != 0.0 || at(s->ntf_range, j) != 0.0 || p->sensor[row(j)] != 0;
        at(s->has_prox, j) = on ? 1 : 0;
        if (on)
            umap_insert(proximity_map(), j, F_PROXIMITY);
        else
            umap_erase(proximity_map(), j);
    }
    // a new ball's: no sensor (period 2 s), no notification range, no tracking, not cloaked, a fresh sensor list
    EBB_HD void reset_sensors(int64_t j) const {
        at(s->srange, j) = 0.0;
        at(s->speriod, j) = 2.0;
        at(s->selapsed, j) = 0.0;
        at(s->sonly, j) = 0;
        at(s->has_prox, j) = 0;
        at(s->ntf_range, j) = 0.0;
        at(s->ntf_in, j) = 0;
        at(s->trk, j) = -1;
        at(s->trk_range, j) = 0.0;
        at(s->trk_in, j) = 0;
        at(s->cloaked, j) = 0;
        umap_clear(sensor_map(j));
        at(s->sbkt, j) = 1;
        p->sensor[row(j)] = 0;
    }
    // AddProximitySensor (Ball.cpp:244; SEN-701): refused when float radius + float range < 0; the list emptied (its
    // buckets kept); a shuffled sensor starts its period at floatrand(0, period), the world's rand() drawn once
    EBB_HD void add_sensor(int64_t j, double range, double period, bool only, bool shuffle) const {
        const int64_t r = row(j);
        const float rng = (float)range;
        if (fadd(p->radius[r], rng) < 0.0f) return;
        umap_clear(sensor_map(j));
        at(s->srange, j) = (double)rng;
        at(s->speriod, j) = period;
        p->sensor[r] = 1;
        at(s->sonly, j) = only ? 1 : 0;
        if (shuffle) {
            int32_t* st = s->rnd + w * EBB_RAND_WORDS;
            int32_t f = st[grand::DEG], rr = st[grand::DEG + 1];
            const int32_t v = grand::draw(st, f, rr);
            st[grand::DEG] = f;
            st[grand::DEG + 1] = rr;
            at(s->selapsed, j) = dadd(0.0, dmul(ddiv((double)v, RAND_MAX_D), dsub(period, 0.0)));
        }
        update_proximity_status(j);
    }
    EBB_HD void remove_sensor(int64_t j) const {
        p->sensor[row(j)] = 0;
        update_proximity_status(j);
    }
    // SetNotificationRange (SEN-704): a negative range ignored; the in-range flag reset
    EBB_HD void set_notification_range(int64_t j, double n) const {
        if (n < 0.0) return;
        at(s->ntf_range, j) = n;
        update_proximity_status(j);
        at(s->ntf_in, j) = 0;
    }
    // SetTargetTracking (SEN-703): a range <= 0 or a target id of 0 turns it off (the proximity status kept)
    EBB_HD void set_tracking(int64_t j, int64_t target, double range, bool target_zero) const {
        if (range <= 0.0 || target_zero) {
            at(s->trk, j) = -1;
            at(s->trk_range, j) = 0.0;
            return;
        }
        if (!slot_ok(target) || !U(s->in_park, target)) return;
        at(s->trk, j) = target;
        at(s->trk_range, j) = range;
        update_proximity_status(j);
        at(s->trk_in, j) = 0;
    }
    // CheckForProximity_NotificationRange (Ball.cpp:520): within the range of the goto point, or within a shell of
    // the range's width around the followed ball's follow range
    EBB_HD void check_notification_range(int64_t j) const {
        const double n = at(s->ntf_range, j);
        if (n == 0.0) return;
        const int64_t r = row(j);
        const int32_t mode = p->mode[r];
        const double rad = (double)p->radius[r];
        bool inside = false;
        if (mode == GOTO) {
            const double lim = dadd(n, rad);
            const double g[3] = {p->goto_pt[r], p->goto_pt[p->n + r], p->goto_pt[2 * p->n + r]};
            inside = dist2(j, g) < dmul(lim, lim);
        } else if (mode == FOLLOW || mode == ORBIT) {
            const int32_t t = p->follow_ptr[r];
            if (t >= 0) {
                const double x[3] = {p->pos[t], p->pos[p->n + t], p->pos[2 * p->n + t]};
                const double len2 = dist2(j, x);
                const double hi = dadd(dadd(dadd((double)p->radius[t], (double)p->follow_range[r]), n), rad);
                double lo = dsub(hi, dmul(2.0, n));
                if (lo < 0.0) lo = 0.0;
                inside = len2 < dmul(hi, hi) && len2 > dmul(lo, lo);
            }
        }
        bool send = false;
        if (inside) {
            if (!at(s->ntf_in, j)) {
                send = true;
                at(s->ntf_in, j) = 1;
            }
        } else if (at(s->ntf_in, j)) {
            send = true;
            at(s->ntf_in, j) = 0;
        }
        if (send) event(EBB_SPACE_EV_RANGE, j, 0, at(s->ntf_in, j));
    }
    // CheckForProximity_TargetTracking (Ball.cpp:595)
    EBB_HD void check_target_tracking(int64_t j) const {
        const double tr = at(s->trk_range, j);
        const int64_t t = at(s->trk, j);
        if (!(tr >= TRACKING_MIN) || t < 0) return;
        const double lim = dadd(tr, (double)p->radius[row(j)]);
        bool send = false;
        if (dist2_slots(j, t) < dmul(lim, lim)) {
            if (!at(s->trk_in, j)) {
                send = true;
                at(s->trk_in, j) = 1;
            }
        } else if (at(s->trk_in, j)) {
            send = true;
            at(s->trk_in, j) = 0;
        }
        if (send) event(EBB_SPACE_EV_TRACKING, j, 0, at(s->trk_in, j));
    }
    // CheckForProximity_Sensor (Ball.cpp:642; SEN-701, SEN-702): every period, GetNearbyBalls with the sensor's
    // radius inflated and the velocity zeroed (the ball re-filed for it and back), the balls no longer near first (in
    // the list's order), then each candidate in the walk's order entering or leaving (the inside test in float sums)
    // CheckSensor's two re-filings (the ball at its radius plus the sensor's range, velocity zeroed; then back) when
    // they leave no trace but BoxAllocator's kept count. That holds when the ball comes back to the filing it has
    // (the same level, keys and sides) and its top box keeps its bubble, the ball's: the live boxes are then those of
    // every ball's filing, as before; each box's ball and child counts follow from them; no bubble, dictionary or set
    // changes; no released box is read. Conditions, each checked (else false, nothing done): the ball filed, neither
    // filing huge, the world unflagged; the top box's bubble the ball's; the inflated box live and not emptied by the
    // ball's leaving, no top box emptied; the inflated sides inside the grid; room in the table for every box the
    // pair makes; the kept count below 256 throughout (every release kept). Then the pair's boxes are counted, not
    // made: `a` released by the ball's leaving (`a1` of them on its own box's chain, re-made by the second GetBox),
    // `b` made for the inflated sides (released again by the second leaving), and the kept count moves as the pair
    // would move it (+a; -b floored at 0; -a1 floored; +b; -(a - a1) floored). `fi`: the inflated filing, for
    // GetNearbyBalls.
    EBB_HDNI bool sensor_fast(int64_t j, const double* x, const double* v, float inflated, Filing* fi) {
        int64_t a = 0, a1 = 0, ak = 0, b = 0;
        bool same = false;
        if (!sensor_plan(j, x, v, inflated, fi, &a, &a1, &ak, &b, &same, true)) return false;
        if (same) EBB_SENSOR_PATH(2);
        return same || sensor_count(a, a1, ak, b);
    }
    // The kept count as the pair would move it, when every release is kept and the table has room (else false): +a
    // (the leaving's releases), -ak floored at 0 (the inflated box's chain made again), -b floored (its sides), -(a1
    // - ak) floored (the ball's own box's chain below it made again), +b (the sides released), -(a - a1) floored (the
    // ball's own sides made again)
    EBB_HD bool sensor_count(int64_t a, int64_t a1, int64_t ak, int64_t b) {
        if (b < 0) return true;                            // (counted as unchanged: see sensor_plan)
        int64_t c = one(s->free_boxes);
        if (!kept_count(c, B - (one(s->box_n) - one(s->box_free_n)), a, a1, ak, b)) return false;
        one(s->free_boxes) = c;
        return true;
    }
    // (the same on a count held by the caller; `room`: the table's free entries)
    EBB_HD static bool kept_count(int64_t& c, int64_t room, int64_t a, int64_t a1, int64_t ak, int64_t b) {
        if (room < b + ak + 8 || c + a + b >= BOX_KEEP) return false;
        c += a;
        c = c > ak ? c - ak : 0;
        c = c > b ? c - b : 0;
        c = c > a1 - ak ? c - (a1 - ak) : 0;
        c += b;
        c = c > a - a1 ? c - (a - a1) : 0;
        return true;
    }
    // sensor_fast's conditions and counts, nothing written: a, a1, b (b = -1 when the kept count cannot move: at
    // least 56 with room, `shortcut`), `same` when the inflated filing is the ball's own. What bounds it is its chain of
    // dependent loads and, a lane a sensor, its divergence: with a list of the entries touched and one of the boxes made
    // (40 and 24 entries of local memory, scanned at every step) a plan took 133,000 cycles in a 4-ship world, 4/5 of
    // the tick there; as corner sets in registers, with the own boxes known without a lookup, the tick of 16,384
    // 4-ship worlds a thread each went from 2.44 to 1.53 ms with it.
    EBB_HDNI bool sensor_plan(int64_t j, const double* x, const double* v, float inflated, Filing* fi, int64_t* a_out,
                              int64_t* a1_out, int64_t* ak_out, int64_t* b_out, bool* same_out, bool shortcut) const {
        *same_out = false;
        if (lvl(j) < 0 || huge(j) || one(s->flags) != 0) return false;
        const int64_t r = row(j);
        const int64_t box0 = I(s->my_box, j), top = I(s->my_top, j);
        if (box0 < 0 || top < 0) return false;
        const int64_t bub = BX(s->box_bubble, top);
        if (bub == -1 || bub != I(s->bubble, j)) return false;
        // the filing it comes back to: its own (known for a fresh one, else made again and compared)
        const int L1 = (int)lvl(j);
        int64_t k1[3], m1[3];
        for (int c = 0; c < 3; ++c) {
            k1[c] = key(j, c);
            m1[c] = mod(j, c);
        }
        if (!is_fresh(j)) {
            const double infl1 = inflated_radius(j, v);
            if (level_for(infl1) != L1 || (L1 == 0 && (double)fmul(p->radius[r], 2.0f) > level_width(0)))
                return false;
            int64_t kk[3], mm[3];
            key_for(L1, x, kk);
            side_mods(L1, kk, infl1, x, mm);
            for (int c = 0; c < 3; ++c)
                if (kk[c] != k1[c] || mm[c] != m1[c]) return false;
        }
        // the inflated filing
        const double rest[3] = {0.0, 0.0, 0.0};
        const double infl = inflated_radius_of(j, inflated, rest);
        const int Li = level_for(infl);
        if (Li == 0 && (double)fmul(inflated, 2.0f) > level_width(0)) return false;
        int64_t ki[3], mi[3];
        key_for(Li, x, ki);
        side_mods(Li, ki, infl, x, mi);
        fi->L = Li;
        for (int c = 0; c < 3; ++c) {
            fi->lo[c] = ki[c] + (mi[c] < 0 ? mi[c] : 0);
            fi->hi[c] = ki[c] + (mi[c] > 0 ? mi[c] : 0);
        }
        if (Li == L1 && ki[0] == k1[0] && ki[1] == k1[1] && ki[2] == k1[2] && mi[0] == m1[0] && mi[1] == m1[1] &&
            mi[2] == m1[2]) {
            *same_out = true;
            return true;                                   // both re-filings return at once
        }
        const int64_t boxi = box_find(Li, ki[0], ki[1], ki[2]);
        if (boxi < 0) return false;
        // A filing's boxes, and their ancestors at each level above, are a product of one or two keys an axis (the
        // ball's and its side's): a cell of them is a corner, bit q set for the side's key on axis q, bit q clear where
        // the two keys have met at that level (`apart`: the axes still apart). So a set of such cells is 8 bits a level,
        // in registers: no list of entries, no scan of one.
        auto apart = [](const int64_t* k, const int64_t* m, int sh) -> unsigned {
            unsigned on = 0;
            for (int q = 0; q < 3; ++q)
                if ((k[q] >> sh) != ((k[q] + m[q]) >> sh)) on |= 1u << q;
            return on;
        };
        // the boxes the ball's leaving empties, level by level: its own that hold it alone and no child, then each
        // parent whose children all went and that holds no ball (`gone`: their corners, 8 bits a level)
        const unsigned sides1 = apart(k1, m1, 0);
        int32_t ent[8];
        uint64_t gone = 0;
        int64_t a = 0;
        unsigned g1 = 0;
        for (unsigned c = 0; c < 8; ++c) {
            if (c & ~sides1) continue;
            const int64_t e = fbox(j, (int)c);
            if (e < 0) return false;
            ent[c] = (int32_t)e;
            if (BX(s->box_balls, e) == 1 && BX(s->box_kids, e) == 0) g1 |= 1u << c;
        }
        for (int L = L1; g1 != 0; --L) {
            gone |= (uint64_t)g1 << (8 * L);
            if (L == 0) {
                for (unsigned c = 0; c < 8; ++c)
                    if ((g1 >> c) & 1) {
                        ++a;
                        if (ent[c] != top) return false;   // another top box emptied: its bubble lost
                    }
                break;
            }
            const unsigned keep = apart(k1, m1, 2 * (L1 - L + 1));
            unsigned up = 0, met = 0;
            for (unsigned c = 0; c < 8; ++c) {
                if (!((g1 >> c) & 1)) continue;
                ++a;
                const unsigned q = c & keep;
                if ((met >> q) & 1) continue;
                met |= 1u << q;
                int64_t kids = 0;
                for (unsigned d = c; d < 8; ++d) kids += ((g1 >> d) & 1) && (d & keep) == q;
                const int64_t e = BX(s->box_parent, ent[c]);
                if (e < 0) continue;
                ent[q] = (int32_t)e;                       // (q <= c: the corners still to come keep theirs)
                if (BX(s->box_balls, e) == 0 && BX(s->box_kids, e) == kids) up |= 1u << q;
            }
            g1 = up;
        }
        // the corner of a cell among the own boxes and their ancestors, or 8
        auto own_corner = [&](int L, int64_t kx, int64_t ky, int64_t kz) -> unsigned {
            if (L > L1) return 8;
            const int64_t k[3] = {kx, ky, kz};
            const int sh = 2 * (L1 - L);
            unsigned c = 0;
            for (int q = 0; q < 3; ++q) {
                if (k[q] == (k1[q] >> sh)) continue;
                if (k[q] != ((k1[q] + m1[q]) >> sh)) return 8;
                c |= 1u << q;
            }
            return c;
        };
        int64_t a1 = 0;                                    // the ball's own box's chain
        for (int L = L1; L >= 0 && ((gone >> (8 * L)) & 1); --L) ++a1;
        // the inflated box emptied: its chain up to a live box made again at once by the inflated filing's GetBox, before
        // the sides, with the top box's bubble set (`gone` keeps the boxes released and not made again)
        int64_t ak = 0;
        for (int L = Li; L >= 0; --L) {
            const int sh = 2 * (Li - L);
            const unsigned c = own_corner(L, ki[0] >> sh, ki[1] >> sh, ki[2] >> sh);
            if (c == 8 || !((gone >> (8 * L + c)) & 1)) break;
            gone &= ~(uint64_t(1) << (8 * L + c));
            ++ak;
        }
        if (ak > 0 && Li == L1) return false;             // (the ball's own box emptied, made again, emptied again)
        const int64_t g = level_grid(Li);
        for (int c = 0; c < 3; ++c)                        // the inflated sides inside the grid
            if (ki[c] + mi[c] < 0 || ki[c] + mi[c] >= g) return false;
        *a_out = a;
        *a1_out = a1;
        *ak_out = ak;
        *b_out = -1;
        const int64_t live = one(s->box_n) - one(s->box_free_n);
        const int64_t c0 = one(s->free_boxes);
        // at most 56 boxes made for the sides (7 chains of 8 levels): with the kept count at least that, and room for
        // them, every making takes one off it and every release puts one back (kept below 256): it ends as it began
        if (shortcut && ak == 0 && c0 >= 56 && c0 + a + 56 < BOX_KEEP && B - live >= 64) return true;
        // else the boxes the inflated sides make, counted level by level: the sides' cells that are missing, then the
        // missing ones' parents (corner 0's chain, the inflated box's, is live). An own box or an ancestor of one is in
        // the table, so only a cell beside them takes a lookup.
        int64_t b = 0;
        unsigned want = 0;
        const unsigned sidesi = apart(ki, mi, 0);
        for (unsigned c = 1; c < 8; ++c)
            if (!(c & ~sidesi)) want |= 1u << c;
        for (int L = Li; L >= 0 && want; --L) {
            const int sh = 2 * (Li - L);
            const unsigned keep = L > 0 ? apart(ki, mi, sh + 2) : 0;
            unsigned up = 0;
            while (want) {
                unsigned c = 0;
                while (!((want >> c) & 1)) ++c;
                want &= want - 1;
                const int64_t kx = (ki[0] + ((c & 1) ? mi[0] : 0)) >> sh, ky = (ki[1] + ((c & 2) ? mi[1] : 0)) >> sh,
                              kz = (ki[2] + ((c & 4) ? mi[2] : 0)) >> sh;
                const unsigned o = own_corner(L, kx, ky, kz);
                const bool have = o < 8 ? !((gone >> (8 * L + o)) & 1) : box_find(L, kx, ky, kz) >= 0;
                if (have) continue;
                ++b;
                up |= 1u << (c & keep);
            }
            want = up & ~1u;
        }
        *b_out = b;
        return true;
    }
    EBB_HDNI void check_sensor(int64_t j) {
        at(s->selapsed, j) = dadd(at(s->selapsed, j), p->dt);
        if (at(s->selapsed, j) < at(s->speriod, j)) return;
        at(s->selapsed, j) = 0.0;
        check_sensor_body(j);
    }
    // the check itself, its period come
    EBB_HDNI void check_sensor_body(int64_t j) {
        const int64_t r = row(j);
        const float radius = p->radius[r];
        const double x[3] = {pos(j, 0), pos(j, 1), pos(j, 2)};
        const double v[3] = {vel(j, 0), vel(j, 1), vel(j, 2)};
        const double rest[3] = {0.0, 0.0, 0.0};
        const float inflated = fadd(radius, (float)at(s->srange, j));
        uint8_t cand[EBB_SPACE_MAX_SLOTS];
        int nc;
        Filing fi;
        EBB_SENSOR_PATH(0);
        if (!(inflated < 0.0f) && !(radius < 0.0f) && sensor_fast(j, x, v, inflated, &fi)) {
            EBB_SENSOR_PATH(1);
            nc = nearby(j, at(s->cloaked, j) == 0, at(s->sonly, j) != 0, false, cand, &fi);
        } else {
            if (!(inflated < 0.0f)) {
                p->radius[r] = inflated;
                insert_in_boxes(j, x, rest);
            }
            nc = nearby(j, at(s->cloaked, j) == 0, at(s->sonly, j) != 0, false, cand);
            set_fresh(j, false);
            if (!(radius < 0.0f)) {
                p->radius[r] = radius;
                insert_in_boxes(j, x, v);
                set_fresh(j, true);
            }
        }
#ifdef __CUDA_ARCH__
        if constexpr (COOP) {
            sensor_events_warp(j, r, cand, nc);
        } else
#endif
        {
            sensor_events_serial(j, r, cand, nc);
        }
    }
    // check_sensor's events by a single thread: the list's balls no longer near leave in its order, then each
    // candidate enters or leaves in the walk's order
    EBB_HDNI void sensor_events_serial(int64_t j, int64_t r, const uint8_t* cand, int nc) const {
        const UMap m = sensor_map(j);
        if (*m.len > 0) {
            uint64_t near[2] = {0, 0};
            for (int i = 0; i < nc; ++i) near[cand[i] >> 6] |= uint64_t(1) << (cand[i] & 63);
            uint8_t keys[EBB_SPACE_MAX_SLOTS];
            const int32_t n0 = *m.len;
            for (int32_t e = 0; e < n0; ++e) keys[e] = m.k[e * m.step];
            for (int32_t e = 0; e < n0; ++e) {
                const int64_t k = keys[e];
                if (k == j || ((near[k >> 6] >> (k & 63)) & 1)) continue;
                umap_erase(m, k);
                event(EBB_SPACE_EV_PROXIMITY, j, k, 0);
                if (!p->sensor[r]) break;
            }
        }
        const float range = (float)at(s->srange, j);
        for (int i = 0; i < nc; ++i) {
            const int64_t o = cand[i];
            if (o == j) continue;
            const bool inside = umap_has(m, o);
            const double ck = (double)fadd(fadd(range, p->radius[row(o)]), p->radius[r]);
            if (dist2_slots(j, o) > dmul(ck, ck)) {
                if (inside) {
                    umap_erase(m, o);
                    event(EBB_SPACE_EV_PROXIMITY, j, o, 0);
                }
            } else if (!inside) {
                umap_insert(m, o, F_SENSOR_LIST);
                event(EBB_SPACE_EV_PROXIMITY, j, o, 1);
            }
            if (!p->sensor[r]) break;
        }
    }
#ifdef __CUDA_ARCH__
    // check_sensor's events in a warp: the lanes read the list's keys and test 32 of them (then 32 candidates) at a
    // time, a ballot naming the ones that change; those are applied one after another in their order, every lane
    // together (a candidate's membership is its own: the changes before it leave it as it was)
    __device__ void sensor_events_warp(int64_t j, int64_t r, const uint8_t* cand, int nc) {
        const UMap m = sensor_map(j);
        uint64_t near[2] = {0, 0};
        for (int i = 0; i < nc; ++i) near[cand[i] >> 6] |= uint64_t(1) << (cand[i] & 63);
        const int32_t n0 = *m.len;
        if (n0 > 0) {
            uint8_t* keys = sh->out;
            for (int32_t e = lane; e < n0; e += 32) keys[e] = m.k[e * m.step];
            __syncwarp();
            for (int32_t base = 0; base < n0; base += 32) {
                bool gone = false;
                if (base + lane < n0) {
                    const int64_t k = keys[base + lane];
                    gone = k != j && !((near[k >> 6] >> (k & 63)) & 1);
                }
                unsigned bits = __ballot_sync(0xffffffffu, gone);
                while (bits) {
                    const int b = __ffs(bits) - 1;
                    bits &= bits - 1;
                    const int64_t k = keys[base + b];
                    umap_erase(m, k);
                    event(EBB_SPACE_EV_PROXIMITY, j, k, 0);
                }
            }
            __syncwarp();
        }
        const float range = (float)at(s->srange, j), rb = p->radius[r];
        const double xj[3] = {pos(j, 0), pos(j, 1), pos(j, 2)};
        for (int base = 0; base < nc; base += 32) {
            int act = 0;                                  // 1 enters, 2 leaves
            if (base + lane < nc) {
                const int64_t o = cand[base + lane];
                if (o != j) {
                    const bool inside = umap_has(m, o);
                    const double ck = (double)fadd(fadd(range, p->radius[row(o)]), rb);
                    const double d0 = dsub(xj[0], pos(o, 0)), d1 = dsub(xj[1], pos(o, 1)), d2 = dsub(xj[2], pos(o, 2));
                    const double len2 = dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
                    if (len2 > dmul(ck, ck)) {
                        if (inside) act = 2;
                    } else if (!inside) {
                        act = 1;
                    }
                }
            }
            unsigned bits = __ballot_sync(0xffffffffu, act != 0);
            const unsigned enter = __ballot_sync(0xffffffffu, act == 1);
            while (bits) {
                const int b = __ffs(bits) - 1;
                bits &= bits - 1;
                const int64_t o = cand[base + b];
                if ((enter >> b) & 1) {
                    umap_insert(m, o, F_SENSOR_LIST);
                    event(EBB_SPACE_EV_PROXIMITY, j, o, 1);
                } else {
                    umap_erase(m, o);
                    event(EBB_SPACE_EV_PROXIMITY, j, o, 0);
                }
            }
        }
    }
#endif
#ifdef __CUDA_ARCH__
    // HandleProximities in a warp, 32 sensors at a time: each lane computes one sensor's check ahead (the fast path's
    // plan, without writing), the lanes together find every sensor's candidates and those in range as slot sets
    // (scan_batch), then the warp takes the map's balls in order as one ball does, using a sensor's ahead-computed check
    // while nothing it read has changed: the world unflagged and no ball's filing or bubble changed by an earlier check's
    // re-filings (then the balls after it are computed ahead again). The kept count moves in the map's order. A 128-slot
    // world's tick, in cycles: the plans 0.88 -> 0.48 million, the candidates 1.17 -> 0.36, the walk 0.92 -> 0.14, the
    // tick's order and moved balls 0.22 -> 0.02 (8,000 partition worlds 10.2 -> 6.4 ms a tick).
    struct Pre {
        int64_t a, a1, ak, b;
        Filing fi;
        uint64_t cand[2], in[2];
        int ok;                                            // 0 none; 1 the fast path's plan; 2 and the filing the ball's own
    };
    // sensor j's plan, and its row for the scan
    __device__ void pre_sensor(int64_t j, Pre& pr, SensorRow* row_out) const {
        const int64_t r = row(j);
        const float radius = p->radius[r];
        const float range = (float)at(s->srange, j);
        const float inflated = fadd(radius, range);
        if (inflated < 0.0f || radius < 0.0f) return;
        const double x[3] = {pos(j, 0), pos(j, 1), pos(j, 2)};
        const double v[3] = {vel(j, 0), vel(j, 1), vel(j, 2)};
        bool same = false;
        if (!sensor_plan(j, x, v, inflated, &pr.fi, &pr.a, &pr.a1, &pr.ak, &pr.b, &same, false)) return;
        pr.ok = same ? 2 : 1;
        const int64_t bub = I(s->bubble, j);
        const bool excl_fixed = at(s->cloaked, j) == 0, excl_inert = at(s->sonly, j) != 0;
        if (excl_inert && !set_any(0, bub)) return;       // (no candidates)
        const int sh = 2 * (NUM_LEVELS - 1 - (int)pr.fi.L);
        for (int q = 0; q < 3; ++q) {
            row_out->lo[q] = pr.fi.lo[q] << sh;
            row_out->hi[q] = ((pr.fi.hi[q] + 1) << sh) - 1;
            row_out->x[q] = x[q];
        }
        row_out->bub = bub;
        row_out->range = range;
        row_out->radius = radius;
        row_out->how = 1 | (excl_fixed ? 2 : 0) | (excl_inert ? 4 : 0) | ((int32_t)j << 8);
    }
    // The batch's candidates and those in range: a lane a slot, its filing, position and filters in registers, against
    // every sensor of the batch (its row a broadcast from shared memory); two ballots a sensor are its sets' words.
    // A lane a sensor instead, walking the slots, spent 4,100 cycles a slot on the slot's dependent loads (three
    // quarters of the check's time in a 128-slot world). Relatedness (related): in the deepest level's units a key
    // range is the interval of the cells it covers, and the finer range shifted up meets the coarser's exactly when
    // the intervals meet.
    __device__ void scan_batch(Pre& mine, unsigned sensors) const {
        uint32_t cw[4] = {0, 0, 0, 0}, iw[4] = {0, 0, 0, 0};
        const int S = occupied < N ? occupied : (int)N;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (32 * q >= S) break;
            const int64_t o = 32 * q + lane;
            bool ok = o < S && slot_ok(o) && U(s->in_park, o) && lvl(o) >= 0;
            int64_t lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0}, bub = 0;
            double x[3] = {0.0, 0.0, 0.0};
            float radius = 0.0f;
            bool free_o = false, inter = false;
            if (ok) {
                const Filing f = filing_of(o);
                const int sh = 2 * (NUM_LEVELS - 1 - (int)f.L);
                const int64_t ro = row(o);
                for (int c = 0; c < 3; ++c) {
                    lo[c] = f.lo[c] << sh;
                    hi[c] = ((f.hi[c] + 1) << sh) - 1;
                    x[c] = pos(o, c);
                }
                bub = I(s->bubble, o);
                radius = p->radius[ro];
                free_o = p->free_[ro] != 0;
                inter = p->interactive[ro] != 0;
            }
            for (unsigned left = sensors; left; left &= left - 1) {
                const int i = __ffs(left) - 1;
                const SensorRow& t = sh->row[i];
                const int how = t.how;
                bool c = ok && (how >> 8) != (int)o && ((how & 4) ? inter : (t.bub == bub && (free_o || !(how & 2))));
                c = c && t.lo[0] <= hi[0] && lo[0] <= t.hi[0] && t.lo[1] <= hi[1] && lo[1] <= t.hi[1] &&
                    t.lo[2] <= hi[2] && lo[2] <= t.hi[2];
                const unsigned cb = __ballot_sync(0xffffffffu, c);
                unsigned ib = 0;
                if (cb) {
                    const double ck = (double)fadd(fadd(t.range, radius), t.radius);
                    const double d0 = dsub(t.x[0], x[0]), d1 = dsub(t.x[1], x[1]), d2 = dsub(t.x[2], x[2]);
                    const double len2 = dadd(dadd(dmul(d0, d0), dmul(d1, d1)), dmul(d2, d2));
                    ib = __ballot_sync(0xffffffffu, c && !(len2 > dmul(ck, ck)));
                }
                if (lane == i) {
                    cw[q] = cb;
                    iw[q] = ib;
                }
            }
        }
        mine.cand[0] = (uint64_t)cw[0] | ((uint64_t)cw[1] << 32);
        mine.cand[1] = (uint64_t)cw[2] | ((uint64_t)cw[3] << 32);
        mine.in[0] = (uint64_t)iw[0] | ((uint64_t)iw[1] << 32);
        mine.in[1] = (uint64_t)iw[2] | ((uint64_t)iw[3] << 32);
    }
    __device__ static Pre pre_of(const Pre& mine, int i) {
        Pre o;
        o.a = __shfl_sync(0xffffffffu, mine.a, i);
        o.a1 = __shfl_sync(0xffffffffu, mine.a1, i);
        o.ak = __shfl_sync(0xffffffffu, mine.ak, i);
        o.b = __shfl_sync(0xffffffffu, mine.b, i);
        o.fi.L = __shfl_sync(0xffffffffu, mine.fi.L, i);
        for (int c = 0; c < 3; ++c) {
            o.fi.lo[c] = __shfl_sync(0xffffffffu, mine.fi.lo[c], i);
            o.fi.hi[c] = __shfl_sync(0xffffffffu, mine.fi.hi[c], i);
        }
        for (int q = 0; q < 2; ++q) {
            o.cand[q] = __shfl_sync(0xffffffffu, mine.cand[q], i);
            o.in[q] = __shfl_sync(0xffffffffu, mine.in[q], i);
        }
        o.ok = __shfl_sync(0xffffffffu, mine.ok, i);
        return o;
    }
    // a sensor's events from its ahead-computed sets: the list's balls no longer candidates leave in the list's order;
    // the candidates whose membership changes enter or leave in the walk's order (their keys made and sorted here)
    __device__ void sensor_events_pre(int64_t j, const Pre& pr) {
        const UMap m = sensor_map(j);
        const int32_t n0 = *m.len;
        if (n0 > 0) {
            uint8_t* keys = sh->out;
            for (int32_t e = lane; e < n0; e += 32) keys[e] = m.k[e * m.step];
            __syncwarp();
            for (int32_t base = 0; base < n0; base += 32) {
                bool gone = false;
                if (base + lane < n0) {
                    const int64_t k = keys[base + lane];
                    gone = k != j && !((pr.cand[k >> 6] >> (k & 63)) & 1);
                }
                unsigned bits = __ballot_sync(0xffffffffu, gone);
                while (bits) {
                    const int b = __ffs(bits) - 1;
                    bits &= bits - 1;
                    const int64_t k = keys[base + b];
                    umap_erase(m, k);
                    event(EBB_SPACE_EV_PROXIMITY, j, k, 0);
                }
            }
            __syncwarp();
        }
        const uint64_t ch[2] = {pr.cand[0] & (pr.in[0] ^ m.m[0]), pr.cand[1] & (pr.in[1] ^ m.m[m.mstep])};
        if ((ch[0] | ch[1]) == 0) return;
        int n = 0;
        for (int base = 0; base < EBB_SPACE_MAX_SLOTS; base += 32) {
            const int o = base + lane;
            const bool is = ((ch[o >> 6] >> (o & 63)) & 1) != 0;
            const unsigned in = __ballot_sync(0xffffffffu, is);
            if (is) {
                const int at_ = n + __popc(in & ((1u << lane) - 1u));
                sh->key[at_] = walk_key(pr.fi, o);
                sh->id[at_] = id(o);
                sh->out[at_] = (uint8_t)o;
            }
            n += __popc(in);
        }
        int P = 1;
        while (P < n) P <<= 1;
        for (int e = n + lane; e < P; e += 32) {
            sh->key[e] = NOT_A_CANDIDATE;
            sh->id[e] = INT64_MAX;
        }
        __syncwarp();
        warp_sort(P);
        for (int i = 0; i < n; ++i) {
            const int64_t o = sh->out[i];
            if ((pr.in[o >> 6] >> (o & 63)) & 1) {
                umap_insert(m, o, F_SENSOR_LIST);
                event(EBB_SPACE_EV_PROXIMITY, j, o, 1);
            } else {
                umap_erase(m, o);
                event(EBB_SPACE_EV_PROXIMITY, j, o, 0);
            }
        }
        __syncwarp();
    }
    // CheckSensor at the ball's turn with its ahead-computed check (else as it runs alone; `dirty` when that
    // changed the ball's filing or bubble)
    __device__ void check_sensor_pre(int64_t j, const Pre& pr, bool& dirty) {
        at(s->selapsed, j) = dadd(at(s->selapsed, j), p->dt);
        if (at(s->selapsed, j) < at(s->speriod, j)) return;
        at(s->selapsed, j) = 0.0;
        if (pr.ok && one(s->flags) == 0 && (pr.ok == 2 || sensor_count(pr.a, pr.a1, pr.ak, pr.b))) {
            EBB_SENSOR_PATH(0);
            EBB_SENSOR_PATH(1);
            if (pr.ok == 2) EBB_SENSOR_PATH(2);
            sensor_events_pre(j, pr);
            return;
        }
        const int64_t l0 = lvl(j), k0 = key(j, 0), k1 = key(j, 1), k2 = key(j, 2), m0 = mod(j, 0), m1 = mod(j, 1),
                      m2 = mod(j, 2), a0 = active(j), b0 = I(s->bubble, j);
        check_sensor_body(j);
        if (lvl(j) != l0 || key(j, 0) != k0 || key(j, 1) != k1 || key(j, 2) != k2 || mod(j, 0) != m0 ||
            mod(j, 1) != m1 || mod(j, 2) != m2 || active(j) != a0 || I(s->bubble, j) != b0)
            dirty = true;
    }
    // The proximity balls in the map's order, its entries 32 q + lane in this lane's byte q of `keys`. Most checks change
    // nothing but the elapsed time and the kept count ("quiet": no notification range or tracking, the sensor's period
    // come or not, the ahead-computed sets equal to its list): the lanes find those at once, and the warp's walk over
    // the order only moves the kept count by each (its four terms packed in a word, at most 64 each); the others are
    // taken whole at their turn.
    __device__ void handle_proximities_warp(uint32_t keys, int32_t n) {
        int32_t batch = 0;
        while (batch < n) {
            Pre mine;
            mine.ok = 0;
            mine.a = mine.a1 = mine.ak = mine.b = 0;
            mine.fi = Filing{};
            const int e_mine = batch + lane;
            int64_t j_mine = -1;
            {
                const uint32_t k = __shfl_sync(0xffffffffu, keys, e_mine & 31);   // (a batch may start anywhere)
                if (e_mine < n) j_mine = (k >> (8 * (e_mine >> 5))) & 255;
            }
            sh->row[lane].how = 0;
            const bool live = j_mine >= 0 && slot_ok(j_mine) && U(s->in_park, j_mine);
            const bool senses = live && p->sensor[row(j_mine)];
            if (senses) pre_sensor(j_mine, mine, &sh->row[lane]);
            __syncwarp();
            scan_batch(mine, __ballot_sync(0xffffffffu, sh->row[lane].how & 1));
            // 0: taken whole at its turn; 1: not due; 2: due, no event
            int quiet = 0;
            double elapsed = 0.0;
            if (senses && at(s->has_prox, j_mine) && at(s->ntf_range, j_mine) == 0.0 &&
                !(at(s->trk_range, j_mine) >= TRACKING_MIN && at(s->trk, j_mine) >= 0) && !in_dead_bubble(j_mine)) {
                elapsed = dadd(at(s->selapsed, j_mine), p->dt);
                if (elapsed < at(s->speriod, j_mine)) {
                    quiet = 1;
                } else if (mine.ok) {
                    elapsed = 0.0;
                    const UMap m = sensor_map(j_mine);
                    const uint64_t m0 = m.m[0], m1 = m.m[m.mstep];
                    const uint64_t self0 = j_mine < 64 ? uint64_t(1) << j_mine : 0,
                                   self1 = j_mine < 64 ? 0 : uint64_t(1) << (j_mine - 64);
                    if (((m0 & ~mine.cand[0] & ~self0) | (m1 & ~mine.cand[1] & ~self1) |
                         (mine.cand[0] & (mine.in[0] ^ m0)) | (mine.cand[1] & (mine.in[1] ^ m1))) == 0)
                        quiet = 2;
                }
            }
            const unsigned not_due = __ballot_sync(0xffffffffu, quiet == 1), calm = __ballot_sync(0xffffffffu, quiet == 2),
                           same = __ballot_sync(0xffffffffu, mine.ok == 2);
            const uint32_t terms = (uint32_t)mine.a | ((uint32_t)mine.a1 << 8) | ((uint32_t)mine.ak << 16) |
                                   ((uint32_t)(mine.b & 255) << 24);
            __syncwarp();
            unsigned taken = 0;                            // the quiet ones passed at their turn
            bool dirty = false;
            const int32_t end = n < batch + 32 ? n : batch + 32;
            int32_t e = batch;
            while (e < end && !dirty) {
                // a run of quiet balls, the kept count in a register
                const int i0 = e - batch;
                if (((not_due | calm) >> i0) & 1) {
                    const bool unflagged = one(s->flags) == 0;
                    const int64_t room = B - (one(s->box_n) - one(s->box_free_n));
                    const int64_t c0 = one(s->free_boxes);
                    int64_t c = c0;
                    bool stop = false;
                    while (e < end && !stop) {
                        const int i = e - batch;
                        if ((not_due >> i) & 1) {
                            taken |= 1u << i;
                            ++e;
                            continue;
                        }
                        if (!((calm >> i) & 1)) break;
                        if (!unflagged) {
                            stop = true;
                            break;
                        }
                        if (!((same >> i) & 1)) {
                            const uint32_t t = __shfl_sync(0xffffffffu, terms, i);
                            const int64_t a = t & 255, a1 = (t >> 8) & 255, ak = (t >> 16) & 255, b = t >> 24;
                            if (!kept_count(c, room, a, a1, ak, b)) {
                                stop = true;
                                break;
                            }
                        } else {
                            EBB_SENSOR_PATH(2);
                        }
                        EBB_SENSOR_PATH(0);
                        EBB_SENSOR_PATH(1);
                        taken |= 1u << i;
                        ++e;
                    }
                    if (c != c0) one(s->free_boxes) = c;
                    if (!stop) continue;
                }
                const Pre pr = pre_of(mine, e - batch);
                const int64_t j = __shfl_sync(0xffffffffu, j_mine, e - batch);
                ++e;
                if (!slot_ok(j) || !U(s->in_park, j)) continue;
                if (in_dead_bubble(j)) {
                    if (at(s->slen, j) > 0) {
                        at(s->selapsed, j) = at(s->speriod, j);
                        check_notification_range(j);
                        check_target_tracking(j);
                        if (p->sensor[row(j)]) check_sensor_pre(j, pr, dirty);
                    }
                    umap_clear(sensor_map(j));
                    continue;
                }
                if (!at(s->has_prox, j)) continue;
                check_notification_range(j);
                check_target_tracking(j);
                if (p->sensor[row(j)]) check_sensor_pre(j, pr, dirty);
            }
            if ((taken >> lane) & 1) at(s->selapsed, j_mine) = elapsed;
            __syncwarp();
            batch = e;
        }
    }
#endif
    EBB_HD void check_for_proximity(int64_t j) {
        check_notification_range(j);
        check_target_tracking(j);
        if (p->sensor[row(j)]) check_sensor(j);
    }
    // Ballpark::HandleProximities (Ballpark.cpp:5822): every proximity ball in the map's order (a copy of it); a ball
    // in a dead bubble gets one forced check when its sensor holds balls, and its list is emptied (TIME-714)
    EBB_HDNI void handle_proximities() {
        const UMap pm = proximity_map();
        const int32_t n = *pm.len;
#ifdef __CUDA_ARCH__
        if constexpr (COOP) {
            uint32_t keys = 0;
            for (int q = 0; q < 4; ++q)
                if (32 * q + lane < n) keys |= (uint32_t)pm.k[(32 * q + lane) * pm.step] << (8 * q);
            handle_proximities_warp(keys, n);
        } else
#endif
        {
            uint8_t keys[EBB_SPACE_MAX_SLOTS];
            for (int32_t e = 0; e < n; ++e) keys[e] = pm.k[e * pm.step];
            for (int32_t e = 0; e < n; ++e) {
                const int64_t j = keys[e];
                if (!slot_ok(j) || !U(s->in_park, j)) continue;
                if (in_dead_bubble(j)) {
                    if (at(s->slen, j) > 0) {
                        at(s->selapsed, j) = at(s->speriod, j);
                        check_for_proximity(j);
                    }
                    umap_clear(sensor_map(j));
                    continue;
                }
                if (!at(s->has_prox, j)) continue;
                check_for_proximity(j);
            }
        }
    }

    // ---- the queries (space.py:1524-1600: CheckVisibility, GetBallIdsInRange, GetBubbleAtCoordinates) ----
    // the slot of a ball of the world by id, -1 for none
    EBB_HD int64_t slot_of(int64_t bid) const {
        for (int64_t j = 0; j < N; ++j)
            if (slot_ok(j) && U(s->in_park, j) && id(j) == bid) return j;
        return -1;
    }
    // Ballpark::CheckVisibility (Ballpark.cpp:5299; SEN-709): -2 between bubbles (or a ball missing); else the first
    // massive, uncloaked ball of the bubble, in the ball dictionary's order, whose sphere the segment enters; else 0
    EBB_HDNI int64_t visibility(int64_t src, int64_t dst) const {
        if (!slot_ok(src) || !slot_ok(dst) || !U(s->in_park, src) || !U(s->in_park, dst)) return -2;
        if (I(s->bubble, src) != I(s->bubble, dst)) return -2;
        const double x0[3] = {pos(src, 0), pos(src, 1), pos(src, 2)};
        double ray[3] = {dsub(pos(dst, 0), x0[0]), dsub(pos(dst, 1), x0[1]), dsub(pos(dst, 2), x0[2])};
        const double len2 = dadd(dadd(dmul(ray[0], ray[0]), dmul(ray[1], ray[1])), dmul(ray[2], ray[2]));
        const double distance = dsqrt(len2), norm = dsqrt(len2);
        if (norm != 0.0) {
            const double inv = ddiv(1.0, norm);
            for (int c = 0; c < 3; ++c) ray[c] = dmul(ray[c], inv);
        }
        int64_t last = -1;
        for (int64_t t = 0; t < N; ++t) {                  // the balls in the order they were added
            int64_t o = -1;
            for (int64_t i = 0; i < N; ++i)
                if (U(s->in_park, i) && slot_ok(i) && I(s->seq, i) > last && (o < 0 || I(s->seq, i) < I(s->seq, o)))
                    o = i;
            if (o < 0) break;
            last = I(s->seq, o);
            const int64_t r = row(o);
            if (I(s->bubble, o) != I(s->bubble, src) || o == src || o == dst || !p->massive[r] ||
                at(s->cloaked, o) != 0)
                continue;
            const double tc[3] = {dsub(pos(o, 0), x0[0]), dsub(pos(o, 1), x0[1]), dsub(pos(o, 2), x0[2])};
            const double v = dadd(dadd(dmul(ray[0], tc[0]), dmul(ray[1], tc[1])), dmul(ray[2], tc[2]));
            const double rad = (double)p->radius[r];
            const double tt = dadd(dadd(dmul(tc[0], tc[0]), dmul(tc[1], tc[1])), dmul(tc[2], tc[2]));
            const double dsq = dsub(dmul(rad, rad), dsub(tt, dmul(v, v)));
            if (dsq < 0.0) continue;
            const double d = dsqrt(dsq);
            const double near = dsub(v, d);
            if (near > 0.0 && near < distance) return id(o);
        }
        return 0;
    }
    // GetBubbleAtCoordinates: the bubble of the existing top box holding the point, -2 for none
    EBB_HD int64_t bubble_at(const double* x) const {
        int64_t k[3];
        key_for(0, x, k);
        const int64_t e = check_box(k[0], k[1], k[2], 0);
        return e < 0 ? -2 : BX(s->box_bubble, e);
    }
    // GetBallIdsInRange (with distances): the balls listed in the bubble's dictionary, in its order (those that left
    // it included until CopyBubbles), within range + radius of the centre; the reference ball itself left out
    EBB_HDNI int64_t in_range(int64_t ref, const double* c, int64_t bub, double range, bool cloaked, int64_t* out,
                            double* outd) const {
        if (bub == -1 || dict_index(bub) < 0) return 0;
        int64_t n = 0;
        const int64_t en = one(s->entry_n);
        for (int64_t e = 0; e < en; ++e) {
            if (I(s->entry_bubble, e) != bub) continue;
            const int64_t o = slot_of(I(s->entry_id, e));
            if (o < 0 || o == ref) continue;
            if (at(s->cloaked, o) != 0 && !cloaked) continue;
            const double d2 = dist2(o, c);
            const double lim = dadd(range, (double)p->radius[row(o)]);
            if (d2 <= dmul(lim, lim)) {
                out[n * W + w] = id(o);
                outd[n * W + w] = d2;
                ++n;
            }
        }
        return n;
    }
    // One query of the world (EbbSpaceQuery): its answer in out[0][w], the balls' ids in out[1 + i][w], their
    // squared distances in outd[i][w]
    EBB_HD void query(int64_t kind, int64_t a, int64_t b, const double* f, int64_t* out, double* outd) {
        int64_t* ids = out + W;
        switch (kind) {
            case EBB_SPACE_Q_VISIBILITY: out[w] = visibility(a, b); break;
            case EBB_SPACE_Q_RANGE_BALL:
                if (!slot_ok(a) || !U(s->in_park, a)) {
                    out[w] = -1;
                } else {
                    const double c[3] = {pos(a, 0), pos(a, 1), pos(a, 2)};
                    out[w] = in_range(a, c, I(s->bubble, a), f[0], (b & 1) != 0, ids, outd);
                }
                break;
            case EBB_SPACE_Q_RANGE_POINT: {
                const int64_t top = bubble_at(f);
                out[w] = in_range(-1, f, top == -2 ? -1 : top, f[3], (b & 1) != 0, ids, outd);
                break;
            }
            case EBB_SPACE_Q_BUBBLE_AT: out[w] = bubble_at(f); break;
            case EBB_SPACE_Q_NEARBY: {
                if (!slot_ok(a) || !U(s->in_park, a)) {
                    out[w] = 0;
                    break;
                }
                uint8_t cand[EBB_SPACE_MAX_SLOTS];
                const int n = nearby(a, (b & 1) != 0, (b & 2) != 0, (b & 4) != 0, cand);
                for (int i = 0; i < n; ++i) ids[(int64_t)i * W + w] = id(cand[i]);
                out[w] = n;
                break;
            }
            default: flag(F_BAD_OP); break;
        }
    }

    // ---- the operations ----
    EBB_HD bool slot_ok(int64_t j) const { return j >= 0 && j < N && row(j) >= 0 && row(j) < p->n; }
    EBB_HD void add(int64_t j) {                           // AddBall's filing (a ball already in: re-filed)
        if (U(s->in_park, j)) {
            delete_from_boxes(j);
        } else {                                           // a new ball: last in the ball dictionary's order
            I(s->seq, j) = one(s->seq_next)++;
            I(s->bubble, j) = -1;
            I(s->old_bubble, j) = -1;
            clear_filing(j);
            reset_sensors(j);
        }
        U(s->in_park, j) = 1;
        insert_in_boxes(j);
    }
    EBB_HD void remove(int64_t j) {                        // RemoveBall outside Evolve: its boxes and bubble left
        if (!U(s->in_park, j)) return;
        delete_from_boxes(j);
        I(s->old_bubble, j) = I(s->bubble, j);
        I(s->bubble, j) = -1;
        add_to_bubble(j);
        if (at(s->has_prox, j)) umap_erase(proximity_map(), j);
        U(s->in_park, j) = 0;
    }
    EBB_HD void set_interactive(int64_t j, bool on) {
        const int64_t r = row(j);
        if (on && !p->interactive[r]) {
            p->interactive[r] = 1;
            if (I(s->bubble, j) != -1) set_insert(0, I(s->bubble, j), id(j));
        } else if (!on && p->interactive[r]) {
            if (I(s->bubble, j) != -1) set_erase(0, I(s->bubble, j), id(j));
            p->interactive[r] = 0;
        }
    }
    // InitializeBubbles: every top box's bubble cleared, the dictionaries and sets emptied, then each ball's top
    // given its bubble (a fill from the first ball to reach it) in the ball dictionary's order
    EBB_HDNI void init_bubbles() {
        const int64_t n = one(s->box_n);
        for (int64_t e = 0; e < n; ++e)
            if (BX(s->box_level, e) == 0) BX(s->box_bubble, e) = -1;
        one(s->bubble_id) = 0;
        one(s->dict_n) = 0;
        one(s->entry_n) = 0;
        one(s->inter_n) = 0;
        one(s->keep_n) = 0;
        for (int64_t j = 0; j < N; ++j) U(s->keep_alive, j) = 0;
        int64_t last = -1;
        for (int64_t t = 0; t < N; ++t) {                  // the slots in the order their balls were added
            int64_t j = -1;
            for (int64_t i = 0; i < N; ++i)
                if (U(s->in_park, i) && I(s->seq, i) > last && (j < 0 || I(s->seq, i) < I(s->seq, j))) j = i;
            if (j < 0) break;
            last = I(s->seq, j);
            if (lvl(j) < 0) {
                I(s->old_bubble, j) = I(s->bubble, j);
                I(s->bubble, j) = -1;
                continue;
            }
            const int64_t top = I(s->my_top, j);
            if (top < 0) continue;
            if (BX(s->box_bubble, top) != -1) {
                I(s->old_bubble, j) = I(s->bubble, j);
                I(s->bubble, j) = BX(s->box_bubble, top);
                add_to_bubble(j);
                continue;
            }
            const int64_t seed = one(s->bubble_id);
            traverse(top, seed);
            I(s->old_bubble, j) = I(s->bubble, j);
            I(s->bubble, j) = seed;
            add_to_bubble(j);
            one(s->bubble_id) = seed + 1;
        }
    }
    // CopyBubbles: each dictionary's entries settle (+1 to 0, -1 gone); an emptied dictionary goes
    EBB_HD void copy_bubbles() {
        for (int64_t e = 0; e < one(s->entry_n);) {
            if (I(s->entry_value, e) == -1) {
                entry_erase(e);
                continue;
            }
            if (I(s->entry_value, e) == 1) I(s->entry_value, e) = 0;
            ++e;
        }
        int64_t m = 0;
        const int64_t n = one(s->dict_n);
        for (int64_t d = 0; d < n; ++d) {
            const int64_t bub = I(s->dict_bubble, d);
            bool any = false;
            for (int64_t e = 0; e < one(s->entry_n) && !any; ++e) any = I(s->entry_bubble, e) == bub;
            if (any) I(s->dict_bubble, m++) = bub;
        }
        one(s->dict_n) = m;
    }
    // phase 1's dead-bubble flags: a free ball of the park in a dead bubble skips the tick
    EBB_HD void dead() {                                   // (in a warp a lane a slot)
        for (int64_t j = COOP ? lane : 0; j < N; j += COOP ? 32 : 1) {
            const bool in = U(s->in_park, j) && slot_ok(j);
            U(s->dead, j) = (in && p->free_[row(j)] && in_dead_bubble(j)) ? 1 : 0;
        }
#ifdef __CUDA_ARCH__
        if constexpr (COOP) __syncwarp();
#endif
    }
    // after the park's tick, in ascending id: each warp drop-out nearly at rest re-filed at its drop-out point (the old
    // state), then each ball that moved at least sqrt(0.1) m
    EBB_HDNI void after_evolve() {
#ifdef __CUDA_ARCH__
        if constexpr (COOP) {
            after_evolve_warp();
        } else
#endif
        {
            int64_t order[EBB_SPACE_MAX_SLOTS];
            int64_t n = 0;
            for (int64_t j = 0; j < N; ++j)
                if (U(s->in_park, j) && slot_ok(j)) order[n++] = j;
            for (int64_t i = 1; i < n; ++i)
                for (int64_t k = i; k > 0 && id(order[k]) < id(order[k - 1]); --k) {
                    const int64_t t = order[k];
                    order[k] = order[k - 1];
                    order[k - 1] = t;
                }
            for (int64_t i = 0; i < n; ++i)
                if (drops_out(order[i])) refile_dropped(order[i]);
            for (int64_t i = 0; i < n; ++i) {
                const int64_t j = order[i];
                if (!moved(j)) continue;
                insert_in_boxes(j);
                set_fresh(j, true);
            }
        }
        handle_proximities();
    }
    // a warp's drop-out nearly at rest; a ball of the tick that moved
    EBB_HD bool drops_out(int64_t j) const {
        const int64_t r = row(j);
        if (!U(s->dropped, j) || U(s->dead, j) || !p->free_[r]) return false;
        const double ov[3] = {p->old_vel[r], p->old_vel[p->n + r], p->old_vel[2 * p->n + r]};
        return dadd(dadd(dmul(ov[0], ov[0]), dmul(ov[1], ov[1])), dmul(ov[2], ov[2])) < 0.1;
    }
    EBB_HD void refile_dropped(int64_t j) {
        const int64_t r = row(j);
        const double ov[3] = {p->old_vel[r], p->old_vel[p->n + r], p->old_vel[2 * p->n + r]};
        const double op[3] = {p->old_pos[r], p->old_pos[p->n + r], p->old_pos[2 * p->n + r]};
        insert_in_boxes(j, op, ov);
    }
    EBB_HD bool moved(int64_t j) const {
        const int64_t r = row(j);
        if (U(s->dead, j) || !p->free_[r]) return false;
        double d[3];
        for (int c = 0; c < 3; ++c) d[c] = dsub(p->pos[c * p->n + r], p->old_pos[c * p->n + r]);
        return !(dadd(dadd(dmul(d[0], d[0]), dmul(d[1], d[1])), dmul(d[2], d[2])) < 0.1);
    }
#ifdef __CUDA_ARCH__
    // after_evolve in a warp: the order, the drop-outs and the balls that moved are found a lane a ball, with those
    // whose re-filing leaves everything as it is (refile_noop: nothing an earlier ball's re-filing writes changes
    // that); the warp files the others one after another in id order
    __device__ void after_evolve_warp() {
        int n = 0, last = -1;
        for (int64_t base = 0; base < N; base += 32) {     // the slots in the park, packed in slot order
            const int64_t j = base + lane;
            const bool in = j < N && U(s->in_park, j) && slot_ok(j);
            const unsigned bits = __ballot_sync(0xffffffffu, in);
            if (in) {
                const int e = n + __popc(bits & ((1u << lane) - 1u));
                sh->key[e] = 0;
                sh->id[e] = id(j);
                sh->out[e] = (uint8_t)j;
            }
            n += __popc(bits);
            if (bits) last = (int)base + 31 - __clz(bits);
        }
        occupied = last + 1;
        __syncwarp();
        bool rising = true;                                // (a world added in id order needs no sort)
        for (int e = lane; e + 1 < n; e += 32) rising = rising && sh->id[e] < sh->id[e + 1];
        if (!__all_sync(0xffffffffu, rising)) {
            int P = 1;
            while (P < n) P <<= 1;
            for (int e = n + lane; e < P; e += 32) {
                sh->key[e] = NOT_A_CANDIDATE;
                sh->id[e] = INT64_MAX;
            }
            __syncwarp();
            warp_sort(P);
        }
        uint32_t order = 0;                                // entry 32 q + lane in byte q
        for (int q = 0; q < 4; ++q)
            if (32 * q + lane < n) order |= (uint32_t)sh->out[32 * q + lane] << (8 * q);
        __syncwarp();
        for (int q = 0; 32 * q < n; ++q) {
            const int64_t j = (order >> (8 * q)) & 255;
            unsigned bits = __ballot_sync(0xffffffffu, 32 * q + lane < n && drops_out(j));
            for (; bits; bits &= bits - 1) refile_dropped(__shfl_sync(0xffffffffu, j, __ffs(bits) - 1));
        }
        for (int q = 0; 32 * q < n; ++q) {
            const int64_t j = (order >> (8 * q)) & 255;
            const bool on = 32 * q + lane < n && moved(j);
            unsigned bits = __ballot_sync(0xffffffffu, on && !refile_noop(j));
            for (; bits; bits &= bits - 1) insert_in_boxes(__shfl_sync(0xffffffffu, j, __ffs(bits) - 1));
            uint32_t f[4];
            for (int c = 0; c < 4; ++c)
                f[c] = __reduce_or_sync(0xffffffffu, on && (int)(j >> 5) == c ? 1u << (j & 31) : 0u);
            fresh[0] |= (uint64_t)f[0] | ((uint64_t)f[1] << 32);
            fresh[1] |= (uint64_t)f[2] | ((uint64_t)f[3] << 32);
        }
    }
#endif
    // Whether InsertInBoxes of ball j at its position and velocity changes nothing: the same box (level and keys) with
    // its entries kept, its top's bubble the ball's, the same sides. Read-only; for the tick's re-filings.
    EBB_HD bool refile_noop(int64_t j) const {
        if (lvl(j) < 0 || I(s->my_box, j) < 0 || I(s->my_top, j) < 0) return false;
        const double x[3] = {pos(j, 0), pos(j, 1), pos(j, 2)}, v[3] = {vel(j, 0), vel(j, 1), vel(j, 2)};
        const double inflated = inflated_radius(j, v);
        const int level0 = level_for(inflated);
        if (level0 != lvl(j)) return false;
        int64_t k[3], m[3];
        key_for(level0, x, k);
        for (int c = 0; c < 3; ++c)
            if (k[c] != key(j, c)) return false;
        const int64_t bub = BX(s->box_bubble, I(s->my_top, j));
        if (bub == -1 || bub != I(s->bubble, j)) return false;
        side_mods(level0, k, inflated, x, m);
        for (int c = 0; c < 3; ++c)
            if (m[c] != mod(j, c)) return false;
        return true;
    }
    EBB_HD void apply(int64_t code, int64_t j, int64_t b, const double* f) {
        fresh[0] = fresh[1] = 0;                           // (an operation's own: AFTER_EVOLVE's re-filings)
        occupied = EBB_SPACE_MAX_SLOTS;
        const bool has_slot = slot_ok(j);
        const bool live = has_slot && U(s->in_park, j);
        switch (code) {
            case EBB_SPACE_NONE: break;
            case EBB_SPACE_ADD: if (has_slot) add(j); else flag(F_BAD_OP); break;
            case EBB_SPACE_REFILE: if (has_slot && U(s->in_park, j)) insert_in_boxes(j); break;
            case EBB_SPACE_INIT_BUBBLES: init_bubbles(); break;
            case EBB_SPACE_COPY_BUBBLES: copy_bubbles(); break;
            case EBB_SPACE_KEEP_ALIVE: if (has_slot) U(s->keep_alive, j) = 1; break;
            case EBB_SPACE_SET_INTERACTIVE: if (has_slot && U(s->in_park, j)) set_interactive(j, b != 0); break;
            case EBB_SPACE_REMOVE_BALL: if (has_slot) remove(j); break;
            case EBB_SPACE_DEAD: dead(); break;
            case EBB_SPACE_AFTER_EVOLVE: after_evolve(); break;
            case EBB_SPACE_ADD_SENSOR: if (live) add_sensor(j, f[0], f[1], (b & 1) != 0, (b & 2) != 0); break;
            case EBB_SPACE_REMOVE_SENSOR: if (live) remove_sensor(j); break;
            case EBB_SPACE_NOTIFY_RANGE: if (live) set_notification_range(j, f[0]); break;
            case EBB_SPACE_TRACK: if (live) set_tracking(j, b, f[0], f[1] != 0.0); break;
            case EBB_SPACE_CLEAR_EVENTS: one(s->evn) = 0; break;
            case EBB_SPACE_HANDLE_PROXIMITIES: handle_proximities(); break;
            case EBB_SPACE_SET_CLOAKED: if (live) at(s->cloaked, j) = b; break;
            default: flag(F_BAD_OP); break;
        }
    }
};

// world w's query (its state read, nothing written but the answer; a flagged world answers nothing)
template <bool WM>
EBB_HD void run_query(const EbbFlightState* p, const EbbSpaceState* s, const EbbSpaceQuery* q, int64_t w) {
    World<WM> wd{p, s, w, s->worlds, s->slots, s->boxes};
    q->out[w] = 0;
    if (wd.one(s->flags) & (F_EDGE | F_BOXES | F_DICTS | F_ENTRIES | F_SETS | F_BAD_OP)) return;
    double f[5];
    for (int c = 0; c < 5; ++c) f[c] = q->f[c * s->worlds + w];
    wd.query(q->kind, q->a[w], q->b[w], f, q->out, q->outd);
}

// world w's K operations of the tape, in order (a flagged world is left alone)
template <bool WM, bool COOP = false>
EBB_HD void run_tape(const EbbFlightState* p, const EbbSpaceState* s, const EbbSpaceTape* t, int64_t w, int lane = -1,
                     Coop* sh = nullptr) {
    World<WM, COOP> wd{p, s, w, s->worlds, s->slots, s->boxes, lane, sh};
    for (int64_t k = 0; k < t->K; ++k) {
        if (wd.one(s->flags) & (F_EDGE | F_BOXES | F_DICTS | F_ENTRIES | F_SETS | F_BAD_OP)) return;
        const int64_t at = k * s->worlds + w;
        double f[4] = {0.0, 0.0, 0.0, 0.0};
        if (t->f != nullptr)
            for (int c = 0; c < 4; ++c) f[c] = t->f[(k * 4 + c) * s->worlds + w];
        wd.apply(t->code[at], t->a[at], t->b[at], f);
    }
}

}  // namespace space
}  // namespace ebb
