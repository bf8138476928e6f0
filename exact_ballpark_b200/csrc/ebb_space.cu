// SPDX-License-Identifier: MIT
// The space layer's tape on the device: one thread (or one warp) a world runs its K operations in order
// (ebb_space.cuh), over the state in either arrangement (interleaved [entry][world], or world-major). The parameter
// structs are __grid_constant__: the program reads its state's pointers through their addresses in the parameter
// space (uniform constant loads) rather than from a per-thread copy in local memory.
#include <cuda_runtime.h>

#include "../../include/ebb.h"
#include "ebb_space.cuh"

// Blocks of 4 warps a multiprocessor that the warp kernel's registers allow. A world's program is a chain of dependent
// loads, so its length counts before the warps in flight: 128 registers (4 blocks) ran 8,000 partition worlds in 6.4 ms a
// tick, 80 (6) in 6.6, 64 (8) in 6.7, 40 (12, with spills) in 7.2.
#ifndef EBB_SPACE_WARP_BLOCKS
#define EBB_SPACE_WARP_BLOCKS 4
#endif

namespace ebb {
namespace space {

// a thread a world, `per_warp` of a warp's lanes (registers: 128, 4 blocks a multiprocessor; 80 ran 16,384 4-ship worlds
// 2-4 % slower)
template <bool WM>
__global__ void __launch_bounds__(128, 4) tape_kernel(const __grid_constant__ EbbFlightState p,
                                                   const __grid_constant__ EbbSpaceState s,
                                                   const __grid_constant__ EbbSpaceTape t, int per_warp) {
    const int lane = (int)(threadIdx.x & 31);
    const int64_t w = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * per_warp + lane;
    if (lane >= per_warp || w >= s.worlds) return;
    run_tape<WM>(&p, &s, &t, w);
}

// a warp a world: the world's index is the warp's, the lanes run its program together (ebb_space.cuh's World)
template <bool WM>
__global__ void __launch_bounds__(128, EBB_SPACE_WARP_BLOCKS) tape_kernel_warp(const __grid_constant__ EbbFlightState p,
                                                         const __grid_constant__ EbbSpaceState s,
                                                         const __grid_constant__ EbbSpaceTape t) {
    __shared__ Coop scratch[4];
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (w >= s.worlds) return;                            // (the whole warp: w is the warp's)
    run_tape<WM, true>(&p, &s, &t, w, (int)(threadIdx.x & 31), &scratch[threadIdx.x >> 5]);
}

// Several layers' tapes in one launch, a warp a world (world-major): a batch's size classes one after another each held
// about a tenth of the chip's warps until its slowest world was done (8,000 partition worlds, 269 blocks a class of 64 or
// 128 slots); side by side the small classes fill the large one's gaps (6.4 -> 5.3 ms a tick). The layers' blocks follow in
// the order given, so that the first layer's (the longest programs) start first. BLOCKS a multiprocessor: while the batch
// is a few waves the tick is its longest programs, which 255 registers (2 blocks) shorten; with more waves the blocks in
// flight count, and 128 registers (4) win. Ms a tick at 2 and 4 blocks: 1,000 worlds of 1 to 128 ships 1.47 and 1.56, 4,000
// 2.29 and 2.56, 8,000 3.52 and 3.94, 10,000 4.40 and 4.53, 11,000 4.84 and 4.80, 14,000 5.95 and 5.80, 24,000 10.0 and
// 9.56 (3 blocks: 8,000 3.78, 24,000 9.80; 5: 4.04 and 9.67): the line is at 9 waves of the 2 (10,656 worlds).
constexpr int64_t LONG_BLOCKS = 9 * 2 * 148;
struct Layers {
    EbbSpaceState s[EBB_SPACE_MAX_LAYERS];
    EbbSpaceTape t[EBB_SPACE_MAX_LAYERS];
    unsigned first[EBB_SPACE_MAX_LAYERS + 1];             // each layer's first block
    int count;
};

template <int BLOCKS>
__global__ void __launch_bounds__(128, BLOCKS) tape_kernel_layers(const __grid_constant__ EbbFlightState p,
                                                                  const __grid_constant__ Layers m) {
    __shared__ Coop scratch[4];
    int l = 0;
    while (l + 1 < m.count && blockIdx.x >= m.first[l + 1]) ++l;
    const int64_t w = (int64_t)(blockIdx.x - m.first[l]) * 4 + (threadIdx.x >> 5);
    if (w >= m.s[l].worlds) return;                       // (the whole warp: w is the warp's)
    run_tape<true, true>(&p, &m.s[l], &m.t[l], w, (int)(threadIdx.x & 31), &scratch[threadIdx.x >> 5]);
}

template <bool WM>
__global__ void __launch_bounds__(128) query_kernel(const __grid_constant__ EbbFlightState p,
                                                    const __grid_constant__ EbbSpaceState s,
                                                    const __grid_constant__ EbbSpaceQuery q) {
    const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= s.worlds) return;
    run_query<WM>(&p, &s, &q, w);
}

}  // namespace space
}  // namespace ebb

extern "C" {

// the sizes and the block (checked first: a call with no worlds then does nothing), then every buffer
static int space_sizes(const EbbFlightState* park, const EbbSpaceState* s, int block) {
    if (park == nullptr || s == nullptr || block <= 0 || block > 128 || block % 32 != 0) return EBB_EINVAL;
    if (s->slots < 1 || s->slots > EBB_SPACE_MAX_SLOTS || s->boxes < 1 || s->dicts < 1 || s->entries < 1 ||
        s->sets < 1)
        return EBB_EINVAL;
    return 0;
}

static int space_buffers(const EbbFlightState* park, const EbbSpaceState* s) {
    if (s->rows == nullptr || s->level == nullptr || s->key == nullptr || s->mod == nullptr || s->active == nullptr ||
        s->bubble == nullptr || s->old_bubble == nullptr || s->seq == nullptr || s->in_park == nullptr ||
        s->keep_alive == nullptr || s->dead == nullptr || s->dropped == nullptr || s->box_level == nullptr ||
        s->box_key == nullptr || s->box_balls == nullptr || s->box_kids == nullptr || s->box_bubble == nullptr ||
        s->my_box == nullptr || s->my_top == nullptr || s->box_hash == nullptr || s->box_free == nullptr ||
        s->box_free_n == nullptr ||
        s->stack == nullptr || s->box_n == nullptr || s->free_boxes == nullptr || s->dict_bubble == nullptr ||
        s->dict_n == nullptr || s->entry_bubble == nullptr || s->entry_id == nullptr || s->entry_value == nullptr ||
        s->entry_n == nullptr || s->inter_bubble == nullptr || s->inter_id == nullptr || s->inter_n == nullptr ||
        s->keep_bubble == nullptr || s->keep_id == nullptr || s->keep_n == nullptr || s->bubble_id == nullptr ||
        s->seq_next == nullptr || s->flags == nullptr)
        return EBB_EINVAL;
    if (s->umap_cap < 1 || s->umap_cap > EBB_SPACE_MAX_SLOTS || s->events < 0 || s->srange == nullptr ||
        s->speriod == nullptr || s->selapsed == nullptr || s->ntf_range == nullptr || s->trk_range == nullptr ||
        s->trk == nullptr || s->cloaked == nullptr || s->sonly == nullptr || s->has_prox == nullptr ||
        s->ntf_in == nullptr || s->trk_in == nullptr || s->slist == nullptr || s->slen == nullptr ||
        s->sbkt == nullptr || s->pmap == nullptr || s->pn == nullptr || s->pbkt == nullptr || s->evn == nullptr ||
        s->rnd == nullptr || (s->events > 0 && s->ev == nullptr) || s->smask == nullptr || s->pmask == nullptr ||
        (s->lanes != 1 && s->lanes != 32) || s->pitch < 0 || s->pitch % 16 != 0 || s->box_parent == nullptr ||
        s->box_top == nullptr || s->box_home == nullptr || s->box_slot == nullptr || s->fbox == nullptr)
        return EBB_EINVAL;
    if (park->pos == nullptr || park->vel == nullptr || park->old_pos == nullptr || park->old_vel == nullptr ||
        park->ids == nullptr || park->radius == nullptr || park->max_vel == nullptr || park->agility == nullptr ||
        park->speed_fraction == nullptr || park->mass == nullptr || park->time_factor == nullptr ||
        park->free_ == nullptr || park->interactive == nullptr || park->mode == nullptr || park->goto_pt == nullptr ||
        park->follow_ptr == nullptr || park->follow_range == nullptr || park->massive == nullptr || park->sensor == nullptr)
        return EBB_EINVAL;
    return 0;
}

int ebb_space_tape(const EbbFlightState* park, const EbbSpaceState* s, const EbbSpaceTape* t, void* stream, int block) {
    if (t == nullptr || t->K < 0) return EBB_EINVAL;
    int rc = space_sizes(park, s, block);
    if (rc) return rc;
    if (s->worlds <= 0 || t->K == 0) return 0;
    rc = space_buffers(park, s);
    if (rc) return rc;
    if (t->code == nullptr || t->a == nullptr || t->b == nullptr) return EBB_EINVAL;
    const cudaStream_t st = (cudaStream_t)stream;
    if (s->lanes == 32) {
        const unsigned grid = (unsigned)((s->worlds * 32 + 127) / 128);
        if (s->pitch > 0)
            ebb::space::tape_kernel_warp<true><<<grid, 128, 0, st>>>(*park, *s, *t);
        else
            ebb::space::tape_kernel_warp<false><<<grid, 128, 0, st>>>(*park, *s, *t);
    } else {
        // Worlds a warp: a warp's time grows with them (their programs diverge: 4 of 32 lanes busy), the worlds' own with the
        // warps in flight (their states contend for the cache), so the worlds a warp rise with the square root of all of
        // them: 2 at 256 worlds, 4 at 1,024, ... 32 from 65,536. Ticks of 4-ship worlds, ms, at 32 a warp and so: 256 worlds
        // 0.94 and 0.36, 1,024 0.96 and 0.47, 4,096 1.03 and 0.65, 16,384 1.40 and 1.31 (8 a warp 1.40, 4 2.06).
        int per = 2;
        while (per < 32 && (int64_t)per * per * 64 < s->worlds) per *= 2;
        const int64_t warps = (s->worlds + per - 1) / per;
        const unsigned grid = (unsigned)((warps + block / 32 - 1) / (block / 32));
        if (s->pitch > 0)
            ebb::space::tape_kernel<true><<<grid, block, 0, st>>>(*park, *s, *t, per);
        else
            ebb::space::tape_kernel<false><<<grid, block, 0, st>>>(*park, *s, *t, per);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : (int)e;
}

int ebb_space_tapes(const EbbFlightState* park, const EbbSpaceState* s, const EbbSpaceTape* t, int count,
                    void* stream) {
    if (s == nullptr || t == nullptr || count < 0 || count > EBB_SPACE_MAX_LAYERS) return EBB_EINVAL;
    ebb::space::Layers m{};
    int64_t blocks = 0;
    for (int l = 0; l < count; ++l) {
        int rc = space_sizes(park, s + l, 128);
        if (rc) return rc;
        if (t[l].K < 0) return EBB_EINVAL;
        if (s[l].worlds <= 0 || t[l].K == 0) continue;
        rc = space_buffers(park, s + l);
        if (rc) return rc;
        if (t[l].code == nullptr || t[l].a == nullptr || t[l].b == nullptr) return EBB_EINVAL;
        if (s[l].lanes != 32 || s[l].pitch <= 0) return EBB_EINVAL;
        m.s[m.count] = s[l];
        m.t[m.count] = t[l];
        m.first[m.count] = (unsigned)blocks;
        blocks += (s[l].worlds + 3) / 4;
        if (blocks > 0x7fffffff) return EBB_EINVAL;
        ++m.count;
    }
    if (m.count == 0) return 0;
    m.first[m.count] = (unsigned)blocks;
    if (blocks <= ebb::space::LONG_BLOCKS)
        ebb::space::tape_kernel_layers<2><<<(unsigned)blocks, 128, 0, (cudaStream_t)stream>>>(*park, m);
    else
        ebb::space::tape_kernel_layers<4><<<(unsigned)blocks, 128, 0, (cudaStream_t)stream>>>(*park, m);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : (int)e;
}

int ebb_space_query(const EbbFlightState* park, const EbbSpaceState* s, const EbbSpaceQuery* q, void* stream,
                    int block) {
    if (q == nullptr || q->kind < EBB_SPACE_Q_VISIBILITY || q->kind > EBB_SPACE_Q_NEARBY) return EBB_EINVAL;
    int rc = space_sizes(park, s, block);
    if (rc) return rc;
    if (s->worlds <= 0) return 0;
    rc = space_buffers(park, s);
    if (rc) return rc;
    if (q->a == nullptr || q->b == nullptr || q->f == nullptr || q->out == nullptr || q->outd == nullptr)
        return EBB_EINVAL;
    const unsigned grid = (unsigned)((s->worlds + block - 1) / block);
    if (s->pitch > 0)
        ebb::space::query_kernel<true><<<grid, block, 0, (cudaStream_t)stream>>>(*park, *s, *q);
    else
        ebb::space::query_kernel<false><<<grid, block, 0, (cudaStream_t)stream>>>(*park, *s, *q);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? 0 : (int)e;
}

}  // extern "C"

EBB_OP_COUNTER(ebb_count_ops_space)

#ifdef EBB_COUNT_OPS
// the counting build's tally of CheckSensor's paths: checks, re-filings skipped, filings unchanged
extern "C" int ebb_count_sensor_paths(unsigned long long* out, int reset) {
    cudaError_t e = cudaMemcpyFromSymbol(out, ebb::space::sensor_paths, sizeof(unsigned long long) * 3);
    if (e == cudaSuccess && reset) {
        const unsigned long long zero[3] = {};
        e = cudaMemcpyToSymbol(ebb::space::sensor_paths, zero, sizeof(zero));
    }
    return e == cudaSuccess ? 0 : (int)e;
}
#endif
