// batch_tmpl.cuh -- per-M H.C and density kernels of the batched engine:
// persistent blocks walk the tile lists of one orbital count M (batch.h),
// each tile a run of rows of one slot, with the building blocks of the
// single-system kernels (pairhc_tmpl.cuh, gram_tmpl.cuh).  One explicit
// instantiation per M (batch_m*.cu).
//
// Every value of a slot is computed by one thread, or summed over the
// slot's own slices in a fixed order, so a slot's result does not depend on
// the other slots of the batch.
#pragma once
#include <algorithm>

#include "batch.h"
#include "gram_tmpl.cuh"
#include "pairhc_tmpl.cuh"

namespace mctdhb {

// H.C of this step's Lanczos iteration runs for the slot; the monitor's
// H.C (iter == kBatchMonIter) for the slots whose eigen residual is due
__device__ __forceinline__ bool bt_hc_active(const BatchSlot& S, int iter) {
    if (iter == kBatchMonIter) return S.flags[BF_MON] != 0;
    return S.flags[BF_STATE] == SLOT_RUNNING && !S.flags[BF_BREAK];
}

// Pair contraction Y = A W^T of V[iter] for every tile of list LIST_HY:
// warp-specialised and double-buffered as hcp_y_kernel.  Consecutive tiles
// may belong to different slots, so the producer warps stage a tile's W with
// its A and publish the tile's output row, size, Y plane and real-W flag in
// shared memory; the consumers start on the tensor cores without a chain of
// global loads.
struct PairTileMeta {
    double2* Y;
    uint32_t row0, D2, ld;
    int active, real;
    int wbuf;  // variant 3: how many times W has been staged before this tile's
};

template <int M, int V, bool NOWAIT = false>
__global__ void __launch_bounds__(PairHcShape<M, V>::THREADS, 1)
    bhcp_y_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                  const int* __restrict__ cnt, int iter) {
    using PS_ = PairHcShape<M, V>;
    constexpr int P = PS_::P, PS = PS_::PS, ROWS = PS_::ROWS, WW = PS_::WWORDS;
    static_assert(ROWS == batch_pair_rows(M), "tile rows of the host lists");
    extern __shared__ double2 smem[];
    double2* Ab = smem;                  // two buffers of ROWS x PS
    double2* Wb = smem + 2 * ROWS * PS;  // two buffers of W
    void* tab = Wb + 2 * WW;
    if (iter == kBatchMonIter && batch_mon(cnt)[M] == 0) return;  // no residual due
    const int nt = batch_cnt(cnt, LIST_HY, M);
    const BatchTile* list = tiles + batch_off(cnt, LIST_HY, M);
    const int t = threadIdx.x, lane = t & 31;
    const int vin = iter < 0 ? 0 : iter;  // input vector V[vin]
    const int pt = t - PS_::CONSUMERS;
    auto tables = [&](const SpaceView& sp) {  // the view on the staged tables
        SpaceView v = sp;
        if (pair_tab_fits(sp.N, M)) {
            v.sq = (const double*)tab;
            v.T = (const uint32_t*)((const double*)tab + sp.N + 3);
        }
        return v;
    };
    if constexpr (PS_::PIPE) {
        // Chunks of 32 rows from producer warp to consumer warp (hcp_y_kernel,
        // variant 3): pair w takes rows 32 w .. 32 w + 31 of every tile.  When
        // the slot changes, all producer warps meet, stage its tables and W
        // (into the buffer of the slot before the last, once every consumer
        // warp has left that slot) and go on; the consumers of a tile wait for
        // its W.  A warp whose wait ran out takes no further part but for the
        // producers' barriers (mbar_wait): it marks the job of every tile it
        // still comes to aborted, since none of their Y is complete.
        __shared__ PairTileMeta meta[PS_::PW][2];
        __shared__ uint64_t full[PS_::PW][2], empty[PS_::PW][2], wfull[2], wdone[2];
        if (t < 2 * PS_::PW) {
            mbar_init(&full[t >> 1][t & 1], 32);
            mbar_init(&empty[t >> 1][t & 1], 32 * PS_::CPP);
        }
        if (t < 2) {
            mbar_init(&wfull[t], PS_::PRODUCERS);
            mbar_init(&wdone[t], PS_::CONSUMERS);
        }
        __syncthreads();
        bool lost = false;
        auto wait = [&](uint64_t* bar, unsigned parity) {
            lost = lost || !__all_sync(0xffffffffu, mbar_wait<NOWAIT>(bar, parity));
        };
        auto give_up = [&](int slot) {
            const BatchSlot& S = slots[slot];
            if (lane != 0 || !bt_hc_active(S, iter)) return;
            if (S.flags[BF_STATE] == SLOT_RUNNING) S.flags[BF_STATE] = SLOT_ABORTED;
            // the monitor's product (the job may have ended in this step): no
            // residual of it, so the stop rule does not pass on old rows
            if (iter == kBatchMonIter) S.flags[BF_MON] = 0;
        };
        const int w = t >= PS_::CONSUMERS ? pt >> 5 : (t >> 5) / PS_::CPP;
        double2* ring = Ab + w * 2 * 32 * PS;
        int i = 0;
        if (t >= PS_::CONSUMERS) {
            pair_regs_dec<PS_::CREG, PS_::PREG>();
            int slot = -1, ver = -1;
            BatchTile next{};
            if ((int)blockIdx.x < nt) next = list[blockIdx.x];
            for (int k = blockIdx.x; k < nt; k += gridDim.x, i++) {
                const BatchTile tl = next;
                if (k + (int)gridDim.x < nt) next = list[k + gridDim.x];
                const BatchSlot& S = slots[tl.slot];
                const int buf = i & 1;
                if (tl.slot != slot) {
                    slot = tl.slot;
                    ver++;
                    pair_producer_barrier<PS_::PRODUCERS>();  // nobody reads the old tables
                    pair_stage_tab(S.sp, tab, pt, PS_::PRODUCERS);
                    if (ver >= 2) wait(&wdone[ver & 1], ((ver >> 1) - 1) & 1);
                    if (!lost) {
                        pair_stage_w<M, V>(S.sp.pair_w, Wb + (ver & 1) * WW, pt, PS_::PRODUCERS);
                        mbar_arrive(&wfull[ver & 1]);
                    }
                    pair_producer_barrier<PS_::PRODUCERS>();
                }
                if (i >= 2) wait(&empty[w][buf], ((i >> 1) - 1) & 1);
                if (lost) {
                    give_up(tl.slot);
                    continue;
                }
                const uint32_t row0 = tl.idx * (uint32_t)ROWS + w * 32;
                const bool active = bt_hc_active(S, iter) && row0 < S.sp.dim2;
                if (lane == 0)
                    meta[w][buf] = PairTileMeta{S.sp.pair_y, row0, S.sp.dim2, S.sp.ldy, active,
                                                active && S.sp.pair_w[P * P].x != 0.0, ver};
                if (active)
                    pair_gather_row<M, V>(tables(S.sp), S.V + (size_t)vin * S.nc, row0 + lane,
                                          ring + buf * 32 * PS, lane);
                mbar_arrive(&full[w][buf]);
            }
        } else {
            pair_regs_inc<PS_::CREG>();
            int ver = -1;
            for (int k = blockIdx.x; k < nt; k += gridDim.x, i++) {
                const int buf = i & 1, slot = list[k].slot;
                wait(&full[w][buf], (i >> 1) & 1);
                if (!lost && meta[w][buf].wbuf != ver) {
                    if (ver >= 0) mbar_arrive(&wdone[ver & 1]);
                    ver = meta[w][buf].wbuf;
                    wait(&wfull[ver & 1], (ver >> 1) & 1);
                }
                if (lost) {
                    give_up(slot);
                    continue;
                }
                const PairTileMeta tm = meta[w][buf];
                if (tm.active)
                    pair_strips<M, V>(ring + buf * 32 * PS, Wb + (ver & 1) * WW,
                                      (t >> 5) % PS_::CPP, PS_::CPP, 2, lane, tm.row0, tm.D2,
                                      tm.ld, tm.Y, tm.real != 0);
                mbar_arrive(&empty[w][buf]);
            }
        }
        return;
    }
    // Producers and consumers run their own loops and meet at one block
    // barrier per tile (named barrier 1 over all threads): the producers
    // fill buffer buf ^ 1 while the consumers contract buffer buf.  W is
    // skipped when the buffer already holds the slot's; the next tile's
    // descriptor is loaded one tile ahead.
    __shared__ PairTileMeta meta[2];
    if (t >= PS_::CONSUMERS) {
        int wslot[2] = {-1, -1};  // slot whose W each buffer holds (same in every producer)
        int tslot = -1;           // slot whose tables the shared table area holds
        auto fill = [&](const BatchTile tl, int buf) {
            const BatchSlot& S = slots[tl.slot];
            const bool active = bt_hc_active(S, iter);
            if (pt == 0)
                meta[buf] = PairTileMeta{S.sp.pair_y, tl.idx * (uint32_t)ROWS, S.sp.dim2, S.sp.ldy,
                                         active, active && S.sp.pair_w[P * P].x != 0.0, 0};
            if (wslot[buf] != tl.slot) {
                pair_stage_w<M, V>(S.sp.pair_w, Wb + buf * WW, pt, PS_::PRODUCERS);
                wslot[buf] = tl.slot;
            }
            // the slot's rank tables: the previous fill's reads ended at the
            // last block barrier; the producers meet before the new reads
            if (tslot != tl.slot) {
                pair_stage_tab(S.sp, tab, pt, PS_::PRODUCERS);
                pair_producer_barrier<PS_::PRODUCERS>();
                tslot = tl.slot;
            }
            if (active)
                pair_gather<M, V>(tables(S.sp), S.V + (size_t)vin * S.nc, tl.idx,
                                  Ab + (size_t)buf * ROWS * PS, pt, PS_::PRODUCERS);
        };
        BatchTile next{};
        if ((int)blockIdx.x < nt) fill(list[blockIdx.x], 0);
        if ((int)(blockIdx.x + gridDim.x) < nt) next = list[blockIdx.x + gridDim.x];
        pair_tile_barrier<PS_::THREADS>();
        int buf = 0;
        for (int k = blockIdx.x; k < nt; k += gridDim.x, buf ^= 1) {
            if (k + (int)gridDim.x < nt) {
                const BatchTile cur = next;
                if (k + 2 * (int)gridDim.x < nt) next = list[k + 2 * gridDim.x];
                fill(cur, buf ^ 1);
            }
            pair_tile_barrier<PS_::THREADS>();
        }
    } else {
        pair_tile_barrier<PS_::THREADS>();
        int buf = 0;
        for (int k = blockIdx.x; k < nt; k += gridDim.x, buf ^= 1) {
            const PairTileMeta tm = meta[buf];
            if (tm.active)
                pair_consume<M, V>(Ab + (size_t)buf * ROWS * PS, Wb + buf * WW, t, tm.row0, tm.D2,
                                   tm.ld, tm.Y, tm.real != 0);
            pair_tile_barrier<PS_::THREADS>();
        }
    }
}

// Lanczos H.C of step iteration `iter`, gathered back from Y:
//   out = H V[iter] - beta_{iter-1} V[iter-1]   (iter > 0)
//   out = H V[0]                                (iter == 0, kBatchMonIter)
// Slots that stopped, or whose Lanczos recurrence broke down in this step,
// are skipped (multiconfig_lanczos.c:70-71); the monitor's launch
// (kBatchMonIter) takes only the slots whose eigen residual is due.
template <int M>
__global__ void __launch_bounds__(kBatchHcRows)
    bhcp_g_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                  const int* __restrict__ cnt, int iter) {
    if (iter == kBatchMonIter && batch_mon(cnt)[M] == 0) return;
    const int nt = batch_cnt(cnt, LIST_HG, M);
    const BatchTile* list = tiles + batch_off(cnt, LIST_HG, M);
    for (int k = blockIdx.x; k < nt; k += gridDim.x) {
        const BatchTile tl = list[k];
        const BatchSlot& S = slots[tl.slot];
        if (!bt_hc_active(S, iter)) continue;
        const uint32_t nc = S.nc;
        const uint32_t row = tl.idx + threadIdx.x;
        if (row >= nc) continue;
        double2 acc = pair_gather_back<M>(S.sp, S.sp.pair_y, row);
        if (iter > 0) {
            const double2 pv = S.V[(size_t)(iter - 1) * nc + row];
            const double b = S.scal[BS_OFFD + iter - 1].x;
            acc.x -= b * pv.x;
            acc.y -= b * pv.y;
        }
        S.out[row] = acc;
    }
}

// rho2 Gram partial of slice `idx` of a slot: its gk consecutive row
// tiles of the (N-2)-boson space, summed into gpart (gram_tmpl.cuh building
// blocks)
template <int M>
__global__ void __launch_bounds__(kGramThreads, 2)
    bgram_kernel(const BatchSlot* __restrict__ slots, const BatchTile* __restrict__ tiles,
                 const int* __restrict__ cnt) {
    using GS = GramShape<M>;
    extern __shared__ double2 As[];
    const int nt = batch_cnt(cnt, LIST_G2, M);
    const BatchTile* list = tiles + batch_off(cnt, LIST_G2, M);
    GramAcc<M> acc(threadIdx.x);
    for (int k = blockIdx.x; k < nt; k += gridDim.x) {
        const BatchTile tl = list[k];
        const BatchSlot& S = slots[tl.slot];
        if (S.flags[BF_STATE] != SLOT_RUNNING) continue;  // block-uniform
        const uint32_t Dp = S.sp.dim2;
        const uint32_t ntr = (Dp + GS::ROWS - 1) / GS::ROWS;
        const uint32_t t0 = tl.idx * (uint32_t)S.gk;
        const uint32_t t1 = min(t0 + (uint32_t)S.gk, ntr);
        acc.clear();
        for (uint32_t tr = t0; tr < t1; tr++) {
            gram_gather<M>(S.sp, Dp, S.V, tr, As, threadIdx.x);
            __syncthreads();
            acc.add(As);
            __syncthreads();
        }
        acc.store(As, S.gpart + (size_t)tl.idx * GS::ENT);
    }
}

// rho2 of the running slots of orbital count M (blockIdx.x), 32 entries a
// block (blockIdx.y): fixed-order sum of the slot's slices and the reference's
// symmetric fill (gram_fill); rho1 follows from rho2 in bt_tail_kernel
template <int M>
__global__ void __launch_bounds__(kBatchVecThreads)
    bgram_finalize_kernel(const BatchSlot* __restrict__ slots, const int* __restrict__ list,
                          const int* __restrict__ nlist) {
    static_assert(kBatchVecThreads == 256, "gram_sum_parts");
    if ((int)blockIdx.x >= *nlist) return;
    const BatchSlot& S = slots[list[blockIdx.x]];
    if (S.M != M || S.flags[BF_STATE] != SLOT_RUNNING) return;  // block-uniform
    constexpr int ENT = gram_entries(M);
    const int e = blockIdx.y * 32 + (threadIdx.x & 31);
    const double2 v = gram_sum_parts(S.gpart + e, S.gs, ENT, e < ENT);
    if (threadIdx.x < 32 && e < ENT) gram_fill<M>(e, v, S.rho2);
}

template <int M, int V>
constexpr size_t batch_y_smem() {
    using PS_ = PairHcShape<M, V>;
    return (2 * (size_t)PS_::WWORDS + 2 * (size_t)PS_::ROWS * PS_::PS) * sizeof(double2) +
           kPairTabBytes;
}

// the batched tile lists fix the rows per tile: variants 0, 2 and 3
__host__ __device__ constexpr bool batch_variant_ok(int M, int V) {
    return V == 3 || ((V == 0 || V == 2) && pair_variant_ok(M, V));
}

template <int M, int V>
int batch_y_attr() {
    static_assert(batch_y_smem<M, V>() <= 227 * 1024, "shared memory of one block (227 KB)");
    if constexpr (batch_variant_ok(M, V))
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(bhcp_y_kernel<M, V>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)batch_y_smem<M, V>()));
    return 0;
}

// the instance without waits, loaded only where it is asked for
template <int M>
int batch_prepare_nowait() {
    MCTDHB_CUDA_TRY(cudaFuncSetAttribute(bhcp_y_kernel<M, 3, true>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)batch_y_smem<M, 3>()));
    return 0;
}

template <int M>
int batch_prepare() {
    static std::atomic<uint64_t> done{0};
    return set_attributes_once(done, []() -> int {
        if (batch_y_attr<M, 0>() || batch_y_attr<M, 2>() || batch_y_attr<M, 3>()) return -1;
        MCTDHB_CUDA_TRY(cudaFuncSetAttribute(bgram_kernel<M>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             gram_smem(M)));
        return 0;
    });
}

template <int M, int V>
int bhcp_y_launch(const BatchSlot* slots, const BatchTile* hy, const int* cnt, int iter,
                  bool nowait, cudaStream_t st) {
    if constexpr (!batch_variant_ok(M, V)) {
        set_error("batched pair contraction variant %d does not exist for %d orbitals", V, M);
        return -1;
    } else {
        auto* kernel = bhcp_y_kernel<M, V>;
        if constexpr (PairHcShape<M, V>::PIPE)
            if (nowait) kernel = bhcp_y_kernel<M, V, true>;
        kernel<<<num_sms(), PairHcShape<M, V>::THREADS, batch_y_smem<M, V>(), st>>>(slots, hy, cnt,
                                                                                   iter);
        MCTDHB_CUDA_TRY(cudaGetLastError());
        return 0;
    }
}

template <int M>
int hcp_batch_launch(const BatchSlot* slots, const BatchTile* hy, const BatchTile* hg,
                     const int* cnt, int iter, int parts, int variant, bool nowait,
                     cudaStream_t st) {
    if (parts & 1) {
        const int rc = variant == 3   ? bhcp_y_launch<M, 3>(slots, hy, cnt, iter, nowait, st)
                       : variant == 2 ? bhcp_y_launch<M, 2>(slots, hy, cnt, iter, nowait, st)
                                      : bhcp_y_launch<M, 0>(slots, hy, cnt, iter, nowait, st);
        if (rc) return -1;
    }
    if (parts & 2) {
        bhcp_g_kernel<M><<<num_sms() * 8, kBatchHcRows, 0, st>>>(slots, hg, cnt, iter);
        MCTDHB_CUDA_TRY(cudaGetLastError());
    }
    return 0;
}

template <int M>
int gram_batch_launch(const BatchSlot* slots, const BatchTile* g2, const int* cnt,
                      const int* list, const int* nlist, int nblocks, cudaStream_t st) {
    bgram_kernel<M><<<num_sms() * 2, kGramThreads, gram_smem(M), st>>>(slots, g2, cnt);
    MCTDHB_CUDA_TRY(cudaGetLastError());
    const dim3 fin(std::max(nblocks, 1), (gram_entries(M) + 31) / 32);
    bgram_finalize_kernel<M><<<fin, kBatchVecThreads, 0, st>>>(slots, list, nlist);
    MCTDHB_CUDA_TRY(cudaGetLastError());
    return 0;
}

}  // namespace mctdhb
