// Accumulator updates of the hash aggregate (accumulator.rs:110-594), shared by the
// ahead-of-time kernels and the runtime-specialized pipeline kernels.
#pragma once

#include "ml_args.hpp"
#include "ml_device.cuh"

namespace mlg {

// ---- hash aggregation ---------------------------------------------------------------------
__device__ __forceinline__ uint64_t agg_identity(int kind) {
    switch (kind) {
        case A_MIN_I64: return 0x7FFFFFFFFFFFFFFFull;
        case A_MAX_I64: return 0x8000000000000000ull;
        case A_MIN_F64:
        case A_MIN_STR: return ~0ull;
        case A_MAX_F64:
        case A_MAX_STR: return 0ull;
        default: return 0ull;
    }
}

// Fold value v into the accumulator word(s) at `w` (shared or global memory).
__device__ __forceinline__ void acc_apply(int kind, uint64_t* w, uint64_t v) {
    switch (kind) {
        case A_SUM_I64: atomicAdd((unsigned long long*)w, (unsigned long long)v); break;
        case A_SUM_F64: atomicAdd((double*)w, as_f64(v)); break;
        case A_AVG:
            atomicAdd((double*)w, as_f64(v));
            atomicAdd((unsigned long long*)w + 1, 1ull);
            break;
        case A_MIN_I64: atomicMin((long long*)w, (long long)v); break;
        case A_MAX_I64: atomicMax((long long*)w, (long long)v); break;
        case A_MIN_F64: atomicMin((unsigned long long*)w, (unsigned long long)f64_order(as_f64(v))); break;
        case A_MAX_F64: atomicMax((unsigned long long*)w, (unsigned long long)f64_order(as_f64(v))); break;
        case A_MIN_STR: atomicMin((unsigned long long*)w, (unsigned long long)v); break;  // v packed (str_pack)
        case A_MAX_STR: atomicMax((unsigned long long*)w, (unsigned long long)v); break;
        default: atomicAdd((unsigned long long*)w, 1ull); break;  // COUNT(x)
    }
}
// A string id as the packed word of A_MIN_STR / A_MAX_STR.
__device__ __forceinline__ uint64_t str_pack(const uint32_t* rank, uint32_t id) {
    return ((uint64_t)(__ldg(rank + id) + 1u) << 32) | id;
}
// acc_apply for accumulators known to be in global memory: fire-and-forget reductions
// (red.global), so no thread waits for the L2 to answer.
__device__ __forceinline__ void acc_apply_global(int kind, uint64_t* w, uint64_t v) {
    switch (kind) {
        case A_SUM_I64: asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(v) : "memory"); break;
        case A_SUM_F64: asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(w), "d"(as_f64(v)) : "memory"); break;
        case A_AVG:
            asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(w), "d"(as_f64(v)) : "memory");
            asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w + 1), "l"(1ull) : "memory");
            break;
        case A_MIN_I64: asm volatile("red.relaxed.gpu.global.min.s64 [%0], %1;" ::"l"(w), "l"(v) : "memory"); break;
        case A_MAX_I64: asm volatile("red.relaxed.gpu.global.max.s64 [%0], %1;" ::"l"(w), "l"(v) : "memory"); break;
        case A_MIN_F64:
            asm volatile("red.relaxed.gpu.global.min.u64 [%0], %1;" ::"l"(w), "l"(f64_order(as_f64(v))) : "memory");
            break;
        case A_MAX_F64:
            asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" ::"l"(w), "l"(f64_order(as_f64(v))) : "memory");
            break;
        default: asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(1ull) : "memory"); break;
    }
}
__device__ __forceinline__ void count_global(uint64_t* w) {
    asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(1ull) : "memory");
}

// Warp-cooperative updates of group blocks (the generated code, emit_coop in ml_jit.cpp): the words of
// a block that take the same reduction are updated by neighbouring lanes of one instruction, because L2
// serves one request per 32-byte sector and instruction, whatever the number of words in it (measured on
// 1.5M 16-byte groups: two reductions by one lane 96 G rows/s, the same two by a pair of lanes 188, one
// reduction alone 188).  Counts join the f64 sums: a count's bits k are the subnormal k * 2^-1074, so an
// f64 add of the subnormal with bits 1 makes them k + 1, exactly, up to 2^53 (IEEE 754 gradual
// underflow; f64 reductions do not flush subnormals).  A NULL argument adds -0.0, which changes no sum.
template <int OP>
__device__ __forceinline__ void coop_red(uint64_t* w, uint64_t v) {
    if (OP == CO_ADD_F64) asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(w), "d"(as_f64(v)) : "memory");
    else if (OP == CO_ADD_U64) asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(w), "l"(v) : "memory");
    else if (OP == CO_MIN_U64) asm volatile("red.relaxed.gpu.global.min.u64 [%0], %1;" ::"l"(w), "l"(v) : "memory");
    else if (OP == CO_MAX_U64) asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" ::"l"(w), "l"(v) : "memory");
    else if (OP == CO_MIN_S64) asm volatile("red.relaxed.gpu.global.min.s64 [%0], %1;" ::"l"(w), "l"(v) : "memory");
    else asm volatile("red.relaxed.gpu.global.max.s64 [%0], %1;" ::"l"(w), "l"(v) : "memory");
}

// A new group's id (kNone when the table takes no more).  The lanes that insert together take theirs
// with one atomic: every insertion counts on the same word.
__device__ __forceinline__ uint32_t new_group(const AggArgs& A) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(A.ngroups, (uint32_t)__popc(m));
    const uint32_t id = __shfl_sync(m, base, leader) + __popc(m & ((1u << lane) - 1u));
    return id < A.gid_cap ? id : kNone;
}

// table_upsert for a whole warp and K keys per lane: every lane calls it, need[k] set where it has a
// key.  g[k] becomes the key's group (kNone: the table is full), bit k of the result is set where this
// lane created it.  `full` is the warp's note that the table takes no more groups.
//
// Bound by the latency of its dependent accesses (slot, claim, group id), so the keys of a lane are taken
// through them together, and the lanes step together instead of splitting into groups that issue the
// same code one after another.  The warp's claims take their group ids with one atomic, once every key is
// resolved or one has to wait: every insertion counts on the same word, which L2 serves one access after
// the other (an atomic per step: 640 and 990 us for the two cases below).
// 4.7M rows with 1.4M new groups and eight words a group: 1,960 us row by row with an atomic and a release
// per insertion, 780 us so (570 us with six words); 14.8M rows with 0.15M new groups 2,530 us and 1,400 us
// (six words 940 us): the table and its accumulators miss L2, 2.1 GB read and 0.6 GB written.
template <int K>
__device__ __forceinline__ uint32_t warp_upsert(const AggArgs& A, bool (&need)[K], const uint64_t (&w)[K][2],
                                                const uint32_t (&nm)[K], const uint64_t (&h)[K], uint32_t (&g)[K], bool& full,
                                                uint32_t* err) {
    const TableView& t = A.t;
    const bool wide = t.nwords > 1;
    const int lane = threadIdx.x & 31;
    uint64_t i[K];
    ulonglong2 v[K];
    uint32_t made = 0, steps = 0, spins = 0, claimed = 0;
    bool any = false;
#pragma unroll
    for (int k = 0; k < K; k++) {
        i[k] = h[k] & t.mask;
        g[k] = kNone;
        any = any || need[k];
    }
    // the warp's claims take their ids, with one atomic, and are published
    auto publish = [&] {
        unsigned m[K];
        uint32_t total = 0;
#pragma unroll
        for (int k = 0; k < K; k++) {
            m[k] = __ballot_sync(0xFFFFFFFFu, (claimed >> k) & 1u);
            total += __popc(m[k]);
        }
        uint32_t id = 0;
        if (lane == 0) id = atomicAdd(A.ngroups, total);
        id = __shfl_sync(0xFFFFFFFFu, id, 0);
        full = id + total > A.gid_cap || id + total < id;
#pragma unroll
        for (int k = 0; k < K; k++) {
            if ((claimed >> k) & 1u) {
                const uint32_t mine = id + __popc(m[k] & ((1u << lane) - 1u));
                uint64_t* s = slot_at(t, i[k]);
                const uint64_t x = (2u | (nm[k] << 8)) | ((uint64_t)mine << 32);
                if (mine >= A.gid_cap) {
                    publish_state((uint32_t*)s, 0);
                } else {
                    if (wide) {
                        s[2] = w[k][1];
                        st_slot_release(s, x, w[k][0]);
                    } else {
                        st_slot(s, x, w[k][0]);
                    }
                    g[k] = mine;
                    made |= 1u << k;
                }
            }
            id += __popc(m[k]);
        }
        claimed = 0;
    };
    while (__any_sync(0xFFFFFFFFu, any)) {
#pragma unroll
        for (int k = 0; k < K; k++)
            if (need[k]) v[k] = wide ? ld_slot_acquire(slot_at(t, i[k])) : ld_slot(slot_at(t, i[k]));
        uint32_t old[K];
#pragma unroll
        for (int k = 0; k < K; k++) {
            old[k] = 1;
            if (need[k] && (uint32_t)v[k].x == 0) {
                if (full) need[k] = false;  // the row overflows
                else old[k] = atomicCAS((uint32_t*)slot_at(t, i[k]), 0u, 1u);
            }
        }
#pragma unroll
        for (int k = 0; k < K; k++)
            if (old[k] == 0) {
                claimed |= 1u << k;
                need[k] = false;
            }
        any = false;
        bool waiting = false;
#pragma unroll
        for (int k = 0; k < K; k++) {
            if (!need[k]) continue;
            const uint32_t st = (uint32_t)v[k].x;
            if (st > 1) {  // a published slot: this key's, or the next one's turn
                g[k] = slot_match(t, i[k], v[k], w[k], nm[k]);
                need[k] = g[k] == kNone;
                i[k] = (i[k] + 1) & t.mask;
            }
            waiting = waiting || st <= 1;
            any = any || need[k];
        }
        // no key of the warp left to resolve, or one waits for a claim (this warp's own, or another's whose
        // warp may wait for this one's)
        if (__any_sync(0xFFFFFFFFu, claimed != 0) && (__any_sync(0xFFFFFFFFu, waiting) || !__any_sync(0xFFFFFFFFu, any))) publish();
        // a claim that is never published, or a table without an empty slot, ends the wait
        if (waiting && ++spins >= kSpinLimit) {
            atomicOr(err, (uint32_t)DE_TIMEOUT);
            any = false;
        }
        if (++steps > t.mask + kSpinLimit) any = false;
        if (!any) {
#pragma unroll
            for (int k = 0; k < K; k++) need[k] = false;
        }
    }
    if (__any_sync(0xFFFFFFFFu, claimed != 0)) publish();  // a lane gave up above
    return made;
}

// Merge a shared-memory partial (word(s) at src) into the global block word(s) at dst.
__device__ __forceinline__ void acc_merge(int kind, uint64_t* dst, const uint64_t* src) {
    uint64_t v = src[0];
    switch (kind) {
        case A_SUM_I64:
        case A_COUNT: if (v) atomicAdd((unsigned long long*)dst, (unsigned long long)v); break;
        case A_SUM_F64: atomicAdd((double*)dst, as_f64(v)); break;
        case A_AVG:
            atomicAdd((double*)dst, as_f64(v));
            if (src[1]) atomicAdd((unsigned long long*)dst + 1, (unsigned long long)src[1]);
            break;
        case A_MIN_I64: atomicMin((long long*)dst, (long long)v); break;
        case A_MAX_I64: atomicMax((long long*)dst, (long long)v); break;
        case A_MIN_F64:
        case A_MIN_STR: atomicMin((unsigned long long*)dst, (unsigned long long)v); break;
        case A_MAX_F64:
        case A_MAX_STR: atomicMax((unsigned long long*)dst, (unsigned long long)v); break;
    }
}

// Append the row combination to the overflow list.  The lanes that overflow together take
// their slots with one atomic per warp (a full table sends every new key here).
__device__ inline void record_overflow(const PipeArgs& P, const AggArgs& A, const RowCtx& x) {
    const unsigned m = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
    unsigned long long base = 0;
    if (lane == leader) base = atomicAdd(A.ovf_count, (unsigned long long)__popc(m));
    base = __shfl_sync(m, base, leader);
    const unsigned long long k = base + __popc(m & ((1u << lane) - 1u));
    if (k >= A.ovf_cap) {
        atomicOr(P.err, (uint32_t)DE_OVERFLOW_LOST);
        return;
    }
    int w = 1 + P.nprobes;
    uint32_t* o = A.ovf + k * (uint64_t)w;
    o[0] = x.r;
    if (w > 1) o[1] = x.b0;
    if (w > 2) o[2] = x.b1;
    if (w > 3) o[3] = x.b2;
    if (w > 4) o[4] = x.b3;
}

// The CTA's direct group index (AggArgs::dslots): entry = group id + 1, 0 until a thread of
// this CTA has looked the slot's key up in the global table.  Every writer of an entry writes
// the same value (a slot stands for one key), so readers need no ordering: a 0 read only sends
// the row to the global table.
__device__ __forceinline__ uint32_t* direct_slots(const AggArgs& A, uint64_t* smem) {
    return (uint32_t*)(smem + (uint64_t)A.smem_groups * A.stride + (uint64_t)A.priv_groups * A.stride * 256);
}

__device__ inline void smem_setup(const AggArgs& A, uint64_t* smem) {
    for (int g = threadIdx.x; g < A.smem_groups; g += blockDim.x) {
        uint64_t* b = smem + (uint64_t)g * A.stride;
        for (int w = 0; w < A.stride; w++) b[w] = 0;
        for (int k = 0; k < A.nagg; k++)
            if (A.aggs[k].func != ML_AGG_COUNT_STAR) b[A.aggs[k].off] = agg_identity(A.aggs[k].kind);
    }
    if (agg_direct_on(A)) {
        uint32_t* d = direct_slots(A, smem);
        for (int i = threadIdx.x; i < kDirectSlots; i += blockDim.x) d[i] = 0;
    }
}

__device__ inline void smem_flush(const AggArgs& A, const uint64_t* smem) {
    for (int g = threadIdx.x; g < A.smem_groups; g += blockDim.x) {
        const uint64_t* b = smem + (uint64_t)g * A.stride;
        if (!b[0]) continue;
        uint64_t* d = A.acc + (uint64_t)g * A.stride;
        atomicAdd((unsigned long long*)d, (unsigned long long)b[0]);
        for (int k = 0; k < A.nagg; k++) {
            const AggDev& a = A.aggs[k];
            if (a.func == ML_AGG_COUNT_STAR) continue;
            acc_merge(a.kind, d + a.off, b + a.off);
        }
    }
}

}  // namespace mlg
