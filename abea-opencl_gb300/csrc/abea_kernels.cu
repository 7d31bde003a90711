// abea_kernels.cu — the three ABEA stages as sm_103a kernels.
//
//   pre   (abea_pre_kernel)    k-mer ranks -> per-position scaled pore-model
//                              parameters; event means; last-column init.
//                              Replaces align_kernel_pre_2d (GPU/align_cuda.cl:162-276).
//   core                       the adaptive banded max-plus fill.
//                              Replaces align_kernel_core_2d_shm (GPU/align_cuda.cl:297-609).
//   post  (post_read_warp)     best end, traceback, reverse, quality checks.
//                              Replaces align_kernel_post (GPU/align_cuda.cl:618-899).
//
// Fill shapes (all bit-exact, same trace layout):
//   warp   — one warp per read, lane l holds k-mer slots 4l..4l+3.  Neighbour
//            scores move by one shuffle per band, the band move is decided from two
//            shuffled end cells; no block barrier.  Most reads per SM.
//   wide   — one read per 512-thread block (fill_chain): a few warps run the band-to-band
//            chain, cells exchanged in shared memory, the others compute the emissions
//            ahead of it.  Shortest band latency.
// Forms:
//   plain   — pre, core (warp shape, one block per read), post (one block per
//             read): the reference's three launches.
//   batched — one persistent kernel of one block per SM (each read's pre runs
//             in the block or warp that fills it): the blocks take the wide reads
//             from a queue, longest first, one after another, each walking its
//             read's traceback with the whole block (post_wide_block); the blocks
//             without a wide read take the first wave of the other reads
//             round-robin, one per warp, and then every warp pulls the rest
//             longest-first from a device queue; a warp-shape read's post runs in the
//             warp that filled it, right after its fill (trace still in L2).
//   The wide shape on a cluster of two blocks (emissions on the second SM) is an
//   option, measured slower.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <stdio.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "abea_cell.cuh"
#include "abea_internal.h"
#include "abea_launch.h"

namespace abea {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kPostChunkBands = 16;  // trace bands per chunk of post's four-chunk shared-memory ring

__host__ __device__ __forceinline__ int round_up_dev(int x) { return (x + kChunk - 1) & ~(kChunk - 1); }

// ---------------------------------------------------------------- helpers
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_group1() { asm volatile("cp.async.wait_group 1;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ float sel4(const float (&v)[4], int j) {
    float r = v[0];
    r = (j == 1) ? v[1] : r;
    r = (j == 2) ? v[2] : r;
    r = (j == 3) ? v[3] : r;
    return r;
}

// k-mer rank, first base most significant; non-ACGT -> 0 (GPU/align_cuda.cl:22-51).
__device__ __forceinline__ uint32_t base_rank(char c) { return c == 'C' ? 1u : c == 'G' ? 2u : c == 'T' ? 3u : 0u; }

__device__ __forceinline__ CellConsts make_consts(const ReadDesc& r, const GlobalConsts& g) {
    CellConsts c;
    c.step_h = r.step_h;
    c.step_l = r.step_l;
    c.stay_h = r.stay_h;
    c.stay_l = r.stay_l;
    c.skip_h = g.skip_h;
    c.skip_l = g.skip_l;
    c.lp_step = r.lp_step;
    c.lp_stay = r.lp_stay;
    c.lp_skip = g.lp_skip;
    return c;
}

// ---------------------------------------------------------------- pre
// One block per read; thread t handles k-mer positions t, t+blockDim, ...
// Pre of read i by nt cooperating threads (thread index t): the read's k-mer
// parameters, event means and last-column initialisation.  The batched form runs
// it in the block or warp that fills the read, just before the fill.
//
// The bases and events come from HBM, or, when the caller's buffers are pinned
// (a.inm), straight from host memory over the CPU-GPU link: no copy of the
// inputs precedes the kernel, and every read's pre stage loads its own (but the
// first few reads the kernel starts, copied to HBM before it: in_hbm).  A thread
// takes kPreUnroll k-mer positions (kEvUnroll events) per pass with every load
// issued before any use (indexes clamped into the read), so that many round trips
// to host memory are in flight at once: a warp-shape read's pre stage is latency-
// bound on them (a k-mer's six bases share the cache lines of its neighbours').
constexpr int kPreUnroll = 4, kEvUnroll = 16;
// kWide: the read's parameters side by side too (km4), for the wide shape; returns whether
// some k-mer of this thread's is none for a grid (grid_kmer_ok).
template <bool kWide>
__device__ __forceinline__ bool pre_read(const PreArgs& a, int i, int t, int nt) {
    const ReadDesc r = a.reads[i];
    if (r.skip) return false;
    const float k1_max = kWide ? grid_k1_max(r.step_h, r.stay_h) : 0.0f;
    bool odd = false;
    const InMirror* m = r.in_hbm ? nullptr : a.inm;
    const char* seq = a.seq;
    const abea_event_t* ev_in = a.ev_in;
    if (m) {
        const InMirror mv = *m;
        if (mv.seq) seq = mv.seq;
        if (mv.ev) ev_in = mv.ev;
    }
    const char* s = seq + r.seq_off;
    const int nk = r.n_kmers, nk_pad = round_up_dev(nk);
    for (int k0 = t; k0 < nk_pad; k0 += kPreUnroll * nt) {
        char base[kPreUnroll][ABEA_KMER_SIZE];
#pragma unroll
        for (int u = 0; u < kPreUnroll; ++u) {
            const int kc = min(k0 + u * nt, nk - 1);  // nk >= 1: the read is not skipped
#pragma unroll
            for (int j = 0; j < ABEA_KMER_SIZE; ++j) base[u][j] = s[kc + j];
        }
#pragma unroll
        for (int u = 0; u < kPreUnroll; ++u) {
            const int k = k0 + u * nt;
            if (k >= nk_pad) break;
            float gm = 0.f, sd = 1.f, rsd = 1.f, k1 = 0.f;
            if (k < nk) {
                uint32_t rank = 0;
#pragma unroll
                for (int j = 0; j < ABEA_KMER_SIZE; ++j) rank = (rank << 2) | base_rank(base[u][j]);
                abea_model_t mm = a.model[rank];
                // gp_mean = scale*level_mean + shift; gp_stdv = level_stdv (scaling.var is
                // ignored by the reference, GPU/align_cuda.cl:509); cached log stdv.
                gm = __fadd_rn(__fmul_rn(r.scale, mm.level_mean), r.shift);
                sd = mm.level_stdv;
                float lsd = mm.level_log_stdv;
                if (a.g.var_aware) {
                    sd = __fmul_rn(sd, r.var);
                    lsd = __fadd_rn(lsd, r.log_var);
                }
                rsd = __frcp_rn(sd);
                k1 = __fsub_rn(kLogInvSqrt2Pi, lsd);
                if (kWide) odd |= !grid_kmer_ok(sd, k1, k1_max);
            }
            a.km_gm[r.km_off + k] = gm;
            a.km_sd[r.km_off + k] = sd;
            a.km_rsd[r.km_off + k] = rsd;
            a.km_k1[r.km_off + k] = k1;
            if (kWide) a.km4[r.km_off + k] = make_float4(gm, sd, rsd, k1);
        }
    }
    const int ne = r.n_events, ne_pad = round_up_dev(ne);
    const abea_event_t* ev = ev_in + r.ev_src;
    for (int e0 = t; e0 < ne_pad; e0 += kEvUnroll * nt) {
        float mean[kEvUnroll];
#pragma unroll
        for (int u = 0; u < kEvUnroll; ++u) mean[u] = ev[min(e0 + u * nt, ne - 1)].mean;  // ne >= 1
#pragma unroll
        for (int u = 0; u < kEvUnroll; ++u) {
            const int e = e0 + u * nt;
            if (e >= ne_pad) break;
            a.ev_mean[r.ev_off + e] = e < ne ? mean[u] : 0.f;
            a.last_col[r.ev_off + e] = -INFINITY;
        }
    }
    return odd;
}

__global__ void __launch_bounds__(128) abea_pre_kernel(PreArgs a) {
    const int i = blockIdx.x;
    if (i >= a.n_reads) return;
    pre_read<false>(a, i, threadIdx.x, blockDim.x);
}

// ---------------------------------------------------------------- prefetch rings
// k-mer parameters live in a 128-entry ring indexed by k-mer & 127 (= the slot),
// event means in a 256-entry ring indexed by event & 255.  Chunks of 16 are
// copied with cp.async as soon as the entries they overwrite have left the band:
// a k-mer chunk [c, c+16) once c+15 <= k0+127, an event chunk once c+15 <= e0+156.
// 16-byte aligned: cp.async copies 16 bytes and the warp shape reads float4s.
struct alignas(16) Rings {
    float gm[kSlots];
    float sd[kSlots];
    float rsd[kSlots];
    float k1[kSlots];
    float ev[kEvRing];
    float4 save[2][32];  // the warp shape's state before a chunk on a grid
};

struct RingState {
    int k_iss, e_iss, k_rdy, e_rdy, km_end, ev_end;
};

// `t` = index of the calling thread among the read's cooperating threads (>= 20).
__device__ __forceinline__ void issue_chunks(Rings& rg, const CoreArgs& a, const ReadDesc& r, int t, bool do_k,
                                             int kc, bool do_e, int ec) {
    if (do_k && t < 16) {
        const int arr = t >> 2, part = t & 3;
        const float* base = arr == 0 ? a.km_gm : arr == 1 ? a.km_sd : arr == 2 ? a.km_rsd : a.km_k1;
        float* dst = arr == 0 ? rg.gm : arr == 1 ? rg.sd : arr == 2 ? rg.rsd : rg.k1;
        cp_async16(dst + ((kc + 4 * part) & (kSlots - 1)), base + r.km_off + kc + 4 * part);
    }
    if (do_e && t >= 16 && t < 20) {
        const int part = t & 3;
        cp_async16(&rg.ev[(ec + 4 * part) & (kEvRing - 1)], a.ev_mean + r.ev_off + ec + 4 * part);
    }
}

// Initial fill for the band-1 window (k0 = -51, e0 = 50).  Caller syncs.
__device__ __forceinline__ void rings_init(Rings& rg, RingState& rs, const CoreArgs& a, const ReadDesc& r, int t,
                                           int k0, int e0) {
    rs.km_end = round_up_dev(r.n_kmers);
    rs.ev_end = round_up_dev(r.n_events);
    rs.k_iss = 0;
    rs.e_iss = 0;
    while (rs.k_iss < rs.km_end && rs.k_iss + 15 <= k0 + 127) {
        issue_chunks(rg, a, r, t, true, rs.k_iss, false, 0);
        rs.k_iss += kChunk;
    }
    while (rs.e_iss < rs.ev_end && rs.e_iss + 15 <= e0 + 156) {
        issue_chunks(rg, a, r, t, false, 0, true, rs.e_iss);
        rs.e_iss += kChunk;
    }
    cp_async_commit();
    cp_async_wait_all();
    rs.k_rdy = rs.k_iss;
    rs.e_rdy = rs.e_iss;
}

// Initial fill for a window (k0, e0) reached in the middle of a read (a resumed
// checkpoint): the chunks that hold the window's k-mers and events, from the
// 16-aligned chunk at or below k0 (events: e0 - 100), at most one ring's worth.
// Caller syncs.
__device__ __forceinline__ void rings_seek(Rings& rg, RingState& rs, const CoreArgs& a, const ReadDesc& r, int t,
                                           int k0, int e0) {
    rs.km_end = round_up_dev(r.n_kmers);
    rs.ev_end = round_up_dev(r.n_events);
    const int k_start = max(k0, 0) & ~(kChunk - 1), e_start = max(e0 - kBand, 0) & ~(kChunk - 1);
    rs.k_iss = k_start;
    rs.e_iss = e_start;
    while (rs.k_iss < rs.km_end && rs.k_iss + 15 <= k0 + 127 && rs.k_iss < k_start + kSlots) {
        issue_chunks(rg, a, r, t, true, rs.k_iss, false, 0);
        rs.k_iss += kChunk;
    }
    while (rs.e_iss < rs.ev_end && rs.e_iss + 15 <= e0 + 156 && rs.e_iss < e_start + kEvRing) {
        issue_chunks(rg, a, r, t, false, 0, true, rs.e_iss);
        rs.e_iss += kChunk;
    }
    cp_async_commit();
    cp_async_wait_all();
    rs.k_rdy = rs.k_iss;
    rs.e_rdy = rs.e_iss;
}

// Called once per group of bands with the current window: waits for the data the
// next `ahead` bands need and issues the chunks whose ring entries are free.
// Returns true when it waited (the caller then syncs the cooperating threads).
__device__ __forceinline__ bool rings_step(Rings& rg, RingState& rs, const CoreArgs& a, const ReadDesc& r, int t,
                                           int k0, int e0, int ahead) {
    bool waited = false;
    const int k_prev = rs.k_iss, e_prev = rs.e_iss;  // issued before this call
    const bool do_k = rs.k_iss < rs.km_end && rs.k_iss + 15 <= k0 + 127;
    const bool do_e = rs.e_iss < rs.ev_end && rs.e_iss + 15 <= e0 + 156;
    if (do_k || do_e) {
        issue_chunks(rg, a, r, t, do_k, rs.k_iss, do_e, rs.e_iss);
        cp_async_commit();
        if (do_k) rs.k_iss += kChunk;
        if (do_e) rs.e_iss += kChunk;
    }
    auto needs = [&](int k_have, int e_have) {
        return (k0 + kBand - 1 + ahead >= k_have && k_have < rs.km_end) || (e0 + ahead >= e_have && e_have < rs.ev_end);
    };
    if (needs(rs.k_rdy, rs.e_rdy)) {
        if ((do_k || do_e) && !needs(k_prev, e_prev)) {
            // the chunks just issued are not needed yet: wait for the older ones only
            cp_async_wait_group1();
            rs.k_rdy = k_prev;
            rs.e_rdy = e_prev;
        } else {
            cp_async_wait_all();
            rs.k_rdy = rs.k_iss;
            rs.e_rdy = rs.e_iss;
        }
        waited = true;
    }
    return waited;
}

// Computed offsets [lo, hi) of a band (GPU/align_cuda.cl:457-470).
__device__ __forceinline__ void band_range(int k0, int e0, int n_events, int n_kmers, int& lo, int& hi) {
    lo = max(max(-k0, e0 - (n_events - 1)), 0);
    hi = min(min(n_kmers - k0, e0 + 1), kBand);
}

// ---------------------------------------------------------------- warp shape
// Slot s of a band holds the cell of k-mer k(s) = k0 + ((s - k0) & 127) and event
// e = (band - 2) - k(s).  A slot inside band b+1 has kept its k-mer since band
// b-1, so its event is two more than under band b-1's placement: the emission of
// band b+1 and its exact diagonal candidate (diagonal = left neighbour of band b)
// are computed during band b, before band b's own placement is decided.  Band b
// itself then only needs its up candidate (from the slot's own previous score),
// the exchange of neighbour cells, the skip candidate and the comparison.

// 4x4 byte transpose: w[j] holds band j's backpointers of slots 0..3 (byte s);
// returns o[s] holding slot s's backpointers of bands 0..3 (byte j).
__device__ __forceinline__ uint4 transpose_bytes(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) {
    const uint32_t a = __byte_perm(w0, w1, 0x5140), c = __byte_perm(w2, w3, 0x5140);
    const uint32_t b = __byte_perm(w0, w1, 0x7362), d = __byte_perm(w2, w3, 0x7362);
    return make_uint4(__byte_perm(a, c, 0x5410), __byte_perm(a, c, 0x7632), __byte_perm(b, d, 0x5410),
                      __byte_perm(b, d, 0x7632));
}

// The bands a fill_warp call computes and where its results go.
//   forward pass: bands [2, n_bands), band-side outputs (last column, band
//     origins, scores, slow-cell count) written, the trace into `trace` (kept
//     traces) or checkpoints into `ck_out` (checkpointed reads);
//   recompute: bands [b_begin, b_end) of a checkpointed read from the record
//     `ck_in` (nullptr: from the start), the trace into a scratch segment.
// Trace band b is stored at trace + trace_index(b - trace_band0, slot).
struct FillSpan {
    int b_begin, b_end;
    const float* ck_in;
    float* ck_out;
    uint8_t* trace;
    int trace_band0;
    int trace_tiles;  // 4-band tiles in the trace region (bounds checks)
    bool side;
};

// Debug builds (ABEA_BOUNDS_CHECK): the global stores of the fill and of the
// traceback check their index against their region; a store out of it is skipped
// and counted (the run then reports ABEA_ERR_INTERNAL).
#ifdef ABEA_BOUNDS_CHECK
__device__ __forceinline__ bool in_bounds(int64_t i, int64_t n, unsigned long long* counters) {
    const bool ok = i >= 0 && i < n;
    if (!ok) atomicAdd(&counters[kCountBounds], 1ull);
    return ok;
}
#else
__device__ __forceinline__ bool in_bounds(int64_t, int64_t, unsigned long long*) { return true; }
#endif

__device__ __forceinline__ FillSpan forward_span(const CoreArgs& a, const ReadDesc& r) {
    FillSpan sp;
    sp.b_begin = 2;
    sp.b_end = r.n_bands;
    sp.ck_in = nullptr;
    sp.ck_out = r.ck ? a.ck + r.ck_off : nullptr;
    sp.trace = r.ck ? nullptr : a.trace + r.trace_off * kSlots;
    sp.trace_band0 = 0;
    sp.trace_tiles = r.ck ? 0 : (r.n_bands + 3) / 4;
    sp.side = true;
    return sp;
}

// kSpan = false: the forward pass of a read that keeps its trace, with none of
// the span's choices left to run time (the common case); kSpan = true: any span.
template <bool kScores, bool kSpan>
__device__ void fill_warp(const CoreArgs& a, const ReadDesc& r, Rings& rg, int lane, const FillSpan& spr) {
    FillSpan sp = spr;
    if (!kSpan) {
        sp.b_begin = 2;
        sp.b_end = r.n_bands;
        sp.ck_in = nullptr;
        sp.ck_out = nullptr;
        sp.trace = a.trace + r.trace_off * kSlots;
        sp.trace_band0 = 0;
        sp.trace_tiles = (r.n_bands + 3) / 4;
        sp.side = true;
    }
    const CellConsts cc = make_consts(r, a.g);
    const int n_events = r.n_events, n_kmers = r.n_kmers, n_bands = sp.b_end;
    uint8_t* trace = sp.trace;
    float* scores = kScores && sp.side ? a.scores + r.band_off * kSlots : nullptr;

    // band 0: start cell (e=-1,k=-1) = 0 in slot 127; band 1: trim cell (e=0,k=-1)
    // = (float)lp_trim, FROM_U, slot 127 (GPU/align_cuda.cl:249-268).  A resumed
    // checkpoint gives band b_begin-1's scores and placement and band
    // b_begin-2's scores shifted by one slot.
    int k0 = -1 - kBand / 2, e0 = kBand / 2;  // band 1 (band 0 is (49,-51), band 1 moved down)
    float S1[4], LP[4];
    if (kSpan && sp.ck_in) {
        const float4 s4 = reinterpret_cast<const float4*>(sp.ck_in)[lane];
        const float4 l4 = reinterpret_cast<const float4*>(sp.ck_in + kSlots)[lane];
        S1[0] = s4.x; S1[1] = s4.y; S1[2] = s4.z; S1[3] = s4.w;
        LP[0] = l4.x; LP[1] = l4.y; LP[2] = l4.z; LP[3] = l4.w;
        k0 = __float_as_int(sp.ck_in[2 * kSlots]);
        e0 = __float_as_int(sp.ck_in[2 * kSlots + 1]);
    }
    RingState rs;
    if (kSpan && sp.ck_in)
        rings_seek(rg, rs, a, r, lane, k0, e0);
    else
        rings_init(rg, rs, a, r, lane, k0, e0);
    __syncwarp();

    int ep[4];  // event of each slot under the previous band's placement
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (!sp.ck_in) S1[j] = LP[j] = -INFINITY;
        ep[j] = e0 - ((4 * lane + j - k0) & 127);
    }
    if (!sp.ck_in) {
        if (lane == 31) S1[3] = a.g.trim_f;
        if (lane == 0) LP[0] = 0.0f;  // band 0 shifted by one slot = diagonal source of band 2
    }
    if (kScores && scores) {
        float4 b0 = make_float4(-INFINITY, -INFINITY, -INFINITY, lane == 31 ? 0.0f : -INFINITY);
        float4 b1 = make_float4(-INFINITY, -INFINITY, -INFINITY, lane == 31 ? a.g.trim_f : -INFINITY);
        reinterpret_cast<float4*>(scores)[lane] = b0;
        reinterpret_cast<float4*>(scores + kSlots)[lane] = b1;
    }
    NextCell nc[4];  // band b's emission side, prepared during band b-1
    {
        const float4 gm4 = *reinterpret_cast<const float4*>(&rg.gm[4 * lane]);
        const float4 sd4 = *reinterpret_cast<const float4*>(&rg.sd[4 * lane]);
        const float4 rs4 = *reinterpret_cast<const float4*>(&rg.rsd[4 * lane]);
        const float4 k14 = *reinterpret_cast<const float4*>(&rg.k1[4 * lane]);
        const float gmv[4] = {gm4.x, gm4.y, gm4.z, gm4.w}, sdv[4] = {sd4.x, sd4.y, sd4.z, sd4.w};
        const float rsv[4] = {rs4.x, rs4.y, rs4.z, rs4.w}, k1v[4] = {k14.x, k14.y, k14.z, k14.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
            nc[j] = next_cell(LP[j], rg.ev[(ep[j] + 1) & (kEvRing - 1)], gmv[j], sdv[j], rsv[j], k1v[j], cc);
    }
    int my_k0 = k0;  // bands 0 and 1 (lanes 0, 1) both have k0 = -51
    unsigned slow = 0;
    const int sl_last = (n_kmers - 1) & 127;
    uint32_t tw0 = 0u, tw1 = (lane == 31 && !sp.ck_in) ? (ABEA_FROM_U << 24) : 0u, tw2 = 0u, tw3 = 0u;

    // Band state kept across the exit to the slow path: a band in which a proof
    // failed in any lane leaves the inner loop (warp-uniform) and is finished
    // below with the reference's FP64 arithmetic, so that the inner loop holds
    // no division routine and no FP64 code.
    int b = sp.b_begin, lo = 0, hi = 0;
    float best[4], left[4];
    uint32_t from[4];
    bool valid[4], bad[4];
    NextCell nn[4];
    auto finish = [&]() {
        uint32_t word = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            best[j] = valid[j] ? best[j] : -INFINITY;
            word |= (valid[j] ? from[j] : 0u) << (8 * j);
        }
        // edges of the read: trim cell (k = -1, slot 127; GPU/align_cuda.cl:431-443)
        // and the last k-mer column read by the post stage (GPU/align_cuda.cl:722-746)
        const int ol = n_kmers - 1 - k0;
        if (k0 <= -1 || ol < kBand) {
            if (k0 <= -1) {  // uniform
                const int e_t = e0 + 1 + k0;
                const bool in = e_t >= 0 && e_t < n_events;
                const float tv = in ? __double2float_rn(__dmul_rn(a.g.lp_trim, (double)(e_t + 1))) : -INFINITY;
                const bool here = lane == 31 && k0 >= -kBand;
                best[3] = here ? tv : best[3];
                word = here ? ((word & 0x00ffffffu) | (in ? (ABEA_FROM_U << 24) : 0u)) : word;
            }
            if (sp.side && ol >= lo && ol < hi && lane == (sl_last >> 2) && in_bounds(e0 - ol, n_events, a.counters))
                (a.last_col + r.ev_off)[e0 - ol] = sel4(best, sl_last & 3);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            LP[j] = left[j];
            S1[j] = best[j];
            nc[j] = nn[j];
        }
        const int jb = b & 3;
        tw0 = jb == 0 ? word : tw0;
        tw1 = jb == 1 ? word : tw1;
        tw2 = jb == 2 ? word : tw2;
        tw3 = jb == 3 ? word : tw3;
        if (jb == 3 || b == n_bands - 1) {
            if ((!kSpan || trace) && in_bounds((b - sp.trace_band0) >> 2, sp.trace_tiles, a.counters))
                reinterpret_cast<uint4*>(trace + (int64_t)((b - sp.trace_band0) >> 2) * 512)[lane] =
                    transpose_bytes(tw0, tw1, tw2, tw3);
            tw0 = tw1 = tw2 = tw3 = 0u;
        }
        if (kScores && scores && in_bounds(b, r.n_bands, a.counters))
            reinterpret_cast<float4*>(scores + (int64_t)b * kSlots)[lane] = make_float4(best[0], best[1], best[2], best[3]);
        my_k0 = ((b & 31) == lane) ? k0 : my_k0;
        if (sp.side && ((b & 31) == 31 || b == n_bands - 1)) {
            if (lane <= (b & 31) && in_bounds((b & ~31) + lane, r.n_bands, a.counters)) (a.band_k0 + r.band_off)[(b & ~31) + lane] = my_k0;
        }
    };
    // Four bands at a time on a grid (abea_cell.cuh, "candidates on a grid") where the
    // band lies inside the read and its scores are in a grid's range: the diagonal and up
    // candidates are one add each, their parts made and proven here, band by band.  The
    // same conditions and the same end-of-chunk check as the wide shape's grid engine; a
    // chunk that fails it runs again in the exact loop below.  Not unrolled over the bands:
    // the loop body stays small (up to sixteen warps on an SM, each at its own place).
    // A read of 20 kb alone: 1,050 cycles per band before, 530 now (the plain form's f5c
    // batch 33.4 -> 17.5 ms); sixteen warps on an SM 131 together.
    //   The exact loop carries no more of it than grid_from, the first band that may try, and
    // pen, the recent failures: a grid is made anew for each run of tiles (kept between runs it
    // cost the exact loop its registers: 300 reads of 0.5-6 kb two to an SM 7.57 ms, now 6.53,
    // with scalings off, where no band tries, 13.0 and 12.2; the exact loop alone had 11.6).
    int grid_from = sp.b_begin, pen = 0;
    auto grid_now = [&]() {
        bool hole = false;
        float mx = -INFINITY, mn = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            hole |= (((4 * lane + j - k0) & 127) < kBand) & (S1[j] == -INFINITY);
            mx = max_nan(max_nan(mx, S1[j]), LP[j]);
            mn = fminf(fminf(mn, S1[j] > -INFINITY ? S1[j] : 0.0f), LP[j] > -INFINITY ? LP[j] : 0.0f);
        }
        const bool none = __any_sync(kFull, hole || mx != mx);
        mx = warp_max(mx);
        mn = warp_min(mn);
        const int m = (__float_as_int(-mx) >> 23) - 127, mlo = (__float_as_int(-mn) >> 23) - 127;
        return !none && m >= kGridMin && m <= kGridMax && mlo < m + 2 ? m : 0;
    };
    // bands b .. b + 3; false (and the state as it was) when the check fails
    auto grid_bands = [&](auto low, const Grid& G) {
        const float k1_max = grid_k1_max(cc.step_h, cc.stay_h);
        constexpr bool kLow = decltype(low)::value;
        constexpr uint32_t kOne = 1u << 25, kIn = (uint32_t)kBand << 25;
        const int k_was = k0, my_was = my_k0;
        rg.save[0][lane] = make_float4(S1[0], S1[1], S1[2], S1[3]);
        rg.save[1][lane] = make_float4(LP[0], LP[1], LP[2], LP[3]);
        float4 km[4];  // {gm, sd, rsd, k1} of the lane's slots
        {
            const float4 gm4 = *reinterpret_cast<const float4*>(&rg.gm[4 * lane]);
            const float4 sd4 = *reinterpret_cast<const float4*>(&rg.sd[4 * lane]);
            const float4 rs4 = *reinterpret_cast<const float4*>(&rg.rsd[4 * lane]);
            const float4 k14 = *reinterpret_cast<const float4*>(&rg.k1[4 * lane]);
            km[0] = make_float4(gm4.x, sd4.x, rs4.x, k14.x);
            km[1] = make_float4(gm4.y, sd4.y, rs4.y, k14.y);
            km[2] = make_float4(gm4.z, sd4.z, rs4.z, k14.z);
            km[3] = make_float4(gm4.w, sd4.w, rs4.w, k14.w);
        }
        int e[4];  // event of each slot in band b
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            km[j].x = grid_kmer_ok(km[j].y, km[j].w, k1_max) ? km[j].x : __int_as_float(0x7fc00000);
            e[j] = b - 2 - (k0 + ((4 * lane + j - k0) & 127));
        }
        const float g_lim = G.lim * kGridLimLo;
        uint32_t vs = (uint32_t)(4 * lane - k0) << 25, w[4] = {0u, 0u, 0u, 0u};
        bool below = false;
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
            const int sl = k0 & 127, su = (k0 + kBand - 1) & 127;
            const float ll = __shfl_sync(kFull, sel4(S1, sl & 3), sl >> 2);
            const float ur = __shfl_sync(kFull, sel4(S1, su & 3), su >> 2);
            const float left0 = __shfl_sync(kFull, S1[3], (lane + 31) & 31);
            const float l4[4] = {left0, S1[0], S1[1], S1[2]};
            float top[4], sk[4], up[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 x = grid_pair<kLow>(rg.ev[(e[j] + q) & (kEvRing - 1)], km[j].x, km[j].y, km[j].z, km[j].w, G);
                const float d = __fadd_rn(LP[j], x.x);
                up[j] = __fadd_rn(S1[j], x.y);
                sk[j] = __fadd_rn(l4[j], G.skip);
                top[j] = max3_nan(d, up[j], sk[j]);
                if (kLow) below |= (x.y < g_lim) & (top[j] != sk[j]);
            }
            const bool right = ll < ur;  // both ends are finite
            k0 += right ? 1 : 0;
            vs -= right ? kOne : 0u;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (top[j] == sk[j]) w[j] |= ABEA_FROM_L << (8 * q);
                if (top[j] == up[j] && top[j] != sk[j]) w[j] |= ABEA_FROM_U << (8 * q);
                LP[j] = l4[j];
                S1[j] = vs + (uint32_t)j * kOne < kIn ? top[j] : -INFINITY;
            }
            my_k0 = (((b + q) & 31) == lane) ? k0 : my_k0;
            if (kScores && scores && in_bounds(b + q, r.n_bands, a.counters))
                reinterpret_cast<float4*>(scores + (int64_t)(b + q) * kSlots)[lane] = make_float4(S1[0], S1[1], S1[2], S1[3]);
        }
        const float mx = max_nan(max_nan(S1[0], S1[1]), max_nan(S1[2], S1[3]));
        if (__any_sync(kFull, below | (mx != mx))) {
            const float4 s4 = rg.save[0][lane], l4 = rg.save[1][lane];
            S1[0] = s4.x; S1[1] = s4.y; S1[2] = s4.z; S1[3] = s4.w;
            LP[0] = l4.x; LP[1] = l4.y; LP[2] = l4.z; LP[3] = l4.w;
            k0 = k_was;
            my_k0 = my_was;
            return false;
        }
        e0 = b + 3 - 2 - k0;
        if ((!kSpan || trace) && in_bounds((b - sp.trace_band0) >> 2, sp.trace_tiles, a.counters))
            reinterpret_cast<uint4*>(trace + (int64_t)((b - sp.trace_band0) >> 2) * 512)[lane] = make_uint4(w[0], w[1], w[2], w[3]);
        if (sp.side && ((b + 3) & 31) == 31) {
            if (in_bounds(((b + 3) & ~31) + lane, r.n_bands, a.counters)) (a.band_k0 + r.band_off)[((b + 3) & ~31) + lane] = my_k0;
        }
        return true;
    };
    // checkpoint b / kCkBands, when band b has one: the state this loop resumes from there
    auto checkpoint = [&]() {
        if (kSpan && sp.ck_out && (b & (kCkBands - 1)) == 0 &&
            in_bounds(b / kCkBands, r.n_bands / kCkBands + 1, a.counters)) {
            float* rec = sp.ck_out + (int64_t)(b / kCkBands) * kCkStride;
            reinterpret_cast<float4*>(rec)[lane] = make_float4(S1[0], S1[1], S1[2], S1[3]);
            reinterpret_cast<float4*>(rec + kSlots)[lane] = make_float4(LP[0], LP[1], LP[2], LP[3]);
            if (lane == 0) {
                rec[2 * kSlots] = __int_as_float(k0);
                rec[2 * kSlots + 1] = __int_as_float(e0);
            }
        }
    };
    // all 100 cells of bands b .. b + 3 are computed, none on the last k-mer column
    auto inside = [&]() {
        return b + 4 <= n_bands && k0 >= 0 && k0 + 4 + kBand <= n_kmers - 1 && e0 >= kBand - 1 && e0 + 4 <= n_events - 1;
    };
    while (true) {
        bool to_slow = false;
        for (; b < n_bands; ++b) {
            checkpoint();
            if ((b & 3) == 0) {
                if (rings_step(rg, rs, a, r, lane, k0, e0, 6)) __syncwarp();
                if (b >= grid_from && inside()) {
                    const int b_first = b;
                    Grid G{};
                    int made = 0, until = 0;
                    do {
                        if (b >= until) {
                            int m = grid_now();
                            until = b + 16;
                            if (m && m != made) {
                                bool ok1, ok2, ok3;
                                grid_step(cc.step_h, cc.step_l, m, ok1);
                                grid_step(cc.stay_h, cc.stay_l, m, ok2);
                                grid_step(cc.skip_h, cc.skip_l, m, ok3);
                                G = make_grid(cc, m);
                                if (!(ok1 && ok2 && ok3)) m = 0;
                            }
                            made = m;
                            if (!m) {
                                grid_from = until;
                                break;
                            }
                        }
                        if (!(made < kGridWide ? grid_bands(std::true_type{}, G) : grid_bands(std::false_type{}, G))) {
                            // these four bands exact; many more after repeated failures
                            pen = pen < 32 ? pen + 8 : min(2 * pen, 4096);
                            grid_from = b + 4 + (pen > 32 ? 4 * pen : 0);
                            if (lane == 0 && sp.side) atomicAdd(&a.counters[kCountGridAgain], 1ull);
                            break;
                        }
                        pen = max(pen - 1, 0);
                        b += 4;
                        checkpoint();
                        if (rings_step(rg, rs, a, r, lane, k0, e0, 6)) __syncwarp();
                    } while (inside());
                    if (lane == 0 && sp.side) atomicAdd(&a.counters[kCountGrid], (unsigned long long)((b - b_first) >> 2));
                    if (b >= n_bands) break;
                    // back to the exact loop: band b's emission side
                    const float4 gm4 = *reinterpret_cast<const float4*>(&rg.gm[4 * lane]);
                    const float4 sd4 = *reinterpret_cast<const float4*>(&rg.sd[4 * lane]);
                    const float4 rs4 = *reinterpret_cast<const float4*>(&rg.rsd[4 * lane]);
                    const float4 k14 = *reinterpret_cast<const float4*>(&rg.k1[4 * lane]);
                    const float gmv[4] = {gm4.x, gm4.y, gm4.z, gm4.w}, sdv[4] = {sd4.x, sd4.y, sd4.z, sd4.w};
                    const float rsv[4] = {rs4.x, rs4.y, rs4.z, rs4.w}, k1v[4] = {k14.x, k14.y, k14.z, k14.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        ep[j] = e0 - ((4 * lane + j - k0) & 127);
                        nc[j] = next_cell(LP[j], rg.ev[(ep[j] + 1) & (kEvRing - 1)], gmv[j], sdv[j], rsv[j], k1v[j], cc);
                    }
                }
            }
            // ---- exchange: end cells for the placement, left neighbour of slot 4*lane
            const int sl = k0 & 127, su = (k0 + kBand - 1) & 127;
            const float ll = __shfl_sync(kFull, sel4(S1, sl & 3), sl >> 2);
            const float ur = __shfl_sync(kFull, sel4(S1, su & 3), su >> 2);
            const float left0 = __shfl_sync(kFull, S1[3], (lane + 31) & 31);
            left[0] = left0;
            left[1] = S1[0];
            left[2] = S1[1];
            left[3] = S1[2];
            // ---- up candidates of band b
            float u[4];
            bool oku[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = cell_u(S1[j], nc[j], cc, oku[j]);
            // ---- band b+1's emission side (placement-independent)
            const float4 gm4 = *reinterpret_cast<const float4*>(&rg.gm[4 * lane]);
            const float4 sd4 = *reinterpret_cast<const float4*>(&rg.sd[4 * lane]);
            const float4 rs4 = *reinterpret_cast<const float4*>(&rg.rsd[4 * lane]);
            const float4 k14 = *reinterpret_cast<const float4*>(&rg.k1[4 * lane]);
            const float gmv[4] = {gm4.x, gm4.y, gm4.z, gm4.w}, sdv[4] = {sd4.x, sd4.y, sd4.z, sd4.w};
            const float rsv[4] = {rs4.x, rs4.y, rs4.z, rs4.w}, k1v[4] = {k14.x, k14.y, k14.z, k14.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                nn[j] = next_cell(left[j], rg.ev[(ep[j] + 2) & (kEvRing - 1)], gmv[j], sdv[j], rsv[j], k1v[j], cc);
            // ---- band placement (Suzuki-Kasahara), GPU/align_cuda.cl:394-430
            const bool right = (ll == -INFINITY && ur == -INFINITY) ? (bool)(b & 1) : (ll < ur);
            k0 += right ? 1 : 0;
            e0 += right ? 0 : 1;
            band_range(k0, e0, n_events, n_kmers, lo, hi);
            // ---- skip candidate (exact), comparison
            bool rare = false;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int o = (4 * lane + j - k0) & 127;
                ep[j] = e0 - o;
                valid[j] = (o >= lo) && (o < hi);
                uint32_t from_du;
                const float best_du = pick_du(nc[j].d, u[j], from_du);
                bool okl;
                const float l = exact_skip(left[j], cc.skip_h, cc.skip_l, okl);
                best[j] = pick_l(best_du, from_du, l, from[j]);
                bad[j] = valid[j] && !(nc[j].ok && oku[j] && okl);
                rare |= bad[j];
            }
            if (__any_sync(kFull, rare)) {
                to_slow = true;
                break;
            }
            finish();
        }
        if (!to_slow) break;
        const CellConsts cs = make_consts(r, a.g);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (bad[j]) {  // a proof failed: the reference's FP64 arithmetic
                const int sj = 4 * lane + j;
                best[j] = cell_slow(LP[j], S1[j], left[j], rg.ev[ep[j] & (kEvRing - 1)], rg.gm[sj], rg.sd[sj],
                                    rg.k1[sj], cs, from[j]);
                ++slow;
            }
        }
        finish();
        ++b;
    }
    cp_async_wait_all();  // no copy may land in shared memory after the read is done
    __syncwarp();
    if (slow && sp.side) {
        atomicAdd(&a.counters[kCountSlow], (unsigned long long)slow);
        atomicAdd(&a.counters[kCountFp64], (unsigned long long)slow);
    }
}

// Shared memory goes into a function by its own address, so that its accesses stay shared ones.
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
template <class T>
__device__ __forceinline__ T& smem_ref(unsigned at) {
    return *reinterpret_cast<T*>(__cvta_shared_to_generic(at));
}

// The one copy of the fill that all warps share when a.one_fill asks for it.
template <bool kScores>
__device__ __noinline__ void fill_span(const CoreArgs& a, const ReadDesc& r, unsigned rg_at, int lane, FillSpan sp) {
    fill_warp<kScores, true>(a, r, smem_ref<Rings>(rg_at), lane, sp);
}

// ---------------------------------------------------------------- wide shape
// A read's fill by one block of 16 warps, in chunks of four bands (a tile of
// backpointers), by two engines over one ring of band scores in shared memory:
//
//   exact (chain_exact): any band.  B, warps 0-3, one k-mer slot per thread, runs the
//     band-to-band chain with the exact sums and their proofs (abea_cell.cuh), E, warps
//     4-11, the emissions and their splits up to 16 bands ahead.  Bound by the chain's own
//     dependent instructions: 390 cycles per band, 440 where a proof fails in most bands.
//   grid (chain_grid): bands inside the read whose scores are all below -2^11.  A
//     candidate is then one add of a part that E makes and proves ahead ("candidates on
//     a grid"), the chain's bound its exchange through shared memory (94 cycles per band on
//     a bare one), and E does the backpointers.  Some 155 cycles per band, bound by the
//     chain's own latency (E waits for it half of its time).  With the exact engine
//     throughout, in an earlier form of 290 cycles per band, align() of a 20 kb read took
//     8.10 ms, now 5.0, the 1.3 Mbase batch of f5c's lengths 7.97, now 5.2, 1,024 reads of
//     1-10 kb 17.3, now 12.1.
//
// A band's cells lie on one anti-diagonal (event + k-mer = band - 2) and each band moves
// k0 by at most one, so the placement of band p gives a window [k0, k0 + 128) that holds
// the k-mers of every band up to p + 28: E works up to 28 bands ahead of B from the
// placements that B leaves in the ring.
constexpr int kWideThreads = 512;   // block size of the batched kernel
constexpr int kWideChunk = 4;       // bands per chunk
constexpr int kScoreRing = 32;      // bands of scores and placements in shared memory
constexpr int kHeadRing = 16;       // chunk headers of the grid engine
static_assert(kWideChunk == 4, "a chunk is a tile of backpointers, one word per slot");

// Exact engine.  Named barriers: 1 = B's per-band barrier, 2 + s = FULL[s] (E arrives, B
// waits; it is also B's barrier before a chunk's first band), 6 + s = EMPTY[s].
constexpr int kExactRing = 4, kExactGroups = 2;
constexpr int kBarChain = 1, kBarFull = 2, kBarExEmpty = 2 + kExactRing;
static_assert(kExactRing % kExactGroups == 0, "each ring slot, and its two barriers, belongs to one E group");

// Grid engine.  B = warps 0 and 1, two slots per thread, E = four groups of two warps:
// the warps w with w & 2.  A warp runs on scheduler (w & 3) of the SM, so B has its two to
// itself; with a fifth group there (warps 4 and 5) a read of 20 kb took 5-8% longer.
// Measured on a bare chain, cycles per band: 87
// with four B warps alone and 134 with E's load on every scheduler; 94 with two, whatever
// runs on the other two schedulers; 141 with one warp of four slots per lane.
//   Named barriers: 1 = B's per-band barrier, 2 + g = E group g's own, 6 + s = EMPTY[s]: B
// has released the chunk of ring slot s (B arrives, the group of the slot's next chunk
// waits; fewer groups than slots, so no two wait on one).  The other way round a header
// in shared memory tells B that a chunk is made: a barrier there costs the chain 68 cycles
// per chunk, a reduction of the failed checks (bar.red) 78; a header read a chunk ahead
// and a flag word next to nothing.  B's polls of a header are bounded by the spin limit:
// when it runs out the run reports a timeout and the read is given up (`dead`), B going on
// with a fixed bound until it can leave in step with E, whose turn by then waits for nothing
// but its own work.  (E polling a word for the released chunks in place of EMPTY, which would
// bound its waits too, took 8% of a long read.)
constexpr int kGridRing = 7;        // chunks in the ring
constexpr int kGridGroups = 4;
constexpr int kPerLane = 2;         // slots per thread of B and of E
constexpr int kTeam = kSlots / kPerLane;  // threads of B, and of an E group
constexpr int kPair = 2 * kTeam;          // B and one E group on EMPTY
constexpr int kBarGroup = 2, kBarEmpty = 2 + kGridGroups;
constexpr int kReadyPolls = 1 << 22;      // B's polls of a header after the spin limit's
static_assert(kWideChunk * kGridRing <= kSlots - kBand && kWideChunk * kExactRing <= kSlots - kBand,
              "E's k-mer window must hold the chunk's bands");
static_assert(kBarEmpty + kGridRing <= 16 && kBarExEmpty + kExactRing <= 16, "named barriers 0-15");
static_assert(kGridGroups < kGridRing, "two groups never wait on one EMPTY barrier");
static_assert(kWideChunk * kGridRing + 2 <= kScoreRing, "bands in use: two before the chunk E closes, to B's");
static_assert(2 * kGridRing <= kHeadRing, "headers in use");

// How long the exact engine runs (chunks) before the grid engine is tried: at the start,
// again, and after failures.  A read's scores pass -2^11 after some 950 bands.
constexpr int kFirstExact = 200, kNextExact = 32;

struct alignas(16) WideSmem {
    union {
        struct {  // exact: band 4j + q of chunk j in slot (j - j0) % kExactRing, entry [q]
            // {p_step, p_stay, w_step, w_stay} and {|em| + |step_h|, |em| + |stay_h|}
            // (NaN when the emission's division was not proven)
            float4 ems[kExactRing][kWideChunk][kSlots];
            float2 emm[kExactRing][kWideChunk][kSlots];
            float trim[kExactRing][kWideChunk];  // the trim cell's value (-inf: past the read's events)
        };
        float2 x[kGridRing][kWideChunk][kSlots];  // grid: {x_step, x_stay} (grid_pair), slot (j - j0) % kGridRing
    };
    float sc[kScoreRing][kSlots];   // scores of band b at [b & 31]
    int32_t kb[kScoreRing];         // 4 * placement of band b at [b & 31]
    // grid engine, of chunk j at [j & 15]
    int32_t head[kHeadRing];        // made: chunk_head(j, its grid or 0 for none)
    float2 skip[kHeadRing];         // {the grid's skip part, 1: B has stored its backpointers and origins}
    int32_t flag;                   // a failed check
    int32_t exit, failing;          // the first chunk not done; failures made it leave
    int32_t dead;                   // a wait ran out of polls
    int32_t k_odd;                  // the next k-mer that is none for a grid
};
__device__ __forceinline__ int chunk_head(int j, int mode) { return (j + 1) << 5 | mode; }  // never 0
static_assert(kGridMax < 32, "five bits of mode");

__device__ __forceinline__ void named_bar_sync(int id, int n) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void named_bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;\n" ::"r"(id), "r"(n) : "memory");
}
// bar.sync that also returns whether p held in any of the n threads
__device__ __forceinline__ bool named_bar_any(int id, int n, bool p) {
    uint32_t r;
    asm volatile(
        "{\n .reg .pred pi, po;\n setp.ne.u32 pi, %1, 0;\n bar.red.or.pred po, %2, %3, pi;\n selp.u32 %0, 1, 0, po;\n}\n"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(id), "r"(n)
        : "memory");
    return r != 0u;
}

__device__ __forceinline__ bool band_moves_right(float ll, float ur, int b) {
    // Suzuki-Kasahara (GPU/align_cuda.cl:394-430); both ends -inf: alternate
    return (ll == -INFINITY && ur == -INFINITY) ? (bool)(b & 1) : (ll < ur);
}

// The reference's arithmetic for one cell whose exactness proof failed, as a
// call: its division routine and FP64 code stay out of the band loop's body.
struct SlowCell {
    float best;
    uint32_t from;
};
__device__ __noinline__ SlowCell slow_cell_call(float diag, float up, float left, float x, float gm, float sd, float k1,
                                                double lp_step, double lp_stay, double lp_skip) {
    CellConsts c{};
    c.lp_step = lp_step;
    c.lp_stay = lp_stay;
    c.lp_skip = lp_skip;
    SlowCell o;
    o.best = cell_slow(diag, up, left, x, gm, sd, k1, c, o.from);
    return o;
}

// A read as the two engines see it.
// kCk: a checkpointed read (code of its own: its tests cost the other reads 3%).
template <bool kCk>
struct WideRead {
    const CoreArgs& a;
    const ReadDesc& r;
    WideSmem& ws;
    CellConsts cc;
    int n_events, n_kmers, n_bands, n_chunks;
    uint8_t* trace;
    int32_t* bk0;
    float* scores;

    // the origins of chunk j's bands, by threads 0-3
    __device__ __forceinline__ void store_origins(int j, int t) const {
        const int band = kWideChunk * j + t;
        if (t < kWideChunk && band < n_bands && in_bounds(band, n_bands, a.counters))
            bk0[band] = ws.kb[band & (kScoreRing - 1)] >> 2;
    }
    // whether tile j of the trace is to be stored
    __device__ __forceinline__ bool tile_in(int j) const { return !kCk && in_bounds(j, (n_bands + 3) / 4, a.counters); }
    // A checkpointed read's record after chunk j, the state before band 4(j + 1), when that
    // band has one (nullptr: none).  The record: the scores of band 4j + 3, those of band
    // 4j + 2 shifted by one slot, and band 4j + 3's placement (record_end, one thread).
    __device__ __forceinline__ float* record(int j) const {
        constexpr int kEvery = kCkBands / kWideChunk;
        const int s = (j + 1) / kEvery;
        return kCk && (j + 1) % kEvery == 0 && in_bounds(s, n_bands / kCkBands + 1, a.counters)
                   ? a.ck + r.ck_off + (int64_t)s * kCkStride
                   : nullptr;
    }
    __device__ __forceinline__ void record_end(float* rec, int j, int k0) const {
        rec[2 * kSlots] = __int_as_float(k0);
        rec[2 * kSlots + 1] = __int_as_float(kWideChunk * j + 1 - k0);  // the event of band 4j + 3
    }
    // the end cells of band b-1 (its row of the ring) and the left neighbour of a slot
    __device__ __forceinline__ void ends(int row, int k0, float& ll, float& ur) const {
        ll = ws.sc[row][k0 & (kSlots - 1)];
        ur = ws.sc[row][(k0 + kBand - 1) & (kSlots - 1)];
    }
};

// ---- exact engine
// E: chunk j's emissions for slot t into ring slot s, from the placement kp of an earlier
// band.
template <bool kCk>
__device__ __forceinline__ void exact_chunk(const WideRead<kCk>& w, int t, int s, int j, int kp) {
    const ReadDesc& r = w.r;
    const int kk = kp + ((t - kp) & (kSlots - 1));  // slot t's k-mer in the window
    const bool kin = kk >= 0 && kk < w.n_kmers;
    const float4 km = w.a.km4[r.km_off + (kin ? kk : 0)];
    const float gm = km.x, sd = km.y, rsd = km.z, k1 = km.w;
    const float* ev = w.a.ev_mean + r.ev_off;
    const int b0 = kWideChunk * j, e_first = b0 - 2 - kk;
    float x[kWideChunk];
#pragma unroll
    for (int q = 0; q < kWideChunk; ++q) {
        // cells outside the read get a finite stand-in; B's in-band test keeps them out
        const int e = e_first + q;
        x[q] = (kin && e >= 0 && e < w.n_events) ? ev[e] : gm;
    }
#pragma unroll
    for (int q = 0; q < kWideChunk; ++q) {
        bool ok;
        const float em = emission_fast(x[q], gm, sd, rsd, k1, ok);
        const EmSplit s1 = em_split(em, w.cc.step_h, w.cc.step_l);
        const EmSplit s2 = em_split(em, w.cc.stay_h, w.cc.stay_l);
        const float nan = __int_as_float(0x7fc00000);
        w.ws.ems[s][q][t] = make_float4(s1.p, s2.p, s1.w, s2.w);
        w.ws.emm[s][q][t] = ok ? make_float2(__fadd_rn(fabsf(em), fabsf(w.cc.step_h)),
                                             __fadd_rn(fabsf(em), fabsf(w.cc.stay_h)))
                               : make_float2(nan, nan);
    }
    if (t < kWideChunk) {
        // the trim cell (k = -1) of band b0 + t: event b0 + t - 1, (float)(lp_trim * (e + 1))
        // (GPU/align_cuda.cl:431-443); B uses it while the band reaches below k-mer 0
        const int e_t = b0 + t - 1;
        w.ws.trim[s][t] = e_t < w.n_events ? __double2float_rn(__dmul_rn(w.a.g.lp_trim, (double)(e_t + 1))) : -INFINITY;
    }
}

// Chunks j0 .. j1 - 1, from the bands before them in the score ring; every thread of the
// block calls it.
template <bool kScores, bool kCk>
__device__ __forceinline__ void chain_exact(const WideRead<kCk>& w, int tid, int j0, int j1) {
    const int warp = tid >> 5;
    if (warp >= 4 + 4 * kExactGroups) return;
    WideSmem& ws = w.ws;
    const ReadDesc& r = w.r;
    const CoreArgs& a = w.a;
    const int n_events = w.n_events, n_kmers = w.n_kmers, n_bands = w.n_bands;
    const int t = tid & (kSlots - 1), tl = (t + kSlots - 1) & (kSlots - 1);
    constexpr int kBoth = 2 * kSlots;  // B and one E group on FULL / EMPTY
    const int before = (kWideChunk * j0 - 1) & (kScoreRing - 1);  // band 4 j0 - 1
    const int k_start = ws.kb[before] >> 2;
    if (warp >= 4) {
        for (int j = j0 + (warp >> 2) - 1; j < j1; j += kExactGroups) {
            const int s = (j - j0) & (kExactRing - 1), jr = j - kExactRing;
            int kp = k_start;
            if (jr >= j0) {
                named_bar_sync(kBarExEmpty + s, kBoth);  // B released chunk jr
                kp = ws.kb[(kWideChunk * jr + kWideChunk - 1) & (kScoreRing - 1)] >> 2;
            }
            exact_chunk(w, t, s, j, kp);
            named_bar_arrive(kBarFull + s, kBoth);
        }
        return;
    }
    // B.  band b's placement: lower-left k-mer k0, event e0 = b - 2 - k0, so only k0 is
    // carried; s1 = band b-1's score of this slot, lp = band b's diagonal (band b-2's score
    // of slot t-1).  Before band 2: bands 1 and 0.
    int k0 = k_start;
    float s1 = ws.sc[j0 ? before : 1][t], lp = ws.sc[j0 ? (before - 1) & (kScoreRing - 1) : 0][tl];
    float* lastc = a.last_col + r.ev_off;
    const int sl_last = (n_kmers - 1) & (kSlots - 1);
    unsigned slow = 0, fp64 = 0;
    // band b's last-column score and, optionally, its scores
    auto keep = [&](int b, bool last_col) {
        if (last_col) {
            const int ol = n_kmers - 1 - k0, e0 = b - 2 - k0;
            int lo, hi;
            band_range(k0, e0, n_events, n_kmers, lo, hi);
            if (t == sl_last && ol >= lo && ol < hi && in_bounds(e0 - ol, n_events, a.counters)) lastc[e0 - ol] = s1;
        }
        if (kScores && in_bounds(b, n_bands, a.counters)) w.scores[(int64_t)b * kSlots + t] = s1;
    };
    // One chunk, its bands unrolled; band b-1's last-column store runs beside band b's
    // loads.  kEdge: the read may begin or end inside it (the only chunks that test for
    // it: a test per band is a branch in the band body, measured 27 cycles per band).
    // kMid: all 100 cells of its bands are computed, none of them the trim cell or on the
    // last k-mer column.
    auto chunk = [&](int j, auto edge, auto mid) {
        constexpr bool kEdge = decltype(edge)::value, kMid = decltype(mid)::value;
        const int s = (j - j0) & (kExactRing - 1), b0 = kWideChunk * j;
        const int r0 = b0 & (kScoreRing - 1);
        uint32_t word = (kEdge && j == 0 && t == 127) ? ABEA_FROM_U << 8 : 0u;  // band 1's trim cell
        bool begun = false;
        named_bar_sync(kBarFull + s, kBoth);  // chunk j's emissions, and band b0-1's scores
#pragma unroll
        for (int q = 0; q < kWideChunk; ++q) {
            const int b = b0 + q;
            if (kEdge && (b < 2 || b >= n_bands)) continue;
            if (q > 0) named_bar_sync(kBarChain, kSlots);  // band b-1's scores are in shared memory
            const int row = q > 0 ? r0 + q - 1 : (r0 - 1) & (kScoreRing - 1);
            float ll, ur;
            w.ends(row, k0, ll, ur);
            const float left = ws.sc[row][tl];
            const float4 ep = ws.ems[s][q][t];
            const float2 mm = ws.emm[s][q][t];
            const float tv = ws.trim[s][q];
            if (kEdge ? begun : q > 0) keep(b - 1, !kMid);
            begun = true;
            // the exact diagonal and up candidates
            bool okd, oku;
            const float d = exact_from_split(lp, EmSplit{ep.x, ep.z}, mm.x, okd);
            const float u = exact_from_split(s1, EmSplit{ep.y, ep.w}, mm.y, oku);
            const bool right = band_moves_right(ll, ur, b);
            k0 += right ? 1 : 0;
            if (t == 0) ws.kb[r0 + q] = 4 * k0;
            const int e0 = b - 2 - k0;
            int lo = 0, hi = kBand;
            if (!kMid) band_range(k0, e0, n_events, n_kmers, lo, hi);
            const int o = (t - k0) & 127;
            const bool valid = kMid ? o < kBand : (o >= lo && o < hi);
            // d vs u (U wins ties), then the skip candidate (L wins ties)
            uint32_t from_du, from;
            const float best_du = pick_du(d, u, from_du);
            bool okl;
            const float l = exact_skip(left, w.cc.skip_h, w.cc.skip_l, okl);
            float best = pick_l(best_du, from_du, l, from);
            const bool bad = valid && !(okd && oku && okl);
            best = valid ? best : -INFINITY;
            if (!kMid) from = valid ? from : 0u;  // a mid chunk's invalid slots are outside the band
            const bool here = !kMid && (t == 127) && (k0 <= -1) && (k0 >= -kBand);  // the trim cell
            best = here ? tv : best;
            from = here ? (tv == -INFINITY ? 0u : ABEA_FROM_U) : from;
            ws.sc[r0 + q][t] = best;  // stored before the check: only the rare path stores again
            if (__any_sync(kFull, bad)) {
                // A proof failed in some lane: in a read's first bands, three of four, where
                // an emission far below its score was added to it (Fast2Sum's condition).
                // TwoSum proves those; with FP64 for them all, the first 800 bands of a read
                // took 710 cycles each and a read of 1 kb 760 us, now 570.  (No vote per band,
                // a failed proof redoing its chunk: 325 cycles per band where all hold, but the
                // tests for it cost the bands with votes 5%.)
                const bool redo = bad && !here;
                bool okd2, oku2;
                const float d2 = exact_from_split<true>(lp, EmSplit{ep.x, ep.z}, mm.x, okd2);
                const float u2 = exact_from_split<true>(s1, EmSplit{ep.y, ep.w}, mm.y, oku2);
                uint32_t from_du2, from2;
                const float best_du2 = pick_du(d2, u2, from_du2);
                const float best2 = pick_l(best_du2, from_du2, l, from2);
                best = redo ? best2 : best;
                from = redo ? from2 : from;
                slow += redo ? 1 : 0;
                const bool still = redo && !(okd2 && oku2 && okl);
                if (__any_sync(kFull, still)) {
                    // Rare: the lane's cell takes the reference's FP64 arithmetic.  The whole
                    // warp calls (a divergent branch around the call cost 20 cycles per
                    // band); the other lanes pass k-mer 0 and event 0 of the read, which
                    // exist because the lane's cell does, and drop the result.
                    const int64_t ko = r.km_off + (still ? k0 + o : 0);
                    const SlowCell c = slow_cell_call(lp, s1, left, a.ev_mean[r.ev_off + (still ? e0 - o : 0)], a.km_gm[ko],
                                                      a.km_sd[ko], a.km_k1[ko], w.cc.lp_step, w.cc.lp_stay, w.cc.lp_skip);
                    best = still ? c.best : best;
                    from = still ? c.from : from;
                    fp64 += still ? 1 : 0;
                }
                ws.sc[r0 + q][t] = best;
            }
            word |= from << (8 * q);
            lp = left;
            s1 = best;
        }
        if (j + kExactRing < j1) named_bar_arrive(kBarExEmpty + s, kBoth);  // E may refill its slot
        keep(min(b0 + kWideChunk, n_bands) - 1, !kMid);
        if (float* rec = kEdge ? nullptr : w.record(j)) {
            rec[t] = s1;
            rec[kSlots + t] = lp;
            if (t == 0) w.record_end(rec, j, k0);
        }
        if (w.tile_in(j)) reinterpret_cast<uint32_t*>(w.trace + (int64_t)j * 512)[t] = word;
        if (warp == 0) {
            __syncwarp();  // thread 0 wrote the placements
            w.store_origins(j, t);
        }
    };
    using F = std::false_type;
    using T = std::true_type;
    for (int j = j0; j < j1; ++j) {
        // band 4j - 1's placement decides for the whole chunk: k0 and e0 each move by at
        // most one per band
        const int e0 = kWideChunk * j - 3 - k0;
        if (j == 0 || kWideChunk * (j + 1) > n_bands)
            chunk(j, T{}, F{});
        else if (k0 >= 0 && k0 + kWideChunk + kBand <= n_kmers - 1 && e0 >= kBand - 1 && e0 + kWideChunk <= n_events - 1)
            chunk(j, F{}, T{});
        else
            chunk(j, F{}, F{});
    }
    if (slow) atomicAdd(&a.counters[kCountSlow], (unsigned long long)slow);
    if (fp64) atomicAdd(&a.counters[kCountFp64], (unsigned long long)fp64);
}

// ---- grid engine
// The trim cell (k = -1) of event e: (float)(lp_trim * (e + 1)) (GPU/align_cuda.cl:431-443).
__device__ __forceinline__ float trim_score(const GlobalConsts& g, int e) {
    return __double2float_rn(__dmul_rn(g.lp_trim, (double)(e + 1)));
}

// E: a chunk's candidate parts (grid_pair) for thread t's slots into ring slot s.
// chunk_mode sees to it that every slot of the window has a k-mer and its four events,
// but for (edge_chunk) k-mer -1 and events past the read's last.
template <bool kLow>
__device__ __forceinline__ void grid_chunk(WideSmem& ws, const float4* km4, const float* ev, const Grid& G, int t, int s,
                                           int b0, int kp) {
    float4 km[kPerLane];
    float x[kPerLane][kWideChunk];
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
        const int kk = kp + ((kPerLane * t + i - kp) & (kSlots - 1));
        km[i] = km4[kk];
        const float* e = ev + (b0 - 2 - kk);
#pragma unroll
        for (int q = 0; q < kWideChunk; ++q) x[i][q] = e[q];
    }
#pragma unroll
    for (int q = 0; q < kWideChunk; ++q) {
        const float2 g0 = grid_pair<kLow>(x[0][q], km[0].x, km[0].y, km[0].z, km[0].w, G);
        const float2 g1 = grid_pair<kLow>(x[1][q], km[1].x, km[1].y, km[1].z, km[1].w, G);
        *reinterpret_cast<float4*>(&ws.x[s][q][kPerLane * t]) = make_float4(g0.x, g0.y, g1.x, g1.y);
    }
}

// The same on a band that has lost the path, at the read's edges: the adaptive band of a
// read whose scalings are off follows the trim cells (k-mer -1, the cheapest way through
// the events) to the last event, then the first invalid event (n_events, its lower left
// cell) through the k-mers.
// Such bands take 440 cycles each on the exact engine, here 160-185 (20,000 bands).
//   The trim cell is the up candidate of the one before it: their difference is a float
// (two neighbours' within a factor of two), and so is their sum; its other two candidates
// come from -inf.  A cell past the last event gets parts of -inf: its score is -inf, its
// left neighbour's event is the same.
__device__ __forceinline__ bool edge_chunk(int b0, int kp, int n_events) {
    return kp < 0 || b0 + kWideChunk - 3 - kp > n_events - 1;
}
template <bool kLow>
__device__ __forceinline__ void grid_chunk_edge(WideSmem& ws, const float4* km4, const float* ev, const Grid& G,
                                                const GlobalConsts& g0, int n_events, int t, int s, int b0, int kp) {
    int kk[kPerLane];
    float4 km[kPerLane];
    float x[kPerLane][kWideChunk];
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
        kk[i] = kp + ((kPerLane * t + i - kp) & (kSlots - 1));
        km[i] = km4[max(kk[i], 0)];
#pragma unroll
        for (int q = 0; q < kWideChunk; ++q) x[i][q] = ev[min(b0 - 2 - kk[i] + q, n_events - 1)];
    }
#pragma unroll
    for (int i = 0; i < kPerLane; ++i) {
        float2 g[kWideChunk];
#pragma unroll
        for (int q = 0; q < kWideChunk; ++q) g[q] = grid_pair<kLow>(x[i][q], km[i].x, km[i].y, km[i].z, km[i].w, G);
        if (kk[i] < 0) {  // one thread
            float last = trim_score(g0, b0 - 2);
#pragma unroll
            for (int q = 0; q < kWideChunk; ++q) {
                const float next = trim_score(g0, b0 - 1 + q);
                g[q].x = g[q].y = __fsub_rn(next, last);
                last = next;
            }
        }
#pragma unroll
        for (int q = 0; q < kWideChunk; ++q) {
            if (b0 - 2 - kk[i] + q >= n_events) g[q].x = g[q].y = -INFINITY;
            ws.x[s][q][kPerLane * t + i] = g[q];
        }
    }
}

// The grid for a band's scores (its row of the ring; 0: none), the same in every warp:
// the binade of the largest one, when the smallest is at most 4 times it.  It serves
// chunks that end up to 68 bands on, whose scores are above -38 * 2^m (-50 * 2^m when a
// run of chunks began on the way, at above -16 * 2^m): a band's scores fall by less than
// 2^(m-1) from its predecessors'.
__device__ __forceinline__ int grid_of(const float* row, int lane, uint32_t modes) {
    const float4 v = reinterpret_cast<const float4*>(row)[lane];
    auto fin = [](float x) { return x > -INFINITY ? x : 0.0f; };
    const float mx = warp_max(fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)));
    const float mn = warp_min(fminf(fminf(fin(v.x), fin(v.y)), fminf(fin(v.z), fin(v.w))));
    const int m = (__float_as_int(-mx) >> 23) - 127;  // a positive mx: negative; -inf: 128
    const int mlo = (__float_as_int(-mn) >> 23) - 127;
    return m >= kGridMin && m <= kGridMax && mlo < m + 2 && ((modes >> (m & 31)) & 1u) ? m : 0;
}
static_assert(kWideChunk * (kGridRing + 2 * kGridGroups) <= 68, "bands from the one that decides a grid to the chunk's last");

// Grid `want` for the chunk of bands b0 .. b0 + 3 if the 128-slot window at the placement
// kp of a band up to 28 bands before its last has its k-mers in the read (or its first is
// the trim cell's; none of the chunk's cells lies on the last k-mer column) and no event
// before the first; else 0.  Events past the last one are only the lower left cell's of a
// band (e0 <= n_events holds where a run of chunks begins, and a band with such a cell
// moves right).
__device__ __forceinline__ int chunk_mode(int want, int kp, int b0, int n_kmers) {
    const bool in = kp >= -1 && kp < n_kmers - kSlots && b0 - 1 - kSlots - kp >= 0;
    return in ? want : 0;
}

// Chunks from j0 on, until one that no grid serves (ws.exit), from the bands before them
// in the score ring; `first`: the grid of those.  Every thread of the block calls it, with
// ws.head and ws.flag zero and ws.exit the largest int.  k_end: the k-mer that E's windows
// stay before (the read's end, or one that is none for a grid).
template <bool kScores, bool kCk>
__device__ __forceinline__ void chain_grid(const WideRead<kCk>& w, int tid, int j0, int first, uint32_t modes, int k_end) {
    const int warp = tid >> 5, lane = tid & 31;
    if ((warp & 3) < 2 && warp >= 2) return;
    WideSmem& ws = w.ws;
    const ReadDesc& r = w.r;
    const CoreArgs& a = w.a;
    const CellConsts& cc = w.cc;
    const int n_events = w.n_events;
    const int t = tid & (kTeam - 1);  // slots 2t and 2t + 1
    const int tl = (kPerLane * t + kSlots - 1) & (kSlots - 1);
    const int k_start = ws.kb[(kWideChunk * j0 - 1) & (kScoreRing - 1)] >> 2;
    auto store_scores = [&](int b, float v0, float v1) {
        if (kScores && in_bounds(b, w.n_bands, a.counters))
            reinterpret_cast<float2*>(w.scores + (int64_t)b * kSlots)[t] = make_float2(v0, v1);
    };
    auto store_tile = [&](int j, uint32_t w0, uint32_t w1) {
        if (w.tile_in(j)) reinterpret_cast<uint2*>(w.trace + (int64_t)j * 512)[t] = make_uint2(w0, w1);
    };

    if (warp >= 2) {
        // ------------------------------------------------ E: closes chunk j - kGridRing and makes chunk j
        const int group = warp >> 2;
        const float4* km4 = a.km4 + r.km_off;
        const float* ev = a.ev_mean + r.ev_off;
        Grid G{};
        int g_mode = 0, want = first;  // want: the grid of the scores at one of the group's last two turns
        for (int j = j0 + group, s = group, turn = 0;; j += kGridGroups, ++turn) {
            const int jr = j - kGridRing, b0 = kWideChunk * j, br = kWideChunk * jr;
            int kp = k_start;
            const bool closes = jr >= j0;
            if (closes) {
                named_bar_sync(kBarEmpty + s, kPair);  // B released chunk jr
                if (jr >= ws.exit) break;
                kp = ws.kb[(br + kWideChunk - 1) & (kScoreRing - 1)] >> 2;
            }
            const int mode = chunk_mode(want, kp, b0, k_end);
            if (closes) {
                const float2 sk = ws.skip[jr & (kHeadRing - 1)];
                if (turn & 1) want = grid_of(ws.sc[(br + 3) & (kScoreRing - 1)], lane, modes);
                if (sk.y == 0.0f) {
                    // the moves from the scores, as the comparison took them
                    const float xl = sk.x;
                    const float* row = ws.sc[(br - 1) & (kScoreRing - 1)];
                    float2 up = *reinterpret_cast<const float2*>(row + kPerLane * t);
                    float left = row[tl];
                    uint32_t w0 = 0u, w1 = 0u;
#pragma unroll
                    for (int q = 0; q < kWideChunk; ++q) {
                        row = ws.sc[(br & (kScoreRing - 1)) + q];
                        const float2 v = *reinterpret_cast<const float2*>(row + kPerLane * t);
                        const float4 x = *reinterpret_cast<const float4*>(&ws.x[s][q][kPerLane * t]);
                        const float l0 = __fadd_rn(left, xl), l1 = __fadd_rn(up.x, xl);
                        const float u0 = __fadd_rn(up.x, x.y), u1 = __fadd_rn(up.y, x.w);
                        if (v.x == l0) w0 |= ABEA_FROM_L << (8 * q);
                        if (v.x == u0 && v.x != l0) w0 |= ABEA_FROM_U << (8 * q);
                        if (v.y == l1) w1 |= ABEA_FROM_L << (8 * q);
                        if (v.y == u1 && v.y != l1) w1 |= ABEA_FROM_U << (8 * q);
                        store_scores(br + q, v.x, v.y);
                        up = v;
                        left = row[tl];
                    }
                    if (br + 1 - kp >= n_events) {  // a cell past the last event has no move
                        for (int q = 0; q < kWideChunk; ++q) {
                            const float* v = ws.sc[(br & (kScoreRing - 1)) + q] + kPerLane * t;
                            if (v[0] == -INFINITY) w0 &= ~(0xffu << (8 * q));
                            if (v[1] == -INFINITY) w1 &= ~(0xffu << (8 * q));
                        }
                    }
                    store_tile(jr, w0, w1);
                    w.store_origins(jr, t);
                }
                if (float* rec = w.record(jr)) {
                    const float* last = ws.sc[(br + 3) & (kScoreRing - 1)];
                    const float* prev = ws.sc[(br + 2) & (kScoreRing - 1)];
                    reinterpret_cast<float2*>(rec)[t] = *reinterpret_cast<const float2*>(last + kPerLane * t);
                    reinterpret_cast<float2*>(rec + kSlots)[t] = make_float2(prev[tl], prev[kPerLane * t]);
                    if (t == 0) w.record_end(rec, jr, kp);
                }
            }
            if (mode) {
                if (mode != g_mode) G = make_grid(cc, mode);
                g_mode = mode;
                if (edge_chunk(b0, kp, n_events)) {
                    if (mode < kGridWide)
                        grid_chunk_edge<true>(ws, km4, ev, G, a.g, n_events, t, s, b0, kp);
                    else
                        grid_chunk_edge<false>(ws, km4, ev, G, a.g, n_events, t, s, b0, kp);
                } else if (mode < kGridWide)
                    grid_chunk<true>(ws, km4, ev, G, t, s, b0, kp);
                else
                    grid_chunk<false>(ws, km4, ev, G, t, s, b0, kp);
            }
            named_bar_sync(kBarGroup + group, kTeam);
            if (t == 0) {
                ws.skip[j & (kHeadRing - 1)] = make_float2(G.skip, 0.0f);
                __threadfence_block();
                *(volatile int32_t*)&ws.head[j & (kHeadRing - 1)] = chunk_head(j, mode);
            }
            s = s + kGridGroups >= kGridRing ? s + kGridGroups - kGridRing : s + kGridGroups;
        }
        return;
    }

    // ------------------------------------------------ B: the chain
    // Every cell of the chunks' bands is computed (100 per band; 99 when the lower left one
    // lies past the last event and is -inf) and finite when the first band's predecessors
    // are (checked on entry): a cell has its up neighbour or, at the band's new right end,
    // its left one.  No score exceeds those before it, E bounds how
    // far they fall, and a NaN in a cell reaches the next band (its own slot's up candidate
    // or, where the slot left the band, its right neighbour's skip): so the scores that a
    // chunk ends with show a failed proof.
    //   A chunk's check runs in the next one: `pend` says that one awaits it, kb_pend and
    // kb_cur are 4 * the placements that it and the current one started from.
    int k0 = k_start;
    float s1[kPerLane], lp[kPerLane];  // band b-1's scores of the slots; band b's diagonals
    float xl = 0.0f, g_lim = 0.0f;
    int g_mode = 0;
    int pen = 0;  // 8 for a failed chunk, -1 for a good one
    unsigned slow = 0, again_n = 0;
    constexpr uint32_t kOne = 1u << 25, kIn = (uint32_t)kBand << 25;
    auto release = [&](int s) { named_bar_arrive(kBarEmpty + s, kPair); };  // E closes the chunk and refills its slot
    // the state before chunk j, from the score ring
    auto restore = [&](int j, int kb) {
        const int row = kWideChunk * j;
        const float2 v = *reinterpret_cast<const float2*>(&ws.sc[(row - 1) & (kScoreRing - 1)][kPerLane * t]);
        k0 = kb >> 2;
        s1[0] = v.x;
        s1[1] = v.y;
        lp[0] = ws.sc[(row - 2) & (kScoreRing - 1)][tl];
        lp[1] = ws.sc[(row - 2) & (kScoreRing - 1)][kPerLane * t];
    };
    // A failed chunk again from its start in the reference's FP64 arithmetic, rare.
    auto redo = [&](int j, int kb) {
        restore(j, kb);
        pen += 8;
        ++again_n;
        uint32_t word[kPerLane] = {0u, 0u};
#pragma unroll 1
        for (int q = 0; q < kWideChunk; ++q) {
            const int b = kWideChunk * j + q, row = (b - 1) & (kScoreRing - 1);
            float ll, ur;
            w.ends(row, k0, ll, ur);
            const float left[kPerLane] = {ws.sc[row][tl], s1[0]};
            k0 += band_moves_right(ll, ur, b) ? 1 : 0;
            if (t == 0) ws.kb[b & (kScoreRing - 1)] = 4 * k0;
#pragma unroll
            for (int i = 0; i < kPerLane; ++i) {
                const int o = (kPerLane * t + i - k0) & (kSlots - 1);
                // all of the band but the trim cell and a cell past the last event, both of
                // them its first; the others compute its second
                const bool trim = o == 0 && k0 < 0, past = o == 0 && b - 2 - k0 >= n_events;
                const bool valid = o < kBand && !trim && !past;
                const int kk = k0 + (valid ? o : 1);
                const int64_t ko = r.km_off + kk;
                const SlowCell c = slow_cell_call(lp[i], s1[i], left[i], a.ev_mean[r.ev_off + (b - 2 - kk)], a.km_gm[ko],
                                                  a.km_sd[ko], a.km_k1[ko], cc.lp_step, cc.lp_stay, cc.lp_skip);
                lp[i] = left[i];
                s1[i] = valid ? c.best : trim && !past ? trim_score(a.g, b - 2 - k0) : -INFINITY;
                word[i] |= (valid ? c.from : trim && !past ? ABEA_FROM_U : 0u) << (8 * q);
                slow += valid ? 1 : 0;
            }
            *reinterpret_cast<float2*>(&ws.sc[b & (kScoreRing - 1)][kPerLane * t]) = make_float2(s1[0], s1[1]);
            store_scores(b, s1[0], s1[1]);
            named_bar_sync(kBarChain, kTeam);
        }
        store_tile(j, word[0], word[1]);
        w.store_origins(j, t);
        if (t == 0) ws.skip[j & (kHeadRing - 1)].y = 1.0f;
    };
    // Chunk j's header, once it is made.
    auto header = [&](int j) {
        volatile int32_t* at = &ws.head[j & (kHeadRing - 1)];
        int h = *at;
        for (long long i = 0; h >> 5 != j + 1 && i < a.spin_limit; ++i) h = *at;
        if (h >> 5 != j + 1) {
            ws.dead = 1;
            if (lane == 0) atomicAdd(&a.counters[kCountTimeouts], 1ull);  // the run reports a timeout
            for (int i = 0; h >> 5 != j + 1 && i < kReadyPolls; ++i) h = *at;
        }
        return h;
    };
    // Runs chunks from chunk j (made, its start checked, every warp past a barrier after
    // band 4j-1) until one that has another grid or none, or a failed check; j is then that
    // chunk.  true: the check of chunk j-1 failed (and chunk j has begun).  The last barrier
    // passed is the one after band 4j-1.
    int kb_cur = 0, kb_pend = 0;
    bool pend = false;
    auto run = [&](int& j, int& s, auto low) {
        constexpr bool kLow = decltype(low)::value;  // emissions may be below the range
        uint32_t vs = (uint32_t)(kPerLane * t - k0) << 25;  // slot 2t's offset in the band, mod 128, at the top of the word
        int kb = 4 * k0;
        bool below = false;
        pend = false;
        char* const sc = reinterpret_cast<char*>(&ws.sc[0][0]);
        constexpr int kRow = 4 * kSlots, kRows = kScoreRing * kRow;
        int rw = (int)((unsigned)(kWideChunk * kRow) * (unsigned)j & (kRows - 1));  // byte offset of the chunk's first score row
        int row0 = (rw - kRow) & (kRows - 1);            // and of the row before it
        while (true) {
            kb_cur = kb;
            int fl = 0, head = 0;
            bool leave = false;
#pragma unroll
            for (int q = 0; q < kWideChunk; ++q) {
                if (q > 0) named_bar_sync(kBarChain, kTeam);
                const char* row = sc + (q > 0 ? rw + (q - 1) * kRow : row0);
                const float ll = *reinterpret_cast<const float*>(row + (kb & (kRow - 4)));
                const float ur = *reinterpret_cast<const float*>(row + ((kb + 4 * (kBand - 1)) & (kRow - 4)));
                const float left[kPerLane] = {*reinterpret_cast<const float*>(row + 4 * tl), s1[0]};
                const float4 x4 = *reinterpret_cast<const float4*>(&ws.x[s][q][kPerLane * t]);
                const float xd[kPerLane] = {x4.x, x4.z}, xu[kPerLane] = {x4.y, x4.w};
                if (q == 0) {
                    const float mx = max_nan(s1[0], s1[1]);
                    if (below | (mx != mx)) ws.flag = 1;
                    below = false;
                }
                if (q == 1) {
                    fl = ws.flag;
                    head = *(volatile int32_t*)&ws.head[(j + 1) & (kHeadRing - 1)];
                }
                if (q == 2) {
                    if (__any_sync(kFull, fl != 0)) return true;
                    if (pend) release(s == 0 ? kGridRing - 1 : s - 1);  // chunk j - 1 stands
                }
                if (q == 3) {
                    // chunk j + 1, usually made by now; both warps leave on another grid
                    if (__any_sync(kFull, head >> 5 != j + 2)) head = header(j + 1);
                    leave = __any_sync(kFull, head != chunk_head(j + 1, g_mode));
                }
                const bool right = ll < ur;  // the upper right end is finite
                const uint32_t vr = vs - kOne;
#pragma unroll
                for (int i = 0; i < kPerLane; ++i) {
                    const float d = __fadd_rn(lp[i], xd[i]), u = __fadd_rn(s1[i], xu[i]), l = __fadd_rn(left[i], xl);
                    const float best = max3_nan(d, u, l);
                    // the slot's in-band test under either placement, chosen last
                    const float b_stay = vs + (uint32_t)i * kOne < kIn ? best : -INFINITY;
                    const float b_right = vr + (uint32_t)i * kOne < kIn ? best : -INFINITY;
                    if (kLow) below |= (xu[i] < g_lim) & (best != l);  // it must not win
                    lp[i] = left[i];
                    s1[i] = right ? b_right : b_stay;
                }
                *reinterpret_cast<float2*>(sc + rw + q * kRow + 8 * t) = make_float2(s1[0], s1[1]);
                vs = right ? vr : vs;
                kb += right ? 4 : 0;
                if (t == 0) ws.kb[((rw / kRow) & (kScoreRing - 1)) + q] = kb;
            }
            pend = true;
            kb_pend = kb_cur;
            ++j;
            s = s + 1 == kGridRing ? 0 : s + 1;
            row0 = rw + (kWideChunk - 1) * kRow;
            rw = (rw + kWideChunk * kRow) & (kRows - 1);
            if (kLow && below) ws.flag = 2;  // (for the check when the run ends here)
            named_bar_sync(kBarChain, kTeam);
            if (leave) {
                k0 = kb >> 2;
                return false;
            }
        }
    };
    restore(j0, 4 * k_start);
    int j = j0, s = 0;
    while (true) {
        // chunk j's header; also the barrier after band 4j-1
        const int h = header(j);
        __threadfence_block();
        const int m = named_bar_any(kBarChain, kTeam, *(volatile int32_t*)&ws.dead != 0) ? 0 : h & 31;
        if (m == 0 || pen > 32) break;
        if (m != g_mode) {
            bool ok;
            g_mode = m;
            xl = grid_step(cc.skip_h, cc.skip_l, m, ok).o0;
            g_lim = -(pow2f(m - 1) - 128.0f) * kGridLimLo;
        }
        // the start: the scores finite in the band and within the grid's range
        const float top = -pow2f(m), bot = -pow2f(m + 4);
        const int past = kWideChunk * j - 3 - k0 >= n_events ? 1 : 0;  // the first cell is none
        bool bad = !(max_nan(max3_nan(s1[0], s1[1], lp[0]), lp[1]) < top);
#pragma unroll
        for (int i = 0; i < kPerLane; ++i) {
            const int o = (kPerLane * t + i - k0) & (kSlots - 1);
            bad |= ((o >= past) & (o < kBand) & !(s1[i] >= bot)) | ((lp[i] < bot) & (lp[i] > -INFINITY));
        }
        if (named_bar_any(kBarChain, kTeam, bad)) {
            redo(j, 4 * k0);
            release(s);
            ++j;
            s = s + 1 == kGridRing ? 0 : s + 1;
            continue;
        }
        const int j1 = j;
        const bool failed = m < kGridWide ? run(j, s, std::true_type{}) : run(j, s, std::false_type{});
        pen = max(pen - (j - j1), 0);
        if (pend) {
            // chunk j - 1 awaits its check (or has failed it)
            const float mx = max_nan(s1[0], s1[1]);
            const bool again = named_bar_any(kBarChain, kTeam, failed | (mx != mx) | (ws.flag != 0));
            if (t == 0) ws.flag = 0;  // every thread has read it
            if (again) redo(j - 1, kb_pend);
            release(s == 0 ? kGridRing - 1 : s - 1);
        }
    }
    // Every chunk before j is released; each E group ends up waiting for one of chunks j ..
    // j + 3, and once chunk j + g is made no group waits for an older chunk of its slot.
    if (t == 0) {
        ws.exit = j;
        ws.failing = pen > 32 ? 1 : 0;
    }
    for (int g = 0; g < kGridGroups; ++g) {
        header(j + g);
        __syncwarp();
        release(s + g >= kGridRing ? s + g - kGridRing : s + g);
    }
    if (slow) {  // a chunk done again: FP64 throughout
        atomicAdd(&a.counters[kCountSlow], (unsigned long long)slow);
        atomicAdd(&a.counters[kCountFp64], (unsigned long long)slow);
    }
    if (t == 0) {
        atomicAdd(&a.counters[kCountGrid], (unsigned long long)(j - j0) - again_n);
        atomicAdd(&a.counters[kCountGridAgain], (unsigned long long)again_n);
    }
}

// One read's fill; false when a wait ran out of polls: the read is given up, the rest of it
// not filled.  `odd`: some k-mer of the read is none for a grid (grid_kmer_ok); the grid
// chain then runs between such k-mers.  A call: it has the block's
// registers to itself.
template <bool kScores, bool kCk>
__device__ __noinline__ bool fill_chain(const CoreArgs& a, const ReadDesc& r, unsigned ws_at, int tid, bool odd) {
    WideSmem& ws = smem_ref<WideSmem>(ws_at);
    const int lane = tid & 31;
    WideRead<kCk> w{a, r, ws, make_consts(r, a.g), r.n_events, r.n_kmers, r.n_bands, (r.n_bands + kWideChunk - 1) / kWideChunk,
               a.trace + r.trace_off * kSlots, a.band_k0 + r.band_off, kScores ? a.scores + r.band_off * kSlots : nullptr};
    const uint32_t modes = grid_modes(w.cc);
    // band 0: the start cell (slot 127) = 0; band 1: the trim cell; both at k0 = -51
    if (tid < kSlots) {
        ws.sc[0][tid] = tid == 127 ? 0.0f : -INFINITY;
        ws.sc[1][tid] = tid == 127 ? a.g.trim_f : -INFINITY;
        if (kScores) {
            w.scores[tid] = ws.sc[0][tid];
            w.scores[kSlots + tid] = ws.sc[1][tid];
        }
    }
    if (tid == 0) {
        ws.kb[0] = ws.kb[1] = ws.kb[kScoreRing - 1] = 4 * (-1 - kBand / 2);
        ws.dead = 0;
    }
    __syncthreads();
    int j = 0, seg = kFirstExact, retry = kNextExact;
    while (true) {
        const int j1 = min(j + seg, w.n_chunks);
        chain_exact<kScores>(w, tid, j, j1);
        j = j1;
        if (tid < kHeadRing) ws.head[tid] = 0;
        if (tid == 0) {
            ws.flag = 0;
            ws.exit = INT32_MAX;
            ws.k_odd = INT32_MAX;
        }
        __syncthreads();
        if (j >= w.n_chunks) return true;
        // the grid engine, if its chunks can begin here and there is room for a run
        const int b0 = kWideChunk * j, kp = ws.kb[(b0 - 1) & (kScoreRing - 1)] >> 2;
        const int first = grid_of(ws.sc[(b0 - 1) & (kScoreRing - 1)], lane, modes);
        int k_end = w.n_kmers;
        if (odd) {
            // up to the next k-mer that is none for a grid, looked for among the next 4,096
            const int k_from = max(kp, 0), k_stop = min(w.n_kmers, k_from + 8 * kWideThreads);
            const float4* km4 = a.km4 + r.km_off;
            const float k1_max = grid_k1_max(r.step_h, r.stay_h);
#pragma unroll 1
            for (int k = k_from + tid; k < k_stop; k += kWideThreads)
                if (!grid_kmer_ok(km4[k].y, km4[k].w, k1_max)) atomicMin(&ws.k_odd, k);
            __syncthreads();
            k_end = min(k_stop, ws.k_odd);
        }
        const bool room = kp >= -1 && b0 - 3 - kp <= w.n_events && chunk_mode(1, kp + 40, b0 + 2 * 40, k_end);
        seg = kp < 0 || kp + 40 <= w.n_kmers - kSlots ? retry : w.n_chunks;  // near the end: to the end
        const bool enter = first && room && chunk_mode(first, kp, b0, k_end);
        // Every warp has decided before the chain may overwrite what they decided from: the
        // warps that the chain leaves idle never wait for it, and all must go the same way.
        __syncthreads();
        if (enter) {
            chain_grid<kScores>(w, tid, j, first, modes, k_end);
            __syncthreads();
            if (ws.dead) return false;
            j = ws.exit;
            if (ws.failing) retry = min(2 * retry, 1 << 20);
            const int k_now = ws.kb[(kWideChunk * j - 1) & (kScoreRing - 1)] >> 2;
            seg = k_now + 64 <= w.n_kmers - kSlots ? retry : w.n_chunks;
            __syncthreads();  // everyone has read the exit
        }
    }
}

// ---------------------------------------------------------------- wide shape on a cluster pair
// The wide fill with its emission work on a second SM: blocks run in clusters
// of two.  The cluster's first block holds the read's band state and runs three
// groups of 128 threads (B: the band-to-band chain, D: diagonal candidates and
// inside flags, K: bookkeeping and the prefetch rings of the FP64 slow path).
// The second block's four groups compute the emissions and their exact splits,
// group g the bands 2+g, 6+g, ..., stage them in their own shared memory and
// bulk-copy them into the first block's (distributed shared memory) up to
// kClRing bands ahead of the chain; one mbarrier per ring slot counts a band's
// bytes.  D waits on it before it prepares the band's diagonal candidates, and
// the block barrier that follows hands the band to B.
// A band's cells lie on one anti-diagonal (event + k-mer = band - 2), so the
// emissions of band bn only need a k-mer window that holds the band: the
// placement k0 of any earlier band p with bn - p <= 28 gives one, [k0, k0+128),
// because each band moves k0 by at most one.  The first block publishes its
// progress, with the placement of the band it names, into the second block's
// shared memory every kClPublish bands (each release is a cluster-scope fence:
// once per band they cost ~400 cycles per band).  E reads its inputs straight
// from the pre stage's arrays (L2), one band ahead.  Every wait is bounded by
// spin_limit polls; a wait that runs out is counted and goes on (the
// batch then reports a timeout).  Measured (64 reads of 1-6 kb): 1,080 cycles per band of
// the longest read against 190 on the single-block wide shape, so the option is off by default.
constexpr int kClRing = 16;    // bands of emissions in flight (<= 28: the k-mer window above)
constexpr int kClPublish = 8;  // block 0 publishes its progress every kClPublish bands (< kClRing)

struct alignas(16) ClSmem {
    Rings rg;                                   // block 0: rings of the FP64 slow path
    float sc[2][kSlots];
    // written by block 1, per band slot and k-mer slot: {pstay, wstay, magu, em} and {pstep, wstep}
    float4 emu[kClRing][kSlots];
    float2 emd[kClRing][kSlots];
    float dc[2][kSlots];
    int32_t flags[2][kSlots];
    float trim[2];
    uint32_t fr[8][kSlots];
    int32_t k0h[8];
};

// Cluster state that outlives the fill (the fill's shared memory is reused
// afterwards; the mbarriers and the partner's stores must not land there).
struct ClShared {
    uint64_t full[kClRing];  // block 0: band b's emissions in slot (b-2) % kClRing have landed
                             // (phase (b-2) / kClRing of that slot's mbarrier)
    int32_t k0ring[64];      // block 1: placement of band b at [b & 63], from block 0
    int32_t progress;        // block 1: block 0 is done with the emissions of bands <= progress
    int32_t pick;
};

__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

// Waits for the phase of parity `parity` of a local mbarrier, at most limit/64
// polls (each poll may itself suspend the thread for a while); false when they
// ran out.  CTA-scope acquire: the data that completes the phase (bulk copies
// counted by complete_tx) is visible to the waiting thread once it observes the
// completion, whichever block issued the copies.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, long long limit) {
    const unsigned a = smem_u32(bar);
    const long long polls = limit > 0 ? (limit >> 6) + 1 : 0;
    for (long long i = 0; i < polls; ++i) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(done)
            : "r"(a), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Remote shared-memory address of `p`'s counterpart in block `rank`.
__device__ __forceinline__ unsigned mapa_u32(const void* p, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}

// Bulk copy of `bytes` (a multiple of 16, both addresses 16-byte aligned) from
// this block's shared memory to another block's (remote address `rdst`),
// counted on that block's mbarrier `rbar` (complete_tx).
__device__ __forceinline__ void bulk_to_remote(unsigned rdst, const void* src, unsigned bytes, unsigned rbar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     rdst),
                 "r"(smem_u32(src)), "r"(bytes), "r"(rbar)
                 : "memory");
}

// One arrival on block `rank`'s mbarrier that also expects `bytes` of
// complete_tx stores in the current phase.
__device__ __forceinline__ void mbar_arrive_expect_remote(unsigned rbar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.release.cluster.shared::cluster.b64 _, [%0], %1;\n" ::"r"(rbar),
                 "r"(bytes)
                 : "memory");
}

// Release store of v to the int at the same place in block `rank`.
__device__ __forceinline__ void st_release_remote(int32_t* p, unsigned rank, int32_t v) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;\n" ::"r"(r), "r"(v) : "memory");
}

__device__ __forceinline__ int32_t ld_acquire_local(const int32_t* p) {
    int32_t v;
    asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];\n" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}

__device__ __forceinline__ void cl_barrier() { asm volatile("bar.sync 1, 384;\n" ::: "memory"); }
__device__ __forceinline__ void e_barrier(int group) { asm volatile("bar.sync %0, 128;\n" ::"r"(2 + group) : "memory"); }
// Called by every thread of both blocks of the cluster (rank = block rank).
template <bool kScores>
__device__ void fill_wide_cl(const CoreArgs& a, const ReadDesc& r, ClSmem& ws, ClShared& cs, int tid,
                             unsigned rank) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const CellConsts cc = make_consts(r, a.g);
    const int n_events = r.n_events, n_kmers = r.n_kmers, n_bands = r.n_bands;
    const int group = tid >> 7;  // block 0: 0 = B, 1 = D, 2 = K, 3 = idle; block 1: E groups 0-3
    const int t = tid & (kSlots - 1);
    const long long lim = a.spin_limit;
    unsigned long long timeouts = 0;
    bool dead = false;  // a wait ran out: later waits do not wait (the batch reports a timeout)

    int k0 = -1 - kBand / 2, e0 = kBand / 2;  // band 1 (band 0 is (49,-51), band 1 moved down)
    RingState rs;
    if (rank == 0 && group == 2) rings_init(ws.rg, rs, a, r, t, k0, e0);
    if (rank == 0 && tid == 0) {
        for (int i = 0; i < kClRing; ++i) mbar_init(&cs.full[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (rank == 1 && tid == 0) {
        cs.k0ring[1] = k0;
        cs.progress = 1;
    }
    cluster.sync();  // barriers initialised, progress 1 published, rings filled

    if (rank == 1) {
        // ------------------------------------------------ E (block 1): group g, bands 2+g, 6+g, ...
        const float* gm_p = a.km_gm + r.km_off;
        const float* sd_p = a.km_sd + r.km_off;
        const float* rsd_p = a.km_rsd + r.km_off;
        const float* k1_p = a.km_k1 + r.km_off;
        const float* ev_p = a.ev_mean + r.ev_off;
        struct In {
            float x, gm, sd, rsd, k1;
        };
        // band bn's inputs in slot t, k-mer window from the latest published placement;
        // waits until that placement is at most kClRing bands back (its ring slot is free)
        auto fetch = [&](int bn) {
            int prog = ld_acquire_local(&cs.progress);
            for (long long i = 0; prog < bn - kClRing && i < (dead ? 0 : lim); ++i)
                prog = ld_acquire_local(&cs.progress);
            if (prog < bn - kClRing) {
                ++timeouts;
                dead = true;
            }
            const int kp = cs.k0ring[prog & 63];
            const int kk = kp + ((t - kp) & 127);
            const int e = bn - 2 - kk;
            // cells outside the read get finite stand-ins; their flags keep them out of the band
            const bool in = kk >= 0 && kk < n_kmers && e >= 0 && e < n_events;
            const int kc = in ? kk : 0, ec = in ? e : 0;
            return In{__ldg(ev_p + ec), __ldg(gm_p + kc), __ldg(sd_p + kc), __ldg(rsd_p + kc), __ldg(k1_p + kc)};
        };
        int bn = 2 + group;
        In cur = bn < n_bands ? fetch(bn) : In{0.0f, 0.0f, 1.0f, 1.0f, 0.0f};
        for (; bn < n_bands; bn += 4) {
            bool ok;
            const float em = emission_fast(cur.x, cur.gm, cur.sd, cur.rsd, cur.k1, ok);
            const EmSplit s1 = em_split(em, cc.step_h, cc.step_l);
            const EmSplit s2 = em_split(em, cc.stay_h, cc.stay_l);
            if (bn + 4 < n_bands) cur = fetch(bn + 4);  // loads in flight across the stores
            // staged in this block's own copy of the slot (free: the band kClRing back
            // was consumed, so its copy has been read), then one bulk copy per array
            const int s = (bn - 2) % kClRing;
            ws.emu[s][t] = make_float4(s2.p, s2.w,
                                       ok ? __fadd_rn(fabsf(em), fabsf(cc.stay_h)) : __int_as_float(0x7fc00000), em);
            ws.emd[s][t] = make_float2(s1.p, s1.w);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // visible to the bulk copy
            e_barrier(group);
            if (t == 0) {
                const unsigned rbar = mapa_u32(&cs.full[s], 0);
                // one arrival and the band's 128 x 24 bytes complete the slot's phase
                mbar_arrive_expect_remote(rbar, kSlots * 24);
                bulk_to_remote(mapa_u32(&ws.emu[s][0], 0), &ws.emu[s][0], kSlots * 16, rbar);
                bulk_to_remote(mapa_u32(&ws.emd[s][0], 0), &ws.emd[s][0], kSlots * 8, rbar);
            }
        }
    } else if (group == 0) {
        // ------------------------------------------------ B (block 0): the chain
        ws.sc[1][t] = (t == 127) ? a.g.trim_f : -INFINITY;
        ws.fr[0][t] = 0u;
        ws.fr[1][t] = (t == 127) ? ABEA_FROM_U : 0u;
        if (t == 0) {
            ws.k0h[0] = k0;
            ws.k0h[1] = k0;
            a.band_k0[r.band_off] = k0;
        }
    }
    if (rank == 0 && group < 3) {
        cl_barrier();  // band 1 in shared memory
        if (group == 0) {
            float* scores = kScores ? a.scores + r.band_off * kSlots : nullptr;
            float s_prev = (t == 127) ? a.g.trim_f : -INFINITY;  // band 1
            float lp = (t == 0) ? 0.0f : -INFINITY;              // band 0 shifted by one slot
            if (kScores) {
                scores[t] = (t == 127) ? 0.0f : -INFINITY;
                scores[kSlots + t] = s_prev;
            }
            unsigned long long slow = 0;
            int b = 2, cb = 0;
            float best = 0.0f, left = 0.0f;
            uint32_t from = 0u;
            bool valid = false, bad = false;
            auto finish = [&]() {
                best = valid ? best : -INFINITY;
                from = valid ? from : 0u;
                if (k0 <= -1) {  // trim cell (k = -1, slot 127) while the band reaches below k-mer 0
                    const bool here = (t == 127) && (k0 >= -kBand);
                    const float tv = ws.trim[cb];
                    best = here ? tv : best;
                    from = here ? (tv == -INFINITY ? 0u : ABEA_FROM_U) : from;
                }
                ws.sc[cb][t] = best;
                ws.fr[b & 7][t] = from;
                if (kScores && in_bounds(b, n_bands, a.counters)) scores[(int64_t)b * kSlots + t] = best;
                lp = left;
                s_prev = best;
            };
            while (true) {
                bool to_slow = false;
                for (; b < n_bands; ++b) {
                    cl_barrier();  // B_{b-1}
                    const int pb = (b - 1) & 1, es = (b - 2) % kClRing;
                    cb = b & 1;
                    // band b's emissions: D saw their mbarrier phase complete before the
                    // barrier above (it prepared band b's diagonal candidates from them)
                    const float ll = ws.sc[pb][k0 & 127];
                    const float ur = ws.sc[pb][(k0 + kBand - 1) & 127];
                    left = ws.sc[pb][(t + 127) & 127];
                    const float d = ws.dc[cb][t];
                    const int f = ws.flags[cb][t];
                    const float4 eu = ws.emu[es][t];
                    const EmSplit su{eu.x, eu.y};
                    const float mu = eu.z;
                    bool oku;
                    const float u = exact_from_split(s_prev, su, mu, oku);
                    const bool right = band_moves_right(ll, ur, b);
                    k0 += right ? 1 : 0;
                    e0 += right ? 0 : 1;
                    valid = (f & (right ? 2 : 1)) != 0;
                    uint32_t from_du;
                    const float best_du = pick_du(d, u, from_du);
                    bool okl;
                    const float l = exact_skip(left, cc.skip_h, cc.skip_l, okl);
                    best = pick_l(best_du, from_du, l, from);
                    bad = valid && !(oku && okl && (f & 4));
                    if (__any_sync(kFull, bad)) {
                        to_slow = true;
                        break;
                    }
                    finish();
                }
                if (!to_slow) break;
                if (bad) {  // a proof failed: the reference's FP64 arithmetic
                    const int ep = e0 - ((t - k0) & 127);
                    best = cell_slow(lp, s_prev, left, ws.rg.ev[ep & (kEvRing - 1)], ws.rg.gm[t], ws.rg.sd[t],
                                     ws.rg.k1[t], cc, from);
                    ++slow;
                }
                finish();
                ++b;
            }
            cl_barrier();  // B_{n_bands-1}
            if (slow) {
                atomicAdd(&a.counters[kCountSlow], slow);
                atomicAdd(&a.counters[kCountFp64], slow);
            }
        } else if (group == 1) {
            // ------------------------------------------------ D (block 0)
            // band bn's diagonal candidates, inside flags and trim value, with the
            // band before it placed at k0
            auto prep = [&](int bn, float diag) {
                const int es = (bn - 2) % kClRing;
                if (!mbar_wait(&cs.full[es], (unsigned)((bn - 2) / kClRing) & 1u, dead ? 0 : lim)) {
                    ++timeouts;
                    dead = true;
                }
                const float em = ws.emu[es][t].w;
                const float2 ed = ws.emd[es][t];
                const EmSplit s1{ed.x, ed.y};
                bool okd;
                const float d = exact_from_split(diag, s1, __fadd_rn(fabsf(em), fabsf(cc.step_h)), okd);
                const int o = (t - k0) & 127;
                const int kk = k0 + o;
                const int e = bn - 2 - kk;
                const bool inb = (kk >= 0) && (kk < n_kmers) && (e >= 0) && (e < n_events);
                ws.dc[bn & 1][t] = d;
                ws.flags[bn & 1][t] =
                    ((inb && o < kBand) ? 1 : 0) | ((inb && o >= 1 && o <= kBand) ? 2 : 0) | (okd ? 4 : 0);
                if (k0 <= 0 && t == 0) {  // trim cell of band bn (GPU/align_cuda.cl:431-443)
                    const int e_t = bn - 1;
                    ws.trim[bn & 1] =
                        (e_t < n_events) ? __double2float_rn(__dmul_rn(a.g.lp_trim, (double)(e_t + 1))) : -INFINITY;
                }
            };
            prep(2, (t == 0) ? 0.0f : -INFINITY);  // band 0 shifted by one slot
            for (int b = 2; b < n_bands; ++b) {
                cl_barrier();  // B_{b-1}
                // B is done with the emissions of bands <= b-1, D with those of band b:
                // E may reuse their ring slots; band b-1's placement was published with them
                // (every kClPublish bands: each release is a cluster-scope fence)
                if (t == 0 && (b & (kClPublish - 1)) == 0) st_release_remote(&cs.progress, 1, b - 1);
                const int pb = (b - 1) & 1;
                const float ll = ws.sc[pb][k0 & 127];
                const float ur = ws.sc[pb][(k0 + kBand - 1) & 127];
                const bool right = band_moves_right(ll, ur, b);
                k0 += right ? 1 : 0;
                if (t == 0) {
                    ws.k0h[b & 7] = k0;
                    // E reads the placement of the published band only (b - 1 at b a multiple of
                    // kClPublish): written with the next progress store's release
                    if (((b + 1) & (kClPublish - 1)) == 0) *cluster.map_shared_rank(&cs.k0ring[b & 63], 1) = k0;
                }
                if (b + 1 < n_bands) prep(b + 1, ws.sc[pb][(t + 127) & 127]);
            }
            cl_barrier();  // B_{n_bands-1}
        } else if (group == 2) {
            // ------------------------------------------------ K (block 0): bookkeeping, rings
            uint8_t* trace = a.trace + r.trace_off * kSlots;
            int32_t* bk0 = a.band_k0 + r.band_off;
            float* lastc = a.last_col + r.ev_off;
            const int sl_last = (n_kmers - 1) & 127;
            for (int b = 2; b <= n_bands; ++b) {
                cl_barrier();  // B_{b-1}
                const int bp = b - 1;
                const int kp = ws.k0h[bp & 7];
                if ((b & 3) == 2) rings_step(ws.rg, rs, a, r, t, kp, bp - 2 - kp, 9);
                const int ep0 = bp - 2 - kp;
                const int ol = n_kmers - 1 - kp;
                if (ol < kBand && t == sl_last && bp >= 2) {  // last k-mer column (GPU/align_cuda.cl:722-746)
                    int lo, hi;
                    band_range(kp, ep0, n_events, n_kmers, lo, hi);
                    if (ol >= lo && ol < hi && in_bounds(ep0 - ol, n_events, a.counters))
                        lastc[ep0 - ol] = ws.sc[bp & 1][t];
                }
                if (t == 0 && in_bounds(bp, n_bands, a.counters)) bk0[bp] = kp;
                if ((bp & 3) == 3 || bp == n_bands - 1) {
                    const int q0 = bp & ~3, nj = bp - q0;
                    uint32_t word = 0u;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        if (j <= nj) word |= (ws.fr[(q0 + j) & 7][t] & 0xffu) << (8 * j);
                    if (in_bounds(bp >> 2, (n_bands + 3) / 4, a.counters))
                        reinterpret_cast<uint32_t*>(trace + (int64_t)(bp >> 2) * 512)[t] = word;
                }
            }
            cp_async_wait_all();
        }
    }
    if (timeouts) atomicAdd(&a.counters[kCountTimeouts], timeouts);
}

// ---------------------------------------------------------------- post
struct alignas(16) PostSmem {
    uint8_t tr[4 * kPostChunkBands * kSlots];  // ring of 64 bands of trace, tile layout
};

__device__ __forceinline__ float path_emission(const PostArgs& a, const ReadDesc& r, int k, int e) {
    const int64_t ko = r.km_off + k;
    return emission_ieee(a.ev_mean[r.ev_off + e], a.km_gm[ko], a.km_sd[ko], a.km_k1[ko]);
}

// One pair's emission for the QC sum as an integer multiple of 2^-24 (exact when
// 0.5 <= |em| < 2^20; `exact` turns false otherwise).  The division is Markstein's
// (div_rn): no routine call, so that the loads of several cells are in flight at once.
__device__ __forceinline__ void qc_term(const PostArgs& a, const ReadDesc& r, abea_aligned_pair_t p, long long& isum,
                                        long long& iabs, bool& exact) {
    const int64_t ko = r.km_off + p.ref_pos;
    bool ok;
    const float em =
        emission_rn(a.ev_mean[r.ev_off + p.read_pos], a.km_gm[ko], a.km_sd[ko], a.km_rsd[ko], a.km_k1[ko], ok);
    const float aem = fabsf(em);
    const long long q = __float2ll_rn(__fmul_rn(em, 16777216.0f));
    const bool in = ok && aem >= 0.5f && aem < 1048576.0f;
    isum += in ? q : 0ll;
    iabs += in ? (q < 0 ? -q : q) : 0ll;
    exact = exact && in;
}

__device__ __forceinline__ void post_write(const PostArgs& a, int ri, int result, float best, int best_e, int status,
                                           int n_out, int cap, bool reversed, int last_from);

// One traceback step: D -> (k-1, e-1), U -> (k, e-1), L -> (k-1, e); gap counting.
__device__ __forceinline__ void step_back(uint32_t from, int& k, int& e, int& gap, int& max_gap) {
    k -= (from != ABEA_FROM_U) ? 1 : 0;
    e -= (from != ABEA_FROM_L) ? 1 : 0;
    gap = (from == ABEA_FROM_L) ? gap + 1 : 0;
    max_gap = max(max_gap, gap);
}

// Serial double sum of the path's emissions in the reference's order (from the
// walk's first cell), re-walking the trace from global memory.  Used only when
// the path is longer than its output slot.  `flat` re-walks through the emulated
// flat band array (no finite end, see post_read_warp).
__device__ double serial_path_sum(const PostArgs& a, const ReadDesc& r, const uint8_t* trace, const int32_t* bk0,
                                  bool flat, int e, int k) {
    double sum = 0.0;
    int gap = 0, mg = 0;
    while (k >= 0 && e >= 0) {
        sum = __dadd_rn(sum, (double)path_emission(a, r, k, e));
        const int64_t band = (int64_t)e + k + 2;
        if (flat) {
            const int64_t f = band * kBand + ((band - 2 - bk0[band]) - e);
            if (f < 0 || f >= (int64_t)r.n_bands * kBand) break;
            const int64_t b2 = f / kBand;
            step_back(trace[trace_index(b2, (bk0[b2] + (int)(f - b2 * kBand)) & 127)], k, e, gap, mg);
        } else {
            step_back(trace[trace_index(band, k & 127)], k, e, gap, mg);
        }
    }
    return sum;
}

// Lane 0's state of a traceback walk.
struct Walk {
    int k, e, n_out, gap, max_gap, last_k, last_from;
    double sum;  // emissions of the walked cells in walk order (kSum)
};

// What a walk does with each cell: store the pair, sum its emission (walk
// order), or record it in a speculative segment map (spec[band - band_lo] =
// k | index << 22 for the cells below band spec_hi).
enum WalkMode { kWalkPairs = 0, kWalkSum = 1, kWalkSpec = 2 };

// Walks the path from (w.k, w.e) while its band is >= band_lo.  The trace tiles
// come from `trace` (band trace_band0 at its start; bands below bands_end exist)
// through a shared-memory ring of kRing 16-band chunks: the chunk being walked
// and the one below it resident, the others in flight.  Each round of loads
// takes the backpointers of the nine cells two moves can reach and takes up to
// three steps from them; the moves are decoded arithmetically (D = 0, U = 1,
// L = 2: the k-mer steps back unless U, the event unless L).  Every lane walks
// the same path; lane 0 stores.  Returns true once the path has ended (k or e
// below 0); false when it left the segment.

template <int kMode, int kRing>
__device__ bool walk_segment(const uint8_t* trace, int trace_band0, int bands_end, int band_lo, uint8_t* ring,
                             int lane, Walk& w, abea_aligned_pair_t* out, int cap, const PostArgs& a,
                             const ReadDesc& r, int32_t* spec = nullptr, int spec_hi = 0) {
    constexpr bool kSum = kMode == kWalkSum;
    static_assert(kRing >= 4 && (kRing & (kRing - 1)) == 0, "ring of a power of two chunks, at least four");
    const int bands_pad = (bands_end + 3) & ~3;
    const int c_lo = band_lo / kPostChunkBands;
    auto stage = [&](int c) {  // chunk c = bands [16c, 16c + 16)
        if (c >= c_lo) {
            const int lo_band = c * kPostChunkBands;
            const int bytes = min(kPostChunkBands, bands_pad - lo_band) * kSlots;
            const uint8_t* src = trace + (int64_t)(lo_band - trace_band0) * kSlots;
            uint8_t* dst = ring + (c & (kRing - 1)) * (kPostChunkBands * kSlots);
            for (int off = lane * 16; off < bytes; off += 32 * 16) cp_async16(dst + off, src + off);
        }
        cp_async_commit();  // an empty group keeps the group count in step
    };
    const uint8_t* tb = ring;
    auto T = [&](int band, int k) -> uint32_t {  // 0, 1 or 2; the clamp keeps every step a move
        const int rb = band & (kRing * kPostChunkBands - 1);
        return min((uint32_t)tb[((rb >> 2) << 9) | ((k & 127) << 2) | (rb & 3)], 2u);
    };
    int k = __shfl_sync(kFull, w.k, 0), e = __shfl_sync(kFull, w.e, 0);
    int c = (e + k + 2) / kPostChunkBands;
    // chunks c and c-1 resident while chunk c is walked, kRing - 2 more in flight
#pragma unroll
    for (int j = 0; j < kRing - 1; ++j) stage(c - j);
    bool ended = false, left_seg = false;
    for (; c >= c_lo && !ended && !left_seg; --c) {
        cp_async_wait_group<kRing - 3>();  // chunks c and c-1 have landed
        __syncwarp();
        stage(c - (kRing - 1));  // into the ring slot of chunk c+1, already walked
        // Every lane walks the same path (warp-uniform branches: the walk in one
        // divergent lane ran slower); lane 0 stores the pairs.
        {
            const int lo = c * kPostChunkBands;
            auto emit = [&](int kk, int ee, uint32_t f) {
                if (kMode == kWalkSpec) {
                    const int band = ee + kk + 2;
                    if (band < spec_hi) {
                        if (lane == 0) spec[band - band_lo] = kk | (w.n_out << 22);
                        ++w.n_out;
                    }
                    return;
                }
                if (kSum)
                    w.sum = __dadd_rn(w.sum, (double)path_emission(a, r, kk, ee));
                else if (w.n_out < cap && lane == 0)
                    out[w.n_out] = abea_aligned_pair_t{kk, ee};
                ++w.n_out;
                w.last_k = kk;
                w.last_from = (int)f;
                w.gap = (f == ABEA_FROM_L) ? w.gap + 1 : 0;
                w.max_gap = max(w.max_gap, w.gap);
            };
            k = w.k;
            e = w.e;
            while (true) {
                const int band = e + k + 2;
                if ((k | e) < 0) {
                    ended = true;
                    break;
                }
                if (band < lo) {
                    left_seg = band < band_lo;
                    break;
                }
                // Up to three steps from one round of loads: the backpointers of every
                // cell two moves can reach (band offset db <= 4, k-mer offset dk <= 2;
                // bands >= lo - 4, resident) packed 2 bits each at position 3*db + dk.
                // A move adds 7 (D: db+2, dk+1), 3 (U: db+1) or 4 (L: db+1, dk+1).
                const uint32_t W = T(band, k) | (T(band - 1, k) << 6) | (T(band - 1, k - 1) << 8) |
                                   (T(band - 2, k) << 12) | (T(band - 2, k - 1) << 14) |
                                   (T(band - 2, k - 2) << 16) | (T(band - 3, k - 1) << 20) |
                                   (T(band - 3, k - 2) << 22) | (T(band - 4, k - 2) << 28);
                uint32_t pos2 = 0;  // 2 * position
#pragma unroll
                for (int st = 0; st < 3; ++st) {
                    const uint32_t f = (W >> pos2) & 3u;
                    emit(k, e, f);
                    k -= (int)((f & 1u) ^ 1u);
                    e -= (int)((f >> 1) ^ 1u);
                    pos2 += (0x86eu >> (4 * f)) & 0xfu;
                    // a step that ends the path or leaves the resident segment stops the round
                    if ((k | e) < 0 || e + k + 2 < band_lo) break;
                }
            }
            w.k = k;
            w.e = e;
        }
    }
    cp_async_wait_all();
    __syncwarp();
    return ended;
}

constexpr int kPostRingDeep = 8;  // trace chunks of a traceback with shared memory to spare (16 KB)
constexpr int kPostRingMany = 4;  // of each of a block's sixteen warps'

// Recomputes the trace of segment seg (bands [seg*kCkBands, (seg+1)*kCkBands)) of
// a checkpointed read into `mem` (kCkBands * kSlots bytes).  The whole warp calls it.
// Inlined at its three calls (as a function: the recompute of 1 kb reads 6-10% slower) but
// for ca.one_fill (kMany: where many warps may run it).
template <bool kMany>
__device__ __forceinline__ void recompute_segment(const CoreArgs& ca, const ReadDesc& r, Rings& rg, int lane, int seg,
                                                  uint8_t* mem) {
    FillSpan sp;
    sp.b_begin = max(2, seg * kCkBands);
    sp.b_end = min((seg + 1) * kCkBands, r.n_bands);
    sp.ck_in = seg > 0 ? ca.ck + r.ck_off + (int64_t)seg * kCkStride : nullptr;
    sp.ck_out = nullptr;
    sp.trace = mem;
    sp.trace_band0 = seg * kCkBands;
    sp.trace_tiles = kCkBands / 4;
    sp.side = false;
    if (kMany && ca.one_fill)
        fill_span<false>(ca, r, smem_u32(&rg), lane, sp);
    else
        fill_warp<false, true>(ca, r, rg, lane, sp);
    __syncwarp();
    __threadfence_block();
}

// One warp per read: best end, traceback, QC, reverse (GPU/align_cuda.cl:618-899).
// Best end (GPU/align_cuda.cl:722-746): the first strict maximum of
// s(e) = (float)(band + (n_events-e)*lp_trim) on the last k-mer column; the
// whole warp calls it and every lane gets the result (best_e = 0 when no end is finite).
__device__ void best_end_warp(const PostArgs& a, const ReadDesc& r, int lane, float& best_out, int& best_e_out) {
    const int n_events = r.n_events;
    const double lp_trim = a.g.lp_trim;
    const float* lastc = a.last_col + r.ev_off;
    float best = -INFINITY;
    int best_e = 0x7fffffff;
    for (int e = lane; e < n_events; e += 32) {
        const float v = lastc[e];
        if (v == -INFINITY) continue;  // -inf + finite is -inf: never a strict maximum
        const float s = __double2float_rn(__dadd_rn((double)v, __dmul_rn((double)(n_events - e), lp_trim)));
        if (s > best) {
            best = s;
            best_e = e;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float ob = __shfl_xor_sync(kFull, best, off);
        const int oe = __shfl_xor_sync(kFull, best_e, off);
        if (ob > best || (ob == best && oe < best_e)) {
            best = ob;
            best_e = oe;
        }
    }
    if (!(best > -INFINITY)) best_e = 0;
    best_out = best;
    best_e_out = best_e;
}


// QC, reverse and the per-read results of a walked path (GPU/align_cuda.cl:830-897).
template <int kRing>
__device__ void post_tail(const CoreArgs& ca, const PostArgs& a, int ri, const ReadDesc& r, uint8_t* ring, Rings& rg,
                          int lane, float best, int best_e, int n_out, int max_gap, int status, int last_k,
                          int last_from, uint8_t* ck_seg);

// `ring`: kRing * 2 KB of shared memory (16-byte aligned) for the traceback's trace chunks.
// A finished read's pairs out[0, n) into the caller's host buffer, when the batch
// mirrors its results there (threads t of nt; the pairs are final and visible to them).
__device__ __forceinline__ void mirror_pairs(const PostArgs& a, const ReadDesc& r, const abea_aligned_pair_t* out,
                                             int n, int t, int nt) {
    abea_aligned_pair_t* h = a.outm ? a.outm->pairs : nullptr;
    if (!h || n <= 0) return;
    h += r.out_off;
    for (int i = t; i < n; i += nt) h[i] = out[i];
}

template <int kRing>
__device__ void post_read_warp(const CoreArgs& ca, const PostArgs& a, int ri, uint8_t* ring, Rings& rg, int lane) {
    const ReadDesc r = a.reads[ri];
    if (r.skip) {
        if (lane == 0) {
            a.n_pairs[ri] = 0;
            if (a.outm && a.outm->n_pairs) a.outm->n_pairs[ri] = 0;
            a.best_scores[ri] = -INFINITY;
            a.status[ri] = 0;
        }
        return;
    }
    const int n_kmers = r.n_kmers, n_bands = r.n_bands;
    float best;
    int best_e;
    best_end_warp(a, r, lane, best, best_e);

    abea_aligned_pair_t* out = a.pairs + r.out_off;
    const uint8_t* trace = a.trace + r.trace_off * kSlots;
    uint8_t* ck_seg = r.ck ? ca.ck_scratch + (int64_t)r.ck_slot * (kCkBands * kSlots) : nullptr;  // recompute scratch
    const int32_t* bk0 = a.band_k0 + r.band_off;
    const int cap = r.out_cap;
    int n_out = 0, max_gap = 0, status = 0, last_k = n_kmers - 1, last_from = 0;

    if (best > -INFINITY) {
        // A finite end: the path only visits computed cells.
        Walk w{n_kmers - 1, best_e, 0, 0, 0, n_kmers - 1, 0, 0.0};
        if (!r.ck) {
            walk_segment<kWalkPairs, kRing>(trace, 0, n_bands, 0, ring, lane, w, out, cap, a, r);
        } else {
            // the trace was not kept: recompute it kCkBands bands at a time from
            // the checkpoints, top segment first, and walk each
            for (int seg = (w.k + w.e + 2) / kCkBands; seg >= 0; --seg) {
                recompute_segment<kRing == kPostRingMany>(ca, r, rg, lane, seg, ck_seg);
                if (walk_segment<kWalkPairs, kRing>(ck_seg, seg * kCkBands, min((seg + 1) * kCkBands, n_bands),
                                               seg * kCkBands, ring, lane, w, out, cap, a, r))
                    break;
            }
        }
        n_out = w.n_out;
        max_gap = w.max_gap;
        last_k = w.last_k;
        last_from = w.last_from;
    } else if (lane == 0 && r.ck) {
        // No finite end on a read whose trace was not kept: the flat-array walk
        // below needs the whole trace.  Reported as undefined.
        status = ABEA_ERR_UNDEFINED;
    } else if (lane == 0) {
        // No finite end: the reference walks from (0, n_kmers-1) through its flat
        // band array, where an offset outside the band reads a neighbouring row.
        // Emulated cell by cell from band_k0; reads outside the read's rows have
        // no defined answer.
        int cur_e = 0, cur_k = n_kmers - 1, gap = 0;
        while (cur_k >= 0 && cur_e >= 0) {
            if (n_out < cap) out[n_out] = abea_aligned_pair_t{cur_k, cur_e};
            ++n_out;
            last_k = cur_k;
            const int64_t band = (int64_t)cur_e + cur_k + 2;
            const int64_t flat = band * kBand + ((band - 2 - bk0[band]) - cur_e);
            if (flat < 0 || flat >= (int64_t)n_bands * kBand) {
                status = ABEA_ERR_UNDEFINED;
                break;
            }
            const int64_t b2 = flat / kBand;
            const uint32_t from = trace[trace_index(b2, (bk0[b2] + (int)(flat - b2 * kBand)) & 127)];
            last_from = (int)from;
            step_back(from, cur_k, cur_e, gap, max_gap);
        }
    }
    n_out = __shfl_sync(kFull, n_out, 0);
    max_gap = __shfl_sync(kFull, max_gap, 0);
    status = __shfl_sync(kFull, status, 0);
    last_k = __shfl_sync(kFull, last_k, 0);
    last_from = __shfl_sync(kFull, last_from, 0);
    __syncwarp();
    __threadfence_block();
    post_tail<kRing>(ca, a, ri, r, ring, rg, lane, best, best_e, n_out, max_gap, status, last_k, last_from, ck_seg);
}

template <int kRing>
__device__ void post_tail(const CoreArgs& ca, const PostArgs& a, int ri, const ReadDesc& r, uint8_t* ring, Rings& rg,
                          int lane, float best, int best_e, int n_out, int max_gap, int status, int last_k,
                          int last_from, uint8_t* ck_seg) {
    const int n_kmers = r.n_kmers, n_bands = r.n_bands;
    abea_aligned_pair_t* out = a.pairs + r.out_off;
    const uint8_t* trace = a.trace + r.trace_off * kSlots;
    const int32_t* bk0 = a.band_k0 + r.band_off;
    const int cap = r.out_cap;
    int result = 0;
    bool reversed = false;
    if (status == 0 && n_out > 0) {
        // QC (GPU/align_cuda.cl:856-882).  After the reversal out[0] is the last
        // cell walked and out[n-1] the first, so spanned <=> last_k == 0.
        double sum;
        if (n_out <= cap) {
            // Every emission with 0.5 <= |em| < 2^20 is a multiple of 2^-24; when the
            // magnitudes sum below 2^53 * 2^-24 all of the reference's partial double
            // sums are exact and equal this integer sum, whatever the order.
            long long isum = 0, iabs = 0;
            bool exact = true;
#pragma unroll 4
            for (int i2 = lane; i2 < n_out; i2 += 32) qc_term(a, r, out[i2], isum, iabs, exact);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                isum += __shfl_xor_sync(kFull, isum, off);
                iabs += __shfl_xor_sync(kFull, iabs, off);
            }
            exact = __all_sync(kFull, exact) && iabs < (1ll << 53);
            if (exact) {
                sum = __dmul_rn((double)isum, 5.9604644775390625e-08);  // * 2^-24
            } else {
                sum = 0.0;  // serial, in walk order (out[0] is the first cell walked)
                if (lane == 0)
                    for (int i2 = 0; i2 < n_out; ++i2)
                        sum = __dadd_rn(sum, (double)path_emission(a, r, out[i2].ref_pos, out[i2].read_pos));
                sum = __shfl_sync(kFull, sum, 0);
            }
        } else if (!r.ck) {
            sum = 0.0;
            if (lane == 0)
                sum = serial_path_sum(a, r, trace, bk0, !(best > -INFINITY), best > -INFINITY ? best_e : 0,
                                      n_kmers - 1);
            sum = __shfl_sync(kFull, sum, 0);
        } else {
            // the path outgrew its output slot on a read whose trace was not kept:
            // recompute and walk again, summing the emissions in walk order
            Walk w{n_kmers - 1, best_e, 0, 0, 0, n_kmers - 1, 0, 0.0};
            for (int seg = (w.k + w.e + 2) / kCkBands; seg >= 0; --seg) {
                recompute_segment<kRing == kPostRingMany>(ca, r, rg, lane, seg, ck_seg);
                if (walk_segment<kWalkSum, kRing>(ck_seg, seg * kCkBands, min((seg + 1) * kCkBands, n_bands),
                                              seg * kCkBands, ring, lane, w, out, cap, a, r))
                    break;
            }
            sum = __shfl_sync(kFull, w.sum, 0);
        }
        const double avg = __ddiv_rn(sum, (double)n_out);
        const bool pass = !(avg < -5.0) && last_k == 0 && max_gap <= 50;
        if (pass && n_out > cap) {
            status = ABEA_ERR_CAPACITY;
            result = ABEA_ERR_CAPACITY;
        } else if (pass) {
            // reverse in place (GPU/align_cuda.cl:830-843)
            for (int i2 = lane; i2 < n_out / 2; i2 += 32) {
                const abea_aligned_pair_t x = out[i2], y = out[n_out - 1 - i2];
                out[i2] = y;
                out[n_out - 1 - i2] = x;
            }
            result = n_out;
            reversed = true;
            __syncwarp();
            mirror_pairs(a, r, out, n_out, lane, 32);
        }
    } else if (status != 0) {
        result = status;
    }
    if (lane == 0) post_write(a, ri, result, best, best_e, status, n_out, cap, reversed, last_from);
}

// The per-read results, and the path the adjoint reads: its length, whether the
// output holds it in walk order or reversed, and the move into its last walked cell.
__device__ __forceinline__ void post_write(const PostArgs& a, int ri, int result, float best, int best_e, int status,
                                           int n_out, int cap, bool reversed, int last_from) {
    {
        a.n_pairs[ri] = result;
        if (a.outm && a.outm->n_pairs) a.outm->n_pairs[ri] = result;
        a.best_scores[ri] = best;
        a.status[ri] = status;
        if (a.path_len) {
            // the path for the adjoint: its length, whether the output holds it in
            // walk order or reversed, and the move into its last walked cell
            a.path_len[ri] = n_out;
            a.path_flags[ri] = (reversed ? kPathReversed : 0) | (n_out > cap ? kPathTruncated : 0) |
                               (best > -INFINITY ? 0 : kPathNoEnd) | (status != 0 ? kPathError : 0) |
                               (last_from << 8);
            a.best_event[ri] = best_e;
        }
    }
}

// ---------------------------------------------------------------- wide read's traceback, block-parallel
// The wide read's traceback is on the batch's critical path while the rest of its
// block waits, so the whole block walks it.  The path is cut into segments of
// kSpecBands bands.  Every thread walks one segment speculatively (up to
// kSpecRound segments at once), from the middle of the band kSpecMargin bands
// above it (paths from different cells of a band merge within a few dozen bands),
// recording its cells in a map in global scratch (L2); warp 0 then walks the true
// path through the round and, at the first cell it shares with a segment's
// speculative path, takes the rest of that segment from the map (the
// backpointers after a shared cell are the same); the block copies those cells
// into the output.  A segment whose speculative path the true one never meets is
// walked cell by cell, so the result never depends on the speculation.  Gaps, the
// last cell and the QC follow from the written pairs.
constexpr int kSpecMargin = 64;
constexpr int kSpecWarps = kWideThreads / 32;

struct WidePostSmem {  // overlays the wide fill's shared memory once the fill is done
    float best;
    int32_t best_e, k, e, n_out, done, max_gap, last_from, last_k, pass, qc_exact, slot;
    float wbest[kSpecWarps];
    int32_t wbest_e[kSpecWarps], qexact[kSpecWarps];
    long long qsum[kSpecWarps], qabs[kSpecWarps];
    union {
        struct {  // per segment of the round: where its speculative walk left, and the splice
            int32_t exit_k[kSpecRound], exit_e[kSpecRound], count[kSpecRound], ended[kSpecRound];
            int32_t task_idx[kSpecRound], task_off[kSpecRound];
        } seg;
        int32_t run[kWideThreads][4];  // per thread: leading L run, trailing L run, longest run, all L
    };
};

// All kWideThreads threads of the block call it.
__device__ void post_wide_block(const CoreArgs& ca, const PostArgs& a, int ri, uint8_t* wide_mem, Rings& rg0, int t,
                                int slot_of_block) {
    const int warp = t >> 5, lane = t & 31;
    WidePostSmem& ps = *reinterpret_cast<WidePostSmem*>(wide_mem);
    const ReadDesc r = a.reads[ri];
    // a path of several segments whose trace was kept and whose k-mers fit the map's 22 bits
    if (r.skip || r.ck || r.n_kmers >= (1 << 22) || r.n_bands < kSpecMinBands) {
        if (warp == 0) post_read_warp<kPostRingDeep>(ca, a, ri, wide_mem, rg0, lane);
        return;
    }
    {
        // best end by the block: the first strict maximum is the largest value at the
        // smallest event among equals, per thread, per warp, then over the warps
        const double lp_trim = a.g.lp_trim;
        const float* lastc = a.last_col + r.ev_off;
        float b = -INFINITY;
        int be = 0x7fffffff;
        for (int e = t; e < r.n_events; e += kWideThreads) {
            const float v = lastc[e];
            if (v == -INFINITY) continue;
            const float sv = __double2float_rn(__dadd_rn((double)v, __dmul_rn((double)(r.n_events - e), lp_trim)));
            if (sv > b) {
                b = sv;
                be = e;
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ob = __shfl_xor_sync(kFull, b, off);
            const int oe = __shfl_xor_sync(kFull, be, off);
            if (ob > b || (ob == b && oe < be)) {
                b = ob;
                be = oe;
            }
        }
        if (lane == 0) {
            ps.wbest[warp] = b;
            ps.wbest_e[warp] = be;
        }
        __syncthreads();
        if (t == 0) {
            for (int w = 1; w < kSpecWarps; ++w)
                if (ps.wbest[w] > b || (ps.wbest[w] == b && ps.wbest_e[w] < be)) {
                    b = ps.wbest[w];
                    be = ps.wbest_e[w];
                }
            ps.best = b;
            ps.best_e = b > -INFINITY ? be : 0;
            ps.slot = slot_of_block;  // the block's scratch slot for the maps (one wide read at a time)
        }
    }
    __syncthreads();
    const float best = ps.best;
    const int best_e = ps.best_e, slot = ps.slot;
    __syncthreads();  // read before warp 0 may reuse the memory below
    if (!(best > -INFINITY) || slot >= ca.n_spec) {
        if (warp == 0) post_read_warp<kPostRingDeep>(ca, a, ri, wide_mem, rg0, lane);
        return;
    }
    const int n_kmers = r.n_kmers, n_events = r.n_events, n_bands = r.n_bands, cap = r.out_cap;
    const uint8_t* trace = a.trace + r.trace_off * kSlots;
    const int32_t* bk0 = a.band_k0 + r.band_off;
    abea_aligned_pair_t* out = a.pairs + r.out_off;
    int32_t* map = ca.spec + (int64_t)slot * (kSpecRound * kSpecBands);
    const int b0 = best_e + n_kmers - 1 + 2;  // band of the path's first cell
    const int jtop = b0 / kSpecBands;
    if (t == 0) {
        ps.k = n_kmers - 1;
        ps.e = best_e;
        ps.n_out = 0;
        ps.done = 0;
    }
    for (int jr = jtop; jr >= 0; jr -= kSpecRound) {
        const int nseg = min(kSpecRound, jr + 1);  // segments jr, jr-1, ..., jr-nseg+1
        for (int i = t; i < nseg * kSpecBands; i += kWideThreads) map[i] = -1;
        __syncthreads();
        // ---- speculative walks: thread t takes segment jr - t, its trace bytes from L2
        if (t < nseg) {
            const int j = jr - t;
            const int seg_lo = j * kSpecBands, seg_hi = min(seg_lo + kSpecBands, n_bands);
            int k = n_kmers - 1, e = best_e;  // the top segment starts at the true start
            if (j != jtop) {
                const int sb = min(seg_hi - 1 + kSpecMargin, b0);
                int kk = bk0[sb] + kBand / 2;  // the middle of band sb, moved inside the read
                kk = max(kk, max(0, sb - 2 - (n_events - 1)));
                kk = min(kk, min(n_kmers - 1, sb - 2));
                k = kk;
                e = sb - 2 - kk;
            }
            int32_t* row = map + t * kSpecBands;
            int cnt = 0, ended = 0;
            while (true) {
                if ((k | e) < 0) {
                    ended = 1;
                    break;
                }
                const int band = e + k + 2;
                if (band < seg_lo) break;
                const uint32_t f = min((uint32_t)trace[trace_index(band, k & 127)], 2u);
                if (band < seg_hi && in_bounds(band - seg_lo, kSpecBands, ca.counters)) row[band - seg_lo] = k | (cnt++ << 22);
                k -= (int)((f & 1u) ^ 1u);
                e -= (int)((f >> 1) ^ 1u);
            }
            ps.seg.exit_k[t] = k;
            ps.seg.exit_e[t] = e;
            ps.seg.count[t] = cnt;
            ps.seg.ended[t] = ended;
            ps.seg.task_idx[t] = -1;
        }
        __syncthreads();
        // ---- the true path through the round (warp 0, every lane alike)
        if (warp == 0) {
            int k = ps.k, e = ps.e, n_out = ps.n_out;
            bool done = ps.done != 0;
            for (int wi = 0; wi < nseg && !done; ++wi) {
                const int seg_lo = (jr - wi) * kSpecBands;
                const int32_t* row = map + wi * kSpecBands;
                while (true) {
                    if ((k | e) < 0) {
                        done = true;
                        break;
                    }
                    const int band = e + k + 2;
                    if (band < seg_lo) break;
                    const int sp = row[band - seg_lo];
                    if (sp >= 0 && (sp & 0x3fffff) == k) {
                        // shared cell: the rest of the segment is the recorded path
                        const int idx = sp >> 22;
                        if (lane == 0) {
                            ps.seg.task_idx[wi] = idx;
                            ps.seg.task_off[wi] = n_out;
                        }
                        n_out += ps.seg.count[wi] - idx;
                        k = ps.seg.exit_k[wi];
                        e = ps.seg.exit_e[wi];
                        done = ps.seg.ended[wi] != 0;
                        break;
                    }
                    const uint32_t f = min((uint32_t)trace[trace_index(band, k & 127)], 2u);
                    if (lane == 0 && n_out < cap) out[n_out] = abea_aligned_pair_t{k, e};
                    ++n_out;
                    k -= (int)((f & 1u) ^ 1u);
                    e -= (int)((f >> 1) ^ 1u);
                }
            }
            if (lane == 0) {
                ps.k = k;
                ps.e = e;
                ps.n_out = n_out;
                ps.done = done ? 1 : 0;
            }
        }
        __syncthreads();
        // ---- the recorded parts, copied by the block
        for (int i = t; i < nseg * kSpecBands; i += kWideThreads) {
            const int wi = i / kSpecBands, idx0 = ps.seg.task_idx[wi];
            if (idx0 < 0) continue;
            const int sp = map[i];
            if (sp < 0 || (sp >> 22) < idx0) continue;
            const int pos = ps.seg.task_off[wi] + (sp >> 22) - idx0, kk = sp & 0x3fffff;
            if (pos < cap) out[pos] = abea_aligned_pair_t{kk, (jr - wi) * kSpecBands + (i % kSpecBands) - 2 - kk};
        }
        __syncthreads();
        if (ps.done) break;
    }
    const int n_out = ps.n_out;
    __syncthreads();  // read before warp 0 may reuse the memory below
    if (n_out > cap) {
        // the path outgrew its output slot: the serial walk handles what the reference does
        if (warp == 0) post_read_warp<kPostRingDeep>(ca, a, ri, wide_mem, rg0, lane);
        return;
    }
    // ---- gaps: the move out of pair i is L iff pair i+1 is the k-mer before at the same event;
    // out of the last pair, its backpointer
    if (t == 0) {
        const abea_aligned_pair_t lp = out[n_out - 1];
        ps.last_from = (int)min((uint32_t)trace[trace_index(lp.read_pos + lp.ref_pos + 2, lp.ref_pos & 127)], 2u);
    }
    __syncthreads();
    {
        const int per = (n_out + kWideThreads - 1) / kWideThreads;
        const int i0 = min(t * per, n_out), i1 = min(i0 + per, n_out);
        int pre = 0, cur = 0, mx = 0;
        bool all = true;
        abea_aligned_pair_t p = i0 < i1 ? out[i0] : abea_aligned_pair_t{0, 0};
        for (int i = i0; i < i1; ++i) {
            bool is_l;
            if (i + 1 < n_out) {
                const abea_aligned_pair_t q = out[i + 1];
                is_l = q.read_pos == p.read_pos && q.ref_pos == p.ref_pos - 1;
                p = q;
            } else {
                is_l = ps.last_from == ABEA_FROM_L;
            }
            cur = is_l ? cur + 1 : 0;
            mx = max(mx, cur);
            if (all && is_l) ++pre;
            all = all && is_l;
        }
        ps.run[t][0] = pre;
        ps.run[t][1] = cur;
        ps.run[t][2] = mx;
        ps.run[t][3] = all ? 1 : 0;
    }
    // ---- QC (GPU/align_cuda.cl:856-882): the exact integer emission sum by the block
    {
        long long isum = 0, iabs = 0;
        bool exact = true;
#pragma unroll 4
        for (int i = t; i < n_out; i += kWideThreads) qc_term(a, r, out[i], isum, iabs, exact);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            isum += __shfl_xor_sync(kFull, isum, off);
            iabs += __shfl_xor_sync(kFull, iabs, off);
        }
        exact = __all_sync(kFull, exact);
        if (lane == 0) {
            ps.qsum[warp] = isum;
            ps.qabs[warp] = iabs;
            ps.qexact[warp] = exact ? 1 : 0;
        }
    }
    __syncthreads();
    if (t == 0) {
        int carry = 0, best_run = 0;
        for (int i = 0; i < kWideThreads; ++i) {
            if (ps.run[i][3]) {
                carry += ps.run[i][0];
            } else {
                best_run = max(best_run, carry + ps.run[i][0]);
                carry = ps.run[i][1];
            }
            best_run = max(best_run, max(carry, ps.run[i][2]));
        }
        long long isum = 0, iabs = 0;
        bool exact = true;
        for (int w = 0; w < kSpecWarps; ++w) {
            isum += ps.qsum[w];
            iabs += ps.qabs[w];
            exact = exact && ps.qexact[w];
        }
        exact = exact && iabs < (1ll << 53);
        const int last_k = out[n_out - 1].ref_pos;  // the last cell walked (before the reversal)
        const double sum = __dmul_rn((double)isum, 5.9604644775390625e-08);  // * 2^-24
        const double avg = __ddiv_rn(sum, (double)n_out);
        ps.max_gap = best_run;
        ps.last_k = last_k;
        ps.qc_exact = exact ? 1 : 0;
        ps.pass = (!(avg < -5.0) && last_k == 0 && best_run <= 50) ? 1 : 0;
    }
    __syncthreads();
    const int max_gap = ps.max_gap, last_from = ps.last_from, last_k = ps.last_k;
    if (!ps.qc_exact) {
        // emissions outside the exact integer form: warp 0 sums serially in walk order
        if (warp == 0)
            post_tail<kPostRingDeep>(ca, a, ri, r, wide_mem, rg0, lane, best, best_e, n_out, max_gap, 0, last_k,
                                     last_from, nullptr);
        return;
    }
    const bool pass = ps.pass != 0;
    if (pass)  // reverse in place (GPU/align_cuda.cl:830-843)
        for (int i = t; i < n_out / 2; i += kWideThreads) {
            const abea_aligned_pair_t x = out[i], y = out[n_out - 1 - i];
            out[i] = y;
            out[n_out - 1 - i] = x;
        }
    if (pass && a.outm) {
        __syncthreads();  // the reversal is done
        mirror_pairs(a, r, out, n_out, t, kWideThreads);
    }
    if (t == 0) post_write(a, ri, pass ? n_out : 0, best, best_e, 0, n_out, cap, pass, last_from);
}

// ---------------------------------------------------------------- wide checkpointed read's traceback
static_assert(sizeof(int32_t) * kSpecRound * kSpecBands >= (size_t)(kWideThreads / 32) * kCkBands * kSlots,
              "a traceback map's memory holds one segment's trace per warp");
// A checkpointed read on the wide shape: the block's 16 warps recompute 16 segments of
// kCkBands bands at a time, top ones first, each into a part of `mem` (a traceback
// map's memory: the two never meet in one read), and warp 0 walks them.  One segment at a time on one warp, the
// recompute alone took 390 cycles per band (560 before the warp shape's grid loop) with
// the SM otherwise idle.  Every thread of the block calls it; `ended` in shared memory.
__device__ void post_ck_block(const CoreArgs& ca, const PostArgs& a, int ri, uint8_t* wide_mem, Rings* rings,
                              int32_t& ended, int t, uint8_t* mem) {
    constexpr int kSegBytes = kCkBands * kSlots;
    const int warp = t >> 5, lane = t & 31;
    const ReadDesc r = a.reads[ri];
    abea_aligned_pair_t* out = a.pairs + r.out_off;
    float best;
    int best_e;
    best_end_warp(a, r, lane, best, best_e);  // every warp alike
    Walk w{r.n_kmers - 1, best_e, 0, 0, 0, r.n_kmers - 1, 0, 0.0};
    if (best > -INFINITY) {
        for (int top = (w.k + w.e + 2) / kCkBands; top >= 0; top -= kWideThreads / 32) {
            if (top - warp >= 0)
                recompute_segment<false>(ca, r, rings[warp], lane, top - warp, mem + (int64_t)warp * kSegBytes);
            if (t == 0) ended = 0;
            __syncthreads();  // the segments are in memory
            if (warp == 0) {
                for (int i = 0; i < kWideThreads / 32 && top - i >= 0; ++i) {
                    const int seg = top - i;
                    if (walk_segment<kWalkPairs, kPostRingDeep>(mem + (int64_t)i * kSegBytes, seg * kCkBands,
                                                                min((seg + 1) * kCkBands, r.n_bands), seg * kCkBands,
                                                                wide_mem, lane, w, out, r.out_cap, a, r)) {
                        if (lane == 0) ended = 1;
                        break;
                    }
                }
            }
            __syncthreads();
            if (ended) break;
        }
    }
    if (warp != 0) return;
    __syncwarp();
    __threadfence_block();
    // without a finite end the reference's flat-array walk needs the whole trace: undefined
    post_tail<kPostRingDeep>(ca, a, ri, r, wide_mem, rings[0], lane, best, best_e, w.n_out, w.max_gap,
                             best > -INFINITY ? 0 : ABEA_ERR_UNDEFINED, w.last_k, w.last_from, mem);
}

// ---------------------------------------------------------------- plain form kernels
template <bool kScores>
__global__ void __launch_bounds__(32) abea_core_warp_kernel(CoreArgs a) {
    __shared__ __align__(16) Rings rg;
    const int i = blockIdx.x;
    if (i >= a.n_reads) return;
    const ReadDesc& r = a.reads[i];
    if (r.skip) return;
    if (r.ck)
        fill_warp<kScores, true>(a, r, rg, threadIdx.x, forward_span(a, r));
    else
        fill_warp<kScores, false>(a, r, rg, threadIdx.x, forward_span(a, r));
}

__global__ void __launch_bounds__(32) abea_post_kernel(const __grid_constant__ CoreArgs ca, const __grid_constant__ PostArgs a) {
    __shared__ __align__(16) uint8_t ring[kPostRingDeep * kPostChunkBands * kSlots];
    __shared__ __align__(16) Rings rg;  // recompute of checkpointed reads
    const int i = blockIdx.x;
    if (i >= a.n_reads) return;
    post_read_warp<kPostRingDeep>(ca, a, i, ring, rg, threadIdx.x);
}

// ---------------------------------------------------------------- batched form
constexpr int kBatchedWarps = kWideThreads / 32;

struct BatchedSmem {
    union {
        WideSmem wide;                 // phase 1: the block's wide read
        PostSmem post[kBatchedWarps];  // phase 2: every warp's post staging
    };
    Rings warp_rings[kBatchedWarps];   // phase 2: one per warp
    int32_t pick;                      // the block's wide read, or -1
    int32_t wide_slot;                 // the block's first pick: its traceback scratch slot
    int32_t free_rank;                 // rank among the blocks without a wide read, or -1
    int32_t ended;                     // a checkpointed read's path has ended
};
static_assert(offsetof(BatchedSmem, warp_rings) % 16 == 0 && offsetof(BatchedSmem, post) % 16 == 0 &&
                  sizeof(Rings) % 16 == 0 && sizeof(PostSmem) % 16 == 0,
              "cp.async destinations must be 16-byte aligned");
static_assert(sizeof(BatchedSmem) <= 227 * 1024, "batched kernel shared memory exceeds the per-block limit");
static_assert(offsetof(WideSmem, ems) % 16 == 0 && offsetof(WideSmem, emm) % 8 == 0 && offsetof(WideSmem, x) % 16 == 0 &&
                  offsetof(WideSmem, sc) % 16 == 0,
              "vector accesses to the emission and score rings must be aligned");
static_assert(sizeof(WideSmem) >= kPostRingDeep * kPostChunkBands * kSlots && alignof(WideSmem) >= 16,
              "the wide read's traceback ring lives in the wide fill's shared memory");
static_assert(sizeof(WidePostSmem) <= sizeof(WideSmem), "the wide read's traceback state fits the fill's memory");

template <bool kScores>
__global__ void __launch_bounds__(kWideThreads, 1) abea_batched_kernel(const __grid_constant__ CoreArgs a, const __grid_constant__ PostArgs p,
                                                                       const __grid_constant__ PreArgs pa) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BatchedSmem& sm = *reinterpret_cast<BatchedSmem*>(smem_raw);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    // phase 1: the wide reads, longest first
    // Each block's first pick decides its role: the first blocks to arrive take a
    // wide read each (and then pull the wide reads past the first wave, one after
    // another); the others the first wave of the warp-shape reads.
    if (t == 0) {
        const int q = atomicAdd(&a.queue[0], 1);
        sm.pick = q < a.n_wide ? a.order[q] : -1;
        sm.wide_slot = q;  // the block's traceback scratch slot: wide reads go longest first, so only
                           // the first blocks' reads (and the reads they pull later) need one
        sm.free_rank = q < a.n_wide ? -1 : q - a.n_wide;
    }
    __syncthreads();
    int wide_read = sm.pick;
    const int free_rank = sm.free_rank, wide_slot = sm.wide_slot;
    while (wide_read >= 0) {
        const ReadDesc& r = a.reads[wide_read];
        const bool odd = __syncthreads_or(pre_read<true>(pa, wide_read, t, kWideThreads));  // and its parameters are in memory
        bool filled = true;
        if (!r.skip) {
            if (r.ck)
                filled = fill_chain<kScores, true>(a, r, smem_u32(&sm.wide), t, odd);
            else
                filled = fill_chain<kScores, false>(a, r, smem_u32(&sm.wide), t, odd);
        }
        __syncthreads();
        __threadfence_block();
        // the whole block walks the wide read's traceback (the fill's shared memory is free)
        if (!filled) {
            if (t == 0) post_write(p, wide_read, ABEA_ERR_TIMEOUT, -INFINITY, 0, ABEA_ERR_TIMEOUT, 0, r.out_cap, false, 0);
        } else if (r.ck && !r.skip && wide_slot < a.n_spec)
            post_ck_block(a, p, wide_read, reinterpret_cast<uint8_t*>(&sm.wide), sm.warp_rings, sm.ended, t,
                          reinterpret_cast<uint8_t*>(a.spec + (int64_t)wide_slot * (kSpecRound * kSpecBands)));
        else
            post_wide_block(a, p, wide_read, reinterpret_cast<uint8_t*>(&sm.wide), sm.warp_rings[0], t, wide_slot);
        // then the next wide read past the first wave (one per block), longest first
        __syncthreads();  // the traceback is done with the block's shared memory and the pick
        if (t == 0) {
            const int q = (int)gridDim.x + atomicAdd(&a.queue[4], 1);
            sm.pick = q < a.n_wide ? a.order[q] : -1;
        }
        __syncthreads();
        wide_read = sm.pick;
    }
    // phase 2: the first wave is static, the blocks without a wide read taking the
    // longest remaining reads round-robin (warp w of free block f:
    // read f + F*w), so that the long ones spread over the SMs; then every warp
    // pulls the rest longest-first.
    const int n_rest = a.n_reads - a.n_wide;
    const int n_free = max((int)gridDim.x - a.n_wide, 0);
    const int wave = min(n_rest, n_free * kBatchedWarps);
    for (int pass = 0;; ++pass) {
        int q;
        if (pass == 0) {
            if (free_rank < 0) continue;
            q = free_rank + n_free * warp;
            if (q >= wave) continue;
        } else {
            q = 0;
            if (lane == 0) q = wave + atomicAdd(&a.queue[1], 1);
            q = __shfl_sync(kFull, q, 0);
            if (q >= n_rest) break;
        }
        const int ri = a.order[a.n_wide + q];
        const ReadDesc& r = a.reads[ri];
        pre_read<false>(pa, ri, lane, 32);
        __syncwarp();  // the read's parameters are in memory for the warp
        if (!r.skip) {
            if (a.one_fill)
                fill_span<kScores>(a, r, smem_u32(&sm.warp_rings[warp]), lane, forward_span(a, r));
            else if (r.ck)
                fill_warp<kScores, true>(a, r, sm.warp_rings[warp], lane, forward_span(a, r));
            else
                fill_warp<kScores, false>(a, r, sm.warp_rings[warp], lane, forward_span(a, r));
        }
        __syncwarp();
        __threadfence_block();
        post_read_warp<kPostRingMany>(a, p, ri, sm.post[warp].tr, sm.warp_rings[warp], lane);
    }
}

struct BatchedClSmem {
    union {
        ClSmem wide;                       // phase 1: the cluster's wide read
        Rings warp_rings[kBatchedWarps];   // then: one per warp
    };
    PostSmem post[kBatchedWarps];          // every warp's post staging
    ClShared cs;
};
static_assert(offsetof(BatchedClSmem, warp_rings) % 16 == 0 && offsetof(BatchedClSmem, post) % 16 == 0,
              "cp.async destinations must be 16-byte aligned");
static_assert(sizeof(BatchedClSmem) <= 227 * 1024, "cluster kernel shared memory exceeds the per-block limit");

// The batched form on clusters of two blocks: phase 1 fills one of the longest
// reads per cluster with the cluster-pair wide shape, phase 2 as the
// single-block kernel.
template <bool kScores>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWideThreads, 1)
    abea_batched_cl_kernel(const __grid_constant__ CoreArgs a, const __grid_constant__ PostArgs p) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    BatchedClSmem& sm = *reinterpret_cast<BatchedClSmem*>(smem_raw);
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned rank = cluster.block_rank();
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (rank == 0 && t == 0) {
        const int q = atomicAdd(&a.queue[0], 1);
        const int pick = q < a.n_wide ? a.order[q] : -1;
        sm.cs.pick = pick;
        *cluster.map_shared_rank(&sm.cs.pick, 1) = pick;
    }
    cluster.sync();
    const int wide_read = sm.cs.pick;
    if (wide_read >= 0) {
        const ReadDesc& r = a.reads[wide_read];
        if (!r.skip) fill_wide_cl<kScores>(a, r, sm.wide, sm.cs, t, rank);
        // every emission copy has landed (block 0 consumed them all) before either
        // block reuses the fill's shared memory
        cluster.sync();
        __threadfence_block();
        if (rank == 0 && warp == 0) post_read_warp<kPostRingMany>(a, p, wide_read, sm.post[0].tr, sm.warp_rings[0], lane);
    }
    // phase 2: every warp pulls reads longest-first
    const int n_rest = a.n_reads - a.n_wide;
    while (true) {
        int q = 0;
        if (lane == 0) q = atomicAdd(&a.queue[1], 1);
        q = __shfl_sync(kFull, q, 0);
        if (q >= n_rest) break;
        const int ri = a.order[a.n_wide + q];
        const ReadDesc& r = a.reads[ri];
        if (!r.skip) {
            if (r.ck)
                fill_warp<kScores, true>(a, r, sm.warp_rings[warp], lane, forward_span(a, r));
            else
                fill_warp<kScores, false>(a, r, sm.warp_rings[warp], lane, forward_span(a, r));
        }
        __syncwarp();
        __threadfence_block();
        post_read_warp<kPostRingMany>(a, p, ri, sm.post[warp].tr, sm.warp_rings[warp], lane);
    }
    cluster.sync();  // neither block leaves while the other may still write its shared memory
}

// ---------------------------------------------------------------- launches
cudaError_t launch_plain(const LaunchArgs& la, int* launches) {
    const int n = la.core.n_reads;
    abea_pre_kernel<<<n, 128, 0, la.stream>>>(la.pre);
    cudaEventRecordWithFlags(la.ev_pre, la.stream, la.capturing ? cudaEventRecordExternal : cudaEventRecordDefault);
    if (la.core.scores)
        abea_core_warp_kernel<true><<<n, 32, 0, la.stream>>>(la.core);
    else
        abea_core_warp_kernel<false><<<n, 32, 0, la.stream>>>(la.core);
    cudaEventRecordWithFlags(la.ev_core, la.stream, la.capturing ? cudaEventRecordExternal : cudaEventRecordDefault);
    abea_post_kernel<<<n, 32, 0, la.stream>>>(la.core, la.post);
    *launches = 3;
    return cudaGetLastError();
}

int batched_blocks_per_sm(bool scores) {
    static int cached[2] = {0, 0};
    int& c = cached[scores ? 1 : 0];
    if (c == 0) {
        const size_t smem = sizeof(BatchedSmem);
        if (scores) {
            cudaFuncSetAttribute(abea_batched_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, abea_batched_kernel<true>, kWideThreads, smem);
        } else {
            cudaFuncSetAttribute(abea_batched_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, abea_batched_kernel<false>, kWideThreads, smem);
        }
        if (c <= 0) c = 1;
    }
    return c;
}

static int cl_max_dyn_smem_set() {
    static int done = 0;
    if (!done) {
        cudaFuncSetAttribute(abea_batched_cl_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(BatchedClSmem));
        cudaFuncSetAttribute(abea_batched_cl_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(BatchedClSmem));
        done = 1;
    }
    return done;
}

cudaError_t launch_batched(const LaunchArgs& la, int* launches) {
    const int n = la.core.n_reads;
    if (la.cluster) abea_pre_kernel<<<n, 128, 0, la.stream>>>(la.pre);  // otherwise pre runs inside the kernel
    cudaEventRecordWithFlags(la.ev_pre, la.stream, la.capturing ? cudaEventRecordExternal : cudaEventRecordDefault);
    const bool scores = la.core.scores != nullptr;
    if (la.cluster) {
        // one wide read per cluster of two blocks; an even grid of one block per SM
        cl_max_dyn_smem_set();
        const int want = 2 * la.core.n_wide + (n - la.core.n_wide + kBatchedWarps - 1) / kBatchedWarps;
        const int grid = 2 * std::max(1, std::min(la.sm_count / 2, (want + 1) / 2));
        const size_t smem = sizeof(BatchedClSmem);
        if (scores)
            abea_batched_cl_kernel<true><<<grid, kWideThreads, smem, la.stream>>>(la.core, la.post);
        else
            abea_batched_cl_kernel<false><<<grid, kWideThreads, smem, la.stream>>>(la.core, la.post);
        cudaEventRecordWithFlags(la.ev_core, la.stream,
                                 la.capturing ? cudaEventRecordExternal : cudaEventRecordDefault);
        *launches = 2;
        return cudaGetLastError();
    }
    // every resident block: the blocks without a wide read share the first wave
    const int max_blocks = batched_blocks_per_sm(scores) * la.sm_count;
    const int grid = std::max(1, std::min(max_blocks, n));
    const size_t smem = sizeof(BatchedSmem);
    if (scores)
        abea_batched_kernel<true><<<grid, kWideThreads, smem, la.stream>>>(la.core, la.post, la.pre);
    else
        abea_batched_kernel<false><<<grid, kWideThreads, smem, la.stream>>>(la.core, la.post, la.pre);
    cudaEventRecordWithFlags(la.ev_core, la.stream, la.capturing ? cudaEventRecordExternal : cudaEventRecordDefault);
    *launches = 1;
    return cudaGetLastError();
}

}  // namespace abea

// ---------------------------------------------------------------- no-allocation entry point
// For callers that cannot allocate device memory: a framework whose own
// allocator owns the whole device and hands out every buffer, or a service whose
// device memory budget is fixed when it starts.  One read goes through the plain
// pre/core/post kernels with every scratch buffer carved out of one file-scope
// device array, which exists on every GPU that loads this library for the life
// of the process.  Calls whose work overlaps on the GPU race on that array.
namespace abea {

constexpr size_t kNoAllocScratchBytes = 32ull << 20;  // 32 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

__global__ void noalloc_write_desc(ReadDesc* dst, ReadDesc d) { *dst = d; }

// The array's device address differs per CUDA context: one per device for the
// runtime's primary contexts, a new one after cudaDeviceReset, and one in each
// context a caller creates itself.  The addresses are kept per context, keyed by
// the context's process-unique id (cuCtxGetId; a context's handle may be reused
// after a reset, its id is not).  The two driver calls are found through the
// runtime (cudaGetDriverEntryPointByVersion), so the library needs no link
// against the driver library.
static std::mutex g_noalloc_mutex;
struct NoAllocSlot {
    unsigned long long ctx_id;
    void* ptr;
};
static NoAllocSlot g_noalloc_slots[64];  // most recently looked up first
typedef int (*CtxGetCurrentFn)(void** ctx);
typedef int (*CtxGetIdFn)(void* ctx, unsigned long long* id);

// Id of the current context, 0 when none is current or the driver calls are missing.
static unsigned long long current_ctx_id() {
    static CtxGetCurrentFn get_current = nullptr;
    static CtxGetIdFn get_id = nullptr;
    static bool looked_up = false;
    if (!looked_up) {
        void* f1 = nullptr;
        void* f2 = nullptr;
        cudaDriverEntryPointQueryResult q1, q2;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) == cudaSuccess &&
            q1 == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) == cudaSuccess &&
            q2 == cudaDriverEntryPointSuccess) {
            get_current = (CtxGetCurrentFn)f1;
            get_id = (CtxGetIdFn)f2;
        }
        looked_up = true;
    }
    void* ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != 0 || !ctx || get_id(ctx, &id) != 0) return 0;
    return id;
}

// Device address of g_noalloc_scratch in the current context: looked up with
// cudaGetSymbolAddress the first time a context asks, then kept.  nullptr on failure.
static void* noalloc_scratch_address(cudaError_t* err) {
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    unsigned long long id = current_ctx_id();
    if (id != 0) {
        for (int i = 0; i < 64 && g_noalloc_slots[i].ptr; ++i)
            if (g_noalloc_slots[i].ctx_id == id) return g_noalloc_slots[i].ptr;
    }
    void* p = nullptr;
    *err = cudaGetSymbolAddress(&p, g_noalloc_scratch);  // makes the device's primary context current if none is
    if (*err != cudaSuccess || !p) return nullptr;
    if (id == 0) id = current_ctx_id();
    if (id != 0) {  // keep it, most recent first (the oldest of a full table is dropped)
        for (int i = 63; i > 0; --i) g_noalloc_slots[i] = g_noalloc_slots[i - 1];
        g_noalloc_slots[0] = NoAllocSlot{id, p};
    }
    return p;
}

static size_t noalloc_align(size_t x) { return (x + 255) & ~(size_t)255; }

// Bytes of scratch one read needs.
static size_t noalloc_bytes(int32_t sequence_len, int32_t n_events) {
    const int64_t nk = std::max<int64_t>(sequence_len - ABEA_KMER_SIZE + 1, 0);
    const int64_t ne = std::max<int64_t>(n_events, 0);
    const int64_t nb = (nk > 0 && ne > 0) ? ne + nk + 2 : 0;
    const size_t ne_pad = (size_t)round_up(std::max<int64_t>(ne, 1), kChunk);
    const size_t nk_pad = (size_t)round_up(std::max<int64_t>(nk, 1), kChunk);
    const size_t nb_pad = (size_t)round_up(std::max<int64_t>(nb, 4), 4);
    return noalloc_align(sizeof(ReadDesc)) + 2 * noalloc_align(4 * ne_pad) + 4 * noalloc_align(4 * nk_pad) +
           noalloc_align(nb_pad * kSlots) + noalloc_align(4 * nb_pad) + noalloc_align(16) +
           noalloc_align(8 * kCounters);
}

}  // namespace abea

extern "C" abea_status_t abea_align_noalloc(abea_aligned_pair_t* pairs, int32_t* n_pairs, int32_t out_capacity,
                                            const char* sequence, int32_t sequence_len, const abea_event_t* events,
                                            int32_t n_events, const abea_model_t* model, abea_scalings_t scaling,
                                            void* stream) {
    using namespace abea;
    if (!pairs || !n_pairs || !sequence || !model || out_capacity < 0 || sequence_len < 0 || n_events < 0 ||
        (n_events > 0 && !events)) {
        abea_internal_set_error("abea_align_noalloc: invalid argument");
        return ABEA_ERR_INVALID_ARG;
    }
    const size_t need = noalloc_bytes(sequence_len, n_events);
    if (need > kNoAllocScratchBytes) {
        char msg[256];
        snprintf(msg, sizeof(msg),
                 "abea_align_noalloc: the read needs %zu bytes of scratch but the fixed scratch holds %zu "
                 "bytes (reads of up to about 230,000 bands, n_events + n_kmers + 2)",
                 need, kNoAllocScratchBytes);
        abea_internal_set_error(msg);
        return ABEA_ERR_INVALID_ARG;
    }
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) {
        abea_internal_set_error("abea_align_noalloc: no current CUDA device");
        return ABEA_ERR_NO_DEVICE;
    }
    // the first call in each context (per device, and again after a device
    // reset) looks up the array's address; later calls reuse it
    cudaError_t serr = cudaSuccess;
    unsigned char* base = (unsigned char*)noalloc_scratch_address(&serr);
    if (!base) {
        char msg[256];
        snprintf(msg, sizeof(msg), "abea_align_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(serr));
        abea_internal_set_error(msg);
        return ABEA_ERR_CUDA;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const int32_t nk = sequence_len - ABEA_KMER_SIZE + 1;
    const int64_t nb = (nk > 0 && n_events > 0) ? (int64_t)n_events + nk + 2 : 0;
    const size_t ne_pad = (size_t)round_up(std::max<int64_t>(n_events, 1), kChunk);
    const size_t nk_pad = (size_t)round_up(std::max<int64_t>(nk, 1), kChunk);
    const size_t nb_pad = (size_t)round_up(std::max<int64_t>(nb, 4), 4);
    unsigned char* p = base;
    auto carve = [&](size_t bytes) {
        unsigned char* q = p;
        p += noalloc_align(bytes);
        return q;
    };
    ReadDesc* d_desc = (ReadDesc*)carve(sizeof(ReadDesc));
    float* ev_mean = (float*)carve(4 * ne_pad);
    float* last_col = (float*)carve(4 * ne_pad);
    float* km_gm = (float*)carve(4 * nk_pad);
    float* km_sd = (float*)carve(4 * nk_pad);
    float* km_rsd = (float*)carve(4 * nk_pad);
    float* km_k1 = (float*)carve(4 * nk_pad);
    uint8_t* trace = (uint8_t*)carve(nb_pad * kSlots);
    int32_t* band_k0 = (int32_t*)carve(4 * nb_pad);
    float* best = (float*)carve(4);
    int32_t* status = (int32_t*)(best + 1);
    unsigned long long* counters = (unsigned long long*)carve(8 * kCounters);

    const ReadDesc desc = describe_single_read(sequence_len, n_events, scaling, out_capacity);
    const GlobalConsts g = parity_consts();
    // every call shares the array: clear what must start at zero
    if (cudaMemsetAsync(counters, 0, 8 * kCounters, st) != cudaSuccess) {
        abea_internal_set_error("abea_align_noalloc: cudaMemsetAsync failed");
        return ABEA_ERR_CUDA;
    }
    noalloc_write_desc<<<1, 1, 0, st>>>(d_desc, desc);
    PreArgs pre{d_desc, 1, g, sequence, events, model, ev_mean, km_gm, km_sd, km_rsd, km_k1, last_col};
    CoreArgs core{d_desc, 1, g, ev_mean, km_gm, km_sd, km_rsd, km_k1, last_col, trace, nullptr, band_k0,
                  counters, nullptr, nullptr, 0, nullptr, nullptr, nullptr, 0, 1ll << 22};
    PostArgs post{d_desc,   1,      g,     ev_mean, km_gm,  km_sd,   km_k1,   km_rsd,  last_col,
                  trace,    band_k0, pairs, n_pairs, best,   status,  nullptr, nullptr, nullptr};
    abea_pre_kernel<<<1, 128, 0, st>>>(pre);
    abea_core_warp_kernel<false><<<1, 32, 0, st>>>(core);
    abea_post_kernel<<<1, 32, 0, st>>>(core, post);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        char msg[256];
        snprintf(msg, sizeof(msg), "abea_align_noalloc: launch failed: %s", cudaGetErrorString(e));
        abea_internal_set_error(msg);
        return ABEA_ERR_CUDA;
    }
    return ABEA_OK;
}

// ---------------------------------------------------------------- adjoint
// Gradient of the best path's log-likelihood along the fixed path of a finished
// forward run: the transitions and trims do not depend on the scalings or the
// pore model, so d(score)/d(theta) is the sum, over the path cells entered by a
// D or U move (the cells whose emission the score contains), of
//   d em/d shift = a/sd, d em/d scale = a*mu/sd, d em/d mu_k = a*scale/sd,
//   d em/d stdv_k = (a^2 - 1)/stdv_k, d em/d var = (a^2 - 1)/var (var-aware only),
// with em = log_inv_sqrt_2pi - log(sd) - a^2/2, a = (x - (scale*mu + shift))/sd,
// sd = stdv (times var when var-aware).  Everything is evaluated and accumulated
// in FP64.  Also accumulated: the Gauss-Newton normal equations of the residuals
// a in (shift, scale) — J^T J and J^T a with J = (-1/sd, -mu/sd) — and the FP64
// emission sum of the path.  One block per read, or a cluster of kAdjSplit blocks
// (a.split), over the path in up to kAdjSplit parts.  The parts and the order in which
// sums are combined (warps, lanes, parts) depend on the path's length alone, so a read's
// result does not depend on its batch.
// Bounded by the FP64 rate (some 60 operations per cell); on one warp per read it was
// the latency of three dependent loads per 32 cells (see launch_adjoint).
namespace abea {

constexpr int kAdjThreads = 256, kAdjSums = 9;

// A read's path as the backward pass walks it.
struct AdjPath {
    const AdjArgs& a;
    const ReadDesc r;
    int len, flags, st, cells;
    __device__ __forceinline__ AdjPath(const AdjArgs& args, int ri) : a(args), r(args.reads[ri]) {
        len = r.skip ? 0 : a.path_len[ri];
        flags = r.skip ? 0 : a.path_flags[ri];
        st = 0;
        if (len > 0 && (flags & (kPathTruncated | kPathNoEnd | kPathError)))
            st = (flags & kPathTruncated) ? ABEA_ERR_CAPACITY : ABEA_ERR_UNDEFINED;
        cells = st == 0 ? max(len, 0) : 0;
    }
    // adds path position j's terms: shift, scale, var, j11, j12, j22, t1, t2, em
    __device__ __forceinline__ void add(int j, double (&acc)[kAdjSums]) const {
        const abea_aligned_pair_t* out = a.pairs + r.out_off;
        const bool rev = (flags & kPathReversed) != 0;
        const int w = rev ? len - 1 - j : j;  // walk position, 0 = best end
        const abea_aligned_pair_t c = out[j];
        bool counted;
        if (w < len - 1) {
            const abea_aligned_pair_t nx = rev ? out[j - 1] : out[j + 1];
            counted = nx.read_pos == c.read_pos - 1;  // D or U: the next walked cell is one event back
        } else {
            counted = flags >> 8 != (int)ABEA_FROM_L;
        }
        if (!counted) return;
        const char* s = a.seq + r.seq_off;
        uint32_t rank = 0;
#pragma unroll
        for (int q = 0; q < ABEA_KMER_SIZE; ++q) rank = (rank << 2) | base_rank(s[c.ref_pos + q]);
        const abea_model_t m = a.model[rank];
        const double scale = r.scale, shift = r.shift, var = r.var, log_var = r.log_var;
        const double mu = m.level_mean, sig = m.level_stdv;
        const double sd = a.var_aware ? sig * var : sig;
        const double lsd = a.var_aware ? (double)m.level_log_stdv + log_var : (double)m.level_log_stdv;
        const double x = a.ev_mean[r.ev_off + c.read_pos];
        const double isd = 1.0 / sd;
        const double av = (x - (scale * mu + shift)) * isd;
        acc[0] += av * isd;
        acc[1] += av * mu * isd;
        if (a.var_aware) acc[2] += (av * av - 1.0) / var;
        acc[3] += isd * isd;
        acc[4] += mu * isd * isd;
        acc[5] += mu * mu * isd * isd;
        acc[6] -= av * isd;
        acc[7] -= av * mu * isd;
        acc[8] += -0.91893853320467274 - lsd - 0.5 * av * av;
        if (a.grad_model) {
            atomicAdd(&a.grad_model[2 * rank], av * scale * isd);
            atomicAdd(&a.grad_model[2 * rank + 1], (av * av - 1.0) / sig);
        }
    }
};
// Sum i of read ri.
__device__ __forceinline__ void adj_write(const AdjArgs& a, int ri, int i, double v) {
    if (i < 3)
        a.grad_scalings[3 * ri + i] = v;
    else if (i < 8)
        a.gn[5 * ri + i - 3] = v;
    else
        a.path_em[ri] = v;
}

template <int kBlocks>
__global__ void __cluster_dims__(kBlocks, 1, 1) __launch_bounds__(kAdjThreads) abea_adjoint_kernel(AdjArgs a) {
    namespace cg = cooperative_groups;
    __shared__ double sums[kAdjSums][kAdjThreads];
    __shared__ double part_sums[kAdjSplit][kAdjSums];  // the cluster's first block's are used
    const int ri = blockIdx.x / kBlocks, rank = blockIdx.x % kBlocks;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    if (kBlocks > 1) cg::this_cluster().sync();  // every block of the cluster runs before its memory is written
    const AdjPath p(a, ri);
    if (kBlocks == 1 && a.n_warp && adj_short(p.r)) return;  // abea_adjoint_warp_kernel's
    const int cells = p.cells;
    const int parts = min(kAdjSplit, 1 + cells / kAdjPart), per_part = (cells + parts - 1) / parts;
    // A short path's cells 256 at a time (a thread's one cell each), their terms added lane by
    // lane over the rows; a longer one's parts whole, each thread's sum first.
    const int step = cells <= kAdjShort ? kAdjThreads : per_part;
    for (int part = rank; part < parts; part += kBlocks) {
        const int first = part * per_part, end = min(cells, first + per_part);
        double v[2] = {0.0, 0.0};  // this warp's one or two sums
        for (int at = first; at < end || at == first; at += step) {
            double acc[kAdjSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            for (int j = at + t; j < min(end, at + step); j += kAdjThreads) p.add(j, acc);
            // A warp per sum: 3,700 additions, a third of butterflies over every warp (which
            // were a fifth of the FP64 work of a 600-base read).
#pragma unroll
            for (int i = 0; i < kAdjSums; ++i) sums[i][t] = acc[i];
            __syncthreads();
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = warp + h * (kAdjThreads / 32);
                if (i < kAdjSums)
#pragma unroll
                    for (int q = 0; q < kAdjThreads; q += 32) v[h] += sums[i][q + lane];
            }
            __syncthreads();  // the sums may be written again
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = warp + h * (kAdjThreads / 32);
            if (i >= kAdjSums) continue;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) v[h] += __shfl_xor_sync(kFull, v[h], off);
            if (lane == 0) {
                if (kBlocks > 1)
                    *cg::this_cluster().map_shared_rank(&part_sums[part][i], 0) = v[h];
                else
                    part_sums[part][i] = v[h];
            }
        }
    }
    __syncthreads();
    if (kBlocks > 1) {
        cg::this_cluster().sync();  // the other blocks' sums are in the first block's memory
        if (rank != 0) return;
    }
    if (t < kAdjSums) {
        double v = 0.0;
        for (int i = 0; i < parts; ++i) v += part_sums[i][t];
        adj_write(a, ri, t, v);
    }
    if (t == 0) a.adj_status[ri] = p.st;
}

// Many short reads: a warp per read.  A block per read leaves eight reads on an SM, and the
// latency of a read's loads and of its reduction is then the bound (20,000 reads of 50-120
// bases 0.60 ms a call, as warps 0.46).
__global__ void __launch_bounds__(32) abea_adjoint_warp_kernel(AdjArgs a) {
    const int ri = blockIdx.x, lane = threadIdx.x;
    const AdjPath p(a, ri);
    if (!adj_short(p.r)) return;
    double v[kAdjSums] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int j = lane; j < p.cells; j += 32) p.add(j, v);
#pragma unroll
    for (int i = 0; i < kAdjSums; ++i)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[i] += __shfl_xor_sync(kFull, v[i], off);
    if (lane == 0) {
#pragma unroll
        for (int i = 0; i < kAdjSums; ++i) adj_write(a, ri, i, v[i]);
        a.adj_status[ri] = p.st;
    }
}

// One warp per read took as long as the longest read: 1.7 ms of 512 reads of 1-10 kb, now
// 0.1-0.2; some 20 ms of a 12 Mb batch with a 65 kb read.
cudaError_t launch_adjoint(const AdjArgs& a, cudaStream_t stream) {
    if (a.n_reads <= 0) return cudaSuccess;
    if (a.split)
        abea_adjoint_kernel<kAdjSplit><<<a.n_reads * kAdjSplit, kAdjThreads, 0, stream>>>(a);
    else if (a.n_warp < a.n_reads)
        abea_adjoint_kernel<1><<<a.n_reads, kAdjThreads, 0, stream>>>(a);
    if (a.n_warp > 0) abea_adjoint_warp_kernel<<<a.n_reads, 32, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace abea

// ---------------------------------------------------------------- method of moments
// f5c's estimate_scalings_using_mom (GPU/f5cmisc.h:47; its body is not part of the
// reference): the scale and shift that map the k-mer levels along the read onto
// the event means' mean and variance.  FP64 sums, one warp per read.
namespace abea {

__global__ void __launch_bounds__(32) abea_mom_kernel(MomArgs a) {
    const int ri = blockIdx.x, lane = threadIdx.x;
    if (ri >= a.n_reads) return;
    const ReadDesc r = a.reads[ri];
    double es = 0.0, es2 = 0.0, ks = 0.0, ks2 = 0.0;
    if (!r.skip) {
        for (int e = lane; e < r.n_events; e += 32) {
            const double x = a.ev[r.ev_src + e].mean;
            es += x;
            es2 += x * x;
        }
        const char* s = a.seq + r.seq_off;
        for (int k = lane; k < r.n_kmers; k += 32) {
            uint32_t rank = 0;
#pragma unroll
            for (int q = 0; q < ABEA_KMER_SIZE; ++q) rank = (rank << 2) | base_rank(s[k + q]);
            const double l = a.model[rank].level_mean;
            ks += l;
            ks2 += l * l;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        es += __shfl_xor_sync(kFull, es, off);
        es2 += __shfl_xor_sync(kFull, es2, off);
        ks += __shfl_xor_sync(kFull, ks, off);
        ks2 += __shfl_xor_sync(kFull, ks2, off);
    }
    if (lane == 0) {
        double scale = 1.0, shift = 0.0;
        if (!r.skip) {
            const double em = es / r.n_events, ev = es2 / r.n_events - em * em;
            const double km = ks / r.n_kmers, kv = ks2 / r.n_kmers - km * km;
            scale = sqrt(ev / kv);
            shift = em - scale * km;
        }
        a.out[2 * ri] = scale;
        a.out[2 * ri + 1] = shift;
    }
}

cudaError_t launch_mom(const MomArgs& a, cudaStream_t stream) {
    if (a.n_reads > 0) abea_mom_kernel<<<a.n_reads, 32, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace abea

// ---------------------------------------------------------------- postalign
// f5c's postalign (GPU/f5cmisc.h:51-52, prototype only; the output types are
// GPU/f5c.h:184-207): the AlignedPairs of a read turned into its base-to-event
// map and its event alignment records.  One warp per read over the pairs in
// order, 32 at a time.
//
// A pair counts for its k-mer when its event differs from the previous pair's;
// such a pair is the first one of its event on the path.  The traceback's path
// moves by one k-mer, one event or both at every step, so the counting pairs
// are exactly one per event from the first event on the path to the last, in
// order: the record of event e sits at e - first event, and a k-mer's map
// entry runs from its first counting pair's event to its last one's.  The first
// pass checks that shape (and the bounds every store below relies on).
namespace abea {

constexpr int kPaUnroll = 8;  // chunks of 32 pairs whose loads are in flight together

__global__ void __launch_bounds__(128) abea_postalign_kernel(PostalignArgs a) {
    const int lane = threadIdx.x & 31;
    const int ri = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (ri >= a.n_reads) return;  // whole warps
    const ReadDesc r = a.reads[ri];
    int n = r.skip ? 0 : a.n_pairs[ri];
    if (n < 0) n = 0;  // a read that ended with an error status has no pairs
    const abea_aligned_pair_t* P = a.pairs + r.out_off;
    bool ok = n <= r.out_cap;
    // pass 1: bounds and unit steps; pair i-1 of lane 0 is lane 31 of the previous chunk
    if (__all_sync(kFull, ok)) {
        int k31 = -1, e31 = -1;
        for (int base = 0; base < n; base += 32 * kPaUnroll) {
            int kk[kPaUnroll], ee[kPaUnroll];
#pragma unroll
            for (int u = 0; u < kPaUnroll; ++u) {
                const int i = base + 32 * u + lane;
                kk[u] = -1;
                ee[u] = -1;
                if (i < n) {
                    const abea_aligned_pair_t p = P[i];
                    kk[u] = p.ref_pos;
                    ee[u] = p.read_pos;
                }
            }
#pragma unroll
            for (int u = 0; u < kPaUnroll; ++u) {
                const int i = base + 32 * u + lane;
                int qk = __shfl_up_sync(kFull, kk[u], 1), qe = __shfl_up_sync(kFull, ee[u], 1);
                if (lane == 0) {
                    qk = k31;
                    qe = e31;
                }
                if (i < n) {
                    if (kk[u] < 0 || kk[u] >= r.n_kmers || ee[u] < 0 || ee[u] >= r.n_events) {
                        ok = false;
                    } else if (i > 0) {
                        const int dk = kk[u] - qk, de = ee[u] - qe;
                        ok = ok && dk >= 0 && dk <= 1 && de >= 0 && de <= 1 && (dk | de) != 0;
                    }
                }
                k31 = __shfl_sync(kFull, kk[u], 31);
                e31 = __shfl_sync(kFull, ee[u], 31);
            }
        }
    }
    ok = __all_sync(kFull, ok);
    if (!ok || n == 0) {
        if (lane == 0) {
            a.count[ri] = ok ? 0 : ABEA_ERR_INTERNAL;
            a.epb[ri] = 0.0;
        }
        return;
    }
    // Pass 1 above accepted only paths whose every step moves the k-mer and the
    // event forward by 0 or 1 (not both 0): the events are non-decreasing along
    // the path, so its first and last pairs hold the smallest and largest event
    // (the oracle takes the minimum and maximum; a path that is not monotone
    // never gets here, it is ABEA_ERR_INTERNAL).
    const int e_first = P[0].read_pos, e_last = P[n - 1].read_pos;
    const char* s = a.seq + r.seq_off;
    abea_index_pair_t* map = a.map + r.seq_off;
    uint4* rec = reinterpret_cast<uint4*>(a.rec + r.ev_src);
    int carry_e = -1, carry_k = -1, carry_rank = -1;  // the previous pair's event; the previous counting pair
    for (int base = 0; base < n; base += 32 * kPaUnroll) {
        int kk[kPaUnroll], ee[kPaUnroll];
#pragma unroll
        for (int u = 0; u < kPaUnroll; ++u) {
            const int i = base + 32 * u + lane;
            kk[u] = -1;
            ee[u] = -1;
            if (i < n) {
                const abea_aligned_pair_t p = P[i];
                kk[u] = p.ref_pos;
                ee[u] = p.read_pos;
            }
        }
        // counting pairs (event differs from the previous pair's) and their k-mers' bases
        bool qq[kPaUnroll];
        uint32_t w0[kPaUnroll], w1[kPaUnroll];  // bases 0-3 and 4-5 of the k-mer, little-endian
#pragma unroll
        for (int u = 0; u < kPaUnroll; ++u) {
            int e_prev = __shfl_up_sync(kFull, ee[u], 1);
            if (lane == 0) e_prev = carry_e;
            qq[u] = base + 32 * u + lane < n && ee[u] != e_prev;
            carry_e = __shfl_sync(kFull, ee[u], 31);
            w0[u] = 0;
            w1[u] = 0;
            if (qq[u]) {
                const uint8_t* sb = reinterpret_cast<const uint8_t*>(s + kk[u]);
                w0[u] = (uint32_t)sb[0] | (uint32_t)sb[1] << 8 | (uint32_t)sb[2] << 16 | (uint32_t)sb[3] << 24;
                w1[u] = (uint32_t)sb[4] | (uint32_t)sb[5] << 8;
            }
        }
#pragma unroll
        for (int u = 0; u < kPaUnroll; ++u) {
            const int k = kk[u], e = ee[u];
            const bool q = qq[u];
            int rank = 0;
            if (q) {
#pragma unroll
                for (int j = 0; j < ABEA_KMER_SIZE; ++j)
                    rank = (rank << 2) | (int)base_rank((char)((j < 4 ? w0[u] >> (8 * j) : w1[u] >> (8 * (j - 4))) & 0xff));
            }
            const unsigned qm = __ballot_sync(kFull, q);
            const unsigned below = qm & ((1u << lane) - 1u);
            const unsigned above = qm & ~((2u << lane) - 1u);  // lane 31: 2u << 31 wraps to 0, so none above
            const int src = below ? 31 - __clz(below) : lane;
            const int dst = above ? __ffs(above) - 1 : lane;
            const int k_below = __shfl_sync(kFull, k, src);
            const int rank_below = __shfl_sync(kFull, rank, src);
            const int k_above = __shfl_sync(kFull, k, dst);
            if (q) {
                const int pk = below ? k_below : carry_k;
                const int pr = below ? rank_below : carry_rank;
                if (pk != k) map[k].start = e;                // first counting pair of this k-mer
                if (!above || k_above != k) map[k].stop = e;  // last one in this chunk; later chunks overwrite
                const uint32_t hmm = rank != pr ? 'M' : 'E';
                // the 32-byte event_alignment_t: ref_kmer[7] + pad, ref_position, read_idx,
                // event_idx, rc, model_kmer[7], hmm_state, pad (little-endian bytes)
                const uint4 lo = make_uint4(w0[u], w1[u], (uint32_t)k, (uint32_t)ri);
                const uint4 hi = make_uint4((uint32_t)e, w0[u] << 8, w0[u] >> 24 | w1[u] << 8, hmm);
                rec[2 * (e - e_first)] = lo;
                rec[2 * (e - e_first) + 1] = hi;
            }
            if (qm) {
                const int lq = 31 - __clz(qm);
                carry_k = __shfl_sync(kFull, k, lq);
                carry_rank = __shfl_sync(kFull, rank, lq);
            }
            __syncwarp();  // orders this chunk's map stores before the next chunk's
        }
    }
    if (lane == 0) {
        a.count[ri] = e_last - e_first + 1;
        a.epb[ri] = (double)(e_last - e_first) / r.n_kmers;
    }
}

cudaError_t launch_postalign(const PostalignArgs& a, cudaStream_t stream) {
    if (a.n_reads > 0) abea_postalign_kernel<<<(a.n_reads + 3) / 4, 128, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace abea
