// fns_rows.cuh - k_rows: the select + draw kernel for batches (k_cap up to 128), a row cut over a cluster of 1 to 8 CTAs.
// Included by fns_sampler.cu after fns_cluster.cuh.
//
// A batch has two bounds: HBM while rows stream, and the chain of dependent steps before and after a row's stream
// (about 10 us for one block).  So the batch is spread over the whole chip - a row is cut over as many CTAs as fill it,
// which meet in distributed shared memory - and up to three CTAs share an SM, whose chains and streams overlap (registers allow
// three; an uncut masked fp32 row of 151,936 needs 90 KB of shared memory, of which two fit).  The row goes from global memory
// straight into registers: 128-bit loads, two cells of four vectors in flight per thread, one three-input maximum per two
// elements, and per cell one 16-bit store that remembers its maximum.
//
//   list     under a mask: the 512-byte segments (what a warp loads with one instruction) that have an allowed id.
//            Segments that are allowed as a whole are streamed without a look at the bit set; in the others a vector
//            without an allowed id is not loaded
//   history  ids set a bit each in a second bit set; the stream does not look at it and nothing is fetched for them
//            (gathering 2,048 logits per row was measured at 13 us of the 62 us that 256 rows took)
//   bound    256 witnesses per row, each the maximum of one group of lanes.  Without penalties the k-th largest is a
//            bound: k elements reach it.  With penalties a witness may be a history id, so the bound is a quarter of k
//            and eight witnesses lower, and it is the count of what was found that proves it.  If it does not, the witnesses
//            are made again from the cells without a history id (or, where these are few, the bound goes down first)
//   pass 2   the cells that reach the bound are read again (L2).  What reaches it goes to the CTA's buffer; a history id
//            among it takes its penalty first, and is dropped if that takes it below the bound.  Penalties that can
//            raise a value (repetition < 1, negative ones) look at every history id instead
//   finish   the CTAs send what they have to the row's CTA 0.  k keys or more are proof that the best k are among them:
//            CTA 0 ranks and draws (rank_draw)
//
// A row may start on any element: whole vectors start at the first 16-byte boundary, what lies before it (and after the
// last whole vector) is taken element by element, and the bit sets are read through a funnel shift.
// Equal values, or no bound, may bring more than the buffer holds: the k-th best of a full buffer is then the next bound.
// No waits but block and hardware cluster barriers.
#pragma once

namespace fnsb {

constexpr int kRowsThreads = 256;
constexpr int kRowsMaxK = 128;
constexpr int kRowsMaxCtas = 8;
constexpr int kRowsCell = 4;       // vectors per thread and cell
constexpr int kRowsMaxCells = 64;  // cells of a slice (one bit each in a thread's work mask)
constexpr int kRowsBuf = 1024;     // keys of a CTA's own buffer
constexpr int kRowsGather = 512;   // keys that all the CTAs of a row may send to CTA 0
constexpr int kWarpList = 96;      // cells of a warp that pass 2 can take
constexpr int kRowsDups = 1024;    // repeated history ids of a slice that are remembered

struct RowsShared {
    SelectShared s;
    fns_b200_params p;                   // the row's parameters
    uint32_t n_hl;                       // cursor of the list of history ids that need their occurrences
    uint32_t count[kRowsMaxCtas];        // how many keys every CTA sent to CTA 0
    uint32_t hl_pos[kRowsThreads];       // the list: positions f
    float hl_raw[kRowsThreads];          // ... and logits
    __align__(16) uint32_t lut[64];      // fill_or_masks
};

// A 16-byte load that happens only if `wanted` is not 0 (then r is replaced).  Written as one predicated instruction: with
// a branch the loaded words would be moved to their place where the paths meet, and the move waits for the load.
__device__ __forceinline__ void load_if(uint4 & r, const uint4 * at, uint32_t wanted) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.u32 p, %4, 0;\n@p ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%5];\n}\n"
                 : "+r"(r.x), "+r"(r.y), "+r"(r.z), "+r"(r.w)
                 : "r"(wanted), "l"(at));
}

template <typename T, int VEC>
__device__ __forceinline__ void raw_values(const uint4 & r, float (&x)[VEC]) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if constexpr (sizeof(T) == 4) {
            x[q] = __uint_as_float(w[q]);
        } else {
            x[2 * q] = __uint_as_float(w[q] << 16);
            x[2 * q + 1] = __uint_as_float(w[q] & 0xffff0000u);
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(kRowsThreads, 3) k_rows(const SelectArgs a) {
    namespace cg = cooperative_groups;
    constexpr int NT = kRowsThreads, kWarps = NT / 32;
    constexpr int VEC = 16 / (int) sizeof(T), NV = kRowsCell;
    constexpr uint32_t kVecBits = (1u << VEC) - 1u;
    constexpr uint32_t kCellBits = VEC * NV == 32 ? 0xffffffffu : (1u << ((VEC * NV) & 31)) - 1u;
    constexpr int TS = 2 * NT, kTShift = 23;  // slots of the occurrence-count table, 32 - log2(TS)
    constexpr uint32_t kNoKey = 0xffffffffu;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    cg::cluster_group cluster = cg::this_cluster();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int C = a.slices, lg_c = __ffs(C) - 1;
    const int row = (int) (blockIdx.x >> lg_c), rank = (int) (blockIdx.x & (unsigned) (C - 1));
    const int W = a.n_draft + 1, win = row / W, col = row - win * W;

    // The slice.  Positions f count from its first word of the bit set: element lo + f.  Whole vectors start at f = h.
    const T * xrow = reinterpret_cast<const T *>(a.logits) + (size_t) row * a.row_stride;
    const int lo = rank * a.slice_len;
    const int h = min((int) (((16u - ((uint32_t) reinterpret_cast<uintptr_t>(xrow) & 15u)) & 15u) / (uint32_t) sizeof(T)), a.vocab);
    const int f0 = rank == 0 ? 0 : h;                                       // the slice is [f0, f1)
    const int f1 = max(f0, min(a.slice_len + h, a.vocab - lo));
    const int nv = max(0, f1 - h) / VEC;                                    // whole vectors
    const int n_head = rank == 0 ? h : 0, n_rag = n_head + max(0, f1 - h - nv * VEC);  // elements outside them
    const int n_segs = (nv + 31) >> 5, n_whole = nv >> 5;
    const int eff_words = a.seg_cap;                                        // with zero words at the end (a multiple of 4)
    const T * x = xrow + lo;                                                // element f
    const T * xv0 = x + h;                                                  // vector 0
    const uint32_t id0 = (uint32_t) (a.id_base + lo);
    const bool listed = a.masks != nullptr;

    RowsShared & rs = *reinterpret_cast<RowsShared *>(smem_raw);
    SelectShared & sh = rs.s;
    constexpr size_t kRsBytes = (sizeof(RowsShared) + 15) & ~(size_t) 15;
    uint64_t * lbuf = reinterpret_cast<uint64_t *>(smem_raw + kRsBytes);    // [kRowsBuf]
    uint64_t * gbuf = lbuf + kRowsBuf;                                      // [kRowsGather] CTA 0's is used
    uint64_t * sel = gbuf + kRowsGather;                                    // [k_cap]
    uint64_t * sorted = sel + a.k_cap;                                      // [k_cap]
    double * pj = reinterpret_cast<double *>(sorted + a.k_cap);             // [k_cap]
    double * acc = pj + a.k_cap;                                            // [k_cap]
    uint32_t * wit = reinterpret_cast<uint32_t *>(acc + a.k_cap);           // [C * NT] the row's witnesses (every CTA gets a copy)
    uint32_t * eff = wit + C * NT;                                          // [eff_words] under a mask: bit f is allowed and in a whole vector
    uint32_t * hb = eff + (listed ? eff_words : 0);                         // [eff_words] with a history: bit f is a history id
    uint32_t * tkey = hb + (a.own_cap > 0 ? eff_words : 0);                 // [TS]
    uint32_t * tcnt = tkey + TS;                                            // [TS]
    uint32_t * vlist = tcnt + TS;                                           // [kWarps * kWarpList] cells to read again
    uint32_t * dups = vlist + kWarps * kWarpList;                           // [kRowsDups] with a history: its ids once for every occurrence after the first
    uint16_t * cmax = reinterpret_cast<uint16_t *>(dups + (a.own_cap > 0 ? kRowsDups : 0));  // [n_stages * NT] maxima of the cells
    uint16_t * seglist = cmax + a.n_stages * NT;                            // [list_cap] segments with an allowed id

    if (tid == 0) {
        sh.n_cand = 0u;
        sh.thr_key = 0ull;
        sh.n_own = 0u;
        sh.n_vl = 0u;
        sh.n_seg = 0u;
        rs.n_hl = 0u;
    }
    for (int i = tid; i < TS; i += NT) tkey[i] = kNoKey;
    if (listed)  // places that no segment takes name a segment behind the slice, whose bits are 0
        for (int i = tid; i < a.list_cap; i += NT) seglist[i] = (uint16_t) (a.slice_len / (32 * VEC));
    fill_or_masks<T>(rs.lut);
    if (a.own_cap > 0)
        for (int i = tid * 4; i < eff_words; i += NT * 4) *reinterpret_cast<uint4 *>(hb + i) = make_uint4(0u, 0u, 0u, 0u);
    if (C > 1) cluster.barrier_arrive();  // (waited for before the first store into another CTA: by then all have started)
    __syncthreads();
    // Launched with programmatic stream serialisation: nothing is read from global memory before the previous kernel of
    // the stream has finished; what precedes this line overlaps its tail.
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");

    // Everything whose address is known is requested before anything is waited for.
    const int32_t * hrow = a.history ? a.history + (size_t) win * a.history_stride : nullptr;
    const int32_t * drow = a.draft ? a.draft + (size_t) win * a.n_draft : nullptr;
    // (the parameters go to shared memory: kept in registers they would not leave enough of those for the stream)
    if (tid < (int) (sizeof(fns_b200_params) / 4))
        reinterpret_cast<uint32_t *>(&rs.p)[tid] = reinterpret_cast<const uint32_t *>(a.params ? a.params + win : &a.p0)[tid];
    int n_hist = (a.history && a.history_len) ? a.history_len[win] : 0;
    constexpr int HB = 8;  // history ids per thread and round
    int32_t ids[HB];
#pragma unroll
    for (int u = 0; u < HB; ++u) {
        const int j = u * NT + tid;
        ids[u] = (hrow && a.own_cap > 0 && j < (int) a.history_stride) ? hrow[j] : -1;
    }
    const uint32_t * mrow = listed ? a.masks + (size_t) (a.mask_rows ? a.mask_rows[row] : row) * a.mask_stride : nullptr;
    auto allowed = [&](uint32_t f) -> bool { return !listed || ((mrow[(lo + (int) f) >> 5] >> (f & 31)) & 1u); };
    float rag_x = 0.0f;  // an element outside the whole vectors
    const int rag_f = tid < n_head ? tid : h + nv * VEC + tid - n_head;
    bool rag_ok = tid < n_rag;
    if (rag_ok) {
        rag_x = to_float(x[rag_f]);
        rag_ok = allowed((uint32_t) rag_f);
    }

    // 1. Under a mask: the bit set, then the list of segments that have an allowed id.
    auto bits_at = [&](const uint32_t * set, int v) -> uint32_t {  // a bit set's bits of vector v
        const int b = h + v * VEC;
        const uint32_t w = h == 0 ? set[b >> 5] >> (b & 31) : __funnelshift_r(set[b >> 5], set[(b >> 5) + 1], b & 31);
        return w & kVecBits;
    };
    auto vector_bits = [&](int v) -> uint32_t {  // the allowed elements of vector v (a listed v: up to the segment behind the slice)
        return listed ? bits_at(eff, v) : (v < nv ? kVecBits : 0u);
    };
    auto at_place = [](int i) -> int { return (i & ~31) | ((i & 7) << 2) | ((i >> 3) & 3); };  // a warp's four places of a cell side by side
    if (listed) {
        const int w0 = lo >> 5, n_words = ((a.vocab + 31) >> 5) - w0;  // words of the row from the slice on
        const uint32_t * mw = mrow + w0;
        const bool wide = (reinterpret_cast<uintptr_t>(mw) & 15u) == 0;
        const int v1 = h + nv * VEC;
        auto slice_bits = [&](int i) -> uint32_t {  // the bits of word i that lie in whole vectors
            const int from = max(h - 32 * i, 0), to = min(v1 - 32 * i, 32);
            return to > from ? (0xffffffffu >> (32 - to)) & (0xffffffffu << from) : 0u;
        };
        constexpr int IT = 5;
#pragma unroll 1
        for (int i0 = tid * 4; i0 < eff_words; i0 += IT * NT * 4) {
            uint4 m[IT];
#pragma unroll
            for (int q = 0; q < IT; ++q) {
                const int i = i0 + q * NT * 4;
                m[q] = make_uint4(0u, 0u, 0u, 0u);
                if (wide && i + 4 <= n_words && i < eff_words) {
                    m[q] = *reinterpret_cast<const uint4 *>(mw + i);
                } else if (i < eff_words) {
                    if (i < n_words) m[q].x = mw[i];
                    if (i + 1 < n_words) m[q].y = mw[i + 1];
                    if (i + 2 < n_words) m[q].z = mw[i + 2];
                    if (i + 3 < n_words) m[q].w = mw[i + 3];
                }
            }
#pragma unroll
            for (int q = 0; q < IT; ++q) {
                const int i = i0 + q * NT * 4;
                if (i >= eff_words) continue;
                if (32 * i < h || 32 * i + 128 > v1) {
                    m[q].x &= slice_bits(i);
                    m[q].y &= slice_bits(i + 1);
                    m[q].z &= slice_bits(i + 2);
                    m[q].w &= slice_bits(i + 3);
                }
                *reinterpret_cast<uint4 *>(eff + i) = m[q];
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int s0 = 0; s0 < n_segs; s0 += NT) {
            const int s = s0 + tid;
            uint32_t any = 0u, all = 0xffffffffu;
            if (s < n_segs) {
#pragma unroll
                for (int q = 0; q < VEC; ++q) {
                    const uint32_t w = h == 0 ? eff[s * VEC + q] : __funnelshift_r(eff[s * VEC + q], eff[s * VEC + q + 1], h);
                    any |= w;
                    all &= w;
                }
            }
            const uint32_t b = __ballot_sync(kFull, any != 0u);
            if (b == 0u) continue;
            uint32_t at = 0u;
            if (lane == 0) at = atomicAdd(&sh.n_seg, (uint32_t) __popc(b));
            at = __shfl_sync(kFull, at, 0) + (uint32_t) __popc(b & ((1u << lane) - 1u));
            if (any != 0u) seglist[at_place((int) at)] = (uint16_t) (s | ((all == 0xffffffffu && s < n_whole) ? 0x8000 : 0));
        }
    }
    __syncthreads();
    const fns_b200_params & p = rs.p;
    const int n_list = listed ? (int) sh.n_seg : n_segs;
    const int n_cells = (n_list + NV * kWarps - 1) / (NV * kWarps);

    // 2. The stream.  Place i of the list belongs to warp i % 8; a cell is four places of a warp.  Without a mask place i
    // is segment i, and all cells but the last few are whole.
    auto entry = [&](int i) -> uint32_t {  // the segment at place i (with 0x8000 when all of it is allowed)
        return listed ? (uint32_t) seglist[at_place(i)] : (uint32_t) i;
    };
    auto vector_at = [&](int v) -> const uint4 * { return reinterpret_cast<const uint4 *>(xv0 + (size_t) v * VEC); };
    const uint4 * x_lane = vector_at(lane);
    const int whole_cells = listed ? 0 : n_whole / (NV * kWarps);
    auto issue = [&](int c, uint4 (&r)[NV], uint32_t & bits) {
        uint32_t o[NV];  // the vectors, from x_lane
        if (c < whole_cells) {
            bits = kCellBits;
#pragma unroll
            for (int u = 0; u < NV; ++u) o[u] = (uint32_t) (((c * NV + u) * kWarps + warp) * 32);
        } else {
            uint32_t en[NV];
            if (listed) {
                const uint2 e = *reinterpret_cast<const uint2 *>(seglist + c * (NV * kWarps) + warp * NV);
                en[0] = e.x & 0xffffu;
                en[1] = e.x >> 16;
                en[2] = e.y & 0xffffu;
                en[3] = e.y >> 16;
            } else {
#pragma unroll
                for (int u = 0; u < NV; ++u) en[u] = (uint32_t) ((c * NV + u) * kWarps + warp);
            }
#pragma unroll
            for (int u = 0; u < NV; ++u) o[u] = (en[u] & 0x7fffu) * 32u;
            bits = kCellBits;
            if (!(en[0] & en[1] & en[2] & en[3] & 0x8000u)) {
                bits = 0u;
#pragma unroll
                for (int u = 0; u < NV; ++u) bits |= vector_bits((int) o[u] + lane) << (u * VEC);
            }
        }
#pragma unroll
        for (int u = 0; u < NV; ++u) load_if(r[u], x_lane + o[u], bits & (kVecBits << (u * VEC)));
    };
    float tmax = -INFINITY;  // this thread's maximum so far (+inf is left to the end)
    auto reduce = [&](int c, uint4 (&r)[NV], uint32_t bits) {
        float m = -INFINITY;
        if (bits) {
            if (bits != kCellBits) {  // excluded elements become NaN, which never wins (a vector not loaded holds old values)
#pragma unroll
                for (int u = 0; u < NV; ++u) exclude<T>(r[u], (bits >> (u * VEC)) & kVecBits, rs.lut);
            }
            float even = -INFINITY;
#pragma unroll
            for (int u = 0; u < NV; ++u) raw_max<T>(r[u], m, even);
            if constexpr (sizeof(T) == 2) m = fmaxf(__uint_as_float(__float_as_uint(m) & 0xffff0000u), even);
            tmax = fmaxf(tmax, m);
        }
        cmax[c * NT + tid] = (uint16_t) (__float_as_uint(m) >> 16);  // (cut towards zero: the order stays)
    };
    uint4 ra[NV], rb[NV];
    uint32_t ba = 0u, bb = 0u;
#pragma unroll
    for (int u = 0; u < NV; ++u) ra[u] = rb[u] = make_uint4(0u, 0u, 0u, 0u);
    if (n_cells > 0) issue(0, ra, ba);
    if (n_cells > 1) issue(1, rb, bb);

    // 3. History ids (and the draft prefix of a verification column) set their bits, with two cells under way.
    const int k = p.temperature <= 0.0f ? 1 : clamp_k(p.top_k, a.k_cap);
    const bool any_pen = p.repetition != 1.0f || p.presence != 0.0f || p.frequency != 0.0f;
    n_hist = n_hist < 0 ? 0 : (n_hist > (int) a.history_stride ? (int) a.history_stride : n_hist);
    const int n_pen = any_pen && a.own_cap > 0 ? n_hist + (a.draft ? col : 0) : 0;
    const bool lowering = p.repetition >= 1.0f && p.presence >= 0.0f && p.frequency >= 0.0f;  // no penalised value is above its logit
    auto pen_pos = [&](int32_t id) -> uint32_t {  // position f of a history id, ~0 if it is not in the slice
        const uint32_t f = (uint32_t) (id - a.id_base - lo);
        return id >= a.id_base && f - (uint32_t) f0 < (uint32_t) (f1 - f0) ? f : 0xffffffffu;
    };
    auto pen_id = [&](int j) -> int32_t { return j < n_hist ? hrow[j] : drow[j - n_hist]; };
#pragma unroll 1
    for (int j0 = 0; j0 < n_pen; j0 += HB * NT) {
#pragma unroll
        for (int u = 0; u < HB; ++u) {
            const int j = j0 + u * NT + tid;
            if (j0 > 0 || j >= n_hist) ids[u] = j < n_pen ? pen_id(j) : -1;
        }
        uint32_t again = 0u;  // bit u: ids[u] is in the slice, and somebody else has set its bit
#pragma unroll
        for (int u = 0; u < HB; ++u) {
            const uint32_t f = pen_pos(ids[u]);
            if (f != 0xffffffffu && ((atomicOr(&hb[f >> 5], 1u << (f & 31)) >> (f & 31)) & 1u)) again |= 1u << u;
        }
        if (p.frequency == 0.0f || !__any_sync(kFull, again != 0u)) continue;
        // (one reservation per warp: a history that repeats itself has more of these than others)
        const uint32_t mine_n = (uint32_t) __popc(again);
        uint32_t upto = mine_n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kFull, upto, o);
            if (lane >= o) upto += t;
        }
        uint32_t at = 0u;
        if (lane == 31) at = atomicAdd(&sh.n_own, upto);
        at = __shfl_sync(kFull, at, 31) + upto - mine_n;
#pragma unroll
        for (int u = 0; u < HB; ++u) {
            if (!((again >> u) & 1u)) continue;
            if (at < (uint32_t) kRowsDups) dups[at] = pen_pos(ids[u]);
            ++at;
        }
    }
    if (rank == 0 && tid == NT - 1) {  // what the draw needs (column c of a window draws with counter + c, src/engine.cu:756)
        rs.p.counter += (uint64_t) col;
        sh.u01 = philox_uniform(p.seed, p.counter);
        sh.inv_t = 1.0 / (double) p.temperature;
    }
#pragma unroll 1
    for (int c = 0; c < n_cells; c += 2) {
        reduce(c, ra, ba);
        if (c + 2 < n_cells) issue(c + 2, ra, ba);
        if (c + 1 >= n_cells) break;
        reduce(c + 1, rb, bb);
        if (c + 3 < n_cells) issue(c + 3, rb, bb);
    }
    if (__builtin_expect(!(tmax <= FLT_MAX), 0)) {
        // +inf among the allowed: never a candidate (src/kernels.cu:629-639).  This thread's cells once more, without it.
        tmax = -INFINITY;
#pragma unroll 1
        for (int c = 0; c < n_cells; ++c) {
            float m = -INFINITY;
#pragma unroll 1
            for (int u = 0; u < NV; ++u) {
                const int v = (int) (entry((c * NV + u) * kWarps + warp) & 0x7fffu) * 32 + lane;
                const uint32_t b = vector_bits(v);
                if (!b) continue;
                float xs[VEC];
                raw_values<T, VEC>(__ldg(vector_at(v)), xs);
#pragma unroll
                for (int j = 0; j < VEC; ++j)
                    if (((b >> j) & 1u) && xs[j] <= FLT_MAX) m = fmaxf(m, xs[j]);
            }
            tmax = fmaxf(tmax, m);
            cmax[c * NT + tid] = (uint16_t) (__float_as_uint(m) >> 16);
        }
    }

    // 4. The witnesses.
    const uint32_t wt = tmax > -INFINITY ? order_word(tmax) : 0u;
    if (C > 1) cluster.barrier_wait();
    {
        uint32_t w = wt;
        for (int o = 1; o < C; o <<= 1) w = max(w, __shfl_xor_sync(kFull, w, o));
        // lane j of a group of C lanes sends the group's maximum to CTA j
        cluster.map_shared_rank(wit, tid & (C - 1))[rank * (NT >> lg_c) + (tid >> lg_c)] = w;
    }
    if (C > 1) cluster.sync();
    else __syncthreads();

    auto penalised = [&](float v, float cnt) -> float {  // each step rounded on its own: no fused multiply-add
        v = v > 0.0f ? __fdiv_rn(v, p.repetition) : __fmul_rn(v, p.repetition);
        v = __fsub_rn(v, __fmul_rn(p.frequency, cnt));
        return __fsub_rn(v, p.presence);
    };
    // How often the id at position f occurs, for at most one id per thread (`live`), all different: once, and once more for
    // every entry of the list of repeats.  The ids enter a table, the block walks the list (the whole history when it holds
    // more repeats than the list) and counts.  Every thread calls it in the same round.
    auto occurrences = [&](bool live, uint32_t f) -> float {
        const uint32_t n_dup = sh.n_own;
        if (n_dup == 0u || !__syncthreads_or(live)) return 1.0f;
        const bool short_list = n_dup <= (uint32_t) kRowsDups;
        uint32_t slot = 0u;
        if (live) {
            slot = (f * 2654435761u) >> kTShift;
            while (atomicCAS(&tkey[slot], kNoKey, f) != kNoKey) slot = (slot + 1u) & (TS - 1);
            tcnt[slot] = short_list ? 1u : 0u;
        }
        __syncthreads();
        auto count = [&](uint32_t o) {
            if (o == 0xffffffffu) return;
            uint32_t q = (o * 2654435761u) >> kTShift;
            for (uint32_t kx = tkey[q]; kx != kNoKey; kx = tkey[q]) {  // at most NT keys in 2 NT slots
                if (kx == o) {
                    atomicAdd(&tcnt[q], 1u);
                    break;
                }
                q = (q + 1u) & (TS - 1);
            }
        };
        const int n_walk = short_list ? (int) n_dup : n_pen;
#pragma unroll 1
        for (int t0 = tid; t0 < n_walk; t0 += 4 * NT) {  // (the ids of a round are requested together)
            uint32_t o[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int t = t0 + u * NT;
                o[u] = t >= n_walk ? 0xffffffffu : (short_list ? dups[t] : pen_pos(pen_id(t)));
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) count(o[u]);
        }
        __syncthreads();
        float n = 1.0f;
        if (live) n = (float) tcnt[slot];
        __syncthreads();
        if (live) tkey[slot] = kNoKey;
        return n;
    };
    auto is_hist = [&](uint32_t f) -> bool { return (hb[f >> 5] >> (f & 31)) & 1u; };

    // What a thread's cells without a history id say for certain: the largest of their maxima, or what the heaviest penalty of
    // the row leaves of the largest of its other cells (penalties that only lower keep the order, so whatever held that
    // maximum does not end below it) - from the cells' 16-bit maxima, cut the other way where they are negative.  About
    // 3 us of a block, which is why only a row takes it whose history shows among the best.
    auto clean_witness = [&]() -> uint32_t {
        uint32_t * mark = vlist;                                 // [2 NT] bit c: cell c of the thread holds a history id
        uint16_t * seg_at = reinterpret_cast<uint16_t *>(lbuf);  // the places of the listed segments
        static_assert(kWarps * kWarpList >= 2 * NT && kRowsBuf * 4 >= kRowsMaxCells * NV * kWarps, "room for the marks");
        __syncthreads();
        mark[tid] = mark[NT + tid] = 0u;
        if (listed)
            for (int i = tid; i < n_list; i += NT) seg_at[entry(i) & 0x7fffu] = (uint16_t) i;
        __syncthreads();
#pragma unroll 4
        for (int j = tid; j < n_pen; j += NT) {
            const uint32_t f = pen_pos(pen_id(j));
            const int e = (int) f - h;  // the element's number in the whole vectors
            if (f == 0xffffffffu || e < 0 || e >= nv * VEC || (listed && !((eff[f >> 5] >> (f & 31)) & 1u))) continue;
            const int seg = e / (32 * VEC), at = listed ? (int) seg_at[seg] : seg;  // (an allowed id: its segment is on the list)
            const int c = at / (NV * kWarps);
            atomicOr(&mark[(c >> 5) * NT + (at % kWarps) * 32 + (e / VEC) % 32], 1u << (c & 31));
        }
        __syncthreads();
        const uint32_t q_lo = mark[tid], q_hi = mark[NT + tid];
        float clean = -INFINITY, other = -INFINITY;
#pragma unroll 2
        for (int c = 0; c < n_cells; ++c) {
            const float m = __uint_as_float((uint32_t) cmax[c * NT + tid] << 16);
            if (((c < 32 ? q_lo >> c : q_hi >> (c - 32)) & 1u) == 0u) clean = fmaxf(clean, m);
            else other = fmaxf(other, m);
        }
        auto down = [](float m) -> float { return __uint_as_float(__float_as_uint(m) | ((int) __float_as_uint(m) < 0 ? 0xffffu : 0u)); };
        float w = clean > other ? tmax : down(clean);  // (NaN for -inf: never wins)
        if (!(clean > other) && lowering) w = fmaxf(w, penalised(down(other), p.frequency != 0.0f ? (float) (1u + sh.n_own) : 1.0f));
        __syncthreads();  // (mark and lbuf are used again)
        return w >= -FLT_MAX ? order_word(w) : 0u;
    };
    int n_wit = NT;  // witnesses of groups, or (C * NT) of threads
    auto send_all = [&](uint32_t w) {  // a thread's witness to every CTA
        if (C > 1) cluster.sync();     // (every CTA has read the ones before)
        else __syncthreads();
        for (int r = 0; r < C; ++r) cluster.map_shared_rank(wit, r)[rank * NT + tid] = w;
        n_wit = C * NT;
        if (C > 1) cluster.sync();
        else __syncthreads();
    };
    // More history ids than six for ten cells leave few cells without one: a lower bound is tried first.
    bool crowded = 5ll * n_pen * (VEC * NV) > 3ll * a.vocab;
    bool sure = n_pen == 0;
    // From here on once, and again with a lower bound if history ids took too many candidates away.
    int witnesses = n_pen > 0 ? min(k + (k >> 2) + 8, 256) : k;  // how many must reach the bound
    float thr_v;
    uint64_t thr_key;
    uint64_t * keys;
    int n_all;
    const int region = kRowsGather >> lg_c;  // what a CTA may send to CTA 0 (k_cap at least)
    for (;;) {
        // 5. The bound.  (Too few groups saw anything, as under a mask that leaves little: every thread speaks for itself.)
        int reach;
        uint32_t bound = block_reach<NT>([&](int i) { return wit[i]; }, n_wit, witnesses, 4, sh.sc, sh.ends, &reach);
        if (C > 1 && bound == 0u && n_wit == NT) {
            send_all(wt);
            bound = block_reach<NT>([&](int i) { return wit[i]; }, n_wit, min(witnesses, k), 4, sh.sc, sh.ends, &reach);
        }
        const bool bounded = bound != 0u;
        thr_v = bounded ? word_value(bound) + 0.0f : -FLT_MAX;  // (-0.0 -> +0.0: one key pattern for both)
        thr_key = (uint64_t) order_word(thr_v) << 32;

        // 6. The candidates.  A history id that reaches the bound: its key, if its penalties are known here; 0 if they take
        // it below the bound, or if its occurrences have to be counted first (then it goes on the list).
        auto history_key = [&](float raw, uint32_t f) -> uint64_t {
            if (!lowering) return 0ull;  // (all history ids are looked at below)
            const float v = penalised(raw, 1.0f);
            if (!(v >= thr_v && is_finite(v))) return 0ull;
            if (p.frequency == 0.0f) return make_key(v, id0 + f);
            const uint32_t at = atomicAdd(&rs.n_hl, 1u);
            if (at < (uint32_t) NT) {
                rs.hl_pos[at] = f;
                rs.hl_raw[at] = raw;
            }
            return 0ull;
        };
        auto offer = [&](uint64_t key) {  // every lane of the warp calls it; 0 = nothing to offer
            const bool has = key != 0ull && key >= thr_key;
            const uint32_t b = __ballot_sync(kFull, has);
            if (b == 0u) return;
            uint32_t at = 0u;
            if (lane == 0) at = atomicAdd(&sh.n_cand, (uint32_t) __popc(b));
            at = __shfl_sync(kFull, at, 0) + (uint32_t) __popc(b & ((1u << lane) - 1u));
            if (has && at < (uint32_t) kRowsBuf) lbuf[at] = key;
        };
        // Every warp reads the cells of its own threads again: no block barrier between the list and the reads.
        uint32_t n_vl;  // cells of this warp that reach the bound
        uint32_t * wlist = vlist + warp * kWarpList;
        {
            const float cut = __uint_as_float(__float_as_uint(thr_v) & 0xffff0000u);
            uint32_t q_lo = 0u, q_hi = 0u;  // bit c: this thread's cell c reaches the bound
            if (tmax >= thr_v) {
#pragma unroll 1
                for (int c0 = 0; c0 < n_cells; c0 += 8) {
                    uint32_t q = 0u;
#pragma unroll
                    for (int u = 0; u < 8; ++u) q |= c0 + u < n_cells && __uint_as_float((uint32_t) cmax[(c0 + u) * NT + tid] << 16) >= cut ? 1u << u : 0u;
                    if (c0 < 32) q_lo |= q << c0;
                    else q_hi |= q << (c0 - 32);
                }
            }
            const uint32_t mine_n = (uint32_t) (__popc(q_lo) + __popc(q_hi));
            uint32_t upto = mine_n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t t = __shfl_up_sync(kFull, upto, o);
                if (lane >= o) upto += t;
            }
            n_vl = __shfl_sync(kFull, upto, 31);
            uint32_t at = upto - mine_n;
            while (q_lo | q_hi) {
                const int c = q_lo ? __ffs(q_lo) - 1 : 31 + __ffs(q_hi);
                if (q_lo) q_lo &= q_lo - 1u;
                else q_hi &= q_hi - 1u;
                if (at < (uint32_t) kWarpList) wlist[at] = (uint32_t) (c << 5 | lane);
                ++at;
            }
            __syncwarp();
        }
        if (n_rag > 0 && warp == 0) {
            uint64_t key = 0ull;
            if (rag_ok && rag_x >= thr_v && rag_x <= FLT_MAX)
                key = n_pen > 0 && is_hist((uint32_t) rag_f) ? history_key(rag_x, (uint32_t) rag_f) : make_key(rag_x, id0 + (uint32_t) rag_f);
            offer(key);
        }
        if (n_vl > (uint32_t) kWarpList) {
            if (lane == 0) sh.n_vl = 1u;  // too many: everything is offered again below
        } else {
            const int total = (int) n_vl * NV;
            constexpr int PB = 4;  // vectors per lane in flight together
#pragma unroll 1
            for (int i0 = 0; i0 < total; i0 += PB * 32) {  // (the same rounds for every lane of a warp)
                uint4 r[PB];
                uint32_t bits[PB];
                int v[PB];
#pragma unroll
                for (int q = 0; q < PB; ++q) {
                    const int i = i0 + q * 32 + lane;
                    bits[q] = 0u;
                    v[q] = 0;
                    r[q] = make_uint4(0u, 0u, 0u, 0u);
                    if (i < total) {
                        const uint32_t cell = wlist[i / NV];
                        v[q] = (int) (entry(((int) (cell >> 5) * NV + i % NV) * kWarps + warp) & 0x7fffu) * 32 + (int) (cell & 31u);
                        bits[q] = vector_bits(v[q]);
                    }
                    load_if(r[q], vector_at(v[q]), bits[q]);
                }
#pragma unroll
                for (int q = 0; q < PB; ++q) {
                    float xs[VEC];
                    raw_values<T, VEC>(r[q], xs);
                    uint32_t hit = 0u;
#pragma unroll
                    for (int j = 0; j < VEC; ++j) hit |= (((bits[q] >> j) & 1u) && xs[j] >= thr_v && xs[j] <= FLT_MAX) ? 1u << j : 0u;
                    if (!__any_sync(kFull, hit != 0u)) continue;
                    const uint32_t pen = n_pen > 0 && hit ? hit & bits_at(hb, v[q]) : 0u;
                    hit &= ~pen;
                    const uint32_t mine_n = (uint32_t) __popc(hit);
                    uint32_t upto = mine_n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t t = __shfl_up_sync(kFull, upto, o);
                        if (lane >= o) upto += t;
                    }
                    uint32_t at = 0u;
                    if (lane == 31) at = atomicAdd(&sh.n_cand, upto);
                    at = __shfl_sync(kFull, at, 31) + upto - mine_n;
#pragma unroll
                    for (int j = 0; j < VEC; ++j) {
                        if (!((hit >> j) & 1u)) continue;
                        if (at < (uint32_t) kRowsBuf) lbuf[at] = make_key(xs[j], id0 + (uint32_t) (h + v[q] * VEC + j));
                        ++at;
                    }
                    if (!__any_sync(kFull, pen != 0u)) continue;
#pragma unroll 1
                    for (int j = 0; j < VEC; ++j) {
                        float xj = xs[0];
#pragma unroll
                        for (int e = 1; e < VEC; ++e) xj = e == j ? xs[e] : xj;
                        offer(((pen >> j) & 1u) ? history_key(xj, (uint32_t) (h + v[q] * VEC + j)) : 0ull);
                    }
                }
            }
        }
        __syncthreads();
        // The history ids that are on the list, whose occurrences are counted now.
        auto listed_history_ids = [&](uint32_t n_hl) {
            const bool live = (uint32_t) tid < n_hl;
            const uint32_t f = live ? rs.hl_pos[tid] : 0u;
            const float cnt = occurrences(live, f), v = live ? penalised(rs.hl_raw[tid], cnt) : -INFINITY;
            offer(v >= thr_v && is_finite(v) ? make_key(v, id0 + f) : 0ull);
            __syncthreads();
        };
        // Every history id, once each (penalties that can raise a value, or more of them than the list holds).
        auto every_history_id = [&]() {  // (the thread that takes an id's bit away owns it)
#pragma unroll 1
            for (int j0 = 0; j0 < n_pen; j0 += NT) {
                const uint32_t f = j0 + tid < n_pen ? pen_pos(pen_id(j0 + tid)) : 0xffffffffu;
                bool live = f != 0xffffffffu && allowed(f);
                if (live) live = (atomicAnd(&hb[f >> 5], ~(1u << (f & 31))) >> (f & 31)) & 1u;
                const float raw = live ? to_float(x[f]) : 0.0f;
                if (lowering) live = live && penalised(raw, 1.0f) >= thr_v;
                const float cnt = p.frequency != 0.0f ? occurrences(live, f) : 1.0f;
                const float v = live ? penalised(raw, cnt) : -INFINITY;
                offer(v >= thr_v && is_finite(v) ? make_key(v, id0 + f) : 0ull);
            }
            __syncthreads();
#pragma unroll 1
            for (int j = tid; j < n_pen; j += NT) {  // (the bits back: this may not have been the last time)
                const uint32_t f = pen_pos(pen_id(j));
                if (f != 0xffffffffu) atomicOr(&hb[f >> 5], 1u << (f & 31));
            }
            __syncthreads();
        };
        if (n_pen > 0) {
            if (lowering) {
                const uint32_t n_hl = rs.n_hl;
                // (too few even if all of them stay: their occurrences can wait for the next bound)
                const bool enough = C > 1 || sure || !bounded || (int) (sh.n_cand + n_hl) >= k;
                if (n_hl > 0u && n_hl <= (uint32_t) NT && enough) listed_history_ids(n_hl);  // uniform
            } else {
                every_history_id();
            }
        }
        int n_loc = (int) sh.n_cand;
        keys = lbuf;
        if (__builtin_expect(n_loc > kRowsBuf || sh.n_vl != 0u || rs.n_hl > (uint32_t) NT, 0)) {  // uniform in the CTA
            // More than the lists or the buffer hold.  The k-th best of a full buffer is a bound that k candidates reach: with it
            // everything is offered again, a cell per thread and round, until it fits.  It is a whole key, so that equal values
            // are cut by their ids, and every time it rises past all but k of the buffer.  (An element per thread between block
            // votes, as k_cluster does it, took 0.4 to 1.7 ms for a batch of rows whose best ids are in the history.)
            for (;;) {
                __syncthreads();
                if (n_loc > kRowsBuf) {
                    thr_key = block_kth_key<NT>(lbuf, kRowsBuf, k, sh.sc);
                    thr_v = key_floor_value(thr_key);
                }
                if (tid == 0) {
                    sh.n_cand = 0u;
                    rs.n_hl = 0u;
                }
                __syncthreads();
                const float cut = __uint_as_float(__float_as_uint(thr_v) & 0xffff0000u);
#pragma unroll 1
                for (int c = -1; c < n_cells; ++c) {  // (-1: the elements outside whole vectors)
                    const bool take = c < 0 ? rag_ok : tmax >= thr_v && __uint_as_float((uint32_t) cmax[c * NT + tid] << 16) >= cut;
                    const bool full = __shfl_sync(kFull, *(volatile uint32_t *) &sh.n_cand, 0) > (uint32_t) kRowsBuf;
                    if (full || !__any_sync(kFull, take)) continue;
                    uint4 r[NV];
                    uint32_t bits[NV];
#pragma unroll
                    for (int u = 0; u < NV; ++u) {
                        const int v = c < 0 ? 0 : (int) (entry((c * NV + u) * kWarps + warp) & 0x7fffu) * 32 + lane;
                        bits[u] = take && c >= 0 ? vector_bits(v) : 0u;
                        r[u] = make_uint4(0u, 0u, 0u, 0u);
                        load_if(r[u], vector_at(v), bits[u]);
                    }
#pragma unroll 1
                    for (int u = 0; u < NV; ++u) {
                        float xs[VEC];
                        raw_values<T, VEC>(u == 0 ? r[0] : (u == 1 ? r[1] : (u == 2 ? r[2] : r[3])), xs);
                        const uint32_t b = u == 0 ? bits[0] : (u == 1 ? bits[1] : (u == 2 ? bits[2] : bits[3]));
                        const int f_v = c < 0 ? 0 : h + ((int) (entry((c * NV + u) * kWarps + warp) & 0x7fffu) * 32 + lane) * VEC;
#pragma unroll 1
                        for (int j = 0; j < VEC; ++j) {
                            float raw = xs[0];
#pragma unroll
                            for (int e = 1; e < VEC; ++e) raw = e == j ? xs[e] : raw;
                            bool ok = (b >> j) & 1u;
                            uint32_t f = (uint32_t) (f_v + j);
                            if (c < 0 && u == 0 && j == 0) {
                                ok = take;
                                raw = rag_x;
                                f = (uint32_t) rag_f;
                            }
                            ok = ok && raw >= thr_v && raw <= FLT_MAX;
                            if (!__any_sync(kFull, ok)) continue;
                            offer(!ok ? 0ull : (n_pen > 0 && is_hist(f) ? history_key(raw, f) : make_key(raw, id0 + f)));
                        }
                    }
                }
                __syncthreads();
                if (n_pen > 0) {
                    const uint32_t n_hl = rs.n_hl;  // uniform
                    if (!lowering || n_hl > (uint32_t) NT) {
                        every_history_id();
                    } else if (n_hl > 0u) {
                        listed_history_ids(n_hl);
                    }
                }
                n_loc = (int) sh.n_cand;
                if (n_loc <= kRowsBuf) break;  // uniform in the CTA
            }
        }
        if (C > 1 && n_loc > region) keys = best_keys<NT>(lbuf, &n_loc, k, a.k_cap - k, sorted, a.k_cap, sel, sh);  // only this CTA's best k can matter
        n_all = n_loc;
        if (C > 1) {
            if (tid < C) cluster.map_shared_rank(&rs, tid)->count[rank] = (uint32_t) n_loc;
            uint64_t * to = cluster.map_shared_rank(gbuf, 0) + rank * region;
            for (int i = tid; i < n_loc; i += NT) to[i] = keys[i];
            cluster.sync();
            n_all = 0;
            for (int q = 0; q < C; ++q) n_all += (int) rs.count[q];
        }
        if (sure || n_all >= k || !bounded) break;  // (the same in every CTA of the cluster)
        // History ids took too many away: once more with a bound that they have no part in, or with a lower one.
        send_all(crowded ? wt : clean_witness());
        sure = !crowded;
        witnesses = crowded ? 2 * witnesses : k;  // (more than there are: no bound at all)
        crowded = false;
        if (tid == 0) {
            sh.n_cand = 0u;
            sh.n_vl = 0u;
            rs.n_hl = 0u;
        }
        __syncthreads();
    }
    if (C > 1) {
        if (rank != 0) return;  // (nobody reads another CTA's memory from here on)
        const int r = tid >> (8 - lg_c);  // 256 / C threads per region
        int before = 0;
        for (int q = 0; q < r; ++q) before += (int) rs.count[q];
        const int n_r = (int) rs.count[r];
        for (int i = tid & ((NT >> lg_c) - 1); i < n_r; i += NT >> lg_c) lbuf[before + i] = gbuf[r * region + i];
        __syncthreads();
        keys = lbuf;
    }
    keys = cut_keys<NT>(keys, &n_all, k, gbuf, sel, sh);
    rank_draw<NT>(keys, n_all, k, sorted, pj, acc, reinterpret_cast<double *>(sel), sh.sc, p, sh.u01, sh.inv_t, a.k_cap,
                  a.out_tokens ? a.out_tokens + row : nullptr, a.out_cands ? a.out_cands + (size_t) row * a.k_cap : nullptr);
}

}  // namespace fnsb
