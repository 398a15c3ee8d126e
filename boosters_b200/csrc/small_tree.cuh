// small_tree.cuh — a whole depth-wise tree in one cooperative launch, for
// training sets whose level kernels are bound by launch and hand-off latency
// (included by kernels.cu: it shares the split search, the leaf solve and the
// partition rule of the level kernels, and grows the same trees bit for bit).
//
// One block per SM. A block owns whole columns: it accumulates a column's
// histograms of a level's smaller children over all rows in shared memory,
// so there are no partial histograms and no merge; the larger children come
// from the parents' histograms (exact integers), and the block searches its
// column's splits at once. Rows are not moved: a 16-bit tree-node id per row
// says where a row is, updated by the block that owns the row's slice. Two
// grid barriers per level: after the splits are known (rows move, children are
// counted) and after the rows moved (histograms, split search).
//
// What bounds it: at 5,000 x 100 the chain of barriers and phases, at 50,000
// rows the row loop: two or four shared atomics per row and column (about 1
// cycle per warp each when the 32 lanes hit 32 banks, 2.5 on 256 random
// words, measured), a node id and a bin of every row and the gradients of the
// rows that count from L2.
// Counters are kept in K copies, lane l adding to copy l mod K, as many as
// fit and as the rows of the level pay for: low-cardinality columns would
// otherwise serialise on a few words.

constexpr int ST_THREADS = 512;
constexpr int ST_WARPS = ST_THREADS / 32;
constexpr uint32_t ST_FRONT = 1u << SMALL_TREE_DEPTH;  // frontier nodes of the deepest level
constexpr uint32_t ST_NODES = 2 * ST_FRONT;            // tree nodes
constexpr uint32_t ST_DYN = 188u * 1024u;              // dynamic shared memory of a block
constexpr int ST_SORT_WARPS = 8;                       // warps that search categorical columns
constexpr uint32_t ST_SORT_BYTES = ST_SORT_WARPS * SORT_N * 12u;  // their sort scratch
constexpr uint32_t ST_POLLS = 1u << 24;  // a barrier gives up after this many polls (seconds)
constexpr uint32_t ST_NONE = 0xFFFFu;

// 32-bit words of a counter: one each for grad and hess while every sum of
// the quantised values fits 31 bits, else two each with an explicit carry (a
// 64-bit shared atomic costs as much as eleven 32-bit ones).
__host__ __device__ constexpr uint32_t st_words(bool wide) { return wide ? 4u : 2u; }
// Shared bytes per histogram bin: the counters (one copy) and the sums.
__host__ __device__ constexpr uint32_t st_bin_bytes(bool wide) { return 2u * st_words(wide) * 4u; }

// ... and per expansion for each 32 bins: sums before them, scores, work list.
__host__ __device__ constexpr uint32_t st_chunk_bytes(bool wide, uint32_t nq) {
    return (nq + 1u) * (wide ? 16u : 8u) + nq * 16u + 16u;
}

__device__ __forceinline__ uint32_t st_level(uint32_t d) { return (1u << d) - 1u; }  // level d's first entry

// All blocks of the launch (co-resident: cooperative launch) wait for each
// other; false after a bounded wait (err set: every block leaves).
__device__ bool st_barrier(uint32_t* bar, uint32_t target, uint32_t* err) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        uint32_t v = 0;
        bool ok = false;
        for (uint32_t it = 0; it < ST_POLLS && !ok; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            ok = v >= target;
        }
        if (!ok) atomicExch(err, 1u);
        s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return s_ok != 0;
}

// q added to the 64-bit sum split over lo[i] / hi[i].
__device__ __forceinline__ void st_add64(uint32_t* lo, uint32_t* hi, uint32_t i, long long q) {
    const uint32_t l = (uint32_t)q;
    const uint32_t old = atomicAdd(&lo[i], l);
    atomicAdd(&hi[i], (uint32_t)((unsigned long long)q >> 32) + (old + l < l ? 1u : 0u));
}

// Row gradients as the row loop reads them.
template <int MODE>
struct StRows : GradLoad<MODE> {  // quantised pairs, one register each
    __device__ explicit StRows(const SmallTree& a) : GradLoad<MODE>(a.gr) {}
};
template <>
struct StRows<GRAD_F32> {  // fixed-point pairs (converted once per tree)
    const longlong2* __restrict__ fix;
    using Raw = longlong2;
    __device__ explicit StRows(const SmallTree& a) : fix(a.fix) {}
    __device__ __forceinline__ Raw raw(uint32_t row) const { return fix[row]; }
    __device__ __forceinline__ void conv(Raw v, long long& g, long long& h) const {
        g = v.x;
        h = v.y;
    }
};

template <bool WIDE>
struct StAcc {
    using T = long long;
    using T2 = longlong2;
    static __device__ __forceinline__ T2 make(long long g, long long h) { return make_longlong2(g, h); }
};
template <>
struct StAcc<false> {
    using T = int;
    using T2 = int2;
    static __device__ __forceinline__ T2 make(long long g, long long h) { return make_int2((int)g, (int)h); }
};

// Best candidates of a numeric column are compared by (gain, scan order); a
// candidate's order tells its bin and direction, so one 64-bit maximum in
// shared memory reduces the warps that search a node. 0: no candidate.
__device__ __forceinline__ unsigned long long st_key(float g, uint32_t order) {
    if (g == 0.0f) g = 0.0f;
    uint32_t u = __float_as_uint(g);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((unsigned long long)u << 32) | (uint32_t)~order;
}

// One lane's candidates at bin b of a node (find.rs:286-407, as scan_column):
// P: the bins' sums up to b, T: the node's totals, M: the totals without the
// last (missing) bin.
template <typename T2>
__device__ __forceinline__ unsigned long long st_candidates(T2 P, T2 T, T2 M, uint32_t b, uint32_t nb, bool hm,
                                                            uint32_t pc, double ig, double ih, const GainCtx& ctx) {
    unsigned long long best = 0ull;
    if (b + 1 < nb) {  // forward candidate: bins <= b go left
        const double lg = (double)P.x * ig, lh = (double)P.y * ih;
        const double rg = (double)((long long)T.x - P.x) * ig, rh = (double)((long long)T.y - P.y) * ih;
        const uint32_t lc = b + 1, rc = sat_sub(pc, lc);
        if (ctx.valid(lh, rh, lc, rc)) {
            const float g = ctx.gain(lg, lh, rg, rh);
            if (g > -INFINITY) best = st_key(g, b);
        }
    }
    if (hm && b + 2 < nb) {  // backward candidate: bins b+1..nb-2 go right
        const long long Rg = (long long)M.x - P.x, Rh = (long long)M.y - P.y;
        const double rg = (double)Rg * ig, rh = (double)Rh * ih;
        const double lg = (double)((long long)T.x - Rg) * ig, lh = (double)((long long)T.y - Rh) * ih;
        const uint32_t rc = nb - 2 - b, lc = sat_sub(pc, rc);
        if (ctx.valid(lh, rh, lc, rc)) {
            const float g = ctx.gain(lg, lh, rg, rh);
            if (g > -INFINITY) best = max(best, st_key(g, 2 * nb - 3 - b));
        }
    }
    return best;
}

struct StShared {  // the level's facts, the same in every block
    PartWork work[ST_FRONT / 2];     // expansions: split rule (begin / count unused)
    uint16_t tl[ST_FRONT / 2], tr[ST_FRONT / 2];  // tree nodes of the training-left / right child
    uint16_t front[ST_FRONT / 2];    // the expansion's index in its frontier
    uint8_t small_left[ST_FRONT / 2];
    uint16_t f_tnode[ST_FRONT];      // frontier: tree nodes
    uint32_t f_cnt[ST_FRONT];        // rows (sampled rows) for the split search
    uint16_t map[ST_NODES];          // tree node -> expansion, or the expansion whose smaller child it is
    uint8_t split[ST_NODES];
    uint32_t cnt[ST_FRONT], scnt[ST_FRONT];  // this block's child counts
    unsigned long long best[ST_FRONT];       // best candidate of a column per node
    uint32_t sh[33];
    uint32_t first_col, n_list;
    longlong2 ptot[ST_FRONT / 2];    // the expansions' totals
    HessMin hmin;
    float lam;                       // lambda in units of the hessian sums
    ScanColumn col;   // of column blockIdx.x
    BColumn bcol;
    double scale[4];  // units of the histogram sums
    unsigned long long small_rows;
};

// Categorical columns: a warp per expansion writes both children's bins and
// searches them from memory (its own writes).
template <int MODE, bool WIDE>
__device__ void st_categories(const SmallTree& a, StShared& s, unsigned char* dyn, uint32_t c, const ScanColumn& cm,
                              uint32_t j0, uint32_t mm, uint32_t level, uint32_t slots, uint32_t parents, bool root,
                              bool searched, const typename StAcc<WIDE>::T2* sum) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, B = cm.n_bins;
    if (warp >= ST_SORT_WARPS) return;
    double* key = reinterpret_cast<double*>(dyn) + warp * SORT_N;
    uint32_t* cat = reinterpret_cast<uint32_t*>(dyn + ST_SORT_WARPS * SORT_N * 8u) + warp * SORT_N;
    HBin* hist = a.hist + cm.hist_off;
    for (uint32_t j = warp; j < mm; j += ST_SORT_WARPS) {
        const uint32_t n0 = root ? 0u : 2u * (j0 + j), kids = root ? 1u : 2u;
        const bool sl = root || s.small_left[j0 + j] != 0;
        HBin* o = hist + (size_t)(slots + n0) * a.slot_bins;
        const HBin* ph = hist + (size_t)(parents + (root ? 0u : s.front[j0 + j])) * a.slot_bins;
        for (uint32_t b = lane; b < B; b += 32u) {
            const longlong2 v = make_longlong2(sum[j * B + b].x, sum[j * B + b].y);
            if (root) {
                *reinterpret_cast<longlong2*>(o + b) = v;
                continue;
            }
            const longlong2 p = __ldcg(reinterpret_cast<const longlong2*>(ph + b));
            const longlong2 w = make_longlong2(p.x - v.x, p.y - v.y);
            *reinterpret_cast<longlong2*>(o + b) = sl ? v : w;
            *reinterpret_cast<longlong2*>(o + a.slot_bins + b) = sl ? w : v;
        }
        __threadfence_block();
        __syncwarp();
        for (uint32_t q = 0; q < kids; ++q) {
            const uint32_t node = n0 + q;
            const HBin* hp = o + (size_t)q * a.slot_bins;
            const ScanNode nd{0u, s.f_cnt[node], 0u, 0u, 0, 0};
            long long tot[2];
            const float g = scan_column<HBin>(
                [hp](uint32_t b) {
                    const longlong2 v = __ldcg(reinterpret_cast<const longlong2*>(hp + b));
                    return HBin{v.x, v.y};
                },
                nd, cm, s.scale, a.gp, a.cand + (size_t)node * a.n_cols + c, tot, key, cat, !searched);
            if (lane == 0) {
                if (c == s.first_col) {
                    a.tot[2 * (st_level(level) + node)] = tot[0];
                    a.tot[2 * (st_level(level) + node) + 1] = tot[1];
                }
                if (g > -INFINITY) atomicMax(&a.keys[st_level(level) + node], cand_key(g, c, a.last_wins));
            }
            __syncwarp();  // key / cat are reused
        }
    }
}

// Histograms and split search of a level (root: the root alone) for the
// columns of this block. m: expansions whose smaller children are built;
// level: the children's level; store: their histograms are needed later.
template <int MODE, bool WIDE>
__device__ void st_histograms(const SmallTree& a, StShared& s, unsigned char* dyn, const StRows<MODE>& load, uint32_t m,
                              uint32_t level, bool root, bool store) {
    using SA = StAcc<WIDE>;
    using Acc = typename SA::T;
    using T2 = typename SA::T2;
    constexpr uint32_t NW = st_words(WIDE);
    // histogram slots: the levels alternate between two halves. A numeric
    // column's slot holds the prefix sums of its bins (larger = parent -
    // smaller holds for them too), a categorical one's the bins' sums.
    const uint32_t slots = (level & 1u) << (a.max_depth - 1u), parents = slots ^ (1u << (a.max_depth - 1u));
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    unsigned char* base = dyn + (a.has_cat ? ST_SORT_BYTES : 0u);
    const uint32_t room = ST_DYN - (a.has_cat ? ST_SORT_BYTES : 0u) - 64u;
    const double ig = s.scale[2], ih = s.scale[3];
    const uint8_t* mask = a.colmask ? a.colmask + (size_t)level * a.n_cols : nullptr;
    // the node totals come from the first column that is searched
    if (mask) {
        if (tid == 0) s.first_col = 0xFFFFFFFFu;
        __syncthreads();
        for (uint32_t c = tid; c < a.n_cols; c += ST_THREADS)
            if (mask[c]) atomicMin(&s.first_col, c);
        __syncthreads();
    }
    for (uint32_t c = blockIdx.x; c < a.n_cols; c += gridDim.x) {
        bool searched = true;
        if (mask) {
            searched = mask[c] != 0;
            bool later = searched;
            for (uint32_t l = level + 1; l < a.max_depth && !later; ++l) later = a.colmask[(size_t)l * a.n_cols + c] != 0;
            if (!later) continue;  // no level from here on searches it
        }
        const bool own = c == blockIdx.x;  // the block's first (often only) column: its facts are at hand
        const ScanColumn cm = own ? s.col : a.cols[c];
        const BColumn bc = own ? s.bcol : a.bcols[c];
        const uint32_t B = cm.n_bins, nq = (B + 31u) / 32u;
        const bool hm = cm.has_missing != 0;
        const uint8_t* col8 = a.fm8 + (size_t)bc.pos * a.n;
        const uint16_t* col16 = a.fm16 + (size_t)bc.pos * a.n;
        const bool u8 = bc.matrix == 0;
        HBin* hist = a.hist + cm.hist_off;
        const uint32_t per_exp = st_bin_bytes(WIDE) * B + st_chunk_bytes(WIDE, nq);
        const uint32_t per_pass = max(1u, min(m, room / per_exp));
        for (uint32_t j0 = 0; j0 < m; j0 += per_pass) {
            const uint32_t mm = min(per_pass, m - j0), cells = mm * B;
            // copies of the counters: a power of two up to 32 that fits, while
            // zeroing and folding them stays below the rows' own work
            uint32_t lk = 0;
            const uint32_t fixed = (uint32_t)sizeof(T2) * cells + mm * st_chunk_bytes(WIDE, nq) + 16u * NW;
            while (lk < 5u && NW * 4u * (cells << (lk + 1)) + fixed <= room && (cells << (lk + 1)) <= max(cells, a.n / 2u)) ++lk;
            const uint32_t plane = ((cells << lk) + 3u) & ~3u;
            T2* sum = reinterpret_cast<T2*>(base);              // [mm][B] the smaller children's bins
            T2* carry = sum + cells;                            // [mm][nq + 1] sums before each 32 bins; totals
            float* score = reinterpret_cast<float*>(carry + mm * (nq + 1u));     // [mm][nq][2] best scores
            uint32_t* list = reinterpret_cast<uint32_t*>(score + 2u * mm * nq);  // [mm * nq * 2] chunks to search
            uint32_t* acc = reinterpret_cast<uint32_t*>(
                base + ((((size_t)cells + mm * (nq + 1u)) * sizeof(T2) + 16u * mm * nq + 15u) & ~(size_t)15u));
            const uint32_t copy = lane & ((1u << lk) - 1u);
            // Rows in steps of V per thread, three steps in flight: the
            // node ids of step k + 2 are loaded while the bins and gradients
            // of step k + 1 (where a row counts) are, and step k is added. A
            // warp's lanes take consecutive rows.
            using Raw = typename StRows<MODE>::Raw;
            constexpr uint32_t V = MODE == GRAD_F32 ? 4u : 8u, STEP = ST_THREADS * V;
            uint32_t t2[V], j1[V], jc[V], b1[V], bc_[V];
            Raw q1[V], qc[V];
            auto ids = [&](uint32_t i0) {
#pragma unroll
                for (uint32_t u = 0; u < V; ++u) {
                    const uint32_t i = i0 + u * ST_THREADS;
                    t2[u] = ST_NONE;
                    if (i < a.n) t2[u] = root ? 0u : (uint32_t)__ldcg(a.rt + i);
                }
            };
            auto fetch = [&](uint32_t i0) {  // t2 -> j1, b1, q1
#pragma unroll
                for (uint32_t u = 0; u < V; ++u) {
                    uint32_t j = t2[u];
                    if (!root && j != ST_NONE) j = BST_IN(j, ST_NODES, CHECK_SMALL_NODE) ? s.map[j] : ST_NONE;
                    j1[u] = j - j0;  // rows of other passes and ST_NONE: past mm
                }
#pragma unroll
                for (uint32_t u = 0; u < V; ++u) {
                    const uint32_t i = i0 + u * ST_THREADS;
                    if (j1[u] < mm) {
                        b1[u] = u8 ? (uint32_t)col8[i] : (uint32_t)col16[i];
                        q1[u] = load.raw(i);
                    }
                }
            };
            ids(tid);
            for (uint32_t i = tid; i < plane * NW / 4u; i += ST_THREADS)
                reinterpret_cast<uint4*>(acc)[i] = make_uint4(0, 0, 0, 0);
            fetch(tid);
            ids(tid + STEP);
            __syncthreads();
            for (uint32_t i = tid; i < a.n; i += STEP) {
#pragma unroll
                for (uint32_t u = 0; u < V; ++u) {
                    jc[u] = j1[u];
                    bc_[u] = b1[u];
                    qc[u] = q1[u];
                }
                fetch(i + STEP);
                ids(i + 2u * STEP);
#pragma unroll
                for (uint32_t u = 0; u < V; ++u) {
                    if (jc[u] < mm && BST_IN(bc_[u], B, CHECK_HIST_ROW)) {
                        long long g, h;
                        load.conv(qc[u], g, h);
                        const uint32_t cell = ((jc[u] * B + bc_[u]) << lk) + copy;
                        if constexpr (WIDE) {
                            st_add64(acc, acc + plane, cell, g);
                            st_add64(acc + 2 * plane, acc + 3 * plane, cell, h);
                        } else {
                            atomicAdd(&acc[cell], (uint32_t)(int32_t)g);
                            atomicAdd(&acc[plane + cell], (uint32_t)(int32_t)h);
                        }
                    }
                }
            }
            __syncthreads();
            // the copies folded; the lanes of a warp start at different
            // copies so that they read 32 banks
            const uint32_t rot = lane >> (5u - lk), km = (1u << lk) - 1u;
            for (uint32_t cell = tid; cell < cells; cell += ST_THREADS) {
                long long g = 0, h = 0;
                for (uint32_t k = 0; k <= km; ++k) {
                    const uint32_t i = (cell << lk) + ((k + rot) & km);
                    if constexpr (WIDE) {
                        g += (long long)(((unsigned long long)acc[plane + i] << 32) | acc[i]);
                        h += (long long)(((unsigned long long)acc[3 * plane + i] << 32) | acc[2 * plane + i]);
                    } else {
                        g += (int32_t)acc[i];
                        h += (int32_t)acc[plane + i];
                    }
                }
                sum[cell] = SA::make(g, h);
            }
            if (tid == 0) s.n_list = 0;
            __syncthreads();
            const uint32_t nodes = root ? 1u : 2u * mm;
            if (cm.is_cat) {
                st_categories<MODE, WIDE>(a, s, dyn, c, cm, j0, mm, level, slots, parents, root, searched, sum);
                __syncthreads();  // the shared counters are reused
                continue;
            }
            // Prefix sums of the smaller children's bins, a warp per
            // (expansion, 32 bins) so that a level of few nodes uses every warp.
            for (uint32_t it = warp; it < mm * nq; it += ST_WARPS) {
                const uint32_t j = it / nq, b = (it % nq) * 32u + lane;
                T2 v = b < B ? sum[j * B + b] : SA::make(0, 0);
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const Acc t0 = __shfl_up_sync(FULL, v.x, d), t1 = __shfl_up_sync(FULL, v.y, d);
                    if (lane >= (uint32_t)d) {
                        v.x += t0;
                        v.y += t1;
                    }
                }
                if (b < B) sum[j * B + b] = v;
                if (lane == 31u) carry[j * (nq + 1u) + it % nq] = v;
            }
            for (uint32_t k = tid; k < nodes; k += ST_THREADS) s.best[k] = 0ull;
            __syncthreads();
            for (uint32_t i = tid; i < 2u * mm; i += ST_THREADS) {  // totals of 32 bins -> the sums before them
                Acc* x = reinterpret_cast<Acc*>(carry + (i >> 1) * (nq + 1u)) + (i & 1u);
                Acc run = 0;
                for (uint32_t q0 = 0; q0 < nq; q0 += 8u) {
                    Acc t[8];
#pragma unroll
                    for (uint32_t q = 0; q < 8u; ++q) t[q] = q0 + q < nq ? x[2u * (q0 + q)] : 0;
#pragma unroll
                    for (uint32_t q = 0; q < 8u; ++q) {
                        if (q0 + q < nq) x[2u * (q0 + q)] = run;
                        run += t[q];
                    }
                }
                x[2u * nq] = run;
            }
            __syncthreads();
            // The sums of a child (kid 0: left) at bin b, and of all its bins
            // and of all but the last one.
            auto parent = [&](uint32_t j, uint32_t b) {
                if (root) return make_longlong2(0, 0);
                return __ldcg(reinterpret_cast<const longlong2*>(hist + (size_t)(parents + s.front[j0 + j]) * a.slot_bins + b));
            };
            auto small_at = [&](uint32_t j, uint32_t b) {
                const T2 v = sum[j * B + b], t = carry[j * (nq + 1u) + b / 32u];
                return make_longlong2((long long)v.x + t.x, (long long)v.y + t.y);
            };
            // 1. The best approximate score of each child per 32 bins; the
            // children's histograms are stored on the way.
            if (searched || store) {
                for (uint32_t it = warp; it < mm * nq; it += ST_WARPS) {
                    const uint32_t j = it / nq, q = it % nq, b = q * 32u + lane;
                    const bool sl = root || s.small_left[j0 + j] != 0;
                    longlong2 pp = make_longlong2(0, 0), mp = pp, ps = pp, ms = pp;
                    if (b < B) pp = parent(j, b);
                    if (hm && B >= 2u) {
                        mp = parent(j, B - 2u);
                        ms = small_at(j, B - 2u);
                    }
                    if (b < B) ps = small_at(j, b);
                    const longlong2 pl = make_longlong2(pp.x - ps.x, pp.y - ps.y);
                    if (store && b < B) {
                        HBin* o = hist + (size_t)(slots + (root ? 0u : 2u * (j0 + j))) * a.slot_bins + b;
                        *reinterpret_cast<longlong2*>(o) = sl ? ps : pl;
                        if (!root) *reinterpret_cast<longlong2*>(o + a.slot_bins) = sl ? pl : ps;
                    }
                    if (!searched) continue;
                    const T2 tt = carry[j * (nq + 1u) + nq];
                    const longlong2 Ts = make_longlong2(tt.x, tt.y), Tp = root ? Ts : s.ptot[j0 + j];
#pragma unroll
                    for (uint32_t kid = 0; kid < 2u; ++kid) {  // kid 0: the smaller child
                        if (root && kid) break;
                        const uint32_t side = (kid == 0u) == sl ? 0u : 1u;
                        const longlong2 T = kid ? make_longlong2(Tp.x - Ts.x, Tp.y - Ts.y) : Ts;
                        const longlong2 M = kid ? make_longlong2(mp.x - ms.x, mp.y - ms.y) : ms;
                        const ScoreRule<long long> rule(s.hmin, s.lam, a.gp, ih,
                                                        s.f_cnt[root ? 0u : 2u * (j0 + j) + side]);
                        float sc = rule.best(kid ? pl : ps, T, M, b, B, hm);
                        if (sc >= 0.0f && (!(a.gp.min_gain >= 0.0) || T.y < 0 || !((float)T.y + s.lam > 0.0f)))
                            sc = INFINITY;  // the offset's sign is not known
                        for (int o = 16; o > 0; o >>= 1) sc = fmaxf(sc, __shfl_xor_sync(FULL, sc, o));
                        if (lane == 0u) score[2u * (j * nq + q) + side] = sc;
                    }
                }
            }
            if (c == s.first_col)
                for (uint32_t k = tid; k < nodes; k += ST_THREADS) {
                    const uint32_t j = k >> 1, node = 2u * j0 + k;
                    const T2 t = carry[(root ? 0u : j) * (nq + 1u) + nq];
                    longlong2 T = make_longlong2(t.x, t.y);
                    if (!root && (s.small_left[j0 + j] != 0) != ((k & 1u) == 0u))
                        T = make_longlong2(s.ptot[j0 + j].x - T.x, s.ptot[j0 + j].y - T.y);
                    a.tot[2 * (st_level(level) + node)] = T.x;
                    a.tot[2 * (st_level(level) + node) + 1] = T.y;
                }
            __syncthreads();
            if (searched && B >= 2u) {
                // 2. Which 32 bins can hold a child's best split: those whose
                // score is within 2^-16 of the child's best. The score
                // gl^2 / (hl + lambda) + gr^2 / (hr + lambda) in f32 (units of
                // the integer sums) is off by less than 2^-19 and the gain is
                // half of it less an offset >= 0, so no other candidate can
                // win or tie: the f64 divisions, which bound the search, run
                // for a chunk or two of a node instead of all. A score that is
                // not finite (a denominator of zero or below, an overflow)
                // lets every chunk through.
                for (uint32_t k = tid; k < nodes; k += ST_THREADS) {
                    const float* sc = score + 2u * (root ? 0u : k >> 1) * nq + (k & 1u);
                    float mx = -1.0f;
                    for (uint32_t q = 0; q < nq; ++q) mx = fmaxf(mx, sc[2u * q]);
                    if (mx < 0.0f) continue;  // no valid candidate
                    const float thr = mx < INFINITY ? mx * (1.0f - 1.0f / 65536.0f) : -1.0f;
                    for (uint32_t q = 0; q < nq; ++q)
                        if (sc[2u * q] >= thr) list[atomicAdd(&s.n_list, 1u)] = k << 16 | q;
                }
                __syncthreads();
                // 3. Their exact gains.
                const uint32_t n_list = s.n_list;
                for (uint32_t e = warp; e < n_list; e += ST_WARPS) {
                    const uint32_t k = list[e] >> 16, q = list[e] & 0xFFFFu, j = root ? 0u : k >> 1, b = q * 32u + lane;
                    const uint32_t node = 2u * j0 + k;
                    const bool small = root || (s.small_left[j0 + j] != 0) == ((k & 1u) == 0u);
                    longlong2 P = make_longlong2(0, 0), M = P;
                    const T2 tt = carry[j * (nq + 1u) + nq];
                    longlong2 T = make_longlong2(tt.x, tt.y);
                    if (b < B) P = small_at(j, b);
                    if (hm) M = small_at(j, B - 2u);
                    if (!small) {
                        if (b < B) {
                            const longlong2 p = parent(j, b);
                            P = make_longlong2(p.x - P.x, p.y - P.y);
                        }
                        if (hm) {
                            const longlong2 p = parent(j, B - 2u);
                            M = make_longlong2(p.x - M.x, p.y - M.y);
                        }
                        T = make_longlong2(s.ptot[j0 + j].x - T.x, s.ptot[j0 + j].y - T.y);
                    }
                    const double tgd = (double)T.x * ig, thd = (double)T.y * ih;
                    GainCtx ctx;
                    ctx.lambda = a.gp.lambda;
                    ctx.offset = 0.5 * (tgd * tgd / (thd + a.gp.lambda)) + a.gp.min_gain;
                    ctx.mcw = a.gp.min_child_weight;
                    ctx.msl = a.gp.min_samples_leaf;
                    unsigned long long best = st_candidates(P, T, M, b, B, hm, s.f_cnt[node], ig, ih, ctx);
                    for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(FULL, best, o));
                    if (lane == 0u && best) atomicMax(&s.best[k], best);
                }
                __syncthreads();
                for (uint32_t k = tid; k < nodes; k += ST_THREADS) {
                    const unsigned long long best = s.best[k];
                    if (!best) continue;
                    const uint32_t node = 2u * j0 + k, order = ~(uint32_t)best;
                    const uint32_t u = (uint32_t)(best >> 32);
                    const float gain = __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
                    const bool fwd = order + 1u < B;
                    ColCand* out = a.cand + (size_t)node * a.n_cols + c;
                    out->gain = gain;
                    out->order = order;
                    out->bin = fwd ? order : 2u * B - 3u - order;
                    out->flags = fwd ? 0u : 1u;
                    out->cats[0] = out->cats[1] = out->cats[2] = out->cats[3] = 0ull;
                    atomicMax(&a.keys[st_level(level) + node], cand_key(gain, c, a.last_wins));
                }
            }
            __syncthreads();  // the shared counters are reused
        }
    }
}

template <int MODE, bool WIDE>
__global__ void __launch_bounds__(ST_THREADS, 1) k_small_tree(const __grid_constant__ SmallTree a) {
    extern __shared__ __align__(16) unsigned char st_smem[];
    __shared__ StShared s;
    const uint32_t tid = threadIdx.x;
    const StRows<MODE> load(a);
    const uint32_t P = gridDim.x;
    uint32_t target = 0;
    uint32_t n_front = 1, n_tn = 1;
    // this block's slice of the rows
    const uint32_t per = (a.n + P - 1) / P;
    const uint32_t r_begin = min(a.n, blockIdx.x * per), r_end = min(a.n, r_begin + per);
    for (uint32_t i = tid; i < ST_NODES; i += ST_THREADS) s.split[i] = 0;
    if (tid < 4u) s.scale[tid] = a.scale[tid];
    if (tid == 64u) {
        s.first_col = 0u;
        s.hmin = hess_min(a.gp.min_child_weight, a.scale[3]);
        s.lam = hess_lambda(a.gp.lambda, a.scale[3]);
    }
    if (tid == 32u && blockIdx.x < a.n_cols) {
        s.col = a.cols[blockIdx.x];
        s.bcol = a.bcols[blockIdx.x];
    }
    if (tid == 0) {
        s.f_tnode[0] = 0;
        s.f_cnt[0] = a.n_root;
        s.small_rows = a.n;
    }
    __syncthreads();
    st_histograms<MODE, WIDE>(a, s, st_smem, load, 1u, 0u, true, a.max_depth > 1u);
    uint32_t d = 0;
    for (;; ++d) {
        target += P;
        if (!st_barrier(a.bar, target, &a.state->err)) return;
        // decisions of level d (grower.rs:353-372, 530-539), the same in every
        // block; block 0 writes the tree
        PartWork w;
        uint32_t tn = 0;
        bool ex = false;
        float gain = 0.0f;
        uint32_t col = 0;
        longlong2 tot = make_longlong2(0, 0);
        if (tid < n_front) {
            tn = s.f_tnode[tid];
            tot.x = __ldcg(a.tot + 2 * (st_level(d) + tid));
            tot.y = __ldcg(a.tot + 2 * (st_level(d) + tid) + 1);
            const unsigned long long key = __ldcg(a.keys + st_level(d) + tid);
            if (key != 0ull) {
                col = a.last_wins ? (uint32_t)key : ~(uint32_t)key;
                const uint4* cp = reinterpret_cast<const uint4*>(a.cand + (size_t)tid * a.n_cols + col);
                const uint4 c0 = __ldcg(cp), c1 = __ldcg(cp + 1), c2 = __ldcg(cp + 2);
                gain = __uint_as_float(c0.x);
                ex = gain > -INFINITY && !((double)gain <= a.lp.min_gain);
                const BColumn bc = a.bcols[col];
                const bool cat = (c0.w & 2u) != 0u;
                w.begin = w.count = w.pad = 0;
                w.matrix = bc.matrix;
                w.pos = bc.pos;
                w.thr_bin = c0.z;
                w.flags = (c0.w & 1u) | (bc.has_missing ? 2u : 0u) | (cat ? 4u : 0u);
                w.default_bin = bc.default_bin;
                w.cats[0] = ((unsigned long long)c1.y << 32) | c1.x;
                w.cats[1] = ((unsigned long long)c1.w << 32) | c1.z;
                w.cats[2] = ((unsigned long long)c2.y << 32) | c2.x;
                w.cats[3] = ((unsigned long long)c2.w << 32) | c2.z;
            }
        }
        for (uint32_t i = tid; i < n_tn; i += ST_THREADS) s.map[i] = ST_NONE;
        for (uint32_t i = tid; i < ST_FRONT; i += ST_THREADS) s.cnt[i] = s.scnt[i] = 0;
        uint32_t n_exp;
        const uint32_t j = block_excl_scan(ex ? 1u : 0u, s.sh, &n_exp);  // (synchronises)
        if (ex) {
            const bool cat = (w.flags & 4u) != 0u;
            const uint32_t tla = n_tn + 2 * j, tra = tla + 1;
            s.map[tn] = (uint16_t)j;
            s.split[tn] = 1;
            s.work[j] = w;
            s.tl[j] = (uint16_t)(cat ? tra : tla);  // categorical: training-left rows go to the stored right child
            s.tr[j] = (uint16_t)(cat ? tla : tra);
            s.front[j] = (uint16_t)tid;
            s.ptot[j] = tot;
            s.f_tnode[2 * j] = s.tl[j];
            s.f_tnode[2 * j + 1] = s.tr[j];
            if (blockIdx.x == 0) {
                BTreeNode t;
                t.col = col;
                t.bin = w.thr_bin;
                t.flags = (w.flags & 1u) | (cat ? 2u : 0u);
                t.left = tla;
                t.right = tra;
                t.gain = gain;
                t.leaf = 0.0f;
                t.G = (double)tot.x * s.scale[2];
                t.H = (double)tot.y * s.scale[3];
                for (int q = 0; q < 4; ++q) t.cats[q] = w.cats[q];
                a.tree[tn] = t;
            }
        }
        __syncthreads();
        if (n_exp == 0) break;
        const bool need_split = d + 1 < a.max_depth;
        // this block's rows move to the children
        for (uint32_t i = r_begin + tid; i < r_end; i += ST_THREADS) {
            const uint32_t t = d ? a.rt[i] : 0u;  // written by this thread's block alone
            if (!BST_IN(t, n_tn, CHECK_SMALL_NODE)) continue;
            const uint32_t jx = s.map[t];
            if (jx == ST_NONE || !BST_IN(jx, n_exp, CHECK_SMALL_NODE)) continue;
            const PartWork& pw = s.work[jx];
            const uint32_t bin = pw.matrix == 0 ? (uint32_t)a.fm8[(size_t)pw.pos * a.n + i]
                                                : (uint32_t)a.fm16[(size_t)pw.pos * a.n + i];
            const bool left = part_left(pw, bin);
            a.rt[i] = left ? s.tl[jx] : s.tr[jx];
            if (need_split) {
                const uint32_t k = 2 * jx + (left ? 0u : 1u);
                atomicAdd(&s.cnt[k], 1u);
                if (a.rmask && a.rmask[i]) atomicAdd(&s.scnt[k], 1u);
            }
        }
        n_tn += 2 * n_exp;
        n_front = 2 * n_exp;
        if (!need_split) {
            ++d;
            break;
        }
        __syncthreads();
        for (uint32_t k = tid; k < n_front; k += ST_THREADS) {
            if (s.cnt[k]) atomicAdd(&a.cnt[st_level(d + 1) + k], s.cnt[k]);
            if (s.scnt[k]) atomicAdd(&a.scnt[st_level(d + 1) + k], s.scnt[k]);
        }
        target += P;
        if (!st_barrier(a.bar, target, &a.state->err)) return;
        // the smaller children (grower.rs:398-402)
        for (uint32_t i = tid; i < n_tn; i += ST_THREADS) s.map[i] = ST_NONE;
        __syncthreads();
        for (uint32_t k = tid; k < n_exp; k += ST_THREADS) {
            const uint32_t lc = __ldcg(a.cnt + st_level(d + 1) + 2 * k), rc = __ldcg(a.cnt + st_level(d + 1) + 2 * k + 1);
            const bool ls = lc <= rc;
            s.small_left[k] = ls ? 1 : 0;
            s.map[ls ? s.tl[k] : s.tr[k]] = (uint16_t)k;
            s.f_cnt[2 * k] = a.rmask ? __ldcg(a.scnt + st_level(d + 1) + 2 * k) : lc;
            s.f_cnt[2 * k + 1] = a.rmask ? __ldcg(a.scnt + st_level(d + 1) + 2 * k + 1) : rc;
            atomicAdd(&s.small_rows, (unsigned long long)(ls ? lc : rc));
        }
        __syncthreads();
        st_histograms<MODE, WIDE>(a, s, st_smem, load, n_exp, d + 1, false, d + 2 < a.max_depth);
    }
    // every leaf's exact sums of the f32 gradients' fixed-point values: in the
    // f32 form the same integers as its histogram's, in the quantised forms
    // what its value is solved from
    uint32_t* xs = reinterpret_cast<uint32_t*>(st_smem);  // [4][ST_NODES]: g lo, g hi, h lo, h hi
    float* val = reinterpret_cast<float*>(st_smem) + 4u * ST_NODES;
    for (uint32_t i = tid; i < 4u * ST_NODES; i += ST_THREADS) xs[i] = 0;
    __syncthreads();
    const double fg = a.fscale[0], fh = a.fscale[1];
    const bool moved = n_tn > 1;
    for (uint32_t i = r_begin + tid; i < r_end; i += ST_THREADS) {
        const uint32_t t = moved ? a.rt[i] : 0u;
        if (!BST_IN(t, n_tn, CHECK_SMALL_NODE)) continue;
        long long g, h;
        if constexpr (MODE == GRAD_F32) {
            load.conv(load.raw(i), g, h);
        } else {
            const float2 v = a.gr.gh[i];
            g = quantize(v.x, fg);
            h = quantize(v.y, fh);
        }
        st_add64(xs, xs + ST_NODES, t, g);
        st_add64(xs + 2 * ST_NODES, xs + 3 * ST_NODES, t, h);
    }
    __syncthreads();
    for (uint32_t t = tid; t < n_tn; t += ST_THREADS) {
        const unsigned long long g = ((unsigned long long)xs[ST_NODES + t] << 32) | xs[t];
        const unsigned long long h = ((unsigned long long)xs[3 * ST_NODES + t] << 32) | xs[2 * ST_NODES + t];
        if (g) atomicAdd(&a.xsum[2 * t], g);
        if (h) atomicAdd(&a.xsum[2 * t + 1], h);
    }
    target += P;
    if (!st_barrier(a.bar, target, &a.state->err)) return;
    for (uint32_t t = tid; t < n_tn; t += ST_THREADS) {
        if (s.split[t]) continue;
        const long long g = (long long)__ldcg(a.xsum + 2 * t), h = (long long)__ldcg(a.xsum + 2 * t + 1);
        const float v = leaf_value_dev(g, h, a.fscale, a.lp);
        val[t] = v;
        if (blockIdx.x == 0) write_leaf(a.tree[t], g, h, a.fscale, v);
    }
    if (blockIdx.x == 0 && tid == 0) {
        a.state->n_tnodes = n_tn;
        a.state->hist_rows = s.small_rows;
    }
    __syncthreads();
    for (uint32_t i = r_begin + tid; i < r_end; i += ST_THREADS) {  // grower.rs:208-219
        const uint32_t t = moved ? a.rt[i] : 0u;
        if (!BST_IN(t, n_tn, CHECK_SMALL_NODE)) continue;
        a.pred[i] = a.pred[i] + val[t];
        if (a.row_leaf) a.row_leaf[i] = t;
    }
}

static const void* small_tree_kernel(int mode, bool wide) {
    if (mode == GRAD_F32) return reinterpret_cast<const void*>(k_small_tree<GRAD_F32, true>);
    if (mode == GRAD_Q16)
        return wide ? reinterpret_cast<const void*>(k_small_tree<GRAD_Q16, true>)
                    : reinterpret_cast<const void*>(k_small_tree<GRAD_Q16, false>);
    return reinterpret_cast<const void*>(k_small_tree<GRAD_Q8, false>);
}

// 32-bit counters hold every sum of n quantised values
static bool small_tree_wide(int mode, uint64_t n) {
    return mode == GRAD_F32 || n * (mode == GRAD_Q16 ? 32767ull : 127ull) > 0x7FFFFFFFull;
}

bool small_tree_fits(int mode, uint64_t n, uint32_t max_bins, bool has_cat) {
    if (mode == GRAD_Q8 && small_tree_wide(mode, n)) return false;
    const bool wide = small_tree_wide(mode, n);
    const uint32_t room = ST_DYN - (has_cat ? ST_SORT_BYTES : 0u) - 64u;
    if (max_bins > 65536u || st_bin_bytes(wide) * max_bins + st_chunk_bytes(wide, (max_bins + 31u) / 32u) > room) return false;
    init_kernel_attributes();
    int dev = 0, coop = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, small_tree_kernel(mode, small_tree_wide(mode, n)),
                                                      ST_THREADS, ST_DYN) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return per_sm >= 1;
}

void launch_small_tree(const SmallTree& a, cudaStream_t st) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(sm_count());
    c.blockDim = dim3(ST_THREADS);
    c.dynamicSmemBytes = ST_DYN;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = 1;
    void* args[] = {(void*)&a};
    cudaLaunchKernelExC(&c, small_tree_kernel(a.gr.mode, small_tree_wide(a.gr.mode, a.n)), args);  // errors: next check
}
