// Column-resident form of the batched FP32 worker: a CTA per forward segment and per traceback window,
// a matrix column per thread, for bands up to column_span(NT) columns.
//
// Why.  The recursion is bound by the latency of its chain of logAdds and by instruction issue, not by
// memory.  With cells spread by their place in the band and exchanged through a shared-memory ring,
// most instructions were not arithmetic: ring addresses, clamps, stores and loads, a look-ahead
// address per operand (24 warp instructions per band cell, issue 19 to 30 % busy).
//
// How.  Column x lives on thread x mod NT, whichever way the band moves.  A cell's neighbours are then
// on the same thread (the same column) or the one beside it (column x - 1 forward, x + 1 backward): one
// shared float4 each (shuffles and an edge per warp took ten instructions a step more).  Threads outside
// the band hold -inf, which makes every absent neighbour drop out of logAdd.  Three anti-diagonals'
// columns never share a thread: the host takes this path for a batch only if any three consecutive
// anti-diagonals span at most NT columns.  Past column_span(NT) the thread beside the band's edge may hold
// its other end: sweeps compiled for that (kFull) leave that neighbour out by its column.  A sweep is a chain of anti-diagonals and its
// warps issue in order, so every instruction that is not the recursion lengthens the chain: four more
// warps take them, each with less to do a step than the sweep, since they issue in order too (one warp
// for all of it made the step 760 cycles; the sweep alone takes under 300).  One works out the
// renormalisation shifts, one brings band facts and copies operands into shared memory kAhead
// anti-diagonals ahead, and two take the results out: forward, the values, bases and publication of
// windows; backward, ten anti-diagonals at a time, one the total probabilities (sequential folds), the
// other posteriors and pairs (one warp for both made a window's step 530 cycles longer than the sweep's
// at 512 threads: 2,300 of them).
//
// The arithmetic is that of ForwardSweep and window_task, operation for operation, so the values are
// theirs bit for bit.
//
// Measured on B200, the worker launch with cells by their place in the band / with four columns a lane,
// a warp per window, and every thread its own copies / with three helper warps / in this form: 8 reads of
// 8 to 12 kb (2.1e7 cells, 71 segments) 3.52 / 2.35 / 1.27 / 1.10 ms, 30 reads of 8 to 30 kb (1.5e8 cells)
// 5.36 / 3.85 / 3.04 / 2.92 ms, 6 reads of 3 to 8 kb at expansion 200 (512 threads) 6.79 / - / 3.88 / 2.98 ms.
#pragma once

namespace sa {
namespace fp32 {

// NT threads hold bands up to column_span(NT) columns (a neighbour's column included), and with kFull NT
__host__ __device__ constexpr int column_span(int nt) { return nt - 2; }

constexpr int kAhead = 6;                // anti-diagonals between a copy and its use
constexpr int kRows = 8;                 // rows of the copy rings
constexpr int kInfoRows = 128;           // rows of band facts kept
constexpr int kBlock = 10;               // anti-diagonals per total probability
constexpr int kPostRows = 64;            // anti-diagonals the posteriors' warp may lag (about 2 kBlock)

extern __shared__ float4 column_smem[];

// lae() with the table at the start of shared memory, in two halves: entries of 8 bytes lie in banks of
// their own, so lanes with different pieces do not conflict (16 bytes an entry put two on a bank: the
// forward sweep's step took 1.3 times as long).  C - 2 d rounded down, C a multiple of 16 large enough
// that the last place is 1/8, holds -ceil(2 d) mod 16 in bits 3..6: the byte offset of the piece,
// without a shift.  The cut-off is a predicated add.
struct LogAddHalves {
    float2 hi[16], lo[16];               // (a3, a2), (a1, a0) of the piece of -ceil(2 d) mod 16
};

__device__ __forceinline__ float4 lac_piece(float d) {
    const int k = __float_as_int(__fmaf_rd(d, -2.0f, 1572864.0f)) & 0x78;
    const char *t = reinterpret_cast<const char *>(column_smem) + k;
    const float2 h = *reinterpret_cast<const float2 *>(t);
    const float2 l = *reinterpret_cast<const float2 *>(t + sizeof(LogAddHalves::hi));
    return make_float4(h.x, h.y, l.x, l.y);
}

__device__ __forceinline__ float lac(float x, float y) {
    float mx = fmaxf(x, y);
    const float d = fabsf(x - y);
    const float4 c = lac_piece(d);
    const float h = fmaf(fmaf(fmaf(c.x, d, c.y), d, c.z), d, c.w);
    asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, 0f40F00000;\n\t@p add.rn.f32 %0, %0, %2;\n\t}"
        : "+f"(mx) : "f"(d), "f"(h));
    return mx;
}

// N independent ones, stage by stage
template <int N>
__device__ __forceinline__ void lacs(const float (&x)[N], const float (&y)[N], float (&r)[N]) {
    float d[N];
    float4 c[N];
#pragma unroll
    for (int j = 0; j < N; ++j) d[j] = fabsf(x[j] - y[j]);
#pragma unroll
    for (int j = 0; j < N; ++j) c[j] = lac_piece(d[j]);
#pragma unroll
    for (int j = 0; j < N; ++j) r[j] = fmaxf(x[j], y[j]);
    float h[N];
#pragma unroll
    for (int j = 0; j < N; ++j) h[j] = fmaf(c[j].x, d[j], c[j].y);
#pragma unroll
    for (int j = 0; j < N; ++j) h[j] = fmaf(h[j], d[j], c[j].z);
#pragma unroll
    for (int j = 0; j < N; ++j) h[j] = fmaf(h[j], d[j], c[j].w);
#pragma unroll
    for (int j = 0; j < N; ++j)
        asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, 0f40F00000;\n\t@p add.rn.f32 %0, %0, %2;\n\t}"
            : "+f"(r[j]) : "f"(d[j]), "f"(h[j]));
}

__device__ __forceinline__ void copy_async4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

__device__ __forceinline__ void copy_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// barrier `id` of the CTA over n threads (the sweep's warps, or they and the warp of the posteriors)
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
// kBarFull + b, kBarTotal + b, kBarEmpty + b: block buffer b
enum { kBarRow = 1, kBarFull = 2, kBarTotal = 4, kBarEmpty = 6, kBarResults = 8 };
// threads of the warps beside a sweep's: shifts, copies, and two of the results (forward: the cells;
// backward: totals, and posteriors)
constexpr int kHelpers = 128;

// ------------------------------------------------------------------------------------------------
// band facts of a sweep, 32 anti-diagonals at a time, by its service warp
// ------------------------------------------------------------------------------------------------
// The k-th anti-diagonal of the sweep is start + DIR k.  A block is loaded when the sweep is 64
// anti-diagonals before it and becomes readable half a block later.
struct InfoRing {
    int4 row[kInfoRows];                 // first column, width | flags, first cell, shift
    double base[kInfoRows];              // forward base (backward sweeps)
};

template <int DIR>
struct RowStream {
    InfoRing *ring;
    const Args *A;
    int64_t db;
    int lane;
    int32_t n, start, acc;               // acc: first cell of the next block (backward: past it)
    int2 raw;
    double base;
    float shift;

    __device__ __forceinline__ void load(int32_t k0) {
        const int32_t d = start + DIR * (k0 + lane), dc = clampi(d, 0, n);
        raw = __ldg(A->meta + db + dc);
        if (d < 0 || d > n) raw.y = 0;   // no such anti-diagonal: no cells
        if (DIR < 0) {
            base = __ldcg(A->base + db + dc);
            shift = __ldcg(A->fshift + db + dc);
        }
    }
    __device__ __forceinline__ void publish(int32_t k0) {
        const int32_t k = k0 + lane, d = start + DIR * k, W = raw.y & kWidthMask;
        int32_t sum = W;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t v = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += v;
        }
        const int32_t first = DIR > 0 ? acc + sum - W : acc - sum;
        ring->row[k & (kInfoRows - 1)] = make_int4((d + raw.x) >> 1, raw.y, first, __float_as_int(shift));
        if (DIR < 0) ring->base[k & (kInfoRows - 1)] = base;
        acc += DIR * __shfl_sync(0xffffffffu, sum, 31);
        __syncwarp();
    }
    // first: first cell of the first anti-diagonal (backward: past it)
    __device__ __forceinline__ void open(InfoRing *r, const Args &a, int64_t diag_base, int32_t nn, int32_t d0,
                                         int32_t first) {
        ring = r;
        A = &a;
        db = diag_base;
        lane = threadIdx.x & 31;
        n = nn;
        start = d0;
        acc = first;
        shift = 0.0f;
        base = 0.0;
        load(0);
        publish(0);
        load(32);
        publish(32);
    }
    __device__ __forceinline__ void advance(int32_t k) {
        if ((k & 31) == 0) load(k + 64);
        else if ((k & 31) == 16) publish(k + 48);
    }
    __device__ __forceinline__ int4 at(int32_t k) const { return ring->row[k & (kInfoRows - 1)]; }
};

// ------------------------------------------------------------------------------------------------
// shared memory
// ------------------------------------------------------------------------------------------------
// what a sweep's thread needs of an anti-diagonal, from the service warp
struct alignas(16) RowFacts {
    int32_t xf, w;                       // first column; width | flags
    float sh1, sh2;                      // the shifts of the values from one and from two anti-diagonals back
};
constexpr int32_t kRowPost = 1 << 23;    // posteriors of the anti-diagonal are the window's

template <int NT>
struct ColumnForwardShared {
    float2 e[kRows][NT];                 // match and extra-event emissions, by cell
    InfoRing info;
    RowFacts row[4];
    float4 v[2][NT];                     // match, gap-X, gap-Y by thread, by parity
    float part[2][NT / 32];              // the warps' largest values, by parity (more than 128 threads)
};

template <int NT>
struct ColumnWindowShared {
    float2 e[kRows][NT];
    InfoRing info;
    RowFacts row[4];
    float f[kRows][NT];                  // forward match values, by cell
    float ops[5][NT];                    // a total's anti-diagonal d: gap-X, gap-Y of d; match, gap-X, gap-Y of d-1
    float4 v[2][NT];                     // match and its emission a row back, gap-X, skip emission by thread,
                                         // by parity
    float part[2][NT / 32];              // the warps' largest values, by parity
    // for the posteriors' warp: by anti-diagonal of the sweep, its base and this window's; and two
    // blocks of kBlock anti-diagonals: F.B of the match state by thread, the two folds' terms, and the
    // shift and gamma of the total's anti-diagonal
    double fb[kPostRows], bb[kPostRows];
    double total[2];                     // the blocks' total probabilities
    int2 post[kPostRows];                // first column, width
    float s[2][kBlock][NT];
    float chain[2][2][NT];
    float2 through[2];
    int2 widths[2];                      // of the two folds
};
static_assert(offsetof(ColumnForwardShared<128>, e) == offsetof(ColumnWindowShared<128>, e), "one emission ring");

template <int NT>
struct alignas(16) ColumnShared {
    LogAddHalves la;
    union {
        ColumnForwardShared<NT> f;
        ColumnWindowShared<NT> w;
    };
    int32_t task;
};

// ------------------------------------------------------------------------------------------------
// one side of a stitch, and its check, by one warp (see stitch_check)
// ------------------------------------------------------------------------------------------------
__device__ __noinline__ void warp_stitch_check(const Args &A, int32_t si) {
    const int lane = threadIdx.x & 31;
    const StitchDesc sd = A.stitch[si];
    StitchRes &res = A.stitch_res[si];
    const double sb0 = __ldcg(&res.sbase[0]), sb1 = __ldcg(&res.sbase[1]);
    const double tb0 = __ldcg(&res.tbase[0]), tb1 = __ldcg(&res.tbase[1]);
    const int32_t nv = 3 * (sd.w0 + sd.w1);
    const float *spec = A.stitch_vals + sd.voff, *tru = spec + nv;
    double amax = -INFINITY, dref = 0.0;
    for (int q = lane; q < nv; q += 32) {
        const bool j = q >= 3 * sd.w0;
        const float tv = __ldcg(tru + q), sv = __ldcg(spec + q);
        if (tv > kNegInf && sv > kNegInf) {
            const double a = (double) tv + (j ? tb1 : tb0);
            if (a > amax) {
                amax = a;
                dref = a - ((double) sv + (j ? sb1 : sb0));
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double a2 = __shfl_xor_sync(0xffffffffu, amax, o), d2 = __shfl_xor_sync(0xffffffffu, dref, o);
        if (a2 > amax || (a2 == amax && d2 < dref)) {
            amax = a2;
            dref = d2;
        }
    }
    const double scale = (double) A.stitch_tol;
    bool ok = scale >= 0.0;
    double spread = 0.0;
    for (int q = lane; q < nv; q += 32) {
        const bool j = q >= 3 * sd.w0;
        const float tv = __ldcg(tru + q), sv = __ldcg(spec + q);
        const bool ft = tv > kNegInf, fs = sv > kNegInf;
        if (ft != fs) {
            ok = false;
        } else if (ft) {
            const double a = (double) tv + (j ? tb1 : tb0);
            const double dev = fabs((a - ((double) sv + (j ? sb1 : sb0))) - dref);
            spread = fmax(spread, dev);
            if (!(dev <= scale * (2e-5 + 1e-6 * (amax - a)))) ok = false;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) spread = fmax(spread, __shfl_xor_sync(0xffffffffu, spread, o));
    ok = __all_sync(0xffffffffu, ok);
    if (lane == 0) {
        res.delta = dref;
        res.spread = (float) spread;
        res.result = ok ? kStitchAgreed : kStitchDisagreed;
        if (!ok) atomicExch(A.seg_fail + sd.read, 1);
        __threadfence();
    }
    __syncwarp();
    read_unit_done<32>(A, sd.read, lane, nullptr);
}

// one side of stitch si has written its values: the second to arrive checks it (one warp)
__device__ __forceinline__ void warp_stitch_arrive(const Args &A, int32_t si) {
    int32_t before = 0;
    if ((threadIdx.x & 31) == 0) {
        __threadfence();
        before = atomicAdd(&A.stitch_res[si].arrive, 1);
        __threadfence();
    }
    if (__shfl_sync(0xffffffffu, before, 0) == 1) warp_stitch_check(A, si);
}

// The largest of the warps' values (part: one row of them), and a warp's share of it.  A sweep of up to
// 128 threads leaves both to the warp of the shifts; wider, that warp would read too long.
template <int NW>
__device__ __forceinline__ float part_max(const float *part) {
    float m[NW];
#pragma unroll
    for (int w = 0; w < NW; ++w) m[w] = part[w];
#pragma unroll
    for (int o = NW / 2; o > 0; o >>= 1)
#pragma unroll
        for (int w = 0; w < NW / 2; ++w)
            if (w < o) m[w] = fmaxf(m[w], m[w + o]);
    return m[0];
}

__device__ __forceinline__ void part_of(float *part, float m, float x, float y) {
    const float mx = warp_max1(fmaxf(m, fmaxf(x, y)));
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = mx;
}

// ------------------------------------------------------------------------------------------------
// forward sweep of one segment
// ------------------------------------------------------------------------------------------------
// On anti-diagonal d a thread folds, side by side: gap-X of d (left column on d-1), gap-Y of d (own
// column on d-1), the match state of d+1 but for its last term (left column on d-1), and the last
// term of d's: one logAdd's latency, a barrier and a shared-memory read a step.
template <int NT, bool kSX, bool kGX, bool kFull>
__device__ __forceinline__ void column_forward_sweep(const Ctx &c, const Segment &S, ColumnForwardShared<NT> *fs) {
    const Args &A = *c.A;
    const RegionDesc &R = c.R;
    const float *t = c.t;
    const int tid = threadIdx.x;
    const int32_t dbeg = S.d_begin, s = dbeg - S.warm + (dbeg == 0 ? 1 : 0), steps = S.d_end - s + 1;
    // own column on d-1, and d's match state but for its last term, and that term
    float M1 = kNegInf, X1 = kNegInf, Y1 = kNegInf, most = kNegInf, last = kNegInf;
    int32_t xf1 = 0;                     // first column of d-1
    if (dbeg == 0) {
        // anti-diagonal 0: startStateProb / raggedStartStateProb (stateMachine.c:1022-1032), column 0
        const float s0 = R.ragged_left ? kNegInf : 0.0f, s1 = R.ragged_left ? 0.0f : kNegInf;
        if (tid == 0) {
            M1 = s0;
            X1 = Y1 = s1;
        }
    } else {
        // a later segment: every band cell of s-2 and s-1 starts at 0
        const int2 r2 = raw_meta(A, R.diag_base, s - 2, R.n), r1 = raw_meta(A, R.diag_base, s - 1, R.n);
        if (((tid - ((s - 1 + r1.x) >> 1)) & (NT - 1)) < (r1.y & kWidthMask)) M1 = X1 = Y1 = 0.0f;
        bool left = ((tid - 1 - ((s - 2 + r2.x) >> 1)) & (NT - 1)) < (r2.y & kWidthMask);
        if (kFull) {
            const int32_t xf = (s + raw_meta(A, R.diag_base, s, R.n).x) >> 1;
            left = left && xf + ((tid - xf) & (NT - 1)) > ((s - 2 + r2.x) >> 1);
            xf1 = (s - 1 + r1.x) >> 1;
        }
        const float z = left ? 0.0f : kNegInf;
        most = lac(z + t[T_MC], z + t[T_MFGX]);
        last = z + t[T_MFGY];
    }
    fs->v[1][tid] = make_float4(M1, X1, Y1, 0.0f);
    if (NT > 128) part_of(fs->part[1], M1, X1, Y1);
    const float4 *left = &fs->v[0][(tid + NT - 1) & (NT - 1)];   // the column before
    bar_sync(kBarRow, NT + kHelpers);          // the first rows are ready
    RowFacts row = fs->row[0];
    bool inb = ((tid - row.xf) & (NT - 1)) < (row.w & kWidthMask);
    int32_t x0 = row.xf + ((tid - row.xf) & (NT - 1));   // own column on d
    float2 e = fs->e[0][(tid - row.xf) & (NT - 1)];
    float gx = 0.0f;
    if (kGX) gx = raw_gapx(c, row.xf + ((tid - row.xf) & (NT - 1)));
#pragma unroll 2
    for (int32_t k = 0; k < steps; ++k) {
        float x[4], y[4], r[4];
        x[1] = M1 + t[T_OY];
        y[1] = Y1 + t[T_EY];
        x[2] = most;
        y[2] = last;
        bar_sync(kBarRow, NT + kHelpers);      // d-1's values; d+1's facts and emissions
        float4 l = left[((k + 1) & 1) * NT];
        const RowFacts next = fs->row[(k + 1) & 3];
        const int32_t i = (tid - next.xf) & (NT - 1);
        if (kFull) {   // no column before d-1's first (a thread in the band on d and on d+1 has one column)
            if ((inb ? x0 : next.xf + i) <= xf1) l.x = l.y = l.z = kNegInf;
            xf1 = row.xf;
            x0 = next.xf + i;
        }
        x[0] = l.x + t[T_OX];
        y[0] = l.y + t[T_EX];
        x[3] = l.x + t[T_MC];
        y[3] = l.y + t[T_MFGX];
        const float2 e_next = fs->e[(k + 1) & (kRows - 1)][i];
        lacs<4>(x, y, r);
        if (kSX) r[0] = lac(r[0], l.z + t[T_SX]);
        const float vX = r[0] + ((kGX ? gx : c.gx) + row.sh1);
        const float vY = r[1] + (e.y + row.sh1);
        const float vM = r[2] + (e.x + row.sh2);
        most = r[3];
        last = l.z + t[T_MFGY];
        M1 = inb ? vM : kNegInf;
        X1 = inb ? vX : kNegInf;
        Y1 = inb ? vY : kNegInf;
        fs->v[k & 1][tid] = make_float4(M1, X1, Y1, 0.0f);
        if (NT > 128) part_of(fs->part[k & 1], M1, X1, Y1);
        row = next;
        inb = i < (next.w & kWidthMask);
        e = e_next;
        if (kGX) gx = raw_gapx(c, row.xf + i);
    }
    bar_sync(kBarRow, NT + kHelpers);          // the last anti-diagonal's values go out
}

// The forward sweep's shifts: at step k (anti-diagonal d) those of d+2, from the maximum of d-1.
// Renormalisation as in ForwardSweep: base(d+1) = base(d-2) + max(d-2); delta(d) = base(d) - base(d-1).
template <int NT>
__device__ __forceinline__ void column_forward_shifts(const Segment &S, ColumnForwardShared<NT> *fs) {
    const int lane = threadIdx.x & 31;
    const int32_t s = S.d_begin - S.warm + (S.d_begin == 0 ? 1 : 0), steps = S.d_end - s + 1;
    float d0 = 0.0f, d1 = 0.0f;          // delta of d and of d+1 (max(s-2) counts as 0)
    if (lane < 2) *reinterpret_cast<float2 *>(&fs->row[lane].sh1) = make_float2(-d0, -d0 - d0);
    bar_sync(kBarRow, NT + kHelpers);
#pragma unroll 2
    for (int32_t k = 0; k < steps; ++k) {
        bar_sync(kBarRow, NT + kHelpers);
        float mx;
        if constexpr (NT > 128) {
            mx = part_max<NT / 32>(fs->part[(k + 1) & 1]);
        } else {
            const float4 *v = &fs->v[(k + 1) & 1][lane];
            float most[NT / 32];
#pragma unroll
            for (int w = 0; w < NT / 32; ++w) {
                const float4 u = v[32 * w];
                most[w] = fmaxf(u.x, fmaxf(u.y, u.z));
            }
            mx = warp_max1(part_max<NT / 32>(most));
        }
        const float d2 = ((mx > kNegInf ? mx : 0.0f) - d1) - d0;
        if (lane == 0) *reinterpret_cast<float2 *>(&fs->row[(k + 2) & 3].sh1) = make_float2(-d2, -d1 - d2);
        d0 = d1;
        d1 = d2;
    }
    bar_sync(kBarRow, NT + kHelpers);
}

// The forward sweep's copies: at step k the emissions of the kAhead-th anti-diagonal after, and the
// place of the second.
template <int NT>
__device__ __forceinline__ void column_forward_copies(const Ctx &c, const Segment &S, ColumnForwardShared<NT> *fs) {
    constexpr int NW = NT / 32;
    const Args &A = *c.A;
    const RegionDesc &R = c.R;
    const int lane = threadIdx.x & 31;
    const int32_t s = S.d_begin - S.warm + (S.d_begin == 0 ? 1 : 0), steps = S.d_end - s + 1;
    const float2 *Ereg = A.E + R.cell_base + lane;
    RowStream<1> info;
    info.open(&fs->info, A, R.diag_base, R.n, s, (int32_t) S.cell0);
    auto issue = [&](int32_t k, const int4 &in) {
        const int32_t W = in.y & kWidthMask;
        const float2 *src = Ereg + in.z;
        float2 *dst = &fs->e[k & (kRows - 1)][lane];
#pragma unroll
        for (int w = 0; w < NW; ++w)
            if (lane + 32 * w < W) copy_async8(dst + 32 * w, src + 32 * w);
        copy_commit();
    };
    auto place = [&](int32_t k) {
        const int4 in = info.at(k);
        if (lane == 0) *reinterpret_cast<int2 *>(&fs->row[k & 3].xf) = make_int2(in.x, in.y);
    };
#pragma unroll
    for (int k = 0; k < kAhead; ++k) issue(k, info.at(k));
    place(0);
    place(1);
    copy_wait<kAhead - 2>();
    int4 in = info.at(kAhead);
    bar_sync(kBarRow, NT + kHelpers);
    for (int32_t k = 0; k < steps; ++k) {
        bar_sync(kBarRow, NT + kHelpers);
        issue(k + kAhead, in);
        place(k + 2);
        info.advance(k);
        in = info.at(k + kAhead + 1);
        copy_wait<kAhead - 2>();         // every copy of d+2 and before has landed
    }
    bar_sync(kBarRow, NT + kHelpers);
    copy_wait<0>();
}

// The forward sweep's results: at step k d-1's values, base and shift go out, a window that closes there
// is published, and a stitch there gets its side.  Two warps, `part` 0 and 1, share the cells.
template <int NT>
__device__ __forceinline__ void column_forward_results(const Ctx &c, const Segment &S, ColumnForwardShared<NT> *fs,
                                                       int part) {
    constexpr int NW = NT / 64;          // cells a lane has, 64 apart
    const Args &A = *c.A;
    const RegionDesc &R = c.R;
    const int lane = threadIdx.x & 31, cell = lane + 32 * part;
    const int64_t db = R.diag_base;
    const int32_t dbeg = S.d_begin, dend = S.d_end;
    const int32_t s = dbeg - S.warm + (dbeg == 0 ? 1 : 0), steps = dend - s + 1;
    float *Freg = A.F + 3 * R.cell_base;
    if (dbeg == 0 && cell == 0) {
        const float s0 = R.ragged_left ? kNegInf : 0.0f, s1 = R.ragged_left ? 0.0f : kNegInf;
        Freg[ST_M] = s0;
        Freg[ST_X] = s1;
        Freg[ST_Y] = s1;
        A.base[db] = 0.0;
        A.fshift[db] = 0.0f;
    }
    double base = 0.0;                   // base(d-1)
    double qbase = 0.0;                  // lane q: base and shift of the last d with d mod 32 == q
    float qshift = 0.0f;
    int32_t wi = S.wi0;
    int32_t cap = S.stitch_in >= 0 ? dbeg - 1 : (S.stitch_out >= 0 ? dend - 1 : INT32_MAX);
    bar_sync(kBarRow, NT + kHelpers);
    bar_sync(kBarRow, NT + kHelpers);    // step 0
    int4 in = fs->info.row[0];
    for (int32_t k = 1; k <= steps; ++k) {
        const int32_t r = s + k - 1;     // the anti-diagonal that goes out
        const int32_t W = in.y & kWidthMask;
        const bool own = r > dbeg, gaps = (in.y & kFlagStoreGaps) != 0;
        float *Fd = Freg + 3 * (int64_t) in.z + cell;
        int at[NW];
#pragma unroll
        for (int w = 0; w < NW; ++w) at[w] = (in.x + cell + 64 * w) & (NT - 1);
        bar_sync(kBarRow, NT + kHelpers);
        const float4 *v = fs->v[(k - 1) & 1];
        if (own) {
            float o[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) o[w] = v[at[w]].x;
#pragma unroll
            for (int w = 0; w < NW; ++w)
                if (cell + 64 * w < W) Fd[64 * w] = o[w];
            if (gaps) {
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    if (cell + 64 * w < W) {
                        Fd[W + 64 * w] = v[at[w]].y;
                        Fd[2 * W + 64 * w] = v[at[w]].z;
                    }
                }
            }
        }
        const float delta = -fs->row[(k - 1) & 3].sh1, delta_next = -fs->row[k & 3].sh1;
        const int4 in_next = fs->info.row[k & (kInfoRows - 1)];
        base += (double) delta;
        const bool window_end = own && (in.y & kFlagWindowEnd) != 0;
        const int q = r & 31;
        if (lane == q) {
            qbase = base;
            qshift = delta;
        }
        if (q == 31 || window_end || r == dend) {
            if (part == 0 && lane <= q && r - q + lane > dbeg) {
                A.base[db + (r - q) + lane] = qbase;
                A.fshift[db + (r - q) + lane] = qshift;
            }
            if (window_end) {
                __threadfence();         // this anti-diagonal and all before it, device-wide
                bar_sync(kBarResults, 64);
                if (cell == 0) {
                    const unsigned p = atomicAdd(&A.ctl->pub, 1u);
                    if ((int64_t) p < A.n_windows) atomicExch(A.ready + p, (int32_t) (R.win_base + wi));
                }
                ++wi;
            }
        }
        if (r == cap) {
            const bool in_side = S.stitch_in >= 0 && r <= dbeg;
            const int32_t si = in_side ? S.stitch_in : S.stitch_out, b = in_side ? dbeg : dend;
            const StitchDesc sd = A.stitch[si];
            float *o = A.stitch_vals + sd.voff + (in_side ? 0 : 3 * (sd.w0 + sd.w1)) + (r == b ? 3 * sd.w0 : 0);
            for (int i = cell; i < W; i += 64) {
                const float4 u = v[(in.x + i) & (NT - 1)];
                o[i] = u.x;
                o[W + i] = u.y;
                o[2 * W + i] = u.z;
            }
            if (r == b && cell == 0) {
                // as ForwardSweep: back from the base past b
                const double past = base + (double) delta_next, base_b = past - (double) delta_next;
                double *bs = in_side ? A.stitch_res[si].sbase : A.stitch_res[si].tbase;
                bs[0] = base_b - (double) delta;
                bs[1] = base_b;
            }
            cap = r < b ? b : (in_side && S.stitch_out >= 0 ? dend - 1 : INT32_MAX);
        }
        in = in_next;
    }
    if (S.stitch_in >= 0 || S.stitch_out >= 0) {
        __threadfence();                 // the stitch's values, before the counts below
        bar_sync(kBarResults, 64);
        if (S.stitch_in >= 0 && part == 0) warp_stitch_arrive(A, S.stitch_in);
        if (S.stitch_out >= 0 && part == 1) warp_stitch_arrive(A, S.stitch_out);
    }
}

// ------------------------------------------------------------------------------------------------
// the two ordered folds of a refresh
// ------------------------------------------------------------------------------------------------
// ordered_fold on chain[0..na) and on chain[32 NC..32 NC + nb), side by side: half the warp folds each, and
// of the values after the first largest one only those within the 7.5 cut-off of it are folded (the
// running result is at least the largest value by then, so logAdd returns it unchanged for any other).
template <int NC>
__device__ __forceinline__ float2 column_folds(float *chain, int na, int nb) {
    const int lane = threadIdx.x & 31;
    float va[NC], vb[NC];
    float ma = kNegInf, mb = kNegInf;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const int i = lane + 32 * k;
        va[k] = i < na ? chain[i] : kNegInf;
        vb[k] = i < nb ? chain[(32 * NC) + i] : kNegInf;
        ma = fmaxf(ma, va[k]);
        mb = fmaxf(mb, vb[k]);
    }
    ma = warp_max1(ma);
    mb = warp_max1(mb);
    // first index within kSeedGap of each maximum, and first index of the maximum
    int sa = na, sb = nb, xa = na, xb = nb;
#pragma unroll
    for (int k = NC - 1; k >= 0; --k) {
        const int i = lane + 32 * k;
        const unsigned a = __ballot_sync(0xffffffffu, i < na && va[k] >= ma - kSeedGap);
        const unsigned b = __ballot_sync(0xffffffffu, i < nb && vb[k] >= mb - kSeedGap);
        const unsigned a1 = __ballot_sync(0xffffffffu, i < na && va[k] == ma);
        const unsigned b1 = __ballot_sync(0xffffffffu, i < nb && vb[k] == mb);
        if (a) sa = 32 * k + __ffs(a) - 1;
        if (b) sb = 32 * k + __ffs(b) - 1;
        if (a1) xa = 32 * k + __ffs(a1) - 1;
        if (b1) xb = 32 * k + __ffs(b1) - 1;
    }
    float seed_a = 0.0f, seed_b = 0.0f;
    if (max(sa, sb) > 0) {
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            const int i = lane + 32 * k;
            seed_a += i < sa && va[k] > kNegInf ? __expf(va[k] - ma) : 0.0f;
            seed_b += i < sb && vb[k] > kNegInf ? __expf(vb[k] - mb) : 0.0f;
        }
        seed_a = warp_sum(seed_a);
        seed_b = warp_sum(seed_b);
    }
    const float ra = ma > kNegInf && seed_a > 0.0f ? ma + __logf(seed_a) : kNegInf;
    const float rb = mb > kNegInf && seed_b > 0.0f ? mb + __logf(seed_b) : kNegInf;
    // candidates, compacted in index order
    __syncwarp();   // every lane has read the chain
    int ca = 0, cb = 0;
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const int i = lane + 32 * k;
        const bool ia = i >= sa && va[k] > ma - kFoldGap && (i <= xa || ma - va[k] < 7.5f);
        const bool ib = i >= sb && vb[k] > mb - kFoldGap && (i <= xb || mb - vb[k] < 7.5f);
        const unsigned a = __ballot_sync(0xffffffffu, ia), b = __ballot_sync(0xffffffffu, ib);
        if (ia) chain[ca + __popc(a & below)] = va[k];
        if (ib) chain[(32 * NC) + cb + __popc(b & below)] = vb[k];
        ca += __popc(a);
        cb += __popc(b);
    }
    __syncwarp();
    const bool second = lane >= 16;
    const int mine = second ? cb : ca, most = max(ca, cb);
    const float *list = chain + (second ? (32 * NC) : 0);
    float r = second ? rb : ra;
    float next = mine > 0 ? list[0] : kNegInf;
    for (int k = 0; k < most; ++k) {
        const float v = next;
        next = k + 1 < mine ? list[k + 1] : kNegInf;
        r = lac(r, v);   // logAdd(r, -inf) is r
    }
    __syncwarp();   // the lists are read before the chain is written again
    return make_float2(__shfl_sync(0xffffffffu, r, 0), __shfl_sync(0xffffffffu, r, 16));
}

// ------------------------------------------------------------------------------------------------
// backward sweep of one traceback window
// ------------------------------------------------------------------------------------------------
template <int NT, bool kSX, bool kGX, bool kFull>
__device__ __forceinline__ void column_window_sweep(const Ctx &c, const Window &Wn, ColumnWindowShared<NT> *ws) {
    const RegionDesc &R = c.R;
    const float *t = c.t;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int32_t steps = Wn.D - Wn.T, rows = Wn.from - Wn.T;
    // end-state values on D (stateMachine.c:1034-1061)
    const bool ragged_end = Wn.at_end && R.ragged_right;
    const float e0 = ragged_end ? (t[T_OX] + t[T_OY]) / 2.0f : t[T_MC];
    const float e1 = ragged_end ? t[T_EX] : t[T_MFGX];
    const float e2 = ragged_end ? t[T_EY] : t[T_MFGY];
    ws->v[1][tid] = make_float4(kNegInf, 0.0f, kNegInf, 0.0f);
    const float4 *right = &ws->v[0][(tid + 1) & (NT - 1)];   // the column after
    // own column: values and emissions of d+1
    float M1 = kNegInf, Y1 = kNegInf;
    float2 e1r = make_float2(0.0f, 0.0f);
    float gx = 0.0f;
    int32_t i1 = 0, W1 = 0, xf1 = 0;     // its cell, the width and the first column of d+1
    int32_t hi1 = -1, hi2 = -1;          // last columns of d+1 and d+2
    int32_t left = rows;                 // posterior anti-diagonals to come
    int32_t block = 0, in_block = 0;
    bar_sync(kBarRow, NT + 64);          // the first rows are ready
    int2 row = *reinterpret_cast<const int2 *>(&ws->row[0].xf);   // first column, width | flags
    int32_t i = (tid - row.x) & (NT - 1);
    float2 e = ws->e[0][i];
    if (kGX) gx = raw_gapx(c, row.x + i);
#pragma unroll 1
    for (int32_t k = 0; k < steps; ++k) {
        const int32_t W = row.y & kWidthMask;
        const bool inb = i < W;
        bar_sync(kBarRow, NT + 64);      // d+1's values, d's shifts; d-1's facts and operands
        float4 n = right[((k + 1) & 1) * NT];
        if (kFull && row.x + i >= max(hi1, hi2)) n.x = n.z = kNegInf;   // no column after their last
        const float2 sh = *reinterpret_cast<const float2 *>(&ws->row[k & 3].sh1);
        const int2 next = *reinterpret_cast<const int2 *>(&ws->row[(k + 1) & 3].xf);
        const float me = n.x + (n.y + sh.y);
        const float ue = Y1 + (e1r.y + sh.x);
        const float le = n.z + ((kGX ? n.w : c.gx) + sh.x);
        float x[3], y[3], r[3];
        x[0] = me + t[T_MC];
        y[0] = ue + t[T_OY];
        x[1] = me + t[T_MFGX];
        y[1] = le + t[T_EX];
        x[2] = me + t[T_MFGY];
        y[2] = ue + t[T_EY];
        const int32_t i_next = (tid - next.x) & (NT - 1);
        const float2 e_next = ws->e[(k + 1) & (kRows - 1)][i_next];
        const float f = ws->f[k & (kRows - 1)][i];
        lacs<3>(x, y, r);
        r[0] = lac(r[0], le + t[T_OX]);
        if (kSX) r[2] = lac(r[2], le + t[T_SX]);
        if (k == 0) {
            r[0] = e0;
            r[1] = e1;
            r[2] = e2;
        }
        const float vM = inb ? r[0] : kNegInf, vX = inb ? r[1] : kNegInf, vY = inb ? r[2] : kNegInf;
        ws->v[k & 1][tid] = make_float4(M1, e1r.x, vX, gx);
        const float mx = warp_max1(fmaxf(vM, fmaxf(vX, vY)));
        if (lane == 0) ws->part[k & 1][warp] = mx;
        if ((row.y & kRowPost) != 0) {
            const int b = block & 1;
            if (in_block == 0 && block >= 2) bar_sync(kBarEmpty + b, NT + 32);   // the block before last is done with
            const float v = f + vM;
            ws->s[b][in_block][tid] = v;
            if (in_block == 0) {
                // diagonalCalculationTotalProbability (pairwiseAligner.c:1182-1200): F.B on d in ascending
                // cell order, then the matches from d-1 over d into d+1, dotted with B(d+1)
                if (inb) {
                    float w = lac(v, ws->ops[0][i] + vX);
                    w = lac(w, ws->ops[1][i] + vY);
                    ws->chain[b][0][i] = w;
                }
                if (k > 0 && i1 < W1) {
                    const int32_t l = xf1 + i1 - 1 - next.x;   // the column before, on d-1
                    const bool there = l >= 0 && l < (next.y & kWidthMask);
                    const int32_t lc = there ? l : 0;
                    float th = (there ? ws->ops[2][lc] : kNegInf) + (e1r.x + t[T_MC]);
                    th = lac(th, (there ? ws->ops[3][lc] : kNegInf) + (e1r.x + t[T_MFGX]));
                    th = lac(th, (there ? ws->ops[4][lc] : kNegInf) + (e1r.x + t[T_MFGY]));
                    ws->chain[b][1][i1] = th + M1;
                }
                if (tid == 0) {
                    ws->through[b] = make_float2(__int_as_float(ws->info.row[k & (kInfoRows - 1)].w), -sh.x);
                    ws->widths[b] = make_int2(W, k > 0 ? W1 : 0);
                }
            }
            ++in_block;
            --left;
            if (in_block == kBlock || left == 0) {
                __threadfence_block();
                bar_arrive(kBarFull + b, NT + 32);
                ++block;
                in_block = 0;
            }
        }
        M1 = vM;
        Y1 = vY;
        e1r = e;
        i1 = i;
        W1 = W;
        xf1 = row.x;
        if (kFull) {
            hi2 = hi1;
            hi1 = row.x + W - 1;
        }
        row = next;
        i = i_next;
        e = e_next;
        if (kGX) gx = raw_gapx(c, row.x + i);
    }
}

// The window sweep's shifts and bases: at step k (anti-diagonal d) those of d-1, from the maximum of d+1:
// base(d-1) - base(d) = max(d+1) - (base(d) - base(d+1)).
template <int NT>
__device__ __forceinline__ void column_window_shifts(const Ctx &c, const Window &Wn, ColumnWindowShared<NT> *ws) {
    const float *t = c.t;
    const int lane = threadIdx.x & 31;
    const int32_t steps = Wn.D - Wn.T;
    const bool ragged_end = Wn.at_end && c.R.ragged_right;
    float mxD = fmaxf(ragged_end ? (t[T_OX] + t[T_OY]) / 2.0f : t[T_MC],
                      fmaxf(ragged_end ? t[T_EX] : t[T_MFGX], ragged_end ? t[T_EY] : t[T_MFGY]));
    if (!(mxD > kNegInf)) mxD = 0.0f;
    float gamma = 0.0f;                  // base(d) - base(d+1)
    double bbase = 0.0;                  // base(d-1) of this window
    if (lane < 2) {                      // D and D-1
        *reinterpret_cast<float2 *>(&ws->row[lane].sh1) = make_float2(-gamma, -gamma - gamma);
        ws->bb[lane] = bbase;
    }
    bar_sync(kBarRow, NT + 64);
    for (int32_t k = 0; k < steps; ++k) {
        bar_sync(kBarRow, NT + 64);
        if (k == 0) continue;
        float m = part_max<NT / 32>(ws->part[(k + 1) & 1]);
        if (k == 1) m = mxD;
        const float g = (m > kNegInf ? m : 0.0f) - gamma;
        if (lane == 0) *reinterpret_cast<float2 *>(&ws->row[(k + 1) & 3].sh1) = make_float2(-g, -gamma - g);
        bbase += (double) g;
        if (lane == 0) ws->bb[(k + 1) & (kPostRows - 1)] = bbase;
        gamma = g;
    }
}

// The window sweep's copies: at step k the operands of the kAhead-th anti-diagonal below, and the place
// of the second (for the sweep and the posteriors).
template <int NT>
__device__ __forceinline__ void column_window_copies(const Ctx &c, const Window &Wn, const WindowTask &wt,
                                                     ColumnWindowShared<NT> *ws) {
    constexpr int NW = NT / 32;
    const Args &A = *c.A;
    const RegionDesc &R = c.R;
    const int lane = threadIdx.x & 31;
    const float2 *Ereg = A.E + R.cell_base + lane;
    const float *Freg = A.F + 3 * R.cell_base + lane;
    const int32_t D = Wn.D, T = Wn.T, from = Wn.from, steps = D - T;
    // a window whose T starts a forward segment reads that segment's own copy of T
    const float *Tside = A.use_side && wt.side >= 0
                             ? A.stitch_vals + A.stitch[wt.side].voff + 3 * A.stitch[wt.side].w0 + lane
                             : nullptr;
    RowStream<-1> info;
    info.open(&ws->info, A, R.diag_base, R.n, D, wt.first_cell + (raw_meta(A, R.diag_base, D, R.n).y & kWidthMask));
    auto issue = [&](int32_t k, const int4 &in) {
        if (k < steps) {
            const int32_t d = D - k, W = in.y & kWidthMask;
            const float2 *es = Ereg + in.z;
            const float *fd = Freg + 3 * (int64_t) in.z;
            float2 *ed = &ws->e[k & (kRows - 1)][lane];
            float *ff = &ws->f[k & (kRows - 1)][lane];
            const int32_t Wf = d <= from ? W : 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                if (lane + 32 * w < W) copy_async8(ed + 32 * w, es + 32 * w);
                if (lane + 32 * w < Wf) copy_async4(ff + 32 * w, fd + 32 * w);
            }
            if (Wf > 0 && (in.y & kFlagRefresh) != 0) {
                const int4 below = info.at(k + 1);
                const int32_t Wm = below.y & kWidthMask;
                const float *fm = Tside && d - 1 == T ? Tside : Freg + 3 * (int64_t) below.z;
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    const int i = lane + 32 * w;
                    if (i < W) {
                        copy_async4(&ws->ops[0][i], fd + W + 32 * w);
                        copy_async4(&ws->ops[1][i], fd + 2 * W + 32 * w);
                    }
                    if (i < Wm) {
                        copy_async4(&ws->ops[2][i], fm + 32 * w);
                        copy_async4(&ws->ops[3][i], fm + Wm + 32 * w);
                        copy_async4(&ws->ops[4][i], fm + 2 * Wm + 32 * w);
                    }
                }
            }
        }
        copy_commit();
    };
    auto place = [&](int32_t k) {
        const int4 in = info.at(k);
        const double fb = ws->info.base[k & (kInfoRows - 1)];
        if (lane == 0) {
            *reinterpret_cast<int2 *>(&ws->row[k & 3].xf) = make_int2(in.x, in.y | (D - k <= from ? kRowPost : 0));
            ws->post[k & (kPostRows - 1)] = make_int2(in.x, in.y & kWidthMask);
            ws->fb[k & (kPostRows - 1)] = fb;
        }
    };
#pragma unroll
    for (int k = 0; k < kAhead; ++k) issue(k, info.at(k));
    place(0);
    place(1);
    copy_wait<kAhead - 2>();
    int4 in = info.at(kAhead);
    bar_sync(kBarRow, NT + 64);
    for (int32_t k = 0; k < steps; ++k) {
        bar_sync(kBarRow, NT + 64);
        issue(k + kAhead, in);
        place(k + 2);
        info.advance(k);
        in = info.at(k + kAhead + 1);
        copy_wait<kAhead - 2>();         // every copy of d-2 and above has landed
    }
    copy_wait<0>();
}

// The window's total probabilities (one warp), a block's at a time.
template <int NT>
__device__ __forceinline__ void column_window_totals(const Window &Wn, ColumnWindowShared<NT> *ws) {
    const int lane = threadIdx.x & 31;
    const int32_t rows = Wn.from - Wn.T, blocks = (rows + kBlock - 1) / kBlock;
    for (int32_t q = 0; q < blocks; ++q) {
        const int b = q & 1;
        bar_sync(kBarFull + b, NT + 32);
        const int2 widths = ws->widths[b];
        const float2 ff = column_folds<NT / 32>(&ws->chain[b][0][0], widths.x, widths.y);
        const float2 th = ws->through[b];
        // the through-part is relative to base_F(d-1) + base_B(d+1)
        const float ptil = lac(ff.x, ff.y - th.x - th.y);
        const int32_t k0 = Wn.D - Wn.from + q * kBlock;   // the total's anti-diagonal
        if (lane == 0) ws->total[b] = (double) ptil + ws->fb[k0 & (kPostRows - 1)] + ws->bb[k0 & (kPostRows - 1)];
        __syncwarp();
        bar_arrive(kBarTotal + b, 64);
    }
}

// The window's posteriors and pairs (one warp): a block's anti-diagonals in the reference's order,
// descending, cells ascending.  Most of an anti-diagonal's cells are far below the threshold, so only
// the groups of 32 that hold one above it are looked at closely.
template <int NT>
__device__ __forceinline__ void column_window_post(const Ctx &c, const Window &Wn, const WindowTask &wt, int64_t gw,
                                                   ColumnWindowShared<NT> *ws) {
    const Args &A = *c.A;
    const RegionDesc &R = c.R;
    constexpr int NW = NT / 32;
    const int lane = threadIdx.x & 31;
    const int32_t rows = Wn.from - Wn.T, blocks = (rows + kBlock - 1) / kBlock;
    // a cell can only reach the threshold if its logarithm does
    const bool every = !(A.threshold > 0.0f);
    const float log_threshold = every ? kNegInf : logf(A.threshold) - 1e-3f;
    double ll = 0.0;
    int64_t n_out = 0;
    for (int32_t q = 0; q < blocks; ++q) {
        const int b = q & 1;
        bar_sync(kBarTotal + b, 64);
        const double pref = ws->total[b];
        const int32_t top = Wn.from - q * kBlock, k0 = Wn.D - top;   // the total's anti-diagonal
        if (top == R.n) ll = pref;
        const int m = min(kBlock, rows - q * kBlock);
        // lane j: what the block's j-th anti-diagonal needs
        const int32_t at_row = (k0 + lane) & (kPostRows - 1);
        const float kd_lane = lane < m ? (float) (ws->fb[at_row] + ws->bb[at_row] - pref) : 0.0f;
        const int2 row_lane = lane < m ? ws->post[at_row] : make_int2(0, 0);
        for (int j = 0; j < m; ++j) {
            const float kd = __shfl_sync(0xffffffffu, kd_lane, j);
            const int32_t xf = __shfl_sync(0xffffffffu, row_lane.x, j), W = __shfl_sync(0xffffffffu, row_lane.y, j);
            const int32_t d = top - j;
            const float *s = ws->s[b][j];
            unsigned mine = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                const int i = lane + 32 * w;
                const float v = s[(xf + i) & (NT - 1)] + kd;
                if (i < W && (v > log_threshold || every)) mine |= 1u << w;
            }
            for (unsigned groups = __reduce_or_sync(0xffffffffu, mine); groups; groups &= groups - 1) {
                const int i = lane + 32 * (__ffs(groups) - 1);
                const int32_t x = xf + i, y = d - x;
                const float p = __expf(s[x & (NT - 1)] + kd);
                const bool hit = i < W && x > 0 && y > 0 && p >= A.threshold;
                const unsigned bal = __ballot_sync(0xffffffffu, hit);
                if (hit) {
                    const int64_t at = n_out + __popc(bal & ((1u << lane) - 1u));
                    if (at < wt.out_cap) {
                        sa_aligned_pair o;
                        o.score = (int64_t) floor((double) fminf(p, 1.0f) * 10000000.0);
                        o.x = R.x1 + x - 1;
                        o.y = R.y1 + y - 1;
                        o.kmer = 0;      // filled in by the gather: a load here would hold the warp up
                        A.out[wt.out_base + at] = o;
                    } else {
                        atomicMax(A.status + R.read, (int32_t) SA_E_OUTPUT);
                    }
                }
                n_out += __popc(bal);
            }
        }
        __syncwarp();
        if (q + 2 < blocks) bar_arrive(kBarEmpty + b, NT + 32);
    }
    if (lane == 0) {
        A.wcount[gw] = n_out;
        if (Wn.at_end) A.loglik[c.region_index] = ll;
    }
    __syncwarp();
}

// ------------------------------------------------------------------------------------------------
// the persistent worker of column-resident batches
// ------------------------------------------------------------------------------------------------
// NT / 32 warps sweep, beside four helper warps.  The first claims are forward segments (longest
// first); once none is left, windows.
template <int NT, bool kSX, bool kGX, bool kFull>
__device__ __forceinline__ void column_forward(const Ctx &c, const Segment &sg, ColumnForwardShared<NT> *fs) {
    if (threadIdx.x < NT) column_forward_sweep<NT, kSX, kGX, kFull>(c, sg, fs);
    else if (threadIdx.x < NT + 32) column_forward_shifts<NT>(sg, fs);
    else if (threadIdx.x < NT + 64) column_forward_copies<NT>(c, sg, fs);
    else column_forward_results<NT>(c, sg, fs, (threadIdx.x - NT - 64) >> 5);
}

template <int NT, bool kSX, bool kGX, bool kFull>
__device__ __forceinline__ void column_window(const Ctx &c, ColumnWindowShared<NT> *ws, int64_t id) {
    const Window Wn = c.A->windows[id];
    const WindowTask wt = c.A->wtask[id];
    if (threadIdx.x < NT) column_window_sweep<NT, kSX, kGX, kFull>(c, Wn, ws);
    else if (threadIdx.x < NT + 32) column_window_shifts<NT>(c, Wn, ws);
    else if (threadIdx.x < NT + 64) column_window_copies<NT>(c, Wn, wt, ws);
    else if (threadIdx.x < NT + 96) column_window_totals<NT>(Wn, ws);
    else column_window_post<NT>(c, Wn, wt, id, ws);
}

template <int NT, int MINB, bool kFull>
__global__ void __launch_bounds__(NT + kHelpers, MINB) column_worker(const __grid_constant__ Args A) {
    ColumnShared<NT> *cs = reinterpret_cast<ColumnShared<NT> *>(column_smem);
    const int tid = threadIdx.x;
    if (tid < 16) {
        float4 c;
        log_add_piece((16 - tid) & 15, c);
        cs->la.hi[tid] = make_float2(c.x, c.y);
        cs->la.lo[tid] = make_float2(c.z, c.w);
    }
    // a thread outside the band adds whatever emission its slot holds to -inf: a number, not what a
    // kernel before this one left there (both unions' members have the ring in one place)
    for (int q = tid; q < kRows * NT; q += NT + kHelpers) (&cs->w.e[0][0])[q] = make_float2(0.0f, 0.0f);
    for (;;) {
        if (tid == 0) {
            const unsigned claim = atomicAdd(&A.ctl->claim, 1u);
            cs->task = claim < (unsigned) A.n_segs ? A.order[claim] : -1;
        }
        __syncthreads();
        const int32_t id = cs->task;
        if (id < 0) break;
        const Segment sg = A.segs[id];
        Ctx c;
        ctx_init(c, A, sg.region);
        const bool sx = c.t[T_SX] > kNegInf;
        if (c.gx_uniform) {
            if (sx) column_forward<NT, true, false, kFull>(c, sg, &cs->f);
            else column_forward<NT, false, false, kFull>(c, sg, &cs->f);
        } else {
            if (sx) column_forward<NT, true, true, kFull>(c, sg, &cs->f);
            else column_forward<NT, false, true, kFull>(c, sg, &cs->f);
        }
        __syncthreads();
    }
    __syncthreads();
    for (;;) {
        if (tid == 0) {
            const unsigned claim = atomicAdd(&A.ctl->wclaim, 1u);
            cs->task = (int64_t) claim < A.n_windows ? wait_ready(A, claim) : -1;
        }
        __syncthreads();
        const int32_t id = cs->task;
        if (id < 0) break;
        Ctx c;
        ctx_init(c, A, A.wtask[id].region);
        const bool sx = c.t[T_SX] > kNegInf;
        if (c.gx_uniform) {
            if (sx) column_window<NT, true, false, kFull>(c, &cs->w, id);
            else column_window<NT, false, false, kFull>(c, &cs->w, id);
        } else {
            if (sx) column_window<NT, true, true, kFull>(c, &cs->w, id);
            else column_window<NT, false, true, kFull>(c, &cs->w, id);
        }
        // the posteriors' warp wrote the window's pairs and counts
        if (tid >= NT + 96) read_unit_done<32>(A, c.R.read, tid & 31, nullptr);
        __syncthreads();
    }
}

}  // namespace fp32
}  // namespace sa
