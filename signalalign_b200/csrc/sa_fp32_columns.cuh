// Column-resident form of the batched FP32 worker, for bands up to column_span(NC) columns: a CTA per
// forward segment (a column per thread), a warp per traceback window (NC columns per lane).
//
// Why.  The recursion is bound by the latency of its chain of logAdds and by instruction issue, not by
// memory.  With cells spread by their place in the band and exchanged through a shared-memory ring,
// most instructions were not arithmetic: ring addresses, clamps, stores and loads, a look-ahead
// address per operand (24 warp instructions per band cell, issue 19 to 30 % busy).
//
// How.  Matrix column x lives in slot x mod 128, whichever way the band moves.  A cell's neighbours are
// then in the same slot (the same column) or in the one beside it (column x - 1 forward, x + 1
// backward): two or three shuffles an anti-diagonal, no ring.  Slots outside the band hold -inf, which
// makes every absent neighbour drop out of logAdd.  Three anti-diagonals' columns never share a slot:
// the host takes this path for a batch only if any three consecutive anti-diagonals span at most
// column_span(NC) columns, so the NC - 1 slots before an anti-diagonal's first column are always
// outside it, and a lane's cells are consecutive elements of each store, addressed from one place.
//
// The arithmetic is that of ForwardSweep and window_task, operation for operation, so the values are
// theirs bit for bit.  Measured on B200, the worker of 8 reads of 8 to 12 kb (2.1e7 cells, 71
// segments): 3.52 -> 2.35 ms; of 30 reads of 8 to 30 kb (1.5e8 cells): 5.36 -> 3.85 ms.  One warp per
// forward segment (NC columns a lane) was slower than the form before it: 5.0 ms on the 8 reads.
#pragma once

namespace sa {
namespace fp32 {

// NC columns per lane: 32 NC slots, bands up to column_span(NC) columns
__host__ __device__ constexpr int column_slots(int nc) { return 32 * nc; }
__host__ __device__ constexpr int column_span(int nc) { return 31 * nc; }


extern __shared__ float4 column_smem[];

// lae() with the table at the start of shared memory.  C - 2 d rounded down, C a multiple of 16 large
// enough that the last place is 1/16, holds -ceil(2 d) mod 16 in bits 4..7: the byte offset of the
// piece, without a shift.  The cut-off is a predicated add.
__device__ __forceinline__ float lac(float x, float y) {
    float mx = fmaxf(x, y);
    const float d = fabsf(x - y);
    const int k = __float_as_int(__fmaf_rd(d, -2.0f, 786432.0f)) & 0xf0;
    const float4 c = *reinterpret_cast<const float4 *>(reinterpret_cast<const char *>(column_smem) + k);
    const float h = fmaf(fmaf(fmaf(c.x, d, c.y), d, c.z), d, c.w);
    asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, 0f40F00000;\n\t@p add.rn.f32 %0, %0, %2;\n\t}"
        : "+f"(mx) : "f"(d), "f"(h));
    return mx;
}

// the element of a lane's first slot on an anti-diagonal whose first column is xf: slots r = 0..3
// hold cells j + r (negative, or at least the width: outside the band)
template <int NC>
__device__ __forceinline__ int32_t first_cell_of_lane(int lane, int32_t xf) {
    return ((NC * lane - (xf & ~(NC - 1))) & (column_slots(NC) - 1)) - (xf & (NC - 1));
}

__device__ __forceinline__ bool cell_in(int32_t j, int r, int32_t W) { return (uint32_t) (j + r) < (uint32_t) W; }

// skip emissions of a lane's columns: the machine's one value, or per column
template <int NC, bool kGX>
struct Skip {
    float v[kGX ? NC : 1];
    __device__ __forceinline__ float operator[](int r) const { return v[kGX ? r : 0]; }
    // columns x0 .. x0 + 3
    __device__ __forceinline__ void load(const Ctx &c, int32_t x0) {
        if (!kGX) {
            v[0] = c.gx;
            return;
        }
#pragma unroll
        for (int r = 0; r < NC; ++r) v[kGX ? r : 0] = raw_gapx(c, x0 + r);
    }
};

// ------------------------------------------------------------------------------------------------
// forward sweep of one segment by a CTA: a column per thread
// ------------------------------------------------------------------------------------------------
// The sweep is a chain of dependent anti-diagonals, so its latency is what counts.  Thread t holds the
// column x with x mod 128 == t.  The recursion needs the column to the left on d-1 (for gap-X) and on
// d-2 (for the match, so a step early), and its own column on d-1 (gap-Y): the left column comes by
// shuffle, across a warp's edge through one shared float4, and only gap-X sits between one
// anti-diagonal's barrier and the next.  Emissions and band facts come in groups of kGroup
// anti-diagonals, a whole group ahead: waits on loads are then for loads of a group ago, not for the
// newest ones (a warp waits for all of its loads that share a scoreboard).
constexpr int kGroup = 4;

struct ColumnForwardShared {
    float4 edge[2][kWarps];             // match, gap-X, gap-Y of a warp's last column, by parity of d
    float part[2][kWarps];              // the warps' largest values, by parity of d
};

template <bool kSX, bool kGX>
struct ColumnForward {
    const Ctx &c;
    const Args &A;
    const RegionDesc &R;
    const Segment &S;
    ColumnForwardShared *fs;
    int tid, lane, warp;
    int64_t db;
    int32_t n, dbeg, dend;
    const float2 *Ereg;
    float *Freg;
    float M1, X1, Y1;             // own column on d-1
    float lM2, lX2, lY2;          // left column on d-2
    float2 e[kGroup], e_next[kGroup];
    float g[kGX ? kGroup : 1], g_next[kGX ? kGroup : 1];
    int2 m[kGroup], m_next[kGroup];   // raw band facts of this group and the next
    int32_t off, off_next;        // first cell of d, and of the next group's first anti-diagonal
    int32_t cap;                  // next anti-diagonal whose values a stitch takes
    float mxw;                    // this warp's largest value on d-1
    float delta0, delta1;         // delta(d) = base(d) - base(d-1), delta(d-1)
    double base0;                 // base(d)
    double qbase;                 // lane q of warp 0: base and shift of the last d with d mod 32 == q
    float qshift;
    int32_t wi;

    __device__ __forceinline__ ColumnForward(const Ctx &cc, const Segment &sg, ColumnForwardShared *f)
        : c(cc), A(*cc.A), R(cc.R), S(sg), fs(f) {}

    __device__ __forceinline__ int32_t cell_of(int32_t d, int2 mt) const {
        return (tid - ((d + mt.x) >> 1)) & (kThreads - 1);
    }

    // band facts of dd .. dd + kGroup - 1
    __device__ __forceinline__ void fetch_meta(int32_t dd, int2 (&o)[kGroup]) const {
#pragma unroll
        for (int k = 0; k < kGroup; ++k) o[k] = raw_meta(A, db, dd + k, n);
    }

    // emissions of dd .. dd + kGroup - 1 (band facts mt, first cell o of dd); returns the first cell after
    __device__ __forceinline__ int32_t fetch(int32_t dd, const int2 (&mt)[kGroup], int32_t o, float2 (&ee)[kGroup],
                                             float (&gg)[kGX ? kGroup : 1]) const {
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
            const int32_t i = cell_of(dd + k, mt[k]);
            ee[k] = __ldg(Ereg + o + i);
            if (kGX) gg[kGX ? k : 0] = raw_gapx(c, ((dd + k + mt[k].x) >> 1) + i);
            o += dd + k <= n ? mt[k].y & kWidthMask : 0;
        }
        return o;
    }

    // the values of d-1 (own column) and the largest values go out, then d is computed; k: d's place
    // in its group, Q: the parity of d
    template <int K, int Q>
    __device__ __forceinline__ void step(int32_t d) {
        const float *t = c.t;
        const int32_t W = m[K].y & kWidthMask, flags = m[K].y & ~kWidthMask;
        const int32_t i = cell_of(d, m[K]);
        const bool in = i < W;
        // d-1 to the right-hand neighbours (Q ^ 1: its parity)
        if (lane == 31) fs->edge[Q ^ 1][warp] = make_float4(M1, X1, Y1, 0.0f);
        if (lane == 0) fs->part[Q ^ 1][warp] = mxw;
        // meanwhile what does not depend on them: match and gap-Y of d
        const float shL = -delta0, shM = -delta1 - delta0;
        float vM = lac(lM2 + t[T_MC], lX2 + t[T_MFGX]);
        vM = lac(vM, lY2 + t[T_MFGY]) + (e[K].x + shM);
        float vY = lac(M1 + t[T_OY], Y1 + t[T_EY]) + (e[K].y + shL);
        float lM = __shfl_up_sync(0xffffffffu, M1, 1), lX = __shfl_up_sync(0xffffffffu, X1, 1),
              lY = __shfl_up_sync(0xffffffffu, Y1, 1);
        // shift of d+1 from the maximum of d-2 (its parity is d's; complete since the last barrier)
        float delta_next = 0.0f;
        if (d >= 2) {
            const float4 fp = *reinterpret_cast<const float4 *>(fs->part[Q]);
            const float mx = fmaxf(fmaxf(fp.x, fp.y), fmaxf(fp.z, fp.w));
            delta_next = ((mx > kNegInf ? mx : 0.0f) - delta0) - delta1;
        }
        __syncthreads();
        const float4 ed = fs->edge[Q ^ 1][(warp + kWarps - 1) & (kWarps - 1)];
        if (lane == 0) {
            lM = ed.x;
            lX = ed.y;
            lY = ed.z;
        }
        float vX = lac(lM + t[T_OX], lX + t[T_EX]);
        if (kSX) vX = lac(vX, lY + t[T_SX]);
        vX = vX + ((kGX ? g[kGX ? K : 0] : c.gx) + shL);
        vM = in ? vM : kNegInf;
        vX = in ? vX : kNegInf;
        vY = in ? vY : kNegInf;
        const bool own = d > dbeg;
        if (in && own) {
            float *Fd = Freg + 3 * (int64_t) off + i;
            Fd[0] = vM;
            if (flags & kFlagStoreGaps) {
                Fd[W] = vX;
                Fd[2 * W] = vY;
            }
        }
        mxw = warp_max1(fmaxf(vM, fmaxf(vX, vY)));
        // base and shift of d: lane d mod 32 of warp 0 keeps them and the warp writes them out 32 at a
        // time and before a window is published (its backward sweep reads them)
        const bool window_end = own && (flags & kFlagWindowEnd) != 0;
        const int q = d & 31;
        if (lane == q) {
            qbase = base0;
            qshift = delta0;
        }
        if (q == 31 || window_end || d == dend) {
            if (warp == 0 && lane <= q && d - q + lane > dbeg) {
                A.base[db + (d - q) + lane] = qbase;
                A.fshift[db + (d - q) + lane] = qshift;
            }
            if (window_end) {
                __threadfence();   // this anti-diagonal and all before it, device-wide
                __syncthreads();
                if (tid == 0) {
                    const unsigned at = atomicAdd(&A.ctl->pub, 1u);
                    if ((int64_t) at < A.n_windows) atomicExch(A.ready + at, (int32_t) (R.win_base + wi));
                }
                ++wi;
            }
        }
        off += W;
        lM2 = lM;
        lX2 = lX;
        lY2 = lY;
        M1 = vM;
        X1 = vX;
        Y1 = vY;
        delta1 = delta0;
        delta0 = delta_next;
        base0 += (double) delta_next;
        if (d == cap) cap = capture(d, i, in);
    }

    // the values of d (now M1, X1, Y1) to their side of a stitch: called on b-1 and on b, where the
    // segment begins or ends; base0 and delta0 / delta1 already describe d+1.  Returns the next such d.
    __device__ __forceinline__ int32_t capture(int32_t d, int32_t i, bool in) const {
        const bool in_side = S.stitch_in >= 0 && d <= dbeg;
        const int32_t si = in_side ? S.stitch_in : S.stitch_out, b = in_side ? dbeg : dend;
        const StitchDesc sd = A.stitch[si];
        float *o = A.stitch_vals + sd.voff + (in_side ? 0 : 3 * (sd.w0 + sd.w1)) + (d == b ? 3 * sd.w0 : 0) + i;
        const int32_t W = d == b ? sd.w1 : sd.w0;
        if (in) {
            o[0] = M1;
            o[W] = X1;
            o[2 * W] = Y1;
        }
        if (d == b && tid == 0) {
            const double base_b = base0 - (double) delta0, base_b1 = base_b - (double) delta1;
            double *bs = in_side ? A.stitch_res[si].sbase : A.stitch_res[si].tbase;
            bs[0] = base_b1;
            bs[1] = base_b;
        }
        return d < b ? b : (in_side && S.stitch_out >= 0 ? dend - 1 : INT32_MAX);
    }

    __device__ __forceinline__ void run(Shared *sh) {
        tid = threadIdx.x;
        lane = tid & 31;
        warp = tid >> 5;
        db = R.diag_base;
        n = R.n;
        dbeg = S.d_begin;
        dend = S.d_end;
        const int32_t s = dbeg - S.warm + (dbeg == 0 ? 1 : 0);
        Ereg = A.E + R.cell_base;
        Freg = A.F + 3 * R.cell_base;
        off = (int32_t) S.cell0;
        M1 = X1 = Y1 = lM2 = lX2 = lY2 = kNegInf;
        // steps run in pairs of parities 0 and 1 (of d - s): s-1 has parity 1, s-2 parity 0
        if (dbeg == 0) {
            // anti-diagonal 0: startStateProb / raggedStartStateProb (stateMachine.c:1022-1032), column 0
            const float s0 = R.ragged_left ? kNegInf : 0.0f, s1 = R.ragged_left ? 0.0f : kNegInf;
            if (tid == 0) {
                M1 = s0;
                X1 = Y1 = s1;
                Freg[ST_M] = s0;
                Freg[ST_X] = s1;
                Freg[ST_Y] = s1;
                A.base[db] = 0.0;
                A.fshift[db] = 0.0f;
            }
            mxw = warp == 0 ? fmaxf(s0, s1) : kNegInf;
        } else {
            // a later segment: every band cell of s-2 and s-1 starts at 0
            const int2 r2 = raw_meta(A, db, s - 2, n), r1 = raw_meta(A, db, s - 1, n);
            if (cell_of(s - 1, r1) < (r1.y & kWidthMask)) M1 = X1 = Y1 = 0.0f;
            if (((cell_of(s - 2, r2) - 1) & (kThreads - 1)) < (r2.y & kWidthMask)) lM2 = lX2 = lY2 = 0.0f;
            mxw = 0.0f;
        }
        if (lane == 0) fs->part[0][warp] = 0.0f;   // maximum of s-2, where there is one
        fetch_meta(s, m);
        off_next = fetch(s, m, off, e, g);
        fetch_meta(s + kGroup, m_next);
        // renormalisation as in ForwardSweep: base(d+1) = base(d-2) + max(d-2)
        delta0 = delta1 = 0.0f;
        base0 = 0.0;
        qbase = 0.0;
        qshift = 0.0f;
        wi = S.wi0;
        cap = S.stitch_in >= 0 ? dbeg - 1 : (S.stitch_out >= 0 ? dend - 1 : INT32_MAX);
        __syncthreads();
        for (int32_t d = s; d <= dend; d += kGroup) {
            off_next = fetch(d + kGroup, m_next, off_next, e_next, g_next);
            int2 m_after[kGroup];
            fetch_meta(d + 2 * kGroup, m_after);
            step<0, 0>(d);
            if (d + 1 > dend) break;
            step<1, 1>(d + 1);
            if (d + 2 > dend) break;
            step<2, 0>(d + 2);
            if (d + 3 > dend) break;
            step<3, 1>(d + 3);
#pragma unroll
            for (int k = 0; k < kGroup; ++k) {
                e[k] = e_next[k];
                if (kGX) g[kGX ? k : 0] = g_next[kGX ? k : 0];
                m[k] = m_next[k];
                m_next[k] = m_after[k];
            }
        }
        if (S.stitch_in >= 0) stitch_arrive(A, sh, S.stitch_in);
        if (S.stitch_out >= 0) stitch_arrive(A, sh, S.stitch_out);
        __syncthreads();
    }
};

// ------------------------------------------------------------------------------------------------
// the two ordered folds of a refresh
// ------------------------------------------------------------------------------------------------
// ordered_fold2 on chain[0..na) and chain[128..128 + nb), with the same result: half the warp folds
// each, and of the values after the first largest one only those within the 7.5 cut-off of it are
// folded (the running result is at least the largest value by then, so logAdd returns it unchanged
// for any other).
template <int NC>
__device__ __forceinline__ float2 column_folds(float *chain, int na, int nb) {
    const int lane = threadIdx.x & 31;
    float va[NC], vb[NC];
    float ma = kNegInf, mb = kNegInf;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const int i = lane + 32 * k;
        va[k] = i < na ? chain[i] : kNegInf;
        vb[k] = i < nb ? chain[column_slots(NC) + i] : kNegInf;
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
        if (ib) chain[column_slots(NC) + cb + __popc(b & below)] = vb[k];
        ca += __popc(a);
        cb += __popc(b);
    }
    __syncwarp();
    const bool second = lane >= 16;
    const int mine = second ? cb : ca, most = max(ca, cb);
    const float *list = chain + (second ? column_slots(NC) : 0);
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
// backward sweep of one traceback window by one warp, posteriors fused
// ------------------------------------------------------------------------------------------------
// A successor's value plus its emission is summed in the successor's own slot and then shifted by one
// column, so an anti-diagonal takes two shuffles.  Emissions and forward values come through shared
// memory, copied asynchronously kAhead anti-diagonals ahead by the lane that reads them (lane-private
// slots, one group of copies per anti-diagonal), so the wait is for copies that old, and no register
// holds an operand that is not in use.  Band facts and bases come 32 anti-diagonals at a time, a lane
// each.
constexpr int kAhead = 5;                // anti-diagonals between a copy and its first use
constexpr int kRows = 8;                 // rows of the copy ring: d + 2 .. d - kAhead

template <int NC>
struct WindowShared {
    float2 e[kRows][NC][32];            // emissions, row d mod kRows, by register and lane
    float f[kRows][NC][32];             // forward match values
    float ops[5][NC][32];               // the next refresh: gap-X, gap-Y of d, match, gap-X, gap-Y of d-1
    int4 info[64];                      // row d mod 64: first column, width | flags, first cell, shift
    double base[64];                    // forward base
    float chain[2 * 32 * NC];           // terms of the two folds
};

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

template <int NC, bool kSX, bool kGX>
struct ColumnWindow {
    const Ctx &c;
    const Args &A;
    const RegionDesc &R;
    WindowShared<NC> *ws;
    int lane;
    int32_t D, T, from;
    const float2 *Ereg;
    const float *Freg, *Tside;
    float vM1[NC], vX1[NC], vY1[NC], vM2[NC];   // backward values of d+1, and match of d+2
    int32_t j1, W1;               // the lane's first cell and the width on d+1
    int32_t xf1;                  // first column of d+1
    int2 raw;                     // band facts, base and shift of the next block of 32, a lane each
    double raw_base;
    float raw_shift;
    int32_t block_top;            // first cell past the next block
    float mx1, mx2, gamma1;
    double bbase, pref;
    int64_t n_out;

    __device__ __forceinline__ ColumnWindow(const Ctx &cc, WindowShared<NC> *w) : c(cc), A(*cc.A), R(cc.R), ws(w) {}

    // band facts and bases of anti-diagonals 32 b + lane
    __device__ __forceinline__ void load_block(int32_t b) {
        const int32_t d = clampi(32 * b + lane, 0, R.n);
        raw = __ldg(A.meta + R.diag_base + d);
        raw_base = __ldcg(A.base + R.diag_base + d);
        raw_shift = __ldcg(A.fshift + R.diag_base + d);
    }

    // the loaded block b becomes readable (anti-diagonals up to `last` of it) and the one below loads
    __device__ __forceinline__ void open_block(int32_t b, int32_t last) {
        const int32_t d = 32 * b + lane, W = d <= last ? raw.y & kWidthMask : 0;
        int32_t sum = W;   // widths of d and the block's later anti-diagonals
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t v = __shfl_down_sync(0xffffffffu, sum, o);
            if (lane + o < 32) sum += v;
        }
        ws->info[d & 63] = make_int4((d + raw.x) >> 1, raw.y, block_top - sum, __float_as_int(raw_shift));
        ws->base[d & 63] = raw_base;
        block_top -= __shfl_sync(0xffffffffu, sum, 0);
        __syncwarp();
        if (b > 0) load_block(b - 1);
    }

    // copies of anti-diagonal d: emissions, forward values, and a refresh's other operands
    __device__ __forceinline__ void issue(int32_t d) {
        if (d > T) {
            if ((d & 31) == 0) open_block((d >> 5) - 1, INT32_MAX);
            const int4 in = ws->info[d & 63];
            const int32_t j = first_cell_of_lane<NC>(lane, in.x), W = in.y & kWidthMask;
            const float2 *es = Ereg + (in.z + j);
            float2(*ed)[32] = ws->e[d & (kRows - 1)];
#pragma unroll
            for (int r = 0; r < NC; ++r) copy_async8(&ed[r][lane], es + r);
            if (d <= from) {
                // only the band's cells: what lies past an anti-diagonal may not be written yet
                const float *fs = Freg + (3 * (int64_t) in.z + j);
                float(*fd)[32] = ws->f[d & (kRows - 1)];
#pragma unroll
                for (int r = 0; r < NC; ++r)
                    if (cell_in(j, r, W)) copy_async4(&fd[r][lane], fs + r);
                if ((in.y & kFlagRefresh) != 0) {
                    const int4 below = ws->info[(d - 1) & 63];
                    const int32_t jm = first_cell_of_lane<NC>(lane, below.x), Wm = below.y & kWidthMask;
                    const float *fm = (Tside && d - 1 == T ? Tside : Freg + 3 * (int64_t) below.z) + jm;
#pragma unroll
                    for (int r = 0; r < NC; ++r) {
                        if (cell_in(j, r, W)) {
                            copy_async4(&ws->ops[0][r][lane], fs + W + r);
                            copy_async4(&ws->ops[1][r][lane], fs + 2 * W + r);
                        }
                        if (cell_in(jm, r, Wm)) {
                            copy_async4(&ws->ops[2][r][lane], fm + r);
                            copy_async4(&ws->ops[3][r][lane], fm + Wm + r);
                            copy_async4(&ws->ops[4][r][lane], fm + 2 * Wm + r);
                        } else {
                            ws->ops[2][r][lane] = ws->ops[3][r][lane] = ws->ops[4][r][lane] = kNegInf;
                        }
                    }
                }
            }
        }
        copy_commit();
    }

    // Total probability through anti-diagonal d (diagonalCalculationTotalProbability,
    // pairwiseAligner.c:1182-1200): F.B on d in ascending cell order, then the matches from d-1 over d
    // into d+1 dotted with B(d+1), relative to base_F(d) + base_B(d).  f, bM, bX, bY: forward match
    // and backward values of d (first cell j, width W).
    __device__ __forceinline__ float refresh(int32_t d, int32_t j, int32_t W, const float (&f)[NC], const float (&bM)[NC],
                                             const float (&bX)[NC], const float (&bY)[NC], float shift, float gamma0) {
        const float *t = c.t;
        const bool have_next = d < D;
        const float2(*en)[32] = ws->e[(d + 1) & (kRows - 1)];
        const int left = (lane + 31) & 31;
        float m = __shfl_sync(0xffffffffu, ws->ops[2][NC - 1][lane], left);
        float x = __shfl_sync(0xffffffffu, ws->ops[3][NC - 1][lane], left);
        float y = __shfl_sync(0xffffffffu, ws->ops[4][NC - 1][lane], left);
#pragma unroll
        for (int r = 0; r < NC; ++r) {
            float v = f[r] + bM[r];
            v = lac(v, ws->ops[0][r][lane] + bX[r]);
            v = lac(v, ws->ops[1][r][lane] + bY[r]);
            if (cell_in(j, r, W)) ws->chain[j + r] = v;
            const float em = en[r][lane].x;
            float th = m + (em + t[T_MC]);
            th = lac(th, x + (em + t[T_MFGX]));
            th = lac(th, y + (em + t[T_MFGY]));
            if (have_next && cell_in(j1, r, W1)) ws->chain[column_slots(NC) + j1 + r] = th + vM1[r];
            m = ws->ops[2][r][lane];
            x = ws->ops[3][r][lane];
            y = ws->ops[4][r][lane];
        }
        __syncwarp();
        const float2 ff = column_folds<NC>(ws->chain, W, have_next ? W1 : 0);
        // the through-part is relative to base_F(d-1) + base_B(d+1)
        return lac(ff.x, ff.y - shift - gamma0);
    }

    // pairs of anti-diagonal d in ascending cell order (the reference's): the lanes rotated so that
    // the one with the first column comes first
    __device__ __forceinline__ void emit(int32_t d, int32_t xf, int32_t j, int32_t W, const float (&s)[NC],
                                         const WindowTask &wt) {
        const int first = (xf / NC) & 31;
        unsigned b[NC], hits = 0;
        float p[NC];
#pragma unroll
        for (int r = 0; r < NC; ++r) {
            const int32_t x = xf + j + r, y = d - x;
            p[r] = __expf(s[r]);
            const bool hit = cell_in(j, r, W) && x > 0 && y > 0 && p[r] >= A.threshold;
            hits |= hit ? 1u << r : 0u;
            const unsigned v = __ballot_sync(0xffffffffu, hit);
            b[r] = __funnelshift_r(v, v, first);
        }
        const unsigned below = (1u << ((lane - first) & 31)) - 1u;
        int64_t q = n_out;
#pragma unroll
        for (int r = 0; r < NC; ++r) q += __popc(b[r] & below);
        if (hits) {
#pragma unroll
            for (int r = 0; r < NC; ++r) {
                if (!((hits >> r) & 1u)) continue;
                const int32_t x = xf + j + r, y = d - x;
                if (q < wt.out_cap) {
                    sa_aligned_pair o;
                    o.score = (int64_t) floor((double) fminf(p[r], 1.0f) * 10000000.0);
                    o.x = R.x1 + x - 1;
                    o.y = R.y1 + y - 1;
                    o.kmer = __ldg(A.kmer + R.kmer_base + x - 1);   // 1 <= x <= lX for a pair
                    A.out[wt.out_base + q] = o;
                } else {
                    atomicMax(A.status + R.read, (int32_t) SA_E_OUTPUT);
                }
                ++q;
            }
        }
#pragma unroll
        for (int r = 0; r < NC; ++r) n_out += __popc(b[r]);
    }

    __device__ __forceinline__ void run(int64_t gw) {
        lane = threadIdx.x & 31;
        Ereg = A.E + R.cell_base;
        Freg = A.F + 3 * R.cell_base;
        const Window Wn = A.windows[gw];
        const WindowTask wt = A.wtask[gw];
        D = Wn.D;
        T = Wn.T;
        from = Wn.from;
        // a window whose T starts a forward segment reads that segment's own copy of T
        Tside = A.use_side && wt.side >= 0 ? A.stitch_vals + A.stitch[wt.side].voff + 3 * A.stitch[wt.side].w0 : nullptr;
        // a cell can only reach the threshold if its logarithm does
        const float log_threshold = A.threshold > 0.0f ? logf(A.threshold) - 1e-3f : kNegInf;
        const float *t = c.t;
        // end-state values on D (stateMachine.c:1034-1061)
        const bool ragged_end = Wn.at_end && R.ragged_right;
        const float e0 = ragged_end ? (t[T_OX] + t[T_OY]) / 2.0f : t[T_MC];
        const float e1 = ragged_end ? t[T_EX] : t[T_MFGX];
        const float e2 = ragged_end ? t[T_EY] : t[T_MFGY];
        float mxD = fmaxf(e0, fmaxf(e1, e2));
        if (!(mxD > kNegInf)) mxD = 0.0f;
        __syncwarp();   // the warp's previous window has read its shared memory
#pragma unroll
        for (int r = 0; r < NC; ++r) {
            vM1[r] = vX1[r] = vY1[r] = vM2[r] = kNegInf;
            ws->e[(D + 1) & (kRows - 1)][r][lane] = ws->e[(D + 2) & (kRows - 1)][r][lane] = make_float2(0.0f, 0.0f);
        }
        load_block(D >> 5);
        block_top = wt.first_cell + (__shfl_sync(0xffffffffu, raw.y, D & 31) & kWidthMask);
        open_block(D >> 5, D);
#pragma unroll
        for (int k = 0; k < kAhead; ++k) issue(D - k);
        j1 = W1 = xf1 = 0;
        mx1 = mx2 = kNegInf;
        gamma1 = 0.0f;
        bbase = pref = 0.0;
        double ll = 0.0;
        n_out = 0;
#pragma unroll 1
        for (int32_t d = D; d > T; --d) {
            issue(d - kAhead);
            copy_wait<kAhead>();   // every copy of d and above has landed
            const int4 in = ws->info[d & 63];
            const int32_t xf = in.x, W = in.y & kWidthMask;
            const int32_t j = first_cell_of_lane<NC>(lane, xf);
            float gamma0 = 0.0f;           // base(d) - base(d+1) = max(d+2) - gamma1
            if (d <= D - 2) gamma0 = (mx2 > kNegInf ? mx2 : 0.0f) - gamma1;
            bbase += (double) gamma0;
            float bM[NC], bX[NC], bY[NC];
            float mx0;
            if (d == D) {
#pragma unroll
                for (int r = 0; r < NC; ++r) {
                    const bool inb = cell_in(j, r, W);
                    bM[r] = inb ? e0 : kNegInf;
                    bX[r] = inb ? e1 : kNegInf;
                    bY[r] = inb ? e2 : kNegInf;
                }
                mx0 = mxD;
            } else {
                const float shU = -gamma0, shM = -gamma1 - gamma0;
                const float2(*ep)[32] = ws->e[(d + 2) & (kRows - 1)], (*eu)[32] = ws->e[(d + 1) & (kRows - 1)];
                Skip<NC, kGX> g;
                g.load(c, xf1 + j1);
                float me[NC + 1], le[NC + 1];
#pragma unroll
                for (int r = 0; r < NC; ++r) {
                    me[r] = vM2[r] + (ep[r][lane].x + shM);
                    le[r] = vX1[r] + (g[r] + shU);
                }
                const int right = (lane + 1) & 31;
                me[NC] = __shfl_sync(0xffffffffu, me[0], right);
                le[NC] = __shfl_sync(0xffffffffu, le[0], right);
                float lm = kNegInf;
#pragma unroll
                for (int r = 0; r < NC; ++r) {
                    float m = me[r + 1] + t[T_MC];
                    float x = me[r + 1] + t[T_MFGX];
                    float y = me[r + 1] + t[T_MFGY];
                    const float ue = vY1[r] + (eu[r][lane].y + shU);
                    m = lac(m, ue + t[T_OY]);
                    y = lac(y, ue + t[T_EY]);
                    m = lac(m, le[r + 1] + t[T_OX]);
                    x = lac(x, le[r + 1] + t[T_EX]);
                    if (kSX) y = lac(y, le[r + 1] + t[T_SX]);
                    const bool inb = cell_in(j, r, W);
                    bM[r] = inb ? m : kNegInf;
                    bX[r] = inb ? x : kNegInf;
                    bY[r] = inb ? y : kNegInf;
                    lm = fmaxf(lm, fmaxf(bM[r], fmaxf(bX[r], bY[r])));
                }
                mx0 = warp_max1(lm);
            }
            if (d <= from) {
                float f[NC];
#pragma unroll
                for (int r = 0; r < NC; ++r) f[r] = ws->f[d & (kRows - 1)][r][lane];
                const double fb = ws->base[d & 63];
                if ((in.y & kFlagRefresh) != 0) {
                    pref = (double) refresh(d, j, W, f, bM, bX, bY, __int_as_float(in.w), gamma0) + fb + bbase;
                    if (d == R.n) ll = pref;
                }
                const float kd = (float) (fb + bbase - pref);
                float s[NC], top = kNegInf;
#pragma unroll
                for (int r = 0; r < NC; ++r) {
                    s[r] = f[r] + bM[r] + kd;
                    top = fmaxf(top, s[r]);
                }
                if (__any_sync(0xffffffffu, top > log_threshold || A.threshold <= 0.0f)) emit(d, xf, j, W, s, wt);
            }
            mx2 = mx1;
            mx1 = mx0;
            gamma1 = gamma0;
            j1 = j;
            W1 = W;
            xf1 = xf;
#pragma unroll
            for (int r = 0; r < NC; ++r) {
                vM2[r] = vM1[r];
                vM1[r] = bM[r];
                vX1[r] = bX[r];
                vY1[r] = bY[r];
            }
        }
        copy_wait<0>();
        if (lane == 0) {
            A.wcount[gw] = n_out;
            if (Wn.at_end) A.loglik[c.region_index] = ll;
        }
        __syncwarp();
    }
};

// ------------------------------------------------------------------------------------------------
// the persistent worker of column-resident batches
// ------------------------------------------------------------------------------------------------
struct alignas(16) ColumnShared {
    float4 la[16];                      // logAdd cubic pieces, indexed by -ceil(2 d) mod 16
    ColumnForwardShared fs;
    Shared sh;                          // the segments' claims and stitch checks
};

// The first claims are forward segments (longest first), one per CTA; once none is left, each warp
// claims windows.
template <bool kSX, bool kGX>
__device__ __forceinline__ void column_forward(const Ctx &c, const Segment &sg, ColumnForwardShared *fs, Shared *sh) {
    ColumnForward<kSX, kGX> f(c, sg, fs);
    f.run(sh);
}

template <int NC, bool kSX, bool kGX>
__device__ __forceinline__ void column_window(const Ctx &c, WindowShared<NC> *ws, int64_t id) {
    ColumnWindow<NC, kSX, kGX> w(c, ws);
    w.run(id);
}

template <int NC, int MINB>
__global__ void __launch_bounds__(kThreads, MINB) column_worker(const __grid_constant__ Args A) {
    ColumnShared *cs = reinterpret_cast<ColumnShared *>(column_smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid < 16) {
        log_add_piece((16 - tid) & 15, cs->la[tid]);
    }
    for (;;) {
        if (tid == 0) {
            const unsigned claim = atomicAdd(&A.ctl->claim, 1u);
            cs->sh.task_id = claim < (unsigned) A.n_segs ? A.order[claim] : -1;
        }
        __syncthreads();
        const int32_t id = cs->sh.task_id;
        if (id < 0) break;
        const Segment sg = A.segs[id];
        Ctx c;
        ctx_init(c, A, sg.region);
        const bool sx = c.t[T_SX] > kNegInf;
        if (c.gx_uniform) {
            if (sx) column_forward<true, false>(c, sg, &cs->fs, &cs->sh);
            else column_forward<false, false>(c, sg, &cs->fs, &cs->sh);
        } else {
            if (sx) column_forward<true, true>(c, sg, &cs->fs, &cs->sh);
            else column_forward<false, true>(c, sg, &cs->fs, &cs->sh);
        }
    }
    WindowShared<NC> *ws = reinterpret_cast<WindowShared<NC> *>(cs + 1) + warp;
    for (;;) {
        int32_t id = -1;
        if (lane == 0) {
            const unsigned claim = atomicAdd(&A.ctl->wclaim, 1u);
            if ((int64_t) claim < A.n_windows) id = wait_ready(A, claim);
        }
        id = __shfl_sync(0xffffffffu, id, 0);
        if (id < 0) break;
        Ctx c;
        ctx_init(c, A, A.wtask[id].region);
        const bool sx = c.t[T_SX] > kNegInf;
        if (c.gx_uniform) {
            if (sx) column_window<NC, true, false>(c, ws, id);
            else column_window<NC, false, false>(c, ws, id);
        } else {
            if (sx) column_window<NC, true, true>(c, ws, id);
            else column_window<NC, false, true>(c, ws, id);
        }
        read_unit_done<32>(A, c.R.read, lane, nullptr);
    }
}

}  // namespace fp32
}  // namespace sa
