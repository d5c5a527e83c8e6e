// Resident kernels of the plain FP64 form: the same recursion, operation for operation, as a chain of
// launches that each have the parallelism their part allows.
//
//   emit64      the emissions of every path slot
//   forward64   a CTA per forward segment, a path per thread: stores every anti-diagonal's values
//   backward64  a CTA per traceback window, a path per thread: stores the match value of every slot, and
//               what the total probabilities need
//   totals64    a warp per total probability (the reference's sequential folds)
//   posterior pairs: outputs64 (counts), scan64, place64, outputs64, in the reference's order; or, in
//   expectations mode, transitions64, kmers64 and finish64 (and the HDP machine's assignments with
//   the pairs' kernels)
//
// Why.  One CTA that walked a region's forward sweep, then window after window backward, then the
// posteriors, with every value in global memory behind four dependent table loads, took ~2.8 us an
// anti-diagonal and sweep: latency, not arithmetic (issue 0.1 a cycle on its SM, FP64 pipe 3 %).
// Here the paths of the reference are numbered along it and path q stays on thread q mod NT, so its own
// column's previous value is in a register and its neighbours' are one shared-memory read away; the
// operands come by asynchronous copy kAhead64 anti-diagonals ahead; and a step's log_adds are
// independent.  Windows run side by side, and logarithms, exponentials, totals and outputs are off the
// sweeps' chain.  Measured on B200: see the rule in plan_route.
//
// A slot not in the band holds log 0 for that anti-diagonal, so an absent neighbour drops out of
// log_add.  No two paths of three consecutive anti-diagonals share a thread: the host takes this
// route only if they span at most NT paths.
#pragma once

constexpr int kAhead64 = 6;            // anti-diagonals between a copy and its use
constexpr int kRing64 = 8;             // rows of the copy rings
constexpr int kInfoRing = 128;         // rows of band facts kept

// neighbours of a path: those of the column before (stride apart) and after (consecutive) that it may
// follow or precede (path_checkLegal), in ascending order
struct Path64 {
    double gapx;                       // its skip emission
    int32_t pred, pred_n;
    int32_t pred_step, col;
    int32_t succ, succ_n;
};

// one traceback window: its task, its place among the region's windows, its first total's terms
struct Window64 {
    int32_t task, win;
    int32_t first_total;               // index of its first total probability
    int32_t pad;
};

struct Total64 {
    int32_t region, d;                 // anti-diagonal
    int32_t win;                       // its window in the region
    int16_t have_next, last;           // d < D; d ends the region
};
// what the backward sweep leaves of a total's anti-diagonal d, by slot: match, gap-X and gap-Y values of
// d, match values of d+1
constexpr int kTotalRows = 4;

__device__ __forceinline__ void copy64_4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy64_8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy64_16(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t) __cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy64_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy64_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------------------------------------
// emissions: a warp per anti-diagonal
// ------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) emit64(const Model64 *models, const Region64 *regions, const int32_t *chunk_region,
                                              const int32_t *chunk_d0) {
    const Region64 &R = regions[chunk_region[blockIdx.x]];
    const Model64 &M = models[R.model];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t d0 = chunk_d0[blockIdx.x];
    for (int32_t d = d0 + warp; d < d0 + 32 && d <= R.n; d += 8) {
        const int4 in = R.info[d];
        for (int32_t k = lane; k < in.y; k += 32) {
            const int32_t q = in.x + k, kid = R.pid[q], y = d - R.path[q].col;
            double em = kNegInf, ey = kNegInf;
            if (y >= 1 && kid >= 0) {
                const double2 ev = R.ev[y - 1];
                em = emit_event(M, kid, ev.x, ev.y, true);
                ey = M.emission == 2 ? em : emit_event(M, kid, ev.x, ev.y, false);
            }
            reinterpret_cast<double2 *>(R.E)[in.z + q] = make_double2(em, ey);
        }
    }
}

__device__ __forceinline__ void bar64(int n) { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }

// ------------------------------------------------------------------------------------------------
// band facts of the sweeps: 32 anti-diagonals at a time, by the warp of the copies
// ------------------------------------------------------------------------------------------------
// DIR: +1 forward, -1 backward.  The block after the current one is loaded at its start and becomes
// readable half way through it, long before anything asks for it.
template <int DIR>
struct InfoStream {
    int4 *ring;
    const int4 *src;
    int32_t n, start;
    int4 next;

    __device__ __forceinline__ int4 fetch(int32_t k) const {   // of the k-th anti-diagonal
        const int32_t d = start + DIR * k;
        int4 v = src[min(max(d, 0), n)];
        if (d < 0 || d > n) v.y = 0;   // no such anti-diagonal: no slots
        return v;
    }
    __device__ __forceinline__ void open(int4 *r, const int4 *s, int32_t nn, int32_t d0) {
        ring = r;
        src = s;
        n = nn;
        start = d0;
        const int lane = threadIdx.x & 31;
        ring[lane] = fetch(lane);
        ring[32 + lane] = fetch(32 + lane);
        __syncwarp();
    }
    // at the k-th step
    __device__ __forceinline__ void advance(int32_t k) {
        const int lane = threadIdx.x & 31;
        if ((k & 31) == 0) next = fetch(k + 64 + lane);
        else if ((k & 31) == 16) {
            ring[((k - 16) + 64 + lane) & (kInfoRing - 1)] = next;
            __syncwarp();
        }
    }
    __device__ __forceinline__ int4 at(int32_t k) const { return ring[k & (kInfoRing - 1)]; }
};

// ------------------------------------------------------------------------------------------------
// log_add on the sweeps' chains
// ------------------------------------------------------------------------------------------------
// dp64::log_add bit for bit, without its select chains: the cubic's piece comes from shared memory,
// indexed as in the FP32 form: C - d rounded down, with C's last place 1/16, holds -8 ceil(2 d) mod
// 128 in bits 3..6, the byte offset of the piece in each coefficient's table (entries of 8 bytes lie in
// banks of their own, so lanes with different pieces do not conflict).  Where the difference is NaN (an
// argument that is NaN, or infinities of one sign) the sum is NaN too and is taken, as log_add takes it,
// unless the smaller argument is -inf.  That test is on its upper word, which no sum's NaN shares with -inf,
// and runs beside the cubic's chain (one 1 kb read 1.078 ms without it, 1.074 with, 1.084 with an FP64
// comparison).
struct LogAdd64 {
    double a[16], b[16], c[16], e[16];   // a3 .. a0 of the piece of -ceil(2 d) mod 16
};

__device__ __forceinline__ void log_add_table64(LogAdd64 &t, int k) {
    const double d = 0.5 * ((16 - k) & 15);   // the upper end of the entry's range
    const bool p0 = d <= 1.0, p1 = d <= 2.5, p2 = d <= 4.5;
    t.a[k] = p0 ? (double) -0.009350833524763f : p1 ? (double) -0.014532321752540f
             : p2 ? (double) -0.004605031767994f : (double) -0.000458661602210f;
    t.b[k] = p0 ? (double) 0.130659527668286f : p1 ? (double) 0.139942324101744f
             : p2 ? (double) 0.063427417320019f : (double) 0.009695946122598f;
    t.c[k] = p0 ? (double) 0.498799810682272f : p1 ? (double) 0.495635523139337f
             : p2 ? (double) 0.695956496475118f : (double) 0.930734667215156f;
    t.e[k] = p0 ? (double) 0.693203116424741f : p1 ? (double) 0.692140569840976f
             : p2 ? (double) 0.514272634594009f : (double) 0.168037164329057f;
}

__device__ __forceinline__ const double *piece64(const LogAdd64 &t, double d) {
    const int k = __double2loint(__dadd_rd(422212465065984.0, -d)) & 0x78;
    return reinterpret_cast<const double *>(reinterpret_cast<const char *>(t.a) + k);
}

// the larger argument alone from the cut-off on and where the smaller is -inf; else the cubic p (of the
// difference d) and the smaller
__device__ __forceinline__ double pick64(double x, double y, double p, double d) {
    double r;
    asm("{\n\t.reg .pred q, n;\n\t.reg .f64 hi, lo, s;\n\t.reg .b32 a, b;\n\tsetp.lt.f64 q, %1, %2;\n\t"
        "selp.f64 hi, %2, %1, q;\n\tselp.f64 lo, %1, %2, q;\n\tadd.rn.f64 s, %3, lo;\n\tmov.b64 {a, b}, lo;\n\t"
        "setp.ltu.f64 n, %4, 0d401E000000000000;\n\tsetp.ne.and.b32 n, b, 0xFFF00000, n;\n\tselp.f64 %0, s, hi, n;\n\t}"
        : "=d"(r) : "d"(x), "d"(y), "d"(p), "d"(d));
    return r;
}

__device__ __forceinline__ double lad(const LogAdd64 &t, double x, double y) {
    const double d = fabs(x - y);
    const double *c = piece64(t, d);
    return pick64(x, y, ((c[0] * d + c[16]) * d + c[32]) * d + c[48], d);
}

// two independent ones, stage by stage
__device__ __forceinline__ void lad2(const LogAdd64 &t, const double (&x)[2], const double (&y)[2], double (&r)[2]) {
    double d[2], p[2], b[2], c[2], e[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) d[j] = fabs(x[j] - y[j]);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const double *q = piece64(t, d[j]);
        p[j] = q[0];
        b[j] = q[16];
        c[j] = q[32];
        e[j] = q[48];
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) p[j] = p[j] * d[j];
#pragma unroll
    for (int j = 0; j < 2; ++j) p[j] = p[j] + b[j];
#pragma unroll
    for (int j = 0; j < 2; ++j) p[j] = p[j] * d[j];
#pragma unroll
    for (int j = 0; j < 2; ++j) p[j] = p[j] + c[j];
#pragma unroll
    for (int j = 0; j < 2; ++j) p[j] = p[j] * d[j];
#pragma unroll
    for (int j = 0; j < 2; ++j) p[j] = p[j] + e[j];
#pragma unroll
    for (int j = 0; j < 2; ++j) r[j] = pick64(x[j], y[j], p[j], d[j]);
}

// ------------------------------------------------------------------------------------------------
// the sweeps' warps
// ------------------------------------------------------------------------------------------------
// A sweep is a chain of anti-diagonals and its warps issue in order, so what counts is how much one
// warp does a step.  Four log_adds of a step are independent of one another; two groups of NT threads
// take two each (gap-X and gap-Y of d; the match state but for its last term, and the last term of the
// anti-diagonal next to it), and more warps take what is not the recursion: the copies, and the stores,
// two of each while a CTA has room.  Operands lie by thread, those of slots outside the band as log 0,
// which makes a path that is not there drop out without a test.  Cycles a step of the forward sweep: one
// group with its own copies and stores 895, with bank conflicts gone 805, with helper warps 600, with two
// groups 465 (250 of them without the log_adds).  Backward, where the terms of the totals were the match
// group's too and one warp copied: 853, with two warps and the totals' terms in a launch of their own 520.
template <int NT>
constexpr int kHelperWarps64 = NT <= 256 ? 2 : 1;   // of the copies, and as many of the stores
template <int NT>
constexpr int kSweepThreads64 = 2 * NT + 64 * kHelperWarps64<NT>;

// Path q stays on thread q mod NT of a group: 128, 256, or (what a CTA of 1,024 threads holds twice, one-path
// sets only) 480.
template <int NT>
constexpr bool kPow2 = (NT & (NT - 1)) == 0;

// the slot that thread t holds on an anti-diagonal whose first path is lo (beyond it: at or past its end)
template <int NT>
__device__ __forceinline__ int32_t slot64(int32_t t, int32_t lo) {
    if constexpr (kPow2<NT>) return (t - lo) & (NT - 1);
    const int32_t i = t - lo % NT;
    return i < 0 ? i + NT : i;
}

// the thread of path q
template <int NT>
__device__ __forceinline__ int32_t thread64(int32_t q) {
    if constexpr (kPow2<NT>) return q & (NT - 1);
    return q % NT;
}

// ------------------------------------------------------------------------------------------------
// forward sweep of one segment
// ------------------------------------------------------------------------------------------------
template <int NT, bool kMulti>
struct Forward64Shared {
    LogAdd64 la;
    int4 info[kInfoRing];
    double2 e[kRing64][NT];            // by thread
    double gx[kRing64][NT];
    int4 pred[kMulti ? kRing64 : 1][kMulti ? NT : 1];   // pred, pred_n, pred_step
    double v[2][3][NT];                // states by thread, by parity of the anti-diagonal
};

// predecessors of a thread's path on the k-th anti-diagonal
template <int NT, bool kMulti>
__device__ __forceinline__ int4 preds64(const Forward64Shared<NT, kMulti> &sh, int32_t k, int tid) {
    if constexpr (kMulti) return sh.pred[k & (kRing64 - 1)][tid];
    return make_int4(tid ? tid - 1 : NT - 1, 1, 0, 0);
}

// gap-X (lower neighbours, d-1) and gap-Y (own path, d-1) of d
template <int NT, bool kMulti, bool kSX>
__device__ __forceinline__ void forward_gaps64(const double *mt, const Region64 &R, Forward64Shared<NT, kMulti> &sh) {
    const double tOX = mt[T_OX], tEX = mt[T_EX], tSX = mt[T_SX], tOY = mt[T_OY], tEY = mt[T_EY];
    const int tid = threadIdx.x;
    const int32_t s = R.s0 <= 1 ? 1 : R.s0, steps = R.win[R.w1 - 1].D - s + 1;
    bar64(kSweepThreads64<NT>);      // s-1's values and the first rows are there
    double Y1 = sh.v[1][S_Y][tid];
    double eY = sh.e[0][tid].y, gx = sh.gx[0][tid];
    int4 pr = preds64(sh, 0, tid);
#pragma unroll 1
    for (int32_t k = 0; k < steps; ++k) {
        const double eOX = gx + tOX, eEX = gx + tEX, eSX = gx + tSX, eOY = eY + tOY;
        double x[2], y[2], r[2];
        y[1] = Y1 + (eY + tEY);
        const int p = kMulti ? pr.x & (NT - 1) : pr.x;
        bar64(kSweepThreads64<NT>);  // d-1's values, d+1's operands
        const double(&v)[3][NT] = sh.v[(k + 1) & 1];
        x[0] = v[S_M][p] + eOX;
        y[0] = v[S_X][p] + eEX;
        x[1] = v[S_M][tid] + eOY;
        double lY = 0.0;
        if (kSX) lY = v[S_Y][p] + eSX;
        eY = sh.e[(k + 1) & (kRing64 - 1)][tid].y;
        gx = sh.gx[(k + 1) & (kRing64 - 1)][tid];
        const int4 pr_next = preds64(sh, k + 1, tid);
        if constexpr (kMulti)
            if (pr.y == 0) x[0] = y[0] = lY = kNegInf;
        lad2(sh.la, x, y, r);
        if (kSX) r[0] = lad(sh.la, r[0], lY);
        if constexpr (kMulti) {
            for (int32_t a = 1, q = pr.x + pr.z; a < pr.y; ++a, q += pr.z) {
                const int w = q & (NT - 1);
                r[0] = lad(sh.la, r[0], v[S_M][w] + eOX);
                r[0] = lad(sh.la, r[0], v[S_X][w] + eEX);
                if (kSX) r[0] = lad(sh.la, r[0], v[S_Y][w] + eSX);
            }
        }
        sh.v[k & 1][S_X][tid] = r[0];
        sh.v[k & 1][S_Y][tid] = r[1];
        Y1 = r[1];
        pr = pr_next;
    }
    bar64(kSweepThreads64<NT>);      // the last anti-diagonal's values go out
}

// the match state (middle neighbours, two anti-diagonals back): of d+1 all terms but the last, of d that
template <int NT, bool kMulti>
__device__ __forceinline__ void forward_match64(const double *mt, const Region64 &R, Forward64Shared<NT, kMulti> &sh) {
    const double tMC = mt[T_MC], tMX = mt[T_MFGX], tMY = mt[T_MFGY];
    const int tid = threadIdx.x - NT;
    const int32_t s = R.s0 <= 1 ? 1 : R.s0, steps = R.win[R.w1 - 1].D - s + 1;
    // the values of s-1 (parity 1); s-2's are log 0, or 0 where a later segment starts
    double z = kNegInf, m = kNegInf, g = kNegInf;
    if (R.s0 <= 1) {
        if (tid == 0) {   // startStateProb / raggedStartStateProb (stateMachine.c:1022-1032) on anti-diagonal 0
            m = R.ragged_left ? kNegInf : 0.0;
            g = R.ragged_left ? 0.0 : kNegInf;
        }
    } else {
        const int4 i2 = R.info[s - 2], i1 = R.info[s - 1];
        if (slot64<NT>(tid, i2.x) < i2.y) z = 0.0;
        if (slot64<NT>(tid, i1.x) < i1.y) m = g = 0.0;
    }
    sh.v[0][S_M][tid] = z;             // s-2's, read before step 0 writes over them
    sh.v[1][S_M][tid] = m;
    sh.v[1][S_X][tid] = g;
    sh.v[1][S_Y][tid] = g;
    bar64(kSweepThreads64<NT>);
    int4 pr = preds64(sh, 0, tid);
    double e = sh.e[0][tid].x, most = kNegInf, last = kNegInf;
    for (int32_t a = 0, q = pr.x; a < pr.y; ++a, q += pr.z) {
        const double b = sh.v[0][S_M][kMulti ? q & (NT - 1) : q];   // every state's value there
        if (a) most = lad(sh.la, most, last);
        most = lad(sh.la, most, b + (e + tMC));
        most = lad(sh.la, most, b + (e + tMX));
        last = b + (e + tMY);
    }
    pr = preds64(sh, 1, tid);
    e = sh.e[1][tid].x;
#pragma unroll 1
    for (int32_t k = 0; k < steps; ++k) {
        const double eMC = e + tMC, eMX = e + tMX, eMY = e + tMY;
        double x[2], y[2], r[2];
        x[0] = most;
        y[0] = last;
        const int p = kMulti ? pr.x & (NT - 1) : pr.x;
        bar64(kSweepThreads64<NT>);  // d-1's values, d+2's operands
        const double(&v)[3][NT] = sh.v[(k + 1) & 1];
        x[1] = v[S_M][p] + eMC;
        y[1] = v[S_X][p] + eMX;
        last = v[S_Y][p] + eMY;
        e = sh.e[(k + 2) & (kRing64 - 1)][tid].x;
        const int4 pr_next = preds64(sh, k + 2, tid);
        if constexpr (kMulti)
            if (pr.y == 0) x[1] = y[1] = last = kNegInf;
        lad2(sh.la, x, y, r);
        most = r[1];
        if constexpr (kMulti) {
            for (int32_t a = 1, q = pr.x + pr.z; a < pr.y; ++a, q += pr.z) {
                const int w = q & (NT - 1);
                most = lad(sh.la, most, last);
                most = lad(sh.la, most, v[S_M][w] + eMC);
                most = lad(sh.la, most, v[S_X][w] + eMX);
                last = v[S_Y][w] + eMY;
            }
        }
        sh.v[k & 1][S_M][tid] = r[0];
        pr = pr_next;
    }
    bar64(kSweepThreads64<NT>);
}

// part: which of the warps of the copies
template <int NT, bool kMulti>
__device__ __forceinline__ void forward_copies64(const Region64 &R, Forward64Shared<NT, kMulti> &sh, InfoStream<1> &info,
                                                 int part) {
    const int lane = threadIdx.x & 31;
    const int32_t s = R.s0 <= 1 ? 1 : R.s0, steps = R.win[R.w1 - 1].D - s + 1;
    auto issue = [&](int32_t k, const int4 &in) {
        const int b = k & (kRing64 - 1);
        const double *e = R.E + 2 * ((int64_t) in.z + in.x);
        const Path64 *path = R.path + in.x;
#pragma unroll
        for (int w = 0; w < NT / 32; w += kHelperWarps64<NT>) {
            const int t = lane + 32 * (w + part), i = slot64<NT>(t, in.x);
            if (i < in.y) {
                copy64_16(&sh.e[b][t], e + 2 * i);
                copy64_8(&sh.gx[b][t], &path[i].gapx);
                if constexpr (kMulti) {
                    copy64_8(&sh.pred[b][t].x, &path[i].pred);
                    copy64_8(&sh.pred[b][t].z, &path[i].pred_step);
                }
            } else {
                sh.e[b][t] = make_double2(kNegInf, kNegInf);
                sh.gx[b][t] = kNegInf;
                if constexpr (kMulti) sh.pred[b][t].y = 0;
            }
        }
        copy64_commit();
    };
#pragma unroll
    for (int k = 0; k < kAhead64; ++k) issue(k, info.at(k));
    copy64_wait<kAhead64 - 3>();
    int4 in = info.at(kAhead64);
    bar64(kSweepThreads64<NT>);
    for (int32_t k = 0; k < steps; ++k) {
        bar64(kSweepThreads64<NT>);
        issue(k + kAhead64, in);
        if (part == 0) info.advance(k);
        in = info.at(k + kAhead64 + 1);
        copy64_wait<kAhead64 - 3>();   // every copy of d+3 and before has landed
    }
    bar64(kSweepThreads64<NT>);
    copy64_wait<0>();
}

// at step k d-1's values go to the store and, where a stitch is, to its side; part: which of the warps
template <int NT, bool kMulti>
__device__ __forceinline__ void forward_results64(const Region64 &R, const SetOut &O, Forward64Shared<NT, kMulti> &sh,
                                                  int part) {
    constexpr int NW = NT / 32 / kHelperWarps64<NT>;
    const int lane = 32 * part + (threadIdx.x & 31), stride = 32 * kHelperWarps64<NT>;
    const int32_t s = R.s0 <= 1 ? 1 : R.s0, steps = R.win[R.w1 - 1].D - s + 1;
    if (R.s0 <= 1 && lane == 0) {
        double *c = R.F + 3 * (int64_t) R.info[0].z;
        c[S_M] = R.ragged_left ? kNegInf : 0.0;
        c[S_X] = c[S_Y] = R.ragged_left ? 0.0 : kNegInf;
    }
    const int32_t b_in = R.st_in >= 0 ? O.stitch[R.st_in].b : -10, b_out = R.st_out >= 0 ? O.stitch[R.st_out].b : -10;
    bar64(kSweepThreads64<NT>);
    bar64(kSweepThreads64<NT>);        // step 0
    int4 in = sh.info[0];
    for (int32_t k = 1; k <= steps; ++k) {
        const int32_t r = s + k - 1;   // the anti-diagonal that goes out
        double *c = R.F + 3 * ((int64_t) in.z + in.x + lane);
        bar64(kSweepThreads64<NT>);
        const double(&v)[3][NT] = sh.v[(k - 1) & 1];
        const int4 in_next = sh.info[k & (kInfoRing - 1)];
#pragma unroll
        for (int w0 = 0; w0 < NW; w0 += 4) {   // as many values in flight as registers allow
            double o[3][4];
#pragma unroll
            for (int w = w0; w < w0 + 4 && w < NW; ++w) {
                const int at = thread64<NT>(in.x + lane + stride * w);
#pragma unroll
                for (int st = 0; st < 3; ++st) o[st][w - w0] = v[st][at];
            }
#pragma unroll
            for (int w = w0; w < w0 + 4 && w < NW; ++w) {
                if (lane + stride * w < in.y) {
#pragma unroll
                    for (int st = 0; st < 3; ++st) c[3 * stride * w + st] = o[st][w - w0];
                }
            }
        }
        if (r == b_in - 1 || r == b_in || r == b_out - 1 || r == b_out) {
            const bool side = r == b_in - 1 || r == b_in;
            const Stitch64 S = O.stitch[side ? R.st_in : R.st_out];
            double *to = S.vals + 3 * (int64_t) (side ? r - (b_in - 1) : 2 + r - (b_out - 1)) * S.stride;
            for (int i = lane; i < in.y; i += stride)
                for (int st = 0; st < 3; ++st) to[3 * i + st] = v[st][thread64<NT>(in.x + i)];
        }
        in = in_next;
    }
}

template <int NT, bool kMulti, bool kSX>
__global__ void __launch_bounds__(kSweepThreads64<NT>) forward64(const Model64 *models, const Region64 *tasks, SetOut O) {
    extern __shared__ double2 smem64[];
    using Sh = Forward64Shared<NT, kMulti>;
    Sh &sh = *reinterpret_cast<Sh *>(smem64);
    const Region64 R = tasks[blockIdx.x];
    const int helper = ((int) threadIdx.x - 2 * NT) >> 5;
    InfoStream<1> info{sh.info, nullptr, 0, 0, make_int4(0, 0, 0, 0)};
    if (threadIdx.x < 16) log_add_table64(sh.la, threadIdx.x);
    if (helper == 0) info.open(sh.info, R.info, R.n, R.s0 <= 1 ? 1 : R.s0);
    __syncthreads();
    if (threadIdx.x < NT) forward_gaps64<NT, kMulti, kSX>(models[R.model].t, R, sh);
    else if (threadIdx.x < 2 * NT) forward_match64<NT, kMulti>(models[R.model].t, R, sh);
    else if (helper < kHelperWarps64<NT>) forward_copies64<NT, kMulti>(R, sh, info, helper);
    else forward_results64<NT, kMulti>(R, O, sh, helper - kHelperWarps64<NT>);
    __syncthreads();
    if (R.st_in >= 0) stitch_arrive64(R, O, R.st_in);
    if (R.st_out >= 0) stitch_arrive64(R, O, R.st_out);
}

// ------------------------------------------------------------------------------------------------
// backward sweep of one traceback window
// ------------------------------------------------------------------------------------------------
// A path's values go to its predecessors already summed with its emission and the transitions (the
// pushed sums of backward_cell), so a predecessor only folds.  The last term of d+1's match state is
// folded at step d, which nothing needs before d-1.  The values go out for the launches after this one:
// the match values of the window's own anti-diagonals, all of an anti-diagonal with a total probability,
// and the match values of the one above it.
template <int NT, bool kMulti>
struct Backward64Shared {
    LogAdd64 la;
    int4 info[kInfoRing];
    double2 e[kRing64][NT];            // by thread
    double gx[NT > 256 ? 1 : kRing64][NT > 256 ? 1 : NT];   // (480 threads read it where it is: no room)
    int2 succ[kMulti ? kRing64 : 1][kMulti ? NT : 1];      // succ, succ_n
    double a[2][3][NT];                // sums for the match predecessors, by parity
    double b[2][3][NT];                // sums for the gap-X predecessors, by parity
    double u[2][NT];                   // the gap-Y sum for the own path's match state, by parity
    double vm[2][NT];                  // match values, by parity of the anti-diagonal
    double vx[4][NT], vy[4][NT];       // gap values
};
static_assert(sizeof(Backward64Shared<480, false>) <= 227 * 1024 && sizeof(Backward64Shared<256, true>) <= 227 * 1024 &&
                  sizeof(Forward64Shared<480, false>) <= 227 * 1024,
              "a CTA's shared memory");

// successors of a thread's path on the k-th anti-diagonal
template <int NT, bool kMulti>
__device__ __forceinline__ int2 succs64(const Backward64Shared<NT, kMulti> &sh, int32_t k, int tid) {
    if constexpr (kMulti) return sh.succ[k & (kRing64 - 1)][tid];
    return make_int2(tid < NT - 1 ? tid + 1 : 0, 1);
}

// gap-X and gap-Y of d
template <int NT, bool kMulti, bool kSX>
__device__ __forceinline__ void backward_gaps64(const double *mt, const Region64 &R, const Window &W,
                                                Backward64Shared<NT, kMulti> &sh) {
    const double tOX = mt[T_OX], tEX = mt[T_EX], tSX = mt[T_SX], tOY = mt[T_OY], tEY = mt[T_EY];
    const int tid = threadIdx.x;
    const int32_t steps = W.D - W.T;
    // endStateProb / raggedEndStateProb (stateMachine.c:1034-1061) on the traceback anti-diagonal
    const bool ragged_end = W.at_end && R.ragged_right;
    const double e1 = ragged_end ? tEX : mt[T_MFGX], e2 = ragged_end ? tEY : mt[T_MFGY];
    for (int st = 0; st < 3; ++st) sh.b[1][st][tid] = kNegInf;
    sh.u[1][tid] = kNegInf;
    auto skip = [&](int32_t k) -> double {
        if constexpr (NT > 256) {
            const int4 in = sh.info[k & (kInfoRing - 1)];
            const int32_t i = slot64<NT>(tid, in.x);
            return k < steps && i < in.y ? __ldg(&R.path[in.x + i].gapx) : kNegInf;
        } else {
            return sh.gx[k & (kRing64 - 1)][tid];
        }
    };
    bar64(kSweepThreads64<NT>);                    // the first rows are ready
    double u1 = kNegInf;                             // own path's gap-Y sum of d+1 for gap-Y
    double eY = sh.e[0][tid].y, gx = skip(0);
    int2 nb = succs64(sh, 0, tid);
#pragma unroll 1
    for (int32_t k = 0; k < steps; ++k) {
        const double gOX = gx + tOX, gEX = gx + tEX, gSX = gx + tSX, eOY = eY + tOY, eEY = eY + tEY;
        double x[2], y[2], r[2];
        const int p = kMulti ? nb.x & (NT - 1) : nb.x;
        y[1] = u1;
        bar64(kSweepThreads64<NT>);                // d+1's sums for gap-X predecessors, d+2's for match predecessors
        const double(&a)[3][NT] = sh.a[k & 1];
        const double(&c)[3][NT] = sh.b[(k + 1) & 1];
        x[0] = a[1][p];
        y[0] = c[1][p];
        x[1] = a[2][p];
        double lY = 0.0;
        if (kSX) lY = c[2][p];
        eY = sh.e[(k + 1) & (kRing64 - 1)][tid].y;
        gx = skip(k + 1);
        const int2 nb_next = succs64(sh, k + 1, tid);
        if constexpr (kMulti) {
            if (nb.y == 0) x[0] = y[0] = x[1] = lY = kNegInf;
            for (int32_t j = 1; j < nb.y; ++j) {
                x[0] = lad(sh.la, x[0], a[1][(nb.x + j) & (NT - 1)]);
                x[1] = lad(sh.la, x[1], a[2][(nb.x + j) & (NT - 1)]);
            }
        }
        lad2(sh.la, x, y, r);
        if (kSX) r[1] = lad(sh.la, r[1], lY);
        if constexpr (kMulti) {
            for (int32_t j = 1; j < nb.y; ++j) {
                r[0] = lad(sh.la, r[0], c[1][(nb.x + j) & (NT - 1)]);
                if (kSX) r[1] = lad(sh.la, r[1], c[2][(nb.x + j) & (NT - 1)]);
            }
        }
        if (k == 0) {
            r[0] = e1;
            r[1] = e2;
        }
        sh.b[k & 1][0][tid] = r[0] + gOX;
        sh.b[k & 1][1][tid] = r[0] + gEX;
        if (kSX) sh.b[k & 1][2][tid] = r[0] + gSX;
        sh.u[k & 1][tid] = r[1] + eOY;
        u1 = r[1] + eEY;
        sh.vx[k & 3][tid] = r[0];
        sh.vy[k & 3][tid] = r[1];
        nb = nb_next;
    }
    bar64(kSweepThreads64<NT>);
    bar64(kSweepThreads64<NT>);
}

// the match state: of d all terms but the last, of d+1 that
template <int NT, bool kMulti>
__device__ __forceinline__ void backward_match64(const double *mt, const Region64 &R, const Window &W,
                                                 Backward64Shared<NT, kMulti> &sh) {
    const double tMC = mt[T_MC], tMX = mt[T_MFGX], tMY = mt[T_MFGY];
    const int tid = threadIdx.x - NT;
    const int32_t steps = W.D - W.T;
    const bool ragged_end = W.at_end && R.ragged_right;
    const double e0 = ragged_end ? (mt[T_OX] + mt[T_OY]) / 2.0 : tMC;
    for (int k = 0; k < 2; ++k)
        for (int st = 0; st < 3; ++st) sh.a[k][st][tid] = kNegInf;
    bar64(kSweepThreads64<NT>);
    double most = kNegInf, last = kNegInf;           // the match state on d+1: all terms but one, and that
    double e1 = kNegInf, e = sh.e[0][tid].x;         // emissions of d+1 and d
    int2 nb = succs64(sh, 0, tid);
#pragma unroll 1
    for (int32_t k = 0; k <= steps; ++k) {           // k == steps: only the last term of the last one
        const double eMC = e1 + tMC, eMX = e1 + tMX, eMY = e1 + tMY;
        double x[2], y[2], r[2];
        x[0] = most;
        y[0] = last;
        const int p = kMulti ? nb.x & (NT - 1) : nb.x;
        bar64(kSweepThreads64<NT>);
        const double(&a)[3][NT] = sh.a[k & 1];
        const double(&c)[3][NT] = sh.b[(k + 1) & 1];
        x[1] = a[0][p];
        y[1] = sh.u[(k + 1) & 1][tid];
        double l = c[0][p];
        const double e_next = sh.e[(k + 1) & (kRing64 - 1)][tid].x;
        const int2 nb_next = succs64(sh, k + 1, tid);
        if constexpr (kMulti) {
            if (nb.y == 0) x[1] = l = kNegInf;
            for (int32_t j = 1; j < nb.y; ++j) x[1] = lad(sh.la, x[1], a[0][(nb.x + j) & (NT - 1)]);
        }
        lad2(sh.la, x, y, r);
        if constexpr (kMulti) {
            for (int32_t j = 1; j < nb.y; ++j) {
                r[1] = lad(sh.la, r[1], l);
                l = c[0][(nb.x + j) & (NT - 1)];
            }
        }
        most = k == 0 ? e0 : r[1];
        last = k == 0 ? kNegInf : l;
        // a buffer's parity is its anti-diagonal's plus one
        sh.a[(k + 1) & 1][0][tid] = r[0] + eMC;
        sh.a[(k + 1) & 1][1][tid] = r[0] + eMX;
        sh.a[(k + 1) & 1][2][tid] = r[0] + eMY;
        sh.vm[(k + 1) & 1][tid] = r[0];
        e1 = e;
        e = e_next;
        nb = nb_next;
    }
    bar64(kSweepThreads64<NT>);                      // the last match values go out
}

template <int NT, bool kMulti>
__device__ __forceinline__ void backward_copies64(const Region64 &R, const Window &W, Backward64Shared<NT, kMulti> &sh,
                                                  InfoStream<-1> &info, int part) {
    const int lane = threadIdx.x & 31;
    const int32_t steps = W.D - W.T;
    auto issue = [&](int32_t k, const int4 &in) {
        const int32_t n = k < steps ? in.y : 0;
        const int b = k & (kRing64 - 1);
        const double *e = R.E + 2 * ((int64_t) in.z + in.x);
        const Path64 *path = R.path + in.x;
#pragma unroll
        for (int w = 0; w < NT / 32; w += kHelperWarps64<NT>) {
            const int t = lane + 32 * (w + part), i = slot64<NT>(t, in.x);
            if (i < n) {
                copy64_16(&sh.e[b][t], e + 2 * i);
                if constexpr (NT <= 256) copy64_8(&sh.gx[b][t], &path[i].gapx);
                if constexpr (kMulti) copy64_8(&sh.succ[b][t], &path[i].succ);
            } else {
                sh.e[b][t] = make_double2(kNegInf, kNegInf);
                if constexpr (NT <= 256) sh.gx[b][t] = kNegInf;
                if constexpr (kMulti) sh.succ[b][t] = make_int2(0, 0);
            }
        }
        copy64_commit();
    };
#pragma unroll
    for (int k = 0; k < kAhead64; ++k) issue(k, info.at(k));
    copy64_wait<kAhead64 - 2>();
    int4 in = info.at(kAhead64);
    bar64(kSweepThreads64<NT>);
    for (int32_t k = 0; k <= steps; ++k) {
        bar64(kSweepThreads64<NT>);
        issue(k + kAhead64, in);
        if (part == 0) info.advance(k);
        in = info.at(k + kAhead64 + 1);
        copy64_wait<kAhead64 - 2>();                 // every copy of d-2 and above has landed
    }
    bar64(kSweepThreads64<NT>);
    copy64_wait<0>();
}

// at step k d+2's values go to their stores
template <int NT, bool kMulti>
__device__ __forceinline__ void backward_results64(const Region64 &R, const Window64 &wt, const Window &W,
                                                   Backward64Shared<NT, kMulti> &sh, double *terms, int64_t term_stride,
                                                   int expect, int part) {
    constexpr int NW = NT / 32 / kHelperWarps64<NT>;
    const int lane = 32 * part + (threadIdx.x & 31), stride = 32 * kHelperWarps64<NT>;
    const int32_t steps = W.D - W.T;
    int32_t until = W.D - W.from;                    // the k of the next total's anti-diagonal
    double *t = terms + (int64_t) wt.first_total * kTotalRows * term_stride + lane;
    bar64(kSweepThreads64<NT>);
    bar64(kSweepThreads64<NT>);
    bar64(kSweepThreads64<NT>);                      // steps 0 and 1 (a match value is there two steps on)
    int4 in = sh.info[0];
    for (int32_t k = 0; k < steps; ++k) {            // the anti-diagonal that goes out
        const int64_t z = (int64_t) in.z + in.x + lane;
        const bool post = W.D - k <= W.from, total = k == until, above = k == until - 1 && until < steps;
        bar64(kSweepThreads64<NT>);
        const int4 in_next = sh.info[(k + 1) & (kInfoRing - 1)];
        if (post || above) {
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                if (lane + stride * w >= in.y) continue;
                const int at = thread64<NT>(in.x + lane + stride * w);
                const double m = sh.vm[k & 1][at];
                if (post) R.S[z + stride * w] = m;
                if (expect && post) {
                    double *b = R.B + 3 * (z + stride * w);
                    b[S_M] = m;
                    b[S_X] = sh.vx[k & 3][at];
                    b[S_Y] = sh.vy[k & 3][at];
                }
                if (total) {
                    t[stride * w] = m;
                    t[term_stride + stride * w] = sh.vx[k & 3][at];
                    t[2 * term_stride + stride * w] = sh.vy[k & 3][at];
                }
                if (above) t[3 * term_stride + stride * w] = m;
            }
        }
        if (total) {
            until += 10;
            t += kTotalRows * term_stride;
        }
        in = in_next;
    }
}

template <int NT, bool kMulti, bool kSX>
__global__ void __launch_bounds__(kSweepThreads64<NT>) backward64(const Model64 *models, const Region64 *tasks,
                                                                 const Window64 *windows, double *terms,
                                                                 int64_t term_stride, int expect) {
    extern __shared__ double2 smem64[];
    using Sh = Backward64Shared<NT, kMulti>;
    Sh &sh = *reinterpret_cast<Sh *>(smem64);
    const Window64 wt = windows[blockIdx.x];
    const Region64 R = tasks[wt.task];
    const Window W = R.win[wt.win];
    const int helper = ((int) threadIdx.x - 2 * NT) >> 5;
    InfoStream<-1> info{sh.info, nullptr, 0, 0, make_int4(0, 0, 0, 0)};
    if (threadIdx.x < 16) log_add_table64(sh.la, threadIdx.x);
    if (helper == 0) info.open(sh.info, R.info, R.n, W.D);
    __syncthreads();
    if (threadIdx.x < NT) backward_gaps64<NT, kMulti, kSX>(models[R.model].t, R, W, sh);
    else if (threadIdx.x < 2 * NT) backward_match64<NT, kMulti>(models[R.model].t, R, W, sh);
    else if (helper < kHelperWarps64<NT>) backward_copies64<NT, kMulti>(R, W, sh, info, helper);
    else backward_results64<NT, kMulti>(R, wt, W, sh, terms, term_stride, expect, helper - kHelperWarps64<NT>);
}

// ------------------------------------------------------------------------------------------------
// total probabilities: a warp each
// ------------------------------------------------------------------------------------------------
// diagonalCalculationTotalProbability (pairwiseAligner.c:1182-1200): F.B on d in ascending cell order, a
// cell's paths folded first (hdCell_totalProbability), then the matches from d-1 over d into d+1, dotted
// with B(d+1).  The lanes make both folds' terms, 128 slots at a time, and two of them fold.
constexpr int kTotalWarps = 2;
constexpr int kTotalSlots = 128;

__global__ void __launch_bounds__(32 * kTotalWarps) totals64(const Model64 *models, const Region64 *regions,
                                                             const Region64 *tasks, const int32_t *task_of,
                                                             const Total64 *totals, int64_t n, const double *terms,
                                                             int64_t term_stride, int multi) {
    __shared__ LogAdd64 la;
    __shared__ double term[kTotalWarps][2][kTotalSlots];
    __shared__ int32_t cols[kTotalWarps][2][kTotalSlots];
    if (threadIdx.x < 16) log_add_table64(la, threadIdx.x);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t at = blockIdx.x * (int64_t) kTotalWarps + warp;
    if (at >= n) return;
    const Total64 T = totals[at];
    const Region64 &R = regions[T.region];
    const double *mt = models[R.model].t;
    const double tMC = mt[T_MC], tMX = mt[T_MFGX], tMY = mt[T_MFGY];
    const double *F = tasks[task_of[R.win_base + T.win]].F;   // the segment that swept the window
    const double *t = terms + at * kTotalRows * term_stride;
    const int4 in = R.info[T.d], in1 = T.have_next ? R.info[T.d + 1] : make_int4(0, 0, 0, 0), bl = R.info[T.d - 1];
    double v = kNegInf, cell = kNegInf;        // lane 0: the fold on d; lane 1: through d
    int32_t col = -1;
    for (int32_t k0 = 0; k0 < max(in.y, in1.y); k0 += kTotalSlots) {
#pragma unroll
        for (int w = 0; w < kTotalSlots / 32; ++w) {
            const int j = lane + 32 * w, i = k0 + j;
            if (i < in.y) {
                const double *f = F + 3 * ((int64_t) in.z + in.x + i);
                double s = f[S_M] + t[i];
                s = lad(la, s, f[S_X] + t[term_stride + i]);
                s = lad(la, s, f[S_Y] + t[2 * term_stride + i]);
                term[warp][0][j] = s;
                if (multi) cols[warp][0][j] = R.path[in.x + i].col;
            }
            if (i < in1.y) {
                const int32_t q = in1.x + i;
                const double e = R.E[2 * ((int64_t) in1.z + q)];
                double s = kNegInf;
                const int32_t cnt = multi ? R.path[q].pred_n : 1, step = multi ? R.path[q].pred_step : 1;
                for (int32_t c = 0, p = multi ? R.path[q].pred : q - 1; c < cnt; ++c, p += step) {
                    const bool there = p >= bl.x && p < bl.x + bl.y;
                    const double *f = F + 3 * ((int64_t) bl.z + (there ? p : bl.x));
                    s = lad(la, s, (there ? f[S_M] : kNegInf) + (e + tMC));
                    s = lad(la, s, (there ? f[S_X] : kNegInf) + (e + tMX));
                    s = lad(la, s, (there ? f[S_Y] : kNegInf) + (e + tMY));
                }
                term[warp][1][j] = s + t[3 * term_stride + i];
                if (multi) cols[warp][1][j] = R.path[q].col;
            }
        }
        __syncwarp();
        if (lane < 2) {
            const int32_t m = min(kTotalSlots, (lane ? in1.y : in.y) - k0);
            const double *s = term[warp][lane];
            if (!multi) {
#pragma unroll 4
                for (int32_t j = 0; j < m; ++j) v = lad(la, v, s[j]);
            } else {
                for (int32_t j = 0; j < m; ++j) {
                    if (cols[warp][lane][j] != col) {
                        v = lad(la, v, cell);
                        cell = kNegInf;
                        col = cols[warp][lane][j];
                    }
                    cell = lad(la, cell, s[j]);
                }
            }
        }
        __syncwarp();
    }
    if (multi) v = lad(la, v, cell);
    const double through = __shfl_sync(0xffffffffu, v, 1);
    if (lane == 0) {
        if (T.have_next) v = lad(la, v, through);
        R.P[T.d] = v;
        if (T.last) *R.loglik = v;
    }
}

// ------------------------------------------------------------------------------------------------
// outputs in the reference's order
// ------------------------------------------------------------------------------------------------
// A region's windows come in ascending order and a window's anti-diagonals (T, from] descending, so
// anti-diagonal d of a window comes T + from - d -th among the region's.
struct Output64 {
    sa_aligned_pair *out;         // pairs, or
    const ExpectOut *reads;       // (expectations of HDP machines) each read's assignments
    int32_t *count;               // per region its anti-diagonals' counts, then their starts
    int64_t *region_total;        // per region its count, then its start
    int64_t cap;
    double threshold;
};

// the number of outputs of slot q on d, and (write) the outputs
template <bool kAssign>
__device__ __forceinline__ int slot_hits(const Region64 &R, const double *F, const Output64 &O, int64_t at, double total,
                                         int32_t x, int32_t y, double &p, unsigned &which) {
    if (kAssign) {   // match transitions at or above the threshold, from match, gap-X, gap-Y
        which = 0;
        if (!(R.B[3 * at] < 0.0))   // -1: no middle neighbour
            for (int j = 0; j < 3; ++j)
                if (R.B[3 * at + j] >= O.threshold) which |= 1u << j;
        return __popc(which);
    }
    if (x <= 0 || y <= 0) return 0;
    p = exp((F[3 * at] + R.S[at]) - total);
    return p >= O.threshold ? 1 : 0;
}

template <bool kAssign, bool kWrite>
__global__ void __launch_bounds__(256) outputs64(const Region64 *regions, const Region64 *tasks, const int32_t *task_of,
                                                 const int32_t *chunk_region, const int32_t *chunk_d0,
                                                 const int64_t *row_base, Output64 O) {
    const int32_t region = chunk_region[blockIdx.x];
    const Region64 &R = regions[region];
    if (kAssign && !O.reads[R.reader].hdp) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t d0 = chunk_d0[blockIdx.x];
    int32_t *count = O.count + row_base[region];
    for (int32_t d = max(d0, 1) + warp; d < d0 + 32 && d <= R.n; d += 8) {
        const int4 in = R.info[d];
        const Window W = R.win[in.w];
        const int32_t place = W.T + W.from - d;
        const double *F = kAssign ? nullptr : tasks[task_of[R.win_base + in.w]].F;   // the segment that swept the window
        const double total = R.P[W.from - 10 * ((W.from - d) / 10)];
        int64_t base = kWrite ? O.region_total[region] + count[place] : 0;
        int32_t found = 0;
        for (int32_t k0 = 0; k0 < in.y; k0 += 32) {
            const int32_t k = k0 + lane, q = in.x + k;
            const int64_t at = (int64_t) in.z + q;
            double p = 0.0;
            unsigned which = 0;
            int hits = 0;
            int32_t x = 0, y = 0;
            if (k < in.y) {
                x = R.path[q].col;
                y = d - x;
                hits = slot_hits<kAssign>(R, F, O, at, total, x, y, p, which);
            }
            if (!__any_sync(0xffffffffu, hits > 0)) continue;
            int32_t inc = hits;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t v = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += v;
            }
            if (kWrite && hits) {
                int64_t to = base + found + inc - hits;
                if (kAssign) {
                    const ExpectOut &X = O.reads[R.reader];
                    for (int j = 0; j < 3; ++j) {
                        if (!((which >> j) & 1u)) continue;
                        if (to < X.assign_cap) {
                            X.assign_kmer[to] = R.pid[q];
                            X.assign_event[to] = R.ev_base + y - 1;
                        }
                        ++to;
                    }
                } else if (to < O.cap) {
                    sa_aligned_pair o;
                    o.score = (int64_t) floor((p > 1.0 ? 1.0 : p) * 10000000.0);
                    o.x = R.x_base + x - 1;
                    o.y = R.ev_base + y - 1;
                    o.kmer = R.pid[q];
                    O.out[to] = o;
                } else {
                    atomicExch(R.status, (int32_t) SA_E_OUTPUT);
                }
            }
            found += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (!kWrite && lane == 0) count[place] = found;
    }
}

// counts of a region's anti-diagonals to their starts, a CTA each
__global__ void __launch_bounds__(1024) scan64(const Region64 *regions, const int64_t *row_base, Output64 O) {
    __shared__ int32_t sums[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int32_t *c = O.count + row_base[blockIdx.x];
    const int32_t n = regions[blockIdx.x].n;   // places 0 .. n-1
    int32_t run = 0;
    for (int32_t k0 = 0; k0 < n; k0 += 4096) {
        int32_t v[4], mine = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t k = k0 + 4 * tid + j;
            v[j] = k < n ? c[k] : 0;
            mine += v[j];
        }
        int32_t inc = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) sums[warp] = inc;
        __syncthreads();
        int32_t before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) before += sums[w];
            all += sums[w];
        }
        int32_t at = run + before + inc - mine;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t k = k0 + 4 * tid + j;
            if (k < n) c[k] = at;
            at += v[j];
        }
        run += all;
        __syncthreads();
    }
    if (tid == 0) O.region_total[blockIdx.x] = run;
}

// regions' counts to their starts, in order; `counts` keeps them, `all` their sum.  `first`: the first
// region of each group that starts again at 0 (a read's assignments), or null for one group
__global__ void place64(int64_t n, int64_t *region_total, int64_t *counts, unsigned long long *all, const int32_t *first) {
    if (threadIdx.x || blockIdx.x) return;
    int64_t at = 0;
    for (int64_t r = 0; r < n; ++r) {
        if (first && first[r] == r) at = 0;
        const int64_t c = region_total[r];
        counts[r] = c;
        region_total[r] = at;
        at += c;
    }
    if (all) *all = (unsigned long long) at;
}

// ------------------------------------------------------------------------------------------------
// expectations
// ------------------------------------------------------------------------------------------------
// The transition posteriors of every slot (cell_signal_updateExpectations, pairwiseAligner.c:763-793;
// see expect_diagonal): summed per block, and the three into the match state kept in place of the
// slot's backward values (-1 where there is no middle neighbour), for the per-k-mer folds.
__global__ void __launch_bounds__(256) transitions64(const Model64 *models, const Region64 *tasks, const int32_t *task_of,
                                                     const int32_t *chunk_region, const int32_t *chunk_d0,
                                                     const Region64 *regions, double *partial) {
    __shared__ double sums[8][9];
    const int32_t region = chunk_region[blockIdx.x];
    const Region64 &R = regions[region];
    const Model64 &M = models[R.model];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t d0 = chunk_d0[blockIdx.x];
    double acc[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) acc[j] = 0.0;
    for (int32_t d = max(d0, 1) + warp; d < d0 + 32 && d <= R.n; d += 8) {
        const int4 in = R.info[d], l1 = R.info[d - 1], l2 = d >= 2 ? R.info[d - 2] : make_int4(0, 0, 0, 0);
        const Window W = R.win[in.w];
        const double total = R.P[W.from - 10 * ((W.from - d) / 10)];
        const double *F = tasks[task_of[R.win_base + in.w]].F;   // the segment that swept this window
        if (lane == 0) acc[8] += total;
        for (int32_t k = lane; k < in.y; k += 32) {
            const int32_t q = in.x + k;
            const int64_t at = (int64_t) in.z + q;
            const double bM = R.B[3 * at], bX = R.B[3 * at + 1], bY = R.B[3 * at + 2];
            const bool lo = q - 1 >= l1.x && q - 1 < l1.x + l1.y && q > 0;
            const bool mi = d - 2 >= W.T && q - 1 >= l2.x && q - 1 < l2.x + l2.y && q > 0;
            const bool up = q >= l1.x && q < l1.x + l1.y;
            if (lo) {
                const double *l = F + 3 * ((int64_t) l1.z + q - 1);
                const double e = R.path[q].gapx;
                acc[0] += exp(l[S_M] + bX + (e + M.t[T_OX]) - total);
                acc[1] += exp(l[S_X] + bX + (e + M.t[T_EX]) - total);
                acc[2] += exp(l[S_Y] + bX + (e + M.t[T_SX]) - total);
            }
            double p3 = -1.0, p4 = 0.0, p5 = 0.0;
            if (mi) {
                const double *m = F + 3 * ((int64_t) l2.z + q - 1);
                const double e = R.E[2 * at];
                p3 = exp(m[S_M] + bM + (e + M.t[T_MC]) - total);
                p4 = exp(m[S_X] + bM + (e + M.t[T_MFGX]) - total);
                p5 = exp(m[S_Y] + bM + (e + M.t[T_MFGY]) - total);
                acc[3] += p3;
                acc[4] += p4;
                acc[5] += p5;
            }
            if (up) {
                const double *u = F + 3 * ((int64_t) l1.z + q);
                const double e = R.E[2 * at + 1];
                acc[6] += exp(u[S_M] + bY + (e + M.t[T_OY]) - total);
                acc[7] += exp(u[S_Y] + bY + (e + M.t[T_EY]) - total);
            }
            R.B[3 * at] = p3;
            R.B[3 * at + 1] = p4;
            R.B[3 * at + 2] = p5;
        }
    }
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
        if (lane == 0) sums[warp][j] = acc[j];
    }
    __syncthreads();
    if (threadIdx.x < 9) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) s += sums[w][threadIdx.x];
        partial[9 * (int64_t) blockIdx.x + threadIdx.x] = s;
    }
}

// a k-mer of a read: the columns it stands at, by region, ascending
struct Kmer64 {
    int32_t read, kid, first, count;   // columns cols[first .. first + count)
};
struct Column64 {
    int32_t region, col, dlo, dhi;     // anti-diagonals the column's cells may be on
};

// continuousPairHmm_addToEmissionExpectation (continuousHmm.c:160-169) for one k-mer of one read, by a
// warp: 32 anti-diagonals at a time in the reference's order.  The running weight and mean sum that
// each update's spread needs are scans over the lanes, a lane's cells of one anti-diagonal in order.
__global__ void __launch_bounds__(128) kmers64(const Model64 *models, const Region64 *regions, const Kmer64 *kmers,
                                               int64_t n_kmers, const Column64 *cols, const ExpectOut *XS) {
    const int64_t at = blockIdx.x * (int64_t) 4 + (threadIdx.x >> 5);
    if (at >= n_kmers) return;
    const int lane = threadIdx.x & 31;
    const Kmer64 K = kmers[at];
    const ExpectOut &X = XS[K.read];
    double e0 = X.event_exp[2 * (int64_t) K.kid], e1 = X.event_exp[2 * (int64_t) K.kid + 1], po = X.posteriors[K.kid];
    bool seen = false;
    for (int32_t c0 = K.first; c0 < K.first + K.count;) {
        // the columns of one region
        const int32_t region = cols[c0].region;
        int32_t c1 = c0 + 1;
        while (c1 < K.first + K.count && cols[c1].region == region) ++c1;
        const Region64 &R = regions[region];
        const Model64 &M = models[R.model];
        const double mu = M.match[(int64_t) K.kid * 5];
        const int32_t dlo = max(cols[c0].dlo, 1), dhi = min(cols[c1 - 1].dhi, R.n);
        for (int32_t w = dlo <= dhi ? R.info[dlo].w : 0; dlo <= dhi && w <= R.info[dhi].w; ++w) {
            const Window W = R.win[w];
            const int32_t bottom = max(W.T + 1, dlo);
            for (int32_t dt = min(W.from, dhi); dt >= bottom; dt -= 32) {
                // down to an anti-diagonal of the last column that begins at or before this one
                int32_t l = c0, h = c1;
                while (l < h) {
                    const int32_t mid = (l + h) >> 1;
                    if (cols[mid].dlo <= dt) l = mid + 1;
                    else h = mid;
                }
                if (l == c0) break;
                dt = min(dt, cols[l - 1].dhi);
                if (dt < bottom) break;
                const int32_t d = dt - lane;
                int32_t a = 0, b = 0;         // columns c0 + a .. c0 + b - 1 are on d
                int4 in = make_int4(0, 0, 0, 0);
                if (d >= bottom) {
                    in = R.info[d];
                    a = 0;
                    b = c1 - c0;
                    if (b == 1) {
                        const int32_t q = cols[c0].col;
                        if (!(q >= in.x && q < in.x + in.y)) b = 0;
                    } else {   // single-path columns: column x is path x
                        int32_t lo = 0, hi = b;
                        while (lo < hi) {
                            const int32_t mid = (lo + hi) >> 1;
                            if (cols[c0 + mid].col < in.x) lo = mid + 1;
                            else hi = mid;
                        }
                        a = lo;
                        hi = b;
                        while (lo < hi) {
                            const int32_t mid = (lo + hi) >> 1;
                            if (cols[c0 + mid].col < in.x + in.y) lo = mid + 1;
                            else hi = mid;
                        }
                        b = lo;
                    }
                }
                double s0 = 0.0, sp = 0.0;
                for (int32_t c = a; c < b; ++c) {
                    const int32_t q = cols[c0 + c].col;
                    const double *p = R.B + 3 * ((int64_t) in.z + q);
                    if (p[0] < 0.0) continue;
                    seen = true;
                    const double xe = (R.ev[d - q - 1].x + M.var * mu - M.scale * mu - M.shift) / M.var;
                    for (int j = 0; j < 3; ++j) {
                        s0 += p[j] * xe;
                        sp += p[j];
                    }
                }
                double i0 = s0, ip = sp;   // inclusive scans in the reference's order (lane 0 first)
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double v0 = __shfl_up_sync(0xffffffffu, i0, o), vp = __shfl_up_sync(0xffffffffu, ip, o);
                    if (lane >= o) {
                        i0 += v0;
                        ip += vp;
                    }
                }
                double r0 = __shfl_up_sync(0xffffffffu, i0, 1), rp = __shfl_up_sync(0xffffffffu, ip, 1);
                r0 = e0 + (lane ? r0 : 0.0);
                rp = po + (lane ? rp : 0.0);
                double spread = 0.0;
                for (int32_t c = a; c < b; ++c) {
                    const int32_t q = cols[c0 + c].col;
                    const double *p = R.B + 3 * ((int64_t) in.z + q);
                    if (p[0] < 0.0) continue;
                    const double xe = (R.ev[d - q - 1].x + M.var * mu - M.scale * mu - M.shift) / M.var;
                    for (int j = 0; j < 3; ++j) {
                        r0 += p[j] * xe;
                        rp += p[j];
                        const double uk = r0 / rp;
                        spread += p[j] * (xe - uk) * (xe - uk);
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) spread += __shfl_xor_sync(0xffffffffu, spread, o);
                e1 += spread;
                e0 += __shfl_sync(0xffffffffu, i0, 31);
                po += __shfl_sync(0xffffffffu, ip, 31);
            }
        }
        c0 = c1;
    }
    seen = __any_sync(0xffffffffu, seen);
    if (lane == 0 && seen) {
        X.event_exp[2 * (int64_t) K.kid] = e0;
        X.event_exp[2 * (int64_t) K.kid + 1] = e1;
        X.posteriors[K.kid] = po;
        X.observed[K.kid] = 1;
    }
}

// A read's likelihood and transition expectations from its blocks' sums, a CTA per read.
__global__ void __launch_bounds__(256) finish64(const ExpectOut *XS, const int64_t *read_chunk, const double *partial) {
    __shared__ double sums[8][9];
    const ExpectOut &X = XS[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    double acc[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) acc[j] = 0.0;
    for (int64_t c = read_chunk[blockIdx.x] + tid; c < read_chunk[blockIdx.x + 1]; c += 256)
#pragma unroll
        for (int j = 0; j < 9; ++j) acc[j] += partial[9 * c + j];
#pragma unroll
    for (int j = 0; j < 9; ++j) {
        for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
        if (lane == 0) sums[warp][j] = acc[j];
    }
    __syncthreads();
    if (tid) return;
    for (int j = 0; j < 9; ++j) {
        acc[j] = 0.0;
        for (int w = 0; w < 8; ++w) acc[j] += sums[w][j];
    }
    X.acc[0] += acc[8];
    constexpr int to[8] = {S_M * 3 + S_X, S_X * 3 + S_X, S_Y * 3 + S_X, S_M * 3 + S_M,
                           S_X * 3 + S_M, S_Y * 3 + S_M, S_M * 3 + S_Y, S_Y * 3 + S_Y};
    for (int j = 0; j < 8; ++j) X.acc[1 + to[j]] += acc[j];
}
