// les_sor_res.cuh -- the whole red-black SOR loop in one launch, the pressure
// kept on the chip.
//
// A pass over HBM (k_sor1, k_sor1p) costs one march over the planes of a k
// chunk, about 1 us a plane: 23 us a pass at 150 x 150 x 90, where its bytes
// take 4, and 11 us at 24 x 20 x 16.  A grid whose p and rhs fit in the SMs'
// registers and shared memory need not move them between iterations at all.
// What fits is a matter of tiles, segments and threads, not of cells alone
// (res_plan): 257 x 203 x 61 does with 3.18 million cells, 195 x 195 x 80 with
// 3.04 does not (its columns are two segments of 40 planes, too many threads, or
// pad to 128).  So here
//   - a CTA owns a ti x tj tile of (i,j) columns, all km planes; the launch is
//     cooperative, one CTA per SM, and runs every iteration of the step;
//   - a thread owns one column's segment of SEG planes, its p in registers;
//     all cells of one colour are independent, so a half-sweep is SEG/2
//     independent updates per thread;
//   - columns are dealt to warps by class (x + y) & 1, so the planes a
//     half-sweep updates have one parity in a whole warp: k neighbours are
//     registers, no lane is idle, and the j and i neighbours of four updates
//     are one 16-byte shared load each.  Shared memory holds p by column, the
//     planes of each parity together, columns padded to an odd number of
//     16-byte words (no bank conflicts between the lanes of a quarter warp);
//   - a tile's edge columns are sent to the neighbouring tile's CTA after the
//     half-sweep that updated them, as 64-bit words {value, tag} written and
//     polled with relaxed loads and stores: the word that arrives is its own
//     flag (the method of NCCL's low-latency protocol), so an exchange costs one
//     trip through L2 and no fence.  The edge
//     columns are the first of each class, so only their warps wait; the other
//     warps work meanwhile.  Two slots per word suffice: a CTA sends
//     half-sweep s+2 only after it has received s+1 from the same neighbour
//     column, which that column sent after it had read s.
// What bounds it: latency.  At 150 x 150 x 90 a half-sweep takes 3.7 us, 6.7
// thousand cycles, with 12 warps an SM of which 29% of the issue slots are used;
// the warps wait at the CTA's barrier for those with edge columns (3.7 cycles per
// issue), for shared memory (1.9), for the neighbours' words (1.4) and for
// instructions (0.7: the unrolled loop is larger than the cache).  51 shared-memory
// wavefronts per four updates of a warp, exchange and bounds included.
// With one CTA (24 x 20 x 16) nothing is exchanged and a half-sweep takes 1.1 us.
// Measured, the SOR of a step (50 iterations), passes -> here: 24 x 20 x 16
// 585 -> 119 us, 61 x 47 x 35 607 -> 160, 150 x 150 x 90 1226 -> 373,
// 257 x 203 x 61 1618 -> 720.  Every segment length spills (12 to 232 bytes of
// stores): its p fills the registers.  Packed two-wide FP32 instructions (18%
// fewer instructions) gave nothing, and need a -0 the assembler cannot see: it
// contracts a packed multiply and add whatever --fmad says.
//
// Ghosts (press.f95:87-115 followed through, les_sor_tb.cuh): the i and k
// ghosts of a cell hold its own value before the update, and the j ghost its
// periodic partner's value before the half-sweep.  For odd jm the rows jm and
// 1 are of one class; the partner's planes of the other parity then arrive one
// half-sweep before they are read, which is the value press.f95 reads.
//
// Stop test: every iteration but the last sums reltmp^2 of one cell in four in
// FP32 (no term is negative, so that is a lower bound of the whole sum), checked
// against the bound of tb_finish_fast (here at most SEG + 32 + 5 + 5 + 5 adds
// from a term to the root).  The CTAs exchange the bounds as words {value, tag}
// and look at them while the loop runs, two iterations late, so that nobody waits;
// after the first four iterations one word carries the least bound of four.
// Where a look does not rule the stop out, all CTAs leave the attempt together
// and the loop runs again from the input p, which is unchanged in memory until
// it ends; from that batch on it sums exactly (les_fix.h) and decides before it
// goes on.  A step that stops after m iterations so costs 2m + 3 to 2m + 8 of them
// instead of the cap's (SOR of a step that stops after 10 of 50, looks at the end
// -> while it runs; the passes: 24 x 20 x 16 167 -> 79 us; 220, 61 x 47 x 35
// 235 -> 118; 235, 150 x 150 x 90 529 -> 271; 352, 257 x 203 x 61 927 -> 380; 440;
// after 10 of 1000 at 150 x 150 x 90 6132 -> 272; 1428).  The looks cost 0 to 4.5%
// of an SOR that runs to its cap (61 x 47 x 35 160 -> 160 us, 150 x 150 x 90
// 365 -> 373, 257 x 203 x 61 688 -> 720) and nothing where no stop is asked for.
// A stop that is only nearly reached (residuals within 4x of the threshold at the
// cap) leaves a batch open early and sums the rest exactly: 150 x 150 x 90 770 us,
// 257 x 203 x 61 1390, still below the passes' 1220 and 1600.
// Iteration counts, the residual and p are those of exact sums throughout.
//
// Every wait is bounded: past a.polls polls a thread gives up, the CTA
// returns without writing p, and the context reports LES_ERR_TIMEOUT.  Such a
// launch leaves words of its own tags behind and does not move ctl[2] on: the
// words and the control words are zeroed before the next step (res_clear), or
// that step would take them for its neighbours'.
#pragma once
#include "les_sor1.cuh"

namespace les {
namespace {

typedef unsigned long long u64;
// a lambda left out of line would move the register window it captures to local memory
#define LES_INLINE __attribute__((always_inline))
constexpr int kResPolls = 1 << 20;   // about a second (ResArgs::polls)
constexpr int kResList = 64;         // halo columns of one warp (at most two per column)
constexpr int kResCtas = 160;        // CTAs of a launch, at most
// Batches of iterations whose FP32 bounds travel as one word: the first four
// iterations one by one, then four each.
constexpr int kResBatch = 4;
__device__ __forceinline__ bool batch_ends(int l) { return l < kResBatch || l % kResBatch == kResBatch - 1; }
__device__ __forceinline__ int batch_of(int l) { return l < kResBatch ? l : kResBatch - 1 + l / kResBatch; }
__device__ __forceinline__ int batch_first(int l) { return l < kResBatch ? l : l / kResBatch * kResBatch; }

struct ResPlan {
    int seg = 0, nseg = 0;           // planes per thread (0: no plan), segments per column
    bool rg = false;                 // rhs in global scratch instead of shared memory
    int nti = 0, ntj = 0, ti = 0, tj = 0;
    int threads = 0, warps = 0;
    int pm = 0, nc = 0;              // columns per stored row and class, per class
    int lch = 0;                     // half the exchange slots along a side
    size_t smem = 0, ll_words = 0;   // shared bytes; 16-byte words of one exchange slot
    size_t rg_words() const { return rg ? (size_t)ncta() * (seg / 4) * threads : 0; }  // float4s of rhs scratch
    int ncta() const { return nti * ntj; }
};

struct ResArgs {
    float *p;
    const float *rhs;
    ulonglong2 *ll;      // exchange words, two slots
    float4 *rg;          // rhs [CTA][parity, group][thread] (RG)
    u64 *resid;          // FP32 bounds [batch of iterations][CTA], words {value, tag}
    FixPart *part;       // exact partial sums, two sets of one per CTA
    unsigned *ctl;       // [0] barrier arrivals, [1] barrier generation, [2] next tag
    int *err;            // host-mapped: a wait gave up
    Scal *sc;
    float c2, c3;        // cn2l = cn2s and cn3l = cn3s of every column
    int itmax, exact0;   // iterations; 1: exact sums from the first on
    int polls;           // of one wait before it gives up
    float pjuge;
    int nti, ntj, ti, tj, nseg, pm, nc, lch, warps;
    int ll_slot;         // words of one slot
    int rstride;         // words of one batch in resid (even)
};

__device__ __forceinline__ void ll_store(ulonglong2 *dst, float v0, float v1, unsigned tag) {
    const u64 t = (u64)tag << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(dst), "l"(t | __float_as_uint(v0)),
                 "l"(t | __float_as_uint(v1))
                 : "memory");
}
__device__ __forceinline__ ulonglong2 ll_load(const ulonglong2 *src) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(src) : "memory");
    return v;
}

// A word {value, tag}: its tag says whose value it is.
__device__ __forceinline__ void word_store(u64 *dst, float v, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(dst), "l"((u64)tag << 32 | __float_as_uint(v)) : "memory");
}
__device__ __forceinline__ u64 word_load(const u64 *src) {
    u64 w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(src) : "memory");
    return w;
}

// Two words into shared memory, from L2, without waiting.
__device__ __forceinline__ void word_fetch2(u64 *dst, const u64 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void word_fetch_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// All CTAs of the launch; true (in every thread) when the wait gave up.
__device__ __forceinline__ bool res_grid_barrier(const ResArgs &a, int ncta, int *s_abort) {
    __syncthreads();
    if (ncta > 1 && threadIdx.x == 0) {
        __threadfence();
        volatile unsigned *gen = a.ctl + 1;
        const unsigned g0 = *gen;
        __threadfence();
        if (atomicAdd(a.ctl, 1u) == (unsigned)ncta - 1u) {
            a.ctl[0] = 0u;
            __threadfence();
            *gen = g0 + 1u;
        } else {
            for (int it = 0; *gen == g0; ++it)
                if (it > a.polls || *(volatile int *)s_abort) {
                    *(volatile int *)s_abort = 1;
                    break;
                }
        }
        __threadfence();
    }
    return __syncthreads_or(*(volatile int *)s_abort);
}

// Threads a CTA may have (registers: SEG of p, the words in flight, about 45 more).
// (registers are dealt to four quarters of an SM: the count matters in steps of four warps)
constexpr int res_threads(int seg) { return seg <= 8 ? 1024 : seg <= 24 ? 768 : seg == 32 ? 640 : seg <= 48 ? 512 : 384; }

// RG (the longest segments): each thread's rhs stays in a global scratch that
// only it reads (16 bytes per four updates out of L2) instead of shared memory,
// which then holds p of up to 24 thousand cells per SM instead of about 20.
template <int SEG, bool RG>
__global__ void __launch_bounds__(res_threads(SEG), 1)
    k_sor_res(Geo g, ResArgs a, const __grid_constant__ TbKCoef kq) {
    constexpr int H = SEG / 2, NG = SEG / 8, NE = SEG / 4, CS = SEG + 4;
    // Long segments unroll to more code than the instruction cache keeps, so what
    // runs between iterations is fetched anew each time: there the bounds are
    // summed once per batch and their loops stay rolled (150 x 150 x 90: SOR to
    // its cap 391 -> 371 us, 257 x 203 x 61 736 -> 719).  Short ones wait for the
    // latencies of a rolled loop instead (24 x 20 x 16: 119 -> 127).
    constexpr bool LONG = SEG >= 40;
    constexpr int UL = LONG ? 1 : 32;  // unrolling of those loops
    extern __shared__ float4 rsm4[];
    __shared__ int s_abort, s_cnt[4], s_stop, s_look[2];
    __shared__ float s_min;
    __shared__ __align__(16) u64 s_words[kResCtas];
    Scal *const sc = a.sc;
    const int im = g.im, jm = g.jm, km = g.km, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int ncta = a.nti * a.ntj, cta = blockIdx.x, tx = cta % a.nti, ty = cta / a.nti;
    const int i0 = 1 + tx * a.ti, j0 = 1 + ty * a.tj;
    const int nx = min(a.ti, im - i0 + 1), ny = min(a.tj, jm - j0 + 1);  // this tile's columns and rows
    // shared memory: p [segment][class][column][parity][plane] and rhs
    // [thread][parity][plane], both padded to an odd number of 16-byte words per
    // column or thread; coefficients [segment][parity][c4l, c4s, cn1][plane], FP32
    // residuals [iteration & 1][thread], halo lists [warp], column lists
    // [class].  Every offset inside a column, thread or segment is a constant.
    float *const S = reinterpret_cast<float *>(rsm4);
    const int SS = 2 * a.nc * CS;  // floats of one segment
    float *const Rs = S + a.nseg * SS;
    float *const T = RG ? Rs : Rs + blockDim.x * CS;
    float4 *const Rg = RG ? a.rg + (size_t)blockIdx.x * 2 * NG * blockDim.x + threadIdx.x : nullptr;
    float *const sumf = T + a.nseg * 6 * H;
    int2 *const hlist = reinterpret_cast<int2 *>(sumf + 2 * blockDim.x);
    short2 *const clist = reinterpret_cast<short2 *>(hlist + a.warps * kResList);
    const int ncl = (a.ti * a.tj + 1) / 2 + 1;  // columns of one class, at most
    auto colof = [&](int x, int y) {            // first float of a column in its segment
        return (((x + y) & 1) * a.nc + (y + 1) * a.pm + ((x + 1) >> 1)) * CS;
    };
    const bool jodd = (jm & 1) != 0, jself = a.ntj == 1 && !jodd;
    // sides 0 west, 1 east, 2 south, 3 north that another tile's column (or,
    // for one tile row and odd jm, this tile's own other end) sends
    auto ext = [&](int x, int y, int side) {
        if (side == 0) return x == 0 && tx > 0;
        if (side == 1) return x == nx - 1 && tx < a.nti - 1;
        if (side == 2) return y == 0 && !jself;
        return y == ny - 1 && !jself;
    };
    if (tid == 0) s_abort = 0, s_look[0] = s_look[1] = -1;
    // coefficient tables and zeroed columns (padded planes stay 0)
    for (int t = tid; t < a.nseg * 6 * H; t += blockDim.x) {
        const int q = t / (3 * H) % 2, w = t / H % 3, k = 1 + t / (6 * H) * SEG + 2 * (t % H) + q;
        T[t] = k > km ? 0.0f : (w == 0 ? kq.c4l[k] : (w == 1 ? kq.c4s[k] : kq.cnk[k]));
    }
    for (int t = tid; t < a.nseg * SS; t += blockDim.x) S[t] = 0.0f;
    // the columns of each class, those with a side to exchange first
    if (wid < 2) {
        int n = 0;
        for (int pass = 0; pass < 2; ++pass) {
            for (int c0 = 0; c0 < nx * ny; c0 += 32) {
                const int c = c0 + lane, x = c % nx, y = c / nx;
                bool take = c < nx * ny && ((x + y) & 1) == wid;
                if (take) {
                    const bool e = ext(x, y, 0) || ext(x, y, 1) || ext(x, y, 2) || ext(x, y, 3);
                    take = e == (pass == 0);
                }
                const unsigned m = __ballot_sync(0xffffffffu, take);
                if (take) clist[wid * ncl + n + __popc(m & ((1u << lane) - 1u))] = make_short2((short)x, (short)y);
                n += __popc(m);
            }
            if (lane == 0) s_cnt[pass * 2 + wid] = n;
        }
    }
    __syncthreads();
    const int nW0 = (s_cnt[2] + 31) / 32, nW1 = (s_cnt[3] + 31) / 32, nWs = nW0 + nW1;
    const int seg = wid / max(nWs, 1), widx = wid % max(nWs, 1);
    const int cls = widx < nW0 ? 0 : 1, cw = cls ? widx - nW0 : widx;
    const bool wact = seg < a.nseg;                          // warps past the tile's columns only keep the barriers
    const int crank = cw * 32 + lane;
    const bool act = wact && crank < s_cnt[2 + cls];
    const bool wedge = wact && cw * 32 < s_cnt[cls];         // the warp has columns with a side to exchange
    const short2 xy = act ? clist[cls * ncl + crank] : (wact ? clist[cls * ncl] : make_short2(0, 0));
    const int x = xy.x, y = xy.y, i = i0 + x, j = j0 + y;
    const int gcls = (i0 + j0 + cls) & 1;                    // (i + j) & 1 of the warp's columns
    const int own = seg * SS + colof(x, y);
    // neighbours: the i ghosts are the cell itself
    const int offW = (i == 1) ? own : seg * SS + colof(x - 1, y);
    const int offE = (i == im) ? own : seg * SS + colof(x + 1, y);
    const int offS = seg * SS + ((y == 0 && jself) ? colof(x, ny - 1) : colof(x, y - 1));
    const int offN = seg * SS + ((y == ny - 1 && jself) ? colof(x, 0) : colof(x, y + 1));
    const float c2 = a.c2, c3 = a.c3;
    // word of one halo column in the receiving CTA's slot (its NE words of a
    // segment lie 2*lch apart)
    auto word = [&](int rcta, int side, int along) {
        return ((rcta * 4 + side) * a.nseg + seg) * NE * 2 * a.lch + (along & 1) * a.lch + (along >> 1);
    };
    // where this column is sent, and the warp's halo columns: {shared column
    // | parity flag, word}
    int dst0 = -1, dst1 = -1, hcnt = 0;
    if (wedge) {
        const int tys = ty == 0 ? a.ntj - 1 : ty - 1, tyn = ty == a.ntj - 1 ? 0 : ty + 1;
        for (int side = 0; side < 4; ++side) {
            const bool e = act && ext(x, y, side);
            if (e) {
                const int rc = side == 0 ? cta - 1 : (side == 1 ? cta + 1 : (side == 2 ? tys : tyn) * a.nti + tx);
                const int d = word(rc, side ^ 1, side < 2 ? y : x);
                if (dst0 < 0)
                    dst0 = d;
                else
                    dst1 = d;
            }
            const unsigned m = __ballot_sync(0xffffffffu, e);
            if (e) {
                const int h = hcnt + __popc(m & ((1u << lane) - 1u));
                const int col = side == 0 ? offW : (side == 1 ? offE : (side == 2 ? offS : offN));
                // odd jm: across the periodic boundary the sender is of this column's class
                const int same = jodd && ((side == 2 && ty == 0) || (side == 3 && ty == a.ntj - 1));
                hlist[wid * kResList + h] = make_int2(col * 2 + same, word(cta, side, side < 2 ? y : x));
            }
            hcnt += __popc(m);
        }
        __syncwarp();
    }
    const int kbase = 1 + seg * SEG;
    const int rt = km - kbase;  // index of plane km in this segment (>= SEG: above it)
    const long long pstride = (long long)g.si * g.sj;
    // the thread's column of a box at plane kbase (looked up again where it is
    // used, so that nothing of it stays in registers through the loop)
    auto column = [&]() {
        const short2 c = clist[cls * ncl + (act ? cw * 32 + lane : 0)];
        return (long long)IX(g, i0 + c.x, j0 + c.y, 0) + pstride * kbase;
    };
    {
        const float rhsav = sc->rhsav;
        const float *const bcol = a.rhs + (act ? column() : 0);
        for (int gq = 0; gq < 2 * NG; ++gq) {
            const int q = gq / NG, gg = gq % NG;
            float b[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int r = 8 * gg + 2 * c + q;
                b[c] = act && r <= rt ? bcol[pstride * r] - rhsav : 0.0f;
            }
            const float4 b4 = make_float4(b[0], b[1], b[2], b[3]);
            if (RG)
                Rg[gq * blockDim.x] = b4;
            else
                *reinterpret_cast<float4 *>(Rs + tid * CS + 4 * gq) = b4;
        }
    }
    const unsigned tag0 = a.ctl[2];  // moved on after the last barrier of the launch
    unsigned tag = tag0;
    int exact_from = a.exact0 ? 0 : a.itmax - 1;
    const bool stops = a.pjuge > 0.0f;  // (a sum of squares is not below 0)
    float P[2][H];  // the column's planes of each parity

    for (int attempt = 0;; ++attempt) {
        // p of the segment and of its halo columns, from memory
        const float *const gin = a.p + (act ? column() : 0);
#pragma unroll
        for (int r = 0; r < SEG; ++r) P[r & 1][r >> 1] = (act && r <= rt) ? gin[pstride * r] : 0.0f;
        if (act)
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int m = 0; m < H; ++m) S[own + q * H + m] = P[q][m];
        if (wedge && act) {
            const short2 c = clist[cls * ncl + cw * 32 + lane];
            const int x = c.x, y = c.y, i = i0 + x, j = j0 + y;
            for (int side = 0; side < 4; ++side)
                if (ext(x, y, side)) {
                    const int ii = side == 0 ? i - 1 : (side == 1 ? i + 1 : i);
                    int jj = side == 2 ? j - 1 : (side == 3 ? j + 1 : j);
                    jj = jj < 1 ? jm : (jj > jm ? 1 : jj);
                    const float *hc = a.p + (IX(g, ii, jj, 0) + pstride * kbase);
                    const int col = side == 0 ? offW : (side == 1 ? offE : (side == 2 ? offS : offN));
                    for (int r = 0; r < SEG; ++r)
                        if (r <= rt) S[col + (r & 1) * H + (r >> 1)] = hc[pstride * r];
                }
        }
        __syncthreads();

        float fs = 0.0f;       // FP32 sum of reltmp^2
        float fm = 0.0f;       // its least in the batch (LONG)
        u64 fh = 0, flo = 0;   // exact sum
        int bad = 0;
        // One half-sweep of the thread's planes of parity Q, sent with tag t;
        // EX: exact sums.
        auto half = [&](auto Qc, auto EXc, unsigned t) LES_INLINE {
            constexpr int Q = decltype(Qc)::value;
            constexpr bool EX = decltype(EXc)::value;
            const float *const Tq = T + seg * 6 * H + Q * 3 * H;
            // the neighbour across the segment's end: below plane kbase (Q 0),
            // above plane kbase+SEG-1 (Q 1)
            float seam = 0.0f;
            if (Q == 0)
                seam = seg == 0 ? P[0][0] : S[own - SS + SEG - 1];
            else if (seg < a.nseg - 1)
                seam = S[own + SS];
            // four updates; TOP: plane km or planes past it among them
            auto four = [&](auto Gc, auto TOPc) LES_INLINE {
                constexpr int gg = decltype(Gc)::value;
                constexpr bool top = decltype(TOPc)::value;
                const float4 vw = *reinterpret_cast<const float4 *>(S + offW + Q * H + 4 * gg);
                const float4 ve = *reinterpret_cast<const float4 *>(S + offE + Q * H + 4 * gg);
                const float4 vs = *reinterpret_cast<const float4 *>(S + offS + Q * H + 4 * gg);
                const float4 vn = *reinterpret_cast<const float4 *>(S + offN + Q * H + 4 * gg);
                const float4 l4 = *reinterpret_cast<const float4 *>(Tq + 4 * gg),
                             s4 = *reinterpret_cast<const float4 *>(Tq + H + 4 * gg),
                             cn = *reinterpret_cast<const float4 *>(Tq + 2 * H + 4 * gg);
                const float4 b = RG ? Rg[(Q * NG + gg) * blockDim.x]
                                    : *reinterpret_cast<const float4 *>(Rs + tid * CS + Q * H + 4 * gg);
                const float w4[4] = {vw.x, vw.y, vw.z, vw.w}, e4[4] = {ve.x, ve.y, ve.z, ve.w},
                            n4[4] = {vn.x, vn.y, vn.z, vn.w}, o4[4] = {vs.x, vs.y, vs.z, vs.w},
                            cl[4] = {l4.x, l4.y, l4.z, l4.w}, cs[4] = {s4.x, s4.y, s4.z, s4.w},
                            cc[4] = {cn.x, cn.y, cn.z, cn.w}, bb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    constexpr int m0 = 4 * gg;
                    const int m = m0 + h;  // plane r = 2m + Q
                    const float pc = P[Q][m];
                    float pu, pd;  // planes above and below
                    if (Q == 0) {
                        pu = P[1][m];
                        pd = m == 0 ? seam : P[1][m == 0 ? 0 : m - 1];
                    } else {
                        pu = m + 1 < H ? P[0][m + 1 < H ? m + 1 : m] : seam;
                        pd = P[0][m];
                    }
                    if (top && 2 * m + Q == rt) pu = pc;  // plane km's upper ghost is the cell itself
                    const float rel = cc[h] * (c2 * e4[h] + c2 * w4[h] + c3 * n4[h] + c3 * o4[h] + cl[h] * pu +
                                               cs[h] * pd - bb[h]) -
                                      pc;  // omega = 1
                    P[Q][m] = pc + rel;
                    if (EX) {
                        if (act) fix_add_nonneg(rel * rel, fh, flo, bad);
                    } else if (h == 0) {
                        fs += rel * rel;  // one cell in four: a lower bound all the same
                    }
                }
            };
            auto group = [&](auto Gc) LES_INLINE {
                constexpr int gg = decltype(Gc)::value;
                if constexpr (gg < NG) {
                    if (8 * gg + 8 <= rt)
                        four(Gc, std::false_type());
                    else if (8 * gg + Q <= rt)
                        four(Gc, std::true_type());
                }
            };
            group(IC<0>());
            group(IC<1>());
            group(IC<2>());
            group(IC<3>());
            group(IC<4>());
            group(IC<5>());
            group(IC<6>());
            group(IC<7>());
            // the stores last: no load of a later group waits behind one
            if (act)
#pragma unroll
                for (int gg = 0; gg < NG; ++gg)
                    *reinterpret_cast<float4 *>(S + own + Q * H + 4 * gg) =
                        make_float4(P[Q][4 * gg], P[Q][4 * gg + 1], P[Q][4 * gg + 2], P[Q][4 * gg + 3]);
            if (wedge) {  // and the neighbours' copies
                ulonglong2 *const dst = a.ll + (size_t)(t & 1u) * a.ll_slot;
                if (dst0 >= 0)
#pragma unroll
                    for (int q = 0; q < NE; ++q) ll_store(dst + dst0 + q * 2 * a.lch, P[Q][2 * q], P[Q][2 * q + 1], t);
                if (dst1 >= 0)
#pragma unroll
                    for (int q = 0; q < NE; ++q) ll_store(dst + dst1 + q * 2 * a.lch, P[Q][2 * q], P[Q][2 * q + 1], t);
            }
        };
        // Receive what the neighbours sent (tag t) for planes of parity Q: all
        // words of a halo column are asked for together, again until each has
        // arrived.
        auto receive = [&](int Q, unsigned t) LES_INLINE {
            const ulonglong2 *const src = a.ll + (size_t)(t & 1u) * a.ll_slot;
            for (int h = lane; h < hcnt; h += 32) {
                const int2 e = hlist[wid * kResList + h];
                ulonglong2 v[NE];
                for (int it = 0;;) {
                    bool ok = true;
#pragma unroll
                    for (int q = 0; q < NE; ++q) v[q] = ll_load(src + e.y + q * 2 * a.lch);
#pragma unroll
                    for (int q = 0; q < NE; ++q)
                        ok = ok && (unsigned)(v[q].x >> 32) == t && (unsigned)(v[q].y >> 32) == t;
                    if (ok) break;
                    if (++it > a.polls || *(volatile int *)&s_abort) {
                        *(volatile int *)&s_abort = 1;
                        break;
                    }
                }
                float *const col = S + (e.x >> 1) + ((e.x & 1) ? 1 - Q : Q) * H;
#pragma unroll
                for (int q = 0; q < NE; ++q)
                    *reinterpret_cast<float2 *>(col + 2 * q) =
                        make_float2(__uint_as_float((unsigned)v[q].x), __uint_as_float((unsigned)v[q].y));
            }
            __syncwarp();
        };
        int restart = -1, done = 0;
        bool gave_up = false;  // the same in every thread
        // Whether a sum over the lanes' v leaves it open that the SOR stops
        // (tb_finish_fast's bound).
        auto open_bound = [&](float v) LES_INLINE {
#pragma unroll UL
            for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const float lb = __fsub_rd(__fmul_rd(v, 0.99609375f), 0x1p-33f);
            return !(lb >= a.pjuge && lb < 0x1p40f);
        };
        // The same for the batch that ends with iteration it, from the words of
        // all CTAs (the same sum in every CTA), by one warp: the words fetched
        // into s_words, or polled where one was not there yet.
        auto words_of = [&](int it) { return a.resid + (size_t)batch_of(it) * a.rstride; };
        auto open_batch = [&](int it, bool fetched) LES_INLINE {
            const unsigned t = tag0 + 2u * (unsigned)(it + 1);
            float v = 0.0f;
            bool there = fetched;
            if (fetched)
#pragma unroll UL
                for (int q = 0; q < kResCtas / 32; ++q)
                    if (lane + 32 * q < ncta) {
                        const u64 w = s_words[lane + 32 * q];
                        v += __uint_as_float((unsigned)w);
                        there = there && (unsigned)(w >> 32) == t;
                    }
            if (!__all_sync(0xffffffffu, there)) {
                v = 0.0f;
#pragma unroll 1
                for (int b = lane; b < ncta; b += 32) {
                    u64 w = word_load(words_of(it) + b);
                    for (int n = 0; (unsigned)(w >> 32) != t; ++n) {
                        if (n > a.polls || *(volatile int *)&s_abort) {
                            *(volatile int *)&s_abort = 1;
                            break;
                        }
                        w = word_load(words_of(it) + b);
                    }
                    v += __uint_as_float((unsigned)w);
                }
                __syncwarp();
            }
            return open_bound(v);
        };
        // At the end of iteration l: the batch that ended two iterations ago, and
        // the fetch of the one that ended in the last.  With short segments, where
        // the warps wait more than they issue, by another warp than the one that
        // sums this CTA's terms (61 x 47 x 35: SOR 161 us, one warp for both 170);
        // with long ones by the same (150 x 150 x 90: 370, two warps 383).
        auto look = [&](int l) LES_INLINE {
            if (l >= 2 && batch_ends(l - 2)) {
                word_fetch_wait();
                __syncwarp();
                if (open_batch(l - 2, true) && lane == 0) s_look[l & 1] = batch_first(l - 2);
                __syncwarp();
            }
            if (l >= 1 && batch_ends(l - 1))
#pragma unroll UL
                for (int b = 2 * lane; b < ncta; b += 64) word_fetch2(s_words + b, words_of(l - 1) + b);
        };
        // One half-sweep; FIRST: of the attempt (its halo columns came from memory).
        auto sweep = [&](auto Qc, auto EXc, bool first) LES_INLINE {
            if (wedge && !first) receive(decltype(Qc)::value, tag);
            ++tag;
            if (wact) half(Qc, EXc, tag);
        };
        // One iteration: colour 0 then colour 1 of press.f95 (a warp's planes of
        // parity gcls, then the others).
        auto iterate = [&](auto EXc, bool first) LES_INLINE {
#pragma unroll 1
            for (int nrd = 0; nrd < 2; ++nrd) {
                if (nrd) __syncthreads();
                if ((gcls + nrd) & 1)
                    sweep(IC<1>(), EXc, first && nrd == 0);
                else
                    sweep(IC<0>(), EXc, first && nrd == 0);
            }
        };
        int l = 0;
        for (; l < exact_from; ++l) {
            fs = 0.0f;
            iterate(std::false_type(), l == 0);
            // this iteration's FP32 terms (LONG: each thread's least of the batch's
            // iterations, whose sum is below the sum of each; a NaN stays): summed by
            // the CTA's last warp while the others go on (the slots are written again
            // two barriers later)
            const bool ends = batch_ends(l) || l == exact_from - 1, sums = !LONG || ends;
            float *f = sumf + (l & 1) * blockDim.x;
            if (LONG && (batch_first(l) == l || fs < fm || fs != fs)) fm = fs;
            if (sums) f[tid] = act ? (LONG ? fm : fs) : 0.0f;  // (idle lanes carry a column's seam values)
            // (or the look that ended in this iteration left a stop open: it was
            // written before the barrier between the half-sweeps, and every CTA's
            // look finds the same, so all leave the attempt here)
            if (__syncthreads_or(*(volatile int *)&s_abort | (s_look[(l + 1) & 1] >= 0))) {
                gave_up = true;
                break;
            }
            if (attempt == 0 && stops) {
                if (wid == a.warps - 1) {
                    if (sums) {
                        float v = 0.0f;
                        if (LONG) {
#pragma unroll 1
                            for (int t = lane; t < (int)blockDim.x; t += 32) v += f[t];
                        } else {
                            for (int t = lane; t < (int)blockDim.x; t += 32) v += f[t];
                        }
                        if (ncta == 1) {
                            if (open_bound(v) && lane == 0) s_look[l & 1] = LONG ? batch_first(l) : l;
                            continue;
                        }
#pragma unroll UL
                        for (int o = 16; o >= 1; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
                        if (lane == 0) {
                            // the least of the batch, summed over the CTAs, is below each
                            // iteration's sum (a NaN stays)
                            if (!LONG) {
                                if (batch_first(l) < l && !(v < s_min) && v == v) v = s_min;
                                s_min = v;
                            }
                            if (ends) word_store(words_of(l) + cta, v, tag);
                        }
                    }
                    if (LONG && ncta > 1) look(l);
                } else if (!LONG && wid == a.warps - 2 && ncta > 1) {
                    look(l);
                }
            }
        }
        word_fetch_wait();
        if (gave_up) {
            restart = s_look[(l + 1) & 1];
            gave_up = restart < 0 || res_grid_barrier(a, ncta, &s_abort);  // all have left the attempt
            if (tid == 0) s_look[0] = s_look[1] = -1;
        }
        for (; l < a.itmax && !gave_up && restart < 0; ++l) {
            fh = flo = 0;
            bad = 0;
            iterate(std::true_type(), l == 0);
            gave_up = __syncthreads_or(*(volatile int *)&s_abort);
            if (gave_up) break;
            // exact sum of iteration l over all CTAs, and its stop test
            FixPart *part = a.part + (size_t)(l & 1) * ncta;
            block_fix_sum_any((i128)(((unsigned __int128)fh << 64) | (unsigned __int128)flo), bad, part + cta);
            gave_up = res_grid_barrier(a, ncta, &s_abort);
            if (gave_up) break;
            if (l == exact_from && attempt == 0 && l > 0 && stops) {
                // the batches whose look is still to come or was not acted on:
                // the first that does not rule the stop out
                if (tid == 0) s_stop = INT_MAX;
                __syncthreads();
                for (int t = max(0, l - 3 - kResBatch) + wid; t < l; t += a.warps) {
                    const bool u = ncta == 1 ? t == l - 1 && s_look[t & 1] >= 0
                                             : (batch_ends(t) || t == l - 1) && open_batch(t, false);
                    if (lane == 0 && u) atomicMin(&s_stop, ncta == 1 ? s_look[t & 1] : batch_first(t));
                }
                __syncthreads();
                if (s_stop != INT_MAX) restart = s_stop;
                __syncthreads();
                if (restart >= 0) break;
            }
            // (read past L1, which keeps what an earlier iteration left in the slot)
            i128 tot = 0;
            int tbad = 0;
            if (wid == 0) {
                for (int b = lane; b < ncta; b += 32) {
                    FixPart fp;
                    fp.lo = __ldcg(&part[b].lo);
                    fp.hi = __ldcg(&part[b].hi);
                    tot += fix_from_part(fp);
                    tbad |= __ldcg(&part[b].bad);
                }
                for (int o = 16; o >= 1; o >>= 1) {
                    tot += shfl_down_i128(tot, o);
                    tbad |= __shfl_down_sync(0xffffffffu, tbad, o);
                }
            }
            if (tid == 0) {
                const float sor = (float)fix_finish(tot, tbad);
                s_stop = sor < a.pjuge ? 1 : 0;
                if (cta == 0) {
                    sc->sor = sor;
                    sc->sor_iters = l + 1;
                    sc->converged = s_stop;
                }
            }
            __syncthreads();
            done = s_stop;
            __syncthreads();
            if (done) break;
        }
        if (gave_up) {
            if (tid == 0) *(volatile int *)a.err = 1;
            return;
        }
        if (restart < 0) break;
        exact_from = restart;
        tag += 2u;  // the abandoned attempt's words are never taken for the next one's
    }
    float *const gout = a.p + (act ? column() : 0);
#pragma unroll
    for (int r = 0; r < SEG; ++r)
        if (act && r <= rt) gout[pstride * r] = P[r & 1][r >> 1];
    if (cta == 0 && tid == 0) a.ctl[2] = tag + 2u;
}

}  // namespace
}  // namespace les
