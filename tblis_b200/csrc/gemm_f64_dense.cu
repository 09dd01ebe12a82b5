// gemm_f64_dense.cu -- the dense FP64 contraction kernel: one persistent,
// warp-specialised CTA per SM over the GEMM view of strided tensors.
//
// Replaces TBLIS's pack + microkernel + scatter-accumulate chain
// (src/nodes/packm.hpp:79-124, src/kernels/3m/packm.hpp:292-403,
// src/nodes/gemm_ukr.hpp:16-126) for one contraction: operand tiles are
// gathered straight from the strided tensors through the scatter vectors, the
// alpha/beta update of C is scattered back from the accumulators, and
// beta == 0 never reads C.
//
// What bounds it: the FP64 tensor pipe (DMMA, 64 FMA per cycle and SM).
// A 64 x 64 tile needs 16 operand bytes per cycle and SM from L2 at that
// rate, 4.5 TB/s over the chip, and its CTA-wide barriers stop all warps once
// per 16 k; it measured 29.7 TFLOP/s at 7680^3. Here a tile is 128 x 128 (8
// bytes per cycle and SM), four producer warps gather it with cp.async into a
// ring of 16-wide k stages whose mbarriers they alone feed, and eight consumer
// warps (two per SM sub-core, so one's fragment loads hide behind the other's
// MMAs) release each stage as soon as its fragments are in registers. No
// barrier spans the CTA after the start. Measured against the 64 x 64 kernel: 7680^3
// in 26.6 ms (30.2; cuBLAS 25.3), 97 x 97 x 93217 in 100 us (283), 3007^3 with permuted
// operands in 1.77 ms (2.88; 1.92 and 2.97 with the copy of a residual before it),
// complex 1728^3 in 1.31 ms (2.50 as four real contractions).
//
// Fragments are dealt to the warps cyclically (16-row fragment f of the tile
// to row-warp f % WGM, 8-column fragment g to column-warp g % WGN), and
// fragments past M or N are neither gathered nor multiplied, so a ragged
// edge costs what it holds, evenly over the sub-cores, instead of a tile.
//
// Work split: whole waves of whole tiles go to the CTAs in launch order
// (neighbouring CTAs share A and B panels in L2); the whole tiles left over, one
// more wave of them and all ragged tiles are cut into runs of k steps of equal
// cost, one per CTA, so no SM idles in the last wave and a contraction of few
// tiles and a long sum still fills the chip. A run that covers part of a
// tile leaves its accumulators in a workspace (at most two per CTA) and
// gemm_f64_fixup sums them in CTA order: the result does not depend on
// scheduling, and no kernel waits for another CTA.
//
// Every wait is bounded (2 s of wall clock): one that gives up ends the CTA's
// work and records the error for the host (gemm_f64_dense_error_flag); part of C
// is then not written.
#include "gemm_f64.hpp"
#include "gemm_f64_dev.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace tb
{

namespace
{

using namespace f64dev;

constexpr int DN_PRODUCERS = 4, DN_CONSUMERS = 8;           // warps (per team of producers)
constexpr int DN_PT = DN_PRODUCERS*32, DN_CT = DN_CONSUMERS*32;
constexpr unsigned long long DN_WAIT_NS = 2000000000ull;    // 2 s
constexpr unsigned long long DN_WAIT_MIN_NS = 10000000ull;  // no limit is below 10 ms: short waits need not read theirs
// registers per thread at launch, and after the split between the roles (a sum
// over the warps above the launch's would wait forever)
constexpr int dn_threads(int teams) { return teams*DN_PT + DN_CT; }
constexpr int dn_reg_launch(int teams) { return teams == 1 ? 168 : 128; }
constexpr int dn_reg_p(int teams) { return teams == 1 ? 104 : 72; }
constexpr int dn_reg_c(int teams) { return teams == 1 ? 200 : 184; }
static_assert(DN_PT*dn_reg_p(1) + DN_CT*dn_reg_c(1) <= dn_threads(1)*dn_reg_launch(1), "register split");
static_assert(2*DN_PT*dn_reg_p(2) + DN_CT*dn_reg_c(2) <= dn_threads(2)*dn_reg_launch(2), "register split");

// the CTA's state of failure, in shared memory: its waits give up together
struct DnFail
{
    int abort;
    unsigned long long limit; // of a wait, ns
};

// records for the host that this CTA gave up (once, at a role's end: the waits are
// inlined in many places, and a longer kernel starts later)
__device__ __forceinline__ void dn_report(int* error)
{
    *(volatile int*)error = 1;            // mapped host memory
    __threadfence_system();
}

// smem position of element (row, k) of an operand tile of R rows and 16 k.
// MODE 0 (gathered along the rows): k rows of R doubles; MODE 1 (along k):
// rows of 16 doubles. XOR swizzles in units of four doubles keep the 8 x 4
// fragment reads free of bank conflicts and element pairs adjacent.
template <int R, int MODE>
__device__ __forceinline__ int tile_pos(int row, int k)
{
    return MODE == 0 ? k*R + (row ^ ((k & 3) << 2)) : row*BK + (k ^ ((row & 3) << 2));
}

__device__ __forceinline__ bool dn_wait_slow(uint64_t* b, uint32_t parity, volatile DnFail* fail)
{
    const unsigned long long t0 = gtimer();
    for (unsigned it = 0;; it++)
    {
        if (mb_try(b, parity)) return true;
        if ((it & 63) == 0)
        {
            if (fail->abort) return false;
            const unsigned long long waited = gtimer() - t0;
            if (waited > DN_WAIT_MIN_NS && waited > fail->limit)
            {
                fail->abort = 1;
                return false;
            }
        }
    }
}

__device__ __forceinline__ bool dn_wait(uint64_t* b, uint32_t parity, volatile DnFail* fail)
{
    const bool ok = mb_try(b, parity) || dn_wait_slow(b, parity, fail);
    return __all_sync(0xffffffffu, ok) != 0;
}

// one run of k steps of one tile
struct Run
{
    unsigned tile;
    int s0, s1;               // k steps [s0, s1)
    int slot;                 // -1: the whole tile (C is updated), else the CTA's workspace slot
};

// Tiles are numbered class by class: whole tiles, the ragged last row of tiles,
// the ragged last column, the corner; a class costs cls_w per k step. The k
// steps ("units") of the cut tiles are dealt so that every CTA gets the same
// cost: CTA c starts at the first unit at or past cost c*sk_per + min(c,
// sk_extra).

// cost of the units before unit u (of the cut tiles)
__device__ __forceinline__ unsigned unit_cost(const GemmF64Args& p, unsigned u)
{
    const unsigned kt = (unsigned)p.kt, tile = u/kt, step = u - tile*kt;
    unsigned cost = 0;
    #pragma unroll
    for (int c = 0; c < 4; c++)
    {
        // the cut tiles of class c, counted from the first cut one
        const unsigned b = p.cls_first[c], e = p.cls_first[c + 1];
        const unsigned n = min(max(tile, b), e) - b;
        cost += n*kt*p.cls_w[c];
        if (tile >= b && tile < e) cost += step*p.cls_w[c];
    }
    return cost;
}

// first unit of CTA c
__device__ __forceinline__ unsigned first_unit(const GemmF64Args& p, unsigned c)
{
    unsigned at = c*p.sk_per + min(c, p.sk_extra);
    const unsigned kt = (unsigned)p.kt;
    #pragma unroll
    for (int k = 0; k < 4; k++)
    {
        const unsigned b = p.cls_first[k], e = p.cls_first[k + 1], w = p.cls_w[k];
        const unsigned all = (e - b)*kt*w;
        if (at <= all && e > b) return b*kt + (at + w - 1)/w;
        at -= all;
    }
    return p.cls_first[4]*kt;
}

// the CTA that holds unit u
__device__ __forceinline__ unsigned cta_of_unit(const GemmF64Args& p, unsigned u)
{
    const unsigned at = unit_cost(p, u), big = p.sk_extra*(p.sk_per + 1);
    return at < big ? at/(p.sk_per + 1) : p.sk_extra + (at - big)/p.sk_per;
}

// Run number r of CTA `cta`: its whole tiles, then its share of the k steps of
// the cut tiles [dp_tiles, dp_tiles + sk_tiles). Computed anew from r where it
// is needed, so that the accumulators have the registers. 32-bit arithmetic:
// the plan keeps tiles and units below 2^31.
__device__ __forceinline__ bool run_at(const GemmF64Args& p, unsigned cta, unsigned r, Run& out)
{
    const unsigned kt = (unsigned)p.kt, dp = (unsigned)p.dp_tiles;
    const unsigned mine = r*gridDim.x + cta;
    if (mine < dp)
    {
        out = Run{mine, 0, (int)kt, -1};
        return true;
    }
    if (cta >= (unsigned)p.sk_ctas) return false;
    const unsigned nd = dp > cta ? (dp - cta - 1)/gridDim.x + 1 : 0;
    const unsigned u0 = first_unit(p, cta), u1 = first_unit(p, cta + 1);
    const unsigned t0 = u0/kt, t = t0 + (r - nd);
    const unsigned b = max(u0, t*kt), e = min(u1, (t + 1)*kt);
    if (b >= e) return false;
    out.tile = dp + t;
    out.s0 = (int)(b - t*kt);
    out.s1 = (int)(e - t*kt);
    // a partial run takes slot 0, the second one (after a first run that is
    // part of an earlier tile) slot 1
    out.slot = e - b == kt ? -1 : t > t0 && u0 != t0*kt ? 1 : 0;
    return true;
}

struct TileAt
{
    i64 m0, n0;
    unsigned l;
    int mrem, nrem;           // rows and columns of the tile inside the GEMM
};

// Whole tiles: groups of 8 tile rows sweep the tile columns together, so
// concurrent CTAs share panels of both operands in L2; then the ragged tiles.
template <int BM, int BN>
__device__ __forceinline__ TileAt tile_at(const GemmF64Args& p, unsigned tile)
{
    const i64 N = p.cplx ? 2*p.N : p.N;                       // real columns
    const unsigned fm = (unsigned)(p.M/BM), fn = (unsigned)(N/BN);
    const unsigned L = (unsigned)p.L, whole = fm*fn, bottom = p.M % BM ? fn : 0, right = N % BN ? fm : 0;
    TileAt t;
    t.l = 0;
    unsigned row = fm, col = fn;
    auto split = [&](unsigned n) { if (L > 1) { t.l = tile/n; tile -= t.l*n; } };
    if (tile < whole*L)
    {
        split(whole);
        const unsigned gid = tile/(8*fn), first = gid*8, in = tile - gid*8*fn;
        const unsigned gs = min(8u, fm - first);
        col = in/gs;
        row = first + in - col*gs;
    }
    else if ((tile -= whole*L) < bottom*L) { split(bottom); col = tile; }
    else if ((tile -= bottom*L) < right*L) { split(right); row = tile; }
    else t.l = tile - right*L;
    t.m0 = (i64)row*BM;
    t.n0 = (i64)col*BN;
    t.mrem = (int)min((i64)BM, p.M - t.m0);
    t.nrem = (int)min((i64)BN, N - t.n0);
    return t;
}

// ---- producers -----------------------------------------------------------------------

// copies of one element or of a pair of elements (16-byte aligned); not ok:
// zero-filled. They write stages that only the consumers read: no memory clobber,
// so that a producer's address loads and arithmetic batch across its copies.
__device__ __forceinline__ void cp_elem(double* dst, const double* src, bool ok = true)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" :: "r"(su32(dst)), "l"(src), "r"(ok ? 8 : 0));
}

__device__ __forceinline__ void cp_pair16(double* dst, const double* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(su32(dst)), "l"(src));
}

// One operand of a run: this thread's share of the gather of a stage. With
// pairs (the host found nearly all pairs of the gathered dimension adjacent and
// 16-byte aligned) a lane takes two neighbouring elements, one 16-byte copy
// where they are adjacent and aligned, else two of 8; without, lanes take
// consecutive elements, so that 8-byte copies still cover whole lines. In mode 0
// a thread's rows are fixed and it copies them at J of the stage's k, in mode 1
// its k are fixed and it copies J rows. The k offsets are loaded four stages at
// a time, four stages ahead (one stage ahead, small tiles waited for them: 0.8
// us a stage), two to a lane, and handed round by shuffles.
//
// A producer warp runs alone on its issue slots, so what bounds it is the
// latency of each copy's address arithmetic: the common case (a warp whose
// copies all lie inside the GEMM, at k of one stride, pairs adjacent and aligned)
// is a run of copies from one pointer; per-copy predicates and shuffles cost 150
// to 200 cycles a copy and capped the gather at 7 to 11 bytes per cycle and SM.
// Rows past the GEMM are not copied: whatever the stage holds there meets no
// stored element of C. k past the end is zero-filled.
template <int R, int MODE>
struct Gather
{
    template <int W>
    struct Geom
    {
        static constexpr int LANES = (MODE == 0 ? R : BK)/W;   // threads along the gathered dimension
        static constexpr int STEP = DN_PT/LANES;               // groups of threads along the other one
        static constexpr int J = (MODE == 0 ? BK : R)/STEP;    // copy slots per thread and stage
        static_assert(DN_PT % LANES == 0 && J >= 1 && J*STEP == (MODE == 0 ? BK : R), "gather geometry");
    };
    const double* X;
    const i64* kvec;
    i64 ro[2];                                                // mode 0: the thread's row offsets
    i64* sro;                                                 // mode 1: row offsets, each read by one warp only
    i64 ko[2], kn[2];                                         // offsets of k lane and lane + 32 of four stages, and of the next four
    int rem;                                                  // rows inside the GEMM
    bool even;                                                // mode 1: this warp's row offsets are even

    template <int W>
    __device__ __forceinline__ void rows(const i64* rvec)
    {
        constexpr int LANES = Geom<W>::LANES, STEP = Geom<W>::STEP, J = Geom<W>::J;
        const int t = threadIdx.x % DN_PT;
        if constexpr (MODE == 0)
        {
            const int r = W*(t % LANES);
            ro[0] = r < rem ? __ldg(rvec + r) : 0;
            if (W == 2) ro[1] = r + 1 < rem ? __ldg(rvec + r + 1) : 0;
        }
        else
        {
            // the rows this warp copies, PER consecutive ones at each of J steps, in
            // its own quarter of sro: which rows they are depends on W, and another
            // warp may still be at a run that was gathered with the other W
            constexpr int PER = 32/LANES;
            static_assert(PER*J == R/DN_PRODUCERS, "a warp's share of the rows");
            int odd = 0;
            __syncwarp();
            for (int x = t % 32; x < PER*J; x += 32)
            {
                const int r = (t/32)*PER + x % PER + x/PER*STEP;
                const i64 o = r < rem ? __ldg(rvec + r) : 0;
                sro[(t/32)*(PER*J) + x] = o;
                odd |= (int)(o & 1);
            }
            even = __all_sync(0xffffffffu, odd == 0) != 0;
            __syncwarp();
        }
    }

    // loads the k offsets of the four stages from k0 on (up to k1) into kn
    __device__ __forceinline__ void fetch(i64 k0, i64 k1)
    {
        const int lane = threadIdx.x & 31;
        kn[0] = k0 + lane < k1 ? __ldg(kvec + k0 + lane) : 0;
        kn[1] = k0 + 32 + lane < k1 ? __ldg(kvec + k0 + 32 + lane) : 0;
    }
    __device__ __forceinline__ void advance() { ko[0] = kn[0]; ko[1] = kn[1]; }

    __device__ __forceinline__ void start(const double* X_, const i64* rvec, const i64* kvec_, i64 r0, int rem_,
                                          bool pairs)
    {
        X = X_; kvec = kvec_;
        rem = rem_;
        if (pairs) rows<2>(rvec + r0);
        else rows<1>(rvec + r0);
    }

    // copies stage u of the current four
    template <int W>
    __device__ __forceinline__ void copy(double* Xs, int u, int kvalid) const
    {
        const i64 mine = u & 2 ? ko[1] : ko[0];               // this stage's offsets, from lane base on
        const int base = (u & 1)*BK;
        constexpr int LANES = Geom<W>::LANES, STEP = Geom<W>::STEP, J = Geom<W>::J;
        const int t = threadIdx.x % DN_PT;
        if (MODE == 0)
        {
            const int lane = t & 31, r = W*(t % LANES), k0 = t/LANES;
            const bool in = r < rem, two = W == 2 && r + 1 < rem, adj = two && ro[1] == ro[0] + 1;
            const i64 first = __shfl_sync(0xffffffffu, mine, base);
            const i64 step = __shfl_sync(0xffffffffu, mine, base + 1) - first;
            const double* src = X + ro[0] + first + k0*step;
            const bool other = ((lane ^ base) & BK) != 0;      // the offset this lane holds belongs to another stage
            const bool fast = kvalid == BK && (other || mine == first + (lane - base)*step) &&
                              (W == 1 || !in || (adj && (((uintptr_t)src | (uintptr_t)(8*STEP*step)) & 15) == 0));
            if (__all_sync(0xffffffffu, fast))
            {
                if (!in) return;
                #pragma unroll
                for (int j = 0; j < J; j++)
                {
                    double* dst = Xs + tile_pos<R, MODE>(r, k0 + j*STEP);
                    if (W == 2) cp_pair16(dst, src);
                    else cp_elem(dst, src);
                    src += STEP*step;
                }
                return;
            }
            // any k offsets: all shuffles before the copies
            i64 k[J];
            #pragma unroll
            for (int j = 0; j < J; j++) k[j] = __shfl_sync(0xffffffffu, mine, base + k0 + j*STEP);
            const bool whole = kvalid == BK && (W == 1 || other || (mine & 1) == 0) &&
                               (W == 1 || !in || (adj && ((uintptr_t)(X + ro[0]) & 15) == 0));
            if (__all_sync(0xffffffffu, whole))
            {
                if (!in) return;
                #pragma unroll
                for (int j = 0; j < J; j++)
                {
                    double* dst = Xs + tile_pos<R, MODE>(r, k0 + j*STEP);
                    if (W == 2) cp_pair16(dst, X + ro[0] + k[j]);
                    else cp_elem(dst, X + ro[0] + k[j]);
                }
                return;
            }
            if (!in) return;
            #pragma unroll
            for (int j = 0; j < J; j++)
            {
                const int kl = k0 + j*STEP;
                const bool ok = kl < kvalid;
                src = X + ro[0] + k[j];
                double* dst = Xs + tile_pos<R, MODE>(r, kl);
                if (W == 2 && ok && adj && ((uintptr_t)src & 15) == 0) cp_pair16(dst, src);
                else
                {
                    cp_elem(dst, src, ok);
                    if (two) cp_elem(dst + 1, X + ro[1] + k[j], ok);
                }
            }
        }
        else
        {
            constexpr int PER = 32/LANES;
            const i64* ros = sro + (t/32)*(PER*J) + (t % 32)/LANES;    // row t/LANES + j*STEP: ros[j*PER]
            const int kl = W*(t % LANES);
            const i64 o0 = __shfl_sync(0xffffffffu, mine, base + kl);
            const i64 o1 = W == 2 ? __shfl_sync(0xffffffffu, mine, base + kl + W - 1) : 0;
            const bool adj = W == 2 && o1 == o0 + 1;
            const double* Xk = X + o0;
            const bool fast = kvalid == BK && (W == 1 || (adj && even && ((uintptr_t)Xk & 15) == 0));
            if (__all_sync(0xffffffffu, fast))
            {
                if (rem < R)
                {
                    #pragma unroll 4
                    for (int j = 0; t/LANES + j*STEP < rem; j++)
                    {
                        double* dst = Xs + tile_pos<R, MODE>(t/LANES + j*STEP, kl);
                        if (W == 2) cp_pair16(dst, Xk + ros[j*PER]);
                        else cp_elem(dst, Xk + ros[j*PER]);
                    }
                    return;
                }
                #pragma unroll
                for (int j = 0; j < J; j++)
                {
                    const int r = t/LANES + j*STEP;
                    double* dst = Xs + tile_pos<R, MODE>(r, kl);
                    if (W == 2) cp_pair16(dst, Xk + ros[j*PER]);
                    else cp_elem(dst, Xk + ros[j*PER]);
                }
                return;
            }
            const bool ok0 = kl < kvalid, ok1 = W == 2 && kl + 1 < kvalid;
            #pragma unroll 4
            for (int j = 0; j < J; j++)
            {
                const int r = t/LANES + j*STEP;
                if (r >= rem) break;
                const i64 row = ros[j*PER];
                double* dst = Xs + tile_pos<R, MODE>(r, kl);
                if (adj && ok1 && ((uintptr_t)(Xk + row) & 15) == 0) cp_pair16(dst, Xk + row);
                else
                {
                    cp_elem(dst, Xk + row, ok0);
                    if (W == 2) cp_elem(dst + 1, X + row + o1, ok1);
                }
            }
        }
    }

    __device__ __forceinline__ void stage(double* Xs, int u, int kvalid, bool pairs) const
    {
        if (pairs) copy<2>(Xs, u, kvalid);
        else copy<1>(Xs, u, kvalid);
    }
};

// The gather of a grouped GEMM, whose direction differs from group to group: one
// stage layout (MODE 1) for both. how: 0 single elements along k, 1 pairs along k,
// 2 single elements along the rows.
template <int R>
struct GatherG : Gather<R, 1>
{
    typedef Gather<R, 1> Base;
    static constexpr int STEP = DN_PT/R, J = BK/STEP;         // along the rows: k per pass, copies per thread
    static_assert(DN_PT % R == 0 && J*STEP == BK, "gather geometry");

    __device__ __forceinline__ void start(const double* X_, const i64* rvec, const i64* kvec_, i64 r0, int rem_, int how)
    {
        if (how < 2) { Base::start(X_, rvec, kvec_, r0, rem_, how == 1); return; }
        this->X = X_; this->kvec = kvec_;
        this->rem = rem_;
        const int r = threadIdx.x % R;
        this->ro[0] = r < rem_ ? __ldg(rvec + r0 + r) : 0;
    }

    __device__ __forceinline__ void stage(double* Xs, int u, int kvalid, int how) const
    {
        if (how < 2) { Base::stage(Xs, u, kvalid, how == 1); return; }
        const i64 mine = u & 2 ? this->ko[1] : this->ko[0];
        const int t = threadIdx.x % DN_PT, base = (u & 1)*BK, r = t % R, k0 = t/R;
        i64 k[J];
        #pragma unroll
        for (int j = 0; j < J; j++) k[j] = __shfl_sync(0xffffffffu, mine, base + k0 + j*STEP);
        if (r >= this->rem) return;
        const double* Xr = this->X + this->ro[0];
        if (kvalid == BK)
        {
            #pragma unroll
            for (int j = 0; j < J; j++) cp_elem(Xs + tile_pos<R, 1>(r, k0 + j*STEP), Xr + k[j]);
            return;
        }
        #pragma unroll
        for (int j = 0; j < J; j++)
            cp_elem(Xs + tile_pos<R, 1>(r, k0 + j*STEP), Xr + k[j], k0 + j*STEP < kvalid);
    }
};

// zero-filled when not ok
__device__ __forceinline__ void cp_pair16(double* dst, const double* src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(su32(dst)), "l"(src), "r"(ok ? 16 : 0));
}

// The gather of a complex operand (R rows of BK/2 complex k; 16-byte aligned
// elements, offsets in elements). Real and imaginary part stay together, so one
// stage layout (tile_pos MODE 1, part p of complex k at real k 2k + p) and one
// 16-byte copy per element serve both gather directions: rows = true takes
// lanes along the rows, else along k.
template <int R>
struct GatherZ
{
    static constexpr int KS = BK/2;                           // complex k per stage
    static constexpr int STEP0 = DN_PT/R, J0 = KS/STEP0;      // along the rows: k per pass, copies per thread
    static constexpr int STEP1 = DN_PT/KS, J1 = R/STEP1;      // along k: rows per pass
    static_assert(DN_PT % R == 0 && J0*STEP0 == KS && J1*STEP1 == R, "gather geometry");
    const double* X;
    const i64* kvec;
    i64 ro;
    i64* sro;                                                 // along k: row offsets, each read by one warp only
    i64 ko, kn;                                               // offset of k lane of four stages, and of the next four
    int rem;

    __device__ __forceinline__ void fetch(i64 k0, i64 k1)
    {
        const int lane = threadIdx.x & 31;
        kn = k0 + lane < k1 ? __ldg(kvec + k0 + lane) : 0;
    }
    __device__ __forceinline__ void advance() { ko = kn; }
    __device__ __forceinline__ void start(const double* X_, const i64* rvec, const i64* kvec_, i64 r0, int rem_,
                                          bool rows)
    {
        X = X_; kvec = kvec_;
        rem = rem_;
        rvec += r0;
        const int t = threadIdx.x % DN_PT;
        ro = rows && t % R < rem ? __ldg(rvec + t % R) : 0;
        if (rows) return;
        constexpr int PER = 32/KS;
        __syncwarp();
        for (int x = t % 32; x < PER*J1; x += 32)
        {
            const int r = (t/32)*PER + x % PER + x/PER*STEP1;
            sro[r] = r < rem ? __ldg(rvec + r) : 0;
        }
        __syncwarp();
    }
    __device__ __forceinline__ void stage(double* Xs, int u, int kvalid, bool rows) const
    {
        const int t = threadIdx.x % DN_PT, base = u*KS;
        if (rows)
        {
            const int r = t % R, k0 = t/R;
            i64 k[J0];
            #pragma unroll
            for (int j = 0; j < J0; j++) k[j] = __shfl_sync(0xffffffffu, ko, base + k0 + j*STEP0);
            if (r >= rem) return;
            #pragma unroll
            for (int j = 0; j < J0; j++)
            {
                const int kl = k0 + j*STEP0;
                cp_pair16(Xs + tile_pos<R, 1>(r, 2*kl), X + 2*(ro + k[j]), kl < kvalid);
            }
        }
        else
        {
            const int kl = t % KS;
            const double* Xk = X + 2*__shfl_sync(0xffffffffu, ko, base + kl);
            #pragma unroll
            for (int j = 0; j < J1; j++)
            {
                const int r = t/KS + j*STEP1;
                if (r >= rem) break;
                cp_pair16(Xs + tile_pos<R, 1>(r, 2*kl), Xk + 2*sro[r], kl < kvalid);
            }
        }
    }
};

// MODE 2: the direction is chosen at run time
template <int R, int MODE, bool CPLX> struct GatherOf { typedef Gather<R, MODE> type; };
template <int R> struct GatherOf<R, 2, false> { typedef GatherG<R> type; };
template <int R, int MODE> struct GatherOf<R, MODE, true> { typedef GatherZ<R> type; };

// ---- kernel ---------------------------------------------------------------------------

// Row-warp and column-warp of a consumer warp. Warps cw and cw + 4 share an SM
// sub-core: shifting the columns of the second row-warp gives a ragged edge's
// longer and shorter shares to the same sub-core.
template <int WGN>
__device__ __forceinline__ void warp_at(int cw, int& wm, int& wn)
{
    wm = cw/WGN;
    wn = (cw + (WGN/2)*wm) % WGN;
}

template <int STAGES>
struct DnShared
{
    uint64_t full[STAGES], empty[STAGES];
    DnFail fail;
};

template <int WGM, int WGN, int MF, int NF, int STAGES, int TEAMS>
constexpr size_t dn_smem()
{
    return (size_t)(STAGES*BK + TEAMS)*(WGM*MF*16 + WGN*NF*8)*sizeof(double) + sizeof(DnShared<STAGES>);
}

// x with its sign bit flipped by the mask
__device__ __forceinline__ double flip(double x, unsigned mask)
{
    return __hiloint2double(__double2hiint(x) ^ (int)mask, __double2loint(x));
}

// alpha*x + beta*op(c) over a complex element of C (beta == 0: c is not read). A
// factor of zero leaves its product out, so that a real alpha or beta scales
// each part by itself: 0 times an infinite part would be NaN in the other one.
// REAL: both are real (tested an element at a time, 4000 x 4000 x 8 took 143 us, not 128).
template <bool REAL>
__device__ __forceinline__ void update_z(const GemmF64Args& p, double* dst, double re, double im)
{
    double vr, vi;
    if (REAL || p.alpha_im == 0.0) { vr = p.alpha*re; vi = p.alpha*im; }
    else if (p.alpha == 0.0) { vr = -p.alpha_im*im; vi = p.alpha_im*re; }
    else { vr = p.alpha*re - p.alpha_im*im; vi = p.alpha*im + p.alpha_im*re; }
    if (p.beta != 0.0 || (!REAL && p.beta_im != 0.0))
    {
        const double cr = dst[0], ci = p.conj_c ? -dst[1] : dst[1];
        if (REAL || p.beta != 0.0) { vr += p.beta*cr; vi += p.beta*ci; }
        if (!REAL && p.beta_im != 0.0) { vr -= p.beta_im*ci; vi += p.beta_im*cr; }
    }
    *reinterpret_cast<double2*>(dst) = make_double2(vr, vi);
}

// the operands of one K segment of a tile; how_a / how_b as the gathers take them
struct Operands
{
    const double *A, *B;
    const i64 *a_m, *a_k, *b_n, *b_k;
    i64 K;
    int how_a, how_b;
};

// where a tile's results go
struct Target
{
    double* C;
    const i64 *c_m, *c_n;
    double alpha, beta;
};

// one contraction (possibly with a batch index)
template <int BM, int BN, bool CPLX>
struct DenseWork
{
    typedef TileAt Tile;
    const GemmF64Args& p;
    __device__ __forceinline__ const GemmF64Args& args() const { return p; }
    __device__ __forceinline__ bool run(unsigned r, Run& out) const { return run_at(p, blockIdx.x, r, out); }
    __device__ __forceinline__ Tile tile(const Run& run) const { return tile_at<BM, BN>(p, run.tile); }
    __device__ __forceinline__ int segments(const Tile&) const { return 1; }
    __device__ __forceinline__ Operands operands(const Tile& t, int) const
    {
        constexpr int ES = CPLX ? 2 : 1;
        return Operands{p.A + ES*p.a_l[t.l], p.B + ES*p.b_l[t.l], p.a_m, p.a_k, p.b_n, p.b_k, p.K,
                        CPLX ? p.amode == 0 : p.pair_a != 0, CPLX ? p.bmode == 0 : p.pair_b != 0};
    }
    __device__ __forceinline__ Target target(const Tile& t) const
    {
        return Target{p.C + (CPLX ? 2 : 1)*p.c_l[t.l], p.c_m, p.c_n, p.alpha, p.beta};
    }
    __device__ __forceinline__ double* partial() const { return p.partial; }
    __device__ __forceinline__ const WaitControl& control() const { return p.ctl; }
};

// The GEMMs of a grouped plan: tiles listed by the plan (group by group), the k
// steps of all of them dealt to the CTAs in runs of equal modelled cost, which the
// plan has worked out too: CTA c takes k steps [start[c], start[c + 1]).
template <int BM, int BN>
struct GroupWork
{
    struct Tile
    {
        i64 m0, n0;
        int mrem, nrem;
        const GroupDesc* g;
    };
    const GroupDesc* groups;
    const GroupTile* tiles;
    const GroupStart* start;
    double* w;
    const WaitControl& ctl;
    __device__ __forceinline__ const WaitControl& control() const { return ctl; }
    __device__ __forceinline__ GemmF64Args args() const { return GemmF64Args(); }     // complex groups do not occur
    __device__ __forceinline__ bool run(unsigned r, Run& out) const
    {
        const GroupStart a = start[blockIdx.x], b = start[blockIdx.x + 1];
        const int t = a.tile + (int)r;
        if (t > b.tile || (t == b.tile && b.step == 0)) return false;
        const int nst = groups[tiles[t].g].nst;
        out.tile = (unsigned)t;
        out.s0 = r == 0 ? a.step : 0;
        out.s1 = t == b.tile ? b.step : nst;
        out.slot = out.s1 - out.s0 == nst ? -1 : r == 0 ? 0 : 1;
        return out.s0 < out.s1;
    }
    __device__ __forceinline__ Tile tile(const Run& run) const
    {
        const GroupTile x = tiles[run.tile];
        Tile t;
        t.g = groups + x.g;
        t.m0 = (i64)x.tm*BM;
        t.n0 = (i64)x.tn*BN;
        t.mrem = (int)min((i64)BM, t.g->M - t.m0);
        t.nrem = (int)min((i64)BN, t.g->N - t.n0);
        return t;
    }
    __device__ __forceinline__ int segments(const Tile& t) const { return t.g->nseg > 0 ? t.g->nseg : 1; }
    __device__ __forceinline__ Operands operands(const Tile& t, int sg) const
    {
        const GroupDesc& g = *t.g;
        if (g.nseg > 0)
        {
            const SegDesc& s = g.segs[sg];
            return Operands{g.A, g.B, s.a_m, s.a_k, s.b_n, s.b_k, s.K, g.how_a, g.how_b};
        }
        return Operands{g.A, g.B, g.a_m, g.a_k, g.b_n, g.b_k, g.K, g.how_a, g.how_b};
    }
    __device__ __forceinline__ Target target(const Tile& t) const
    {
        return Target{t.g->C, t.g->c_m, t.g->c_n, t.g->alpha, t.g->beta};
    }
    __device__ __forceinline__ double* partial() const { return w; }
};

// calls f with the fragment counts as constants: an MMA under a run-time
// condition is predicated, and the pipe takes as long for one that is off
template <int MF, int NF, typename F>
__device__ __forceinline__ bool dn_fragments(int ni, int nj, F&& f)
{
    if (ni <= 0 || nj <= 0) return f(std::integral_constant<int, 0>(), std::integral_constant<int, 0>());
    bool ok = true;
    auto columns = [&](auto i)
    {
        if (nj == 1) ok = f(i, std::integral_constant<int, 1>());
        else if (NF <= 2 || nj == 2) ok = f(i, std::integral_constant<int, (NF < 2 ? NF : 2)>());
        else if (nj == 3) ok = f(i, std::integral_constant<int, (NF < 3 ? NF : 3)>());
        else ok = f(i, std::integral_constant<int, NF>());
    };
    if (ni == 1) columns(std::integral_constant<int, 1>());
    else if (MF <= 2 || ni == 2) columns(std::integral_constant<int, (MF < 2 ? MF : 2)>());
    else if (ni == 3) columns(std::integral_constant<int, (MF < 3 ? MF : 3)>());
    else columns(std::integral_constant<int, MF>());
    return ok;
}

// CPLX: a complex contraction as a real one of M x 2N x 2K: the columns of C
// and the k of A are (real, imaginary) pairs as they lie in memory, and the 2 x 2
// real block of each element of B, ((re, im), (-im, re)), is formed from the one
// stored copy as the fragments are read: column parity q and k parity p pick
// part p ^ q and a sign. N, K and the scatter vectors stay in complex units in
// the arguments; M x 2N tiles of 16 real k (8 complex) are what the tile loop
// sees.
//
// Work: the source of runs, tiles and operands (DenseWork, GroupWork).
template <int WGM, int WGN, int MF, int NF, int STAGES, int LAG, int TEAMS, int AMODE, int BMODE, bool CPLX,
          typename Work>
__device__ __forceinline__ void dn_body(const Work& work)
{
    static_assert(WGM*WGN == DN_CONSUMERS, "consumer warps");
    static_assert(STAGES % TEAMS == 0 && LAG*TEAMS < STAGES, "ring");
    constexpr bool SPLIT = MF*NF > 4;             // small accumulators: the launch's registers serve both roles
    constexpr int BM = WGM*MF*16, BN = WGN*NF*8;
    constexpr int STAGE = BK*(BM + BN);
    extern __shared__ __align__(128) double smem[];
    i64* sro = reinterpret_cast<i64*>(smem + STAGES*STAGE);        // each team's row offsets of A, then of B
    DnShared<STAGES>& sh = *reinterpret_cast<DnShared<STAGES>*>(sro + TEAMS*(BM + BN));
    volatile DnFail* fail = &sh.fail;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < STAGES; s++)
        {
            // one arrival per producer warp, its copies landed
            mb_init(&sh.full[s], DN_PRODUCERS + (s == work.control().hold_stage ? 1 : 0));
            mb_init(&sh.empty[s], DN_CONSUMERS);      // one arrival per consumer warp
        }
        sh.fail.abort = 0;
        sh.fail.limit = work.control().wait_ns;
    }
    __syncthreads();
    // from here on the roles never wait on a CTA-wide barrier

    Run run;
    uint32_t st = 0, phase = 0;                       // ring position
    if (warp < TEAMS*DN_PRODUCERS)
    {
        if (SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(dn_reg_p(TEAMS)));
        // two teams take the stages in turn
        const int team = warp/DN_PRODUCERS;
        int turn = 0;
        bool ok = true;
        bool wrapped = false;                         // the first round of stages starts empty
        // A warp publishes a stage LAG stages after it issued it, when its copies
        // have landed: LAG stages are in flight. (An mbarrier arrival tied to the
        // copies, cp.async.mbarrier.arrive, held the warp's later copies back
        // until it had fired.) LAG covers the memory latency at the tile's cycles
        // per stage; a longer one only delays a run's first stage.
        int lag = 0;
        uint32_t pub = team;                          // the team's next stage to publish
        for (unsigned r = 0; ok && work.run(r, run); r++)
        {
            const typename Work::Tile t = work.tile(run);
            constexpr int KS = CPLX ? BK/2 : BK;               // k of the scatter vectors per stage
            constexpr int ES = CPLX ? 2 : 1;                   // doubles per element
            int base = 0;                                      // first k step of the segment
            for (int sg = 0; ok && sg < work.segments(t); sg++)
            {
            const Operands o = work.operands(t, sg);
            const int steps = (int)((o.K + KS - 1)/KS), lo = max(run.s0, base), hi = min(run.s1, base + steps);
            if (lo < hi)
            {
            typename GatherOf<BM, AMODE, CPLX>::type ga;
            typename GatherOf<CPLX ? BN/2 : BN, BMODE, CPLX>::type gb;
            ga.sro = sro + team*(BM + BN);
            gb.sro = ga.sro + BM;
            const i64 k_begin = (i64)(lo - base)*KS, k_end = min(o.K, (i64)(hi - base)*KS);
            ga.start(o.A, o.a_m, o.a_k, t.m0, t.mrem, o.how_a);
            gb.start(o.B, o.b_n, o.b_k, t.n0/ES, t.nrem/ES, o.how_b);
            ga.fetch(k_begin, k_end);
            gb.fetch(k_begin, k_end);
            int u = 0;
            for (i64 k0 = k_begin; k0 < k_end; k0 += KS)
            {
                if (u == 0)
                {
                    ga.advance();
                    gb.advance();
                    ga.fetch(k0 + 4*KS, k_end);
                    gb.fetch(k0 + 4*KS, k_end);
                }
                if (turn == team)
                {
                    if (wrapped && !dn_wait(&sh.empty[st], phase ^ 1, fail))
                    {
                        ok = false;
                        break;
                    }
                    const int kvalid = (int)min((i64)KS, k_end - k0);
                    double* As = smem + st*STAGE;
                    ga.stage(As, u, kvalid, o.how_a);
                    gb.stage(As + BK*BM, u, kvalid, o.how_b);
                    cp_async_commit();
                    if (lag < LAG) lag++;
                    else
                    {
                        cp_async_wait<LAG>();
                        __syncwarp();
                        if (lane == 0) mb_arrive(&sh.full[pub]);
                        pub = (pub + TEAMS) % STAGES;
                    }
                }
                if (TEAMS > 1) turn ^= 1;
                u = (u + 1) & 3;
                if (++st == STAGES) { st = 0; phase ^= 1; wrapped = true; }
            }
            }
            base += steps;
            }
        }
        // the last stages (also after a wait that gave up: the copies land before
        // the CTA is gone)
        cp_async_wait<0>();
        if (!ok) dn_report(work.control().error);
        __syncwarp();
        for (; ok && lag > 0; lag--)
        {
            if (lane == 0) mb_arrive(&sh.full[pub]);
            pub = (pub + TEAMS) % STAGES;
        }
        return;
    }

    if (SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(dn_reg_c(TEAMS)));
    int wm, wn;
    warp_at<WGN>(warp - TEAMS*DN_PRODUCERS, wm, wn);
    const int fr = lane >> 2, fc = lane & 3;
    // (Ar + i sa Ai)(Br + i sb Bi): sign of the part of B at this lane's column
    // parity fr & 1 (0: real) and k parity fc & 1 (0: Ar)
    unsigned sign = 0;
    if (CPLX)
    {
        const bool col_im = fr & 1, k_im = fc & 1;
        const GemmF64Args& p = work.args();
        const bool neg = k_im ? (col_im ? p.conj_a != 0 : (p.conj_a != 0) == (p.conj_b != 0)) : col_im && p.conj_b;
        sign = neg ? 0x80000000u : 0u;
    }
    for (unsigned r = 0; work.run(r, run); r++)
    {
        typename Work::Tile t = work.tile(run);
        // fragments of this warp inside the GEMM: 16-row fragment i*WGM + wm, 8-column fragment j*WGN + wn
        const int ni = min(MF, max(0, ((t.mrem + 15)/16 - wm + WGM - 1)/WGM));
        const int nj = min(NF, max(0, ((t.nrem + 7)/8 - wn + WGN - 1)/WGN));
        double acc[MF][NF][4];
        #pragma unroll
        for (int i = 0; i < MF; i++)
            #pragma unroll
            for (int j = 0; j < NF; j++)
                #pragma unroll
                for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0;

        const bool ok = dn_fragments<MF, NF>(ni, nj, [&](auto ni_, auto nj_)
        {
            constexpr int NI = decltype(ni_)::value, NJ = decltype(nj_)::value;
            for (int left = run.s1 - run.s0; left > 0; left--)
            {
                if (!dn_wait(&sh.full[st], phase, fail)) return false;
                if (NI*NJ > 0)
                {
                    const double* As = smem + st*STAGE;
                    const double* Bs = As + BK*BM;
                    #pragma unroll
                    for (int kk = 0; kk < BK; kk += 8)
                    {
                        double af[NI > 0 ? NI : 1][4], bf[NJ > 0 ? NJ : 1][2];
                        #pragma unroll
                        for (int j = 0; j < NJ; j++)
                            #pragma unroll
                            for (int q = 0; q < 2; q++)
                            {
                                if (CPLX)
                                    bf[j][q] = flip(Bs[tile_pos<BN/2, 1>((j*WGN + wn)*4 + (fr >> 1),
                                                                         (kk + fc + 4*q) ^ (fr & 1))], sign);
                                else bf[j][q] = Bs[tile_pos<BN, BMODE != 0>((j*WGN + wn)*8 + fr, kk + fc + 4*q)];
                            }
                        #pragma unroll
                        for (int i = 0; i < NI; i++)
                            #pragma unroll
                            for (int q = 0; q < 4; q++)
                                af[i][q] = As[tile_pos<BM, AMODE != 0>((i*WGM + wm)*16 + fr + 8*(q & 1),
                                                                  kk + fc + 4*(q >> 1))];
                        if (kk + 8 == BK)
                        {
                            // the stage's last fragments are read: it may be refilled
                            __syncwarp();
                            if (lane == 0) mb_arrive(&sh.empty[st]);
                        }
                        #pragma unroll
                        for (int i = 0; i < NI; i++)
                            #pragma unroll
                            for (int j = 0; j < NJ; j++) dmma16(acc[i][j], af[i], bf[j]);
                    }
                }
                else if (lane == 0) mb_arrive(&sh.empty[st]);
                if (++st == STAGES) { st = 0; phase ^= 1; }
            }
            return true;
        });
        if (!ok)
        {
            dn_report(work.control().error);
            break;
        }

        // the run and its tile again (not kept over the loop above)
        asm volatile("" : "+r"(r));
        work.run(r, run);
        t = work.tile(run);
        if (run.slot >= 0)
        {
            // this run's sums, thread by thread, for gemm_f64_fixup
            double* w = work.partial() + ((i64)blockIdx.x*2 + run.slot)*(BM*BN) + (threadIdx.x - TEAMS*DN_PT);
            #pragma unroll
            for (int i = 0; i < MF; i++)
                #pragma unroll
                for (int j = 0; j < NF; j++)
                    if (i < ni && j < nj)
                    {
                        #pragma unroll
                        for (int q = 0; q < 4; q++) w[((i*NF + j)*4 + q)*DN_CT] = acc[i][j][q];
                    }
            continue;
        }
        const Target c = work.target(t);
        double* C = c.C;
        const double alpha = c.alpha, beta = c.beta;
        #pragma unroll
        for (int j = 0; j < NF; j++)
        {
            const int n = (j*WGN + wn)*8 + 2*fc;
            if (n >= t.nrem) continue;
            if (CPLX)
            {
                double* C0 = C + 2*__ldg(c.c_n + (t.n0 + n)/2);
                const GemmF64Args& p = work.args();
                auto rows = [&](auto real)
                {
                    #pragma unroll
                    for (int i = 0; i < MF; i++)
                        #pragma unroll
                        for (int hh = 0; hh < 2; hh++)
                        {
                            const int m = (i*WGM + wm)*16 + 8*hh + fr;
                            if (m < t.mrem)
                                update_z<decltype(real)::value>(p, C0 + 2*__ldg(c.c_m + t.m0 + m), acc[i][j][2*hh],
                                                                acc[i][j][2*hh + 1]);
                        }
                };
                if (p.alpha_im == 0.0 && p.beta_im == 0.0) rows(std::true_type());
                else rows(std::false_type());
                continue;
            }
            const bool two = n + 1 < t.nrem;
            double* C0 = C + __ldg(c.c_n + t.n0 + n);
            double* C1 = C + (two ? __ldg(c.c_n + t.n0 + n + 1) : 0);
            // The old values of IB fragments' rows are loaded before the first of them is
            // stored: one by one, each load behind the store before it, the update
            // took a memory latency an element, and a load from a sector just stored to
            // waits for the store. With small accumulators all rows of a column pair
            // go together (656^3 with permuted operands and beta: 51 us, 59 a fragment at
            // a time); with 128 x 128 tiles the registers for more would spill. Past L1,
            // which has no room for that many lines beside the stages.
            constexpr int IB = MF*NF > 4 ? 1 : MF;
            #pragma unroll
            for (int i0 = 0; i0 < MF; i0 += IB)
            {
                bool in[IB][2];
                i64 ro[IB][2];
                double v[IB][2][2];
                #pragma unroll
                for (int x = 0; x < IB; x++)
                    #pragma unroll
                    for (int hh = 0; hh < 2; hh++)
                    {
                        const int m = ((i0 + x)*WGM + wm)*16 + 8*hh + fr;
                        in[x][hh] = m < t.mrem;
                        ro[x][hh] = in[x][hh] ? __ldg(c.c_m + t.m0 + m) : 0;
                    }
                if (beta != 0.0)
                {
                    #pragma unroll
                    for (int x = 0; x < IB; x++)
                        #pragma unroll
                        for (int hh = 0; hh < 2; hh++)
                        {
                            v[x][hh][0] = in[x][hh] ? __ldcg(C0 + ro[x][hh]) : 0.0;
                            v[x][hh][1] = in[x][hh] && two ? __ldcg(C1 + ro[x][hh]) : 0.0;
                        }
                    #pragma unroll
                    for (int x = 0; x < IB; x++)
                        #pragma unroll
                        for (int hh = 0; hh < 2; hh++)
                            #pragma unroll
                            for (int q = 0; q < 2; q++) v[x][hh][q] = alpha*acc[i0 + x][j][2*hh + q] + beta*v[x][hh][q];
                }
                else
                {
                    #pragma unroll
                    for (int x = 0; x < IB; x++)
                        #pragma unroll
                        for (int hh = 0; hh < 2; hh++)
                            #pragma unroll
                            for (int q = 0; q < 2; q++) v[x][hh][q] = alpha*acc[i0 + x][j][2*hh + q];
                }
                #pragma unroll
                for (int x = 0; x < IB; x++)
                    #pragma unroll
                    for (int hh = 0; hh < 2; hh++)
                    {
                        if (in[x][hh]) C0[ro[x][hh]] = v[x][hh][0];
                        if (in[x][hh] && two) C1[ro[x][hh]] = v[x][hh][1];
                    }
            }
        }
    }
}

template <int WGM, int WGN, int MF, int NF, int STAGES, int LAG, int TEAMS, int AMODE, int BMODE, bool CPLX>
__global__ void __launch_bounds__(dn_threads(TEAMS), 1)
gemm_f64_dense_kernel(const GemmF64Args p)
{
    if (p.gate && *p.gate <= p.gate_above) return;
    const DenseWork<WGM*MF*16, WGN*NF*8, CPLX> work{p};
    dn_body<WGM, WGN, MF, NF, STAGES, LAG, TEAMS, AMODE, BMODE, CPLX>(work);
}

// the GEMMs of a grouped plan, 128 x 128 tiles (GroupWork). AMODE, BMODE: the
// gather directions where all groups share them, else 2 (chosen per group, one
// stage layout for both, single elements along the rows)
constexpr int GD_BM = 128, GD_BN = 128;
template <int AMODE, int BMODE>
__global__ void __launch_bounds__(dn_threads(1), 1)
gemm_f64_group_dense_kernel(const GroupDesc* __restrict__ groups, const GroupTile* __restrict__ tiles,
                            const GroupStart* __restrict__ start, double* __restrict__ partial, const WaitControl ctl)
{
    const GroupWork<GD_BM, GD_BN> work{groups, tiles, start, partial, ctl};
    dn_body<2, 4, 4, 4, 6, 1, 1, AMODE, BMODE, false>(work);
}

// sums the runs of a cut tile of a grouped plan in CTA order; block (cut tile,
// fragment), thread t the elements of consumer thread t
__global__ void __launch_bounds__(DN_CT)
gemm_f64_group_fixup(const GroupDesc* __restrict__ groups, const GroupTile* __restrict__ tiles,
                     const GroupCut* __restrict__ cuts, const double* __restrict__ partial)
{
    constexpr int NF = 4, WGM = 2, WGN = 4, SLOT = GD_BM*GD_BN;
    const GroupCut x = cuts[blockIdx.x];
    const GroupTile tl = tiles[x.tile];
    const GroupDesc& g = groups[tl.g];
    const int lane = threadIdx.x & 31, e = blockIdx.y, j = e % NF, i = e/NF;
    int wm, wn;
    warp_at<WGN>(threadIdx.x >> 5, wm, wn);
    #pragma unroll
    for (int q = 0; q < 4; q++)
    {
        const i64 m = (i64)tl.tm*GD_BM + (i*WGM + wm)*16 + 8*(q >> 1) + (lane >> 2);
        const i64 n = (i64)tl.tn*GD_BN + (j*WGN + wn)*8 + 2*(lane & 3) + (q & 1);
        if (m >= g.M || n >= g.N) continue;
        const i64 at = (i64)(4*e + q)*DN_CT + threadIdx.x;
        double s = partial[((i64)x.cta*2 + x.slot)*SLOT + at];
        for (int c = 1; c < x.count; c++) s += partial[(i64)(x.cta + c)*2*SLOT + at];
        double* dst = g.C + __ldg(g.c_m + m) + __ldg(g.c_n + n);
        const double v = g.alpha*s;
        *dst = g.beta == 0.0 ? v : v + g.beta*(*dst);
    }
}

// Sums the runs of the cut tiles in CTA order and applies alpha and beta.
// blockIdx.x: the tile; thread t of a group of DN_CT holds the elements of
// consumer thread t, a few of the MF*NF*2 pairs per block. GROUPS groups of threads
// take interleaved CTAs and combine in a fixed order: a tile cut over all SMs
// then still has enough loads in flight.
template <int WGM, int WGN, int MF, int NF, int GROUPS, bool CPLX>
__global__ void __launch_bounds__(DN_CT*GROUPS)
gemm_f64_fixup(const GemmF64Args p)
{
    constexpr int BM = WGM*MF*16, BN = WGN*NF*8;
    if (p.gate && *p.gate <= p.gate_above)
    {
        asm volatile("griddepcontrol.wait;" ::: "memory");     // as below
        return;
    }
    __shared__ double sums[GROUPS][2][DN_CT];
    const int tc = threadIdx.x % DN_CT, grp = threadIdx.x/DN_CT;
    const int lane = tc & 31;
    int wm, wn;
    warp_at<WGN>(tc >> 5, wm, wn);
    const TileAt t = tile_at<BM, BN>(p, p.dp_tiles + blockIdx.x);

    // the CTAs [c0, c1) whose runs meet this tile's k steps [ub, ue)
    const unsigned kt = (unsigned)p.kt, ub = blockIdx.x*kt, ue = ub + kt;
    const unsigned c0 = cta_of_unit(p, ub), c1 = cta_of_unit(p, ue - 1) + 1;
    // the CTA's second slot when its first run is part of an earlier tile
    // (whole tiles take no slot); only the first CTA can have such a run
    const unsigned uf = first_unit(p, c0);
    const double* first = p.partial + (i64)(c0*2 + (uf < ub && uf % kt != 0 ? 1 : 0))*(BM*BN) + tc;
    // launched while the kernel above runs: its sums are complete from here on.
    // Every block waits, also one with nothing to add: else a launch whose blocks
    // all return could end, and the next kernel start, before that kernel's writes
    // to C are visible.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (c1 - c0 == 1) return;                        // one CTA did the whole tile
    for (int e = blockIdx.y; e < MF*NF*2; e += gridDim.y)
    {
        // elements 2e and 2e + 1: neighbouring columns of one row (complex: the
        // parts of one element)
        const int hh = e & 1, j = (e >> 1) % NF, i = e/(2*NF);
        const int m = (i*WGM + wm)*16 + 8*hh + (lane >> 2), n = (j*WGN + wn)*8 + 2*(lane & 3);
        const bool in = m < t.mrem && n < t.nrem;
        double s0 = 0.0, s1 = 0.0;
        if (in)
        {
            const i64 at = (i64)2*e*DN_CT;
            if (grp == 0) { s0 = first[at]; s1 = first[at + DN_CT]; }
            #pragma unroll 4
            for (unsigned c = c0 + (grp == 0 ? GROUPS : grp); c < c1; c += GROUPS)
            {
                const double* w = p.partial + (i64)c*2*(BM*BN) + at + tc;
                s0 += w[0];
                s1 += w[DN_CT];
            }
        }
        if (GROUPS > 1)
        {
            __syncthreads();
            sums[grp][0][tc] = s0;
            sums[grp][1][tc] = s1;
            __syncthreads();
            if (grp > 0) continue;
            #pragma unroll
            for (int g = 1; g < GROUPS; g++) { s0 += sums[g][0][tc]; s1 += sums[g][1][tc]; }
        }
        if (!in) continue;
        if (CPLX)
        {
            update_z<false>(p, p.C + 2*(p.c_l[t.l] + __ldg(p.c_m + t.m0 + m) + __ldg(p.c_n + (t.n0 + n)/2)), s0, s1);
            continue;
        }
        double* Cm = p.C + p.c_l[t.l] + __ldg(p.c_m + t.m0 + m);
        double* d0 = Cm + __ldg(p.c_n + t.n0 + n);
        const double v0 = p.alpha*s0;
        *d0 = p.beta == 0.0 ? v0 : v0 + p.beta*(*d0);
        if (n + 1 < t.nrem)
        {
            double* d1 = Cm + __ldg(p.c_n + t.n0 + n + 1);
            const double v1 = p.alpha*s1;
            *d1 = p.beta == 0.0 ? v1 : v1 + p.beta*(*d1);
        }
    }
}

// a kernel's shared memory above 48 KB is allowed once per device (asked for before
// every launch it took 0.3 us of them)
static void dn_allow(std::atomic<unsigned long long>& done, const void* kern, size_t bytes)
{
    int dev = 0;
    TB_CUDA(cudaGetDevice(&dev));
    const unsigned long long bit = dev < 64 ? 1ull << dev : 0;
    if (done.load(std::memory_order_relaxed) & bit) return;
    TB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done |= bit;
}

template <int WGM, int WGN, int MF, int NF, int STAGES, int LAG, int TEAMS>
struct DenseTile
{
    static constexpr int BM = WGM*MF*16, BN = WGN*NF*8, GM = WGM, GN = WGN;
    template <int AM, int BMd, bool CPLX = false>
    static void go(const GemmF64Args& a, cudaStream_t s)
    {
        auto kern = gemm_f64_dense_kernel<WGM, WGN, MF, NF, STAGES, LAG, TEAMS, AM, BMd, CPLX>;
        constexpr size_t bytes = dn_smem<WGM, WGN, MF, NF, STAGES, TEAMS>();
        static std::atomic<unsigned long long> done{0};
        dn_allow(done, (const void*)kern, bytes);
        TimedLaunch t("gemm_f64_kernel", s);
        kern<<<(unsigned)a.grid, dn_threads(TEAMS), bytes, s>>>(a);
        check_launch("gemm_f64_dense_kernel");
    }
    // starts as the dense kernel's CTAs leave (its index arithmetic and launch
    // overlap them), and waits for all of them before it reads their sums
    template <int GROUPS>
    static void fixup(const GemmF64Args& a, int y, cudaStream_t s)
    {
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3((unsigned)a.sk_tiles, (unsigned)y);
        c.blockDim = dim3(DN_CT*GROUPS);
        c.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        c.attrs = at;
        c.numAttrs = 1;
        if (a.cplx) TB_CUDA(cudaLaunchKernelEx(&c, gemm_f64_fixup<WGM, WGN, MF, NF, GROUPS, true>, a));
        else TB_CUDA(cudaLaunchKernelEx(&c, gemm_f64_fixup<WGM, WGN, MF, NF, GROUPS, false>, a));
    }
    static void launch(const GemmF64Args& a, cudaStream_t s)
    {
        if (a.cplx) go<1, 1, true>(a, s);
        else switch (a.amode*2 + a.bmode)
        {
            case 0: go<0, 0>(a, s); break;
            case 1: go<0, 1>(a, s); break;
            case 2: go<1, 0>(a, s); break;
            default: go<1, 1>(a, s); break;
        }
        if (a.cut)
        {
            // few runs per tile: several elements a thread; many: the loads of
            // one element spread over four groups of threads
            if (a.sk_ctas >= 8*a.sk_tiles) fixup<4>(a, MF*NF*2, s);
            else fixup<1>(a, MF*NF, s);
            check_launch("gemm_f64_fixup");
        }
    }
};

typedef DenseTile<2, 4, 4, 4, 6, 1, 1> Tile128;      // 128 x 128, 192 KB of stages
typedef DenseTile<2, 4, 2, 2, 12, 1, 2> Tile64;      // 64 x 64, the same ring in bytes
typedef DenseTile<8, 1, 1, 4, 8, 2, 2> TileTall;     // 128 x 32, 180 KB

// Cycles of one k step of a tile with m rows and n columns, as measured: 128 for
// each 16 x 8 fragment pair of the busiest SM sub-core (the DMMA rate) and about
// 350 more, at least the gather of its operands (12 bytes per cycle and SM) and
// the time a producer warp takes to issue a stage (kFloor).
template <typename T>
double step_cycles(int m, int n)
{
    constexpr double kGather = 12.0, kFloor = T::BM == 128 && T::BN == 128 ? 1450.0 : 900.0;
    double load[4] = {0, 0, 0, 0};
    for (int cw = 0; cw < DN_CONSUMERS; cw++)
    {
        const int wm = cw/T::GN, wn = (cw + (T::GN/2)*wm) % T::GN;
        const int ni = std::max(0, ((m + 15)/16 - wm + T::GM - 1)/T::GM);
        const int nj = std::max(0, ((n + 7)/8 - wn + T::GN - 1)/T::GN);
        load[cw % 4] += 128.0*ni*nj;
    }
    return std::max({350.0 + std::max({load[0], load[1], load[2], load[3]}), (double)(m + n)*BK*8/kGather, kFloor});
}

// the work split of one tile shape and its modelled cycles
template <typename T>
double split_work(GemmF64Args& a, int sms, size_t ws_limit)
{
    // A tile's C update, or the way of its partial sums to the workspace, takes
    // kOut bytes per cycle and SM after its last step (its warps do nothing else
    // meanwhile) and kRun for its tables; the fixup starts kFixup late and moves
    // kChip bytes per cycle. Fitted to forced splits (us, uncut and cut): 4000 x
    // 4000 with k 16 64 and 64, k 64 109 and 135, k 500 557 and 559; 2000 x 2000 with k
    // 200 77 and 98; 40000 x 100 with k 500 217 and 190. (2000 cycles a tile and 26000 a
    // cut, as assumed before, cut 2000 x 2000 from k 200 on.)
    constexpr double kOut = 9, kRun = 700, kFixup = 15000, kChip = 1700, kUnit = 32;
    constexpr size_t kSlot = (size_t)T::BM*T::BN*sizeof(double);
    const i64 N = a.cplx ? 2*a.N : a.N;
    const i64 fm = a.M/T::BM, fn = N/T::BN, L = a.L;
    const int rm = (int)(a.M - fm*T::BM), rn = (int)(N - fn*T::BN);
    const i64 count[4] = {fm*fn*L, rm ? fn*L : 0, rn ? fm*L : 0, rm && rn ? L : 0};
    const int rows[4] = {T::BM, std::max(rm, 1), T::BM, std::max(rm, 1)};
    const int cols[4] = {T::BN, T::BN, std::max(rn, 1), std::max(rn, 1)};
    const double elem = a.beta != 0.0 || a.beta_im != 0.0 ? 16.0 : 8.0;      // C is read too
    const double kt = (double)a.kt;
    double cyc[4], update[4];
    i64 tiles = 0;
    double total = 0, longest = 0;
    for (int c = 0; c < 4; c++)
    {
        cyc[c] = step_cycles<T>(rows[c], cols[c]);
        update[c] = kRun + elem*rows[c]*cols[c]/kOut;
        tiles += count[c];
        total += (double)count[c]*(kt*cyc[c] + update[c]);
        if (count[c]) longest = std::max(longest, kt*cyc[c] + update[c]);
    }
    a.dp_tiles = tiles; a.sk_tiles = 0; a.sk_ctas = 0; a.cut = 0;
    a.sk_per = a.sk_extra = 0;
    a.grid = (int)std::min<i64>(tiles, sms);
    a.ws_bytes = 0;
    // tiles dealt in turn: whole rounds of them, or a part of one above the mean
    const double whole = tiles <= sms ? longest : std::max((double)((tiles + sms - 1)/sms)*total/(double)tiles,
                                                           total/sms + 0.25*longest);
    // A batch that fills the SMs is not cut: dealt in turn, neighbouring CTAs hold
    // neighbouring batch indices at the same k, and what they share (32-byte sectors
    // where the batch label is the fastest) is fetched once. Cut, every CTA has a run
    // of its own: 100 matrices of 300 x 300 x 300 took 378 us where uncut ones take 238,
    // and 1034 against 489 with the batch label fastest.
    if (L > 1 && tiles > sms) return whole;
    // cut: all but the last whole wave of whole tiles stays uncut
    const i64 dp = std::max<i64>(0, (count[0]/sms - 1)*sms);
    double units = 0;
    unsigned first = 0, wmax = 1;
    for (int c = 0; c < 4; c++)
    {
        const unsigned n = (unsigned)(count[c] - (c == 0 ? dp : 0));
        a.cls_first[c] = first;
        a.cls_w[c] = (unsigned)std::max(1.0, std::round(cyc[c]/kUnit));
        first += n;
        units += (double)n*kt*a.cls_w[c];
        if (n) wmax = std::max(wmax, a.cls_w[c]);
    }
    a.cls_first[4] = first;
    // no run below 1500 cycles (its pipeline start) or two steps of any class
    i64 ctas = std::min<i64>({(i64)sms, (i64)(units*kUnit/1500.0), (i64)(units/(2.0*wmax)), (i64)(ws_limit/(2*kSlot))});
    if (units >= (double)(1ll << 31) || ctas < 2 || (dp > 0 && ctas < sms)) return whole;
    const double sk = (double)(tiles - dp), fixed = std::min(sk, (double)ctas);      // tiles that the fixup sums
    const double slots = std::min((double)ctas + sk, 2.0*(double)ctas);
    double steps = 0, updates = 0, elements = 0;       // of the cut tiles
    for (int c = 0; c < 4; c++)
    {
        const double n = (double)(count[c] - (c == 0 ? dp : 0));
        steps += n*kt*cyc[c];
        updates += n*update[c];
        elements += n*rows[c]*cols[c];
    }
    const double mean = elements/sk;                   // elements of a tile
    const double cut = (double)(dp/sms)*(kt*cyc[0] + update[0]) + (steps + (sk - fixed)*updates/sk)/(double)ctas +
                       slots/(double)ctas*mean*8.0/kOut + kFixup + (slots*8.0 + fixed*elem)*mean/kChip;
    if (cut >= whole) return whole;
    a.dp_tiles = dp;
    a.sk_tiles = tiles - dp;
    a.sk_ctas = (int)ctas;
    a.sk_per = (unsigned)units/(unsigned)ctas;
    a.sk_extra = (unsigned)units - a.sk_per*(unsigned)ctas;
    a.cut = 1;
    a.grid = (int)ctas;
    a.ws_bytes = (size_t)ctas*2*kSlot;
    return cut;
}

} // namespace

// The tile shape and work split of least modelled time: 128 x 128 for most; 64
// x 64 (twice the operand bytes per FMA, a quarter of the partial sums) where a
// GEMM has few tiles or ragged ones; 128 x 32 where one extent is small, the
// operands swapped if that is the rows.
void gemm_f64_dense_plan(GemmF64Args& a, int sms, size_t ws_limit)
{
    const i64 per = a.cplx ? 2 : 1;                 // real columns and k per element
    if (a.N > a.M && per*a.M <= TileTall::BN)
    {
        // C^T = B^T A^T: the small extent becomes the columns
        std::swap(a.A, a.B);
        std::swap(a.a_m, a.b_n); std::swap(a.a_k, a.b_k); std::swap(a.a_l, a.b_l);
        std::swap(a.c_m, a.c_n); std::swap(a.M, a.N);
        std::swap(a.amode, a.bmode); std::swap(a.pair_a, a.pair_b);
        std::swap(a.conj_a, a.conj_b);
    }
    a.kt = (per*a.K + BK - 1)/BK;
    GemmF64Args b = a, c = a;
    a.tile = 0; b.tile = 1; c.tile = 2;
    const double t128 = split_work<Tile128>(a, sms, ws_limit), t64 = split_work<Tile64>(b, sms, ws_limit);
    const double tall = per*a.N <= TileTall::BN ? split_work<TileTall>(c, sms, ws_limit) : 1e300;
    // equal steps of a thin real GEMM: 128 x 32 where it fills more than 32 rows (us, 64 x
    // 64 and 128 x 32 tiles: 100 of 20 x 200 x 1000 103 and 87, 30000 of 5 x 40 x 40 506
    // and 457; 10000 of 32 x 32 x 40 171 and 217, 30000 complex of 5 x 40 x 3 574 and 683)
    const double bias = a.M > 32 && !a.cplx ? 1.03 : 1.0;
    if (t64 < t128 && t64*bias <= tall) a = b;
    else if (tall < t128) a = c;
}

// what gemm_f64_dense_inject_wait_timeout has set, and how often
static std::atomic<int> g_dn_hold{-1}, g_dn_changes{0};
static std::atomic<unsigned long long> g_dn_wait_ns{DN_WAIT_NS};

// The host's flag: one int of pinned memory that every device can write, so that
// reading it costs nothing.
static int* dn_error()
{
    static int* const flag = []
    {
        int* p = nullptr;
        TB_CUDA(cudaHostAlloc(&p, sizeof(int), cudaHostAllocPortable | cudaHostAllocMapped));
        *p = 0;
        return p;
    }();
    return flag;
}

void gemm_f64_dense_prepare() { dn_error(); }

static WaitControl wait_control() { return {dn_error(), g_dn_wait_ns.load(), g_dn_hold.load()}; }

void gemm_f64_dense_launch(GemmF64Args& a, cudaStream_t stream)
{
    a.ctl = wait_control();
    if (a.M == 0 || a.N == 0 || a.L == 0 || a.K == 0) return;
    TB_CHECK(a.L <= 65535, TB_ERR_SIZE, "batch extent too large");
    TB_CHECK(((a.M + 63)/64)*((a.N + 63)/64) < (1ll << 31), TB_ERR_SIZE, "tile grid too large");
    TB_CHECK(!a.cut || a.partial, TB_ERR_ARG, "cut tiles need a workspace");
    TB_CHECK(a.dp_tiles + a.sk_tiles < (1ll << 31), TB_ERR_SIZE, "tile grid too large");
    if (a.tile == 0) Tile128::launch(a, stream);
    else if (a.tile == 1) Tile64::launch(a, stream);
    else TileTall::launch(a, stream);
}

void gemm_f64_group_dense_tile(int& bm, int& bn) { bm = GD_BM; bn = GD_BN; }

size_t gemm_f64_group_dense_bytes(int ctas) { return (size_t)ctas*2*GD_BM*GD_BN*sizeof(double); }

void gemm_f64_group_dense_plan(const std::vector<GroupTile>& tiles, const std::vector<GroupExtents>& groups, int sms,
                               std::vector<GroupStart>& start, std::vector<GroupCut>& cuts)
{
    constexpr double kRun = 2500;                     // a tile's C update and operand tables
    std::vector<double> cyc(tiles.size());            // per k step
    double total = 0;
    for (size_t t = 0; t < tiles.size(); t++)
    {
        const GroupExtents& g = groups[tiles[t].g];
        const int m = (int)std::min<i64>(GD_BM, g.M - (i64)tiles[t].tm*GD_BM);
        const int n = (int)std::min<i64>(GD_BN, g.N - (i64)tiles[t].tn*GD_BN);
        cyc[t] = step_cycles<Tile128>(m, n);
        total += cyc[t]*g.nst + kRun;
    }
    // few CTAs where the work is small: no run below 3000 cycles
    const int ctas = (int)std::max(1.0, std::min((double)sms, total/3000.0));
    start.assign(1, GroupStart{0, 0});
    cuts.clear();
    double at = 0;                                    // cost before tile t
    size_t t = 0;
    for (int c = 1; c < ctas; c++)
    {
        const double want = total*c/ctas;
        while (t < tiles.size() && at + cyc[t]*groups[tiles[t].g].nst + kRun <= want)
        {
            at += cyc[t]*groups[tiles[t].g].nst + kRun;
            t++;
        }
        GroupStart s{(int)t, 0};
        if (t < tiles.size())
        {
            // a boundary inside a tile, at a whole step; close to an end it moves there
            const int nst = groups[tiles[t].g].nst;
            int step = (int)std::lround((want - at)/cyc[t]);
            if (step < 2) step = 0;
            if (step > nst - 2) { s.tile = (int)t + 1; step = 0; }
            s.step = step;
        }
        const GroupStart& last = start.back();
        if (s.tile < last.tile || (s.tile == last.tile && s.step < last.step)) s = last;
        start.push_back(s);
    }
    start.push_back(GroupStart{(int)tiles.size(), 0});
    // CTAs without work are dropped, so that a cut tile's runs are consecutive CTAs'
    std::vector<GroupStart> kept(1, start[0]);
    for (size_t c = 1; c < start.size(); c++)
        if (start[c].tile != kept.back().tile || start[c].step != kept.back().step) kept.push_back(start[c]);
    start.swap(kept);
    // a tile is cut where a boundary falls inside it: its runs are the last of the
    // CTA before (slot 0 if that is also that CTA's first) and the first of the others
    for (size_t c = 1; c + 1 < start.size(); c++)
    {
        if (start[c].step == 0) continue;
        if (!cuts.empty() && cuts.back().tile == start[c].tile) { cuts.back().count++; continue; }
        cuts.push_back(GroupCut{start[c].tile, (int)c - 1, 2, start[c - 1].tile == start[c].tile ? 0 : 1});
    }
}

void gemm_f64_group_dense_launch(const GroupDesc* d_groups, const GroupTile* d_tiles, const GroupStart* d_start, int ctas,
                                 const GroupCut* d_cuts, int ncuts, double* partial, int modes, cudaStream_t s)
{
    if (ctas <= 0) return;
    constexpr size_t bytes = dn_smem<2, 4, 4, 4, 6, 1>();
    auto go = [&](auto kern)
    {
        TB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
        TimedLaunch t("gemm_f64_group_dense_kernel", s);
        kern<<<(unsigned)ctas, dn_threads(1), bytes, s>>>(d_groups, d_tiles, d_start, partial, wait_control());
        check_launch("gemm_f64_group_dense_kernel");
    };
    switch (modes)
    {
        case 0: go(gemm_f64_group_dense_kernel<0, 0>); break;
        case 1: go(gemm_f64_group_dense_kernel<0, 1>); break;
        case 2: go(gemm_f64_group_dense_kernel<1, 0>); break;
        case 3: go(gemm_f64_group_dense_kernel<1, 1>); break;
        default: go(gemm_f64_group_dense_kernel<2, 2>);
    }
    if (ncuts > 0)
    {
        gemm_f64_group_fixup<<<dim3((unsigned)ncuts, 16), DN_CT, 0, s>>>(d_groups, d_tiles, d_cuts, partial);
        check_launch("gemm_f64_group_fixup");
    }
}

int gemm_f64_dense_error_flag()
{
    // reported once: the next check starts clean
    return __atomic_exchange_n(dn_error(), 0, __ATOMIC_ACQ_REL);
}

void gemm_f64_dense_inject_wait_timeout(int stage, double wait_seconds)
{
    const unsigned long long ns = wait_seconds > 0.0 ? (unsigned long long)(wait_seconds*1e9) : DN_WAIT_NS;
    g_dn_hold.store(stage);
    g_dn_wait_ns.store(ns);
    g_dn_changes++;
}

int gemm_f64_dense_control_changes() { return g_dn_changes.load(std::memory_order_relaxed); }

} // namespace tb
