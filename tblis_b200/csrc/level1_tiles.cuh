// level1_tiles.cuh -- level-1 kernels over pieces of two tensors whose fastest
// dimensions differ, are short or are ragged (included by level1.cu).
//
// A piece is a dense index space shared by A and B (a whole tensor, or one
// stored block of a block-sparse one). Dimension p is A's fastest, q is B's, the
// others are "outer". A tile covers tp x tq indices of (p, q) at tr consecutive
// outer indices, up to 256 threads x pc_ne elements, its extents chosen to divide
// the piece evenly: a 97 x 97 transpose takes 33 x 49 tiles, a 5 x 7 one takes 58
// outer indices at once, where fixed 64 x 64 tiles left 43% and 99% of the lanes
// idle. Lanes run along p for A and along q for B, and the tile turns around in
// shared memory (row length odd: no bank conflicts); where p is also B's fastest
// dimension (q absent) a thread reads back what it fetched.
//
// Where a thread's elements lie in a tile is the same for every tile of a piece,
// so it is worked out once a piece and kept in registers: a 32-bit offset within
// the tile, the outer index and the place in shared memory, and one bit an element
// and edge for the tiles that are cut short. Three divisions an element and pass
// instead made the kernel issue-bound. A's elements of the next tile travel to
// shared memory (cp.async) while the tile at hand is written, two or three CTAs an
// SM. Pieces come by value (one) or from a table
// (many: all blocks of a block-sparse tensor in one launch); a CTA takes a
// contiguous run of tiles, so it changes pieces rarely.
//
// Measured (FP64): B[baji] = A[abij] - B, extents 97, 97, 31, 31, 43.6 us = 5.0
// TB/s (113 us with 64 x 64 tiles); without reading B 32.7 us = 4.4 TB/s (64.7). The
// 512 blocks of an 8-irrep tensor of 30M elements: add 128 us, with beta 166, dot
// 140, norm 73 (a launch a block: 25 ms and more); their runs of 3 to 60 elements
// leave a tenth of the fetched sectors unused and the last CTAs a sixth behind.
#pragma once

struct Piece
{
    i64 np, nq, sap, saq, sbp, sbq;          // extents and strides (elements) of p and q
    i64 offa, offb;
    int nd;                                  // outer dimensions
    i64 len[L1_MAX_DIM], sa[L1_MAX_DIM], sb[L1_MAX_DIM];
    unsigned outer, tiles_p, tiles_q, first; // tiles: p fastest, then q, then outer; first tile of the piece
    int tp, tq, tr, turn;                    // turn: q present, through shared memory
};

constexpr int PC_THREADS = 256;
template <int OP> constexpr int pc_blocks() { return OP == 1 || OP == 2 ? 2 : 3; }  // CTAs an SM (B's elements in registers too)
template <typename T> constexpr int pc_ne() { return sizeof(T) >= 16 ? 4 : 8; }     // elements a thread and tile
template <typename T> constexpr int pc_tile() { return PC_THREADS*pc_ne<T>(); }
template <typename T> constexpr int pc_smem() { return pc_tile<T>()*9/8; }          // a tile with odd rows
constexpr int PC_TR = 256;
constexpr i64 PC_FEW = 148*2;                                // smaller tiles below this many

// accumulators of sums over pieces: at least double
template <typename T> struct PcAcc { typedef double type; };
template <typename R> struct PcAcc<cplx<R>> { typedef cplx<double> type; };
__host__ __device__ inline double pc_widen(double x) { return x; }
__host__ __device__ inline double pc_widen(float x) { return x; }
template <typename R> __host__ __device__ inline cplx<double> pc_widen(cplx<R> x)
{
    return cplx<double>((double)x.re, (double)x.im);
}

// the elements of a tile: all that a CTA takes, or a share of a small problem
template <typename T>
i64 pc_size(i64 elements)
{
    return std::max<i64>(PC_THREADS, std::min<i64>(pc_tile<T>(), (elements + PC_FEW - 1)/PC_FEW));
}

// chooses the tile of a piece, up to E elements; returns its number of tiles
template <typename T>
i64 pc_tiles(Piece& c, i64 E)
{
    constexpr i64 SM = pc_smem<T>();
    auto up = [](i64 a, i64 b) { return (a + b - 1)/b; };
    i64 tp = 1, tq = 1, tr = 1;
    if (!c.turn)
    {
        tp = up(c.np, up(c.np, E));
        tr = std::min<i64>({(i64)c.outer, E/tp, PC_TR});
    }
    else
    {
        // a few widths, the first that fills the tile (a few hundred pieces a call:
        // 32-bit divisions); for a small problem one width, since the call costs more
        // than the kernel
        typedef unsigned u32;
        auto evenly = [](i64 n, u32 w) -> u32        // n in the fewest equal parts of at most w
        {
            if (n <= (i64)w) return (u32)n;
            if (n >> 31) return w;
            const u32 parts = ((u32)n + w - 1)/w;
            return ((u32)n + parts - 1)/parts;
        };
        double best = -1;
        u32 seen = 0;
        const bool small = E < pc_tile<T>()/2;
        for (u32 w : {48u, 64u, 32u, 96u, 24u, 16u})
        {
            if (small) w = E < 512 ? 16 : 28;
            const u32 a = evenly(c.np, w);
            if (a == seen) continue;
            seen = a;
            const u32 b = evenly(c.nq, std::min(128u, std::max(1u, std::min((u32)E/a, (u32)SM/(a | 1)))));
            u32 r = 1;
            if (c.outer > 1) r = std::max(1u, std::min({c.outer, (u32)E/(a*b), (u32)SM/((a | 1)*b), (u32)PC_TR}));
            // filled share of the tile's elements, runs below 32 elements at a discount
            auto run = [](u32 x, i64 all) { return x >= 32 || all <= 32 ? 1.0 : (double)x*(1.0/32.0); };
            const double fill = (double)(a*b*r)*run(a, c.np)*run(b, c.nq);
            if (fill > best) { best = fill; tp = a; tq = b; tr = r; }
            if (small || fill >= 0.85*(double)E) break;
        }
    }
    // offsets within a tile are kept in 32 bits
    auto far = [&](i64 a, i64 b)
    {
        const double lim = 2147483647.0;
        return (double)(a - 1)*std::fabs((double)c.sap) + (double)(b - 1)*std::fabs((double)c.saq) > lim ||
               (double)(a - 1)*std::fabs((double)c.sbp) + (double)(b - 1)*std::fabs((double)c.sbq) > lim;
    };
    while (far(tp, tq))
        if (tq > 1 && (tp == 1 || far(1, tq))) tq = (tq + 1)/2;
        else tp = (tp + 1)/2;
    c.tp = (int)tp; c.tq = (int)tq; c.tr = (int)tr;
    c.tiles_p = (unsigned)up(c.np, tp);
    c.tiles_q = (unsigned)up(c.nq, tq);
    return up(c.np, tp)*up(c.nq, tq)*up(c.outer, tr);
}

// the tile at hand, shared by the CTA: offsets of its outer indices (p0 and q0
// included); bits 0, 1, 2 of edge: the last tile along p, q, outer
struct PcTile
{
    i64 oa[PC_TR], ob[PC_TR];
    int edge;
};

// fills t for tile number `tile` of piece c (all threads; ends with a barrier)
__device__ __forceinline__ void pc_setup(const Piece& c, unsigned tile, PcTile& t)
{
    const unsigned pq = c.tiles_p*c.tiles_q;
    const unsigned ro = tile/pq, in = tile - ro*pq, iq = in/c.tiles_p, ip = in - iq*c.tiles_p;
    const i64 p0 = (i64)ip*c.tp, q0 = (i64)iq*c.tq;
    const unsigned r0 = ro*(unsigned)c.tr;
    for (int r = threadIdx.x; r < c.tr && r < c.outer - r0; r += PC_THREADS)
    {
        unsigned o = r0 + r;
        i64 oa = c.offa + p0*c.sap + q0*c.saq, ob = c.offb + p0*c.sbp + q0*c.sbq;
        for (int d = 0; d < c.nd; d++)
        {
            const unsigned ld = (unsigned)c.len[d], qq = o/ld, i = o - qq*ld;
            oa += (i64)i*c.sa[d];
            ob += (i64)i*c.sb[d];
            o = qq;
        }
        t.oa[r] = oa;
        t.ob[r] = ob;
    }
    if (threadIdx.x == 0)
        t.edge = (ip + 1 == c.tiles_p) | (iq + 1 == c.tiles_q) << 1 | (c.outer - r0 <= (unsigned)c.tr) << 2;
    __syncthreads();
}

// e/d for e below 2^11 and inv = ceil(2^32/d)
__device__ __forceinline__ int pc_div(int e, unsigned inv, int d) { return d == 1 ? e : (int)__umulhi((unsigned)e, inv); }

// where this thread's elements lie in the tiles of a piece, in A's order (p
// fastest) or B's
template <int NE>
struct PcSpots
{
    int rel[NE];                             // offset within the tile
    unsigned at[NE];                         // place in shared memory << 8 | outer index
    unsigned in;                             // a bit an element, by bytes: in the tile; in the last one along p, q, outer

    // element u's offset from the tensor's base (o: those of the tile's outer
    // indices). The empty asm keeps the compiler from holding 64-bit addresses of
    // all elements from tile to tile, which spilled.
    __device__ __forceinline__ i64 offset(int u, const i64* o) const
    {
        int x = rel[u];
        asm volatile("" : "+r"(x));
        return o[at[u] & 255] + x;
    }
};
template <int NE>
__device__ __forceinline__ void pc_spots(const Piece& c, bool q_fast, i64 sp, i64 sq, PcSpots<NE>& w)
{
    const int lp = (int)(c.np - (i64)(c.tiles_p - 1)*c.tp), lq = (int)(c.nq - (i64)(c.tiles_q - 1)*c.tq);
    const int lr = (int)(c.outer - (c.outer - 1)/(unsigned)c.tr*(unsigned)c.tr);
    const int fast = q_fast ? c.tq : c.tp, slow = q_fast ? c.tp : c.tq, n = c.tp*c.tq*c.tr;
    const int ld = c.turn ? c.tp | 1 : c.tp;             // rows of a tile that turns: odd (pc_tiles holds them to pc_smem)
    const unsigned inv_f = 0xffffffffu/(unsigned)fast + 1u, inv_s = 0xffffffffu/(unsigned)slow + 1u;
    w.in = 0;
    #pragma unroll
    for (int u = 0; u < NE; u++)
    {
        w.rel[u] = 0;
        w.at[u] = 0;
        if (PC_THREADS*u >= n) continue;
        const int e = threadIdx.x + PC_THREADS*u, x = pc_div(e, inv_f, fast), f = e - x*fast;
        const int r = pc_div(x, inv_s, slow), g = x - r*slow;
        const int i = q_fast ? g : f, j = q_fast ? f : g;
        w.rel[u] = (int)(i*sp + j*sq);
        w.at[u] = (unsigned)((r*c.tq + j)*ld + i) << 8 | (unsigned)r;
        w.in |= ((unsigned)(r < c.tr) | (unsigned)(i < lp) << 8 | (unsigned)(j < lq) << 16 | (unsigned)(r < lr) << 24) << u;
    }
}
// the elements that a tile has
template <int NE>
__device__ __forceinline__ unsigned pc_mask(const PcSpots<NE>& w, int edge)
{
    unsigned m = w.in;
    if (edge & 1) m &= w.in >> 8;
    if (edge & 2) m &= w.in >> 16;
    if (edge & 4) m &= w.in >> 24;
    return m & 255;
}

template <typename T>
__device__ __forceinline__ void pc_copy(T* to, const T* from)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;"
                 :: "r"((unsigned)__cvta_generic_to_shared(to)), "l"(from), "n"((int)sizeof(T)) : "memory");
}

// OP 0: B = alpha*op(A) (B not read), 1: B = alpha*op(A) + beta*op(B),
// 2: sum of op(A)*op(B), 3: sum of red_val(op, A), both in at least double precision
template <typename T, int OP>
__global__ void __launch_bounds__(PC_THREADS, pc_blocks<OP>())
k_pieces(const T* __restrict__ A, T* __restrict__ B, const Piece one, const Piece* __restrict__ many, int npieces,
         unsigned ntiles, T alpha, T beta, bool conj_a, bool conj_b, int red_op, typename PcAcc<T>::type* partial)
{
    constexpr int NE = pc_ne<T>();
    typedef typename PcAcc<T>::type Acc;
    __shared__ T buf[2][pc_smem<T>()];
    __shared__ PcTile ts[2];
    __shared__ Piece held;
    Acc acc = Acc(0);
    // this CTA's run of tiles
    const unsigned t0 = (unsigned)((unsigned long long)ntiles*blockIdx.x/gridDim.x);
    const unsigned t1 = (unsigned)((unsigned long long)ntiles*(blockIdx.x + 1)/gridDim.x);
    int pi = 0;
    if (many && t0 < t1)
    {
        int lo = 0, hi = npieces - 1;
        while (lo < hi)
        {
            const int mid = (lo + hi + 1) >> 1;
            if (many[mid].first <= t0) lo = mid; else hi = mid - 1;
        }
        pi = lo;
    }
    PcSpots<NE> wa, wb;
    const Piece& c = held;
    for (unsigned tile = t0; tile < t1; pi++)
    {
        // the piece into shared memory (the last tile's readers are past their barrier)
        const int* src = many ? reinterpret_cast<const int*>(many + pi) : reinterpret_cast<const int*>(&one);
        for (int w = threadIdx.x; w < (int)(sizeof(Piece)/4); w += PC_THREADS) reinterpret_cast<int*>(&held)[w] = src[w];
        __syncthreads();
        const unsigned first = c.first, end = pi + 1 < npieces ? min(t1, many[pi + 1].first) : t1;
        pc_spots(c, false, c.sap, c.saq, wa);
        if (OP != 3) pc_spots(c, c.turn != 0, c.sbp, c.sbq, wb);
        auto fetch = [&](const PcTile& t, T* to)
        {
            const unsigned m = pc_mask(wa, t.edge);
            #pragma unroll
            for (int u = 0; u < NE; u++)
                if (m >> u & 1) pc_copy(to + (wa.at[u] >> 8), A + wa.offset(u, t.oa));
        };
        int b = 0;
        if (tile < end)
        {
            pc_setup(c, tile - first, ts[0]);
            fetch(ts[0], buf[0]);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (; tile < end; tile++, b ^= 1)
        {
            const PcTile& t = ts[b];
            const PcSpots<NE>& w = OP == 3 ? wa : wb;
            const unsigned m = pc_mask(w, t.edge);
            T y[NE];
            if (OP == 1 || OP == 2)
            {
                #pragma unroll
                for (int u = 0; u < NE; u++)
                    if (m >> u & 1) y[u] = B[w.offset(u, t.ob)];
            }
            if (tile + 1 < end)
            {
                pc_setup(c, tile + 1 - first, ts[b ^ 1]);
                fetch(ts[b ^ 1], buf[b ^ 1]);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            #pragma unroll
            for (int u = 0; u < NE; u++)
            {
                if (!(m >> u & 1)) continue;
                const T x = buf[b][w.at[u] >> 8];
                if (OP == 2) acc += pc_widen(cj(x, conj_a))*pc_widen(cj(y[u], conj_b));
                else if (OP == 3) acc += red_val(red_op, pc_widen(x));     // float squares leave its range
                else
                {
                    const T v = alpha*cj(x, conj_a);
                    B[w.offset(u, t.ob)] = OP == 0 ? v : v + beta*cj(y[u], conj_b);
                }
            }
            __syncthreads();                 // this tile's buffers, and held, may change
        }
    }
    if (OP >= 2)
    {
        for (int o = 16; o > 0; o >>= 1) acc += shfl_down(acc, o);
        __shared__ Acc ws[PC_THREADS/32];
        if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = acc;
        __syncthreads();
        if (threadIdx.x == 0)
        {
            Acc s = Acc(0);
            for (int w = 0; w < PC_THREADS/32; w++) s += ws[w];
            partial[blockIdx.x] = s;
        }
    }
}
