// gemm_f64.hpp -- FP64 DMMA block-scatter contraction kernel (see gemm_f64.cu)
#pragma once

#include "common.hpp"

namespace tb
{

// the bounded waits of the dense kernel: the host's flag of one that gave up, their
// limit, and a ring stage that never fills up (test support, -1: none)
struct WaitControl
{
    int* error;
    unsigned long long wait_ns;
    int hold_stage;
};

// A kernel argument: 376 bytes took the host 0.7 us a launch more than 352 (11.6 and
// 10.9 us for the whole call of a small contraction), so the fields that only one
// of the launchers uses share their place.
struct GemmF64Args
{
    const double* A;
    const double* B;
    double* C;
    // scatter vectors (device): element offsets per GEMM index
    const i64 *a_m, *a_k, *b_k, *b_n, *c_m, *c_n, *a_l, *b_l, *c_l;
    union
    {
        // gemm_f64_launch: per-BK-block common k strides of A and B (0 = irregular
        // block), and its own share of k
        struct { const i64 *a_kbs, *b_kbs; i64 k_per_split; };
        WaitControl ctl;     // the dense kernel's launcher sets it
    };
    i64 M, N, K, L;
    double alpha, beta;
    int amode, bmode;        // gather directions (see GemmView)
    int splits;              // split-K factor
    double* partial;         // split-K workspace (splits*L*M*N doubles)
    int variant;             // tile configuration, 0 = automatic
    // complex contraction (dense kernel only; offsets and extents in complex
    // elements, every element 16-byte aligned)
    int cplx, conj_a, conj_b, conj_c;
    double alpha_im, beta_im;
    // dense kernel: run only if the word at gate is above gate_above (null: always)
    const unsigned* gate;
    unsigned gate_above;
    int pair_a, pair_b;      // gather the operand's contiguous dimension in pairs (16-byte copies)
    // set by gemm_f64_dense_plan: k steps of a tile, tiles done whole, tiles
    // whose k steps are cut into equal runs over sk_ctas CTAs, CTAs, workspace
    // (tile: 0 = 128 x 128, 1 = 64 x 64, 2 = 128 x 32), and of the cut tiles the
    // first of each class, its cost per k step and the cost per CTA
    i64 kt, dp_tiles, sk_tiles;
    int sk_ctas, cut, grid, tile;
    unsigned sk_per, sk_extra, cls_first[5], cls_w[4];
    size_t ws_bytes;
};

static_assert(sizeof(GemmF64Args) <= 352, "GemmF64Args as a kernel argument");

// one K segment of a grouped GEMM: the rows of A / columns of B it reads
// and its k range (all segments of a group accumulate into the same C tile)
struct SegDesc
{
    const i64 *a_m, *a_k, *b_k, *b_n, *a_kbs, *b_kbs;
    i64 K;
};

// one GEMM of a grouped launch (no batch dimension: one entry per batch index).
// With nseg == 0 the group has a single segment given by the inline fields;
// otherwise segs[0..nseg) replace them (A and B offsets per segment).
struct GroupDesc
{
    const double* A;
    const double* B;
    double* C;
    const i64 *a_m, *a_k, *b_k, *b_n, *c_m, *c_n, *a_kbs, *b_kbs;
    i64 M, N, K;
    double alpha, beta;
    int amode, bmode;
    int nseg;
    const SegDesc* segs;
    // packed path (gemm_f64_ws.cu): tile shape (gemm_f64_ws_shape), k steps
    // over all segments, and the offsets (in doubles) of the group's packed A
    // panels and B panels
    int shape;
    int nst;
    i64 pa, pb;
    // dense grouped path: gather of A and B: 0 single elements, 1 pairs; in a plan
    // whose groups differ in direction 0 and 1 along k, 2 single elements along the
    // rows
    int how_a, how_b;
};

// The dense grouped path (gemm_f64_dense.cu): a plan lists the 128 x 128 tiles
// of its groups (those with k steps), and gemm_f64_group_dense_plan deals their k
// steps to CTAs in runs of equal modelled cost: CTA c starts at start[c] and ends
// at start[c + 1]; cuts lists the tiles that several CTAs share.
struct GroupTile { int g, tm, tn; };
struct GroupStart { int tile, step; };
struct GroupCut { int tile, cta, count, slot; };     // runs of CTAs [cta, cta + count), the first in `slot`
struct GroupExtents { i64 M, N; int nst; };
void gemm_f64_group_dense_tile(int& bm, int& bn);
size_t gemm_f64_group_dense_bytes(int ctas);         // workspace for the partial sums
void gemm_f64_group_dense_plan(const std::vector<GroupTile>& tiles, const std::vector<GroupExtents>& groups, int sms,
                               std::vector<GroupStart>& start, std::vector<GroupCut>& cuts);
void gemm_f64_group_dense_launch(const GroupDesc* d_groups, const GroupTile* d_tiles, const GroupStart* d_start, int ctas,
                                 const GroupCut* d_cuts, int ncuts, double* partial, int modes, cudaStream_t s);
// (modes: 2*amode + bmode shared by all groups, or 4)

// one piece of a panel to pack: k steps [s0, s0 + ns) of rows
// [panel*BM, ...) of group g's A (side 0), or of columns [panel*BN, ...) of
// its B (side 1); steps are counted over all segments of the group
struct PackItem
{
    int g, side, panel, s0, ns, pad;
};

int gemm_f64_num_variants();
void gemm_f64_variant_tile(int variant, int& bm, int& bn);
// variants of a grouped launch: the tile family above, the packed path
// (variant gemm_f64_num_variants() + 1, tiles of each group's own shape; run
// by the grouped plan, not by gemm_f64_grouped_launch)
int gemm_f64_grouped_num_variants();
bool gemm_f64_is_ws_variant(int variant);
// the dense grouped path, the last variant
bool gemm_f64_is_dense_variant(int variant);

// The packed grouped path (gemm_f64_ws.cu): gemm_f64_ws_pack gathers the A
// row panels and B column panels of every group into contiguous, swizzled
// 16-wide k steps (panel p of group g at pa / pb + p*nst*P*16, P the panel
// width of the group's shape); gemm_f64_ws_launch then runs the groups' tiles
// on them, one producer lane streaming the blocks with bulk copies and four
// consumer warps running the MMAs, consecutive tiles overlapping.
// shape: bit 1 = 32 rows (else 64), bit 0 = 32 columns (else 64)
int gemm_f64_ws_shape(i64 M, i64 N, i64 K);
void gemm_f64_ws_tile(int shape, int& bm, int& bn);
void gemm_f64_ws_pack(const GroupDesc* d_groups, const PackItem* d_items, int nitems, double* packA,
                      double* packB, cudaStream_t stream);
// tile_begin[g] = first tile of group g in tiles of its own shape; d_counter
// as for gemm_f64_grouped_launch
void gemm_f64_ws_launch(const GroupDesc* d_groups, const i64* d_tile_begin, int ngroups, i64 total_tiles,
                        const double* packA, const double* packB, cudaStream_t stream,
                        unsigned long long* d_counter);
// 1 when a kernel of gemm_f64_ws.cu gave up a bounded wait since the last
// call (the flag is cleared by reading it)
int gemm_f64_error_flag();
// test support: the packed GEMM's producer issues no copy for the CTA's
// stage number `step` (-1: none) and every bounded wait gives up after
// wait_seconds (<= 0: the default 2 s)
void gemm_f64_inject_wait_timeout(int step, double wait_seconds);
// tile_begin[g] = first global tile of group g (tiles of BM x BN of the variant).
// d_counter (optional, one 64-bit word of device memory, zeroed by the launch)
// turns the static tile striding into a dynamic queue.
void gemm_f64_grouped_launch(const GroupDesc* d_groups, const i64* d_tile_begin, int ngroups,
                             i64 total_tiles, int variant, cudaStream_t stream,
                             unsigned long long* d_counter = nullptr);

i64 gemm_f64_tile_m();
i64 gemm_f64_tile_n();
i64 gemm_f64_tile_k();
int gemm_f64_choose_splits(i64 M, i64 N, i64 K, i64 L, int num_sms);
size_t gemm_f64_workspace_bytes(i64 M, i64 N, i64 L, int splits);
void gemm_f64_launch(GemmF64Args a, cudaStream_t stream);

// The dense kernel (gemm_f64_dense.cu): plan sets the work split for `sms` SMs
// and a.ws_bytes, at most ws_limit bytes of workspace for a.partial; launch
// runs it.
void gemm_f64_dense_plan(GemmF64Args& a, int sms, size_t ws_limit);
void gemm_f64_dense_launch(GemmF64Args& a, cudaStream_t stream);
void gemm_f64_dense_prepare();             // the launches' one allocation, made once
// nonzero once after a dense kernel (also a grouped one) gave up a wait
int gemm_f64_dense_error_flag();
// test support: ring stage `stage` never fills (-1: none) and waits give up after wait_seconds (0: 2 s)
void gemm_f64_dense_inject_wait_timeout(int stage, double wait_seconds);
int gemm_f64_dense_control_changes();      // times that was called: a captured launch holds older values

} // namespace tb
