// fse_tick.cu -- the cell update of world::tick() (source/engine/world.cpp:1036-1948)
// as one colour-pass kernel.
//
// A launch handles one chunk colour of one iteration (world.cpp:1050-1077) for a
// list of chunks, possibly of many worlds, or every pass of a tick (the fused tick).
// Each CTA stages its chunk plus a halo in shared memory (a word per cell, scalar,
// colour; the pending fluid diff stays in HBM and is touched only by SOUP cells), runs
// sweeps A, B and C as sequences of lattice sub-phases separated by __syncthreads(), and
// writes back only the cells it changed. The lattice spacing makes every write set of a
// sub-phase disjoint from every other cell's read and write sets, so the result does not
// depend on thread timing.
//
// What bounds it: the slowest warp of each of the 30 sub-phases, one after another, as the
// tile takes an SM's shared memory and a chunk-pass its SM. A wet 128 x 128 chunk takes 95 us
// a pass (140 us before the steps below), of which sweep A's rules take about 45%,
// finding and listing its cells and its barriers 20%, sweep B 25%, staging and write-back
// 10%; DRAM moves 3% of what it could. So what counts is the length of the chain of
// dependent instructions and loads that a warp goes through in a sub-phase:
// - one word per cell answers what a rule asks of a neighbour (see CW_*);
// - a sub-phase first finds the cells that a rule may change and deals them to the threads,
//   liquids to the first warps and the others to the last, so that a warp runs one rule
//   with most of its lanes; the rare cases (free fall, another liquid beside, fire,
//   reactions) are with the others, so that they do not lengthen the flowing liquids' rule;
// - what comes from HBM (the diff of a displaced or falling liquid, a staging slot) is asked
//   for as soon as its address is known, and used after the next barrier where it can be.
// Tried and slower: blocks of the chunk that wait only for their neighbours (mbarrier
// arrivals release, and so wait for the diff reductions in flight: 215 us a pass against
// 131 then), requesting the next sub-phase's diffs a sub-phase ahead (512 x 512 tick 1.005 ->
// 1.052 ms).
//
// The reference copies neighbour cells into locals and writes those copies back
// later; no rule modifies such a neighbour between the copy and the write-back, so
// here the write-back is a move inside shared memory at write time (move()), which
// keeps only the active cell in registers.
//
// The kernel is built twice (template TEMP): worlds that keep liquid temperatures
// (FSE_CFG_TEMPERATURE) copy them with every liquid move; the others run code with
// no trace of that plane. fse_tick_temp.cu compiles the TEMP instantiation as a
// translation unit of its own (including this file with FSE_TICK_TEMP_TU), so the
// two build in parallel.
#include <algorithm>

#include "fse_internal.cuh"

// Optional per-phase cycle counters of the colour pass (build with
// -DFSE_PHASE_CLOCKS): thread 0 of each CTA accumulates clock64() deltas between
// barriers; fse_debug_phase_clocks() reads the totals. Off by default: no cost.
#ifdef FSE_PHASE_CLOCKS
static __device__ unsigned long long g_phase_clk[16];  // per translation unit
static __device__ unsigned long long g_phase_max[16];  // per phase: the largest CTA total; [15]: largest CTA
#define FSE_PT_DECL                       \
    __shared__ long long pt_acc[16];      \
    long long pt_last = clock64();        \
    const long long pt_first = pt_last;   \
    if (threadIdx.x < 16) pt_acc[threadIdx.x] = 0;
#define FSE_PT(k)                           \
    if (threadIdx.x == 0) {                 \
        long long t_ = clock64();           \
        pt_acc[(k)] += t_ - pt_last;        \
        pt_last = t_;                       \
    }
#define FSE_PT_FLUSH                                                                                   \
    __syncthreads();                                                                                   \
    if (threadIdx.x < 15) {                                                                            \
        atomicAdd(&g_phase_clk[threadIdx.x], (unsigned long long)pt_acc[threadIdx.x]);                 \
        atomicMax(&g_phase_max[threadIdx.x], (unsigned long long)pt_acc[threadIdx.x]);                 \
    }                                                                                                  \
    if (threadIdx.x == 15) atomicMax(&g_phase_max[15], (unsigned long long)(clock64() - pt_first));
#else
#define FSE_PT_DECL
#define FSE_PT(k)
#define FSE_PT_FLUSH
#endif

namespace fse {

constexpr int MAXRW = 160;        // tile row width bound (chunk <= 128, halo <= 5), a multiple of 32

// 4-byte global -> shared copy that does not pass through registers (sm_80+ cp.async)
__device__ __forceinline__ void cp_async4(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// q = e / n and r = e % n for 0 <= e < 2^16, 1 <= n <= 256, from a float reciprocal
// of n: (e + 0.5) / n sits at least 0.5 / n from an integer, far more than the
// float error, so the truncation is exact.
__device__ __forceinline__ void divmod_small(int e, int n, float rn, int &q, int &r) {
    q = (int)(((float)e + 0.5f) * rn);
    r = e - q * n;
}

// ------------------------------------------------------------- cell words
// A cell of the shared-memory tile is one 32-bit word beside its scalar and colour
// planes: the material id, the flags byte, what the rules ask of the material (its
// type, whether it is updated in this iteration, whether it burns or reacts) and its
// density rank. One load then answers every question a rule asks of a neighbour;
// with id and flags in planes of their own and the material's type and density looked
// up in tables, each question was a chain of two or three dependent shared loads, and
// those chains set the length of a sub-phase.
//
// Ranks order the materials by density: AIR 0, SOLID 255 and the others by increasing
// density from 1, equal densities equal ranks (MatTable::word, built on the host), so
// that "AIR, or not SOLID and less dense" is one unsigned comparison (cw_sink).
constexpr uint32_t CW_ID = 0xFFu;
constexpr uint32_t CW_FLAGS = 0xFF00u;  // the flags byte: MOVED, VISITED, settle count
constexpr uint32_t CW_SETTLE = (uint32_t)SETTLE_MASK << 8;
constexpr uint32_t CW_VIS = (uint32_t)VISITED << 8;
constexpr uint32_t CW_MOVED = (uint32_t)MOVED << 8;
constexpr uint32_t CW_TYPE = MW_TYPE;
constexpr uint32_t CW_LIVE = 1u << 19;   // the material's iterations exceed this pass's
constexpr uint32_t CW_DIRTY = 1u << 20;  // the cell must be written back
constexpr uint32_t CW_FIRE = MW_FIRE;
constexpr uint32_t CW_REACT = MW_REACT;
constexpr uint32_t CW_RANK = MW_RANK;
// the bits a cell takes from its material
constexpr uint32_t CW_MAT = ~(CW_FLAGS | CW_DIRTY);

__device__ __forceinline__ int cw_id(uint32_t w) { return (int)(w & CW_ID); }
__device__ __forceinline__ bool cw_is(uint32_t w, int type) { return (w & CW_TYPE) == (uint32_t)type << MW_TYPE_SHIFT; }
__device__ __forceinline__ bool cw_air(uint32_t w) { return (w & CW_TYPE) == 0; }
__device__ __forceinline__ bool cw_same(uint32_t a, uint32_t b) { return ((a ^ b) & CW_ID) == 0; }
// cells that sand `w` sinks into have words below this: AIR, or not SOLID and less
// dense (a SAND of rank 255 has no density to compare, a NaN: only AIR is below it)
__device__ __forceinline__ uint32_t cw_sink(uint32_t w) { return w >= CW_RANK ? 1u << 24 : w & CW_RANK; }

struct Cell {
    uint32_t w;  // its word; the VISITED and DIRTY bits mean nothing here
    int32_t sc;
    uint32_t col;
    int32_t df;
};

// ------------------------------------------------------- shared-memory tile
// Region: x in [cx - 2, cx + C + HALO), full state for y in [cy - 2, cy + C + HALO),
// words only down to y < cy + C + 10 (the deepest read, the friction pillar of
// world.cpp:1619-1627).
//
// Every access of the rules stays inside the tile: relative to the active cell
// they reach x +- 2 (fire), y - 2 .. y + 2 in the full planes, words down to y + 4
// (sand and liquid free fall), and the interaction boxes, which lie right of and
// below the cell (a box with a negative corner is not visited) with offset + radius
// <= 5 enforced at registration and run with HALO = 5; the sweep-B pillar reads
// words down to cy + C + 9. So the tile needs no bounds checks. Where the tile
// crosses the world edge it holds GENERIC_SOLID, which is what world.cpp:999-1002
// reads there; the only writes that can reach such cells are those of fire and
// interactions, which check the world bounds themselves (world.cpp:1003-1008 drops
// them).
constexpr int HALO_LO = 2;  // cells staged left of and above the chunk

struct TileData {
    uint32_t *s_w;
    int32_t *s_sc;
    uint32_t *s_col;
    const uint32_t *mw;  // material id -> word of a new cell (flags clear)
    int32_t *df;         // HBM diff plane
    int16_t *tp;         // HBM temperature plane of SOUP cells (NULL: not kept)
    int x0, y0, RW, RHF, RHI;
    int W, H;
    int id_air;
    // sweep-B pillar snapshot: AIR bits of columns ax0.., rows ay0.., 5 words per column
    const uint32_t *s_air;
    int ax0, ay0, aw;
    // a chunk split over a CTA pair: the partner's copy of the planes (shared::cluster
    // addresses); cell i of this tile is cell i + pd of the partner's, both of RW
    // columns and RHF, RHI rows
    uint32_t p_w, p_sc, p_col;
    int pd;
};

// --------------------------------------------------- CTA-pair (cluster) helpers
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// the address of this CTA's shared location `a` in the shared memory of cluster rank r
__device__ __forceinline__ uint32_t mapa_rank(uint32_t a, uint32_t r) {
    uint32_t o;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(r));
    return o;
}
__device__ __forceinline__ void st_cluster_u32(uint32_t a, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// every thread of both CTAs of the pair; the partner's shared-memory stores made
// before it are visible after it
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// ------------------------------------------------------ TMA staging helpers
// The 4-byte planes of a tile come in as two 2D tensor copies (cp.async.bulk.tensor)
// completing on one mbarrier; thread 0 issues them, every thread waits.
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// orders this thread's generic shared-memory accesses before later async-proxy ones
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// the same for global memory
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// box of the tensor map at (x, y) (x a multiple of 4 cells: a 16-byte boundary) into
// dst (128-byte aligned); complete_tx on bar
__device__ __forceinline__ void tma_load_2d(void *dst, const void *tmap, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(smem_addr(dst)),
        "l"(tmap), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

// ------------------------------------------------- fused-tick flag helpers
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_gpu(uint32_t *p, uint32_t v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
constexpr unsigned long long FUSED_WAIT_NS = 2000000000ull;  // a dependency wait gives up after 2 s

// LIVE: the pillar reads the tile as it stands (the reference's own order, where
// one thread updates the chunk's cells in turn) instead of the sweep-B snapshot.
// F32: liquid amounts and diffs are f32 bit patterns (FSE_CFG_F32_FLUID).
// PAIR: the chunk is split over a CTA pair; every write to a row the partner's tile
// holds is made in both copies (reads are always local), so both copies of the
// shared rows stay equal; at the end of a sub-phase the cluster barrier makes them
// visible.
//
// Cells are named by their tile index i (neighbours i +- 1, i +- RW) and, for the
// planes in HBM, their world index g (neighbours g +- 1, g +- W).
template <bool TEMP, bool LIVE = false, bool F32 = false, bool PAIR = false>
struct Tile : TileData {
    static constexpr bool kTemp = TEMP;
    static constexpr bool kF32 = F32;
    __device__ __forceinline__ explicit Tile(const TileData &d) : TileData(d) {}

    __device__ __forceinline__ int li(int x, int y) const { return (y - y0) * RW + (x - x0); }
    __device__ __forceinline__ int gi(int x, int y) const { return y * W + x; }
    __device__ __forceinline__ uint32_t at(int i) const { return s_w[i]; }
    __device__ __forceinline__ bool air(int i) const { return cw_air(s_w[i]); }
    // inside the world: the writes of fire and interactions can reach cells outside it,
    // where world.cpp:1003-1008 drops them
    __device__ __forceinline__ bool in_world(int x, int y) const {
        return (unsigned)x < (unsigned)W && (unsigned)y < (unsigned)H;
    }

    // store a cell's word, and its planes, in both copies of a pair
    __device__ __forceinline__ void set_word(int i, uint32_t w) const {
        s_w[i] = w;
        if constexpr (PAIR) {
            const int j = i + pd;
            if (j >= 0 && j < RW * RHI) st_cluster_u32(p_w + 4u * (uint32_t)j, w);
        }
    }
    __device__ __forceinline__ void set_planes(int i, int32_t sc, uint32_t col) const {
        s_sc[i] = sc;
        s_col[i] = col;
        if constexpr (PAIR) {
            const int j = i + pd;
            if (j >= 0 && j < RW * RHF) {
                st_cluster_u32(p_sc + 4u * (uint32_t)j, (uint32_t)sc);
                st_cluster_u32(p_col + 4u * (uint32_t)j, col);
            }
        }
    }
    __device__ __forceinline__ void set_sc(int i, int32_t sc) const {
        s_sc[i] = sc;
        if constexpr (PAIR) {
            const int j = i + pd;
            if (j >= 0 && j < RW * RHF) st_cluster_u32(p_sc + 4u * (uint32_t)j, (uint32_t)sc);
        }
    }

    // 10 AIR bits of the column of cell i (at (x, y)) starting at it: from the snapshot
    // (0 outside it), or live
    __device__ __forceinline__ uint32_t air10(int i, int x, int y) const {
        if constexpr (LIVE) {
            uint32_t bits = 0;
            for (int k = 0; k < 10; k++)
                if (air(i + k * RW)) bits |= 1u << k;
            return bits;
        }
        int sx = x - ax0, sy = y - ay0;
        if ((unsigned)sx >= (unsigned)aw || sy < 0) return 0u;
        const uint32_t *col = s_air + sx * 5;
        int wi = sy >> 5, b = sy & 31;
        if (wi >= 5) return 0u;
        unsigned long long v = col[wi] | ((unsigned long long)(wi + 1 < 5 ? col[wi + 1] : 0u) << 32);
        return (uint32_t)(v >> b) & 0x3FFu;
    }

    __device__ __forceinline__ int32_t df_load(int g) const { return df[g]; }
    // the pending diff of cell i (0 where it is not SOUP)
    __device__ __forceinline__ int32_t df_of(int i, int g) const { return cw_is(s_w[i], T_SOUP) ? df[g] : 0; }
    // cell i becomes `c`; the visited mark stays with the position
    __device__ __forceinline__ void put(int i, int g, const Cell &c) const {
        set_word(i, (c.w & ~CW_VIS) | CW_DIRTY | (s_w[i] & CW_VIS));
        set_planes(i, c.sc, c.col);
        if (cw_is(c.w, T_SOUP)) df[g] = c.df;
    }
    // the same, for a cell known not to be SOUP
    __device__ __forceinline__ void put_dry(int i, uint32_t w, int32_t sc, uint32_t col) const {
        set_word(i, (w & ~CW_VIS) | CW_DIRTY | (s_w[i] & CW_VIS));
        set_planes(i, sc, col);
    }
    __device__ __forceinline__ void set_nothing(int i) const { put_dry(i, mw[id_air], 0, 0); }
    // write the cell at s, of word v and (a SOUP cell) pending diff dfv, over d; the visited
    // mark stays with the position
    __device__ __forceinline__ void move(int d, int dg, int s, int sg, uint32_t v, int32_t dfv) const {
        set_word(d, (v & ~CW_VIS) | CW_DIRTY | (s_w[d] & CW_VIS));
        set_planes(d, s_sc[s], s_col[s]);
        if (cw_is(v, T_SOUP)) {
            df[dg] = dfv;
            if (TEMP && tp) tp[dg] = tp[sg];
        }
    }
    // the pending diff of the cell of word v at g, if it is SOUP (it comes from HBM: load it
    // well before its use)
    __device__ __forceinline__ int32_t df_if_soup(uint32_t v, int g) const { return cw_is(v, T_SOUP) ? df[g] : 0; }
    // Temperatures of SOUP cells live in HBM beside the diff; the tile's scalar is
    // their amount. They move only where a SOUP cell moves or is made, so the
    // rules touch them at those few places and nowhere else.
    __device__ __forceinline__ int16_t tp_load(int g) const { return (TEMP && tp) ? tp[g] : (int16_t)0; }
    __device__ __forceinline__ void tp_store(int g, int16_t v) const {
        if (TEMP && tp) tp[g] = v;
    }
    // put a tile just made by a factory (TilesCreate): a SOUP tile takes the
    // factory temperature, or `keep` (a reaction keeps the old temperature)
    __device__ __forceinline__ void put_new(int i, int g, const Cell &c, const MatTable *mt, bool keep = false,
                                            int32_t keep_t = 0) const {
        put(i, g, c);
        if (TEMP && tp && cw_is(c.w, T_SOUP)) tp[g] = keep ? (int16_t)keep_t : (int16_t)__ldg(&mt->f_temp[cw_id(c.w)]);
    }
    // only a change marks the cell for write-back (settled sand clears an already
    // clear flag every pass); w: the cell's word
    __device__ __forceinline__ void set_moved_w(int i, uint32_t w, bool on) const {
        const uint32_t n = on ? w | CW_MOVED : w & ~CW_MOVED;
        if (n != w) set_word(i, n | CW_DIRTY);
    }
    // clear the moved flag of cell i if it is a liquid that has settled
    __device__ __forceinline__ void wake_soup(int i, uint32_t w) const {
        if ((w & (CW_TYPE | CW_MOVED)) == ((uint32_t)T_SOUP << MW_TYPE_SHIFT | CW_MOVED))
            set_word(i, (w & ~CW_MOVED) | CW_DIRTY);
    }
    __device__ __forceinline__ void set_moved(int i, bool on) const { set_moved_w(i, s_w[i], on); }
    // f32 worlds: fluidAmountDiff += v as the reference's float add. No other cell of
    // the sub-phase (or wavefront step) touches this diff, and the ones that touched
    // it before did so in the reference's order, so a plain read-modify-write adds in
    // that order.
    __device__ __forceinline__ void add_diff_f(int g, float v) const {
        df[g] = __float_as_int(__fadd_rn(__int_as_float(df[g]), v));
    }
    __device__ __forceinline__ void setvis(int i) const { set_word(i, s_w[i] | CW_VIS); }
};

// ------------------------------------------------------------- rule context
struct Ctx {
    uint32_t pk, ck, k;
    int kx, ky;   // the active cell, whose key ck is derived on the first draw
    bool have_ck;
    int iter;
    int id_fire, id_water, id_lava, id_steam, id_obsidian, has_inter;
    bool f32;  // f32 liquid amounts: the ledger keeps no fluid rows (a compile-time constant)
    const MatTable *mt;
    int32_t *led_s;        // shared ledger [LED_TICK][64] of the chunk-pass
    long long *led_g;      // global ledger [LED_ROWS][MAXMAT]
    const uint32_t *mw;    // material words (shared)
    const uint16_t *fr;    // slipperiness | stability << 8 (shared)
    const uint2 *fric;     // by drop over stability (at most 11): 1000 / d, 2^32 / that (shared)
    // the cell's spawn event: its particles' kind (1 sand, 2 soup, 3 fire), id and flags as
    // in their records, colour, scalar, temperature, and the velocity of the first
    int ev_kind;
    uint32_t ev_idfl, ev_col;
    int32_t ev_sc;
    float ev_vx, ev_vy;
    int16_t ev_tp;
    int ev_n;  // particles the cell emits (0: none)
    // the pending diff that a liquid in free fall loses: counted when its particles are
    // emitted, so that the rule does not wait for the load
    int32_t ev_df;
    // start the draws of the cell at (x, y); most cells never draw, so the key
    // (two hash rounds) is computed only when the first draw needs it
    __device__ __forceinline__ void at(int x, int y) {
        kx = x;
        ky = y;
        have_ck = false;
        k = 0;
    }
    __device__ __forceinline__ uint32_t key() {
        if (!have_ck) {
            ck = cell_key(pk, (uint32_t)kx, (uint32_t)ky);
            have_ck = true;
        }
        return ck;
    }
    __device__ __forceinline__ uint32_t D() { return draw_k(key(), k++); }
};

// Ledger counts of one chunk-pass are 32-bit shared counters (native shared atomics;
// 64-bit ones are compare-and-swap loops), added to the world's 64-bit ledger when the
// chunk-pass ends. A counter takes amounts below LED_SMALL only, larger ones go to the
// world's ledger at once, so that a chunk-pass cannot overflow it: a cell's turns make at
// most LED_ENTRIES entries in a row. In sweep A a sand's interactions make the most, at most
// 4 of a pair (fse_material_set_interaction) with boxes of at most 25 cells each (a visited
// box has no negative corner and reaches 5 cells at the farthest); fire converts at most 27
// cells, water on lava 11, a reaction 4, a flow makes 4 new cells; sweeps B and C convert
// the cell itself.
constexpr int LED_SMALL = 1024, LED_ENTRIES = 128;
static_assert(4 * 25 + 2 <= LED_ENTRIES && 27 + 2 <= LED_ENTRIES, "entries of a cell");
static_assert((long long)LED_ENTRIES * 128 * 128 * (LED_SMALL - 1) <= INT32_MAX, "a counter holds a chunk-pass");
constexpr int LED_TICK = 4;  // the rows the cell update counts in: all but LED_XN and LED_XF
__host__ __device__ constexpr int led_slot(int row) { return row > LED_XN ? row - 1 : row; }
__device__ __forceinline__ void led_add(Ctx &c, int row, uint32_t w, int32_t v) {
    if (v == 0 || cw_air(w)) return;
    const int mat = cw_id(w);
    if (mat < 64 && v > -LED_SMALL && v < LED_SMALL)
        atomicAdd(&c.led_s[led_slot(row) * 64 + mat], v);
    else
        atomicAdd((unsigned long long *)&c.led_g[row * MAXMAT + mat], (unsigned long long)(long long)v);
}
__device__ __forceinline__ void led_add64(Ctx &c, int row, uint32_t w, long long v) {
    if (v > -LED_SMALL && v < LED_SMALL)
        led_add(c, row, w, (int32_t)v);
    else if (!cw_air(w))
        atomicAdd((unsigned long long *)&c.led_g[row * MAXMAT + cw_id(w)], (unsigned long long)v);
}
// a conversion (not a move) of the content old -> nw
__device__ __forceinline__ void led_swap(Ctx &c, uint32_t old_w, long long old_fluid, uint32_t new_w,
                                         long long new_fluid) {
    led_add(c, LED_DN, old_w, 1);
    if (!c.f32 && cw_is(old_w, T_SOUP)) led_add64(c, LED_DF, old_w, old_fluid);
    led_add(c, LED_CN, new_w, 1);
    if (!c.f32 && cw_is(new_w, T_SOUP)) led_add64(c, LED_CF, new_w, new_fluid);
}
// conversion of whatever is at cell i into nw
template <class TL>
__device__ __forceinline__ void led_replace_at(const TL &T, Ctx &c, int i, int g, const Cell &nw) {
    const uint32_t o = T.at(i);
    const long long of = (!c.f32 && cw_is(o, T_SOUP)) ? (long long)T.s_sc[i] + T.df_of(i, g) : 0;
    led_swap(c, o, of, nw.w, (long long)nw.sc + nw.df);
}

// TilesCreate(id, x, y), game_datastruct.cpp:494-574
__device__ __forceinline__ Cell create_tile(Ctx &c, int mid) {
    Cell t;
    t.w = c.mw[mid];
    t.df = 0;
    t.sc = soup_scalar(c.mt, mid, c.f32);  // a temperature, or a SOUP tile's amount
    t.col = __ldg(&c.mt->f_base[mid]);
    uint32_t fp = __ldg(&c.mt->f_pack[mid]);
    int mod = (int)(fp >> 20);
    if (mod > 0) {
        int shift = (int)(fp & 0xFF), lo = (int)((fp >> 8) & 0xFFF);
        t.col = t.col + ((uint32_t)(lo + (int)(c.D() % (uint32_t)mod)) << shift);
    }
    return t;
}

// CalculateVerticalFlowValue, world.cpp:1021-1034, Q16.16
// rem > 0. The sum in 32 bits: unsigned it is exact for dst >= 0, and for dst < 0 it is
// a signed number below 2^31.
__device__ __forceinline__ int32_t vflow(int32_t rem, int32_t dst) {
    const uint32_t sum = (uint32_t)rem + (uint32_t)dst;
    if (sum <= (uint32_t)Q_MAXV || (dst < 0 && (int32_t)sum < 0)) return Q_MAXV;
    // MAXV^2 + sum * MAXCOMP < 2^31 below the bound; MAXCOMP is even above it
    if (sum < (uint32_t)(2 * Q_MAXV + Q_MAXCOMP))
        return (int32_t)(((uint32_t)Q_MAXV * Q_MAXV + sum * Q_MAXCOMP) / (uint32_t)(Q_MAXV + Q_MAXCOMP));
    return (int32_t)((sum >> 1) + Q_MAXCOMP / 2);
}
__device__ __forceinline__ int32_t clampflow(int32_t flow, int32_t rem) {
    return min(max(flow, 0), min(rem, Q_MAXFLOW));  // rem > 0
}

// CalculateVerticalFlowValue, world.cpp:1021-1034, in the reference's f32: every
// operation separately rounded as the reference's x86-64 build does (no contraction)
__device__ __forceinline__ float vflow_f(float rem, float dst) {
    const float sum = __fadd_rn(rem, dst);
    if (sum <= F_MAXV) return F_MAXV;
    if (sum < __fadd_rn(2.0f * F_MAXV, F_MAXCOMP))
        return __fdiv_rn(__fadd_rn(F_MAXV * F_MAXV, __fmul_rn(sum, F_MAXCOMP)), __fadd_rn(F_MAXV, F_MAXCOMP));
    return __fdiv_rn(__fadd_rn(sum, F_MAXCOMP), 2.0f);
}
// flow = std::max(flow, 0.0f); if (flow > std::min(FLUID_MaxFlow, rem)) flow = ...
// (world.cpp:1320-1321 and its three copies), with std::max/min's own comparisons;
// the FLUID_FlowSpeed factor of 1.0f before it changes no float and is left out
__device__ __forceinline__ float clampflow_f(float flow, float rem) {
    if (flow < 0.0f) flow = 0.0f;
    const float lim = (rem < F_MAXFLOW) ? rem : F_MAXFLOW;
    return (flow > lim) ? lim : flow;
}

// the world of the CTA's current chunk
__shared__ WorldDev s_w;

// a liquid cell's flow in a rendering world, added to the flow of its cell (flowX -= /
// += flow for left / right, flowY += / -= for down / up, world.cpp:1334,1374,1402,1432):
// a reduction no other cell of the sub-phase makes
__device__ __forceinline__ void render_flow(int32_t *fw, int g, int axis, int32_t v) {
    atomicAdd(&fw[2 * (size_t)g + axis], v);
}
__device__ __forceinline__ void render_flow_f(int32_t *fw, int g, int axis, float v, bool add) {
    float *q = reinterpret_cast<float *>(fw) + 2 * (size_t)g + axis;
    *q = add ? __fadd_rn(*q, v) : __fsub_rn(*q, v);
}

// the cell a liquid `w0` of colour `col` makes where it flows into the AIR cell n
// (word wn): MaterialInstance(tile.mat, tile.color, tile.temperature) with amount 0 and
// the flow as its pending diff
template <class TL>
__device__ __forceinline__ void flow_into_air(const TL &T, uint32_t w0, uint32_t col, int n, uint32_t wn, int gn,
                                              int32_t diff, int g) {
    T.set_word(n, (w0 & CW_MAT) | CW_DIRTY | (wn & CW_VIS));
    T.set_planes(n, 0, col);
    T.df[gn] = diff;
    T.tp_store(gn, T.tp_load(g));
}

// the active liquid trades places with its liquid neighbour n (world.cpp:1341-1350,
// 1439-1448), carrying its whole pending diff
template <class TL>
__device__ __forceinline__ void swap_liquid(const TL &T, uint32_t w0, int32_t sc, uint32_t col, int32_t diff, int i,
                                            int g, int n, int gn) {
    const int16_t tv = T.tp_load(g);
    T.move(i, g, n, gn, T.at(n), T.df_load(gn));
    Cell t;
    t.w = w0;
    t.sc = sc;
    t.col = col;
    t.df = diff;
    T.put(n, gn, t);
    T.tp_store(gn, tv);
}

// WATER on LAVA, world.cpp:1519-1537; old_fluid: the water's amount and diff
template <class TL>
__device__ __forceinline__ void water_on_lava(const TL &T, Ctx &c, uint32_t w0, long long old_fluid, int i, int g) {
    const MatTable *mt = c.mt;
    Cell st = create_tile(c, c.id_steam);
    led_swap(c, w0, old_fluid, st.w, c.f32 ? 0 : (long long)st.sc);
    T.put_new(i, g, st, mt);
    const int n = i + T.RW, gn = g + T.W;
    Cell ob = create_tile(c, c.id_obsidian);
    led_replace_at(T, c, n, gn, ob);
    T.put_new(n, gn, ob, mt);
    T.setvis(n);
    for (int xx = -1; xx <= 1; xx++)
        for (int yy = 0; yy <= 2; yy++) {
            const int m = i + yy * T.RW + xx, gm = g + yy * T.W + xx;
            if (cw_id(T.at(m)) == c.id_lava) {
                Cell o2 = create_tile(c, c.id_obsidian);
                led_replace_at(T, c, m, gm, o2);
                T.put_new(m, gm, o2, mt);
                T.setvis(m);
            }
        }
}

// velocities of spawned particles by their draws, as the reference's divisions give them
// (world.cpp:1222,1298; divided once per CTA, as a division is a dozen instructions)
struct SpawnVel {
    float sand_vx[10];  // (k - 5) / 20.0f
    float soup_vx[10];  // (k - 5) / 30.0f
    float sand_vy[2];   // -(k + 3) / 10.0f + 1.5f
    float soup_vy[2];   // -(k + 3) / 10.0f + 1.0f
};
__shared__ SpawnVel s_vel;
__device__ __forceinline__ void spawn_vel_init(int tid) {
    if (tid < 10) {
        s_vel.sand_vx[tid] = (float)(tid - 5) / 20.0f;
        s_vel.soup_vx[tid] = (float)(tid - 5) / 30.0f;
    }
    if (tid < 2) {
        s_vel.sand_vy[tid] = (float)(-(tid + 3)) / 10.0f + 1.5f;
        s_vel.soup_vy[tid] = (float)(-(tid + 3)) / 10.0f + 1.0f;
    }
}

__device__ __forceinline__ void spawn_one(Ctx &c, int kind, uint32_t w, int32_t sc, uint32_t col, float vx, float vy) {
    c.ev_n = 1;
    c.ev_kind = kind;
    c.ev_idfl = (w & CW_ID) | ((w & (CW_FLAGS & ~CW_VIS)) << 8);
    c.ev_col = col;
    c.ev_sc = sc;
    c.ev_vx = vx;
    c.ev_vy = vy;
}

// a liquid cell in free fall becomes n particles (world.cpp:1283-1305)
template <class TL>
__device__ __forceinline__ void free_fall(const TL &T, Ctx &c, uint32_t w0, int32_t sc, uint32_t col, int n, int i,
                                          int g, int x, int y) {
    T.set_nothing(i);
    if (n < 1) n = 1;
    led_add(c, LED_CN, w0, n - 1);
    c.ev_n = n;
    c.ev_kind = 2;
    c.ev_idfl = w0 & CW_ID;
    c.ev_col = col;
    c.ev_sc = sc;
    if (TL::kTemp) c.ev_tp = T.tp_load(g);
    // the cell's first draws (its other particles draw theirs when they are written)
    c.ev_vx = s_vel.soup_vx[draw_k(c.key(), 0u) % 10];
    c.ev_vy = s_vel.soup_vy[draw_k(c.key(), 1u) % 2];
    c.k += 2 * n;
}

// settle counts and the moved flags around a liquid that has had its turn
// (world.cpp:1472-1483): unchanged amounts count, flows wake the liquid neighbours
__device__ __forceinline__ uint32_t settle_word(uint32_t w0) {
    uint32_t s = w0 & CW_SETTLE;
    if (s < CW_SETTLE) s += 0x100u;
    uint32_t w = (w0 & ~CW_SETTLE) | s;
    if (s >= 10u << 8) w |= CW_MOVED;
    return w;
}

// ------------------------------------------------- sweep A, liquids
// world.cpp:1269-1567 but for the free fall (class_a finds the cells in free fall, and leaves
// out those that have settled). The neighbours are read first, all together (nothing the cell
// writes before it reads them is among them: a flow writes only the cell it enters).
// Q16.16 amounts, or with F32 the reference's own float amounts: the same branches
// in f32 with every operation rounded on its own, and the cell's fluidAmountDiff read
// when its turn begins (it already holds the flows of the cells updated before it) and
// written back with its own flows subtracted in order, as the reference's copy of the
// tile does.
//
// MIXED: the cell above or below may be another liquid, to trade places with or to react
// with (few are: class_a lists those with the other cells; the way through the trades,
// though no lane took it, made the rule of a single liquid a third slower).
template <bool MIXED, class TL>
__device__ __forceinline__ void rule_a_soup(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    const int32_t sc = T.s_sc[i];
    if (sc == 0) return;
    if (sc < Q_MINV) {
        led_add64(c, LED_DF, w0, sc);
        T.set_word(i, w0 | CW_DIRTY);
        T.set_sc(i, 0);
        return;
    }
    const int RW = T.RW;
    const uint32_t col = T.s_col[i];
    const uint32_t wb = T.at(i + RW);
    const bool airBelow = cw_air(wb);
    const int g = T.gi(x, y);
    const uint32_t wl = T.at(i - 1), wr = T.at(i + 1), wt = T.at(i - RW);
    const int32_t sb = T.s_sc[i + RW], sl = T.s_sc[i - 1], sr = T.s_sc[i + 1], su = T.s_sc[i - RW];
    int32_t rem = sc, down = 0, left = 0, right = 0, up = 0;
    bool gone = false;
    if ((airBelow && c.iter <= 2) || cw_same(wb, w0)) {
        const int32_t dst = airBelow ? 0 : sb;
        down = clampflow(vflow(sc, dst) - dst, sc);
        rem -= down;
    } else if (MIXED && c.iter == 0 && cw_is(wb, T_SOUP)) {
        if (c.D() % 10 == 0) {
            swap_liquid(T, w0, sc, col, T.df_load(g), i, g, i + RW, g + T.W);
            return;
        }
    }
    const bool canL = (cw_air(wl) || cw_same(wl, w0)) && !airBelow;
    const bool canR = (cw_air(wr) || cw_same(wr, w0)) && !airBelow;
    gone = rem < Q_MINV;
    if (!gone && canL) {
        const int32_t d = rem - (cw_air(wl) ? 0 : sl);
        left = clampflow(canR ? d / 3 : d / 2, rem);
        rem -= left;
        gone = rem < Q_MINV;
    }
    if (!gone && canR) {
        const int32_t d = rem - (cw_air(wr) ? 0 : sr);
        right = clampflow(d / 2, rem);
        rem -= right;
        gone = rem < Q_MINV;
    }
    bool swap_up = false;
    if (!gone) {
        if (cw_air(wt) || cw_same(wt, w0)) {
            const int32_t dst = cw_air(wt) ? 0 : su;
            up = clampflow(rem - vflow(rem, dst), rem);
            rem -= up;
            gone = rem < Q_MINV;
        } else if (MIXED && c.iter == 0 && cw_is(wt, T_SOUP)) {
            swap_up = c.D() % 10 == 0;
        }
    }
    int32_t *pd = T.df + g;
    if (int32_t *fw = s_w.flow) {
        if (down != 0) render_flow(fw, g, 1, down);
        if (left != 0) render_flow(fw, g, 0, -left);
        if (right != 0) render_flow(fw, g, 0, right);
        if (up != 0) render_flow(fw, g, 1, -up);
    }
    // the flows: pending diffs (reductions, nothing waits for them), and where they enter
    // AIR new cells, which few of a liquid's flows do
    const bool mb = down != 0 && airBelow, ml = left != 0 && cw_air(wl), mr = right != 0 && cw_air(wr);
    const bool mu = up != 0 && cw_air(wt);
    if (down != 0 && !airBelow) atomicAdd(pd + T.W, down);
    if (left != 0 && !ml) atomicAdd(pd - 1, left);
    if (right != 0 && !mr) atomicAdd(pd + 1, right);
    if (up != 0 && !mu) atomicAdd(pd - T.W, up);
    if (mb || ml || mr || mu) {
        if (mb) flow_into_air(T, w0, col, i + RW, wb, g + T.W, down, g);
        if (ml) flow_into_air(T, w0, col, i - 1, wl, g - 1, left, g);
        if (mr) flow_into_air(T, w0, col, i + 1, wr, g + 1, right, g);
        if (mu) flow_into_air(T, w0, col, i - RW, wt, g - T.W, up, g);
        led_add(c, LED_CN, w0, (int)mb + (int)ml + (int)mr + (int)mu);
    }
    const int32_t dd = rem - sc;  // the change of its own pending diff
    if (swap_up) {
        swap_liquid(T, w0, sc, col, dd + T.df_load(g), i, g, i - RW, g - T.W);
        return;
    }
    if (gone) {  // the remainder evaporates
        led_add64(c, LED_DF, w0, rem);
        T.set_word(i, w0 | CW_DIRTY);
        atomicAdd(pd, -sc);
        return;
    }
    uint32_t wn = w0;
    if (dd == 0) {
        wn = settle_word(w0);
    } else {
        T.wake_soup(i - RW, wt);
        T.wake_soup(i + RW, wb);
        T.wake_soup(i - 1, wl);
        T.wake_soup(i + 1, wr);
        atomicAdd(pd, dd);
    }
    T.set_word(i, wn | CW_DIRTY);
    if (MIXED && cw_id(w0) == c.id_water && cw_id(wb) == c.id_lava)
        water_on_lava(T, c, wn, (long long)sc + T.df_load(g), i, g);
}

template <bool MIXED, class TL>
__device__ __forceinline__ void rule_a_soup_f32(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    const int32_t sc = T.s_sc[i];
    const float amount = __int_as_float(sc);
    if (amount == 0.0f) return;
    if (amount < F_MINV) {
        T.set_word(i, w0 | CW_DIRTY);  // the diff stays as it is
        T.set_sc(i, __float_as_int(0.0f));
        return;
    }
    const int RW = T.RW;
    const uint32_t col = T.s_col[i];
    const uint32_t wb = T.at(i + RW);
    const bool airBelow = cw_air(wb);
    const int g = T.gi(x, y);
    float dfv = __int_as_float(T.df_load(g));
    const uint32_t wl = T.at(i - 1), wr = T.at(i + 1), wt = T.at(i - RW);
    const float sb = __int_as_float(T.s_sc[i + RW]), sl = __int_as_float(T.s_sc[i - 1]);
    const float sr = __int_as_float(T.s_sc[i + 1]), su = __int_as_float(T.s_sc[i - RW]);
    const float start = amount;
    float rem = amount;
    int made = 0;
    int32_t *fw = s_w.flow;
    // one flow (world.cpp:1309-1460) into neighbour n
    auto flow_to = [&](float flow, int n, uint32_t wn, int gn, int axis, bool add) {
        if (flow == 0.0f) return;
        if (fw) render_flow_f(fw, g, axis, flow, add);
        rem = __fsub_rn(rem, flow);
        dfv = __fsub_rn(dfv, flow);
        if (cw_air(wn)) {
            // fluidAmount 0, then fluidAmountDiff (0) += flow
            flow_into_air(T, w0, col, n, wn, gn, __float_as_int(__fadd_rn(0.0f, flow)), g);
            made++;
        } else {
            T.add_diff_f(gn, flow);
        }
    };
    bool done = false;  // the remainder evaporates
    if ((airBelow && c.iter <= 2) || cw_same(wb, w0)) {
        const float dst = airBelow ? 0.0f : sb;
        flow_to(clampflow_f(__fsub_rn(vflow_f(start, dst), dst), start), i + RW, wb, g + T.W, 1, true);
    } else if (MIXED && c.iter == 0 && cw_is(wb, T_SOUP)) {
        if (c.D() % 10 == 0) {  // the cell leaves its position with its diff
            swap_liquid(T, w0, sc, col, __float_as_int(dfv), i, g, i + RW, g + T.W);
            return;
        }
    }
    const bool canL = (cw_air(wl) || cw_same(wl, w0)) && !airBelow;
    const bool canR = (cw_air(wr) || cw_same(wr, w0)) && !airBelow;
    done = rem < F_MINV;
    if (!done && canL) {
        const float dst = cw_air(wl) ? 0.0f : sl;
        flow_to(clampflow_f(__fdiv_rn(__fsub_rn(rem, dst), canR ? 3.0f : 2.0f), rem), i - 1, wl, g - 1, 0, false);
        done = rem < F_MINV;
    }
    if (!done && canR) {
        const float dst = cw_air(wr) ? 0.0f : sr;
        flow_to(clampflow_f(__fdiv_rn(__fsub_rn(rem, dst), 2.0f), rem), i + 1, wr, g + 1, 0, true);
        done = rem < F_MINV;
    }
    bool swap_up = false;
    if (!done) {
        if (cw_air(wt) || cw_same(wt, w0)) {
            const float dst = cw_air(wt) ? 0.0f : su;
            flow_to(clampflow_f(__fsub_rn(rem, vflow_f(rem, dst)), rem), i - RW, wt, g - T.W, 1, false);
            done = rem < F_MINV;
        } else if (MIXED && c.iter == 0 && cw_is(wt, T_SOUP)) {
            swap_up = c.D() % 10 == 0;
        }
    }
    led_add(c, LED_CN, w0, made);
    if (swap_up) {
        swap_liquid(T, w0, sc, col, __float_as_int(dfv), i, g, i - RW, g - T.W);
        return;
    }
    uint32_t wn = w0;
    if (done) {
        dfv = __fsub_rn(dfv, rem);
    } else if (start == rem) {
        wn = settle_word(w0);
    } else {
        T.wake_soup(i - RW, wt);
        T.wake_soup(i + RW, wb);
        T.wake_soup(i - 1, wl);
        T.wake_soup(i + 1, wr);
    }
    T.set_word(i, wn | CW_DIRTY);
    T.df[g] = __float_as_int(dfv);
    if (MIXED && !done && cw_id(w0) == c.id_water && cw_id(wb) == c.id_lava) water_on_lava(T, c, wn, 0, i, g);
}

// fire, world.cpp:1101-1146. Returns false where the cell burnt out (the sweep goes on
// to its material's own rule either way, which for FIRE is none)
template <class TL>
__device__ __forceinline__ void rule_a_fire(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    const MatTable *mt = c.mt;
    const int g = T.gi(x, y);
    const int32_t sc = T.s_sc[i];
    uint32_t col = T.s_col[i];
    if (c.D() % 10 == 0) col = (255u << 16) | ((uint32_t)(100 + (int)(c.D() % 50)) << 8) | 50u;
    if (c.D() % 10 == 0) {
        float vx = (float)((int)(c.D() % 10) - 5) / 20.0f;
        float vy = -((float)(int)(c.D() % 10) / 10.0f) / 3.0f + -0.5f;
        spawn_one(c, 3, w0, sc, col, vx, vy);
        led_add(c, LED_CN, w0, 1);
    }
    if (c.D() % 150 == 0) {
        led_swap(c, w0, (long long)sc, T.mw[T.id_air], 0);
        T.set_nothing(i);
        T.setvis(i);
    } else {
        bool found = false;
        for (int xx = -2; xx <= 2; xx++)
            for (int yy = -2; yy <= 2; yy++) {
                const int n = i + yy * T.RW + xx;
                if (cw_is(T.at(n), T_SOLID)) {
                    found = true;
                    if (c.D() % 500 == 0) {
                        Cell f = create_tile(c, c.id_fire);
                        if (T.in_world(x + xx, y + yy)) {
                            const int gn = g + yy * T.W + xx;
                            led_replace_at(T, c, n, gn, f);
                            T.put_new(n, gn, f, mt);
                            T.setvis(n);
                        }
                    }
                }
            }
        if (!found && c.D() % 120 == 0) {
            led_swap(c, w0, (long long)sc, T.mw[T.id_air], 0);
            T.set_nothing(i);
            T.setvis(i);
        }
    }
}

// interactions of sand with the cell below it, world.cpp:1153-1179: true where the
// pair of materials has any (the sand's turn then ends)
template <class TL>
__device__ __forceinline__ bool rule_a_inter(const TL &T, Ctx &c, uint32_t w0, int bid, int i, int x, int y) {
    const MatTable *mt = c.mt;
    const int sid = cw_id(w0), g = T.gi(x, y);
    int hit = -1;
    for (int k = 0; k < mt->n_inter; k++)
        if (mt->inter[k][0] == sid && mt->inter[k][1] == bid) hit = k;
    if (hit < 0) return false;
    for (int k = 0; k < mt->n_inter; k++) {
        if (mt->inter[k][0] != sid || mt->inter[k][1] != bid) continue;
        int kind = mt->inter[k][2], d1 = mt->inter[k][3], d2 = mt->inter[k][4];
        int ox = mt->inter[k][5], oy = mt->inter[k][6];
        // the radius is a u32 in the reference, so its loops compare
        // unsigned: a box whose low corner is negative is not visited
        if (ox - d2 < 0 || oy - d2 < 0) continue;
        for (int xx = ox - d2; xx <= ox + d2; xx++)
            for (int yy = oy - d2; yy <= oy + d2; yy++) {
                const int n = i + yy * T.RW + xx;
                const int nid = cw_id(T.at(n));
                bool doit = (kind == INTER_TRANSFORM) ? (nid == bid) : ((xx == 0 && yy == 0) || nid == T.id_air);
                if (doit) {
                    Cell nt = create_tile(c, d1);
                    if (T.in_world(x + xx, y + yy)) {
                        const int gn = g + yy * T.W + xx;
                        led_replace_at(T, c, n, gn, nt);
                        T.put_new(n, gn, nt, mt);
                        T.setvis(n);
                    }
                }
            }
    }
    return true;
}

// temperature reactions of a SAND cell, world.cpp:1181-1204: true where one happened
template <class TL>
__device__ __forceinline__ bool rule_a_react(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    const MatTable *mt = c.mt;
    const int sid = cw_id(w0), g = T.gi(x, y);
    const int32_t sc = T.s_sc[i];
    const int nr = mt->n_react[sid];
    bool react = false;
    for (int k = 0; k < nr; k++) {
        int kind = mt->react[sid][k][0], temp = mt->react[sid][k][1], res = mt->react[sid][k][2];
        bool hit = (kind == REACT_BELOW) ? (sc < temp) : (sc > temp);
        if (hit) {
            Cell nt = create_tile(c, res);
            // the temperature is kept (world.cpp:1188,1196): in the scalar,
            // or beside the amount of a SOUP result
            if (!cw_is(nt.w, T_SOUP)) nt.sc = sc;
            led_replace_at(T, c, i, g, nt);
            T.put_new(i, g, nt, mt, true, sc);
            T.setvis(i);
            react = true;
        }
    }
    return react;
}

// ----------------------------------------------------------------- sweep A
// a liquid of amount sc with four AIR cells below (world.cpp:1283-1284)
template <class TL>
__device__ __forceinline__ bool soup_falls(const TL &T, int i, int32_t sc) {
    bool enough;
    if constexpr (TL::kF32)
        enough = (double)__int_as_float(sc) > 0.005;  // in double: 0.005 is a double literal
    else
        enough = sc > Q_FREEFALL;
    return enough && cw_air(T.at(i + T.RW) | T.at(i + 2 * T.RW) | T.at(i + 3 * T.RW) | T.at(i + 4 * T.RW));
}

// Whether sweep A may change cell i (a superset of the cells that its rule changes):
// 0 no, 1 a liquid, 2 another cell, a liquid in free fall (world.cpp:1283-1305) or one with
// another liquid above or below, so that the warps of liquids that flow do not take the
// long ways through an emission or a trade of places. Cells whose material is not updated in this
// iteration are marked visited here (world.cpp:1093-1096).
template <class TL>
__device__ __forceinline__ int class_a(const TL &T, const Ctx &c, int i) {
    // what any class asks, in one round of loads
    const uint32_t w0 = T.at(i), wn = T.at(i + T.RW), wt = T.at(i - T.RW);
    const int32_t sc = T.s_sc[i];
    if (w0 & CW_VIS) return 0;
    if (!(w0 & CW_LIVE)) {
        T.set_word(i, w0 | CW_VIS);
        return 0;
    }
    if (cw_is(w0, T_SOUP)) {
        bool none, small;
        if constexpr (TL::kF32) {
            const float amount = __int_as_float(sc);
            none = amount == 0.0f;
            small = amount < F_MINV;
        } else {
            none = sc == 0;
            small = sc < Q_MINV;
        }
        if (none) return 0;
        if (small) return 1;
        if (cw_air(wn) && soup_falls(T, i, sc)) return 2;
        if (w0 & CW_MOVED) return 0;  // a settled liquid only falls or dries up
        const bool mixed = (cw_is(wn, T_SOUP) && !cw_same(wn, w0)) || (cw_is(wt, T_SOUP) && !cw_same(wt, w0));
        return mixed ? 2 : 1;
    }
    bool act = (w0 & CW_FIRE) != 0;
    if (cw_is(w0, T_SAND)) act = c.has_inter || (w0 & CW_REACT) || wn < cw_sink(w0);
    if (cw_is(w0, T_GAS)) act = cw_air(wt);
    return act ? 2 : 0;
}

// the rules: c.ev_n = the particles the cell emits
template <bool MIXED, class TL>
__device__ __forceinline__ void rule_a_liquid(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    if constexpr (TL::kF32)
        rule_a_soup_f32<MIXED>(T, c, w0, i, x, y);
    else
        rule_a_soup<MIXED>(T, c, w0, i, x, y);
}
// a cell of class 2, of word w0
template <class TL>
__device__ __forceinline__ void rule_a(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    if (w0 & CW_FIRE) rule_a_fire(T, c, w0, i, x, y);
    if (cw_is(w0, T_SAND)) {
        const uint32_t wb = T.at(i + T.RW);  // world.cpp:1150
        const uint32_t lim = cw_sink(w0);
        if (c.has_inter && rule_a_inter(T, c, w0, cw_id(wb), i, x, y)) return;
        if ((w0 & CW_REACT) && rule_a_react(T, c, w0, i, x, y)) return;
        // world.cpp:1206-1267
        if (!(wb < lim)) return;
        c.key();  // it will draw: the hashes run while the loads are under way
        const int g = T.gi(x, y);
        const int32_t dfb = T.df_if_soup(wb, g + T.W);
        const bool canL = T.at(i + T.RW - 1) < lim, canR = T.at(i + T.RW + 1) < lim;
        if (!((canL || canR) && c.D() % 20 == 0)) {
            const int n = i + T.RW;
            const int32_t sc = T.s_sc[i];
            const uint32_t col = T.s_col[i];
            bool falls = cw_air(wb);
            if (falls) {
                const uint32_t w2 = T.at(i + 2 * T.RW), w3 = T.at(i + 3 * T.RW), w4 = T.at(i + 4 * T.RW);
                falls = cw_air(w2) && cw_air(w3) && cw_air(w4);
            }
            T.move(i, g, n, g + T.W, wb, dfb);
            if (falls) {
                const float vx = s_vel.sand_vx[c.D() % 10];
                const float vy = s_vel.sand_vy[c.D() % 2];
                spawn_one(c, 1, w0, sc, col, vx, vy);
            } else {
                const uint32_t t = c.D() % 2 == 0 ? w0 | CW_MOVED : w0;
                T.set_word(n, t | CW_DIRTY | CW_VIS);
                T.set_planes(n, sc, col);
            }
            if (c.D() % 2 == 0) {
                if (x > 0 && cw_is(T.at(n - 1), T_SAND)) {
                    if (c.D() % 2 == 0) T.set_moved(n - 1, true);
                }
                if (x < T.W - 1 && cw_is(T.at(n + 1), T_SAND)) {
                    if (c.D() % 2 == 0) T.set_moved(n + 1, true);
                }
            }
        }
    } else if (cw_is(w0, T_SOUP)) {
        const int32_t sc = T.s_sc[i];
        if (!soup_falls(T, i, sc)) {  // another liquid above or below
            rule_a_liquid<true>(T, c, w0, i, x, y);
            return;
        }
        const int g = T.gi(x, y);
        if constexpr (TL::kF32) {
            free_fall(T, c, w0, sc, T.s_col[i], (int)__fdiv_rn(__int_as_float(sc), 4.0f), i, g, x, y);  // int n = tile.fluidAmount / 4
        } else {
            c.ev_df = T.df_load(g);
            free_fall(T, c, w0, sc, T.s_col[i], sc >> 18, i, g, x, y);
        }
    } else if (cw_is(w0, T_GAS)) {  // world.cpp:1569-1585
        const int n = i - T.RW;
        const uint32_t above = T.at(n), aboveL = T.at(n - 1), aboveR = T.at(n + 1);
        if (cw_air(above) && !((cw_air(aboveL) || cw_air(aboveR)) && c.D() % 2 == 0)) {
            const int32_t sc = T.s_sc[i];
            const uint32_t col = T.s_col[i];
            // the AIR cell above and the gas trade places
            T.put_dry(i, above, T.s_sc[n], T.s_col[n]);
            T.set_word(n, w0 | CW_DIRTY | CW_VIS);
            T.set_planes(n, sc, col);
        }
    }
}

// ----------------------------------------------------------------- sweep B
// a liquid takes its pending diff, world.cpp:1728-1745. w0: the cell's word; dfv: its
// pending diff, read when the sub-phase began (no other cell of the sub-phase writes it)
template <class TL>
__device__ __forceinline__ void rule_b_soup(const TL &T, Ctx &c, uint32_t w0, int i, int g, int32_t dfv) {
    int32_t a;
    bool dry;
    if constexpr (TL::kF32) {
        const float f = __fadd_rn(__int_as_float(T.s_sc[i]), __int_as_float(dfv));
        a = __float_as_int(f);
        dry = f < F_MINV;
    } else {
        a = T.s_sc[i] + dfv;
        dry = a < Q_MINV;
    }
    if (dry) {
        led_add(c, LED_DN, w0, 1);
        if constexpr (!TL::kF32) led_add64(c, LED_DF, w0, a);
        T.set_word(i, T.mw[T.id_air] | CW_DIRTY | CW_VIS);
        T.set_planes(i, 0, 0);
    } else {
        T.set_word(i, w0 | CW_DIRTY | CW_VIS);
        T.set_sc(i, a);
        if (dfv != 0) T.df[g] = 0;
    }
}

// Whether sweep B may move cell i of word w0 (not SOUP; a superset). Sand that nothing
// beside it lets slide only clears its moved flag, which happens here: the friction
// draw of a stopped one could set the flag, but it is cleared again before the turn
// ends, and leaves only the mark that the cell was written, which rendering worlds
// (render: they count the written cells) keep exactly.
template <class TL>
__device__ __forceinline__ bool class_b(const TL &T, uint32_t w0, int i, bool render) {
    const bool sand = cw_is(w0, T_SAND);
    if (!sand && !cw_is(w0, T_GAS)) return false;
    const int n = sand ? i + T.RW : i - T.RW;
    const uint32_t lim = sand ? cw_sink(w0) : 1u << 24;  // gas rises into AIR
    const bool slides = T.at(n - 1) < lim || T.at(n + 1) < lim;
    if (sand && !slides && !render) T.set_moved_w(i, w0, false);
    return slides || (sand && render);
}

// w0: the cell's word (sand or gas)
template <class TL>
__device__ __forceinline__ void rule_b(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    if (cw_is(w0, T_SAND)) {  // world.cpp:1602-1727
        const int RW = T.RW;
        const uint32_t lim = cw_sink(w0);
        const uint32_t wl = T.at(i + RW - 1), wr = T.at(i + RW + 1);
        const bool canL = wl < lim, canR = wr < lim;
        const int g = T.gi(x, y);
        const int32_t dfl = canL ? T.df_if_soup(wl, g + T.W - 1) : 0, dfr = canR ? T.df_if_soup(wr, g + T.W + 1) : 0;
        bool stopped = !(w0 & CW_MOVED);
        c.at(x, y);
        c.key();  // it will draw: the hashes run while the loads are under way
        const int a = c.fr[cw_id(w0)];
        if (stopped) {
            // world.cpp:1619-1627 over the AIR snapshot taken when sweep B began
            const int drop = __popc(T.air10(i + RW - 1, x - 1, y + 1) | T.air10(i + RW + 1, x + 1, y + 1));
            int d = drop + 1 - (a >> 8);
            if (d > 0) {
                // chance = 1000 / d, 2 <= d <= 11 (1000 or more never): draw % chance == 0,
                // with the quotient by multiplication, which is at most one short
                if (d >= 2) {
                    const uint2 f = c.fric[d];
                    const uint32_t draw = c.D(), rest = draw - __umulhi(draw, f.y) * f.x;
                    if (rest == 0 || rest == f.x) {
                        stopped = false;
                        T.set_moved_w(i, w0, true);
                    }
                }
            }
        }
        if (stopped || !(canL || canR)) {
            T.set_moved(i, false);
            return;
        }
        // the moving cell as it was when its turn began
        uint32_t t = w0;
        const int32_t sc = T.s_sc[i];
        const uint32_t col = T.s_col[i];
        const int slip = a & 0xFF;
        const bool shouldMove = (slip > 0) ? (c.D() % (uint32_t)(2 * slip) != 0) : true;
        if (shouldMove && (canL || canR)) {
            if (c.D() % 2 == 0) {
                if (cw_is(T.at(i + RW), T_SAND)) {
                    if (c.D() % 2 == 0) T.set_moved(i + RW, true);
                }
            }
        }
        const bool goL = shouldMove && canL && (!canR || c.D() % 2 == 0);
        if (!goL && !(shouldMove && canR)) {
            T.set_moved(i, false);
            return;
        }
        const int o = goL ? -1 : 1;  // towards the left or the right
        const int s = i + o, d = i + RW + o, gd = g + T.W + o;
        const uint32_t wd = T.at(d);
        const int32_t dfd = goL ? dfl : dfr;
        if (T.air(s)) {
            T.move(s, g + o, d, gd, wd, dfd);
            if (goL) T.setvis(s);
            T.set_nothing(i);
        } else {
            T.move(i, g, d, gd, wd, dfd);
            T.setvis(i);
        }
        if (slip > 0 && c.D() % (uint32_t)(20 * slip) == 0) t &= ~CW_MOVED;
        T.set_word(d, t | CW_DIRTY | CW_VIS);
        T.set_planes(d, sc, col);
    } else if (cw_is(w0, T_GAS)) {  // world.cpp:1799-1818
        const int n = i - T.RW;
        const bool aboveL = T.air(n - 1), aboveR = T.air(n + 1);
        if (!aboveL && !aboveR) return;
        c.at(x, y);
        const int32_t sc = T.s_sc[i];
        const uint32_t col = T.s_col[i];
        const bool goL = aboveL && !(aboveR && c.D() % 2 == 0);
        if (!goL && !aboveR) return;
        const int d = goL ? n - 1 : n + 1;  // the AIR cell and the gas trade places
        T.put_dry(i, T.at(d), T.s_sc[d], T.s_col[d]);
        T.set_word(d, w0 | CW_DIRTY | CW_VIS);
        T.set_planes(d, sc, col);
    }
}

// ----------------------------------------------------------------- sweep C
// w0: the word of a GAS cell not yet visited
template <class TL>
__device__ __forceinline__ void rule_c(const TL &T, Ctx &c, uint32_t w0, int i, int x, int y) {
    // world.cpp:1862-1889
    const bool l = T.air(i - 1), r = T.air(i + 1), steam = cw_id(w0) == c.id_steam;
    if (!l && !r && !steam) return;
    c.at(x, y);
    const bool goL = l && !(r && c.D() % 2 == 0);
    if (goL || r) {
        const int d = goL ? i - 1 : i + 1;  // the AIR cell and the gas trade places
        const int32_t sc = T.s_sc[i];
        const uint32_t col = T.s_col[i];
        T.put_dry(i, T.at(d), T.s_sc[d], T.s_col[d]);
        T.set_word(d, w0 | CW_DIRTY | CW_VIS);
        T.set_planes(d, sc, col);
    } else if (steam) {
        if (c.D() % 10 == 0) {
            const int g = T.gi(x, y);
            Cell wt = create_tile(c, c.id_water);
            led_swap(c, w0, 0, wt.w, (long long)wt.sc);
            T.put_new(i, g, wt, c.mt);
        }
    }
}

// --------------------------------------------------------------- lattices
// (Px, Py) per sweep and chunk mode; see the oracle's lattice() for the derivation.
__device__ __forceinline__ void lattice(int sweep, int mode, int &px, int &py) {
    if (sweep == 0) {
        if (mode == 2) {
            px = 11;
            py = 11;
        } else if (mode == 1) {
            px = 5;
            py = 7;
        } else {
            px = 3;
            py = 6;
        }
    } else if (sweep == 1) {
        // the friction pillar reads the sweep-B snapshot, so only rows y-1..y+1 are live
        px = 3;
        py = 3;
    } else {
        px = 3;
        py = 1;
    }
}

// write the particles of the active cell's spawn event (world.cpp:1110-1119,1222,1298), three
// 16-byte stores each
static_assert(sizeof(SpawnRec) == 48, "three 16-byte stores");
template <bool TEMP, bool F32>
__device__ __forceinline__ void emit_spawns(const WorldDev &w, Ctx &c, uint32_t cp, uint32_t rank0, int base) {
    const int n = c.ev_n;
    int32_t amount = c.ev_sc, extra = 0;
    if (c.ev_kind == 2 && n > 1) {
        if (F32) {
            // f32 amt = tile.fluidAmount / n for every particle (world.cpp:1292)
            amount = __float_as_int(__fdiv_rn(__int_as_float(c.ev_sc), (float)n));
        } else {
            amount = c.ev_sc / n;
            extra = c.ev_sc % n;
        }
    }
    const uint32_t bits = c.ev_kind == 3 ? 2u << 24 : 0u;
    const uint32_t life = c.ev_kind == 3 ? 30u | 10u << 16 : 60u << 16;  // lifetime, fade
    const uint32_t temp = (TEMP && c.ev_kind == 2) ? (uint32_t)(uint16_t)c.ev_tp : 0u;
    const float x = (float)c.kx, y = (float)(c.ev_kind == 3 ? c.ky - 1 : c.ky + 1);
    float vx = c.ev_vx, vy = c.ev_vy;
#pragma unroll 1
    for (int i = 0; i < n; i++) {
        const int slot = base + i;
        if (slot >= w.stage_cap) {
            atomicOr(w.err, ERR_SPAWN_CAP);
            return;
        }
        if (i > 0) {
            vx = s_vel.soup_vx[draw_k(c.key(), 2u * (uint32_t)i) % 10];
            vy = s_vel.soup_vy[draw_k(c.key(), 2u * (uint32_t)i + 1u) % 2];
        }
        uint4 *r = reinterpret_cast<uint4 *>(&w.stage[slot]);
        r[0] = make_uint4(cp, rank0 + (uint32_t)i, __float_as_uint(x), __float_as_uint(y));
        r[1] = make_uint4(__float_as_uint(vx), __float_as_uint(vy), __float_as_uint(c.ev_kind == 3 ? 0.01f : 0.1f),
                          c.ev_col);
        r[2] = make_uint4((uint32_t)(amount + (i < extra ? 1 : 0)), c.ev_idfl | bits, life, temp);
    }
}

// -------------------------------------------------------------- the kernel
// shared memory besides the tile planes
template <int NT>
struct SmemHeadT {
    uint32_t mw[MAXMAT];  // material -> cell word of this iteration
    uint16_t fr[MAXMAT];  // slipperiness | stability << 8
    uint2 fric[12];       // d: 1000 / d and 2^32 / that
    int32_t led[LED_TICK * 64];   // the chunk-pass's ledger counts (led_slot)
    union {
        uint32_t vote[32];  // each warp's activity (bit 0) and fire (bit 1) votes of the chunk-pass
        int scan[32];       // in its sweeps: the warps' spawn totals of a sub-phase
    };
    // the pillar snapshot of sweep B (chunk edge <= 128)
    uint32_t air[(128 + 2) * 5];
    // the cells of a sub-phase that a rule may change (dx | dy << 8); after a sweep-A
    // sub-phase where a cell spawned several particles, the spawn counts, then ranks
    union {
        uint16_t list[2 * NT];
        uint32_t cnt[NT];
    };
    // which cells of a sweep-A sub-phase spawn, by enumeration index, in the same turn; and
    // the last sub-phase in which a cell spawned more than one particle
    uint32_t spawn_bits[3][NT / 32];
    int many;
    int running[2];  // spawns of the chunk-pass so far, in turn
    uint32_t n_list[3];  // lengths of the lists of this sub-phase and of the next two, in turn
    // CTA pair: what the partner wrote here: [0..1] its chunk flags, [2..3] its spawn
    // count of a sweep-A sub-phase (alternate slots)
    uint32_t xch[4];
};

// Dynamic shared memory of a CTA that updates `own` rows of a chunk of edge C: the
// head, up to 128 bytes of padding (the planes start on a 128-byte boundary of the
// window) and the planes of the largest tile
template <int NT>
constexpr size_t tile_smem(int C, int own, int halo, int width) {
    const size_t RW = (size_t)(width > C + HALO_LO + halo ? width : C + HALO_LO + halo);
    const size_t RHF = (size_t)own + HALO_LO + halo;
    const size_t RHI = (size_t)own + HALO_LO + 10;
    const size_t head = (sizeof(SmemHeadT<NT>) + 127) & ~(size_t)127;
    const size_t plane = (RW * RHF + 31) & ~(size_t)31;
    return 128 + head + (2 * plane + RW * RHI) * 4;
}
// The largest tile, a chunk of 128 with the 5-cell halo, beside the kernel's static
// variables (the world's descriptor, the spawn velocities, the mbarrier and the fused
// tick's words): a CTA takes at most 227 KB, and a launch that asks for more fails.
constexpr size_t COLOUR_STATIC = ((sizeof(WorldDev) + 15) & ~(size_t)15) + ((sizeof(SpawnVel) + 15) & ~(size_t)15) + 32;
static_assert(tile_smem<CP_THREADS>(128, 128, 5, 0) + COLOUR_STATIC <= 227 * 1024, "the 5-cell halo's tile");
static_assert(tile_smem<CP_THREADS>(128, 128, 2, tma_tile_width(128)) + COLOUR_STATIC <= 227 * 1024,
              "the tile of the tensor copies");

// items: (world << 20) | chunk slot within the colour; iter, tk select the pass.
// FUSED: every pass of the tick in one launch (iter, tk, items and n_items unused;
// ft holds the work). CTAs take chunk-passes in pass order from a ticket counter; a
// chunk-pass starts when the last earlier pass of each chunk of its 3 x 3
// neighbourhood is done (a chunk-pass reads and writes its chunk plus a halo of at
// most 5 cells, and each pass's chunks tile the zone, so these are all the
// chunk-passes it can conflict with, directly or through a chain), and publishes
// its own completion with a release store. A CTA only waits for tickets taken
// before its own by CTAs that are running, so the launch cannot deadlock whatever
// its grid; each wait is also bounded (ERR_TIMEOUT). The last CTA to finish clears
// the flags and the counters for the next launch.
// SEQ: the reference's own order inside each chunk (bottom row first, left to right,
// sweep by sweep; world.cpp:1084-1087, 1589, 1823), with the same rules, run as a
// wavefront of one thread per chunk row (see sweeps_seq)
// PAIR: each chunk is split over the two CTAs of a cluster, 512 threads each: rank 0
// updates the top half of its rows, rank 1 the bottom half, each staging its half
// plus the rows its rules reach (the shared rows are kept equal by mirrored writes)
// and writing back its own rows; sub-phases end with a cluster barrier. A chunk's
// sub-phases then run on two SMs.
// CC: the chunk edge where it is known when compiling (128, the reference's), else 0:
// the tile's rows, planes and lattices are then constants. Two CTAs of pairs share an SM up
// to edge 124, so they are held to 64 registers each; one of edge 128 takes 120 KB, an SM of
// its own and all the registers it asks for (4096 x 2048 step on pairs 3.02 -> 2.47 ms,
// 512 x 512 1.58 -> 1.33; at edge 64, where two fit, 4.0 ms against 5.0 with one)
template <int HALO, bool TEMP, bool SEQ, bool F32, bool PAIR = false, bool FUSED = false, int CC = 0>
__global__ void __launch_bounds__(PAIR ? CP_THREADS / 2 : CP_THREADS, PAIR && CC != 128 ? 2 : 1)
    k_colour_pass(const WorldDev *__restrict__ worlds, const uint32_t *__restrict__ items, int n_items, int iter_arg,
                  int tk_arg, const MatTable *__restrict__ mt, const FusedTick ft) {
    static_assert(!(PAIR && SEQ), "the reference order runs a chunk in one CTA");
    static_assert(!(FUSED && (PAIR || SEQ)), "the fused tick runs partitioned chunk-passes in one CTA each");
    constexpr int T = PAIR ? CP_THREADS / 2 : CP_THREADS;
    using Head = SmemHeadT<T>;
    extern __shared__ __align__(16) unsigned char smem[];
    Head &S = *reinterpret_cast<Head *>(smem);
    // the planes start on a 128-byte boundary of the shared window (TMA destinations)
    const uint32_t sbase = smem_addr(smem);
    unsigned char *planes = smem + (((sbase + (uint32_t)sizeof(Head) + 127u) & ~127u) - sbase);
    // TMA staging of the 4-byte planes: the partitioned order with a 2-cell halo, in
    // worlds with tensor maps (one phase of s_tma_bar per staged chunk-pass)
    constexpr bool kTma = HALO == 2 && !PAIR && !SEQ;
    __shared__ __align__(8) uint64_t s_tma_bar;
    uint32_t tma_phase = 0;

    const int tid = threadIdx.x;
    const int rank = PAIR ? (int)cluster_rank() : 0;
    int npass = 0;  // chunks taken so far (the same count in both CTAs of a pair)
    int mw_iter = -1;  // the iteration S.mw was built for
    if (tid >= 1 && tid < 12) S.fric[tid] = make_uint2(1000u / tid, 0xFFFFFFFFu / (1000u / tid));
    for (int i = tid; i < MAXMAT; i += T)
        S.fr[i] = (uint16_t)(i < mt->n ? mt_slip(mt->a[i]) | (mt_stab(mt->a[i]) << 8) : 0);
    for (int i = tid; i < LED_TICK * 64; i += T) S.led[i] = 0;
    if (tid < 3) S.n_list[tid] = 0;
    if (tid < T / 32)
        for (int k = 0; k < 3; k++) S.spawn_bits[k][tid] = 0;
    if (tid == 0) S.many = 0;
    int seq = 0;  // sub-phases of sweep A so far
    int nsub = 0;  // the list count of the next sub-phase of sweeps A and B
    Ctx c;
    spawn_vel_init(tid);
    c.iter = iter_arg;
    c.mt = mt;
    c.led_s = S.led;
    c.mw = S.mw;
    c.fr = S.fr;
    c.fric = S.fric;
    c.id_fire = mt->id_fire;
    c.id_water = mt->id_water;
    c.id_lava = mt->id_lava;
    c.id_steam = mt->id_steam;
    c.id_obsidian = mt->id_obsidian;
    // interactions exist exactly when the launch runs the 5-cell halo (tick_halo)
    c.has_inter = HALO == 5;
    c.f32 = F32;
    const int id_air = mt->id_air, id_solid = mt->id_solid;
    if (kTma && tid == 0) mbar_init(&s_tma_bar, 1);
    FSE_PT_DECL
    __syncthreads();

    int iter = iter_arg, tk = tk_arg;

    const int wstart = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
    const int wstride = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
    // FUSED: the ticket taken, and the completion flag this CTA publishes before it
    // takes the next one (kept in shared memory: the tile code needs the registers)
    __shared__ int s_ticket;
    __shared__ uint32_t *s_done_flag;
    __shared__ uint32_t s_done_value;
    if (FUSED && tid == 0) s_done_flag = nullptr;
    for (int it = wstart;; it += wstride) {
        uint32_t item;
        if constexpr (FUSED) {
            if (tid == 0) {
                if (s_done_flag) {
                    __threadfence();
                    st_release_gpu(s_done_flag, s_done_value);
                    s_done_flag = nullptr;
                }
                s_ticket = (int)atomicAdd(&worlds[0].sched[0], 1u);
            }
            __syncthreads();
            int t = s_ticket;
            const int per_iter = ft.n[0] + ft.n[1] + ft.n[2] + ft.n[3];
            if (t >= per_iter * (ft.passes / 4)) break;
            iter = t / per_iter;
            t -= iter * per_iter;
            // the colour and the index within it (no dynamic indexing of the parameters)
            const uint32_t *li = ft.items[0];
            tk = 0;
            if (t >= ft.n[0]) {
                t -= ft.n[0];
                tk = 1;
                li = ft.items[1];
                if (t >= ft.n[1]) {
                    t -= ft.n[1];
                    tk = 2;
                    li = ft.items[2];
                    if (t >= ft.n[2]) {
                        t -= ft.n[2];
                        tk = 3;
                        li = ft.items[3];
                    }
                }
            }
            item = __ldg(&li[t]);
        } else {
            if (it >= n_items) break;
            item = __ldg(&items[it]);
        }
        const int ox = tk % 2, oy = 1 - tk / 2;
        c.iter = iter;
        // the last chunk-pass's generic accesses to the planes come before this one's
        // tensor copies into them
        if constexpr (kTma) fence_proxy_async_smem();
        {
            // the world's descriptor into shared memory, 8 bytes a thread (one thread
            // copying it load by load took ~5% of a chunk-pass)
            static_assert(sizeof(WorldDev) % 8 == 0, "the descriptor is copied in 8-byte words");
            constexpr int NW8 = (int)(sizeof(WorldDev) / 8);
            static_assert(NW8 <= T, "one word per thread");
            if (tid < NW8)
                reinterpret_cast<uint2 *>(&s_w)[tid] =
                    __ldg(reinterpret_cast<const uint2 *>(&worlds[item >> 20]) + tid);
        }
        if (iter != mw_iter) {
            // the cell words of this iteration's materials
            mw_iter = iter;
            for (int i = tid; i < MAXMAT; i += T)
                S.mw[i] = i < mt->n ? mt->word[i] | (iter < mt_iter(mt->a[i]) ? CW_LIVE : 0u) : (uint32_t)i;
        }
        __syncthreads();
        FSE_PT(0)
        const WorldDev &w = s_w;
        const int slot = (int)(item & 0xFFFFF);
        if constexpr (FUSED) {
            // wait until the chunk-passes this one depends on are done: for each chunk
            // of the 3 x 3 neighbourhood, its last pass before this one
            const int nbq = (w.nCy - oy + 1) / 2;
            const int a = ox + 2 * (slot / nbq), b = oy + 2 * (slot % nbq);
            const int q = iter * 4 + tk;
            if (tid < 9) {
                const int a2 = a + tid % 3 - 1, b2 = b + tid / 3 - 1;
                if (a2 >= 0 && a2 < w.nCx && b2 >= 0 && b2 < w.nCy) {
                    const int tn = (a2 & 1) + 2 * (1 - (b2 & 1));
                    const int p = tn < tk ? iter * 4 + tn : (iter - 1) * 4 + tn;
                    if (p >= 0) {
                        const uint32_t *f = &w.cdone[(size_t)b2 * w.nCx + a2];
                        // sched[2]: a wait of this launch gave up; the others do not wait
                        volatile uint32_t *abort = &worlds[0].sched[2];
                        if (ld_acquire_gpu(f) <= (uint32_t)p && !*abort) {
                            const unsigned long long t0 = global_ns();
                            while (ld_acquire_gpu(f) <= (uint32_t)p && !*abort) {
                                if (global_ns() - t0 > FUSED_WAIT_NS) {
                                    atomicOr(w.err, ERR_TIMEOUT);
                                    *abort = 1u;
                                    break;
                                }
                                __nanosleep(64);
                            }
                        }
                    }
                }
            }
            if (tid == 0) {
                s_done_flag = &w.cdone[(size_t)b * w.nCx + a];
                s_done_value = (uint32_t)q + 1u;
            }
            __syncthreads();
        }
        if (iter >= w.cell_iter) {
            __syncthreads();
            continue;
        }
        const int C = CC ? CC : w.C, W = w.W, H = w.H;
        const int nb = (w.nCy - oy + 1) / 2;
        const int cx = w.zx + (ox + 2 * (slot / nb)) * C, cy = w.zy + (oy + 2 * (slot % nb)) * C;
        const uint32_t cp = (uint32_t)((iter * 4 + tk) * w.max_slots + slot);

        // the chunk rows this CTA updates, [o0, o1)
        const int half = C / 2;
        const int o0 = PAIR ? rank * half : 0, o1 = PAIR ? (rank ? C : half) : C;
        const int own = o1 - o0;
        TileData Tl;
        const bool tma = kTma && w.tmap != nullptr;
        // with TMA the rows start on a 16-byte boundary and are tma_tile_width wide
        Tl.RW = (CC && !PAIR) || tma ? tma_tile_width(C) : C + HALO_LO + HALO;
        Tl.RHF = own + HALO_LO + HALO;
        Tl.RHI = own + HALO_LO + 10;
        Tl.x0 = tma ? ((cx - HALO_LO) & ~3) : cx - HALO_LO;
        Tl.y0 = cy + o0 - HALO_LO;
        Tl.W = W;
        Tl.H = H;
        Tl.mw = S.mw;
        Tl.df = w.df;
        Tl.tp = w.tp;
        Tl.id_air = id_air;
        Tl.s_air = S.air;
        Tl.ax0 = cx - 1;
        Tl.ay0 = cy + o0 + 1;
        Tl.aw = C + 2;
        const int nfull = Tl.RW * Tl.RHF, plane = (nfull + 31) & ~31;  // 128-byte aligned planes
        Tl.s_sc = (int32_t *)planes;
        Tl.s_col = (uint32_t *)(Tl.s_sc + plane);
        Tl.s_w = Tl.s_col + plane;
        if constexpr (PAIR) {
            // the partner's planes lie at the same offsets of its shared memory
            const uint32_t pr = (uint32_t)(rank ^ 1);
            Tl.p_w = mapa_rank(smem_addr(Tl.s_w), pr);
            Tl.p_sc = mapa_rank(smem_addr(Tl.s_sc), pr);
            Tl.p_col = mapa_rank(smem_addr(Tl.s_col), pr);
            Tl.pd = (rank ? half : -half) * Tl.RW;
        }

        if (tid == 0) S.running[0] = 0;

        // ---- stage the tile, one warp per row. The 4-byte planes go straight to
        // shared memory, as two tensor copies (TMA) or with cp.async; ids and flags
        // are loaded a row at a time, all loads of a row in flight together. The
        // chunk's ids decide the skip and the lattice mode.
        if (tma && tid == 0) {
            const char *tm = static_cast<const char *>(w.tmap);
            // what the neighbours wrote (seen through their flags and the barrier above) comes
            // before these copies, which read it through the async proxy
            if constexpr (FUSED) fence_proxy_async_global();
            mbar_expect_tx(&s_tma_bar, 2u * (uint32_t)nfull * 4u);
            tma_load_2d(Tl.s_sc, tm, Tl.x0, Tl.y0, &s_tma_bar);
            tma_load_2d(Tl.s_col, tm + 128, Tl.x0, Tl.y0, &s_tma_bar);
        }
        int active = 0, fire = 0;
        if (tma) {
            // ids and flags four cells at a time: a group starts on a multiple of four cells, so
            // it lies wholly inside or outside a world that is a multiple of four cells wide.
            // All of a thread's loads are in flight together: one round trip to memory where
            // the row-by-row form below waits for five.
            constexpr int NG = 5;  // 140 rows of 34 groups over 1024 threads
            const int gpr = Tl.RW / 4, groups = gpr * Tl.RHI;
            const float rgpr = __frcp_rn((float)gpr);
            uint2 v[NG];
            uint32_t f[NG];
            int rows[NG];
#pragma unroll
            for (int k = 0; k < NG; k++) {
                const int e = tid + k * T;
                int r, q4;
                divmod_small(e, gpr, rgpr, r, q4);
                const int gx = Tl.x0 + 4 * q4, gy = Tl.y0 + r;
                rows[k] = r;
                const bool in = e < groups && (unsigned)gy < (unsigned)H && (unsigned)gx < (unsigned)W;
                const uint32_t so = (uint32_t)id_solid * 0x10001u;
                v[k] = make_uint2(so, so);
                f[k] = 0;
                if (in) {
                    const size_t gi = (size_t)gy * W + gx;
                    v[k] = *reinterpret_cast<const uint2 *>(&w.id[gi]);
                    if (r < Tl.RHF) f[k] = *reinterpret_cast<const uint32_t *>(&w.fl[gi]);
                }
            }
#pragma unroll
            for (int k = 0; k < NG; k++) {
                const int e = tid + k * T;
                if (e >= groups) break;
                const int q4 = e - rows[k] * gpr, gx = Tl.x0 + 4 * q4, gy = Tl.y0 + rows[k];
                const uint32_t fl = f[k] & ~((uint32_t)VISITED * 0x01010101u);
                uint4 o;
                o.x = S.mw[v[k].x & CW_ID] | ((fl & 0xFFu) << 8);
                o.y = S.mw[(v[k].x >> 16) & CW_ID] | (fl & 0xFF00u);
                o.z = S.mw[v[k].y & CW_ID] | ((fl >> 8) & 0xFF00u);
                o.w = S.mw[(v[k].y >> 16) & CW_ID] | ((fl >> 16) & 0xFF00u);
                *reinterpret_cast<uint4 *>(&Tl.s_w[4 * e]) = o;
                // the chunk's cells inside the world vote
                if (gy >= cy && gy < cy + C && gy < H && gx < W) {
                    const int l = cx - gx, u = cx + C - gx;  // cells l .. u - 1 of the group
                    uint32_t any = 0;
                    if (l <= 0 && u > 0) any |= o.x;
                    if (l <= 1 && u > 1) any |= o.y;
                    if (l <= 2 && u > 2) any |= o.z;
                    if (l <= 3 && u > 3) any |= o.w;
                    if (any & CW_LIVE) active = 1;
                    if (any & CW_FIRE) fire = 1;
                }
            }
        } else {
            const int lane = tid & 31, wid = tid >> 5;
            constexpr int NW = T / 32;
            for (int r = wid; r < Tl.RHI; r += NW) {
                const int gy = Tl.y0 + r;
                const bool rin = (unsigned)gy < (unsigned)H;
                const size_t gb = (size_t)gy * W;
                const bool full = r < Tl.RHF;
                uint16_t v[MAXRW / 32];
                uint8_t f[MAXRW / 32];
#pragma unroll
                for (int k = 0; k < MAXRW / 32; k++) {
                    const int lx = lane + 32 * k, gx = Tl.x0 + lx;
                    v[k] = (uint16_t)id_solid;
                    f[k] = 0;
                    if (lx < Tl.RW && rin && (unsigned)gx < (unsigned)W) {
                        v[k] = w.id[gb + gx];
                        if (full) f[k] = w.fl[gb + gx];
                    }
                }
                if (full) {
#pragma unroll
                    for (int k = 0; k < MAXRW / 32; k++) {
                        const int lx = lane + 32 * k, gx = Tl.x0 + lx;
                        if (lx >= Tl.RW) continue;
                        const int i = r * Tl.RW + lx;
                        if (rin && (unsigned)gx < (unsigned)W) {
                            cp_async4(&Tl.s_sc[i], &w.sc[gb + gx]);
                            cp_async4(&Tl.s_col[i], &w.col[gb + gx]);
                        } else {
                            Tl.s_sc[i] = 0;
                            Tl.s_col[i] = 0xff0000u;
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < MAXRW / 32; k++) {
                    const int lx = lane + 32 * k, gx = Tl.x0 + lx;
                    if (lx >= Tl.RW) continue;
                    const int i = r * Tl.RW + lx;
                    const uint32_t cw_ = S.mw[v[k] & CW_ID];
                    Tl.s_w[i] = cw_ | ((uint32_t)(f[k] & (uint8_t)~VISITED) << 8);
                    if (gx >= cx && gx < cx + C && gy >= cy + o0 && gy < cy + o1 && rin && gx < W) {
                        if (cw_ & CW_LIVE) active = 1;
                        if (cw_ & CW_FIRE) fire = 1;
                    }
                }
            }
        }
        if (tma) {
            // the tensor copies have landed (a bounded wait); cells outside the world
            // read as zero there and take the outside colour
            long long spins = 0;
            while (!mbar_try_wait(&s_tma_bar, tma_phase)) {
                if (++spins > (1LL << 26)) {
                    atomicOr(w.err, ERR_TIMEOUT);
                    break;
                }
            }
            tma_phase ^= 1u;
            if (Tl.x0 < 0 || Tl.y0 < 0 || Tl.x0 + Tl.RW > W || Tl.y0 + Tl.RHF > H) {
                for (int i = tid; i < nfull; i += T) {
                    const int r = i / Tl.RW, gx = Tl.x0 + (i - r * Tl.RW), gy = Tl.y0 + r;
                    if ((unsigned)gx >= (unsigned)W || (unsigned)gy >= (unsigned)H) Tl.s_col[i] = 0xff0000u;
                }
            }
        }
        if constexpr (PAIR) {
            active = __syncthreads_or(active);
            fire = __syncthreads_or(fire);
            cp_async_wait_all();
            // the pair decides together whether the chunk runs and with which lattice
            const int slot_x = npass & 1;
            if (tid == 0) st_cluster_u32(mapa_rank(smem_addr(&S.xch[slot_x]), (uint32_t)(rank ^ 1)),
                                         (uint32_t)(active | (fire << 1)));
            cluster_sync();
            const uint32_t o = S.xch[slot_x];
            active |= (int)(o & 1u);
            fire |= (int)((o >> 1) & 1u);
        } else {
            // the copies are in and the chunk's votes are taken with one barrier: each
            // warp's leader writes its warp's votes, every warp ORs the 32 words after
            cp_async_wait_all();
            const unsigned bits = (__any_sync(0xffffffffu, active) ? 1u : 0u) | (__any_sync(0xffffffffu, fire) ? 2u : 0u);
            if ((tid & 31) == 0) S.vote[tid >> 5] = bits;
            __syncthreads();
            const unsigned vv = __reduce_or_sync(0xffffffffu, (tid & 31) < T / 32 ? S.vote[tid & 31] : 0u);
            active = (int)(vv & 1u);
            fire = (int)((vv >> 1) & 1u);
        }
        npass++;
        FSE_PT(1)
        if (!active) {
            // every chunk cell has iterations <= iter: the pass only marks cells visited
            if constexpr (SEQ) {
                if (tid < w.cp_rows) w.cp_count[cp * w.cp_rows + tid] = 0;
            } else if (tid == 0 && rank == 0) {
                w.cp_count[cp] = 0;
            }
            __syncthreads();
            continue;
        }
        FSE_PT(2)

        const int mode = c.has_inter ? 2 : (fire ? 1 : 0);
        const int cw = min(C, W - cx), chh = min(C, H - cy);
        int rb = 0;       // which of S.running holds the spawns of the chunk-pass so far
        int nsub_a = 0;   // CTA pair: the exchange slot of the sweep-A sub-phase
        c.led_g = w.ledger;
        // The reference's order as a wavefront: thread k updates chunk row k counted
        // from the bottom (the row world.cpp's loop takes k-th), cell dx at step
        // dx + s*k. A cell reads and writes at most RX columns to either side
        // (RX = 1; 2 with fire; 5 with interactions, whose boxes lie right of the
        // cell), so two cells whose accesses meet are at least 2*RX+1 = s steps apart
        // in the reference's order's direction: every cell still sees exactly the
        // cells the sequential loop would have updated before it, and no two cells
        // of one step touch the same cell. Each row ranks its own spawns.
        auto sweeps_seq = [&](const auto &Tl) {
            const int s = mode == 2 ? 11 : (mode == 1 ? 5 : 3);
            // row k on lane k / 32 of warp k % 32: a warp runs the rules of its lanes' cells one
            // after another, so four rows a warp on all warps end a step sooner than 32 rows on
            // four (1024 x 512 with f32 amounts: 18.7 against 15.2 ms a step)
            static_assert(CP_THREADS >= 1024, "a thread for each of 32 rows on each of 32 lanes");
            const int k = (tid & 31) * 32 + (tid >> 5), dy = chh - 1 - k;
            const bool row = k < chh;
            int spawned = 0;
            for (int sweep = 0; sweep < 3; sweep++) {
                c.pk = pass_key(w.seed, *w.tick, (uint32_t)(c.iter * 3 + sweep));
                const int steps = cw + s * (chh - 1);
                for (int t = 0; t < steps; t++) {
                    const int dx = t - s * k;
                    if (row && dx >= 0 && dx < cw) {
                        const int x = cx + dx, y = cy + dy, i = Tl.li(x, y);
                        if (sweep == 0) {
                            c.ev_n = 0;
                            c.at(x, y);
                            const int cls = class_a(Tl, c, i);
                            if (cls == 1)
                                rule_a_liquid<false>(Tl, c, Tl.at(i), i, x, y);
                            else if (cls == 2)
                                rule_a(Tl, c, Tl.at(i), i, x, y);
                            if (c.ev_n > 0) {
                                if (!F32 && c.ev_kind == 2) led_add64(c, LED_DF, S.mw[c.ev_idfl & CW_ID], c.ev_df);
                                const int base = atomicAdd(w.stage_count, c.ev_n);
                                emit_spawns<TEMP, F32>(w, c, cp * (uint32_t)w.cp_rows + (uint32_t)k, (uint32_t)spawned,
                                                       base);
                                spawned += c.ev_n;
                            }
                        } else if (sweep == 1) {
                            const uint32_t w0 = Tl.at(i);
                            if (w0 & CW_VIS) {  // world.cpp:1597
                            } else if (cw_is(w0, T_SOUP)) {
                                rule_b_soup(Tl, c, w0, i, Tl.gi(x, y), w.df[Tl.gi(x, y)]);
                            } else {
                                rule_b(Tl, c, w0, i, x, y);
                            }
                        } else {
                            const uint32_t w0 = Tl.at(i);
                            if (!(w0 & CW_VIS) && cw_is(w0, T_GAS)) rule_c(Tl, c, w0, i, x, y);  // world.cpp:1831
                        }
                    }
                    __syncthreads();
                }
            }
            if (k < w.cp_rows) w.cp_count[cp * w.cp_rows + k] = spawned;
        };
        auto sweeps = [&](const auto &Tl) {
#pragma unroll 1
        for (int sweep = 0; sweep < 3; sweep++) {
            c.pk = pass_key(w.seed, *w.tick, (uint32_t)(c.iter * 3 + sweep));
            if (sweep == 1) {
                // AIR snapshot for the friction pillar: columns cx-1..cx+C, rows cy+1..cy+C+9
                // (consecutive threads take consecutive columns, which lie in different banks)
                for (int task = tid; task < (C + 2) * 5; task += T) {
                    const int wi = task / (C + 2), sx = task - wi * (C + 2);
                    const int rows = min(32, own + 9 - wi * 32);
                    int i = Tl.li(cx - 1 + sx, Tl.ay0 + wi * 32);
                    uint32_t bits = 0;
                    for (int b = 0; b < rows; b++, i += Tl.RW)
                        if (Tl.air(i)) bits |= 1u << b;
                    S.air[sx * 5 + wi] = bits;
                }
                // a pair waits for both snapshots: each reads rows that the partner's first
                // sub-phase already changes (a liquid that dries up is mirrored into this tile)
                if constexpr (PAIR)
                    cluster_sync();
                else
                    __syncthreads();
            }
            int px, py;
            lattice(sweep, mode, px, py);
            // A sub-phase's cells are enumerated row by row, nxm to a row for every one of
            // its columns (the last may lie beyond the chunk), so that the threads keep
            // their places in the lattice for the whole sweep.
            const int nxm = (C + px - 1) / px;
            int q, r, dq, dr;
            divmod_small(tid, nxm, __frcp_rn((float)nxm), q, r);
            divmod_small(T, nxm, __frcp_rn((float)nxm), dq, dr);
            const int q1 = q + dq + (r + dr >= nxm ? 1 : 0);  // and of index tid + T
            const int r1 = r + dr - (r + dr >= nxm ? nxm : 0);
#pragma unroll 1
            for (int ry = py - 1; ry >= 0; ry--) {
                // this CTA's rows of the sub-phase: dyb, dyb + py, ... below o1
                const int dyb = ry + (o0 > ry ? (o0 - ry + py - 1) / py * py : 0);
                const int yend = min(o1, chh);
#pragma unroll 1
                for (int rx = 0; rx < px; rx++) {
                    const int dx = rx + r * px, dy = dyb + q * py;
                    const bool v0 = dx < cw && dy < yend;
                    if (sweep == 0) {
                        // at most 43 x 22 <= T cells: one per thread
                        const int cls = v0 ? class_a(Tl, c, Tl.li(cx + dx, cy + dy)) : 0;
                        const unsigned ml = __ballot_sync(0xffffffffu, cls == 1);
                        const unsigned mo = __ballot_sync(0xffffffffu, cls == 2);
                        if (ml | mo) {
                            const int lane = tid & 31;
                            const unsigned lt = (1u << lane) - 1u;
                            unsigned at = 0;
                            if (lane == 0)
                                at = atomicAdd(&S.n_list[nsub], (unsigned)__popc(ml) | ((unsigned)__popc(mo) << 16));
                            at = __shfl_sync(0xffffffffu, at, 0);
                            const uint16_t item = (uint16_t)(dx | (dy << 8));
                            if (cls == 1) S.list[(at & 0xFFFF) + __popc(ml & lt)] = item;
                            if (cls == 2) S.list[T - 1 - (at >> 16) - __popc(mo & lt)] = item;
                        }
                        __syncthreads();
                        const unsigned nl = S.n_list[nsub];
                        const int sub = nsub, nnext = nsub == 2 ? 0 : nsub + 1;
                        // last read before this sub-phase's barrier, next used after the next one's
                        if (tid == 0) S.n_list[nnext == 2 ? 0 : nnext + 1] = 0;
                        if (tid < T / 32) S.spawn_bits[nnext == 2 ? 0 : nnext + 1][tid] = 0;
                        nsub = nnext;
                        if constexpr (!PAIR) {
                            if (nl == 0) continue;  // nothing to do, nothing written but visited marks
                        }
                        FSE_PT(2)
                        c.ev_n = 0;
                        int e = 0;
                        const bool liquid = tid < (int)(nl & 0xFFFF);
                        if (liquid || tid >= T - (int)(nl >> 16)) {
                            const int item = S.list[tid];
                            const int ix = item & 0xFF, iy = item >> 8;
                            const int x = cx + ix, y = cy + iy, i = Tl.li(x, y);
                            const uint32_t w0 = Tl.at(i);
                            c.at(x, y);
                            if (liquid)
                                rule_a_liquid<false>(Tl, c, w0, i, x, y);
                            else
                                rule_a(Tl, c, w0, i, x, y);
                            if (c.ev_n > 0) {
                                int qe, re, t_;
                                divmod_small(iy - dyb, py, __frcp_rn((float)py), qe, t_);
                                divmod_small(ix - rx, px, __frcp_rn((float)px), re, t_);
                                e = qe * nxm + re;
                            }
                        }
                        // The spawns take staging slots a warp at a time, in any order; the atomic
                        // returns while the sub-phase's barrier waits for other warps.
                        __syncwarp();
                        const int lane = tid & 31, wid = tid >> 5;
                        const unsigned sp = __ballot_sync(0xffffffffu, c.ev_n > 0);
                        int slot = 0, spi = 0;
                        seq++;
                        if (sp) {
                            spi = c.ev_n;
#pragma unroll
                            for (int o = 1; o < 32; o <<= 1) {
                                const int t = __shfl_up_sync(0xffffffffu, spi, o);
                                if (lane >= o) spi += t;
                            }
                            if (lane == 31) slot = atomicAdd(w.stage_count, spi);
                            if (c.ev_n > 0) atomicOr(&S.spawn_bits[sub][e >> 5], 1u << (e & 31));
                            if (c.ev_n > 1) S.many = seq;
                        }
                        FSE_PT(3)
                        // spawned particles are ranked in enumeration order: from the bits of the
                        // spawning cells, a word per lane of every warp, without another barrier
                        const bool any = __syncthreads_or(c.ev_n > 0);
                        // (only the warps that need them, and the first, which keeps the count)
                        int tot = 0, rank_e = 0, before = S.running[rb];
                        if (any) {
                            if (S.many != seq) {
                                if (sp || wid == 0) {
                                    const uint32_t word = lane < T / 32 ? S.spawn_bits[sub][lane] : 0u;
                                    int inc = __popc(word);
#pragma unroll
                                    for (int o = 1; o < 32; o <<= 1) {
                                        const int t = __shfl_up_sync(0xffffffffu, inc, o);
                                        if (lane >= o) inc += t;
                                    }
                                    tot = __shfl_sync(0xffffffffu, inc, 31);
                                    const uint32_t we = __shfl_sync(0xffffffffu, word, e >> 5);
                                    rank_e = __shfl_sync(0xffffffffu, inc - __popc(word), e >> 5) +
                                             __popc(we & ((1u << (e & 31)) - 1u));
                                }
                            } else {
                                // some cell spawns several: a scan over their counts
                                S.cnt[tid] = 0;
                                __syncthreads();
                                if (c.ev_n > 0) S.cnt[e] = (uint32_t)c.ev_n;
                                __syncthreads();
                                const int v = (int)S.cnt[tid];
                                int inc = v;
#pragma unroll
                                for (int o = 1; o < 32; o <<= 1) {
                                    const int t = __shfl_up_sync(0xffffffffu, inc, o);
                                    if (lane >= o) inc += t;
                                }
                                if (lane == 31) S.scan[wid] = inc;
                                __syncthreads();
                                const int ws = lane < T / 32 ? S.scan[lane] : 0;
                                tot = (int)__reduce_add_sync(0xffffffffu, (unsigned)ws);
                                S.cnt[tid] = __reduce_add_sync(0xffffffffu, lane < wid ? (unsigned)ws : 0u) +
                                             (unsigned)(inc - v);
                                __syncthreads();
                                rank_e = (int)S.cnt[e];
                                __syncthreads();
                            }
                        }
                        if constexpr (PAIR) {
                            // the sub-phase's enumeration runs through rank 0's rows first:
                            // each CTA ranks its own spawns, the partner's count of the
                            // sub-phase comes through the cluster barrier that ends it
                            const int slot_t = 2 + nsub_a;
                            nsub_a ^= 1;
                            if (tid == 0)
                                st_cluster_u32(mapa_rank(smem_addr(&S.xch[slot_t]), (uint32_t)(rank ^ 1)),
                                               (uint32_t)tot);
                            cluster_sync();
                            const int tot_p = (int)S.xch[slot_t];
                            if (any || tot_p) {
                                if (tid == 0) S.running[rb ^ 1] = before + tot + tot_p;
                                rb ^= 1;
                            }
                            if (rank) before += tot_p;
                        } else if (any) {
                            // read after the next barrier at the earliest
                            if (tid == 0) S.running[rb ^ 1] = before + tot;
                            rb ^= 1;
                        }
                        // the (chunk-pass, rank) key orders the particles later
                        if (sp) {
                            slot = __shfl_sync(0xffffffffu, slot, 31) + spi - c.ev_n;
                            if (c.ev_n > 0) {
                                emit_spawns<TEMP, F32>(w, c, cp, (uint32_t)(before + rank_e), slot);
                                if (!F32 && c.ev_kind == 2) led_add64(c, LED_DF, S.mw[c.ev_idfl & CW_ID], c.ev_df);
                            }
                        }
                        FSE_PT(4)
                    } else if (sweep == 1) {
                        // at most 43 x 43 < 2 T cells: two per thread. Liquids take their
                        // pending diffs, requested together; sand and gas that may move are
                        // listed and dealt to the threads
                        const int dx1 = rx + r1 * px, dy1 = dyb + q1 * py;
                        const bool v1 = dx1 < cw && dy1 < yend;
                        const int i0 = Tl.li(cx + dx, cy + dy), i1 = Tl.li(cx + dx1, cy + dy1);
                        const uint32_t w0 = v0 ? Tl.at(i0) : CW_VIS, w1 = v1 ? Tl.at(i1) : CW_VIS;
                        const int g0 = Tl.gi(cx + dx, cy + dy), g1 = Tl.gi(cx + dx1, cy + dy1);
                        const bool s0 = (w0 & (CW_TYPE | CW_VIS)) == (uint32_t)T_SOUP << MW_TYPE_SHIFT;
                        const bool s1 = (w1 & (CW_TYPE | CW_VIS)) == (uint32_t)T_SOUP << MW_TYPE_SHIFT;
                        const int32_t df0 = s0 ? w.df[g0] : 0, df1 = s1 ? w.df[g1] : 0;
                        const bool a0 = !(w0 & CW_VIS) && class_b(Tl, w0, i0, w.dirty != nullptr);
                        const bool a1 = !(w1 & CW_VIS) && class_b(Tl, w1, i1, w.dirty != nullptr);
                        const unsigned m0 = __ballot_sync(0xffffffffu, a0), m1 = __ballot_sync(0xffffffffu, a1);
                        if (m0 | m1) {
                            const int lane = tid & 31;
                            const unsigned lt = (1u << lane) - 1u;
                            unsigned at = 0;
                            if (lane == 0) at = atomicAdd(&S.n_list[nsub], (unsigned)(__popc(m0) + __popc(m1)));
                            at = __shfl_sync(0xffffffffu, at, 0);
                            if (a0) S.list[at + __popc(m0 & lt)] = (uint16_t)(dx | (dy << 8));
                            if (a1) S.list[at + __popc(m0) + __popc(m1 & lt)] = (uint16_t)(dx1 | (dy1 << 8));
                        }
                        if (s0) rule_b_soup(Tl, c, w0, i0, g0, df0);
                        if (s1) rule_b_soup(Tl, c, w1, i1, g1, df1);
                        FSE_PT(5)
                        __syncthreads();
                        const int nl = (int)S.n_list[nsub];
                        const int nnext = nsub == 2 ? 0 : nsub + 1;
                        if (tid == 0) S.n_list[nnext == 2 ? 0 : nnext + 1] = 0;
                        if (tid < T / 32) S.spawn_bits[nnext == 2 ? 0 : nnext + 1][tid] = 0;
                        nsub = nnext;
                        if constexpr (!PAIR) {
                            if (nl == 0) continue;
                        }
#pragma unroll 1
                        for (int k = tid; k < nl; k += T) {
                            const int item = S.list[k];
                            const int ix = item & 0xFF, iy = item >> 8;
                            const int i = Tl.li(cx + ix, cy + iy);
                            rule_b(Tl, c, Tl.at(i), i, cx + ix, cy + iy);
                        }
                        if constexpr (PAIR)
                            cluster_sync();
                        else
                            __syncthreads();
                        FSE_PT(6)
                    } else {
                        // every row of the chunk, its columns 3 apart: each thread takes all of
                        // its cells in turn
                        // (three words loaded at a time: most cells are no gas)
                        int qe = q, re = r;
#pragma unroll 1
                        while (dyb + qe * py < yend) {
                            int i3[3], x3[3], y3[3];
                            uint32_t w3[3];
#pragma unroll
                            for (int k = 0; k < 3; k++) {
                                const int ex = rx + re * px, ey = dyb + qe * py;
                                x3[k] = cx + ex;
                                y3[k] = cy + ey;
                                i3[k] = Tl.li(x3[k], y3[k]);
                                w3[k] = ex < cw && ey < yend ? Tl.at(i3[k]) : CW_VIS;
                                qe += dq;
                                re += dr;
                                if (re >= nxm) {
                                    re -= nxm;
                                    qe++;
                                }
                            }
#pragma unroll
                            for (int k = 0; k < 3; k++)
                                if (!(w3[k] & CW_VIS) && cw_is(w3[k], T_GAS)) rule_c(Tl, c, w3[k], i3[k], x3[k], y3[k]);
                        }
                        FSE_PT(7)
                        if constexpr (PAIR)
                            cluster_sync();
                        else
                            __syncthreads();
                        FSE_PT(8)
                    }
                }
            }
        }
        };
        if constexpr (SEQ)
            sweeps_seq(Tile<TEMP, true, F32>(Tl));
        else
            sweeps(Tile<TEMP, false, F32, PAIR>(Tl));

        // ---- write back the cells this CTA changed (full-state rows inside the world),
        // one warp per row
        if (tma) {
            // four cells at a time, whole groups that hold a changed cell: the other cells of
            // the tile go back as they were staged (no other chunk-pass runs on them meanwhile)
            const int gpr = Tl.RW / 4, groups = gpr * Tl.RHF;
            const float rgpr = __frcp_rn((float)gpr);
            for (int e = tid; e < groups; e += T) {
                const uint4 o = *reinterpret_cast<const uint4 *>(&Tl.s_w[4 * e]);
                if (!((o.x | o.y | o.z | o.w) & CW_DIRTY)) continue;
                int r, q4;
                divmod_small(e, gpr, rgpr, r, q4);
                const int gx = Tl.x0 + 4 * q4, gy = Tl.y0 + r;
                if ((unsigned)gy >= (unsigned)H || (unsigned)gx >= (unsigned)W) continue;
                const size_t gi = (size_t)gy * W + gx;
                constexpr uint32_t FL = (CW_FLAGS & ~CW_VIS) >> 8;
                *reinterpret_cast<uint2 *>(&w.id[gi]) =
                    make_uint2((o.x & CW_ID) | (o.y & CW_ID) << 16, (o.z & CW_ID) | (o.w & CW_ID) << 16);
                *reinterpret_cast<uint32_t *>(&w.fl[gi]) = (o.x >> 8 & FL) | (o.y >> 8 & FL) << 8 |
                                                           (o.z >> 8 & FL) << 16 | (o.w >> 8 & FL) << 24;
                *reinterpret_cast<uint4 *>(&w.sc[gi]) = *reinterpret_cast<const uint4 *>(&Tl.s_sc[4 * e]);
                *reinterpret_cast<uint4 *>(&w.col[gi]) = *reinterpret_cast<const uint4 *>(&Tl.s_col[4 * e]);
                if (w.dirty) {
                    if (o.x & CW_DIRTY) w.dirty[gi] = 1;
                    if (o.y & CW_DIRTY) w.dirty[gi + 1] = 1;
                    if (o.z & CW_DIRTY) w.dirty[gi + 2] = 1;
                    if (o.w & CW_DIRTY) w.dirty[gi + 3] = 1;
                }
            }
        } else {
            const int lane = tid & 31, wid = tid >> 5;
            for (int r = wid; r < Tl.RHF; r += T / 32) {
                const int gy = Tl.y0 + r;
                if ((unsigned)gy >= (unsigned)H) continue;
                // a CTA pair: rank 0 writes rows above the chunk's middle, rank 1 the
                // others (each row is written by the CTA that owns it)
                if (PAIR && (rank == 0 ? gy >= cy + half : gy < cy + half)) continue;
                const size_t gb = (size_t)gy * W;
#pragma unroll
                for (int k = 0; k < MAXRW / 32; k++) {
                    const int lx = lane + 32 * k, gx = Tl.x0 + lx;
                    if (lx >= Tl.RW || (unsigned)gx >= (unsigned)W) continue;
                    const int i = r * Tl.RW + lx;
                    const uint32_t v = Tl.s_w[i];
                    if (!(v & CW_DIRTY)) continue;
                    w.id[gb + gx] = (uint16_t)cw_id(v);
                    w.fl[gb + gx] = (uint8_t)((v & (CW_FLAGS & ~CW_VIS)) >> 8);
                    w.sc[gb + gx] = Tl.s_sc[i];
                    w.col[gb + gx] = Tl.s_col[i];
                    if (w.dirty) w.dirty[gb + gx] = 1;
                }
            }
        }
        // the written cells come before the tensor copies of the chunk-passes that wait for this one
        if constexpr (FUSED && kTma) fence_proxy_async_global();
        if (!SEQ && tid == 0 && rank == 0) w.cp_count[cp] = S.running[rb];
        // the chunk-pass's ledger counts (the sweeps ended with a barrier)
        for (int i = tid; i < LED_TICK * 64; i += T) {
            const int32_t v = S.led[i];
            if (v == 0) continue;
            S.led[i] = 0;
            const int row = i / 64 < LED_XN ? i / 64 : i / 64 + 1;
            atomicAdd((unsigned long long *)&w.ledger[row * MAXMAT + (i % 64)], (unsigned long long)(long long)v);
        }
        __syncthreads();
        FSE_PT(9)
    }
    // a CTA of a pair leaves only when its partner no longer writes to it
    if constexpr (PAIR) cluster_sync();
    if constexpr (FUSED) {
        // the last CTA out clears the completion flags and the counters
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            s_ticket = (atomicAdd(&worlds[0].sched[1], 1u) == gridDim.x - 1) ? 1 : 0;
        }
        __syncthreads();
        if (s_ticket) {
            __threadfence();
            for (int wi = 0; wi < ft.n_worlds; wi++) {
                uint32_t *f = worlds[wi].cdone;
                const int nc = worlds[wi].nCx * worlds[wi].nCy;
                for (int i = tid; i < nc; i += T) f[i] = 0u;
            }
            if (tid == 0) {
                worlds[0].sched[0] = 0u;
                worlds[0].sched[1] = 0u;
                worlds[0].sched[2] = 0u;
            }
        }
    }
    FSE_PT_FLUSH
}

#if !defined(FSE_TICK_TEMP_TU) && !defined(FSE_TICK_SEQ_TU) && !defined(FSE_TICK_F32_TU) && \
    !defined(FSE_TICK_PAIR_TU) && !defined(FSE_TICK_FUSED_TU)
size_t colour_pass_smem(int C, int halo) {
    // a 2-cell halo leaves room for the TMA-staged tile's wider rows
    return tile_smem<CP_THREADS>(C, C, halo, halo == 2 ? tma_tile_width(C) : 0);
}

#endif

template <int HALO, bool TEMP, bool SEQ = false, bool F32 = false, int CC = 0>
static cudaError_t launch_cc(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                            const MatTable *mt, size_t sm, int grid, cudaStream_t s) {
    auto *kernel = k_colour_pass<HALO, TEMP, SEQ, F32, false, false, CC>;
    static SmemOptIn opt_in;
    if (const cudaError_t e = opt_in(kernel, sm)) return e;
    kernel<<<grid, CP_THREADS, sm, s>>>(worlds, items, n_items, iter, tk, mt, FusedTick{});
    return cudaGetLastError();
}

// chunks of 128 with a 2-cell halo run the instantiation that knows its chunk edge
template <int HALO, bool TEMP, bool SEQ = false, bool F32 = false>
static cudaError_t launch_t(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                            const MatTable *mt, int C, size_t sm, int grid, cudaStream_t s) {
    if constexpr (HALO == 2 && !SEQ) {
        if (C == 128) return launch_cc<HALO, TEMP, SEQ, F32, 128>(worlds, items, n_items, iter, tk, mt, sm, grid, s);
    }
    return launch_cc<HALO, TEMP, SEQ, F32>(worlds, items, n_items, iter, tk, mt, sm, grid, s);
}

// the fused tick: one CTA per SM (the tile takes most of an SM's shared memory)
template <int HALO, bool TEMP, bool F32, int CC>
static cudaError_t launch_fused_cc(const WorldDev *worlds, const FusedTick &ft, const MatTable *mt, size_t sm,
                                  int grid, cudaStream_t s) {
    auto *kernel = k_colour_pass<HALO, TEMP, false, F32, false, true, CC>;
    static SmemOptIn opt_in;
    if (const cudaError_t e = opt_in(kernel, sm)) return e;
    kernel<<<grid, CP_THREADS, sm, s>>>(worlds, nullptr, 0, 0, 0, mt, ft);
    return cudaGetLastError();
}

template <int HALO, bool TEMP, bool F32>
static cudaError_t launch_fused_t(const WorldDev *worlds, const FusedTick &ft, const MatTable *mt, int C, size_t sm,
                                  int grid, cudaStream_t s) {
    if constexpr (HALO == 2) {
        if (C == 128) return launch_fused_cc<HALO, TEMP, F32, 128>(worlds, ft, mt, sm, grid, s);
    }
    return launch_fused_cc<HALO, TEMP, F32, 0>(worlds, ft, mt, sm, grid, s);
}

// shared memory of one CTA of a pair: half the chunk's rows plus the reach of its rules
static size_t colour_pass_smem_pair(int C, int halo) { return tile_smem<CP_THREADS / 2>(C, C / 2, halo, 0); }

// the chunks split over CTA pairs (thread-block clusters of two): `clusters` pairs
template <int HALO, bool TEMP, bool F32, int CC>
static cudaError_t launch_pair_cc(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                  const MatTable *mt, size_t sm, int clusters, cudaStream_t s) {
    auto *kernel = k_colour_pass<HALO, TEMP, false, F32, true, false, CC>;
    // all of the unified L1/shared storage as shared memory, so that two CTAs share an SM
    // where they fit
    static SmemOptIn opt_in;
    if (const cudaError_t e = opt_in(kernel, sm, cudaSharedmemCarveoutMaxShared)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * clusters);
    cfg.blockDim = dim3(CP_THREADS / 2);
    cfg.dynamicSmemBytes = sm;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, worlds, items, n_items, iter, tk, mt, FusedTick{});
}

template <int HALO, bool TEMP, bool F32>
static cudaError_t launch_pair_t(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                 const MatTable *mt, int C, size_t sm, int clusters, cudaStream_t s) {
    if (C == 128) return launch_pair_cc<HALO, TEMP, F32, 128>(worlds, items, n_items, iter, tk, mt, sm, clusters, s);
    return launch_pair_cc<HALO, TEMP, F32, 0>(worlds, items, n_items, iter, tk, mt, sm, clusters, s);
}

// Each translation unit that includes this file with one of the defines below
// compiles one family of instantiations, so that they build in parallel.
#if defined(FSE_TICK_FUSED_TU)
// the fused tick, Q16.16 amounts (FSE_TICK_FUSED_TU = 1) or f32 (2)
#define FSE_FUSED_F32 (FSE_TICK_FUSED_TU == 2)
size_t colour_pass_smem(int C, int halo);
#if FSE_TICK_FUSED_TU == 2
cudaError_t launch_colour_fused_f32(const WorldDev *worlds, const FusedTick &ft, const MatTable *mt, int halo, int C,
                                    int grid, cudaStream_t s, bool temp) {
#else
cudaError_t launch_colour_fused(const WorldDev *worlds, const FusedTick &ft, const MatTable *mt, int halo, int C,
                                int grid, cudaStream_t s, bool temp) {
#endif
    const size_t sm = colour_pass_smem(C, halo);
    if (temp) {
        if (halo == 5) return launch_fused_t<5, true, FSE_FUSED_F32>(worlds, ft, mt, C, sm, grid, s);
        return launch_fused_t<2, true, FSE_FUSED_F32>(worlds, ft, mt, C, sm, grid, s);
    }
    if (halo == 5) return launch_fused_t<5, false, FSE_FUSED_F32>(worlds, ft, mt, C, sm, grid, s);
    return launch_fused_t<2, false, FSE_FUSED_F32>(worlds, ft, mt, C, sm, grid, s);
}
#elif defined(FSE_TICK_PAIR_TU)
// chunks split over CTA pairs, Q16.16 amounts (FSE_TICK_PAIR_TU = 1) or f32 (2)
#define FSE_PAIR_F32 (FSE_TICK_PAIR_TU == 2)
#if FSE_TICK_PAIR_TU == 2
cudaError_t launch_colour_pass_pair_f32(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                        const MatTable *mt, int halo, int C, int clusters, cudaStream_t s, bool temp) {
#else
cudaError_t launch_colour_pass_pair(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                    const MatTable *mt, int halo, int C, int clusters, cudaStream_t s, bool temp) {
#endif
    const size_t sm = colour_pass_smem_pair(C, halo);
    if (temp) {
        if (halo == 5)
            return launch_pair_t<5, true, FSE_PAIR_F32>(worlds, items, n_items, iter, tk, mt, C, sm, clusters, s);
        return launch_pair_t<2, true, FSE_PAIR_F32>(worlds, items, n_items, iter, tk, mt, C, sm, clusters, s);
    }
    if (halo == 5) return launch_pair_t<5, false, FSE_PAIR_F32>(worlds, items, n_items, iter, tk, mt, C, sm, clusters, s);
    return launch_pair_t<2, false, FSE_PAIR_F32>(worlds, items, n_items, iter, tk, mt, C, sm, clusters, s);
}
#elif defined(FSE_TICK_F32_TU)
// f32 liquid amounts (FSE_CFG_F32_FLUID), in the partitioned order (FSE_TICK_F32_TU
// = 1) or in the reference's order (2)
#define FSE_F32_SEQ (FSE_TICK_F32_TU == 2)
#if FSE_TICK_F32_TU == 2
cudaError_t launch_colour_pass_f32_seq(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                       const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s, bool temp) {
#else
cudaError_t launch_colour_pass_f32(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                   const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s, bool temp) {
#endif
    if (temp) {
        if (halo == 5) return launch_t<5, true, FSE_F32_SEQ, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
        return launch_t<2, true, FSE_F32_SEQ, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
    }
    if (halo == 5) return launch_t<5, false, FSE_F32_SEQ, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
    return launch_t<2, false, FSE_F32_SEQ, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
}
#elif defined(FSE_TICK_SEQ_TU)
cudaError_t launch_colour_pass_seq(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                   const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s, bool temp) {
    if (temp) {
        if (halo == 5) return launch_t<5, true, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
        return launch_t<2, true, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
    }
    if (halo == 5) return launch_t<5, false, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
    return launch_t<2, false, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
}
#elif defined(FSE_TICK_TEMP_TU)
cudaError_t launch_colour_pass_temp(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                    const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s) {
    if (halo == 5) return launch_t<5, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
    return launch_t<2, true>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
}
#else
cudaError_t launch_colour_pass_temp(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                    const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s);
cudaError_t launch_colour_pass_seq(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                   const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s, bool temp);
cudaError_t launch_colour_pass_f32(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                   const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s, bool temp);
cudaError_t launch_colour_pass_f32_seq(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                       const MatTable *mt, int halo, int C, size_t sm, int grid, cudaStream_t s, bool temp);

cudaError_t launch_colour_pass_pair(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                    const MatTable *mt, int halo, int C, int clusters, cudaStream_t s, bool temp);
cudaError_t launch_colour_pass_pair_f32(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                                        const MatTable *mt, int halo, int C, int clusters, cudaStream_t s, bool temp);

// threads: CP_THREADS (one CTA per chunk) or CP_THREADS / 2 (each chunk split over a
// CTA pair; the partitioned order and an even chunk edge only); grid: chunk workers
// (CTAs, or pairs), 0 = one per chunk
cudaError_t launch_colour_pass(const WorldDev *worlds, const uint32_t *items, int n_items, int iter, int tk,
                               const MatTable *mt, int halo, int C, int threads, int grid, cudaStream_t s,
                               bool temp, bool seq, bool f32) {
    size_t sm = colour_pass_smem(C, halo);
    if (n_items <= 0) return cudaSuccess;
    if (grid <= 0 || grid > n_items) grid = n_items;
    if (threads == CP_THREADS / 2 && !seq && C % 2 == 0) {
        if (f32) return launch_colour_pass_pair_f32(worlds, items, n_items, iter, tk, mt, halo, C, grid, s, temp);
        return launch_colour_pass_pair(worlds, items, n_items, iter, tk, mt, halo, C, grid, s, temp);
    }
    if (f32 && seq) return launch_colour_pass_f32_seq(worlds, items, n_items, iter, tk, mt, halo, C, sm, grid, s, temp);
    if (f32) return launch_colour_pass_f32(worlds, items, n_items, iter, tk, mt, halo, C, sm, grid, s, temp);
    if (seq) return launch_colour_pass_seq(worlds, items, n_items, iter, tk, mt, halo, C, sm, grid, s, temp);
    if (temp) return launch_colour_pass_temp(worlds, items, n_items, iter, tk, mt, halo, C, sm, grid, s);
    if (halo == 5) return launch_t<5, false>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
    return launch_t<2, false>(worlds, items, n_items, iter, tk, mt, C, sm, grid, s);
}
#endif

}  // namespace fse

#if defined(FSE_PHASE_CLOCKS) && !defined(FSE_TICK_TEMP_TU) && !defined(FSE_TICK_SEQ_TU) && !defined(FSE_TICK_F32_TU) && \
    !defined(FSE_TICK_PAIR_TU) && !defined(FSE_TICK_FUSED_TU)
extern "C" int fse_debug_phase_clocks(unsigned long long out[16], int reset) {
    cudaDeviceSynchronize();
    cudaMemcpyFromSymbol(out, g_phase_clk, 16 * sizeof(unsigned long long));
    if (reset) {
        unsigned long long z[16] = {0};
        cudaMemcpyToSymbol(g_phase_clk, z, sizeof(z));
    }
    return 0;
}
// the per-phase maxima over CTAs (out[15]: the longest CTA, start to end)
extern "C" int fse_debug_phase_max(unsigned long long out[16], int reset) {
    cudaDeviceSynchronize();
    cudaMemcpyFromSymbol(out, g_phase_max, 16 * sizeof(unsigned long long));
    if (reset) {
        unsigned long long z[16] = {0};
        cudaMemcpyToSymbol(g_phase_max, z, sizeof(z));
    }
    return 0;
}
#endif
