// fse_objects.cu -- rigid-body OBJECT tiles: stamping before the tick
// (source/engine/game.cpp:1768-1814), readback after it (game.cpp:1896-1983) and
// the per-tick OBJECT-cell export to the host-side rigid-body solver.
//
// Stamp and readback resolve body tiles by deferred acceptance (see k_obj_settle): the result is the reference's tile-by-tile one,
// and displaced particles are appended in (body, tile) order.
#include <algorithm>
#include <vector>

#include "fse_host.cuh"

namespace fse {

__constant__ int c_dirs[5][2] = {{0, 0}, {1, 0}, {-1, 0}, {0, 1}, {0, -1}};

__device__ __forceinline__ void body_pos(const fse_body &b, int tx, int ty, int &wx, int &wy) {
    // int wx = (int)(tx * c - (ty + 1) * s + x); int wy = (int)(tx * s + (ty + 1) * c + y);
    float fx = __fadd_rn(__fsub_rn(__fmul_rn((float)tx, b.cos_a), __fmul_rn((float)(ty + 1), b.sin_a)), b.x);
    float fy = __fadd_rn(__fadd_rn(__fmul_rn((float)tx, b.sin_a), __fmul_rn((float)(ty + 1), b.cos_a)), b.y);
    wx = (int)fx;
    wy = (int)fy;
}

__device__ __forceinline__ int block_scan_excl(int v, int *s, int *total) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int inc = v;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) s[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int a = lane < nw ? s[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, a, o);
            if (lane >= o) a += t;
        }
        if (lane < nw) s[lane] = a;
    }
    __syncthreads();
    int before = wid > 0 ? s[wid - 1] : 0;
    *total = s[nw - 1];
    __syncthreads();
    return before + inc - v;
}

__device__ __forceinline__ int body_of(const uint32_t *__restrict__ prefix, int nb, uint32_t g) {
    int lo = 0, hi = nb - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= g) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ bool tile_usable(const WorldDev &w, const MatTable *__restrict__ mt, int mode, int c,
                                            int body_id) {
    const int cid = w.id[c];
    if (mode == 0) {
        const int ty = mt_type(mt->a[cid]);
        return ty == T_AIR || ty == T_SAND || ty == T_SOUP;
    }
    return cid == body_id;
}

// mode 0 = stamp, 1 = readback; prefix[b] = first global tile index of body b.
//
// The reference walks the tiles one after another (bodies in order, tx-major,
// ty-minor): each takes the first of its five cells that is usable at that moment
// (stamp: AIR, SAND or SOUP; readback: the body's material), and a taken cell is
// not usable by the tiles after it. Here the tiles propose in parallel, each cell
// keeping its lowest proposer (claim = atomicMin of the tile index) and displacing
// higher ones, a rejected or displaced tile proposing its next cell: deferred
// acceptance with the same priority order at every cell, whose outcome is the
// sequential one, in whatever order the proposals are made. Usability is read from the
// grid before any write, since only the taking itself makes a cell unusable. Displaced
// particles are then appended in tile order.

// a tile's own cell and which of its five cells it may take
struct ObjTile {
    int32_t x, y;  // may lie outside the world
    uint32_t use;  // bit d: the cell at c_dirs[d]
    int32_t pad;
};

__global__ void __launch_bounds__(256) k_obj_tiles(const WorldDev *__restrict__ wd, const MatTable *__restrict__ mt,
                                                   const fse_body *__restrict__ bodies,
                                                   const uint32_t *__restrict__ prefix, int nb, int mode,
                                                   ObjTile *tiles) {
    const WorldDev &w = *wd;
    const uint32_t total = prefix[nb];
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const int bi = body_of(prefix, nb, g);
        const fse_body &b = bodies[bi];
        const int t = (int)(g - prefix[bi]);
        ObjTile o;
        body_pos(b, t / b.h, t % b.h, o.x, o.y);
        o.use = 0;
        o.pad = 0;
#pragma unroll
        for (int d = 0; d < 5; d++) {
            const long long x = (long long)o.x + c_dirs[d][0], y = (long long)o.y + c_dirs[d][1];
            if (x < 0 || y < 0 || x >= w.W || y >= w.H) continue;
            if (tile_usable(w, mt, mode, (int)y * w.W + (int)x, (int)b.id)) o.use |= 1u << d;
        }
        tiles[g] = o;
    }
}

// Every thread takes a tile through its proposals; a tile that it displaces from a cell is
// taken through its further ones by the same thread, from the cell that it lost (which of
// its five that was follows from its position). So a chain of displacements, up to some
// hundred tiles long where boxes read back overlapping cells, waits for two memory round
// trips a link and for no other tile. (Rounds over work lists in one CTA, with a barrier and a
// dozen dependent loads a round, took 1.9 ms of a call with 260,000 tiles.)
__global__ void __launch_bounds__(256) k_obj_settle(const WorldDev *__restrict__ wd, uint32_t total,
                                                    const ObjTile *__restrict__ tiles, uint32_t *claim) {
    const int W = wd->W;
    for (uint32_t first = blockIdx.x * blockDim.x + threadIdx.x; first < total; first += gridDim.x * blockDim.x) {
        uint32_t g = first;
        ObjTile o = tiles[g];
        uint32_t left = o.use;  // the cells not yet proposed to
        // ends: each step uses up one of some tile's five cells, for good
        while (left) {
            const int d = __ffs(left) - 1;
            left &= left - 1;
            const int c = (o.y + c_dirs[d][1]) * W + o.x + c_dirs[d][0];
            const uint32_t old = atomicMin(&claim[c], g);
            if (old < g) continue;  // taken by an earlier tile
            if (old == 0xffffffffu) break;
            g = old;  // displaced from c
            o = tiles[g];
            const int x = c % W - o.x, y = c / W - o.y;
            int lost = 0;
#pragma unroll
            for (int k = 0; k < 5; k++)
                if (c_dirs[k][0] == x && c_dirs[k][1] == y) lost = k;
            left = o.use & ~((2u << lost) - 1u);
        }
    }
}

// the cell a tile holds in the end (-1: none)
__global__ void __launch_bounds__(256) k_obj_held(const WorldDev *__restrict__ wd, uint32_t total,
                                                  const ObjTile *__restrict__ tiles, const uint32_t *__restrict__ claim,
                                                  int32_t *held) {
    const int W = wd->W;
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < total; g += gridDim.x * blockDim.x) {
        const ObjTile o = tiles[g];
        int h = -1;
#pragma unroll
        for (int d = 0; d < 5; d++) {
            if (!(o.use >> d & 1)) continue;
            const int c = (o.y + c_dirs[d][1]) * W + o.x + c_dirs[d][0];
            if (claim[c] == g) h = c;
        }
        held[g] = h;
    }
}

// blocks of the two kernels below: contiguous ranges of tiles in order; two a SM, as many as
// the scan of their counts by one block allows for many times over (a stamp and readback of
// 2 million tiles took 0.71 ms with 152, 304 and 608 blocks, of 12 million 4.1, 3.9 and 3.8)
constexpr int OBJ_BLOCKS = 304;
__device__ __forceinline__ void obj_range(uint32_t total, uint32_t *b0, uint32_t *b1) {
    const uint32_t seg = (total + gridDim.x - 1) / gridDim.x;
    *b0 = min(total, blockIdx.x * seg);
    *b1 = min(total, *b0 + seg);
}

// stamp: the particles that the range's tiles displace
__global__ void __launch_bounds__(1024) k_obj_count(const WorldDev *__restrict__ wd, const MatTable *__restrict__ mt,
                                                    uint32_t total, const int32_t *__restrict__ held, int32_t *blk) {
    __shared__ int s_scan[40];
    uint32_t b0, b1;
    obj_range(total, &b0, &b1);
    int n = 0;
    for (uint32_t g = b0 + threadIdx.x; g < b1; g += blockDim.x) {
        const int c = held[g];
        if (c < 0) continue;
        const int ty = mt_type(mt->a[wd->id[c]]);
        n += ty == T_SAND || ty == T_SOUP;
    }
    int tot;
    block_scan_excl(n, s_scan, &tot);
    if (threadIdx.x == 0) blk[blockIdx.x] = tot;
}

// add one to the counter a thread's address names, once per group of a warp's lanes of
// the same key (equal keys mean equal addresses; `on` lanes only)
template <class F>
__device__ __forceinline__ void warp_count(bool on, int key, F add) {
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (!on) return;
    const unsigned same = __match_any_sync(m, key);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) add(__popc(same));
}

// the outcome: displaced particles in tile order (a tile reads and writes the cell it
// holds, which no other tile holds), then the tile's cell
__global__ void __launch_bounds__(1024) k_obj_apply(WorldDev *wd, const MatTable *__restrict__ mt, fse_body *bodies,
                                                    const uint32_t *__restrict__ prefix, int nb,
                                                    const int32_t *__restrict__ held, uint32_t *claim, int mode,
                                                    const int32_t *__restrict__ blk, long long *removed) {
    const WorldDev &w = *wd;
    const int W = w.W;
    __shared__ int s_scan[40];
    const uint32_t total = prefix[nb];
    uint32_t b0, b1;
    obj_range(total, &b0, &b1);
    const uint32_t pk = pass_key(w.seed, *w.tick, PH_STAMP);
    int run = 0;
    if (mode == 0) {
        const int v = (int)threadIdx.x < (int)blockIdx.x ? blk[threadIdx.x] : 0;
        int before;
        block_scan_excl(v, s_scan, &before);
        run = *w.part_count + before;
    }
    int rem_local = 0;
    for (uint32_t base = b0; base < b1; base += blockDim.x) {
        const uint32_t g = base + threadIdx.x;
        const int tg = g < b1 ? held[g] : -1;
        int id = 0, ty = -1, bi = 0;
        if (tg >= 0) {
            id = w.id[tg];
            ty = mt_type(mt->a[id]);
            bi = body_of(prefix, nb, g);
        }
        if (mode == 0) {
            const bool spawn = ty == T_SAND || ty == T_SOUP;
            int tot_s;
            const int ex_s = block_scan_excl(spawn ? 1 : 0, s_scan, &tot_s);
            if (spawn) {
                const int pos = run + ex_s;
                if (pos < w.part_cap) {
                    const uint32_t ck = cell_key(pk, (uint32_t)bi, g - prefix[bi]);
                    // CellData(tile, wxd, wyd - 3, (rand()%10-5)/10.0f, -(rand()%5+5)/10.0f, 0, 0.1)
                    w.p.x[pos] = (float)(tg % W);
                    w.p.y[pos] = (float)(tg / W - 3);
                    w.p.vx[pos] = (float)((int)(draw_k(ck, 0) % 10) - 5) / 10.0f;
                    w.p.vy[pos] = (float)(-((int)(draw_k(ck, 1) % 5) + 5)) / 10.0f;
                    w.p.ax[pos] = 0.f;
                    w.p.ay[pos] = 0.1f;
                    w.p.tx[pos] = 0.f;
                    w.p.ty[pos] = 0.f;
                    w.p.tf[pos] = 0.f;
                    w.p.life[pos] = 0;
                    w.p.fade[pos] = 60;
                    w.p.col[pos] = w.col[tg];
                    w.p.sc[pos] = w.sc[tg];
                    if (w.tp) w.p.tp[pos] = ty == T_SOUP ? w.tp[tg] : (int16_t)0;
                    w.p.id[pos] = (uint16_t)id;
                    w.p.fl[pos] = w.fl[tg];
                    w.p.bits[pos] = 0;
                } else {
                    atomicOr(w.err, ERR_PART_CAP);
                }
                if (ty == T_SOUP && !w.f32)  // f32 amounts: no fluid rows
                    atomicAdd((unsigned long long *)&w.ledger[LED_DF * MAXMAT + id],
                              (unsigned long long)(long long)w.df[tg]);
            }
            run += tot_s;
            warp_count(ty == T_SOUP, bi, [&](int n) { atomicAdd(&bodies[bi].n_soup, n); });
            warp_count(ty == T_SAND, bi, [&](int n) { atomicAdd(&bodies[bi].n_sand, n); });
        }
        // a body's tiles are of one material, and on readback the cells they hold as well
        warp_count(tg >= 0, bi, [&](int n) {
            fse_body &b = bodies[bi];
            const int row = mode == 0 ? LED_CN : LED_DN, m = mode == 0 ? b.id : id;
            atomicAdd(mode == 0 ? &b.n_placed : &b.n_recovered, n);
            atomicAdd((unsigned long long *)&w.ledger[row * MAXMAT + m], (unsigned long long)n);
        });
        if (tg < 0) continue;
        w.id[tg] = mode == 0 ? bodies[bi].id : (uint16_t)mt->id_air;
        w.col[tg] = mode == 0 ? bodies[bi].colour : 0u;
        w.sc[tg] = 0;
        w.fl[tg] = 0;
        w.df[tg] = 0;
        if (w.dirty) w.dirty[tg] = 1;
        claim[tg] = 0xffffffffu;  // every claimed cell has its lowest proposer as holder
        rem_local++;
    }
    if (mode == 1) {
        rem_local = (int)__reduce_add_sync(0xffffffffu, (unsigned)rem_local);
        if ((threadIdx.x & 31) == 0 && rem_local)
            atomicAdd((unsigned long long *)removed, (unsigned long long)rem_local);
    }
}

// stamp: the particle count with the displaced ones (one warp)
__global__ void k_obj_end(const WorldDev *wd, const int32_t *__restrict__ blk, int nblocks) {
    int n = 0;
    for (int k = threadIdx.x; k < nblocks; k += 32) n += blk[k];
    n = (int)__reduce_add_sync(0xffffffffu, (unsigned)n);
    if (threadIdx.x == 0) *wd->part_count = min(*wd->part_count + n, wd->part_cap);
}

// 1 bit per cell, LSB first: one warp vote per 32 cells
__global__ void k_obj_mask(const WorldDev *__restrict__ wd, const MatTable *__restrict__ mt, uint32_t *bits) {
    const WorldDev &w = *wd;
    const size_t n = (size_t)w.W * w.H;
    const size_t nwords = (n + 31) / 32;
    const int lane = threadIdx.x & 31;
    const size_t warp = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5;
    const size_t nwarps = ((size_t)gridDim.x * blockDim.x) >> 5;
    for (size_t wd_i = warp; wd_i < nwords; wd_i += nwarps) {
        size_t c = wd_i * 32 + lane;
        bool obj = c < n && mt_type(mt->a[w.id[c]]) == T_OBJECT;
        unsigned m = __ballot_sync(0xffffffffu, obj);
        if (lane == 0) bits[wd_i] = m;
    }
}

// ascending list of OBJECT cells from the mask: per-block word ranges, scanned
__global__ void k_obj_list_count(const uint32_t *bits, size_t nwords, int32_t *blk) {
    size_t seg = (nwords + gridDim.x - 1) / gridDim.x;
    size_t b0 = blockIdx.x * seg, b1 = min(nwords, b0 + seg);
    int c = 0;
    for (size_t i = b0 + threadIdx.x; i < b1; i += blockDim.x) c += __popc(bits[i]);
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    __shared__ int s[32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); k++) t += s[k];
        blk[blockIdx.x] = t;
    }
}
__global__ void k_obj_list_scan(int32_t *blk, int nb, long long *total) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        long long run = 0;
        for (int b = 0; b < nb; b++) {
            long long v = blk[b];
            blk[b] = (int32_t)run;
            run += v;
        }
        *total = run;
    }
}
__global__ void k_obj_list_scatter(const uint32_t *bits, size_t nwords, const int32_t *blk, uint32_t *out, long long cap) {
    size_t seg = (nwords + gridDim.x - 1) / gridDim.x;
    size_t b0 = blockIdx.x * seg, b1 = min(nwords, b0 + seg);
    __shared__ int s[32];
    __shared__ long long s_carry;
    if (threadIdx.x == 0) s_carry = blk[blockIdx.x];
    __syncthreads();
    for (size_t base = b0; base < b1; base += blockDim.x) {
        size_t i = base + threadIdx.x;
        uint32_t m = i < b1 ? bits[i] : 0u;
        int v = __popc(m);
        int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
        int inc = v;
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
        }
        if (lane == 31) s[wid] = inc;
        __syncthreads();
        long long pos = s_carry + inc - v;
        for (int k = 0; k < wid; k++) pos += s[k];
        while (m) {
            int b = __ffs(m) - 1;
            m &= m - 1;
            if (pos < cap) out[pos] = (uint32_t)(i * 32 + b);
            pos++;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            long long t = 0;
            for (int k = 0; k < nw; k++) t += s[k];
            s_carry += t;
        }
        __syncthreads();
    }
}

}  // namespace fse

using namespace fse;

static int obj_prepare(fse_world *w) {
    size_t n = (size_t)w->W * w->H;
    if (!w->claim) {
        if (device_alloc(&w->claim, n * 4) != cudaSuccess) {
            w->claim = nullptr;
            return FSE_E_NOMEM;
        }
        w->bytes += n * 4;
        // in the order of the world's stream, which does not wait for the default stream
        FSE_CUDA_TRY(cudaMemsetAsync(w->claim, 0xff, n * 4, w->stream));
    }
    return FSE_OK;
}

static int obj_run(fse_world *w, fse_body *bodies, int n, int mode, int64_t *out_removed) {
    if (!w || n < 0 || (n > 0 && !bodies)) return FSE_E_INVAL;
    int rc = ensure_materials_pushed();
    if (rc) return rc;
    rc = obj_prepare(w);
    if (rc) return rc;
    if (n == 0) {
        if (out_removed) *out_removed = 0;
        return FSE_OK;
    }
    std::vector<uint32_t> prefix(n + 1, 0);
    const MatTable &t = host_table();
    for (int b = 0; b < n; b++) {
        if (bodies[b].w < 0 || bodies[b].h <= 0 || bodies[b].id >= t.n) return FSE_E_INVAL;
        if (mode == 0) bodies[b].n_sand = bodies[b].n_soup = bodies[b].n_placed = 0;
        else bodies[b].n_recovered = 0;
        prefix[b + 1] = prefix[b] + (uint32_t)(bodies[b].w * bodies[b].h);
    }
    size_t total = prefix[n];
    // the call's workspace
    size_t bytes = 0;
    auto part = [&](size_t b) {
        const size_t at = bytes;
        bytes += (b + 255) & ~(size_t)255;
        return at;
    };
    const size_t o_b = part(n * sizeof(fse_body)), o_pref = part((size_t)(n + 1) * 4);
    const size_t o_tiles = part(total * sizeof(ObjTile)), o_held = part(total * 4);
    const size_t o_blk = part(OBJ_BLOCKS * 4), o_rem = part(8);
    CallScratch scr(w->stream);
    if (!scr.take(bytes)) return FSE_E_NOMEM;
    uint8_t *s = scr.p;
    fse_body *d_b = (fse_body *)(s + o_b);
    uint32_t *d_pref = (uint32_t *)(s + o_pref);
    ObjTile *d_tiles = (ObjTile *)(s + o_tiles);
    int32_t *d_held = (int32_t *)(s + o_held), *d_blk = (int32_t *)(s + o_blk);
    long long *d_rem = (long long *)(s + o_rem), rem = 0;
    cudaMemcpyAsync(d_b, bodies, n * sizeof(fse_body), cudaMemcpyHostToDevice, w->stream);
    cudaMemcpyAsync(d_pref, prefix.data(), (size_t)(n + 1) * 4, cudaMemcpyHostToDevice, w->stream);
    cudaMemsetAsync(d_rem, 0, 8, w->stream);
    const int wide = (int)std::max<size_t>(1, std::min<size_t>((total + 255) / 256, (size_t)sm_count() * 8));
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>((total + 1023) / 1024, OBJ_BLOCKS));
    k_obj_tiles<<<wide, 256, 0, w->stream>>>(w->d, g_dev_mt, d_b, d_pref, n, mode, d_tiles);
    k_obj_settle<<<wide, 256, 0, w->stream>>>(w->d, (uint32_t)total, d_tiles, w->claim);
    k_obj_held<<<wide, 256, 0, w->stream>>>(w->d, (uint32_t)total, d_tiles, w->claim, d_held);
    if (mode == 0)
        k_obj_count<<<blocks, 1024, 0, w->stream>>>(w->d, g_dev_mt, (uint32_t)total, d_held, d_blk);
    k_obj_apply<<<blocks, 1024, 0, w->stream>>>(w->d, g_dev_mt, d_b, d_pref, n, d_held, w->claim, mode, d_blk, d_rem);
    if (mode == 0) k_obj_end<<<1, 32, 0, w->stream>>>(w->d, d_blk, blocks);
    int result = cudaGetLastError() == cudaSuccess ? FSE_OK : FSE_E_CUDA;
    cudaMemcpyAsync(bodies, d_b, n * sizeof(fse_body), cudaMemcpyDeviceToHost, w->stream);
    cudaMemcpyAsync(&rem, d_rem, 8, cudaMemcpyDeviceToHost, w->stream);
    if (cudaStreamSynchronize(w->stream) != cudaSuccess) result = FSE_E_CUDA;
    if (out_removed) *out_removed = rem;
    if (result) return result;
    return fse_world_sync(w);
}

extern "C" {

int fse_object_stamp(fse_world *w, fse_body *bodies, int n) { return obj_run(w, bodies, n, 0, nullptr); }

int fse_object_readback(fse_world *w, fse_body *bodies, int n, int64_t *out_removed) {
    return obj_run(w, bodies, n, 1, out_removed);
}

static int obj_mask_dev(fse_world *w) {
    size_t n = (size_t)w->W * w->H;
    size_t nwords = (n + 31) / 32;
    if (!w->mask_bits) {
        if (device_alloc(&w->mask_bits, nwords * 4) != cudaSuccess) {
            w->mask_bits = nullptr;
            return FSE_E_NOMEM;
        }
        w->bytes += nwords * 4;
    }
    int rc = ensure_materials_pushed();
    if (rc) return rc;
    int blocks = (int)std::min<size_t>((nwords * 32 + 255) / 256, (size_t)sm_count() * 8);
    k_obj_mask<<<std::max(blocks, 1), 256, 0, w->stream>>>(w->d, g_dev_mt, (uint32_t *)w->mask_bits);
    return cudaGetLastError() == cudaSuccess ? FSE_OK : FSE_E_CUDA;
}

int fse_object_mask_export(fse_world *w, uint8_t *host_bits) {
    if (!w || !host_bits) return FSE_E_INVAL;
    int rc = obj_mask_dev(w);
    if (rc) return rc;
    size_t n = (size_t)w->W * w->H;
    FSE_CUDA_TRY(cudaMemcpyAsync(host_bits, w->mask_bits, (n + 7) / 8, cudaMemcpyDeviceToHost, w->stream));
    FSE_CUDA_TRY(cudaStreamSynchronize(w->stream));
    return FSE_OK;
}

int fse_object_list_export(fse_world *w, uint32_t *host_idx, int64_t cap, int64_t *out_n) {
    if (!w || cap < 0 || (cap > 0 && !host_idx)) return FSE_E_INVAL;
    int rc = obj_mask_dev(w);
    if (rc) return rc;
    size_t n = (size_t)w->W * w->H, nwords = (n + 31) / 32;
    const int NB = 256;
    if (!w->obj_n) {
        if (device_alloc(&w->obj_n, 8 + (NB + 1) * 4) != cudaSuccess) return FSE_E_NOMEM;
    }
    int32_t *blk = (int32_t *)((char *)w->obj_n + 8);
    long long cap_dev = std::max<long long>(cap, 1);
    if (!w->obj_list || w->obj_list_cap < (size_t)cap_dev) {
        if (w->obj_list) cudaFree(w->obj_list);
        if (device_alloc(&w->obj_list, (size_t)cap_dev * 4) != cudaSuccess) {
            w->obj_list = nullptr;
            w->obj_list_cap = 0;
            return FSE_E_NOMEM;
        }
        w->obj_list_cap = (size_t)cap_dev;
    }
    k_obj_list_count<<<NB, 256, 0, w->stream>>>((uint32_t *)w->mask_bits, nwords, blk);
    k_obj_list_scan<<<1, 32, 0, w->stream>>>(blk, NB, (long long *)w->obj_n);
    k_obj_list_scatter<<<NB, 256, 0, w->stream>>>((uint32_t *)w->mask_bits, nwords, blk, w->obj_list, cap);
    long long total = 0;
    FSE_CUDA_TRY(cudaMemcpyAsync(&total, w->obj_n, 8, cudaMemcpyDeviceToHost, w->stream));
    FSE_CUDA_TRY(cudaStreamSynchronize(w->stream));
    long long m = std::min<long long>(total, cap);
    if (m > 0) {
        FSE_CUDA_TRY(cudaMemcpyAsync(host_idx, w->obj_list, (size_t)m * 4, cudaMemcpyDeviceToHost, w->stream));
        FSE_CUDA_TRY(cudaStreamSynchronize(w->stream));
    }
    if (out_n) *out_n = total;
    return FSE_OK;
}

}  // extern "C"
