// verify.cu -- manifold labels by tile roots and pointer jumping, and
// re-verification.
//
// Replaces PathCompression (pMSz.cu:255-271): the reference walks every
// vertex's pointer chain to its root one step at a time.  Here the chains are
// shortened where memory is near first:
//   k_tile_roots  every 32 x 16 x 16 tile resolves its chains in shared memory:
//                 a voxel's label becomes its local root, an extremum or a
//                 voxel whose neighbour lies in another tile (an exit); an
//                 exit's label is that neighbour, and exits are listed
//   k_exit_walk   every listed exit walks on, from tile to tile, to its root
//   k_finish      every voxel takes its local root's label
// Global memory sees each code once, each label twice and one gather per
// voxel, which its tile shares; the walks start from the few percent of voxels
// that are exits.  Whole-field three-hop jumping (k_jump) needed five launches
// over all voxels and a host read after each: 32.4 M voxels, codes and both label
// kinds as int64, 1850 -> 722 us.  It remains as the general form, for fields a few
// voxels thick and for what the walks leave: a flag tells the host, the labels
// so far are valid ancestors, and jumping goes on from them to the fixpoint.
// Chains beyond one walk's bound are walked on first, where the labels are not
// yet finished.
//
// Verification replaces the reference's disabled check_consistency block
// (pMSz.cu:3038-3126) and count_false_cases (pMSz.cu:1852-1870).
#include "common.cuh"
#include "internal.h"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace pmsz {

__global__ void __launch_bounds__(256) k_init_ptr(const uint8_t *__restrict__ codes, uint32_t *__restrict__ as,
                                                  uint32_t *__restrict__ ds, Geom g) {
    const int x = blockIdx.x * 32 + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int z = blockIdx.z;
    if (x >= g.nx || y >= g.ny) return;
    const size_t i = flat(g, x, y, z);
    const uint8_t c = codes[i];
    const int a = c & 15, d = c >> 4;
    const uint32_t valid = valid_mask(x, y, z, g.nx, g.ny, g.nz);
    auto target = [&](int r) {  // a step out of the domain (not the codes of a field) stays put
        return static_cast<uint32_t>((valid >> r) & 1u ? flat(g, x + rank_dx(r), y + rank_dy(r), z + rank_dz(r)) : i);
    };
    if (as) as[i] = target(a);
    if (ds) ds[i] = target(d);
}

__global__ void __launch_bounds__(256) k_jump(uint32_t *__restrict__ L, size_t n, unsigned int *changed,
                                              int rounds) {
    bool any = false;
    const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint32_t l = L[i];
        bool moved = false;
        for (int r = 0; r < rounds; ++r) {
            const uint32_t ll = L[l];
            if (ll == l) break;
            // three hops: a pointer spanning d chain steps now spans at least 3d
            l = L[ll];
            moved = true;
        }
        if (moved) {
            L[i] = l;
            any = true;
        }
    }
    if (__any_sync(0xFFFFFFFFu, any) && (threadIdx.x & 31) == 0) atomicOr(changed, 1u);
}

static inline unsigned grid_for(size_t n) {
    return static_cast<unsigned>(std::max<size_t>(1, std::min<size_t>((n + 255) / 256, 152 * 16)));
}

// The labels of `kinds` arrays to their roots: together, with one read-back a round,
// where they share the 129 MB L2, else one after the other (17 M voxels, both kinds
// of a ramp: 564 us, together 595; 20 000 voxels 150 and 120).
static int jump_to_roots(uint32_t *const *L, int kinds, size_t n, unsigned int *d_flag, cudaStream_t s, int rounds) {
    if (kinds > 1 && kinds * n * sizeof(uint32_t) > (static_cast<size_t>(64) << 20)) {
        for (int l = 0; l < kinds; ++l) {
            const int rc = jump_to_roots(L + l, 1, n, d_flag, s, rounds);
            if (rc) return rc;
        }
        return PMSZ_OK;
    }
    unsigned int *h = static_cast<unsigned int *>(host_pinned(sizeof(unsigned int)));
    if (!h) return set_error(PMSZ_ERR_OOM, "pinned host allocation failed");
    for (int launch = 0; launch < 64; ++launch) {
        PMSZ_CUDA(cudaMemsetAsync(d_flag, 0, sizeof(unsigned int), s));
        for (int l = 0; l < kinds; ++l) k_jump<<<grid_for(n), 256, 0, s>>>(L[l], n, d_flag, rounds);
        PMSZ_CUDA(cudaGetLastError());
        PMSZ_CUDA(cudaMemcpyAsync(h, d_flag, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
        PMSZ_CUDA(cudaStreamSynchronize(s));
        if (*h == 0) return PMSZ_OK;
    }
    return set_error(PMSZ_ERR_CUDA, "pointer jumping did not reach its fixpoint");
}

constexpr int kLX = 32, kLY = 16, kLZ = 16, kLTile = kLX * kLY * kLZ;
constexpr int kLWarps = 16, kLThreads = 32 * kLWarps;
constexpr uint32_t kLShell = kLTile - (kLX - 2) * (kLY - 2) * (kLZ - 2);  // most exits a tile can have
constexpr int kWalkHops = 64;  // hops of an exit per launch (two per tile crossed)
constexpr int kWalks = 8;      // launches: each goes on from where the last one's chains ended
constexpr unsigned int kOpen = 1, kCycle = 2;  // flags: a walk ran out of hops; a chain in a tile does not end

struct TileGrid {
    dim3 grid;         // tiles
    uint32_t stride;   // list entries per tile
    size_t tiles() const { return static_cast<size_t>(grid.x) * grid.y * grid.z; }
};
static TileGrid tile_grid(const Geom &g) {
    TileGrid t;
    t.grid = dim3(static_cast<unsigned>((g.nx + kLX - 1) / kLX), static_cast<unsigned>((g.ny + kLY - 1) / kLY),
                  static_cast<unsigned>((g.nz + kLZ - 1) / kLZ));
    t.stride = std::min<uint32_t>(kLShell, static_cast<uint32_t>(std::min(g.nx, kLX) * std::min(g.ny, kLY) * std::min(g.nz, kLZ)));
    return t;
}

template <int NL>
struct TileRootsSmem {
    uint16_t p[NL][kLTile];   // twice the local index of a voxel's pointer: its byte offset here
    uint16_t exits[NL][kLShell];  // local indices
    uint32_t n[NL];
};

// One block of 16 warps per tile; warp w owns the row y = w of every plane (with
// 8 warps and two rows each the chase has half the chains in flight: both
// labels of 32 M voxels 545 us, now 494); planes beyond the field are left out.
// L[l][i] receives the label so far of nibble lo[l] (0: ascent, 4: descent),
// exits[l] the tile's exits (global indices) and count[l] their number.  *flag is set if a chain does not end within the tile's voxel count
// (a cycle: not the codes of a field).  gate (or null): nothing is done where it is
// set.  Bound by shared-memory latency and
// conflicts of the pointer chase (L1 78 % busy, issue 63 %): pointers are stored
// as byte offsets, steps come from a shuffle, the in-tile test from rank masks,
// and exits are handled by full warps behind the loop.  71.5 M voxels, one kind, with 8
// warps: 250 us and 87 warp instructions per voxel (312 us and 152 with
// coordinates decoded per voxel and exits handled in the loop).
template <int NL>
__global__ void __launch_bounds__(kLThreads) k_tile_roots(const uint8_t *__restrict__ codes, uint32_t *__restrict__ l0,
                                                          uint32_t *__restrict__ l1, int lo0, int lo1,
                                                          uint32_t *__restrict__ exits0, uint32_t *__restrict__ exits1,
                                                          uint32_t stride, uint32_t *__restrict__ count0,
                                                          uint32_t *__restrict__ count1, unsigned int *flag,
                                                          const unsigned int *gate, Geom g) {
    if (gate && *gate) return;
    constexpr int NW = kLWarps, H = kLY / NW;  // rows of a plane per thread
    __shared__ TileRootsSmem<NL> sm;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int x0 = blockIdx.x * kLX, y0 = blockIdx.y * kLY, z0 = blockIdx.z * kLZ;
    const int ex = min(kLX, g.nx - x0), ey = min(kLY, g.ny - y0), ez = min(kLZ, g.nz - z0);  // the tile's extent
    const uint32_t sy = static_cast<uint32_t>(g.nx), sz = static_cast<uint32_t>(g.nx) * static_cast<uint32_t>(g.ny);
    const uint32_t origin = static_cast<uint32_t>(x0) + sy * static_cast<uint32_t>(y0) + sz * static_cast<uint32_t>(z0);
    const uint32_t tile = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    auto at = [&](int l, uint32_t off) -> uint16_t & {
        return *reinterpret_cast<uint16_t *>(reinterpret_cast<unsigned char *>(sm.p[l]) + off);
    };
    if (threadIdx.x < NL) sm.n[threadIdx.x] = 0;
    __syncthreads();
    // lane r: the step of rank r, in bytes; ranks whose target lies in the tile.
    // A nibble of 15 (no rank, and not the code of a field) stays put, which is
    // in the tile: only voxels of its shell are exits, at most kLShell.
    constexpr uint32_t kStay = kAllValid | 1u << 15;
    const int r16 = lane & 15;
    const int step = r16 < 15 ? 2 * (rank_dx(r16) + kLX * rank_dy(r16) + kLX * kLY * rank_dz(r16)) : 0;
    const uint32_t xmask = kStay & ~(lane == 0 ? kNegX : 0u) & ~(lane + 1 >= ex ? kPosX : 0u);
    uint32_t ymask[H];
    bool in_row[H];
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const int y = w + NW * h;
        ymask[h] = xmask & ~(y == 0 ? kNegY : 0u) & ~(y + 1 >= ey ? kPosY : 0u);
        in_row[h] = lane < ex && y < ey;
    }
    const uint32_t v0 = static_cast<uint32_t>(lane + kLX * w);                       // row w of plane 0
    const uint32_t i0 = origin + static_cast<uint32_t>(lane) + sy * static_cast<uint32_t>(w);
#pragma unroll 4
    for (int z = 0; z < ez; ++z) {
        const uint32_t zmask = kStay & ~(z == 0 ? kNegZ : 0u) & ~(z + 1 >= ez ? kPosZ : 0u);
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const uint32_t v = v0 + static_cast<uint32_t>(kLX * NW * h + kLX * kLY * z);
            const uint32_t c = in_row[h] ? codes[i0 + sy * static_cast<uint32_t>(NW * h) + sz * static_cast<uint32_t>(z)] : 0x77u;
            const uint32_t mask = ymask[h] & zmask;
#pragma unroll
            for (int l = 0; l < NL; ++l) {
                const uint32_t r = (c >> (l == 0 ? lo0 : lo1)) & 15u;
                const int s = __shfl_sync(0xFFFFFFFFu, step, static_cast<int>(r));
                const bool inside = ((mask >> r) & 1u) != 0u;
                at(l, 2 * v) = static_cast<uint16_t>(static_cast<int>(2 * v) + (inside ? s : 0));
                // a step out of the tile (or of the domain: found below)
                if (!inside) sm.exits[l][atomicAdd(&sm.n[l], 1u)] = static_cast<uint16_t>(v);
            }
        }
    }
    __syncthreads();
    // in place: whatever a concurrent reader sees is an ancestor
#pragma unroll 1
    for (int round = 0; round < 2; ++round) {
#pragma unroll 8
        for (int k = 0; k < H * ez; ++k) {
            const uint32_t off = 2 * v0 + static_cast<uint32_t>(2 * kLX * NW * k);
#pragma unroll
            for (int l = 0; l < NL; ++l) at(l, off) = at(l, at(l, at(l, off)));
        }
        __syncthreads();
    }
    bool stuck = false;
#pragma unroll 2
    for (int k = 0; k < H * ez; ++k) {
        const int z = k / H;
        const uint32_t off = 2 * v0 + static_cast<uint32_t>(2 * kLX * NW * k);
        const bool in = in_row[k % H];
        const uint32_t i = i0 + sy * static_cast<uint32_t>(NW * (k % H)) + sz * static_cast<uint32_t>(z);
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            uint32_t p = at(l, off), q = at(l, p);
            if (q != p) {  // rare after the two rounds
                int hops = 0;
                do {
                    p = q;
                    q = at(l, p);
                } while (q != p && ++hops < kLTile);
                at(l, off) = static_cast<uint16_t>(p);
                stuck |= q != p;
            }
            // (an exit's label is written below)
            if (in) (l == 0 ? l0 : l1)[i] = origin + ((p >> 1) & 31u) + sy * ((p >> 6) & 15u) + sz * (p >> 10);
        }
    }
    if (stuck) atomicOr(flag, kCycle);
    __syncthreads();  // the exits' labels come after the loop's
    // dx + 1, dy + 1, dz + 1 of every rank, two bits each (nibble 15 is no exit)
    constexpr auto steps = [](int axis) {
        uint32_t t = 1u << 30;
        for (int r = 0; r < 15; ++r)
            t |= static_cast<uint32_t>((axis == 0 ? rank_dx(r) : axis == 1 ? rank_dy(r) : rank_dz(r)) + 1) << (2 * r);
        return t;
    };
    constexpr uint32_t tx = steps(0), ty = steps(1), tz = steps(2);
#pragma unroll
    for (int l = 0; l < NL; ++l) {
        uint32_t *L = l == 0 ? l0 : l1;
        uint32_t *list = (l == 0 ? exits0 : exits1) + static_cast<size_t>(tile) * stride;
        for (uint32_t j = threadIdx.x; j < sm.n[l]; j += kLThreads) {
            const uint32_t v = sm.exits[l][j];
            const int x = x0 + static_cast<int>(v & 31u), y = y0 + static_cast<int>((v >> 5) & 15u),
                      z = z0 + static_cast<int>(v >> 9);
            const uint32_t i = static_cast<uint32_t>(x) + sy * static_cast<uint32_t>(y) + sz * static_cast<uint32_t>(z);
            const uint32_t r2 = 2u * ((static_cast<uint32_t>(codes[i]) >> (l == 0 ? lo0 : lo1)) & 15u);
            const int gx = x + static_cast<int>((tx >> r2) & 3u) - 1, gy = y + static_cast<int>((ty >> r2) & 3u) - 1,
                      gz = z + static_cast<int>((tz >> r2) & 3u) - 1;
            uint32_t label = i;
            if (static_cast<unsigned>(gx) < static_cast<unsigned>(g.nx) && static_cast<unsigned>(gy) < static_cast<unsigned>(g.ny) &&
                static_cast<unsigned>(gz) < static_cast<unsigned>(g.nz))
                label = static_cast<uint32_t>(gx) + sy * static_cast<uint32_t>(gy) + sz * static_cast<uint32_t>(gz);
            L[i] = label;
            list[j] = i;
        }
    }
    if (threadIdx.x == 0) {
        count0[tile] = sm.n[0];
        if (NL == 2) count1[tile] = sm.n[NL - 1];
    }
}

// Every exit of a tile (one block for each kind of label, blockIdx.y) walks to
// its root; *flag is set where the hops run out.
__global__ void __launch_bounds__(512) k_exit_walk(uint32_t *l0, uint32_t *l1, const uint32_t *__restrict__ exits0,
                                                   const uint32_t *__restrict__ exits1, uint32_t stride,
                                                   const uint32_t *__restrict__ count0,
                                                   const uint32_t *__restrict__ count1, unsigned int *flag,
                                                   const unsigned int *gate) {
    if (gate && *gate) return;
    uint32_t *L = blockIdx.y ? l1 : l0;
    const uint32_t m = (blockIdx.y ? count1 : count0)[blockIdx.x];
    const uint32_t *list = (blockIdx.y ? exits1 : exits0) + static_cast<size_t>(blockIdx.x) * stride;
    bool open = false;
    for (uint32_t j = threadIdx.x; j < m; j += blockDim.x) {
        const uint32_t e = list[j];
        uint32_t l = L[e];
        int hop = 0;
        for (; hop < kWalkHops; ++hop) {
            const uint32_t n = L[l];
            if (n == l) break;
            l = n;
        }
        L[e] = l;
        open |= hop == kWalkHops;
    }
    if (__any_sync(0xFFFFFFFFu, open) && (threadIdx.x & 31) == 0) atomicOr(flag, kOpen);
}

// Every voxel's label: that of its local root (roots and exits already hold
// theirs).  OUT: the labels' type; uint32_t may be in place.  Four voxels per
// thread and step, so that their gathers are in flight together.
template <typename OUT>
__global__ void __launch_bounds__(256) k_finish(const uint32_t *L, OUT *out, size_t n) {
    const size_t step = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i0 = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < n; i0 += 4 * step) {
        uint32_t a[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] = i0 + j * step < n ? L[i0 + j * step] : 0u;
#pragma unroll
        for (int j = 0; j < 4; ++j) a[j] = L[a[j]];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (i0 + j * step < n) out[i0 + j * step] = static_cast<OUT>(a[j]);
    }
}

// Scratch and launches of one label computation; AS first where both are asked.
struct LabelRun {
    Geom g;
    TileGrid t;
    uint32_t *L[2] = {nullptr, nullptr};
    int lo[2] = {0, 4};
    int nl = 0;
    uint32_t *lists = nullptr;      // per label kind: the tiles' counts, then their exits
    unsigned int *flag = nullptr, *jump = nullptr;  // chains beyond the bounds; the jumping's
    static size_t list_words(const TileGrid &t) { return t.tiles() * (static_cast<size_t>(t.stride) + 1); }
    uint32_t *counts(int l) const { return lists + static_cast<size_t>(l) * list_words(t); }
    uint32_t *exits(int l) const { return counts(l) + t.tiles(); }
    // Lines, and fields a few rows thick: a tile holds 16 to 96 voxels, and
    // nearly every chain leaves its tile.  They go to the general jumping at once
    // (2 M voxels in a line: codes and labels 694 us by tiles, 562 so; 500 000 along
    // y verified, 986 and 720; a plane of 2048 x 2000: 206 by tiles, 577 so).
    static bool general(const Geom &g) {
        const int rows = std::min(g.ny, kLY) * std::min(g.nz, kLZ);
        return rows < 4 || rows * std::min(g.nx, kLX) <= 16;
    }
    int init(const uint8_t *codes, cudaStream_t s) {  // every voxel's neighbour
        const dim3 grid(static_cast<unsigned>(g.wpr), static_cast<unsigned>((g.ny + 7) / 8), static_cast<unsigned>(g.nz));
        k_init_ptr<<<grid, dim3(32, 8, 1), 0, s>>>(codes, lo[0] == 0 ? L[0] : nullptr, nl == 2 ? L[1] : lo[0] == 4 ? L[0] : nullptr, g);
        PMSZ_CUDA(cudaGetLastError());
        return PMSZ_OK;
    }
    int tile_roots(const uint8_t *codes, const unsigned int *gate, cudaStream_t s) {  // *flag |= 1 where chains go on
        if (nl == 2)
            k_tile_roots<2><<<t.grid, kLThreads, 0, s>>>(codes, L[0], L[1], lo[0], lo[1], exits(0), exits(1), t.stride,
                                                         counts(0), counts(1), flag, gate, g);
        else
            k_tile_roots<1><<<t.grid, kLThreads, 0, s>>>(codes, L[0], nullptr, lo[0], 0, exits(0), nullptr, t.stride,
                                                         counts(0), nullptr, flag, gate, g);
        return walk(flag, gate, s);
    }
    int walk(unsigned int *f, const unsigned int *gate, cudaStream_t s) {  // one more walk of the exits
        const int last = nl - 1;
        k_exit_walk<<<dim3(static_cast<unsigned>(t.tiles()), static_cast<unsigned>(nl)), 512, 0, s>>>(
            L[0], L[last], exits(0), exits(last), t.stride, counts(0), counts(last), f, gate);
        PMSZ_CUDA(cudaGetLastError());
        return PMSZ_OK;
    }
    int roots(const uint8_t *codes, cudaStream_t s) {  // everything up to k_finish
        PMSZ_CUDA(cudaMemsetAsync(flag, 0, sizeof(unsigned int), s));
        if (!general(g)) return tile_roots(codes, nullptr, s);
        const int rc = init(codes, s);
        if (rc) return rc;
        PMSZ_CUDA(cudaMemsetAsync(flag, 1, 1, s));  // (little-endian int 1)
        return PMSZ_OK;
    }
    template <typename OUT>
    int finish(int l, OUT *out, cudaStream_t s) {
        k_finish<OUT><<<grid_for((g.n + 3) / 4), 256, 0, s>>>(L[l], out, g.n);
        PMSZ_CUDA(cudaGetLastError());
        return PMSZ_OK;
    }
    // Chains beyond the walks' bounds, of `m` runs that have not been finished: more
    // walks of their exits, each from the last one's ends (so 64 times as far), until
    // none is open (*left 0) or, as on a cycle, for kWalks launches.  The other
    // voxels need none: 8 M voxels in a ramp 4 x 4 wide, verified, 1850 us by jumping,
    // 1488 so; 17 M of 64 planes 1502 and 1256.
    static int walk_on(LabelRun *r, int m, unsigned int *left, cudaStream_t s) {
        unsigned int *h = static_cast<unsigned int *>(host_pinned(sizeof(unsigned int)));
        if (!h) return set_error(PMSZ_ERR_OOM, "pinned host allocation failed");
        for (int launch = 0; launch < kWalks; ++launch) {
            int rc;
            PMSZ_CUDA(cudaMemsetAsync(r->jump, 0, sizeof(unsigned int), s));
            for (int k = 0; k < m; ++k)
                if ((rc = r[k].walk(r->jump, nullptr, s))) return rc;
            PMSZ_CUDA(cudaMemcpyAsync(h, r->jump, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
            PMSZ_CUDA(cudaStreamSynchronize(s));
            *left = *h;
            if (!*left) break;
        }
        return PMSZ_OK;
    }
    // The general jumping, from the labels so far.
    int complete(cudaStream_t s, int rounds) { return jump_to_roots(L, nl, g.n, jump, s, rounds); }
};

template <typename OUT>
static int labels_run(const uint8_t *codes, size_t nx, size_t ny, size_t nz, OUT *as, OUT *ds, cudaStream_t s) {
    if (!codes) return set_error(PMSZ_ERR_ARG, "null codes pointer");
    int rc = check_geom(nx, ny, nz);
    if (rc) return rc;
    LabelRun r;
    r.g = make_geom(nx, ny, nz);
    if (r.g.n >= (static_cast<size_t>(1) << 32)) return set_error(PMSZ_ERR_ARG, "labels need fewer than 2^32 voxels");
    if (!as && !ds) return PMSZ_OK;
    constexpr bool kInPlace = sizeof(OUT) == 4;
    OUT *out[2] = {as ? as : ds, ds};
    r.nl = as && ds ? 2 : 1;
    r.lo[0] = as ? 0 : 4;
    r.t = tile_grid(r.g);
    Workspace ws(s);
    const size_t o_w = ws.reserve<unsigned int>(2), o_e = ws.reserve<uint32_t>(LabelRun::list_words(r.t) * r.nl);
    const size_t o_l = ws.reserve<uint32_t>(kInPlace ? 0 : r.g.n * r.nl);
    if ((rc = ws.commit())) return rc;
    r.flag = ws.at<unsigned int>(o_w);
    r.jump = r.flag + 1;
    r.lists = ws.at<uint32_t>(o_e);
    for (int l = 0; l < r.nl; ++l)
        r.L[l] = kInPlace ? reinterpret_cast<uint32_t *>(out[l]) : ws.at<uint32_t>(o_l) + static_cast<size_t>(l) * r.g.n;
    unsigned int *h = static_cast<unsigned int *>(host_pinned(sizeof(unsigned int)));
    if (!h) return set_error(PMSZ_ERR_OOM, "pinned host allocation failed");
    if ((rc = r.roots(codes, s))) return rc;
    PMSZ_CUDA(cudaMemcpyAsync(h, r.flag, sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    for (int l = 0; l < r.nl; ++l)
        if ((rc = r.finish<OUT>(l, out[l], s))) return rc;
    PMSZ_CUDA(cudaStreamSynchronize(s));
    if (unsigned int left = *h) {
        if (!kInPlace && !LabelRun::general(r.g) && left == kOpen && (rc = LabelRun::walk_on(&r, 1, &left, s))) return rc;
        if (left && (rc = r.complete(s, tuned_jump_rounds(nx, ny, nz)))) return rc;
        for (int l = 0; l < r.nl && !kInPlace; ++l)
            if ((rc = r.finish<OUT>(l, out[l], s))) return rc;
    }
    return ws.release();
}

int labels_impl(const uint8_t *codes, size_t nx, size_t ny, size_t nz, uint32_t *as, uint32_t *ds, cudaStream_t s) {
    return labels_run<uint32_t>(codes, nx, ny, nz, as, ds, s);
}

static LabelRun both_kinds(size_t nx, size_t ny, size_t nz, uint32_t *as, uint32_t *ds, uint32_t *lists,
                           unsigned int *words) {
    LabelRun r;
    r.g = make_geom(nx, ny, nz);
    r.t = tile_grid(r.g);
    r.L[0] = as;
    r.L[1] = ds;
    r.nl = 2;
    r.lists = lists;
    r.flag = words;
    r.jump = words + 1;
    return r;
}
size_t label_list_words(size_t nx, size_t ny, size_t nz) {
    return 2 * LabelRun::list_words(tile_grid(make_geom(nx, ny, nz)));
}
int labels_roots(const uint8_t *codes, size_t nx, size_t ny, size_t nz, uint32_t *as, uint32_t *ds, uint32_t *lists,
                 unsigned int *words, cudaStream_t s) {
    return both_kinds(nx, ny, nz, as, ds, lists, words).roots(codes, s);
}
int labels_finish(size_t nx, size_t ny, size_t nz, uint32_t *as, uint32_t *ds, cudaStream_t s) {
    LabelRun r = both_kinds(nx, ny, nz, as, ds, nullptr, nullptr);
    const int rc = r.finish<uint32_t>(0, as, s);
    return rc ? rc : r.finish<uint32_t>(1, ds, s);
}
int labels_complete(size_t nx, size_t ny, size_t nz, uint32_t *as, uint32_t *ds, unsigned int *words, cudaStream_t s) {
    return both_kinds(nx, ny, nz, as, ds, nullptr, words).complete(s, tuned_jump_rounds(nx, ny, nz));
}

int time_jump_rounds(const uint8_t *codes, size_t nx, size_t ny, size_t nz, const int *rounds, int m, float *ms,
                     cudaStream_t s) {
    const Geom g = make_geom(nx, ny, nz);
    for (int k = 0; k < m; ++k) ms[k] = 0.f;
    if (g.n >= (static_cast<size_t>(1) << 32)) return PMSZ_OK;  // no labels at this size
    Workspace ws(s);
    const size_t o_l = ws.reserve<uint32_t>(g.n), o_flag = ws.reserve<unsigned int>(1);
    int rc = ws.commit();
    if (rc) return rc;
    uint32_t *L = ws.at<uint32_t>(o_l);
    EventTimer et;
    if ((rc = et.init())) return rc;
    const dim3 grid(static_cast<unsigned>(g.wpr), static_cast<unsigned>((g.ny + 7) / 8), static_cast<unsigned>(g.nz));
    for (int k = 0; k < m; ++k) {
        float best = 0.f;
        for (int rep = 0; rep < 3; ++rep) {  // the first run of each candidate is a warm-up
            k_init_ptr<<<grid, dim3(32, 8, 1), 0, s>>>(codes, L, nullptr, g);
            PMSZ_CUDA(cudaEventRecord(et.ev[0], s));
            if ((rc = jump_to_roots(&L, 1, g.n, ws.at<unsigned int>(o_flag), s, rounds[k]))) return rc;
            PMSZ_CUDA(cudaEventRecord(et.ev[1], s));
            PMSZ_CUDA(cudaEventSynchronize(et.ev[1]));
            float t = 0.f;
            PMSZ_CUDA(cudaEventElapsedTime(&t, et.ev[0], et.ev[1]));
            if (rep > 0 && (best == 0.f || t < best)) best = t;
        }
        ms[k] = best;
    }
    return ws.release();
}

// Voxels whose labels differ, the labels of both fields finished on the way
// (hop: L holds local roots as before k_finish; else the labels themselves);
// nothing where *gate is set.
__global__ void __launch_bounds__(256) k_count_diff(const uint32_t *__restrict__ a, const uint32_t *__restrict__ b,
                                                    size_t n, int hop, const unsigned int *gate, unsigned long long *out) {
    if (gate && *gate) return;
    constexpr int kPer = 8;
    uint32_t c = 0;
    const size_t step = static_cast<size_t>(gridDim.x) * blockDim.x;
    for (size_t i0 = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < n; i0 += kPer * step) {
        uint32_t u[kPer], v[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const size_t i = i0 + j * step;
            u[j] = i < n ? a[i] : 0u;
            v[j] = i < n ? b[i] : 0u;
        }
        if (hop) {
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                u[j] = a[u[j]];
                v[j] = b[v[j]];
            }
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) c += i0 + j * step < n && u[j] != v[j];
    }
    c = warp_sum_u32(c);
    if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, (unsigned long long)c);
}

template <typename T>
int verify_impl(const T *f, const T *fp, size_t nx, size_t ny, size_t nz, double eb, pmsz_verify_result *out,
                cudaStream_t s) {
    if (!f || !fp || !out) return set_error(PMSZ_ERR_ARG, "null pointer");
    int rc = check_geom(nx, ny, nz);
    if (rc) return rc;
    const Geom g = make_geom(nx, ny, nz);
    const bool with_labels = g.n < (static_cast<size_t>(1) << 32);
    const TileGrid tiles = tile_grid(g);
    Workspace ws(s);
    const size_t o_c0 = ws.reserve<uint8_t>(g.n), o_c1 = ws.reserve<uint8_t>(g.n);
    const size_t o_l0 = ws.reserve<uint32_t>(with_labels ? g.n : 0), o_l1 = ws.reserve<uint32_t>(with_labels ? g.n : 0);
    const size_t o_e = ws.reserve<uint32_t>(with_labels ? 2 * LabelRun::list_words(tiles) : 0), o_w = ws.reserve<unsigned int>(3);
    const size_t o_cnt = ws.reserve<unsigned long long>(9);
    if ((rc = ws.commit())) return rc;
    uint8_t *c0 = ws.at<uint8_t>(o_c0), *c1 = ws.at<uint8_t>(o_c1);
    unsigned long long *cnt = ws.at<unsigned long long>(o_cnt);
    constexpr size_t kCounts = 9 * sizeof(unsigned long long);
    unsigned long long *h = static_cast<unsigned long long *>(host_pinned(kCounts + 2 * sizeof(unsigned int)));
    if (!h) return set_error(PMSZ_ERR_OOM, "pinned host allocation failed");
    PMSZ_CUDA(cudaMemsetAsync(cnt, 0, kCounts, s));
    const T eps = static_cast<T>(eb);
    uint64_t sure = 0;
    if (eps > T(0) && std::isfinite(eps)) {
        if (sizeof(T) == 8) std::memcpy(&sure, &eps, 8);
        else std::memcpy(&sure, &eps, 4);  // little-endian: the low word
    }
    // cnt: codes, extrema, beyond the bound, beyond the clamp, some ascent, some
    // descent differ; then the label mismatches of either kind, and the copies' flag
    if ((rc = pair_impl<T>(f, fp, nx, ny, nz, eps, sure, c0, c1, cnt, reinterpret_cast<uint32_t *>(cnt + 8), s))) return rc;
    PMSZ_CUDA(cudaMemcpyAsync(h, cnt, kCounts, cudaMemcpyDeviceToHost, s));
    PMSZ_CUDA(cudaStreamSynchronize(s));
    unsigned long long got[9];  // what follows reads back through the same pinned block
    std::memcpy(got, h, kCounts);
    if (got[8]) return set_error(PMSZ_ERR_CUDA, "verification: a tile plane's tensor copy did not arrive within the bounded wait");
    // A label is the end of a voxel's chain of steepest neighbours, so fields
    // whose directions agree at every voxel have the same labels: a kind is
    // labelled only if some direction of it differs.  A corrected field, the
    // usual one to be checked, agrees in all of them (71.5 M voxels fp64 2809 ->
    // 1017 us, and 727 with both codes and the comparison in one pass); reading
    // that back first costs the others 15 us.
    const bool wanted[2] = {with_labels && got[4] != 0, with_labels && got[5] != 0};
    // AS, then DS labels of both fields in the same two arrays
    uint32_t *const L[2] = {ws.at<uint32_t>(o_l0), ws.at<uint32_t>(o_l1)};
    unsigned int *flags = ws.at<unsigned int>(o_w);  // per kind: chains go on beyond the walks' bounds; then the jumping's
    auto run_of = [&](int kind, int field) {
        LabelRun r;
        r.g = g;
        r.nl = 1;
        r.lo[0] = 4 * kind;
        r.L[0] = L[field];
        r.t = tiles;
        r.lists = ws.at<uint32_t>(o_e) + static_cast<size_t>(field) * LabelRun::list_words(tiles);
        r.flag = flags + kind;
        r.jump = flags + 2;
        return r;
    };
    auto count = [&](int kind, int hop, const unsigned int *gate) -> int {
        k_count_diff<<<grid_for((g.n + 3) / 4), 256, 0, s>>>(L[0], L[1], g.n, hop, gate, cnt + 6 + kind);
        PMSZ_CUDA(cudaGetLastError());
        return PMSZ_OK;
    };
    auto walk = [&](int kind, const unsigned int *gate) -> int {
        for (int field = 0; field < 2; ++field)
            if ((rc = run_of(kind, field).tile_roots(field ? c1 : c0, gate, s))) return rc;
        return count(kind, 1, gate);
    };
    auto go_on = [&](int kind, bool tiled) -> int {  // from the labels so far to the end
        unsigned int left = kOpen;
        LabelRun r[2] = {run_of(kind, 0), run_of(kind, 1)};
        if (tiled && (rc = LabelRun::walk_on(r, 2, &left, s))) return rc;
        if (left && (rc = jump_to_roots(L, 2, g.n, flags + 2, s, tuned_jump_rounds(nx, ny, nz)))) return rc;
        PMSZ_CUDA(cudaMemsetAsync(cnt + 6 + kind, 0, sizeof(unsigned long long), s));
        return count(kind, left ? 0 : 1, nullptr);
    };
    unsigned int open[2] = {0, 0};
    auto read_counts = [&]() -> int {
        unsigned int *hw = reinterpret_cast<unsigned int *>(h + 9);
        PMSZ_CUDA(cudaMemcpyAsync(h, cnt, kCounts, cudaMemcpyDeviceToHost, s));
        PMSZ_CUDA(cudaMemcpyAsync(hw, flags, sizeof(open), cudaMemcpyDeviceToHost, s));
        PMSZ_CUDA(cudaStreamSynchronize(s));
        std::memcpy(open, hw, sizeof(open));
        got[6] = h[6];
        got[7] = h[7];
        return PMSZ_OK;
    };
    if (wanted[0] || wanted[1]) {
        PMSZ_CUDA(cudaMemsetAsync(flags, 0, sizeof(open), s));
        if (LabelRun::general(g)) {
            for (int kind = 0; kind < 2; ++kind) {
                if (!wanted[kind]) continue;
                for (int field = 0; field < 2; ++field)
                    if ((rc = run_of(kind, field).init(field ? c1 : c0, s))) return rc;
                if ((rc = go_on(kind, false))) return rc;
            }
            if ((rc = read_counts())) return rc;
        } else {
            // both kinds, the second only where the first is done; else the arrays
            // keep the first one's labels so far, and the walks go on from them
            if (wanted[0] && (rc = walk(0, nullptr))) return rc;
            if (wanted[1] && (rc = walk(1, wanted[0] ? flags : nullptr))) return rc;
            if ((rc = read_counts())) return rc;
            if (open[0]) {
                if ((rc = go_on(0, true)) || (wanted[1] && (rc = walk(1, nullptr))) || (rc = read_counts())) return rc;
            }
            if (open[1] && ((rc = go_on(1, true)) || (rc = read_counts()))) return rc;
        }
    }
    out->dir_mismatch = got[0];
    out->ext_mismatch = got[1];
    out->as_mismatch = with_labels ? got[6] : UINT64_MAX;
    out->ds_mismatch = with_labels ? got[7] : UINT64_MAX;
    out->bound_strict = got[2];
    out->bound_beyond_clamp = got[3];
    return ws.release();
}

template int verify_impl<float>(const float *, const float *, size_t, size_t, size_t, double, pmsz_verify_result *, cudaStream_t);
template int verify_impl<double>(const double *, const double *, size_t, size_t, size_t, double, pmsz_verify_result *, cudaStream_t);

}  // namespace pmsz

using namespace pmsz;

extern "C" int pmsz_labels(const uint8_t *codes, size_t nx, size_t ny, size_t nz, uint32_t *as_label,
                           uint32_t *ds_label, void *stream) {
    return guarded([&] { return labels_impl(codes, nx, ny, nz, as_label, ds_label, as_stream(stream)); });
}
extern "C" int pmsz_labels_i64(const uint8_t *codes, size_t nx, size_t ny, size_t nz, int64_t *as_label,
                               int64_t *ds_label, void *stream) {
    return guarded([&] { return labels_run<int64_t>(codes, nx, ny, nz, as_label, ds_label, as_stream(stream)); });
}
extern "C" int pmsz_verify_f32(const float *f, const float *fp, size_t nx, size_t ny, size_t nz, double eb,
                               pmsz_verify_result *out, void *stream) {
    return guarded([&] { return verify_impl<float>(f, fp, nx, ny, nz, eb, out, as_stream(stream)); });
}
extern "C" int pmsz_verify_f64(const double *f, const double *fp, size_t nx, size_t ny, size_t nz, double eb,
                               pmsz_verify_result *out, void *stream) {
    return guarded([&] { return verify_impl<double>(f, fp, nx, ny, nz, eb, out, as_stream(stream)); });
}
