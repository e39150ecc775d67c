// el_extrap.cu -- extrapolation (src/project/3d/fluid/extrapolation.cpp:5-51): the reference's
// layer loop over a bitmask of the valid cells.
//
// extrapolate() runs `layers` Jacobi layers: in layer l every cell that is not valid yet and
// has a valid cell among its 26 neighbours (valid when the layer began) takes the mean of those
// neighbours (summed in z, y, x order) and becomes valid.  Here the valid set S of a field is a
// bitmask, one bit per cell and 32 cells of a row per word, with a zero word before and after
// every row and zero rows and planes around the grid, so that a neighbour outside the grid is a
// zero bit and needs no bounds test.  Per layer:
//   1. S' = S dilated by the 3 x 3 x 3 cube is written to the other buffer; the cells of S' \ S
//      are this layer's.
//   2. each of them takes the mean of its neighbours in S, summed in z, y, x order, and is marked
//      valid (extrapolate) or not (extrapolate_const).  No such cell reads another.
// One kernel does both, a block a tile of 64 x 8 x 8 cells in shared memory, whose cells of the layer
// its threads share out: a large layer is bound by the instructions of the means (about 250 a cell), a
// small one by the chain of latencies.  A dilation kernel that left a list to a kernel of means took,
// both together, 41 us a layer at 256^3 (2 million cells in four fields) and 22 at 48^3; this one 28
// and 8.  256 threads a tile: 31 and 8.7; tiles of four planes: 34 and 9.
// The results are those of the reference loop bit for bit: the same cells, the same sums in the
// same order and the same division.  Up to four fields go through each launch (velocity u, v,
// w and the level set of a step), each with its own scratch slot.
#include "el_internal.cuh"

namespace el {

namespace {

constexpr int kExMaxFields = 4;
constexpr int kExThreads = 256;     // of the streaming passes
constexpr int kLayerThreads = 128;  // of a layer's kernel
// the tile: 2 words (64 cells) of a row x 8 rows x 8 planes, and its one-word / one-row /
// one-plane halo
constexpr int kTW = 2, kTY = 8, kTZ = 8;
constexpr int kHW = kTW + 2, kHY = kTY + 2, kHZ = kTZ + 2;
constexpr int kTileWords = kTW * kTY * kTZ;
constexpr int kHaloWords = kHW * kHY * kHZ;
constexpr int kHaloLoads = (kHaloWords + kLayerThreads - 1) / kLayerThreads;
static_assert(kTileWords <= kLayerThreads && kTileWords % 32 == 0, "a thread a word");

// what S holds on a tile
enum : uint8_t { kTileZero = 0, kTileMixed = 1, kTileFull = 2 };

struct ExField {
    void* g;            // the field (float or double), i-fastest n0 x n1 x n2
    uint8_t* valid;     // its valid mask (written for the layers' cells when write_back)
    unsigned* s;        // the valid set before the layer: padded bitmask
    unsigned* s_next;   // and after it
    unsigned* flat;     // the valid mask as a flat bit stream
    uint8_t* st0;       // the first layer's st and ch
    uint8_t* ch0;
    const uint8_t* st;  // per tile: S before the layer (kTile*)
    uint8_t* st_next;   // and after it
    const uint8_t* ch;  // per tile: the layer before changed S there
    uint8_t* ch_next;   // this layer does
    int n0, n1, n2;
    int rw;             // words per row, ceil(n0 / 32); a padded row holds rw + 2
    int ntx, nty, ntz;  // tiles along x, y, z
    int write_back;
};

struct ExArgs {
    ExField f[kExMaxFields];
    int nf;
    int ntiles;       // of the field with the most
    int per;          // tiles a block of ex_layer_kernel
    int blocks;       // of ex_layer_kernel a field
};

// word (wp, yp, zp) of a padded bitmask: wp = word + 1, yp = y + 1, zp = z + 1
__device__ __forceinline__ long long pad_at(const ExField& F, int wp, int yp, int zp) {
    return wp + (long long)(F.rw + 2) * (yp + (long long)(F.n1 + 2) * zp);
}

// the bits of word w of a row that are cells of the grid
__device__ __forceinline__ unsigned row_mask(int n0, int w) {
    const int rem = n0 - 32 * w;
    return rem >= 32 ? 0xffffffffu : ((1u << rem) - 1u);
}

// ---- the valid masks as bitmasks, in two passes over all fields: the mask's bytes as a flat
// bit stream (32 cells per word, 16-byte loads), then that stream cut into the padded rows.

// bit q of the result: byte q of x is not zero
__device__ __forceinline__ unsigned nonzero_bytes(unsigned x) {
    const unsigned h = (((x & 0x7f7f7f7fu) + 0x7f7f7f7fu) | x) & 0x80808080u;
    return ((h >> 7) & 1u) | ((h >> 14) & 2u) | ((h >> 21) & 4u) | ((h >> 28) & 8u);
}

__global__ void __launch_bounds__(kExThreads) ex_flat_kernel(const ExArgs a) {
    const ExField& F = a.f[blockIdx.y];
    const long long n = (long long)F.n0 * F.n1 * F.n2;
    const long long words = (n + 31) / 32;
    unsigned* flat = F.flat;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < words;
         t += (long long)gridDim.x * blockDim.x) {
        unsigned word = 0u;
        if (32 * t + 32 <= n) {
            const uint4* v4 = reinterpret_cast<const uint4*>(F.valid) + 2 * t;
            const uint4 p = v4[0], q = v4[1];
            word = nonzero_bytes(p.x) | (nonzero_bytes(p.y) << 4) | (nonzero_bytes(p.z) << 8) |
                   (nonzero_bytes(p.w) << 12) | (nonzero_bytes(q.x) << 16) | (nonzero_bytes(q.y) << 20) |
                   (nonzero_bytes(q.z) << 24) | (nonzero_bytes(q.w) << 28);
        } else {
            for (int b = 0; 32 * t + b < n; ++b) word |= (F.valid[32 * t + b] != 0 ? 1u : 0u) << b;
        }
        flat[t] = word;
    }
}

// The tiles of a field in an order whose equal shares (a block's, ex_layer_kernel) differ in y: a liquid's surface,
// and with it the layer's cells, crosses the rows of tiles of one y or few.
struct Tile {
    int index, x, y, z;  // index: of its states
};
__device__ __forceinline__ Tile tile_at(const ExField& F, int t) {
    Tile r;
    r.x = t % F.ntx;
    t /= F.ntx;
    r.z = t % F.ntz;
    r.y = t / F.ntz;
    r.index = t * F.ntx + r.x;
    return r;
}
__device__ __forceinline__ int state_at(const ExField& F, int x, int y, int z) {
    return x + F.ntx * (z + F.ntz * y);
}

// what the words sn of a tile's threads hold, `mask` the bits that are cells; all warps' flags or-ed
__device__ __forceinline__ unsigned word_flags(unsigned sn, unsigned mask) {
    return (__any_sync(0xffffffffu, sn != 0u) ? 1u : 0u) | (__any_sync(0xffffffffu, sn != mask) ? 2u : 0u);
}
__device__ __forceinline__ uint8_t tile_state(unsigned flags) {
    return !(flags & 2u) ? kTileFull : (!(flags & 1u) ? kTileZero : kTileMixed);
}

// S_0, a block a tile: its words into both buffers (so that no tile counts as changed), the padding
// words around it as zeros (a slot may have held another field's layout), and its state
__global__ void __launch_bounds__(kLayerThreads) ex_rows_kernel(const __grid_constant__ ExArgs a) {
    __shared__ unsigned wflag[kLayerThreads / 32];
    pdl_wait();
    pdl_trigger();
    const int f = blockIdx.x / a.ntiles;
    const ExField& F = a.f[f];
    if ((int)blockIdx.x - f * a.ntiles >= F.ntx * F.nty * F.ntz) return;  // uniform over the CTA
    const Tile t = tile_at(F, blockIdx.x - f * a.ntiles);
    const int w0 = t.x * kTW, y0 = t.y * kTY, z0 = t.z * kTZ;
    const int tid = threadIdx.x;
    const int w = w0 + tid % kTW, y = y0 + tid / kTW % kTY, z = z0 + tid / (kTW * kTY);
    unsigned word = 0u, mask = 0u;
    if (tid < kTileWords && w < F.rw && y < F.n1 && z < F.n2) {
        // cells 32 w .. + 31 of row (y, z) in the flat stream
        const long long words = ((long long)F.n0 * F.n1 * F.n2 + 31) / 32;
        const long long c0 = 32ll * w + (long long)F.n0 * (y + (long long)F.n1 * z), lo = c0 >> 5;
        const unsigned a0 = F.flat[lo], a1 = lo + 1 < words ? F.flat[lo + 1] : 0u;
        mask = row_mask(F.n0, w);
        word = __funnelshift_r(a0, a1, (unsigned)(c0 & 31)) & mask;
        const long long q = pad_at(F, w + 1, y + 1, z + 1);
        F.s[q] = word;
        F.s_next[q] = word;
    }
    if (t.x == 0 || t.x == F.ntx - 1 || t.y == 0 || t.y == F.nty - 1 || t.z == 0 || t.z == F.ntz - 1) {
        for (int e = tid; e < kHaloWords; e += kLayerThreads) {
            const int wp = w0 + e % kHW, yp = y0 + e / kHW % kHY, zp = z0 + e / (kHW * kHY);
            if (wp > F.rw + 1 || yp > F.n1 + 1 || zp > F.n2 + 1) continue;
            if (wp == 0 || wp == F.rw + 1 || yp == 0 || yp == F.n1 + 1 || zp == 0 || zp == F.n2 + 1) {
                const long long q = pad_at(F, wp, yp, zp);
                F.s[q] = 0u;
                F.s_next[q] = 0u;
            }
        }
    }
    const unsigned flags = word_flags(word, mask);
    if ((tid & 31) == 0) wflag[tid >> 5] = flags;
    __syncthreads();
    if (tid == 0) {
        unsigned all = 0u;
        for (int q = 0; q < kLayerThreads / 32; ++q) all |= wflag[q];
        F.st0[t.index] = tile_state(all);
        F.ch0[t.index] = 0;
    }
}

// (extrapolation.cpp:24-33)
__device__ __forceinline__ float ex_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double ex_add(double a, double b) { return __dadd_rn(a, b); }

// the words of a tile, unchanged, into the other buffer
__device__ __forceinline__ void copy_tile(const ExField& F, const Tile& t) {
    const int tid = threadIdx.x;
    const int w = t.x * kTW + tid % kTW, y = t.y * kTY + tid / kTW % kTY, z = t.z * kTZ + tid / (kTW * kTY);
    if (tid < kTileWords && w < F.rw && y < F.n1 && z < F.n2) {
        const long long q = pad_at(F, w + 1, y + 1, z + 1);
        F.s_next[q] = F.s[q];
    }
}

template <typename T>
__device__ __forceinline__ void layer_tile(const ExField& F, const Tile& t) {
    __shared__ unsigned sm[kHZ][kHY][kHW];               // S over the tile and its halo
    __shared__ unsigned short list[kTileWords * 32];     // the layer's cells: word of the tile, bit
    __shared__ int wtot[kLayerThreads / 32];
    __shared__ unsigned wflag[kLayerThreads / 32];
    const int w0 = t.x * kTW, y0 = t.y * kTY, z0 = t.z * kTZ;
    const int tid = threadIdx.x;
    // the thread's word of the tile
    const int tw = tid % kTW, ty = tid / kTW % kTY, tz = tid / (kTW * kTY);
    const bool live = tid < kTileWords && w0 + tw < F.rw && y0 + ty < F.n1 && z0 + tz < F.n2;
    const long long q0 = pad_at(F, w0 + tw + 1, y0 + ty + 1, z0 + tz + 1);
    // padded coordinates of halo entry (hw, hy, hz): (w0 + hw, y0 + hy, z0 + hz); the entry's
    // place in sm is its index e.  Every load of the thread is issued before the first store.
    const int pw = F.rw + 2, py = F.n1 + 2, pz = F.n2 + 2;
    unsigned hv[kHaloLoads];
#pragma unroll
    for (int u = 0; u < kHaloLoads; ++u) {
        const int e = tid + kLayerThreads * u;
        const int hw = e % kHW, r = e / kHW, hy = r % kHY, hz = r / kHY;
        const int wp = w0 + hw, yp = y0 + hy, zp = z0 + hz;
        hv[u] = 0u;
        if (e < kHaloWords && wp < pw && yp < py && zp < pz) hv[u] = F.s[pad_at(F, wp, yp, zp)];
    }
    unsigned* smf = &sm[0][0][0];
    __syncthreads();  // the block's tile before is done with the shared memory
#pragma unroll
    for (int u = 0; u < kHaloLoads; ++u) {
        const int e = tid + kLayerThreads * u;
        if (e < kHaloWords) smf[e] = hv[u];
    }
    __syncthreads();
    // the layer's cells in the word: the dilation along x (a cell's left and right neighbours,
    // across the word's edges) of the OR over its nine rows, less S, inside the row
    unsigned nw = 0u, sn = 0u;
    const unsigned mask = live ? row_mask(F.n0, w0 + tw) : 0u;
    if (live) {
        unsigned cm = 0u, c0 = 0u, cp = 0u;
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const unsigned* row = sm[tz + r / 3][ty + r % 3] + tw;
            cm |= row[0];
            c0 |= row[1];
            cp |= row[2];
        }
        const unsigned old = sm[tz + 1][ty + 1][tw + 1];
        nw = (c0 | (c0 << 1) | (cm >> 31) | (c0 >> 1) | (cp << 31)) & ~old & mask;
        sn = old | nw;
        F.s_next[q0] = sn;
    }
    // the tile's list, in the order of the threads' words
    const int lane = tid & 31, warp = tid >> 5, cnt = __popc(nw);
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
    }
    const unsigned flags = word_flags(sn, mask);
    if (lane == 31) {
        wtot[warp] = incl;
        wflag[warp] = flags;
    }
    __syncthreads();
    int off = incl - cnt, total = 0;
    unsigned flag = 0u;
#pragma unroll
    for (int q = 0; q < kLayerThreads / 32; ++q) {
        off += q < warp ? wtot[q] : 0;
        total += wtot[q];
        flag |= wflag[q];
    }
    if (tid == 0) {
        F.st_next[t.index] = tile_state(flag);
        F.ch_next[t.index] = total ? 1 : 0;
    }
    if (!total) return;
    while (nw) {
        const int b = __ffs(nw) - 1;
        nw &= nw - 1;
        list[off++] = (unsigned short)(tid * 32 + b);
    }
    __syncthreads();
    T* g = static_cast<T*>(F.g);
    const long long plane = (long long)F.n0 * F.n1;
    [[maybe_unused]] const long long ncell = plane * F.n2;  // read by the index checks of the debug build
    for (int q = tid; q < total; q += kLayerThreads) {
        const int code = list[q], wd = code >> 5, b = code & 31;
        const int cw = wd % kTW, cy = wd / kTW % kTY, cz = wd / (kTW * kTY);
        // which of the 27 are in S: cells x - 1, x, x + 1 of a row are bits sh.. from word lo
        const int lb = 32 * (cw + 1) + b - 1, lo = lb >> 5, sh = lb & 31;
        unsigned m = 0u;
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const unsigned* row = sm[cz + r / 3][cy + r % 3];
            m |= (__funnelshift_r(row[lo], row[lo + 1], sh) & 7u) << (3 * r);
        }
        const long long c = 32 * (w0 + cw) + b + (long long)F.n0 * (y0 + cy) + plane * (z0 + cz);
        if (!EL_IN(c, ncell, 22)) continue;
        // every value's load is issued before the first is summed
        T v[27];
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const T* row = g + c + (long long)F.n0 * (r % 3 - 1) + plane * (r / 3 - 1);
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) v[3 * r + dx] = (m >> (3 * r + dx)) & 1u ? row[dx - 1] : T(0);
        }
        T sum = T(0);
#pragma unroll
        for (int n = 0; n < 27; ++n)
            if ((m >> n) & 1u) sum = ex_add(sum, v[n]);
        g[c] = sum / (T)__popc(m);  // at least one: the cell has a neighbour in S
        if (F.write_back) F.valid[c] = 1;
    }
}

// ---- one layer: a block takes up to four tiles of a field, whose states its warps look
// up first, one a warp; then the block takes each that has work
template <typename T>
__global__ void __launch_bounds__(kLayerThreads) ex_layer_kernel(const __grid_constant__ ExArgs a) {
    constexpr int kWarps = kLayerThreads / 32;
    __shared__ unsigned char work[kWarps];               // 0 none, 1 S' = S to be copied, 2 staged
    pdl_wait();
    pdl_trigger();
    const int f = blockIdx.x / a.blocks, first = blockIdx.x - f * a.blocks;
    const ExField& F = a.f[f];
    const int ntiles = F.ntx * F.nty * F.ntz;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < a.per) {
        const int ti = first + warp * a.blocks;
        int w = 0;
        if (ti < ntiles) {
            // a tile that S fills, or that S leaves empty with its neighbour tiles, has no cell of
            // this layer and is not staged: S' = S there, and the buffer S' goes to holds S of two
            // layers back, so its words are copied only if the layer before changed them
            const Tile t = tile_at(F, ti);
            const int nx = t.x + lane % 3 - 1, ny = t.y + lane / 3 % 3 - 1, nz = t.z + lane / 9 - 1;
            uint8_t st = kTileZero;
            if (lane < 27 && nx >= 0 && nx < F.ntx && ny >= 0 && ny < F.nty && nz >= 0 && nz < F.ntz)
                st = F.st[state_at(F, nx, ny, nz)];
            const uint8_t changed = F.ch[t.index];
            const bool busy = __any_sync(0xffffffffu, st != kTileZero);
            const uint8_t own = (uint8_t)__shfl_sync(0xffffffffu, (int)st, 13);
            w = own != kTileFull && busy ? 2 : (changed ? 1 : 0);
            if (lane == 0 && w < 2) {
                F.st_next[t.index] = own;
                F.ch_next[t.index] = 0;
            }
        }
        if (lane == 0) work[warp] = (unsigned char)w;
    }
    __syncthreads();
    for (int p = 0; p < a.per; ++p) {
        const int w = work[p];
        if (w == 0) continue;
        const Tile t = tile_at(F, first + p * a.blocks);
        if (w == 1)
            copy_tile(F, t);
        else
            layer_tile<T>(F, t);
    }
}

}  // namespace

// bytes of one padded bitmask of an n0 x n1 x n2 field
size_t extrapolation_bits_bytes(int n0, int n1, int n2) {
    return (size_t)((n0 + 31) / 32 + 2) * (size_t)(n1 + 2) * (size_t)(n2 + 2) * sizeof(unsigned);
}

// tiles over an n0 x n1 x n2 field
size_t extrapolation_tiles(int n0, int n1, int n2) {
    return (size_t)(((n0 + 31) / 32 + kTW - 1) / kTW) * (size_t)((n1 + kTY - 1) / kTY) *
           (size_t)((n2 + kTZ - 1) / kTZ);
}

// bytes of the flat bit stream of an n0 x n1 x n2 mask
size_t extrapolation_flat_bytes(int n0, int n1, int n2) {
    return ((size_t)n0 * n1 * n2 + 31) / 32 * sizeof(unsigned);
}

// Scratch of one field slot: two padded bitmasks, the mask as a flat bit stream and four arrays
// of tile states (S on each tile after an even / odd layer, and whether that layer changed it).
static int ensure_ex_slot(el_ctx* ctx, int slot) {
    if (ctx->ex_bits[slot][0]) return EL_OK;
    ctx->ex_bits[slot][0] = (unsigned*)ctx_alloc(ctx, ctx->ex_bits_bytes);
    ctx->ex_bits[slot][1] = (unsigned*)ctx_alloc(ctx, ctx->ex_bits_bytes);
    ctx->ex_flat[slot] = (unsigned*)ctx_alloc(ctx, ctx->ex_flat_bytes);
    ctx->ex_tiles[slot] = (uint8_t*)ctx_alloc(ctx, 4 * ctx->ex_tile_count);
    if (!ctx->ex_bits[slot][0] || !ctx->ex_bits[slot][1] || !ctx->ex_flat[slot] || !ctx->ex_tiles[slot])
        return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "extrapolation scratch");
    return EL_OK;
}

// Allocates the scratch of `nfields` slots (outside any stream capture).
int ensure_extrapolation(el_ctx* ctx, int nfields) {
    for (int q = 0; q < nfields && q < kExMaxFields; ++q) {
        const int rc = ensure_ex_slot(ctx, q);
        if (rc != EL_OK) return rc;
    }
    return EL_OK;
}

// Extrapolates up to four fields together; fields[q] is a field id, valid[q] its mask and
// write_back[q] whether the mask is updated (extrapolate) or left alone (extrapolate_const).
// Returns the kernels launched.
int launch_extrapolate_fields(el_ctx* ctx, int nf, const int* fields, uint8_t* const* valid, const bool* write_back,
                              int layers) {
    if (nf < 1 || layers < 1) return 0;
    ExArgs a{};
    a.nf = nf;
    long long max_cells = 0;
    for (int q = 0; q < nf; ++q) {
        ExField& F = a.f[q];
        int n0, n1, n2;
        field_dims(ctx, fields[q], n0, n1, n2);
        F.g = ctx->field[fields[q]];
        F.valid = valid[q];
        F.flat = ctx->ex_flat[q];
        F.st0 = ctx->ex_tiles[q];
        F.ch0 = ctx->ex_tiles[q] + 2 * ctx->ex_tile_count;
        F.n0 = n0;
        F.n1 = n1;
        F.n2 = n2;
        F.rw = (n0 + 31) / 32;
        F.ntx = (F.rw + kTW - 1) / kTW;
        F.nty = (n1 + kTY - 1) / kTY;
        F.ntz = (n2 + kTZ - 1) / kTZ;
        F.write_back = write_back[q] ? 1 : 0;
        a.ntiles = std::max(a.ntiles, F.ntx * F.nty * F.ntz);
        max_cells = std::max(max_cells, (long long)n0 * n1 * n2);
    }
    auto set_layer = [&](int k) {  // layer k reads buffer (k - 1) & 1 and writes buffer k & 1
        const size_t nt = ctx->ex_tile_count;
        for (int q = 0; q < nf; ++q) {
            ExField& F = a.f[q];
            const int r = (k - 1) & 1, w = k & 1;
            F.s = ctx->ex_bits[q][r];
            F.s_next = ctx->ex_bits[q][w];
            F.st = ctx->ex_tiles[q] + r * nt;
            F.st_next = ctx->ex_tiles[q] + w * nt;
            F.ch = ctx->ex_tiles[q] + (2 + r) * nt;
            F.ch_next = ctx->ex_tiles[q] + (2 + w) * nt;
        }
    };
    // one tile a block where all blocks are resident at once (by threads), else up to four: most tiles
    // have no work, and a wave of blocks that find none costs a few microseconds (256^3:
    // 29.4 us a layer with one, 27.8 with four).
    const long long wave = (long long)ctx->num_sms * (2048 / kLayerThreads);
    a.per = (int)std::min<long long>(4, ((long long)nf * a.ntiles + wave - 1) / wave);
    a.blocks = (a.ntiles + a.per - 1) / a.per;
    set_layer(1);
    const int wide = ctx->num_sms * std::max(1, ctx->extrap_per_sm);  // blocks of the streaming pass
    ex_flat_kernel<<<dim3((unsigned)std::min<long long>(wide, (max_cells / 32 + kExThreads) / kExThreads), nf),
                     kExThreads, 0, ctx->stream>>>(a);
    launch_dependent(ctx, ex_rows_kernel, dim3((unsigned)(nf * a.ntiles)), dim3(kLayerThreads), 0, a);
    int n = 2;
    for (int k = 1; k <= layers; ++k) {
        set_layer(k);
        launch_dependent(ctx, ctx->dtype == EL_F64 ? ex_layer_kernel<double> : ex_layer_kernel<float>,
                         dim3((unsigned)(nf * a.blocks)), dim3(kLayerThreads), 0, a);
        ++n;
    }
    return n;
}

EL_CHECK_EXPORT(extrap)

}  // namespace el
