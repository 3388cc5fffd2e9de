// Kernels of the learned warm start's 3D U-Net (declared in warmnet.h).
//
// The 3x3x3 convolutions are implicit GEMMs on the BF16 tensor cores with FP32
// accumulation.  Levels whose x-rows hold 128 nodes run on tcgen05 (TMA staging, TMEM
// accumulators; convRowsKernel and convTcKernel below); the others on mma.sync m16n8k16:
//   * forward and input-gradient: M = output nodes (one 16-node x-row per MMA row block),
//     N = output channels, K = 27 taps x input channels.  A block stages a haloed
//     4 x 10 x 18-node tile of 16 input channels and the 27-tap weight slice of its
//     output channels in shared memory (cp.async, zero fill outside the grid), and the A
//     operands are ldmatrix loads from the shifted halo, so each input value is read from
//     global memory once per block;
//   * weight gradient: M = 16 output channels, N = 16 input channels, K = nodes; the A
//     operand (dy transposed) and the B operand (shifted input) come from the same two
//     tiles through ldmatrix.trans; each block loops over node tiles and adds its partial
//     sums to the FP32 gradient with one atomic per warp and element at the end.
// Shared-memory rows are 48 bytes (an odd number of 16-byte segments) or 32 bytes with their halves
// swapped in turn, so the eight row addresses of every ldmatrix phase fall in distinct banks.
#include <cuda.h>
#include <cuda_bf16.h>

#include "warmnet.h"

namespace eikx {
namespace net {
namespace {

__device__ __forceinline__ unsigned smemAddr(const void *p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// 16-byte global -> shared copy; zero fill when !valid (src is then not read).
__device__ __forceinline__ void cpAsync16At(unsigned dst, const void *src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

struct TileCoord {
    int gx0, gy0, gz0;
};
__device__ __forceinline__ TileCoord tileOf(int t, int D, int H, int W) {
    (void)D;
    const int tx = (W + kTileX - 1) / kTileX, ty = (H + kTileY - 1) / kTileY;
    TileCoord c;
    c.gx0 = (t % tx) * kTileX;
    t /= tx;
    c.gy0 = (t % ty) * kTileY;
    c.gz0 = (t / ty) * kTileZ;
    return c;
}
__host__ __device__ inline int tilesPerSample(int D, int H, int W) {
    return ((D + kTileZ - 1) / kTileZ) * ((H + kTileY - 1) / kTileY) * ((W + kTileX - 1) / kTileX);
}

// Forward and input-gradient convolution on mma.sync.  A warp owns four x-rows of the tile along y.
// Per dz it loads the six haloed rows that they read, at three shifts along x, as 18 A fragments, and
// every tap's weights (operand B) meet four of them: 18 fragments of x and 18 of weights (N = 32) for
// 144 MMAs, where a warp of two rows loading A anew for every tap took 108 of each kind.  Rows of 16
// channels are 32 bytes in shared memory, the two halves swapped where bit 2 of the node (weights:
// channel) is set, so that eight consecutive rows fall in distinct banks at any shift; haloed rows
// are 24 nodes apart.  Sums run over chunk, dz, dy, dx.  8 x 32 x 64 x 64 nodes, us: 32 to 32 channels
// 216, 155 now; 96 to 32 611, 419 now.
constexpr int kCvThreads = 128, kCvRow = 24 * 32, kCvHaloB = kHaloZ * kHaloY * kCvRow;
__device__ __forceinline__ void ldsm4At(unsigned (&r)[4], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}
template <int NB>
__global__ void __launch_bounds__(kCvThreads, 3) convKernel(ConvArgs a) {
    extern __shared__ __align__(128) unsigned char smemRaw[];   // [halo][weights: tap, channel out]
    const unsigned xAt = smemAddr(smemRaw), wAt = xAt + kCvHaloB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const TileCoord c = tileOf(blockIdx.x, a.D, a.H, a.W);
    const int b = blockIdx.z, co0 = blockIdx.y * NB;
    const long long V = static_cast<long long>(a.D) * a.H * a.W;
    const bf16 *xb = a.x + (b * V + (static_cast<long long>(c.gz0 - 1) * a.H + c.gy0 - 1) * a.W + c.gx0 - 1) * a.cin;

    float acc[4][NB / 8][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < NB / 8; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;

    const int li = lane >> 3, lj = lane & 7;
    const int tz = warp >> 1, ty0 = 4 * (warp & 1);
    // A: matrix li = (nodes 8*(li&1) .. of the shifted row, k half li>>1)
    unsigned aAt[3];
#pragma unroll
    for (int dx = 0; dx < 3; ++dx) {
        const int hx = lj + 8 * (li & 1) + dx;
        aAt[dx] = xAt + (tz * kHaloY + ty0) * kCvRow + hx * 32 + 16 * ((li >> 1) ^ (hx >> 2 & 1));
    }
    // B: matrix li = (channels 16p + 8*(li>>1) .. +7, k half li&1)
    const unsigned bAt = wAt + (lj + 8 * (li >> 1)) * 32 + 16 * ((li & 1) ^ (lj >> 2 & 1));
    const int half = threadIdx.x & 1;
    for (int ci0 = 0; ci0 < a.cin; ci0 += 16) {
#pragma unroll
        for (int i = 0; i < (2 * kHaloNodes + kCvThreads - 1) / kCvThreads; ++i) {
            const int hv = (threadIdx.x + i * kCvThreads) >> 1;
            const int hx = hv % kHaloX, hr = hv / kHaloX, hy = hr % kHaloY, hz = hr / kHaloY;
            const bool in = static_cast<unsigned>(c.gx0 - 1 + hx) < static_cast<unsigned>(a.W) &&
                            static_cast<unsigned>(c.gy0 - 1 + hy) < static_cast<unsigned>(a.H) &&
                            static_cast<unsigned>(c.gz0 - 1 + hz) < static_cast<unsigned>(a.D);
            if (hv < kHaloNodes)
                cpAsync16At(xAt + hr * kCvRow + hx * 32 + 16 * (half ^ (hx >> 2 & 1)),
                            in ? xb + ((static_cast<long long>(hz) * a.H + hy) * a.W + hx) * a.cin + ci0 + 8 * half : a.x, in);
        }
#pragma unroll
        for (int i = 0; i < (27 * NB * 2 + kCvThreads - 1) / kCvThreads; ++i) {
            const int row = (threadIdx.x + i * kCvThreads) >> 1, tap = row / NB, co = row % NB;   // row = tap * NB + co
            if (row < 27 * NB)
                cpAsync16At(wAt + row * 32 + 16 * (half ^ (row >> 2 & 1)),
                            a.w + (static_cast<long long>(tap) * a.cout + co0 + co) * a.cin + ci0 + 8 * half, true);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
#pragma unroll 1
        for (int dz = 0; dz < 3; ++dz) {
            unsigned x[6][3][4];   // [row][dx]
#pragma unroll
            for (int r = 0; r < 6; ++r)
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) ldsm4At(x[r][dx], aAt[dx] + (dz * kHaloY + r) * kCvRow);
#pragma unroll
            for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    unsigned w[NB / 16][4];
#pragma unroll
                    for (int p = 0; p < NB / 16; ++p) ldsm4At(w[p], bAt + ((9 * dz + 3 * dy + dx) * NB + 16 * p) * 32);
#pragma unroll
                    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
                        for (int nt = 0; nt < NB / 8; ++nt)
                            mma16816(acc[mt][nt], x[mt + dy][dx], w[nt >> 1][(nt & 1) * 2], w[nt >> 1][(nt & 1) * 2 + 1]);
                }
        }
        __syncthreads();
    }

    // Epilogue: accumulator (row lane/4 [+8], columns 2*(lane%4), +1) of each 16x8 block.
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
        const int gz = c.gz0 + tz, gy = c.gy0 + ty0 + mt;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int gx = c.gx0 + (lane >> 2) + 8 * h;
            if (gz >= a.D || gy >= a.H || gx >= a.W) continue;
            const long long node = b * V + (static_cast<long long>(gz) * a.H + gy) * a.W + gx;
#pragma unroll
            for (int nt = 0; nt < NB / 8; ++nt) {
                const int co = co0 + 8 * nt + 2 * (lane & 3);
                float y0 = acc[mt][nt][2 * h], y1 = acc[mt][nt][2 * h + 1];
                if (a.bias) {
                    y0 += a.bias[co];
                    y1 += a.bias[co + 1];
                }
                if (a.relu) {
                    y0 = fmaxf(y0, 0.f);
                    y1 = fmaxf(y1, 0.f);
                }
                if (a.mask) {
                    const __nv_bfloat162 m = *reinterpret_cast<const __nv_bfloat162 *>(a.mask + node * a.cout + co);
                    if (!(__bfloat162float(m.x) > 0.f)) y0 = 0.f;
                    if (!(__bfloat162float(m.y) > 0.f)) y1 = 0.f;
                }
                *reinterpret_cast<__nv_bfloat162 *>(a.y + node * a.cout + co) = __floats2bfloat162_rn(y0, y1);
            }
        }
    }
}

// Weight gradient.  A block sums, over its share of the node tiles, the 27 x 16 (co) x 16 (ci) values
// of one block of output channels (blockIdx.y) and one of input channels (blockIdx.z).  Warp w takes
// the taps of one dz = w % 3 on the tile's plane tz = w / 3: nine accumulators of 16 x 16.  Down the
// plane's rows along y a row of dy (operand A, transposed) meets three rows of x at three shifts along
// x (operand B), and two of those rows were there for the row of dy before: three new fragments of x
// and one of dy for 18 MMAs.  What bounds it is shared memory (ldmatrix) with the copies' latency, so
// a tile's copies run while the one before is worked on.  8 x 64 x 128 x 128 nodes, 16 to 16 and 48
// to 16 channels: 620 and 2134 us with four taps a warp (five fragments for eight MMAs), their
// addresses formed per tap and row and more blocks than fit; 450 and 1355 with constant offsets and
// the resident blocks; 354 and 1044 now.
constexpr int kWgThreads = 192;
constexpr int kWgRowB = kRowHalfs * 2, kWgXB = kHaloNodes * kWgRowB, kWgBufB = kWgXB + 256 * kWgRowB;
constexpr int kWgX = (2 * kHaloNodes + kWgThreads - 1) / kWgThreads, kWgDy = (512 + kWgThreads - 1) / kWgThreads;   // 16-byte pieces a thread
__device__ __forceinline__ void ldsm4tAt(unsigned (&r)[4], unsigned a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a)
                 : "memory");
}
__global__ void __launch_bounds__(kWgThreads, 2) wgradKernel(WGradArgs a) {
    extern __shared__ __align__(128) unsigned char smemRaw[];   // two buffers: [x halo][dy]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int li = lane >> 3, lj = lane & 7;
    const int co0 = blockIdx.y * 16, ci0 = blockIdx.z * 16;
    const int dz = warp % 3, tz = warp / 3;
    const long long V = static_cast<long long>(a.D) * a.H * a.W;
    const int tps = tilesPerSample(a.D, a.H, a.W);
    const int nTiles = tps * a.B;
    const unsigned smem = smemAddr(smemRaw);

    float acc[9][2][4];
#pragma unroll
    for (int i = 0; i < 9; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.f;

    // the halo nodes that this thread copies one half of: x, y, z in bytes
    const int half = threadIdx.x & 1;
    int place[kWgX];
#pragma unroll
    for (int i = 0; i < kWgX; ++i) {
        const int hv = (threadIdx.x + i * kWgThreads) >> 1;
        place[i] = hv % kHaloX | (hv / kHaloX % kHaloY) << 8 | hv / (kHaloX * kHaloY) << 16;
    }
    const unsigned xTo = smem + (threadIdx.x >> 1) * kWgRowB + 16 * half, dyTo = xTo + kWgXB;
    auto stage = [&](int t, unsigned buf) {
        const int b = t / tps;
        const TileCoord c = tileOf(t % tps, a.D, a.H, a.W);
        const bf16 *xb = a.x + (b * V + (static_cast<long long>(c.gz0 - 1) * a.H + c.gy0 - 1) * a.W + c.gx0 - 1) * a.cin + ci0 + 8 * half;
#pragma unroll
        for (int i = 0; i < kWgX; ++i) {
            const int hx = place[i] & 255, hy = place[i] >> 8 & 255, hz = place[i] >> 16;
            const bool in = static_cast<unsigned>(c.gx0 - 1 + hx) < static_cast<unsigned>(a.W) &&
                            static_cast<unsigned>(c.gy0 - 1 + hy) < static_cast<unsigned>(a.H) &&
                            static_cast<unsigned>(c.gz0 - 1 + hz) < static_cast<unsigned>(a.D);
            if (i + 1 < kWgX || threadIdx.x < 2 * kHaloNodes - (kWgX - 1) * kWgThreads)
                cpAsync16At(xTo + buf + i * (kWgThreads / 2) * kWgRowB,
                            in ? xb + ((static_cast<long long>(hz) * a.H + hy) * a.W + hx) * a.cin : a.x, in);
        }
        const bf16 *db = a.dy + (b * V + (static_cast<long long>(c.gz0) * a.H + c.gy0) * a.W + c.gx0) * a.cout + co0 + 8 * half;
#pragma unroll
        for (int i = 0; i < kWgDy; ++i) {
            const int node = (threadIdx.x + i * kWgThreads) >> 1, z = node >> 7, y = node >> 4 & 7, x = node & 15;
            const bool in = c.gz0 + z < a.D && c.gy0 + y < a.H && c.gx0 + x < a.W;
            if (node < 256)
                cpAsync16At(dyTo + buf + i * (kWgThreads / 2) * kWgRowB,
                            in ? db + ((static_cast<long long>(z) * a.H + y) * a.W + x) * a.cout : a.dy, in);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // B: matrix li = (nodes 8*(li&1) .., channels 8*(li>>1) ..); A: (co 8*(li&1) .., nodes 8*(li>>1) ..)
    const unsigned bAt = smem + (((tz + dz) * kHaloY * kHaloX + lj + 8 * (li & 1)) * kWgRowB + 16 * (li >> 1));
    const unsigned aAt = smem + kWgXB + (128 * tz + lj + 8 * (li >> 1)) * kWgRowB + 16 * (li & 1);

    unsigned buf = 0;
    if (static_cast<int>(blockIdx.x) < nTiles) stage(blockIdx.x, 0);
    for (int t = blockIdx.x; t < nTiles; t += gridDim.x) {
        const int next = t + gridDim.x;
        if (next < nTiles) {
            stage(next, kWgBufB - buf);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        unsigned x[3][3][4];   // [row mod 3][dx]
        auto row = [&](int hy) {
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) ldsm4tAt(x[hy % 3][dx], bAt + buf + (hy * kHaloX + dx) * kWgRowB);
        };
        row(0);
        row(1);
#pragma unroll
        for (int ty = 0; ty < kTileY; ++ty) {
            row(ty + 2);
            unsigned d[4];
            ldsm4tAt(d, aAt + buf + 16 * ty * kWgRowB);
#pragma unroll
            for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    const unsigned(&f)[4] = x[(ty + dy) % 3][dx];
                    mma16816(acc[3 * dy + dx][0], d, f[0], f[1]);
                    mma16816(acc[3 * dy + dx][1], d, f[2], f[3]);
                }
        }
        __syncthreads();
        buf = kWgBufB - buf;
    }
#pragma unroll
    for (int k = 0; k < 9; ++k)
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int ci = ci0 + 8 * nt + 2 * (lane & 3);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int co = co0 + (lane >> 2) + 8 * h;
                float *d = a.dw + (static_cast<long long>(9 * dz + k) * a.cout + co) * a.cin + ci;
                atomicAdd(d, acc[k][nt][2 * h]);
                atomicAdd(d + 1, acc[k][nt][2 * h + 1]);
            }
        }
}

struct alignas(16) Vec8 {
    __nv_bfloat162 h[4];
};
__device__ __forceinline__ void unpack8(float (&f)[8], const Vec8 &v) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f[2 * i] = __bfloat162float(v.h[i].x);
        f[2 * i + 1] = __bfloat162float(v.h[i].y);
    }
}
__device__ __forceinline__ void load8(float (&f)[8], const bf16 *p) { unpack8(f, *reinterpret_cast<const Vec8 *>(p)); }
__device__ __forceinline__ void store8(bf16 *p, const float (&f)[8]) {
    Vec8 v;
#pragma unroll
    for (int i = 0; i < 4; ++i) v.h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    *reinterpret_cast<Vec8 *>(p) = v;
}

// 16 channels, 32 bytes: a whole sector in one instruction.
__device__ __forceinline__ unsigned pack2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const unsigned *>(&h);
}
__device__ __forceinline__ void store16(bf16 *p, const float (&f)[16]) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(pack2(f[0], f[1])), "r"(pack2(f[2], f[3])),
                 "r"(pack2(f[4], f[5])), "r"(pack2(f[6], f[7])), "r"(pack2(f[8], f[9])), "r"(pack2(f[10], f[11])),
                 "r"(pack2(f[12], f[13])), "r"(pack2(f[14], f[15]))
                 : "memory");
}
__device__ __forceinline__ void load16(float (&f)[16], const bf16 *p) {
    unsigned u[8];
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "l"(p)
                 : "memory");
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        f[2 * k] = __uint_as_float(u[k] << 16);
        f[2 * k + 1] = __uint_as_float(u[k] & 0xffff0000u);
    }
}

// db[c] += sum over nodes of dy[.][c].  Bound by reading dy: a thread sums eight channels, 16 bytes
// a node (8.4 M nodes of 16 channels: 131 us with one channel a thread, 61 now).
__global__ void __launch_bounds__(kThreads) biasGradKernel(const bf16 *dy, int C, long long nodes, float *db) {
    __shared__ float part[kThreads][9];   // 9: the sums below read 8 rows apart without bank conflicts
    const int groups = C / 8, g = threadIdx.x % groups, slot = threadIdx.x / groups, slots = kThreads / groups;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 4
    for (long long v = static_cast<long long>(blockIdx.x) * slots + slot; v < nodes;
         v += static_cast<long long>(gridDim.x) * slots) {
        float f[8];
        load8(f, dy + v * C + 8 * g);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += f[j];
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) part[threadIdx.x][j] = s[j];
    __syncthreads();
    if (threadIdx.x < C) {
        float t = 0.f;
        for (int k = 0; k < slots; ++k) t += part[k * groups + threadIdx.x / 8][threadIdx.x % 8];
        atomicAdd(db + threadIdx.x, t);
    }
}

// The element-wise kernels below move whole 16-byte pieces of 8 channels and are bound by memory.
// A block takes pieces of one x-row of the tensor that it writes (grid: pieces of a row, rows of a
// plane, planes of all samples, the latter two up to what a launch takes and in steps of it), so that a thread needs one 32-bit division to find its place
// (upsampling and concatenation at 8 x 64 x 128 x 128 nodes: 445 us with five 64-bit ones, 183 now).
struct Piece {
    int g, x, y, z, b;   // 8-channel group, node, sample
};
__device__ __forceinline__ bool pieceOf(Piece &p, int groups, int W, int D, long long plane) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    p.x = static_cast<int>(i / static_cast<unsigned>(groups));
    p.g = static_cast<int>(i - static_cast<unsigned>(p.x) * groups);
    p.y = blockIdx.y;
    p.b = static_cast<int>(plane / D);
    p.z = static_cast<int>(plane - static_cast<long long>(p.b) * D);
    return p.x < W;
}

__global__ void __launch_bounds__(kThreads) poolKernel(const bf16 *x, int C, int D, int H, int W, int B, bf16 *y) {
    const int Dl = D / 2, Hl = H / 2, Wl = W / 2, groups = C / 8;
    for (long long plane = blockIdx.z; plane < static_cast<long long>(B) * Dl; plane += gridDim.z) {
        Piece p;
        if (!pieceOf(p, groups, Wl, Dl, plane)) continue;
        for (; p.y < Hl; p.y += gridDim.y) {
            const bf16 *src = x + ((((static_cast<long long>(p.b) * D + 2 * p.z) * H + 2 * p.y) * W + 2 * p.x) * C + 8 * p.g);
            float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                float f[8];
                load8(f, src + ((static_cast<long long>(k >> 2) * H + ((k >> 1) & 1)) * W + (k & 1)) * C);
#pragma unroll
                for (int j = 0; j < 8; ++j) s[j] += f[j];
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j] *= 0.125f;
            store8(y + ((plane * Hl + p.y) * Wl + p.x) * C + 8 * p.g, s);
        }
    }
}

// (kRowsEach rows a thread, their loads all in flight before the first store.)
constexpr int kRowsEach = 4;
__global__ void __launch_bounds__(kThreads) upcatKernel(const bf16 *low, int c1, const bf16 *skip, int c2, int D, int H, int W,
                                                        int B, bf16 *out) {
    const int C = c1 + c2, groups = C / 8;
    const int rows = (H + kRowsEach - 1) / kRowsEach;
    for (long long plane = blockIdx.z; plane < static_cast<long long>(B) * D; plane += gridDim.z) {
        Piece p;
        if (!pieceOf(p, groups, W, D, plane)) continue;
        for (; p.y < rows; p.y += gridDim.y) {
            Vec8 v[kRowsEach];
#pragma unroll
            for (int k = 0; k < kRowsEach; ++k) {
                const int y = kRowsEach * p.y + k;
                if (y >= H) break;
                const bf16 *src = skip + ((plane * H + y) * W + p.x) * c2 + 8 * p.g - c1;
                if (8 * p.g < c1)
                    src = low + (((static_cast<long long>(p.b) * (D / 2) + p.z / 2) * (H / 2) + y / 2) * (W / 2) + p.x / 2) * c1 + 8 * p.g;
                v[k] = *reinterpret_cast<const Vec8 *>(src);
            }
#pragma unroll
            for (int k = 0; k < kRowsEach; ++k) {
                const int y = kRowsEach * p.y + k;
                if (y < H) *reinterpret_cast<Vec8 *>(out + ((plane * H + y) * W + p.x) * C + 8 * p.g) = v[k];
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads) upSumMaskKernel(const bf16 *dcat, int ccat, const bf16 *act, int c1, int Dl, int Hl,
                                                            int Wl, int B, bf16 *dpre) {
    const int groups = c1 / 8, D = 2 * Dl, H = 2 * Hl, W = 2 * Wl;
    for (long long plane = blockIdx.z; plane < static_cast<long long>(B) * Dl; plane += gridDim.z) {
        Piece p;
        if (!pieceOf(p, groups, Wl, Dl, plane)) continue;
        for (; p.y < Hl; p.y += gridDim.y) {
            const bf16 *src = dcat + ((((static_cast<long long>(p.b) * D + 2 * p.z) * H + 2 * p.y) * W + 2 * p.x) * ccat + 8 * p.g);
            const long long u = (plane * Hl + p.y) * Wl + p.x;
            float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                float f[8];
                load8(f, src + ((static_cast<long long>(k >> 2) * H + ((k >> 1) & 1)) * W + (k & 1)) * ccat);
#pragma unroll
                for (int j = 0; j < 8; ++j) s[j] += f[j];
            }
            float m[8];
            load8(m, act + u * c1 + 8 * p.g);
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (!(m[j] > 0.f)) s[j] = 0.f;
            store8(dpre + u * c1 + 8 * p.g, s);
        }
    }
}

__global__ void __launch_bounds__(kThreads) combineSkipKernel(const bf16 *dcat, int ccat, int c1, const bf16 *dpool,
                                                              const bf16 *skip, int c2, int D, int H, int W, int B, bf16 *dpre) {
    const int groups = c2 / 8;
    const int rows = (H + kRowsEach - 1) / kRowsEach;
    for (long long plane = blockIdx.z; plane < static_cast<long long>(B) * D; plane += gridDim.z) {
        Piece q;
        if (!pieceOf(q, groups, W, D, plane)) continue;
        for (; q.y < rows; q.y += gridDim.y) {
            Vec8 a[kRowsEach], p[kRowsEach], m[kRowsEach];
#pragma unroll
            for (int k = 0; k < kRowsEach; ++k) {
                const int y = kRowsEach * q.y + k;
                if (y >= H) break;
                const long long v = (plane * H + y) * W + q.x;
                const long long u = ((static_cast<long long>(q.b) * (D / 2) + q.z / 2) * (H / 2) + y / 2) * (W / 2) + q.x / 2;
                a[k] = *reinterpret_cast<const Vec8 *>(dcat + v * ccat + c1 + 8 * q.g);
                p[k] = *reinterpret_cast<const Vec8 *>(dpool + u * c2 + 8 * q.g);
                m[k] = *reinterpret_cast<const Vec8 *>(skip + v * c2 + 8 * q.g);
            }
#pragma unroll
            for (int k = 0; k < kRowsEach; ++k) {
                const int y = kRowsEach * q.y + k;
                if (y >= H) break;
                float f[8], g[8], r[8];
                unpack8(f, a[k]);
                unpack8(g, p[k]);
                unpack8(r, m[k]);
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] = (r[j] > 0.f) ? f[j] + 0.125f * g[j] : 0.f;
                store8(dpre + ((plane * H + y) * W + q.x) * c2 + 8 * q.g, f);
            }
        }
    }
}

// Per-node geometry, FP32: the offsets from the source are FP64 differences rounded to
// FP32, the distance an FP32 square root; s_src is the slowness at the node nearest the
// source.  An FP64 instruction takes 64 cycles a warp and scheduler here, so what is FP64 in them
// is taken once per sample and axis position, into the sample's table (warmnet.h).
__global__ void __launch_bounds__(kThreads) slownessKernel(const Sample *samples, Geometry g, float *slow, float *tables) {
    const long long V = static_cast<long long>(g.nx) * g.ny * g.nz;
    const Sample s = samples[blockIdx.y];
    float *table = tables + blockIdx.y * tableLength(g);
    const long long first = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x, step = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long i = first; i < V; i += step) slow[blockIdx.y * V + i] = 1.f / s.velocity[i];
    for (long long i = first; i < tableLength(g); i += step) {
        float v;
        if (i == 0) {
            const int ix = min(g.nx - 1, max(0, __double2int_rn((s.xs - g.x0) / g.dx)));
            const int iy = min(g.ny - 1, max(0, __double2int_rn((s.ys - g.y0) / g.dy)));
            const int iz = min(g.nz - 1, max(0, __double2int_rn((s.zs - g.z0) / g.dz)));
            v = 1.f / s.velocity[(static_cast<long long>(iz) * g.ny + iy) * g.nx + ix];
        } else if (i < 4) {
            v = static_cast<float>(i == 1 ? (s.xs - g.x0) / g.dx : i == 2 ? (s.ys - g.y0) / g.dy : (s.zs - g.z0) / g.dz);
        } else {
            const int k = static_cast<int>(i) - 4;
            v = k < g.nx            ? static_cast<float>((g.x0 + k * g.dx) - s.xs)
                : k < g.nx + g.ny ? static_cast<float>((g.y0 + (k - g.nx) * g.dy) - s.ys)
                                  : static_cast<float>((g.z0 + (k - g.nx - g.ny) * g.dz) - s.zs);
        }
        table[i] = v;
    }
}
struct NodeGeom {
    float ddx, ddy, ddz, dist;
};
__device__ __forceinline__ NodeGeom nodeGeom(const float *table, const Geometry &g, int x, int y, int z) {
    NodeGeom n;
    n.ddx = table[4 + x];
    n.ddy = table[4 + g.nx + y];
    n.ddz = table[4 + g.nx + g.ny + z];
    n.dist = sqrtf(n.ddx * n.ddx + n.ddy * n.ddy + n.ddz * n.ddz);
    return n;
}

// Straight-ray estimate of tau - 1 at node (x, y, z): the mean of s/s_src - 1 over
// kRaySamples midpoints of the segment from the source to the node, the slowness
// trilinear in the nodal 1/v.  FP32, in an operation order the oracle repeats.  What bounds it is
// issue slots (72 % taken): two midpoints are in flight together, floor is an addition
// rounded down (px + 2^23, whose low bits are the index; the conversions run at a quarter of the
// rate), and the clamps to the grid are left out where the source lies inside (INSIDE: then so do
// the rounded points of the segment: with w = RN(t e), |w| <= (63/64) |e| (1 + 2^-23) leaves s + w
// between s and x, and rounding keeps that).
constexpr int kRaySamples = 32;
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return add2(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float2 f) { return add2(a, mul2(f, sub2(b, a))); }
template <bool INSIDE>
__device__ __forceinline__ float straightRayContrast(const float *sl, const Geometry &g, const float *table, int x, int y, int z) {
    const float sSrc = table[0], sx = table[1], sy = table[2], sz = table[3];
    const float ex = static_cast<float>(x) - sx, ey = static_cast<float>(y) - sy, ez = static_cast<float>(z) - sz;
    constexpr float kTwo23 = 8388608.f;
    // cell index along one axis (two midpoints), and the positions within the cells
    auto cell = [&](float s, float e, float2 t, int n, int (&i)[2]) {
        float2 p = add2(make_float2(s, s), mul2(t, make_float2(e, e)));
        if (!INSIDE) {
            p.x = fminf(fmaxf(p.x, 0.f), static_cast<float>(n - 1));
            p.y = fminf(fmaxf(p.y, 0.f), static_cast<float>(n - 1));
        }
        const float top = kTwo23 + static_cast<float>(n - 2);   // exact: n <= 2^23
        const float2 m = make_float2(fminf(__fadd_rd(p.x, kTwo23), top), fminf(__fadd_rd(p.y, kTwo23), top));
        i[0] = __float_as_int(m.x) & 0x7fffff;
        i[1] = __float_as_int(m.y) & 0x7fffff;
        return sub2(p, sub2(m, make_float2(kTwo23, kTwo23)));
    };
    const int ny = g.nx, nz = g.nx * g.ny;   // strides (a sample holds fewer than 2^31 nodes)
    const float *slY = sl + ny, *slZ = sl + nz, *slYZ = slY + nz;
    float acc = 0.f;
#pragma unroll 2
    for (int k = 0; k < kRaySamples; k += 2) {
        const float2 t = make_float2((static_cast<float>(k) + 0.5f) / static_cast<float>(kRaySamples),
                                     (static_cast<float>(k + 1) + 0.5f) / static_cast<float>(kRaySamples));
        int ix[2], iy[2], iz[2];
        const float2 fx = cell(sx, ex, t, g.nx, ix), fy = cell(sy, ey, t, g.ny, iy), fz = cell(sz, ez, t, g.nz, iz);
        const int o = iz[0] * nz + iy[0] * ny + ix[0], q = iz[1] * nz + iy[1] * ny + ix[1];
        const float2 c00 = lerp2(make_float2(sl[o], sl[q]), make_float2(sl[o + 1], sl[q + 1]), fx);
        const float2 c10 = lerp2(make_float2(slY[o], slY[q]), make_float2(slY[o + 1], slY[q + 1]), fx);
        const float2 c01 = lerp2(make_float2(slZ[o], slZ[q]), make_float2(slZ[o + 1], slZ[q + 1]), fx);
        const float2 c11 = lerp2(make_float2(slYZ[o], slYZ[q]), make_float2(slYZ[o + 1], slYZ[q + 1]), fx);
        const float2 c = lerp2(lerp2(c00, c10, fy), lerp2(c01, c11, fy), fz);
        acc += c.x / sSrc - 1.f;
        acc += c.y / sSrc - 1.f;
    }
    return acc / static_cast<float>(kRaySamples);
}

// Input features.  8 x 64 x 128 x 128 nodes: 1169 us with FP64 per node and one midpoint at a time,
// 694 now; the 16 bytes a node reads and the 32 it writes would take 60.
__global__ void __launch_bounds__(kThreads) featuresKernel(const float *slow, const float *tables, Geometry g, bf16 *feat) {
    const long long V = static_cast<long long>(g.nx) * g.ny * g.nz;
    const int b = blockIdx.z;
    const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = static_cast<int>(p / static_cast<unsigned>(g.nx)), x = static_cast<int>(p - static_cast<unsigned>(y) * g.nx);
    if (y >= g.ny) return;
    const float *sl = slow + b * V, *table = tables + b * tableLength(g);
    const float invL = static_cast<float>(g.invL);
    const bool inside = table[1] >= 0.f && table[1] <= static_cast<float>(g.nx - 1) && table[2] >= 0.f &&
                        table[2] <= static_cast<float>(g.ny - 1) && table[3] >= 0.f && table[3] <= static_cast<float>(g.nz - 1);
    for (int z = blockIdx.y; z < g.nz; z += gridDim.y) {   // one plane, unless there are more than a launch takes
        const long long v = static_cast<long long>(z) * g.nx * g.ny + p;
        const NodeGeom n = nodeGeom(table, g, x, y, z);
        float f[8] = {sl[v] / table[0] - 1.f,
                      n.dist * invL,
                      n.ddx * invL,
                      n.ddy * invL,
                      n.ddz * invL,
                      inside ? straightRayContrast<true>(sl, g, table, x, y, z) : straightRayContrast<false>(sl, g, table, x, y, z),
                      0.f,
                      0.f};
        store8(feat + (b * V + v) * 16, f);
        const float zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        store8(feat + (b * V + v) * 16 + 8, zero);
    }
}

__device__ __forceinline__ float warpSum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warpSumD(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float headOut(const float (&h)[16], const float (&hw)[17]) {
    float o = hw[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) o += hw[c] * h[c];
    return o;
}

// Nodes of sample blockIdx.y, strided over the sample's blocks: f(node, x, y, z).
template <class F> __device__ __forceinline__ void forNodes(const Geometry &g, F f) {
    const unsigned nx = g.nx, ny = g.ny, V = nx * ny * static_cast<unsigned>(g.nz);   // < 2^31
    for (unsigned v = blockIdx.x * blockDim.x + threadIdx.x; v < V; v += gridDim.x * blockDim.x) {
        const unsigned r = v / nx, z = r / ny;
        f(v, static_cast<int>(v - r * nx), static_cast<int>(r - z * ny), static_cast<int>(z));
    }
}

// Head and loss.  Bound by the activations it reads and the gradients it writes (8 x 64 x 128 x 128
// nodes, 537 MB: 885 us with the source's FP64 geometry per node and a block per 256 nodes, each
// adding its 18 sums to the same words, 170 now): a thread sums over many nodes, a block adds once.
__global__ void __launch_bounds__(kThreads) headLossKernel(const bf16 *h, const float *hw, const Sample *samples,
                                                           const float *tables, Geometry g, double invN, float *dhw,
                                                           bf16 *dpre, double *lossSum) {
    __shared__ float red[kThreads / 32][17];
    __shared__ double redL[kThreads / 32];
    const long long V = static_cast<long long>(g.nx) * g.ny * g.nz;
    const int b = blockIdx.y;
    const float *table = tables + b * tableLength(g);
    const float *travelTime = samples[b].travelTime;
    float w[17], sum[17];
#pragma unroll
    for (int k = 0; k < 17; ++k) {
        w[k] = hw[k];
        sum[k] = 0.f;
    }
    double l = 0.0;
    forNodes(g, [&](unsigned v, int x, int y, int z) {
        const long long i = b * V + v;
        float hv[16], a[8], c[8];
        load8(a, h + i * 16);
        load8(c, h + i * 16 + 8);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            hv[k] = a[k];
            hv[8 + k] = c[k];
        }
        float dout = 0.f;
        const float o = headOut(hv, w);
        const float T0 = table[0] * nodeGeom(table, g, x, y, z).dist;
        if (T0 > 0.f) {
            const float tgt = travelTime[v] / T0 - 1.f;
            const float diff = o - tgt;
            const double d = diff;
            l = fma(d, d, l);
            dout = static_cast<float>(2.0 * d * invN);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            a[k] = hv[k] > 0.f ? dout * w[k] : 0.f;
            c[k] = hv[8 + k] > 0.f ? dout * w[8 + k] : 0.f;
        }
        store8(dpre + i * 16, a);
        store8(dpre + i * 16 + 8, c);
#pragma unroll
        for (int k = 0; k < 16; ++k) sum[k] += dout * hv[k];
        sum[16] += dout;
    });
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < 17; ++k) {
        const float t = warpSum(sum[k]);
        if (lane == 0) red[warp][k] = t;
    }
    const double tl = warpSumD(l);
    if (lane == 0) redL[warp] = tl;
    __syncthreads();
    if (threadIdx.x < 17) {
        float s = 0.f;
        for (int q = 0; q < kThreads / 32; ++q) s += red[q][threadIdx.x];
        atomicAdd(dhw + threadIdx.x, s);
    } else if (threadIdx.x == 32) {
        double s = 0.0;
        for (int q = 0; q < kThreads / 32; ++q) s += redL[q];
        atomicAdd(lossSum, s);
    }
}

// Predicted times (4 x 64 x 128 x 128 nodes, 151 MB: 412 us with the FP64 geometry per node, 49 now).
__global__ void __launch_bounds__(kThreads) predictKernel(const bf16 *h, const float *hw, const Sample *samples,
                                                          const float *tables, Geometry g, float inflate, float *out,
                                                          double *lossSum) {
    __shared__ double redL[kThreads / 32];
    const long long V = static_cast<long long>(g.nx) * g.ny * g.nz;
    const int b = blockIdx.y;
    const float *table = tables + b * tableLength(g);
    const float *travelTime = samples[b].travelTime;
    float w[17];
#pragma unroll
    for (int k = 0; k < 17; ++k) w[k] = hw[k];
    double l = 0.0;
    forNodes(g, [&](unsigned v, int x, int y, int z) {
        const long long i = b * V + v;
        float hv[16], a[8], c[8];
        load8(a, h + i * 16);
        load8(c, h + i * 16 + 8);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            hv[k] = a[k];
            hv[8 + k] = c[k];
        }
        const float o = headOut(hv, w);
        const float T0 = table[0] * nodeGeom(table, g, x, y, z).dist;
        out[i] = T0 * (1.f + o) * inflate;
        if (lossSum && travelTime && T0 > 0.f) {
            const double diff = o - (travelTime[v] / T0 - 1.f);
            l = fma(diff, diff, l);
        }
    });
    if (!lossSum) return;
    const double t = warpSumD(l);
    if ((threadIdx.x & 31) == 0) redL[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int q = 0; q < kThreads / 32; ++q) s += redL[q];
        atomicAdd(lossSum, s);
    }
}

__global__ void adamKernel(float *p, const float *g, float *m, float *v, bf16 *pb, long long n, float lr, float b1,
                           float b2, float eps, float bc1, float bc2) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        const float pi = p[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
        p[i] = pi;
        pb[i] = __float2bfloat16_rn(pi);
    }
}

__global__ void toBF16Kernel(const float *p, bf16 *pb, long long n) {
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        pb[i] = __float2bfloat16_rn(p[i]);
}

__global__ void flipTransposeKernel(const bf16 *w, int cout, int cin, bf16 *wt) {
    const long long n = 27LL * cout * cin;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int co = i % cout;
        const int ci = (i / cout) % cin;
        const int tap = i / (static_cast<long long>(cout) * cin);
        wt[i] = w[(static_cast<long long>(26 - tap) * cout + co) * cin + ci];
    }
}

// ---- tcgen05 convolution for x-rows of 128 nodes ------------------------------------------
// A block computes 8 output x-rows (4 along y, 2 along z), each a full row of 128 nodes, for
// N output channels.  Each row accumulates in its own TMEM region (128 lanes = the row's
// nodes, N FP32 columns).  Per 16-channel input chunk, one thread stages with TMA
// (cp.async.bulk.tensor, zero fill outside the grid):
//   * the 6 x 4 haloed input rows of 130 nodes, one box per 8-channel group: in shared memory
//     [group][row][node][8 channels], so a node's 8 channels are one 16-byte row of a core
//     matrix and node r + dx starts 16 * dx bytes later;
//   * the 27-tap weight slice, one box per group: [group][tap][channel out][8 channels in].
// Both are the no-swizzle K-major canonical layout (K-direction core matrices one group
// apart, 8-row core matrices 128 bytes apart).  The same thread then issues 8 rows x 27 taps
// MMAs (M = 128 nodes, N channels, K = 16): every tap's A operand is the staged row, shifted.
// mbarriers (bounded waits) signal the TMA bytes' arrival and the MMAs' completion; the
// epilogue reads TMEM with tcgen05.ld (warp w: lanes 32w..32w+31).
namespace tc {
constexpr int kRY = 4, kRZ = 2, kRows = kRY * kRZ;
constexpr int kHY = kRY + 2, kHZ = kRZ + 2, kHaloRows = kHY * kHZ;
constexpr int kXN = 130;                          // a 128-node row with its two halo nodes
constexpr int kRowB = kXN * 16;                   // one staged row of one 8-channel group (bytes)
constexpr int kGroupB = kHaloRows * kRowB;        // one group of the halo: 49,920
constexpr int kHaloB = 2 * kGroupB;               // 99,840
constexpr long long kSpin = 1ll << 24;

__device__ __forceinline__ unsigned long long sdesc(unsigned addr, unsigned lbo, unsigned sbo) {
    // start address, leading (K-direction core-matrix) and stride (8-row) byte offsets, all
    // in 16-byte units; bit 46: descriptor version of tcgen05; no swizzle
    return static_cast<unsigned long long>((addr >> 4) & 0x3FFF) |
           (static_cast<unsigned long long>((lbo >> 4) & 0x3FFF) << 16) |
           (static_cast<unsigned long long>((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}
__device__ __forceinline__ void mma(unsigned d, unsigned long long ad, unsigned long long bd, unsigned idesc,
                                    unsigned accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ bool waitParity(unsigned mbar, unsigned parity, long long spin) {
    unsigned done = 0;
    for (long long it = 0; it < spin && !done; ++it)
        asm volatile(
            "{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n selp.u32 %0, 1, 0, q;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
    return done != 0;
}
__device__ __forceinline__ void fenceBefore() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fenceAfter() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tma5(unsigned dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, int c4,
                                     unsigned mbar) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
        "%6}], [%7];" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(mbar)
        : "memory");
}
__device__ __forceinline__ void tma3(unsigned dst, const CUtensorMap *map, int c0, int c1, int c2, unsigned mbar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(dst),
        "l"(reinterpret_cast<unsigned long long>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(mbar)
        : "memory");
}

template <int N> __host__ __device__ constexpr int colStride() { return N <= 32 ? 32 : 64; }
template <int N> __host__ __device__ constexpr int weightGroupB() { return 27 * N * 16; }
template <int N> __host__ __device__ constexpr int smemBytes() { return kHaloB + 2 * weightGroupB<N>() + 32; }

template <int N>
__global__ void __launch_bounds__(128) convTcKernel(ConvArgs a, const __grid_constant__ CUtensorMap mapX,
                                                    const __grid_constant__ CUtensorMap mapW) {
    constexpr int CS = colStride<N>(), NCOL = kRows * CS, WG = weightGroupB<N>();
    static_assert(N % 16 == 0 && N <= 64 && (NCOL & (NCOL - 1)) == 0 && NCOL <= 512, "TMEM layout");
    extern __shared__ __align__(1024) unsigned char smemRaw[];
    unsigned char *halo = smemRaw;                 // [2 groups][24 rows][130 nodes][16 B]
    unsigned char *wsm = smemRaw + kHaloB;         // [2 groups][27 taps][N][16 B]
    unsigned long long *full = reinterpret_cast<unsigned long long *>(wsm + 2 * WG);
    unsigned long long *mmaDone = full + 1;
    unsigned *tslot = reinterpret_cast<unsigned *>(full + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tilesY = a.H / kRY;
    const int z0 = (blockIdx.x / tilesY) * kRZ, y0 = (blockIdx.x % tilesY) * kRY;
    const int b = blockIdx.z, co0 = blockIdx.y * N;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(tslot)),
                     "r"(NCOL)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smemAddr(full)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smemAddr(mmaDone)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fenceBefore();
    __syncthreads();
    fenceAfter();
    const unsigned tmem = *tslot;
    // kind::f16: D FP32 (bit 4), A and B BF16 (bits 7, 10), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<unsigned>(N >> 3) << 17) | ((128u >> 4) << 24);
    const unsigned hb = smemAddr(halo), wb = smemAddr(wsm);
    const long long spin = a.spin > 0 ? a.spin : kSpin;
    // A wait that runs out must not leave the CTA while its copies or MMAs may still write
    // its shared memory or TMEM: before it leaves, the CTA drains -- it waits again on the
    // same barrier phase with a bound kDrain times as long -- and only then frees TMEM.
    constexpr long long kDrain = 64;
    bool ok = true;
    int chunk = 0;
    for (int ci0 = 0; ci0 < a.cin; ci0 += 16, ++chunk) {
        const bool lateTx = a.testLate == 1 && chunk == 0, lateCommit = a.testLate == 2 && chunk == 0;
        if (tid == 0) {
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(full)),
                         "r"(static_cast<unsigned>(kHaloB + 2 * WG + (lateTx ? 16 : 0)))
                         : "memory");
            for (int g = 0; g < 2; ++g) {
                tma5(hb + g * kGroupB, &mapX, ci0 + 8 * g, -1, y0 - 1, z0 - 1, b, smemAddr(full));
                tma3(wb + g * WG, &mapW, ci0 + 8 * g, co0, 0, smemAddr(full));
            }
        }
        const bool landed = waitParity(smemAddr(full), static_cast<unsigned>(chunk & 1), spin);
        if (!__syncthreads_and(landed)) {
            // drain: the copies of this chunk land before the CTA leaves (the test hook's
            // extra bytes are declared complete here, as late bytes would arrive)
            if (tid == 0 && lateTx)
                asm volatile("mbarrier.complete_tx.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(full)), "r"(16u)
                             : "memory");
            waitParity(smemAddr(full), static_cast<unsigned>(chunk & 1), kDrain * spin);
            __syncthreads();
            ok = false;
            break;
        }
        if (tid == 0) {
            for (int rr = 0; rr < kRows; ++rr) {
                const int oz = rr / kRY, oy = rr % kRY;
                for (int tap = 0; tap < 27; ++tap) {
                    const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
                    const int hr = (oz + dz) * kHY + oy + dy;
                    mma(tmem + static_cast<unsigned>(rr * CS),
                        sdesc(hb + static_cast<unsigned>(hr * kRowB + dx * 16), kGroupB, 128),
                        sdesc(wb + static_cast<unsigned>(tap * N * 16), WG, 128), idesc,
                        (ci0 > 0 || tap > 0) ? 1u : 0u);
                }
            }
            if (!lateCommit)
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smemAddr(mmaDone))
                             : "memory");
        }
        // this chunk's MMAs have read the buffers once the barrier's phase completes
        const bool done = waitParity(smemAddr(mmaDone), static_cast<unsigned>(chunk & 1), spin);
        ok = __syncthreads_and(done) != 0;
        if (!ok) {
            // drain: the MMAs issued for this chunk complete before TMEM is freed (the test
            // hook commits their completion only now, as a late completion would arrive)
            if (tid == 0 && lateCommit)
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smemAddr(mmaDone))
                             : "memory");
            waitParity(smemAddr(mmaDone), static_cast<unsigned>(chunk & 1), kDrain * spin);
            __syncthreads();
        }
        fenceAfter();
        if (!ok) break;
    }
    if (ok) {
        const int x = warp * 32 + lane;
        for (int rr = 0; rr < kRows; ++rr) {
            const int gz = z0 + rr / kRY, gy = y0 + rr % kRY;
            const long long node = ((static_cast<long long>(b) * a.D + gz) * a.H + gy) * 128 + x;
#pragma unroll
            for (int c0 = 0; c0 < N; c0 += 16) {
                unsigned r[16];
                const unsigned addr = tmem + ((static_cast<unsigned>(warp) * 32u) << 16) + static_cast<unsigned>(rr * CS + c0);
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                      "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                      "=r"(r[15])
                    : "r"(addr)
                    : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                float v[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    v[j] = __uint_as_float(r[j]);
                    if (a.bias) v[j] += a.bias[co0 + c0 + j];
                    if (a.relu) v[j] = fmaxf(v[j], 0.f);
                }
                bf16 *dst = a.y + node * a.cout + co0 + c0;
                if (a.mask) {
                    float m0[8], m1[8];
                    load8(m0, a.mask + node * a.cout + co0 + c0);
                    load8(m1, a.mask + node * a.cout + co0 + c0 + 8);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        if (!(m0[j] > 0.f)) v[j] = 0.f;
                        if (!(m1[j] > 0.f)) v[8 + j] = 0.f;
                    }
                }
                float lo[8], hi[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    lo[j] = v[j];
                    hi[j] = v[8 + j];
                }
                store8(dst, lo);
                store8(dst + 8, hi);
            }
        }
    } else if (tid == 0 && a.status) {
        atomicExch(a.status, 1);
    }
    fenceBefore();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOL) : "memory");
}

// The same convolution as a persistent kernel, where all weights and a ring of four or more input
// planes fit in shared memory: loads, MMAs and output run at the same time, in three roles (a
// loading thread, an issuing thread, eight output warps).  A tile is four x-rows along y; a block
// walks tiles along z (a segment), so that a plane of six haloed rows is loaded once for the three
// tiles that read it.
//
// What bounds an MMA at few channels is reading A (128 nodes of 16 channels, 4 KB), so one takes an
// input row's A for all output rows that it reaches: row r contributes through tap dy to row r - dy,
// and with the accumulators of the output rows side by side and the weights ordered
// [dz][dx][dy = 2, 1, 0][channel out], the two or three taps are one operand B of two or three times
// N columns.  That is 54 MMAs a tile instead of 108; at 68 cycles each, whatever N is, they are what
// bounds the kernel.  With several 16-channel chunks a segment is walked once per chunk, its tiles'
// accumulators staying in TMEM.  The output warps free the accumulators once they are in registers
// and store whole 32-byte sectors (with 16-byte stores before the arrival: 408 us where 222 is now,
// and 1140 where 298 is).  Every output still sums its products in the order chunk, dz, dy, dx: the
// results are those of convTcKernel, bit for bit.  8 x 64 x 128 x 128 nodes, us, convTcKernel and now:
// 16 to 16 channels 530, 222; 48 to 16 1137, 606; 16 to 48 1448, 298.
namespace rows {
constexpr int kY = 4, kIn = kY + 2, kOutWarps = 8, kThreadsR = 64 + 32 * kOutWarps, kRing = 8;
constexpr int kGroup = (kIn * kRowB + 127) / 128 * 128;   // one 8-channel group of a plane: 12,544
constexpr int kPlane = 2 * kGroup;
constexpr int kSmemMax = 232448, kBarB = 512;             // shared memory per block; barriers
template <int N> __host__ __device__ constexpr int chunkWeights() { return 2 * 27 * N * 16; }
// columns from one tile's accumulators to the next, and how many tiles TMEM holds
template <int N> __host__ __device__ constexpr int accStep() { return N <= 16 ? 64 : N <= 32 ? 128 : 256; }
template <int N> __host__ __device__ constexpr int accCount() { return 512 / accStep<N>(); }
template <int N> __host__ int ringOf(int cin) {
    const int r = (kSmemMax - kBarB - cin / 16 * chunkWeights<N>()) / kPlane;
    return r < kRing ? r : kRing;
}

__device__ __forceinline__ void arrive(unsigned mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void expect(unsigned mbar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void commit(unsigned mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
// A bounded wait that also ends when another role has given up.
__device__ __forceinline__ bool wait(unsigned mbar, unsigned parity, long long spin, volatile int *stop) {
    for (long long it = 0; it < spin; ++it) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred q;\n mbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n selp.u32 %0, 1, 0, q;\n}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
        if (*stop) return false;
    }
    *stop = 1;
    return false;
}

// The MMAs of one dz: the six input rows of a plane (A at `a`, group stride kGroup) with the weights
// at `b` onto the accumulators at `acc`; FIRST: these are the first products of every output row.
template <int N, bool FIRST>
__device__ __forceinline__ void issuePlane(unsigned acc, unsigned long long a, unsigned long long b) {
#pragma unroll
    for (int r = 0; r < kIn; ++r)
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) {
            const int lo = r < 2 ? 0 : r - 2, hi = r < kY ? r : kY - 1;   // output rows reached
            const unsigned long long ad = a + static_cast<unsigned long long>((r * kRowB + dx * 16) >> 4);
            auto part = [&](int y0, int y1, unsigned accumulate) {
                if (y1 < y0) return;
                const int first = dx * 3 + 2 - (r - y0);   // [dx][dy = 2, 1, 0], dy = r - y0
                const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) |
                                       (static_cast<unsigned>((y1 - y0 + 1) * N >> 3) << 17) | ((128u >> 4) << 24);
                mma(acc + static_cast<unsigned>(y0 * N), ad, b + static_cast<unsigned long long>(first * N), idesc, accumulate);
            };
            if (FIRST && dx == 0 && r < kY) {   // row r starts here
                part(lo, r - 1, 1u);
                part(r, r, 0u);
            } else {
                part(lo, hi, 1u);
            }
        }
}

// A slot of the ring and the parity of its barriers' present phase.
struct Slot {
    int at = 0, parity = 0;
    __device__ __forceinline__ void next(int ring) {
        if (++at == ring) {
            at = 0;
            parity ^= 1;
        }
    }
};
// Segment `s`: up to `len` tiles along z from z0, of rows y0 .. y0 + 3.
struct Segment {
    int b, y0, z0, n;
    __device__ __forceinline__ Segment(int s, int len, const ConvArgs &a) {
        const int tilesY = a.H / kY, segsZ = (a.D + len - 1) / len;
        y0 = (s % tilesY) * kY;
        z0 = (s / tilesY) % segsZ * len;
        b = s / tilesY / segsZ;
        n = a.D - z0 < len ? a.D - z0 : len;
    }
};

template <int N>
__global__ void __launch_bounds__(kThreadsR, 1) convRowsKernel(ConvArgs a, const __grid_constant__ CUtensorMap mapX,
                                                            const __grid_constant__ CUtensorMap mapW, int segments, int len,
                                                            int ring) {
    constexpr int STEP = accStep<N>(), ACCS = accCount<N>(), WC = chunkWeights<N>(), WG = WC / 2;
    static_assert(kY * N <= STEP && (ACCS & (ACCS - 1)) == 0, "TMEM layout");
    extern __shared__ __align__(1024) unsigned char smemRaw[];
    const int chunks = a.cin / 16;
    unsigned char *wsm = smemRaw + ring * kPlane;   // [chunk][2 groups][dz][dx][dy = 2, 1, 0][N][16 B]
    const unsigned full = smemAddr(wsm + chunks * WC), empty = full + 64, accFull = full + 128, accEmpty = full + 192,
                   wFull = full + 256, drained = full + 264;
    unsigned *tslot = reinterpret_cast<unsigned *>(wsm + chunks * WC + 272);
    volatile int *stop = reinterpret_cast<volatile int *>(tslot + 1);
    volatile int *issued = stop + 1;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int co0 = blockIdx.y * N;
    const long long spin = a.spin > 0 ? a.spin : kSpin;
    const unsigned hb = smemAddr(smemRaw), wb = smemAddr(wsm);

    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smemAddr(tslot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int k = 0; k < 34; ++k)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full + 8 * k), "r"(k >= 24 && k < 32 ? kOutWarps : 1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        *stop = 0;
        *issued = 0;
    }
    fenceBefore();
    __syncthreads();
    fenceAfter();
    const unsigned tmem = *tslot;

    if (warp == 0) {
        if (lane == 0) {
            expect(wFull, static_cast<unsigned>(chunks * WC));
            for (int c = 0; c < chunks; ++c)
                for (int g = 0; g < 2; ++g)
                    for (int tap = 0; tap < 27; ++tap) {
                        const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
                        tma3(wb + c * WC + g * WG + ((dz * 3 + dx) * 3 + 2 - dy) * N * 16, &mapW, 16 * c + 8 * g, co0, tap, wFull);
                    }
            Slot slot;
            int k = 0;   // planes loaded
            bool ok = true;
            for (int s = blockIdx.x; s < segments && ok; s += gridDim.x) {
                const Segment sg(s, len, a);
                for (int c = 0; c < chunks && ok; ++c)
                    for (int p = 0; p < sg.n + 2; ++p) {
                        if (k >= ring && !wait(empty + 8 * slot.at, slot.parity ^ 1, spin, stop)) {
                            ok = false;
                            break;
                        }
                        expect(full + 8 * slot.at, static_cast<unsigned>(2 * kIn * kRowB + (a.testLate == 1 && k == 0 ? 16 : 0)));
                        for (int g = 0; g < 2; ++g)
                            tma5(hb + slot.at * kPlane + g * kGroup, &mapX, 16 * c + 8 * g, -1, sg.y0 - 1, sg.z0 - 1 + p, sg.b,
                                 full + 8 * slot.at);
                        *issued = ++k;
                        slot.next(ring);
                    }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = wait(wFull, 0, spin, stop);
            Slot slot;     // the next plane to arrive
            int first = 0;   // tiles of the segments before
            for (int s = blockIdx.x; s < segments && ok; s += gridDim.x) {
                const Segment sg(s, len, a);
                for (int c = 0; c < chunks && ok; ++c) {
                    const unsigned long long bd = sdesc(wb + c * WC, WG, 128);
                    constexpr unsigned long long bPlane = 9 * N;
                    int s0 = 0, s1 = slot.at;   // the slots of the tile's planes z - 1 and z
                    ok = wait(full + 8 * slot.at, slot.parity, spin, stop);
                    slot.next(ring);
                    int s2 = slot.at;
                    ok = ok && wait(full + 8 * slot.at, slot.parity, spin, stop);
                    slot.next(ring);
                    for (int j = 0; j < sg.n && ok; ++j) {
                        s0 = s1;
                        s1 = s2;
                        s2 = slot.at;
                        ok = wait(full + 8 * slot.at, slot.parity, spin, stop);
                        slot.next(ring);
                        const int t = first + j, at = t & (ACCS - 1);
                        if (ok && c == 0 && t >= ACCS) ok = wait(accEmpty + 8 * at, (t / ACCS + 1) & 1, spin, stop);
                        if (!ok) break;
                        fenceAfter();
                        const unsigned acc = tmem + static_cast<unsigned>(at * STEP);
                        const unsigned long long d0 = sdesc(hb + s0 * kPlane, kGroup, 128);
                        if (c == 0) issuePlane<N, true>(acc, d0, bd);
                        else issuePlane<N, false>(acc, d0, bd);
#pragma unroll 1
                        for (int dz = 1; dz < 3; ++dz)
                            issuePlane<N, false>(acc, sdesc(hb + (dz == 1 ? s1 : s2) * kPlane, kGroup, 128), bd + dz * bPlane);
                        commit(empty + 8 * s0);   // once they have read it
                        if (j == sg.n - 1) {
                            commit(empty + 8 * s1);
                            commit(empty + 8 * s2);
                        }
                        if (c == chunks - 1 && !(a.testLate == 2 && t == 0)) commit(accFull + 8 * at);
                    }
                }
                first += sg.n;
            }
        }
    } else {
        // warp w reads TMEM lanes 32 (w & 3) .., the first four warps rows 0 and 1, the others 2 and 3
        const int q = warp & 3, x = q * 32 + lane, yFirst = warp < 6 ? 0 : 2;
        float bias[N];
#pragma unroll
        for (int j = 0; j < N; ++j) bias[j] = a.bias ? a.bias[co0 + j] : 0.f;
        int t = 0;
        bool ok = true;
        for (int s = blockIdx.x; s < segments && ok; s += gridDim.x) {
            const Segment sg(s, len, a);
            for (int j = 0; j < sg.n; ++j, ++t) {
                const int at = t & (ACCS - 1);
                ok = __all_sync(0xffffffffu, wait(accFull + 8 * at, (t / ACCS) & 1, spin, stop));
                if (!ok) break;
                fenceAfter();
                // both rows into registers, the accumulators free at once, then the output
                unsigned r[2 * N];
#pragma unroll
                for (int c0 = 0; c0 < 2 * N; c0 += 16)
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                        : "=r"(r[c0]), "=r"(r[c0 + 1]), "=r"(r[c0 + 2]), "=r"(r[c0 + 3]), "=r"(r[c0 + 4]), "=r"(r[c0 + 5]),
                          "=r"(r[c0 + 6]), "=r"(r[c0 + 7]), "=r"(r[c0 + 8]), "=r"(r[c0 + 9]), "=r"(r[c0 + 10]), "=r"(r[c0 + 11]),
                          "=r"(r[c0 + 12]), "=r"(r[c0 + 13]), "=r"(r[c0 + 14]), "=r"(r[c0 + 15])
                        : "r"(tmem + ((static_cast<unsigned>(q) * 32u) << 16) + static_cast<unsigned>(at * STEP + yFirst * N + c0))
                        : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                fenceBefore();
                __syncwarp();
                if (lane == 0) arrive(accEmpty + 8 * at);
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const long long node = ((static_cast<long long>(sg.b) * a.D + sg.z0 + j) * a.H + sg.y0 + yFirst + y) * 128 + x;
#pragma unroll
                    for (int c0 = 0; c0 < N; c0 += 16) {
                        float v[16];
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            v[k] = __uint_as_float(r[y * N + c0 + k]);
                            if (a.bias) v[k] += bias[c0 + k];
                            if (a.relu) v[k] = fmaxf(v[k], 0.f);
                        }
                        if (a.mask) {
                            float m[16];
                            load16(m, a.mask + node * a.cout + co0 + c0);
#pragma unroll
                            for (int k = 0; k < 16; ++k)
                                if (!(m[k] > 0.f)) v[k] = 0.f;
                        }
                        store16(a.y + node * a.cout + co0 + c0, v);
                    }
                }
            }
        }
    }
    __syncwarp();
    __syncthreads();
    if (*stop) {
        // A wait ran out: the block leaves only when its copies have landed and its MMAs are done
        // (waits again, kDrain times as long; the test hook's late bytes and completion come now).
        constexpr long long kDrain = 64;
        if (tid == 0) {
            if (a.testLate == 1)
                asm volatile("mbarrier.complete_tx.shared::cta.b64 [%0], %1;" ::"r"(full), "r"(16u) : "memory");
            waitParity(wFull, 0, kDrain * spin);
            const int n = *issued;
            for (int k = n > ring ? n - ring : 0; k < n; ++k) waitParity(full + 8 * (k % ring), (k / ring) & 1, kDrain * spin);
            if (a.status) atomicExch(a.status, 1);
        } else if (tid == 32) {
            commit(drained);
            waitParity(drained, 0, kDrain * spin);
        }
    }
    fenceBefore();
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

template <int N>
cudaError_t launch(const ConvArgs &a, const CUtensorMap &mapX, const CUtensorMap &mapW, cudaStream_t s) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int ring = ringOf<N>(a.cin), smem = ring * kPlane + a.cin / 16 * chunkWeights<N>() + kBarB;
    // the shared-memory limit is a per-device attribute: set it for the current device
    if (e == cudaSuccess) e = cudaFuncSetAttribute(convRowsKernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    // Tiles per segment: with several chunks as many as TMEM holds; with one, what leaves the blocks
    // least to do (two planes more per segment, about half a tile's time each).
    auto segmentsOf = [&](int len) { return static_cast<long long>(a.B) * (a.H / kY) * ((a.D + len - 1) / len); };
    int len = accCount<N>();
    if (a.cin == 16) {
        long long best = 0;
        for (int l = 4; l <= 64; l += 4) {
            const long long cost = (segmentsOf(l) + sms - 1) / sms * (l + 1);
            if (!best || cost < best) {
                best = cost;
                len = l;
            }
        }
    }
    const long long segments = segmentsOf(len);
    if (segments > 2147483647LL - 65536) return cudaErrorInvalidValue;
    const dim3 grid(static_cast<unsigned>(segments < sms ? segments : sms), a.cout / N);
    convRowsKernel<N><<<grid, kThreadsR, smem, s>>>(a, mapX, mapW, static_cast<int>(segments), len, ring);
    return cudaGetLastError();
}
}  // namespace rows

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encodeTiled() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    }
    return fn;
}

template <int N>
cudaError_t launchTc(const ConvArgs &a, cudaStream_t s) {
    EncodeTiled enc = encodeTiled();
    if (!enc) return cudaErrorNotSupported;
    const bool rowsFit = rows::ringOf<N>(a.cin) >= 4;
    // activations [B][D][H][128][cin] BF16: box of 8 channels x 130 nodes x 6 rows x 4 planes (1) x 1 sample
    CUtensorMap mapX, mapW;
    const cuuint64_t dimX[5] = {static_cast<cuuint64_t>(a.cin), 128, static_cast<cuuint64_t>(a.H),
                                static_cast<cuuint64_t>(a.D), static_cast<cuuint64_t>(a.B)};
    const cuuint64_t strideX[4] = {static_cast<cuuint64_t>(a.cin) * 2, 128ull * a.cin * 2,
                                   static_cast<cuuint64_t>(a.H) * 128 * a.cin * 2,
                                   static_cast<cuuint64_t>(a.D) * a.H * 128 * a.cin * 2};
    const cuuint32_t boxX[5] = {8, kXN, kHY, static_cast<cuuint32_t>(rowsFit ? 1 : kHZ), 1}, ones[5] = {1, 1, 1, 1, 1};
    static_assert(kHY == rows::kIn, "one box height");
    if (enc(&mapX, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16 *>(a.x), dimX, strideX, boxX, ones,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    // weights [27][cout][cin] BF16: box of 8 channels in x N channels out x 27 taps (1 tap)
    const cuuint64_t dimW[3] = {static_cast<cuuint64_t>(a.cin), static_cast<cuuint64_t>(a.cout), 27};
    const cuuint64_t strideW[2] = {static_cast<cuuint64_t>(a.cin) * 2, static_cast<cuuint64_t>(a.cout) * a.cin * 2};
    const cuuint32_t boxW[3] = {8, static_cast<cuuint32_t>(N), rowsFit ? 1u : 27u};
    if (enc(&mapW, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16 *>(a.w), dimW, strideW, boxW, ones,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    if (rowsFit) return rows::launch<N>(a, mapX, mapW, s);
    // the shared-memory limit is a per-device attribute: set it for the current device
    cudaError_t e = cudaFuncSetAttribute(convTcKernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smemBytes<N>());
    if (e != cudaSuccess) return e;
    dim3 grid((a.D / kRZ) * (a.H / kRY), a.cout / N, a.B);
    convTcKernel<N><<<grid, 128, smemBytes<N>(), s>>>(a, mapX, mapW);
    return cudaGetLastError();
}
}  // namespace tc

int gridFor(long long n, int cap = 1 << 20) {
    long long b = (n + kThreads - 1) / kThreads;
    if (b < 1) b = 1;
    return static_cast<int>(b < cap ? b : cap);
}

template <int NB>
cudaError_t convOne(const ConvArgs &a, cudaStream_t s) {
    const int smem = kCvHaloB + 27 * NB * 32;
    // the shared-memory limit is a per-device attribute: set it for the current device
    cudaError_t e = cudaFuncSetAttribute(convKernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    dim3 grid(tilesPerSample(a.D, a.H, a.W), a.cout / NB, a.B);
    convKernel<NB><<<grid, kCvThreads, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launchConv(const ConvArgs &a, cudaStream_t s) {
    if (a.cin % 16 || a.cout % 16 || a.B < 1) return cudaErrorInvalidValue;
    if (a.W == 128 && a.H % tc::kRY == 0 && a.D % tc::kRZ == 0) {
        switch (a.cout) {
            case 16: return tc::launchTc<16>(a, s);
            case 32: return tc::launchTc<32>(a, s);
            case 48: return tc::launchTc<48>(a, s);
            default:
                if (a.cout % 64 == 0) return tc::launchTc<64>(a, s);
                if (a.cout % 32 == 0) return tc::launchTc<32>(a, s);
                return tc::launchTc<16>(a, s);
        }
    }
    return a.cout % 32 == 0 ? convOne<32>(a, s) : convOne<16>(a, s);
}

cudaError_t launchWGrad(const WGradArgs &a, int numSMs, cudaStream_t s) {
    if (a.cin % 16 || a.cout % 16 || a.B < 1) return cudaErrorInvalidValue;
    const int smem = 2 * kWgBufB;
    // the shared-memory limit is a per-device attribute: set it for the current device
    cudaError_t e = cudaFuncSetAttribute(wgradKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    const int gy = a.cout / 16, gz = a.cin / 16;
    const int nTiles = tilesPerSample(a.D, a.H, a.W) * a.B;
    // as many blocks as are resident (two per SM): a block's share of the tiles is fixed, so a second
    // wave takes as long as the first
    int gx = 2 * numSMs / (gy * gz);
    gx = gx < 1 ? 1 : (gx > nTiles ? nTiles : gx);
    wgradKernel<<<dim3(gx, gy, gz), kWgThreads, smem, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launchBiasGrad(const bf16 *dy, int c, long long nodes, float *db, int numSMs, cudaStream_t s) {
    if (c < 8 || c > kThreads || kThreads % c) return cudaErrorInvalidValue;
    const long long slots = kThreads / (c / 8);
    long long blocks = (nodes + slots * 16 - 1) / (slots * 16);
    if (blocks > 4LL * numSMs) blocks = 4LL * numSMs;
    if (blocks < 1) blocks = 1;
    biasGradKernel<<<static_cast<int>(blocks), kThreads, 0, s>>>(dy, c, nodes, db);
    return cudaGetLastError();
}

namespace {
// The y or z extent of a launch grid for n of something that the kernel steps through by it: a
// launch takes up to 65535.
unsigned gridYZ(long long n) { return static_cast<unsigned>(n < 65535 ? n : 65535); }
// Grid of the kernels over 16-byte pieces (pieceOf): W x H rows, `planes` planes.
dim3 pieceGrid(int W, int C, int H, long long planes) {
    return dim3((W * (C / 8) + kThreads - 1) / kThreads, gridYZ(H), gridYZ(planes));
}
// Blocks of a sample in the kernels with sums (forNodes): eight per SM over all samples.
dim3 nodeGrid(const Geometry &g, int B, int numSMs) {
    const long long all = (static_cast<long long>(g.nx) * g.ny * g.nz + kThreads - 1) / kThreads, want = (8LL * numSMs + B - 1) / B;
    return dim3(static_cast<unsigned>(all < want ? all : want), B);
}
}  // namespace

cudaError_t launchPool(const bf16 *x, int C, int D, int H, int W, int B, bf16 *y, cudaStream_t s) {
    poolKernel<<<pieceGrid(W / 2, C, H / 2, static_cast<long long>(B) * (D / 2)), kThreads, 0, s>>>(x, C, D, H, W, B, y);
    return cudaGetLastError();
}

cudaError_t launchUpcat(const bf16 *low, int c1, const bf16 *skip, int c2, int D, int H, int W, int B, bf16 *out,
                        cudaStream_t s) {
    upcatKernel<<<pieceGrid(W, c1 + c2, (H + kRowsEach - 1) / kRowsEach, static_cast<long long>(B) * D), kThreads, 0, s>>>(low, c1, skip, c2, D, H, W, B, out);
    return cudaGetLastError();
}

cudaError_t launchUpSumMask(const bf16 *dcat, int ccat, const bf16 *act, int c1, int Dl, int Hl, int Wl, int B,
                            bf16 *dpre, cudaStream_t s) {
    upSumMaskKernel<<<pieceGrid(Wl, c1, Hl, static_cast<long long>(B) * Dl), kThreads, 0, s>>>(dcat, ccat, act, c1, Dl, Hl, Wl, B, dpre);
    return cudaGetLastError();
}

cudaError_t launchCombineSkip(const bf16 *dcat, int ccat, int c1, const bf16 *dpool, const bf16 *skip, int c2,
                              int D, int H, int W, int B, bf16 *dpre, cudaStream_t s) {
    combineSkipKernel<<<pieceGrid(W, c2, (H + kRowsEach - 1) / kRowsEach, static_cast<long long>(B) * D), kThreads, 0, s>>>(dcat, ccat, c1, dpool, skip, c2, D, H, W,
                                                                                             B, dpre);
    return cudaGetLastError();
}

cudaError_t launchSlowness(const Sample *samples, Geometry g, int B, float *slow, float *tables, cudaStream_t s) {
    slownessKernel<<<dim3(gridFor(static_cast<long long>(g.nx) * g.ny * g.nz), B), kThreads, 0, s>>>(samples, g, slow, tables);
    return cudaGetLastError();
}

cudaError_t launchFeatures(const float *slow, const float *tables, Geometry g, int B, bf16 *feat, cudaStream_t s) {
    const dim3 grid(static_cast<unsigned>((static_cast<long long>(g.nx) * g.ny + kThreads - 1) / kThreads), gridYZ(g.nz), B);
    featuresKernel<<<grid, kThreads, 0, s>>>(slow, tables, g, feat);
    return cudaGetLastError();
}

cudaError_t launchHeadLoss(const bf16 *h, const float *hw, const Sample *samples, const float *tables, Geometry g,
                           int B, double invN, float *dhw, bf16 *dpre, double *lossSum, int numSMs, cudaStream_t s) {
    headLossKernel<<<nodeGrid(g, B, numSMs), kThreads, 0, s>>>(h, hw, samples, tables, g, invN, dhw, dpre, lossSum);
    return cudaGetLastError();
}

cudaError_t launchPredict(const bf16 *h, const float *hw, const Sample *samples, const float *tables, Geometry g, int B,
                          double inflate, float *out, double *lossSum, int numSMs, cudaStream_t s) {
    predictKernel<<<nodeGrid(g, B, numSMs), kThreads, 0, s>>>(h, hw, samples, tables, g, static_cast<float>(inflate), out, lossSum);
    return cudaGetLastError();
}

cudaError_t launchAdam(float *p, const float *g, float *m, float *v, bf16 *pb, long long n, float lr, float b1,
                       float b2, float eps, float bc1, float bc2, cudaStream_t s) {
    adamKernel<<<gridFor(n, 4096), kThreads, 0, s>>>(p, g, m, v, pb, n, lr, b1, b2, eps, bc1, bc2);
    return cudaGetLastError();
}

cudaError_t launchToBF16(const float *p, bf16 *pb, long long n, cudaStream_t s) {
    toBF16Kernel<<<gridFor(n, 4096), kThreads, 0, s>>>(p, pb, n);
    return cudaGetLastError();
}

cudaError_t launchFlipTranspose(const bf16 *w, int cout, int cin, bf16 *wt, cudaStream_t s) {
    flipTransposeKernel<<<gridFor(27LL * cout * cin, 4096), kThreads, 0, s>>>(w, cout, cin, wt);
    return cudaGetLastError();
}

}  // namespace net
}  // namespace eikx
