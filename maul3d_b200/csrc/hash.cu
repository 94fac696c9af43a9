// World hash on the device, one thread block per world, the byte stream
// hashed in parallel.
//
// FNV-1a 64 folds one byte at a time, h = (h ^ b) * P with
// P = 2^40 + 435, which is a chain of dependent multiplies: folded by one
// thread it runs at the multiply latency per byte, several milliseconds
// for a world of a few thousand bodies.  The block instead splits the
// stream into 32-byte chunks, one per thread, and uses three facts about
// the recurrence (all arithmetic mod 2^32, on the two 32-bit halves
// lo/hi of h):
//
//  1. The low byte s of lo evolves on its own: s' = ((s ^ b) * 435) & 255.
//     Multiplication by an odd constant and XOR are triangular in the
//     bits (bit j of the result depends on bits <= j only), and bit j of
//     s' is bit j of s XOR a function of b and the bits below j.  So bit j
//     of s over the whole stream is an exclusive prefix XOR, computable
//     by a block-wide scan once bits 0..j-1 are known: eight rounds, one
//     per bit, each a bit-sliced update of 32 bytes per thread plus a
//     ballot-and-popcount XOR scan across the block.
//  2. With s known at every byte, lo ^ b = lo + ((s ^ b) - s), so
//     lo' = 435 * (lo + d) is affine in lo: each chunk is one map
//     x -> A x + C, and an ordered scan of those maps gives every chunk's
//     starting lo.
//  3. hi' = 435 * hi + umulhi(x, 435) + (x << 8) with x = lo ^ b is affine
//     in hi once the lo sequence is known: one more ordered composition
//     gives the block's final hi.
//
// The stream itself is the record sequence of m3_hash.h (header, bodies,
// shapes, joints, pair count, pairs).  Each round of the outer loop
// stages up to one record per thread of the block's first half into
// shared memory (lengths by a counting pass and a block scan, then the
// bytes) and hashes the staged bytes tile by tile, carrying (lo, hi)
// across tiles and rounds.  The
// result is bit-identical to m3WorldHashView.
//
// A large world among few is hashed over many blocks instead (one block
// took 36 ms for a world of 20,000 bodies, 46,000 joints and 121,000 pairs,
// on one SM of 148): its stream is written out once, and each of the
// facts above becomes a pass over the stream's 8 KB tiles, a block a
// tile: eight passes for the low byte's bits (a tile's bit toggles are
// one parity, and a tile's start is the parity of the tiles before it),
// one for the tiles' lo maps, one for their hi maps, and one block that
// composes them.
#include "m3_world.h"
#include "m3_hash.h"

#include <cuda_runtime.h>

#define M3H_BLOCK 256
#define M3H_WARPS (M3H_BLOCK / 32)
#define M3H_RECORD_MAX 256 // longest record of the stream
// The longest record of each kind (m3_hash.h, every optional field there).
#define M3H_BODY_MAX 196
#define M3H_SHAPE_MAX 125
#define M3H_JOINT_MAX 171
// Records staged per round: half the block, so that the stage (32 KB)
// lets four blocks share an SM (the registers allow four; a 64 KB stage
// allowed three).
#define M3H_ROUND_RECORDS (M3H_BLOCK / 2)
#define M3H_STAGE_BYTES (M3H_ROUND_RECORDS * M3H_RECORD_MAX)
#define M3H_CHUNK 32
#define M3H_TILE (M3H_BLOCK * M3H_CHUNK)
#define M3H_MUL 435u // P = 2^40 + 435

static_assert(M3H_STAGE_BYTES % M3H_TILE == 0, "tiles must cover the stage exactly");

// Writes emitted bytes into the shared-memory stage at a running offset.
struct m3StageSink
{
    uint8_t* dst;
    int32_t off;
    __device__ void put(const void* p, int32_t n)
    {
        const uint8_t* s = (const uint8_t*)p;
        uint8_t* d = dst + off;
        int32_t k = 0;
        if (((uintptr_t)s & 3u) == 0)
        {
            for (; k + 4 <= n; k += 4)
            {
                const uint32_t v = *(const uint32_t*)(s + k);
                d[k] = (uint8_t)v;
                d[k + 1] = (uint8_t)(v >> 8);
                d[k + 2] = (uint8_t)(v >> 16);
                d[k + 3] = (uint8_t)(v >> 24);
            }
        }
        for (; k < n; ++k)
        {
            d[k] = s[k];
        }
        off += n;
    }
};

struct m3HashShared
{
    uint32_t warpBits[8][M3H_WARPS];
    uint32_t warpA[M3H_WARPS];
    uint32_t warpC[M3H_WARPS];
    int32_t warpSum[M3H_WARPS];
    uint32_t pow435[M3H_CHUNK + 1];
    int32_t bad;
};

// Transpose of an 8x8 bit matrix held in a 64-bit word, rows = bytes:
// bit c of byte r moves to bit r of byte c.
__device__ __forceinline__ uint64_t Transpose8(uint64_t x)
{
    uint64_t t = (x ^ (x >> 7)) & 0x00AA00AA00AA00AAull;
    x = x ^ t ^ (t << 7);
    t = (x ^ (x >> 14)) & 0x0000CCCC0000CCCCull;
    x = x ^ t ^ (t << 14);
    t = (x ^ (x >> 28)) & 0x00000000F0F0F0F0ull;
    x = x ^ t ^ (t << 28);
    return x;
}

// Exclusive block scan of one int per thread; every thread gets its
// offset and the total.
__device__ int32_t HashBlockScan(int32_t v, int32_t* total, m3HashShared& sh)
{
    const int32_t lane = threadIdx.x & 31;
    const int32_t warp = threadIdx.x >> 5;
    int32_t x = v;
    for (int32_t o = 1; o < 32; o <<= 1)
    {
        const int32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o)
        {
            x += y;
        }
    }
    if (lane == 31)
    {
        sh.warpSum[warp] = x;
    }
    __syncthreads();
    int32_t before = 0;
    int32_t all = 0;
    for (int32_t k = 0; k < M3H_WARPS; ++k)
    {
        const int32_t s = sh.warpSum[k];
        before += k < warp ? s : 0;
        all += s;
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

// Ordered composition of the threads' affine maps x -> A x + C (thread 0
// first).  Returns, per thread, the composition of all earlier threads'
// maps (exA, exC) and, to every thread, the composition of all of them.
__device__ void AffineBlockScan(uint32_t A, uint32_t C, uint32_t* exA, uint32_t* exC,
                                uint32_t* totA, uint32_t* totC, m3HashShared& sh)
{
    const int32_t lane = threadIdx.x & 31;
    const int32_t warp = threadIdx.x >> 5;
    uint32_t iA = A;
    uint32_t iC = C;
    for (int32_t o = 1; o < 32; o <<= 1)
    {
        const uint32_t a2 = __shfl_up_sync(0xFFFFFFFFu, iA, o);
        const uint32_t c2 = __shfl_up_sync(0xFFFFFFFFu, iC, o);
        if (lane >= o)
        {
            // Earlier map first, then this one.
            iC = iA * c2 + iC;
            iA = iA * a2;
        }
    }
    uint32_t eA = __shfl_up_sync(0xFFFFFFFFu, iA, 1);
    uint32_t eC = __shfl_up_sync(0xFFFFFFFFu, iC, 1);
    if (lane == 0)
    {
        eA = 1u;
        eC = 0u;
    }
    if (lane == 31)
    {
        sh.warpA[warp] = iA;
        sh.warpC[warp] = iC;
    }
    __syncthreads();
    uint32_t pA = 1u;
    uint32_t pC = 0u;
    uint32_t tA = 1u;
    uint32_t tC = 0u;
    for (int32_t k = 0; k < M3H_WARPS; ++k)
    {
        const uint32_t a2 = sh.warpA[k];
        const uint32_t c2 = sh.warpC[k];
        if (k < warp)
        {
            pC = a2 * pC + c2;
            pA = a2 * pA;
        }
        tC = a2 * tC + c2;
        tA = a2 * tA;
    }
    __syncthreads();
    *exC = eA * pC + eC;
    *exA = eA * pA;
    *totA = tA;
    *totC = tC;
}

// One thread's 32-byte chunk of a tile of n bytes: its words, its bit
// planes (bit i of B[j] = bit j of byte i) and which bytes exist.
struct m3HashChunk
{
    uint32_t wd[8];
    uint32_t B[8];
    uint32_t valid;
    int32_t cnt;
};

__device__ __forceinline__ void LoadChunk(const uint8_t* tile, int32_t n, m3HashChunk& c)
{
    const int32_t tid = threadIdx.x;
    int32_t cnt = n - tid * M3H_CHUNK;
    cnt = cnt < 0 ? 0 : (cnt > M3H_CHUNK ? M3H_CHUNK : cnt);
    c.cnt = cnt;
    c.valid = cnt >= 32 ? 0xFFFFFFFFu : ((1u << cnt) - 1u);
    if (cnt > 0)
    {
        const uint4* src = (const uint4*)(tile + tid * M3H_CHUNK);
        const uint4 q0 = src[0];
        const uint4 q1 = src[1];
        c.wd[0] = q0.x;
        c.wd[1] = q0.y;
        c.wd[2] = q0.z;
        c.wd[3] = q0.w;
        c.wd[4] = q1.x;
        c.wd[5] = q1.y;
        c.wd[6] = q1.z;
        c.wd[7] = q1.w;
    }
    else
    {
#pragma unroll
        for (int32_t k = 0; k < 8; ++k)
        {
            c.wd[k] = 0u;
        }
    }
#pragma unroll
    for (int32_t j = 0; j < 8; ++j)
    {
        c.B[j] = 0u;
    }
#pragma unroll
    for (int32_t g = 0; g < 4; ++g)
    {
        const uint64_t y = Transpose8((uint64_t)c.wd[2 * g] | ((uint64_t)c.wd[2 * g + 1] << 32));
#pragma unroll
        for (int32_t j = 0; j < 8; ++j)
        {
            c.B[j] |= (uint32_t)((y >> (8 * j)) & 0xFFu) << (8 * g);
        }
    }
}

// Rounds 0 .. ROUNDS - 1: plane j of S is bit j of the low byte before
// every byte of the tile, which starts at the low byte s0 (its bits below
// ROUNDS matter).  Returns the parity of the tile's toggles in the last
// round's bit.
template <int ROUNDS>
__device__ __forceinline__ uint32_t LowPlanes(const m3HashChunk& chunk, uint32_t s0, uint32_t S[8],
                                              m3HashShared& sh)
{
    const int32_t lane = threadIdx.x & 31;
    const int32_t warp = threadIdx.x >> 5;
    // acc holds, bit-sliced, ((s ^ b) mod 2^j) * 435 mod 256 for every
    // byte, i.e. the part of the product known from the lower bits.
    uint32_t acc[8];
#pragma unroll
    for (int32_t j = 0; j < 8; ++j)
    {
        acc[j] = 0u;
    }
    uint32_t parity = 0u;
    const uint32_t ltMask = (1u << lane) - 1u;
#pragma unroll
    for (int32_t j = 0; j < ROUNDS; ++j)
    {
        // s'_j = s_j ^ b_j ^ acc_j: the toggles, prefix-XORed.
        const uint32_t T = (chunk.B[j] ^ acc[j]) & chunk.valid;
        uint32_t Q = T << 1;
        Q ^= Q << 1;
        Q ^= Q << 2;
        Q ^= Q << 4;
        Q ^= Q << 8;
        Q ^= Q << 16;
        const uint32_t ballot = __ballot_sync(0xFFFFFFFFu, (__popc(T) & 1) != 0);
        if (lane == 0)
        {
            sh.warpBits[j][warp] = (uint32_t)(__popc(ballot) & 1);
        }
        __syncthreads();
        if (j == ROUNDS - 1)
        {
            for (int32_t k = 0; k < M3H_WARPS; ++k)
            {
                parity ^= sh.warpBits[j][k];
            }
        }
        uint32_t carry = ((s0 >> j) & 1u) ^ ((uint32_t)__popc(ballot & ltMask) & 1u);
        for (int32_t k = 0; k < warp; ++k)
        {
            carry ^= sh.warpBits[j][k];
        }
        S[j] = Q ^ (0u - carry);
        // Add x_j * 435 * 2^j (435 = 0b110110011 = 256 + 179; mod 256 the
        // multiplier is 179 = 2^7 + 2^5 + 2^4 + 2^1 + 2^0).
        const uint32_t X = S[j] ^ chunk.B[j];
#pragma unroll
        for (int32_t o = 0; o < 8; ++o)
        {
            if (((179 >> o) & 1) == 0 || j + o >= 8)
            {
                continue;
            }
            uint32_t c = X;
#pragma unroll
            for (int32_t q = j + o; q < 8; ++q)
            {
                const uint32_t t2 = acc[q] & c;
                acc[q] ^= c;
                c = t2;
            }
        }
    }
    return parity;
}

// The chunk's lo map from its low-byte planes: lo' = 435 * (lo + ((s ^ b)
// - s)) per byte, A lo + C in all (A is 435 to the chunk's length).
__device__ __forceinline__ uint32_t ChunkLo(const m3HashChunk& chunk, const uint32_t S[8])
{
    // Low bytes back to byte order.
    uint32_t sw[8];
#pragma unroll
    for (int32_t g = 0; g < 4; ++g)
    {
        uint64_t z = 0;
#pragma unroll
        for (int32_t j = 0; j < 8; ++j)
        {
            z |= (uint64_t)((S[j] >> (8 * g)) & 0xFFu) << (8 * j);
        }
        const uint64_t y = Transpose8(z);
        sw[2 * g] = (uint32_t)y;
        sw[2 * g + 1] = (uint32_t)(y >> 32);
    }
    uint32_t C = 0u;
#pragma unroll
    for (int32_t k = 0; k < M3H_CHUNK; ++k)
    {
        if (k < chunk.cnt)
        {
            const uint32_t s = (sw[k >> 2] >> (8 * (k & 3))) & 0xFFu;
            const uint32_t b = (chunk.wd[k >> 2] >> (8 * (k & 3))) & 0xFFu;
            C = M3H_MUL * (C + ((s ^ b) - s));
        }
    }
    return C;
}

// The chunk's hi map from lo before it: hi' = 435 * hi + umulhi(x, 435) +
// (x << 8) per byte with x = lo ^ b.
__device__ __forceinline__ uint32_t ChunkHi(const m3HashChunk& chunk, uint32_t lo)
{
    uint32_t H = 0u;
#pragma unroll
    for (int32_t k = 0; k < M3H_CHUNK; ++k)
    {
        if (k < chunk.cnt)
        {
            const uint32_t b = (chunk.wd[k >> 2] >> (8 * (k & 3))) & 0xFFu;
            const uint32_t x = lo ^ b;
            H = M3H_MUL * H + (__umulhi(x, M3H_MUL) + (x << 8));
            lo = x * M3H_MUL;
        }
    }
    return H;
}

// Folds tile[0, n) (n <= M3H_TILE) into (lo, hi); every thread of the
// block calls it with the same arguments and gets the same result.
__device__ void FnvTile(const uint8_t* tile, int32_t n, uint32_t& lo, uint32_t& hi,
                        m3HashShared& sh)
{
    m3HashChunk chunk;
    uint32_t S[8];
    LoadChunk(tile, n, chunk);
    LowPlanes<8>(chunk, lo & 0xFFu, S, sh);
    const uint32_t C = ChunkLo(chunk, S);
    const uint32_t A = sh.pow435[chunk.cnt];
    uint32_t exA;
    uint32_t exC;
    uint32_t totA;
    uint32_t totC;
    AffineBlockScan(A, C, &exA, &exC, &totA, &totC, sh);
    const uint32_t H = ChunkHi(chunk, exA * lo + exC);
    const uint32_t loEnd = totA * lo + totC;
    uint32_t hA;
    uint32_t hC;
    AffineBlockScan(A, H, &exA, &exC, &hA, &hC, sh);
    lo = loEnd;
    hi = hA * hi + hC;
}

// The powers of 435 a chunk's length needs; read after a barrier.
__device__ __forceinline__ void HashPowers(m3HashShared& sh)
{
    const int32_t tid = threadIdx.x;
    if (tid <= M3H_CHUNK)
    {
        uint32_t p = 1u;
        for (int32_t k = 0; k < tid; ++k)
        {
            p *= M3H_MUL;
        }
        sh.pow435[tid] = p;
    }
}

__global__ void __launch_bounds__(M3H_BLOCK, 5) m3HashKernel(const m3WorldView* views,
                                                          const int32_t* order, int32_t count,
                                                          uint64_t* out)
{
    const int32_t wi = order[blockIdx.x];
    const m3WorldView* w = &views[wi];
    extern __shared__ __align__(16) uint8_t s_stage[];
    __shared__ m3HashShared sh;
    const int32_t tid = threadIdx.x;
    HashPowers(sh);
    if (tid == 0)
    {
        sh.bad = 0;
    }
    __syncthreads();
    const int32_t records = m3HashRecordCount(w);
    uint32_t lo = (uint32_t)M3_HASH_INIT;
    uint32_t hi = (uint32_t)(M3_HASH_INIT >> 32);
    for (int32_t r0 = 0; r0 < records; r0 += M3H_ROUND_RECORDS)
    {
        const int32_t r = r0 + tid;
        int32_t len = 0;
        if (tid < M3H_ROUND_RECORDS && r < records)
        {
            m3CountSink c{0};
            m3HashRecord(w, r, c);
            len = c.n;
            if (len > M3H_RECORD_MAX)
            {
                // Cannot happen with this record set; never overrun the stage.
                sh.bad = 1;
                len = 0;
            }
        }
        int32_t total = 0;
        const int32_t off = HashBlockScan(len, &total, sh);
        if (len > 0)
        {
            m3StageSink k{s_stage, off};
            m3HashRecord(w, r, k);
        }
        __syncthreads();
        for (int32_t base = 0; base < total; base += M3H_TILE)
        {
            const int32_t n = total - base < M3H_TILE ? total - base : M3H_TILE;
            FnvTile(s_stage + base, n, lo, hi, sh);
        }
        __syncthreads();
    }
    if (tid == 0)
    {
        out[wi] = sh.bad != 0 ? 0ull : (((uint64_t)hi << 32) | lo);
    }
}

// ---------------------------------------------------------------------
// Large worlds over many blocks.  blockIdx.y is the world's job, the
// blocks of a row stride over its record blocks or tiles.  The job's
// working words: [0] the stream's bytes, then one sum per record block,
// eight bit arrays of the tiles' parities, and the tiles' maps.
// ---------------------------------------------------------------------
struct m3HashWork
{
    uint32_t* bytes;
    uint32_t* sums;  // per M3H_ROUND_RECORDS records: their bytes
    uint32_t* bits;  // 8 arrays of `words`: a tile's parity a bit
    uint32_t* mapA;  // per tile: lo' = A lo + C, hi' = A hi + H
    uint32_t* mapC;
    uint32_t* mapH;
    int32_t words;
};

// The stream's bytes; a stream beyond the job's tiles cannot happen with
// this record set (it would end as the hash 0, and never overrun them).
__device__ __forceinline__ int32_t StreamBytes(const m3HashJob& job, const m3HashWork& work)
{
    const uint32_t cap = (uint32_t)job.tiles * M3H_TILE;
    return (int32_t)(*work.bytes < cap ? *work.bytes : cap);
}

__device__ __forceinline__ m3HashWork HashWork(const m3HashJob& job)
{
    const int32_t tiles = job.tiles;
    m3HashWork k;
    k.words = (tiles + 31) / 32;
    k.bytes = job.work;
    k.sums = job.work + 8;
    k.bits = k.sums + job.recordBlocks;
    k.mapA = k.bits + 8 * k.words;
    k.mapC = k.mapA + tiles;
    k.mapH = k.mapC + tiles;
    return k;
}

// Words of a job of at most `tiles` tiles and `recordBlocks` record blocks.
static int64_t HashWorkWords(int64_t tiles, int64_t recordBlocks)
{
    return 8 + recordBlocks + 8 * ((tiles + 31) / 32) + 3 * tiles;
}

__global__ void __launch_bounds__(M3H_BLOCK) m3HashLengthKernel(const __grid_constant__ m3HashJobs jobs)
{
    const m3HashJob& job = jobs.job[blockIdx.y];
    const m3WorldView* w = job.view;
    const m3HashWork work = HashWork(job);
    __shared__ int32_t s_warp[M3H_WARPS];
    const int32_t records = m3HashRecordCount(w);
    const int32_t lane = threadIdx.x & 31;
    const int32_t warp = threadIdx.x >> 5;
    for (int32_t i = blockIdx.x * M3H_BLOCK + threadIdx.x; i < 8 * work.words;
         i += gridDim.x * M3H_BLOCK)
    {
        work.bits[i] = 0u;
    }
    for (int32_t r0 = blockIdx.x * M3H_BLOCK; r0 < records; r0 += gridDim.x * M3H_BLOCK)
    {
        const int32_t r = r0 + threadIdx.x;
        int32_t len = 0;
        if (r < records)
        {
            m3CountSink c{0};
            m3HashRecord(w, r, c);
            len = c.n;
        }
        for (int32_t o = 16; o > 0; o >>= 1)
        {
            len += __shfl_xor_sync(0xFFFFFFFFu, len, o);
        }
        if (lane == 0)
        {
            s_warp[warp] = len;
        }
        __syncthreads();
        const int32_t half = M3H_WARPS / 2;
        if (threadIdx.x < 2 && r0 + (int32_t)threadIdx.x * M3H_ROUND_RECORDS < records)
        {
            int32_t sum = 0;
            for (int32_t k = 0; k < half; ++k)
            {
                sum += s_warp[threadIdx.x * half + k];
            }
            work.sums[r0 / M3H_ROUND_RECORDS + threadIdx.x] = (uint32_t)sum;
        }
        __syncthreads();
    }
}

// Sum of v over the block, the same in every thread.
__device__ uint32_t HashBlockSum(uint32_t v, m3HashShared& sh)
{
    for (int32_t o = 16; o > 0; o >>= 1)
    {
        v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        sh.warpA[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    uint32_t all = 0;
    for (int32_t k = 0; k < M3H_WARPS; ++k)
    {
        all += sh.warpA[k];
    }
    __syncthreads();
    return all;
}

// Writes the stream: a record block is laid out in shared memory at its
// place's alignment, then copied 16 bytes at a time.
__global__ void __launch_bounds__(M3H_BLOCK) m3HashStreamKernel(const __grid_constant__ m3HashJobs jobs)
{
    const m3HashJob& job = jobs.job[blockIdx.y];
    const m3WorldView* w = job.view;
    const m3HashWork work = HashWork(job);
    extern __shared__ __align__(16) uint8_t s_stage[];
    __shared__ m3HashShared sh;
    const int32_t tid = threadIdx.x;
    const int32_t records = m3HashRecordCount(w);
    const int32_t recordBlocks = (records + M3H_ROUND_RECORDS - 1) / M3H_ROUND_RECORDS;
    for (int32_t rb = blockIdx.x; rb < recordBlocks; rb += gridDim.x)
    {
        uint32_t before = 0;
        for (int32_t k = tid; k < rb; k += M3H_BLOCK)
        {
            before += work.sums[k];
        }
        const uint32_t base = HashBlockSum(before, sh);
        const int32_t r = rb * M3H_ROUND_RECORDS + tid;
        int32_t len = 0;
        if (tid < M3H_ROUND_RECORDS && r < records)
        {
            m3CountSink c{0};
            m3HashRecord(w, r, c);
            len = c.n;
        }
        int32_t total = 0;
        const int32_t off = HashBlockScan(len, &total, sh);
        const int32_t shift = (int32_t)(base & 15u);
        if (len > 0)
        {
            m3StageSink k{s_stage + shift, off};
            m3HashRecord(w, r, k);
        }
        __syncthreads();
        // Stream bytes [base, base + total) = stage bytes [shift, end).
        uint8_t* to = job.stream + (base - (uint32_t)shift);
        const bool fits = (int64_t)base + total <= (int64_t)job.tiles * M3H_TILE;
        const int32_t end = fits ? shift + total : shift;
        const int32_t head = shift == 0 ? 0 : 16;
        const int32_t tail = end & ~15;
        for (int32_t k = head + 16 * tid; k < tail; k += 16 * M3H_BLOCK)
        {
            *(uint4*)(to + k) = *(const uint4*)(s_stage + k);
        }
        if (tid < 16 && tid >= shift && tid < head && tid < end)
        {
            to[tid] = s_stage[tid];
        }
        if (tid >= 16 && tid < 32 && tail >= head && tail + tid - 16 < end)
        {
            to[tail + tid - 16] = s_stage[tail + tid - 16];
        }
        if (rb == recordBlocks - 1 && tid == 0)
        {
            *work.bytes = base + (uint32_t)total;
        }
        __syncthreads();
    }
}

// The low byte's bits below BITS at the start of tile t: the parities of
// the tiles before it, on the stream's first low byte (warp j counts bit j).
template <int BITS>
__device__ uint32_t TileLow(const m3HashWork& work, int32_t t, m3HashShared& sh)
{
    const int32_t lane = threadIdx.x & 31;
    const int32_t warp = threadIdx.x >> 5;
    uint32_t odd = 0;
    if (warp < BITS)
    {
        const uint32_t* bits = work.bits + warp * work.words;
        for (int32_t k = lane; k <= t >> 5; k += 32)
        {
            const uint32_t mask = k < t >> 5 ? 0xFFFFFFFFu : (1u << (t & 31)) - 1u;
            odd ^= (uint32_t)__popc(bits[k] & mask) & 1u;
        }
        odd = (uint32_t)__popc(__ballot_sync(0xFFFFFFFFu, odd != 0)) & 1u;
    }
    if (lane == 0)
    {
        sh.warpC[warp] = odd << warp;
    }
    __syncthreads();
    uint32_t low = (uint32_t)M3_HASH_INIT & 0xFFu;
    for (int32_t k = 0; k < M3H_WARPS; ++k)
    {
        low ^= sh.warpC[k];
    }
    __syncthreads();
    return low;
}

template <int BIT>
__global__ void __launch_bounds__(M3H_BLOCK) m3HashBitKernel(const __grid_constant__ m3HashJobs jobs)
{
    const m3HashJob& job = jobs.job[blockIdx.y];
    const m3HashWork work = HashWork(job);
    __shared__ m3HashShared sh;
    const int32_t bytes = StreamBytes(job, work);
    for (int32_t t = blockIdx.x; t * (int64_t)M3H_TILE < bytes; t += gridDim.x)
    {
        const int32_t base = t * M3H_TILE;
        const uint32_t low = TileLow<BIT>(work, t, sh);
        m3HashChunk chunk;
        uint32_t S[8];
        LoadChunk(job.stream + base, bytes - base < M3H_TILE ? bytes - base : M3H_TILE, chunk);
        const uint32_t parity = LowPlanes<BIT + 1>(chunk, low, S, sh);
        if (threadIdx.x == 0 && parity != 0)
        {
            atomicOr(&work.bits[BIT * work.words + (t >> 5)], 1u << (t & 31));
        }
        __syncthreads();
    }
}

// Each tile's lo map (HI false), or its hi map from the lo its start has
// (the maps of the tiles before it, composed).
template <bool HI>
__global__ void __launch_bounds__(M3H_BLOCK) m3HashMapKernel(const __grid_constant__ m3HashJobs jobs)
{
    const m3HashJob& job = jobs.job[blockIdx.y];
    const m3HashWork work = HashWork(job);
    __shared__ m3HashShared sh;
    HashPowers(sh);
    __syncthreads();
    const int32_t bytes = StreamBytes(job, work);
    for (int32_t t = blockIdx.x; t * (int64_t)M3H_TILE < bytes; t += gridDim.x)
    {
        const int32_t base = t * M3H_TILE;
        uint32_t exA;
        uint32_t exC;
        uint32_t totA;
        uint32_t totC;
        uint32_t lo = (uint32_t)M3_HASH_INIT;
        if (HI)
        {
            const int32_t per = (t + M3H_BLOCK - 1) / M3H_BLOCK;
            uint32_t A = 1u;
            uint32_t C = 0u;
            for (int32_t k = threadIdx.x * per; k < ((int32_t)threadIdx.x + 1) * per && k < t; ++k)
            {
                C = work.mapA[k] * C + work.mapC[k];
                A = work.mapA[k] * A;
            }
            AffineBlockScan(A, C, &exA, &exC, &totA, &totC, sh);
            lo = totA * lo + totC;
        }
        const uint32_t low = TileLow<8>(work, t, sh);
        m3HashChunk chunk;
        uint32_t S[8];
        LoadChunk(job.stream + base, bytes - base < M3H_TILE ? bytes - base : M3H_TILE, chunk);
        LowPlanes<8>(chunk, low, S, sh);
        const uint32_t A = sh.pow435[chunk.cnt];
        AffineBlockScan(A, ChunkLo(chunk, S), &exA, &exC, &totA, &totC, sh);
        if (HI)
        {
            AffineBlockScan(A, ChunkHi(chunk, exA * lo + exC), &exA, &exC, &totA, &totC, sh);
        }
        if (threadIdx.x == 0)
        {
            work.mapA[t] = totA;
            (HI ? work.mapH : work.mapC)[t] = totC;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(M3H_BLOCK) m3HashFinalKernel(const __grid_constant__ m3HashJobs jobs)
{
    const m3HashJob& job = jobs.job[blockIdx.x];
    const m3HashWork work = HashWork(job);
    __shared__ m3HashShared sh;
    const int32_t tiles = (StreamBytes(job, work) + M3H_TILE - 1) / M3H_TILE;
    const int32_t per = (tiles + M3H_BLOCK - 1) / M3H_BLOCK;
    uint32_t A = 1u;
    uint32_t C = 0u;
    uint32_t H = 0u;
    for (int32_t k = threadIdx.x * per; k < ((int32_t)threadIdx.x + 1) * per && k < tiles; ++k)
    {
        C = work.mapA[k] * C + work.mapC[k];
        H = work.mapA[k] * H + work.mapH[k];
        A = work.mapA[k] * A;
    }
    uint32_t exA;
    uint32_t exC;
    uint32_t totA;
    uint32_t loC;
    uint32_t hiC;
    AffineBlockScan(A, C, &exA, &exC, &totA, &loC, sh);
    AffineBlockScan(A, H, &exA, &exC, &totA, &hiC, sh);
    if (threadIdx.x == 0)
    {
        const uint32_t lo = totA * (uint32_t)M3_HASH_INIT + loC;
        const uint32_t hi = totA * (uint32_t)(M3_HASH_INIT >> 32) + hiC;
        *job.out = *work.bytes <= (uint32_t)job.tiles * M3H_TILE ? ((uint64_t)hi << 32) | lo : 0ull;
    }
}

// Fills in a job's sizes; false when the working memory cannot hold the
// world's longest stream.
bool m3gpuHashJobFits(m3HashJob* job, int64_t streamBytes, int64_t workBytes, int64_t bodies,
                      int64_t shapes, int64_t joints, int64_t pairs)
{
    const int64_t records = 2 + bodies + shapes + joints + pairs;
    const int64_t bytes = 2 * M3H_RECORD_MAX + M3H_BODY_MAX * bodies + M3H_SHAPE_MAX * shapes +
                          M3H_JOINT_MAX * joints +
                          (int64_t)(sizeof(uint64_t) + sizeof(m3Manifold)) * pairs;
    const int64_t tiles = (bytes + M3H_TILE - 1) / M3H_TILE;
    const int64_t recordBlocks = (records + M3H_ROUND_RECORDS - 1) / M3H_ROUND_RECORDS;
    job->tiles = (int32_t)tiles;
    job->recordBlocks = (int32_t)recordBlocks;
    // The last tile's chunks are read whole.
    return bytes < INT32_MAX - M3H_TILE && tiles * M3H_TILE <= streamBytes &&
           4 * HashWorkWords(tiles, recordBlocks) <= workBytes;
}

// Launches the passes of `count` jobs; the number of kernels, or a negative
// error code.
int32_t m3gpuLaunchHashJobs(const m3HashJobs& jobs, int32_t count)
{
    static int s_configured = -1;
    const int32_t stage = M3H_STAGE_BYTES + 16;
    int device = 0;
    cudaGetDevice(&device);
    if (s_configured != device)
    {
        const cudaError_t e = cudaFuncSetAttribute(
            m3HashStreamKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, stage);
        if (e != cudaSuccess)
        {
            return -m3gpuSetError(M3GPU_ERR_CUDA, "cudaFuncSetAttribute(hash stage): %s",
                                  cudaGetErrorString(e));
        }
        s_configured = device;
    }
    // Blocks a job: all of its tiles at once, up to four blocks an SM over
    // the jobs.
    int32_t most = 1;
    for (int32_t k = 0; k < count; ++k)
    {
        most = jobs.job[k].tiles > most ? jobs.job[k].tiles : most;
    }
    const int32_t share = (148 * 4 + count - 1) / count;
    const dim3 grid((uint32_t)(most < share ? most : share), (uint32_t)count);
    m3HashLengthKernel<<<grid, M3H_BLOCK>>>(jobs);
    m3HashStreamKernel<<<grid, M3H_BLOCK, stage>>>(jobs);
    m3HashBitKernel<0><<<grid, M3H_BLOCK>>>(jobs);
    m3HashBitKernel<1><<<grid, M3H_BLOCK>>>(jobs);
    m3HashBitKernel<2><<<grid, M3H_BLOCK>>>(jobs);
    m3HashBitKernel<3><<<grid, M3H_BLOCK>>>(jobs);
    m3HashBitKernel<4><<<grid, M3H_BLOCK>>>(jobs);
    m3HashBitKernel<5><<<grid, M3H_BLOCK>>>(jobs);
    m3HashBitKernel<6><<<grid, M3H_BLOCK>>>(jobs);
    m3HashBitKernel<7><<<grid, M3H_BLOCK>>>(jobs);
    m3HashMapKernel<false><<<grid, M3H_BLOCK>>>(jobs);
    m3HashMapKernel<true><<<grid, M3H_BLOCK>>>(jobs);
    m3HashFinalKernel<<<count, M3H_BLOCK>>>(jobs);
    return 13;
}

int32_t m3gpuLaunchHash(const m3WorldView* views, const int32_t* order, int32_t count,
                        uint64_t* out)
{
    static int s_configured = -1;
    int device = 0;
    cudaGetDevice(&device);
    if (s_configured != device)
    {
        cudaError_t e = cudaFuncSetAttribute(
            m3HashKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, M3H_STAGE_BYTES);
        if (e != cudaSuccess)
        {
            return m3gpuSetError(M3GPU_ERR_CUDA, "cudaFuncSetAttribute(hash smem): %s",
                                 cudaGetErrorString(e));
        }
        s_configured = device;
    }
    if (count > 0)
    {
        m3HashKernel<<<count, M3H_BLOCK, M3H_STAGE_BYTES>>>(views, order, count, out);
    }
    return M3GPU_OK;
}
