// partition.cu -- stable multi-split radix sort of (key, index) pairs and the
// partition (split) search of MRay's RayPartitioner::MultiPartition
// (Source/Tracer/RayPartitioner.cu:263-411, split kernels :19-75).
//
// MRay sorts with CUB's radix sort and finds the splits with a binary
// partition, waiting on the host in between.  Here one radix digit (up to 8
// bits, 256 buckets) is one pass of three kernels:
//   hist     per-tile bucket counts (shared-memory atomics) and bucket totals
//   rows     a block per bucket scans its row of the (bucket, tile) count table
//   scatter  stable ranks inside each tile (warp match against per-warp counts
//            in shared memory), written to the bucket's global offset
// The element count may live in device memory (a path tracer's alive count),
// so a pass is enqueued without knowing it; the grid is sized for an upper
// bound and tiles past the count contribute nothing.
#include "mrg_partition.h"

namespace mrg {

namespace {

constexpr int kMsTPB = 256;
constexpr int kMsItems = 8;
constexpr int kMsTile = kMsTPB * kMsItems;     // 2048 elements per tile
constexpr int kMsWarps = kMsTPB / 32;
constexpr int kScanTPB = 1024;
constexpr uint32_t kMsEmpty = 0xFFFFFFFFu;      // an empty key (DigitSpec::dropEmpty)

__device__ __forceinline__ uint32_t bits_of(uint32_t v, uint32_t shift, uint32_t width)
{
    return (width >= 32u) ? (v >> shift) : ((v >> shift) & ((1u << width) - 1u));
}

// Composite sort key: batch bits above data bits (or batch bits alone).
__device__ __forceinline__ uint32_t digit_of(const DigitSpec& s, uint32_t key)
{
    uint32_t c = bits_of(key, s.batchShift, s.batchWidth);
    if(s.dataWidth) c = (c << s.dataWidth) | bits_of(key, s.dataShift, s.dataWidth);
    return bits_of(c, s.digitShift, s.digitBits);
}

__device__ __forceinline__ uint32_t count_of(const uint32_t* nDevice, uint32_t nHost)
{
    return nDevice ? *nDevice : nHost;
}

// Bucket counts of one tile, and their sums over all tiles.
__global__ void __launch_bounds__(kMsTPB)
k_ms_hist(const uint32_t* __restrict__ keys, const uint32_t* nDevice, uint32_t nHost, DigitSpec spec,
          uint32_t* __restrict__ hist, uint32_t numTiles, uint32_t* __restrict__ totals)
{
    __shared__ uint32_t sHist[256];
    const uint32_t nb = 1u << spec.digitBits;
    for(uint32_t b = threadIdx.x; b < nb; b += kMsTPB) sHist[b] = 0u;
    __syncthreads();
    const uint32_t n = count_of(nDevice, nHost);
    const uint32_t tileStart = blockIdx.x * (uint32_t)kMsTile;
    uint32_t key[kMsItems];
#pragma unroll
    for(int r = 0; r < kMsItems; r++)
    {
        const uint32_t e = tileStart + (uint32_t)r * kMsTPB + threadIdx.x;
        key[r] = (e < n) ? __ldg(&keys[e]) : kMsEmpty;
    }
#pragma unroll
    for(int r = 0; r < kMsItems; r++)
    {
        const uint32_t e = tileStart + (uint32_t)r * kMsTPB + threadIdx.x;
        if(e < n && !(spec.dropEmpty && key[r] == kMsEmpty)) atomicAdd(&sHist[digit_of(spec, key[r])], 1u);
    }
    __syncthreads();
    for(uint32_t b = threadIdx.x; b < nb; b += kMsTPB)
    {
        hist[(size_t)b * numTiles + blockIdx.x] = sHist[b];
        if(sHist[b]) atomicAdd(&totals[b], sHist[b]);
    }
}

// Exclusive scan of v across the block; the block's total in *total.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t sWarp[kScanTPB / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for(int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if(lane >= (uint32_t)o) x += y;
    }
    if(lane == 31u) sWarp[warp] = x;
    __syncthreads();
    if(warp == 0)
    {
        uint32_t w = (lane < kScanTPB / 32) ? sWarp[lane] : 0u;
#pragma unroll
        for(int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if(lane >= (uint32_t)o) w += y;
        }
        if(lane < kScanTPB / 32) sWarp[lane] = w;
    }
    __syncthreads();
    const uint32_t before = (warp ? sWarp[warp - 1] : 0u) + x - v;
    *total = sWarp[kScanTPB / 32 - 1];
    __syncthreads();
    return before;
}

// Output offsets: block b turns bucket b's row of tile counts into positions,
// from the sum of the buckets before it.  One launch for any table size; a
// one-block scan, or three kernels over tables past 65,536 counts (6.6 us for
// 262,144), did this before.
__global__ void __launch_bounds__(kScanTPB)
k_ms_rows(uint32_t* __restrict__ hist, uint32_t numTiles, const uint32_t* __restrict__ totals, uint32_t* nOut)
{
    const uint32_t b = blockIdx.x;
    uint32_t carry;
    block_exclusive(threadIdx.x < b ? totals[threadIdx.x] : 0u, &carry);      // at most 256 buckets
    if(nOut && b == gridDim.x - 1u && threadIdx.x == 0u) *nOut = carry + totals[b];
    uint32_t* row = hist + (size_t)b * numTiles;
    for(uint32_t t = 0; t < numTiles; t += kScanTPB)
    {
        const uint32_t i = t + threadIdx.x;
        const uint32_t v = (i < numTiles) ? row[i] : 0u;
        uint32_t total;
        const uint32_t before = block_exclusive(v, &total);
        if(i < numTiles) row[i] = carry + before;
        carry += total;
    }
}

// Stable scatter of one tile.  Each warp takes 256 consecutive elements and
// ranks them against its own counters (no block barrier), one pass over the
// buckets turns the eight warps' counts into output positions, and every
// element goes to its position.  Bound by latency and the scattered writes:
// 2.1M elements, 8 bits, in 9.0 us; ranking 256 elements of the whole
// block at a time, with four barriers each, took 17.8 us.
__global__ void __launch_bounds__(kMsTPB)
k_ms_scatter(const uint32_t* keysIn, const uint32_t* __restrict__ idxIn,
             uint32_t* __restrict__ keysOut, uint32_t* __restrict__ idxOut,
             const uint32_t* nDevice, uint32_t nHost, DigitSpec spec,
             const uint32_t* __restrict__ hist, uint32_t numTiles, uint32_t* emptied)
{
    __shared__ uint32_t sCount[kMsWarps][256];
    const uint32_t nb = 1u << spec.digitBits;
    const uint32_t n = count_of(nDevice, nHost);
    const uint32_t tileStart = blockIdx.x * (uint32_t)kMsTile;
    if(tileStart >= n) return;                              // block-uniform
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lowerMask = (1u << lane) - 1u;
    for(uint32_t b = lane; b < nb; b += 32u) sCount[warp][b] = 0u;
    __syncwarp();
    const uint32_t first = tileStart + warp * (uint32_t)(kMsTile / kMsWarps);
    uint32_t key[kMsItems], digit[kMsItems], rank[kMsItems];
#pragma unroll
    for(int r = 0; r < kMsItems; r++)
    {
        const uint32_t e = first + (uint32_t)r * 32u + lane;
        key[r] = (e < n) ? keysIn[e] : kMsEmpty;
    }
#pragma unroll
    for(int r = 0; r < kMsItems; r++)
    {
        const uint32_t e = first + (uint32_t)r * 32u + lane;
        const bool valid = e < n && !(spec.dropEmpty && key[r] == kMsEmpty);
        const uint32_t d = valid ? digit_of(spec, key[r]) : 0xFFFFFFFFu;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t before = valid ? sCount[warp][d] : 0u;
        __syncwarp();
        if(valid && (peers & lowerMask) == 0u) sCount[warp][d] = before + (uint32_t)__popc(peers);
        __syncwarp();
        digit[r] = d;
        rank[r] = before + (uint32_t)__popc(peers & lowerMask);
        if(spec.dropEmpty && valid) emptied[e] = kMsEmpty;
    }
    __syncthreads();
    for(uint32_t b = threadIdx.x; b < nb; b += kMsTPB)
    {
        uint32_t at = hist[(size_t)b * numTiles + blockIdx.x];
#pragma unroll
        for(int w = 0; w < kMsWarps; w++)
        {
            const uint32_t c = sCount[w][b];
            sCount[w][b] = at;
            at += c;
        }
    }
    __syncthreads();
#pragma unroll
    for(int r = 0; r < kMsItems; r++)
    {
        if(digit[r] == 0xFFFFFFFFu) continue;
        const uint32_t e = first + (uint32_t)r * 32u + lane;
        const uint32_t pos = sCount[warp][digit[r]] + rank[r];
        keysOut[pos] = key[r];
        idxOut[pos] = idxIn ? idxIn[e] : e;
    }
}

// KCFindSplits: mark 1 where the batch portion changes (and at 0).
__global__ void k_find_splits(const uint32_t* __restrict__ sortedKeys, const uint32_t* nDevice, uint32_t nHost,
                              uint32_t batchShift, uint32_t batchWidth, uint32_t* __restrict__ marks)
{
    const uint32_t n = count_of(nDevice, nHost);
    for(uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x)
    {
        const uint32_t k = bits_of(sortedKeys[j], batchShift, batchWidth);
        marks[j] = (j == 0u) ? 1u : (k != bits_of(sortedKeys[j - 1], batchShift, batchWidth) ? 1u : 0u);
    }
}

// KCFindBinMatIds: partition start offsets and keys from the compacted split
// positions (bucket 1 of a one-bit multi-split of the marks).
__global__ void k_bins(const uint32_t* __restrict__ splitPos, const uint32_t* __restrict__ sortedKeys,
                       const uint32_t* nDevice, uint32_t nHost, const uint32_t* __restrict__ scannedHist,
                       uint32_t numTiles, uint32_t maxPartitions,
                       uint32_t* __restrict__ count, uint32_t* __restrict__ offsets, uint32_t* __restrict__ binKeys)
{
    const uint32_t n = count_of(nDevice, nHost);
    // bucket 1 starts after every zero mark
    const uint32_t ones = (n == 0u) ? 0u : n - scannedHist[(size_t)1 * numTiles];
    const uint32_t first = n - ones;
    for(uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < ones && i < maxPartitions;
        i += gridDim.x * blockDim.x)
    {
        const uint32_t p = splitPos[first + i];
        offsets[i] = p;
        binKeys[i] = sortedKeys[p];
    }
    if(blockIdx.x == 0 && threadIdx.x == 0)
    {
        *count = ones;
        if(ones <= maxPartitions) offsets[ones] = n;
    }
}

} // namespace

namespace {

// Coherence key of a ray: direction octant above a 27-bit Morton code of the
// origin quantised (9 bits per axis) in the scene box.
__global__ void k_ray_keys(const float4* __restrict__ rays, const uint32_t* __restrict__ idx, uint32_t n,
                           float3 lo, float3 scale, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals)
{
    for(uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const uint32_t r = idx ? idx[i] : i;
        const float4 o = __ldg(rays + 2 * (size_t)r), d = __ldg(rays + 2 * (size_t)r + 1);
        auto q = [](float v, float l, float s) {
            const float t = fminf(fmaxf((v - l) * s, 0.0f), 511.0f);
            uint32_t x = (uint32_t)t;
            x = (x | (x << 16)) & 0x030000FFu;
            x = (x | (x << 8)) & 0x0300F00Fu;
            x = (x | (x << 4)) & 0x030C30C3u;
            x = (x | (x << 2)) & 0x09249249u;
            return x;
        };
        const uint32_t m = q(o.x, lo.x, scale.x) | (q(o.y, lo.y, scale.y) << 1) | (q(o.z, lo.z, scale.z) << 2);
        const uint32_t oct = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
        keys[i] = (oct << 27) | m;
        vals[i] = r;
    }
}

} // namespace

cudaError_t ray_coherence_order(const void* rays, const uint32_t* idx, uint32_t n, const float box[6],
                                uint32_t* keysA, uint32_t* valsA, uint32_t* keysB, uint32_t* valsB,
                                uint32_t* hist, uint32_t*& order, int smCount, cudaStream_t st)
{
    float3 lo = make_float3(box[0], box[1], box[2]), sc;
    const float ext[3] = { box[3] - box[0], box[4] - box[1], box[5] - box[2] };
    sc.x = ext[0] > 0.0f ? 511.0f / ext[0] : 0.0f;
    sc.y = ext[1] > 0.0f ? 511.0f / ext[1] : 0.0f;
    sc.z = ext[2] > 0.0f ? 511.0f / ext[2] : 0.0f;
    k_ray_keys<<<std::max(1, smCount * 8), 256, 0, st>>>(static_cast<const float4*>(rays), idx, n, lo, sc, keysA, valsA);
    cudaError_t e = cudaGetLastError();
    uint32_t* kin = keysA; uint32_t* vin = valsA;
    uint32_t* kout = keysB; uint32_t* vout = valsB;
    for(uint32_t p = 0; p < 4 && e == cudaSuccess; p++)
    {
        DigitSpec s;
        s.batchShift = 0; s.batchWidth = 30;
        s.digitShift = 8u * p; s.digitBits = (p == 3) ? 6u : 8u;
        e = multisplit_pass(kin, vin, kout, vout, nullptr, n, s, hist, st);
        std::swap(kin, kout); std::swap(vin, vout);
    }
    order = vin;
    return e;
}

size_t multisplit_hist_words(uint32_t nMax, uint32_t digitBits)
{
    const uint32_t tiles = (nMax + kMsTile - 1) / kMsTile;
    // the count table, then the bucket totals
    return ((size_t)(tiles ? tiles : 1u) << digitBits) + 256u;
}

cudaError_t multisplit_pass(const uint32_t* keysIn, const uint32_t* idxIn, uint32_t* keysOut, uint32_t* idxOut,
                            const uint32_t* nDevice, uint32_t nMax, const DigitSpec& spec, uint32_t* hist,
                            cudaStream_t st, uint32_t* emptied, uint32_t* nOut)
{
    if(spec.dropEmpty && (!emptied || !nOut)) return cudaErrorInvalidValue;
    if(spec.digitBits == 0 || spec.digitBits > 8) return cudaErrorInvalidValue;
    uint32_t tiles = (nMax + kMsTile - 1) / kMsTile;
    if(tiles == 0) tiles = 1;
    const uint32_t nb = 1u << spec.digitBits;
    uint32_t* totals = hist + ((size_t)tiles << spec.digitBits);
    cudaError_t e = cudaMemsetAsync(totals, 0, sizeof(uint32_t) * nb, st);
    if(e != cudaSuccess) return e;
    k_ms_hist<<<tiles, kMsTPB, 0, st>>>(keysIn, nDevice, nMax, spec, hist, tiles, totals);
    k_ms_rows<<<nb, kScanTPB, 0, st>>>(hist, tiles, totals, nOut);
    k_ms_scatter<<<tiles, kMsTPB, 0, st>>>(keysIn, idxIn, keysOut, idxOut, nDevice, nMax, spec, hist, tiles, emptied);
    return cudaGetLastError();
}

cudaError_t multi_partition(const uint32_t* keys, const uint32_t* indices, const uint32_t* nDevice, uint32_t nMax,
                            uint32_t dataShift, uint32_t dataWidth, uint32_t batchShift, uint32_t batchWidth,
                            uint32_t* sortedKeys, uint32_t* sortedIdx, uint32_t* tmpKeys, uint32_t* tmpIdx,
                            uint32_t* hist, uint32_t* count, uint32_t* offsets, uint32_t* binKeys,
                            uint32_t maxPartitions, int smCount, cudaStream_t st)
{
    const uint32_t total = batchWidth + dataWidth;
    const uint32_t passes = (total + 7u) / 8u;
    // ping-pong so that the last pass lands in the outputs
    const uint32_t* kIn = keys;
    const uint32_t* iIn = indices;
    for(uint32_t p = 0; p < passes; p++)
    {
        const bool toOut = ((passes - 1u - p) & 1u) == 0u;
        uint32_t* kOut = toOut ? sortedKeys : tmpKeys;
        uint32_t* iOut = toOut ? sortedIdx : tmpIdx;
        DigitSpec s;
        s.batchShift = batchShift; s.batchWidth = batchWidth;
        s.dataShift = dataShift; s.dataWidth = dataWidth;
        s.digitShift = 8u * p;
        s.digitBits = std::min(8u, total - 8u * p);
        cudaError_t e = multisplit_pass(kIn, iIn, kOut, iOut, nDevice, nMax, s, hist, st);
        if(e != cudaSuccess) return e;
        kIn = kOut; iIn = iOut;
    }
    // splits of the batch portion, compacted in order with a one-bit pass
    k_find_splits<<<std::max(1, smCount * 4), 256, 0, st>>>(sortedKeys, nDevice, nMax, batchShift, batchWidth, tmpKeys);
    DigitSpec m;
    m.batchShift = 0; m.batchWidth = 1; m.dataShift = 0; m.dataWidth = 0;
    m.digitShift = 0; m.digitBits = 1;
    uint32_t* marksOut = hist + multisplit_hist_words(nMax, 8);      // past the widest count table
    cudaError_t e = multisplit_pass(tmpKeys, nullptr, marksOut, tmpIdx, nDevice, nMax, m, hist, st);
    if(e != cudaSuccess) return e;
    uint32_t tiles = (nMax + kMsTile - 1) / kMsTile;
    if(tiles == 0) tiles = 1;
    k_bins<<<std::max(1, smCount), 256, 0, st>>>(tmpIdx, sortedKeys, nDevice, nMax, hist, tiles, maxPartitions,
                                                 count, offsets, binKeys);
    return cudaGetLastError();
}

} // namespace mrg
