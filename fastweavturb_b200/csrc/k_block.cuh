// k_block.cuh -- tile-owned FP32 deposition by blocks of 64 grid points, two points per lane.
//
// A CTA owns a tile (or a part of one) and walks the tile's candidate records in chunks staged in
// shared memory by bulk asynchronous copies, two chunks in flight.  The tile is cut into blocks
// of 4 x 4 x 4 points; a task is one block against one chunk.  A warp that takes a task culls
// the chunk's records against the block, one record per lane, and then goes through the records
// that may hold accepted points: each lane tests its own two points (neighbours along z) and
// evaluates the vorticity, and adds it to its own points' sums.  No two warps hold the same
// block during a chunk, so the sums are plain registers (kept in shared memory between chunks)
// and need no atomics.
//
// Why this shape: the earlier form spread the grid rows of every record over the lanes, queued
// the accepted points and added each with three shared-memory int64 atomics.  It issued 13.6
// warp instructions per accepted pair over levels 0-3 of the 8-level family on 512^3 (solving
// the rows, testing, queueing and the atomics, which run at 1.8 lanes per clock and SM), where
// the vorticity itself is about 2.2.  Here a block that a record covers costs one pass of tests
// and evaluation, and a block that it misses one lane of a cull.  Two points per lane share the
// record's loads and the loop, and their vorticity is evaluated in packed FP32 (f32x2): the
// kernel is bound by instruction issue, and a packed operation takes one slot for two points.
//
// The tests, the evaluation and the int64 fixed-point sums are those of the record (the Policy):
// integer sums do not depend on the order, so the field is the same bit for bit whatever the
// split into blocks, parts and chunks.
#pragma once

#include <type_traits>

#include "k_tile_common.cuh"

namespace fwt {

constexpr int kBX = 4, kBY = 4, kBZ = 4;                       // block of 64 points
constexpr int kBlocksX = TX / kBX, kBlocksY = TY / kBY, kBlocksZ = TZ / kBZ;
constexpr int kTileBlocks = kBlocksX * kBlocksY * kBlocksZ;    // 16
constexpr float kBlockHalfDiag = 2.6f;                         // sqrt(3) * 1.5 = 2.598 grid spacings

__device__ __forceinline__ void block_origin(int blk, int &bx, int &by, int &bz)
{
    bx = (blk % kBlocksX) * kBX;
    by = ((blk / kBlocksX) % kBlocksY) * kBY;
    bz = (blk / (kBlocksX * kBlocksY)) * kBZ;
}

// What a record is to a block (Policy::may_hit), and the form of its visit.
enum BlockHit { kMiss = 0, kPlain = 1, kBoxed = 2, kWrapped = 3 };

template <class Policy>
struct BlockStage {
    typename Policy::Rec rec[2][Policy::kChunk];
    typename Policy::Prep prep;
    uint32_t id[2][Policy::kChunk];   // record id | image << 26
    uint64_t bar[2];
    int next[2];                      // next unclaimed block of the chunk in each buffer
    int failed;
};

template <class Policy>
constexpr size_t block_smem()
{
    return kAccBytes + sizeof(BlockStage<Policy>);
}

// Constant-core lines without a twist (sigma_ratio = 1, eta = 0): the vorticity has no
// curvature term, so no pair is deferred for its conditioning.  (Lines with a varying core take
// deposit_tile_kernel: their vorticity is five times the work, and is better evaluated with all
// lanes busy from a queue than by the third of a block's lanes that hold accepted points.)
// One CTA per tile part: D.w0 + blockIdx.x / parts is the tile; parts (1 or 2) cut it along z.
template <class Policy, bool Accumulate>
__global__ void __launch_bounds__(kDepThreads, Policy::kCtas) deposit_block_kernel(
    const typename Policy::Rec *__restrict__ rec, int N, int ntx, int nty, int tz0, int parts,
    const int64_t *__restrict__ tile_off, const uint32_t *__restrict__ list, double scale, float *__restrict__ wx,
    float *__restrict__ wy, float *__restrict__ wz, int *__restrict__ err, int zs, int zlim, float dx,
    unsigned long long *__restrict__ tally, const DeferList D)
{
    extern __shared__ __align__(16) unsigned char dsm[];
    long long(*acc)[kAccN] = reinterpret_cast<long long(*)[kAccN]>(dsm);
    BlockStage<Policy> &S = *reinterpret_cast<BlockStage<Policy> *>(dsm + kAccBytes);
    const int tile = (int)D.w0 + (int)blockIdx.x / parts, part = (int)blockIdx.x % parts;
    const int64_t c0 = tile_off[tile], c1 = tile_off[tile + 1];
    // a tile that no record of this batch meets keeps its values: earlier batches wrote them,
    // or the field was cleared before the first
    if (c0 == c1) return;
    const int tx = tile % ntx, ty = (tile / ntx) % nty, tz = tz0 + tile / (ntx * nty);
    const int x0 = tx * TX, y0 = ty * TY, z0 = tz * TZ;
    const int nblk = kTileBlocks / parts, blk0 = part * nblk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nrec = (int)(c1 - c0);
    const int nchunks = (nrec + Policy::kChunk - 1) / Policy::kChunk;

    // warp 0: the chunk's record ids, then one bulk copy per record.  The ids are plain stores, and what
    // the other warps wait for is the mbarrier: they are written before lane 0 arrives on it (a release,
    // which the wait's acquire meets; the copies' bytes alone would not publish them).  A barrier after the
    // sums' set-up does it too, but spills registers: 512^3, radius 122 to 15: 307 ms, 296 so.
    auto issue = [&](int ch) {
        const int b = ch & 1;
        const int64_t base = c0 + (int64_t)ch * Policy::kChunk;
        const int nc = min(Policy::kChunk, nrec - ch * Policy::kChunk);
        for (int t = lane; t < nc; t += 32) S.id[b][t] = __ldg(list + base + t);
        __syncwarp();
        if (lane == 0) mbar_expect(&S.bar[b], (uint32_t)(nc * sizeof(typename Policy::Rec)));
        __syncwarp();
        for (int t = lane; t < nc; t += 32)
            bulk_g2s(&S.rec[b][t], rec + (S.id[b][t] & ((1u << 26) - 1u)), (uint32_t)sizeof(typename Policy::Rec), &S.bar[b]);
    };
    if (tid == 0) {
        mbar_init(&S.bar[0]);
        mbar_init(&S.bar[1]);
        S.failed = 0;
    }
    __syncthreads();
    if (warp == 0) {
        issue(0);
        if (nchunks > 1) issue(1);
    }
    // every point of the tile is on the context's grid
    const bool full = (x0 + TX <= N) && (y0 + TY <= N) && (z0 + TZ <= zlim);
    // the part's points: its cells are loaded (Accumulate) or zeroed
    const int npts = nblk * 64;
    auto point_of = [&](int q, int &lx, int &ly, int &lz) {   // q-th point of the part, x fastest
        const int p = blk0 * 64 + q;   // whole xy planes: 8 blocks fill four of them
        lx = p % TX;
        ly = (p / TX) % TY;
        lz = p / (TX * TY);
    };
    for (int q = tid; q < npts; q += kDepThreads) {
        int lx, ly, lz;
        point_of(q, lx, ly, lz);
        const int gx = x0 + lx, gy = y0 + ly, gz = z0 + lz;
        long long a0 = 0, a1 = 0, a2 = 0;
        if (Accumulate && gx < N && gy < N && gz < zlim) {
            const size_t g = (size_t)gx + (size_t)N * ((size_t)gy + (size_t)N * (gz - zs));
            a0 = __double2ll_rn((double)wx[g] * scale);
            a1 = __double2ll_rn((double)wy[g] * scale);
            a2 = __double2ll_rn((double)wz[g] * scale);
        }
        const int pa = lx + kSY * ly + kSZ * lz;
        acc[0][pa] = a0;
        acc[1][pa] = a1;
        acc[2][pa] = a2;
    }

    // an emit-only pass lists the deferred pairs again and discards its sums
    const float fscale = D.emit_only ? 0.0f : (float)scale;
    unsigned nacc = 0;       // pairs evaluated by this lane
    f32x2 poison = pk(0.0f, 0.0f);   // turns NaN with any contribution that is not finite
    const int plx = lane & 3, ply = (lane >> 2) & 3, plz = 2 * (lane >> 4);
    const f32x2 zero2 = pk(0.0f, 0.0f);
    uint32_t phases = 0u;    // bit b: parity of buffer b's next wait
    for (int ch = 0; ch < nchunks; ++ch) {
        const int b = ch & 1;
        const int nc = min(Policy::kChunk, nrec - ch * Policy::kChunk);
        if (!mbar_wait(&S.bar[b], (phases >> b) & 1u)) S.failed = 1;
        phases ^= 1u << b;
        // kDepThreads / kChunk threads share a record's preparation
        if (tid % Policy::kChunk < nc)
            Policy::prepare(S.prep, tid % Policy::kChunk, tid / Policy::kChunk, S.rec[b][tid % Policy::kChunk],
                            S.id[b][tid % Policy::kChunk] >> 26, N, x0, y0, z0);
        if (tid == 0) S.next[b] = kDepWarps;
        __syncthreads();
        if (S.failed) {   // the other buffer's copies land before the CTA ends
            if (ch + 1 < nchunks) mbar_wait(&S.bar[b ^ 1], (phases >> (b ^ 1)) & 1u);
            break;
        }
        for (int blk = warp; blk < nblk;) {
            int bx, by, bz;
            block_origin(blk0 + blk, bx, by, bz);
            const float fbx = (float)bx, fby = (float)by, fbz = (float)bz;
            const int lx = bx + plx, ly = by + ply, lz = bz + plz;
            const bool in_xy = x0 + lx < N && y0 + ly < N;
            const bool in0 = in_xy && z0 + lz < zlim, in1 = in_xy && z0 + lz + 1 < zlim;
            const float flx = (float)lx, fly = (float)ly, flz = (float)lz;
            const int pa = lx + kSY * ly + kSZ * lz;
            long long a00 = acc[0][pa], a01 = acc[1][pa], a02 = acc[2][pa];
            long long a10 = acc[0][pa + kSZ], a11 = acc[1][pa + kSZ], a12 = acc[2][pa + kSZ];
            // one record against the block's points: test, evaluate, add (every lane computes;
            // points that are not accepted add zero)
            auto one = [&](int k, auto form) {
                Policy::template visit<decltype(form)::value>(
                    S.prep, S.rec[b][k], k, dx, flx, fly, flz, in0, in1,
                    [&](bool ok0, bool ok1, bool dec0, bool dec1, const f32x2 *v) {
                        // dec: left to the reference's FP64 tests
                        nacc += ok0;
                        nacc += ok1;
                        const f32x2 fs = pk(ok0 ? fscale : 0.0f, ok1 ? fscale : 0.0f);
                        const f32x2 s0 = mul2(v[0], fs), s1 = mul2(v[1], fs), s2 = mul2(v[2], fs);
                        float s00, s01, s02, s10, s11, s12;
                        unpk(s0, s00, s10);
                        unpk(s1, s01, s11);
                        unpk(s2, s02, s12);
                        // |tp T| <= amp, and amp times the scale is at most 2^44 by the choice of the
                        // scale: only a value that is not a number can leave the fixed-point range, and
                        // then all three components are none (they share tp / |c'|)
                        poison = fma2(s0, zero2, poison);
                        a00 += __float2ll_rn(s00);
                        a01 += __float2ll_rn(s01);
                        a02 += __float2ll_rn(s02);
                        a10 += __float2ll_rn(s10);
                        a11 += __float2ll_rn(s11);
                        a12 += __float2ll_rn(s12);
                        if (__any_sync(0xffffffffu, dec0 || dec1)) {
                            const uint32_t id = (S.id[b][k] & ((1u << 26) - 1u)) | kDeferDecide;
                            defer_push(D, lane, dec0, id, x0 + lx, y0 + ly, z0 + lz);
                            defer_push(D, lane, dec1, id, x0 + lx, y0 + ly, z0 + lz + 1);
                        }
                    });
            };
            for (int k0 = 0; k0 < nc; k0 += 32) {
                const int kc = k0 + lane;
                int hit = kc < nc ? Policy::may_hit(S.prep, kc, dx, fbx, fby, fbz) : kMiss;
                if (hit == kPlain && !full) hit = kBoxed;
                const unsigned plain = __ballot_sync(0xffffffffu, hit == kPlain);
                const unsigned boxed = __ballot_sync(0xffffffffu, hit == kBoxed);
                const unsigned wrapped = __ballot_sync(0xffffffffu, hit == kWrapped);
                for (unsigned m = plain; m; m &= m - 1)
                    one(k0 + __ffs(m) - 1, std::integral_constant<int, kPlain>{});
                for (unsigned m = boxed; m; m &= m - 1)
                    one(k0 + __ffs(m) - 1, std::integral_constant<int, kBoxed>{});
                for (unsigned m = wrapped; m; m &= m - 1)
                    one(k0 + __ffs(m) - 1, std::integral_constant<int, kWrapped>{});
            }
            acc[0][pa] = a00;
            acc[1][pa] = a01;
            acc[2][pa] = a02;
            acc[0][pa + kSZ] = a10;
            acc[1][pa + kSZ] = a11;
            acc[2][pa + kSZ] = a12;
            int nxt = 0;
            if (lane == 0) nxt = atomicAdd(&S.next[b], 1);
            blk = __shfl_sync(0xffffffffu, nxt, 0);
        }
        __syncthreads();   // the buffer's records and the prepared culls are free again
        if (warp == 0 && ch + 2 < nchunks) issue(ch + 2);
    }
    float p0, p1;
    unpk(poison, p0, p1);
    if ((!(p0 == p0) || !(p1 == p1)) && !D.emit_only) atomicOr(err, 4);
    // a lane's pairs: at most 2 points x 16 blocks x 2^26 records; the warp's do not fit 32 bits
    const unsigned long long wacc = warp_sum((unsigned long long)nacc);
    if (lane == 0 && tally && !D.emit_only && wacc) atomicAdd(tally, wacc);
    __syncthreads();
    if (S.failed && tid == 0) atomicOr(err, 2);
    if (D.emit_only) return;
    // fixed point -> float, 16-byte stores where the rows of omega start on 16 bytes
    const double inv = 1.0 / scale;
    if (full && (N & 3) == 0) {
        for (int q4 = tid; q4 < npts / 4; q4 += kDepThreads) {
            int lx, ly, lz;
            point_of(4 * q4, lx, ly, lz);
            const size_t g = (size_t)(x0 + lx) + (size_t)N * ((size_t)(y0 + ly) + (size_t)N * (z0 + lz - zs));
            const int pa = lx + kSY * ly + kSZ * lz;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float4 v4;
                v4.x = (float)((double)acc[d][pa] * inv);
                v4.y = (float)((double)acc[d][pa + 1] * inv);
                v4.z = (float)((double)acc[d][pa + 2] * inv);
                v4.w = (float)((double)acc[d][pa + 3] * inv);
                float *w = d == 0 ? wx : (d == 1 ? wy : wz);
                *reinterpret_cast<float4 *>(w + g) = v4;
            }
        }
    } else {
        for (int q = tid; q < npts; q += kDepThreads) {
            int lx, ly, lz;
            point_of(q, lx, ly, lz);
            const int gx = x0 + lx, gy = y0 + ly, gz = z0 + lz;
            if (gx >= N || gy >= N || gz >= zlim) continue;
            const size_t g = (size_t)gx + (size_t)N * ((size_t)gy + (size_t)N * (gz - zs));
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                float *w = d == 0 ? wx : (d == 1 ? wy : wz);
                w[g] = (float)((double)acc[d][lx + kSY * ly + kSZ * lz] * inv);
            }
        }
    }
}

// Parts per tile: one where the tiles alone fill the GPU several times over, two on small grids
// (64^3 has 256 tiles for 148 SMs x 3 CTAs).
inline int block_parts(int64_t ntiles, int sms, int ctas) { return ntiles < (int64_t)4 * sms * ctas ? 2 : 1; }

}  // namespace fwt
