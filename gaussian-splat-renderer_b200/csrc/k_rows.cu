// The binning list built row by row (the reference's binning order: depth, then gaussian, inside every
// tile), in the place of the scan, the emission of one entry a tile, the tile sort and the ranges.
//
// The depth sort has put each view's records in (depth, index) order. From there two stable partitions
// build the list, both from the runs [x0, x1) that a splat covers in a tile row, so that the entries
// moved are half as many (a run is about two tiles wide) and the per-tile entry is written once:
//
//   rowPlan       one block: the rows' sizes, counted by the preprocess, into the places of their
//                 buckets and of their tiles' part of the list. When the list overflows its capacity,
//                 all blocks find the record it ends in (a scan of the counts in depth order) and
//                 count the rows of the kept records instead; they and the partition end at that record (four
//                 720p views of 1.24 M, a capacity of 219,136: 286 -> 79 us; of 3.5 M: 333 -> 153)
//   rowPartition  1,024 records a block in depth order: a row entry (x0, x1, gaussian) for every run
//                 into its row's bucket, stable, with the onesweep sort's digit look-back (the digit is
//                 the row)
//   rowTiles      eight blocks (a cluster) a bucket: the tiles' counts from the runs' ends, exchanged
//                 through distributed shared memory, give the row's ranges; then every run writes its
//                 gaussian to its tiles' places, again stable
//
// Bound by the records' scattered reads (a hint a record, 13 M L2 sectors a 1080p view in the partition,
// 5 TB/s) and, in the tiles, by the scattered 4-byte stores. From the depth sort to the ranges,
// against the scan, emission, tile sort and ranges it replaces (us): 10,000 gaussians at 641 x 359
// 57 -> 28, 100,000 at 720p 78 -> 38, 1.24 M at 1080p 177 -> 126, eight such views 1,025 -> 714, 24
// uneven views of 559,000 1,560 -> 900, 6 M at 4K 630 -> 503; the rasterizer reads 4 bytes an entry
// instead of 8.
// Built with -fmad=false: the runs of large splats are computed again (splat_math.cuh).
#include <cooperative_groups.h>

#include "kernels.cuh"
#include "splat_math.cuh"

namespace gsr {

namespace {

namespace cg = cooperative_groups;

constexpr uint32_t kRowThreads = 256, kRowWarps = kRowThreads / 32;
constexpr uint32_t kRowSteps = kRowTile / kRowThreads;  // a warp's steps of 32 records
constexpr uint32_t kRowCluster = 8;
constexpr uint32_t kPartThreads = 256, kPartWarps = kPartThreads / 32;  // rowPartition: a block
constexpr uint32_t kTileThreads = 512, kTileWarps = kTileThreads / 32;  // rowTiles: a block
static_assert(kRowBins == kRowThreads, "a thread owns a row");

__device__ __forceinline__ uint32_t lanesBelow() {
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Where a record's runs are, beside an index of the spilled ones: its hint, one run for every row, or
// nowhere (computed again from the ellipse).
constexpr uint32_t kRunsInHint = 0xFFFFFFFFu, kRunsSame = 0xFFFFFFFEu, kRunsEllipse = 0xFFFFFFFDu;

// The coverage of a record whose hint holds no runs, as the preprocess had it.
__device__ __forceinline__ Coverage recordCoverage(const FrontArgs& a, const DevView& vw, size_t rec, RowGeom& g) {
    float cx, cy, cA, cB, cC;
    TileRect rect;
    if (a.renderSplat == kRenderSplatFull) {
        const DevSplat s = reinterpret_cast<const DevSplat*>(a.splats)[rec];
        cx = s.cx;
        cy = s.cy;
        cA = s.conicA;
        cB = s.conicB;
        cC = s.conicC;
        rect = tileRect(s.cx, s.cy, s.radius, (vw.width + 15) / 16, (vw.height + 15) / 16);
    } else {
        rect = unpackRect(a.rects[rec]);
        if (a.renderSplat == kRenderSplatP32) {
            const uint4 w = reinterpret_cast<const uint4*>(a.packed)[rec * 2];
            cx = __uint_as_float(w.x);
            cy = __uint_as_float(w.y);
            cA = __uint_as_float(w.z);
            cB = __uint_as_float(w.w);
            cC = __uint_as_float(reinterpret_cast<const uint32_t*>(a.packed)[rec * 8 + 4]);
        } else {
            const uint2 w0 = reinterpret_cast<const uint2*>(a.packed)[rec * 3];
            const uint2 w1 = reinterpret_cast<const uint2*>(a.packed)[rec * 3 + 1];
            cx = __uint_as_float(w0.x);
            cy = __uint_as_float(w0.y);
            float o;
            p24DecodeConic(w1.x, w1.y, cA, cB, cC, o);
        }
    }
    const float4 hint = a.bounds != kBoundsRect ? a.hints[rec] : make_float4(-2.0f, 0.0f, 0.0f, 0.0f);
    return coverageFromHint(a.bounds, rect, binShapeOf(a.binSize), int(vw.tilesX), int(vw.tilesY), cx, cy, cA, cB, cC,
                            hint, g);
}
__device__ __noinline__ uint32_t ellipseRun(const FrontArgs& a, const DevView& vw, size_t rec, uint32_t row) {
    RowGeom g;
    const Coverage cv = recordCoverage(a, vw, rec, g);
    int x0, x1;
    coverageRowSpan(cv, g, int(row), binShapeOf(a.binSize), x0, x1);
    return packRun(x0, x1);
}
__device__ __noinline__ uint4 ellipseRows(const FrontArgs& a, const DevView& vw, size_t rec) {  // r0, rows, first run, rest
    RowGeom g;
    const Coverage cv = recordCoverage(a, vw, rec, g);
    int r0, r1;
    coverageRows(cv, binShapeOf(a.binSize), r0, r1);
    return make_uint4(uint32_t(r0), uint32_t(r1 - r0),
                      packRun(cv.bins.x0, cv.bins.x1),
                      cv.useEllipse ? kRunsEllipse : kRunsSame);
}

// The rows of a record: r0, their number, and where their runs are: an index of the spilled runs, the
// hint, one run for every row (`same`), or the ellipse.
struct RecordRows {
    uint32_t r0, rows, at;
    uint32_t run[kSpanRows];  // a hint's runs; run[0] also the run of every row (kRunsSame)
};
// Of a thread's COUNT records (their loads in flight together: the hints, then the runs beside them).
template <uint32_t COUNT>
__device__ __forceinline__ void recordRows(const FrontArgs& a, const DevView& vw, const size_t (&rec)[COUNT],
                                           const uint32_t (&kept)[COUNT], RecordRows (&R)[COUNT]) {
    uint4 hint[COUNT];
#pragma unroll
    for (uint32_t j = 0; j < COUNT; ++j) {
        hint[j] = make_uint4(0u, 0u, 0u, 0u);
        if (kept[j] && a.bounds != kBoundsRect) hint[j] = *reinterpret_cast<const uint4*>(&a.hints[rec[j]]);
    }
#pragma unroll
    for (uint32_t j = 0; j < COUNT; ++j) {
        const bool spilled = (hint[j].x & kSpanSpilled) != 0, runs = (hint[j].x & 0xFFC00000u) == kSpanMarker;
        R[j].r0 = hint[j].x & 0xFFFFu;
        R[j].rows = !runs ? 0u : spilled ? hint[j].y : (hint[j].x >> 16) & 0x7u;
        R[j].at = runs && spilled ? hint[j].z : kRunsInHint;
        R[j].run[0] = hint[j].y;
        R[j].run[1] = hint[j].z;
        R[j].run[2] = hint[j].w;
        if (runs && !spilled && R[j].rows > 3) {
            const uint4 more = a.spanRows[rec[j]];
            R[j].run[3] = more.x;
            R[j].run[4] = more.y;
            R[j].run[5] = more.z;
            R[j].run[6] = more.w;
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < COUNT; ++j)
        if (kept[j] && (hint[j].x & 0xFFC00000u) != kSpanMarker) {
            const uint4 e = ellipseRows(a, vw, rec[j]);
            R[j].r0 = e.x;
            R[j].rows = e.y;
            R[j].run[0] = e.z;
            R[j].at = e.w;
        }
}
// Run r of the record (x0 | x1 << 16); `kept` tiles of it, cut at them if it is the list's last record.
__device__ __noinline__ uint32_t runOf(const FrontArgs& a, const DevView& vw, size_t rec, uint32_t r0, uint32_t r, uint32_t at,
                                       uint32_t same) {
    if (at == kRunsInHint)
        return r < 3 ? reinterpret_cast<const uint32_t*>(a.hints + rec)[1 + r]
                     : reinterpret_cast<const uint32_t*>(a.spanRows + rec)[r - 3];
    if (at == kRunsSame) return same;
    if (at == kRunsEllipse) return ellipseRun(a, vw, rec, r0 + r);
    return a.spill[at + r];
}
__device__ __noinline__ uint32_t cutRun(const FrontArgs& a, const DevView& vw, size_t rec, uint32_t r0, uint32_t r, uint32_t at,
                                        uint32_t same, uint32_t kept) {
    for (uint32_t q = 0;; ++q) {
        const uint32_t run = runOf(a, vw, rec, r0, q, at, same), wide = (run >> 16) - (run & 0xFFFFu);
        const uint32_t w = wide < kept ? wide : kept;
        if (q == r) return (run & 0xFFFFu) | (((run & 0xFFFFu) + w) << 16);
        kept -= w;
    }
}

// A warp's work, shared out evenly: lane l brings n items; pairs (lane, item) are numbered lane by lane
// and taken 32 at a time, one a lane. (A lane walking its own items leaves most lanes waiting for the
// longest: the partition executed five times the instructions.)
struct WarpPairs {
    uint32_t n, begin, total, place;  // place: the lane's position among those with items
    uint32_t before;                  // lanes whose items begin before the current 32
    __device__ __forceinline__ WarpPairs(uint32_t items) : n(items), before(0) {
        const uint32_t lane = threadIdx.x & 31;
        uint32_t end = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, end, o);
            if (lane >= uint32_t(o)) end += t;
        }
        begin = end - n;
        total = __shfl_sync(0xFFFFFFFFu, end, 31);
        place = __popc(__ballot_sync(0xFFFFFFFFu, n != 0) & lanesBelow());
    }
    // the position (among the lanes with items) of the lane that brought pair p0 + lane
    __device__ __forceinline__ uint32_t owner(uint32_t p0) {
        const uint32_t heads = __reduce_or_sync(0xFFFFFFFFu, n && begin - p0 < 32u ? 1u << (begin - p0) : 0u);
        const uint32_t q = before + __popc(heads & (lanesBelow() | (1u << (threadIdx.x & 31)))) - 1u;
        before += __popc(heads);
        return q;
    }
};

// fn(valid, row, run x0 | x1 << 16, gaussian) for the runs of the warp's 32 records in (record, row)
// order, 32 at a time, all lanes together (valid: not empty, and inside the view whatever the word holds);
// terms = kTermWords x 32 words of the warp's shared memory.
constexpr uint32_t kTermWords = 4 + kSpanRows;
template <typename Fn>
__device__ __forceinline__ void forWarpRuns(const FrontArgs& a, const DevView& vw, uint32_t view, size_t rec, const RecordRows& R,
                                            uint32_t kept, bool cut, uint32_t (*terms)[32], Fn fn) {
    const uint32_t lane = threadIdx.x & 31;
    WarpPairs w(R.rows);
    __syncwarp();
    if (R.rows) {
        terms[0][w.place] = R.r0 - w.begin;  // row = pair + this
        terms[1][w.place] = R.at;
        terms[2][w.place] = uint32_t(rec - size_t(view) * a.count);
        terms[3][w.place] = w.begin;
#pragma unroll
        for (uint32_t r = 0; r < uint32_t(kSpanRows); ++r)
            if (r == 0 || (R.at == kRunsInHint && r < R.rows)) terms[4 + r][w.place] = R.run[r];
    }
    const uint32_t cutAt = __shfl_sync(0xFFFFFFFFu, w.place, __ffs(__ballot_sync(0xFFFFFFFFu, cut) | 0x80000000u) - 1);
    const uint32_t cutKept = __reduce_max_sync(0xFFFFFFFFu, cut ? kept : 0u);  // 0: the record is not here
    __syncwarp();
    for (uint32_t p0 = 0; p0 < w.total; p0 += 32) {
        const uint32_t q = w.owner(p0), p = p0 + lane;
        uint32_t row = 0, run = 0, gaussian = 0;
        if (p < w.total) {
            row = p + terms[0][q];
            gaussian = terms[2][q];
            const uint32_t at = terms[1][q], r = p - terms[3][q];
            const size_t owner = size_t(view) * a.count + gaussian;
            if (cutKept && q == cutAt) run = cutRun(a, vw, owner, row - r, r, at, terms[4][q], cutKept);
            else if (at == kRunsInHint) run = terms[4 + r][q];
            else if (at == kRunsSame) run = terms[4][q];
            else if (at == kRunsEllipse) run = ellipseRun(a, vw, owner, row);
            else run = a.spill[at + r];
        }
        fn((run >> 16) > (run & 0xFFFFu) && (run >> 16) <= vw.tilesX && row < vw.tilesY, row, run, gaussian);
    }
}

// The sorted records of a thread's slots of a view, and whether they have tiles (not past the view's end,
// for records without tiles, whose depth bits are all ones, nor for a word that names no record of the
// view: a frame whose look-back gave up).
template <uint32_t COUNT>
__device__ __forceinline__ void slotRecords(const FrontArgs& a, const uint64_t* sorted, uint32_t view, uint32_t slot,
                                            uint32_t stride, size_t (&rec)[COUNT], bool (&tiles)[COUNT]) {
    const size_t first = size_t(view) * a.count, end = first + a.count;
    uint64_t word[COUNT];
#pragma unroll
    for (uint32_t j = 0; j < COUNT; ++j) word[j] = slot + j * stride < end ? sorted[slot + j * stride] : ~0ull;
#pragma unroll
    for (uint32_t j = 0; j < COUNT; ++j) {
        rec[j] = word[j] & ((1ull << a.recordBits) - 1ull);
        tiles[j] = uint32_t(word[j] >> a.recordBits) != 0xFFFFFFFFu && rec[j] >= first && rec[j] < end;
        if (!tiles[j]) rec[j] = first;
    }
}

// Block-wide exclusive scan of a 64-bit value a thread; *total = the sum.
template <uint32_t WARPS = kRowWarps>
__device__ __forceinline__ uint64_t blockScan64(uint64_t v, uint64_t* sWarp, uint64_t* total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t o = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= uint32_t(d)) incl += o;
    }
    if (lane == 31) sWarp[warp] = incl;
    __syncthreads();
    uint64_t base = 0, sum = 0;
#pragma unroll
    for (uint32_t w = 0; w < WARPS; ++w) {
        const uint64_t t = sWarp[w];
        if (w < warp) base += t;
        sum += t;
    }
    __syncthreads();
    *total = sum;
    return base + incl - v;
}

// The buckets' places from the rows' sizes, by one block (row entries in the high word, tiles in the
// low): a thread's share is viewCount consecutive buckets.
__device__ void planRows(const FrontArgs& a, const unsigned long long* hist, uint64_t* sWarp) {
    const size_t first = size_t(threadIdx.x) * a.viewCount;
    uint64_t sum = 0, total;
#pragma unroll 8
    for (uint32_t j = 0; j < a.viewCount; ++j) sum += __ldcg(&hist[first + j]);
    uint64_t at = blockScan64(sum, sWarp, &total);
#pragma unroll 8
    for (uint32_t j = 0; j < a.viewCount; ++j) {
        const uint64_t h = __ldcg(&hist[first + j]);
        a.rowPlan[first + j] = make_uint4(uint32_t(at >> 32), uint32_t(h >> 32), uint32_t(at), uint32_t(h));
        at += h;
    }
    if (threadIdx.x == 0) a.ctl->c.ext_pad[0] = uint32_t(total >> 32);  // the row entries
}

// A full list's largest tile id is that of all records, kept or not: the end of the longest run in the last
// row with tiles, found by all blocks together from the view's hints as they lie (16 bytes a record; 1.24 M: 17
// us).
__device__ void reportLastTile(const FrontArgs& a, uint32_t view, uint32_t row) {
    const DevView vw = a.views[view];
    uint32_t end = 0;
    for (uint32_t i0 = blockIdx.x * kRowTile + threadIdx.x; i0 < a.count; i0 += gridDim.x * kRowTile) {
        size_t rec[kRowSteps];
        uint32_t kept[kRowSteps];
        RecordRows R[kRowSteps];
#pragma unroll
        for (uint32_t j = 0; j < kRowSteps; ++j) {
            const uint32_t i = i0 + j * kRowThreads;
            rec[j] = size_t(view) * a.count + (i < a.count ? i : 0u);
            kept[j] = i < a.count ? a.tileCounts[rec[j]] : 0u;
        }
        recordRows(a, vw, rec, kept, R);
#pragma unroll
        for (uint32_t j = 0; j < kRowSteps; ++j) {
            const uint32_t r = row - R[j].r0;
            if (kept[j] && r < R[j].rows) {
                const uint32_t run = runOf(a, vw, rec[j], R[j].r0, r, R[j].at, R[j].run[0]);
                if ((run >> 16) > (run & 0xFFFFu) && (run >> 16) <= vw.tilesX) end = end > (run >> 16) ? end : run >> 16;
            }
        }
    }
    end = __reduce_max_sync(0xFFFFFFFFu, end);
    if ((threadIdx.x & 31) == 0 && end && row < vw.tilesY) {
        const uint32_t tile = vw.tileBase + row * vw.tilesX + end - 1;
        atomicMax(&a.ctl->c.tile_max, tile);
        atomicMax(&a.ctl->c.key_bits, bitWidth32(tile));
    }
}

__global__ void __launch_bounds__(kRowThreads) rowPlanKernel(const __grid_constant__ FrontArgs a) {
    __shared__ uint64_t sWarp[kRowWarps];
    __shared__ uint32_t sTicket, sPast, sExclusive, sRows[kRowBins], sLast;
    __shared__ uint32_t sTerms[kRowWarps][kTermWords][32];
    gridWait();
    DeviceControl* ctl = a.ctl;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // every block adds up the frame's tiles from the rows' low words, unless one of them may have gone past
    // 2^32 and carried into its entries (which are not read then: a full list is planned from its kept records)
    uint64_t sum = 0, all;
    uint32_t lastRow = 0;  // the last bucket with tiles
#pragma unroll 8
    for (uint32_t j = tid; j < a.viewCount * kRowBins; j += kRowThreads) {
        const uint64_t h = __ldcg(&a.rowHist[j]);
        sum += h & 0xFFFFFFFFull;
        if (h) lastRow = j;
    }
    blockScan64(sum, sWarp, &all);
    if (a.rowTilesWide) all = *rowTilesOf(ctl);
    const uint32_t tiles = uint32_t(all < 0xFFFFFFFFull ? all : 0xFFFFFFFFull);
    const bool full = tiles > a.capacity;
    if (blockIdx.x == 0 && tid == 0) {
        GsrControl& c = ctl->c;
        const uint32_t entries = full ? a.capacity : tiles;
        c.duplicates = tiles;
        c.entries = entries;
        c.overflow = tiles - entries;
        c.ranges_groups[0] = (entries + 255u) / 256u;
        c.visible = c.cull_counts[0];
        c.packed_entries = 1;
        c.index_bits = a.count > 1 ? bitWidth32(a.count - 1) : 1u;
        c.sort_passes = a.totalTiles > 1 ? 1 : 0;  // (tile_max and key_bits: rowTiles)
        c.depth_low_bits = 0;
        c.sorted_buffer = 0;
    }
    if (!full) {
        if (blockIdx.x == 0) planRows(a, a.rowHist, sWarp);
        return;
    }
    if (tid == 0) sLast = 0;
    __syncthreads();
    atomicMax(&sLast, lastRow);
    __syncthreads();
    reportLastTile(a, sLast / kRowBins, sLast % kRowBins);
    // the list ends inside the record at which the counts' prefix in depth order reaches the capacity
    const uint64_t* sorted = a.depthKeys[a.depthPlan->sortedBuffer & 1u];
    const uint32_t epoch = ctl->c.epoch, perView = (a.count + kRowTile - 1) / kRowTile;
    for (;;) {
        if (tid == 0) {
            sTicket = atomicAdd(&ctl->tickets[kRowCutTicket], 1u);
            sPast = __ldcg(&ctl->rowCutSlot) != 0xFFFFFFFFu;
        }
        sRows[tid] = 0;
        __syncthreads();
        const uint32_t t = sTicket;
        if (t >= perView * a.viewCount) break;
        if (sPast) {  // the cut lies before this tile (it is found after every tile up to it has published)
            if (tid == 0) stRelaxed(&a.scanStatus[t], packStatus(epoch, kFlagInclusive, 0xFFFFFFFFu));
            __syncthreads();
            continue;
        }
        const uint32_t view = t / perView, base = view * a.count + (t - view * perView) * kRowTile + tid * kRowSteps;
        const DevView vw = a.views[view];
        size_t rec[kRowSteps];
        uint32_t n[kRowSteps], mine = 0;
        bool some[kRowSteps];
        slotRecords(a, sorted, view, base, 1u, rec, some);
#pragma unroll
        for (uint32_t j = 0; j < kRowSteps; ++j) {
            n[j] = some[j] ? a.tileCounts[rec[j]] : 0u;
            mine += n[j];
        }
        // (a prefix past 2^32 - 1 stays there: it is past every capacity)
        uint64_t total, at = blockScan64(mine, sWarp, &total);
        if (warp == 0) {
            if (lane == 0) stRelaxed(&a.scanStatus[t], packStatus(epoch, t == 0 ? kFlagInclusive : kFlagAggregate, uint32_t(total)));
            const uint32_t before = t ? warpLookback<true>(a.scanStatus, int(t), epoch, ctl, kWaitScan) : 0u;
            const uint64_t through = before + total;
            if (lane == 0) {
                if (t) stRelaxed(&a.scanStatus[t], packStatus(epoch, kFlagInclusive, through < 0xFFFFFFFFull ? uint32_t(through) : 0xFFFFFFFFu));
                sExclusive = before;
            }
        }
        __syncthreads();
        at += sExclusive;
        uint32_t kept[kRowSteps];
        RecordRows R[kRowSteps];
#pragma unroll
        for (uint32_t j = 0; j < kRowSteps; ++j) {
            const uint32_t room = at < a.capacity ? a.capacity - uint32_t(at) : 0u;
            kept[j] = n[j] < room ? n[j] : room;
            if (room && n[j] >= room) {  // one record of the frame
                ctl->rowCutSlot = base + j;
                ctl->rowCutTiles = kept[j];
            }
            at += n[j];
        }
        recordRows(a, vw, rec, kept, R);
#pragma unroll
        for (uint32_t j = 0; j < kRowSteps; ++j)
            forWarpRuns(a, vw, view, rec[j], R[j], kept[j], kept[j] != 0 && kept[j] != n[j], sTerms[warp],
                        [&](bool valid, uint32_t row, uint32_t run, uint32_t) {
                            if (valid) atomicAdd(&sRows[row], (1u << 20) | ((run >> 16) - (run & 0xFFFFu)));
                        });
        __syncthreads();
        if (sRows[tid])
            atomicAdd(&a.rowKept[size_t(view) * kRowBins + tid],
                      (static_cast<unsigned long long>(sRows[tid] >> 20) << 32) | (sRows[tid] & 0xFFFFFu));
        __syncthreads();
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) sLast = atomicAdd(&ctl->histDone[0], 1u) == gridDim.x - 1;
    __syncthreads();
    if (!sLast) return;
    __threadfence();
    planRows(a, a.rowKept, sWarp);
}

// Look-back words of the partition: a row's count of one tile, or of all of the view's tiles up to it.
// 32 bits, so that one load takes four rows'; zero (the frame's start) is not published yet.
constexpr uint32_t kRowAggregate = 1u << 30, kRowInclusive = 2u << 30, kRowValue = kRowAggregate - 1u;
__device__ __forceinline__ uint4 ldRelaxed4(const uint32_t* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ void stRelaxed32(uint32_t* p, uint32_t v) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Decoupled look-back of the rows of partition tile t (of a view whose tiles begin at t0 < t) by the whole
// block: thread (four rows, slice) sums eight earlier tiles of its slice's window, the slices' windows
// one after another, until a window holds the rows' inclusive counts. (All blocks start together, so the
// first ones read hundreds of tiles: with a thread a row and two windows of 16, plan and partition of
// eight 1080p views took 521 us instead of 508.) Returns the exclusive prefix of row threadIdx.x < bins. Waits are bounded as digitLookback's.
__device__ __forceinline__ uint32_t rowLookback(const uint32_t* status, uint32_t t, uint32_t t0, uint32_t bins,
                                                DeviceControl* ctl, uint4* sSum, uint32_t* sFound) {
    constexpr int kWindow = 8;
    const uint32_t quads = bins / 4, slices = kPartThreads / quads, quad = threadIdx.x % quads, slice = threadIdx.x / quads;
    const uint32_t forced = ctl->forceTimeout;
    uint32_t exclusive = 0;
    bool open = threadIdx.x < bins;
    for (int q = int(t) - 1;; q -= kWindow * int(slices)) {
        if (slice < slices) {
            const int base = q - kWindow * int(slice);
            uint4 w[kWindow];
#pragma unroll
            for (int j = 0; j < kWindow; ++j)
                w[j] = base - j >= int(t0) ? ldRelaxed4(&status[size_t(base - j) * kRowBins + quad * 4])
                                           : make_uint4(kRowInclusive, kRowInclusive, kRowInclusive, kRowInclusive);
            uint4 sum = make_uint4(0u, 0u, 0u, 0u);
            uint32_t found = 0, spins = 0;
            auto take = [&](uint32_t word, uint32_t bit, uint32_t& s) {
                if (found & bit) return;
                s += word & kRowValue;
                if (word & kRowInclusive) found |= bit;
            };
#pragma unroll
            for (int j = 0; j < kWindow; ++j) {
                while (found != 15u && (!w[j].x || !w[j].y || !w[j].z || !w[j].w || (forced && spins < forced))) {
                    if (++spins >= kSpinLimit || (forced && spins >= forced)) {
                        reportTimeout(ctl, kWaitSort);
                        found = 15u;
                        break;
                    }
                    __nanosleep(32);
                    w[j] = ldRelaxed4(&status[size_t(base - j >= 0 ? base - j : 0) * kRowBins + quad * 4]);
                }
                take(w[j].x, 1u, sum.x);
                take(w[j].y, 2u, sum.y);
                take(w[j].z, 4u, sum.z);
                take(w[j].w, 8u, sum.w);
            }
            sSum[slice * quads + quad] = sum;
            sFound[slice * quads + quad] = found;
        }
        __syncthreads();
        if (open) {
            const uint32_t at = threadIdx.x / 4, c = threadIdx.x % 4;
            for (uint32_t s = 0; s < slices && open; ++s) {
                exclusive += reinterpret_cast<const uint32_t*>(&sSum[s * quads + at])[c];
                open = !((sFound[s * quads + at] >> c) & 1u);
            }
        }
        if (!__syncthreads_or(open)) return exclusive;
    }
}

// STEPS x 256 records a block, a warp's in STEPS steps of 32. The warp's runs are listed in order in
// shared memory (the first kWarpRuns of them; a warp with more looks the others up again), counted by
// row, and after the look-back written 32 at a time: ranks among them come from lane masks in shared
// memory, one word a row (as the sort's multisplit). (Put into row order in shared memory first and
// written out in runs: no faster, 83 us, and 434 instead of 381 at 6 M records, where its space costs
// a block a SM.) bins = the rows, a multiple of 32.
template <uint32_t STEPS>
struct RowPartSmem {
    static constexpr uint32_t kWarpRuns = 80 * STEPS;
    uint2 runs[kPartWarps][kWarpRuns];  // x0 | x1 << 10 | row << 20, gaussian
    uint32_t terms[kPartWarps][kTermWords][32];
    uint4 sum[kPartThreads];
    uint32_t found[kPartThreads];
};
static_assert(kRowMaxTilesX < 1024 && kRowBins <= 4096, "a packed run");
template <uint32_t STEPS>
size_t rowPartBytes(uint32_t bins) { return sizeof(RowPartSmem<STEPS>) + kPartWarps * bins * 2 * 4; }

template <uint32_t STEPS>
__global__ void __launch_bounds__(kPartThreads, 4) rowPartitionKernel(const __grid_constant__ FrontArgs a, uint32_t bins) {
    extern __shared__ __align__(16) unsigned char sRowPart[];
    RowPartSmem<STEPS>& S = *reinterpret_cast<RowPartSmem<STEPS>*>(sRowPart);
    uint32_t* sCount = reinterpret_cast<uint32_t*>(sRowPart + sizeof(RowPartSmem<STEPS>));  // [warp][row]
    uint32_t* sMask = sCount + kPartWarps * bins;
    constexpr uint32_t kWarpRuns = RowPartSmem<STEPS>::kWarpRuns, kTile = STEPS * kPartThreads, kBatch = 2;
    __shared__ uint32_t sTicket;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, below = lanesBelow();
    for (uint32_t j = tid; j < kPartWarps * bins; j += kPartThreads) sMask[j] = 0;
    gridWait();
    DeviceControl* ctl = a.ctl;
    const uint64_t* sorted = a.depthKeys[a.depthPlan->sortedBuffer & 1u];
    const uint32_t cutSlot = ctl->rowCutSlot, cutTiles = ctl->rowCutTiles;
    const uint32_t perView = (a.count + kTile - 1) / kTile, tiles = perView * a.viewCount;
    uint32_t* count = sCount + warp * bins;
    uint32_t* mask = sMask + warp * bins;
    uint2* runs = S.runs[warp];
    for (;;) {
        if (tid == 0) sTicket = atomicAdd(&ctl->tickets[kRowPartTicket], 1u);
        for (uint32_t j = tid; j < kPartWarps * bins; j += kPartThreads) sCount[j] = 0;
        __syncthreads();
        const uint32_t t = sTicket;
        if (t >= tiles) return;
        const uint32_t view = t / perView, local = t - view * perView;
        if (view * a.count + local * kTile > cutSlot) return;  // past a full list's last record, as all tiles after it
        const DevView vw = a.views[view];
        uint32_t listed = 0;
        // the records' runs, the loads of kBatch steps in flight together
        auto forRuns = [&](auto fn) {
#pragma unroll 1
            for (uint32_t s0 = 0; s0 < STEPS; s0 += kBatch) {
                const uint32_t slot0 = view * a.count + local * kTile + warp * (32 * STEPS) + s0 * 32 + lane;
                size_t rec[kBatch];
                bool some[kBatch];
                uint32_t kept[kBatch];  // cutTiles of the list's last record, nothing of those after it
                RecordRows R[kBatch];
                slotRecords(a, sorted, view, slot0, 32u, rec, some);
#pragma unroll
                for (uint32_t j = 0; j < kBatch; ++j) {
                    const uint32_t slot = slot0 + j * 32;
                    kept[j] = some[j] && slot <= cutSlot ? (slot == cutSlot ? cutTiles : 1u) : 0u;
                }
                recordRows(a, vw, rec, kept, R);
#pragma unroll
                for (uint32_t j = 0; j < kBatch; ++j)
                    forWarpRuns(a, vw, view, rec[j], R[j], kept[j], slot0 + j * 32 == cutSlot && kept[j] != 0, S.terms[warp], fn);
            }
        };
        forRuns([&](bool valid, uint32_t row, uint32_t run, uint32_t gaussian) {
            valid = valid && row < bins;
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, valid);
            const uint32_t at = listed + __popc(m & below);
            if (valid) {
                atomicAdd(&count[row], 1u);
                if (at < kWarpRuns) runs[at] = make_uint2((run & 0xFFFFu) | ((run >> 16) << 10) | (row << 20), gaussian);
            }
            listed += __popc(m);
        });
        __syncthreads();
        // thread tid's row: the block's entries, then their place after the earlier blocks'
        uint32_t mine = 0;
        uint32_t* status = a.rowStatus + size_t(t) * kRowBins;
        if (tid < bins) {
#pragma unroll
            for (uint32_t w = 0; w < kPartWarps; ++w) {
                const uint32_t c = sCount[w * bins + tid];
                sCount[w * bins + tid] = mine;
                mine += c;
            }
            stRelaxed32(&status[tid], (local == 0 ? kRowInclusive : kRowAggregate) | mine);
        }
        const uint32_t before = local ? rowLookback(a.rowStatus, t, t - local, bins, ctl, S.sum, S.found) : 0u;
        if (tid < bins) {
            if (local) stRelaxed32(&status[tid], kRowInclusive | ((before + mine) & kRowValue));
            const uint32_t place = a.rowPlan[size_t(view) * kRowBins + tid].x + before;
#pragma unroll
            for (uint32_t w = 0; w < kPartWarps; ++w) sCount[w * bins + tid] += place;
        }
        __syncthreads();
        auto write = [&](bool valid, uint32_t row, uint32_t run, uint32_t gaussian) {
            if (valid) atomicOr(&mask[row], 1u << lane);
            __syncwarp();
            uint32_t peers = 0, first = 0;
            if (valid) {
                peers = mask[row];
                first = count[row];
                const uint32_t place = first + __popc(peers & below);
                if (place < a.capacity) a.rowEntries[place] = make_uint2(run, gaussian);
                else atomicOr(&ctl->c.status, uint32_t(GSR_CONTROL_BOUNDS));
            }
            __syncwarp();
            if (valid && (peers & below) == 0) {  // the first of them
                count[row] = first + __popc(peers);
                mask[row] = 0;
            }
            __syncwarp();
        };
        const uint32_t inList = listed < kWarpRuns ? listed : kWarpRuns;
        for (uint32_t p = lane; p - lane < inList; p += 32) {
            const uint2 e = p < inList ? runs[p] : make_uint2(0u, 0u);
            write(p < inList, e.x >> 20, (e.x & 0x3FFu) | (((e.x >> 10) & 0x3FFu) << 16), e.y);
        }
        if (listed > kWarpRuns) {  // the runs that found no place in the list, in the same order
            uint32_t seen = 0;
            forRuns([&](bool valid, uint32_t row, uint32_t run, uint32_t gaussian) {
                valid = valid && row < bins;
                const uint32_t m = __ballot_sync(0xFFFFFFFFu, valid);
                const bool late = valid && seen + __popc(m & below) >= kWarpRuns;
                seen += __popc(m);
                write(late, row, run, gaussian);
            });
        }
        if (tiles <= gridDim.x) return;  // every block's first ticket was its only one
        __syncthreads();
    }
}

// One bucket (a view's tile row) a cluster. Shared memory, W = the widest view's tiles of a row:
// counts [warps][W + 1] (ends of runs, then the warps' places), masks [warps][W], the block's tile
// counts [W] that the cluster's other blocks read.
__global__ void __cluster_dims__(kRowCluster, 1, 1) __launch_bounds__(kTileThreads)
    rowTilesKernel(const __grid_constant__ FrontArgs a, uint32_t W) {
    extern __shared__ uint32_t sRowTiles[];
    __shared__ uint64_t sWarp[kTileWarps];
    uint32_t* counts = sRowTiles;
    uint32_t* masks = counts + kTileWarps * (W + 1);
    uint32_t* tileCount = masks + kTileWarps * W;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, below = lanesBelow();
    for (uint32_t j = tid; j < kTileWarps * (2 * W + 1) + W; j += kTileThreads) sRowTiles[j] = 0;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t part = cluster.block_rank(), bucket = blockIdx.x / kRowCluster;
    gridWait();
    const uint32_t view = a.buckets[bucket] >> 8, row = a.buckets[bucket] & 0xFFu;
    const DevView vw = a.views[view];
    const uint4 plan = a.rowPlan[size_t(view) * kRowBins + row];
    const uint32_t entries = plan.x < a.capacity ? (plan.y < a.capacity - plan.x ? plan.y : a.capacity - plan.x) : 0u;
    // the warp's contiguous share of the bucket, in steps of 32
    const uint32_t share = ((entries + kRowCluster * kTileThreads - 1) / (kRowCluster * kTileThreads)) * 32u;
    const uint32_t w0 = (part * kTileWarps + warp) * share;
    const uint32_t w1 = w0 + share < entries ? w0 + share : entries;
    const uint2* in = a.rowEntries + plan.x;
    uint32_t* count = counts + warp * (W + 1);
    uint32_t* mask = masks + warp * W;
    const uint32_t tilesX = vw.tilesX;
    // a run's ends, inside the row whatever the word holds
    auto ends = [&](uint2 e, uint32_t& x0, uint32_t& x1) {
        x0 = e.x & 0xFFFFu;
        x1 = e.x >> 16;
        x1 = x1 < tilesX ? x1 : tilesX;
        x0 = x0 < x1 ? x0 : x1;
    };
    __syncthreads();
#pragma unroll 4
    for (uint32_t k = w0 + lane; k < w1; k += 32) {
        uint32_t x0, x1;
        ends(__ldcg(&in[k]), x0, x1);
        atomicAdd(&count[x0], 1u);
        atomicSub(&count[x1], 1u);
    }
    __syncwarp();
    // the warp's tile counts: the running sum of the ends
    uint32_t carry = 0;
    for (uint32_t x = lane; x < (tilesX + 31u) / 32u * 32u; x += 32) {
        uint32_t v = x < tilesX ? count[x] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
            if (lane >= uint32_t(o)) v += u;
        }
        v += carry;
        if (x < tilesX) count[x] = v;
        carry = __shfl_sync(0xFFFFFFFFu, v, 31);
    }
    __syncthreads();
    for (uint32_t x = tid; x < tilesX; x += kTileThreads) {
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t w = 0; w < kTileWarps; ++w) {
            const uint32_t c = counts[w * (W + 1) + x];
            counts[w * (W + 1) + x] = sum;
            sum += c;
        }
        tileCount[x] = sum;
    }
    cluster.sync();
    // the row's tiles: their sizes over the cluster, their places in the list, the ranges
    uint32_t run = 0, last = 0;
    for (uint32_t x0 = 0; x0 < tilesX; x0 += kTileThreads) {
        const uint32_t x = x0 + tid;
        uint32_t all = 0, before = 0;
        if (x < tilesX) {
            uint32_t c[kRowCluster];
#pragma unroll
            for (uint32_t p = 0; p < kRowCluster; ++p) c[p] = cluster.map_shared_rank(tileCount, p)[x];
#pragma unroll
            for (uint32_t p = 0; p < kRowCluster; ++p) {
                if (p < part) before += c[p];
                all += c[p];
            }
        }
        uint64_t total;
        const uint32_t start = plan.z + run + uint32_t(blockScan64<kTileWarps>(all, sWarp, &total));
        run += uint32_t(total);
        if (x < tilesX) {
            if (part == 0) {
                reinterpret_cast<uint2*>(a.ranges)[vw.tileBase + row * tilesX + x] =
                    all ? make_uint2(start, start + all) : make_uint2(0u, 0u);
                if (all) last = x;
            }
#pragma unroll
            for (uint32_t w = 0; w < kTileWarps; ++w) counts[w * (W + 1) + x] += start + before;
        }
    }
    last = __reduce_max_sync(0xFFFFFFFFu, last);
    if (part == 0 && run && lane == 0) {  // (the warp's last tile with an entry; tile 0 of the row for the others)
        const uint32_t tile = vw.tileBase + row * tilesX + last;
        atomicMax(&a.ctl->c.tile_max, tile);
        atomicMax(&a.ctl->c.key_bits, bitWidth32(tile));
    }
    cluster.barrier_arrive();  // this block has read the others' counts (waited for before it ends)
    __syncthreads();
    // every run's gaussian to its tiles' places, the (run, tile) pairs shared out over the lanes
    uint32_t* terms = tileCount + W + warp * 64;
    uint2 next = w0 + lane < w1 ? __ldcg(&in[w0 + lane]) : make_uint2(0u, 0u);
    for (uint32_t k0 = w0; k0 < w1; k0 += 32) {
        const uint2 e = next;  // a step ahead
        next = k0 + 32 + lane < w1 ? __ldcg(&in[k0 + 32 + lane]) : make_uint2(0u, 0u);
        uint32_t x0, x1;
        ends(e, x0, x1);
        WarpPairs pairs(x1 - x0);
        __syncwarp();
        if (x1 > x0) {
            terms[pairs.place] = x0 - pairs.begin;  // tile = pair + this
            terms[32 + pairs.place] = e.y;
        }
        __syncwarp();
        for (uint32_t p0 = 0; p0 < pairs.total; p0 += 32) {
            const uint32_t q = pairs.owner(p0), p = p0 + lane;
            const bool valid = p < pairs.total;
            uint32_t x = 0, peers = 0, first = 0, gaussian = 0;
            if (valid) {
                x = p + terms[q];
                gaussian = terms[32 + q];
                atomicOr(&mask[x], 1u << lane);
            }
            __syncwarp();
            if (valid) {
                peers = mask[x];
                first = count[x];
                const uint32_t place = first + __popc(peers & below);
                if (place < a.capacity) a.list[place] = gaussian;
            }
            __syncwarp();
            if (valid && (peers & below) == 0) {  // the first of them
                count[x] = first + __popc(peers);
                mask[x] = 0;
            }
            __syncwarp();
        }
    }
    cluster.barrier_wait();
}

}  // namespace

namespace {
template <uint32_t STEPS>
cudaError_t launchRowPartitionT(const FrontArgs& a, cudaStream_t s) {
    static std::atomic<int> grids[64] = {};
    std::atomic<int>& grid = perDevice(grids);
    const uint32_t bins = (a.rowsPerView + 31u) / 32u * 32u;
    if (!grid) {
        const cudaError_t e = cudaFuncSetAttribute(rowPartitionKernel<STEPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   int(rowPartBytes<STEPS>(kRowBins)));
        if (e != cudaSuccess) return e;
        int dev = 0, sms = 148, perSm = 2;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, rowPartitionKernel<STEPS>, kPartThreads, rowPartBytes<STEPS>(kRowBins));
        grid = sms * (perSm > 0 ? perSm : 1);
    }
    const uint32_t tile = STEPS * kPartThreads, tiles = (a.count + tile - 1) / tile * a.viewCount;
    return launchDependent(rowPartitionKernel<STEPS>, dim3(tiles < uint32_t(grid) ? tiles : uint32_t(grid)), kPartThreads,
                           rowPartBytes<STEPS>(bins), s, a, bins);
}
}  // namespace

cudaError_t launchRowPartition(const FrontArgs& a, cudaStream_t s) {
    const uint64_t records = uint64_t(a.count) * a.viewCount;
    const uint32_t planBlocks = uint32_t((records + kRowTile - 1) / kRowTile);
    const cudaError_t e = launchDependent(rowPlanKernel, dim3(planBlocks < 148u ? planBlocks : 148u), kRowThreads, 0, s, a);
    if (e != cudaSuccess) return e;
    if (rowPartitionTile(records) == kRowPartTile) return launchRowPartitionT<2>(a, s);
    return launchRowPartitionT<4>(a, s);
}

// 512 records a block where 1,024 would leave SMs without one (100,000 records: 23.6 against 25.9 us for
// the plan and the partition); 1,024 otherwise (1.24 M: 77 us; 2,048: 96; 512 threads and 2,048: 83).
uint32_t rowPartitionTile(uint64_t records) { return records < 148 * 1024 ? kRowPartTile : 4 * kPartThreads; }
static_assert(kRowPartTile == 2 * kPartThreads, "the small blocks");

cudaError_t launchRowTiles(const FrontArgs& a, uint32_t maxTilesX, cudaStream_t s) {
    static std::atomic<bool> configuredOn[64] = {};
    std::atomic<bool>& configured = perDevice(configuredOn);
    auto bytes = [](uint32_t w) { return size_t(kTileWarps * (2 * w + 1) + w + kTileWarps * 64) * 4; };
    if (!configured) {
        const cudaError_t e =
            cudaFuncSetAttribute(rowTilesKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes(kRowMaxTilesX)));
        if (e != cudaSuccess) return e;
        configured = true;
    }
    return launchDependent(rowTilesKernel, dim3(a.bucketCount * kRowCluster), kTileThreads, bytes(maxTilesX), s, a,
                           maxTilesX);
}

}  // namespace gsr
