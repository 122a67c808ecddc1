// Launch interface of the kernels of the DFPSR triangle path (host side).
//
// Every launch covers a whole batch: any number of frames (target image pairs), each drawn by
// any number of tasks (models with a transform and a camera).  model_render is a batch of one
// frame with one task, renderer_begin/giveTask/end one frame with several tasks.
#ifndef DSRG_KERNELS_H
#define DSRG_KERNELS_H

#include <cuda_runtime.h>
#include <stdint.h>
#include "dsrg_types.h"

namespace dsrg {

// One model submitted to a frame: model_render / renderer_giveTask (api/modelAPI.cpp:197-281).
struct TaskParams {
	const float *positions;   // pointCount x 3
	const int32_t *polygons;  // polygonCount x 4
	const float *texCoords;   // polygonCount x 4 x 4
	const float *colors;      // polygonCount x 4 x 4
	const int32_t *triSource; // per fan triangle: polygon * 2 + fan index
	int32_t pointCount;
	int32_t triangleCount;
	uint32_t pointBase;       // this task's first projected point in the batch
	uint32_t triangleBase;    // this task's first fan triangle in the batch
	uint32_t orderBase;       // fan triangles submitted earlier to the same frame
	int32_t frame;            // the frame this task draws into
	float modelToWorld[12];
	CameraData camera;
	int32_t filter;           // 0 Solid, 1 Alpha
	int32_t diffuse, light;   // indices into the batch's texture table, -1 for none
	int32_t depthOnly;        // model_renderDepth: 1x1 alignment, no shading (renderCore.cpp:343-443)
	const GivenPoint *given;  // renderer_giveTask_triangle: the corners come projected (positions unused)
};

// One frame of a batch: its target images, its key image and its range of tiles.
struct FrameTarget {
	uint32_t *color;          // device pointer or null
	int32_t colorStride;      // in pixels
	int32_t packOrder;
	float *depth;             // device pointer or null
	int32_t depthStride;
	int32_t width, height;
	int32_t affine;           // orthogonal camera: depth test '<' on linear depth
	unsigned long long *keys; // width * height winning (depth, record) keys, written by the tile pass
	uint32_t *coverage;       // optional per-pixel fragment counts (width * height, dense)
	uint32_t tileBase;        // the frame's first tile in the batch
	int32_t tilesX, tilesY;
	float *occlusion;         // the renderer's occlusion grid (gridWidth x gridHeight cells) or null
	int32_t gridWidth, gridHeight, gridStride;
};

// Device tables of a batch.
struct BatchParams {
	const TaskParams *tasks;
	const uint32_t *taskPointBase;    // taskCount + 1 prefix sums of point counts
	const uint32_t *taskTriangleBase; // taskCount + 1 prefix sums of fan-triangle counts
	int32_t taskCount;
	const FrameTarget *frames;
	const uint32_t *frameTileBase;    // frameCount + 1 prefix sums of tile counts
	int32_t frameCount;
	uint32_t totalPoints, totalTriangles, totalTiles;
	const TextureData *textures;
	unsigned long long *fragments;    // optional fragment total
	unsigned long long *walked;       // optional running total of the fragments the tile kernels depth-tested
	int32_t smallRows;                // records whose raster bound is at most smallRows x smallWidth pixels
	int32_t smallWidth;               // are walked by one lane each instead of by the whole warp
	int32_t depthOnly;                // the whole batch is model_renderDepth (1x1 walk)
	int32_t oddDepthFrames;           // frames of odd height with a depth buffer (their last row: odd_row_kernel)
	int32_t maxTilesX;                // the widest frame's tile columns
	uint32_t *tileQueue;              // work counter of the persistent tile kernel
	uint4 *tileList;                  // the tiles that have list entries (written at the end of phase C) as tile, first
	                                  // entry, entries and frame, or null: every tile
	uint32_t *tileListCount;          // their number
	uint32_t recordShift;             // 3: records numbered 8 * fan triangle + piece, 0: as they are stored (record_slot)
	const uint32_t *extraBase;        // per fan triangle: where the further pieces of a clipped triangle begin
	const int32_t *errorFlag;         // device error bits; tile and resolve kernels return when an overflow is set
};

// Projected corners (implementation/render/ProjectedPoint.h:33-49): the camera-space position and
// the image x in one 16-byte vector, the image y with the camera planes that the point lies outside
// of, and both sub-pixel coordinates in one 16-byte vector, so that the triangle setup gathers a
// corner with three loads.
struct ProjectedPoints {
	float4 *csis;     // cs.x, cs.y, cs.z, is.x
	uint2 *isyOut;    // is.y (bits) and the planes the point is outside of (outside_planes)
	longlong2 *flat;  // flat x, flat y
};

// What the one-pass setup writes beside the records.  Counters in device memory, zeroed by the
// batch's first launch: draw records, row intervals taken, extra slots taken.
enum EmitCounter : uint32_t { EMIT_DRAWN = 0, EMIT_ROWS = 1, EMIT_EXTRAS = 2, EMIT_COUNTERS = 3 };
static const uint32_t ROW_SEGMENT = 16; // rows one thread of rows_segment_kernel computes
// A slot's mark: 0 no record, else its tiles + 1 (of a record over at most four) or DRAWN_BIG, and half
// its rows (always even) above, DRAWN_ROWS_MAX standing for that many or more.
static const uint32_t DRAWN_BITS = 3, DRAWN_MASK = 7, DRAWN_BIG = 6, DRAWN_ROWS_MAX = (1u << (16 - DRAWN_BITS)) - 1u;
__host__ __device__ inline uint16_t drawn_mark(uint32_t tiles, int32_t rows) {
	const uint32_t half = (uint32_t)rows / 2u;
	return (uint16_t)(tiles | ((half < DRAWN_ROWS_MAX ? half : DRAWN_ROWS_MAX) << DRAWN_BITS));
}

struct EmitBuffers {
	uint32_t *counters;      // EMIT_COUNTERS values
	uint16_t *drawn;         // per slot: drawn_mark; null: the two-pass setup
	uint32_t triangles;      // slots of the fan triangles, which come first,
	uint32_t capacity;       // and all slots
	uint32_t *extraBase;     // per fan triangle with further pieces: their first extra slot
	uint32_t *extraIds;      // per extra slot: its record's number
	uint4 *tileHeads;        // per slot of a record over at most four tiles: its first tile-list slot, tilesX | columns << 16,
	                         // and its places in the first two tiles' lists
	uint2 *tileRanks;        // over more than two tiles: its places in the third and fourth
	uint32_t *segmentSlots;  // tall triangles: the record of every segment of ROW_SEGMENT rows; null: rows are packed in pairs
	uint32_t *tileCursors;   // 2 * totalTiles: the places taken in each tile's lists
	uint32_t *bigList, *bigCount; // records over more than four tiles, for bin_big_kernel
};

struct FrameBuffers {
	ProjectedPoints points;
	uint32_t *triCounts;      // two-pass setup: draw records that each fan triangle emits,
	uint32_t *triOffsets;     // their exclusive scan, total at [totalTriangles],
	uint32_t *rowOffsets;     // and per record its first row interval (+ total at [recordCount])
	DrawRecord *records;
	uint32_t *rows;           // row intervals of every record, left | right << 16
	int32_t *errorFlag;       // device error bits
	uint32_t *scanScratch;
	size_t scanScratchElems;
	// when set, the record count is read on the device (at most the host count given to the
	// launches, which then bounds the grids), and rows hold at most rowCapacity entries
	const uint32_t *recordCountDevice;
	uint32_t rowCapacity;
	EmitBuffers emit;         // the one-pass setup (emit.drawn set)
};

// Counters zeroed by a batch's first launch (launch_project).
struct ClearedCounters {
	uint32_t *tileCounts, *tileCursors; // tileSlots values each
	uint32_t *thresholds;               // tileSlots / 2 values, or null
	uint32_t tileSlots;
	uint32_t *control;                  // words values: tile queue, error bits, emit counters, list lengths
	uint32_t words;
};

// Two lists per tile: slot 2 * tile holds the records walked one lane each (small), slot
// 2 * tile + 1 the ones walked by a whole warp (large).
struct TileBins {
	uint32_t *counts;   // 2 * totalTiles: entries of each list (one-pass setup: of its big records)
	uint32_t *offsets;  // 2 * totalTiles + 1
	uint32_t *cursors;  // 2 * totalTiles: places taken in each list
	uint32_t *lists;
	size_t listCapacity;
	uint32_t *scratch;  // alpha filter: as long as lists, where long ones are sorted
	// records over more than four tiles, listed by setup_emit_kernel and binned by whole blocks
	uint32_t *bigList;
	uint32_t *bigCount;
	// per tile: a key (upper word) that every pixel of the tile reaches, from the big records covering it
	// completely; large records below it are not listed.  null: nothing is culled while binning
	uint32_t *thresholds;
	uint32_t *culled; // (tile, record) pairs left out of the count; null: nothing is culled
	// tiles weighing more than partWeight as (tile, part) items, and per tile the parts done; null: every
	// tile is drawn by one CTA
	uint2 *parts;
	uint32_t partWeight;
	uint32_t *partCount;
	uint32_t partCapacity;
	uint32_t *partsDone;
	// the tile queue is zeroed by the batch's first launch (0: launch_raster zeroes it with a memset)
	int32_t cleared;
};

// What a tile's lists cost to draw, and the share of it that one CTA takes.  A large entry is walked by
// a whole warp, small ones 32 at a time: about eight times the time.  Shares of 2,048 to 8,192 take a
// batch of small frames of many triangles the same time; dense terrain seen from afar (a thousand
// small entries in a tile of the horizon) should not be cut, which cost 3 to 10 % of its frame.
// Depth-only tiles are drawn by single warps, whose share is smaller.
static const uint32_t LARGE_WEIGHT = 8, PART_WEIGHT = 4096, DEPTH_PART_WEIGHT = 1024;
__host__ __device__ inline uint32_t part_weight(uint32_t smalls, uint32_t larges) { return smalls + LARGE_WEIGHT * larges; }
// At most this many parts for lists of `entries` entries in all: a cut tile weighs more than partWeight.
inline uint32_t max_parts(uint64_t entries, uint32_t partWeight) { return (uint32_t)(2 * LARGE_WEIGHT * entries / partWeight) + 1u; }

// True when one lane walks the whole record inside a tile (small-triangle path).
__host__ __device__ inline bool bound_is_small(int32_t left, int32_t top, int32_t right, int32_t bottom, int32_t smallRows,
                                               int32_t smallWidth) {
	return (bottom - top) <= smallRows && (right - left) <= smallWidth;
}
__host__ __device__ inline bool record_is_small(const DrawRecord &r, int32_t smallRows, int32_t smallWidth) {
	return bound_is_small(r.left, r.top, r.right, r.bottom, smallRows, smallWidth);
}

enum ErrorBits : int32_t {
	ERROR_RECORD_OVERFLOW = 1,
	ERROR_COORDINATE_RANGE = 2,
	ERROR_BIN_OVERFLOW = 4,
	ERROR_ROW_OVERFLOW = 8,
	ERROR_INTERNAL = 16,
	// a buffer sized before its count was known was too small: the frame is redone with larger
	// buffers, and the kernels that would read past them or write the targets return at once
	ERROR_OVERFLOW_BITS = ERROR_RECORD_OVERFLOW | ERROR_BIN_OVERFLOW | ERROR_ROW_OVERFLOW,
};

// Phase A: projection (zeroing the counters of the launches behind it when `clear` is given).
void launch_project(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream, const ClearedCounters *clear = nullptr);
// The one-pass setup (fb.emit): every fan triangle's records with their places in the tile lists.  Needs fewer than MAX_EMIT_TRIANGLES fan triangles.
static const uint32_t MAX_EMIT_TRIANGLES = 1u << 29;
void launch_setup_emit(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream);
// The two-pass setup: the count of draw records per fan triangle, scanned so that the record count
// ends at triOffsets[totalTriangles], then the records in submission order (per frame: the order of
// its tasks, then of their triangles), row offsets (total at rowOffsets[recordCount]).
void launch_setup_count(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream);
void launch_setup_write(const BatchParams &b, const FrameBuffers &fb, uint32_t recordCapacity, cudaStream_t stream);
// occludeFromExistingTriangles (api/rendererAPI.cpp:240-255): every solid draw command of the batch
// whose bound exceeds one cell lowers the occlusion grid of its frame over the cells it covers.
void launch_setup_occlude(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream);
// occludeFromTopRows (api/rendererAPI.cpp:417-476) from a device depth image.
void launch_occlusion_top_rows(float *grid, int32_t gridWidth, int32_t gridHeight, int32_t gridStride, const float *depth,
                               int32_t depthStride, int32_t width, bool perspective, cudaStream_t stream);
void launch_row_offsets(const FrameBuffers &fb, uint32_t recordCount, uint32_t *rowCounts, cudaStream_t stream);
// Phase B: tile counts and where each tile's lists begin (total at offsets[2 * totalTiles]).
void launch_bin_count(const BatchParams &b, const FrameBuffers &fb, uint32_t recordCount, TileBins &bins, cudaStream_t stream);
// Phase C: row intervals, tile lists, the persistent tile raster and the per-pixel resolve.
void launch_rows(const FrameBuffers &fb, uint32_t recordCount, cudaStream_t stream);
void launch_bin_fill(const BatchParams &b, const FrameBuffers &fb, uint32_t recordCount, TileBins &bins, cudaStream_t stream);
// Launch shape of the persistent tile kernel.
struct RasterConfig {
	int32_t threadsPerTile; // 64, 128 or 256
	int32_t ctasPerSm;      // resident CTAs per SM pulling tiles (at most 1024 / threadsPerTile)
	int32_t resolveMode;    // 0 one pixel per thread in a pass of its own, 1 per pixel inside the tile
	                        // kernel, 2 one 2x2 quad per thread in a pass of its own (same results)
};
// resolve = false leaves the winners in the key images (the differentiable renderer reads them).
void launch_raster(const BatchParams &b, const FrameBuffers &fb, const TileBins &bins, const RasterConfig &config, bool resolve,
                   cudaStream_t stream);
// Buffers of launch_stable_sort for n items: keys and ids twice n; hist and offsets
// 256 * sort_blocks(n) + 1; scan scratch for 256 * sort_blocks(n) + 1 values.
struct SortBuffers {
	uint32_t *keysA, *keysB, *idsA, *idsB, *hist, *offsets;
	uint32_t *scanScratch;
	size_t scanScratchElems;
};
uint32_t sort_blocks(uint64_t n); // n >= 1
// Stable LSD radix sort of the indices of the n >= 1 items by their keys, leaving out the items whose
// key is not below keyEnd; *keptDevice is the number of the others.  *sortedIds points at the buffer
// holding the result.
void launch_stable_sort(const uint32_t *keys, uint64_t n, uint32_t keyEnd, const uint32_t *keptDevice, const SortBuffers &b,
                        cudaStream_t stream, const uint32_t **sortedIds);
// The alpha filter over the binned records (in place of launch_raster): colour blends in
// submission order, depth read only.
void launch_alpha(const BatchParams &b, const FrameBuffers &fb, const TileBins &bins, cudaStream_t stream);
// Debug overlays: the three edges of every record as lines in pixels (flat / 256), and draw_line
// (api/drawAPI.cpp:176-279) of many lines of one packed colour into a device image.
// (drawn: the records' marks per slot, null for the first `slots` records; counter: zero, counts them.)
void launch_wire_lines(const DrawRecord *records, const uint16_t *drawn, uint32_t slots, uint32_t capacity, uint32_t *counter, int4 *lines,
                       cudaStream_t stream);
void launch_draw_lines(uint32_t *image, int32_t stride, int32_t width, int32_t height, const int4 *lines, uint32_t count,
                       uint32_t color, cudaStream_t stream);
// out[0..3] = record count, row count, tile-list entry count, error bits of a batch, and the extra
// slots at out[TOTALS_EXTRAS], the pairs that binning culled before counting at out[TOTALS_CULLED].
static const uint32_t TOTALS_EXTRAS = 9, TOTALS_CULLED = 10;
struct TotalsSources {
	const uint32_t *records, *rows, *extras, *culled;
	const uint32_t *rowOffsets;   // the two-pass setup: the row count is rowOffsets[records]
	uint32_t recordCapacity;
	const int32_t *errorFlag;
};
void launch_gather_totals(const BatchParams &b, const TotalsSources &from, const TileBins &bins, uint32_t *out, cudaStream_t stream);
// Exclusive scan of n uint32 values into out (out[n] = total); two launches, scratch of
// scan_scratch_elems(n) values.
void launch_scan(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *scratch, size_t scratchElems, cudaStream_t stream);
// The same for a length written on the device (*nDevice, at most capacity; scratch for capacity).
void launch_scan_device(const uint32_t *in, uint32_t *out, const uint32_t *nDevice, uint32_t capacity, uint32_t *scratch,
                        size_t scratchElems, cudaStream_t stream);
size_t scan_scratch_elems(uint32_t n);
// The first memset the launchers above failed to enqueue on this thread since the last call
// (cudaSuccess if none), cleared by the call; callers check it with cudaGetLastError after launching.
cudaError_t take_enqueue_error();
// Makes `to` wait for what `from` has queued so far (an event recorded on `from`); inside a stream
// capture this forks or joins branches of the graph.  A failure is kept for take_enqueue_error.
void enqueue_join(cudaStream_t from, cudaStream_t to, cudaEvent_t event);
// Kernels launched by this library in this process (host-side count).
uint64_t launch_count();
// Adds kernels launched through a replayed CUDA graph to that count.
void add_launches(uint64_t n);
int32_t sm_count();

} // namespace dsrg

#endif
