// Host side of one batch through the kernels: table layout, scratch sizing and the launch phases,
// shared by the renderer (one frame), the batch API (many frames) and the differentiable renderer.
// All phases are queued before the host reads their totals, once: buffers are sized from the largest
// totals seen, and a batch that outgrows them is redone.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "dsrg_internal.h"

namespace dsrg {

static size_t align16(size_t x) { return (x + 15) & ~(size_t)15; }

size_t layout_tables(TaskParams *tasks, size_t taskCount, FrameTarget *frames, size_t frameCount, const TextureData *textures,
                     size_t textureCount, bool depthOnly, unsigned long long *keysBase, unsigned char *host,
                     unsigned char *deviceBase, BatchParams &params, BatchTotals &totals) {
	// bases
	uint32_t points = 0, triangles = 0, tiles = 0;
	size_t pixels = 0;
	for (size_t i = 0; i < taskCount; i++) {
		TaskParams &t = tasks[i];
		t.pointBase = points;
		t.triangleBase = triangles;
		points += (uint32_t)t.pointCount;
		triangles += (uint32_t)t.triangleCount;
	}
	for (size_t i = 0; i < frameCount; i++) {
		FrameTarget &f = frames[i];
		f.tilesX = (f.width + TILE_W - 1) / TILE_W;
		f.tilesY = (f.height + TILE_H - 1) / TILE_H;
		f.tileBase = tiles;
		tiles += (uint32_t)(f.tilesX * f.tilesY);
		f.keys = keysBase ? keysBase + pixels : nullptr;
		pixels += (size_t)f.width * f.height;
	}
	totals.points = points;
	totals.triangles = triangles;
	totals.tiles = tiles;
	totals.pixels = pixels;
	// layout
	const size_t taskOffset = 0;
	const size_t pointBaseOffset = align16(taskOffset + taskCount * sizeof(TaskParams));
	const size_t triangleBaseOffset = align16(pointBaseOffset + (taskCount + 1) * sizeof(uint32_t));
	const size_t frameOffset = align16(triangleBaseOffset + (taskCount + 1) * sizeof(uint32_t));
	const size_t frameTileOffset = align16(frameOffset + frameCount * sizeof(FrameTarget));
	const size_t textureOffset = align16(frameTileOffset + (frameCount + 1) * sizeof(uint32_t));
	const size_t bytes = align16(textureOffset + (textureCount + 1) * sizeof(TextureData));
	if (host) {
		memset(host, 0, bytes);
		if (taskCount) memcpy(host + taskOffset, tasks, taskCount * sizeof(TaskParams));
		uint32_t *pointBase = (uint32_t *)(host + pointBaseOffset), *triangleBase = (uint32_t *)(host + triangleBaseOffset);
		for (size_t i = 0; i < taskCount; i++) { pointBase[i] = tasks[i].pointBase; triangleBase[i] = tasks[i].triangleBase; }
		pointBase[taskCount] = points;
		triangleBase[taskCount] = triangles;
		if (frameCount) memcpy(host + frameOffset, frames, frameCount * sizeof(FrameTarget));
		uint32_t *frameTile = (uint32_t *)(host + frameTileOffset);
		for (size_t i = 0; i < frameCount; i++) frameTile[i] = frames[i].tileBase;
		frameTile[frameCount] = tiles;
		if (textureCount) memcpy(host + textureOffset, textures, textureCount * sizeof(TextureData));
	}
	params.tasks = (const TaskParams *)(deviceBase + taskOffset);
	params.taskPointBase = (const uint32_t *)(deviceBase + pointBaseOffset);
	params.taskTriangleBase = (const uint32_t *)(deviceBase + triangleBaseOffset);
	params.taskCount = (int32_t)taskCount;
	params.frames = (const FrameTarget *)(deviceBase + frameOffset);
	params.frameTileBase = (const uint32_t *)(deviceBase + frameTileOffset);
	params.frameCount = (int32_t)frameCount;
	params.textures = (const TextureData *)(deviceBase + textureOffset);
	params.totalPoints = points;
	params.totalTriangles = triangles;
	params.totalTiles = tiles;
	params.depthOnly = depthOnly ? 1 : 0;
	params.oddDepthFrames = 0;
	params.maxTilesX = 0;
	for (size_t i = 0; i < frameCount; i++) {
		if ((frames[i].height & 1) && frames[i].depth) params.oddDepthFrames++;
		params.maxTilesX = std::max(params.maxTilesX, frames[i].tilesX);
	}
	return bytes;
}

size_t layout_tables(BatchJob &job, unsigned long long *keysBase, unsigned char *host, unsigned char *deviceBase,
                     BatchParams &params, BatchTotals &totals) {
	return layout_tables(job.tasks.data(), job.tasks.size(), job.frames.data(), job.frames.size(), job.textures.data(),
	                     job.textures.size(), job.depthOnly, keysBase, host, deviceBase, params, totals);
}

#define TRY(expr) DSRG_CUDA_TRY(ctx, expr)

// Launch parameters of one phase; compared byte for byte, so it is cleared before it is filled.
struct PhaseKey {
	int32_t phase;
	int32_t resolve;
	int32_t alpha;
	uint32_t recordCount;
	RasterConfig config;
	BatchParams params;
	FrameBuffers fb;
	TileBins bins;
	uint32_t *rowCounts;
};

// Runs one phase's launches on the context's stream, through its graph when the phase repeats.
template <typename Launches>
static cudaError_t run_phase(dsrg_context ctx, PhaseGraph &g, const PhaseKey &key, Launches launches) {
	const unsigned char *k = reinterpret_cast<const unsigned char *>(&key);
	const bool same = g.key.size() == sizeof(key) && memcmp(g.key.data(), k, sizeof(key)) == 0;
	if (!ctx->useGraphs || !same) {
		if (!same) {
			if (g.exec) cudaGraphExecDestroy(g.exec);
			g.exec = nullptr;
			g.key.assign(k, k + sizeof(key));
		}
		launches();
		const cudaError_t enqueued = take_enqueue_error();
		const cudaError_t launched = cudaGetLastError();
		return enqueued != cudaSuccess ? enqueued : launched;
	}
	if (g.exec) {
		add_launches(g.launches);
		return cudaGraphLaunch(g.exec, ctx->stream);
	}
	const uint64_t before = launch_count();
	cudaError_t e = cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal);
	if (e != cudaSuccess) return e;
	launches();
	const cudaError_t enqueued = take_enqueue_error();
	const cudaError_t refused = cudaGetLastError(); // a launch refused while capturing
	const cudaError_t launched = enqueued != cudaSuccess ? enqueued : refused;
	cudaGraph_t graph = nullptr;
	e = cudaStreamEndCapture(ctx->stream, &graph);
	if (e != cudaSuccess) return e;
	if (launched != cudaSuccess) {
		cudaGraphDestroy(graph);
		return launched;
	}
	g.launches = launch_count() - before;
	e = cudaGraphInstantiate(&g.exec, graph, 0);
	cudaGraphDestroy(graph);
	if (e != cudaSuccess) {
		g.exec = nullptr;
		return e;
	}
	return cudaGraphLaunch(g.exec, ctx->stream);
}

static int enqueue_phases(dsrg_context ctx, BatchJob &job, BatchTotals &totals, BatchOutputs *outputs) {
	cudaStream_t stream = ctx->stream;
	ctx->stopRecorded = false;
	totals = BatchTotals();
	BatchParams params;
	memset(&params, 0, sizeof(params));
	// sizes first, then the buffers, then the tables with their final device addresses
	const size_t tableBytes = layout_tables(job, nullptr, nullptr, nullptr, params, totals);
	if (totals.pixels > 0) TRY(ctx->keys.reserve(totals.pixels));
	TRY(ctx->tables.reserve(tableBytes));
	if (job.depthOnly) TRY(ctx->tileList.reserve((size_t)totals.tiles + 1));
	if (ctx->pinnedCapacity < tableBytes) {
		if (ctx->pinnedTables) cudaFreeHost(ctx->pinnedTables);
		ctx->pinnedTables = nullptr;
		ctx->pinnedCapacity = 0;
		size_t capacity = 4096;
		while (capacity < tableBytes) capacity *= 2;
		TRY(cudaMallocHost((void **)&ctx->pinnedTables, capacity));
		ctx->pinnedCapacity = capacity;
	}
	layout_tables(job, ctx->keys.ptr, ctx->pinnedTables, ctx->tables.ptr, params, totals);
	TRY(cudaMemcpyAsync(ctx->tables.ptr, ctx->pinnedTables, tableBytes, cudaMemcpyHostToDevice, stream));
	// without the resolve pass the caller reads every key, also where no tile was drawn
	if (!job.resolve && totals.pixels > 0) TRY(cudaMemsetAsync(ctx->keys.ptr, 0, totals.pixels * sizeof(unsigned long long), stream));
	params.smallRows = ctx->smallRows;
	params.smallWidth = ctx->smallWidth;
	params.tileQueue = ctx->control.ptr + CONTROL_TILE_QUEUE;
	// depth-only batches (shadow-cube faces) are mostly empty tiles: their tile kernel pulls only
	// the listed ones.  Colour frames pull every tile in order, which measured faster for them
	// (the listed order is not the tile order, and the list costs a wider totals launch).
	params.tileList = job.depthOnly ? ctx->tileList.ptr : nullptr;
	params.tileListCount = job.depthOnly ? ctx->control.ptr + CONTROL_LISTED_TILES : nullptr;
	params.fragments = nullptr;
	params.walked = ctx->fragmentCounter.ptr + 1;
	if (ctx->counting && !job.clearCounters) {
		params.fragments = ctx->fragmentCounter.ptr;
	} else if (ctx->counting) {
		TRY(cudaMemsetAsync(ctx->fragmentCounter.ptr, 0, sizeof(unsigned long long), stream));
		params.fragments = ctx->fragmentCounter.ptr;
		for (const FrameTarget &f : job.frames)
			if (f.coverage) TRY(cudaMemsetAsync(f.coverage, 0, (size_t)f.width * f.height * sizeof(uint32_t), stream));
	}
	if (totals.triangles == 0) return DSRG_OK; // nothing reaches the tiles: the targets stay as they are
	params.errorFlag = (const int32_t *)(ctx->control.ptr + CONTROL_ERROR);
	RasterConfig config;
	config.threadsPerTile = ctx->threadsPerTile;
	config.ctasPerSm = ctx->ctasPerSm;
	// Fewer triangles than one per 8 pixels: tall triangles, whose rows are dealt in segments
	// (rows_segment_kernel); the others' rows are stepped record by record in the launch that places them
	// (rows_place_kernel).  By segments and by records: 300 random triangles at 800x600 124 and 203 us, 20,000 187
	// and 425, terrain of 130,000 at 1920x1080 (16 pixels each) 163 and 179, meshes of 10 to 40 pixels a triangle
	// alike; below the line the terrain of 522,000 at 1920x1080 (4 pixels) 257 and 241, while random triangles, whose
	// size has nothing to do with their number, would still gain (100,000 at 800x600: 356 and 716).
	const bool tallTriangles = (uint64_t)totals.triangles * 8u <= (uint64_t)totals.pixels;
	// how winners are shaded (the context's tuning); targets in host memory take the per-pixel
	// stores inside the tile kernel (2x2 quads scatter small writes over the link)
	config.resolveMode = ctx->resolveMode == 2 && job.hostTargets ? 1 : ctx->resolveMode;

	// Buffers whose sizes depend on earlier phases are sized from the context's capacities (the
	// largest totals seen, with slack); the phases then run back to back with no host round trip.
	// A total above its capacity sets an overflow bit, the tile and resolve kernels return at once,
	// and batch_enqueue redoes the batch with the capacities the totals asked for.
	const size_t np = totals.points, nt = totals.triangles;
	// the one-pass setup keeps a slot per fan triangle and extra ones for the pieces of clipped
	// triangles; beyond its record numbers' range the two-pass setup counts first
	const bool onePass = nt < ctx->onePassLimit;
	const uint32_t recordCap = onePass ? (uint32_t)(nt + std::max<uint64_t>(ctx->extraCapacity, nt / 8 + 1024))
	                                   : (uint32_t)std::max<uint64_t>(ctx->recordCapacity, nt + nt / 8 + 1024);
	// Four rows per record at first, and where rows are placed in whole segments (tall triangles) what rounding
	// up can add to each, so that a frame of a new context is not drawn twice for the padding alone: a mesh
	// of 57,600 triangles at 1281x719 has 223,000 rows, 402,000 in segments, and four a record are 263,000.
	const uint64_t rowsAtFirst = (uint64_t)recordCap * (onePass && tallTriangles ? 4 + ROW_SEGMENT - 2 : 4);
	const uint32_t rowCap = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(ctx->rowCapacity, rowsAtFirst), 0xFFFFFFF0u);
	const uint32_t binCap = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(ctx->binCapacity, (uint64_t)recordCap * 2), 0xFFFFFFF0u);
	if (!onePass) {
		TRY(ctx->triCounts.reserve(nt + 1));
		TRY(ctx->triOffsets.reserve(nt + 1));
		TRY(ctx->rowCounts.reserve((size_t)recordCap + 1));
		TRY(ctx->rowOffsets.reserve((size_t)recordCap + 1));
	}
	// The arrays of a batch lie in one allocation, which a new context maps once and a redo once more: with
	// buffers of their own for the records, rows and lists the first frame of 57,600 triangles at 1281x719 took 374 us
	// instead of 311, of 20,000 random triangles at 800x600 685 instead of 577, with one for each array 100 us more.
	size_t scratchBytes = 0;
	const auto part = [&](size_t bytes) {
		const size_t at = scratchBytes;
		scratchBytes = (at + bytes + 255) & ~(size_t)255;
		return at;
	};
	const uint32_t partWeight = job.depthOnly ? DEPTH_PART_WEIGHT : PART_WEIGHT;
	const size_t slots = 2 * (size_t)totals.tiles + 1;
	const size_t csisAt = part(np * sizeof(*ctx->pointCsis.ptr)), isyOutAt = part(np * sizeof(*ctx->pointIsyOut.ptr));
	const size_t flatAt = part(np * sizeof(*ctx->pointFlat.ptr));
	const size_t countsAt = part(slots * sizeof(uint32_t)), offsetsAt = part(slots * sizeof(uint32_t)), cursorsAt = part(slots * sizeof(uint32_t));
	const size_t bigListAt = part(((size_t)recordCap + 1) * sizeof(uint32_t)), thresholdsAt = part(((size_t)totals.tiles + 1) * sizeof(uint32_t));
	const size_t partsAt = part(((size_t)max_parts(binCap, partWeight) + 1) * sizeof(uint2)), partsDoneAt = part(((size_t)totals.tiles + 1) * sizeof(uint32_t));
	const size_t sortAt = job.alpha ? part((size_t)binCap * sizeof(uint32_t)) : 0;
	size_t marksAt = 0, extraBaseAt = 0, extraIdsAt = 0, headsAt = 0, ranksAt = 0, segmentsAt = 0;
	if (onePass) {
		marksAt = part(((size_t)recordCap + 4) * sizeof(uint16_t)); // read four at a time
		extraBaseAt = part((nt + 1) * sizeof(uint32_t));
		extraIdsAt = part(((size_t)recordCap - nt + 1) * sizeof(uint32_t));
		headsAt = part(((size_t)recordCap + 1) * sizeof(uint4));
		ranksAt = part(((size_t)recordCap + 1) * sizeof(uint2));
		if (tallTriangles) segmentsAt = part(((size_t)rowCap / ROW_SEGMENT + 1) * sizeof(uint32_t));
	}
	const uint64_t scanned = std::max<uint64_t>(onePass ? 0 : recordCap, 2 * (uint64_t)totals.tiles);
	const size_t scanElems = scan_scratch_elems((uint32_t)scanned + 1), scanAt = part(scanElems * sizeof(uint32_t));
	// the large arrays after the small ones (before them the frame of two million triangles at 3840x2160 took 768 us on
	// the GPU instead of 763)
	const size_t rowsAt = part(((size_t)rowCap + 2) * sizeof(uint32_t)), listsAt = part(((size_t)binCap + 1) * sizeof(uint32_t));
	const size_t recordsAt = part(((size_t)recordCap + 1) * sizeof(DrawRecord));
	TRY(ctx->batchScratch.replace(scratchBytes / sizeof(uint4)));
	uint8_t *scratch = reinterpret_cast<uint8_t *>(ctx->batchScratch.ptr);
	const auto words = [&](size_t at) { return reinterpret_cast<uint32_t *>(scratch + at); };
	FrameBuffers fb;
	memset(&fb, 0, sizeof(fb));
	fb.points.csis = reinterpret_cast<decltype(fb.points.csis)>(scratch + csisAt);
	fb.points.isyOut = reinterpret_cast<decltype(fb.points.isyOut)>(scratch + isyOutAt);
	fb.points.flat = reinterpret_cast<decltype(fb.points.flat)>(scratch + flatAt);
	fb.records = reinterpret_cast<DrawRecord *>(scratch + recordsAt);
	fb.rows = words(rowsAt);
	fb.errorFlag = (int32_t *)(ctx->control.ptr + CONTROL_ERROR);
	fb.scanScratch = words(scanAt);
	fb.scanScratchElems = scanElems;
	fb.rowCapacity = rowCap;
	if (onePass) {
		fb.emit.counters = ctx->control.ptr + CONTROL_EMIT;
		fb.emit.drawn = reinterpret_cast<uint16_t *>(scratch + marksAt);
		fb.emit.triangles = (uint32_t)nt;
		fb.emit.capacity = recordCap;
		fb.emit.extraBase = words(extraBaseAt);
		fb.emit.extraIds = words(extraIdsAt);
		fb.emit.tileHeads = reinterpret_cast<uint4 *>(scratch + headsAt);
		fb.emit.tileRanks = reinterpret_cast<uint2 *>(scratch + ranksAt);
		fb.emit.segmentSlots = tallTriangles ? words(segmentsAt) : nullptr;
		fb.emit.tileCursors = words(cursorsAt);
		fb.emit.bigList = words(bigListAt);
		fb.emit.bigCount = ctx->control.ptr + CONTROL_BIG_RECORDS;
		fb.recordCountDevice = fb.emit.counters + EMIT_DRAWN;
		params.recordShift = 3;
		params.extraBase = words(extraBaseAt);
	} else {
		fb.triCounts = ctx->triCounts.ptr;
		fb.triOffsets = ctx->triOffsets.ptr;
		fb.rowOffsets = ctx->rowOffsets.ptr;
		fb.recordCountDevice = fb.triOffsets + nt;
	}
	TileBins bins;
	memset(&bins, 0, sizeof(bins));
	bins.counts = words(countsAt);
	bins.offsets = words(offsetsAt);
	bins.cursors = words(cursorsAt);
	bins.lists = words(listsAt);
	bins.listCapacity = binCap;
	bins.scratch = job.alpha ? words(sortAt) : nullptr;
	bins.bigList = words(bigListAt);
	bins.bigCount = ctx->control.ptr + CONTROL_BIG_RECORDS;
	bins.cleared = 1; // by the first launch of phase A
	// records are culled while binning where only the best key of a pixel counts: not where every
	// fragment is counted, nor for the alpha filter, which blends them all
	bins.thresholds = (job.alpha || params.fragments) ? nullptr : words(thresholdsAt);
	bins.culled = bins.thresholds ? ctx->control.ptr + CONTROL_CULLED : nullptr;
	if (!job.alpha) {
		bins.parts = reinterpret_cast<uint2 *>(scratch + partsAt);
		bins.partCount = ctx->control.ptr + CONTROL_TILE_PARTS;
		bins.partWeight = partWeight;
		bins.partCapacity = max_parts(binCap, partWeight);
		bins.partsDone = words(partsDoneAt);
	}
	ClearedCounters clear;
	memset(&clear, 0, sizeof(clear));
	clear.tileCounts = bins.counts;
	clear.tileCursors = bins.cursors;
	clear.tileSlots = 2 * totals.tiles;
	clear.thresholds = bins.thresholds;
	clear.control = ctx->control.ptr;
	clear.words = CONTROL_WORDS;
	TotalsSources from;
	memset(&from, 0, sizeof(from));
	from.records = fb.recordCountDevice;
	from.rows = onePass ? fb.emit.counters + EMIT_ROWS : nullptr;
	from.extras = onePass ? fb.emit.counters + EMIT_EXTRAS : nullptr;
	from.culled = ctx->control.ptr + CONTROL_CULLED;
	from.rowOffsets = fb.rowOffsets;
	from.recordCapacity = recordCap;
	from.errorFlag = fb.errorFlag;
	uint32_t *rowCounts = ctx->rowCounts.ptr;
	uint32_t *gathered = ctx->readbackDevice; // records, rows, bin entries, error bits: written into host memory
	PhaseKey key;
	memset(&key, 0, sizeof(key));
	key.resolve = job.resolve ? 1 : 0;
	key.alpha = job.alpha ? 1 : 0;
	key.config = config;
	key.params = params;
	key.fb = fb;
	key.bins = bins;
	key.rowCounts = rowCounts;
	key.recordCount = recordCap;
	key.phase = 0;
	// phases A (projection, records), B (tile counts and list offsets) and C (row intervals, tile
	// lists) as one graph, then D (tiles and resolve, or the alpha filter) as another
	const int graph = job.alpha ? 2 : 0; // a frame's solid and alpha-filtered runs each keep their graphs
	TRY(run_phase(ctx, ctx->graphs[graph], key, [&] {
		launch_project(params, fb, stream, &clear);
		if (onePass) {
			launch_setup_emit(params, fb, stream);
			// the row intervals on a second branch right after the records, the tile counts, offsets
			// and lists on this one: neither needs the other; joined before the totals
			enqueue_join(stream, ctx->branchStream, ctx->branchFork);
			launch_rows(fb, recordCap, ctx->branchStream);
			launch_bin_count(params, fb, recordCap, bins, stream);
			launch_bin_fill(params, fb, recordCap, bins, stream);
			enqueue_join(ctx->branchStream, stream, ctx->branchJoin);
		} else {
			launch_setup_count(params, fb, stream);
			launch_setup_write(params, fb, recordCap, stream);
			launch_row_offsets(fb, recordCap, rowCounts, stream);
			launch_rows(fb, recordCap, stream);
			launch_bin_count(params, fb, recordCap, bins, stream);
			launch_bin_fill(params, fb, recordCap, bins, stream);
		}
		launch_gather_totals(params, from, bins, gathered, stream);
	}));
	// phase D right behind, timed on the stream between the two graphs; after an overflow its
	// kernels return at once and the targets stay untouched
	TRY(cudaEventRecord(ctx->eventRasterStart, stream));
	key.phase = 1;
	TRY(run_phase(ctx, ctx->graphs[graph + 1], key, [&] {
		if (job.alpha) launch_alpha(params, fb, bins, stream);
		else launch_raster(params, fb, bins, config, job.resolve, stream);
	}));
	TRY(cudaEventRecord(ctx->eventRasterStop, stream));
	// the batch's own work ends here: the one host wait below also completes the timing events
	TRY(cudaEventRecord(ctx->eventStop, stream));
	if (ctx->counting)
		TRY(cudaMemcpyAsync(ctx->pinnedReadback + 4, ctx->fragmentCounter.ptr, sizeof(unsigned long long), cudaMemcpyDeviceToHost,
		                    stream));
	if (ctx->beforeWait) { // once, also when the batch is redone
		const std::function<void()> work = std::move(ctx->beforeWait);
		ctx->beforeWait = nullptr;
		work();
	}
	TRY(cudaStreamSynchronize(stream));
	ctx->stopRecorded = true;
	totals.records = ctx->pinnedReadback[0];
	totals.rows = ctx->pinnedReadback[1];
	const uint32_t counted = ctx->pinnedReadback[2]; // the tile lists' entries
	totals.binEntries = counted + ctx->pinnedReadback[TOTALS_CULLED];
	const uint32_t errorBits = ctx->pinnedReadback[3];
	if (errorBits & ERROR_OVERFLOW_BITS) {
		// the capacities the totals ask for; a total counted past an overflowed buffer is a lower bound
		const uint64_t extras = onePass ? ctx->pinnedReadback[TOTALS_EXTRAS] : 0;
		const bool recordsOver = onePass ? nt + extras > recordCap : totals.records > recordCap;
		if (onePass) ctx->extraCapacity = std::max<uint64_t>(ctx->extraCapacity, extras + extras / 4 + 1024);
		else ctx->recordCapacity = std::max<uint64_t>(ctx->recordCapacity, (uint64_t)totals.records + totals.records / 4 + 1024);
		// rows and entries of the pieces that found no slot: as many each as the others have, so that one redo
		// is mostly enough (the two-pass setup's own totals say nothing about them)
		const uint64_t missing = onePass && recordsOver ? nt + extras - recordCap : 0;
		const double scale = missing && totals.records ? 1.0 + (double)missing / totals.records : 1.0;
		if (!recordsOver || missing) {
			const uint64_t rows = (uint64_t)(scale * totals.rows), entries = (uint64_t)(scale * counted);
			ctx->rowCapacity = std::max<uint64_t>(ctx->rowCapacity, rows + rows / 4 + 1024);
			// the entries counted depend on how early the tiles' thresholds rose (bin_big_kernel), by a third from
			// run to run for 20,000 random triangles at 800x600: twice the total, so that a frame that has
			// been drawn once is not redone for it
			ctx->binCapacity = std::max<uint64_t>(ctx->binCapacity, entries * 2 + 1024);
		}
		return DSRG_RETRY;
	}
	if (errorBits != 0) return fail(ctx, DSRG_ERROR_DEVICE, "triangle setup reported device error bits " + std::to_string(errorBits));
	if (outputs) {
		outputs->params = params;
		outputs->fb = fb;
		outputs->slots = onePass ? (uint32_t)nt + ctx->pinnedReadback[TOTALS_EXTRAS] : totals.records;
	}
	return DSRG_OK;
}

int batch_enqueue(dsrg_context ctx, BatchJob &job, BatchTotals &totals, BatchOutputs *outputs) {
	if (outputs) memset(outputs, 0, sizeof(*outputs));
	int status = DSRG_RETRY;
	// a batch whose totals outgrow the capacities is redone with larger ones
	for (int attempt = 0; attempt < 4 && status == DSRG_RETRY; attempt++) status = enqueue_phases(ctx, job, totals, outputs);
	if (status == DSRG_RETRY) return fail(ctx, DSRG_ERROR_DEVICE, "batch buffers kept overflowing");
	if (status == DSRG_OK && !ctx->stopRecorded) TRY(cudaEventRecord(ctx->eventStop, ctx->stream));
	return status;
}

int occlude_enqueue(dsrg_context ctx, BatchJob &job) {
	cudaStream_t stream = ctx->stream;
	BatchTotals totals;
	BatchParams params;
	memset(&params, 0, sizeof(params));
	const size_t tableBytes = layout_tables(job, nullptr, nullptr, nullptr, params, totals);
	if (totals.triangles == 0) return DSRG_OK;
	TRY(ctx->tables.reserve(tableBytes));
	if (ctx->pinnedCapacity < tableBytes) {
		if (ctx->pinnedTables) cudaFreeHost(ctx->pinnedTables);
		ctx->pinnedTables = nullptr;
		ctx->pinnedCapacity = 0;
		size_t capacity = 4096;
		while (capacity < tableBytes) capacity *= 2;
		TRY(cudaMallocHost((void **)&ctx->pinnedTables, capacity));
		ctx->pinnedCapacity = capacity;
	}
	layout_tables(job, nullptr, ctx->pinnedTables, ctx->tables.ptr, params, totals);
	TRY(cudaMemcpyAsync(ctx->tables.ptr, ctx->pinnedTables, tableBytes, cudaMemcpyHostToDevice, stream));
	const size_t np = totals.points;
	TRY(ctx->pointCsis.reserve(np)); TRY(ctx->pointIsyOut.reserve(np)); TRY(ctx->pointFlat.reserve(np));
	FrameBuffers fb;
	memset(&fb, 0, sizeof(fb));
	fb.points.csis = ctx->pointCsis.ptr; fb.points.isyOut = ctx->pointIsyOut.ptr; fb.points.flat = ctx->pointFlat.ptr;
	fb.errorFlag = (int32_t *)(ctx->control.ptr + CONTROL_ERROR);
	launch_project(params, fb, stream);
	launch_setup_occlude(params, fb, stream);
	TRY(take_enqueue_error());
	TRY(cudaGetLastError());
	// the page-locked tables are rewritten by the next batch: wait for their copy (and the grid)
	TRY(cudaStreamSynchronize(stream));
	return DSRG_OK;
}

// Only the setup, row and binning kernels raise error bits, and enqueue_phases has read them
// after those (gather_totals_kernel): what is left is the fragment count and one wait for the
// work the caller queued after the batch (image copies, overlays), if any.
int batch_finish(dsrg_context ctx, const BatchTotals &totals) {
	cudaStream_t stream = ctx->stream;
	unsigned long long fragments = 0;
	uint32_t *readback = ctx->pinnedReadback + 4;
	if (ctx->counting && !ctx->stopRecorded)
		TRY(cudaMemcpyAsync(readback, ctx->fragmentCounter.ptr, sizeof(fragments), cudaMemcpyDeviceToHost, stream));
	TRY(cudaStreamSynchronize(stream));
	if (ctx->counting) memcpy(&fragments, readback, sizeof(fragments));
	ctx->stopRecorded = false;
	ctx->timingPending = true;
	ctx->timingHasRaster = totals.triangles > 0;
	ctx->stats.fragments = fragments;
	ctx->stats.drawRecords = totals.records;
	ctx->stats.binEntries = totals.binEntries;
	ctx->stats.kernelLaunches = launch_count();
	return DSRG_OK;
}

} // namespace dsrg
