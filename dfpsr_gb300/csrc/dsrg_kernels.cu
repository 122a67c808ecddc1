// CUDA kernels of the DFPSR triangle path for sm_103a.
//
// Every launch covers a whole batch of frames (see dsrg_kernels.h).  Per batch:
//   A  project_kernel       Camera::worldToScreen for every model point (implementation/render/Camera.h:157-190),
//                           and the counters of the launches behind it zeroed
//      setup_emit_kernel    per fan triangle: cull, clip, front-face; writes the DrawRecords (bound, sub-pixel
//                           corners, projection), takes their rows and counts their tiles
//   B  bin_big_kernel       (tile, record) pairs of the records over more than four tiles
//      scan                 where each tile's list begins
//   C  rows_*_kernel        row intervals of every record (rasterizeTriangle)
//      bin_fill_kernel      per-tile record lists
//   D  raster_kernel        persistent CTAs pull tiles from a queue; every fragment competes for
//                           64-bit depth keys in shared memory; every pixel re-evaluates and shades its winner
//
// Why the depth test can run out of order: the reference writes a fragment when its depth is
// strictly greater (1/W, perspective) or smaller (linear, orthogonal) than the stored one
// (implementation/render/shader/fillerTemplates.h:108-152).  After any sequence of opaque
// triangles the stored value is the extreme depth over all fragments that beat the initial
// value, and the colour is the earliest fragment reaching it.  Packing (depth, ~record index)
// into one 64-bit key and taking the maximum reproduces exactly that, in any order, because
// record numbers grow in submission order.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <utility>

#include "dsrg_exact.h"
#include "dsrg_geometry.h"
#include "dsrg_shade.h"
#include "dsrg_kernels.h"
#include "dsrg_raster.cuh"
#include "dsrg_occlusion.h"

namespace dsrg {

static uint64_t g_launches = 0;

// The first failed enqueue of a memset inside the launchers of this thread, reported to the caller
// of the launches by take_enqueue_error (the launchers themselves return nothing).
static thread_local cudaError_t t_enqueueError = cudaSuccess;

static void memset_async(void *p, int value, size_t bytes, cudaStream_t stream) {
	const cudaError_t e = cudaMemsetAsync(p, value, bytes, stream);
	if (e != cudaSuccess && t_enqueueError == cudaSuccess) t_enqueueError = e;
}

void enqueue_join(cudaStream_t from, cudaStream_t to, cudaEvent_t event) {
	cudaError_t e = cudaEventRecord(event, from);
	if (e == cudaSuccess) e = cudaStreamWaitEvent(to, event, 0);
	if (e != cudaSuccess && t_enqueueError == cudaSuccess) t_enqueueError = e;
}

cudaError_t take_enqueue_error() {
	const cudaError_t e = t_enqueueError;
	t_enqueueError = cudaSuccess;
	return e;
}
uint64_t launch_count() { return g_launches; }
void add_launches(uint64_t n) { g_launches += n; }
#define COUNT_LAUNCH() (g_launches++)

int32_t sm_count() {
	static int32_t count = 0;
	if (count == 0) {
		int device = 0, value = 0;
		cudaGetDevice(&device);
		cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device);
		count = value > 0 ? value : 1;
	}
	return count;
}

// Grid of a grid-stride kernel over n items: enough CTAs to fill the GPU, never more than needed.
static int grid_for(uint64_t n, int threads) {
	uint64_t blocks = (n + threads - 1) / threads;
	const uint64_t cap = (uint64_t)sm_count() * 16;
	if (blocks > cap) blocks = cap;
	return (int)(blocks > 0 ? blocks : 1);
}

// Programmatic dependent launch.  A kernel launched with launch_chained may be scheduled while
// the kernel before it on the stream is still running: that kernel lets it in once all of its
// CTAs have started (the release in chain_enter), and chain_enter, the first statement of every
// chained kernel, holds its threads until the predecessor has completed with its writes visible.
// Captured into a graph the pair becomes a programmatic edge, so the launch of each dependent
// kernel overlaps the last CTAs of the one before.  Kernels launched the ordinary way pass the
// wait at once.  Every CTA of a chained kernel runs chain_enter before anything else, so a kernel
// completes only after its predecessor did and the chain stays ordered end to end.
__device__ __forceinline__ void chain_enter() {
	asm volatile("griddepcontrol.wait;" ::: "memory");
	asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... Params, typename... Args>
static void launch_chained(void (*kernel)(Params...), dim3 grid, uint32_t block, cudaStream_t stream, Args &&...args) {
	cudaLaunchAttribute attribute[1];
	attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
	attribute[0].val.programmaticStreamSerializationAllowed = 1;
	cudaLaunchConfig_t config;
	memset(&config, 0, sizeof(config));
	config.gridDim = grid;
	config.blockDim = dim3(block);
	config.stream = stream;
	config.attrs = attribute;
	config.numAttrs = 1;
	cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

// A count written on the device, bounded by the capacity the host sized the buffers for.
__device__ __forceinline__ uint32_t device_count(uint32_t capacity, const uint32_t *countDevice) {
	if (!countDevice) return capacity;
	const uint32_t n = *countDevice;
	return n < capacity ? n : capacity;
}

__device__ __forceinline__ bool overflowed(const BatchParams &b) {
	return b.errorFlag && (*(volatile const int32_t *)b.errorFlag & ERROR_OVERFLOW_BITS) != 0;
}

// ------------------------------------------------------------------ projection

// The planes that a camera-space point lies outside of: bit s for culling plane s, bit
// OUTSIDE_CLIP_SHIFT + s for clipping plane s (at most six of each).  Tested once per point instead
// of for every corner of every triangle (some six corners share a point of a mesh), the planes cost the
// triangle setup three loads it makes anyway: 64 views of 50,000 triangles went from 938 to 913 us, a 4k
// terrain frame of two million from 908 to 871 us.
static const uint32_t OUTSIDE_CLIP_SHIFT = 6, OUTSIDE_CULL_MASK = (1u << OUTSIDE_CLIP_SHIFT) - 1u;

__device__ __forceinline__ uint32_t outside_planes(const CameraData &c, const Vec3 &p) {
	uint32_t out = 0;
	for (int s = 0; s < c.cullCount; s++) out |= plane_inside(c.cull[s], p) ? 0u : 1u << s;
	for (int s = 0; s < c.clipCount; s++) out |= plane_inside(c.clip[s], p) ? 0u : 1u << (OUTSIDE_CLIP_SHIFT + s);
	return out;
}

// The counters of a batch's later launches, zeroed by its first one (`clear`, see ClearedCounters):
// no launch or memset of their own sits in the chain.
__device__ __forceinline__ void clear_counters(const ClearedCounters &c) {
	const uint32_t at = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
	for (uint32_t i = at; i < c.tileSlots; i += stride) {
		c.tileCounts[i] = 0u;
		c.tileCursors[i] = 0u;
		if (c.thresholds && !(i & 1u)) c.thresholds[i >> 1] = 0u;
	}
	for (uint32_t i = at; i < c.words; i += stride) c.control[i] = 0u;
}

__global__ void project_kernel(BatchParams b, ProjectedPoints out, ClearedCounters clear) {
	chain_enter();
	clear_counters(clear);
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < b.totalPoints; i += gridDim.x * blockDim.x) {
		const TaskParams &task = b.tasks[find_segment(b.taskPointBase, b.taskCount, i)];
		const uint32_t local = i - task.pointBase;
		if (task.given) { // renderer_giveTask_triangle: projected by the caller
			const GivenPoint &g = task.given[local];
			out.csis[i] = make_float4(g.cs[0], g.cs[1], g.cs[2], g.is[0]);
			out.isyOut[i] = make_uint2(fbits(g.is[1]), outside_planes(task.camera, vec3(g.cs[0], g.cs[1], g.cs[2])));
			out.flat[i] = make_longlong2(g.flat[0], g.flat[1]);
			continue;
		}
		Vec3 p = vec3(task.positions[local * 3], task.positions[local * 3 + 1], task.positions[local * 3 + 2]);
		Projected pr = camera_to_screen(task.camera, world_to_camera(task.camera, transform_point(task.modelToWorld, p)));
		out.csis[i] = make_float4(pr.cs.x, pr.cs.y, pr.cs.z, pr.isx);
		out.isyOut[i] = make_uint2(fbits(pr.isy), outside_planes(task.camera, pr.cs));
		out.flat[i] = make_longlong2(pr.flatx, pr.flaty);
	}
}

void launch_project(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream, const ClearedCounters *clear) {
	ClearedCounters none;
	memset(&none, 0, sizeof(none));
	if (!clear) clear = &none;
	if (b.totalPoints == 0 && clear->words == 0) return;
	COUNT_LAUNCH();
	launch_chained(project_kernel, grid_for(std::max(b.totalPoints, clear->tileSlots), 256), 256, stream, b, fb.points, *clear);
}

// ------------------------------------------------------------------ triangle setup

struct Corner {
	Vec3 cs;
	float isx, isy;
	int64_t fx, fy;
};

// Emits one draw command (renderCore.cpp:203-217 executeTriangleDrawing against the whole target):
// the triangle bound cut to the target with rows aligned to pairs (ITriangle2D.cpp:70-75).
enum SetupMode { SETUP_COUNT = 0, SETUP_WRITE = 1, SETUP_OCCLUDE = 2 };

// Lowers a frame's occlusion grid to the command's farthest corner over the cells its triangle
// covers (occludeFromSortedHull with the triangle as the hull, rendererAPI.cpp:216-239, 240-255).
// Cells only ever decrease, so the order of the commands does not matter.
__device__ void occlude_cells(const FrameTarget &f, const int64_t *fx, const int64_t *fy, const int32_t *bd, const Corner *c) {
	if (!((bd[2] - bd[0]) > OCCLUSION_CELL && (bd[3] - bd[1]) > OCCLUSION_CELL)) return;
	float distance = 0.0f;
	for (int i = 0; i < 3; i++) if (c[i].cs.z > distance) distance = c[i].cs.z;
	const CellRect cells = outer_cell_bound(bd[0], bd[1], bd[2], bd[3], f.gridWidth, f.gridHeight);
	for (int32_t cy = cells.top; cy < cells.bottom; cy++) {
		for (int32_t cx = cells.left; cx < cells.right; cx++) {
			if (!cell_inside_hull(fx, fy, 3, cx, cy)) continue;
			// float minimum by compare-and-swap; it stops as soon as the cell holds a smaller value
			int *cell = reinterpret_cast<int *>(f.occlusion + (size_t)cy * f.gridStride + cx);
			int old = *cell;
			while (distance < __int_as_float(old)) {
				const int seen = atomicCAS(cell, old, __float_as_int(distance));
				if (seen == old) break;
				old = seen;
			}
		}
	}
}

template <int MODE>
__device__ void emit_record(const TaskParams &task, uint32_t taskIndex, const FrameTarget &frame, const FrameBuffers &fb,
                            uint32_t recordCapacity, const Corner *c, const float *subB, const float *subC, uint32_t tri,
                            uint32_t base, uint32_t &emitted) {
	const int32_t width = frame.width, height = frame.height;
	int64_t fx[3] = {c[0].fx, c[1].fx, c[2].fx}, fy[3] = {c[0].fy, c[1].fy, c[2].fy};
	int32_t bd[4];
	triangle_bound(fx, fy, bd);
	if (MODE == SETUP_OCCLUDE) {
		if (task.filter == 0 && frame.occlusion) occlude_cells(frame, fx, fy, bd, c);
		return;
	}
	// completeOcclusion: commands behind every cell of the grid are not drawn
	if (frame.occlusion &&
	    !command_survives(frame.occlusion, frame.gridWidth, frame.gridHeight, frame.gridStride, bd,
	                      nearest_corner(c[0].cs.z, c[1].cs.z, c[2].cs.z)))
		return;
	if (!(bd[0] < width && bd[2] > 0 && bd[1] < height && bd[3] > 0)) return;
	if (MODE == SETUP_WRITE) {
		const uint32_t index = base + emitted;
		if (index >= recordCapacity) {
			atomicOr(fb.errorFlag, ERROR_RECORD_OVERFLOW);
		} else {
			DrawRecord r;
			bool inRange = true;
			for (int i = 0; i < 3; i++) {
				if (fx[i] < -(1ll << 30) || fx[i] > (1ll << 30) || fy[i] < -(1ll << 30) || fy[i] > (1ll << 30)) inRange = false;
				r.flat[i * 2] = (int32_t)fx[i];
				r.flat[i * 2 + 1] = (int32_t)fy[i];
			}
			if (!inRange) atomicOr(fb.errorFlag, ERROR_COORDINATE_RANGE);
			r.left = bd[0] > 0 ? bd[0] : 0;
			r.top = (bd[1] > 0 ? bd[1] : 0) & ~1;                           // roundDown(top, 2)
			r.right = bd[2] < width ? bd[2] : width;
			r.bottom = ((bd[3] < height ? bd[3] : height) + 1) & ~1;        // roundUp(bottom, 2)
			float isx[3] = {c[0].isx, c[1].isx, c[2].isx}, isy[3] = {c[0].isy, c[1].isy, c[2].isy};
			float csz[3] = {c[0].cs.z, c[1].cs.z, c[2].cs.z};
			triangle_projection(isx, isy, csz, subB, subC, task.camera.perspective != 0, r.start, r.dx, r.dy);
			r.rowStart = 0; // written with the rows (rows_group_kernel)
			r.tri = tri;
			r.task = taskIndex;
			r.frame = (uint32_t)task.frame;
			r.source = task.triSource[tri];
			fb.records[index] = r;
		}
	}
	emitted++;
}

// The projected corners of fan triangle t of a task, and whether it is drawn at all: seen by the
// camera, and not an alpha-filtered triangle whose three alphas are almost zero (renderCore.cpp:319).
// *whole: no corner lies outside a clipping plane.  A triangle is hidden when one culling plane has
// all three corners outside (getTriangleVisibility, renderCore.cpp:172-198), which the corners' plane
// bits (outside_planes) tell without touching the planes again.
__device__ __forceinline__ bool load_triangle(const TaskParams &task, uint32_t t, const ProjectedPoints &points, Corner *c, bool *whole) {
	const int32_t src = task.triSource[t];
	const int32_t p = src >> 1, fan = src & 1;
	const int corner[3] = {0, 1 + fan, 2 + fan}; // fan 0-1-2, 0-2-3 (model/Model.cpp:135-162, 164-183)
	uint32_t all = 0xFFFFFFFFu, any = 0u;
	for (int i = 0; i < 3; i++) {
		const uint32_t pi = task.pointBase + (uint32_t)task.polygons[p * 4 + corner[i]];
		const float4 a = points.csis[pi];
		const uint2 y = points.isyOut[pi];
		const longlong2 f = points.flat[pi];
		c[i].cs = vec3(a.x, a.y, a.z);
		c[i].isx = a.w; c[i].isy = bitsf(y.x);
		c[i].fx = f.x; c[i].fy = f.y;
		all &= y.y;
		any |= y.y;
	}
	*whole = (any >> OUTSIDE_CLIP_SHIFT) == 0u;
	if ((all & OUTSIDE_CULL_MASK) != 0u) return false;
	if (!task.depthOnly && task.filter == 1) {
		const float *col = task.colors + p * 16;
		if (almost_zero(col[corner[0] * 4 + 3]) && almost_zero(col[corner[1] * 4 + 3]) && almost_zero(col[corner[2] * 4 + 3])) return false;
	}
	return true;
}

// renderTriangleFromData / renderTriangleFromDataDepth for one fan triangle (renderCore.cpp:220-341, 400-443).
template <int MODE>
__global__ void __launch_bounds__(256) setup_kernel(BatchParams b, FrameBuffers fb, uint32_t recordCapacity) {
	chain_enter();
	const bool WRITE = MODE == SETUP_WRITE;
	for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < b.totalTriangles; g += gridDim.x * blockDim.x) {
		const uint32_t k = (uint32_t)find_segment(b.taskTriangleBase, b.taskCount, g);
		const TaskParams &task = b.tasks[k];
		const FrameTarget &frame = b.frames[task.frame];
		const bool hasTarget = frame.color != nullptr || frame.depth != nullptr;
		const uint32_t t = g - task.triangleBase;
		uint32_t emitted = 0;
		const uint32_t base = WRITE ? fb.triOffsets[g] : 0u;
		if (WRITE && fb.triOffsets[g + 1] == base) continue; // the count pass emitted nothing for it
		Corner c[3];
		bool whole;
		const bool visible = load_triangle(task, t, fb.points, c, &whole);
		if (visible && hasTarget) {
			const float defaultB[3] = {0.0f, 1.0f, 0.0f}, defaultC[3] = {0.0f, 0.0f, 1.0f};
			const float zero3[3] = {0.0f, 0.0f, 0.0f};
			if (whole) {
				int64_t fx[3] = {c[0].fx, c[1].fx, c[2].fx}, fy[3] = {c[0].fy, c[1].fy, c[2].fy};
				if (is_frontfacing(fx, fy)) {
					emit_record<MODE>(task, k, frame, fb, recordCapacity, c, task.depthOnly ? zero3 : defaultB,
					                   task.depthOnly ? zero3 : defaultC, t, base, emitted);
				}
			} else {
				ClippedPolygon poly;
				poly.count = 3;
				for (int i = 0; i < 3; i++) { poly.v[i].cs = c[i].cs; poly.v[i].state = 0; poly.v[i].value = 0.0f; }
				poly.v[0].subB = 0.0f; poly.v[0].subC = 0.0f;
				poly.v[1].subB = 1.0f; poly.v[1].subC = 0.0f;
				poly.v[2].subB = 0.0f; poly.v[2].subC = 1.0f;
				for (int s = 0; s < task.camera.clipCount; s++) poly.clip(task.camera.clip[s]);
				for (int f = 0; f < poly.count - 2; f++) {
					const SubVertex *sv[3] = {&poly.v[0], &poly.v[1 + f], &poly.v[2 + f]};
					Corner sc[3];
					for (int i = 0; i < 3; i++) {
						Projected pr = camera_to_screen(task.camera, sv[i]->cs);
						sc[i].cs = pr.cs; sc[i].isx = pr.isx; sc[i].isy = pr.isy; sc[i].fx = pr.flatx; sc[i].fy = pr.flaty;
					}
					int64_t fx[3] = {sc[0].fx, sc[1].fx, sc[2].fx}, fy[3] = {sc[0].fy, sc[1].fy, sc[2].fy};
					if (is_frontfacing(fx, fy)) {
						float sb[3] = {sv[0]->subB, sv[1]->subB, sv[2]->subB};
						float scc[3] = {sv[0]->subC, sv[1]->subC, sv[2]->subC};
						emit_record<MODE>(task, k, frame, fb, recordCapacity, sc, task.depthOnly ? zero3 : sb,
						                   task.depthOnly ? zero3 : scc, t, base, emitted);
					}
				}
			}
		}
		if (MODE == SETUP_COUNT) fb.triCounts[g] = emitted;
	}
}

void launch_setup_count(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream) {
	if (b.totalTriangles == 0) {
		memset_async(fb.triOffsets, 0, sizeof(uint32_t), stream);
		return;
	}
	COUNT_LAUNCH();
	launch_chained(setup_kernel<SETUP_COUNT>, grid_for(b.totalTriangles, 256), 256, stream, b, fb, 0u);
	launch_scan(fb.triCounts, fb.triOffsets, b.totalTriangles, fb.scanScratch, fb.scanScratchElems, stream);
}

void launch_setup_write(const BatchParams &b, const FrameBuffers &fb, uint32_t recordCapacity, cudaStream_t stream) {
	if (b.totalTriangles == 0) return;
	COUNT_LAUNCH();
	launch_chained(setup_kernel<SETUP_WRITE>, grid_for(b.totalTriangles, 256), 256, stream, b, fb, recordCapacity);
}

void launch_setup_occlude(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream) {
	if (b.totalTriangles == 0) return;
	COUNT_LAUNCH();
	launch_chained(setup_kernel<SETUP_OCCLUDE>, grid_for(b.totalTriangles, 256), 256, stream, b, fb, 0u);
}

// ------------------------------------------------------------------ one-pass triangle setup

// One draw command on its way to a record: its corners and its raster bound.
struct Command {
	float isx[3], isy[3], csz[3];
	int32_t flat[6];
	int32_t left, top, right, bottom;
};

// Takes the corners over and cuts their bound to the target with rows aligned to pairs
// (ITriangle2D.cpp:70-75); false when the command faces away, lies outside or lies behind every
// cell of the occlusion grid.
__device__ __forceinline__ bool make_command(const FrameTarget &f, const Corner *c, int32_t *errorFlag, Command &m) {
	const int64_t fx[3] = {c[0].fx, c[1].fx, c[2].fx}, fy[3] = {c[0].fy, c[1].fy, c[2].fy};
	if (!is_frontfacing(fx, fy)) return false;
	int32_t bd[4];
	triangle_bound(fx, fy, bd);
	if (f.occlusion &&
	    !command_survives(f.occlusion, f.gridWidth, f.gridHeight, f.gridStride, bd, nearest_corner(c[0].cs.z, c[1].cs.z, c[2].cs.z)))
		return false;
	if (!(bd[0] < f.width && bd[2] > 0 && bd[1] < f.height && bd[3] > 0)) return false;
	bool inRange = true;
	for (int i = 0; i < 3; i++) {
		if (fx[i] < -(1ll << 30) || fx[i] > (1ll << 30) || fy[i] < -(1ll << 30) || fy[i] > (1ll << 30)) inRange = false;
		m.flat[2 * i] = (int32_t)fx[i];
		m.flat[2 * i + 1] = (int32_t)fy[i];
		m.isx[i] = c[i].isx;
		m.isy[i] = c[i].isy;
		m.csz[i] = c[i].cs.z;
	}
	if (!inRange) atomicOr(errorFlag, ERROR_COORDINATE_RANGE);
	m.left = bd[0] > 0 ? bd[0] : 0;
	m.top = (bd[1] > 0 ? bd[1] : 0) & ~1;                           // roundDown(top, 2)
	m.right = bd[2] < f.width ? bd[2] : f.width;
	m.bottom = ((bd[3] < f.height ? bd[3] : f.height) + 1) & ~1;    // roundUp(bottom, 2)
	return true;
}

__device__ __forceinline__ int32_t command_tiles(const Command &m, const FrameTarget &f, int32_t &tx0, int32_t &ty0, int32_t &w) {
	tx0 = m.left >> 4;
	ty0 = m.top >> 4;
	w = min((m.right - 1) >> 4, f.tilesX - 1) - tx0 + 1;
	const int32_t h = min((m.bottom - 1) >> 4, f.tilesY - 1) - ty0 + 1;
	return (w > 0 && h > 0) ? w * h : 0;
}

// Writes a command's record and what the launches behind it need (its rows are placed by
// rows_place_kernel).  subB, subC: its corners' places in the fan triangle.
__device__ __forceinline__ void store_command(const BatchParams &b, const FrameBuffers &fb, const TaskParams &task, uint32_t taskIndex,
                                              const FrameTarget &f, uint32_t tri, const Command &m, const float *subB, const float *subC,
                                              uint32_t slot) {
	const EmitBuffers &emit = fb.emit;
	int32_t tx0, ty0, w;
	const int32_t tiles = command_tiles(m, f, tx0, ty0, w);
	if (tiles > 4) {
		emit.drawn[slot] = drawn_mark(DRAWN_BIG, m.bottom - m.top);
		// one atomic for the lanes that are here together
		const unsigned together = __activemask();
		const uint32_t lane = threadIdx.x & 31u, leader = __ffs(together) - 1;
		uint32_t at = 0;
		if (lane == leader) at = atomicAdd(emit.bigCount, (uint32_t)__popc(together));
		at = __shfl_sync(together, at, leader);
		emit.bigList[at + __popc(together & ((1u << lane) - 1u))] = slot;
	} else {
		emit.drawn[slot] = drawn_mark((uint32_t)tiles + 1u, m.bottom - m.top);
		// a place in each tile's list: the atomics' answers arrive while the record is made
		const uint32_t large = (b.depthOnly || !bound_is_small(m.left, m.top, m.right, m.bottom, b.smallRows, b.smallWidth)) ? 1u : 0u;
		const uint32_t first = 2u * (f.tileBase + (uint32_t)(ty0 * f.tilesX + tx0)) + large;
		uint32_t rank[4] = {0u, 0u, 0u, 0u};
		// tile i at column i % w, row i / w (w at most 4)
#pragma unroll
		for (int32_t i = 0; i < 4; i++) {
			const int32_t row = w == 1 ? i : (w == 2 ? i >> 1 : (i >= w ? 1 : 0));
			if (i < tiles) rank[i] = atomicAdd(&emit.tileCursors[first + 2u * (uint32_t)(row * f.tilesX + i - row * w)], 1u);
		}
		emit.tileHeads[slot] = make_uint4(first, (uint32_t)f.tilesX | ((uint32_t)w << 16), rank[0], rank[1]);
		if (tiles > 2) emit.tileRanks[slot] = make_uint2(rank[2], rank[3]);
	}
	DrawRecord r;
	for (int i = 0; i < 6; i++) r.flat[i] = m.flat[i];
	r.left = m.left; r.top = m.top; r.right = m.right; r.bottom = m.bottom;
	triangle_projection(m.isx, m.isy, m.csz, subB, subC, task.camera.perspective != 0, r.start, r.dx, r.dy);
	r.rowStart = 0;
	r.tri = tri;
	r.task = taskIndex;
	r.frame = (uint32_t)task.frame;
	r.source = task.triSource[tri];
	fb.records[slot] = r;
}

// A fan triangle that crosses a clipping plane: every piece is stored on its own, the first at the
// triangle's slot (renderTriangleFromData, renderCore.cpp:220-341).  Returns whether there was one.  Out of line: few triangles come
// here, and the polygon would cost the others their registers.
__device__ __noinline__ bool emit_clipped(const BatchParams &b, const FrameBuffers &fb, uint32_t g, uint32_t k, const Corner *corners) {
	const TaskParams &task = b.tasks[k];
	const FrameTarget &f = b.frames[task.frame];
	const EmitBuffers &emit = fb.emit;
	const uint32_t t = g - task.triangleBase;
	ClippedPolygon poly;
	poly.count = 3;
	for (int i = 0; i < 3; i++) { poly.v[i].cs = corners[i].cs; poly.v[i].state = 0; poly.v[i].value = 0.0f; }
	poly.v[0].subB = 0.0f; poly.v[0].subC = 0.0f;
	poly.v[1].subB = 1.0f; poly.v[1].subC = 0.0f;
	poly.v[2].subB = 0.0f; poly.v[2].subC = 1.0f;
	for (int s = 0; s < task.camera.clipCount; s++) poly.clip(task.camera.clip[s]);
	uint32_t pieces = 0, base = 0;
	bool first = false;
	for (int n = 0; n < poly.count - 2; n++) {
		const SubVertex *sv[3] = {&poly.v[0], &poly.v[1 + n], &poly.v[2 + n]};
		Corner c[3];
		float subB[3], subC[3];
		for (int i = 0; i < 3; i++) {
			const Projected pr = camera_to_screen(task.camera, sv[i]->cs);
			c[i].cs = pr.cs; c[i].isx = pr.isx; c[i].isy = pr.isy; c[i].fx = pr.flatx; c[i].fy = pr.flaty;
			subB[i] = task.depthOnly ? 0.0f : sv[i]->subB;
			subC[i] = task.depthOnly ? 0.0f : sv[i]->subC;
		}
		Command m;
		if (!make_command(f, c, fb.errorFlag, m)) continue;
		uint64_t slot = g;
		if (pieces == 1) { // extra slots for this piece and all that can follow it
			const uint32_t taken = (uint32_t)(poly.count - 2 - n);
			base = atomicAdd(&emit.counters[EMIT_EXTRAS], taken);
			emit.extraBase[g] = base;
			for (uint32_t i = 0; i < taken; i++)
				if ((uint64_t)b.totalTriangles + base + i < emit.capacity) emit.drawn[b.totalTriangles + base + i] = 0;
		}
		if (pieces > 0) {
			slot = (uint64_t)b.totalTriangles + base + (pieces - 1);
			if (slot < emit.capacity) emit.extraIds[base + (pieces - 1)] = (g << 3) | pieces;
		}
		pieces++;
		if (slot >= emit.capacity) {
			atomicOr(fb.errorFlag, ERROR_RECORD_OVERFLOW);
			continue;
		}
		if (pieces == 1) first = true;
		store_command(b, fb, task, k, f, t, m, subB, subC, (uint32_t)slot);
	}
	return first;
}

// One thread per fan triangle (renderTriangleFromData, renderCore.cpp:220-341, 400-443).  The record
// of triangle g goes to slot g and is numbered 8 * g; further pieces of a clipped triangle go to
// extra slots as numbers 8 * g + 1 .. 8 * g + 6 (record_slot), so that record numbers grow in
// submission order wherever the records lie, and nothing has to be counted and scanned before they
// can be written.  `drawn` tells per slot whether there is a record, over how many tiles and rows; a record
// over at most four tiles takes its place in their lists at once (what the atomic on the list's cursor
// returns).  The rows are placed by the launch behind it (rows_place_kernel).
// This pass takes the place of a counting pass over the same triangles, two scans (of the
// triangles' records and of the records' rows) and the atomics of the list-filling pass:
// a terrain frame of 522,242 triangles went from 304 to 290 us, 64 views of 50,000 triangles (forward,
// loss and adjoint) from 960 to 938 us, a frame of 400 triangles (64x64) from 114 to 107 us with 7 launches
// less.  It is bound by the latency of its gathers, so four blocks of 256 per SM with a few spilled
// registers beat half as many with none.  Counters that every warp adds to are kept out of it: an
// atomic on one address takes 1.6 to 1.9 ns, and with one per warp of 32 triangles (for a list of the
// drawn records and their rows) it took
// exactly that time per warp. Without them: terrain 48 -> 33 us of the setup, the 64 views 162 -> 120 us.
static const uint32_t EMIT_THREADS = 256;

__global__ void __launch_bounds__(EMIT_THREADS, 1024 / EMIT_THREADS) setup_emit_kernel(BatchParams b, FrameBuffers fb) {
	chain_enter();
	for (uint32_t g = blockIdx.x * EMIT_THREADS + threadIdx.x; g < b.totalTriangles; g += gridDim.x * EMIT_THREADS) {
		const uint32_t k = (uint32_t)find_segment(b.taskTriangleBase, b.taskCount, g);
		const TaskParams &task = b.tasks[k];
		const FrameTarget &f = b.frames[task.frame];
		Corner c[3];
		bool whole, drawn = false;
		if (load_triangle(task, g - task.triangleBase, fb.points, c, &whole) && (f.color != nullptr || f.depth != nullptr)) {
			Command m;
			if (!whole) {
				Corner copy[3] = {c[0], c[1], c[2]};
				drawn = emit_clipped(b, fb, g, k, copy);
			} else if (make_command(f, c, fb.errorFlag, m)) {
				drawn = true;
				const float one = task.depthOnly ? 0.0f : 1.0f; // depth only: no weights
				const float subB[3] = {0.0f, one, 0.0f}, subC[3] = {0.0f, 0.0f, one};
				store_command(b, fb, task, k, f, g - task.triangleBase, m, subB, subC, g);
			}
		}
		if (!drawn) fb.emit.drawn[g] = 0;
	}
}

void launch_setup_emit(const BatchParams &b, const FrameBuffers &fb, cudaStream_t stream) {
	if (b.totalTriangles == 0) return;
	COUNT_LAUNCH();
	launch_chained(setup_emit_kernel, grid_for(b.totalTriangles, EMIT_THREADS), EMIT_THREADS, stream, b, fb);
}

// One thread per cell of the grid: the cell's run of the top pixel row of its cell row.  The
// reference's runs are [0, 15) for the first cell and [16 g - 1, 16 g + 15) after it, cut at the
// image's width; perspective depth holds 1 / distance, orthogonal depth the distance itself.
__global__ void occlusion_top_rows_kernel(float *grid, int32_t gridWidth, int32_t gridHeight, int32_t gridStride,
                                          const float *__restrict__ depth, int32_t depthStride, int32_t width, int32_t perspective) {
	const int32_t i = blockIdx.x * blockDim.x + threadIdx.x;
	if (i >= gridWidth * gridHeight) return;
	const int32_t gx = i % gridWidth, gy = i / gridWidth;
	const float *row = depth + (size_t)(gy * OCCLUSION_CELL) * depthStride;
	const int32_t start = gx == 0 ? 0 : gx * OCCLUSION_CELL - 1;
	int32_t end = gx * OCCLUSION_CELL + OCCLUSION_CELL - 1;
	if (end >= width) end = width;
	float value;
	if (perspective) {
		float maxInv = __int_as_float(0x7F800000);
		for (int32_t x = start; x < end; x++) if (row[x] < maxInv) maxInv = row[x];
		value = __fdiv_rn(1.0f, maxInv);
	} else {
		value = 0.0f;
		for (int32_t x = start; x < end; x++) if (row[x] > value) value = row[x];
	}
	float &cell = grid[(size_t)gy * gridStride + gx];
	if (value < cell) cell = value;
}

void launch_occlusion_top_rows(float *grid, int32_t gridWidth, int32_t gridHeight, int32_t gridStride, const float *depth,
                               int32_t depthStride, int32_t width, bool perspective, cudaStream_t stream) {
	const int32_t cells = gridWidth * gridHeight;
	if (cells <= 0) return;
	COUNT_LAUNCH();
	occlusion_top_rows_kernel<<<(cells + 127) / 128, 128, 0, stream>>>(grid, gridWidth, gridHeight, gridStride, depth, depthStride,
	                                                                 width, perspective ? 1 : 0);
}

// ------------------------------------------------------------------ scan

// Exclusive scan in two launches and no host round trip: the first writes one sum per chunk of
// SCAN_CHUNK values, the second gives every chunk the sum of the chunk sums before it (read by
// the whole block) and scans the chunk through shared memory.  The length may live on the
// device (a count written by an earlier kernel), with `capacity` bounding it for the grid.  With
// `plus` the scan is over in[i] + plus[i].
static const int SCAN_THREADS = 256;
static const int SCAN_PER_THREAD = 16;
static const uint32_t SCAN_CHUNK = SCAN_THREADS * SCAN_PER_THREAD;

__device__ __forceinline__ uint32_t scan_length(uint32_t n, const uint32_t *nDevice, uint32_t capacity) {
	if (!nDevice) return n;
	const uint32_t d = *nDevice;
	return d < capacity ? d : capacity;
}

__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t *shared) {
	for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
	if ((threadIdx.x & 31) == 0) shared[threadIdx.x >> 5] = v;
	__syncthreads();
	uint32_t total = 0;
	for (int w = 0; w < SCAN_THREADS / 32; w++) total += shared[w];
	__syncthreads();
	return total;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_reduce_kernel(const uint32_t *__restrict__ in, const uint32_t *__restrict__ plus,
                                                                   uint32_t n, const uint32_t *nDevice,
                                                                   uint32_t capacity, uint32_t *chunkSums) {
	chain_enter();
	__shared__ uint32_t warpSums[SCAN_THREADS / 32];
	const uint32_t count = scan_length(n, nDevice, capacity);
	const uint32_t begin = blockIdx.x * SCAN_CHUNK;
	uint32_t v = 0;
	for (uint32_t i = begin + threadIdx.x; i < begin + SCAN_CHUNK && i < count; i += SCAN_THREADS) v += in[i] + (plus ? plus[i] : 0u);
	const uint32_t total = block_sum(v, warpSums);
	if (threadIdx.x == 0) chunkSums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_apply_kernel(const uint32_t *__restrict__ in, const uint32_t *__restrict__ plus, uint32_t *out,
                                                                  uint32_t n,
                                                                  const uint32_t *nDevice, uint32_t capacity,
                                                                  const uint32_t *__restrict__ chunkSums) {
	chain_enter();
	__shared__ uint32_t values[SCAN_CHUNK + SCAN_CHUNK / 32]; // one padding word per 32: a thread's 16 values hit 16 banks
	__shared__ uint32_t warpSums[SCAN_THREADS / 32];
	const uint32_t count = scan_length(n, nDevice, capacity);
	const uint32_t begin = blockIdx.x * SCAN_CHUNK;
	if (begin > count || (begin == count && count != 0)) return;
	// the sum of every chunk before this one
	uint32_t p = 0;
	for (uint32_t c = threadIdx.x; c < blockIdx.x; c += SCAN_THREADS) p += chunkSums[c];
	const uint32_t prefix = block_sum(p, warpSums);
	for (int k = 0; k < SCAN_PER_THREAD; k++) {
		const uint32_t i = begin + k * SCAN_THREADS + threadIdx.x;
		const uint32_t at = k * SCAN_THREADS + threadIdx.x;
		values[at + (at >> 5)] = i < count ? in[i] + (plus ? plus[i] : 0u) : 0u;
	}
	__syncthreads();
	uint32_t local[SCAN_PER_THREAD];
	uint32_t mine = 0;
	for (int k = 0; k < SCAN_PER_THREAD; k++) {
		local[k] = mine;
		const uint32_t at = threadIdx.x * SCAN_PER_THREAD + k;
		mine += values[at + (at >> 5)];
	}
	// exclusive scan of the threads' sums
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	uint32_t x = mine;
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
		if (lane >= o) x += y;
	}
	if (lane == 31) warpSums[warp] = x;
	__syncthreads();
	uint32_t before = prefix + x - mine;
	for (int w = 0; w < warp; w++) before += warpSums[w];
	for (int k = 0; k < SCAN_PER_THREAD; k++) {
		const uint32_t at = threadIdx.x * SCAN_PER_THREAD + k;
		values[at + (at >> 5)] = before + local[k];
	}
	__syncthreads();
	for (int k = 0; k < SCAN_PER_THREAD; k++) {
		const uint32_t i = begin + k * SCAN_THREADS + threadIdx.x;
		const uint32_t at = k * SCAN_THREADS + threadIdx.x;
		if (i < count) out[i] = values[at + (at >> 5)];
	}
	// the total after the last value, by the block holding it
	if (threadIdx.x == SCAN_THREADS - 1 && (count == 0 || (count - 1) / SCAN_CHUNK == blockIdx.x)) {
		uint32_t total = prefix;
		for (int w = 0; w < SCAN_THREADS / 32; w++) total += warpSums[w];
		out[count] = total;
	}
}

size_t scan_scratch_elems(uint32_t n) { return (size_t)(n / SCAN_CHUNK) + 16; }

static void scan_launch(const uint32_t *in, const uint32_t *plus, uint32_t *out, uint32_t n, const uint32_t *nDevice, uint32_t *scratch, size_t scratchElems,
                        cudaStream_t stream) {
	const uint32_t blocks = n / SCAN_CHUNK + 1; // n = the length, or the capacity bounding a device length
	if (blocks > scratchElems) {
		memset_async(out, 0xFF, sizeof(uint32_t), stream); // never reached: callers size the scratch
		return;
	}
	COUNT_LAUNCH();
	launch_chained(scan_reduce_kernel, blocks, SCAN_THREADS, stream, in, plus, n, nDevice, n, scratch);
	COUNT_LAUNCH();
	launch_chained(scan_apply_kernel, blocks, SCAN_THREADS, stream, in, plus, out, n, nDevice, n, scratch);
}


void launch_scan(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *scratch, size_t scratchElems, cudaStream_t stream) {
	scan_launch(in, nullptr, out, n, nullptr, scratch, scratchElems, stream);
}

void launch_scan_device(const uint32_t *in, uint32_t *out, const uint32_t *nDevice, uint32_t capacity, uint32_t *scratch,
                        size_t scratchElems, cudaStream_t stream) {
	scan_launch(in, nullptr, out, capacity, nDevice, scratch, scratchElems, stream);
}

// The totals a batch's host side reads once its phases ran: records, rows, tile-list entries, the
// error bits and the extra records of clipped triangles, gathered into one small block.  The same
// launch lists the tiles that have entries (one thread per tile, warp-aggregated appends), so that
// the persistent tile kernel pulls only those: frames that are mostly empty (shadow-cube faces) no
// longer send every CTA through thousands of empty tiles.  And it cuts tiles weighing more than
// bins.partWeight into parts, which the tile kernel draws before the other tiles (raster_kernel).
__global__ void gather_totals_kernel(BatchParams b, TotalsSources from, TileBins bins, uint32_t *out) {
	const uint32_t *binOffsets = bins.offsets;
	const uint32_t tiles = b.totalTiles;
	uint4 *tileList = b.tileList;
	uint32_t *tileListCount = b.tileListCount;
	chain_enter();
	if (blockIdx.x == 0 && threadIdx.x == 0) {
		const uint32_t records = *from.records;
		out[0] = records;
		out[1] = from.rowOffsets ? from.rowOffsets[records < from.recordCapacity ? records : from.recordCapacity] : *from.rows;
		out[2] = binOffsets[2 * tiles];
		out[3] = (uint32_t)*from.errorFlag;
		out[TOTALS_EXTRAS] = from.extras ? *from.extras : 0u;
		out[TOTALS_CULLED] = from.culled ? *from.culled : 0u;
	}
	const uint32_t lane = threadIdx.x & 31u;
	if (bins.parts) {
		for (uint32_t first = blockIdx.x * blockDim.x; first < tiles; first += gridDim.x * blockDim.x) { // uniform per block
			const uint32_t t = first + threadIdx.x;
			const uint32_t weight = t < tiles ? part_weight(bins.cursors[2 * t], bins.cursors[2 * t + 1]) : 0u;
			const bool cut = weight > bins.partWeight;
			const uint32_t cutMask = __ballot_sync(0xFFFFFFFFu, cut);
			if (!cutMask) continue;
			// the warp's parts from one atomic
			const uint32_t parts = cut ? (weight + bins.partWeight - 1) / bins.partWeight : 0u;
			uint32_t inclusive = parts;
			for (int o = 1; o < 32; o <<= 1) {
				const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inclusive, o);
				if (lane >= (uint32_t)o) inclusive += v;
			}
			uint32_t at = 0;
			if (lane == 31) at = atomicAdd(bins.partCount, inclusive);
			at = __shfl_sync(0xFFFFFFFFu, at, 31) + inclusive - parts;
			unsigned long long *keys = nullptr;
			int32_t width = 0, columns = 0, rows = 0;
			if (cut) {
				for (uint32_t p = 0; p < parts; p++)
					if (at + p < bins.partCapacity) bins.parts[at + p] = make_uint2(t, p); // always true unless the lists overflowed
				bins.partsDone[t] = 0u;
				const FrameTarget &f = b.frames[find_segment(b.frameTileBase, b.frameCount, t)];
				const int32_t local = (int32_t)(t - f.tileBase), x = (local % f.tilesX) * TILE_W, y = (local / f.tilesX) * TILE_H;
				width = f.width;
				columns = min(TILE_W, width - x);
				rows = min(TILE_H, f.height - y);
				keys = f.keys + (size_t)y * width + x;
			}
			// the parts' keys meet in the key image: zeroed tile by tile, two rows a time
			for (uint32_t left = cutMask; left; left &= left - 1u) {
				const int src = __ffs(left) - 1;
				unsigned long long *to = reinterpret_cast<unsigned long long *>(__shfl_sync(0xFFFFFFFFu, reinterpret_cast<unsigned long long>(keys), src));
				const int32_t stride = __shfl_sync(0xFFFFFFFFu, width, src), c = __shfl_sync(0xFFFFFFFFu, columns, src);
				const int32_t r = __shfl_sync(0xFFFFFFFFu, rows, src);
				const int32_t x = (int32_t)(lane & 15u);
				for (int32_t y = (int32_t)(lane >> 4); y < r; y += 2)
					if (x < c) to[(size_t)y * stride + x] = 0ull;
			}
		}
	}
	if (!tileList) return;
	for (uint32_t first = blockIdx.x * blockDim.x; first < tiles; first += gridDim.x * blockDim.x) { // uniform per block
		const uint32_t t = first + threadIdx.x;
		const bool drawn = t < tiles && binOffsets[2 * t] != binOffsets[2 * t + 2];
		const uint32_t mask = __ballot_sync(0xFFFFFFFFu, drawn);
		if (!mask) continue;
		const uint32_t leader = __ffs(mask) - 1;
		uint32_t at = 0;
		if (lane == leader) at = atomicAdd(tileListCount, (uint32_t)__popc(mask));
		at = __shfl_sync(0xFFFFFFFFu, at, leader);
		if (drawn) // large entries only: depth-only batches have no small ones
			tileList[at + __popc(mask & ((1u << lane) - 1u))] =
				make_uint4(t, binOffsets[2 * t + 1], bins.cursors[2 * t + 1], (uint32_t)find_segment(b.frameTileBase, b.frameCount, t));
	}
}

void launch_gather_totals(const BatchParams &b, const TotalsSources &from, const TileBins &bins, uint32_t *out, cudaStream_t stream) {
	COUNT_LAUNCH();
	const bool tiles = b.tileList || bins.parts;
	launch_chained(gather_totals_kernel, tiles ? grid_for(b.totalTiles, 256) : 1u, tiles ? 256u : 1u, stream, b, from, bins, out);
}

// ------------------------------------------------------------------ row intervals

__global__ void row_count_kernel(const DrawRecord *__restrict__ records, uint32_t capacity, const uint32_t *countDevice,
                                 uint32_t *counts) {
	chain_enter();
	const uint32_t recordCount = device_count(capacity, countDevice);
	for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < recordCount; i += gridDim.x * blockDim.x)
		counts[i] = (uint32_t)(records[i].bottom - records[i].top);
}

void launch_row_offsets(const FrameBuffers &fb, uint32_t recordCount, uint32_t *rowCounts, cudaStream_t stream) {
	if (recordCount > 0) {
		COUNT_LAUNCH();
		launch_chained(row_count_kernel, grid_for(recordCount, 256), 256, stream, fb.records, recordCount, fb.recordCountDevice, rowCounts);
	}
	if (fb.recordCountDevice)
		launch_scan_device(rowCounts, fb.rowOffsets, fb.recordCountDevice, recordCount, fb.scanScratch, fb.scanScratchElems, stream);
	else
		launch_scan(rowCounts, fb.rowOffsets, recordCount, fb.scanScratch, fb.scanScratchElems, stream);
}

static const int32_t ROWS_STEPPED_MAX = 16; // records of at most this many rows are stepped by one lane each
static_assert(ROWS_STEPPED_MAX == ROW_SEGMENT, "a segment is what one lane steps");

// The row intervals of a warp's 32 records (count 0: none in the lane), stepped exactly
// (row_intervals_stepped: two floor divisions per edge start a segment of rows, then one carry step
// per edge and row).  a, b and c hold the record's corners and bound, out its first row.  When all of them have at most ROWS_STEPPED_MAX rows (dense meshes) each lane steps its
// own record; otherwise the records are cut into segments of up to ROWS_STEPPED_MAX rows that are
// spread over the lanes (a lane finds its record by a search over the warp's prefix sums of
// segment counts and fetches its corners with shuffles), so tall triangles keep every lane busy.
__device__ __noinline__ void step_rows(int4 a, int4 b, int2 c, int32_t count, uint32_t out, uint32_t *rows,
                                          uint32_t rowCapacity, int32_t *errorFlag) {
	const int lane = threadIdx.x & 31;
	const int32_t f0 = a.x, f1 = a.y, f2 = a.z, f3 = a.w, f4 = b.x, f5 = b.y, L = b.z, top = b.w, R = c.x;
	const bool short_ = __all_sync(0xFFFFFFFFu, count <= ROWS_STEPPED_MAX);
	const int32_t segments = short_ ? 1 : (count + ROWS_STEPPED_MAX - 1) / ROWS_STEPPED_MAX;
	int32_t inclusive = segments, total = 32;
	if (!short_) {
		for (int o = 1; o < 32; o <<= 1) {
			const int32_t v = __shfl_up_sync(0xFFFFFFFFu, inclusive, o);
			if (lane >= o) inclusive += v;
		}
		total = __shfl_sync(0xFFFFFFFFu, inclusive, 31);
	}
	for (int32_t base = 0; base < total; base += 32) {
		// this lane's segment: the rows [first, first + rowsHere) of the record held by lane k
		int32_t x0 = f0, y0 = f1, x1 = f2, y1 = f3, x2 = f4, y2 = f5, kTop = top, kL = L, kR = R, kCount = count;
		uint32_t kOut = out;
		int32_t first = 0;
		const int32_t j = base + lane;
		if (!short_) {
			int k = 0; // first lane whose inclusive sum exceeds j
			for (int step = 16; step >= 1; step >>= 1)
				if (__shfl_sync(0xFFFFFFFFu, inclusive, k + step - 1) <= j) k += step;
			const int32_t start = __shfl_sync(0xFFFFFFFFu, inclusive, k) - __shfl_sync(0xFFFFFFFFu, segments, k);
			x0 = __shfl_sync(0xFFFFFFFFu, f0, k); y0 = __shfl_sync(0xFFFFFFFFu, f1, k);
			x1 = __shfl_sync(0xFFFFFFFFu, f2, k); y1 = __shfl_sync(0xFFFFFFFFu, f3, k);
			x2 = __shfl_sync(0xFFFFFFFFu, f4, k); y2 = __shfl_sync(0xFFFFFFFFu, f5, k);
			kTop = __shfl_sync(0xFFFFFFFFu, top, k); kL = __shfl_sync(0xFFFFFFFFu, L, k);
			kR = __shfl_sync(0xFFFFFFFFu, R, k); kCount = __shfl_sync(0xFFFFFFFFu, count, k);
			kOut = __shfl_sync(0xFFFFFFFFu, out, k);
			first = (j - start) * ROWS_STEPPED_MAX;
		}
		if (j >= total) continue;
		const int32_t rowsHere = min(ROWS_STEPPED_MAX, kCount - first);
		if (rowsHere <= 0) continue;
		const bool degenerate = (x0 == x1 && y0 == y1) || (x1 == x2 && y1 == y2) || (x2 == x0 && y2 == y0);
		EdgeStepper st[3];
		if (!degenerate) {
			st[0] = edge_stepper(make_edge(x0, y0, x1, y1), kTop + first);
			st[1] = edge_stepper(make_edge(x1, y1, x2, y2), kTop + first);
			st[2] = edge_stepper(make_edge(x2, y2, x0, y0), kTop + first);
		}
		for (int32_t r = 0; r < rowsHere; r++) {
			int32_t left = kR, right = kL;
			if (!degenerate) {
				left = kL; right = kR;
				edge_step(st[0], kL, kR, left, right);
				edge_step(st[1], kL, kR, left, right);
				edge_step(st[2], kL, kR, left, right);
			}
			const uint32_t at = kOut + (uint32_t)(first + r);
			if (at < rowCapacity) rows[at] = (uint32_t)(left & 0xFFFF) | ((uint32_t)right << 16);
			else atomicOr(errorFlag, ERROR_ROW_OVERFLOW);
		}
	}
}

// The two-pass setup's rows: one lane per record, placed by the scan of their row counts.
__global__ void __launch_bounds__(256, 3) rows_group_kernel(DrawRecord *records, uint32_t capacity, const uint32_t *countDevice,
                                                            const uint32_t *__restrict__ rowOffsets, uint32_t *rows, uint32_t rowCapacity,
                                                            int32_t *errorFlag) {
	chain_enter();
	const uint32_t recordCount = device_count(capacity, countDevice);
	const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
	for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w * 32u < recordCount; w += warps) {
		const uint32_t i = w * 32u + (threadIdx.x & 31u);
		int4 a = make_int4(0, 0, 0, 0), b = a;
		int2 c = make_int2(0, 0);
		uint32_t out = 0;
		if (i < recordCount) {
			a = *reinterpret_cast<const int4 *>(&records[i].flat[0]); // flat[0..3]
			b = *reinterpret_cast<const int4 *>(&records[i].flat[4]); // flat[4..5], left, top
			c = *reinterpret_cast<const int2 *>(&records[i].right);   // right, bottom
			out = rowOffsets[i];
			records[i].rowStart = out;
		}
		step_rows(a, b, c, c.y - b.w, out, rows, rowCapacity, errorFlag);
	}
}

// The one-pass setup's rows.  A block takes PLACE_SLOTS slots at a time, makes a dense list of the
// records among them in shared memory (in a closed mesh half the triangles face away), adds their
// rows up, takes that many with one atomic and writes each record's first one.  With `segments`
// (tall triangles) it lists the segments of ROW_SEGMENT rows for rows_segment_kernel; otherwise it
// computes the rows itself, a warp stepping 32 of the listed records: in 32-bit arithmetic where all are
// small (a 64-bit product or remainder costs several times as much, and there are three edges), with
// step_rows otherwise.  With both, placing and computing the rows of the 1.4 M records of
// 64 views takes 56 to 68 us (computing them alone in 64 bits took 72), and a step of the 64 views went
// from 874 to 845 us, a terrain frame from 281 to 266 us, 4k from 908 to 872 us.
static const uint32_t PLACE_BLOCKS = 4; // per SM
static const uint32_t PLACE_THREADS = 256, PLACE_SLOTS = 4 * PLACE_THREADS;

// Exclusive prefix sums of two values over the block's threads, and their totals.  `sums` holds a pair
// of values per warp.
__device__ __forceinline__ uint2 block_prefix(uint2 v, uint2 *sums, uint2 &total) {
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	uint2 inclusive = v;
	for (int o = 1; o < 32; o <<= 1) {
		const uint32_t x = __shfl_up_sync(0xFFFFFFFFu, inclusive.x, o), y = __shfl_up_sync(0xFFFFFFFFu, inclusive.y, o);
		if (lane >= (uint32_t)o) { inclusive.x += x; inclusive.y += y; }
	}
	if (lane == 31) sums[warp] = inclusive;
	__syncthreads();
	uint2 before = make_uint2(0u, 0u);
	total = before;
	for (uint32_t w = 0; w < PLACE_THREADS / 32; w++) {
		const uint2 s = sums[w];
		if (w < warp) { before.x += s.x; before.y += s.y; }
		total.x += s.x;
		total.y += s.y;
	}
	return make_uint2(before.x + inclusive.x - v.x, before.y + inclusive.y - v.y);
}

__global__ void __launch_bounds__(PLACE_THREADS, PLACE_BLOCKS) rows_place_kernel(DrawRecord *records, uint32_t triangles, EmitBuffers emit,
                                                                                 uint32_t *rows, uint32_t rowCapacity, int32_t *errorFlag) {
	chain_enter();
	__shared__ uint32_t slots[PLACE_SLOTS], starts[PLACE_SLOTS], taken;
	__shared__ uint2 sums[PLACE_THREADS / 32];
	const uint32_t end = min(triangles + emit.counters[EMIT_EXTRAS], emit.capacity);
	for (uint32_t base = blockIdx.x * PLACE_SLOTS; base < end; base += gridDim.x * PLACE_SLOTS) { // uniform per block
		// four slots per thread: their records and rows
		const uint32_t at = base + 4u * threadIdx.x;
		const ushort4 marks = at < end ? *reinterpret_cast<const ushort4 *>(emit.drawn + at) : make_ushort4(0, 0, 0, 0); // (padded)
		const uint32_t mark[4] = {marks.x, marks.y, marks.z, marks.w};
		uint32_t count[4];
		uint2 mine = make_uint2(0u, 0u);
#pragma unroll
		for (uint32_t i = 0; i < 4; i++) {
			count[i] = 0;
			if (at + i >= end || (mark[i] & DRAWN_MASK) == 0u) continue;
			count[i] = 2u * (mark[i] >> DRAWN_BITS);
			if (count[i] == 2u * DRAWN_ROWS_MAX) count[i] = (uint32_t)(records[at + i].bottom - records[at + i].top);
			if (emit.segmentSlots) count[i] = (count[i] + ROW_SEGMENT - 1) / ROW_SEGMENT * ROW_SEGMENT;
			mine.x++;
			mine.y += count[i];
		}
		uint2 total;
		const uint2 place = block_prefix(mine, sums, total);
		const uint32_t n = total.x;
		if (threadIdx.x == 0) {
			taken = total.y ? atomicAdd(&emit.counters[EMIT_ROWS], total.y) : 0u;
			if (n) atomicAdd(&emit.counters[EMIT_DRAWN], n);
			if (taken + total.y > rowCapacity) atomicOr(errorFlag, ERROR_ROW_OVERFLOW);
		}
		__syncthreads();
		uint32_t e = place.x, start = taken + place.y;
#pragma unroll
		for (uint32_t i = 0; i < 4; i++) {
			if (count[i] == 0u) continue; // (a record has two rows at least)
			slots[e] = at + i;
			starts[e] = start;
			records[at + i].rowStart = start;
			if (emit.segmentSlots)
				for (uint32_t s = start / ROW_SEGMENT; s < (start + count[i]) / ROW_SEGMENT && s < rowCapacity / ROW_SEGMENT; s++)
					emit.segmentSlots[s] = at + i;
			e++;
			start += count[i];
		}
		__syncthreads();
		if (emit.segmentSlots) continue;
		for (uint32_t first = threadIdx.x & ~31u; first < n; first += PLACE_THREADS) { // uniform per warp
			const uint32_t e = first + (threadIdx.x & 31u);
			int4 a = make_int4(0, 0, 0, 0), b = a;
			int2 c = make_int2(0, 0);
			uint32_t out = 0;
			if (e < n) {
				const DrawRecord &r = records[slots[e]];
				a = *reinterpret_cast<const int4 *>(&r.flat[0]); // flat[0..3]
				b = *reinterpret_cast<const int4 *>(&r.flat[4]); // flat[4..5], left, top
				c = *reinterpret_cast<const int2 *>(&r.right);   // right, bottom
				out = starts[e];
			}
			const int32_t count = c.y - b.w;
			const int32_t flat[6] = {a.x, a.y, a.z, a.w, b.x, b.y};
			if (!__all_sync(0xFFFFFFFFu, count <= NEAR_ROWS && near_corners(flat, b.z, b.w))) {
				step_rows(a, b, c, count, out, rows, rowCapacity, errorFlag);
				continue;
			}
			// a warp of small triangles: each lane steps its record in 32-bit arithmetic
			const int32_t dx = 256 * b.z, dy = 256 * b.w;
			const bool degenerate = (a.x == a.z && a.y == a.w) || (a.z == b.x && a.w == b.y) || (b.x == a.x && b.y == a.y);
			NearEdge e0 = near_edge(a.x - dx, a.y - dy, a.z - dx, a.w - dy), e1 = near_edge(a.z - dx, a.w - dy, b.x - dx, b.y - dy);
			NearEdge e2 = near_edge(b.x - dx, b.y - dy, a.x - dx, a.y - dy);
			for (int32_t r = 0; r < count; r += 2) { // rows come in pairs
				uint32_t packed[2];
#pragma unroll
				for (int j = 0; j < 2; j++) {
					int32_t left = degenerate ? c.x : b.z, right = degenerate ? b.z : c.x;
					if (!degenerate) {
						near_step(e0, b.z, b.z, c.x, left, right);
						near_step(e1, b.z, b.z, c.x, left, right);
						near_step(e2, b.z, b.z, c.x, left, right);
					}
					packed[j] = (uint32_t)(left & 0xFFFF) | ((uint32_t)right << 16);
				}
				// (past the capacity: the block has set the overflow bit and the frame is redone)
				if (out + (uint32_t)r + 2u <= rowCapacity) *reinterpret_cast<uint2 *>(rows + out + r) = make_uint2(packed[0], packed[1]);
			}
		}
		__syncthreads(); // the lists are done with
	}
}

// The rows of frames of tall triangles: one thread per segment of ROW_SEGMENT rows, whose record
// rows_place_kernel wrote down (segmentSlots) as it placed the rows.  Two floor divisions per edge
// start the segment and each row then steps, so the work is spread evenly whatever the records'
// heights and no thread searches for its record.  A kernel that cut the concatenated rows into
// chunks of 1,024, searched the records of each chunk with one warp and stepped four rows per thread
// took 43 us for the 2.5 M rows of 20,000 random triangles at 800x600; this one takes 17 us.
__global__ void __launch_bounds__(128) rows_segment_kernel(const DrawRecord *__restrict__ records, const uint32_t *__restrict__ segmentSlots,
                                                           const uint32_t *rowTotal, uint32_t rowCapacity, uint32_t *rows) {
	chain_enter();
	const uint32_t total = min(*rowTotal, rowCapacity) / ROW_SEGMENT; // rows past the capacity: the frame is redone
	for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < total; s += gridDim.x * blockDim.x) {
		const DrawRecord &r = records[segmentSlots[s]];
		const int4 a = __ldg(reinterpret_cast<const int4 *>(&r.flat[0]));   // flat[0..3]
		const int4 b = __ldg(reinterpret_cast<const int4 *>(&r.flat[4]));   // flat[4..5], left, top
		const int2 c = __ldg(reinterpret_cast<const int2 *>(&r.right));     // right, bottom
		const int32_t first = (int32_t)(s * ROW_SEGMENT - __ldg(&r.rowStart));
		const int32_t count = min((int32_t)ROW_SEGMENT, c.y - b.w - first);
		const bool degenerate = (a.x == a.z && a.y == a.w) || (a.z == b.x && a.w == b.y) || (b.x == a.x && b.y == a.y);
		EdgeStepper st[3];
		if (!degenerate) {
			st[0] = edge_stepper(make_edge(a.x, a.y, a.z, a.w), b.w + first);
			st[1] = edge_stepper(make_edge(a.z, a.w, b.x, b.y), b.w + first);
			st[2] = edge_stepper(make_edge(b.x, b.y, a.x, a.y), b.w + first);
		}
		uint32_t *out = rows + (size_t)s * ROW_SEGMENT;
		// rows come in pairs (raster bounds cover row pairs)
		for (int32_t k = 0; k < count; k += 2) {
			uint32_t packed[2];
#pragma unroll
			for (int j = 0; j < 2; j++) {
				int32_t left = c.x, right = b.z;
				if (!degenerate) {
					left = b.z; right = c.x;
					edge_step(st[0], b.z, c.x, left, right);
					edge_step(st[1], b.z, c.x, left, right);
					edge_step(st[2], b.z, c.x, left, right);
				}
				packed[j] = (uint32_t)(left & 0xFFFF) | ((uint32_t)right << 16);
			}
			*reinterpret_cast<uint2 *>(out + k) = make_uint2(packed[0], packed[1]);
		}
	}
}

void launch_rows(const FrameBuffers &fb, uint32_t recordCount, cudaStream_t stream) {
	if (recordCount == 0) return;
	COUNT_LAUNCH();
	const uint32_t rowCapacity = fb.rowCapacity ? fb.rowCapacity : 0xFFFFFFFFu;
	if (fb.emit.drawn) {
		launch_chained(rows_place_kernel, grid_for((uint64_t)fb.emit.capacity / 4u + 1u, PLACE_THREADS), PLACE_THREADS, stream, fb.records,
		               fb.emit.triangles, fb.emit, fb.rows, rowCapacity, fb.errorFlag);
		if (!fb.emit.segmentSlots) return;
		COUNT_LAUNCH();
		launch_chained(rows_segment_kernel, grid_for(fb.rowCapacity / ROW_SEGMENT, 128), 128, stream, fb.records, fb.emit.segmentSlots,
		               fb.emit.counters + EMIT_ROWS, rowCapacity, fb.rows);
		return;
	}
	launch_chained(rows_group_kernel, grid_for((uint64_t)((recordCount + 31) / 32) * 32, 256), 256, stream, fb.records, recordCount,
	               fb.recordCountDevice, fb.rowOffsets, fb.rows, rowCapacity, fb.errorFlag);
}

// ------------------------------------------------------------------ binning

// Conservative test of whether any pixel of the tile whose top-left pixel is (px0, py0) can be
// inside the record's row intervals: a pixel (x, y) passes edge i of cutConvexEdge when
//   (128 + 256x - sx)*nx + (128 + 256y - sy)*ny <= threshold      (ITriangle2D.cpp:96-146)
// and that linear function is largest at a corner of any rectangle, so a tile is out when one
// edge rejects all four corners of the tile grown by two pixels (the growth covers the rows
// where the reference's truncating division admits a pixel just outside an edge).
__device__ __forceinline__ bool tile_may_overlap(const DrawRecord &r, int32_t px0, int32_t py0) {
	const int64_t X0 = 128 + 256 * (int64_t)(px0 - 2), X1 = 128 + 256 * (int64_t)(px0 + TILE_W + 1);
	const int64_t Y0 = 128 + 256 * (int64_t)(py0 - 2), Y1 = 128 + 256 * (int64_t)(py0 + TILE_H + 1);
	for (int i = 0; i < 3; i++) {
		const int j = (i + 1) % 3;
		const Edge e = make_edge(r.flat[i * 2], r.flat[i * 2 + 1], r.flat[j * 2], r.flat[j * 2 + 1]);
		const int64_t a = (X0 - e.sx) * e.nx, bb = (X1 - e.sx) * e.nx;
		const int64_t c = (Y0 - e.sy) * e.ny, d = (Y1 - e.sy) * e.ny;
		const int64_t lowest = (a < bb ? a : bb) + (c < d ? c : d);
		if (lowest > e.threshold) return false;
	}
	return true;
}

// The corner test above is exact only when no row of the record makes the reference cast a
// quotient beyond 32 bits (a nearly horizontal edge whose row crossings lie 2^30 pixels away),
// because such a row's interval comes from the wrapped value, not from the edge.
__device__ __forceinline__ bool edge_test_is_exact(const Edge &e, int32_t top, int32_t bottom) {
	if (e.nx == 0) return true;
	const float den = fabsf(i64_to_float(e.nx * 256));
	for (int k = 0; k < 2; k++) {
		const int64_t y = k ? (int64_t)bottom : (int64_t)top;
		const int64_t limit = e.threshold - (128 - e.sx) * e.nx - (128 + 256 * y - e.sy) * e.ny;
		if (fabsf(i64_to_float(limit)) >= 5.0e8f * den) return false;
	}
	return true;
}

__device__ __forceinline__ bool tile_test_is_exact(const DrawRecord &r) {
	for (int i = 0; i < 3; i++) {
		const int j = (i + 1) % 3;
		if (!edge_test_is_exact(make_edge(r.flat[i * 2], r.flat[i * 2 + 1], r.flat[j * 2], r.flat[j * 2 + 1]), r.top, r.bottom)) return false;
	}
	return true;
}

// Counts (FILL = false) or writes (FILL = true) the (tile, record) pairs.  Every tile has two lists,
// slot 2 * tile for the records the tile kernel walks one lane each (small) and slot 2 * tile + 1
// for the ones it walks with a whole warp (large).  Records touching at most 4 tiles are binned by
// their own thread, with the atomics of threads that hit the same slot merged into one; larger
// ones by the whole warp, tested tile by tile.  A list keeps submission order only per warp, which
// the order-free depth keys do not need.
// This is the two-pass setup's binning (its records are stored one after another).
template <bool FILL>
__global__ void bin_kernel(BatchParams b, const DrawRecord *__restrict__ records, uint32_t capacity, const uint32_t *countDevice,
                           TileBins bins, int32_t *errorFlag) {
	chain_enter();
	const uint32_t recordCount = device_count(capacity, countDevice);
	const uint32_t lane = threadIdx.x & 31;
	const uint32_t stride = gridDim.x * blockDim.x;
	for (uint32_t r0 = blockIdx.x * blockDim.x; r0 < recordCount; r0 += stride) {
		const uint32_t r = r0 + threadIdx.x;
		int32_t tx0 = 0, tx1 = -1, ty0 = 0, ty1 = -1, tilesX = 0;
		uint32_t tileBase = 0, large = 1;
		if (r < recordCount) {
			const DrawRecord rec = records[r];
			const FrameTarget &f = b.frames[rec.frame];
			large = (b.depthOnly || !record_is_small(rec, b.smallRows, b.smallWidth)) ? 1u : 0u;
			tilesX = f.tilesX;
			tileBase = f.tileBase;
			tx0 = rec.left >> 4; tx1 = (rec.right - 1) >> 4;
			ty0 = rec.top >> 4; ty1 = (rec.bottom - 1) >> 4;
			if (tx1 >= f.tilesX) tx1 = f.tilesX - 1;
			if (ty1 >= f.tilesY) ty1 = f.tilesY - 1;
		}
		const int32_t w = tx1 - tx0 + 1, h = ty1 - ty0 + 1;
		const int32_t tiles = (w > 0 && h > 0) ? w * h : 0;
		const bool big = tiles > 4;
		for (int32_t i = 0; i < 4; i++) {
			const bool active = !big && i < tiles;
			const uint32_t tile = active ? 2u * (tileBase + (uint32_t)((ty0 + i / w) * tilesX + tx0 + i % w)) + large : 0xFFFFFFFFu;
			const uint32_t peers = __match_any_sync(0xFFFFFFFFu, tile);
			if (active) {
				const uint32_t leader = __ffs(peers) - 1;
				const uint32_t rank = __popc(peers & ((1u << lane) - 1u));
				uint32_t baseSlot = 0;
				if (lane == leader) baseSlot = atomicAdd(FILL ? &bins.cursors[tile] : &bins.counts[tile], (uint32_t)__popc(peers));
				baseSlot = __shfl_sync(peers, baseSlot, leader);
				if (FILL) {
					const uint32_t slot = bins.offsets[tile] + baseSlot + rank;
					if (slot < bins.listCapacity) bins.lists[slot] = r; else atomicOr(errorFlag, ERROR_BIN_OVERFLOW);
				}
			}
		}
		uint32_t bigMask = __ballot_sync(0xFFFFFFFFu, big);
		while (bigMask) {
			const uint32_t src = __ffs(bigMask) - 1;
			bigMask &= bigMask - 1;
			const int32_t bx0 = __shfl_sync(0xFFFFFFFFu, tx0, src), by0 = __shfl_sync(0xFFFFFFFFu, ty0, src);
			const int32_t bw = __shfl_sync(0xFFFFFFFFu, w, src), bt = __shfl_sync(0xFFFFFFFFu, tiles, src);
			const int32_t btx = __shfl_sync(0xFFFFFFFFu, tilesX, src);
			const uint32_t bbase = __shfl_sync(0xFFFFFFFFu, tileBase, src);
			const uint32_t br = __shfl_sync(0xFFFFFFFFu, r, src);
			const uint32_t blarge = __shfl_sync(0xFFFFFFFFu, large, src);
			const DrawRecord rec = records[br];
			const bool exact = tile_test_is_exact(rec);
			for (int32_t i = (int32_t)lane; i < bt; i += 32) {
				const int32_t tx = bx0 + i % bw, ty = by0 + i / bw;
				if (exact && !tile_may_overlap(rec, tx * TILE_W, ty * TILE_H)) continue;
				const uint32_t tile = 2u * (bbase + (uint32_t)(ty * btx + tx)) + blarge;
				uint32_t slot = atomicAdd(FILL ? &bins.cursors[tile] : &bins.counts[tile], 1u);
				if (FILL) {
					slot += bins.offsets[tile];
					if (slot < bins.listCapacity) bins.lists[slot] = br; else atomicOr(errorFlag, ERROR_BIN_OVERFLOW);
				}
			}
		}
	}
}

// Bound on how far a fragment's depth can lie from the record's plane.  The reference accumulates
// depth along rows (start + dx*(x0 + 0.5) + dy*(y + 0.5), then one addition per quad or per pixel),
// so a fragment differs from the plane's value at its centre by at most (3 + steps) roundings of at
// most 2^-24 * M each, where M bounds every partial sum and steps is the length of the row walk;
// this is four times that.
__device__ __forceinline__ float plane_margin(const DrawRecord &r, bool pixelSteps) {
	const float bound = __fadd_rn(__fadd_rn(fabsf(r.start[0]), __fmul_rn(fabsf(r.dx[0]), (float)(abs(r.right) + abs(r.left) + 2))),
	                              __fmul_rn(fabsf(r.dy[0]), (float)(abs(r.bottom) + abs(r.top) + 2)));
	const int32_t steps = (pixelSteps ? (r.right - r.left) : ((r.right - r.left) >> 1)) + 16;
	return __fmul_rn(__fmul_rn(bound, (float)steps), 2.384185791015625e-7f); // 2^-22 per step
}

// Upper word of the best (BEST) or worst key that a fragment of the plane can have over the pixels
// [xa, xb] x [ya, yb]: the plane's extreme over their centres lies at a corner, widened by the
// margin.  Not finite: 0xFFFFFFFF, never culled, or 0, culls nothing.
template <bool BEST>
__device__ __forceinline__ uint32_t plane_hi(float s, float dx, float dy, float margin, int32_t xa, int32_t xb, int32_t ya, int32_t yb,
                                             bool affine) {
	const bool up = BEST ? !affine : affine; // perspective: the largest 1/W wins; orthogonal: the smallest W
	const float px = (float)((dx >= 0.0f) == up ? xb : xa) + 0.5f;
	const float py = (float)((dy >= 0.0f) == up ? yb : ya) + 0.5f;
	const float extreme = __fadd_rn(__fadd_rn(s, __fmul_rn(dx, px)), __fmul_rn(dy, py));
	const float value = up ? __fadd_rn(extreme, margin) : __fsub_rn(extreme, margin);
	if (!isfinite(value) || !isfinite(margin)) return BEST ? 0xFFFFFFFFu : 0u;
	const uint32_t hi = ordered_depth(value);
	return affine ? ~hi : hi;
}

// The records over more than four tiles, which setup_emit_kernel listed.  A block takes BIG_GROUP of
// them at a time.  Four lanes load each record (one per edge, one for the plane), the (record, tile
// row) pairs are dealt to the warps in turn, each lane finds the columns of one row, and the warp's
// lanes share the (record, tile) pairs of its 32 rows evenly: one record spanning a whole frame is
// spread over the block, and no lane is spent on the tiles of a bound that the triangle misses.
//
// The edge test of tile_may_overlap is a linear function of the tile's column and row, so an edge is
// kept as base + row * stepY + column * stepX (the value at the tile's most inside corner less the
// threshold, at most 0 when the edge admits it), and in one row it admits the columns on one side of
// a crossing.  Adding `full`, the function's change from that corner to the opposite one, gives the
// same for the most outside corner: a tile whose grown rectangle passes it for all three edges is
// covered by the record completely (the growth by two pixels also keeps clear of the column where
// the reference's truncating division rejects a pixel that is inside).  The row's value is exact; the
// crossing is a binary32 quotient (four roundings, under 2^-21 of itself) widened by 2^-20 of itself
// and 2^-10 of a tile: towards a tile too many to list, which the exact value at that tile then settles,
// and towards covering one too few.
//
// Culling while binning: the count pass raises a tile's threshold to the worst key (plane_hi) of
// each record that covers it completely and leaves out a large record whose best key does not reach
// the threshold so far.  The fill pass runs when every record has been counted and tests against the
// final threshold, so what it lists was counted, whatever the order; the count is an upper bound that
// differs from run to run.  (The pairs left out are counted apart, for the statistics.)  Every pixel of the tile then holds a better key than a record left out
// could give.  Scenes of large triangles drawn over one another keep a few entries per tile of
// hundreds or thousands: of the 1.07 M entries of 20,000 random triangles at 800x600, which the tile
// kernel fetched and rejected one by one, about 62,000 are listed (frame 375 -> 277 us, a batch of 32 mixed
// frames 10.4 -> 8.7 ms).  With every tile of a bound tested by itself and culling in the fill pass
// only, the batch's two passes took 970 and 940 us; they take 350 and 320 (frame 277 -> 250 us, batch
// 5.73 -> 4.72 ms).
static const int BIG_GROUP = 32;
static const int BIG_WARPS = 8; // warps of a block

struct BigEdge {
	long long base, stepX, stepY, full;
	float recip; // 1 / stepX
	int32_t side; // sign of stepX
};

struct BigRecord {
	BigEdge edge[3];
	float start, dx, dy, margin;
	int32_t left, top, right, bottom;
	uint32_t id, tileBase, large;
	int32_t tx0, tx1, ty0, tilesX, exact, affine, width, height;
	int32_t coverLeft, coverRight; // columns within the record's bounds
	int32_t cullRows; // tile rows from the top in which keys decide (0: none)
};

// One row of tiles of a big record, as its warp's lanes read it.
struct __align__(16) BigRow {
	int32_t shift;   // column of a pair less its number
	uint32_t covers; // first column covered completely, and the last one << 16
	uint32_t place;  // the row, its record in the group << 16, and whether keys decide << 31
	uint32_t tile;   // tile number of column 0
};

// Tile rows of a frame in which the largest key decides every pixel, so that records may be culled:
// none without a depth buffer, and not the bottom one of an odd height, whose last row
// odd_row_kernel replays in submission order (depth-only frames have no such row).
__device__ __forceinline__ int32_t key_decided_rows(const FrameTarget &f, bool depthOnly) {
	if (!f.depth) return 0;
	return (!depthOnly && (f.height & 1)) ? f.tilesY - 1 : f.tilesY;
}

// Columns of the tile row ty that the record may touch (lo..hi) and that it covers (cl..ch).
__device__ __forceinline__ void big_row_columns(const BigRecord &h, int32_t ty, int32_t &lo, int32_t &hi, int32_t &cl, int32_t &ch) {
	lo = h.tx0; hi = h.tx1;
	cl = h.coverLeft; ch = h.coverRight;
	const int32_t py0 = ty * TILE_H;
	if (!h.exact || ty >= h.cullRows || h.top > py0 || h.bottom < min(py0 + TILE_H, h.height)) ch = -1;
	if (!h.exact) return;
#pragma unroll
	for (int e = 0; e < 3; e++) {
		const BigEdge &edge = h.edge[e];
		const long long outer = edge.base + (long long)ty * edge.stepY, inner = outer + edge.full;
		if (edge.side == 0) {
			if (outer > 0) hi = -1;
			if (inner > 0) ch = -1;
			continue;
		}
		const float qo = -__fmul_rn(i64_to_float(outer), edge.recip), qi = -__fmul_rn(i64_to_float(inner), edge.recip);
		const float mo = __fadd_rn(__fmul_rn(fabsf(qo), 9.5367431640625e-7f), 9.765625e-4f);
		const float mi = __fadd_rn(__fmul_rn(fabsf(qi), 9.5367431640625e-7f), 9.765625e-4f);
		if (edge.side > 0) {
			const int32_t x = max(__float2int_rd(__fadd_rn(qo, mo)), -1);
			if (x <= hi) hi = outer + x * edge.stepX > 0 ? x - 1 : x;
			ch = min(ch, __float2int_rd(__fsub_rn(qi, mi)));
		} else {
			const int32_t x = min(__float2int_ru(__fsub_rn(qo, mo)), h.tx1 + 1);
			if (x >= lo) lo = outer + x * edge.stepX > 0 ? x + 1 : x;
			cl = max(cl, __float2int_ru(__fadd_rn(qi, mi)));
		}
	}
}

template <bool FILL>
__device__ __forceinline__ void bin_big(const BatchParams &b, const DrawRecord *__restrict__ records, const TileBins &bins,
                                        const uint32_t *extraIds, int32_t *errorFlag) {
	__shared__ BigRecord held[BIG_GROUP];
	__shared__ BigRow heldRows[BIG_WARPS][32];
	__shared__ int32_t firstRow[BIG_GROUP + 1];
	const uint32_t count = *bins.bigCount;
	const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
	const uint32_t upTo = 0xFFFFFFFFu >> (31u - lane); // this lane and those before
	// two groups per block where that leaves a group 8 to BIG_GROUP records: fewer barriers per record where
	// there are many (32 mixed frames: groups of 8, 16 and 32 take 3.73, 3.58 and 3.52 ms), more blocks at
	// work where there are few (20,000 random triangles: 205, 211 and 213 us)
	const uint32_t group = min(max(count / (gridDim.x * 2u), 8u), (uint32_t)BIG_GROUP);
	uint32_t culled = 0;
	for (uint32_t first = blockIdx.x * group; first < count; first += gridDim.x * group) { // uniform per block
		const uint32_t taken = min(group, count - first);
		if (threadIdx.x < BIG_GROUP * 4) {
			const uint32_t q = threadIdx.x >> 2, role = threadIdx.x & 3u;
			bool wrapped = false; // an edge whose test is not exact
			if (q < taken) {
				BigRecord &h = held[q];
				const uint32_t slot = bins.bigList[first + q];
				const DrawRecord &rec = records[slot];
				if (role < 3u) {
					const uint32_t j = role == 2u ? 0u : role + 1u;
					const Edge e = make_edge(rec.flat[role * 2], rec.flat[role * 2 + 1], rec.flat[j * 2], rec.flat[j * 2 + 1]);
					// the grown rectangle of tile (0, 0): pixel centres -2 .. TILE_W + 1 and -2 .. TILE_H + 1
					const long long x = 128 + 256 * (long long)(e.nx >= 0 ? -2 : TILE_W + 1);
					const long long y = 128 + 256 * (long long)(e.ny >= 0 ? -2 : TILE_H + 1);
					BigEdge &edge = h.edge[role];
					edge.base = (x - e.sx) * e.nx + (y - e.sy) * e.ny - e.threshold;
					edge.stepX = 256 * TILE_W * (long long)e.nx;
					edge.stepY = 256 * TILE_H * (long long)e.ny;
					edge.full = 256 * (TILE_W + 3) * (long long)(e.nx >= 0 ? e.nx : -e.nx) + 256 * (TILE_H + 3) * (long long)(e.ny >= 0 ? e.ny : -e.ny);
					edge.side = e.nx > 0 ? 1 : (e.nx < 0 ? -1 : 0);
					edge.recip = e.nx != 0 ? __fdiv_rn(1.0f, i64_to_float(256 * TILE_W * (long long)e.nx)) : 0.0f;
					wrapped = !edge_test_is_exact(e, rec.top, rec.bottom);
				} else {
					const FrameTarget &f = b.frames[rec.frame];
					h.id = record_id(b, extraIds, slot);
					h.large = (b.depthOnly || !record_is_small(rec, b.smallRows, b.smallWidth)) ? 1u : 0u;
					h.left = rec.left; h.top = rec.top; h.right = rec.right; h.bottom = rec.bottom;
					h.tx0 = rec.left >> 4;
					h.ty0 = rec.top >> 4;
					h.tx1 = min((rec.right - 1) >> 4, f.tilesX - 1);
					h.tilesX = f.tilesX;
					h.tileBase = f.tileBase;
					h.width = f.width;
					h.height = f.height;
					h.affine = f.affine;
					h.coverLeft = (rec.left + TILE_W - 1) >> 4;
					h.coverRight = rec.right >= f.width ? f.tilesX - 1 : (rec.right >> 4) - 1;
					h.cullRows = bins.thresholds ? key_decided_rows(f, b.depthOnly != 0) : 0;
					h.start = rec.start[0]; h.dx = rec.dx[0]; h.dy = rec.dy[0];
					h.margin = plane_margin(rec, b.depthOnly != 0);
				}
			}
			const uint32_t wrappedMask = __ballot_sync(0xFFFFFFFFu, wrapped);
			if (q < taken && role == 3u) held[q].exact = (wrappedMask >> (lane & 28u) & 7u) == 0u ? 1 : 0;
		}
		__syncthreads();
		if (threadIdx.x < 32) { // the group's rows
			int32_t rows = 0;
			if (lane < taken) {
				const BigRecord &h = held[lane];
				const int32_t ty1 = min((h.bottom - 1) >> 4, ((h.height + TILE_H - 1) >> 4) - 1);
				if (h.tx1 >= h.tx0 && ty1 >= h.ty0) rows = ty1 - h.ty0 + 1;
			}
			int32_t inclusive = rows;
			for (int o = 1; o < BIG_GROUP; o <<= 1) {
				const int32_t v = __shfl_up_sync(0xFFFFFFFFu, inclusive, o);
				if ((int)lane >= o) inclusive += v;
			}
			if (lane < BIG_GROUP) firstRow[lane + 1] = inclusive;
			if (lane == 0) firstRow[0] = 0;
		}
		__syncthreads();
		const int32_t totalRows = firstRow[BIG_GROUP];
		for (int32_t item0 = (int32_t)warp; item0 < totalRows; item0 += 32 * BIG_WARPS) { // uniform per warp
			const int32_t item = item0 + (int32_t)lane * BIG_WARPS;
			int32_t lo = 0, hi = -1, cl = 0, ch = -1, ty = 0, q = 0;
			if (item < totalRows) {
				for (int o = BIG_GROUP / 2; o > 0; o >>= 1) // the record: firstRow[q] <= item < firstRow[q + 1]
					if (firstRow[q + o] <= item) q += o;
				ty = held[q].ty0 + item - firstRow[q];
				big_row_columns(held[q], ty, lo, hi, cl, ch);
			}
			const int32_t length = max(hi - lo + 1, 0);
			int32_t inclusive = length;
			for (int o = 1; o < 32; o <<= 1) {
				const int32_t v = __shfl_up_sync(0xFFFFFFFFu, inclusive, o);
				if ((int)lane >= o) inclusive += v;
			}
			const int32_t total = __shfl_sync(0xFFFFFFFFu, inclusive, 31), begin = inclusive - length;
			const uint32_t some = __ballot_sync(0xFFFFFFFFu, length > 0);
			if (length > 0) {
				const BigRecord &h = held[q];
				BigRow row;
				row.shift = lo - begin;
				row.covers = ch >= cl ? (uint32_t)cl | (uint32_t)ch << 16 : 0x0000FFFFu;
				row.place = (uint32_t)ty | (uint32_t)q << 16 | (ty < h.cullRows ? 0x80000000u : 0u);
				row.tile = h.tileBase + (uint32_t)(ty * h.tilesX);
				heldRows[warp][__popc(some & (upTo >> 1))] = row;
			}
			__syncwarp();
			int32_t before = -1; // rows begun so far, less one
			for (int32_t base = 0; base < total; base += 32) {
				// which of the next 32 pairs begin a row
				const uint32_t at = (uint32_t)(begin - base);
				const uint32_t starts = __reduce_or_sync(0xFFFFFFFFu, length > 0 && at < 32u ? 1u << at : 0u);
				const int32_t i = base + (int32_t)lane;
				const int32_t mine = before + __popc(starts & upTo);
				before += __popc(starts);
				if (i >= total) continue;
				const BigRow row = heldRows[warp][mine];
				const BigRecord &h = held[row.place >> 16 & 0x7FFFu];
				const int32_t tx = i + row.shift, py0 = (int32_t)(row.place & 0xFFFFu) * TILE_H, px0 = tx * TILE_W;
				const uint32_t tile = row.tile + (uint32_t)tx, slotOf = 2u * tile + h.large;
				if ((row.place >> 31) && h.large) {
					const uint32_t best =
						plane_hi<true>(h.start, h.dx, h.dy, h.margin, max(px0, h.left), min(px0 + TILE_W, h.right) - 1, max(py0, h.top),
						               min(py0 + TILE_H, h.bottom) - 1, h.affine != 0);
					if (best < bins.thresholds[tile]) {
						culled++;
						continue;
					}
				}
				if (!FILL) {
					atomicAdd(&bins.counts[slotOf], 1u);
					if ((uint32_t)tx >= (row.covers & 0xFFFFu) && (uint32_t)tx <= row.covers >> 16) {
						const uint32_t worst = plane_hi<false>(h.start, h.dx, h.dy, h.margin, px0, min(px0 + TILE_W, h.width) - 1, py0,
						                                       min(py0 + TILE_H, h.height) - 1, h.affine != 0);
						if (worst > bins.thresholds[tile]) atomicMax(&bins.thresholds[tile], worst);
					}
				} else {
					const uint32_t slot = bins.offsets[slotOf] + atomicAdd(&bins.cursors[slotOf], 1u);
					if (slot < bins.listCapacity) bins.lists[slot] = h.id; else atomicOr(errorFlag, ERROR_BIN_OVERFLOW);
				}
			}
			__syncwarp(); // the rows are done with before the next ones are written
		}
		__syncthreads(); // the group is done with before the next one is loaded
	}
	if (!FILL && bins.culled && blockIdx.x * group < count) { // uniform per block: one that had a group
		culled = __reduce_add_sync(0xFFFFFFFFu, culled);
		if (lane == 0) firstRow[warp] = (int32_t)culled;
		__syncthreads();
		if (threadIdx.x == 0) {
			for (int w = 1; w < BIG_WARPS; w++) culled += (uint32_t)firstRow[w];
			if (culled) atomicAdd(bins.culled, culled);
		}
	}
}

__global__ void __launch_bounds__(256) bin_big_kernel(BatchParams b, const DrawRecord *__restrict__ records, TileBins bins,
                                                      const uint32_t *extraIds, int32_t *errorFlag) {
	chain_enter();
	bin_big<false>(b, records, bins, extraIds, errorFlag);
}

// The tile lists once their offsets are known.  A record over at most four tiles took its place in
// each of them in setup_emit_kernel, so listing it is plain stores; the big records, whose places
// follow (the cursors go on), are listed in the same launch.
__global__ void __launch_bounds__(256) bin_fill_kernel(BatchParams b, const DrawRecord *__restrict__ records, TileBins bins, EmitBuffers emit,
                                                       int32_t *errorFlag) {
	chain_enter();
	const uint32_t end = min(b.totalTriangles + emit.counters[EMIT_EXTRAS], emit.capacity);
	for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < end; slot += gridDim.x * blockDim.x) {
		const uint32_t mark = emit.drawn[slot] & DRAWN_MASK;
		if (mark == 0u || mark == DRAWN_BIG) continue;
		const uint32_t tiles = mark - 1u;
		const uint4 head = emit.tileHeads[slot];
		const uint2 more = tiles > 2u ? emit.tileRanks[slot] : make_uint2(0u, 0u);
		const uint32_t id = record_id(b, emit.extraIds, slot);
		const uint32_t tilesX = head.y & 0xFFFFu, w = head.y >> 16;
		const uint32_t rank[4] = {head.z, head.w, more.x, more.y};
#pragma unroll
		for (uint32_t k = 0; k < 4; k++) {
			if (k >= tiles) break;
			const uint32_t row = w == 1u ? k : (w == 2u ? k >> 1 : (k >= w ? 1u : 0u));
			const uint32_t at = bins.offsets[head.x + 2u * (row * tilesX + k - row * w)] + rank[k];
			if (at < bins.listCapacity) bins.lists[at] = id; else atomicOr(errorFlag, ERROR_BIN_OVERFLOW);
		}
	}
	bin_big<true>(b, records, bins, emit.extraIds, errorFlag);
}

void launch_bin_count(const BatchParams &b, const FrameBuffers &fb, uint32_t recordCount, TileBins &bins, cudaStream_t stream) {
	if (fb.emit.drawn) { // the others were counted as they were written
		COUNT_LAUNCH();
		launch_chained(bin_big_kernel, sm_count() * 8, 256, stream, b, fb.records, bins, fb.emit.extraIds, fb.errorFlag);
	} else {
		memset_async(bins.counts, 0, sizeof(uint32_t) * 2 * b.totalTiles, stream);
		if (recordCount > 0) {
			COUNT_LAUNCH();
			launch_chained(bin_kernel<false>, grid_for(recordCount, 256), 256, stream, b, fb.records, recordCount, fb.recordCountDevice, bins,
			               fb.errorFlag);
		}
	}
	scan_launch(bins.counts, fb.emit.drawn ? bins.cursors : nullptr, bins.offsets, 2 * b.totalTiles, nullptr, fb.scanScratch,
	            fb.scanScratchElems, stream);
}

void launch_bin_fill(const BatchParams &b, const FrameBuffers &fb, uint32_t recordCount, TileBins &bins, cudaStream_t stream) {
	if (fb.emit.drawn) {
		COUNT_LAUNCH();
		launch_chained(bin_fill_kernel, sm_count() * 8, 256, stream, b, fb.records, bins, fb.emit, fb.errorFlag);
		return;
	}
	memset_async(bins.cursors, 0, sizeof(uint32_t) * 2 * b.totalTiles, stream);
	if (recordCount > 0) {
		COUNT_LAUNCH();
		launch_chained(bin_kernel<true>, grid_for(recordCount, 256), 256, stream, b, fb.records, recordCount, fb.recordCountDevice, bins,
		               fb.errorFlag);
	}
}

// RgbaMultiply_data and its variant (shader/RgbaMultiply.h:37-58, 110-173) for the fan triangle whose
// triSource entry is `src` (polygon * 2 + fan).
__device__ __forceinline__ void make_shade(const TaskParams &task, int32_t src, ShadeRecord &s) {
	const int32_t p = src >> 1, k = src & 1;
	const int corner[3] = {0, 1 + k, 2 + k};
	float scale = 255.0f;
	if (task.diffuse >= 0) scale = fmul(scale, 1.0f / 255.0f);
	if (task.light >= 0) scale = fmul(scale, 1.0f / 255.0f);
	for (int i = 0; i < 3; i++) {
		const float4 col = *reinterpret_cast<const float4 *>(task.colors + (p * 4 + corner[i]) * 4);
		const float4 tc = *reinterpret_cast<const float4 *>(task.texCoords + (p * 4 + corner[i]) * 4);
		s.red[i] = fmul(col.x, scale); s.green[i] = fmul(col.y, scale);
		s.blue[i] = fmul(col.z, scale); s.alpha[i] = fmul(col.w, scale);
		s.u1[i] = tc.x; s.v1[i] = tc.y; s.u2[i] = tc.z; s.v2[i] = tc.w;
	}
	bool fade = !(almost_same3(s.red) && almost_same3(s.green) && almost_same3(s.blue) && almost_same3(s.alpha));
	bool colorless = almost_one3(s.red) && almost_one3(s.green) && almost_one3(s.blue) && almost_one3(s.alpha);
	const bool hasDiffuse = task.diffuse >= 0, hasLight = task.light >= 0;
	if (fade || (hasDiffuse == hasLight)) colorless = false;
	s.flags = (hasDiffuse ? SHADE_DIFFUSE : 0u) | (hasLight ? SHADE_LIGHT : 0u) | (fade ? SHADE_VERTEX_FADE : 0u) |
	          (colorless ? SHADE_COLORLESS : 0u) | (task.filter == 1 ? SHADE_ALPHA_FILTER : 0u);
	s.diffuse = task.diffuse;
	s.light = task.light;
}

// ------------------------------------------------------------------ tiles

// Depth test of one fragment against the tile's shared keys.
__device__ __forceinline__ void tile_fragment(unsigned long long *keys, const float *initialDepth, uint32_t *coverage,
                                              bool counting, int pix, float z, uint32_t record, bool depthTest,
                                              bool affine, uint32_t &fragments) {
	fragments++;
	if (counting) atomicAdd(&coverage[pix], 1u);
	const bool pass = !depthTest || (affine ? (z < initialDepth[pix]) : (z > initialDepth[pix]));
	if (pass) {
		const unsigned long long key = make_key(z, record, depthTest, affine);
		if (key > keys[pix]) atomicMax(&keys[pix], key);
	}
}

// Early depth culling.  A fragment can only change a pixel when its key beats the pixel's key
// and its depth passes the test against the initial depth buffer.  In key order (the upper 32
// bits of make_key) the pixel therefore has a threshold max(key hi, initial depth hi), and a
// record whose best key hi anywhere in the tile is below the smallest threshold of the tile's
// pixels cannot change the tile.  Keys only grow while a tile is drawn, so a threshold read
// early (or read while other warps write) is smaller than the true one: culling stays safe.

// Smallest threshold over the tile's pixels inside the frame, reduced over the warp.
__device__ __forceinline__ uint32_t warp_tile_threshold(const unsigned long long *keys, const float *initialDepth, int lane,
                                                        int32_t validW, int32_t validH, bool affine) {
	uint32_t m = 0xFFFFFFFFu;
#pragma unroll
	for (int k = 0; k < TILE_W * TILE_H / 32; k++) {
		const int p = lane + 32 * k;
		const int row = p >> 4, col = p & 15;
		if (col < validW && row < validH) {
			const int at = row * TILE_STRIDE + col;
			const uint32_t keyHi = (uint32_t)(keys[at] >> 32);
			uint32_t initialHi = ordered_depth(initialDepth[at]);
			if (affine) initialHi = ~initialHi;
			m = min(m, max(keyHi, initialHi));
		}
	}
	return __reduce_min_sync(0xFFFFFFFFu, m);
}

// Largest key hi any fragment of the record can have inside the tile (plane_hi over the pixels of
// the tile and the record's bound).  Returns 0xFFFFFFFF (never culled) for non-finite planes.
__device__ __forceinline__ uint32_t record_best_hi(const DrawRecord &r, int32_t tx0, int32_t ty0, bool affine, bool pixelSteps) {
	return plane_hi<true>(r.start[0], r.dx[0], r.dy[0], plane_margin(r, pixelSteps), max(tx0, r.left), min(tx0 + TILE_W, r.right) - 1,
	                      max(ty0, r.top), min(ty0 + TILE_H, r.bottom) - 1, affine);
}

// Lane `lane` of the record's quad at (x, y1), shaded and written to pixel (px, py): the
// reference's running sums of the quad (quad_lanes), the vertex weights, RgbaMultiply and the
// packed colour and depth.
__device__ __forceinline__ void write_lane(const BatchParams &b, const FrameTarget &f, const DrawRecord &r, const RowPair &pair,
                                           int32_t y1, int32_t x, int lane, int32_t px, int32_t py, bool affine) {
	float w[3][4];
	const int components = f.color ? 3 : 1;
	for (int c = 0; c < components; c++) quad_lanes(r.start[c], r.dx[c], r.dy[c], pair, y1, x, w[c]);
	const float depthValue = (lane == 0) ? w[0][0] : (lane == 1) ? w[0][1] : (lane == 2) ? w[0][2] : w[0][3];
	if (f.color) {
		float wa[4], wb[4], wc[4];
		lane_weights(w, affine, wa, wb, wc);
		ShadeRecord shade;
		make_shade(b.tasks[r.task], r.source, shade);
		float rgba[4];
		shade_lane_inline(shade, b.textures, wa, wb, wc, lane, rgba);
		f.color[(size_t)py * f.colorStride + px] = pack_saturated(rgba, f.packOrder);
	}
	if (f.depth) f.depth[(size_t)py * f.depthStride + px] = depthValue;
}

// The depth model_renderDepth leaves at (px, py) when record ri wins the pixel: the reference's
// 1 x 1 walk from its row's left end (executeTriangleDrawingDepth, renderCore.cpp:343-387).
__device__ __forceinline__ float depth_walk_value(const BatchParams &b, const DrawRecord *__restrict__ records,
                                                  const uint32_t *__restrict__ rows, uint32_t ri, int32_t px, int32_t py) {
	const DrawRecord r = records[record_slot(b, ri)];
	int32_t left, right;
	unpack_row(rows[r.rowStart + (uint32_t)(py - r.top)], left, right);
	const float value = fadd(fadd(r.start[0], fmul(r.dx[0], (float)left + 0.5f)), fmul(r.dy[0], (float)py + 0.5f));
	return chain_add(value, r.dx[0], px - left);
}

// The depth of a depth-only winner from its key: the key's upper word is the ordered bits of the
// very value the walk wrote (make_key), so it decodes to that value, except that +0 and -0 share
// one key word; that word is walked again.
__device__ __forceinline__ float depth_from_key(const BatchParams &b, unsigned long long key, bool affine,
                                                const DrawRecord *__restrict__ records, const uint32_t *__restrict__ rows,
                                                int32_t px, int32_t py) {
	uint32_t hi = (uint32_t)(key >> 32);
	if (affine) hi = ~hi;
	if (hi == 0x80000000u) return depth_walk_value(b, records, rows, key_record(key, true), px, py);
	return bitsf((hi & 0x80000000u) ? (hi & 0x7FFFFFFFu) : ~hi);
}

// The winner of one pixel, shaded and written: the reference's running sums of its quad
// (quad_lanes), the vertex weights, RgbaMultiply and the packed colour and depth.  On the last row
// of an odd-height target the depth-tested pixels are left to odd_row_kernel (their result depends
// on the order of the triangles); without a depth buffer the last triangle drawn wins there as
// anywhere, with its lower lane's value where the pixel lies in its run of full quads.
__device__ __forceinline__ void resolve_pixel(const BatchParams &b, const FrameTarget &f, const DrawRecord *__restrict__ records,
                                              const uint32_t *__restrict__ rows, int32_t px, int32_t py, unsigned long long key) {
	const bool depthTest = f.depth != nullptr, affine = f.affine != 0;
	const bool oddRow = odd_last_row(py, f.height);
	if (oddRow && depthTest) return;
	const DrawRecord r = records[record_slot(b, key_record(key, depthTest))];
	const int32_t y1 = py & ~1, x = px & ~1;
	const RowPair pair = record_row_pair(r, rows, y1, f.height);
	const int lane4 = ((py & 1) << 1) | (px & 1) | ((oddRow && full_quad(pair, x)) ? 2 : 0);
	write_lane(b, f, r, pair, y1, x, lane4, px, py, affine);
}

// The winners of the eight quads that a warp holds (lanes 4q..4q+3 the positions of quad q), shaded and
// written; the values are those of resolve_pixel.  A pixel's mip level needs the vertex weights of
// three positions of its quad besides its own.  Far from a triangle's left end the running sums are
// most of what a pixel costs (up to 18 chains of additions when one lane evaluates its whole quad),
// so there the quad's lanes work together: in each round they take one winner of their quad, every
// lane evaluates the sums (quad_lane, up to 6 chains) and weights of its own position for it, and the
// pixels with that winner collect the positions' weights by shuffles.  There are as many rounds as
// the warp's most divided quad has winners.  One round is always the better way; of several, only
// where the tile has large triangles (largeCount) and a pixel of the warp lies LONG_CHAIN from its
// triangle's left bound: in meshes of small triangles the chains are short and the rounds' own work
// costs more than they save.
// 20,000 random triangles at 800x600: 228 us when every divided quad's pixels go alone, 204 with
// rounds; 32 mixed frames 4.03 and 3.55 ms.  Limits of 16, 32, 64 and 128 pixels: the batch 3.59, 3.59,
// 3.64 and 3.73 ms, the random triangles 206, 203, 210 and 216 us.
// `key` 0: nothing to write.  All 32 lanes call it.
static const int LONG_CHAIN = 32; // pixels from the record's left bound

__device__ __forceinline__ void resolve_quads(const BatchParams &b, const FrameTarget &f, const DrawRecord *__restrict__ records,
                                              const uint32_t *__restrict__ rows, int32_t px, int32_t py, unsigned long long key,
                                              const uint32_t *largeCount) {
	const bool depthTest = f.depth != nullptr, affine = f.affine != 0;
	const bool oddRow = odd_last_row(py, f.height);
	const int lane = (int)(threadIdx.x & 31u), base = lane & ~3;
	const bool mine = key != 0ull && !(oddRow && depthTest); // that row's depth-tested pixels are odd_row_kernel's
	const uint32_t winner = mine ? key_record(key, depthTest) : 0u;
	const int32_t y1 = py & ~1, x = px & ~1;
	float depthValue = 0.0f;
	float wa[4], wb[4], wc[4]; // of positions 0..2, and of the pixel's own
	const uint32_t drawn = __ballot_sync(0xFFFFFFFFu, mine);
	bool first = mine; // no earlier position of the quad has the pixel's winner
#pragma unroll
	for (int l = 1; l < 4; l++) {
		const int other = lane ^ l;
		const uint32_t theirs = __shfl_sync(0xFFFFFFFFu, winner, other);
		if (other < lane && (drawn >> other & 1u) && theirs == winner) first = false;
	}
	const int winners = __popc(__ballot_sync(0xFFFFFFFFu, first) >> base & 15u);
	const DrawRecord &r = records[record_slot(b, winner)];
	const uint32_t rounds = __reduce_max_sync(0xFFFFFFFFu, (uint32_t)winners);
	const bool distant = rounds > 1u && *largeCount != 0u && __any_sync(0xFFFFFFFFu, mine && x - r.left >= LONG_CHAIN);
	if (rounds > 1u && !distant) { // every pixel for itself
		if (!mine) return;
		const RowPair pair = record_row_pair(r, rows, y1, f.height);
		float w[3][4];
		const int components = f.color ? 3 : 1;
		for (int c = 0; c < components; c++) quad_lanes(r.start[c], r.dx[c], r.dy[c], pair, y1, x, w[c]);
		const int at = (lane & 3) | (oddRow && full_quad(pair, x) ? 2 : 0);
		depthValue = pick4(w[0], at);
		if (f.color) {
			lane_weights(w, affine, wa, wb, wc);
			wa[3] = pick4(wa, at); wb[3] = pick4(wb, at); wc[3] = pick4(wc, at);
		}
	} else {
		bool waiting = mine;
		for (;;) {
			const uint32_t pending = __ballot_sync(0xFFFFFFFFu, waiting);
			if (!pending) break;
			const uint32_t quad = pending >> base & 15u;
			const uint32_t round = __shfl_sync(0xFFFFFFFFu, winner, base + (quad ? __ffs(quad) - 1 : 0));
			float z = 0.0f, a = 0.0f, bw = 0.0f, c = 0.0f;
			int at = lane;
			if (quad) {
				const DrawRecord &t = records[record_slot(b, round)];
				const RowPair pair = record_row_pair(t, rows, y1, f.height);
				// without a depth buffer the last row of an odd height holds the lower lanes of full quads
				if (oddRow && full_quad(pair, x)) at |= 2;
				z = quad_lane(t.start[0], t.dx[0], t.dy[0], pair, y1, x, lane & 3);
				if (f.color)
					lane_weight(z, quad_lane(t.start[1], t.dx[1], t.dy[1], pair, y1, x, lane & 3),
					            quad_lane(t.start[2], t.dx[2], t.dy[2], pair, y1, x, lane & 3), affine, a, bw, c);
			}
			const bool taken = waiting && winner == round;
#pragma unroll
			for (int l = 0; l < 4; l++) {
				const int from = l < 3 ? base + l : at;
				const float va = __shfl_sync(0xFFFFFFFFu, a, from), vb = __shfl_sync(0xFFFFFFFFu, bw, from);
				const float vc = __shfl_sync(0xFFFFFFFFu, c, from);
				if (taken) { wa[l] = va; wb[l] = vb; wc[l] = vc; }
			}
			if (taken) {
				depthValue = z;
				waiting = false;
			}
		}
		if (!mine) return;
	}
	if (f.color) {
		ShadeRecord shade;
		make_shade(b.tasks[r.task], r.source, shade);
		float rgba[4];
		shade_lane_inline(shade, b.textures, wa, wb, wc, 3, rgba);
		f.color[(size_t)py * f.colorStride + px] = pack_saturated(rgba, f.packOrder);
	}
	if (f.depth) f.depth[(size_t)py * f.depthStride + px] = depthValue;
}

// Persistent CTAs pull 16x16 tiles of the batch from a device queue.  The binning split every
// tile's list into small and large records.  Both are dealt round-robin over the warps (warp w of
// W takes entries w, w + W, ...): the quads of a warp's 32 small records inside the tile are spread
// over its lanes, one quad each (the reference's running sums at that quad, quad_lanes); large
// records are rasterised by the whole warp, one lane per (row pair, position in the 2x2 quad),
// which evaluates the running sums once at the tile's left edge and then walks on.
// All fragments compete for the tile's shared keys; the winners go to the frame's key image.
// Tiles that nothing covers write nothing: the resolve pass skips them too.
// A tile weighing more than bins.partWeight is drawn in parts by several CTAs at once: each draws its
// share of the lists, merges its keys into the key image with 64-bit maxima (the same order-free
// argument as inside a CTA) and counts itself done; the last part to finish resolves the tile.  No
// CTA waits for another.  Small frames of many triangles have a few tiles with thousands of entries,
// and one CTA walking such a list alone was what the whole batch waited for: 32 frames of up to
// 200,000 triangles at 64x64 to 1024x768 went from 8.7 to 5.9 ms (this launch from 5.5 to 3.0).
static const int SHARED_FRAMES = 256;
static const uint32_t WHOLE_TILE = 0xFFFFFFFFu;

template <bool DEPTH_ONLY_1X1, int THREADS, bool RESOLVE>
__global__ void __launch_bounds__(THREADS, 1024 / THREADS) raster_kernel(BatchParams b, const DrawRecord *__restrict__ records,
                                                                         TileBins bins, const uint32_t *__restrict__ rows) {
	chain_enter();
	constexpr int WARPS = THREADS / 32;
	if (overflowed(b)) return; // the lists or rows are incomplete: the frame is redone
	constexpr int PIXELS = TILE_W * TILE_H / THREADS; // tile pixels owned by each thread
	__shared__ unsigned long long keys[TILE_H * TILE_STRIDE];
	__shared__ float initialDepth[TILE_H * TILE_STRIDE];
	__shared__ uint32_t coverage[TILE_H * TILE_STRIDE];
	__shared__ uint32_t sharedTile, sharedPart, sharedParts, sharedLast;
	__shared__ unsigned long long fragmentSum;
	__shared__ uint32_t frameBases[SHARED_FRAMES]; // the frames' first tiles, for batches of up to SHARED_FRAMES frames
	const int tid = threadIdx.x;
	const int warp = tid >> 5, lane = tid & 31;
	const bool framesShared = b.frameCount <= SHARED_FRAMES;
	if (framesShared)
		for (int i = tid; i < b.frameCount; i += THREADS) frameBases[i] = b.frameTileBase[i];
	const uint32_t listed = (tid == 0 && b.tileList) ? *b.tileListCount : 0u;
	const uint32_t partItems = (tid == 0 && bins.parts) ? *bins.partCount : 0u;
	for (;;) {
		if (tid == 0) {
			// the listed tiles (those with entries), or every tile.  (A ticket taken one tile ahead
			// hides the atomic's round trip but holds a tile back from idle CTAs: slower overall.)
			// The parts of cut tiles come first, so that the longest work starts earliest.
			uint32_t ticket = atomicAdd(b.tileQueue, 1u);
			sharedPart = WHOLE_TILE;
			if (ticket < partItems) {
				const uint2 item = bins.parts[ticket];
				sharedTile = item.x;
				sharedPart = item.y;
			} else {
				ticket -= partItems;
				sharedTile = !b.tileList ? ticket : (ticket < listed ? b.tileList[ticket].x : 0xFFFFFFFFu);
			}
			fragmentSum = 0ull;
		}
		__syncthreads();
		const uint32_t tile = sharedTile;
		if (tile >= b.totalTiles) break;
		uint32_t smallBegin = bins.offsets[2 * tile], largeBegin = bins.offsets[2 * tile + 1];
		uint32_t smallEnd = largeBegin;
		uint32_t end = largeBegin + bins.cursors[2 * tile + 1]; // the large records that binning did not cull
		const uint32_t smalls = smallEnd - smallBegin;
		// nothing to draw, or drawn in parts
		const uint32_t weight = part_weight(smalls, end - largeBegin);
		if (weight == 0u || (sharedPart == WHOLE_TILE && bins.parts && weight > bins.partWeight)) { __syncthreads(); continue; }
		if (sharedPart != WHOLE_TILE) { // (read where it is needed: a register for it costs the resolve spills)
			// this part's share of the small list followed by the large one
			if (tid == 0) sharedParts = (weight + bins.partWeight - 1) / bins.partWeight;
			const uint32_t lo = sharedPart * bins.partWeight, hi = min(lo + bins.partWeight, weight);
			end = largeBegin + (max(hi, smalls) - smalls) / LARGE_WEIGHT;
			largeBegin += (max(lo, smalls) - smalls) / LARGE_WEIGHT;
			smallEnd = smallBegin + min(hi, smalls);
			smallBegin += min(lo, smalls);
		}
		const FrameTarget &f = b.frames[framesShared ? find_segment_shared(frameBases, b.frameCount, tile)
		                                             : find_segment(b.frameTileBase, b.frameCount, tile)];
		const int32_t width = f.width, height = f.height;
		const float *depthImage = f.depth;
		const bool depthTest = depthImage != nullptr;
		const bool affine = f.affine != 0;
		uint32_t *coverageImage = f.coverage;
		const bool counting = coverageImage != nullptr;
		unsigned long long *keyImage = f.keys;
		const int32_t local = (int32_t)(tile - f.tileBase);
		const int32_t tx0 = (local % f.tilesX) * TILE_W, ty0 = (local / f.tilesX) * TILE_H;
		for (int k = 0; k < PIXELS; k++) {
			const int p = tid + k * THREADS;
			const int32_t px = tx0 + (p & 15), py = ty0 + (p >> 4);
			const int me = (p >> 4) * TILE_STRIDE + (p & 15); // the pixel in the padded tile arrays
			initialDepth[me] = (depthTest && px < width && py < height) ? depthImage[(size_t)py * f.depthStride + px] : 0.0f;
			// a part starts from what other parts have already merged: keys only grow
			keys[me] = (sharedPart != WHOLE_TILE && px < width && py < height) ? __ldcg(&keyImage[(size_t)py * width + px]) : 0ull;
			coverage[me] = 0u;
		}
		__syncthreads();

		uint32_t fragments = 0;
		// early depth culling needs a depth buffer and is off while fragments are being counted; the
		// 1x1 depth walk of depth-only frames is cheaper than the culling test itself
		const bool cull = depthTest && b.fragments == nullptr && !DEPTH_ONLY_1X1;
		const int32_t validW = min(TILE_W, width - tx0), validH = min(TILE_H, height - ty0);
		// what every pixel of the tile reaches by the records that cover it (also culls the large records
		// over at most four tiles, which were listed before the thresholds were known)
		const uint32_t tileFloor = (cull && bins.thresholds) ? bins.thresholds[tile] : 0u;
		uint32_t tileMin = 0u; // this warp's view of the tile's depth threshold (0: nothing culled yet)
		// small records: dealt round-robin over the warps (warp w of W takes entries w, w + W, ...).
		// A warp's 32 records are cut into their quads inside the tile, (row pair, quad column)
		// slots of each record's bound, and the slots are spread evenly over the lanes: a lane finds
		// its record by a search over the warp's prefix sums, builds the row pair from the record's
		// two rows and evaluates the reference's running sums at its quad (quad_lanes), so records
		// of different sizes no longer keep lanes idle.  Small records are not culled early: in dense
		// meshes a tile's small list is walked about once per pixel, and the bound test per record
		// cost more than it saved (large records keep the culling; a scene of small triangles with
		// heavy overdraw can send every record down that path with a small bound of 0 x 0).
		for (uint32_t chunk = smallBegin; chunk < smallEnd; chunk += (uint32_t)THREADS) {
			const uint32_t e = chunk + (uint32_t)warp + (uint32_t)WARPS * (uint32_t)lane;
			uint32_t ri = 0, rowOffset = 0;
			int32_t slots = 0, cols = 1, rowStart = 0, colStart = 0, top = 0, colsRecip = 65536;
			float s0 = 0.0f, dx0 = 0.0f, dy0 = 0.0f;
			if (e < smallEnd) {
				ri = bins.lists[e];
				const DrawRecord &r = records[record_slot(b, ri)];
				const int32_t left = r.left, right = r.right;
				top = r.top;
				const int32_t bottom = r.bottom;
				s0 = r.start[0]; dx0 = r.dx[0]; dy0 = r.dy[0];
				rowOffset = r.rowStart;
				rowStart = max(top, ty0);
				const int32_t rowEnd = min(bottom, ty0 + TILE_H);
				colStart = max(left & ~1, tx0);
				const int32_t colEnd = min((right + 1) & ~1, tx0 + TILE_W);
				if (rowEnd > rowStart && colEnd > colStart) {
					cols = (colEnd - colStart) >> 1;
					slots = ((rowEnd - rowStart) >> 1) * cols;
				}
				colsRecip = (65536 + cols - 1) / cols;
			}
			int32_t inclusive = slots;
			for (int o = 1; o < 32; o <<= 1) {
				const int32_t v = __shfl_up_sync(0xFFFFFFFFu, inclusive, o);
				if (lane >= o) inclusive += v;
			}
			const int32_t total = __shfl_sync(0xFFFFFFFFu, inclusive, 31);
			for (int32_t base = 0; base < total; base += 32) {
				const int32_t j = base + lane;
				int k = 0; // the first lane whose inclusive sum exceeds j
				for (int step = 16; step >= 1; step >>= 1)
					if (__shfl_sync(0xFFFFFFFFu, inclusive, k + step - 1) <= j) k += step;
				const int32_t first = __shfl_sync(0xFFFFFFFFu, inclusive, k) - __shfl_sync(0xFFFFFFFFu, slots, k);
				const int32_t kCols = __shfl_sync(0xFFFFFFFFu, cols, k), kRecip = __shfl_sync(0xFFFFFFFFu, colsRecip, k);
				const int32_t kRowStart = __shfl_sync(0xFFFFFFFFu, rowStart, k), kColStart = __shfl_sync(0xFFFFFFFFu, colStart, k);
				const int32_t kTop = __shfl_sync(0xFFFFFFFFu, top, k);
				const uint32_t kRecord = __shfl_sync(0xFFFFFFFFu, ri, k), kRowOffset = __shfl_sync(0xFFFFFFFFu, rowOffset, k);
				const float kS = __shfl_sync(0xFFFFFFFFu, s0, k), kDx = __shfl_sync(0xFFFFFFFFu, dx0, k);
				const float kDy = __shfl_sync(0xFFFFFFFFu, dy0, k);
				if (j >= total) continue;
				const int32_t slot = j - first;
				const int32_t pairIndex = (slot * kRecip) >> 16; // slot / kCols: slots < 64, columns <= 8
				const int32_t y1 = kRowStart + 2 * pairIndex, x = kColStart + 2 * (slot - pairIndex * kCols);
				// the record's rows y1 and y1 + 1 (row offsets are even: one 8-byte load)
				const uint2 two = *reinterpret_cast<const uint2 *>(rows + kRowOffset + (uint32_t)(y1 - kTop));
				int32_t uL, uR, lL, lR;
				unpack_row(two.x, uL, uR);
				unpack_row(two.y, lL, lR);
				const RowPair pair = make_row_pair(uL, uR, lL, lR, y1 + 1, height);
				if (!pair.any || x < pair.obs || x >= pair.obe) continue;
				const bool edge = pair.ibe <= pair.ibs || x < pair.ibs || x >= pair.ibe;
				float v[4];
				quad_lanes(kS, kDx, kDy, pair, y1, x, v);
				for (int l = 0; l < 4; l++) {
					const int32_t xx = x + (l & 1), yy = y1 + (l >> 1);
					if (yy >= height || xx >= width) continue;
					if (!lane_covered(pair, x, edge, l)) continue;
					tile_fragment(keys, initialDepth, coverage, counting, (yy - ty0) * TILE_STRIDE + (xx - tx0), v[l], kRecord,
					              depthTest, affine, fragments);
				}
			}
		}
		// large records: dealt round-robin over the warps (warp w of W takes entries w, w + W, ...),
		// each rasterised by the whole warp
		for (uint32_t chunk = largeBegin; chunk < end; chunk += 32u * WARPS) {
			const uint32_t e = chunk + (uint32_t)warp + (uint32_t)WARPS * (uint32_t)lane;
			const bool valid = e < end;
			const uint32_t myRecord = valid ? bins.lists[e] : 0u;
			bool culled = false;
			uint32_t myBest = 0u;
			if (cull) tileMin = max(tileFloor, warp_tile_threshold(keys, initialDepth, lane, validW, validH, affine));
			if (valid && cull) {
				myBest = record_best_hi(records[record_slot(b, myRecord)], tx0, ty0, affine, DEPTH_ONLY_1X1);
				culled = myBest < tileMin;
			}
			uint32_t largeMask = __ballot_sync(0xFFFFFFFFu, valid && !culled);
			int sinceRefresh = 0;
			while (largeMask) {
				int src = __ffs(largeMask) - 1;
				if (cull) {
					// the threshold only rises while the tile is drawn: refresh it every few records (8: against
					// 4, a batch of 32 mixed frames takes 4.03 ms instead of 4.16; 1 costs more than it culls)
					if (++sinceRefresh == 8) {
						sinceRefresh = 0;
						tileMin = max(tileFloor, warp_tile_threshold(keys, initialDepth, lane, validW, validH, affine));
					}
					// nearest first, until the nearest one left is below the threshold: what is drawn early hides
					// what would have come before it in the list (a frame of 20,000 random triangles took
					// 250 us in the list's order and 231 in this one, 32 mixed frames 4.72 and 4.07 ms)
					const bool left = (largeMask >> lane & 1u) != 0u;
					const uint32_t nearest = __reduce_max_sync(0xFFFFFFFFu, left ? myBest : 0u);
					if (nearest < tileMin) break;
					src = __ffs(__ballot_sync(0xFFFFFFFFu, left && myBest == nearest)) - 1;
				}
				largeMask &= ~(1u << src);
				const uint32_t ri = __shfl_sync(0xFFFFFFFFu, myRecord, src);
				const DrawRecord r = records[record_slot(b, ri)];
				// every lane reads one of the tile's 16 rows (lanes 16..31 repeat 0..15)
				int32_t rowLeft = 0, rowRight = 0;
				const int32_t ry = ty0 + (lane & 15);
				if (ry >= r.top && ry < r.bottom) unpack_row(rows[r.rowStart + (uint32_t)(ry - r.top)], rowLeft, rowRight);
				if (DEPTH_ONLY_1X1) {
					// executeTriangleDrawingDepth (renderCore.cpp:343-387): depth starts at the row's left
					// pixel and grows by dx one pixel at a time.
					if (ry >= r.top && ry < r.bottom && ry < height && rowRight > rowLeft) {
						const int32_t xs = tx0 + (lane >> 4) * 8;
						const int32_t x0 = max(xs, rowLeft), x1 = min(xs + 8, rowRight);
						if (x0 < x1) {
							float value = fadd(fadd(r.start[0], fmul(r.dx[0], (float)rowLeft + 0.5f)), fmul(r.dy[0], (float)ry + 0.5f));
							value = chain_add(value, r.dx[0], x0 - rowLeft);
							for (int32_t x = x0; x < x1; x++) {
								tile_fragment(keys, initialDepth, coverage, counting, (ry - ty0) * TILE_STRIDE + (x - tx0), value, ri, true,
								              affine, fragments);
								value = fadd(value, r.dx[0]);
							}
						}
					}
					continue;
				}
				// lane = (row pair, position in the 2x2 quad); it walks its position across the tile's quads
				const int rp = lane >> 2, pos = lane & 3;
				const int32_t y1 = ty0 + 2 * rp;
				const int32_t uL = __shfl_sync(0xFFFFFFFFu, rowLeft, 2 * rp), uR = __shfl_sync(0xFFFFFFFFu, rowRight, 2 * rp);
				const int32_t lL = __shfl_sync(0xFFFFFFFFu, rowLeft, 2 * rp + 1), lR = __shfl_sync(0xFFFFFFFFu, rowRight, 2 * rp + 1);
				if (y1 < r.top || y1 >= r.bottom) continue;
				const RowPair pair = make_row_pair(uL, uR, lL, lR, y1 + 1, height);
				if (!pair.any) continue;
				const int32_t x0 = max(tx0, pair.obs), x1 = min(tx0 + TILE_W, pair.obe);
				if (x0 >= x1) continue;
				const int32_t yy = y1 + (pos >> 1);
				if (yy >= height) continue;
				const bool odd = (pos & 1) != 0;
				const int32_t rowL = (pos < 2) ? pair.upperLeft : pair.lowerLeft, rowR = (pos < 2) ? pair.upperRight : pair.lowerRight;
				const float dx = r.dx[0], d2 = fmul(dx, 2.0f);
				const float P0 = fadd(fadd(r.start[0], fmul(dx, (float)pair.obs + 0.5f)), fmul(r.dy[0], (float)y1 + 0.5f));
				const float R0 = (pos < 2) ? P0 : fadd(P0, r.dy[0]);
				const bool allEdge = pair.ibe <= pair.ibs;
				const int32_t nL = (pair.ibs - pair.obs) >> 1;
				const float m = fmul(d2, (float)((pair.ibe - pair.ibs) >> 1));
				// state of the reference's running sums at quad x0 (fillerTemplates.h:328-373)
				int region; // 0 left edge, 1 full quads, 2 right edge
				float R, V = 0.0f, Rb = 0.0f;
				if (allEdge || x0 < pair.ibs) {
					region = 0;
					R = chain_add_short(R0, d2, (x0 - pair.obs) >> 1);
				} else {
					Rb = chain_add_short(R0, d2, nL);
					if (x0 < pair.ibe) {
						region = 1;
						R = Rb;
						V = chain_add_short(odd ? fadd(Rb, dx) : Rb, d2, (x0 - pair.ibs) >> 1);
					} else {
						region = 2;
						R = chain_add_short(fadd(Rb, m), d2, (x0 - pair.ibe) >> 1);
					}
				}
				const int pixRow = (yy - ty0) * TILE_STRIDE;
				for (int32_t x = x0; x < x1; x += 2) {
					const int32_t xx = x + (odd ? 1 : 0);
					const float z = (region == 1) ? V : (odd ? fadd(R, dx) : R);
					const bool covered = (region == 1) || (xx >= rowL && xx < rowR);
					if (covered && xx < width)
						tile_fragment(keys, initialDepth, coverage, counting, pixRow + (xx - tx0), z, ri, depthTest, affine, fragments);
					if (region == 0) {
						R = fadd(R, d2);
						if (!allEdge && x + 2 == pair.ibs) { region = 1; Rb = R; V = odd ? fadd(R, dx) : R; }
					} else if (region == 1) {
						V = fadd(V, d2);
						if (x + 2 == pair.ibe) { region = 2; R = fadd(Rb, m); }
					} else {
						R = fadd(R, d2);
					}
				}
			}
		}
		if (b.fragments || b.walked) {
			for (int o = 16; o > 0; o >>= 1) fragments += __shfl_xor_sync(0xFFFFFFFFu, fragments, o);
			if (lane == 0) atomicAdd(&fragmentSum, (unsigned long long)fragments);
		}
		__syncthreads();
		if (sharedPart != WHOLE_TILE) {
			// the part's keys into the key image; the tile's last part goes on with all of them
			for (int k = 0; k < PIXELS; k++) {
				const int p = tid + k * THREADS;
				const int32_t px = tx0 + (p & 15), py = ty0 + (p >> 4);
				if (px >= width || py >= height) continue;
				const int me = (p >> 4) * TILE_STRIDE + (p & 15);
				unsigned long long *merged = &keyImage[(size_t)py * width + px];
				if (keys[me] > __ldcg(merged)) atomicMax(merged, keys[me]);
				if (counting && coverage[me]) atomicAdd(&coverageImage[(size_t)py * width + px], coverage[me]);
			}
			__threadfence();
			__syncthreads();
			if (tid == 0) sharedLast = atomicAdd(&bins.partsDone[sharedTile], 1u) + 1u == sharedParts ? 1u : 0u;
			__syncthreads();
			if (sharedLast) {
				__threadfence();
				for (int k = 0; k < PIXELS; k++) {
					const int p = tid + k * THREADS;
					const int32_t px = tx0 + (p & 15), py = ty0 + (p >> 4);
					if (px < width && py < height) keys[(p >> 4) * TILE_STRIDE + (p & 15)] = __ldcg(&keyImage[(size_t)py * width + px]);
				}
				__syncthreads();
			}
		}
#pragma unroll 1
		for (int k = 0; k < PIXELS && (sharedPart == WHOLE_TILE || sharedLast != 0u); k++) { // one copy of the (inlined) resolve code, not PIXELS
			// quad-major: lanes 4q..4q+3 hold the four pixels of quad q, and a warp holds a 16 x 2 strip
			const int p = tid + k * THREADS, q = p >> 2, l4 = p & 3;
			const int lx = 2 * (q & 7) + (l4 & 1), ly = 2 * (q >> 3) + (l4 >> 1);
			const int32_t px = tx0 + lx, py = ty0 + ly;
			const int me = ly * TILE_STRIDE + lx;
			const bool inside = px < width && py < height;
			const unsigned long long key = inside ? keys[me] : 0ull;
			if (inside) {
				if (counting && sharedPart == WHOLE_TILE) coverageImage[(size_t)py * width + px] += coverage[me]; // zeroed before a frame's first run
				if (!RESOLVE) keyImage[(size_t)py * width + px] = key;
				// model_renderDepth: the winner's depth straight from its key, written by the tile pass itself
				else if (DEPTH_ONLY_1X1 && key != 0ull)
					f.depth[(size_t)py * f.depthStride + px] = depth_from_key(b, key, affine, records, rows, px, py);
			}
			if (!RESOLVE || DEPTH_ONLY_1X1) continue;
			// the tile's winners shaded right away (resolve_pixels_kernel fused into the tile pass)
			if (__any_sync(0xFFFFFFFFu, key != 0ull)) resolve_quads(b, f, records, rows, px, py, key, &bins.cursors[2 * tile + 1]);
		}
		if (tid == 0 && fragmentSum) {
			if (b.fragments) atomicAdd(b.fragments, fragmentSum);
			if (b.walked) atomicAdd(b.walked, fragmentSum);
		}
		__syncthreads();
	}
}

// Depth-only batches (shadow-cube faces, model_renderDepth): one warp per tile.  Lane l owns eight
// pixels of row l / 2 (the left half of the tile for even lanes, the right one for odd), which is how the
// reference's 1 x 1 walk runs along a row, so the tile's keys stay in the lanes' registers: no shared
// memory, no barriers and no atomics.  A lane starts each pixel from the key of the depth already in
// the image with the largest low word, which no record has, so a fragment replaces it exactly when it
// passes the reference's strict test; a NaN in the image is never passed.  What bounds it is the latency
// of a tile's few dependent loads (shadow faces have two or three entries per drawn tile), hence many
// small independent warps, a descriptor per listed tile, the next ticket taken a tile ahead and each
// record's row interval loaded one record ahead.  With a block of 64 threads per tile and keys in
// shared memory the 96 faces of the 1080p light frame took 180 us; they now take 83 us (frame 710 -> 616 us).
// Tiles cut into parts (raster_kernel) meet in the key image as there.
static const int DEPTH_PIXELS = 8; // of one lane
static const int DEPTH_BLOCKS = 8; // of four warps, per SM

__global__ void __launch_bounds__(128) raster_depth_kernel(BatchParams b, const DrawRecord *__restrict__ records, TileBins bins,
                                                           const uint32_t *__restrict__ rows) {
	chain_enter();
	if (overflowed(b)) return;
	const int lane = threadIdx.x & 31;
	const uint32_t partItems = bins.parts ? *bins.partCount : 0u, items = partItems + *b.tileListCount;
	uint32_t walked = 0;
	uint32_t ticket = 0;
	if (lane == 0) ticket = atomicAdd(b.tileQueue, 1u);
	ticket = __shfl_sync(0xFFFFFFFFu, ticket, 0);
	while (ticket < items) { // every condition on the ticket's tile is the same for the whole warp
		uint32_t following = 0;
		if (lane == 0) following = atomicAdd(b.tileQueue, 1u);
		uint32_t part = WHOLE_TILE, parts = 1;
		uint4 item; // tile, first entry, entries, frame
		if (ticket < partItems) {
			const uint2 p = bins.parts[ticket];
			part = p.y;
			item.x = p.x;
			item.y = bins.offsets[2 * p.x + 1];
			item.z = bins.cursors[2 * p.x + 1];
			item.w = (uint32_t)find_segment(b.frameTileBase, b.frameCount, p.x);
			const uint32_t weight = part_weight(0u, item.z);
			parts = (weight + bins.partWeight - 1) / bins.partWeight;
			const uint32_t lo = part * bins.partWeight / LARGE_WEIGHT, hi = min((part + 1) * bins.partWeight, weight) / LARGE_WEIGHT;
			item.y += lo;
			item.z = hi - lo;
		} else {
			item = b.tileList[ticket - partItems];
			if (bins.parts && part_weight(0u, item.z) > bins.partWeight) { // drawn in parts
				ticket = __shfl_sync(0xFFFFFFFFu, following, 0);
				continue;
			}
		}
		const FrameTarget &f = b.frames[item.w];
		const int32_t width = f.width, height = f.height, tilesX = f.tilesX;
		const bool affine = f.affine != 0;
		const int32_t local = (int32_t)(item.x - f.tileBase);
		const int32_t y = (local / tilesX) * TILE_H + (lane >> 1), xs = (local % tilesX) * TILE_W + (lane & 1) * DEPTH_PIXELS;
		float *pixels = f.depth + (size_t)y * f.depthStride + xs; // (used inside the image only)
		const int32_t valid = y < height ? min(DEPTH_PIXELS, width - xs) : 0;
		const bool vector = valid == DEPTH_PIXELS && (reinterpret_cast<unsigned long long>(pixels) & 15ull) == 0ull;
		unsigned long long key[DEPTH_PIXELS];
		{
			float initial[DEPTH_PIXELS];
			if (vector) {
				const float4 a = reinterpret_cast<const float4 *>(pixels)[0], c = reinterpret_cast<const float4 *>(pixels)[1];
				initial[0] = a.x; initial[1] = a.y; initial[2] = a.z; initial[3] = a.w;
				initial[4] = c.x; initial[5] = c.y; initial[6] = c.z; initial[7] = c.w;
			} else {
#pragma unroll
				for (int k = 0; k < DEPTH_PIXELS; k++) initial[k] = k < valid ? pixels[k] : 0.0f;
			}
#pragma unroll
			for (int k = 0; k < DEPTH_PIXELS; k++) {
				uint32_t hi = ordered_depth(initial[k]);
				if (affine) hi = ~hi;
				if (k >= valid || initial[k] != initial[k]) hi = 0xFFFFFFFFu;
				key[k] = ((unsigned long long)hi << 32) | 0xFFFFFFFFull;
			}
		}
		uint32_t drawn = 0; // pixels some record has won
		for (uint32_t first = 0; first < item.z; first += 32u) {
			const uint32_t count = min(32u, item.z - first);
			uint32_t id = 0, rowStart = 0;
			int32_t top = 0, bottom = 0;
			float start = 0.0f, dx = 0.0f, dy = 0.0f;
			if ((uint32_t)lane < count) {
				id = bins.lists[item.y + first + (uint32_t)lane];
				const DrawRecord &r = records[record_slot(b, id)];
				top = r.top; bottom = r.bottom;
				start = r.start[0]; dx = r.dx[0]; dy = r.dy[0];
				rowStart = r.rowStart;
			}
			// this lane's row of record j
			auto interval = [&](uint32_t j) -> uint32_t {
				const int32_t t = __shfl_sync(0xFFFFFFFFu, top, j), o = __shfl_sync(0xFFFFFFFFu, bottom, j);
				const uint32_t at = __shfl_sync(0xFFFFFFFFu, rowStart, j);
				return (valid > 0 && y >= t && y < o) ? rows[at + (uint32_t)(y - t)] : 0u;
			};
			uint32_t ahead = interval(0);
			for (uint32_t j = 0; j < count; j++) {
				const uint32_t packed = ahead;
				if (j + 1 < count) ahead = interval(j + 1);
				const float s = __shfl_sync(0xFFFFFFFFu, start, j), sx = __shfl_sync(0xFFFFFFFFu, dx, j), sy = __shfl_sync(0xFFFFFFFFu, dy, j);
				const uint32_t record = __shfl_sync(0xFFFFFFFFu, id, j);
				int32_t left, right;
				unpack_row(packed, left, right);
				const int32_t x0 = max(xs, left), x1 = min(xs + valid, right);
				if (x0 >= x1) continue;
				walked += (uint32_t)(x1 - x0);
				// executeTriangleDrawingDepth (renderCore.cpp:343-387): depth starts at the row's left pixel
				// and grows by dx one pixel at a time
				float z = fadd(fadd(s, fmul(sx, (float)left + 0.5f)), fmul(sy, (float)y + 0.5f));
				z = chain_add(z, sx, x0 - left);
#pragma unroll
				for (int k = 0; k < DEPTH_PIXELS; k++) {
					if (xs + k < x0 || xs + k >= x1) continue;
					const unsigned long long candidate = make_key(z, record, true, affine);
					if (z == z && candidate > key[k]) {
						key[k] = candidate;
						drawn |= 1u << k;
					}
					z = fadd(z, sx);
				}
			}
		}
		if (part != WHOLE_TILE) {
			// the part's keys into the key image; the tile's last part writes the depths of all of them
			unsigned long long *merged = f.keys + (size_t)y * width + xs;
#pragma unroll
			for (int k = 0; k < DEPTH_PIXELS; k++)
				if ((drawn >> k) & 1u) atomicMax(merged + k, key[k]);
			__threadfence();
			__syncwarp();
			uint32_t done = 0;
			if (lane == 0) done = atomicAdd(&bins.partsDone[item.x], 1u) + 1u;
			done = __shfl_sync(0xFFFFFFFFu, done, 0);
			drawn = 0;
			if (done == parts) {
				__threadfence();
#pragma unroll
				for (int k = 0; k < DEPTH_PIXELS; k++) {
					key[k] = k < valid ? __ldcg(merged + k) : 0ull;
					if (key[k] != 0ull) drawn |= 1u << k;
				}
			}
		}
		if (vector && drawn == 0xFFu) {
			float z[DEPTH_PIXELS];
#pragma unroll
			for (int k = 0; k < DEPTH_PIXELS; k++) z[k] = depth_from_key(b, key[k], affine, records, rows, xs + k, y);
			reinterpret_cast<float4 *>(pixels)[0] = make_float4(z[0], z[1], z[2], z[3]);
			reinterpret_cast<float4 *>(pixels)[1] = make_float4(z[4], z[5], z[6], z[7]);
		} else {
#pragma unroll
			for (int k = 0; k < DEPTH_PIXELS; k++)
				if ((drawn >> k) & 1u) pixels[k] = depth_from_key(b, key[k], affine, records, rows, xs + k, y);
		}
		ticket = __shfl_sync(0xFFFFFFFFu, following, 0);
	}
	if (b.walked) {
		for (int o = 16; o > 0; o >>= 1) walked += __shfl_xor_sync(0xFFFFFFFFu, walked, o);
		if (lane == 0 && walked) atomicAdd(b.walked, (unsigned long long)walked);
	}
}

// One thread per pixel: the winning fragment's quad is re-evaluated exactly (its row pair's
// intervals and the reference's running sums at that quad) and the pixel is shaded.  Used for
// frames of small triangles, where the pixels of a quad mostly have different winners.  One CTA
// of 256 threads per 16x16 tile.
__global__ void __launch_bounds__(256, 4) resolve_pixels_kernel(BatchParams b, const DrawRecord *__restrict__ records,
                                                                const uint32_t *__restrict__ binOffsets, const uint32_t *__restrict__ rows) {
	chain_enter();
	if (overflowed(b)) return;
	const uint32_t tile = blockIdx.x;
	if (binOffsets[2 * tile] == binOffsets[2 * tile + 2]) return;
	const FrameTarget &f = b.frames[find_segment(b.frameTileBase, b.frameCount, tile)];
	const int32_t local = (int32_t)(tile - f.tileBase);
	const int32_t px = (local % f.tilesX) * TILE_W + (threadIdx.x & 15), py = (local / f.tilesX) * TILE_H + (threadIdx.x >> 4);
	if (px >= f.width || py >= f.height) return;
	const unsigned long long key = f.keys[(size_t)py * f.width + px];
	if (key != 0ull) resolve_pixel(b, f, records, rows, px, py, key);
}

// One thread per 2x2 quad: the winners of its pixels are grouped by record, and for each record
// the reference's running sums of the quad (its row pair's intervals and chains), the vertex
// weights, the shader inputs and the mip level are evaluated once for all the pixels it won
// (deferred shading: only winners are shaded).  Used for frames of larger triangles, where a
// quad's pixels mostly share their winner.  One CTA of 64 threads per 16x16 tile.
__global__ void __launch_bounds__(64) resolve_quads_kernel(BatchParams b, const DrawRecord *__restrict__ records,
                                                     const uint32_t *__restrict__ binOffsets, const uint32_t *__restrict__ rows) {
	chain_enter();
	if (overflowed(b)) return;
	const uint32_t tile = blockIdx.x;
	if (binOffsets[2 * tile] == binOffsets[2 * tile + 2]) return;
	const FrameTarget &f = b.frames[find_segment(b.frameTileBase, b.frameCount, tile)];
	const int32_t local = (int32_t)(tile - f.tileBase);
	const int32_t x = (local % f.tilesX) * TILE_W + 2 * (threadIdx.x & 7), y1 = (local / f.tilesX) * TILE_H + 2 * (threadIdx.x >> 3);
	const int32_t width = f.width, height = f.height;
	if (x >= width || y1 >= height) return;
	const bool depthTest = f.depth != nullptr, affine = f.affine != 0;
	uint32_t record[4];
	uint32_t pending = 0;
	for (int l = 0; l < 4; l++) {
		const int32_t px = x + (l & 1), py = y1 + (l >> 1);
		record[l] = 0;
		// depth-tested pixels of an odd-height target's last row: odd_row_kernel
		if (px < width && py < height && !(depthTest && odd_last_row(py, height))) {
			const unsigned long long key = f.keys[(size_t)py * width + px];
			if (key != 0ull) {
				record[l] = key_record(key, depthTest);
				pending |= 1u << l;
			}
		}
	}
	while (pending) {
		const int first = __ffs(pending) - 1;
		const uint32_t ri = record[first];
		uint32_t mask = 0;
		for (int l = first; l < 4; l++)
			if ((pending & (1u << l)) && record[l] == ri) mask |= 1u << l;
		pending &= ~mask;
		const DrawRecord r = records[record_slot(b, ri)];
		const RowPair pair = record_row_pair(r, rows, y1, height);
		float w[3][4];
		const int components = f.color ? 3 : 1;
		for (int c = 0; c < components; c++) quad_lanes(r.start[c], r.dx[c], r.dy[c], pair, y1, x, w[c]);
		if (f.color) {
			float wa[4], wb[4], wc[4];
			lane_weights(w, affine, wa, wb, wc);
			ShadeRecord shade;
			make_shade(b.tasks[r.task], r.source, shade);
			float u[4], v[4];
			const uint32_t mip = quad_diffuse_coordinates(shade, b.textures, wa, wb, wc, u, v);
			// no depth buffer, last row of an odd height: the lower lanes of full quads are written last
			const int lower = (odd_last_row(y1, height) && full_quad(pair, x)) ? 2 : 0;
#pragma unroll
			for (int l = 0; l < 4; l++) {
				if (!(mask & (1u << l))) continue;
				float rgba[4];
				shade_quad_lane(shade, b.textures, wa, wb, wc, u, v, mip, l + lower, rgba);
				f.color[(size_t)(y1 + (l >> 1)) * f.colorStride + x + (l & 1)] = pack_saturated(rgba, f.packOrder);
			}
		}
		if (depthTest)
			for (int l = 0; l < 4; l++)
				if (mask & (1u << l)) f.depth[(size_t)(y1 + (l >> 1)) * f.depthStride + x + (l & 1)] = w[0][l];
	}
}

// ------------------------------------------------------------------ last row of odd heights

// Records one odd_row_kernel window holds (candidates of all 16 columns in shared memory).
static const int ODD_WINDOW = 320;
static const int ODD_SORT = 512; // ODD_WINDOW rounded up to a power of two, for the bitonic sort

// Whether a record can touch row y of the 16 columns from tx0 (its bound, which holds every pixel
// it writes, the lower lanes of the last row's full quads included).
__device__ __forceinline__ bool odd_row_relevant(const BatchParams &b, const DrawRecord *__restrict__ records, uint32_t ri, int32_t y,
                                                 int32_t tx0) {
	const DrawRecord &r = records[record_slot(b, ri)];
	const int4 bound = *reinterpret_cast<const int4 *>(&r.flat[4]); // flat[4], flat[5], left, top
	const int2 rb = *reinterpret_cast<const int2 *>(&r.right);
	return bound.w <= y && rb.y > y && bound.z < tx0 + TILE_W && rb.x > tx0;
}

// Relevant records of the tile's list with index in [lo, hi): counted, and the largest one.
__device__ __forceinline__ void odd_row_count(const BatchParams &b, const DrawRecord *__restrict__ records, const uint32_t *__restrict__ lists,
                                              uint32_t begin, uint32_t end, uint32_t lo, uint32_t hi, int32_t y, int32_t tx0,
                                              uint32_t *count, uint32_t *largest) {
	__syncthreads(); // every thread has read the previous totals
	if (threadIdx.x == 0) { *count = 0u; *largest = 0u; }
	__syncthreads();
	uint32_t n = 0, m = 0;
	for (uint32_t e = begin + threadIdx.x; e < end; e += blockDim.x) {
		const uint32_t ri = lists[e];
		if (ri >= lo && ri < hi && odd_row_relevant(b, records, ri, y, tx0)) { n++; m = max(m, ri); }
	}
	if (n) { atomicAdd(count, n); atomicMax(largest, m); }
	__syncthreads();
}

// The last row of a depth-tested frame of odd height, in submission order (odd_last_row).  Along
// the run of full quads of that row pair a triangle writes its lower lane's value over its upper
// lane's whenever the lower lane passes the depth test, even where the upper lane is nearer, so
// the row's result is not the nearest fragment and the max-key argument of the tile pass does not
// hold: the tile pass leaves the row alone and this kernel replays it.  One CTA per tile of the
// frame's bottom tile row (blockIdx.x the tile column, blockIdx.y the frame).  The tile's records
// that reach the row are taken in windows of at most ODD_WINDOW in increasing record index (the
// submission order); a window is sorted in shared memory, every (record, column) pair evaluates its
// upper and lower candidates in parallel (quad_lanes, as the tile pass does), and one thread per
// column folds them in order with the reference's strict tests: the lower lane if it beats the
// stored depth, else the upper one if it does.  The winner is shaded once at the end.
__global__ void __launch_bounds__(256) odd_row_kernel(BatchParams b, const DrawRecord *__restrict__ records,
                                                      const uint32_t *__restrict__ binOffsets, const uint32_t *__restrict__ lists,
                                                      const uint32_t *__restrict__ rows) {
	chain_enter();
	if (overflowed(b)) return;
	__shared__ uint32_t ids[ODD_SORT];
	__shared__ float2 candidates[ODD_WINDOW * TILE_W];
	__shared__ uint32_t count, largest;
	// every condition that skips a frame or tile is the same for the whole CTA
	for (int32_t frame = (int32_t)blockIdx.y; frame < b.frameCount; frame += (int32_t)gridDim.y) {
		const FrameTarget &f = b.frames[frame];
		if (!(f.height & 1) || f.depth == nullptr || (int32_t)blockIdx.x >= f.tilesX) continue;
		const uint32_t tile = f.tileBase + (uint32_t)((f.tilesY - 1) * f.tilesX) + blockIdx.x;
		const uint32_t begin = binOffsets[2 * tile], end = binOffsets[2 * tile + 2];
		if (begin == end) continue;
		const int32_t y = f.height - 1, tx0 = (int32_t)blockIdx.x * TILE_W, width = f.width;
		const bool affine = f.affine != 0;
		const int tid = threadIdx.x;
		// fold state of column tid (threads 0..15); orthogonal depths are negated so that the nearer
		// one is always the greater (x < y exactly when -x > -y, and NaN fails both)
		const int32_t px = tx0 + tid;
		float stored = 0.0f;
		uint32_t winner = 0xFFFFFFFFu;
		int winnerLower = 0;
		if (tid < TILE_W && px < width) {
			stored = f.depth[(size_t)y * f.depthStride + px];
			if (affine) stored = -stored;
		}
		uint32_t lo = 0;
		for (;;) {
			odd_row_count(b, records, lists, begin, end, lo, 0xFFFFFFFFu, y, tx0, &count, &largest);
			uint32_t n = count;
			if (n == 0) break;
			uint32_t hi = 0xFFFFFFFFu;
			if (n > (uint32_t)ODD_WINDOW) {
				// the largest hi whose window [lo, hi) holds at most ODD_WINDOW records (bisection;
				// [lo, lo + 1) holds at most one, [lo, largest + 1) too many)
				uint32_t good = lo + 1, bad = largest + 1;
				while (bad - good > 1) {
					const uint32_t mid = good + (bad - good) / 2;
					odd_row_count(b, records, lists, begin, end, lo, mid, y, tx0, &count, &largest);
					if (count <= (uint32_t)ODD_WINDOW) good = mid; else bad = mid;
				}
				hi = good;
			}
			// gather the window (any order), then sort it ascending
			__syncthreads();
			if (tid == 0) count = 0u;
			__syncthreads();
			for (uint32_t e = begin + tid; e < end; e += blockDim.x) {
				const uint32_t ri = lists[e];
				if (ri >= lo && ri < hi && odd_row_relevant(b, records, ri, y, tx0)) {
					const uint32_t slot = atomicAdd(&count, 1u);
					if (slot < (uint32_t)ODD_WINDOW) ids[slot] = ri; // always true: the window was sized by the same test
				}
			}
			__syncthreads();
			n = min(count, (uint32_t)ODD_WINDOW);
			for (uint32_t i = n + tid; i < (uint32_t)ODD_SORT; i += blockDim.x) ids[i] = 0xFFFFFFFFu;
			__syncthreads();
			for (uint32_t k = 2; k <= (uint32_t)ODD_SORT; k <<= 1) {
				for (uint32_t j = k >> 1; j > 0; j >>= 1) {
					for (uint32_t i = tid; i < (uint32_t)ODD_SORT; i += blockDim.x) {
						const uint32_t partner = i ^ j;
						if (partner > i) {
							const uint32_t a = ids[i], c = ids[partner];
							const bool ascending = (i & k) == 0;
							if ((a > c) == ascending) { ids[i] = c; ids[partner] = a; }
						}
					}
					__syncthreads();
				}
			}
			// candidates of every (record, column): upper lane where covered, lower lane in full quads
			for (uint32_t p = tid; p < n * TILE_W; p += blockDim.x) {
				const uint32_t j = p >> 4;
				const int32_t cx = tx0 + (int32_t)(p & 15);
				const float none = __int_as_float(0x7FC00000); // quiet NaN: fails every depth test
				float2 cand = make_float2(none, none);
				if (cx < width) {
					const uint32_t ri = ids[j];
					const DrawRecord r = records[record_slot(b, ri)];
					const RowPair pair = record_row_pair(r, rows, y, f.height);
					const int32_t x = cx & ~1;
					if (pair.any && x >= pair.obs && x < pair.obe) {
						float v[4];
						quad_lanes(r.start[0], r.dx[0], r.dy[0], pair, y, x, v);
						const bool full = full_quad(pair, x);
						const int l = cx & 1;
						if (lane_covered(pair, x, !full, l)) cand.x = affine ? -v[l] : v[l];
						if (full) cand.y = affine ? -v[l + 2] : v[l + 2];
					}
				}
				candidates[p] = cand;
			}
			__syncthreads();
			if (tid < TILE_W) {
				for (uint32_t j = 0; j < n; j++) {
					const float2 cand = candidates[j * TILE_W + tid];
					if (cand.y > stored) { stored = cand.y; winner = ids[j]; winnerLower = 1; }
					else if (cand.x > stored) { stored = cand.x; winner = ids[j]; winnerLower = 0; }
				}
			}
			__syncthreads();
			if (hi == 0xFFFFFFFFu) break;
			lo = hi;
		}
		if (tid < TILE_W && px < width && winner != 0xFFFFFFFFu) {
			const DrawRecord r = records[record_slot(b, winner)];
			const int32_t x = px & ~1;
			const RowPair pair = record_row_pair(r, rows, y, f.height);
			write_lane(b, f, r, pair, y, x, (px & 1) + (winnerLower ? 2 : 0), px, y, affine);
		}
		__syncthreads(); // the next frame reuses the shared arrays
	}
}

// ------------------------------------------------------------------ alpha filter

static const uint32_t ALPHA_THREADS = 256, ALPHA_WARPS = ALPHA_THREADS / 32;
static const uint32_t ALPHA_LIST = 2048; // list entries sorted in shared memory at once
static const uint32_t ALPHA_CHUNK = 32;  // records staged at once, one bit of a pixel's mask each
static const uint32_t ALPHA_ITEMS = 8;   // entries of a thread in one step of a long list's sort
static_assert(ALPHA_LIST == ALPHA_WARPS * 256 && ALPHA_THREADS == 256, "a digit's counts of every warp, a digit per thread");

// Sorts the n entries of one tile's list by record number (each is there once), by one CTA: least
// significant digits first, eight bits of the number less the smallest one a pass, from one array to
// the other.  Returns the array that holds the result.  `counts` (ALPHA_LIST words) and `next` (256)
// are shared memory.  The time grows with the entries: 240,000 small triangles over one 16x16 tile are
// sorted and blended in 39 ms, 30,000 in 4.3 ms (taking windows of the list, each found by reading all of
// it some twenty times, took 467 and 7.3 ms).
__device__ __noinline__ const uint32_t *sort_long_list(uint32_t *list, uint32_t *other, uint32_t n, uint32_t *counts, uint32_t *next) {
	const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
	uint32_t *mine = counts + 256u * warp; // this warp's counts
	if (tid < 2u) next[tid] = tid == 0u ? 0xFFFFFFFFu : 0u;
	__syncthreads();
	uint32_t low = 0xFFFFFFFFu, high = 0u;
#pragma unroll 8
	for (uint32_t i = tid; i < n; i += ALPHA_THREADS) {
		low = min(low, list[i]);
		high = max(high, list[i]);
	}
	low = __reduce_min_sync(0xFFFFFFFFu, low);
	high = __reduce_max_sync(0xFFFFFFFFu, high);
	if (lane == 0u) { atomicMin(&next[0], low); atomicMax(&next[1], high); }
	__syncthreads();
	low = next[0];
	const uint32_t range = next[1] - low;
	for (uint32_t shift = 0; shift < 32u && (range >> shift) != 0u; shift += 8u) {
		// the entries of each digit, by every warp for its share, then where each digit begins
		for (uint32_t k = lane; k < 256u; k += 32u) mine[k] = 0u;
		__syncthreads(); // (and `next` is read)
		for (uint32_t base = tid; base < n; base += ALPHA_THREADS * ALPHA_ITEMS) {
			uint32_t id[ALPHA_ITEMS];
#pragma unroll
			for (uint32_t k = 0; k < ALPHA_ITEMS; k++) id[k] = base + ALPHA_THREADS * k < n ? list[base + ALPHA_THREADS * k] : 0u;
#pragma unroll
			for (uint32_t k = 0; k < ALPHA_ITEMS; k++)
				if (base + ALPHA_THREADS * k < n) atomicAdd(&mine[((id[k] - low) >> shift) & 255u], 1u);
		}
		__syncthreads();
		uint32_t total = 0;
		for (uint32_t w = 0; w < ALPHA_WARPS; w++) total += counts[256u * w + tid];
		uint32_t inclusive = total;
		for (int o = 1; o < 32; o <<= 1) {
			const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inclusive, o);
			if (lane >= (uint32_t)o) inclusive += v;
		}
		__syncthreads(); // the counts are read
		if (lane == 31u) counts[warp] = inclusive;
		__syncthreads();
		uint32_t begin = inclusive - total;
		for (uint32_t w = 0; w < warp; w++) begin += counts[w];
		next[tid] = begin;
		__syncthreads();
		// every warp takes 32 * ALPHA_ITEMS consecutive entries a step and ranks them among its entries of
		// the same digit; the warps' counts then give every warp its first place of each digit
		for (uint32_t base = 0; base < n; base += ALPHA_THREADS * ALPHA_ITEMS) {
			const uint32_t first = base + warp * 32u * ALPHA_ITEMS + lane;
			uint32_t id[ALPHA_ITEMS], rank[ALPHA_ITEMS];
			for (uint32_t k = lane; k < 256u; k += 32u) mine[k] = 0u;
			__syncwarp();
#pragma unroll
			for (uint32_t k = 0; k < ALPHA_ITEMS; k++) id[k] = first + 32u * k < n ? list[first + 32u * k] : 0u;
#pragma unroll
			for (uint32_t k = 0; k < ALPHA_ITEMS; k++) {
				const bool valid = first + 32u * k < n;
				const uint32_t digit = ((id[k] - low) >> shift) & 255u;
				const uint32_t peers = __match_any_sync(0xFFFFFFFFu, valid ? digit : 256u);
				const uint32_t before = __popc(peers & ((1u << lane) - 1u));
				const uint32_t earlier = valid ? mine[digit] : 0u;
				rank[k] = earlier + before;
				__syncwarp();
				if (valid && before == 0u) mine[digit] = earlier + __popc(peers);
				__syncwarp();
			}
			__syncthreads();
			uint32_t place = next[tid];
			for (uint32_t w = 0; w < ALPHA_WARPS; w++) {
				const uint32_t count = counts[256u * w + tid];
				counts[256u * w + tid] = place;
				place += count;
			}
			next[tid] = place;
			__syncthreads();
#pragma unroll
			for (uint32_t k = 0; k < ALPHA_ITEMS; k++)
				if (first + 32u * k < n) other[mine[((id[k] - low) >> shift) & 255u] + rank[k]] = id[k];
			__syncwarp(); // the warp's places are read before its next counts
		}
		__syncthreads(); // the pass is written
		uint32_t *sorted = other;
		other = list;
		list = sorted;
	}
	return list;
}

// Alpha-filtered triangles (fillQuadSuper with Filter::Alpha, fillerTemplates.h:160-186, read-only
// depth: fillerTemplates.h:386-441): every covered fragment that passes the depth test blends its
// colour over the pixel, source * (alpha / 255) + target * (1 - alpha / 255), packed with
// saturation after each blend, and writes no depth.  The order matters, so a tile's records are taken
// in submission order, and each pixel's colour stays in a register of its thread.
//
// One CTA of 256 threads per 16x16 tile, a warp holding a 16 x 2 strip as eight quads.  The tile's
// list is sorted by record number (lists are in no order), in shared memory up to ALPHA_LIST entries and
// by sort_long_list beyond.  Records are staged 32 at a time
// with their rows inside the tile and their shader inputs.  Each pixel marks the staged records that
// cover it, and then every quad takes its own marked records one after another: the quads of a warp
// work on different records at the same time, and the four lanes of a quad evaluate one position
// each and share the weights by shuffles.  What bounds it is instruction issue, and most records of a
// tile (small particles) cover a small part of it: when the whole warp walked every record of the
// tile, each lane evaluating the four positions of its quad, a frame of 1,500 particles over a
// 1281x719 image spent 474 us here and 160 us in four global sorting passes before it; it now
// takes 140 us in all (frame 834 -> 358 us).
__global__ void __launch_bounds__(ALPHA_THREADS) alpha_kernel(BatchParams b, const DrawRecord *__restrict__ records, TileBins bins,
                                                    const uint32_t *__restrict__ rows) {
	chain_enter();
	// lists or rows that overflowed (the run is redone), or a coordinate out of range (the call fails): nothing
	// is blended over the image
	if (b.errorFlag && *(volatile const int32_t *)b.errorFlag != 0) return;
	__shared__ uint32_t ids[ALPHA_LIST];
	__shared__ DrawRecord staged[ALPHA_CHUNK];
	__shared__ ShadeRecord shades[ALPHA_CHUNK];
	__shared__ uint32_t stagedRows[ALPHA_CHUNK][TILE_H];
	static_assert(ALPHA_CHUNK * TILE_H >= 256, "sort_long_list's digits");
	const uint32_t tile = blockIdx.x;
	const uint32_t begin = bins.offsets[2 * tile], end = bins.offsets[2 * tile + 2];
	if (begin == end) return; // the same for the whole CTA, as every condition around a barrier below
	const FrameTarget &f = b.frames[find_segment(b.frameTileBase, b.frameCount, tile)];
	if (!f.color) return;
	// the list in submission order, before the pixels take their registers
	const int tid = threadIdx.x;
	const uint32_t n = end - begin;
	const uint32_t *order = ids;
	if (n > ALPHA_LIST) {
		order = sort_long_list(bins.lists + begin, bins.scratch + begin, n, ids, &stagedRows[0][0]);
	} else {
		uint32_t size = 2;
		while (size < n) size <<= 1;
		for (uint32_t i = tid; i < size; i += ALPHA_THREADS) ids[i] = i < n ? bins.lists[begin + i] : 0xFFFFFFFFu;
		__syncthreads();
		for (uint32_t k = 2; k <= size; k <<= 1) {
			for (uint32_t j = k >> 1; j > 0; j >>= 1) {
				for (uint32_t i = tid; i < size; i += ALPHA_THREADS) {
					const uint32_t partner = i ^ j;
					if (partner > i) {
						const uint32_t a = ids[i], c = ids[partner];
						if ((a > c) == ((i & k) == 0)) { ids[i] = c; ids[partner] = a; }
					}
				}
				__syncthreads();
			}
		}
	}
	const int lane = tid & 31, l4 = tid & 3, quadBase = lane & ~3;
	const int32_t local = (int32_t)(tile - f.tileBase), tx0 = (local % f.tilesX) * TILE_W, ty0 = (local / f.tilesX) * TILE_H;
	const int32_t width = f.width, height = f.height, packOrder = f.packOrder;
	const int q = tid >> 2;
	const int32_t x = tx0 + 2 * (q & 7), y1 = ty0 + 2 * (q >> 3), px = x + (l4 & 1), py = y1 + (l4 >> 1);
	const bool inside = px < width && py < height;
	const bool depthTest = f.depth != nullptr, affine = f.affine != 0, oddRow = odd_last_row(y1, height);
	const float stored = (depthTest && inside) ? f.depth[(size_t)py * f.depthStride + px] : 0.0f;
	uint32_t *target = f.color + (size_t)py * f.colorStride + px;
	uint32_t packed = inside ? *target : 0u;
	uint32_t fragments = 0;
	for (uint32_t base = 0; base < n; base += ALPHA_CHUNK) {
		const uint32_t m = min(ALPHA_CHUNK, n - base);
		__syncthreads(); // the chunk before is done with
		for (uint32_t i = tid; i < m * (sizeof(DrawRecord) / 16); i += blockDim.x) {
			const uint32_t j = i / (sizeof(DrawRecord) / 16), w = i % (sizeof(DrawRecord) / 16);
			reinterpret_cast<int4 *>(&staged[j])[w] = reinterpret_cast<const int4 *>(&records[record_slot(b, order[base + j])])[w];
		}
		__syncthreads();
		for (uint32_t i = tid; i < m * TILE_H; i += blockDim.x) {
			const uint32_t j = i / TILE_H, y = i % TILE_H;
			const int32_t py2 = ty0 + (int32_t)y;
			const DrawRecord &r = staged[j];
			stagedRows[j][y] = (py2 >= r.top && py2 < r.bottom) ? rows[r.rowStart + (uint32_t)(py2 - r.top)] : 0u;
		}
		if ((uint32_t)tid < m) make_shade(b.tasks[staged[tid].task], staged[tid].source, shades[tid]);
		__syncthreads();
		uint32_t mine = 0; // the staged records that cover this pixel
		for (uint32_t j = 0; j < m; j++) {
			int32_t left, right;
			unpack_row(stagedRows[j][py - ty0], left, right);
			if (inside && px >= left && px < right) mine |= 1u << j;
		}
		fragments += __popc(mine);
		uint32_t todo = mine | __shfl_xor_sync(0xFFFFFFFFu, mine, 1);
		todo |= __shfl_xor_sync(0xFFFFFFFFu, todo, 2); // the quad's
		for (;;) {
			const unsigned active = __ballot_sync(0xFFFFFFFFu, todo != 0u);
			if (!active) break;
			if (todo == 0u) continue;
			const int j = __ffs(todo) - 1;
			todo &= todo - 1u;
			const DrawRecord &r = staged[j];
			int32_t uL, uR, lL, lR;
			unpack_row(stagedRows[j][y1 - ty0], uL, uR);
			unpack_row(stagedRows[j][y1 - ty0 + 1], lL, lR);
			const RowPair pair = make_row_pair(uL, uR, lL, lR, y1 + 1, height);
			const float z = quad_lane(r.start[0], r.dx[0], r.dy[0], pair, y1, x, l4);
			const bool covered = (mine >> j) & 1u;
			bool draws = covered && (!depthTest || (affine ? (z < stored) : (z > stored)));
			int position = l4;
			if (oddRow) {
				// the lower lane reads the same target colour and is written after the upper one: it
				// decides the pixel when it passes the depth test (odd_last_row)
				const float zl = __shfl_sync(active, z, quadBase + (l4 & 1) + 2);
				if (covered && full_quad(pair, x) && (!depthTest || (affine ? (zl < stored) : (zl > stored)))) {
					draws = true;
					position = (l4 & 1) + 2;
				}
			}
			const unsigned drawing = __ballot_sync(active, draws);
			if (!((drawing >> quadBase) & 15u)) continue; // no pixel of the quad
			unsigned shading = drawing | (drawing >> 1); // every lane of the quads that go on
			shading = (shading | (shading >> 2)) & 0x11111111u;
			shading *= 15u;
			float a, bw, c;
			lane_weight(z, quad_lane(r.start[1], r.dx[1], r.dy[1], pair, y1, x, l4), quad_lane(r.start[2], r.dx[2], r.dy[2], pair, y1, x, l4),
			            affine, a, bw, c);
			float wa[4], wb[4], wc[4];
			for (int l = 0; l < 4; l++) {
				wa[l] = __shfl_sync(shading, a, quadBase + l);
				wb[l] = __shfl_sync(shading, bw, quadBase + l);
				wc[l] = __shfl_sync(shading, c, quadBase + l);
			}
			float rgba[4];
			shade_lane_inline(shades[j], b.textures, wa, wb, wc, position, rgba);
			if (!draws) continue;
			const float opacity = fmul(rgba[3], 1.0f / 255.0f);
			const float keep = fsub(1.0f, opacity);
			float blended[4];
			for (int ch = 0; ch < 4; ch++) {
				const float t = (float)((packed >> pack_shift(packOrder, ch)) & 0xFFu);
				blended[ch] = fadd(fmul(rgba[ch], opacity), fmul(t, keep));
			}
			packed = pack_saturated(blended, packOrder);
		}
	}
	if (inside) {
		*target = packed;
		if (f.coverage) f.coverage[(size_t)py * width + px] += fragments;
	}
	if (b.fragments || b.walked) {
		for (int o = 16; o > 0; o >>= 1) fragments += __shfl_xor_sync(0xFFFFFFFFu, fragments, o);
		if (lane == 0 && fragments) {
			if (b.fragments) atomicAdd(b.fragments, (unsigned long long)fragments);
			if (b.walked) atomicAdd(b.walked, (unsigned long long)fragments);
		}
	}
}

void launch_alpha(const BatchParams &b, const FrameBuffers &fb, const TileBins &bins, cudaStream_t stream) {
	if (b.totalTiles == 0) return;
	COUNT_LAUNCH();
	launch_chained(alpha_kernel, b.totalTiles, ALPHA_THREADS, stream, b, fb.records, bins, fb.rows);
}

void launch_odd_rows(const BatchParams &b, const FrameBuffers &fb, const TileBins &bins, cudaStream_t stream) {
	if (b.depthOnly || b.oddDepthFrames == 0 || b.totalTiles == 0) return;
	COUNT_LAUNCH();
	const unsigned frames = (unsigned)std::min<int32_t>(b.frameCount, 65535);
	launch_chained(odd_row_kernel, dim3((unsigned)b.maxTilesX, frames), 256, stream, b, fb.records, bins.offsets,
	               bins.lists, fb.rows);
}

void launch_raster(const BatchParams &b, const FrameBuffers &fb, const TileBins &bins, const RasterConfig &config, bool resolve,
                   cudaStream_t stream) {
	if (b.totalTiles == 0) return;
	if (!bins.cleared) memset_async(b.tileQueue, 0, sizeof(uint32_t), stream);
	const int threads = config.threadsPerTile == 64 ? 64 : (config.threadsPerTile == 128 ? 128 : 256);
	const int maxPerSm = 1024 / threads;
	const int perSm = config.ctasPerSm < 1 ? 1 : (config.ctasPerSm > maxPerSm ? maxPerSm : config.ctasPerSm);
	uint32_t ctas = (uint32_t)sm_count() * (uint32_t)perSm;
	const uint64_t items = (uint64_t)b.totalTiles + (bins.parts ? bins.partCapacity : 0u);
	if (ctas > items) ctas = (uint32_t)items;
	COUNT_LAUNCH();
	if (b.depthOnly && resolve && b.tileList && !b.fragments) { // counting fragments, and batches without a tile list: raster_kernel
		launch_chained(raster_depth_kernel, sm_count() * DEPTH_BLOCKS, 128, stream, b, fb.records, bins, fb.rows);
		return;
	}
	// small triangles resolve per pixel inside the tile pass; the keys then never leave the chip
	const bool fused = resolve && !b.depthOnly && config.resolveMode == 1;
#define DSRG_RASTER(T)                                                                                            \
	if (b.depthOnly && resolve) launch_chained(raster_kernel<true, T, true>, ctas, T, stream, b, fb.records, bins, fb.rows); \
	else if (b.depthOnly) launch_chained(raster_kernel<true, T, false>, ctas, T, stream, b, fb.records, bins, fb.rows); \
	else if (fused) launch_chained(raster_kernel<false, T, true>, ctas, T, stream, b, fb.records, bins, fb.rows); \
	else launch_chained(raster_kernel<false, T, false>, ctas, T, stream, b, fb.records, bins, fb.rows);
	if (threads == 64) { DSRG_RASTER(64) }
	else if (threads == 128) { DSRG_RASTER(128) }
	else { DSRG_RASTER(256) }
#undef DSRG_RASTER
	if (!resolve) return;
	if (!fused && !b.depthOnly) { // depth-only batches resolve inside the tile pass (depth_from_key)
		COUNT_LAUNCH();
		if (config.resolveMode == 2) launch_chained(resolve_quads_kernel, b.totalTiles, 64, stream, b, fb.records, bins.offsets, fb.rows);
		else launch_chained(resolve_pixels_kernel, b.totalTiles, 256, stream, b, fb.records, bins.offsets, fb.rows);
	}
	// the last rows of depth-tested odd-height frames, which every resolve above leaves alone
	launch_odd_rows(b, fb, bins, stream);
}

} // namespace dsrg
