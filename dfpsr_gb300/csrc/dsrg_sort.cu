// Stable LSD radix sort of (key, id) pairs, up to 8 bits per pass: per-block digit histograms, one scan
// over (digit, block) in digit-major order, and a scatter that keeps each block's items in input
// order.  Items whose key is not below keyEnd are left out by the first pass.
// Used by the deterministic adjoint of the differentiable renderer.
#include <cuda_runtime.h>
#include <stdint.h>

#include "dsrg_kernels.h"

namespace dsrg {

namespace {

const int SORT_THREADS = 256, SORT_WARPS = SORT_THREADS / 32;
// Items per thread: few for small sorts, whose blocks would not fill the GPU otherwise (a pass over
// 500,000 items took 44 us with 121 blocks of 4,096 items stepping together, and takes 20 us), and 16 for
// large ones, whose digit counts would grow into more work than the items.  The deterministic adjoint with
// 4 and with 16 items: 3.7 M entries 213 and 225 us, 14.7 M 420 and 413, 73 M 1,648 and 1,581; the line lies between
// the first two.
const int SORT_ITEMS_SMALL = 4, SORT_ITEMS_LARGE = 16;
const uint64_t SORT_LARGE = 1u << 22;

int items_per_block(uint64_t n) { return SORT_THREADS * (n > SORT_LARGE ? SORT_ITEMS_LARGE : SORT_ITEMS_SMALL); }

template <int ITEMS>
__global__ void __launch_bounds__(SORT_THREADS) radix_histogram_kernel(const uint32_t *__restrict__ keys, uint64_t n, const uint32_t *nDevice,
                                                                       uint32_t keyEnd, int shift, uint32_t bins, uint32_t *hist,
                                                                       uint32_t blocks) {
	__shared__ uint32_t counts[256];
	counts[threadIdx.x] = 0u;
	__syncthreads();
	if (nDevice) n = *nDevice;
	const uint64_t begin = (uint64_t)blockIdx.x * (SORT_THREADS * ITEMS);
#pragma unroll
	for (int k = 0; k < ITEMS; k++) {
		const uint64_t i = begin + (uint64_t)(k * SORT_THREADS) + threadIdx.x;
		const uint32_t key = i < n ? keys[i] : 0xFFFFFFFFu;
		if (key < keyEnd) atomicAdd(&counts[(key >> shift) & (bins - 1u)], 1u);
	}
	__syncthreads();
	if (threadIdx.x < bins) hist[(size_t)threadIdx.x * blocks + blockIdx.x] = counts[threadIdx.x]; // digit-major
}

// Writes the block's items to their digit's slots in input order.  A warp takes consecutive items,
// 32 at a time, and ranks each among the warp's items of its digit (the lanes before it from
// __match_any_sync, the steps before it from the warp's own counts, without a barrier); the
// warps' counts then give every warp its first slot of each digit.
template <int ITEMS>
__global__ void __launch_bounds__(SORT_THREADS) radix_scatter_kernel(const uint32_t *__restrict__ keysIn, const uint32_t *__restrict__ idsIn,
                                                                     uint64_t n, const uint32_t *nDevice, uint32_t keyEnd, int shift,
                                                                     uint32_t bins, const uint32_t *__restrict__ offsets, uint32_t blocks,
                                                                     uint32_t *keysOut, uint32_t *idsOut) {
	__shared__ uint32_t first[SORT_WARPS][256]; // the warps' counts, then their first slots
	if (nDevice) n = *nDevice;
	const uint64_t begin = (uint64_t)blockIdx.x * (SORT_THREADS * ITEMS);
	if (begin >= n) return;
	const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
	for (int w = 0; w < SORT_WARPS; w++) first[w][threadIdx.x] = 0u;
	__syncthreads();
	uint32_t key[ITEMS], rank[ITEMS];
	const uint64_t mine = begin + (uint64_t)(warp * 32 * ITEMS) + lane;
#pragma unroll
	for (int k = 0; k < ITEMS; k++) {
		const uint64_t i = mine + (uint64_t)(k * 32);
		key[k] = i < n ? keysIn[i] : 0xFFFFFFFFu;
	}
#pragma unroll
	for (int k = 0; k < ITEMS; k++) {
		const bool valid = key[k] < keyEnd;
		const uint32_t digit = valid ? (key[k] >> shift) & (bins - 1u) : 0x100u; // left-out items form their own group
		const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
		const uint32_t before = __popc(peers & ((1u << lane) - 1u));
		const uint32_t earlier = valid ? first[warp][digit] : 0u;
		rank[k] = earlier + before;
		__syncwarp();
		if (valid && before == 0u) first[warp][digit] = earlier + __popc(peers);
		__syncwarp();
	}
	__syncthreads();
	if (threadIdx.x < bins) {
		uint32_t next = offsets[(size_t)threadIdx.x * blocks + blockIdx.x];
		for (int w = 0; w < SORT_WARPS; w++) {
			const uint32_t count = first[w][threadIdx.x];
			first[w][threadIdx.x] = next;
			next += count;
		}
	}
	__syncthreads();
#pragma unroll
	for (int k = 0; k < ITEMS; k++) {
		if (!(key[k] < keyEnd)) continue;
		const uint64_t i = mine + (uint64_t)(k * 32);
		const uint32_t at = first[warp][(key[k] >> shift) & (bins - 1u)] + rank[k];
		keysOut[at] = key[k];
		idsOut[at] = idsIn ? idsIn[i] : (uint32_t)i;
	}
}

} // namespace

uint32_t sort_blocks(uint64_t n) { return (uint32_t)((n + items_per_block(n) - 1) / items_per_block(n)); }

void launch_stable_sort(const uint32_t *keys, uint64_t n, uint32_t keyEnd, const uint32_t *keptDevice, const SortBuffers &b,
                        cudaStream_t stream, const uint32_t **sortedIds) {
	const uint32_t blocks = sort_blocks(n);
	int keyBits = 1;
	while (keyBits < 32 && (1ull << keyBits) < (uint64_t)keyEnd) keyBits++;
	const int passes = (keyBits + 7) / 8, digitBits = (keyBits + passes - 1) / passes;
	const uint32_t bins = 1u << digitBits;
	const uint32_t *kin = keys, *iin = nullptr;
	uint32_t *kout = b.keysA, *iout = b.idsA;
	for (int p = 0; p < passes; p++) {
		const int shift = digitBits * p;
		const uint32_t *count = p == 0 ? nullptr : keptDevice;
		if (n > SORT_LARGE)
			radix_histogram_kernel<SORT_ITEMS_LARGE><<<blocks, SORT_THREADS, 0, stream>>>(kin, n, count, keyEnd, shift, bins, b.hist, blocks);
		else
			radix_histogram_kernel<SORT_ITEMS_SMALL><<<blocks, SORT_THREADS, 0, stream>>>(kin, n, count, keyEnd, shift, bins, b.hist, blocks);
		launch_scan(b.hist, b.offsets, bins * blocks, b.scanScratch, b.scanScratchElems, stream);
		if (n > SORT_LARGE)
			radix_scatter_kernel<SORT_ITEMS_LARGE><<<blocks, SORT_THREADS, 0, stream>>>(kin, iin, n, count, keyEnd, shift, bins, b.offsets, blocks,
			                                                                            kout, iout);
		else
			radix_scatter_kernel<SORT_ITEMS_SMALL><<<blocks, SORT_THREADS, 0, stream>>>(kin, iin, n, count, keyEnd, shift, bins, b.offsets, blocks,
			                                                                            kout, iout);
		add_launches(2);
		kin = kout;
		iin = iout;
		kout = (kout == b.keysA) ? b.keysB : b.keysA;
		iout = (iout == b.idsA) ? b.idsB : b.idsA;
	}
	*sortedIds = iin;
}

} // namespace dsrg
