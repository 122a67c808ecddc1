// Host build of the exact arithmetic that the kernels use (dsrg_exact.h, dsrg_geometry.h),
// exported for CPU-side checks of the closed-form accumulation and the row intervals.
// Built with -ffp-contract=off so that it computes the same bits as the device code.
#include <stdint.h>

// Estimates of integer quotients 2^-21 off, at least as far as the device's: the host checks then
// exercise the exact corrections that follow them.
#define DSRG_HOST_ESTIMATE_ERROR 4.76837158203125e-7f
#include "dsrg_exact.h"
#include "dsrg_fill.h"
#include "dsrg_geometry.h"

extern "C" {

// out[i] = s[i] after n[i] additions of d[i] (dsrg::chain_add).
void dsrg_host_chain_add(const float *s, const float *d, const int32_t *n, float *out, int64_t count) {
	for (int64_t i = 0; i < count; i++) out[i] = dsrg::chain_add(s[i], d[i], n[i]);
}

// out[i] = min(max(L, (int32)(a/b + 1)), R) (dsrg::clamp_quotient_plus_one).
void dsrg_host_clamp_quotient(const int64_t *a, const int64_t *b, const int32_t *L, const int32_t *R, int32_t *out, int64_t count) {
	for (int64_t i = 0; i < count; i++) out[i] = dsrg::clamp_quotient_plus_one(a[i], b[i], L[i], R[i]);
}

// Row intervals of one triangle (sub-pixel corners flat[6]) for rows [y0, y0 + rows), clamped to [L, R).
void dsrg_host_row_intervals(const int32_t *flat, int32_t y0, int32_t rows, int32_t L, int32_t R, int32_t *lefts, int32_t *rights) {
	for (int32_t r = 0; r < rows; r++) dsrg::row_interval(flat, y0 + r, L, R, lefts[r], rights[r]);
}

// The same rows in 32-bit arithmetic where the triangle allows it (dsrg::near_edge, near_step), as
// rows_place_kernel steps them; 0 when it does not.
int32_t dsrg_host_row_intervals_near(const int32_t *flat, int32_t y0, int32_t rows, int32_t L, int32_t R, int32_t *lefts, int32_t *rights) {
	if (rows > dsrg::NEAR_ROWS || !dsrg::near_corners(flat, L, y0)) return 0;
	int32_t p[6];
	for (int i = 0; i < 3; i++) { p[2 * i] = flat[2 * i] - 256 * L; p[2 * i + 1] = flat[2 * i + 1] - 256 * y0; }
	const bool degenerate = (p[0] == p[2] && p[1] == p[3]) || (p[2] == p[4] && p[3] == p[5]) || (p[4] == p[0] && p[5] == p[1]);
	dsrg::NearEdge e[3] = {dsrg::near_edge(p[0], p[1], p[2], p[3]), dsrg::near_edge(p[2], p[3], p[4], p[5]), dsrg::near_edge(p[4], p[5], p[0], p[1])};
	for (int32_t k = 0; k < rows; k++) {
		lefts[k] = degenerate ? R : L;
		rights[k] = degenerate ? L : R;
		if (!degenerate)
			for (int i = 0; i < 3; i++) dsrg::near_step(e[i], L, L, R, lefts[k], rights[k]);
	}
	return 1;
}

// The same rows by exact stepping (dsrg::row_intervals_stepped).
void dsrg_host_row_intervals_stepped(const int32_t *flat, int32_t y0, int32_t rows, int32_t L, int32_t R, int32_t *lefts,
                                     int32_t *rights) {
	dsrg::row_intervals_stepped(flat, y0, rows, L, R, lefts, rights);
}

// The pieces that a rectangle is filled in (dsrg::add_fill_pieces): per piece its first byte, stride, width
// and height in words, and whether it is written 16 bytes at a time.  Returns their number.
int32_t dsrg_host_fill_pieces(uint64_t address, int32_t strideWords, int32_t width, int32_t height, uint64_t *out, int32_t capacity) {
	std::vector<dsrg::FillRect> pieces;
	dsrg::add_fill_pieces(dsrg::fill_rect((void *)(uintptr_t)address, strideWords, width, height, 0u), pieces);
	for (size_t i = 0; i < pieces.size() && (int32_t)i < capacity; i++) {
		const dsrg::FillRect &p = pieces[i];
		const uint64_t row[5] = {(uint64_t)(uintptr_t)p.words, p.stride, p.width, p.height, (uint64_t)p.vector};
		for (int k = 0; k < 5; k++) out[5 * i + k] = row[k];
	}
	return (int32_t)pieces.size();
}

} // extern "C"
