// Rectangles of 32-bit words that are each set to one value (a frame's clears).
#ifndef DSRG_FILL_H
#define DSRG_FILL_H

#include <stdint.h>

#include <vector>

namespace dsrg {

static const int FILL_RECTS = 32; // rectangles of one launch
// Words of a rectangle of a launch: the kernel counts them in 32 bits and steps past the end by up to
// the threads of its grid.
static const uint64_t FILL_WORDS_MAX = 1ull << 31;

struct FillRect {
	uint32_t *words;
	uint32_t stride, width, height; // in words
	uint32_t value;
	int32_t vector;                 // 16 bytes at a time (set by add_fill_pieces)
};

inline FillRect fill_rect(void *image, int32_t strideWords, int32_t width, int32_t height, uint32_t value) {
	FillRect r;
	r.words = (uint32_t *)image;
	r.stride = (uint32_t)strideWords;
	r.width = (uint32_t)width;
	r.height = (uint32_t)height;
	r.value = value;
	r.vector = 0;
	return r;
}

// Appends the rectangle in pieces of whole rows below FILL_WORDS_MAX words (a row is at most 2^29:
// strides in bytes fit 31 bits).  Rows without a gap between them become one row, and where rows begin
// on 16 bytes and are whole multiples of them the piece is written 16 bytes at a time.
inline void add_fill_pieces(FillRect r, std::vector<FillRect> &out) {
	if (r.width == 0 || r.height == 0) return;
	const uint32_t rowsMax = (uint32_t)((FILL_WORDS_MAX - 1) / r.width);
	while (r.height > 0) {
		FillRect piece = r;
		if (piece.height > rowsMax) piece.height = rowsMax;
		r.words += (uint64_t)piece.height * r.stride;
		r.height -= piece.height;
		if (piece.stride == piece.width) {
			piece.width *= piece.height;
			piece.height = 1;
		}
		piece.vector = ((uintptr_t)piece.words & 15u) == 0 && piece.width % 4u == 0 && (piece.height == 1 || piece.stride % 4u == 0);
		out.push_back(piece);
	}
}

} // namespace dsrg

#endif
