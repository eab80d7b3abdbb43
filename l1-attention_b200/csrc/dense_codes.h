// Order codes of q and k (dense_codes.cu), which the tensor-core backward (dense_bwd_tc.cu) compares instead of the values.
//
// Per (batch, head, column) the keys are taken in blocks of CODE_BLOCK tokens and sorted; then, with rank(x) = number of the block's
// keys below x,
//     code(k) = 2 rank(k) + 1        code(q) = 2 rank(q) + (1 if q equals one of the keys, else 0)
// so that code(q) >= code(k) exactly where q >= k, and code(q) = code(k) exactly where q = k.  The tables hold 16-bit words
//     Q = 4 code(q) + tied(q)        K = 0x8000 - 4 code(k) + tied(k)        tied: equals a value of the other side in this block
// so that bit 15 of Q + K says q >= k, and bit 15 of Q + K - 3 says q > k.  No sum leaves its 16 bits: one 32-bit addition
// compares two pairs.  NaN is below and above nothing: Q = 0 and K = 0x8000 - 4 * NAN_CODE never reach 0x8000.
#pragma once
#include <stddef.h>
#include <stdint.h>
#include <cuda_runtime.h>
namespace l1b {
constexpr int CODE_BLOCK = 1024;
constexpr int NAN_CODE = 2 * CODE_BLOCK + 2;

// Tables in the scratch: [batch][head][token / 8][column][token % 8]; k once, q once for every block of keys.
struct CodeTables {
	size_t hdr, k, q, q_block; // byte offsets; bytes of one q table
	size_t bytes;
	int t8, nb; // groups of eight tokens, blocks of keys
};
inline CodeTables code_tables(int bs, int n_tok, int n_heads, int width)
{
	CodeTables c;
	c.t8 = (n_tok + 7) / 8;
	c.nb = (n_tok + CODE_BLOCK - 1) / CODE_BLOCK;
	const size_t n = size_t(bs) * n_heads * c.t8 * width * 16;
	c.q_block = (n + 255) / 256 * 256;
	c.hdr = 0;
	c.k = 256;
	c.q = c.k + c.q_block;
	c.bytes = c.q + size_t(c.nb) * c.q_block;
	return c;
}
// The widths that the tensor-core backward takes: a row of codes fits its stages.
constexpr int CODE_MAX_WIDTH = 128;
// Word of the header that sends a call to the exact kernel: a gradient is not finite, or so large that sums might overflow.
constexpr int CODE_HDR_EXACT = 1; // = BWD_HDR_OVERFLOW, on which the exact kernels wait

int dense_codes_launch(const float *q, const float *k, void *scratch, int bs, int n_tok, int n_heads, int width, cudaStream_t st);
// Gradients of the scores: element (batch, s, t, head) at b * stride_b + s * stride_s + t * stride_t + h * stride_h
struct GradStrides {
	long long b, s, t, h;
};
int dense_bwd_tc_launch(const float *g, GradStrides gs, float *d_q, float *d_k, void *scratch, int bs, int n_tok, int n_heads, int width, cudaStream_t st);
} // namespace l1b
