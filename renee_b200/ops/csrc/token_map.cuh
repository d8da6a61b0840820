// Packed tokens: the encoder's activations hold only the tokens that can influence the pooled output.
//
// A token (b, s) of the padded [B, S] batch is KEPT if it is attended (mask != 0), if it is the first of its row (the
// CLS token, which pooling may read whatever its mask says), or if its whole row is masked (softmax is then uniform over
// all S keys).  Every other token is a masked key (probability exactly 0, so neither it nor its gradient reaches a kept
// one) whose own output nobody reads.  Kept tokens sit in packed rows in (b, s) order; the row count is rounded up to a
// multiple of TOK_ALIGN by rows of zeros so that the weight-gradient GEMMs, which contract over the rows in blocks of 64,
// read defined data.  The count lives on the device, so a captured graph serves every batch of its padded shape.
//   meta  [TOK_VALID] kept tokens, [TOK_ROWS] rows incl. the zero rows (never more than B S), [2] block counter (0)
//   tok   [B S]  packed row -> padded index b S + s (-1 for the zero rows): dropout counters number the padded layout
//   slot  [B S]  padded index -> packed row, or -1
//   off / len / cnt [B]  first packed row, last kept position + 1, attended tokens of a sequence
#pragma once
enum TokMeta : int { TOK_VALID = 0, TOK_ROWS = 1, TOK_COUNTER = 2, TOK_META_WORDS = 4 };
constexpr int TOK_ALIGN = 64;
