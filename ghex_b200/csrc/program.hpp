// The differentiable program in fused passes (program.cu): a pass is one halo exchange and one
// 7-point update (or the transpose of the two) of every domain, in one kernel.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "core.hpp"

namespace ghexb
{
// One domain of a program: interior extents, the caller's element strides, and its rows in a
// packed buffer (interior only, x fastest, rows on 32-byte boundaries).
struct program_domain
{
    int32_t n[3];
    int64_t s[3];
    int64_t row, plane, offset; // packed: elements per row and plane, first element in the buffer
    int32_t from[6];            // the domain whose far face the halo beyond face x-, x+, y-, y+, z-, z+ copies, or -1
    int32_t to[6];              // the domain whose halo copies this face, or -1
    uint32_t ranks;             // per face, 3 bits: the place of its image in the order images are added, 7 without one
    uint32_t images;            // bit (a + 3 b + 9 c): the halo region (a, b, c in 0..2 = before, inside, after) is written by the exchange
};
} // namespace ghexb

struct ghexb_program_s
{
    bool f64 = true;
    int32_t halo = 1;
    int64_t packed_elements = 0;
    std::vector<ghexb::program_domain> domains; // one per field
    // page-locked host word that the passes write and the host reads without waiting: 1, a load of a
    // pass did not arrive in time (what depended on it is not a number)
    unsigned* status = nullptr;

    ~ghexb_program_s();
};

namespace ghexb
{
// Status words (0 when taken), shared out by all programs from pages of 1024: page-locking one for
// each took 1 to 7 ms, as much as the rest of a graphed program's set-up (4.2 ms for 500 x 510 x 250;
// 5.5 to 7 with a word allocated on the device each). A page stays until the process ends, its words
// are used again.
unsigned* take_status_word();
void return_status_word(unsigned* word);

// The program's geometry from the fields of an exchange (n >= 1; their memory is not kept): every
// halo region must be written whole by the exchange or not at all, and every face of a domain must
// be a whole face of one neighbour. Throws ghexb::error (GHEXB_ERR_INVALID, with the reason) for
// any other exchange.
void build_program(ghexb_program_s& program, const ghexb_field* fields, int n, int halo);

// `steps` passes over the domains: from the caller's fields (`fields`, halo included) or, where
// it is null, from the packed buffer `source`; each pass but the last writes one of the packed
// buffers `a` and `b` in turn (the one it does not read), the last one `out` (the caller's layout;
// its halo zero, or for the transpose the gradient of the halo) or, where that is null, a packed
// buffer too. adjoint: the transpose. twice: the source is read times two (the gradient of a sum
// of squares).
cudaError_t launch_passes(const ghexb_program_s& program, const void* const* fields, const void* source, void* const* out,
    void* a, void* b, int steps, double alpha, bool adjoint, bool twice, cudaStream_t stream);

// Sum of squares of n interiors, in 64-bit partial sums of fixed blocks added in a fixed order:
// the same bits for the caller's layout and for a packed buffer. `partials` has room for
// sumsq_blocks doubles; the result goes to *out (float or double).
struct interior
{
    const void* p; // first interior cell
    int32_t n[3];
    int64_t s[3];
};
int64_t sumsq_blocks(bool f64, const int32_t (*extents)[3], int n);
cudaError_t launch_sumsq(bool f64, const interior* d, int n, bool packed, double* partials, void* out, cudaStream_t stream);
// The gradient of the sum of squares: out = g * (2 x) on the interior, 0 on the halo; p and out
// address the whole arrays (extents with the halo), *g is the gradient of the sum.
cudaError_t launch_sumsq_grad(bool f64, const interior* d, void* const* out, int n, int halo, const void* g, cudaStream_t stream);
} // namespace ghexb
