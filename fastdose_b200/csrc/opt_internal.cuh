// opt_internal.cuh -- device CSR matrix of the optimizer, shared by the SpMV,
// VOI-restriction and solver translation units.
#pragma once
#include <cstdint>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../../include/fd2_opt.h"
#include "fd2_internal.cuh"

namespace fd2 {

constexpr int kChunk = 256;           // nonzeros per SpMV chunk (32 lanes x 8)
constexpr int kChunkWords = kChunk / 32;

// Storage position of logical nonzero k.  A matrix of long rows whose x is
// gathered from global memory, or whose values are 16 bits and x is large, is
// interleaved inside a chunk: logical element
// 32 i + l is stored at 8 l + i, so that lane l's two 16-byte loads bring it
// elements l, l + 32, ..., l + 224, and each of the warp's x-gathers covers 32
// consecutive nonzeros of the row instead of 32 elements 8 apart.  In the other
// matrices lane l holds elements 8 l .. 8 l + 7, rotated by l / 4: a gather of
// consecutive columns from shared memory then meets every bank once.
__host__ __device__ __forceinline__ int64_t slot(int64_t k, bool interleaved) {
    const int64_t c = k / kChunk;
    const int e = (int)(k % kChunk);
    return c * kChunk + (interleaved ? (e % 32) * 8 + e / 32 : (e & ~7) + ((e - (e >> 5)) & 7));
}

// Column index of logical nonzero k in either index format (after finalize).
struct ColView {
    const int32_t* col;     // I32: [nnz_pad], storage order
    const uint16_t* col16;  // PACKED16: [nnz_pad] offset from the chunk base, storage order
    const int32_t* cbase;   // PACKED16: per chunk base, or -(1 + exception slot)
    const int32_t* exc;     // PACKED16: [slots * kChunk] columns of exception chunks, storage order
    bool interleaved;       // storage order: slot()
    __device__ __forceinline__ int64_t at_slot(int64_t k) const { return slot(k, interleaved); }
    __device__ __forceinline__ int at(int64_t k) const {
        const int64_t q = at_slot(k);
        if (col) return col[q];
        const int32_t b = cbase[k / kChunk];
        return b >= 0 ? b + (int)col16[q] : exc[(int64_t)(-1 - b) * kChunk + (q % kChunk)];
    }
};

inline size_t value_size(int vt) { return vt == FD2_VALUES_F32 ? 4 : 2; }
inline int64_t round_chunk(int64_t n) { return (n + kChunk - 1) / kChunk * kChunk; }
inline int current_device() {
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

}  // namespace fd2

struct fd2_matrix {
    fd2_context* ctx = nullptr;
    int device = fd2::current_device();  // where its memory is; it may outlive the context
    int64_t rows = 0, cols = 0, nnz = 0;
    int value_type = FD2_VALUES_F32;
    int scale_axis = FD2_SCALE_NONE;
    int index_format = FD2_INDEX_I32;
    int64_t* d_off = nullptr;      // [rows + 1]
    // Builders write d_col / d_val in logical order; matrix_finalize moves them
    // to storage order (slot()), after which readers index through slot().
    int32_t* d_col = nullptr;      // I32: [nnz_pad]; PACKED16: released after packing
    uint16_t* d_col16 = nullptr;   // PACKED16: [nnz_pad]
    int32_t* d_cbase = nullptr;    // PACKED16: [n_chunks]
    int32_t* d_exc = nullptr;      // PACKED16: [n_exc * kChunk]
    int64_t n_exc = 0;
    void* d_val = nullptr;         // [nnz_pad] float / __half / __nv_bfloat16, zero past nnz
    float* d_scale = nullptr;      // [rows] or [cols] when scale_axis != NONE
    // stream SpMV plan
    int64_t n_chunks = 0;          // nnz_pad / kChunk
    uint32_t* d_head = nullptr;    // [n_chunks * kChunkWords] row starts: per chunk 32 bytes, one per
                                   // lane; bit i of byte l: the lane's element i starts its row
    int32_t* d_chunk_h = nullptr;  // [n_chunks] row starts before the chunk
    int32_t* d_chunk_row0 = nullptr;  // [n_chunks] first row starting in the chunk if its starts are
                                      // consecutive rows, else -1 - d_chunk_h[c]
    int32_t* d_nzrow = nullptr;    // [n_nzrows] rows with nonzeros, in order
    int64_t n_nzrows = 0;
    int n_warps = 0;               // SpMV warps
    int n_ranges = 0;              // contiguous chunk ranges, n_warps or a multiple of it
    bool x_in_smem = false;        // SpMV instance: x staged in shared memory (cols small enough)
    bool interleaved = true;       // storage order inside a chunk (slot())
    int64_t* d_carry_row = nullptr;  // [n_ranges] row open at each range's end
    float* d_carry_val = nullptr;    // [n_ranges] its partial sum
    float* d_xs = nullptr;           // [cols] x times the column scale, where the product does not scale x itself
    int32_t* d_zrow = nullptr;       // rows the product itself does not write: empty, or only in carries
    int* d_nz = nullptr;             // [2] number of those rows, and n_nzrows
    int n_zrows = 0;                 // the first on the host

    fd2::ColView cols_view() const { return fd2::ColView{d_col, d_col16, d_cbase, d_exc, interleaved}; }
};

namespace fd2 {

// Device memory of matrices and problems and of what builds them, in the order
// of a stream, from a pool the library keeps per device (as densities are): a
// matrix makes some thirty allocations, and cudaMalloc and cudaFree, which wait
// for the device, took most of the time of the orientation loop's phases.  The
// pool keeps at most 4 GiB of freed memory (with 1 GiB, the transpose of 5e7
// nonzeros gave its buffers back and took them again: 15 % of the build);
// fd2_context_release empties it.  Blocks of kPlainBlock and more are plain
// allocations: past what it keeps, a pool maps and unmaps 3 to 11 ms a GiB, where
// cudaMalloc and cudaFree take 0.6 and 1.2.  Transpose of 2e8 nonzeros in 16 bits,
// all from cudaMalloc / from the pool / as now: 24.6 / 98 / 22 ms, of 8e8 91 / 590 /
// 84, of 5e7 10.1 / 2.7 / 3.8; the VOI matrices of 2.7e8: 0.11 / 0.6 to 1 / 0.10 s.
constexpr size_t kPlainBlock = (size_t)512 << 20;
cudaError_t mat_malloc_bytes(void** p, size_t bytes, cudaStream_t stream);
template <typename T>
cudaError_t mat_malloc(T** p, size_t bytes, cudaStream_t stream) {
    return mat_malloc_bytes((void**)p, bytes, stream);
}
// Returns memory whose last use is before this point of the stream.
void mat_free(void* p, cudaStream_t stream);

// Allocates d_off (rows + 1), d_col (int32, nnz padded to kChunk), d_val
// (padded, zeroed past nnz) and d_scale for the sizes in m.
int matrix_alloc(fd2_matrix* m, cudaStream_t stream);
// The same without d_off (for builders that write the offsets first).
int matrix_alloc_entries(fd2_matrix* m, cudaStream_t stream);
// Builds the SpMV plan (row-start bitmap, chunk row counts, non-empty rows,
// warp partition) from d_off, and packs the columns when m->index_format is
// PACKED16.  Call once the offsets, columns and values are written.
int matrix_finalize(fd2_matrix* m, cudaStream_t stream);
// Frees what m holds, after all work of its device (a product may run on any
// stream, the matrix may outlive its context, and another device may be current).
void matrix_free(fd2_matrix* m);
// Transpose into a matrix of the given index format.
int matrix_transpose_fmt(const fd2_matrix* m, int index_format, fd2_matrix** out);
// Row blocks of m in a given order (fd2_matrix_select_blocks).
int matrix_select_blocks(const fd2_matrix* m, int64_t n_blocks, const int64_t* h_rows, const int64_t* h_cols,
                         int64_t n_keep, const int64_t* h_order, fd2_matrix** out);
// y = M x on `stream`.  Not re-entrant per matrix: a column-scaled matrix
// stages the scaled x, and every product its carries, in the matrix's buffers.
int matrix_spmv(const fd2_matrix* m, const float* d_x, float* d_y, cudaStream_t stream);
// The context a dose-loading matrix was built on.
fd2_context* ensemble_context(const fd2_csr_ensemble* e);
// The stream a dose-loading matrix's arrays are ordered on.
cudaStream_t ensemble_stream(const fd2_csr_ensemble* e);

}  // namespace fd2
