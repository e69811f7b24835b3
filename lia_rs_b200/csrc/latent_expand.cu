// Prompt portions of attention through a latent, ahead of their products: the pages that the portions' tokens can see are
// laid side by side, so that one product against [W_uk | unit matrix] and one against W_uv expand every record into whole
// keys and values per head, which the tcgen05 prompt kernel then attends over as over any pages.
//
// For portion s the blocks b0 .. b1 of its request's table hold the keys from its first token's earliest visible position to
// its last token's own; block b becomes page base_s + b - b0 of the side-by-side rows (the portions in order) and `table`, laid
// out like the step's block table, says so.  A record is copied as [latent: rank | rotated part: dr]: the unit matrix behind
// a head's share of W_uk then carries the rotated part through the product unchanged (a bfloat16 times one in 32-bit).
//
// A CTA copies one page (16-byte pieces where the sizes allow).  2,048 records of 512 + 64 are 4.7 MB, in and out of L2.
#include "common.cuh"

namespace {
template <typename V>
__global__ void __launch_bounds__(128)
latent_gather_kernel(const int* __restrict__ segments, int n_segments, const int* __restrict__ slots,
                     const int* __restrict__ block_table, int table_stride, const V* __restrict__ latent_pages,
                     const V* __restrict__ part_pages, V* __restrict__ records, int* __restrict__ table, int latent_words,
                     int part_words, int page_size, int window, int num_pages, int* __restrict__ error_flag) {
    pdl_launch_dependents();
    pdl_wait();
    int page = blockIdx.x, block = -1, slot = -1;
    for (int s = 0; s < n_segments; ++s) {
        const int start = segments[3 * s + 1], last = start + segments[3 * s + 2] - 1;
        const int first = window > 0 && start - window + 1 > 0 ? start - window + 1 : 0;
        const int b0 = first / page_size, blocks = last / page_size - b0 + 1;
        if (page < blocks) {
            block = b0 + page;
            slot = slots[segments[3 * s]];
            break;
        }
        page -= blocks;
    }
    if (block < 0 || block >= table_stride || slot < 0) return;
    const size_t at = (size_t)slot * table_stride + block;
    const int source = block_table[at];
    const bool there = source >= 0 && source < num_pages;
    if (threadIdx.x == 0) {
        table[at] = there ? (int)blockIdx.x : -1;
        if (!there && error_flag) atomicExch(error_flag, 2);
    }
    if (!there) return;
    const int words = latent_words + part_words;
    const V* latent = latent_pages + (size_t)source * page_size * latent_words;
    const V* part = part_pages + (size_t)source * page_size * part_words;
    V* out = records + (size_t)blockIdx.x * page_size * words;
#pragma unroll 4
    for (int e = threadIdx.x; e < page_size * words; e += blockDim.x) {
        const int row = e / words, c = e - row * words;
        out[e] = c < latent_words ? latent[(size_t)row * latent_words + c] : part[(size_t)row * part_words + (c - latent_words)];
    }
}
}  // namespace

// latent_pages [num_pages, page_size, rank] and part_pages [num_pages, page_size, dr] (16-bit elements), records [pages,
// page_size, rank + dr], table [slots, table_stride].  `pages`: at least the blocks that all portions see (pages beyond them are
// left as they are).  segments [n_segments][3]: first token's batch index, its position, count.
LIA_EXPORT int lia_latent_gather(const int* segments, int n_segments, const int* slots, const int* block_table, int table_stride,
                                 const void* latent_pages, const void* part_pages, void* records, int* table, int pages, int rank,
                                 int dr, int page_size, int window, int num_pages, int* error_flag, cudaStream_t stream) {
    if (n_segments <= 0 || pages <= 0) return LIA_OK;
    if (rank <= 0 || dr <= 0 || page_size <= 0 || table_stride <= 0 || num_pages <= 0) return LIA_ERR_SIZE;
    const bool wide = rank % 8 == 0 && dr % 8 == 0 &&
                      (((uintptr_t)latent_pages | (uintptr_t)part_pages | (uintptr_t)records) & 15u) == 0;
    if (wide)
        return lia_launch(latent_gather_kernel<uint4>, dim3(pages), dim3(128), 0, stream, segments, n_segments, slots, block_table,
                          table_stride, (const uint4*)latent_pages, (const uint4*)part_pages, (uint4*)records, table, rank / 8,
                          dr / 8, page_size, window, num_pages, error_flag);
    return lia_launch(latent_gather_kernel<uint16_t>, dim3(pages), dim3(128), 0, stream, segments, n_segments, slots, block_table,
                      table_stride, (const uint16_t*)latent_pages, (const uint16_t*)part_pages, (uint16_t*)records, table, rank, dr,
                      page_size, window, num_pages, error_flag);
}
