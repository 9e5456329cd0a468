// Host-side launchers of the chunked canonical-Huffman kernels (huffman.cu).
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

#include "stz_internal.h"

namespace stz {

// A chunk holding unpredictable values and where its values sit in the
// stream's compact list.
struct UnpredWork {
    uint32_t stream;
    uint32_t chunk;
    uint64_t list_off;
    uint64_t count;  // values of this chunk in the list
};

// Run-symbol counts per stream (streams with run_n > 0): stats[s * kRunStats]
// gets the centre codes left as single symbols, stats[s * kRunStats + 1 + i]
// the uses of run slot i. stats must be zeroed.
constexpr int kRunStats = 64;
// Per stream: the bits of a run of r centre codes, r < kRunBitsStride
// (launch_codebooks; planes of up to 1024 codes).
constexpr uint32_t kRunBitsStride = 1025;
void launch_run_stats(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                      const uint16_t* codes, unsigned long long* stats, cudaStream_t st);
// Codebooks of every stream from its code histogram (2 radius bins a stream),
// the counts of codes outside the host window's range and the run-symbol
// counts (codebook.cu): patches each descriptor's cb_off, n_used, run_base
// and run_n, and writes the code tables (ctab: 2 radius entries a stream, code
// << 5 | length), the bits of a run of r centre codes (rbits: nstreams x
// kRunBitsStride bytes; streams with runs and planes of up to 1024 codes),
// the canonical (symbol, length) lists of all streams back to back, and what
// the host needs to find them. scratch_off[q]: first scratch item of stream
// q, codebook_items(stream) items each; items: their total.
struct CodebookInfo {
    uint32_t cb_off, n_used, run_base, run_n;
};
uint64_t codebook_items(const StreamDesc& s, uint64_t codes);
size_t codebook_scratch_bytes(uint64_t items, int nstreams);
void launch_codebooks(StreamDesc* sd, int nstreams, const uint32_t* hist, const uint32_t* outside,
                      const unsigned long long* rstats, const uint64_t* scratch_off, uint64_t items, void* scratch,
                      uint32_t* ctab, uint8_t* rbits, uint16_t* cb_sym, uint8_t* cb_len, CodebookInfo* info,
                      cudaStream_t st);
void launch_sub_bits(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                     const uint16_t* codes, const uint32_t* ctab, const uint8_t* rbits, uint32_t* sub_bits,
                     cudaStream_t st);
// Plane bit offsets, chunk word offsets and stream word counts from the
// plane bit counts; clears every plane's boundary words (max_chunks: the
// most chunks of any stream).
void launch_scan_streams(const StreamDesc* sd, int nstreams, uint32_t max_chunks, const uint32_t* sub_bits,
                         uint32_t* sub_off, uint64_t* chunk_word_off, uint64_t* stream_words, uint32_t* payload,
                         cudaStream_t st);
void launch_encode(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                   const uint16_t* codes, const uint32_t* ctab, const uint8_t* rbits, const uint32_t* sub_bits,
                   const uint32_t* sub_off, const uint64_t* chunk_word_off, uint32_t* payload, cudaStream_t st);
void launch_decode(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                   const uint16_t* cb_sym, const void* tables, const uint32_t* sub_off, const uint64_t* chunk_word_off,
                   const uint32_t* payload, uint16_t* codes, cudaStream_t st);
// The same for items marked by_plane.
void launch_decode_planes(const CtaWork* work, const uint32_t* chunk_ids, int nwork, const StreamDesc* sd,
                          const uint16_t* cb_sym, const void* tables, const uint32_t* sub_off,
                          const uint64_t* chunk_word_off, const uint32_t* payload, uint16_t* codes, cudaStream_t st);
// Decode tables of every stream (read by the decoders): decode_tables_bytes()
// each, stream i at byte i * decode_tables_bytes() of `tables`.
size_t decode_tables_bytes();
void launch_build_tables(const StreamDesc* sd, int nstreams, const uint16_t* cb_sym, const uint8_t* cb_len,
                         void* tables, cudaStream_t st);
// The payload words of streams [s0, s1) back to back in stream order into dst
// (each stream's count from stream_words, as k_scan_stream leaves it), so a
// group of small streams goes to the host in one transfer.
void launch_pack_streams(const StreamDesc* sd, const uint64_t* stream_words, int s0, int s1, const uint32_t* payload,
                         uint32_t* dst, cudaStream_t st);
// codes_most: the codes of the largest listed chunk.
template <typename T>
void launch_unpred_move(bool gather, uint32_t codes_most, const UnpredWork* work, int nwork, const StreamDesc* sd,
                        const uint16_t* codes, T* dense, T* list, cudaStream_t st);

// Persistent variants for captured graphs: `grid` CTAs walk the lists of a
// batch held in device memory (BatchHdr at meta: n_work/o_work/o_ids,
// n_uwork/o_uwork).
void launch_decode_dyn(int grid, const uint8_t* meta, const StreamDesc* sd, const uint16_t* cb_sym,
                       const void* tables, const uint32_t* sub_off, const uint64_t* chunk_word_off,
                       const uint32_t* payload, uint16_t* codes, cudaStream_t st);
template <typename T>
void launch_unpred_scatter_dyn(int grid, const uint8_t* meta, const StreamDesc* sd, const uint16_t* codes, T* dense,
                               T* list, cudaStream_t st);

}  // namespace stz
