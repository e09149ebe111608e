// hash.cuh -- per-slice MD5 + CRC32 launcher.
#pragma once
#include "common.cuh"

namespace p2g {

// The four slicing-by-4 tables of CRC-32/ISO-HDLC (reflected 0xEDB88320).
void crc32_tables(uint32_t tab[4][256]);
size_t hash_smem_bytes();

// MD5 (16 bytes per slice, d_md5) and CRC32 (d_crc) of n slices of S bytes;
// d_slices is a DEVICE array of 16-byte aligned device pointers.
int hash_run(p2g_ctx *ctx, const uint8_t *const *d_slices, int n, size_t S, uint8_t *d_md5,
             uint32_t *d_crc);

// ok[i] = 1 where both checksums of slice i are the expected ones, else 0 (md5
// and want_md5 16-byte aligned).
int hash_compare(cudaStream_t st, const uint8_t *d_md5, const uint32_t *d_crc, const uint8_t *d_want_md5,
                 const uint32_t *d_want_crc, int n, uint8_t *d_ok);

// Up to 32 slices of one size, hashed by one team; results at md5 (16-byte
// aligned, 16 bytes a slice) and crc.
struct HashWarp {
    const uint8_t *const *slices;
    size_t S;
    uint8_t *md5;
    uint32_t *crc;
    int count;
};
// All groups (a DEVICE array, longest first) in one launch.
int hash_groups(cudaStream_t st, int sms, const uint32_t *crc_tables, const HashWarp *d_groups, int n);

}  // namespace p2g
