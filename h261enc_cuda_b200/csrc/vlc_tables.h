/* H.261 variable-length code tables for the macroblock headers of the device
 * bitstream writer (the coefficients' are in vlc_coder.h).
 *
 * The codes are the standard's (ITU-T H.261 Tables 1-4), the same values
 * the reference's src/h261_tables.c holds; the writer must reproduce the
 * reference's bytes, so nothing here may differ from the standard.  Layouts
 * are ours: (length << 8) | code in 16 bits, 0 = no entry. */
#pragma once

#include <cstdint>

namespace h261b {

#define VLC(code, len) (uint16_t)(((len) << 8) | (code))

/* MBA, address increment 1..33 */
static __device__ __constant__ uint16_t c_vlc_mba[34] = {
    0,           VLC(1, 1),   VLC(3, 3),   VLC(2, 3),   VLC(3, 4),   VLC(2, 4),   VLC(3, 5),
    VLC(2, 5),   VLC(7, 7),   VLC(6, 7),   VLC(11, 8),  VLC(10, 8),  VLC(9, 8),   VLC(8, 8),
    VLC(7, 8),   VLC(6, 8),   VLC(23, 10), VLC(22, 10), VLC(21, 10), VLC(20, 10), VLC(19, 10),
    VLC(18, 10), VLC(35, 11), VLC(34, 11), VLC(33, 11), VLC(32, 11), VLC(31, 11), VLC(30, 11),
    VLC(29, 11), VLC(28, 11), VLC(27, 11), VLC(26, 11), VLC(25, 11), VLC(24, 11),
};

/* MVD by magnitude 0..16 of the wrapped difference: the negative value's
 * code (the positive value's is one less; 0 has the code 1) */
static __device__ __constant__ uint16_t c_vlc_mvd[17] = {
    VLC(1, 1),   VLC(3, 3),   VLC(3, 4),   VLC(3, 5),   VLC(7, 7),   VLC(11, 8),
    VLC(9, 8),   VLC(7, 8),   VLC(23, 10), VLC(21, 10), VLC(19, 10), VLC(35, 11),
    VLC(33, 11), VLC(31, 11), VLC(29, 11), VLC(27, 11), VLC(25, 11),
};

/* CBP 1..63 */
static __device__ __constant__ uint16_t c_vlc_cbp[64] = {
    0,          VLC(11, 5), VLC(9, 5),  VLC(13, 6), VLC(13, 4), VLC(23, 7), VLC(19, 7), VLC(31, 8),
    VLC(12, 4), VLC(22, 7), VLC(18, 7), VLC(30, 8), VLC(19, 5), VLC(27, 8), VLC(23, 8), VLC(19, 8),
    VLC(11, 4), VLC(21, 7), VLC(17, 7), VLC(29, 8), VLC(17, 5), VLC(25, 8), VLC(21, 8), VLC(17, 8),
    VLC(15, 6), VLC(15, 8), VLC(13, 8), VLC(3, 9),  VLC(15, 5), VLC(11, 8), VLC(7, 8),  VLC(7, 9),
    VLC(10, 4), VLC(20, 7), VLC(16, 7), VLC(28, 8), VLC(14, 6), VLC(14, 8), VLC(12, 8), VLC(2, 9),
    VLC(16, 5), VLC(24, 8), VLC(20, 8), VLC(16, 8), VLC(14, 5), VLC(10, 8), VLC(6, 8),  VLC(6, 9),
    VLC(18, 5), VLC(26, 8), VLC(22, 8), VLC(18, 8), VLC(13, 5), VLC(9, 8),  VLC(5, 8),  VLC(5, 9),
    VLC(12, 5), VLC(8, 8),  VLC(4, 8),  VLC(4, 9),  VLC(7, 3),  VLC(10, 5), VLC(8, 5),  VLC(12, 6),
};

#undef VLC

/* MTYPE lengths (every code is a single 1 after zeros), indexed by the
 * reference's macroblock type numbers 0..9 (src/h261_types.h:15-24) */
enum {
    MT_INTRA = 0, MT_INTRA_MQ, MT_INTER, MT_INTER_MQ, MT_MC, MT_MC_CBP, MT_MC_CBP_MQ,
    MT_MC_FIL, MT_MC_FIL_CBP, MT_MC_FIL_CBP_MQ
};
static __device__ __constant__ uint8_t c_vlc_mtype_len[10] = { 4, 7, 1, 5, 9, 8, 10, 3, 2, 6 };

} // namespace h261b
