// Geometry of the plane-streaming kernels (efm_stream.cu).
//
// A block owns one (x, z) tile of tw x th cells at a time and marches it along y; each of its
// consumer threads computes a pair of x-neighbours (one 8-byte shared-memory access per operand
// and pair) of every plane.  Two block sizes are built: 224 consumer threads (tiles up to 448
// cells, two blocks per SM) and 96 (up to 192 cells, four): with the producer warp that is 16
// warps per SM, four per scheduler, and 128 registers per thread (a ninth warp per block would
// leave 96).  The large blocks are the default on every grid: their wider tiles load fewer
// neighbours per cell and hide more behind one another (forward + gradient, ms, large and the
// better of the small ones' two rings: 64 x 64 x 64 1.92, 2.14; 96 x 96 x 64 3.36, 3.50; 128 x 128 x 96
// 7.21, 8.23; 256 x 256 x 128 19.3, 21.2); the small ones are an option the autotuner times.  The
// tile's shape is chosen per grid (shape_of in efm_capi.cu) so that ragged grids do not leave
// threads idle; the shared-memory slots below bound it.
#pragma once

#define EFM_MAX_YCHUNK 64
#define EFM_IMG 3  // the imaging pass, beside EFM_FWD, EFM_ADJ, EFM_REV

// Consumer threads of the variant with `rows` (EFM_OPT_TILE_ROWS); a producer warp comes on top.
__host__ __device__ constexpr int efm_st_nt(int rows) { return rows == 1 ? 96 : 224; }
__host__ __device__ constexpr int efm_st_cells(int nt) { return 2 * nt; }
// Shared-memory slot of one plane's field: the cells alone, or a box with x neighbours (tw + 4
// columns, so that the TMA x start stays 16-byte aligned), with one z neighbour row, with both,
// or with x neighbours and two z rows.
__host__ __device__ constexpr int efm_slot_c(int nt) { return 8 * nt; }
__host__ __device__ constexpr int efm_slot_x(int nt) { return nt == 224 ? 2048 : 1024; }
__host__ __device__ constexpr int efm_slot_z(int nt) { return nt == 224 ? 2304 : 1024; }
__host__ __device__ constexpr int efm_slot_xz(int nt) { return nt == 224 ? 2432 : 1152; }
__host__ __device__ constexpr int efm_slot_xz2(int nt) { return nt == 224 ? 2816 : 1408; }

// Whether a tile of tw x th cells fits the slots.
__host__ __device__ constexpr bool efm_shape_ok(int nt, int tw, int th) {
    return tw >= 4 && tw % 4 == 0 && tw <= 252 && th >= 1 && tw * th <= efm_st_cells(nt) &&
           (tw + 4) * th * 4 <= efm_slot_x(nt) && tw * (th + 1) * 4 <= efm_slot_z(nt) &&
           (tw + 4) * (th + 1) * 4 <= efm_slot_xz(nt) && (tw + 4) * (th + 2) * 4 <= efm_slot_xz2(nt);
}

// Bytes of one plane: fields with neighbours (kept for planes j and j+1) and cell-only fields.
__host__ __device__ constexpr int efm_halo_s(int nt) { return 4 * efm_slot_xz(nt); }
__host__ __device__ constexpr int efm_cell_s(int nt) { return 7 * efm_slot_c(nt); }
__host__ __device__ constexpr int efm_halo_v(int nt) {
    return 2 * efm_slot_x(nt) + 2 * efm_slot_z(nt) + 2 * efm_slot_xz(nt) + efm_slot_c(nt);
}
__host__ __device__ constexpr int efm_cell_v(int nt) { return 3 * efm_slot_c(nt); }
__host__ __device__ constexpr int efm_halo_i(int nt) { return 3 * efm_slot_xz(nt) + efm_slot_xz2(nt); }
__host__ __device__ constexpr int efm_cell_i(int nt) { return 7 * efm_slot_c(nt); }
// One ring slot: a plane's neighbour and cell fields (of the stress and velocity passes, or of the imaging).
__host__ __device__ constexpr int efm_slot_bytes(int nt, bool image) {
    return image                                                                ? efm_halo_i(nt) + efm_cell_i(nt)
           : efm_halo_s(nt) + efm_cell_s(nt) > efm_halo_v(nt) + efm_cell_v(nt) ? efm_halo_s(nt) + efm_cell_s(nt)
                                                                                 : efm_halo_v(nt) + efm_cell_v(nt);
}
// resident blocks per SM the launch bounds promise (d: ring depth)
__host__ __device__ constexpr int efm_stream_blocks(int nt, int d) { return nt == 96 ? (d > 3 ? 3 : 4) : 2; }
