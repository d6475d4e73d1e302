// sweep_bytes.h -- device bytes of the LU-SGS sweeps' arrays in their two orders, and which one a context
// takes.  Host code only (no CUDA), so that the rule is tested without a device.
#pragma once
#include <stddef.h>

namespace tg {

// Hyperplane order, per interior cell: a case's share as case_bytes charges it.  rec: record entries, ndq:
// DeltaQ arrays (the sweep's, the tuner's copy, the two-plane schedule's), pc: PrecondDW entries (doubles);
// six neighbour positions, two flags and the cell.
inline size_t plane_cell_bytes(size_t rec, size_t ndq, size_t dq_stride, size_t elem, size_t pc) {
    return (rec + ndq * dq_stride) * elem + 8 * 4 + 16 + pc * 8;
}

// Marching order of one block: every tile of J x K lines takes ni + J + K - 2 steps of J K places.
// edge: bytes of a lane's edge words of a step; tile: bytes of a tile's entry; run: bytes of an entry of
// jac_steps steps (0: none).
struct MarchBytes { size_t steps, bytes; };
inline MarchBytes march_block_bytes(int ni, int nj, int nk, int J, int K, size_t rec, size_t dq_stride, size_t elem, size_t edge,
                                    size_t tile, size_t run, int jac_steps) {
    const size_t tiles = (size_t)((nj + J - 1) / J) * (size_t)((nk + K - 1) / K), steps = (size_t)(ni + J + K - 2);
    const size_t per_step = (size_t)J * K * (rec + dq_stride) * elem + (size_t)(J + K) * edge;
    const size_t runs = run ? (steps + jac_steps - 1) / jac_steps : 0;
    return {tiles * steps, tiles * (steps * per_step + tile + runs * run)};
}

// The marching order, unless the hyperplane order is the smaller (blocks whose lines fill their tiles badly, or
// that are short along i: it is padded to whole tiles and steps) and the difference does not fit the
// budget that is left (left < 0: no budget), or the marching arrays would take more than half of the free
// device memory, which the context's other lists, the next cases and their fields need too.  Where the marching
// arrays are the smaller, as on every large FP64 block (656 bytes of record a place against 1,280 a cell), the
// other order could only need more.
inline bool march_fits(size_t march, size_t planes, size_t free_bytes, long long left) {
    if (march <= planes) return true;
    if (left >= 0 && march - planes > (size_t)left) return false;
    return march <= free_bytes / 2;
}

}  // namespace tg
