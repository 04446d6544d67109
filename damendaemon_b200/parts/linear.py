"""Matrix products of the parts: one call that picks the kernel for the engine dtype."""
from __future__ import annotations

import functools

import torch

from .. import kernels


def splits_float32(out, reduction):
    """Whether a float32 product with a matrix of this size goes to the tensor cores, every operand as three bfloat16
    numbers (its error against 64-bit sums is below that of float32 multiply-adds one after the other at every size tried,
    K = 4 to 6,400). Smaller matrices stream through the CUDA-core kernel in fewer steps than the split one needs to
    start (split / CUDA cores, us): 1024 x 256 at 8 rows 7.2 / 3.4, 512 x 512 at 8 and 64 rows 7.3 / 4.8 and 12.4 / 11.9;
    1024 x 1024 7.5 / 8.1 and 11.3 / 21.8, 6400 -> 1600 15 / 41 and 21.5 / 125. The line goes by the matrix alone, so that
    a row of a small model has the same bits whatever else is in the batch. The split product cuts its sums by the number of
    tiles: a row of a larger model has other bits beside more than 128 tokens than alone, within the same error (gemm='simt'
    keeps them)."""
    return out * reduction >= 1 << 20


RESIDENT_CLUSTERS = (148, 74, 45, 33, 26, 22, 15, 15)       # clusters of 1 to 8 blocks that a B200 holds at once, one block an SM
STREAM_BOX_US = (0.32, 0.40, 0.46, 0.32, 0.46, 0.46, 0.37, 0.35)       # gemm_stream by blocks of a cluster: us a row and box of 256 k


@functools.lru_cache(maxsize=4096)
def stream_is_ahead(out, reduction):
    """Whether gemm_stream is estimated to take less time than gemm_split for up to eight rows. Neither is ahead over a whole
    range: both cut their work into rounds of what the GPU holds, at different sizes. The estimates, in us, were fitted to 217
    shapes (out 300 to 100,000, reduction 128 to 14,336, 12 to 200 MB) that were timed with both. The product that they take
    is the slower one by up to 8 % (1,024 x 11,008: 20.9 for 19.4), mostly by none; the stream alone is by up to 70 %
    (split / stream at 8 rows: 4,096 x 4,096 18.4 / 27.6, 11,008 x 4,096 51.4 / 66.7, 65,536 x 128 14.5 / 24.7, 32,000 x 1,536
    41.8 / 42.9; but 2,048 x 2,048 15.6 / 8.0, 9,000 x 1,280 13.3 / 11.9, 1,600 x 6,400 15.2 / 14.4)."""
    up = lambda a, b: -(-a // b)
    # split: a block takes its share of a tile's k blocks; tiles beyond the resident clusters wait for a second wave
    blocks = up(reduction, 32)
    share = up(blocks, kernels._split_plan(kernels.GEMM_STREAM_ROWS, out, reduction, RESIDENT_CLUSTERS[0])[0])
    cluster = up(blocks, share)
    waves = up(up(out, 128), RESIDENT_CLUSTERS[cluster - 1])
    split = 5.4 + 0.37 * share * waves + (3.7 * (waves - 1) if cluster > 1 else 0)
    # stream: a warp takes two to four rows of the matrix at a time, the fewest in all; the blocks that share K wait for one another
    # in every round
    part = up(up(reduction, up(reduction, 7 * 256)), 128) * 128
    cluster, boxes = up(reduction, part), up(part, 256)
    warps = 16 * RESIDENT_CLUSTERS[cluster - 1]
    at_once = min((4, 3, 2), key=lambda r: up(up(out, r), warps) * r)
    rounds = up(up(out, at_once), warps)
    start, row = (1.9, 0.66) if cluster == 1 else (1.0 + 2.2 * rounds, 0.55)
    stream = start + (row + STREAM_BOX_US[cluster - 1] * boxes) * rounds * at_once
    return max(stream, out * reduction * 4 / 4.7e6) < split


def streams_float32(rows, out, reduction):
    """Whether a float32 product that splits_float32 takes streams its matrix through the CUDA cores (kernels.gemm_stream)
    instead: up to eight rows and a matrix of 12 to 200 MB, where that is ahead (split / stream, us at 8 rows: 3072 x 1024
    13.7 / 5.8, 4096 x 1024 9.0 / 6.8, 1024 x 4096 11.0 / 8.4, 4800 x 1600 11.9 / 9.3, 6400 x 1600 14.2 / 11.0, 1600 x 6400
    14.8 / 14.2, 25600 x 1600 41.7 / 34.6; 50257 x 1600 60.6 / 68.3: the stream's warps reach 4.7 TB/s, what their reads of X from
    shared memory leave them, the split product 5.3). Smaller matrices stay with the split product. A row of a streamed
    product has other bits beside more than seven others, where the split product takes over, than beside fewer, within
    the error of either (gemm='simt' keeps them)."""
    return rows <= kernels.GEMM_STREAM_ROWS and 3 << 20 <= out * reduction <= 3 << 24 and reduction <= kernels.GEMM_STREAM_REDUCTION \
        and stream_is_ahead(out, reduction)


def linear(runtime, a, w, bias=None, residual=None, activation=None, out_dtype=None, out=None):
    """act(a @ w.T + bias) (+ residual). float32 engine: the split product on the tensor cores, or for up to eight rows the
    product that streams the matrix (a row's last bits may change between eight rows and nine, see streams_float32, and
    beyond 128, see splits_float32); for small matrices and rows that are not 16-byte aligned, or if the runtime asks for 'simt',
    the CUDA-core float32 kernel, whose rows do not depend on what is beside them.
    bfloat16 engine: the tcgen05 tensor-core kernel, unless the runtime asks for 'simt' or the
    reduction width is no multiple of 8 (then the CUDA-core kernel with bfloat16 operands)."""
    if a.dtype == torch.float32 and runtime.gemm != "simt" and out_dtype in (None, torch.float32) and \
            splits_float32(w.shape[0], a.shape[1]) and kernels.gemm_split_fits(a, w):
        if streams_float32(a.shape[0], w.shape[0], a.shape[1]):
            return kernels.gemm_stream(a, w, bias, residual, activation, out)
        return kernels.gemm_split(a, w, bias, residual, activation, out)
    if a.dtype == torch.float32 or runtime.gemm == "simt":
        return kernels.gemm_simt(a, w, bias, residual, activation, out_dtype, out)
    if a.shape[1] % 8 or a.stride(0) % 8 or w.stride(0) % 8:
        # TMA wants 16-byte rows; a reduction width that is no multiple of 8 runs on the CUDA cores instead
        return kernels.gemm_simt(a, w, bias, residual, activation, out_dtype or torch.bfloat16, out)
    return kernels.gemm_tcgen05(a, w, bias, residual, activation, out_dtype, out)


def grouped_on_tensor_cores(runtime, dtype, *reductions):
    """Whether grouped products over these reduction widths run on the tensor cores: bfloat16, and every width a
    multiple of 8 (TMA needs 16-byte rows). One answer for all products of a part: they share the rows' tiles."""
    return dtype == torch.bfloat16 and runtime.gemm != "simt" and all(k % 8 == 0 for k in reductions)


def grouped_tile(tensor_cores, pairs, groups):
    """Rows per tile of the grouped products: every group's rows start on a multiple of it. The tensor-core kernel
    takes 16 to 128: about twice the rows a group gets on average, so that few tiles are mostly padding and few groups
    need several. The CUDA-core kernel has one tile size."""
    if not tensor_cores:
        return kernels.simt_group_tile()
    want = 2 * pairs // max(1, groups)
    return next((t for t in kernels.GROUPED_TCGEN05_TILES if t >= want), kernels.GROUPED_TCGEN05_TILES[-1])


def grouped_linear(tensor_cores, a, w, tile_group, tile, out_dtype=None, activation=None, row_scale=None):
    """Rows of a in tiles of ``tile``; tile i is multiplied with w[tile_group[i]] (w: [groups, out, in]); tiles whose
    group is negative are skipped. act(row_scale[r] * product), row_scale float32 [rows] or None, in the product's epilogue."""
    if tensor_cores:
        return kernels.gemm_grouped_tcgen05(a, w, tile_group, tile, out_dtype=out_dtype or a.dtype, activation=activation, row_scale=row_scale)
    return kernels.gemm_simt_grouped(a, w, tile_group, activation=activation, out_dtype=out_dtype or a.dtype, row_scale=row_scale)


def grouped_gated_unit(tensor_cores, a, gate_up, tile_group, tile, limit, alpha, form="clamped_swish"):
    """The gated unit (form: one of kernels.GATED_FORMS) over grouped rows: gate_up [groups, 2 * inner, in] holds a group's
    gate rows, then its up rows. On the tensor cores both products and the unit are one kernel; else a grouped product and
    the unit's own kernel."""
    if tensor_cores:
        return kernels.gemm_grouped_tcgen05(a, gate_up, tile_group, tile, gated=(limit, alpha, form))
    return kernels.gated_unit(kernels.gemm_simt_grouped(a, gate_up, tile_group), limit, alpha, form=form)
