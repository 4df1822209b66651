"""psi_decode_plan_preview as the tests call it (no GPU needed)."""
import ctypes as C

import numpy as np

import __graft_entry__ as entry

pkg = entry.load_package()


def config(dtype, heads, head_dim, page, mode):
    size = 4 if dtype == pkg.F32 else 2
    return pkg.GQAConfig(*heads, head_dim, 1.0, 2 * heads[1] * head_dim * page * size, dtype, pkg.GQAPageTableLayout(1, 1, 1, 1), 1, pkg.PLAN_BALANCED, mode, 0)


def status_of(cfg, token_indices, cu_tokens, max_ctas, items, ctas, counts):
    u32 = lambda a: None if a is None else a.ctypes.data_as(C.POINTER(C.c_uint32))  # noqa: E731
    return pkg.library().psi_decode_plan_preview(C.byref(cfg), u32(token_indices), u32(cu_tokens), C.c_uint32(len(token_indices)), C.c_uint32(max_ctas),
                                                 u32(items), C.c_uint64(0 if items is None else len(items)), u32(ctas),
                                                 C.c_uint64(0 if ctas is None else len(ctas)), u32(counts))


def preview(cfg, token_indices, cu_tokens, max_ctas):
    ti, cu = (np.ascontiguousarray(x, dtype=np.uint32) for x in (token_indices, cu_tokens))
    counts = np.zeros(6, dtype=np.uint32)
    assert status_of(cfg, ti, cu, max_ctas, None, None, counts) == 0
    items, ctas = np.zeros((int(counts[0]), 6), dtype=np.uint32), np.zeros(int(counts[1]) + 1, dtype=np.uint32)
    assert status_of(cfg, ti, cu, max_ctas, items, ctas, counts) == 0
    return items, ctas, counts
