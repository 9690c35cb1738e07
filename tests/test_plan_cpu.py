"""Host-side layout bookkeeping of the kernels' plan, on CPU tensors built with the oracle's layouts."""
import numpy as np
import torch

from oracle import dkernel_oracle as O


def _plan(mask: np.ndarray):
    from dkernel_b200.ops import _Plan
    crow, col = O.dense_to_crow_col(mask)
    ccol, row = O.dense_to_ccol_row(mask)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(torch.int32)
    nnz = int((crow[:, 1:] - crow[:, :-1]).max())
    return _Plan(t(crow), t(col), t(ccol), t(row), 64, nnz)


def test_csc_to_csr_names_the_same_block():
    rng = np.random.default_rng(0)
    for H, R, Cn, dens in ((1, 5, 5, 0.5), (3, 16, 16, 0.3), (2, 7, 12, 0.6), (2, 9, 4, 0.0)):
        mask = (rng.random((H, R, Cn)) < dens).astype(np.uint8)
        if dens > 0:
            mask[:, 0, 0] = 1
        plan = _plan(mask)
        m = plan.csc_to_csr()
        assert m.shape == plan.row.shape and m.dtype == torch.int32
        crow, col, ccol, row = (x.numpy() for x in (plan.crow, plan.col, plan.ccol, plan.row))
        for h in range(H):
            for c in range(Cn):
                for j in range(ccol[h, c], ccol[h, c + 1]):
                    r = row[h, j]
                    i = int(m[h, j])
                    assert crow[h, r] <= i < crow[h, r + 1] and col[h, i] == c
            assert (m[h, ccol[h, Cn]:] == -1).all()
        assert plan.max_head_nnz() == int(mask.reshape(H, -1).sum(1).max())


def test_packed_parameter_values_land_in_their_fields():
    """The parameter structures are filled with one pack() of positional values: every value must end up in
    the field of its name."""
    import torch
    from dkernel_b200 import _lib, ops
    i32 = dict(dtype=torch.int32)
    crow, col = torch.arange(3 * 5, **i32).view(3, 5), torch.arange(3 * 7, **i32).view(3, 7)
    plan = ops._Plan(crow, col, crow, col, 64, 4)
    q, k, v = torch.zeros(2, 10, 6, 64).half(), torch.zeros(2, 20, 3, 64).half(), torch.zeros(2, 20, 4, 64).half()[:, :, :3]
    o, lse = torch.zeros(2, 10, 6, 64).half(), torch.zeros(2, 6, 10)
    rng = [torch.zeros(2, **i32) for _ in range(4)]
    p = ops._fwd_params(q, k, v, o, lse, 1, plan, 0.25, True, _lib.ROWS_BY_POSITION, *rng, total_q=11, impl=2)
    want = dict(q=q.data_ptr(), k=k.data_ptr(), v=v.data_ptr(), o=o.data_ptr(), lse=lse.data_ptr(),
                q_sb=3840, q_ss=384, q_sh=64, k_sb=3840, k_ss=192, k_sh=64, v_sb=5120, v_ss=256, v_sh=64,
                o_sb=3840, o_ss=384, o_sh=64, lse_sb=60, lse_sh=10, batch=2, hq=6, hkv=3, d=64, sq=10, sk=20, total_q=11,
                q_start=rng[0].data_ptr(), q_end=rng[1].data_ptr(), k_start=rng[2].data_ptr(), k_end=rng[3].data_ptr(),
                crow=crow.data_ptr(), col=col.data_ptr(), crow_sh=5, col_sh=7, h_pat=3, n_rows=4, block_size=64,
                causal=1, row_mode=1, dtype=_lib.BSA_F16, impl=2, sm_scale=0.25, col_bits=None, col_bits_sh=0,
                fine_block=0, tile_counter=None)
    assert set(want) == {n for n, _ in _lib.FwdParams._fields_}
    assert {n: getattr(p, n) for n in want} == want
