"""C tiles of the block-row SpGEMM kernel with alpha and beta and on a boundary
of 8 bytes only, in every output type, four and eight warps, tiles without
products among them: against the dense product, exact; what lies around the
tiles stays as it was."""
import numpy as np
import pytest
import torch

from kami_b200 import api

pytestmark = pytest.mark.gpu


def _bsr(rng, rows, cols, per):
    cnt = np.minimum(rng.integers(0, 2 * per + 1, rows), cols)
    ci = np.concatenate([np.sort(rng.choice(cols, c, replace=False)) for c in cnt]).astype(np.int32)
    rp = np.zeros(rows + 1, np.int32)
    np.cumsum(cnt, out=rp[1:])
    v = rng.integers(-2, 3, (len(ci), 16, 16))
    dense = np.zeros((rows, cols, 16, 16))
    dense[np.repeat(np.arange(rows), cnt), ci] = v
    dense = torch.from_numpy(dense.transpose(0, 2, 1, 3).reshape(rows * 16, cols * 16)).cuda()
    return api.BSR(torch.from_numpy(rp).cuda(), torch.from_numpy(ci).cuda(),
                   torch.tensor(v, dtype=torch.float16, device="cuda"), cols), dense


@pytest.mark.parametrize("rows", [50, 900])
@pytest.mark.parametrize("out", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("shift_bytes", [0, 8])
def test_alpha_beta(cuda, rows, out, shift_bytes):
    rng = np.random.default_rng(rows)
    (A, da), (B, db) = _bsr(rng, rows, 20, 3), _bsr(rng, 20, 24, 3)
    rp = torch.arange(0, (rows + 1) * 24, 24, dtype=torch.int32, device="cuda")  # every tile of C
    ci = torch.arange(24, dtype=torch.int32, device="cuda").repeat(rows)
    want = (da @ db).reshape(rows, 16, 24, 16).permute(0, 2, 1, 3).reshape(-1, 16, 16)
    n, shift = rows * 24 * 256, shift_bytes // out.itemsize
    for alpha, beta in ((1.0, 0.0), (2.0, -3.0), (-1.0, 0.0)):
        flat = torch.randint(-3, 4, (n + 16,), device="cuda").to(out)
        exact = flat.clone()
        old = exact[shift:shift + n].view(-1, 16, 16)
        old.copy_((alpha * want + beta * old.double()).float().to(out))
        if beta == 0.0:
            flat[shift:shift + n].fill_(float("nan"))  # not read
        api.spgemm_numeric(A, B, rp, ci, out, flat[shift:shift + n].view(-1, 16, 16), alpha=alpha, beta=beta)
        assert torch.equal(flat, exact)
