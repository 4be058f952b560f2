"""A timestep whose array ends before the size the stream's descriptor gives is
refused, as the copy it takes the place of was, and the stream goes on; arrays
that end with their allocation are taken."""
import numpy as np
import pytest

from ftk2_b200 import api
import test_stream_gpu as ts
import cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("short", [0, 1])
def test_short_component_array_is_refused(ctx, short):
    import torch
    # whole allocations of their own, so that their ends are the tensors' ends
    dims, nt, n = [2048, 1025], 3, 2048 * 1025
    rng = np.random.default_rng(4)
    v = np.full((2, nt, dims[1], dims[0]), 1.0, np.float32)
    v[:, :, -40:, -30:] = rng.standard_normal((2, nt, 40, 30))  # the features lie in the last rows
    keep: list = []
    with api.Stream(ctx, api.regular_mesh_desc(dims + [1]),
                    api.field_desc(list(v[:, 0]), api.LAYOUT_SEPARATE, 2, keep=keep), api.params(2.0 ** 20)) as st:
        torch.cuda.empty_cache()
        # 32 MB each: the steps lie at the very end of their blocks
        blocks = [torch.zeros(8 << 20, dtype=torch.float32, device="cuda") for _ in range(2)]
        for t in range(nt):
            step = []
            for j in range(2):
                blocks[j][-n:] = torch.from_numpy(v[j, t].ravel()).cuda()
                step.append(blocks[j][-n:].view(dims[1], dims[0]))
            torch.cuda.synchronize()
            fld = api.field_desc(step, api.LAYOUT_SEPARATE, 2, keep=keep)
            if t == 1:
                bad = api.field_desc(step, api.LAYOUT_SEPARATE, 2, keep=keep)
                bad.comp[short] = blocks[short].data_ptr() + 4 * ((8 << 20) - 1024)
                with pytest.raises(api.Ftk2bError) as e:
                    st.push(bad)
                assert e.value.status == api.CUDA_ERROR
            st.push(fld)
        got = st.result()
    case = cases.Case("noise", "regular", 2, cases.SEPARATE, list(v), 2.0 ** 20, dims + [nt])
    ts.assert_identical(got, ts.one_shot(ctx, case, nt, False))
