"""QuadDirect inside the Stereo pipeline reads the solver's C1 where it needs it: on the BF16 path too (the CRF's
16-bit unary copy), the refined map equals the fit on the written-out C1 of the same solve, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 40])
def test_bf16_quadfit_equals_fit_on_c1(cuda, D):
    torch = cuda
    from cnncrf import api, scenes, _lib as L
    from test_gpu_bf16 import q16_unary
    W, H = 120, 33
    s = scenes.kitti_scene(W, H, D, seed=4, ground_max=D * 0.8, box_range=(4.0, D * 0.9))
    st = api.Stereo(precision=L.BF16, unary=L.UNARY_ONE_MINUS_DOT, topology=L.TOPO_ALL3X3, ref_depth_rounding=False,
                    crf_shape=L.RHO_LINEAR)
    st.initialize(W, H, 0.0, 1.0, float(D - 1))
    st.set_matching_function(L.MATCH_COLORCNN_PAIRWISE)
    st.set_num_layers(3)
    st.set_xavier_seed(0)
    st.set_color_images(s["left"], s["right"])
    st.compute_slack_propagation(0.5, 1.5, 3, 4, 0.0, 0.0, 1.0)
    vol, (wx, wy) = st.volume_device().clone(), (t.clone() for t in st.weights_device())
    u = st.output_device().clone()
    st.fuse_quad_fit_direct()
    sp, labels = api.SlackProp(), torch.empty((H, W), device="cuda", dtype=torch.int32)
    sp.init(q16_unary(torch, vol, 1) if D % 64 == 0 else vol, labels)
    for k, v in dict(L1=0.5, L2=1.5, delta=3, total_it=4, shape=L.RHO_LINEAR, slack=0.5).items():
        sp.ops[k] = v
    sp.update_W(wx, wy)
    sp.execute()
    want = api.quad_fit_direct(u, sp.get_C1(), 0.0, 1.0)
    assert np.array_equal(st.output_device().cpu().numpy(), want.cpu().numpy())
    assert not torch.equal(want, u)
