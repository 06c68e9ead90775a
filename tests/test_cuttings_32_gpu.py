"""32-bit models give equal bits however a prompt is cut into steps: 700 tokens whole, in portions and beside other requests.  The layers'
kernels for many tokens start at 148 to 592 tokens, so that these cuttings lie on both sides of every line."""

import pytest
import torch

from tests import helpers as H
from tests import kolisun_configs as K
from tests import ravapel_configs as R
from tests import rugedra_configs as U
from tests import vofanex_configs as V

pytestmark = pytest.mark.gpu


def _rugedra():  # the delta rule, latent attention, routed experts
    return U, U.config(72, 131, [("channel_delta", U.delta(16, 8, 64, 64, 4), U.moe(40, 6, 3, 3, 2)),
                                 ("latent_attention", U.latent(8, 32, 16, 32, 64), U.dense(264))], max_positions=1024)


def _vofanex():  # linear attention with low-rank decays, attention with a sink and a window
    return V, V.config(264, 131, [(V.gla(8, 64, 64, tau=8.0), V.dense(96)), (V.attention(6, 2, 32, 32, window=100), V.moe(5, 2, 24)),
                                  (V.gla(16, 32, 128, tau=3.5), None)])


def _ravapel():  # HGRN2
    return R, R.config(72, 131, [(R.hgrn2(8, 64, 64), R.dense(40)), (R.hgrn2(16, 32, 128), None)], max_positions=1024)


def _kolisun():  # latent attention whose queries have a latent of their own
    return K, K.config(72, 131, [(K.latent(8, 32, 16, 32, 64, 48), K.dense(96)), (K.latent(4, 16, 8, 16, 32, 20), None)])


@pytest.mark.parametrize("model", [_rugedra, _vofanex, _ravapel, _kolisun])
def test_equal_bits_however_it_is_cut(tmp_path, model):
    from inference_engine_b200.engine.replay import ReplaySession
    from inference_engine_b200.kernels import get_ops

    configs, cfg = model()
    weights = configs.make_weights(cfg, seed=5, **({"ranks": {0: 16, 2: 24}} if configs is V else {}))
    folder = H.write_model_dir(tmp_path / "model", cfg, weights)
    tokens = {rid: torch.randint(0, cfg["vocab"], (n,), generator=torch.Generator().manual_seed(n)).tolist()
              for rid, n in (("a", 700), ("b", 90), ("c", 1))}
    one = {"a": tokens["a"]}
    beside = [{"step": 0, "entries": [{"id": rid, "tokens": tokens[rid], "want": list(range(len(tokens[rid])))} for rid in ("b", "a", "c")],
               "end": ["a", "b", "c"]}]
    results = {}
    for how, steps in {"whole": H.trace_whole(one), "portions": H.trace_portions(one, (300, 150, 7)), "beside": beside}.items():
        session = ReplaySession(folder, "float32", 1024, device="cuda", ops=get_ops("cuda"), page_size=16)
        results[how] = H.collect(session, steps)["a"]
    get_ops("cuda").check_errors()
    assert torch.isfinite(results["whole"]).all() and results["whole"].shape[0] == 700
    for how in ("portions", "beside"):
        assert torch.equal(results["whole"], results[how]), how
