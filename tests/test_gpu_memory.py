"""Device memory that is not to be had: what fails, what goes on, and what the calls after it see."""
import numpy as np
import pytest

from helpers import write_model
from mini_llm_cuda_b200.model_file import ModelSpec, periodic_layer_types

pytestmark = pytest.mark.gpu

SPEC = ModelSpec(dim=128, layers=3, heads=2, head_dim=64, ffn_dim=256, ple_dim=32, vocab=512, max_context=128, rms_eps=1e-5,
                 layer_types=periodic_layer_types(3, 2), weight_dtype="bfloat16", kv_dtype="bfloat16")


@pytest.fixture(scope="module")
def api(built_lib):
    from mini_llm_cuda_b200 import api as _api
    return _api


def test_refused_session_leaves_the_others_alone(api, tmp_path):
    """A K/V pool of terabytes is refused; the next call of another session, whose launches ask the runtime for its last error,
    must not be blamed for it."""
    model = api.Model(write_model(tmp_path, SPEC, seed=81))
    sess = api.Session(model, 2)
    prompts = [[1, 2, 3], [4, 5]]
    sess.prefill(prompts)
    want = sess.decode(4)
    with pytest.raises(api.MlbError) as e:
        api.Session(model, 1, kv_pages=2 ** 31 - 1)
    assert e.value.status == api.MLB_E_NOMEM
    sess.prefill(prompts)
    assert np.array_equal(sess.decode(4), want)
    sess.close()
    model.close()
