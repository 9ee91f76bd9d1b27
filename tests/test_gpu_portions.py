"""Attention of prompt portions on tcgen05 tiles at the sizes where it can go wrong: edges of tiles (128 rows of tokens x
heads, 128 keys, 64 columns), windows and kept tokens that start and end inside a block of keys, one tile or two a CTA."""
import pytest

import bamudra_case
import nadilorn_case as case
from test_gpu_ragged import executor, run_cut

pytestmark = pytest.mark.gpu

# (heads, key heads, key size, value size, rotated, window): heads that divide a tile's rows and do not, columns that fill
# chunks of 64 and do not, values wider and narrower than keys, windows inside, at and beyond a block of keys
LAYERS = {
    "full": (4, 1, 128, 128, 64, 300), "half": (8, 8, 64, 64, 64, 129), "wide keys": (2, 2, 192, 128, 64, 128), "thirds": (6, 2, 72, 96, 24, 127),
    "odd": (5, 1, 44, 26, 20, 65), "many": (32, 2, 136, 40, 8, 1000), "one": (1, 1, 24, 120, 24, 1),
}
CUTS = ([300], [127, 1, 130, 42], [128, 172], [129, 2, 169], [33, 31, 64, 172], [1, 1, 298])


def check(module, config, tensors, plan_dir):
    ids = module.tokens(config, 300)
    want, _ = module.truth(config, tensors, ids)
    padded = any(layer["mixer"]["dim"] % 16 for layer in config["layers"])
    with executor(config, tensors, plan_dir, "bf16", max_wanted=512) as ex:
        for name, tensor in ex.state.items():
            if name.startswith("kv_pool"):
                tensor.fill_(3.0 if padded else float("nan"))      # (rows of used pages hold anything, columns behind a key's a number)
        for cuts in CUTS:
            assert case.error(run_cut(ex, ids, cuts), want) < case.TOLERANCE["bf16"], cuts


@pytest.mark.parametrize("name", sorted(LAYERS))
def test_windows_and_sizes(name, plan_dir):
    heads, kv_heads, dim, vdim, rot, window = LAYERS[name]
    config = case.model(96, 131, [case.layer(heads, kv_heads, dim, vdim, rot, window), case.layer(heads, kv_heads, dim, vdim, rot, 1000)])
    check(case, config, case.weights(config), plan_dir)


@pytest.mark.parametrize("window,keep", [(40, 5), (128, 128), (150, 200), (64, 1)])
def test_kept_tokens(window, keep, plan_dir):
    config = bamudra_case.model(96, 131, [bamudra_case.attention_layer(8, 2, 64, 32, window, keep), bamudra_case.attention_layer(3, 1, 128, 64, window, keep)])
    check(bamudra_case, config, bamudra_case.weights(config), plan_dir)


def test_two_tiles_a_cta(plan_dir):
    """Enough key heads that pairs of tiles fill the device."""
    config = case.model(64, 67, [case.layer(80, 80, 64, 64, 32, 200), case.layer(80, 80, 128, 72, 32, 500), case.layer(80, 80, 160, 128, 32, 70)])
    check(case, config, case.weights(config), plan_dir)
