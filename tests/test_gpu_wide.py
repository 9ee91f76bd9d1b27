"""Products of long portions on tiles of 256 tokens, a CTA taking several tiles in turn: remainders of both sides, one and
many tiles a CTA, every kind of epilogue, experts with fewer rows than a tile and with more."""
import pytest

import bamudra_case
import benarax_case
import nadilorn_case
from test_gpu_ragged import executor, run_cut
from tilemega_b200.serving.ragged import Portion

pytestmark = pytest.mark.gpu


def check(module, config, tensors, plan_dir, cuts, length=530):
    ids = module.tokens(config, length)
    want, _ = module.truth(config, tensors, ids)
    with executor(config, tensors, plan_dir, "bf16", capacity=640, max_rows=640, max_wanted=640) as ex:
        for sizes in cuts:
            assert module.error(run_cut(ex, ids, sizes), want) < module.TOLERANCE["bf16"], sizes


@pytest.mark.parametrize("vocab,ff", [(20011, 9000), (45000, 15300)])
def test_store_unit_and_head(vocab, ff, plan_dir):
    """Projections of 80 heads, a wide gated unit, a vocabulary of up to ten tiles a CTA; rows that fill two tiles, nearly and not at all."""
    case = nadilorn_case
    config = case.model(96, vocab, [case.layer(80, 80, 32, 48, 32, 200, case.dense(ff))])
    check(case, config, case.weights(config), plan_dir, ([512, 18], [257, 256, 17], [129, 401]))


def test_sums_into_the_stream(plan_dir):
    """A stream so wide that outputs are added to it by wide tiles (with a bias)."""
    case = bamudra_case
    config = case.model(7704, 131, [case.attention_layer(4, 2, 64, 32, 100, 3, mlp=case.mlp(80, 1.5))])
    check(case, config, case.weights(config), plan_dir, ([300], [257, 43]), length=300)


def test_rotation(plan_dir):
    """Latent attention whose queries turn on their way out, for enough heads."""
    case = benarax_case
    config = case.model(96, 131, [case.latent(60, 120, 40, 40, 130, 72), case.latent(60, 96, 64, 24, 260, 40, neighbours=False)], groups=2, taps=3)
    check(case, config, case.weights_for(config, "bf16"), plan_dir, ([512, 18], [300, 230]))


def test_products_by_heads(plan_dir):
    """Latent attention whose latent rows are small enough that portions are not expanded: every row's queries and values pass through
    products by heads, of 128 rows a head, 200 and 48. And one of 308 rows a head, where only a decoded token beside the portion does."""
    case = benarax_case
    config = case.model(96, 131, [case.latent(64, 64, 8, 128, 40, 24), case.latent(32, 56, 8, 200, 40, 24, neighbours=False), case.latent(24, 40, 8, 72, 300, 24)],
                        groups=2)
    tensors = case.weights_for(config, "bf16")
    check(case, config, tensors, plan_dir, ([512, 18], [300, 230]))
    single, portion = case.tokens(config, 41, seed=3), case.tokens(config, 530, seed=4)
    with executor(config, tensors, plan_dir, "bf16", capacity=640, max_rows=640, max_wanted=640) as ex:
        slots = ex.open(), ex.open()
        ex.run([Portion(slots[0], single[:40])])
        logits = ex.run([Portion(slots[0], single[40:], [0]), Portion(slots[1], portion, list(range(530)))])
    assert case.error(logits[:1], case.truth(config, tensors, single)[0][40:]) < case.TOLERANCE["bf16"]
    assert case.error(logits[1:], case.truth(config, tensors, portion)[0]) < case.TOLERANCE["bf16"]


def test_pairs_that_would_take_a_round_more(plan_dir):
    """49 tiles of weight rows by three of tokens: single CTAs, for the gated unit and the head, a stream's sums, and rotated queries."""
    case = nadilorn_case
    config = case.model(96, 6272, [case.layer(4, 2, 32, 32, 16, 90, case.dense(3136))])
    check(case, config, case.weights(config), plan_dir, ([530],))
    case = bamudra_case
    config = case.model(6272, 131, [case.attention_layer(4, 2, 64, 32, 100, 3, mlp=case.mlp(80, 1.5))])
    check(case, config, case.weights(config), plan_dir, ([530],))
    case = benarax_case
    config = case.model(96, 131, [case.latent(56, 80, 32, 40, 130, 72)], groups=2)
    check(case, config, case.weights_for(config, "bf16"), plan_dir, ([530],))


@pytest.mark.parametrize("side", [5100, 6272])
def test_side_inputs(side, plan_dir):
    """Parts of the second embedding so wide that their gate runs on wide tiles, by pairs of CTAs and by single ones."""
    case = benarax_case
    config = case.model(96, 131, [case.latent(4, 32, 16, 32, 64, 48)], groups=2, side=side)
    check(case, config, case.weights_for(config, "bf16"), plan_dir, ([530],))


@pytest.mark.parametrize("module", [nadilorn_case, benarax_case], ids=["input weighted", "output weighted"])
@pytest.mark.parametrize("experts,top", [(3, 2), (5, 1), (2, 2), (7, 3)])
def test_experts_of_many_rows(module, experts, top, plan_dir):
    """About 100 to 530 rows an expert: tiles of 256 rows not full, just over one, two and more."""
    mlp = module.moe(experts, top, 300)
    if module is nadilorn_case:
        config = module.model(264, 131, [module.layer(4, 2, 32, 32, 16, 90, mlp)])
    else:
        config = module.model(264, 131, [module.latent(4, 32, 16, 32, 64, 48, mlp)], groups=2)
    check(module, config, module.weights_for(config, "bf16"), plan_dir, ([530], [300, 230]))


# (experts, top, their gate and up rows together, or the up rows) whose products take tiles of 256 rows for 530 tokens of width 2056, as
# test_linear_rules.py checks: less than a tile an expert, and just over one
WIDE_EXPERTS = [(8, 2, 1800), (4, 2, 3000)]


@pytest.mark.parametrize("module", [nadilorn_case, benarax_case], ids=["input weighted", "output weighted"])
@pytest.mark.parametrize("experts,top,rows", WIDE_EXPERTS)
def test_experts_on_wide_tiles(module, experts, top, rows, plan_dir):
    if module is nadilorn_case:
        config = module.model(2056, 131, [module.layer(4, 2, 32, 32, 16, 90, module.moe(experts, top, rows))])
    else:
        config = module.model(2056, 131, [module.latent(4, 32, 16, 32, 64, 48, module.moe(experts, top, rows // 2))], groups=2)
    check(module, config, module.weights_for(config, "bf16"), plan_dir, ([530],))
