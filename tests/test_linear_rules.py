"""The rules that cut a ragged step's products into tiles (tilemega_b200/csrc/linear_rules.h), compiled for the host."""
import shutil
import subprocess
from pathlib import Path

import pytest

from test_gpu_wide import WIDE_EXPERTS

ROOT = Path(__file__).resolve().parents[1]
SMS = 148


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    binary = tmp_path_factory.mktemp("rules") / "linear_rules"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{ROOT / 'tilemega_b200' / 'csrc'}", str(ROOT / "tests" / "linear_rules.cpp"), "-o", str(binary)], check=True)

    def ask(lines):
        text = subprocess.run([str(binary)], input="\n".join(" ".join(map(str, line)) for line in lines), capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in text.splitlines()]

    return ask


def rounds(tiles, at_once):
    return -(-tiles // at_once)


def test_pairs_of_ctas_never_take_a_round_more(rules):
    asked = [("linear", t, n, 0, 32, SMS) for t in (129, 256, 300, 513, 769, 1000, 1500, 2048) for n in range(128, 30000, 392)]
    wide = 0
    for (_, t, n, _, _, _), (index, splits, pair) in zip(asked, rules(asked)):
        tokens, single = -(-t // 256), rounds(-(-n // 128) * -(-t // 256), SMS)
        paired = rounds(-(-n // 256) * tokens, SMS // 2)
        assert (index == 4) == (-(-n // 128) * tokens * 10 >= SMS * 8) and (index < 4 or splits == 1)
        if index == 4:
            wide += 1
            assert pair == (paired <= single), (t, n)
    assert wide > 100


@pytest.mark.parametrize("n", [64, 128, 200, 256, 320, 384, 576])
def test_products_by_heads_stay_with_single_ctas(rules, n):
    """A pair would take 256 rows of one head, 128 of them for nothing where the head has no more."""
    asked = [("linear", t, n, heads, 5, SMS) for t in (129, 700, 1024, 1800, 2048) for heads in (4, 16, 32, 64)]
    for (_, t, _, heads, _, _), (index, _, pair) in zip(asked, rules(asked)):
        assert not pair
        assert (index == 4) == (heads * -(-n // 128) * -(-t // 256) * 10 >= SMS * 8)


def test_experts_take_the_wider_tiles_only_where_they_end_sooner(rules):
    """(experts, their rows, slots) with both widths measured at 2048 columns: those whose difference is more than a twentieth."""
    narrow = [(8, 512, 1000), (8, 1024, 4000), (32, 768, 4000)]
    wide = [(128, 1152, 16384), (32, 768, 8000), (16, 2048, 2000), (16, 1024, 2000), (8, 2048, 1000), (8, 4096, 1000)]
    asked = [("experts", slots, experts, ff, 2048, ff) for experts, ff, slots in narrow + wide]
    assert [rows for rows, _, _ in rules(asked)] == [128] * len(narrow) + [256] * len(wide)


def test_experts_of_the_wide_tests_are_wide(rules):
    asked = [("experts", 530 * top, experts, rows, 2056, ff) for experts, top, rows in WIDE_EXPERTS for ff in (rows, rows // 2)]
    assert {rows for rows, _, _ in rules(asked)} == {256}


def test_few_tiles_of_experts_are_split_over_k(rules):
    """Many rows for few experts with few weight rows: 128-row tiles, K in parts, not a fifth of the SMs busy."""
    (rows, index, splits), = rules([("experts", 1000, 8, 512, 2048, 512)])
    assert (rows, index) == (128, 3) and splits > 1


def test_few_slots_of_an_expert_take_tiles_as_before(rules):
    asked = [("experts", share * 16, 16, 1024, 2048, 1024) for share in (1, 9, 12, 13, 24, 25, 48, 49, 96)]
    assert [rows for rows, _, _ in rules(asked)] == [16, 16, 16, 32, 32, 64, 64, 128, 128]
