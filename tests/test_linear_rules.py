"""The rules that cut a ragged step's products into tiles (tilemega_b200/csrc/linear_rules.h), compiled for the host."""
import shutil
import subprocess
from pathlib import Path

import pytest

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
