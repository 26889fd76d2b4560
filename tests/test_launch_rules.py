"""CPU check of the rule that takes the FP32K sums to the shape without a register bound
(csrc/interact32.cuh, few_waves32), evaluated as written: on 152 SMs it takes that shape at the
sizes where the step was measured faster with it, and leaves it where slower, without and with
the learned warm start in the epilogue."""
import re
from pathlib import Path

SOURCE = (Path(__file__).resolve().parents[1] / "sph_fem_2d_cutting_gpu_gb300" / "csrc" / "interact32.cuh").read_text()


def chosen(n, mlp):
    body = re.search(r"inline bool few_waves32\(int N\) \{(.*?)\n\}", SOURCE, re.S).group(1)
    names = {"N": n, "kMlp": mlp, "sm_count": lambda: 152, "div_up": lambda a, b: -(-a // b)}
    for statement in re.sub(r"//.*", "", body).replace("\n", " ").split(";"):
        code = statement.strip().replace("&&", " and ").replace("||", " or ").replace(" / ", " // ")
        if code.startswith("if (kMlp) return"):
            if mlp:
                return bool(eval(code[len("if (kMlp) return"):].strip(), {}, names))
        elif code.startswith("return"):
            return bool(eval(code[len("return"):].strip(), {}, names))
        elif code.startswith("const int"):
            for part in code[len("const int"):].split(","):
                name, value = part.split("=")
                names[name.strip()] = eval(value.strip(), {}, names)
    raise AssertionError("no rule")


def test_plain_sums():
    for n in (1_600, 12_000, 90_000, 96_100, 132_496, 160_000, 193_600, 250_000, 270_400, 291_600):
        assert chosen(n, False), n
    for n in (99_225, 105_625, 115_600, 202_500, 215_296, 230_400, 313_600, 336_400, 422_500, 4_194_304):
        assert not chosen(n, False), n


def test_with_the_warm_start():
    for n in (1_600, 12_000, 22_500, 38_809):
        assert chosen(n, True), n
    for n in (40_000, 62_500, 90_000, 160_000, 250_000, 291_600, 640_000):
        assert not chosen(n, True), n
