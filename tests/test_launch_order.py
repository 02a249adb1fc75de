"""Source check (no GPU) of the rule that keeps stream order with programmatic dependent launches: a kernel lets its
successor start only after its own wait for its predecessor, so that whatever a kernel reads before its wait can be
stale only through its direct predecessor.  The activation quantisers alone do it first."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "gewell_b200" / "csrc"


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_successors_start_only_after_the_wait():
    sources = {path.name: code(path) for path in sorted(CSRC.iterdir())}
    common = sources.pop("common.cuh")
    body = re.search(r"void griddep_enter\(\) \{(.*?)\n\}", common, re.S).group(1)
    assert body.index("griddep_wait();") < body.index("griddep_launch();")
    for name, text in sources.items():
        assert "launch_dependents" not in text and "griddep_launch" not in text, name
        assert text.count("griddep_enter_first();") == (2 if name == "quant_kernels.cu" else 0), name


def test_every_programmatic_kernel_waits():
    """A kernel launched with the attribute enters; one launched with <<<>>> needs no wait."""
    checked = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = code(path)
        launches = re.findall(r"(?:launch_pdl(?:_shared)?|cudaLaunchKernelEx)\(.*?;", text, re.S)
        names = set(re.findall(r"\b\w+_kernel\b", " ".join(launches)))
        names |= {name for name in re.findall(r"const auto kernel = [^;]*;", text) for name in re.findall(r"\b\w+_kernel\b", name)}
        for name in names:
            start = re.search(r"__global__[^;{]*?\b%s\(" % name, text)
            assert start, f"{path.name}: {name}"
            body = text[start.start():]
            assert "griddep_enter" in body[:body.index("\n}\n")], f"{path.name}: {name}"
            checked += 1
    assert checked > 30
