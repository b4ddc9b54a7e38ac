"""Rules of the kernel sources that no run shows: loads from global memory in inline assembly are volatile, 16-bit scalars
do not go through the __ldg overloads of cuda_fp16.h / cuda_bf16.h (asm statements that are not: the compiler may evaluate
either ahead of the bounds test in front of it), and kernels whose launch overlaps the one before them wait for its end
ahead of every access to global memory and keep off the read-only path."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "mflux_b200" / "csrc"
SOURCES = sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh"))
# Started by an ordinary launch, so that everything before them in the stream has finished.
ORDINARY = {"qmv_kernel", "decode_kernel", "qmm_t_kernel", "pack_scales_kernel", "interleave_codes_kernel",
            "widen_codes_kernel", "tp_fuse_kernel", "tp_signal_kernel", "tp_wait_kernel"}
READ_ONLY = re.compile(r"__ldg|__restrict__|\.nc\b|__ldc[asgv]\b")


def _code(src: Path) -> str:
    return re.sub(r"/\*.*?\*/", "", re.sub(r"//[^\n]*", "", src.read_text()), flags=re.S)


def _kernels(text: str):
    """(name, start, start of the body, end) of every kernel definition."""
    for m in re.finditer(r"__global__", text):
        head = re.compile(r"(\w+)\s*\((?=[^;{]*\)\s*\{)").finditer(text, m.end())
        name = next(h for h in head if not h.group(1).startswith("__") and h.group(1) != "launch_bounds")
        depth, i = 0, text.index("{", name.end())
        body = i
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield name.group(1), m.start(), body, i


def test_loads_in_assembly_are_volatile():
    found = 0
    for src in SOURCES:
        for m in re.finditer(r"asm\s*(volatile)?\s*\(\s*\"([^\"]*)", src.read_text()):
            if re.search(r"\bld(u)?\.(global|shared|weak|relaxed|acquire)|\bld\.param|prefetch", m.group(2)):
                found += 1
                assert m.group(1), f"{src.name}: {m.group(2)[:60]}"
    assert found


def test_no_16_bit_ldg():
    for src in SOURCES:
        assert not re.search(r"__ldg\((static_cast|reinterpret_cast)<const (__half|__nv_bfloat16)", src.read_text()), src.name


def test_ordinary_launches():
    """Whether a kernel is of the one kind or the other: a <<<>>> launch makes it an ordinary one."""
    names = {k[0] for src in SOURCES for k in _kernels(_code(src))}
    assert len(names) > 15 and ORDINARY <= names, ORDINARY - names
    for src in SOURCES:
        text = _code(src)
        for m in re.finditer(r"(\w+)(?:<[^;<>]*>)?<<<", text):
            if m.group(1) != "kern":
                assert m.group(1) in ORDINARY, m.group(1)
            else:   # the kernel of the last assignment in front of it
                kern = re.findall(r"auto kern = (.*?);", text[:m.start()], flags=re.S)[-1]
                assert set(re.findall(r"\w+_kernel", kern)) <= ORDINARY, kern
        for m in re.finditer(r"launch_overlapped\(([^,]+?),", text):
            assert not ORDINARY & set(re.findall(r"\w+_kernel", m.group(1))), m.group(1)


def test_overlapped_kernels_wait_before_they_touch_memory():
    """Ahead of the wait a kernel may use its parameters and indices, set up barriers, shared and tensor memory and fetch
    descriptors: no other call, no dereference."""
    setup = {"mbar_init", "fence_mbar_init", "tma_prefetch_desc", "tmem_alloc", "tmem_relinquish", "tmem_alloc_pair",
             "tmem_relinquish_pair", "tc_fence_before", "tc_fence_after", "__syncthreads", "cluster_sync_all",
             "cluster_ctarank", "smem_u32", "__align__", "if", "for"}
    waited = 0
    for src in SOURCES:
        text = _code(src)
        for name, _, body, end in _kernels(text):
            if name in ORDINARY:
                continue
            waited += 1
            assert text.count("wait_for_predecessor()", body, end) == 1, name
            before = text[body:text.index("wait_for_predecessor()", body)]
            before = re.sub(r"auto (\w+) = \[&\].*?\};", lambda m: setup.add(m.group(1)) or "", before, flags=re.S)
            calls = set(re.findall(r"(?<![\w>])([a-zA-Z_]\w*)\s*\(", before)) - setup
            assert not calls, f"{src.name}: {name}: {calls}"
            assert not re.search(r"\bp\.\w+\s*\[|->|(?<!volatile)\s\*\s*(reinterpret|static)_cast", before), name
    assert waited >= 12


def test_read_only_loads_stay_in_ordinary_kernels():
    """Nothing but the text of ordinary kernels names the read-only path: not the other kernels, and no helper, which they
    could call."""
    for src in SOURCES:
        text = _code(src)
        for name, start, _, end in sorted(_kernels(text), key=lambda k: -k[1]):
            if name in ORDINARY:
                text = text[:start] + text[end:]
        assert not READ_ONLY.search(text), f"{src.name}: {READ_ONLY.search(text).group()}"
