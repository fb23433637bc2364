"""The C-ABI library loads without a GPU and exports every symbol include/inpc_b200.h declares;
argument validation that needs no device works."""
import ctypes as C
import re
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def _declared():
    text = (ROOT / "include" / "inpc_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    names = set(re.findall(r"\b(inpc_[a-z0-9_]+)\s*\(", text))
    names -= {"inpc_alloc_fn"}
    return sorted(names)


def test_header_declares_the_expected_surface():
    names = _declared()
    for must in ("inpc_rasterize_forward", "inpc_rasterize_backward", "inpc_render", "inpc_render_preextracted",
                 "inpc_generate_training_samples", "inpc_generate_samples", "inpc_generate_expected_samples_count",
                 "inpc_compute_viewpoint_weights", "inpc_sort_pairs", "inpc_weight_decay_grads", "inpc_spherical_contraction",
                 "inpc_cauchy_loss", "inpc_cauchy_loss_backward"):
        assert must in names


def test_library_exports_every_declared_symbol():
    from inpc_b200 import _build, _cabi
    _build.build()
    handle = C.CDLL(str(_cabi.LIB_PATH))
    missing = [n for n in _declared() if not hasattr(handle, n)]
    assert not missing, f"declared in include/inpc_b200.h but not exported: {missing}"
    # and the binding declares a prototype for each of them
    unbound = [n for n in _declared() if n not in _cabi.PROTOTYPES]
    assert not unbound, f"no ctypes prototype for: {unbound}"


def test_every_declaration_cites_the_reference():
    text = (ROOT / "include" / "inpc_b200.h").read_text()
    # every documented entry point names a reference file:line (or says it has no counterpart)
    blocks = re.findall(r"/\*(.*?)\*/\s*(?:size_t|int|uint64_t|void|long long|const char\*|inpc_sampler\*)\s+(inpc_[a-z0-9_]+)\s*\(", text, flags=re.S)
    assert len(blocks) >= 15
    for comment, name in blocks:
        assert re.search(r"\.(h|cu|cuh|py|cpp):\d+", comment) or "no counterpart" in comment or name in (
            "inpc_version", "inpc_launch_count", "inpc_sampler_get_counter", "inpc_sampler_workspace_bytes"), name


@pytest.mark.parametrize("name", ["inpc_sort_workspace_bytes", "inpc_morton_workspace_bytes", "inpc_sampler_workspace_bytes"])
def test_a_workspace_for_more_serves_fewer(name):
    """A caller sizes one workspace for its largest n: the size must not fall as n grows, in particular not where the sort
    goes over to larger tiles (2^18 pairs)."""
    from inpc_b200 import _cabi
    size = getattr(_cabi.lib(), name)
    edge = 1 << 18
    ns = sorted({1, 2, 100, 2047, 2048, 2049, 8192, 100_003, 200_000, edge - 2049, edge - 1, edge, edge + 1, edge + 8192, 300_000, 500_000,
                 3 * edge, 4 * edge - 1, 4 * edge, 4 * edge + 1, 5 * edge, 1 << 22, 1 << 23} | {edge + 2048 * k for k in range(-8, 40)})
    if name == "inpc_sampler_workspace_bytes":
        ns = [n for n in ns if n <= 1 << 22]
    sizes = [int(size(n)) for n in ns]
    fell = [(a, b) for (a, x), (b, y) in zip(zip(ns, sizes), zip(ns[1:], sizes[1:])) if y < x]
    assert not fell, f"{name} falls between {fell}"


def test_host_side_validation_without_gpu():
    from inpc_b200 import _cabi
    L = _cabi.lib()
    assert L.inpc_version() >= 100
    assert L.inpc_sort_workspace_bytes(1 << 20) > 0
    assert L.inpc_sampler_workspace_bytes(1 << 18) > 2 * 4 * (1 << 18)
    assert L.inpc_cauchy_workspace_bytes(10) > 0
    assert L.inpc_sort_pairs(None, None, None, None, 10, 99, None, None, None) == -1
    assert b"end_bit" in L.inpc_last_error()
    h = L.inpc_sampler_create(7)
    assert h
    L.inpc_sampler_set_counter(h, 41)
    assert L.inpc_sampler_get_counter(h) == 41
    L.inpc_sampler_destroy(h)
    with pytest.raises(_cabi.InpcError):
        _cabi.check(-1)


def test_failed_launches_are_reported_under_the_name_of_their_kernel():
    sources = "".join(p.read_text() for p in sorted((ROOT / "inpc_b200" / "csrc").glob("*.cu")))
    kernels = set(re.findall(r"\b(\w+_kernel)\s*\(", sources))
    named = [name for check in re.findall(r"INPC_LAUNCH_CHECK\((.*)\);", sources) for name in re.findall(r'"([^"]*)"', check)]
    assert len(named) > 40 and not [name for name in named if name not in kernels]


def test_product_never_touches_the_oracle():
    """The package must not import, load or execute anything under oracle/ (no CPU fallback)."""
    for path in (ROOT / "inpc_b200").rglob("*"):
        if path.suffix in (".py", ".cu", ".cuh", ".h") and "_obj" not in path.parts:
            text = path.read_text()
            assert "oracle" not in text.lower(), f"{path} mentions the oracle"


@pytest.mark.parametrize("leaves", [4096, 100_003, 1 << 18, 1 << 20, 1 << 22, 1 << 24])
def test_sampler_workspace_is_no_larger_than_its_largest_call(leaves):
    """A training view takes one per step and stream.  No call needs more than a CDF, a weight, a 16-byte record, a count and an
    offset per leaf, and a guide of 32-byte records, at most 2^20 and one per leaf rounded up to a power of two."""
    from inpc_b200 import _cabi
    buckets = min(1 << 20, 1 << (leaves - 1).bit_length())
    assert _cabi.lib().inpc_sampler_workspace_bytes(leaves) <= 32 * leaves + 32 * buckets + leaves // 64 + 8192
