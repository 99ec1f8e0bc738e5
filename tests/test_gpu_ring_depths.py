"""The ring depth that a kernel runs with where the caller sets none, and a depth
that the caller sets."""
import pytest

pytestmark = pytest.mark.gpu


def kernel(pkg, kind, nk=57, ncol=4096):
    import torch
    B = kind or 1
    z = lambda n: torch.ones((n, ncol), dtype=torch.float64, device="cuda")  # noqa: E731
    seg = dict(kind=kind or pkg.TG_KIND_SCALAR, nk=nk, k2=nk, ncol=ncol, ld=ncol, a=z(nk * B * B), b=z(nk * B * B),
               c=z(nk * B * B), f=z(nk * B), x=z(nk * B))
    plan = pkg.Plan([seg], pkg.TG_PREC_F64)
    text = plan.describe()
    plan.close()
    return text.split(" ")[0]


@pytest.fixture
def settings(pkg):
    yield pkg
    for k in (2, 3):
        pkg.set_block_width(k, 0)
        pkg.set_column_residency(k, pkg.TG_PREC_F64, -1)
        pkg.set_pipeline(k, pkg.TG_PREC_F64, -1, 0)
    pkg.set_column_residency(pkg.TG_KIND_SCALAR, pkg.TG_PREC_F64, -1)
    pkg.set_pipeline(pkg.TG_KIND_SCALAR, pkg.TG_PREC_F64, -1, 0)


@pytest.mark.parametrize("kind", [2, 3])
@pytest.mark.parametrize("width", [16, 8])
@pytest.mark.parametrize("res", [0, 1])
def test_narrow_block_rings(settings, kind, width, res):
    pkg = settings
    pkg.set_block_width(kind, width)
    pkg.set_column_residency(kind, pkg.TG_PREC_F64, res)
    assert kernel(pkg, kind) == f"k_block_f64_ring<{kind},4,{width}{',1' if res else ''}>"
    pkg.set_pipeline(kind, pkg.TG_PREC_F64, 8, 0)
    if (kind, width, res) != (3, 16, 1):       # 8 levels are not built with Gamma of 3x3 blocks on chip in 16 columns
        assert kernel(pkg, kind) == f"k_block_f64_ring<{kind},8,{width}{',1' if res else ''}>"


@pytest.mark.parametrize("res", [1, 2])
def test_scalar_scratch_on_chip(settings, res):
    pkg = settings
    pkg.set_column_residency(pkg.TG_KIND_SCALAR, pkg.TG_PREC_F64, res)
    assert kernel(pkg, 0) == f"k_scalar_f64_res<2,4,{res - 1}>"
    pkg.set_pipeline(pkg.TG_KIND_SCALAR, pkg.TG_PREC_F64, 4, 0)
    assert kernel(pkg, 0) == f"k_scalar_f64_res<4,4,{res - 1}>"


def test_defaults(settings):
    pkg = settings
    assert kernel(pkg, 0) == "k_scalar_f64_chunk<3,4>"
    assert [kernel(pkg, k).startswith(f"k_block_f64_chunk<{k},") for k in (2, 3)] == [True, True]


@pytest.mark.parametrize("kind", [2, 3])
def test_columns_of_few_levels(settings, kind):
    pkg = settings
    depth = lambda nk: kernel(pkg, kind, nk, 4096)  # noqa: E731
    four, eight = depth(10), depth(11)
    assert four != eight and depth(1) == four and depth(57) == eight
    pkg.set_pipeline(kind, pkg.TG_PREC_F64, 4, 0)
    assert depth(57) == four
    pkg.set_pipeline(kind, pkg.TG_PREC_F64, 8, 0)
    assert depth(10) == eight


@pytest.mark.parametrize("kind,depth,name", [(2, 4, "2,2,2"), (2, 8, "2,4,2"), (2, 16, "2,8,2"), (3, 4, "3,4,1"), (3, 8, "3,4,2"),
                                             (3, 16, "3,8,2")])
def test_describe_names_the_kernel(settings, kind, depth, name):
    """The template's arguments, as a profiler's kernel filter takes them."""
    pkg = settings
    pkg.set_pipeline(kind, pkg.TG_PREC_F64, depth, 0)
    assert kernel(pkg, kind) == f"k_block_f64_chunk<{name}>"
