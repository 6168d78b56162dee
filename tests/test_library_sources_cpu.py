"""The source lists of the libraries."""
from pisceslx_b200.ops import build


def test_every_source_is_listed_once_and_exists():
    for extra in ([], *build.FAMILIES.values()):
        names = (build.LAYERED_CUDA_SOURCES + extra if extra else build.CUDA_SOURCES)
        assert len(names) == len(set(names)) and all((build.CSRC / n).exists() for n in names)
