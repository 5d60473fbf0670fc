"""Building the oracle where the reference's sources are missing."""
from oracle import oracle


def test_build_with_an_empty_reference_tree(tmp_path):
    oracle.build(ref_tree=str(tmp_path))
