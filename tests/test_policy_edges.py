"""The rule that chooses between the two tensor-core forms, at its edges, on both sides of the library boundary."""
import pytest

from actlizela_b200 import device, sm100_policy

B200 = device.DeviceProfile("NVIDIA B200", 148, (10, 0))


@pytest.mark.parametrize("shape,family", [((1, 192, 2, 4), "fused"), ((1, 193, 2, 4), "umma"), ((1, 449, 9, 63), "umma"),
                                          ((1, 449, 16, 64), "fused"), ((1, 64 * 319, 2, 4), "umma"), ((1, 64 * 319 + 1, 2, 4), "fused"),
                                          ((31, 64 * 41, 1, 1), "umma"), ((31, 64 * 41 + 1, 1, 1), "fused")])
def test_family_rule(shape, family, native_library):
    choice = sm100_policy.select((*shape, 128, 128), B200)
    assert choice.configuration == family and choice.segments == 1
    assert native_library.lib.actlize_la_sm100_select(*shape, 1) == choice.configuration_id


def test_rows_say_what_the_rule_says():
    """The measured rows and the rule for all other shapes cannot drift apart."""
    for row in sm100_policy.policy()["rows"]:
        b, t, _, hv = row["shape"]
        assert row["configuration"] == sm100_policy.default_configuration(b, t, hv)
        assert row["parallel"] == sm100_policy.default_parallel(b, t, hv) and row["segments"] == 1
