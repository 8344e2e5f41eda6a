"""Materials packed with one call give the bytes that setting each field gives,
whatever the fields hold, and what was refused stays refused."""
import ctypes as C
import dataclasses

import numpy as np
import pytest

from shiro_gb300 import Material
from shiro_gb300.abi import MarshalledScene, MaterialDesc, Scene

INF, NAN = float("inf"), float("nan")
MATERIALS = {
    "defaults": Material(),
    "values": Material(base_color=(0.1, -0.0, 1e-45), roughness=1 / 3, thin_walled=True, has_normal_override=True,
                       normal_override=(0.0, 1.0, 0.0)),
    "numpy": Material(base_color=tuple(np.array([0.1, 0.2, 0.3])), emission_color=(np.float32(0.7),) * 3,
                      ior=np.float64(1.4), metallic=np.float16(0.25), opacity=np.float32(1)),
    "whole numbers": Material(base_color=(1, 0, 2), emission_strength=3, opacity=True),
    "short triples": Material(base_color=(0.5,), coat_color=(), sheen_color=(0.25, 0.5)),
    "past a float": Material(base_color=(1e39, -1e300, 3.4028235677973366e38), emission_strength=1e40),
    "special values": Material(base_color=(INF, -INF, NAN), roughness=NAN),
    "text": Material(roughness="0.25", base_color=("0.1", 0.2, 0.3)),
}


def _bytes(material):
    ms = MarshalledScene(Scene(materials=[Material(), material]))
    return C.string_at(C.addressof(ms.desc.materials[1]), C.sizeof(MaterialDesc))


@pytest.mark.parametrize("name", list(MATERIALS))
def test_packed_bytes_are_the_fields_bytes(name):
    desc = MATERIALS[name].to_desc()
    assert _bytes(MATERIALS[name]) == C.string_at(C.addressof(desc), C.sizeof(desc))


@pytest.mark.parametrize("kw", [dict(base_color=(1.0, 2.0, 3.0, 4.0)), dict(base_color=0.5), dict(base_color=[0.1, 0.2, 0.3]),
                                dict(base_color=np.array([0.1, 0.2, 0.3])), dict(base_color=("a", "b", "c")),
                                dict(roughness=None), dict(thin_walled=0.5), dict(thin_walled=1),
                                dict(has_normal_override=np.int32(1)), dict(thin_walled=2**32 + 3)], ids=str)
def test_refused_values_stay_refused(kw):
    material = Material(**kw)
    with pytest.raises(Exception) as fields:
        material.to_desc()
    with pytest.raises(type(fields.value)):
        MarshalledScene(Scene(materials=[material]))


def test_a_material_that_describes_itself():
    """Other types than Material are asked for their descriptor."""

    @dataclasses.dataclass
    class Tinted(Material):
        tint: float = 0.5

        def to_desc(self):
            return dataclasses.replace(Material(), base_color=tuple(self.tint * c for c in self.base_color)).to_desc()

    class Bare:
        def to_desc(self):
            return Material(roughness=0.75).to_desc()

    for m in (Tinted(base_color=(0.2, 0.4, 0.6)), Bare()):
        desc = m.to_desc()
        assert _bytes(m) == C.string_at(C.addressof(desc), C.sizeof(desc))
