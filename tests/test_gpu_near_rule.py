"""Who walks the near-first trees (orn_near_trees): the kernels for which they
are the faster ones.  And what each kernel renders on them is what a counting
render, which walks the blob's trees, does."""
import numpy as np
import pytest

from zig_ornament_gb300 import _lib, ornament, scenes

pytestmark = pytest.mark.gpu

RAYS, BATCH, MEGA, WAVE = 1, 2, 3, 4


def _instanced(n_blas, n_instances, triangles):
    return scenes.instanced_meshes_scene(96, 54, seed=5, n_blas=n_blas, n_instances=n_instances,
                                         tri_range=(0.9 * triangles, 1.1 * triangles), n_textures=2, texture_size=16)


def _on_ground(scene):
    scene.attachSphere(scene.createSphere((0, -3060, 0, 1), 3000.0, scene.lambertian((0.5, 0.5, 0.5, 1))))
    return scene


@pytest.mark.parametrize("scene,builder,who", [
    (lambda: _instanced(1, 4, 60), "reference", RAYS),         # a handful of visits
    (lambda: _instanced(1, 4, 60), "sah", RAYS),
    (lambda: _instanced(1, 16, 200), "reference", BATCH),      # more visits than with new trees, but few
    (lambda: _instanced(1, 16, 200), "sah", RAYS),
    (lambda: _instanced(2, 64, 1500), "reference", MEGA),      # many visits, and half again as many
    (lambda: _instanced(2, 64, 1500), "sah", RAYS),            # trees as good
    (lambda: _instanced(2, 64, 1500), "lbvh", RAYS),
    (lambda: _instanced(4, 128, 40_000), "reference", WAVE),
    (lambda: _instanced(4, 128, 40_000), "lbvh", RAYS),
    (lambda: _on_ground(_instanced(1, 16, 200)), "sah", MEGA), # little to walk: shading counts
    (scenes.spheres_scene, "reference", MEGA),                 # nothing of it in meshes
    (scenes.spheres_scene, "sah", MEGA),
    (scenes.cornell_box_scene, "reference", MEGA),
    (lambda: scenes.small_test_scene(96, 64), "sah", MEGA)])
def test_who_walks_them(scene, builder, who):
    r = ornament.Renderer(ornament.Bvh(scene(), builder=builder), device=0)
    got = r.near_trees()
    r.close()
    assert got == who


@pytest.mark.parametrize("semantics", [_lib.SEMANTICS_HIP, _lib.SEMANTICS_WGSL], ids=["hip", "wgsl"])
@pytest.mark.parametrize("scene", [lambda: _instanced(4, 128, 20_000), scenes.spheres_scene,
                                   lambda: _on_ground(_instanced(1, 16, 200))], ids=["instanced", "spheres", "ground"])
def test_pictures(scene, semantics):
    s = scene()
    bvh = ornament.Bvh(s)
    state = ornament.State()
    state.setDepth(8)
    state.setIterations(5)
    state.semantics = semantics
    frames = []
    for kernel, count in ((_lib.KERNEL_MEGA, True), (_lib.KERNEL_MEGA, False), (_lib.KERNEL_WAVEFRONT, False),
                          (None, False)):
        r = ornament.Renderer(bvh, device=0)
        assert r.near_trees() >= MEGA
        if kernel is not None:
            state.kernel = kernel
        r.set_state(state.to_struct())
        r.set_resolution(83, 47)
        r.set_camera(s.camera.to_struct())
        r.enable_counters(count)
        if kernel is not None:
            r.render()
        else:
            batch = ornament.Batch([r])
            batch.render()
            batch.synchronize()
            batch.close()
        acc, rng, _ = r.progress()
        frames.append((acc.view(np.uint32), rng, r.framebuffer().view(np.uint32)))
        r.close()
    for got in frames[1:]:
        for a, b in zip(frames[0], got):
            assert np.array_equal(a, b)
