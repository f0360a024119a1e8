// The mesh build (st_update_mesh_bvh) on the stand-in runtime; one scenario a process.
#include <cstdio>
#include <cstring>
#include <vector>
#include "runtime.h"
#include "slimtracin_b200.h"

namespace st {
int batch_blocks_per_sm(int) { return 7; }       // (st_render.cu is not linked)
}

#define EXPECT(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

// A mesh of `n` triangles over four vertices, its arrays for the build's results.
struct MeshArrays {
    std::vector<vec3> positions, normals;
    std::vector<TriangleVertexIndices> ids;
    std::vector<Triangle> triangles;
    std::vector<BVHNode> nodes;
    std::vector<u32> leaf_ids;
    Mesh mesh;
    explicit MeshArrays(u32 n) : positions(4), normals(4), ids(n), triangles(n), nodes(2 * n), leaf_ids(n) {
        memset(&mesh, 0, sizeof(mesh));
        mesh.triangle_count = n;
        mesh.vertex_count = mesh.normals_count = 4;
        mesh.vertex_positions = positions.data();
        mesh.vertex_normals = normals.data();
        mesh.vertex_position_indices = mesh.vertex_normal_indices = ids.data();
        mesh.triangles = triangles.data();
        mesh.bvh.nodes = nodes.data();
        mesh.bvh.leaf_ids = leaf_ids.data();
        mesh.bvh.node_count = 77;
    }
};

// A launch that is refused fails the build, and nothing after it reads what it should have made.
static int refused_launch(st_ctx *ctx, const char *kernel, const char *must_not_follow) {
    MeshArrays a(5000);
    for (int mode : {ST_BVH_BINNED_SAH, ST_BVH_LBVH30}) {
        fake.log.clear();
        fake.refuse_kernel = kernel;
        EXPECT(st_update_mesh_bvh(ctx, &a.mesh, mode) == ST_ERR_CUDA);
        EXPECT(a.mesh.bvh.node_count == 77);
        EXPECT(!*must_not_follow || fake.log.find(must_not_follow) == std::string::npos);
        fake.refuse_kernel.clear();
        EXPECT(st_update_mesh_bvh(ctx, &a.mesh, mode) == ST_OK);
        a.mesh.bvh.node_count = 77;
    }
    return 0;
}

// An allocation that one call is refused, wherever it is, is that call's error and no later one's.
static int refused_allocation(st_ctx *ctx) {
    const size_t all = fake.device_bytes;
    for (u32 n : {2000u, 5000u, 40000u}) {           // (larger each time, so that the builder's scratch grows)
        MeshArrays a(n);
        for (size_t room : {(size_t)1000, (size_t)40 * n, (size_t)300 * n, (size_t)1 << 20}) {
            fake.device_bytes = fake.device_held + room;
            const int r = st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_BINNED_SAH);
            EXPECT(r == ST_OK || r == ST_ERR_OUT_OF_MEMORY);
            fake.device_bytes = all;
            if (r == ST_OK) break;
        }
        EXPECT(st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_LBVH30) == ST_OK);
    }
    return 0;
}

// A scene of n boxes, their TLAS, and one mesh of n triangles, each tree one split and two leaves; `extra`
// nodes more, which no other leads to.
struct SceneArrays {
    std::vector<Primitive> prims;
    std::vector<Material> materials;
    std::vector<BVHNode> nodes;
    std::vector<u32> ids;
    MeshArrays mesh;
    Scene scene;
    SceneArrays(u32 n, u32 extra) : prims(n), materials(1), nodes(3 + extra), ids(n), mesh(n) {
        memset(&scene, 0, sizeof(scene));
        for (u32 i = 0; i < n; i++) {
            prims[i].type = PrimitiveType_Box;
            ids[i] = i;
        }
        nodes[0].first_child_id = 1;
        nodes[1].child_count = 1;
        nodes[2].first_child_id = 1;
        nodes[2].child_count = (u16)(n - 1);
        for (u32 k = 3; k < 3 + extra; k++) nodes[k] = nodes[1];
        mesh.mesh.bvh.nodes = scene.bvh.nodes = nodes.data();
        mesh.mesh.bvh.node_count = scene.bvh.node_count = 3 + extra;
        mesh.mesh.bvh.height = scene.bvh.height = 1;
        mesh.mesh.bvh.leaf_ids = scene.bvh.leaf_ids = ids.data();
        scene.primitives = prims.data();
        scene.materials = materials.data();
        scene.meshes = &mesh.mesh;
        scene.settings.primitives = n;
        scene.settings.materials = scene.settings.meshes = 1;
    }
};

// A tree with more nodes than a tree over its items has, and the library has room for, is refused.
static int oversized_trees(st_ctx *ctx) {
    for (u32 n : {2u, 3u, 700u}) {
        for (u32 extra : {0u, 2 * n - 3, 2 * n - 2, 2 * n, 40 * n}) {
            SceneArrays a(n, extra);
            const bool fits = 3 + extra <= 2 * n, pairs_fit = (2 + extra) / 2 <= n;
            EXPECT(st_upload_scene(ctx, 0, &a.scene) == ST_OK);
            EXPECT(st_upload_mesh_bvhs(ctx, 0, &a.scene) == (pairs_fit ? ST_OK : ST_ERR_BAD_SCENE));
            EXPECT(st_upload_scene_bvh(ctx, 0, &a.scene) == (fits ? ST_OK : ST_ERR_BAD_SCENE));
            EXPECT(fake.out_of_range == 0);
            EXPECT(st_free_scene(ctx, 0) == ST_OK);
        }
    }
    return 0;
}

// What a build takes for its own time is within the budget, the binned builder's scratch too, and so is
// what is kept of it; it is reported, and given back for memory that stays and for serving.
static int budget() {
    const size_t MB = (size_t)1 << 20;
    st_ctx *ctx = nullptr;
    st_config cfg = {};
    cfg.memory_budget = 30 * MB;
    EXPECT(st_init(&ctx, &cfg) == ST_OK);
    const uint64_t empty = st_device_bytes_in_use(ctx);
    MeshArrays a(100000);                              // 23 MB, and 18 of scratch
    EXPECT(st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_BINNED_SAH) == ST_ERR_BUDGET);
    EXPECT(a.mesh.bvh.node_count == 77);
    std::vector<float> boxes(6 * 200000);
    std::vector<u32> order(200000);
    std::vector<BVHNode> nodes(400000);
    u32 info[2];
    EXPECT(st_build_bvh(ctx, ST_BVH_BINNED_SAH, boxes.data(), 200000, 2, nullptr, order.data(), nodes.data(), info) == ST_ERR_BUDGET);
    EXPECT(st_build_bvh(ctx, ST_BVH_LBVH30, boxes.data(), 200000, 2, nullptr, order.data(), nodes.data(), info) == ST_OK);
    EXPECT(st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_LBVH30) == ST_OK);
    EXPECT(st_device_bytes_in_use(ctx) > empty + 20 * MB && st_device_bytes_in_use(ctx) <= 30 * MB);
    // a scene takes the room that was kept, and leaves the builds what it does not need
    SceneArrays s(20000, 0);                           // 12 MB with its mesh of as many triangles
    EXPECT(st_upload_scene(ctx, 0, &s.scene) == ST_OK);
    EXPECT(st_upload_mesh_bvhs(ctx, 0, &s.scene) == ST_OK);
    EXPECT(st_upload_scene_bvh(ctx, 0, &s.scene) == ST_OK);
    EXPECT(st_device_bytes_in_use(ctx) <= 30 * MB);
    EXPECT(st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_LBVH30) == ST_ERR_BUDGET);
    EXPECT(st_update_mesh_bvh(ctx, &s.mesh.mesh, ST_BVH_LBVH30) == ST_OK);
    EXPECT(st_device_bytes_in_use(ctx) <= 30 * MB);
    EXPECT(st_free_scene(ctx, 0) == ST_OK);
    EXPECT(st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_LBVH30) == ST_OK);
    // serving has what no scene holds for its frames
    st_serve_config serve = {};
    serve.frame_budget = 2 * MB;
    EXPECT(st_serve_start(ctx, &serve) == ST_OK);
    EXPECT(st_device_bytes_in_use(ctx) < 3 * MB);
    EXPECT(st_serve_stop(ctx) == ST_OK);
    st_shutdown(ctx);
    EXPECT(fake.device_held == 0);
    return 0;
}

// Memory that is only kept is no reason to refuse a call: not the builders' scratch, nor a scene's arrays,
// nor a transient block.
static int kept_memory(st_ctx *ctx) {
    MeshArrays a(100000), b(150000);
    EXPECT(st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_BINNED_SAH) == ST_OK);     // 41 MB kept
    const size_t all = fake.device_bytes, MB = (size_t)1 << 20;
    fake.device_bytes = fake.device_held + 4 * MB;
    std::vector<float> boxes(6 * 150000);
    std::vector<u32> order(150000);
    std::vector<BVHNode> nodes(300000);
    u32 info[2];
    EXPECT(st_build_bvh(ctx, ST_BVH_LBVH30, boxes.data(), 150000, 2, nullptr, order.data(), nodes.data(), info) == ST_OK);
    fake.device_bytes = fake.device_held + 25 * MB;
    EXPECT(st_update_mesh_bvh(ctx, &a.mesh, ST_BVH_LBVH30) == ST_OK);
    fake.device_bytes = fake.device_held + 4 * MB;
    SceneArrays s(20000, 0);                                                  // 12 MB
    EXPECT(st_upload_scene(ctx, 0, &s.scene) == ST_OK);
    // and what does not fit without it is refused as before
    fake.device_bytes = fake.device_held + MB;
    EXPECT(st_update_mesh_bvh(ctx, &b.mesh, ST_BVH_LBVH30) == ST_ERR_OUT_OF_MEMORY);
    fake.device_bytes = all;
    EXPECT(st_update_mesh_bvh(ctx, &b.mesh, ST_BVH_LBVH30) == ST_OK);
    return 0;
}

// What a TLAS update page-locks is what it writes there: not the tree's arrays where the host wants none,
// or gets them by copies.
static int update_staging(st_ctx *ctx) {
    for (u32 n : {700u, 40000u}) {
        SceneArrays a(n, 0);
        EXPECT(st_upload_scene(ctx, 0, &a.scene) == ST_OK);
        EXPECT(st_upload_scene_bvh(ctx, 0, &a.scene) == ST_OK);
        size_t before = fake.host_bytes;
        EXPECT(st_update_scene_bvh(ctx, 0, nullptr, ST_BVH_REFIT) == ST_OK);
        EXPECT(st_update_scene_bvh(ctx, 0, nullptr, ST_BVH_LBVH30) == ST_OK);
        EXPECT(fake.host_bytes - before <= 4096);
        EXPECT(st_upload_scene_bvh(ctx, 0, &a.scene) == ST_OK);
        before = fake.host_bytes;
        EXPECT(st_update_scene_bvh(ctx, 0, &a.scene, ST_BVH_REFIT) == ST_OK);
        EXPECT(n <= 16384 || fake.host_bytes - before <= 4096);
        EXPECT(a.scene.bvh.node_count == 3);
        EXPECT(st_free_scene(ctx, 0) == ST_OK);
    }
    return 0;
}

// Serving that cannot start leaves nothing but its scene's spare arrays, which go with the scene, and starts
// once there is room.
static int refused_serving(st_ctx *ctx) {
    const size_t all = fake.device_bytes, empty = fake.device_held, MB = (size_t)1 << 20;
    const int streams = fake.streams;
    for (size_t room : {0 * MB, 1 * MB, 3 * MB, 9 * MB, 19 * MB, 50 * MB}) {     // (three spares take 14 MB)
        SceneArrays a(20000, 0);
        EXPECT(st_upload_scene(ctx, 0, &a.scene) == ST_OK);
        EXPECT(st_upload_scene_bvh(ctx, 0, &a.scene) == ST_OK);
        st_serve_config cfg = {};
        cfg.frame_budget = MB;
        fake.device_bytes = fake.device_held + room;
        fake.no_threads = room == 19 * MB;
        EXPECT(st_serve_start(ctx, &cfg) == (room == 50 * MB ? ST_OK : ST_ERR_OUT_OF_MEMORY));
        fake.device_bytes = all;
        fake.no_threads = false;
        if (room == 50 * MB) {
            EXPECT(st_serve_start(ctx, &cfg) == ST_ERR_INVALID_ARG);
            EXPECT(st_serve_stop(ctx) == ST_OK);
        }
        EXPECT(fake.streams == streams);
        EXPECT(st_free_scene(ctx, 0) == ST_OK);
        EXPECT(fake.device_held == empty);
    }
    return 0;
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    st_ctx *ctx = nullptr;
    int r = 2;
    if (what == "budget") return budget();
    EXPECT(st_init(&ctx, nullptr) == ST_OK);
    if (what == "refused_launch") r = refused_launch(ctx, argv[2], argv[3]);
    else if (what == "refused_allocation") r = refused_allocation(ctx);
    else if (what == "oversized_trees") r = oversized_trees(ctx);
    else if (what == "kept_memory") r = kept_memory(ctx);
    else if (what == "update_staging") r = update_staging(ctx);
    else if (what == "refused_serving") r = refused_serving(ctx);
    else printf("no such scenario\n");
    st_shutdown(ctx);
    return r;
}
