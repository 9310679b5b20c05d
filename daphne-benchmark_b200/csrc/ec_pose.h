// Box yaw of a cluster's bounding box (host code, ec_pose.cpp).
#pragma once

namespace ec {
// xyz: the cluster's n points (3 floats each); min_x / min_y: their smallest
// x and y.  Writes the z and w of the yaw quaternion (x = y = 0).
void box_yaw(const float *xyz, int n, float min_x, float min_y, double *qz, double *qw);

// Many clusters at once, spread over up to kYawThreads host threads.
constexpr int kYawThreads = 8;
struct YawJob {
    const float *xyz;
    int n;
    float min_x, min_y;
    double *qz, *qw;
};
void box_yaws(const YawJob *jobs, int count);

// One cluster of the segmentation: the n points idx[] of xyz are written to out
// in that order, with their centroid and, where the reference keeps one
// (clusterAndColor, kernel.cpp:652-765), their box: position, orientation
// (x, y, z, w) and dimensions.  Spread over the same host threads.
struct ClusterJob {
    const int *idx;
    int n;
    float *out;
    bool kept;
    double centroid[3];
    double box[10];
};
void finish_clusters(const float *xyz, ClusterJob *jobs, int count);
}  // namespace ec
