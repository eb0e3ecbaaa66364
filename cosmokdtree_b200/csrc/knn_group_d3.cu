// knn_group_d3.cu -- the kNN kernel with a group of lanes per query, d = 3.
#include "ckd_knn_group.cuh"

namespace ckd {
CKD_KNN_GROUP(3)
}  // namespace ckd
